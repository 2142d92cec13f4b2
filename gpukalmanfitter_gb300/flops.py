"""Algorithmic FP64 operation counts of the fit, per counted event.

Of the fit kernels' formulation (csrc/kf_fit.cuh: covariance in the start
frame, leg transport as scalars or columns): one add, multiply, divide, square
root or transcendental call = 1 FLOP, a fused multiply-add = 2, as the kernel
executes them (DFMA, DMUL and DADD counters of batches with 1, 10 and 20
planes and with half the hits missing, solved for the events).  The kernel
reports, per track, the RK trials, the accepted RK steps and the measurement
states, so the FLOPs of a batch are

    F = trials*RK_TRIAL + steps*RK_STEP + states*FILTER + tracks*FIXED

with POLY_TRIAL/POLY_STEP in place of RK_TRIAL/RK_STEP in a uniform field.
The smoothed first state is a running sum inside FILTER.

The dense formulation of the reference (8x8 D*J per step, 8x8*8x6 and 6x8*8x6
per surface, dense 6x6 products in updater and smoother) would count about
8x more for the same events; DENSE_* give those figures for context.
"""
from __future__ import annotations

import numpy as np

# the fit kernels (what runs on the GPU)
RK_TRIAL = 225     # field map: two field points, k2..k4, error estimate
RK_STEP = 415      # field map: accepted step: field point, k1, three transport columns, motion, navigation
POLY_TRIAL = 4     # uniform field: y = h q/p B, h y, acceptance bound
POLY_STEP = 120    # uniform field: motion, five transport scalars, q/p column, navigation
FILTER = 712       # bound Jacobian, F <- J F, update of C0 and D, stepper update
FIXED = 1139       # start state on the perigee line, first state, transport to the line

# dense reference formulation, same events
DENSE_RK_TRIAL = 94
DENSE_RK_STEP = 1024 + 400 + 60
DENSE_FILTER = 768 + 96 + 576 + 864 + 432 + 300
DENSE_SMOOTH = 6 * 6 * 6 * 2 * 4 + 500
DENSE_FIXED = 2400


def batch_flops(n_trials, n_steps, n_meas, status, dense: bool = False,
                uniform: bool = False) -> float:
    """FP64 FLOPs of one fit of a batch from the kernel's per-track counters
    (uniform: the uniform-field step formulation)."""
    t = np.asarray(n_trials, dtype=np.float64).sum()
    s = np.asarray(n_steps, dtype=np.float64).sum()
    m = np.asarray(n_meas, dtype=np.float64)
    if dense:
        smooth = np.clip(m - 1, 0, None)[np.asarray(status) == 0].sum()
        return (t * DENSE_RK_TRIAL + s * DENSE_RK_STEP + m.sum() * DENSE_FILTER
                + smooth * DENSE_SMOOTH + len(m) * DENSE_FIXED)
    trial, step = (POLY_TRIAL, POLY_STEP) if uniform else (RK_TRIAL, RK_STEP)
    return t * trial + s * step + m.sum() * FILTER + len(m) * FIXED


def batch_bytes(n_tracks: int, n_surfaces: int) -> dict:
    """Algorithmic HBM bytes of one fit: inputs read once, outputs written
    once, the first state's record written and read back once."""
    inputs = n_tracks * (n_surfaces * 5 * 8 + 8 + 4 + 6 * 8 + 21 * 8 + 3 * 8)
    outputs = n_tracks * (6 * 8 + 21 * 8 + 8 + 4 * 4)
    workspace = 2 * n_tracks * 35 * 8  # the first state's record (x, F, trigonometry)
    return {"inputs": inputs, "outputs": outputs, "workspace": workspace,
            "total": inputs + outputs + workspace}
