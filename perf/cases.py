"""The workloads whose speed is measured, through the package's public entry points.

listed() and draw() give cases (dicts of plain values); prepare() makes a case's
inputs on the GPU (or on the host, where the entry point takes host arrays) and
the batch or plan a program keeps; run() is one pass; work() the bytes and
operations a pass cannot do without; exact() the same results from a plain torch
restatement of the fit in 64 bits.

Every case is a batch of simulated tracks in a telescope of planes, as the
benchmark and the tests make them:

  uniform   planes over 1 m, uniform 2 T, a hit on every plane
  holes     planes over 1.5 m, uniform 2 T, uneven lengths, holes, outliers and
            an outlier cut
  map       planes over 1.5 m in a trilinear field map of 101^3 points
  material  planes over 1 m with 0.5 mm of silicon each: energy loss and scattering
  align     planes over 1 m, truth planes misaligned (the alignment's workload)
"""
from __future__ import annotations

import math

import numpy as np
import torch

import gpukalmanfitter_gb300 as kf

OVERSTEP = 0.1   # mm; with the default 0.01 mm a quarter of these tracks skip planes
MUON = 105.6583755e-3
SILICON_MM = 0.5


def _case(name, form, telescope, n, planes, mixed=False, smoothed=False):
    return {"name": name, "form": form, "telescope": telescope, "n": n, "planes": planes,
            "mixed": mixed, "smoothed": smoothed}


def listed():
    return [
        # a handful of tracks, as an interactive check or one event's few candidates
        _case("plain_5_uniform10", "plain", "uniform", 5, 10),
        # one event's worth of tracks in host memory, fitted and read back (the
        # reference driver's own 1000 tracks)
        _case("host_1000_uniform10", "host", "uniform", 1000, 10),
        # one event's worth in the field map, device resident, queue form, mixed precision
        _case("sorted_1000_map30_mixed", "sorted", "map", 1000, 30, mixed=True),
        # a large plain batch, one kernel launch (the reference's 1e5 tracks)
        _case("plain_100k_uniform10", "plain", "uniform", 100_000, 10),
        # the headline: a million tracks through a captured plan
        _case("plan_1M_uniform10", "plan", "uniform", 1_000_000, 10),
        # uneven tracks with holes and outliers, captured plan
        _case("plan_1M_holes30", "plan", "holes", 1_000_000, 30),
        # the same kind of tracks in a ragged middle-sized batch, mixed precision
        _case("sorted_65537_holes30_mixed", "sorted", "holes", 65_537, 30, mixed=True),
        # production precision mode: a million tracks in the field map, mixed
        _case("plan_1M_map30_mixed", "plan", "map", 1_000_000, 30, mixed=True),
        # FP64 in the field map, plain form, ragged size
        _case("plain_50021_map30", "plain", "map", 50_021, 30),
        # a tracker with material, queue form
        _case("sorted_100003_material10", "sorted", "material", 100_003, 10),
        # smoothed states of every measurement kept (alignment and residual studies)
        _case("plain_20011_holes30_smoothed", "plain", "holes", 20_011, 30, smoothed=True),
        # one gradient pass of the alignment: chi2 and its derivatives
        _case("adjoint_65536_align20", "adjoint", "align", 65_536, 20),
    ]


# telescope: planes (least, most), most tracks
_RANGE = {"uniform": (5, 20, 1_000_000), "holes": (15, 30, 1_000_000), "map": (10, 30, 600_000),
          "material": (5, 20, 300_000), "align": (10, 20, 65_536)}


def draw(rng):
    telescope = rng.choice(["uniform", "uniform", "holes", "holes", "map", "map", "material", "align"])
    low, high, most = _RANGE[telescope]
    planes = rng.randint(low, high)
    smoothed = False
    if telescope == "align":
        form, mixed = "adjoint", False
    else:
        form = rng.choice(["plain", "sorted", "plan", "host"])
        mixed = rng.random() < 0.4
        smoothed = form in ("plain", "sorted") and not mixed and rng.random() < 0.2
    if form == "host":
        most = 20_000
    if smoothed:
        most = 40_000
    least = 64 if form == "adjoint" else 1
    n = int(round(math.exp(rng.uniform(math.log(least), math.log(most)))))
    c = _case("", form, telescope, n, planes, mixed, smoothed)
    del c["name"]
    return c


def _telescope_args(case):
    p = case["planes"]
    t = case["telescope"]
    length = 1500.0 if t in ("holes", "map") else 1000.0
    kw = dict(n_planes=p, x_first=length / p, x_step=length / p)
    if t == "holes":
        kw.update(min_len=5, max_len=p, hit_prob=0.9, outlier_prob=0.02)
    elif t == "map":
        kw.update(field_map=True)
    elif t == "material":
        kw.update(material=SILICON_MM)
    elif t == "align":
        kw.update(mis_shift=0.1, mis_rot=1e-3)
    return kw


def _config_args(case):
    kw = dict(overstep_limit=OVERSTEP, precision=1 if case["mixed"] else 0)
    if case["telescope"] == "holes":
        kw.update(outlier_chi2_cut=25.0)
    elif case["telescope"] == "material":
        kw.update(material_effects=3)
    return kw


def _telescope(case, seed, device):
    return kf.make_telescope(case["n"], seed=1_000_003 + 7919 * seed, device=device,
                             **_telescope_args(case))


def prepare(case, seed):
    form = case["form"]
    cfg = kf.default_config(**_config_args(case))
    if form == "host":
        tel = _telescope(case, seed, None)
        size = kf.load().kf_host_staging_size(cfg, case["n"], case["planes"], 0)
        state = {"tel": tel, "cfg": cfg,
                 "staging": torch.empty(size, dtype=torch.uint8, device="cuda")}
        if tel.field_grid is not None:
            state["grid"] = torch.from_numpy(tel.field_grid).cuda()
        return {"form": form, **state}
    tel = _telescope(case, seed, "cuda")
    torch.cuda.synchronize()
    if form == "adjoint":
        return {"form": form, "batch": kf.AdjointBatch(tel, cfg)}
    batch = kf.DeviceBatch(tel, cfg, smoothed=case["smoothed"])
    state = {"form": form, "batch": batch}
    if form == "plan":
        stream = torch.cuda.Stream()
        batch.make_plan(stream)
        state["stream"] = stream
    return state


def run(state):
    form = state["form"]
    if form == "host":
        return kf.fit_host(state["tel"], state["cfg"], staging=state["staging"],
                           field_grid_dev=state.get("grid"))
    batch = state["batch"]
    if form == "adjoint":
        return batch.run(grad=True)
    if form == "plain":
        batch.fit()
    elif form == "sorted":
        batch.fit_sorted()
    else:
        batch.launch_plan(state["stream"])
    return batch.out


def work(case):
    """Bytes: every input read once, every output written once.  Operations: a
    track needs about 2.6 RK steps a plane (a step to the straight-line
    estimate and its corrections), a measurement update a hit, and its start
    and end on the perigee line."""
    n, p = case["n"], case["planes"]
    planes = 0.5 * (5 + p) if case["telescope"] == "holes" else p
    hits = planes * (0.9 if case["telescope"] == "holes" else 1.0)
    step = 500 if case["telescope"] == "map" else 120
    flops = 2.6 * planes * step + hits * 600 + 1000
    data = hits * 40 + 8 + 4 + 30 * 8 + 28 * 8 + 16
    if case["smoothed"]:
        data += hits * 27 * 8
        flops += hits * 250
    if case["telescope"] == "material":
        flops += hits * 500
    if case["form"] == "adjoint":
        # a reverse sweep costs about twice the forward evaluation
        flops = 3 * (flops + hits * 250)
        data = hits * 40 + 8 + 4 + 30 * 8 + 8 * 8 + 4
    extra = 101 ** 3 * 16 if case["telescope"] == "map" and n > 10_000 else 0
    return {"bytes": n * data + extra, "flops": n * flops}


# ---------------------------------------------------------------------------
# The fit in plain torch, 64 bits: a vector of tracks taken plane by plane.
# Reference algorithm: RK4 with step control (Propagator/EigenStepper.ipp),
# covariance transport (Propagator/detail/CovarianceEngine.hpp), gain-matrix
# filter and smoother (Fitter/GainMatrixUpdater.hpp, GainMatrixSmoother.hpp).
# ---------------------------------------------------------------------------
_TOL, _SURF = 1e-4, 1e-4
_BIG = 1.7976931348623157e308


def _cross(a, b):
    return torch.linalg.cross(a, b, dim=-1)


def _dot(a, b):
    return (a * b).sum(-1)


def _skew(B):
    """M with M v = v x B."""
    z = torch.zeros_like(B[:, 0])
    return torch.stack([torch.stack([z, B[:, 2], -B[:, 1]], -1),
                        torch.stack([-B[:, 2], z, B[:, 0]], -1),
                        torch.stack([B[:, 1], -B[:, 0], z], -1)], -2)


class _Fit:
    """One batch of tracks; every array has the track as its first axis."""

    def __init__(self, inp, opt, scale=None):
        self.i, self.o = inp, opt
        self.n = inp["start"].shape[1]
        self.dev = inp["start"].device
        self.scale = scale if scale is not None else torch.ones(self.n, dtype=torch.float64, device=self.dev)
        self.eye3 = torch.eye(3, dtype=torch.float64, device=self.dev)

    def field(self, pos):
        g = self.i.get("grid")
        if g is None:
            B = torch.zeros((self.n, 3), dtype=torch.float64, device=self.dev)
            B[:, 2] = self.i["bz"]
            return B * self.scale[:, None]
        m, half = g.shape[0], self.i["half"]
        u = (pos + half) * ((m - 1) / (2.0 * half))
        c = torch.clamp(torch.floor(u), 0, m - 2)
        f = u - c
        c = c.long()
        B = 0.0
        for dx in (0, 1):
            for dy in (0, 1):
                for dz in (0, 1):
                    w = ((f[:, 0] if dx else 1 - f[:, 0]) * (f[:, 1] if dy else 1 - f[:, 1])
                         * (f[:, 2] if dz else 1 - f[:, 2]))
                    B = B + w[:, None] * g[c[:, 2] + dz, c[:, 1] + dy, c[:, 0] + dx]
        return B * self.scale[:, None]

    def set_p(self, ip):
        """Constants of a leg from 1 / |p|."""
        self.ip = ip
        self.qop = self.q * ip
        x = MUON * ip
        self.dtds = torch.sqrt(1 + x * x)
        self.d37 = MUON * MUON * self.qop / self.dtds

    def step(self, todo, acc, other, backward):
        """One accepted RK step of the tracks `todo`; the step is the smaller
        (in size, of its direction) of the accuracy limit and `other`."""
        pos, d, q = self.pos, self.dir, self.qop[:, None]
        pick = torch.maximum if backward else torch.minimum
        one = torch.ones_like(acc)
        h = torch.where(todo, pick(acc, other), one)
        Bf = self.field(pos)
        k1 = q * _cross(d, Bf)
        for _ in range(100):
            H = h[:, None]
            Bm = self.field(pos + 0.5 * H * d + 0.125 * H * H * k1)
            k2 = q * _cross(d + 0.5 * H * k1, Bm)
            k3 = q * _cross(d + 0.5 * H * k2, Bm)
            Bl = self.field(pos + H * d + 0.5 * H * H * k3)
            k4 = q * _cross(d + H * k3, Bl)
            e = torch.clamp(h * h * (k1 - k2 - k3 + k4).abs().sum(-1), min=1e-20)
            bad = todo & (e > _TOL)
            if not bool(bad.any()):
                break
            s = torch.clamp(torch.pow(_TOL / (2 * e), 0.25), 0.25, 4.0)
            acc = torch.where(bad, h * s, acc)
            h = torch.where(bad, pick(acc, other), h)
        H, Q = h[:, None], q
        a1 = _cross(d, Bf)
        a2 = _cross(d + 0.5 * H * k1, Bm) + Q * 0.5 * H * _cross(a1, Bm)
        a3 = _cross(d + 0.5 * H * k2, Bm) + Q * 0.5 * H * _cross(a2, Bm)
        a4 = _cross(d + H * k3, Bl) + Q * H * _cross(a3, Bl)
        H3, Q3 = H[:, :, None], q[:, :, None]
        T1 = Q3 * _skew(Bf)
        T2 = Q3 * (_skew(Bm) @ (self.eye3 + 0.5 * H3 * T1))
        T3 = Q3 * (_skew(Bm) @ (self.eye3 + 0.5 * H3 * T2))
        T4 = Q3 * (_skew(Bl) @ (self.eye3 + H3 * T3))
        DA = H3 * (self.eye3 + H3 / 6 * (T1 + T2 + T3))
        DB = self.eye3 + H3 / 6 * (T1 + 2 * (T2 + T3) + T4)
        Da = H * H / 6 * (a1 + a2 + a3)
        Dc = H / 6 * (a1 + 2 * (a2 + a3) + a4)
        t1, t2, t3 = todo, todo[:, None], todo[:, None, None]
        Zq = self.Zq[:, None, :]
        Zp = self.Zp + DA @ self.Zd + Da[:, :, None] * Zq
        Zd = DB @ self.Zd + Dc[:, :, None] * Zq
        self.Zt = torch.where(t2, self.Zt + (h * self.d37)[:, None] * self.Zq, self.Zt)
        self.Zp, self.Zd = torch.where(t3, Zp, self.Zp), torch.where(t3, Zd, self.Zd)
        np_ = pos + H * d + H * H / 6 * (k1 + k2 + k3)
        nd = d + H / 6 * (k1 + 2 * (k2 + k3) + k4)
        nd = nd / torch.sqrt(_dot(nd, nd))[:, None]
        self.pos, self.dir = torch.where(t2, np_, pos), torch.where(t2, nd, d)
        self.k4 = torch.where(t2, k4, self.k4)
        self.t = torch.where(t1, self.t + h * self.dtds, self.t)
        self.stepped = self.stepped | todo
        return acc

    def trig(self):
        d = self.dir
        s = torch.sqrt(d[:, 0] ** 2 + d[:, 1] ** 2)
        return d[:, 2], s, d[:, 0] / s, d[:, 1] / s

    def direction_columns(self):
        c, s, cp, sp = self.trig()
        z = torch.zeros_like(c)
        return torch.stack([-s * sp, s * cp, z], -1), torch.stack([c * cp, c * sp, -s], -1)

    def reset_plane(self, who, U, V):
        """Jacobian of the free state by bound parameters on a plane."""
        n = self.n
        z = torch.zeros((n, 6), dtype=torch.float64, device=self.dev)
        z3 = torch.zeros((n, 3), dtype=torch.float64, device=self.dev)
        ph, th = self.direction_columns()
        Zp = torch.stack([U.expand(n, 3), V.expand(n, 3), z3, z3, z3, z3], -1)
        Zd = torch.stack([z3, z3, ph, th, z3, z3], -1)
        Zq, Zt = z.clone(), z.clone()
        Zq[:, 4] = 1.0
        Zt[:, 5] = 1.0
        w2, w3 = who[:, None], who[:, None, None]
        self.Zp, self.Zd = torch.where(w3, Zp, self.Zp), torch.where(w3, Zd, self.Zd)
        self.Zq, self.Zt = torch.where(w2, Zq, self.Zq), torch.where(w2, Zt, self.Zt)
        self.k4 = torch.where(w2, torch.zeros_like(self.k4), self.k4)
        self.stepped = self.stepped & ~who

    def project(self, s, ax0, ax1):
        """Bound-to-bound Jacobian at a surface; s: path correction by parameter."""
        on = self.stepped.to(torch.float64)[:, None]
        Zp = self.Zp - (self.dir * on)[:, :, None] * s[:, None, :]
        Zd = self.Zd - (self.k4 * on)[:, :, None] * s[:, None, :]
        Zt = self.Zt - (self.dtds[:, None] * on) * s
        c, sn, cp, sp = self.trig()
        z = torch.zeros_like(c)
        f = torch.stack([-sp / sn, cp / sn, z], -1)
        g = torch.stack([cp * c, sp * c, -sn], -1)
        return torch.stack([(ax0[:, :, None] * Zp).sum(1), (ax1[:, :, None] * Zp).sum(1),
                            (f[:, :, None] * Zd).sum(1), (g[:, :, None] * Zd).sum(1),
                            self.Zq, Zt], 1)

    def update(self, who, x, U, V, c):
        """Free state from bound parameters on a plane."""
        pos = c + x[:, 0:1] * U + x[:, 1:2] * V
        sp, cp, st, ct = torch.sin(x[:, 2]), torch.cos(x[:, 2]), torch.sin(x[:, 3]), torch.cos(x[:, 3])
        d = torch.stack([cp * st, sp * st, ct], -1)
        self.pos = torch.where(who[:, None], pos, self.pos)
        self.dir = torch.where(who[:, None], d, self.dir)
        self.t = torch.where(who, x[:, 5], self.t)
        self.set_p(torch.where(who, x[:, 4].abs(), self.ip))

    def start(self):
        i, n = self.i, self.n
        s = i["start"].T
        self.q = torch.where(s[:, 4] > 0, 1.0, -1.0).to(torch.float64)
        st, ct = torch.sin(s[:, 3]), torch.cos(s[:, 3])
        sp, cp = torch.sin(s[:, 2]), torch.cos(s[:, 2])
        self.dir = torch.stack([cp * st, sp * st, ct], -1)
        z = torch.zeros(n, dtype=torch.float64, device=self.dev)
        X = torch.stack([-sp, cp, z], -1)
        per = i["perigee"].T
        Y = torch.stack([z, z, z + 1], -1)
        self.pos = per + s[:, 0:1] * X + s[:, 1:2] * Y
        self.t = s[:, 5]
        self.set_p(s[:, 4].abs())
        self.k4 = torch.zeros((n, 3), dtype=torch.float64, device=self.dev)
        self.stepped = torch.zeros(n, dtype=torch.bool, device=self.dev)
        ph, th = self.direction_columns()
        D = _cross(X, Y)
        ipdn = 1.0 / _dot(self.dir, D)
        cols = []
        for col in (ph, th):
            w = _cross(Y, col)
            w = w - _dot(X, w)[:, None] * X
            cols.append(w * (s[:, 0] * ipdn)[:, None])
        z3 = torch.zeros_like(X)
        self.Zp = torch.stack([X, Y, cols[0], cols[1], z3, z3], -1)
        self.Zd = torch.stack([z3, z3, ph, th, z3, z3], -1)
        self.Zq = torch.zeros((n, 6), dtype=torch.float64, device=self.dev)
        self.Zt = self.Zq.clone()
        self.Zq[:, 4] = 1.0
        self.Zt[:, 5] = 1.0
        iu = torch.triu_indices(6, 6, device=self.dev)
        C = torch.zeros((n, 6, 6), dtype=torch.float64, device=self.dev)
        C[:, iu[0], iu[1]] = i["scov"].T
        C[:, iu[1], iu[0]] = i["scov"].T
        self.C = C

    def material(self, who, T):
        """Energy loss and scattering after an update (Material/detail/Interactions.ipp)."""
        t0, X0, _, _, Z, rho = self.i["material"]
        m, me = MUON, 0.5109989461e-3
        d, p = self.dir, 1.0 / self.ip
        pc = 1.0 / _dot(d, T.expand(self.n, 3)).abs()
        mop = m * self.ip
        beta2 = 1.0 / (1.0 + mop * mop)
        bg = 1.0 / mop
        gamma = torch.sqrt(1 + bg * bg)
        q2b = 1.0 + mop * mop
        Ne, I = Z * rho, 16e-9 * Z ** float(np.float32(0.9))
        eps = 0.5 * (0.307075e-3 * 100.0) * Ne * t0 * pc * q2b
        dh = torch.log(bg) + math.log(28.816e-9 * math.sqrt(Ne) / I) - 0.5
        dh = torch.where(bg < 10.0, torch.zeros_like(dh), dh)
        u = 2 * me * bg * bg
        mf = me / m
        wmax = u / (1.0 + 2 * gamma * mf + mf * mf)
        loss = eps * (0.5 * torch.log(u / I) + 0.5 * torch.log(wmax / I) - beta2 - dh)
        sq = torch.sqrt(q2b) * self.ip * self.ip * (4 * eps / (2 * math.sqrt(2 * math.log(2.0))))
        t = torch.sqrt(t0 / X0 * pc * q2b)
        th0 = 13.6e-3 * self.ip * t * (1.0 + float(np.float32(0.038)) * 2 * torch.log(t))
        sphi = th0 / torch.sqrt(d[:, 0] ** 2 + d[:, 1] ** 2)
        E = torch.sqrt(m * m + p * p) - loss
        pn = torch.sqrt(torch.clamp(E * E - m * m, min=1e-30))
        self.set_p(torch.where(who, 1.0 / pn, self.ip))
        add = torch.zeros((self.n, 6), dtype=torch.float64, device=self.dev)
        add[:, 2], add[:, 3], add[:, 4] = sphi * sphi, th0 * th0, sq * sq
        self.C = self.C + torch.diag_embed(add * who[:, None])

    def forward(self, planes):
        """planes: (centre, U, V, T) per plane.  Filters every track; keeps each
        plane's state: who has one, predicted and filtered parameters and
        covariances, Jacobian from the state before, outlier."""
        i, o, n = self.i, self.o, self.n
        S = len(planes)
        bits = torch.stack([((i["mask"] >> k) & 1).bool() & (i["nplanes"] > k) for k in range(S)])
        hits = bits.sum(0)
        self.hits = hits
        self.start()
        acc = torch.full((n,), _BIG, dtype=torch.float64, device=self.dev)
        self.chi2 = torch.zeros(n, dtype=torch.float64, device=self.dev)
        seen = torch.zeros_like(hits)
        self.states = []
        noise = i.get("material") is not None
        for k, (c, U, V, T) in enumerate(planes):
            live = (i["nplanes"] > k) & (seen < hits)
            on = torch.zeros_like(live)
            go = live.clone()

            def distance():
                den = (self.dir * T).sum(-1)
                path = ((c - self.pos) * T).sum(-1) / den
                return path

            path = distance()
            go = go & (path > -OVERSTEP)
            for _ in range(300):
                if not bool(go.any()):
                    break
                acc = self.step(go, acc, path, False)
                path = distance()
                here = go & (path * path < _SURF * _SURF)
                on = on | here
                go = go & ~here & (path > -OVERSTEP)
            who = on & bits[k]
            if not bool(who.any()):
                self.states.append(None)
                continue
            s = ((T / _dot(self.dir, T.expand(n, 3))[:, None])[:, :, None] * self.Zp).sum(1)
            J = self.project(s, U.expand(n, 3), V.expand(n, 3))
            w3 = who[:, None, None]
            Cp = J @ self.C @ J.transpose(1, 2)
            rel = self.pos - c
            pred = torch.stack([(rel * U).sum(-1), (rel * V).sum(-1),
                                torch.atan2(self.dir[:, 1], self.dir[:, 0]),
                                torch.atan2(torch.sqrt(self.dir[:, 0] ** 2 + self.dir[:, 1] ** 2),
                                            self.dir[:, 2]), self.qop, self.t], -1)
            self.reset_plane(who, U, V)
            m = i["meas"][k]
            # tracks without a hit here hold no numbers: harmless ones in their place
            r = torch.where(who[:, None], m[:2].T - pred[:, :2], torch.zeros_like(pred[:, :2]))
            v = [torch.where(who, m[2 + e], torch.full_like(m[2], (1.0, 0.0, 1.0)[e])) for e in range(3)]
            Vm = torch.stack([torch.stack([v[0], v[1]], -1), torch.stack([v[1], v[2]], -1)], -2)
            Sm = Cp[:, :2, :2] + Vm
            det = Sm[:, 0, 0] * Sm[:, 1, 1] - Sm[:, 0, 1] * Sm[:, 1, 0]
            Si = torch.stack([torch.stack([Sm[:, 1, 1], -Sm[:, 0, 1]], -1),
                              torch.stack([-Sm[:, 1, 0], Sm[:, 0, 0]], -1)], -2) / det[:, None, None]
            chi2 = _dot(r, (Si @ r[:, :, None])[:, :, 0])
            out = torch.zeros_like(who)
            if o["cut"] > 0:
                out = who & (chi2 > o["cut"])
            upd = who & ~out
            K = Cp[:, :, :2] @ Si
            filt = torch.where(upd[:, None], pred + (K @ r[:, :, None])[:, :, 0], pred)
            Cf = torch.where(upd[:, None, None], Cp - K @ Cp[:, :2, :], Cp)
            self.chi2 = torch.where(upd, self.chi2 + chi2, self.chi2)
            self.C = torch.where(w3, Cf, self.C)
            self.update(upd, filt, U, V, c)
            st = {"who": who, "out": out, "xp": pred, "xf": filt, "J": J, "r": m, "V": v, "no": seen.clone()}
            if noise:
                st.update(Cp=Cp, Cf=Cf)
                self.material(who, T)
            st["C"] = Cf if noise or o["keep"] else None
            self.states.append(st)
            seen = seen + who.to(seen.dtype)
        self.seen = seen
        self.last = self.C

    def smooth(self, planes, each=None):
        """Smoothed states, last first; each(k, state, x, C) sees every one."""
        n = self.n
        x = C = None
        later = None
        for k in range(len(planes) - 1, -1, -1):
            st = self.states[k]
            if st is None:
                continue
            who = st["who"]
            last = st["no"] == self.seen - 1
            noise = "Cp" in st
            if x is None:
                x, C = st["xf"], (st["Cf"] if noise else self.last)
                later = {m: st[m] for m in ("xp", "J", "Cp") if m in st}
                started = who & last
            else:
                J = later["J"]
                if noise:
                    # scaled to a unit diagonal: the variances span fourteen orders
                    w = later["Cp"].diagonal(dim1=1, dim2=2).rsqrt()
                    A = later["Cp"] * w[:, :, None] * w[:, None, :]
                    G = (torch.linalg.solve(A, w[:, :, None] * (J @ st["Cf"])) * w[:, :, None]).transpose(1, 2)
                    Cn = st["Cf"] - G @ (later["Cp"] - C) @ G.transpose(1, 2)
                else:
                    G = torch.linalg.inv(torch.where(started[:, None, None], J, torch.eye(6, dtype=J.dtype, device=self.dev)))
                    Cn = G @ C @ G.transpose(1, 2)
                xn = st["xf"] + (G @ (x - later["xp"])[:, :, None])[:, :, 0]
                go = who & started
                new = who & last
                first = st["Cf"] if noise else self.last
                x = torch.where(go[:, None], xn, torch.where(new[:, None], st["xf"], x))
                C = torch.where(go[:, None, None], Cn, torch.where(new[:, None, None], first, C))
                for m in list(later):
                    w = who.view([n] + [1] * (later[m].dim() - 1))
                    later[m] = torch.where(w, st[m], later[m])
                started = started | new
            if each is not None:
                each(k, st, x, C)
        return x, C

    def backward(self, planes, x, C):
        """From the smoothed first state back to the perigee line."""
        n = self.n
        ok = self.seen > 0
        first = torch.zeros(n, dtype=torch.long, device=self.dev)
        for k in range(len(planes) - 1, -1, -1):
            if self.states[k] is not None:
                first = torch.where(self.states[k]["who"], torch.full_like(first, k), first)
        c, U, V, _ = (torch.stack([p[e] for p in planes])[first] for e in range(4))
        self.update(ok, x, U, V, c)
        self.C = C
        per = self.i["perigee"].T
        acc = torch.full((n,), -_BIG, dtype=torch.float64, device=self.dev)
        best = torch.full((n,), -_BIG, dtype=torch.float64, device=self.dev)
        go = ok.clone()
        for _ in range(300):
            ea, m = -self.dir, per - self.pos
            den = 1 - ea[:, 2] ** 2
            u = (_dot(m, ea) - m[:, 2] * ea[:, 2]) / den
            go = go & ~(u * u < _SURF * _SURF)
            if not bool(go.any()):
                break
            best = torch.where(go & (u.abs() < best.abs()), -u, best)
            acc = self.step(go, acc, best, True)
        d = self.dir
        z = torch.zeros(n, dtype=torch.float64, device=self.dev)
        Y = torch.stack([z, z, z + 1], -1)
        X = _cross(Y, d)
        X = X / torch.sqrt(_dot(X, X))[:, None]
        pc = self.pos - per
        lc = d[:, 2]
        nv = d - lc[:, None] * Y
        nrm = 1.0 / (1.0 - lc * lc)
        sk = (nv[:, :, None] * self.Zp).sum(1)
        row = (pc[:, :, None] * (Y[:, :, None] * sk[:, None, :] - self.Zd)).sum(1)
        J = self.project(nrm[:, None] * (sk - row), X, Y)
        Cl = J @ self.C @ J.transpose(1, 2)
        sign = torch.where(-d[:, 1] * pc[:, 0] + d[:, 0] * pc[:, 1] < 0, -1.0, 1.0)
        r = torch.sqrt(pc[:, 0] ** 2 + pc[:, 1] ** 2)
        par = torch.stack([r * sign, pc[:, 2], torch.atan2(d[:, 1], d[:, 0]),
                           torch.atan2(torch.sqrt(d[:, 0] ** 2 + d[:, 1] ** 2), d[:, 2]),
                           self.qop, self.t], 0)
        iu = torch.triu_indices(6, 6, device=self.dev)
        cov = Cl[:, iu[0], iu[1]].T
        return par * ok, cov * ok


def _inputs(case, seed, dev):
    """The case's inputs as torch tensors (the same numbers run() is given)."""
    tel = _telescope(case, seed, "cuda" if dev == "cuda" and case["form"] != "host" else None)
    t = lambda a: a if isinstance(a, torch.Tensor) else torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    mask = tel.hit_mask
    mask = mask if isinstance(mask, torch.Tensor) else torch.from_numpy(mask.view(np.int64)).to(dev)
    inp = {"meas": t(tel.meas), "mask": mask, "nplanes": t(tel.n_planes).long(), "start": t(tel.start),
           "scov": t(tel.start_cov), "perigee": t(tel.perigee),
           "bz": 2.0 * 0.000299792458}
    if case["telescope"] == "map":
        m = tel.field_n
        inp["grid"] = t(tel.field_grid).reshape(m, m, m, 4)[..., :3].double()
        inp["half"] = tel.field_half
    if case["telescope"] == "material":
        inp["material"] = [float(v) for v in tel.material[0]]
    c = torch.from_numpy(np.array(tel.center, dtype=np.float64)).to(dev)
    r = torch.from_numpy(np.array(tel.rotation, dtype=np.float64)).to(dev).reshape(-1, 3, 3)
    return inp, c, r


def _part(inp, lo, hi):
    cut = {"meas": inp["meas"][:, :, lo:hi], "mask": inp["mask"][lo:hi], "nplanes": inp["nplanes"][lo:hi],
           "start": inp["start"][:, lo:hi], "scov": inp["scov"][:, lo:hi], "perigee": inp["perigee"][:, lo:hi]}
    return {**inp, **cut}


def _exact_fit(case, seed, dev):
    inp, c, r = _inputs(case, seed, dev)
    n, S = case["n"], case["planes"]
    planes = [(c[k], r[k, :, 0], r[k, :, 1], r[k, :, 2]) for k in range(S)]
    opt = {"cut": _config_args(case).get("outlier_chi2_cut", 0.0), "keep": case["smoothed"]}
    out = {"params": torch.zeros((6, n), dtype=torch.float64, device=dev),
           "cov": torch.zeros((21, n), dtype=torch.float64, device=dev),
           "chi2": torch.zeros(n, dtype=torch.float64, device=dev)}
    if case["smoothed"]:
        out["smoothed"] = torch.zeros((S, 27, n), dtype=torch.float64, device=dev)
    for lo in range(0, n, 250_000):
        hi = min(n, lo + 250_000)
        f = _Fit(_part(inp, lo, hi), opt)
        f.forward(planes)
        each = None
        if case["smoothed"]:
            iu = torch.triu_indices(6, 6, device=dev)

            def each(k, st, x, C):
                at = st["who"].nonzero()[:, 0]
                out["smoothed"][st["no"][at], :6, lo + at] = x[at]
                out["smoothed"][st["no"][at], 6:, lo + at] = C[at][:, iu[0], iu[1]]

        x, C = f.smooth(planes, each)
        chi2 = f.chi2
        par, cov = f.backward(planes, x, C)
        out["params"][:, lo:hi], out["cov"][:, lo:hi], out["chi2"][lo:hi] = par, cov, chi2
    return out


def _exact_adjoint(case, seed, dev):
    """Total smoothed chi2 and its derivatives, by autograd of the fit above."""
    inp, c, r = _inputs(case, seed, dev)
    n, S = case["n"], case["planes"]
    opt = {"cut": 0.0, "keep": False}
    out = {"chi2": torch.zeros(n, dtype=torch.float64, device=dev),
           "grad_start": torch.zeros((6, n), dtype=torch.float64, device=dev),
           "grad_align": torch.zeros((S, 6), dtype=torch.float64, device=dev),
           "grad_field_scale_track": torch.zeros(n, dtype=torch.float64, device=dev)}
    for lo in range(0, n, 16_384):
        hi = min(n, lo + 16_384)
        part = _part(inp, lo, hi)
        start = part["start"].clone().requires_grad_()
        scale = torch.ones(hi - lo, dtype=torch.float64, device=dev, requires_grad=True)
        a = torch.zeros((S, 6), dtype=torch.float64, device=dev, requires_grad=True)
        part["start"] = start
        planes = []
        for k in range(S):
            w = a[k, 3:]
            axes = [r[k, :, e] + torch.linalg.cross(w, r[k, :, e]) for e in range(3)]
            planes.append((c[k] + a[k, :3], *axes))
        f = _Fit(part, opt, scale)
        f.forward(planes)
        terms = []

        def each(k, st, x, C):
            m, (v0, v1, v2) = st["r"], st["V"]
            r0 = torch.where(st["who"], m[0] - x[:, 0], torch.zeros_like(x[:, 0]))
            r1 = torch.where(st["who"], m[1] - x[:, 1], torch.zeros_like(x[:, 0]))
            det = v0 * v2 - v1 * v1
            terms.append(torch.where(st["who"], (r0 * (v2 * r0 - v1 * r1) + r1 * (v0 * r1 - v1 * r0)) / det,
                                     torch.zeros_like(r0)))

        f.smooth(planes, each)
        chi2 = torch.stack(terms).sum(0)
        chi2.sum().backward()
        out["chi2"][lo:hi] = chi2.detach()
        out["grad_start"][:, lo:hi] = start.grad
        out["grad_align"] += a.grad
        out["grad_field_scale_track"][lo:hi] = scale.grad
    out["grad_field_scale"] = out["grad_field_scale_track"].sum().reshape(1)
    out["chi2_total"] = out["chi2"].sum().reshape(1)
    return out


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if case["form"] == "adjoint":
        return _exact_adjoint(case, seed, dev)
    with torch.no_grad():
        return _exact_fit(case, seed, dev)
