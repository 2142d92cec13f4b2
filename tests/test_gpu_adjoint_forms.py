"""The two kernels of the chi2 adjoint against each other: the one for a field
along z (adjointZ) and the general one (adjointKernel), which serves a field in
any other direction and the tracks whose tape runs over its capacity.  Both
differentiate the same function; they agree to rounding."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEYS = ("chi2", "grad_start", "grad_align", "grad_field_scale", "chi2_total", "grad_field_scale_track")


def _run(kf, tel, tilt=0.0, **opt):
    plain = tel.field

    def field(grid_ptr=None, scale=1.0):
        f = plain(grid_ptr, scale)
        f.value[0] = tilt * kf.TESLA
        return f

    b = kf.AdjointBatch(tel, kf.default_config(overstep_limit=0.1, **opt))
    tel.field = field
    try:
        return b.run(grad=True)
    finally:
        tel.field = plain


def _agree(a, b):
    assert np.array_equal(a["status"], b["status"]) and np.mean(a["status"] == 0) > 0.9
    for k in KEYS:
        # one step's acceptance, or a constraint that ties with another, may
        # fall the other way: a few tracks in a thousand
        x, y = a[k], b[k]
        if k in ("grad_align", "grad_field_scale", "chi2_total"):
            assert np.linalg.norm(x - y) <= 1e-6 * np.linalg.norm(y), k
        else:
            scale = np.maximum(np.abs(y), np.sqrt(np.mean(y * y, axis=-1, keepdims=True)))
            rel = np.abs(x - y) / np.maximum(scale, 1e-300)
            assert np.quantile(rel, 0.995) < 1e-8, (k, np.sort(rel.ravel())[-8:])


@pytest.mark.parametrize("kw", [dict(n_planes=20, x_first=50., x_step=50., mis_shift=0.1, mis_rot=1e-3),
                                dict(n_planes=12, x_first=40., x_step=40., min_len=3, max_len=12,
                                     hit_prob=0.8, outlier_prob=0.05, p_min=0.4, p_max=2.0),
                                dict(n_planes=1), dict(n_planes=10, bz_tesla=-1.0)])
@pytest.mark.parametrize("n", [1, 33, 700])
def test_kernels_agree(kf, kw, n):
    tel = kf.make_telescope(n, seed=61 + n, **kw)
    cut = dict(outlier_chi2_cut=25.0) if "outlier_prob" in kw else {}
    _agree(_run(kf, tel, **cut), _run(kf, tel, tilt=1e-13, **cut))


def test_tape_overflow_falls_back(kf):
    """64 planes: the segment mode's tape (3072 words) cannot hold the tracks."""
    tel = kf.make_telescope(300, seed=71, n_planes=64, x_first=15., x_step=15.)
    _agree(_run(kf, tel, adjoint_tape=1), _run(kf, tel, adjoint_tape=0))
