"""The FP64 fit kernels' branches that the workloads of the parity tests do
not reach, against the precise oracle at the same 1e-9 bar: a uniform field
off the z axis (the fit's own frame), along -z, absent; low momenta (rejected
steps, large turning angles); a start covariance that correlates the time with
the other parameters; the Jacobian rebuilt after each update; all of them with
smoothed states; in the field map too."""
import numpy as np
import pytest

from conftest import parity_report

pytestmark = pytest.mark.gpu

TOL = 1e-9
DIAG = [0, 6, 11, 15, 18, 20]


def _with_field(tel, tesla, kf):
    """The telescope with a uniform fit field of the given components."""
    plain = tel.field

    def field(grid_ptr=None, scale=1.0):
        f = plain(grid_ptr, scale)
        for a in range(3):
            f.value[a] = tesla[a] * kf.TESLA
        return f

    tel.field = field
    return tel


def _correlate_time(tel):
    """Correlation 0.3 ... 0.5 of the start time with every other parameter
    (and of the first two with each other): positive definite."""
    sig = np.sqrt(tel.start_cov[DIAG])
    row = {0: 5, 1: 10, 2: 14, 3: 17, 4: 19}  # (i, 5) in the upper triangle
    for i, e in row.items():
        tel.start_cov[e] = (0.3 + 0.05 * i) * (-1) ** i * sig[i] * sig[5]
    tel.start_cov[1] = 0.2 * sig[0] * sig[1]
    return tel


def _check(kf, orc, tel, smoothed=False, **opt):
    cfg = kf.default_config(overstep_limit=0.1, **opt)
    o = orc.fit(tel, cfg, threads=0, smoothed=smoothed, variant="precise")
    b = kf.DeviceBatch(tel, cfg, smoothed=smoothed)
    ok = o["status"] == 0
    assert ok.mean() > 0.5
    for form in ("plain", "sorted"):
        b.fit() if form == "plain" else b.fit_sorted()
        g = b.results()
        for k in ("status", "n_meas", "n_steps", "n_trials"):
            assert np.array_equal(g[k], o[k]), (form, k)
        rep = parity_report(g, o, TOL, mask=ok)
        print(form, rep)
        assert rep["params"] <= 1 and rep["chi2"] <= 1 and rep["cov"] <= 1, (form, rep)
        if not smoothed:
            continue
        for s in range(tel.n_surfaces):
            at = ok & (o["n_meas"] > s)
            if not at.any():
                continue
            so, sg = o["smoothed"][s][:, at], g["smoothed"][s][:, at]
            sig = np.sqrt(so[6 + np.array(DIAG)])
            assert np.max(np.abs(sg[:6] - so[:6]) / np.maximum(np.abs(so[:6]), sig)) < TOL, (form, s)
            assert np.max(np.abs(sg[6 + np.array(DIAG)] / so[6 + np.array(DIAG)] - 1)) < TOL, (form, s)


@pytest.mark.parametrize("tesla", [(0.03, 0.05, 0.19), (0.1, 0., 0.), (0., -0.05, -0.18), (0., 0., 0.)])
@pytest.mark.parametrize("smoothed", [False, True])
def test_field_off_axis(kf, orc, tesla, smoothed):
    tel = _with_field(kf.make_telescope(777, seed=31, n_planes=12, bz_tesla=0.2), tesla, kf)
    _check(kf, orc, tel, smoothed)


@pytest.mark.parametrize("kw", [dict(bz_tesla=-2.0), dict(p_min=0.25, p_max=0.8, n_planes=8, x_first=30., x_step=30.),
                                dict(n_planes=1), dict(n_planes=64, x_first=12., x_step=12.)])
def test_uniform_field_ranges(kf, orc, kw):
    _check(kf, orc, kf.make_telescope(555, seed=32, **kw), smoothed=True)


@pytest.mark.parametrize("field_map", [False, True])
@pytest.mark.parametrize("faithful", [0, 1])
@pytest.mark.parametrize("smoothed", [False, True])
def test_time_correlated_start(kf, orc, field_map, faithful, smoothed):
    tel = kf.make_telescope(600, seed=33, n_planes=15, x_first=80., x_step=80., min_len=5, max_len=15,
                            hit_prob=0.9, outlier_prob=0.02, field_map=field_map)
    _check(kf, orc, _correlate_time(tel), smoothed, faithful_jacobian=faithful, outlier_chi2_cut=25.0)


@pytest.mark.parametrize("kw", [dict(tesla=(0.03, 0.05, 0.19)), dict(field_map=True), dict()])
def test_material_forms(kf, orc, kw):
    """Process noise (fixed-point smoother of the first state): parameters and
    chi2 at 1e-9, covariance at the 1e-8 of the material parity test."""
    tel = kf.make_telescope(400, seed=34, n_planes=10, material=0.5 if "field_map" not in kw else 0.,
                            field_map=kw.get("field_map", False),
                            **(dict(bz_tesla=0.2) if "tesla" in kw else {}))
    if "field_map" in kw:  # (the generator has no material truth in a map)
        tel.material = np.tile(kf.silicon(0.3), (10, 1))
    if "tesla" in kw:
        _with_field(tel, kw["tesla"], kf)
    _correlate_time(tel)
    cfg = kf.default_config(overstep_limit=0.1, material_effects=3)
    g = kf.fit_device(tel, cfg)
    o = orc.fit(tel, cfg, threads=0, variant="precise")
    assert np.array_equal(g["status"], o["status"]) and np.array_equal(g["n_steps"], o["n_steps"])
    rep = parity_report(g, o, TOL, mask=o["status"] == 0)
    print(rep)
    assert rep["params"] <= 1 and rep["chi2"] <= 1 and rep["cov"] <= 10, rep


@pytest.mark.parametrize("n", [1, 3, 5, 31, 700, 3041])
@pytest.mark.parametrize("kind", ["uniform", "map", "mixed"])
def test_lanes_per_track_do_not_change_the_bits(kf, n, kind):
    """Small batches run eight lanes a track, larger ones a lane a track with
    fewer or more tracks a warp, in or out of order: the first n tracks of a
    larger batch come out bitwise as a batch of n does."""
    kw = dict(n_planes=15, x_first=80., x_step=80., min_len=5, max_len=15, hit_prob=0.9,
              outlier_prob=0.02, field_map=kind == "map")
    tel = _correlate_time(kf.make_telescope(6000, seed=35, **kw))
    from gpukalmanfitter_gb300 import shard
    cfg = kf.default_config(overstep_limit=0.1, outlier_chi2_cut=25.0, precision=int(kind == "mixed"))
    whole = kf.fit_device(tel, cfg)
    part = kf.fit_device(shard.subset(tel, np.arange(n)), cfg)
    for k, v in part.items():
        assert np.array_equal(v, whole[k][..., :n]), k


@pytest.mark.parametrize("n", [19456, 19457, 30011, 38912, 38913])
@pytest.mark.parametrize("uneven", [False, True])
@pytest.mark.parametrize("precision", [0, 1])
def test_shares_or_queue_do_not_change_the_bits(kf, n, uneven, precision):
    """Batches of 4 ... 8 warps an SM take static shares or, with uneven
    lengths, a queue of 4 warps an SM; larger ones a queue of 8: the last
    tracks of the batch come out bitwise as a batch of their own."""
    kw = dict(n_planes=12, x_first=80., x_step=80., min_len=4 if uneven else 12, max_len=12, hit_prob=0.9)
    tel = kf.make_telescope(n, seed=36, **kw)
    from gpukalmanfitter_gb300 import shard
    cfg = kf.default_config(overstep_limit=0.1, precision=precision)
    whole = kf.fit_device(tel, cfg)
    part = kf.fit_device(shard.subset(tel, np.arange(n - 2000, n)), cfg)
    for k, v in part.items():
        assert np.array_equal(v, whole[k][..., -2000:]), k
