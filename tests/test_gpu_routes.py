"""Which kernel and launch serve a call does not change its bits: the routes
whose forms the other tests do not reach.  Sizes follow the device's SM count,
by which launches are chosen; the general adjoint kernel in a field that it
alone serves."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


def _same_bits(kf, tel, rows, cfg, **kw):
    """The rows fitted in the whole batch and by themselves."""
    from gpukalmanfitter_gb300 import shard
    whole = kf.fit_device(tel, cfg, **kw)
    part = kf.fit_device(shard.subset(tel, rows), cfg, **kw)
    assert np.mean(whole["status"] == 0) > 0.9
    for k, v in part.items():
        w = whole[k][..., rows]
        if k == "smoothed":  # (only the states that a track has are written)
            has = np.arange(tel.n_surfaces)[:, None] < part["n_meas"]
            v, w = (np.moveaxis(a, 1, 2)[has] for a in (v, w))
        assert np.array_equal(v, w), k


# eight lanes a track (up to 20 tracks an SM) against one lane a track
@pytest.mark.parametrize("tracks", ["1", "3", "5", "31", "700", "20 an SM", "20 an SM + 1"])
@pytest.mark.parametrize("uneven", [False, True])
def test_lanes_per_track_mixed_map(kf, sms, tracks, uneven):
    n = 20 * sms + ("+" in tracks) if "SM" in tracks else int(tracks)
    tel = kf.make_telescope(40 * sms, seed=91, n_planes=15, x_first=80., x_step=80., min_len=5 if uneven else 15,
                            max_len=15, hit_prob=0.9, outlier_prob=0.02, field_map=True, field_n=21)
    cfg = kf.default_config(overstep_limit=0.1, outlier_chi2_cut=25.0, precision=1)
    _same_bits(kf, tel, np.arange(n), cfg)


# static shares, a queue of 4 warps an SM (uneven lengths) and one of 8 (whose
# blocks of the mixed form run their events together) against a small batch
@pytest.mark.parametrize("warps, more", [(4, 0), (4, 1), (6, 11), (8, 0), (8, 1)])
@pytest.mark.parametrize("uneven", [False, True])
@pytest.mark.parametrize("kind", ["smoothed", "material", "map", "mixed map"])
def test_shares_or_queue(kf, sms, warps, more, uneven, kind):
    n = 32 * warps * sms + more
    tel = kf.make_telescope(n, seed=92, n_planes=12, x_first=80., x_step=80., min_len=4 if uneven else 12,
                            max_len=12, hit_prob=0.9, field_map="map" in kind, field_n=21)
    if kind == "material":
        tel.material = np.tile(kf.silicon(0.3), (12, 1))
    cfg = kf.default_config(overstep_limit=0.1, precision=int(kind == "mixed map"),
                            material_effects=3 if kind == "material" else 0)
    _same_bits(kf, tel, np.arange(n - 2000, n), cfg, smoothed=kind == "smoothed")


# The general adjoint kernel in a field off the z axis, against fourth-order
# central differences of the plain fit's smoothed chi2: steps and bounds of the
# test along z (test_gpu_adjoint.py).
def test_adjoint_off_axis(kf):
    import copy
    tel = kf.make_telescope(600, seed=93, n_planes=12, x_first=50., x_step=50., mis_shift=0.1, mis_rot=1e-3,
                            bz_tesla=0.2)
    along_z = tel.field

    def field(grid_ptr=None, scale=1.0):
        f = along_z(grid_ptr, scale)
        for a, b in enumerate((0.3, -0.5, 1.9)):
            f.value[a] = b * 0.1 * kf.TESLA
        return f

    tel.field = field
    cfg = kf.default_config(overstep_limit=0.1)
    r = kf.AdjointBatch(tel, cfg).run(grad=True)
    ok = r["status"] == 0
    assert ok.mean() > 0.95

    def chi2(t):
        o = kf.fit_device(t, cfg, smoothed=True)
        c = np.zeros(t.n)
        for k in range(t.n_surfaces):
            x = o["smoothed"][k]
            r0, r1 = t.meas[k, 0] - x[0], t.meas[k, 1] - x[1]
            v00, v01, v11 = t.meas[k, 2:]
            c += (v11 * r0 * r0 - 2 * v01 * r0 * r1 + v00 * r1 * r1) / (v00 * v11 - v01 * v01)
        return c

    base = chi2(tel)
    assert np.allclose(base[ok], r["chi2"][ok], rtol=1e-9)

    def fd4(f, h):
        return (f(-2 * h) - 8 * f(-h) + 8 * f(h) - f(2 * h)) / (12 * h)

    def close(g, fd):
        rel = np.abs(g - fd)[ok] / np.maximum(np.abs(fd[ok]), np.median(np.abs(fd[ok])))
        assert np.median(rel) < 3e-7 and np.quantile(rel, 0.98) < 3e-6, np.sort(rel)[-4:]

    for e, scale in enumerate((0.05, 0.05, 1e-3, 1e-3, 0.05)):
        def f(d):
            t = copy.copy(tel)
            t.start = tel.start.copy()
            t.start[e] += d
            return chi2(t)
        close(r["grad_start"][e], fd4(f, 1e-4 * np.maximum(np.abs(tel.start[e]), scale)))

    def f(d):
        t = copy.copy(tel)
        t.field = lambda grid_ptr=None, scale=1.0: field(grid_ptr, scale + d)
        return chi2(t)
    close(r["grad_field_scale_track"], fd4(f, 1e-4))
    al = np.zeros((tel.n_surfaces, 6))
    for k in (0, 7):
        for a, scale in enumerate((0.1, 0.1, 0.1, 1e-3, 1e-3, 1e-3)):
            def f(d):
                t = copy.copy(tel)
                m = al.copy()
                m[k, a] = d
                t.center, t.rotation = kf.align_geometry(tel.center, tel.rotation, m)
                return chi2(t)[ok].sum()
            fd = fd4(f, 3e-4 * scale)
            g = r["grad_align"][k, a]
            assert abs(g - fd) <= 1e-6 * max(abs(fd), 1e-3 * np.max(np.abs(r["grad_align"][:, a]))), (k, a, g, fd)
