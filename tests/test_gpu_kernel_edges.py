"""Sizes at which the rewritten kernels can go wrong: mode counts around the warp and the group of eight,
noise scales from fewer cells than texels to a cell per texel, and the tracer's variants with and
without the coordinate time."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _torus(so, n, modes, **prec):
    sh = so.Shot("synchrotron_1024.ini", [f"camera.width={n}", f"camera.height={n}", "flow.n0=1594262.8",
                                          f"so.modes={modes}"])
    r = so.Renderer(sh.scene, sh.tables, sh.settings)
    r.set_plasma(sh.plasma())
    r.set_precision(prec.pop("precision"), **prec)
    img, _, st = r.render(sh.frame(0))
    r.close()
    return img, st


@pytest.mark.parametrize("modes", [1, 31, 33, 200, 1024])
def test_fp64_sums_any_mode_count(so, modes):
    """k_turb64_records (a position per thread, tree over the partial sums) equals the tracer's own warp
    sums bit for bit: the frame with a record pool against the one whose pool is too small."""
    a, sa = _torus(so, 72, modes, precision=so.abi.SO_PREC_FP64)
    b, sb = _torus(so, 72, modes, precision=so.abi.SO_PREC_FP64, pool_mb=0.001)
    assert sa.rec64_short == 0 and sb.rec64_short > 0
    assert a[..., 0].max() > 0 and np.array_equal(a, b)


@pytest.mark.parametrize("modes", [3, 8, 100, 1024])
def test_fp32_sums_any_mode_count(so, modes):
    """mode_sums2 (packed, every eighth mode on the FMA pipe) against the tracer's SFU sums: both are within
    1.3e-5 of the sums' norm (0.3) of the 64-bit value, so an emission exp(delta) differs by at most
    about 1e-5 and the image by less than 5e-5 of its norm."""
    a, _ = _torus(so, 64, modes, precision=so.abi.SO_PREC_MIXED)
    b, _ = _torus(so, 64, modes, precision=so.abi.SO_PREC_MIXED, turbulence=1)
    a, b = a[..., 0].astype(np.float64), b[..., 0].astype(np.float64)
    assert b.max() > 0 and np.abs(a - b).sum() <= 5e-5 * b.sum()


@pytest.mark.parametrize("scale", [0.02, 0.1, 3.0])
def test_bake_any_noise_scale(so, orc, scale):
    """The bake at noise scales whose cells along phi run from one or two a row to one a texel (the octave
    by octave form), against the oracle's texels: the bar of the shipped scale's test."""
    n = 20
    sh = so.Shot("m87_reference_flow.ini", [f"camera.width={n}", f"camera.height={n}",
                                            f"flow.turbulence_scale={scale}"])
    r = so.Renderer(sh.scene, sh.tables, sh.settings)
    r.set_flow_noise(so.abi.SO_FLOW_NOISE_BAKED_FP32)
    f = sh.frame(0)
    X, Y = so.pixel_centres(f, n, n)
    k = r.trace_rays(f, X, Y)
    o = orc.orc_trace(orc.baked(sh.scene), f, X, Y)
    r.close()
    I0, I1 = o["I"].astype(np.float64), k["I"].astype(np.float64)
    assert I0[:, 0].max() > 0
    assert np.abs(I0 - I1).max() <= 1e-6 * I0[:, 0].max()


@pytest.mark.parametrize("turb", [0.0, 0.6])
def test_disk_with_and_without_time(so, orc, turb):
    """The disk tracer leaves the coordinate time out unless the disk's turbulence reads it."""
    n = 48
    sh = so.Shot("thin_disk_4096.ini", [f"camera.width={n}", f"camera.height={n}", f"disk.turbulence={turb}"])
    r = so.Renderer(sh.scene, sh.tables, sh.settings)
    f = sh.frame(0)
    X, Y = so.pixel_centres(f, n, n)
    k = r.trace_rays(f, X, Y)
    o = orc.orc_trace(sh.scene, f, X, Y)
    r.close()
    for key in ("fate", "ncross", "n_accepted", "n_attempts"):
        assert np.array_equal(k[key], o[key]), key
    I0, I1 = o["I"].astype(np.float64), k["I"].astype(np.float64)
    assert I0.max() > 0 and np.abs(I0 - I1).max() <= 1e-5 * I0.max()


@pytest.mark.parametrize("spp", [2, 3, 4, 32])
def test_transfer_samples_per_job(so, spp):
    """The ordered transfer takes a lane per sample at 2, 4, .. 32 samples a job and one thread otherwise: the
    frame with a record pool (4320 jobs: enough to defer) equals the one whose pool is too small (the replay
    pass) bit for bit."""
    imgs = []
    for pool in ({}, {"pool_mb": 0.001}):
        sh = so.Shot("m87_reference_flow.ini", ["camera.width=72", "camera.height=60", f"render.spp={spp}",
                                                f"render.spp_max={spp}"])
        r = so.Renderer(sh.scene, sh.tables, sh.settings)
        r.set_precision(so.abi.SO_PREC_FP64, **pool)
        img, _, st = r.render(sh.frame(0))
        r.close()
        assert (st.rec64_short > 0) == bool(pool)
        imgs.append(img)
    assert imgs[0][..., 0].max() > 0 and np.array_equal(*imgs)


@pytest.mark.parametrize("band_m", [0.05, 0.6])
def test_mixed_flow_band_deferred(so, band_m):
    """A mixed reference-flow frame's band rays, their emission deferred to passes of their own, equal bit for
    bit the same rays of a frame whose band covers the field (emission in the tracer)."""
    n = 128
    sh = so.Shot("m87_reference_flow.ini", [f"camera.width={n}", f"camera.height={n}", "render.spp=1",
                                            "render.spp_max=1"])
    r = so.Renderer(sh.scene, sh.tables, sh.settings)
    f = sh.frame(0)
    r.set_precision(so.abi.SO_PREC_MIXED, band_m=band_m)
    a, _, _ = r.render(f)
    fa, band = r.last_fates(n * n)
    r.set_precision(so.abi.SO_PREC_MIXED, band_m=1e6)
    b, _, _ = r.render(f)
    fb, every = r.last_fates(n * n)
    r.close()
    assert every.all() and 0 < band.sum() < n * n // 4
    a, b = a.reshape(n * n, -1), b.reshape(n * n, -1)
    assert b[band, 0].max() > 0 and np.array_equal(a[band], b[band]) and np.array_equal(fa[band], fb[band])


@pytest.mark.parametrize("ini,over", [("thin_disk_4096.ini", "disk.turbulence=0"), ("thin_disk_4096.ini", "disk.turbulence=0.6"),
                                      ("m87_reference_flow.ini", "camera.incl=163"),
                                      ("synchrotron_1024.ini", "so.modes=8")])
def test_launch_shape_changes_no_ray(so, ini, over):
    """A list that three CTAs per SM hold at once runs with 168 registers, a longer one with 128: every output
    of 60,000 rays in one call equals that of the same rays in calls of 20,000 bit for bit."""
    sh = so.Shot(ini, ["camera.width=250", "camera.height=240", over])
    r = so.Renderer(sh.scene, sh.tables, sh.settings)
    r.set_plasma(sh.plasma())
    r.set_flow_noise(so.abi.SO_FLOW_NOISE_INLINE)
    f = sh.frame(0)
    X, Y = so.pixel_centres(f, 250, 240)
    a = r.trace_rays(f, X, Y)
    parts = [r.trace_rays(f, X[i:i + 20000], Y[i:i + 20000]) for i in range(0, 60000, 20000)]
    r.close()
    for key in ("fate", "ncross", "theta", "phi", "I", "n_accepted", "n_attempts"):
        assert np.array_equal(a[key], np.concatenate([p[key] for p in parts]), equal_nan=True), key
