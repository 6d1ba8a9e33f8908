"""Torus turbulence whose phases leave the range of the FMA-pipe cosine (2^21 turns; FP32 phases of that size are
all rounding): the sums must stay sums of cosines."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [False, True])
def test_fp32_sums_stay_bounded(so, batch):
    """16 modes of amplitude 0.05 and |k| = 3e7 rad/M: |delta| <= 0.8 whatever the phases, so the density is within
    a factor exp(0.8) of the smooth torus's and the frame's flux well within 30 of the one with every sum in the
    tracer (frame) or in FP64 (batch)."""
    n = 72
    sh = so.Shot("synchrotron_1024.ini", [f"camera.width={n}", f"camera.height={n}", "flow.n0=1594262.8", "so.modes=16"])
    rs = np.random.default_rng(5)
    modes = (so.abi.Mode * 16)()
    for m in modes:
        d = rs.normal(size=3)
        d *= 3e7 / np.linalg.norm(d)
        m.kx, m.ky, m.kz, m.phase, m.amp = *d, rs.uniform(0.0, 2 * np.pi), 0.05
    r = so.Renderer(sh.scene, sh.tables, sh.settings)
    r.set_plasma(sh.plasma(), modes)
    f = sh.frame(0)
    imgs = []
    for far in (False, True):
        if batch:
            import torch
            r.set_precision(so.abi.SO_PREC_MIXED if far else so.abi.SO_PREC_FP64)
            px = torch.zeros((n, n, 4), device="cuda")
            torch.cuda.synchronize()
            b = so.Batch(r, [sh.scene], [f], [0], n, n)
            st = b.render(px.data_ptr(), stats=True)
            b.close()
            assert st.rec64_records > 0
            imgs.append(px.cpu().numpy())
        else:
            r.set_precision(so.abi.SO_PREC_MIXED, turbulence=0 if far else 1)
            img, _, st = r.render(f)
            assert (st.turb_records > 0) == far
            imgs.append(img)
    r.close()
    near, far = (i[..., 0].astype(np.float64) for i in imgs)
    assert np.isfinite(near).all() and np.isfinite(far).all()
    assert near.sum() / 30 < far.sum() < near.sum() * 30
