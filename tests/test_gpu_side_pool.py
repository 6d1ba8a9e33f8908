"""Record pool of a mixed reference-flow frame's band and re-traced rays: large enough, too small, and given up."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _renderer(so, pool_mb):
    sh = so.Shot("m87_reference_flow.ini", ["camera.width=128", "camera.height=128", "render.spp=1",
                                            "render.spp_max=1"])
    r = so.Renderer(sh.scene, sh.tables, sh.settings)
    r.set_precision(so.abi.SO_PREC_MIXED, band_m=0.6, pool_mb=pool_mb)
    return r, sh.frame(0)


def test_side_pool_shortage_changes_no_pixel(so):
    """The statistics tell which way the lists went: an ample pool holds every ray's records; one of 2 MiB runs
    short, so the replay pass traces the lists again; the next frame keeps them in the tracer.  All images are equal
    bit for bit (the FP32 rays' pool has the same limit and takes waves instead)."""
    r, f = _renderer(so, 0.0)
    a, _, sa = r.render(f)
    r.close()
    r, f = _renderer(so, 2.0)
    b, _, sb = r.render(f)
    c, _, sc = r.render(f)
    r.close()
    assert sa.rec64_records > 0 and sa.rec64_short == 0 and sa.rec64_slots >= sa.rec64_records
    assert sb.rec64_short > 0 and sb.rec64_slots < sa.rec64_slots and sb.record_waves > 1 and sb.redo_records == 0
    assert sc.rec64_slots == sc.rec64_short == sc.rec64_records == 0
    assert sa.band_rays == sb.band_rays == sc.band_rays > 0 and sa.flow_steps == sb.flow_steps == sc.flow_steps
    assert a[..., 0].max() > 0 and np.array_equal(a, b) and np.array_equal(a, c)
