"""Record pools of the deferred passes: what the host code does when memory is short, limited or has run out.
The library runs in a child process on a CUDA runtime without a device (fake_cudart.cpp): kernels do
nothing, so only allocations, launches and statuses mean anything."""
import json
import os
import shutil
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))

PRELUDE = """
import ctypes as C, json, sys
import numpy as np
sys.path.insert(0, %r)
import conftest
so = conftest.load_package()
rt = C.CDLL(sys.argv[1])
for name in ("fake_mallocs", "fake_graphs", "fake_launches"):
    getattr(rt, name).restype = C.c_longlong
for name in ("fake_held", "fake_largest"):
    getattr(rt, name).restype = C.c_size_t
rt.fake_memory.argtypes = [C.c_size_t]
rt.fake_fail_in.argtypes = [C.c_longlong]
rt.fake_counts.argtypes = [C.c_size_t] + [C.c_ulonglong] * 3
MIXED, FP64 = so.abi.SO_PREC_MIXED, so.abi.SO_PREC_FP64
def flow(n):
    sh = so.Shot("m87_reference_flow.ini", ["camera.width=%%d" %% n, "camera.height=%%d" %% n, "render.spp=1",
                                            "render.spp_max=1"])
    return so.Renderer(sh.scene, sh.tables, sh.settings), sh.frame(0)
def frame(r, f):
    # status of one frame into a buffer of the renderer's size, and what it allocated and launched
    px = np.zeros(r.settings.W * r.settings.H * 4, np.float32)
    m, l = rt.fake_mallocs(), rt.fake_launches()
    rc = so.lib().so_render_device(r.h, C.byref(f), px.ctypes.data_as(C.c_void_p), None)
    return rc, rt.fake_mallocs() - m, rt.fake_launches() - l
"""


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("needs g++")
    lib = str(tmp_path_factory.mktemp("rt") / "fake_cudart.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-o", lib, os.path.join(HERE, "fake_cudart.cpp")],
                   check=True)

    def run(body):
        p = subprocess.run([sys.executable, "-c", PRELUDE % HERE + body, lib], env=dict(os.environ, LD_PRELOAD=lib),
                           capture_output=True, text=True, timeout=300)
        assert p.returncode == 0, p.stderr[-3000:]
        return json.loads(p.stdout)
    return run


@pytest.mark.parametrize("prec,spare", [("MIXED", 8), ("FP64", 8)])
def test_failed_allocation_leaves_no_error(host, prec, spare):
    """Whichever allocation of a first reference flow frame fails, the frame is rendered (those of the FP64
    passes' pools, `spare` of them: the rays then run in the tracer) or refused, and the next one is rendered."""
    out, codes = host("""
out = []
for k in range(40):
    r, f = flow(64)
    r.set_precision(%s)
    rt.fake_fail_in(k)
    first = frame(r, f)[0]
    rt.fake_fail_in(-1)
    out.append((first, frame(r, f)[0]))
    r.close()
print(json.dumps([out, [0, so.abi.SO_ERR_ALLOC, so.abi.SO_ERR_CUDA]]))
""" % prec)
    n = max([i + 1 for i, (a, b) in enumerate(out) if a] + [0])
    assert all(a in codes and b == 0 for a, b in out)
    assert sum(a == 0 for a, _ in out[:max(n, spare)]) >= spare


def test_pool_limit_holds_for_every_pool(host):
    """so_mixed_opts.pool_mb = 2 on a mixed reference-flow frame: no block above 2 MiB (the frame's own are
    smaller), neither on a new renderer nor on one that rendered without a limit before."""
    fresh, free, lowered = host("""
r, f = flow(64)
r.set_precision(MIXED, pool_mb=2.0)
out = [(frame(r, f)[0], rt.fake_largest())]
r.close()
r, f = flow(64)
r.set_precision(MIXED)
out.append((frame(r, f)[0], rt.fake_largest()))
r.set_precision(MIXED, pool_mb=2.0)
out.append((frame(r, f)[0], rt.fake_largest()))
print(json.dumps(out))
""")
    assert fresh[0] == free[0] == lowered[0] == 0
    assert fresh[1] <= 2 << 20 and lowered[1] <= 2 << 20 < free[1]


def test_side_pool_is_kept_from_frame_to_frame(host):
    """Later frames of a renderer allocate nothing: where free memory (300 MB) bounds the side passes' pool, and,
    but for one or two steps of growth, where each of 24 frames zooms in by 1 %."""
    capped, zoomed = host("""
rt.fake_memory(rt.fake_held() + (300 << 20))
r, f = flow(64)
r.set_precision(MIXED)
capped = [frame(r, f)[:2] for i in range(5)]
r.close()
rt.fake_memory(64 << 30)
r, f = flow(512)
r.set_precision(MIXED)
zoomed = []
for i in range(24):
    zoomed.append(frame(r, f)[:2])
    f.pix *= 0.99
print(json.dumps([capped, zoomed]))
""")
    assert all(rc == 0 for rc, _ in capped + zoomed)
    assert capped[0][1] > 0 and sum(m for _, m in capped[1:]) == 0
    assert sum(m > 0 for _, m in zoomed[1:]) <= 2


def test_side_pool_that_cannot_grow(host):
    """Every list of every frame runs short.  A pool that may grow doubles; one bounded by free memory (300 MB) or by
    pool_mb neither grows nor records in vain: from the second frame on the rays run in the tracer (six
    launches fewer a frame, three a list), until so_set_precision gives another limit."""
    grown, free, limited, again = host("""
rt.fake_counts(24, 1, 1, 1)
r, f = flow(64)
r.set_precision(MIXED)
grown = []
for i in range(3):
    frame(r, f)
    grown.append(rt.fake_largest())
r.close()
def run(pool_mb):
    r, f = flow(64)
    r.set_precision(MIXED, pool_mb=pool_mb)
    out = [frame(r, f) for i in range(70)]
    r.set_precision(MIXED, pool_mb=pool_mb)
    return out, frame(r, f)[2]
limited, again = run(2.0)
rt.fake_memory(rt.fake_held() + (300 << 20))
free, _ = run(0.0)
print(json.dumps([grown, free, limited, again]))
""")
    assert 1.8 * grown[0] < grown[1] < 2.2 * grown[0] and 1.8 * grown[1] < grown[2] < 2.2 * grown[1]
    for frames in (free, limited):
        assert all(rc == 0 for rc, _, _ in frames)
        assert all(m == 0 and n == frames[0][2] - 6 for _, m, n in frames[2:])
    assert again == limited[0][2]


def test_shortage_under_other_options_is_forgotten(host):
    """A shortage under pool_mb = 2 says nothing about the pool that so_set_precision allows next: the first frame
    after it defers, with the launches of a new renderer's first frame."""
    new, after = host("""
rt.fake_counts(24, 1, 1, 1)
r, f = flow(64)
r.set_precision(MIXED, pool_mb=64.0)
new = frame(r, f)
r.close()
r, f = flow(64)
r.set_precision(MIXED, pool_mb=2.0)
frame(r, f)
r.set_precision(MIXED, pool_mb=64.0)
print(json.dumps([new, frame(r, f)]))
""")
    assert new[0] == after[0] == 0 and new[2] == after[2]


BATCH = """
def batch(r, f, size, frames):
    px = np.zeros(frames * size * size * 4, np.float32)
    b = so.Batch(r, [r.scene], [f] * frames, [0] * frames, size, size)
    def render():
        g = rt.fake_graphs()
        st = b.render(px.ctypes.data, stats=True)
        return rt.fake_graphs() - g, st.rec64_waves
    return render
"""


def test_batch_graph_follows_its_buffers(host):
    """A batch's graph holds the pointers of its launches, so it is captured again when the record pool has been
    replaced (a larger frame or batch on the renderer) or the modes (so_set_plasma), and only then: two
    batches under one pool_mb do not replace each other's pool."""
    got = host(BATCH + """
r, f = flow(128)
r.set_precision(FP64)
a = batch(r, f, 32, 5)
out = [a()[0], a()[0], frame(r, f)[0], a()[0], frame(r, f)[0], a()[0]]
sh = so.Shot("synchrotron_1024.ini", ["so.modes=8", "camera.width=32", "camera.height=32"])
t = so.Renderer(sh.scene, sh.tables, sh.settings)
t.set_plasma(sh.plasma())
b = batch(t, sh.frame(0), 32, 5)
out += [b()[0], b()[0]]
t.set_plasma(sh.plasma())
out += [b()[0], b()[0]]
r.set_precision(FP64, pool_mb=64.0)
c, d = batch(r, f, 32, 5), batch(r, f, 32, 12)
c(), d(), c(), d()
out += [c()[0], d()[0], c()[0], d()[0]]
print(json.dumps(out))
""")
    assert got == [1, 0, 0, 1, 0, 0, 1, 0, 1, 0, 0, 0, 0, 0]


def test_batch_counts_its_own_waves(host):
    """A batch in waves reports (and looks for shortages in) its own number of waves, also when the renderer traced
    a frame in another number since its graph was captured."""
    got = host(BATCH + """
r, f = flow(72)
r.set_precision(FP64, pool_mb=100.0)
b = batch(r, f, 32, 20)
first = b()[1]
st = so.abi.Stats()
px = np.zeros(72 * 72 * 4, np.float32)
so.lib().so_render_device(r.h, C.byref(f), px.ctypes.data_as(C.c_void_p), C.byref(st))
print(json.dumps([first, st.rec64_waves, b()]))
""")
    first, between, (graphs, again) = got
    assert first > 1 and between != first and graphs == 0 and again == first


@pytest.mark.parametrize("prec,size", [("FP64", 24), ("MIXED", 16)])
def test_estimates_stay_finite(host, prec, size):
    """70 frames under a pool_mb too small for any of them double the estimate of records per ray or sample; it stays
    within what a ray can have, so that the first frame without the limit gets a pool (it had overflowed)."""
    largest, frames = host("""
r, f = flow(72)
r.set_precision(%s, pool_mb=0.001)
rt.fake_counts(%d, 1, 1, 1)
frames = [frame(r, f)[0] for i in range(70)]
rt.fake_counts(0, 0, 0, 0)
r.set_precision(%s)
frames.append(frame(r, f)[0])
print(json.dumps([rt.fake_largest(), frames]))
""" % (prec, size, prec))
    assert not any(frames) and largest > 1 << 28


def test_refused_plasma_changes_nothing(host):
    """so_set_plasma that cannot allocate its modes keeps the renderer's plasma, modes and all."""
    rc, alloc, before, after, frames = host("""
sh = so.Shot("synchrotron_1024.ini", ["so.modes=8", "camera.width=32", "camera.height=32"])
r = so.Renderer(sh.scene, sh.tables, sh.settings)
r.set_plasma(sh.plasma())
first = frame(r, sh.frame(0))[0]
held = rt.fake_held()
p = sh.plasma()
p.n_modes = 512
rt.fake_fail_in(0)
rc = so.lib().so_set_plasma(r.h, C.byref(p), so.plasma_modes(p))
rt.fake_fail_in(-1)
print(json.dumps([rc, so.abi.SO_ERR_ALLOC, held, rt.fake_held(), [first, frame(r, sh.frame(0))[0]]]))
""")
    assert rc == alloc and before == after and frames == [0, 0]
