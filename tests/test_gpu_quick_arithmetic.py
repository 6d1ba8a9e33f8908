"""The tracers' straight-line division, reciprocal and square root as the device runs them (so_probe_quick: its own
seeds, the flags of the tracers' files) against the IEEE operators, over the ranges they are stated for."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _quick(so, op, a, b=None):
    import torch
    d = [torch.tensor(v, dtype=torch.float64, device="cuda") for v in ((a, b) if b is not None else (a,))]
    out = torch.empty_like(d[0])
    torch.cuda.synchronize()
    rc = so.lib().so_probe_quick(op, C.c_void_p(d[0].data_ptr()), C.c_void_p(d[-1].data_ptr()),
                                 C.c_void_p(out.data_ptr()), d[0].numel())
    assert rc == 0
    return out.cpu().numpy()


def _operands(rng, n, span, bits=52):
    """Signed values of random significands (a few short, a few just under a power of two, none of all ones) and
    exponents in [-span, span]."""
    one = 1 << bits
    m = rng.integers(0, one - 1, n)
    m[::5] &= ~((1 << (bits // 2)) - 1)
    m[1::11] |= (one - 1) ^ ((1 << (bits // 4)) - 1)
    m[m == one - 1] = 0
    return np.ldexp(1.0 + m / one, rng.integers(-span, span + 1, n)) * rng.choice([-1.0, 1.0], n)


def test_fp64_reciprocal_and_quotient(so):
    rng = np.random.default_rng(1)
    a, b = _operands(rng, 2000000, 300), _operands(rng, 2000000, 300)
    a[::7] = b[::7] * rng.integers(1, 1000, a[::7].size)  # quotients near whole numbers
    b[::13] = 1e-300
    a[::13] = rng.uniform(-20.0, 20.0, a[::13].size)  # the pole's sin^2
    a[3] = 0.0
    assert np.array_equal(_quick(so, 0, b), 1.0 / b)
    assert np.array_equal(_quick(so, 1, a, b), a / b)


def test_fp64_square_root(so):
    rng = np.random.default_rng(2)
    x = np.abs(_operands(rng, 2000000, 200))
    x[::3] = rng.uniform(0.0, 1.0, x[::3].size) ** 2
    x[0], x[1] = 0.0, 2.0 ** -106
    assert np.array_equal(_quick(so, 2, x), np.sqrt(x))


def test_fp32_reciprocal(so):
    """Rounded to nearest for normal operands and results; 0 and infinity give each other."""
    rng = np.random.default_rng(3)
    x = _operands(rng, 2000000, 125, bits=23)
    x[0], x[1], x[2], x[3] = 0.0, np.inf, 1.0, -2.0
    got = _quick(so, 3, x)
    with np.errstate(divide="ignore"):
        want = (1.0 / x).astype(np.float32).astype(np.float64)
    assert np.array_equal(got, want)
