"""Coefficients of cos_turns (so_kerr.cuh; the oracle repeats them) and of its packed FP32 form cos_turns2
(so_packed32.cuh): near-minimax polynomials of degree 8 and 4 in z = g^2 for cos(2 pi g) on |g| <= 1/4
turn, from Chebyshev interpolation of cos(2 pi sqrt(z)) on [0, 1/16] at 60-digit precision, printed as C
hex-float literals (ascending powers of z).  Run: python fit_cos_turns.py"""
import mpmath as mp
import numpy as np

mp.mp.dps = 60


def fit(degree, rounded, name):
    poly, err = mp.chebyfit(lambda z: mp.cos(2 * mp.pi * mp.sqrt(z)), [mp.mpf(0), mp.mpf(1) / 16], degree + 1,
                            error=True)
    coef = [rounded(float(c)) for c in reversed(poly)]
    # error of the rounded coefficients on a fine grid of g
    worst = max(abs(sum(mp.mpf(float(c)) * (g * g) ** j for j, c in enumerate(coef)) - mp.cos(2 * mp.pi * g))
                for g in (mp.mpf(k) / 4096 / 4 for k in range(0, 4097)))
    print(f"// max abs error: exact-coefficient fit {mp.nstr(err, 3)}, {name} coefficients {mp.nstr(worst, 3)}")
    print("{" + ", ".join(float(c).hex() for c in coef) + "}")
    return coef


fit(8, float, "double")
coef = fit(4, np.float32, "float")
# evaluated in FP32 (each fma rounded once: the product of two floats is exact in double, and the double
# rounding of the sum does not show at this size)
g = np.linspace(-0.25, 0.25, 400001).astype(np.float32)
z = g * g
p = np.full_like(z, coef[4])
for c in coef[3::-1]:
    p = (p.astype(np.float64) * z + np.float64(c)).astype(np.float32)
print(f"// in FP32 arithmetic {np.abs(p - np.cos(2 * np.pi * g.astype(np.float64))).max():.3g}")
