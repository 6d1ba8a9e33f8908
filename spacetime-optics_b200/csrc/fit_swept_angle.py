"""Coefficients of swept_angle (so_fast64.cuh): minimax polynomials (Chebyshev interpolation at 60-digit
precision) of sin(g)/g in g^2 on |g| <= pi/2 (degree 7) and of 2 asin(sqrt(w)/2) / sqrt(w) in w on
[0, 1/2] (degree 9), printed as C hex-float literals (ascending powers).  Run: python fit_swept_angle.py"""
import mpmath as mp

mp.mp.dps = 60


def fit(name, f, hi, n):
    lo = mp.mpf("1e-12")
    coef = [mp.mpf(float(c)) for c in reversed(mp.chebyfit(f, [lo, hi], n))]
    worst = max(abs(sum(c * z ** j for j, c in enumerate(coef)) / f(z) - 1)
                for z in (lo + (hi - lo) * mp.mpf(k) / 2000 for k in range(2001)))
    print(f"// {name}: max relative error with double coefficients {mp.nstr(worst, 3)}")
    print("{" + ", ".join(float(c).hex() for c in coef) + "}")


fit("sin(g)/g", lambda z: mp.sin(mp.sqrt(z)) / mp.sqrt(z), (mp.pi / 2) ** 2 * mp.mpf("1.0001"), 8)
fit("angle/chord", lambda w: 2 * mp.asin(mp.sqrt(w) / 2) / mp.sqrt(w), mp.mpf("0.5"), 10)
