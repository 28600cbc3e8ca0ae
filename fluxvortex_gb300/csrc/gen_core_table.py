"""Writes fvx_core_table.cuh: the Gaussian core's polynomials (fvx_x3.cuh).

F(x) = g(rho) / rho^3 with x = rho^2 and g(rho) = erf(rho / sqrt 2) -
sqrt(2 / pi) rho exp(-rho^2 / 2) (src/fluxvortex/kernel.py:16-18), and G(x) =
2 F'(x) = (sqrt(2 / pi) rho^3 exp(-rho^2 / 2) - 3 g) / rho^5, are interpolated
on every interval [i / 4, (i + 1) / 4) of [0, 90) at ten Chebyshev nodes in
60-digit arithmetic; beyond 90 the core is the singular one to 1e-18, F =
x^-3/2, interpolated on the intervals [j, j + 1) of [64, 256), to which a power
of four brings every x.  Each polynomial about the interval's middle is stored as 20 floats (see Row).

    python gen_core_table.py > fvx_core_table.cuh
"""
import mpmath as mp
import numpy as np

mp.mp.dps = 60
ROWS, DEG = 360, 9


def g(x):
    rho = mp.sqrt(x)
    return mp.erf(rho / mp.sqrt(2)) - mp.sqrt(2 / mp.pi) * rho * mp.exp(-x / 2)


def F(x):
    return g(x) / mp.sqrt(x) ** 3


def G(x):
    rho = mp.sqrt(x)
    return (mp.sqrt(2 / mp.pi) * rho ** 3 * mp.exp(-x / 2) - 3 * g(x)) / rho ** 5


def F_far(x):
    return x ** mp.mpf(-1.5)


def G_far(x):
    return -3 * x ** mp.mpf(-2.5)


def coefficients(fn, mid, half):
    n = DEG + 1
    nodes = [half * mp.cos(mp.pi * (2 * k + 1) / (2 * n)) for k in range(n)]
    a = mp.matrix(n, n)
    b = mp.matrix(n, 1)
    for i, t in enumerate(nodes):
        for j in range(n):
            a[i, j] = (t / half) ** j
        b[i] = fn(mid + t)
    c = mp.lu_solve(a, b)
    return [c[j] / half ** j for j in range(n)]


def split(v, parts):
    out = []
    for _ in range(parts):
        f = np.float32(float(v))
        # float() rounds to FP64 first; the float nearest to that is within its
        # last place, and the next part takes the difference up
        out.append(f)
        v -= mp.mpf(float(f))
    return out


def row(c):
    out = []
    for k, v in enumerate(c):
        out += split(v, 3 if k < 2 else (2 if k < 6 else 1))
    return out + [np.float32(0)] * (20 - len(out))


def text(fn, mid, half):
    return "  " + ", ".join(float(v).hex() + "f" for v in row(coefficients(fn, mid, half)))


def main():
    print("// Generated by gen_core_table.py: the Gaussian core's polynomials.")
    print("#pragma once\n")
    print("namespace fvx {\nnamespace x3 {\n")
    print("constexpr int kCoreRows = %d;" % ROWS)
    print("constexpr float kCoreEnd = 90.0f;")
    print("constexpr int kFarRows = 192;  // [64, 256), after the others")
    print("// [interval][F, G][20 floats]")
    print("#define FVX_CORE_TABLE \\")
    lines = []
    for i in range(ROWS):
        mid = mp.mpf(2 * i + 1) / 8
        for fn in (F, G):
            lines.append(text(fn, mid, mp.mpf(1) / 8))
    for j in range(64, 256):
        for fn in (F_far, G_far):
            lines.append(text(fn, mp.mpf(2 * j + 1) / 2, mp.mpf(1) / 2))
    print(", \\\n".join(lines))
    print("\n}  // namespace x3\n}  // namespace fvx")


if __name__ == "__main__":
    main()
