"""Generate csrc/boys_table_data.inc: the polynomials of the Boys evaluation
(boys_fm in csrc/pfk_os.cuh), by Chebyshev interpolation in 40-digit
arithmetic, converted to the monomial basis the kernels evaluate.

  kBoysMid[M]    F_0(T) sqrt(T + 16), 0 <= T <= TA(M), in y = 2x/x1 - 1 with
                 x = T / (T + 16), x1 = TA / (TA + 16).  The factor and the
                 variable make the function nearly straight (4.0 at T = 0 to
                 about 1.1 at TA), so the degree is 25 to 32 over the whole
                 range and the coefficients add up to 4: no cancellation.
  kBoysSmall[M]  F_M(T), 0 <= T <= TS(M), in T - TS/2: about the middle the
                 coefficients fall off, where those in T alternate and cancel
                 (relative error 1.2e-14 for M = 5 and 6, now 1.2e-15).
  kBoysExp       e^r, |r| <= ln 2 / 2.

    python gen_boys_table.py > csrc/boys_table_data.inc
"""
import mpmath as mp

C = 16
TA = [34, 38, 42, 44, 46, 60, 60]
TS = [1, 1, 2.125, 2.125, 2.25, 3.25, 3.25]
MID_DEG = [25, 26, 28, 28, 29, 32, 32]
SMALL_DEG = [12, 12, 15, 15, 15, 17, 17]
EXP_DEG = 11


def boys(m, T):
    if T < mp.mpf(10) ** -35:
        return mp.mpf(1) / (2 * m + 1)
    return mp.gammainc(m + mp.mpf(1) / 2, 0, T) / (2 * T ** (m + mp.mpf(1) / 2))


def interpolate(f, lo, hi, deg, var):
    """Monomial coefficients, in var(t) of t in [lo, hi] mapped from the
    Chebyshev nodes of [-1, 1], of the degree-deg interpolant of f."""
    n = deg + 1
    nodes = [mp.cos(mp.pi * (k + mp.mpf(1) / 2) / n) for k in range(n)]
    pts = [(lo + hi) / 2 + (hi - lo) / 2 * y for y in nodes]
    A = mp.matrix(n, n)
    for i in range(n):
        for j in range(n):
            A[i, j] = var(pts[i]) ** j
    return list(mp.lu_solve(A, mp.matrix([f(p) for p in pts])))


def mid(M):
    ta, c = mp.mpf(TA[M]), mp.mpf(C)
    x1 = ta / (ta + c)

    def f(y):
        x = (y + 1) / 2 * x1
        T = c * x / (1 - x)
        return boys(0, T) * mp.sqrt(T + c)
    return interpolate(f, mp.mpf(-1), mp.mpf(1), MID_DEG[M], lambda y: y), 2 / x1


def small(M):
    return interpolate(lambda T: boys(M, T), mp.mpf(0), mp.mpf(TS[M]), SMALL_DEG[M], lambda T: T - mp.mpf(TS[M]) / 2)


def tables():
    mp.mp.dps = 40
    h = mp.log(2) / 2
    m = [mid(M) for M in range(7)]
    return {"mid": [[float(v) for v in r[0]] for r in m], "mid_scale": [float(r[1]) for r in m],
            "small": [[float(v) for v in small(M)] for M in range(7)],
            "exp": [float(v) for v in interpolate(mp.exp, -h, h, EXP_DEG, lambda r: r)]}


def main():
    t = tables()

    def rows(name, vals, width):
        print(f"static __constant__ double {name}[7][{width}] = {{")
        for v in vals:
            print("    {" + ", ".join(repr(x) for x in v + [0.0] * (width - len(v))) + "},")
        print("};")
    print("// Written by gen_boys_table.py: do not edit.")
    print("constexpr double kBoysShift = %d.0;" % C)
    for name, v in (("kBoysTA", TA), ("kBoysTS", TS)):
        print(f"constexpr double {name}[7] = {{" + ", ".join(repr(float(x)) for x in v) + "};")
    for name, v in (("kBoysMidDeg", MID_DEG), ("kBoysSmallDeg", SMALL_DEG)):
        print(f"constexpr int {name}[7] = {{" + ", ".join(map(str, v)) + "};")
    print("constexpr int kBoysExpDeg = %d;" % EXP_DEG)
    print("constexpr double kBoysMidScale[7] = {" + ", ".join(repr(x) for x in t["mid_scale"]) + "};")
    rows("kBoysMid", t["mid"], max(MID_DEG) + 1)
    rows("kBoysSmall", t["small"], max(SMALL_DEG) + 1)
    print(f"static __constant__ double kBoysExp[{EXP_DEG + 1}] = {{")
    print("    " + ", ".join(repr(x) for x in t["exp"]) + "};")


if __name__ == "__main__":
    main()
