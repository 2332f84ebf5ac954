"""Generate cl_tables.h: constants for the device's Float32 elementary functions.

Every value is computed here from its mathematical definition with Python's
``decimal`` module at 60 significant digits and rounded once to IEEE double
(``float(Decimal)`` rounds correctly):

* the table (sin, cos)(j/64) over one turn and the short polynomials in the
  remainder that go with it (Taylor coefficients; the last cosine term
  economised, C. Lanczos, "Applied Analysis", 1956);
* ln 2 and, for F_j = 1 + j/64 (j = -19..27), the pairs (1/F_j, ln F_j) of a
  table-driven logarithm in the manner of P. T. P. Tang, "Table-driven
  implementation of the logarithm function in IEEE floating-point arithmetic",
  ACM TOMS 16(4), 1990;
* the Taylor coefficients (-1)^(k+1)/k of log1p.

Run: python gen_tables.py > cl_tables.h
"""
from decimal import Decimal, getcontext
import math

getcontext().prec = 60

LOG_JMIN, LOG_JMAX = -19, 27   # round(64*(m-1)) for m in [sqrt(1/2), sqrt(2))


def d_sin_cos(x: Decimal) -> tuple:
    """sin and cos by their Taylor series at 60 digits (|x| <= 2 pi)."""
    eps = Decimal(10) ** (-(getcontext().prec + 2))
    s, c = Decimal(0), Decimal(0)
    term, n = Decimal(1), 0          # x^n / n!
    while True:
        if n % 4 == 0: c += term
        elif n % 4 == 1: s += term
        elif n % 4 == 2: c -= term
        else: s -= term
        n += 1
        term = term * x / n
        if abs(term) < eps and n > 4:
            break
    return s, c


def dbl(x: Decimal) -> float:
    return float(x)


def hexd(v: float) -> str:
    return float.hex(v)


def main() -> None:
    ln2 = dbl(Decimal(2).ln())

    out = []
    out.append("/* Generated by gen_tables.py from exact arithmetic (decimal, 60 digits). */")
    out.append("#pragma once")
    out.append("")
    out.append(f"#define CLM_LN2 {hexd(ln2)}  /* {ln2!r} */")
    out.append("")
    # log1p(r) = r + r^2 (L2 + r (L3 + ... + r L8)), L_k = (-1)^(k+1)/k
    for k in range(2, 9):
        c = Decimal((-1) ** (k + 1)) / Decimal(k)
        out.append(f"#define CLM_L{k} {hexd(dbl(c))}")
    out.append("")
    out.append(f"#define CLM_LOG_JMIN ({LOG_JMIN})")
    out.append(f"#define CLM_LOG_NTAB {LOG_JMAX - LOG_JMIN + 1}")
    out.append("/* (1/F_j, ln F_j), F_j = 1 + j/64, j = CLM_LOG_JMIN .. */")
    out.append("#define CLM_LOG_TAB_INIT \\")
    for j in range(LOG_JMIN, LOG_JMAX + 1):
        F = Decimal(64 + j) / Decimal(64)
        inv = dbl(1 / F)
        lg = dbl(F.ln()) if j != 0 else 0.0
        out.append(f"    {hexd(inv)}, {hexd(lg)},  /* j = {j} */ \\")
    out.append("")
    # table-driven sincos: x = j/64 + r, |r| <= 1/128 (both exact in Float32)
    n_sc = 404                       # j/64 up to 403/64 > 2 pi
    out.append("")
    out.append(f"#define CLM_SC_N {n_sc}")
    for n in (3, 5):
        c = Decimal((-1) ** ((n - 1) // 2)) / Decimal(math.factorial(n))
        out.append(f"#define CLM_TS{n} {hexd(dbl(c))}")
    # cos r - 1 = C2 r^2 + C4 r^4 + C6 r^6 economised to two terms: with t = r^2
    # in [0, T], t^3 is replaced by the quadratic that leaves the least error
    # (t^3 minus it is the cubic Chebyshev polynomial with its first root moved
    # to t = 0), 0.0385 T^3 instead of T^3: 2^-56 of the result
    T = Decimal(1) / Decimal(128 * 128)
    root3 = Decimal(3).sqrt()
    sc = T / (1 + root3 / 2)
    c2, c4, c6 = Decimal(-1) / 2, Decimal(1) / 24, Decimal(-1) / 720
    out.append(f"#define CLM_TC2 {hexd(dbl(c2 - c6 * (3 * sc * sc / 2)))}")
    out.append(f"#define CLM_TC4 {hexd(dbl(c4 + c6 * (3 * root3 / 2 * sc)))}")
    out.append("/* (sin, cos)(j / 64), j = 0..403 */")
    out.append("#define CLM_SC_TAB_INIT \\")
    for j in range(n_sc):
        sd, cd = d_sin_cos(Decimal(j) / 64)
        out.append(f"    {hexd(dbl(sd))}, {hexd(dbl(cd))},  /* j = {j} */ \\")
    out.append("")
    print("\n".join(out))


if __name__ == "__main__":
    main()
