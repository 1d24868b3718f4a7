"""Piecewise fixed-point polynomials for the FP64 pair force of the P2P
kernels: with u = r / 2rs, q = u^2 and

    f(q) = (erfc(u) + (2/sqrt(pi)) u exp(-u^2)) / u^3,

the pair force of src/fmm.c:846-855 is m f(q) dx / (2rs)^3.  The kernels
evaluate f on q in [2^-14, 2^6) from q's bits: each octave is cut into 64
intervals (the exponent and the top 6 mantissa bits of q number them), the
remaining mantissa bits are the position d in [-1/2, 1/2) within the
interval, and

    f = 2^E sum_k P[k] d^k,   degree 7,

is summed in integers: P[0..3] are 64-bit with 62 fraction bits, P[4..7]
32-bit with S fraction bits (S falls for q >= 4, where f's derivatives grow
and g is below 0.05).  Coefficients are f's Taylor coefficients at the
interval's centre from the recurrence that f's differential equation gives,

    q f' = -3/2 f - (2/sqrt(pi)) exp(-q),

at 60 digits, with the degree-8 term folded into the lower even ones by its
Chebyshev polynomial (x^8 = x^8 - T8/128 + O(T8/128)).  The script replays
the integer evaluation on random q and prints the largest error.

Run:  python fit_pair_fp64.py > pair_fp64_table.h
"""
import random

import mpmath as mp

OCT_LO, OCT_HI, MB = -14, 6, 6  # octaves [2^-14, 2^6), 64 intervals each
NI = (OCT_HI - OCT_LO) << MB


def tail_bits(e):
    return 52 if e < 2 else 56 - 4 * e  # fraction bits of P[4..7]


def g_over_u3(q):
    u = mp.sqrt(q)
    return (mp.erfc(u) + 2 / mp.sqrt(mp.pi) * u * mp.exp(-q)) / (u * q)


def interval(i):
    """(exponent E, the integers P[0..7], S) of interval i."""
    e = OCT_LO + (i >> MB)
    w = mp.mpf(2) ** (e - MB)
    qc = mp.mpf(2) ** e + ((i & ((1 << MB) - 1)) + mp.mpf(1) / 2) * w
    E0 = 2 / mp.sqrt(mp.pi) * mp.exp(-qc)
    a = [g_over_u3(qc)]
    for k in range(8):
        a.append((-(k + mp.mpf(3) / 2) * a[k] - E0 * (-1) ** k / mp.factorial(k)) / (qc * (k + 1)))
    a = [a[k] * w ** k for k in range(9)]
    # x = 2 d: x^8 - T8(x)/128 = 2 x^6 - 5/4 x^4 + 1/4 x^2 - 1/128
    top = a[8] / 2 ** 8
    for k, c in ((6, mp.mpf(2)), (4, -mp.mpf(5) / 4), (2, mp.mpf(1) / 4), (0, -mp.mpf(1) / 128)):
        a[k] += top * c * 2 ** k
    ex = int(mp.floor(mp.log(a[0], 2))) + 1  # a[0] / 2^ex in [1/2, 1)
    s = tail_bits(e)
    p = [int(mp.nint(a[k] * mp.mpf(2) ** ((62 if k < 4 else s) - ex))) for k in range(8)]
    assert all(abs(v) < (1 << 62 if k < 4 else 15 << 27) for k, v in enumerate(p)), (i, p)
    return ex, p, s


def wrap32(v):
    v &= 0xffffffff
    return v - (1 << 32) if v >> 31 else v


def evaluate(tab, bits):
    """The kernels' integer evaluation: f(q) as a double, from q's bits."""
    ex, p, s = tab[(bits >> (52 - MB)) - ((1023 + OCT_LO) << MB)]
    d = ((bits << (12 + MB)) & ((1 << 64) - 1)) ^ (1 << 63)
    d = d - (1 << 64) if d >> 63 else d
    dh = d >> 32
    t = p[7]
    for k in (6, 5, 4):
        t = wrap32(p[k] + ((t * dh) >> 32))
    acc = p[3] + ((t * dh) >> (s - 30))
    for k in (2, 1, 0):
        acc = p[k] + ((acc * d) >> 64)
    lz = 64 - acc.bit_length()
    m = ((acc << lz) + (1 << 10)) >> 11
    return float(m) * 2.0 ** (1 - lz + ex - 52)


def main():
    mp.mp.dps = 60
    tab = [interval(i) for i in range(NI)]
    mp.mp.dps = 40
    rng = random.Random(7)
    worst = {"q < 4": 0.0, "q >= 4, times g": 0.0}
    for i in range(NI):
        for _ in range(12):
            q = 2.0 ** (OCT_LO + (i >> MB)) * (1 + ((i & 63) + rng.random()) / 64)
            bits = int.from_bytes(__import__("struct").pack("<d", q), "little")
            f = g_over_u3(mp.mpf(q))
            rel = float(abs(mp.mpf(evaluate(tab, bits)) - f) / f)
            if q < 4:
                worst["q < 4"] = max(worst["q < 4"], rel)
            else:
                worst["q >= 4, times g"] = max(worst["q >= 4, times g"], rel * float(f * mp.mpf(q) ** 1.5))
    print("// Generated by fit_pair_fp64.py -- do not edit.")
    print("// f(q) = (erfc(u) + (2/sqrt(pi)) u exp(-u^2)) / u^3, q = u^2, on [2^%d, 2^%d): 64 intervals" % (OCT_LO, OCT_HI))
    print("// an octave, f = 2^E sum_k P[k] d^k (see the script).  Largest error of the rounded double over")
    print("// 12 random q per interval: relative %.3e (q < 4), times g %.3e (q >= 4)." % (
        worst["q < 4"], worst["q >= 4, times g"]))
    print("#pragma once")
    print("#define PAIR64_LO %d" % OCT_LO)
    print("#define PAIR64_MB %d" % MB)
    print("#define PAIR64_NI %d" % NI)

    def rows(name, what, cols):
        print("// " + what)
        print("#define %s \\" % name)
        cells = ["{" + ", ".join(c(t) for c in cols) + "}" if len(cols) > 1 else cols[0](t) for t in tab]
        per = {1: 16, 2: 3, 4: 3}[len(cols)]
        for i in range(0, NI, per):
            print("    %s%s, \\" % ("{" if i == 0 else " ", ", ".join(cells[i:i + per])))
        print("    }")

    rows("PAIR64_P01_INIT", "P[0], P[1]", [lambda t, k=k: "%dLL" % t[1][k] for k in (0, 1)])
    rows("PAIR64_P23_INIT", "P[2], P[3]", [lambda t, k=k: "%dLL" % t[1][k] for k in (2, 3)])
    rows("PAIR64_T_INIT", "P[4..7]", [lambda t, k=k: "%d" % t[1][k] for k in (4, 5, 6, 7)])
    rows("PAIR64_E_INIT", "(1023 + E) | (S - 30) << 16", [lambda t: "%d" % ((1023 + t[0]) | (t[2] - 30) << 16)])


if __name__ == "__main__":
    main()
