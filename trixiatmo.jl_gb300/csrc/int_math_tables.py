"""Constants of int_math.cuh, from their definitions in 60-digit arithmetic.

Run as a script to print int_math_tables.cuh:
  kLogTable[i] = (-log2(y_i / 512) in Q0.63, y_i), y_i = round(512 / (1 + (i + 1/2)/128)):
      the reciprocal table of a table-driven logarithm (P. T. P. Tang, ACM TOMS 16 (1990) 378-400);
  kExp2Table[j] = 2^(j/128) in Q1.63 (P. T. P. Tang, ACM TOMS 15 (1989) 144-157);
  the Taylor coefficients of log2(1 + f), 2^r, tanh(x)/x and x/sinh(x) in the forms the code uses.
"""
import mpmath as mp

mp.mp.dps = 60
LN2 = mp.log(2)
TERMS = 13  # of the even series; the first FIXED in integers, the others in binary32
FIXED = 7


def fix(x, bits):
    return int(mp.nint(mp.mpf(x) * mp.mpf(2) ** bits))


def log_table():
    rows = []
    for i in range(128):
        y = int(mp.nint(512 / (1 + (mp.mpf(i) + mp.mpf("0.5")) / 128)))
        rows.append((fix(-mp.log(mp.mpf(y) / 512, 2), 63), y))
    return rows


def exp2_table():
    return [fix(mp.mpf(2) ** (mp.mpf(j) / 128), 63) for j in range(128)]


def series_coefficients(name):
    """tanh(x)/x at x = d ln2 / 2 ("ln") and x/sinh(x) at x = d ln2 ("inv"), in z = d^2."""
    # tanh(x)/x = sum 2^(2n)(2^(2n)-1) B_2n / (2n)! x^(2n-2); x/sinh(x) = sum 2(1-2^(2n-1)) B_2n x^2n/(2n)!
    out = []
    for k in range(TERMS):
        n = k + 1
        if name == "ln":
            m = n + 1
            c = mp.mpf(4) ** m * (mp.mpf(4) ** m - 1) * mp.bernoulli(2 * m) / mp.factorial(2 * m)
            out.append(-c * (LN2 / 2) ** (2 * n))
        else:
            c = 2 * (1 - mp.mpf(2) ** (2 * n - 1)) * mp.bernoulli(2 * n) / mp.factorial(2 * n)
            out.append(-c * LN2 ** (2 * n))
    return out


def main():
    print("// Written by int_math_tables.py; do not edit.")
    print("#pragma once")
    print("namespace tag {")
    print("#define TAG_LOG_TABLE \\")
    print(", \\\n".join("  {%dull, %dull}" % r for r in log_table()))
    print("#define TAG_EXP2_TABLE \\")
    print(", \\\n".join("  %dull" % v for v in exp2_table()))
    for name in ("ln", "inv"):
        a = series_coefficients(name)
        # alternating series: the magnitudes, Q0.64 and binary32
        for k in range(FIXED):
            print("#define TAG_%s_A%d %dull" % (name.upper(), k, fix(abs(a[k]), 64)))
        for k in range(FIXED, TERMS):
            print("#define TAG_%s_B%d %sf" % (name.upper(), k - FIXED, mp.nstr(abs(a[k]), 10)))
    for k in (1, 2, 3):
        print("#define TAG_LOG2_C%d %dll" % (k, fix((-1) ** (k + 1) / (k * LN2), 62)))
    for k in (4, 5, 6, 7):
        print("#define TAG_LOG2_C%d %sf" % (k, mp.nstr((-1) ** (k + 1) / (k * LN2), 10)))
    for k in (1, 2, 3):
        print("#define TAG_EXP2_C%d %dll" % (k, fix(LN2 ** k / mp.factorial(k), 63)))
    for k in (4, 5, 6):
        print("#define TAG_EXP2_C%d %sf" % (k, mp.nstr(LN2 ** k / mp.factorial(k), 10)))
    print("#define TAG_LOG2E_Q62 %dll" % fix(1 / LN2, 62))
    print("#define TAG_RAINY_LOG2_REF %dll" % fix(mp.log(mp.mpf("273.15"), 2), 58))
    print("#define TAG_LN2_Q64 %dull" % fix(LN2, 64))
    print("}  // namespace tag")


if __name__ == "__main__":
    main()
