"""Writes fq_log_table.h for fq_log's quick phase (fq_math.h): table-driven reduction after Tang (1990),
"Table-driven implementation of the logarithm function in IEEE floating-point arithmetic".  Row i serves the
significands m in [1 + i/128, 1 + (i+1)/128); from i = 53 on, m/2 is taken, so that the logarithm of a number
just below 1 needs no cancellation.  c = 1/centre rounded to 20 bits (1 in the two rows beside 1), and -log(c)
as a double-double, from 60-digit mpmath.  Also ln 2 as a 40-bit part and the rest.
Run: python gen_log_table.py > fq_log_table.h"""

import mpmath as mp

mp.mp.dps = 60
N = 128
HALF = 53  # first row whose significands exceed sqrt(2)


def row(i):
    centre = 1 + (mp.mpf(i) + mp.mpf(1) / 2) / N
    if i >= HALF:
        centre /= 2
    c = mp.mpf(1) if i in (0, N - 1) else mp.nint((1 / centre) * 2**19) / 2**19
    v = -mp.log(c)
    hi = float(v)
    return float(c).hex(), hi.hex(), float(v - mp.mpf(hi)).hex()


def main():
    ln2 = mp.log(2)
    hi = mp.nint(ln2 * 2**40) / 2**40
    print("/* Generated by gen_log_table.py: c, -log(c) (hi, lo) per row, for fq_log's quick phase. */")
    print("#ifndef FQSB_FQ_LOG_TABLE_H\n#define FQSB_FQ_LOG_TABLE_H\n")
    print(f"#define FQ_LOG_N {N}\n#define FQ_LOG_HALF {HALF}")
    print(f"#define FQ_LOG_LN2_HI {float(hi).hex()}\n#define FQ_LOG_LN2_LO {float(ln2 - hi).hex()}\n")
    print("#define FQ_LOG_TABLE_INIT { \\")
    for i in range(N):
        c, h, lo = row(i)
        print(f"    {{{c}, {h}, {lo}, 0.0}}, \\")
    print("}\n\n#endif")


if __name__ == "__main__":
    main()
