"""Writes rnj_logtab_q.h: the table of the fused epilogue's logarithm
(rnj_device.cuh, neg_quarter_ln).  Table-driven reduction after P. T. P. Tang, ACM
TOMS 16(4), 1990, with 128 intervals of [kLnLow, 2 kLnLow), kLnLow =
0.70703125: the high word of z minus that of kLnLow, shifted, is the interval.
Per interval the reciprocal of its midpoint c (the double nearest to 1 / c)
and a quarter of that double's own logarithm, rounded once; the two intervals
that meet at 1 take the reciprocal 1 and the logarithm -0.0, so that arguments
next to 1 keep their relative precision and 1 itself gives -0.0.

Usage: python rapidnj_b200/csrc/gen_log_table_q.py > rapidnj_b200/csrc/rnj_logtab_q.h
"""
import struct
from decimal import Decimal
from fractions import Fraction

from gen_log_table import ln_decimal, nearest_double

OFF = 0x3FE6A000  # high word of kLnLow; (0x3FF00000 - OFF) / 8192 = 75 exactly


def double_of(hi: int) -> float:
    return struct.unpack("<d", struct.pack("<Q", hi << 32))[0]


def ln_any(x: Fraction) -> Decimal:
    d = Decimal(x.numerator) / Decimal(x.denominator)
    return ln_decimal(d) if d >= 1 else -ln_decimal(1 / d)


def main():
    print("// rnj_logtab_q.h -- generated by gen_log_table_q.py; do not edit.")
    print("// Per interval j of the fused epilogue's logarithm: {ln(inv) / 4, inv}, inv the double")
    print("// nearest to 1 / midpoint (1 and -0.0 in the two intervals that meet at 1).")
    print("#pragma once")
    print(f"constexpr unsigned int kLnOff = 0x{OFF:08X}u;  // high word of 0.70703125")
    print("constexpr int kLnIntervals = 128;")
    ln2 = 2 * ln_decimal(Decimal(2).sqrt())
    print(f"constexpr double kNegQuarterLn2 = {nearest_double(-ln2 / 4).hex()};")
    print("static __device__ __align__(16) const double c_log_tab_q[kLnIntervals][2] = {")
    for j in range(128):
        lo, hi = Fraction(double_of(OFF + j * 8192)), Fraction(double_of(OFF + (j + 1) * 8192))
        inv = 1.0 if j in (74, 75) else float(2 / (lo + hi))
        q = -0.0 if inv == 1.0 else nearest_double(ln_any(Fraction(inv)) / 4)
        print(f"    {{{q.hex()}, {inv.hex()}}},")
    print("};")


if __name__ == "__main__":
    main()
