"""Writes mpgb_fixed_tables.h: the series coefficients and tables of the
fixed-point exponential, logarithm and reciprocal in mpgb_fixed.cuh, from
60-digit decimal arithmetic (Python's decimal module), rounded once.

    python gen_fixed_tables.py > mpgb_fixed_tables.h
"""
from decimal import ROUND_CEILING, ROUND_HALF_EVEN, Decimal, getcontext

getcontext().prec = 60
LN2 = Decimal(2).ln()


def q(x, bits):
    return int((x * (Decimal(2) ** bits)).to_integral_value(ROUND_HALF_EVEN))


def main():
    out = ["// Generated by gen_fixed_tables.py; do not edit.", "#pragma once", "namespace mpgb {", "namespace fx {"]
    out.append(f"constexpr uint64_t kLog2e63 = 0x{q(1 / LN2, 63):016x}ull;  // log2(e), 63 fraction bits")
    # 1 - 2^-r = s (d1 - s (d2 - ...)), s = 16 r, d_n = (ln2/16)^n / n!
    fact, d = 1, []
    for n in range(1, 8):
        fact *= n
        d.append((LN2 / 16) ** n / fact)
    # log(1 + r) = s (l1 - s (l2 - ...)), s = 16 r, l_n = 1 / (n 16^n)
    lg = [Decimal(1) / (n * Decimal(16) ** n) for n in range(1, 11)]
    for name, v, wide in (("kE", d, 3), ("kL", lg, 4)):
        for n, x in enumerate(v, 1):
            if n <= wide:
                out.append(f"constexpr uint64_t {name}{n} = 0x{q(x, 64):016x}ull;  // 64 fraction bits")
            else:
                out.append(f"constexpr uint32_t {name}{n} = 0x{q(x, 53):08x}u;  // 53 fraction bits")
    out.append("// 2^(-j/32), 63 fraction bits (1 as the largest value below it).")
    t = [min(q((-LN2 * j / 32).exp(), 63), 2 ** 63 - 1) for j in range(32)]
    out.append("MPGB_FX_TABLE uint64_t kExpTab[32] = {")
    for i in range(0, 32, 4):
        out.append("    " + ", ".join(f"0x{v:016x}ull" for v in t[i:i + 4]) + ",")
    out.append("};")
    out.append("// inv: the smallest multiple of 2^-31 not below 1 / (1 + j/32), 31 fraction bits;")
    out.append("// lg: -log(inv), 63 fraction bits.")
    out.append("struct alignas(16) LogEntry { uint64_t lg; uint32_t inv, pad; };")
    out.append("MPGB_FX_TABLE LogEntry kLogTab[32] = {")
    for j in range(32):
        iv = int((Decimal(2) ** 31 / (1 + Decimal(j) / 32)).to_integral_value(ROUND_CEILING))
        out.append(f"    {{0x{q(-(Decimal(iv) / 2 ** 31).ln(), 63):016x}ull, 0x{iv:08x}u, 0u}},")
    out.append("};")
    out += ["}  // namespace fx", "}  // namespace mpgb"]
    print("\n".join(out))


if __name__ == "__main__":
    main()
