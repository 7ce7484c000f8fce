"""Writes trig_table_data.h: the quarter wave sin(2 pi j / N), j = 0 .. N/4, in Q62 (nearest), and the constants of
trig_table.h, from 60-digit arithmetic. Run: python gen_trig_table.py > trig_table_data.h"""
from mpmath import mp, mpf, floor, pi, sin

mp.dps = 60
LOG_N = 10
N = 1 << LOG_N


def q(v, bits):
    return int(floor(mpf(v) * mpf(2) ** bits + mpf(1) / 2))


a = pi / N  # half a table step, in radians
k = 1 / (2 * pi) / mpf(2) ** 16
words = [int(floor(k * mpf(2) ** (32 * (i + 1)))) & 0xFFFFFFFF for i in range(4)]
print("// Written by gen_trig_table.py: the quarter wave and the constants of trig_table.h.")
print("#pragma once\n\n#include <cstdint>\n")
print("namespace pgx\n{\nnamespace trigtab\n{\n")
print(f"constexpr int kLogN = {LOG_N};")
print("// sin and 1 - cos of t a, a = pi / N, as polynomials in z = t^2 (Taylor coefficients: |t a| <= 0.0031, the first")
print("// dropped terms are below 2^-75 and 2^-82)")
a1 = q(a ** 3 / 6, 73)
low = (a1 + 2 ** 31) % 2 ** 32 - 2 ** 31
print(f"constexpr int64_t kFineA0 = {q(a, 67)}LL;          // a, Q67")
print(f"constexpr int32_t kFineA1High = {(a1 - low) >> 32}, kFineA1Low = {low}; // a^3 / 6, Q73, in signed words")
print(f"constexpr uint32_t kFineA2 = {q(a ** 5 / 120, 74)}u;             // a^5 / 120, Q74")
print(f"constexpr int64_t kA0 = {q(a, 67) - 280}LL;              // a, Q67, less what the floored products below it take too little")
print(f"constexpr uint32_t kA1 = {q(a ** 3 / 6, 59)}u;               // a^3 / 6, Q59")
print(f"constexpr uint32_t kA2 = {q(a ** 5 / 120, 60)}u;                     // a^5 / 120, Q60")
print(f"constexpr int64_t kB0 = {q(a ** 2 / 2, 70) + 2}LL;               // a^2 / 2, Q70, likewise")
print(f"constexpr uint32_t kB1 = {q(a ** 4 / 24, 69)}u;               // a^4 / 24, Q69")
print(f"constexpr uint32_t kB2 = {q(a ** 6 / 720, 70)}u;                     // a^6 / 720, Q70")
print("// 2^-16 / (2 pi): its first 96 bits after the point, most significant word first")
print("constexpr uint32_t " + ", ".join(f"kInv2Pi{i} = 0x{w:08x}u" for i, w in enumerate(words[:3])) + ";")
hi = float(k)
print(f"constexpr double kInv2PiHi = {hi.hex()}, kInv2PiLo = {float(k - mpf(hi)).hex()}; // their sum, two doubles\n")
print(f"// sin(2 pi j / {N}) in Q62, j = 0 .. {N // 4}")
print(f"#define PGX_TRIG_QUARTER_WAVE \\")
vals = [q(sin(2 * pi * j / N), 62) for j in range(N // 4 + 1)]
lines = []
for i in range(0, len(vals), 5):
    lines.append("    " + " ".join(f"{v}LL," for v in vals[i:i + 5]))
print(" \\\n".join(lines))
print("\n} // namespace trigtab\n} // namespace pgx")
