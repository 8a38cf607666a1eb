"""Generate iexp_table.h: constants of the engine's fixed-point exponential.

exp(x), x <= 0, is evaluated on the integer pipes as 2^-|y| with
|y| = |x| log2(e) held with 64 fractional bits, m = ceil(|y|),
g = m - |y| = j/256 + s:  2^-|y| = 2^-m 2^(j/256) exp(s ln2).
Constants (computed here with mpmath at 80 digits, each rounded once):

  L2E_HI, L2E_LO  floor(log2(e) 2^127) as two 64-bit words
  L2E32           floor(log2(e) 2^31)
  LN2             nearest integer to ln2 2^64
  C2 .. C5        nearest integers to 2^63 / k!  (Taylor coefficients of exp)
  table[j]        nearest integer to 2^(j/256) 2^63, j = 0..255
  table1024[j]    nearest integer to exp(j/1024 - 2^-32) 2^62, j = 0..1023 (the
                  kernel-matrix build's variant, whose argument is reduced
                  by m ln2 and not scaled by log2(e); 0..710 are reached)
  fine1024[k]     nearest integer to expm1((k + 1/2)/2^20 + 2^-32) (2^64 + 2^12) + 1,
                  k = 0..1023 (its second table: the rest, within +-2^-21,
                  needs a degree-2 polynomial only).  The 2^-32 keeps
                  exp - 1 of both lower parts together positive; 2^12 and 1
                  centre the truncations of their product and of the square

Run: python gen_iexp_table.py > iexp_table.h
"""
import mpmath as mp

mp.mp.dps = 80
L = int(mp.floor(mp.mpf(2) ** 127 / mp.log(2)))
LN2 = int(mp.nint(mp.log(2) * mp.mpf(2) ** 64))
C = {k: int(mp.nint(mp.mpf(2) ** 63 / mp.factorial(k))) for k in range(2, 6)}
tab = [int(mp.nint(mp.mpf(2) ** (mp.mpf(j) / 256 + 63))) for j in range(256)]
SHIFT = mp.mpf(2) ** -32
tab1024 = [int(mp.nint(mp.exp(mp.mpf(j) / 1024 - SHIFT) * mp.mpf(2) ** 62)) for j in range(1024)]
fine1024 = [int(mp.nint(mp.expm1((mp.mpf(k) + 0.5) / 2 ** 20 + SHIFT) * (mp.mpf(2) ** 64 + 2 ** 12) + 1))
            for k in range(1024)]
L2E32 = int(mp.floor(mp.mpf(2) ** 31 / mp.log(2)))
print("// Generated by gen_iexp_table.py (constants of the fixed-point exponential).")
print("#pragma once")
print(f"#define IEXP_L2E_HI 0x{L >> 64:016x}ULL  // floor(log2(e) 2^127), high word")
print(f"#define IEXP_L2E_LO 0x{L & ((1 << 64) - 1):016x}ULL  // low word")
print(f"#define IEXP_L2E32 0x{L2E32:08x}u  // floor(log2(e) 2^31)")
print(f"#define IEXP_LN2 0x{LN2:016x}ULL     // ln2 2^64")
for k in range(2, 6):
    print(f"#define IEXP_C{k} 0x{C[k]:016x}ULL      // 2^63 / {k}!")
print("// 2^(j/256) 2^63")
print("static __device__ const unsigned long long g_iexp_tab[256] = {")
for j in range(0, 256, 4):
    print("    " + ", ".join(f"0x{t:016x}ULL" for t in tab[j:j + 4]) + ",")
print("};")
print("// exp(j/1024 - 2^-32) 2^62")
print("static __device__ const unsigned long long g_iexp_tab1024[1024] = {")
for j in range(0, 1024, 4):
    print("    " + ", ".join(f"0x{t:016x}ULL" for t in tab1024[j:j + 4]) + ",")
print("};")
print("// expm1((k + 1/2)/2^20 + 2^-32) (2^64 + 2^12) + 1")
print("static __device__ const unsigned long long g_iexp_fine1024[1024] = {")
for k in range(0, 1024, 4):
    print("    " + ", ".join(f"0x{t:016x}ULL" for t in fine1024[k:k + 4]) + ",")
print("};")
