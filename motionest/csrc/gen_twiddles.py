"""Generate dft_consts.cuh: DFT twiddle constants as literals.

  python motionest/csrc/gen_twiddles.py   (run by motionest/build.py when the header is stale)

Emits, for every line length the compile-time FFT kernels support, a global device table
tw<N>[m] = exp(-2 pi i m / N) (m < N), initialised in the module image (no set-up kernel), the
same values in the order of the second FFT stage (twp<N>), and
for every small radix R the constants cos(2 pi m / R), sin(2 pi m / R) used by the register
DFTs.  The values are plain float64 evaluations of cos/sin rounded to float32.
"""
from pathlib import Path

import numpy as np

HERE = Path(__file__).resolve().parent
OUT = HERE / "dft_consts.cuh"

# Line lengths with a compile-time two-stage plan N = G * R1, G = 8 up to 128 points, else 16.
LENGTHS = [16, 24, 32, 48, 56, 64, 72, 88, 96, 112, 128, 144, 176, 192, 224, 256]
RADICES = [2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15, 16, 18, 20, 21, 22, 24, 25, 26, 27,
           28, 30, 32]


def f32(v):
    s = repr(float(np.float32(v)))
    if "e" not in s and "." not in s:
        s += ".0"
    return s + "f"


def main():
    lines = ["// Generated by gen_twiddles.py -- do not edit.", "#pragma once", "",
             "namespace me {", ""]
    lines.append("// Lengths with a compile-time plan (LineFft, fft_reg.cuh).")
    lines.append("#define ME_FAST_LENGTHS(X) \\")
    lines.append(" \\\n".join(f"  X({n})" for n in LENGTHS))
    lines.append("")
    for n in LENGTHS:
        m = np.arange(n)
        ang = -2.0 * np.pi * m / n
        vals = ", ".join(f"{{{f32(np.cos(a))}, {f32(np.sin(a))}}}" for a in ang)
        lines.append(f"__device__ const float2 tw{n}[{n}] = {{{vals}}};")
    lines.append("")
    lines.append("// The second-stage twiddles of each plan in the order the threads read them:")
    lines.append("// twp<N>[r R1 + k] = exp(-2 pi i r k / N), r < G, k < R1 = N / G.")
    for n in LENGTHS:
        g = 8 if n <= 128 else 16
        ang = [-2.0 * np.pi * (r * k) / n for r in range(g) for k in range(n // g)]
        vals = ", ".join(f"{{{f32(np.cos(a))}, {f32(np.sin(a))}}}" for a in ang)
        lines.append(f"__device__ const float2 twp{n}[{n}] = {{{vals}}};")
    lines.append("")
    lines.append("// cos / sin of 2 pi m / R for the register DFTs (m is a compile-time constant at")
    lines.append("// every call site after unrolling, so these fold to immediates)")
    lines.append("template <int R> struct RadixConst;")
    for r in RADICES:
        m = np.arange(r)
        c = ", ".join(f32(np.cos(2 * np.pi * k / r)) for k in m)
        s = ", ".join(f32(np.sin(2 * np.pi * k / r)) for k in m)
        lines.append(f"template <> struct RadixConst<{r}> {{")
        lines.append(f"  static __host__ __device__ __forceinline__ float c(int m) {{")
        lines.append(f"    constexpr float t[{r}] = {{{c}}};")
        lines.append("    return t[m];")
        lines.append("  }")
        lines.append(f"  static __host__ __device__ __forceinline__ float s(int m) {{")
        lines.append(f"    constexpr float t[{r}] = {{{s}}};")
        lines.append("    return t[m];")
        lines.append("  }")
        lines.append("};")
    lines.append("")
    lines.append("}  // namespace me")
    OUT.write_text("\n".join(lines) + "\n")
    return OUT


if __name__ == "__main__":
    print(main())
