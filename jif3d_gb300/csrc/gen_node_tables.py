"""Generate node_tables.h: the breakpoint tables of the fixed-point logarithm
and arctangent in node_fixed.cuh, computed here at 60 significant digits with
mpmath.

* Logarithm -- for m in [1, 2) and j = floor((m - 1) 512): a 32-bit
  multiplier G_j = round(2^32 / (1 + (j + 1/2) / 512)), so that m G_j 2^-32 - 1
  is below 2^-9.99 in magnitude, and -log(G_j 2^-32) at scale 2^57.
* Arctangent -- atan(j/1024) at scale 2^63, j = 0..1024.

Run:  python jif3d_gb300/csrc/gen_node_tables.py   (rewrites node_tables.h)
"""
import os

import mpmath as mp

mp.mp.dps = 60
HERE = os.path.dirname(os.path.abspath(__file__))
LOG_N, ATAN_N, LOG_BIAS = 512, 1024, 128


def main():
    ln2 = int(mp.floor(mp.log(2) * 2 ** 89))  # scale 2^57, 32 further bits
    G = [int(mp.nint(2 ** 32 / (1 + (mp.mpf(j) + 0.5) / LOG_N))) for j in range(LOG_N)]
    L = [int(mp.nint(-mp.log(mp.mpf(g) / 2 ** 32) * 2 ** 57)) for g in G]
    A = [int(mp.nint(mp.atan(mp.mpf(j) / ATAN_N) * 2 ** 63)) for j in range(ATAN_N + 1)]

    def rows(v, width, suffix):
        out = []
        for i in range(0, len(v), 4):
            out.append("    " + ", ".join(f"0x{x:0{width}x}{suffix}" for x in v[i:i + 4]) + ",")
        return out
    lines = [
        "// node_tables.h -- generated by gen_node_tables.py; do not edit.",
        "// Tables of the fixed-point logarithm (multipliers G_j at scale 2^32 and",
        "// -log G_j at scale 2^57) and arctangent (atan(j/1024) at scale 2^63).",
        "#pragma once",
        "#include <cstdint>",
        "",
        "#ifdef __CUDACC__",
        "#define J3G_TABLE __device__ const",
        "#else",
        "#define J3G_TABLE static const",
        "#endif",
        "",
        "namespace j3g {",
        "namespace nodetab {",
        "",
        f"constexpr int kLogN = {LOG_N};",
        f"constexpr int kAtanN = {ATAN_N};",
        f"constexpr int kLogBias = {LOG_BIAS};",
        f"constexpr uint64_t kLn2 = 0x{ln2 >> 32:016x}ull;   // log 2, scale 2^57",
        f"constexpr uint32_t kLn2Low = 0x{ln2 & 0xffffffff:08x}u;  // its next 32 bits",
        f"constexpr uint64_t kPio2S61 = 0x{int(mp.nint(mp.pi / 2 * 2 ** 61)):016x}ull;  // pi/2, scale 2^61",
        f"constexpr uint64_t kPiS61 = 0x{int(mp.nint(mp.pi * 2 ** 61)):016x}ull;    // pi, scale 2^61",
        "",
        f"J3G_TABLE uint32_t kLogG[{LOG_N}] = {{",
    ] + rows(G, 8, "u") + ["};", f"J3G_TABLE uint64_t kLogL[{LOG_N}] = {{"] + rows(L, 16, "ull") + [
        "};", f"J3G_TABLE uint64_t kAtan[{ATAN_N + 1}] = {{"] + rows(A, 16, "ull") + [
        "};", "", "}  // namespace nodetab", "}  // namespace j3g", "", "#undef J3G_TABLE", ""]
    with open(os.path.join(HERE, "node_tables.h"), "w") as f:
        f.write("\n".join(lines))


if __name__ == "__main__":
    main()
