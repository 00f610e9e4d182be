"""Writes joker_trig_table.cuh: sin and cos of 2 pi k / 2048, k = 0..1024, and
2^(k / 512), k = 0..511, as integers at scale 2^61, each the integer nearest to
the exact value (60-digit mpmath evaluation).

The fixed-point Kepler solver starts its sin and cos series from these nodes,
the period draws their exponential series.  Run from any directory:

    python thejoker_gb300/csrc/gen_trig_table.py
"""
import os

import mpmath

N = 1025         # half a turn in steps of 1/2048 turn


def main():
    mpmath.mp.dps = 60
    rows = []
    for k in range(N):
        a = 2 * mpmath.pi * k / 2048
        s, c = (int(mpmath.nint(v * mpmath.mpf(2) ** 61)) for v in (mpmath.sin(a), mpmath.cos(a)))
        rows.append(f"    {{{s}LL, {c}LL}},")
    body = "\n".join(rows)
    powers = "\n".join(f"    {int(mpmath.nint(mpmath.mpf(2) ** (61 + mpmath.mpf(k) / 512)))}LL,"
                       for k in range(512))
    text = f"""// Generated by gen_trig_table.py: sin and cos of 2 pi k / 2048, k = 0..{N - 1},
// and 2^(k / 512), k = 0..511, times 2^61, each the nearest integer.  Do not
// edit.
#pragma once
#include <cstdint>

namespace joker {{
namespace fx {{

constexpr int TRIG_N = {N};

struct alignas(16) trig_entry {{ long long s, c; }};

#ifdef __CUDACC__
static __device__ const trig_entry kTrig[TRIG_N] = {{
#else
static const trig_entry kTrig[TRIG_N] = {{
#endif
{body}
}};

#ifdef __CUDACC__
static __device__ const long long kExp2[512] = {{
#else
static const long long kExp2[512] = {{
#endif
{powers}
}};

}}  // namespace fx
}}  // namespace joker
"""
    out = os.path.join(os.path.dirname(os.path.abspath(__file__)), "joker_trig_table.cuh")
    with open(out, "w") as f:
        f.write(text)
    print(f"wrote {out}")


if __name__ == "__main__":
    main()
