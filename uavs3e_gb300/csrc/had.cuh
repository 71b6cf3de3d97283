// Hadamard magnitudes of com_had tiles on packed sample pairs, a tile row per lane.
//
// Columns c and c + 2 of a row travel in one register as d[c + 2] * 2^16 + d[c] (PRMT spreads the two
// bytes of a word into 16-bit lanes, one subtract of the packed org and prediction gives both
// differences; every value stays below 2^15 in magnitude, so integer adds, subtracts and negations keep
// both halves exact).  The stages of the transform commute: the row stages of distance 1 and 4 and the
// column stages (butterflies across the lanes of the tile) run on the pairs, and the row stage of
// distance 2, the one between the halves, is left to the end, where |lo + hi| + |lo - hi| =
// 2 max(|lo|, |hi|).
//
// Tiles of 2:1 shape: the 16-point (8-point) transform of [first | second] is [H(first) + H(second),
// H(first) - H(second)], so the tile's magnitudes are those of the two square transforms of the sum and
// of the difference of its halves.
#pragma once
#include "common.cuh"

namespace uc {

// signs of the three column butterflies of a lane: its own value enters with -1 where its bit is set
struct HadSigns { int s1, s2, s4; };
__device__ __forceinline__ HadSigns had_signs(int lane)
{
    return HadSigns{ 1 - 2 * (lane & 1), 1 - (lane & 2), 1 - ((lane & 4) >> 1) };
}

// the packed differences of 8 samples: columns (0, 2), (1, 3), (4, 6), (5, 7)
__device__ __forceinline__ void had_diff8(u32 ol, u32 oh, u32 pl, u32 ph, int (&q)[4])
{
    q[0] = (int)(__byte_perm(ol, 0u, 0x4240) - __byte_perm(pl, 0u, 0x4240));
    q[1] = (int)(__byte_perm(ol, 0u, 0x4341) - __byte_perm(pl, 0u, 0x4341));
    q[2] = (int)(__byte_perm(oh, 0u, 0x4240) - __byte_perm(ph, 0u, 0x4240));
    q[3] = (int)(__byte_perm(oh, 0u, 0x4341) - __byte_perm(ph, 0u, 0x4341));
}

// max(|lo|, |hi|) of a packed pair
__device__ __forceinline__ int had_pair_max(int v)
{
    const int lo = (int)(s16)(v & 0xFFFF), hi = (v - lo) >> 16;
    return max(abs(lo), abs(hi));
}

// a lane's share (its row after the transform) of the 8x8 magnitude sum, halved: 8 aligned lanes hold
// the 8 rows; the caller sums over them and doubles
__device__ __forceinline__ int had8_lane(const int (&q)[4], const HadSigns &S)
{
    const int a = q[0] + q[1], b = q[0] - q[1], c = q[2] + q[3], d = q[2] - q[3];
    int r[4] = { a + c, b + d, a - c, b - d };
#pragma unroll
    for (int i = 0; i < 4; i++) {
        r[i] = __shfl_xor_sync(0xffffffffu, r[i], 1) + S.s1 * r[i];
        r[i] = __shfl_xor_sync(0xffffffffu, r[i], 2) + S.s2 * r[i];
        r[i] = __shfl_xor_sync(0xffffffffu, r[i], 4) + S.s4 * r[i];
    }
    return had_pair_max(r[0]) + had_pair_max(r[1]) + had_pair_max(r[2]) + had_pair_max(r[3]);
}

// the same for 4x4: 4 aligned lanes hold the rows, q = columns (0, 2), (1, 3)
__device__ __forceinline__ int had4_lane(int q0, int q1, const HadSigns &S)
{
    int r[2] = { q0 + q1, q0 - q1 };
#pragma unroll
    for (int i = 0; i < 2; i++) {
        r[i] = __shfl_xor_sync(0xffffffffu, r[i], 1) + S.s1 * r[i];
        r[i] = __shfl_xor_sync(0xffffffffu, r[i], 2) + S.s2 * r[i];
    }
    return had_pair_max(r[0]) + had_pair_max(r[1]);
}

// 4 or 8 samples at p (any alignment) as little-endian words; only words that hold them are read
__device__ __forceinline__ u32 had_load4(const pel *p)
{
    const uintptr_t a = (uintptr_t)p;
    const u32 *q = (const u32 *)(a & ~(uintptr_t)3);
    const u32 sh = (u32)(a & 3) * 8;
    const u32 w0 = __ldg(q), w1 = sh ? __ldg(q + 1) : 0u;
    return __funnelshift_r(w0, w1, sh);
}
// (two 8-byte loads rather than three of 4: a warp's rows lie on 32 cache lines, and the L1 takes as
// long for either)
__device__ __forceinline__ void had_load8(const pel *p, u32 &lo, u32 &hi)
{
    const uintptr_t a = (uintptr_t)p;
    const uint2 *q = (const uint2 *)(a & ~(uintptr_t)7);
    const u32 off = (u32)(a & 7), sh = (off & 3) * 8;
    const uint2 x = __ldg(q), y = off ? __ldg(q + 1) : make_uint2(0u, 0u);
    const bool up = off >= 4;
    const u32 w0 = up ? x.y : x.x, w1 = up ? y.x : x.y, w2 = up ? y.y : y.x;
    lo = __funnelshift_r(w0, w1, sh);
    hi = __funnelshift_r(w1, w2, sh);
}

}  // namespace uc
