// Per-call motion search of the encoder, batched: me_search_tz (src/me.c:529-568) for a list of
// independent calls (block, reference, predictor, MV resolution, bi-prediction state), each
// bit-exact with the reference's call on the same state.
//
// One warp per call.  The org block (or, for a bi call, 2 org - the other list's prediction,
// create_bi_org src/inter.c:55) sits in shared memory.  The search's stages run one after the
// other -- first diamond, raster grids, refinement diamond (search_diamond :199, search_raster
// :103, get_raster_range :65) -- and each stage's candidates, in the reference's visit order,
// are costed 32 at a time (a SAD per lane; the rows of few candidates split between the lanes); the
// stage keeps the minimum of (cost << 20 | visit position) and moves the running best only when that
// minimum is strictly smaller, as the reference's sequence of strict updates does.  The fractional
// refinement (me_sub_pel_search :366-500) costs its centre and 8 half-sample points in one batch, then
// 8 quarter-sample points, with the rows of the com_had tiles spread over the lanes (had.cuh; per-lane
// SADs for subpel_cost_type 1), and keeps the first of the smallest.
//
// The 170,220 calls of a 1080p frame (10 shapes, 2 references, 30 % bi) take 1.68 ms, bound by the L1
// (81 % of its throughput: a warp's loads lie on up to 32 lines).  With every stage its own inlined copy
// of the SAD and of six SATD tile shapes (204 KB of code, half the time spent waiting for
// instructions), SATD samples read byte by byte and small stages on 9 of 32 lanes it was 3.35 ms.
#include "common.cuh"
#include "had.cuh"
#include "uavs3e_cuda_internal.h"
#include "../../include/uavs3e_cuda.h"

#include <algorithm>
#include <math.h>
#include <string.h>

namespace uc {

constexpr int TZ_KEY_BITS = 20;

struct TzReq {
    s16 x, y; u8 w, h; u8 ref_slot; s8 refi; u8 num_refp; u8 mvr; u8 bi; u8 flags;
    s16 mvp[2]; s16 mv[2]; s16 mv_ipel[2]; s16 other_mv[2]; u8 other_slot; u8 pad0[3];
    s32 mot_bits_other; u32 lambda_mv; s32 dist; s32 pad1;
};
struct TzOut { s16 mv[2]; s16 mv_ipel[2]; u64 cost; };
static_assert(sizeof(TzReq) == sizeof(uavs3e_cuda_tz_req_t), "request layout");
static_assert(sizeof(TzOut) == sizeof(uavs3e_cuda_tz_out_t), "result layout");

struct TzParams {
    const pel *planes[UAVS3E_CUDA_TZ_MAX_SLOTS * 16];   // sample (0,0) of each slot's 16 planes
    const pel *org;
    int i_org, i_ref, n_slots;
    int W, H, is_padding, max_search_range, gop_size, mto;
    const TzReq *reqs;
    int n;
    TzOut *out;
    double sq32, sq128;
    u64 k32, k128;       // had_scale_k of sq32, sq128
};

// search_diamond's ring points (src/me.c:307-331) at MV resolution <= integer: step 4, 8, 16
__device__ __constant__ static const s8 kTzRing[28][3] = {
    { -4, 0, 4 }, { 0, 4, 4 }, { 4, 0, 4 }, { 0, -4, 4 },
    { -8, 0, 8 }, { -4, 4, 8 }, { 0, 8, 8 }, { 4, 4, 8 }, { 8, 0, 8 }, { 4, -4, 8 }, { 0, -8, 8 }, { -4, -4, 8 },
    { -16, 0, 16 }, { -12, 4, 16 }, { -8, 8, 16 }, { -4, 12, 16 }, { 0, 16, 16 }, { 4, 12, 16 }, { 8, 8, 16 },
    { 12, 4, 16 }, { 16, 0, 16 }, { 12, -4, 16 }, { 8, -8, 16 }, { 4, -12, 16 }, { 0, -16, 16 }, { -4, -12, 16 },
    { -8, -8, 16 }, { -12, -4, 16 },
};
// me_sub_pel_search's patterns (src/me.c:413-415, :451-453)
__device__ __constant__ static const s8 kTzHalf[8][2] = { { -2, 0 }, { -2, 2 }, { 0, 2 }, { 2, 2 },
                                                         { 2, 0 }, { 2, -2 }, { 0, -2 }, { -2, -2 } };
__device__ __constant__ static const s8 kTzQuar[8][2] = { { -1, 0 }, { 0, 1 }, { 1, 0 }, { 0, -1 },
                                                         { -1, 1 }, { 1, 1 }, { -1, -1 }, { 1, -1 } };

// MV bits at table index v (inter_search_create, src/inter.c:2029-2057)
__device__ __forceinline__ u32 tz_bits(int v)
{
    return v == 0 ? 1u : 2u * (32u - (u32)__clz(abs(v) + 1));
}

// a refinement batch's candidates: sample (0, 0) of the block in the plane of each
struct TzShared {
    __align__(16) u32 org[64 * 64 / 4];   // the block searched against, wq words per row
    const pel *ptr[9];
    u32 sum[9];
};

// the N + 1 words that hold 4 N samples from address a on, from aligned 8-byte loads
template <int N>
__device__ __forceinline__ void tz_row(uintptr_t a, u32 (&w)[N + 1])
{
    const uint2 *q = (const uint2 *)(a & ~(uintptr_t)7);
    const bool up = a & 4;            // the first word is the upper one of its 8 bytes
    uint2 x[N / 2 + 1];
#pragma unroll
    for (int i = 0; i < N / 2 + 1; i++) x[i] = __ldg(q + i);
#pragma unroll
    for (int i = 0; i < N + 1; i++) {
        const u32 lo = i & 1 ? x[i / 2].y : x[i / 2].x;
        const u32 hi = i == N ? x[N / 2].y : (i & 1 ? x[i / 2 + 1].x : x[i / 2].y);
        w[i] = up ? hi : lo;
    }
}

// SAD of rows [0, rows) of a block of wq words per row: org at so, candidate at p (its rows `stride` samples
// apart, a multiple of 4).  The reads span at most 8 samples beyond either end of a row, inside the planes'
// padding.  The L1 is the busiest unit of the search (a row's load touches up to 32 lines): 8-byte loads
// halve its requests.  Two rows of narrow blocks, 32 samples of wide ones are in flight together.
__device__ __noinline__ u32 tz_sad(const u32 *so, int wq, int rows, const pel *p, int stride)
{
    uintptr_t a = (uintptr_t)p;
    const u32 sh = (u32)(a & 3) * 8;
    u32 s = 0;
    if (wq >= 8) {
#pragma unroll 1
        for (int r = 0; r < rows; r++, a += stride, so += wq) {
#pragma unroll 1
            for (int c = 0; c < wq; c += 8) {
                u32 w[9];
                tz_row<8>(a + 4 * c, w);
                const uint4 oa = *reinterpret_cast<const uint4 *>(so + c), ob = *reinterpret_cast<const uint4 *>(so + c + 4);
                s = sad4(oa.x, __funnelshift_r(w[0], w[1], sh), s);
                s = sad4(oa.y, __funnelshift_r(w[1], w[2], sh), s);
                s = sad4(oa.z, __funnelshift_r(w[2], w[3], sh), s);
                s = sad4(oa.w, __funnelshift_r(w[3], w[4], sh), s);
                s = sad4(ob.x, __funnelshift_r(w[4], w[5], sh), s);
                s = sad4(ob.y, __funnelshift_r(w[5], w[6], sh), s);
                s = sad4(ob.z, __funnelshift_r(w[6], w[7], sh), s);
                s = sad4(ob.w, __funnelshift_r(w[7], w[8], sh), s);
            }
        }
    } else if (wq == 4) {
#pragma unroll 1
        for (int r = 0; r < rows; r += 2, a += 2 * stride, so += 8) {
#pragma unroll
            for (int k = 0; k < 2; k++) {
                u32 w[5];
                tz_row<4>(a + k * stride, w);
                const uint4 o = *reinterpret_cast<const uint4 *>(so + 4 * k);
                s = sad4(o.x, __funnelshift_r(w[0], w[1], sh), s);
                s = sad4(o.y, __funnelshift_r(w[1], w[2], sh), s);
                s = sad4(o.z, __funnelshift_r(w[2], w[3], sh), s);
                s = sad4(o.w, __funnelshift_r(w[3], w[4], sh), s);
            }
        }
    } else if (wq == 2) {
#pragma unroll 1
        for (int r = 0; r < rows; r += 2, a += 2 * stride, so += 4) {
            const uint4 o = *reinterpret_cast<const uint4 *>(so);
            u32 v[3], w[3];
            tz_row<2>(a, v);
            tz_row<2>(a + stride, w);
            s = sad4(o.x, __funnelshift_r(v[0], v[1], sh), s);
            s = sad4(o.y, __funnelshift_r(v[1], v[2], sh), s);
            s = sad4(o.z, __funnelshift_r(w[0], w[1], sh), s);
            s = sad4(o.w, __funnelshift_r(w[1], w[2], sh), s);
        }
    } else {
#pragma unroll 1
        for (int r = 0; r < rows; r++, a += stride, so++) {
            const u32 *q = (const u32 *)(a & ~(uintptr_t)3);
            s = sad4(*so, __funnelshift_r(__ldg(q), __ldg(q + 1), sh), s);
        }
    }
    return s;
}

// how many lanes (as a power of two) share a candidate when n are costed: the block's rows are split
// between them while all candidates still fit the warp and a lane keeps 4 rows
__device__ __forceinline__ int tz_split(int n, int h)
{
    int lg = 0;
    while (lg < 3 && (n << (lg + 1)) <= 32 && (h >> (lg + 1)) >= 4) lg++;
    return lg;
}

// sum over the 2^lg lanes that share a candidate
__device__ __forceinline__ u32 tz_split_sum(u32 v, int lg)
{
    for (int d = 1; d < (1 << lg); d <<= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
    return v;
}

__device__ __forceinline__ u64 tz_key(u64 cost, int k) { return (cost << TZ_KEY_BITS) | (u64)k; }

// com_mc_blk_luma_pointer (src/com_mc.c:89-101) into a slot's planes
__device__ __forceinline__ const pel *tz_mc_ptr(const TzParams &P, int slot, int qx, int qy)
{
    const int px = min(max(qx >> 2, -128 - 4), P.W + 4), py = min(max(qy >> 2, -128 - 4), P.H + 4);
    return P.planes[slot * 16 + (qy & 3) * 4 + (qx & 3)] + (long long)py * P.i_ref + px;
}

// candidate k of a refinement batch: pattern 0 = centre + the 8 half-sample points, 1 = the 8
// quarter-sample points, 2 = the centre alone
__device__ __forceinline__ void tz_sub_mv(int pattern, int k, int cx, int cy, int &vx, int &vy)
{
    if (pattern == 1) { vx = cx + kTzQuar[k][0]; vy = cy + kTzQuar[k][1]; }
    else if (pattern == 0 && k > 0) { vx = cx + kTzHalf[k - 1][0]; vy = cy + kTzHalf[k - 1][1]; }
    else { vx = cx; vy = cy; }
}

// com_had of nc candidates (com_had_4x4 .. _16x8, src/com_cost.c:176-812): the rows of every
// candidate's tiles spread over the lanes (had.cuh), R = 8 or 4 lanes to a tile.  Sides are powers of
// two, so a task number splits into (candidate, tile, row) by shifts.
template <int R>
__device__ __forceinline__ void tz_had(TzShared &S, const TzParams &P, int lw, int lh, int nc, int lane)
{
    constexpr int LR = R == 8 ? 3 : 2;
    const HadSigns G = had_signs(lane);
    const bool wide = lw > lh, pair = lw != lh;
    const int lntx = lw - LR - (wide ? 1 : 0), lnt = lntx + lh - LR - (pair && !wide ? 1 : 0);
    const int w = 1 << lw, i_ref = P.i_ref;
    const int po = wide ? R : R << lw, pr = wide ? R : R * i_ref;   // the second half of a 2:1 tile
    const pel *org = (const pel *)S.org;
    const int total = nc << (lnt + LR);
#pragma unroll 1
    for (int base = 0; base < total; base += 32) {
        const int t = base + lane;
        const bool active = t < total;                 // a tile's lanes are active together
        const int tt = active ? t : (lane & (R - 1));
        const int row = tt & (R - 1), tile = (tt >> LR) & ((1 << lnt) - 1), k = tt >> (LR + lnt);
        const int ox = (tile & ((1 << lntx) - 1)) << (LR + (wide ? 1 : 0));
        const int oy = ((tile >> lntx) << (LR + (pair && !wide ? 1 : 0))) + row;
        const pel *o = org + oy * w + ox, *p = S.ptr[k] + oy * i_ref + ox;
        int s;
        if (R == 8) {
            u32 pl, ph;
            int q[4];
            had_load8(p, pl, ph);
            const uint2 ov = *reinterpret_cast<const uint2 *>(o);
            had_diff8(ov.x, ov.y, pl, ph, q);
            if (pair) {
                int e[4], d[4];
                had_load8(p + pr, pl, ph);
                const uint2 ow = *reinterpret_cast<const uint2 *>(o + po);
                had_diff8(ow.x, ow.y, pl, ph, e);
#pragma unroll
                for (int i = 0; i < 4; i++) { d[i] = q[i] - e[i]; q[i] += e[i]; }
                s = had8_lane(d, G);
                s += had8_lane(q, G);
            } else {
                s = had8_lane(q, G);
            }
        } else {
            const u32 pv = had_load4(p), ov = *reinterpret_cast<const u32 *>(o);
            int q0 = (int)(__byte_perm(ov, 0u, 0x4240) - __byte_perm(pv, 0u, 0x4240));
            int q1 = (int)(__byte_perm(ov, 0u, 0x4341) - __byte_perm(pv, 0u, 0x4341));
            if (pair) {
                const u32 pw = had_load4(p + pr), ow = *reinterpret_cast<const u32 *>(o + po);
                const int e0 = (int)(__byte_perm(ow, 0u, 0x4240) - __byte_perm(pw, 0u, 0x4240));
                const int e1 = (int)(__byte_perm(ow, 0u, 0x4341) - __byte_perm(pw, 0u, 0x4341));
                s = had4_lane(q0 - e0, q1 - e1, G);
                s += had4_lane(q0 + e0, q1 + e1, G);
            } else {
                s = had4_lane(q0, q1, G);
            }
        }
#pragma unroll
        for (int m = 1; m < R; m <<= 1) s += __shfl_xor_sync(0xffffffffu, s, m);
        s *= 2;
        if (active && row == 0) {
            const u32 v = !pair ? (u32)(R == 8 ? (s + 2) >> 2 : (s + 1) >> 1)
                                : (R == 8 ? had_scale(s, P.sq128, P.k128) : had_scale(s, P.sq32, P.k32));
            atomicAdd(&S.sum[k], v);
        }
    }
}

// One warp per CTA: calls differ widely in length, and a warp's slot frees as soon as its call ends.
// The search is one loop over its stages and the refinement one loop over its batches, each with a
// single copy of the SAD and SATD code: with the stages as separate inlined copies the kernel was 204 KB
// of code and waited for instructions half of its time.
__global__ void __launch_bounds__(32, 32) k_me_tz(const TzParams P)
{
    __shared__ TzShared S;
    const int lane = threadIdx.x;
    const int r = blockIdx.x;
    const TzReq q = P.reqs[r];
    TzOut o;
    o.mv[0] = q.mv[0]; o.mv[1] = q.mv[1];
    o.mv_ipel[0] = q.mv_ipel[0]; o.mv_ipel[1] = q.mv_ipel[1];
    const int x = q.x, y = q.y, w = q.w, h = q.h, mvr = q.mvr, bi = q.bi;
    // The predictor by two 16-bit loads of its own.  As q.mvp[1], the upper halfword of a loaded word, it was 0
    // in every use of one version of this kernel, while a second read of the record gave the right value:
    // with ptxas 13.0 at -O2 and -O3, not at -O1 and -O0, whatever nvcc's own level; a register made opaque
    // where the value is used was 0 too.
    const volatile s16 *mvp = P.reqs[r].mvp;
    const int mvpx = mvp[0], mvpy = mvp[1];
    // calls outside the supported domain (block inside the picture, sides 4..64 powers of two,
    // known slots, resolution 0..4) come back with cost UINT64_MAX and their MVs unchanged
    const bool pow2 = (w & (w - 1)) == 0 && (h & (h - 1)) == 0;
    if (!pow2 || w < 4 || w > 64 || h < 4 || h > 64 || x < 0 || y < 0 || x + w > P.W || y + h > P.H || mvr > 4 ||
        q.ref_slot >= P.n_slots || (bi && q.other_slot >= P.n_slots) || q.refi < 0 || q.refi > 15 ||
        q.num_refp > 16) {
        o.cost = ~0ull;
        if (lane == 0) P.out[r] = o;
        return;
    }
    // get_max_search_range (src/me.c:502-527), com_ipel_range_rounding above integer resolution
    const int mt = (P.mto << mvr) >> 2, px = mvpx >> 2, py = mvpy >> 2;
    int minx, maxx, miny, maxy;
    if (P.is_padding) {
        minx = max(-127 - x, px - mt + 4); miny = max(-127 - y, py - mt + 4);
        maxx = min(P.W - 1 - x, px + mt - 4); maxy = min(P.H - 1 - y, py + mt - 4);
    } else {
        minx = max(-x, px - mt + 4); miny = max(-y, py - mt + 4);
        maxx = min(P.W - 1 - x - w, px + mt - 4); maxy = min(P.H - 1 - y - h, py + mt - 4);
    }
    const int msh = max(mvr - 2, 0);          // log2 of the MV step in samples
    if (msh) {
        minx = minx >= 0 ? (minx >> msh) << msh : -(((-minx) >> msh) << msh);
        miny = miny >= 0 ? (miny >> msh) << msh : -(((-miny) >> msh) << msh);
        maxx = maxx >= 0 ? (maxx >> msh) << msh : -(((-maxx) >> msh) << msh);
        maxy = maxy >= 0 ? (maxy >> msh) << msh : -(((-maxy) >> msh) << msh);
    }
    if (minx > maxx || miny > maxy) {
        o.cost = ~0ull;
        if (lane == 0) P.out[r] = o;
        return;
    }
    const int lw = 31 - __clz(w), lh = 31 - __clz(h), wq = w >> 2;
    // the block searched against: org, or 2 org - the other list's prediction (clipped, byte-wise:
    // s + (s - p) where s >= p, else s - (p - s))
    {
        const pel *og = P.org + (long long)y * P.i_org + x;
        const pel *pr = bi ? tz_mc_ptr(P, q.other_slot, (x << 2) + q.other_mv[0], (y << 2) + q.other_mv[1]) : og;
#pragma unroll 1
        for (int i = lane; i < wq * h; i += 32) {
            const int rr = i >> (lw - 2), c = (i & (wq - 1)) * 4;
            u32 v = had_load4(og + rr * P.i_org + c);
            if (bi) {
                const u32 pv = had_load4(pr + rr * P.i_ref + c);
                v = __vsubus4(__vaddus4(v, __vsubus4(v, pv)), __vsubus4(pv, v));
            }
            S.org[i] = v;
        }
    }
    __syncwarp();
    const pel *ref = P.planes[q.ref_slot * 16] + (long long)y * P.i_ref + x;
    const int shift = 16 - bi;
    const int bpx = mvpx >> mvr, bpy = mvpy >> mvr;   // predictor at the MV-bits table's resolution
    const u32 lambda = q.lambda_mv;
    int mvx = min(max(((bi ? q.mv[0] : mvpx) + 2) >> 2, minx), maxx);
    int mvy = min(max(((bi ? q.mv[1] : mvpy) + 2) >> 2, miny), maxy);
    u64 best = ~0ull;
    // The stages: a diamond (search_diamond, src/me.c:199-334: centre, core square, rings below its
    // largest step), for far winners the raster grids (search_raster :103-197) with get_raster_range's
    // window, then a small diamond.  Each is a list of candidates in the reference's visit order: the
    // centre (n0 = 1), the grid x0 + i g, y0 + j g (nx x ny, rows outer), the ring points.
    int stage = 0, step = 0, smin = 1, rx = 0, ry = 0;
    for (;;) {
        const int cx = mvx, cy = mvy;
        int x0, y0, x1, y1, g, n0, n_ring;
        if (stage == 1) {                     // a raster grid: the whole window, then around the best
            x0 = max(cx - rx, minx); x1 = min(cx + rx, maxx);
            y0 = max(cy - ry, miny); y1 = min(cy + ry, maxy);
            g = step; n0 = 0; n_ring = 0;
        } else {
            int core = bi ? 5 : 2;
            if (bi) {
                if (mvr > 2) core++;
                const int ix = (mvpx + 2) >> 2, iy = (mvpy + 2) >> 2;
                const int diff = max(abs(ix - cx), abs(iy - cy)) >> msh;
                core = min(max(diff, 2), core);
            }
            core <<= msh;
            g = 1 << msh;
            x0 = cx - core; y0 = cy - core; x1 = cx + core; y1 = cy + core;
            while (x0 <= minx) x0 += g;
            while (y0 <= miny) y0 += g;
            while (x1 >= maxx) x1 -= g;
            while (y1 >= maxy) y1 -= g;
            n0 = 1;
            n_ring = bi ? 0 : (stage == 0 ? 28 : 4);     // largest step 32 / 8
        }
        const int nx = x1 >= x0 ? (x1 - x0) / g + 1 : 0, ny = y1 >= y0 ? (y1 - y0) / g + 1 : 0;
        const int ngrid = nx * ny, n = n0 + ngrid + n_ring;
        // j / nx = umulhi(j, inv) for j nx < 2^32 and nx > 1
        const u32 inv = nx > 1 ? 0xFFFFFFFFu / (u32)nx + 1u : 0u;
        const auto place = [&](int k, int &mx, int &my) {
            const int j = k - n0, jr = j - ngrid;
            const int row = nx > 1 ? (int)__umulhi((u32)j, inv) : j;
            mx = x0 + (j - row * nx) * g;
            my = y0 + row * g;
            if (j < 0) { mx = cx; my = cy; }
            if (jr >= 0) { mx = cx + (kTzRing[jr][0] << msh); my = cy + (kTzRing[jr][1] << msh); }
        };
        const int lg = tz_split(n, h), rows = h >> lg, part = lane & ((1 << lg) - 1);
        const u32 *so = S.org + part * rows * wq;
        u64 kmin = ~0ull;
#pragma unroll 1
        for (int base = 0; base < n; base += 32) {       // more than 32 candidates are never split
            const int k = base + (lane >> lg);
            int mx = cx, my = cy;
            bool in = k < n;
            if (in) {
                place(k, mx, my);
                in = mx >= minx && mx <= maxx && my >= miny && my <= maxy;   // ring points past the limits
            }
            u32 sad = in ? tz_sad(so, wq, rows, ref + (my + part * rows) * P.i_ref + mx, P.i_ref) : 0u;
            sad = tz_split_sum(sad, lg);
            if (in) {
                const u32 bits = tz_bits(((mx * 4) >> mvr) - bpx) + tz_bits(((my * 4) >> mvr) - bpy);
                const u64 key = tz_key(((u64)sad << shift) + (u64)(bits * lambda), k);
                kmin = key < kmin ? key : kmin;
            }
        }
        kmin = warp_min_u64(kmin);
        int ring_step = -1;
        if (kmin != ~0ull && (kmin >> TZ_KEY_BITS) < best) {
            const int k = (int)(kmin & ((1u << TZ_KEY_BITS) - 1));
            best = kmin >> TZ_KEY_BITS;
            place(k, mvx, mvy);
            if (k >= n0 + ngrid) ring_step = kTzRing[k - n0 - ngrid][2];
        }
        if (stage == 0) {
            const int found = ring_step >= 0 ? ring_step : (mvx != cx || mvy != cy) ? 2 : 0;   // best_step
            if (bi || (abs(mvpx - (mvx << 2)) <= 2 && abs(mvpy - (mvy << 2)) <= 2)) break;
            stage = 2;
            if (found > 5) {
                // get_raster_range (src/me.c:65-100)
                smin = 1 << msh;
                step = max(mvr < 3 ? 5 : mvr == 3 ? 6 : 8, min(w >> 1, h >> 1)) * (q.refi + 1);
                const int max_sr = P.max_search_range >> max(3 - mvr, 0);
                const int rxy = min(max((max_sr * q.dist + (P.gop_size >> 1)) / P.gop_size, max_sr >> 2), max_sr);
                rx = ry = rxy;
                if (mvr && (q.flags & 2)) {
                    rx = min(max(max(abs(q.mv_ipel[0] - mvx) * 4, max_sr >> 2), step * 8), rxy);
                    ry = min(max(max(abs(q.mv_ipel[1] - mvy) * 2, max_sr >> 2), step * 4), rxy);
                }
                if (msh) { rx = (rx >> msh) << msh; ry = (ry >> msh) << msh; }
                if (step >= smin) stage = 1;
            }
        } else if (stage == 1) {
            step >>= 1;
            if (msh) step = (step >> msh) << msh;
            rx = ry = step;
            if (step < smin) stage = 2;
        } else {
            break;
        }
    }
    if (!bi) { o.mv_ipel[0] = (s16)mvx; o.mv_ipel[1] = (s16)mvy; }
    int qx = mvx << 2, qy = mvy << 2;
    u64 cost = best;
    if (mvr < 2) {
        // me_sub_pel_search: centre + 8 half-sample points, then 8 quarter-sample points; with SAD
        // costs, the SATD of the winner closes
        const bool sad = q.flags & 1;
        const int bx = x << 2, by = y << 2;
#pragma unroll 1
        for (int pattern = 0; pattern < 3; pattern++) {
            if ((pattern == 1 && mvr != 0) || (pattern == 2 && !sad)) continue;
            const int cx = qx, cy = qy, nc = pattern == 0 ? 9 : pattern == 1 ? 8 : 1;
            __syncwarp();                    // the previous batch's sums have been read
            if (lane < nc) {
                int vx, vy;
                tz_sub_mv(pattern, lane, cx, cy, vx, vy);
                S.ptr[lane] = tz_mc_ptr(P, q.ref_slot, bx + vx, by + vy);
                S.sum[lane] = 0;
            }
            __syncwarp();
            if (sad && pattern < 2) {
                const int lg = tz_split(nc, h), rows = h >> lg, part = lane & ((1 << lg) - 1), k = lane >> lg;
                u32 v = k < nc ? tz_sad(S.org + part * rows * wq, wq, rows, S.ptr[k] + part * rows * P.i_ref, P.i_ref) : 0u;
                v = tz_split_sum(v, lg);
                if (k < nc && part == 0) S.sum[k] = v;
            } else if (min(w, h) >= 8) {
                tz_had<8>(S, P, lw, lh, nc, lane);
            } else {
                tz_had<4>(S, P, lw, lh, nc, lane);
            }
            __syncwarp();
            const int sh = pattern == 2 ? 16 - bi : shift;
            // lane i holds candidate i; the first of the smallest costs, as strict updates in order keep
            // it; the centre (of pattern 0, or alone) sets the cost that pattern 1 has to beat
            u64 key = ~0ull;
            if (lane < nc) {
                int vx, vy;
                tz_sub_mv(pattern, lane, cx, cy, vx, vy);
                key = ((u64)(lambda * (tz_bits((vx >> mvr) - bpx) + tz_bits((vy >> mvr) - bpy))) +
                       ((u64)S.sum[lane] << sh)) << 4 | (u64)lane;
            }
            key = warp_min_u64(key);
            if (pattern != 1 || (key >> 4) < cost) {
                cost = key >> 4;
                tz_sub_mv(pattern, (int)(key & 15), cx, cy, qx, qy);
            }
        }
    }
    const int rb = q.num_refp <= 1 ? 0 : min(q.refi + 1, q.num_refp - 1);   // tbl_refi_bits, src/tables.c:52
    const int extra = rb + mvr + (mvr < 4) + (bi ? q.mot_bits_other + 1 : 2);
    cost += (u64)(q.lambda_mv * (u32)extra);
    o.mv[0] = (s16)qx; o.mv[1] = (s16)qy;
    o.cost = (u32)((cost + (1u << 15)) >> 16);
    if (lane == 0) P.out[r] = o;
}

int launch_me_tz(const uavs3e_cuda_tz_pic_t *pic, const pel *org, int i_org, const pel *const *planes, int n_slots,
                 int i_ref, int pad, const void *reqs, int n, void *out, cudaStream_t st)
{
    if (!pic || !org || !planes || !reqs || !out || n < 0) return set_status(UC_ERR_ARG, "me_tz: null argument");
    if (n_slots < 1 || n_slots > UAVS3E_CUDA_TZ_MAX_SLOTS) return set_status(UC_ERR_ARG, "me_tz: slot count");
    if (pic->width < 8 || pic->height < 8 || pic->gop_size < 1 || pic->max_search_range < 4 ||
        pic->max_search_range > 1024)
        return set_status(UC_ERR_ARG, "me_tz: picture parameters");
    if ((i_ref & 3) || i_ref < pic->width + 2 * pad || pad < 144 || i_org < pic->width)
        return set_status(UC_ERR_ARG, "me_tz: strides / padding (planes padded by >= 144, stride a multiple of 4)");
    if (n == 0) return UC_OK;
    TzParams P;
    memset(&P, 0, sizeof(P));
    for (int i = 0; i < n_slots * 16; i++) {
        if (!planes[i]) return set_status(UC_ERR_ARG, "me_tz: null plane");
        P.planes[i] = planes[i];
    }
    P.org = org; P.i_org = i_org; P.i_ref = i_ref; P.n_slots = n_slots;
    P.W = pic->width; P.H = pic->height; P.is_padding = pic->is_padding ? 1 : 0;
    P.max_search_range = pic->max_search_range; P.gop_size = pic->gop_size;
    P.mto = (std::max(pic->width, pic->height) << 2) + 3;
    P.reqs = (const TzReq *)reqs; P.n = n; P.out = (TzOut *)out;
    P.sq32 = sqrt(32.0); P.sq128 = sqrt(128.0);
    P.k32 = had_scale_k(P.sq32); P.k128 = had_scale_k(P.sq128);
    prof_begin(PROF_TZ, st);
    k_me_tz<<<(unsigned)n, 32, 0, st>>>(P);
    UC_CHECK(cudaGetLastError());
    count_launch(1);
    prof_end(PROF_TZ, st);
    return UC_OK;
}

}  // namespace uc

using namespace uc;

extern "C" UAVS3E_CUDA_API int uavs3e_cuda_me_tz_device(const uavs3e_cuda_tz_pic_t *pic, const uint8_t *d_org, int i_org,
                                                        const uint8_t *const *d_planes, int n_slots, int i_ref, int pad,
                                                        const uavs3e_cuda_tz_req_t *d_reqs, int n,
                                                        uavs3e_cuda_tz_out_t *d_out, void *stream)
{
    int rc = ensure_init();
    if (rc) return rc;
    return launch_me_tz(pic, d_org, i_org, d_planes, n_slots, i_ref, pad, d_reqs, n, d_out, (cudaStream_t)stream);
}
