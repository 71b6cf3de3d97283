// Affine motion search for lists of calls: affine_me_gradient (src/inter.c:1339-1470) -- up to 7
// (uni) / 5 (bi) Gauss-Newton steps of the 4-parameter affine model, each from the normal
// equations of the residual and the Sobel gradients of the current prediction, its CPMV change
// rounded to the AMVR step and kept when the SATD + MV cost drops -- with the start CPMVs of
// analyze_affine_uni (:1607-1647) or the bi org of analyze_affine_bi (:1730-1790) on request.
// Bit-exact with the reference, including its double-precision solve.
//
// One warp per call.  The CU's org (or bi org) and the current prediction sit in shared memory;
// the prediction (com_mc_blk_affine_luma, src/com_mc.c:202-250) is rebuilt there after every
// step, the lanes walk its samples for the SATD tiles (packed rows, had.cuh) and, a column each, for the
// equation sums, which reduce across the warp in 64-bit integers.  The 4x4 solve runs over the warp's
// lanes in IEEE double with every operation rounded on its own (no fused multiply-add), in the
// reference's order; its divisions run on the integer pipe (f64div.cuh).
//
// The 40,860 calls of a 1080p frame take 1.91 ms (6.3 steps a call), issue-bound (61 % of the slots): by
// cycles the prediction is the largest part, then the solve and the sums.  With the divisions on the FP64
// pipe (45 % busy), the sums as 14 64-bit products per sample, SATD samples read byte by byte and one
// column per lane in the prediction it was 2.95 ms.  Solving 32 calls per warp in launches of their own,
// between launches of one step of every call, took 1.87 ms at this size and twice the time of this kernel
// below 5,000 calls.
#include "affine.cuh"
#include "common.cuh"
#include "f64div.cuh"
#include "had.cuh"
#include "uavs3e_cuda_internal.h"
#include "../../include/uavs3e_cuda.h"

#include <math.h>
#include <string.h>

namespace uc {

constexpr s32 CPMV_MIN = -131072, CPMV_MAX = 131071;

struct AffMeReq {
    s16 x, y; u8 w, h; u8 ref_slot; s8 refi; u8 num_refp; u8 mvr; u8 flags; u8 other_slot;
    u32 lambda_mv; s32 mot_bits_other; s32 pad;
    s32 mvp[2][2]; s32 mv[2][2]; s32 other_mv[2][2];
};
struct AffMeOut { s32 mv[2][2]; u32 satd; s32 bits; u64 cost; };
static_assert(sizeof(AffMeReq) == sizeof(uavs3e_cuda_affme_req_t), "affine search request layout");
static_assert(sizeof(AffMeOut) == sizeof(uavs3e_cuda_affme_out_t), "affine search result layout");

struct AffMeParams {
    const pel *planes[UAVS3E_CUDA_TZ_MAX_SLOTS];   // integer plane of each slot
    const pel *org;
    int i_org, i_ref, n_slots, W, H, n;
    double sq32, sq128;
    u64 k32, k128;       // had_scale_k of sq32, sq128
    const AffMeReq *reqs;
    AffMeOut *out;
};

// Tab_Affine_AMVR (inc/com_define.h:203)
__device__ __forceinline__ int ame_shift(int mvr) { return mvr == 0 ? 2 : (mvr == 1 ? 4 : 0); }

// MV_COST (src/inter.c:41): unsigned 32-bit product, rounded
__device__ __forceinline__ u32 ame_mv_cost(u32 lambda, int bits) { return (lambda * (u32)bits + 32768u) >> 16; }

__device__ __forceinline__ int ame_log2(int v) { return 31 - __clz(v); }

// affine_mv_bits (src/inter.c:1317-1337), tbl_refi_bits (src/tables.c:52) in closed form
__device__ __forceinline__ int ame_bits(const s32 *mv, const s32 *mvp, int num_refp, int refi, int sh)
{
    int bits = num_refp <= 1 ? 0 : min(refi + 1, num_refp - 1);
#pragma unroll
    for (int v = 0; v < 2; v++) {
        const int dx = abs((mv[2 * v] - mvp[2 * v]) >> sh), dy = abs((mv[2 * v + 1] - mvp[2 * v + 1]) >> sh);
        bits += ((ame_log2(dx + 1) + ame_log2(dy + 1)) << 1) + 2 + (dx != 0) + (dy != 0);
    }
    return bits;
}

// com_mc_blk_affine_luma (src/com_mc.c:202-250) into dst (w x h, stride w): each sample takes the
// MV of its SUB x SUB block (centre, or the control point for the two top corner blocks), rounded
// to 1/16 and clipped to 18 bits, and is filtered from the integer plane (com_mc_blk_luma, hp).
// A lane takes two columns of a band of 4 rows, or 8 where the sub-blocks are 8x8 and that leaves every
// lane a task, four rows of both at a time (aff_luma_pair).  One copy of the filter for both sizes: with
// unrolled variants the kernel waited for instructions a third of its time.
__device__ __noinline__ void ame_pred(const AffMeParams &P, const pel *plane, int x, int y, int w, int h, int lw,
                                      const s32 *mv, int sub, pel *dst, int lane)
{
    const s32 dhx = ((mv[2] - mv[0]) * 128) >> lw, dhy = ((mv[3] - mv[1]) * 128) >> lw;
    const s32 dvx = -dhy, dvy = dhx;
    const int lr = sub == 8 && w * h >= 512 ? 3 : 2;       // log2 of a task's rows
    const int tasks = (w * h) >> (1 + lr);
#pragma unroll 1
    for (int t = lane; t < tasks; t += 32) {
        const int c = (2 * t) & (w - 1), row = ((2 * t) >> lw) << lr, bx = c & -sub, by = row & -sub;
        int px = bx + (sub >> 1), py = by + (sub >> 1);
        if (bx == 0 && by == 0) { px = 0; py = 0; }
        else if (bx + sub == w && by == 0) { px = w; py = 0; }
        const s32 mx = min(max(aff_round7(mv[0] * 128 + dhx * px + dvx * py), CPMV_MIN), CPMV_MAX);
        const s32 my = min(max(aff_round7(mv[1] * 128 + dhy * px + dvy * py), CPMV_MIN), CPMV_MAX);
        const int qx = ((x + bx) << 4) + mx, qy = ((y + by) << 4) + my;
        pel *d = dst + row * w + c;
        aff_luma_pair(plane, P.i_ref, P.W, P.H, qx, qy, c - bx, row - by, 1 << (lr - 2), [&](int o, int v0, int v1) {
            *reinterpret_cast<u16 *>(d + o * w) = (u16)(v0 | v1 << 8);
        });
    }
}

// com_had (src/com_cost.c:712-812) of the 2^lw x 2^lh block o - p (both in shared memory, dense rows):
// 8x8 tiles of square blocks, 16x8 / 8x16 of the others, 8 lanes to a tile (had.cuh)
__device__ __noinline__ u32 ame_had(const pel *o, const pel *p, int lw, int lh, int lane, const AffMeParams &P)
{
    const HadSigns G = had_signs(lane);
    const bool wide = lw > lh, pair = lw != lh;
    const int lx = wide ? 4 : 3, ly = pair && !wide ? 4 : 3, lntx = lw - lx;
    const int po = wide ? 8 : 8 << lw;                 // the second half of a 2:1 tile
    const int total = 8 << (lntx + lh - ly);           // rows of all tiles: a multiple of 32
    u32 acc = 0;
#pragma unroll 1
    for (int t = lane; t < total; t += 32) {
        const int row = t & 7, tile = t >> 3;
        const int at = (((tile >> lntx) << ly) + row) * (1 << lw) + ((tile & ((1 << lntx) - 1)) << lx);
        const uint2 ov = *reinterpret_cast<const uint2 *>(o + at), pv = *reinterpret_cast<const uint2 *>(p + at);
        int q[4], s;
        had_diff8(ov.x, ov.y, pv.x, pv.y, q);
        if (pair) {
            const uint2 ow = *reinterpret_cast<const uint2 *>(o + at + po), pw = *reinterpret_cast<const uint2 *>(p + at + po);
            int e[4], d[4];
            had_diff8(ow.x, ow.y, pw.x, pw.y, e);
#pragma unroll
            for (int i = 0; i < 4; i++) { d[i] = q[i] - e[i]; q[i] += e[i]; }
            s = had8_lane(d, G);
            s += had8_lane(q, G);
        } else {
            s = had8_lane(q, G);
        }
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        s += __shfl_xor_sync(0xffffffffu, s, 4);
        if (row == 0) acc += pair ? had_scale(2 * s, P.sq128, P.k128) : (u32)((2 * s + 2) >> 2);
    }
    return __reduce_add_sync(0xffffffffu, acc);
}

// The sums of one gradient step (affine_sobel_flt_hor / _ver and affine_coef_computer,
// src/com_util.c:2966-3045): per sample (j, k) the Sobel gradients gx, gy of the prediction at the
// nearest interior position, the four model columns c0 = gx, c1 = k gx + j gy, c2 = gy, c3 = j gx - k gy
// and the residual r; e[0..9] = the sums of the products c_i c_j (i <= j), e[10..13] of c_i r, written
// to dst by the lanes that hold them.
//
// A lane walks a column (for 16 columns, half of one), so k is a factor of its sums and only gx gx,
// gx gy, gy gy (each also times j and j^2) and gx r, gy r (also times j) are summed per sample; a row
// costs three new samples.  All but the j^2 sums stay below 2^31: |gx|, |gy| <= 1020 and the sum of j
// over 64 rows is 2016.
__device__ __noinline__ void ame_equations(const pel *o, const pel *p, int lw, int lh, int lane, s64 *dst)
{
    const int w = 1 << lw, h = 1 << lh;
    s64 e[16];
#pragma unroll
    for (int i = 0; i < 16; i++) e[i] = 0;
    const int halves = w < 32 ? 2 : 1, rows = h / halves, j0 = halves == 2 ? (lane >> 4) * rows : 0;
#pragma unroll 1
    for (int k = lane & (w - 1); k < w; k += 32) {
        const int kk = min(max(k, 1), w - 2);
        const pel *pc = p + kk;
        s32 xx = 0, xy = 0, yy = 0, jxx = 0, jxy = 0, jyy = 0, xr = 0, yr = 0, jxr = 0, jyr = 0;
        s64 jjxx = 0, jjxy = 0, jjyy = 0;
        // rows of the window around the gradient's row: horizontal difference d and smoothing s
        int jj = min(max(j0, 1), h - 2);
        const auto load = [&](int row, int &d, int &s) {
            const pel *q = pc + (row << lw);
            const int l = q[-1], c = q[0], r = q[1];
            d = r - l;
            s = l + 2 * c + r;
        };
        int d0, d1, d2, s0, s1, s2;
        load(jj - 1, d0, s0);
        load(jj, d1, s1);
        load(jj + 1, d2, s2);
#pragma unroll 1
        for (int j = j0; j < j0 + rows; j++) {
            const int gx = d0 + 2 * d1 + d2, gy = s2 - s0;
            const int r = (int)o[(j << lw) + k] - (int)p[(j << lw) + k];
            const int a = gx * gx, b = gx * gy, c = gy * gy, g = j * r;
            const int ja = j * a, jb = j * b, jc = j * c;
            xx += a; xy += b; yy += c;
            jxx += ja; jxy += jb; jyy += jc;
            jjxx += (s64)ja * j; jjxy += (s64)jb * j; jjyy += (s64)jc * j;
            xr += gx * r; yr += gy * r;
            jxr += gx * g; jyr += gy * g;
            // the next sample's gradient row is the next one inside the block
            if (j >= 1 && j < h - 2) {
                d0 = d1; d1 = d2; s0 = s1; s1 = s2;
                load(j + 2, d2, s2);
            }
        }
        const s64 K = k, K2 = k * k;
        e[0] += xx;
        e[1] += K * xx + jxy;
        e[2] += xy;
        e[3] += jxx - K * xy;
        e[4] += K2 * xx + 2 * K * jxy + jjyy;
        e[5] += K * xy + jyy;
        e[6] += K * jxx - K2 * xy + jjxy - K * jyy;
        e[7] += yy;
        e[8] += jxy - K * yy;
        e[9] += jjxx - 2 * K * jxy + K2 * yy;
        e[10] += xr;
        e[11] += K * xr + jyr;
        e[12] += yr;
        e[13] += jxr - K * yr;
    }
    // the 16 sums over the warp: at each step a lane keeps the half of its sums that its bit selects
    // and sends the other, so 16 exchanges leave sum (bit 4, 3, 2, 1 of the lane) on each lane pair
#pragma unroll
    for (int st = 0; st < 4; st++) {
        const int m = 16 >> st, half = 8 >> st;
        const bool up = lane & m;
#pragma unroll
        for (int i = 0; i < half; i++) {
            const s64 keep = up ? e[i + half] : e[i], send = up ? e[i] : e[i + half];
            e[i] = keep + __shfl_xor_sync(0xffffffffu, send, m);
        }
    }
    e[0] += __shfl_xor_sync(0xffffffffu, e[0], 1);
    const int idx = (lane >> 1) & 15;                  // bits 4, 3, 2, 1 of the lane, highest first
    if (!(lane & 1) && idx < 14) dst[idx] = e[0];
}

// IEEE division on the integer pipe (f64div.cuh); zeros, infinities, NaNs, denormals and results outside
// the normal range take the hardware's.  The elimination's divisions go this way, the back substitution's
// four (one lane each) to the FP64 pipe: 10 issue slots against 90, and the pipe has room for them -- not
// for all seven, with which it was busy 45 % of the search and its latency bound the solve.
__device__ __noinline__ double ame_div_hw(double a, double b) { return __ddiv_rn(a, b); }
__device__ __noinline__ double ame_div(double a, double b)
{
    uint64_t r;
    if (f64_div_bits((uint64_t)__double_as_longlong(a), (uint64_t)__double_as_longlong(b), &r)) return __longlong_as_double((long long)r);
    return ame_div_hw(a, b);
}

// (s16) of a double as x86-64 code converts it (the reference's platform): truncation to 32 bits
// by cvttsd2si -- NaN and values outside the 32-bit range give INT_MIN -- then the low 16 bits
// (the range test on the exponent bits: |v| >= 2^31, infinities and NaN all give INT_MIN, and
// the values in (-2^31 - 1, -2^31] that truncate to INT_MIN give it too)
__device__ __forceinline__ s16 ame_to_s16(double v)
{
    const int e = (int)((unsigned long long)__double_as_longlong(v) >> 52) & 0x7ff;
    const int i = e < 1023 + 31 ? __double2int_rz(v) : (int)0x80000000u;
    return (s16)(u16)(u32)i;
}

// the bits of |v| as an unsigned integer: for non-NaN values |a| > |b| exactly when
// ame_mag(a) > ame_mag(b); NaN maps above every finite value
__device__ __forceinline__ unsigned long long ame_mag(double v)
{
    return (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
}

// a component of the solution as a CPMV change at AMVR shift sh (src/inter.c:1412-1436): scaled, rounded
// half away from zero (d >= 0: +0, -0 and positive values, not NaN) and rounded to the AMVR step
__device__ __forceinline__ s16 ame_step_mv(double d, int sh)
{
    const long long db = __double_as_longlong(d);
    const bool ge0 = db == (long long)0x8000000000000000ull ||
                     (db >= 0 && (unsigned long long)db <= 0x7ff0000000000000ull);
    const double half = ge0 ? 0.5 : -0.5;
    if (sh == 0) return ame_to_s16(__dadd_rn(__dmul_rn(d, 16.0), half));
    s16 q = ame_to_s16(__dadd_rn(__dmul_rn(d, 4.0), half));
    q = (s16)(q << 2);
    return (s16)(((q + (1 << (sh - 1))) >> sh) << sh);   // com_mv_rounding_s16
}

// solve_equal (src/inter.c:1280-1315) over the warp and the conversion of its solution to the four
// CPMV changes (x0, y0, x1, y1) at AMVR shift sh.  Lane 5 r + k (< 25) holds element (r, k) of the
// augmented matrix (rows 1..4, row 0 being the reference's swap buffer); in step i every element
// (j > i, k >= i) of the elimination is one lane's a[j][k] - a[i][k] * a[j][i-1] / a[i][i-1], each
// operation rounded on its own, so the values are the reference's; the back substitution runs on
// lane 0 in the reference's order.  e[] = the equation sums in shared memory.
__device__ __noinline__ void ame_solve(const s64 *e, int w, int sh, int lane, s16 *mvd)
{
    const bool mine = lane < 25;
    const int r = mine ? lane / 5 : 0, col = mine ? lane - 5 * (lane / 5) : 0;
    // coef[c + 1][k] = e[ix(c, k)] for k < 4 (the symmetric products), coef[c + 1][4] = 8 e[10 + c]
    const int c = r - 1;
    const int lo = min(c, col), hi = max(c, col);
    const int idx = col == 4 ? 10 + c : (lo == 0 ? hi : (lo == 1 ? 3 + hi : (lo == 2 ? 5 + hi : 9)));
    double v = (mine && r >= 1) ? __ll2double_rn(col == 4 ? 8 * e[idx] : e[idx]) : 0.0;
#pragma unroll 1
    for (int i = 1; i < 4; i++) {
        // fabs(cand) > best in integers: false when cand is NaN, and nothing exceeds a NaN best
        unsigned long long best = ame_mag(__shfl_sync(0xffffffffu, v, i * 5 + i - 1));
        int bi = i;
#pragma unroll 1
        for (int j = i + 1; j < 5; j++) {
            const unsigned long long cand = ame_mag(__shfl_sync(0xffffffffu, v, j * 5 + i - 1));
            if (cand <= 0x7ff0000000000000ull && cand > best) { best = cand; bi = j; }
        }
        if (bi != i) {
            const int src = (mine && r == i) ? bi * 5 + col : ((mine && r == bi) ? i * 5 + col : lane);
            v = __shfl_sync(0xffffffffu, v, src);
        }
        const double aik = __shfl_sync(0xffffffffu, v, i * 5 + col);
        const double aji = __shfl_sync(0xffffffffu, v, r * 5 + i - 1);
        const double aii = __shfl_sync(0xffffffffu, v, i * 5 + i - 1);
        if (mine && r > i && col >= i) v = __dsub_rn(v, ame_div(__dmul_rn(aik, aji), aii));
    }
    double m[25];
#pragma unroll
    for (int k = 5; k < 25; k++) m[k] = __shfl_sync(0xffffffffu, v, k);
    double x[4] = { 0, 0, 0, 0 };
    if (lane == 0) {
#define A(i, j) m[(i) * 5 + (j)]
        x[3] = ame_div_hw(A(4, 4), A(4, 3));
#pragma unroll
        for (int i = 2; i >= 0; i--) {
            double t = 0;
#pragma unroll
            for (int j = i + 1; j < 4; j++) t = __dadd_rn(t, __dmul_rn(A(i + 1, j), x[j]));
            x[i] = ame_div_hw(__dsub_rn(A(i + 1, 4), t), A(i + 1, i));
        }
#undef A
    }
    // lanes 0..3 convert x0 -> mvd x0, x2 -> y0, x1 w + x0 -> x1, -x3 w + x2 -> y1
    const double x0 = __shfl_sync(0xffffffffu, x[0], 0), x1 = __shfl_sync(0xffffffffu, x[1], 0);
    const double x2 = __shfl_sync(0xffffffffu, x[2], 0), x3 = __shfl_sync(0xffffffffu, x[3], 0);
    u32 o = 0;
    if (lane < 4) {
        const double wd = (double)w;
        const double d = lane == 0 ? x0 : (lane == 1 ? x2 : (lane == 2 ? __dadd_rn(__dmul_rn(x1, wd), x0)
                                                                        : __dadd_rn(__dmul_rn(-x3, wd), x2)));
        o = (u32)(u16)ame_step_mv(d, sh);
    }
    u32 packed[2];
    packed[0] = __shfl_sync(0xffffffffu, o, 0) | (__shfl_sync(0xffffffffu, o, 1) << 16);
    packed[1] = __shfl_sync(0xffffffffu, o, 2) | (__shfl_sync(0xffffffffu, o, 3) << 16);
    mvd[0] = (s16)(u16)packed[0];
    mvd[1] = (s16)(u16)(packed[0] >> 16);
    mvd[2] = (s16)(u16)packed[1];
    mvd[3] = (s16)(u16)(packed[1] >> 16);
}

__device__ __forceinline__ bool ame_cpmv_ok(const s32 (*m)[2])
{
    return m[0][0] >= CPMV_MIN && m[0][0] <= CPMV_MAX && m[0][1] >= CPMV_MIN && m[0][1] <= CPMV_MAX &&
           m[1][0] >= CPMV_MIN && m[1][0] <= CPMV_MAX && m[1][1] >= CPMV_MIN && m[1][1] <= CPMV_MAX;
}

// calls outside the supported domain (CU inside the picture, sides 16..64, slots, AMVR index,
// reference index, CPMVs within 18 bits) return cost ~0 with the start CPMVs
__device__ __forceinline__ bool ame_valid(const AffMeParams &P, const AffMeReq &q)
{
    const int w = q.w, h = q.h, bi = q.flags & UAVS3E_CUDA_AFFME_BI;
    return !((w != 16 && w != 32 && w != 64) || (h != 16 && h != 32 && h != 64) || q.x < 0 || q.y < 0 ||
             q.x + w > P.W || q.y + h > P.H || q.ref_slot >= P.n_slots || (bi && q.other_slot >= P.n_slots) ||
             q.mvr > 2 || q.refi < 0 || q.refi >= q.num_refp || !ame_cpmv_ok(q.mvp) ||
             (!(q.flags & UAVS3E_CUDA_AFFME_UNI_START) && !ame_cpmv_ok(q.mv)) || (bi && !ame_cpmv_ok(q.other_mv)));
}

__device__ __forceinline__ void ame_write_invalid(const AffMeReq &q, AffMeOut *out)
{
    for (int v = 0; v < 2; v++) { out->mv[v][0] = q.mv[v][0]; out->mv[v][1] = q.mv[v][1]; }
    out->satd = 0;
    out->bits = 0;
    out->cost = ~0ull;
}

__device__ __forceinline__ void ame_write_result(const AffMeReq &q, const s32 *mv, u64 best, int best_bits, AffMeOut *out)
{
    const u64 satd = best - ame_mv_cost(q.lambda_mv, best_bits);
    for (int v = 0; v < 2; v++) { out->mv[v][0] = mv[2 * v]; out->mv[v][1] = mv[2 * v + 1]; }
    out->satd = (u32)satd;
    out->bits = best_bits;
    out->cost = satd + ame_mv_cost(q.lambda_mv, best_bits);
}

// a call's search state: the CPMVs of the last step, the best ones with their cost and bits
struct AmeState { s32 mvt[4], mv[4]; u64 best; s32 bits, pad; };

// steps of a call at most
__device__ __forceinline__ int ame_steps(const AffMeReq &q) { return (q.flags & UAVS3E_CUDA_AFFME_BI) ? 5 : 7; }

__device__ __forceinline__ int ame_sub(const AffMeReq &q)
{
    return (q.flags & (UAVS3E_CUDA_AFFME_BI | UAVS3E_CUDA_AFFME_SUB8)) ? 8 : 4;
}

// the org block in so; for a bi call create_bi_org (src/inter.c:55) with the 8x8 prediction of the other
// list, formed in sp
__device__ __noinline__ void ame_org(const AffMeParams &P, const AffMeReq &q, pel *so, pel *sp, int lane)
{
    const int w = q.w, h = q.h, lw = 31 - __clz(w), n4 = (w * h) >> 2;
    const pel *org = P.org + (long long)q.y * P.i_org + q.x;
    u32 *so4 = reinterpret_cast<u32 *>(so);
#pragma unroll 1
    for (int i = lane; i < n4; i += 32)
        so4[i] = had_load4(org + (long long)(i >> (lw - 2)) * P.i_org + ((i << 2) & (w - 1)));
    if (q.flags & UAVS3E_CUDA_AFFME_BI) {
        const s32 om[4] = { q.other_mv[0][0], q.other_mv[0][1], q.other_mv[1][0], q.other_mv[1][1] };
        ame_pred(P, P.planes[q.other_slot], q.x, q.y, w, h, lw, om, 8, sp, lane);
        __syncwarp();
        const u32 *sp4 = reinterpret_cast<const u32 *>(sp);
#pragma unroll 1
        for (int i = lane; i < n4; i += 32) {
            // 2 org - prediction, clipped, byte-wise: s + (s - p) where s >= p, else s - (p - s)
            const u32 v = so4[i], pv = sp4[i];
            so4[i] = __vsubus4(__vaddus4(v, __vsubus4(v, pv)), __vsubus4(pv, v));
        }
    }
    __syncwarp();
}

// the prediction at CPMVs mv into sp, and its com_had against so
__device__ __forceinline__ u32 ame_cost(const AffMeParams &P, const AffMeReq &q, const s32 *mv, const pel *so, pel *sp, int lane)
{
    const int lw = 31 - __clz((int)q.w), lh = 31 - __clz((int)q.h);
    __syncwarp();
    ame_pred(P, P.planes[q.ref_slot], q.x, q.y, q.w, q.h, lw, mv, ame_sub(q), sp, lane);
    __syncwarp();
    return ame_had(so, sp, lw, lh, lane, P);
}

// the state before the first step, its prediction in sp: the start CPMVs (for an UNI_START call
// analyze_affine_uni's choice) and their cost
__device__ __forceinline__ void ame_start(const AffMeParams &P, const AffMeReq &q, const pel *so, pel *sp, int lane, AmeState &T)
{
    const int w = q.w, h = q.h, bi = q.flags & UAVS3E_CUDA_AFFME_BI, sh = ame_shift(q.mvr);
    const s32 mvp[4] = { q.mvp[0][0], q.mvp[0][1], q.mvp[1][0], q.mvp[1][1] };
    s32 mv[4] = { q.mv[0][0], q.mv[0][1], q.mv[1][0], q.mv[1][1] };
    u32 had = 0;
    // candidates in order: for UNI_START the MVP (0), the uni MV (1) and, where the MVP won, its
    // prediction again (2); else only the start CPMVs (2)
    u64 c_mvp = 0;
#pragma unroll 1
    for (int k = (!bi && (q.flags & UAVS3E_CUDA_AFFME_UNI_START)) ? 0 : 2; k < 3; k++) {
        s32 m[4];
        if (k == 1) {
            // the uni MV clipped (mv_clip, src/inter.c:1472) and scaled to 1/16 sample (rounded to
            // whole samples at AMVR index 1)
            const int x4 = q.x << 2, y4 = q.y << 2, w4 = w << 2, h4 = h << 2;
            const int min_c = (-128 - 4) << 2, max_x = (P.W - 1 + 128 + 4) << 2, max_y = (P.H - 1 + 128 + 4) << 2;
            s16 mx = (s16)q.mv[0][0], my = (s16)q.mv[0][1];
            if (x4 + mx < min_c) mx = (s16)(min_c - x4);
            if (y4 + my < min_c) my = (s16)(min_c - y4);
            if (x4 + mx + w4 - 4 > max_x) mx = (s16)(max_x - x4 - w4 + 4);
            if (y4 + my + h4 - 4 > max_y) my = (s16)(max_y - y4 - h4 + 4);
            s32 tx = (s32)mx * 4, ty = (s32)my * 4;
            if (q.mvr == 1) {
                tx = tx >= 0 ? ((tx + 8) >> 4) << 4 : -(((-tx + 8) >> 4) << 4);
                ty = ty >= 0 ? ((ty + 8) >> 4) << 4 : -(((-ty + 8) >> 4) << 4);
            }
            m[0] = m[2] = min(max(tx, CPMV_MIN), CPMV_MAX);
            m[1] = m[3] = min(max(ty, CPMV_MIN), CPMV_MAX);
        } else {
#pragma unroll
            for (int v = 0; v < 4; v++) m[v] = k == 0 ? mvp[v] : mv[v];
        }
        had = ame_cost(P, q, m, so, sp, lane);
        const u64 c = (u64)had + ame_mv_cost(q.lambda_mv, ame_bits(m, mvp, q.num_refp, q.refi, sh));
        if (k == 0) c_mvp = c;
        if (k == 1) {
            const bool uni = c < c_mvp;
#pragma unroll
            for (int v = 0; v < 4; v++) mv[v] = uni ? m[v] : mvp[v];
            if (uni) break;
        }
    }
#pragma unroll
    for (int v = 0; v < 4; v++) T.mv[v] = T.mvt[v] = mv[v];
    T.bits = ame_bits(mv, mvp, q.num_refp, q.refi, sh) + (bi ? q.mot_bits_other : 0);
    T.best = (u64)ame_mv_cost(q.lambda_mv, T.bits) + (had >> bi);
}

// the CPMVs after a step's change
__device__ __forceinline__ void ame_move(const AffMeReq &q, const s16 *mvd, s32 *mvt)
{
    const int sh = ame_shift(q.mvr);
#pragma unroll
    for (int v = 0; v < 4; v++) {
        s32 m = min(max(mvt[v] + (s32)mvd[v], CPMV_MIN), CPMV_MAX);
        if (m == CPMV_MAX) m = m >> sh << sh;
        mvt[v] = m;
    }
}

// the cost of the moved CPMVs (their prediction in sp); the best is kept
__device__ __forceinline__ void ame_try(const AffMeParams &P, const AffMeReq &q, const pel *so, pel *sp, int lane, AmeState &T)
{
    const int bi = q.flags & UAVS3E_CUDA_AFFME_BI;
    const s32 mvp[4] = { q.mvp[0][0], q.mvp[0][1], q.mvp[1][0], q.mvp[1][1] };
    const u32 had = ame_cost(P, q, T.mvt, so, sp, lane);
    const int bits = ame_bits(T.mvt, mvp, q.num_refp, q.refi, ame_shift(q.mvr)) + (bi ? q.mot_bits_other : 0);
    const u64 cost = (u64)ame_mv_cost(q.lambda_mv, bits) + (had >> bi);
    if (cost < T.best) {
        T.best = cost;
        T.bits = bits;
#pragma unroll
        for (int v = 0; v < 4; v++) T.mv[v] = T.mvt[v];
    }
}

// One warp per CTA: calls differ 16-fold in size, and a slot frees as soon as its call ends.  9 KB of
// shared memory and 80 registers let 24 warps share an SM.
__global__ void __launch_bounds__(32, 24) k_me_affine(const AffMeParams P)
{
    __shared__ __align__(16) pel s_org[64 * 64];
    __shared__ __align__(16) pel s_pred[64 * 64];
    __shared__ s64 s_eq[14];
    const int lane = threadIdx.x, r = blockIdx.x;
    const AffMeReq q = P.reqs[r];
    AffMeOut *out = P.out + r;
    if (!ame_valid(P, q)) {
        if (lane == 0) ame_write_invalid(q, out);
        return;
    }
    pel *so = s_org, *sp = s_pred;
    AmeState T;
    ame_org(P, q, so, sp, lane);
    ame_start(P, q, so, sp, lane, T);
    const int steps = ame_steps(q);
#pragma unroll 1
    for (int iter = 0; iter < steps; iter++) {
        ame_equations(so, sp, 31 - __clz((int)q.w), 31 - __clz((int)q.h), lane, s_eq);
        __syncwarp();
        s16 mvd[4];
        ame_solve(s_eq, q.w, ame_shift(q.mvr), lane, mvd);
        if (!mvd[0] && !mvd[1] && !mvd[2] && !mvd[3]) break;
        ame_move(q, mvd, T.mvt);
        ame_try(P, q, so, sp, lane, T);
    }
    if (lane == 0) ame_write_result(q, T.mv, T.best, T.bits, out);
}

int launch_me_affine(int W, int H, const pel *org, int i_org, const pel *const *planes, int n_slots, int i_ref,
                     int pad, const void *reqs, int n, void *out, cudaStream_t st)
{
    if (!org || !planes || (n > 0 && (!reqs || !out)) || n < 0) return set_status(UC_ERR_ARG, "me_affine: null argument");
    if (n_slots < 1 || n_slots > UAVS3E_CUDA_TZ_MAX_SLOTS || W < 16 || H < 16 || i_org < W)
        return set_status(UC_ERR_ARG, "me_affine: slots / picture size / org stride");
    // 8-tap windows reach 132 + 3 samples before the picture and W + 4 + 7 + 4 after it
    if (pad < 144 || i_ref < W + 2 * pad) return set_status(UC_ERR_ARG, "me_affine: padding (>= 144) / stride");
    if (n == 0) return UC_OK;
    AffMeParams P;
    memset(&P, 0, sizeof(P));
    for (int s = 0; s < n_slots; s++) {
        if (!planes[s * 16]) return set_status(UC_ERR_ARG, "me_affine: null plane");
        P.planes[s] = planes[s * 16];
    }
    P.org = org; P.i_org = i_org; P.i_ref = i_ref; P.n_slots = n_slots; P.W = W; P.H = H; P.n = n;
    P.sq32 = sqrt(32.0);
    P.sq128 = sqrt(128.0);
    P.k32 = had_scale_k(P.sq32);
    P.k128 = had_scale_k(P.sq128);
    P.reqs = (const AffMeReq *)reqs;
    P.out = (AffMeOut *)out;
    prof_begin(PROF_AFFME, st);
    k_me_affine<<<(unsigned)n, 32, 0, st>>>(P);
    UC_CHECK(cudaGetLastError());
    count_launch(1);
    prof_end(PROF_AFFME, st);
    return UC_OK;
}

}  // namespace uc

using namespace uc;

UAVS3E_CUDA_API int uavs3e_cuda_me_affine_device(int width, int height, const uint8_t *d_org, int i_org,
                                                 const uint8_t *const *d_planes, int n_slots, int i_ref, int pad,
                                                 const uavs3e_cuda_affme_req_t *d_reqs, int n,
                                                 uavs3e_cuda_affme_out_t *d_out, void *stream)
{
    if (ensure_init()) return uavs3e_cuda_status();
    return launch_me_affine(width, height, d_org, i_org, d_planes, n_slots, i_ref, pad, d_reqs, n, d_out,
                            (cudaStream_t)stream);
}

// ---------------------------------------------------------------------------------------------
// Affine control-point MVP: one thread per CU.  The neighbour walk, the POC-distance scaling
// (ratio = (2^14 / t_neb) * t_cur, C's truncating division first; symmetric rounding shift by
// 14; s16 clip) and the AMVR rounding of the 1/16-sample value (magnitude rounded, sign kept;
// 18-bit clip) are integer and follow com_get_affine_mvp_scaling step for step.
// ---------------------------------------------------------------------------------------------
static_assert(sizeof(uavs3e_cuda_affmvp_req_t) == 12, "affine MVP request layout");
static_assert(sizeof(uavs3e_cuda_affmvp_out_t) == 16, "affine MVP result layout");

__device__ __forceinline__ int amvp_scale(int mv, int ratio)
{
    const long long t = (long long)mv * ratio;
    const long long r = t == 0 ? 0 : t > 0 ? (t + 8192) >> 14 : -((-t + 8192) >> 14);
    return (int)max(-32768ll, min(32767ll, r));
}

__device__ __forceinline__ int amvp_round(int v, int shift)
{
    const int x = v * 4, add = shift > 0 ? 1 << (shift - 1) : 0;
    const int r = x >= 0 ? ((x + add) >> shift) << shift : -(((-x + add) >> shift) << shift);
    return max(-131072, min(131071, r));
}

__global__ void __launch_bounds__(256) k_affine_mvp(long long ptr, const long long *ref_ptr, int n_ref,
                                                    const short *map_mv, const signed char *map_refi, int i_scu,
                                                    long long n_field, const uavs3e_cuda_affmvp_req_t *reqs, int n,
                                                    uavs3e_cuda_affmvp_out_t *out, int *err)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uavs3e_cuda_affmvp_req_t q = reqs[i];
    uavs3e_cuda_affmvp_out_t o = {};
    bool bad = q.lidx < 0 || q.lidx > 1 || q.cur_refi < 0 || q.cur_refi >= n_ref || q.mvr < 0 || q.mvr > 2 ||
               q.cu_width < 4;
    int t_cur = 0;
    if (!bad) {
        t_cur = (int)(ptr * 2 - ref_ptr[q.cur_refi * 2 + q.lidx] * 2);
        bad = t_cur == 0;
    }
    int mv[2][2] = { { 0, 0 }, { 0, 0 } };
    if (!bad) {
        const long long base = (long long)i_scu + 1 + q.scup - i_scu;   // the row above the CU
        const int wsc = q.cu_width >> 2;
        // A (left, same row), B (above), D (above-left); G (above the last column), C (above-right)
        const long long nb[5] = { base + i_scu - 1, base, base - 1, base + wsc - 1, base + wsc };
#pragma unroll
        for (int g = 0; g < 2; g++) {
            bool found = false;
#pragma unroll
            for (int k = g == 0 ? 0 : 3; k < (g == 0 ? 3 : 5); k++) {
                if (found || bad) continue;
                const long long a = nb[k];
                if (a < 0 || a >= n_field) { bad = true; continue; }
                const int refi = map_refi[a * 2 + q.lidx];
                if (refi < 0) continue;
                if (refi >= n_ref) { bad = true; continue; }
                const int t_neb = (int)(ptr * 2 - ref_ptr[refi * 2 + q.lidx] * 2);
                if (t_neb == 0) { bad = true; continue; }
                const int ratio = (1 << 14) / t_neb * t_cur;
                const short2 v = *(const short2 *)(map_mv + (a * 2 + q.lidx) * 2);
                mv[g][0] = amvp_scale(v.x, ratio);
                mv[g][1] = amvp_scale(v.y, ratio);
                found = true;
            }
        }
    }
    if (!bad) {
        const int shift = q.mvr == 0 ? 2 : q.mvr == 1 ? 4 : 0;
#pragma unroll
        for (int g = 0; g < 2; g++) {
            o.mvp[g][0] = amvp_round(mv[g][0], shift);
            o.mvp[g][1] = amvp_round(mv[g][1], shift);
        }
    } else if (err) {
        atomicAdd(err, 1);
    }
    out[i] = o;
}

int launch_affine_mvp(long long ptr, const long long *d_ref_ptr, int n_ref, const short *d_map_mv,
                      const signed char *d_map_refi, int i_scu, int rows, const void *d_reqs, int n, void *d_out,
                      int *d_err, cudaStream_t st)
{
    if (n < 0 || n_ref < 1 || i_scu < 3 || rows < 2 || (n > 0 && (!d_ref_ptr || !d_map_mv || !d_map_refi || !d_reqs || !d_out)))
        return set_status(UC_ERR_ARG, "affine_mvp: bad argument");
    if (((uintptr_t)d_map_mv & 3) != 0) return set_status(UC_ERR_ARG, "affine_mvp: map_mv not 4-byte aligned");
    if (n == 0) return UC_OK;
    k_affine_mvp<<<(n + 255) / 256, 256, 0, st>>>(ptr, d_ref_ptr, n_ref, d_map_mv, d_map_refi, i_scu,
                                                  (long long)rows * i_scu, (const uavs3e_cuda_affmvp_req_t *)d_reqs, n,
                                                  (uavs3e_cuda_affmvp_out_t *)d_out, d_err);
    UC_CHECK(cudaGetLastError());
    count_launch(1);
    return UC_OK;
}

UAVS3E_CUDA_API int uavs3e_cuda_affine_mvp_device(int64_t ptr, const int64_t *d_ref_ptr, int n_ref,
                                                  const int16_t *d_map_mv, const int8_t *d_map_refi, int i_scu,
                                                  int rows, const uavs3e_cuda_affmvp_req_t *d_reqs, int n,
                                                  uavs3e_cuda_affmvp_out_t *d_out, int32_t *d_err, void *stream)
{
    int rc = ensure_init();
    if (rc) return rc;
    return launch_affine_mvp(ptr, (const long long *)d_ref_ptr, n_ref, d_map_mv, (const signed char *)d_map_refi,
                             i_scu, rows, d_reqs, n, d_out, (int *)d_err, (cudaStream_t)stream);
}

UAVS3E_CUDA_API int uavs3e_cuda_affine_mvp(int64_t ptr, const int64_t *ref_ptr, int n_ref, const int16_t *map_mv,
                                           const int8_t *map_refi, int i_scu, int rows,
                                           const uavs3e_cuda_affmvp_req_t *reqs, int n,
                                           uavs3e_cuda_affmvp_out_t *out)
{
    int rc = ensure_init();
    if (rc) return rc;
    if (n < 0 || n_ref < 1 || i_scu < 3 || rows < 2 || (n > 0 && (!ref_ptr || !map_mv || !map_refi || !reqs || !out)))
        return set_status(UC_ERR_ARG, "affine_mvp: bad argument");
    if (n == 0) return UC_OK;
    cudaStream_t st = nullptr;
    UC_CHECK(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    const size_t field = (size_t)rows * i_scu;
    const size_t b_ref = (size_t)n_ref * 16, b_mv = field * 8, b_refi = (field * 2 + 255) & ~(size_t)255;
    const size_t b_req = (size_t)n * sizeof(uavs3e_cuda_affmvp_req_t), b_out = (size_t)n * sizeof(uavs3e_cuda_affmvp_out_t);
    auto up = [](size_t b) { return (b + 255) & ~(size_t)255; };
    char *buf = nullptr;
    cudaError_t ce = cudaMallocAsync((void **)&buf, up(b_ref) + up(b_mv) + b_refi + up(b_req) + up(b_out) + 256, st);
    if (ce != cudaSuccess) { cudaStreamDestroy(st); return check_cuda(ce, "affine_mvp: allocate"); }
    char *d_ref = buf, *d_mv = d_ref + up(b_ref), *d_refi = d_mv + up(b_mv), *d_req = d_refi + b_refi;
    char *d_out = d_req + up(b_req), *d_err = d_out + up(b_out);
    int bad = 0;
    rc = UC_OK;
    if ((ce = cudaMemcpyAsync(d_ref, ref_ptr, b_ref, cudaMemcpyHostToDevice, st)) != cudaSuccess ||
        (ce = cudaMemcpyAsync(d_mv, map_mv, b_mv, cudaMemcpyHostToDevice, st)) != cudaSuccess ||
        (ce = cudaMemcpyAsync(d_refi, map_refi, field * 2, cudaMemcpyHostToDevice, st)) != cudaSuccess ||
        (ce = cudaMemcpyAsync(d_req, reqs, b_req, cudaMemcpyHostToDevice, st)) != cudaSuccess ||
        (ce = cudaMemsetAsync(d_err, 0, 4, st)) != cudaSuccess)
        rc = check_cuda(ce, "affine_mvp: upload");
    if (!rc) rc = launch_affine_mvp(ptr, (const long long *)d_ref, n_ref, (const short *)d_mv,
                                    (const signed char *)d_refi, i_scu, rows, d_req, n, d_out, (int *)d_err, st);
    if (!rc && ((ce = cudaMemcpyAsync(out, d_out, b_out, cudaMemcpyDeviceToHost, st)) != cudaSuccess ||
                (ce = cudaMemcpyAsync(&bad, d_err, 4, cudaMemcpyDeviceToHost, st)) != cudaSuccess))
        rc = check_cuda(ce, "affine_mvp: download");
    cudaFreeAsync(buf, st);
    ce = cudaStreamSynchronize(st);
    cudaStreamDestroy(st);
    if (rc) return rc;
    if (ce != cudaSuccess) return check_cuda(ce, "affine_mvp: synchronise");
    if (bad) return set_status(UC_ERR_ARG, "affine_mvp: requests outside the domain");
    return UC_OK;
}

// ---------------------------------------------------------------------------------------------
// Affine merge candidates: one thread per CU, the reference's derivation order.  Model-based
// candidates: the first two affine neighbours among F, G, C, A, D (same-CU duplicates dropped),
// each neighbour CU's corner MVs (found through its map_pos entry) extrapolated to the CU's
// corners in 1/128 units with the magnitude-rounding shift, a 4-parameter model when the
// neighbour's bottom edge is the CTU row boundary above the CU.  Constructed candidates: LT, RT,
// LB from the first inter neighbour of each corner, RB from the colocated picture (scaled by POC
// distances), combined in the 6 model orders while the list has room.  Every read of the maps is
// bounds-checked; a request with an out-of-field read gets a zeroed result and is counted.
// Records are assembled in shared memory and written out by the CTA as contiguous words.
// ---------------------------------------------------------------------------------------------
static_assert(sizeof(uavs3e_cuda_affmrg_req_t) == 8, "affine merge request layout");
static_assert(sizeof(uavs3e_cuda_affmrg_out_t) == 260, "affine merge result layout");
static_assert(sizeof(uavs3e_cuda_affmrg_pic_t) == 184, "affine merge picture layout");

struct AmrgMaps {
    const short *mv; const signed char *refi; const unsigned char *scu; const unsigned *pos;
    const short *col_mv; const signed char *col_refi;
    long long origin, nf;
};

struct AmrgReader {
    const AmrgMaps &M;
    bool bad;
    __device__ bool in(long long a)
    {
        const long long k = a + M.origin;
        if (k < 0 || k >= M.nf) { bad = true; return false; }
        return true;
    }
    __device__ int scu(long long a) { return in(a) ? M.scu[a + M.origin] : 0; }
    __device__ unsigned pos(long long a) { return in(a) ? M.pos[a + M.origin] : 0u; }
    __device__ int refi(long long a, int l) { return in(a) ? M.refi[(a + M.origin) * 2 + l] : -1; }
    __device__ int mv(long long a, int l, int d) { return in(a) ? M.mv[((a + M.origin) * 2 + l) * 2 + d] : 0; }
};

__device__ __forceinline__ int amrg_round7(int v)
{
    return v >= 0 ? (int)(((unsigned)v + 64u) >> 7) : -(int)(((unsigned)(-(long long)v) + 64u) >> 7);
}

__device__ __forceinline__ int amrg_clip18(int v) { return max(-131072, min(131071, v)); }

__device__ __forceinline__ int amrg_shl(int v, int s) { return (int)((unsigned)v << s); }

// scaling_mv1 of an MV (x, y): false on a zero POC distance
__device__ __forceinline__ bool amrg_scale(long long cur, long long cur_ref, long long neb, long long neb_ref, int mx,
                                           int my, int &ox, int &oy)
{
    const int t0 = (int)(neb * 2 - neb_ref * 2), t1 = (int)(cur * 2 - cur_ref * 2);
    if (t0 == 0 || t1 == 0) return false;
    const int ratio = (1 << 14) / t0 * t1;
    ox = amvp_scale(mx, ratio);
    oy = amvp_scale(my, ratio);
    return true;
}

// com_derive_affine_model_mv: control points of the CU at scup from the affine CU covering scun
__device__ void amrg_model(AmrgReader &R, const uavs3e_cuda_affmrg_pic_t &P, int scup, int scun, int l, int cw, int ch,
                           int (*mvp)[2], int &vn)
{
    const int i_scu = P.i_scu;
    const unsigned pos = R.pos(scun);
    const int lw = (int)(pos & 7), lh = (int)((pos >> 3) & 7), nw = 1 << lw, nh = 1 << lh;
    const int a0 = (int)(pos >> 6), a1 = a0 + ((nw >> 2) - 1), a2 = a0 + ((nh >> 2) - 1) * i_scu, a3 = a2 + ((nw >> 2) - 1);
    const int neb_x = (a0 % i_scu) << 2;
    int neb_y = (a0 / i_scu) << 2;
    const int cur_x = (scup % i_scu) << 2, cur_y = (scup / i_scu) << 2;
    int m0x = R.mv(a0, l, 0), m0y = R.mv(a0, l, 1), m1x = R.mv(a1, l, 0), m1y = R.mv(a1, l, 1);
    const int m2x = R.mv(a2, l, 0), m2y = R.mv(a2, l, 1), m3x = R.mv(a3, l, 0), m3y = R.mv(a3, l, 1);
    bool top = false;
    if ((neb_y + nh) % (1 << P.log2_max_cuwh) == 0 && neb_y + nh == cur_y) {
        top = true;
        neb_y += nh;
        m0x = m2x; m0y = m2y; m1x = m3x; m1y = m3y;
    }
    const int dhx = amrg_shl(m1x - m0x, 7 - lw), dhy = amrg_shl(m1y - m0y, 7 - lw);
    int dvx, dvy;
    if (vn == 3 && !top) {
        dvx = amrg_shl(m2x - m0x, 7 - lh);
        dvy = amrg_shl(m2y - m0y, 7 - lh);
    } else {
        dvx = -dhy;
        dvy = dhx;
        vn = 2;
    }
    const int hb = amrg_shl(m0x, 7), vb = amrg_shl(m0y, 7);
    for (int k = 0; k < vn; k++) {
        const int ox = cur_x - neb_x + (k == 1 ? cw : 0), oy = cur_y - neb_y + (k == 2 ? ch : 0);
        const int th = (int)((unsigned)dhx * (unsigned)ox + (unsigned)dvx * (unsigned)oy + (unsigned)hb);
        const int tv = (int)((unsigned)dhy * (unsigned)ox + (unsigned)dvy * (unsigned)oy + (unsigned)vb);
        mvp[k][0] = amrg_clip18(amrg_shl(amrg_round7(th), 2));
        mvp[k][1] = amrg_clip18(amrg_shl(amrg_round7(tv), 2));
    }
}

// com_derive_affine_constructed_candidate for the control points c0, c1[, c2] of model m
__device__ void amrg_construct(uavs3e_cuda_affmrg_out_t &o, int &cnt, int cw, int ch, const bool *valid,
                               const int (*cmv)[4][2], const int (*crefi)[4], int c0, int c1, int c2, int m, int ver)
{
    if (cnt >= 5) return;
    const int idx[3] = { c0, c1, c2 };
    for (int i = 0; i < ver; i++)
        if (!valid[idx[i]]) return;
    bool vm[2];
    for (int l = 0; l < 2; l++) {
        bool ok = true;
        for (int i = 0; i < ver; i++) ok = ok && crefi[l][idx[i]] >= 0 && crefi[l][idx[i]] == crefi[l][c0];
        vm[l] = ok;
    }
    if (!vm[0] && !vm[1]) return;
    o.cp_num[cnt] = (signed char)ver;
    const int sh = 7 + (31 - __clz(cw)) - (31 - __clz(ch));
    for (int l = 0; l < 2; l++) {
        if (!vm[l]) {
            o.refi[cnt][l] = -1;
            for (int i = 0; i < ver; i++) o.cpmv[cnt][l][i][0] = o.cpmv[cnt][l][i][1] = 0;
            continue;
        }
        int t[4][2] = { { 0, 0 }, { 0, 0 }, { 0, 0 }, { 0, 0 } };
        for (int i = 0; i < ver; i++) { t[idx[i]][0] = cmv[l][idx[i]][0]; t[idx[i]][1] = cmv[l][idx[i]][1]; }
        for (int d = 0; d < 2; d++) {
            if (m == 1) t[2][d] = t[3][d] + t[0][d] - t[1][d];
            if (m == 2) t[1][d] = t[3][d] + t[0][d] - t[2][d];
            if (m == 3) t[0][d] = t[1][d] + t[2][d] - t[3][d];
        }
        if (m == 5) {
            const int th = (int)((unsigned)amrg_shl(t[2][1] - t[0][1], sh) + (unsigned)amrg_shl(t[0][0], 7));
            const int tv = (int)((unsigned)(-amrg_shl(t[2][0] - t[0][0], sh)) + (unsigned)amrg_shl(t[0][1], 7));
            t[1][0] = amrg_round7(th);
            t[1][1] = amrg_round7(tv);
        }
        o.refi[cnt][l] = (signed char)crefi[l][c0];
        for (int i = 0; i < ver; i++)
            for (int d = 0; d < 2; d++) o.cpmv[cnt][l][i][d] = amrg_clip18(amrg_shl(t[i][d], 2));
    }
    cnt++;
}

__device__ bool amrg_one(const uavs3e_cuda_affmrg_pic_t &P, const AmrgMaps &M, const uavs3e_cuda_affmrg_req_t q,
                         uavs3e_cuda_affmrg_out_t &o)
{
    const int cw = q.cu_width, ch = q.cu_height;
    if ((cw != 16 && cw != 32 && cw != 64 && cw != 128) || (ch != 16 && ch != 32 && ch != 64 && ch != 128)) return false;
    AmrgReader R{ M, false };
    const int i_scu = P.i_scu, scup = q.scup, wsc = cw >> 2, hsc = ch >> 2;
    int cnt = 0;
    {
        const int nb[5] = { scup + i_scu * (hsc - 1) - 1, scup - i_scu + wsc - 1, scup - i_scu + wsc, scup - 1,
                            scup - i_scu - 1 };
        int aff[5], tl[5];
        bool valid[5];
        for (int k = 0; k < 5; k++) {
            aff[k] = (R.scu(nb[k]) >> 4) & 3;
            valid[k] = aff[k] != 0;
            tl[k] = valid[k] ? (int)(R.pos(nb[k]) >> 6) : 0;
        }
        if (valid[2] && valid[1] && tl[1] == tl[2]) valid[2] = false;
        const bool v3 = valid[3];
        if (valid[3] && valid[0] && tl[0] == tl[3]) valid[3] = false;
        if ((valid[4] && v3 && tl[4] == tl[3]) || (valid[4] && valid[1] && tl[4] == tl[1])) valid[4] = false;
        for (int k = 0; k < 5 && cnt < 2; k++) {
            if (!valid[k]) continue;
            int vn = aff[k] == 1 ? 2 : 3;
            for (int l = 0; l < 2; l++) {
                const int r = R.refi(nb[k], l);
                if (r >= 0) {
                    o.refi[cnt][l] = (signed char)r;
                    amrg_model(R, P, scup, nb[k], l, cw, ch, o.cpmv[cnt][l], vn);
                } else {
                    o.refi[cnt][l] = -1;
                    for (int i = 0; i < 3; i++) o.cpmv[cnt][l][i][0] = o.cpmv[cnt][l][i][1] = 0;
                }
            }
            o.cp_num[cnt] = (signed char)vn;
            cnt++;
        }
    }
    {
        int cmv[2][4][2], crefi[2][4];
        bool valid[4] = { false, false, false, false };
        for (int l = 0; l < 2; l++)
            for (int i = 0; i < 4; i++) { cmv[l][i][0] = cmv[l][i][1] = 0; crefi[l][i] = -1; }
        const int corner[6] = { scup - 1, scup - i_scu, scup - i_scu - 1, scup - i_scu + wsc - 1, scup - i_scu + wsc,
                                scup + i_scu * (hsc - 1) - 1 };
        const int first[4] = { 0, 3, 5, 6 };
        for (int g = 0; g < 3; g++) {
            for (int k = first[g]; k < first[g + 1]; k++) {
                const int a = corner[k];
                if ((R.scu(a) & 3) != 1) continue;
                for (int l = 0; l < 2; l++) {
                    crefi[l][g] = R.refi(a, l);
                    cmv[l][g][0] = R.mv(a, l, 0);
                    cmv[l][g][1] = R.mv(a, l, 1);
                }
                valid[g] = true;
                break;
            }
        }
        const int rb = scup + i_scu * (hsc - 1) + (wsc - 1);
        const int bx = rb % i_scu, by = rb / i_scu;
        int xpos = (bx & ~3) + 2, ypos = (by & ~3) + 2;
        if (ypos >= P.pic_height_in_scu) ypos = ((by & ~3) + P.pic_height_in_scu) >> 1;
        if (xpos >= P.pic_width_in_scu) xpos = ((bx & ~3) + P.pic_width_in_scu) >> 1;
        const long long co = (long long)ypos * i_scu + xpos + M.origin;
        if (co < 0 || co >= M.nf) return false;
        const int cr = M.col_refi[co * 2];
        const int cx = M.col_mv[co * 4 + 0], cy = M.col_mv[co * 4 + 1];
        if (cr >= 17) return false;
        if (cr >= 0) {
            if (P.slice_type == 3) {
                for (int l = 0; l < 2; l++) {
                    if (!amrg_scale(P.ptr, P.ref0_ptr[l], P.ref0_ptr[1], P.col_list_ptr[cr], cx, cy, cmv[l][3][0], cmv[l][3][1]))
                        return false;
                    crefi[l][3] = 0;
                }
            } else {
                if (!amrg_scale(P.ptr, P.ref0_ptr[0], P.ref0_ptr[0], P.col_list_ptr[cr], cx, cy, cmv[0][3][0], cmv[0][3][1]))
                    return false;
                crefi[0][3] = 0;
                crefi[1][3] = -1;
            }
            valid[3] = true;
        }
        amrg_construct(o, cnt, cw, ch, valid, cmv, crefi, 0, 1, 2, 0, 3);
        amrg_construct(o, cnt, cw, ch, valid, cmv, crefi, 0, 1, 3, 1, 3);
        amrg_construct(o, cnt, cw, ch, valid, cmv, crefi, 0, 2, 3, 2, 3);
        amrg_construct(o, cnt, cw, ch, valid, cmv, crefi, 1, 2, 3, 3, 3);
        amrg_construct(o, cnt, cw, ch, valid, cmv, crefi, 0, 1, 0, 4, 2);
        amrg_construct(o, cnt, cw, ch, valid, cmv, crefi, 0, 2, 0, 5, 2);
    }
    o.num = cnt;
    for (int k = cnt; k < 5; k++) {
        o.cp_num[k] = 2;
        o.refi[k][0] = 0;
        o.refi[k][1] = -1;
    }
    for (int k = 0; k < 5; k++)
        for (int l = 0; l < 2; l++)
            for (int i = (k < cnt ? o.cp_num[k] : 0); i < 3; i++) o.cpmv[k][l][i][0] = o.cpmv[k][l][i][1] = 0;
    return !R.bad;
}

constexpr int AMRG_THREADS = 128;

__global__ void __launch_bounds__(AMRG_THREADS) k_affine_merge(const uavs3e_cuda_affmrg_pic_t P, AmrgMaps M,
                                                              const uavs3e_cuda_affmrg_req_t *reqs, int n,
                                                              uavs3e_cuda_affmrg_out_t *out, int *err)
{
    __shared__ uavs3e_cuda_affmrg_out_t s_out[AMRG_THREADS];
    const int base = blockIdx.x * AMRG_THREADS, i = base + threadIdx.x;
    if (i < n) {
        uavs3e_cuda_affmrg_out_t o;
        memset(&o, 0, sizeof(o));
        if (!amrg_one(P, M, reqs[i], o)) {
            memset(&o, 0, sizeof(o));
            if (err) atomicAdd(err, 1);
        }
        s_out[threadIdx.x] = o;
    }
    __syncthreads();
    // the CTA's records are contiguous: copy them out as words
    const int nrec = min(AMRG_THREADS, n - base);
    const unsigned *src = reinterpret_cast<const unsigned *>(s_out);
    unsigned *dst = reinterpret_cast<unsigned *>(out + base);
    const int words = nrec * (int)(sizeof(uavs3e_cuda_affmrg_out_t) / 4);
    for (int w = threadIdx.x; w < words; w += AMRG_THREADS) dst[w] = src[w];
}

int launch_affine_merge(const uavs3e_cuda_affmrg_pic_t &pic, const short *d_mv, const signed char *d_refi,
                        const unsigned char *d_scu, const unsigned *d_pos, const short *d_col_mv,
                        const signed char *d_col_refi, const uavs3e_cuda_affmrg_req_t *d_reqs, int n,
                        uavs3e_cuda_affmrg_out_t *d_out, int *d_err, cudaStream_t st)
{
    if (n < 0 || pic.i_scu < 3 || pic.rows < 2 || pic.pic_width_in_scu < 1 || pic.pic_height_in_scu < 1 ||
        pic.log2_max_cuwh < 2 || pic.log2_max_cuwh > 7 ||
        (n > 0 && (!d_mv || !d_refi || !d_scu || !d_pos || !d_col_mv || !d_col_refi || !d_reqs || !d_out)))
        return set_status(UC_ERR_ARG, "affine_merge: bad argument");
    if (((uintptr_t)d_mv & 3) || ((uintptr_t)d_col_mv & 3) || ((uintptr_t)d_pos & 3) || ((uintptr_t)d_out & 3))
        return set_status(UC_ERR_ARG, "affine_merge: map_mv, col_mv, map_pos or out not 4-byte aligned");
    if (n == 0) return UC_OK;
    AmrgMaps M{ d_mv, d_refi, d_scu, d_pos, d_col_mv, d_col_refi, (long long)pic.i_scu + 1,
                (long long)pic.rows * pic.i_scu };
    k_affine_merge<<<(n + AMRG_THREADS - 1) / AMRG_THREADS, AMRG_THREADS, 0, st>>>(pic, M, d_reqs, n, d_out, d_err);
    UC_CHECK(cudaGetLastError());
    count_launch(1);
    return UC_OK;
}

UAVS3E_CUDA_API int uavs3e_cuda_affine_merge_device(const uavs3e_cuda_affmrg_pic_t *pic, const int16_t *d_map_mv,
                                                    const int8_t *d_map_refi, const uint8_t *d_map_scu,
                                                    const uint32_t *d_map_pos, const int16_t *d_col_mv,
                                                    const int8_t *d_col_refi, const uavs3e_cuda_affmrg_req_t *d_reqs,
                                                    int n, uavs3e_cuda_affmrg_out_t *d_out, int32_t *d_err,
                                                    void *stream)
{
    if (ensure_init()) return uavs3e_cuda_status();
    if (!pic) return set_status(UC_ERR_ARG, "affine_merge: bad argument");
    return launch_affine_merge(*pic, d_map_mv, (const signed char *)d_map_refi, d_map_scu, d_map_pos, d_col_mv,
                               (const signed char *)d_col_refi, d_reqs, n, d_out, (int *)d_err, (cudaStream_t)stream);
}

UAVS3E_CUDA_API int uavs3e_cuda_affine_merge(const uavs3e_cuda_affmrg_pic_t *pic, const int16_t *map_mv,
                                             const int8_t *map_refi, const uint8_t *map_scu,
                                             const uint32_t *map_pos, const int16_t *col_mv, const int8_t *col_refi,
                                             const uavs3e_cuda_affmrg_req_t *reqs, int n,
                                             uavs3e_cuda_affmrg_out_t *out)
{
    int rc = ensure_init();
    if (rc) return rc;
    if (!pic || n < 0 || pic->i_scu < 3 || pic->rows < 2 ||
        (n > 0 && (!map_mv || !map_refi || !map_scu || !map_pos || !col_mv || !col_refi || !reqs || !out)))
        return set_status(UC_ERR_ARG, "affine_merge: bad argument");
    if (n == 0) return UC_OK;
    const size_t field = (size_t)pic->rows * pic->i_scu;
    auto up = [](size_t b) { return (b + 255) & ~(size_t)255; };
    const size_t b_mv = up(field * 8), b_refi = up(field * 2), b_scu = up(field), b_pos = up(field * 4);
    const size_t b_req = up((size_t)n * sizeof(uavs3e_cuda_affmrg_req_t)), b_out = up((size_t)n * sizeof(uavs3e_cuda_affmrg_out_t));
    cudaStream_t st = nullptr;
    UC_CHECK(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    char *buf = nullptr;
    cudaError_t ce = cudaMallocAsync((void **)&buf, 2 * b_mv + 2 * b_refi + b_scu + b_pos + b_req + b_out + 256, st);
    if (ce != cudaSuccess) { cudaStreamDestroy(st); return check_cuda(ce, "affine_merge: allocate"); }
    char *d_mv = buf, *d_refi = d_mv + b_mv, *d_scu = d_refi + b_refi, *d_pos = d_scu + b_scu;
    char *d_cmv = d_pos + b_pos, *d_crefi = d_cmv + b_mv, *d_req = d_crefi + b_refi, *d_out = d_req + b_req;
    char *d_err = d_out + b_out;
    int bad = 0;
    rc = UC_OK;
    if ((ce = cudaMemcpyAsync(d_mv, map_mv, field * 8, cudaMemcpyHostToDevice, st)) != cudaSuccess ||
        (ce = cudaMemcpyAsync(d_refi, map_refi, field * 2, cudaMemcpyHostToDevice, st)) != cudaSuccess ||
        (ce = cudaMemcpyAsync(d_scu, map_scu, field, cudaMemcpyHostToDevice, st)) != cudaSuccess ||
        (ce = cudaMemcpyAsync(d_pos, map_pos, field * 4, cudaMemcpyHostToDevice, st)) != cudaSuccess ||
        (ce = cudaMemcpyAsync(d_cmv, col_mv, field * 8, cudaMemcpyHostToDevice, st)) != cudaSuccess ||
        (ce = cudaMemcpyAsync(d_crefi, col_refi, field * 2, cudaMemcpyHostToDevice, st)) != cudaSuccess ||
        (ce = cudaMemcpyAsync(d_req, reqs, (size_t)n * sizeof(uavs3e_cuda_affmrg_req_t), cudaMemcpyHostToDevice, st)) !=
            cudaSuccess ||
        (ce = cudaMemsetAsync(d_err, 0, 4, st)) != cudaSuccess)
        rc = check_cuda(ce, "affine_merge: upload");
    if (!rc)
        rc = launch_affine_merge(*pic, (const short *)d_mv, (const signed char *)d_refi, (const unsigned char *)d_scu,
                                 (const unsigned *)d_pos, (const short *)d_cmv, (const signed char *)d_crefi,
                                 (const uavs3e_cuda_affmrg_req_t *)d_req, n, (uavs3e_cuda_affmrg_out_t *)d_out,
                                 (int *)d_err, st);
    if (!rc && ((ce = cudaMemcpyAsync(out, d_out, (size_t)n * sizeof(uavs3e_cuda_affmrg_out_t), cudaMemcpyDeviceToHost,
                                      st)) != cudaSuccess ||
                (ce = cudaMemcpyAsync(&bad, d_err, 4, cudaMemcpyDeviceToHost, st)) != cudaSuccess))
        rc = check_cuda(ce, "affine_merge: download");
    cudaFreeAsync(buf, st);
    ce = cudaStreamSynchronize(st);
    cudaStreamDestroy(st);
    if (rc) return rc;
    if (ce != cudaSuccess) return check_cuda(ce, "affine_merge: synchronise");
    if (bad) return set_status(UC_ERR_ARG, "affine_merge: requests outside the domain");
    return UC_OK;
}
