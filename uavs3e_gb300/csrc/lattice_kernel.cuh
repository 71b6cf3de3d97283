// Device side of the batched intra lattice: the tile body of every CU shape class; the
// persistent kernel, the device work queue, the layout tuner and the C ABI are in lattice.cu.
#pragma once
#include "common.cuh"
#include "had.cuh"
#include "intra.cuh"
#include "tables.h"
#include "uavs3e_cuda_internal.h"
#include "quant_tables.cuh"

#include <type_traits>

namespace uc {

static const u32 hDqScale[80] = {
    32768, 36061, 38968, 42495, 46341, 50535, 55437, 60424, 32932, 35734, 38968, 42495, 46177, 50535, 55109, 59933,
    65535, 35734, 38968, 42577, 46341, 50617, 55027, 60097, 32809, 35734, 38968, 42454, 46382, 50576, 55109, 60056,
    65535, 35734, 38968, 42495, 46320, 50515, 55109, 60076, 65535, 35744, 38968, 42495, 46341, 50535, 55099, 60087,
    65535, 35734, 38973, 42500, 46341, 50535, 55109, 60097, 32771, 35734, 38965, 42497, 46341, 50535, 55109, 60099,
    32768, 36061, 38968, 42495, 46341, 50535, 55437, 60424, 32932, 35734, 38968, 42495, 46177, 50535, 55109, 59933,
};
static const u8 hDqShift[80] = {
    14, 14, 14, 14, 14, 14, 14, 14, 13, 13, 13, 13, 13, 13, 13, 13, 13, 12, 12, 12, 12, 12, 12, 12,
    11, 11, 11, 11, 11, 11, 11, 11, 11, 10, 10, 10, 10, 10, 10, 10, 10, 9, 9, 9, 9, 9, 9, 9,
    9, 8, 8, 8, 8, 8, 8, 8, 7, 7, 7, 7, 7, 7, 7, 7, 6, 6, 6, 6, 6, 6, 6, 6, 5, 5, 5, 5, 5, 5, 5, 5,
};

// sum of 4 (unsigned byte of a) x (signed byte of b) products + c
__device__ __forceinline__ int dp4a_us(u32 a, u32 b, int c)
{
    int d;
    asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
// sum of the 2 signed halfwords of a times signed bytes 0,1 (lo) or 2,3 (hi) of b, + c
__device__ __forceinline__ int dp2a_lo(u32 a, u32 b, int c)
{
    int d;
    asm("dp2a.lo.s32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
__device__ __forceinline__ int dp2a_hi(u32 a, u32 b, int c)
{
    int d;
    asm("dp2a.hi.s32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}

struct LatCu { s16 x, y; u8 w, h; u16 pad; };
struct LatQ { u32 ssd; u32 coef_hash; u16 num_nz; s16 last_nz; u32 sum_abs; };

struct alignas(8) LatPerm { int id; s16 x, y; };   // a CU of a class: its index and position

constexpr int LAT_THREADS = 256;
constexpr int LAT_BUDGET = 50 * 1024;   // default dynamic shared bytes per CTA (4 CTAs per SM with the static part)
constexpr int LAT_MAX_QP = 4;
constexpr int LAT_SMEM_MAX = 96 * 1024;   // dynamic shared memory admitted by the kernel attribute
constexpr int LAT_MAX_G = 8;            // CUs per CTA
constexpr int LAT_MAX_JOBS = 132;       // (CU, mode) jobs of a tile: 4 CUs of 33 modes
constexpr int LAT_NB = 592;             // neighbour buffer per CU (INTRA_NEIB_SIZE + pad)
constexpr int LAT_SHAPES = 25;          // log2 sides 2..6
constexpr int LAT_NO_MODE = 33;         // a list entry that is no mode (above 32): a job without records

// shared-memory layout of one shape's CTAs (host and device compute it the same way)
struct LatLayout {
    int w, h, lw, lh, kw, kh, lkw;
    int ps;            // prediction / org row stride (bytes): 16-byte aligned rows
    int ts;            // forward row-pass output row stride (s16): 16-byte aligned rows
    int cs;            // coefficient row stride (s16): 16-byte aligned rows
    int ds;            // transposed dequantised row stride (s16): 16-byte aligned rows
    int t2s;           // inverse column-pass output row stride (s16): 16-byte aligned rows
    int fw_ws, fh_ws, fht_ws, fwt_ws;   // table row strides in words
    int o_fw, o_fh, o_fht, o_fwt;       // table offsets
    int o_scan;                         // scan index of each kept coefficient, [v][u] (u16)
    int o_cu, cu_bytes;                 // per-CU blocks: org, neighbours, org row-pass sums
    int c_org, c_nb, c_torg;
    int o_job, job_bytes;               // per-job blocks: prediction, T, C, DQ^T, T2
    int j_pred, j_t, j_c, j_dqt, j_t2;
    int G, MC, nchunk;                  // CUs per CTA, modes per CTA, mode chunks per CU
    int smem;
};

__host__ __device__ __forceinline__ int lat_up16(int v) { return (v + 15) & ~15; }

// row stride for rows of n words (n = 2, 4, 8, 16) read 8 bytes per lane: n + 2 is twice an odd number but
// for n = 2
__host__ __device__ constexpr int lat_pair_stride(int n) { return n == 2 ? 6 : n + 2; }

// the layout of a CTA for (2^lw) x (2^lh) CUs, nm modes and n_qp QPs within `budget` bytes of dynamic
// shared memory: how many CUs (or which chunk of one CU's modes) a CTA takes
__host__ __device__ inline void lat_layout(int lw, int lh, int nm, int n_qp, int budget, LatLayout &L)
{
    L.lw = lw; L.lh = lh; L.w = 1 << lw; L.h = 1 << lh;
    L.kw = L.w < 32 ? L.w : 32; L.kh = L.h < 32 ? L.h : 32;
    L.lkw = lw < 5 ? lw : 5;
    // rows that are read whole by every lane of a warp (broadcast) start on 16 bytes; the
    // strides also keep the rows 8 lanes read at once on distinct banks
    L.ps = L.w <= 8 ? 16 : L.w <= 32 ? 48 : 80;
    L.ts = L.h >= 8 ? L.h + 8 : 8;
    L.cs = L.kw >= 8 ? L.kw + 8 : 8;
    L.ds = L.kh >= 8 ? L.kh + 8 : 8;
    L.t2s = L.kw >= 8 ? L.kw + 8 : 8;
    // matrix rows are read one per lane, a chunk in one load: 16 bytes of a forward row matrix, 8 of the
    // others, at strides (in words) that keep those loads on distinct banks
    L.fw_ws = L.w >= 32 ? L.w / 4 + 4 : L.w == 16 ? 12 : L.w == 8 ? 6 : 1;
    L.fh_ws = L.h >= 8 ? lat_pair_stride(L.h / 4) : 1;
    L.fht_ws = L.kh >= 8 ? lat_pair_stride(L.kh / 4) : 1;
    L.fwt_ws = L.kw >= 8 ? lat_pair_stride(L.kw / 4) : 1;
    int o = 0;
    // without a QP (SATD records only) a tile has neither tables nor transform buffers
    const int tr = n_qp > 0 ? 1 : 0;
    L.o_fw = o; o += tr * lat_up16(L.kw * L.fw_ws * 4);
    L.o_fh = o; o += tr * lat_up16(L.kh * L.fh_ws * 4);
    L.o_fht = o; o += tr * lat_up16(L.h / 2 * L.fht_ws * 4);
    L.o_fwt = o; o += tr * lat_up16(L.w / 2 * L.fwt_ws * 4);
    L.o_scan = o; o += tr * lat_up16(L.kw * L.kh * 2);
    int c = 0;
    L.c_org = c; c += lat_up16(L.h * L.ps);
    L.c_nb = c; c += lat_up16(LAT_NB);
    L.c_torg = c; c += tr * lat_up16(L.kw * L.h * 4);
    L.cu_bytes = c;
    int j = 0;
    L.j_pred = j; j += lat_up16(L.h * L.ps);
    const int b_t = lat_up16(L.kw * L.ts * 2), b_t2 = lat_up16(L.h * L.t2s * 2);
    // T is dead once C is formed, and C once the levels of the last QP are: T2 takes T's place, and with one
    // QP DQT^T takes T's and T2 C's.  (Two QPs at a time, sharing the reads of C, took 24 % more bytes a
    // job and was slower.)
    const int b_c = lat_up16(L.kh * L.cs * 2), b_dqt = lat_up16(L.kw * L.ds * 2);
    if (n_qp > 1) {
        L.j_t = L.j_t2 = j; j += b_t2 > b_t ? b_t2 : b_t;
        L.j_c = j; j += b_c;
        L.j_dqt = j; j += b_dqt;
    } else {
        L.j_t = L.j_dqt = j; j += tr * (b_dqt > b_t ? b_dqt : b_t);
        L.j_c = L.j_t2 = j; j += tr * (b_t2 > b_c ? b_t2 : b_c);
    }
    // an odd multiple of 16 bytes: where a warp holds several jobs, their rows lie on different banks
    // (at a multiple of 128 the quantisation of 4x4 blocks took twice the time)
    L.job_bytes = j | 16;
    const int avail = budget - o;
    // several whole CUs when nm jobs of the shape fit, else one CU and a chunk of its modes
    int G = avail / (nm * L.job_bytes + L.cu_bytes);
    if (G >= 1) {
        L.G = G < LAT_MAX_G ? G : LAT_MAX_G;
        if (L.G * nm > LAT_MAX_JOBS) L.G = LAT_MAX_JOBS / nm;
        L.MC = nm; L.nchunk = 1;
    } else {
        int J = (avail - L.cu_bytes) / L.job_bytes;
        J = J < 1 ? 1 : J;
        L.G = 1;
        L.nchunk = (nm + J - 1) / J;
        L.MC = (nm + L.nchunk - 1) / L.nchunk;
    }
    L.o_cu = o; o += L.G * L.cu_bytes;
    L.o_job = o; o += L.G * L.MC * L.job_bytes;
    L.smem = o;
}

// what a QP means for a CU size: the quantisation multiplier, the magnitude above which a coefficient makes
// quant_check code the block, and the dequantisation.  Formed on the host: a division and four table reads
// per QP, thread and tile otherwise.
struct LatQp { int q_value, thr, dq_scale, dq_shift; };
__host__ __device__ constexpr int lat_q_bits(int log2_size) { return 14 + (15 - 8 - log2_size); }

inline LatQp lat_qp(int qp, int l_samples, int is_intra)
{
    const int odd = l_samples & 1, log2_size = l_samples >> 1, q_bits = lat_q_bits(log2_size);
    const int offset = (is_intra ? 201 : 153) << (q_bits - 9);
    LatQp o;
    o.q_value = ((int)hQScale[qp] * (odd ? 181 : 1) + (odd ? 64 : 0)) >> (odd ? 7 : 0);
    o.thr = ((((1 << q_bits) - offset) << 10) / o.q_value - 1) >> 10;
    o.dq_scale = (int)hDqScale[qp];
    o.dq_shift = (int)hDqShift[qp] - (15 - 8 - log2_size) + 1;
    return o;
}

struct LatParams {
    const pel *org; int i_org;
    int org_words;            // org and i_org are multiples of 4: org blocks are read by words
    const pel *rec; int i_rec;
    int W, H;
    int ipf, n_qp;
    LatQp qp[9][LAT_MAX_QP];  // [log2 of the samples of a CU - 4][QP]
    u32 *satd_out; LatQ *q_out;
    const u8 *images;         // [class][LAT_IMAGE_BYTES] transform and scan tables (lat_image_fill)
    const u32 *ipred;         // the prediction table (lat_table_at)
    const u8 *modes;          // [CU][n_modes] modes to evaluate, or null for all 33 in order
    int n_modes;
    int budget[LAT_SHAPES];   // dynamic shared bytes of each shape class's layout (lat_layout)
    double sq32, sq128;
    u64 k32, k128;       // had_scale_k of sq32, sq128
    // the device work queue (written by k_lat_plan for each launch)
    const int *counts;        // [LAT_SHAPES] CUs per shape class
    const int *cu_off;        // [LAT_SHAPES] first entry of each class in perm
    const int *tile_off;      // [LAT_SHAPES + 1] first tile of the class of each launch rank; [25] = total
    const LatPerm *perm;      // the CUs grouped by class
    int *next;                // the next tile to take
};

// per-CTA shared scalars of a tile (the static part of the tile's shared memory)
struct LatShared {
    IpredBlock B[LAT_MAX_G];
    LatPerm cu[LAT_MAX_G];
    u8 mode[LAT_MAX_JOBS];
    u32 satd[LAT_MAX_JOBS], ssd0[LAT_MAX_JOBS];   // ssd0: of the prediction, for QPs that code nothing
    u32 flag[LAT_MAX_JOBS];   // bit q: QP q codes the job
    // of the QP at hand: the statistics and the SSD.  nz also has bits 16 + k / 20 + k: chunk k of eight
    // columns / rows holds a level
    u32 nz[LAT_MAX_JOBS], sum[LAT_MAX_JOBS], hash[LAT_MAX_JOBS], ssd[LAT_MAX_JOBS];
    int last[LAT_MAX_JOBS];
    u8 list[LAT_MAX_QP][LAT_MAX_JOBS];   // the jobs that each QP codes
    int coded[LAT_MAX_QP];               // and how many
    int tile_off[LAT_SHAPES + 1], cu_off[LAT_SHAPES], counts[LAT_SHAPES];   // of the queue (LatParams)
    int next[2], rank[2];           // the tile after this one and its launch rank, by the tile's parity
    int tables;   // shape class whose matrices and scan table are in place (-1: none)
};

// lanes [k*seg, (k+1)*seg) of a warp hold one job's elements (seg = 16 or 32): the sum or
// max over the lane's segment, with the warp-wide reduction instructions
__device__ __forceinline__ u32 seg_sum(u32 v, int seg, int lane)
{
    if (seg == 32) return __reduce_add_sync(0xFFFFFFFFu, v);
    const u32 lo = __reduce_add_sync(0xFFFFFFFFu, lane < 16 ? v : 0u);
    const u32 hi = __reduce_add_sync(0xFFFFFFFFu, lane < 16 ? 0u : v);
    return lane < 16 ? lo : hi;
}
__device__ __forceinline__ int seg_max(int v, int seg, int lane)
{
    if (seg == 32) return __reduce_max_sync(0xFFFFFFFFu, v);
    const int lo = __reduce_max_sync(0xFFFFFFFFu, lane < 16 ? v : -1);
    const int hi = __reduce_max_sync(0xFFFFFFFFu, lane < 16 ? -1 : v);
    return lane < 16 ? lo : hi;
}

// NW words of a row that every lane of a warp reads (16-byte aligned): vector loads
template <int NW>
__device__ __forceinline__ void lat_row(const void *p, u32 (&r)[NW])
{
    if constexpr (NW >= 4) {
#pragma unroll
        for (int k = 0; k < NW / 4; k++) {
            const uint4 v = reinterpret_cast<const uint4 *>(p)[k];
            r[4 * k] = v.x; r[4 * k + 1] = v.y; r[4 * k + 2] = v.z; r[4 * k + 3] = v.w;
        }
    } else if constexpr (NW == 2) {
        const uint2 v = *reinterpret_cast<const uint2 *>(p);
        r[0] = v.x; r[1] = v.y;
    } else {
        r[0] = *reinterpret_cast<const u32 *>(p);
    }
}

// position of index k in a row of n entries stored for the even/odd sums: chunks of eight entries (or
// the row of four), in each the even k first and the odd k after them
__host__ __device__ __forceinline__ constexpr int lat_eo(int k, int n)
{
    return n == 4 ? (k & 1) * 2 + (k >> 1) : (k & ~7) + (k & 1) * 4 + ((k & 7) >> 1);
}

// the even parts e[r] and the odd parts o[r] of sum_k F[k] D_r[k] over the first 8 nch of N entries of R rows
// D_r (s16, `pitch` apart) and the row F (bytes at f), both in lat_eo order.  The loop over the chunks is
// not unrolled: the code stays small, and rows that end in zeros cost what they hold.
template <int N, int R>
__device__ __forceinline__ void lat_eo_sums(const s16 *d, int pitch, const u32 *f, int nch, int (&e)[R], int (&o)[R])
{
#pragma unroll
    for (int r = 0; r < R; r++) e[r] = o[r] = 0;
    if constexpr (N == 4) {
        const u32 fw = f[0];
#pragma unroll
        for (int r = 0; r < R; r++) {
            const uint2 v = *reinterpret_cast<const uint2 *>(d + r * pitch);
            e[r] = dp2a_lo(v.x, fw, 0); o[r] = dp2a_hi(v.y, fw, 0);
        }
    } else {
#pragma unroll 1
        for (int c = 0; c < nch; c++, d += 8, f += 2) {
            const uint2 fv = *reinterpret_cast<const uint2 *>(f);
            const u32 fe = fv.x, fo = fv.y;
#pragma unroll
            for (int r = 0; r < R; r++) {
                const uint4 v = *reinterpret_cast<const uint4 *>(d + r * pitch);
                e[r] = dp2a_hi(v.y, fe, dp2a_lo(v.x, fe, e[r]));
                o[r] = dp2a_hi(v.w, fo, dp2a_lo(v.z, fo, o[r]));
            }
        }
    }
}

// two values clipped to s16 and packed, lo in the low half
__device__ __forceinline__ u32 lat_pack16(int lo, int hi)
{
    u32 d;
    asm("cvt.pack.sat.s16.s32 %0, %1, %2;" : "=r"(d) : "r"(hi), "r"(lo));
    return d;
}
// stores NW words of a row (aligned to its size)
template <int NW>
__device__ __forceinline__ void lat_store(void *p, const u32 (&v)[NW])
{
    if constexpr (NW == 4) *reinterpret_cast<uint4 *>(p) = make_uint4(v[0], v[1], v[2], v[3]);
    else *reinterpret_cast<uint2 *>(p) = make_uint2(v[0], v[1]);
}

// sum over aligned groups of SEG lanes (SEG a power of two <= 32)
template <int SEG>
__device__ __forceinline__ u32 lat_seg_sum(u32 v, int lane)
{
    if constexpr (SEG >= 16) {
        return seg_sum(v, SEG, lane);
    } else {
#pragma unroll
        for (int d = 1; d < SEG; d <<= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, d);
        return v;
    }
}

// maximum over aligned groups of SEG lanes
template <int SEG>
__device__ __forceinline__ int lat_seg_max(int v, int lane)
{
    if constexpr (SEG >= 16) {
        return seg_max(v, SEG, lane);
    } else {
#pragma unroll
        for (int d = 1; d < SEG; d <<= 1) v = max(v, __shfl_xor_sync(0xFFFFFFFFu, v, d));
        return v;
    }
}

// com_had tile of a (2^LW) x (2^LH) block (src/com_cost.c:712-812), as constants
constexpr int lat_tw(int w, int h)
{
    return w == h ? (w == 4 ? 4 : 8) : w > h ? (h == 4 ? 8 : 16) : (w == 4 ? 4 : 8);
}
constexpr int lat_th(int w, int h)
{
    return w == h ? (w == 4 ? 4 : 8) : w > h ? (h == 4 ? 4 : 8) : (w == 4 ? 8 : 16);
}

// sum of the squares of the four byte differences of a and b, plus c
__device__ __forceinline__ u32 lat_sq4(u32 a, u32 b, u32 c)
{
    const u32 d = __vabsdiffu4(a, b);
    return __dp4a(d, d, c);
}

// SATD of every (job, tile), a tile row per lane (had.cuh): R = 8 or 4 lanes to a tile, whose two
// squares (16x8 / 8x16 / 8x4 / 4x8 tiles) a lane holds a row of each.  With SSD, the sum of squared
// differences of the prediction, which every QP that codes no level of the job keeps, is added to
// s_ssd0[j] too.
template <int TW, int TH, bool SSD>
__device__ __forceinline__ void lat_satd_tiles(int n_tiles, int lnt, int ntx,
                                               const u8 *cub, int cu_bytes, int c_org,
                                               const u8 *jobb, int job_bytes, int j_pred, int ps, u32 mc_magic,
                                               u32 *s_satd, u32 *s_ssd0, double sq32, double sq128, u64 k32,
                                               u64 k128)
{
    constexpr int R = (TW == 4 || TH == 4) ? 4 : 8;
    constexpr bool PAIR = TW != TH, SIDE = TW > TH;
    constexpr int GPW = 32 / R;                       // groups per warp
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int k = lane % R, grp = lane / R;
    const HadSigns G = had_signs(lane);
    for (int base = warp * GPW; base < n_tiles; base += (LAT_THREADS / 32) * GPW) {
        const int ti = base + grp;
        const bool act = ti < n_tiles;
        const int tt = act ? ti : base;
        const int j = tt >> lnt, t = tt & ((1 << lnt) - 1);
        const int ox = (t % ntx) * TW, oy = (t / ntx) * TH;
        const u8 *o = cub + ((u32)j * mc_magic >> 16) * cu_bytes + c_org + (oy + k) * ps + ox;
        const u8 *p = jobb + j * job_bytes + j_pred + (oy + k) * ps + ox;
        const int bo = SIDE ? R : R * ps;
        int sum;
        u32 sq = 0;
        if constexpr (R == 8) {
            const uint2 ov = *reinterpret_cast<const uint2 *>(o), pv = *reinterpret_cast<const uint2 *>(p);
            int q[4];
            had_diff8(ov.x, ov.y, pv.x, pv.y, q);
            if (SSD) sq = lat_sq4(ov.y, pv.y, lat_sq4(ov.x, pv.x, 0u));
            if constexpr (PAIR) {
                const uint2 ow = *reinterpret_cast<const uint2 *>(o + bo), pw = *reinterpret_cast<const uint2 *>(p + bo);
                int e[4], d[4];
                had_diff8(ow.x, ow.y, pw.x, pw.y, e);
                if (SSD) sq = lat_sq4(ow.y, pw.y, lat_sq4(ow.x, pw.x, sq));
#pragma unroll
                for (int i = 0; i < 4; i++) { d[i] = q[i] - e[i]; q[i] += e[i]; }
                sum = had8_lane(d, G) + had8_lane(q, G);
            } else {
                sum = had8_lane(q, G);
            }
        } else {
            const u32 ov = *reinterpret_cast<const u32 *>(o), pv = *reinterpret_cast<const u32 *>(p);
            const int q0 = (int)(__byte_perm(ov, 0u, 0x4240) - __byte_perm(pv, 0u, 0x4240));
            const int q1 = (int)(__byte_perm(ov, 0u, 0x4341) - __byte_perm(pv, 0u, 0x4341));
            if (SSD) sq = lat_sq4(ov, pv, 0u);
            if constexpr (PAIR) {
                const u32 ow = *reinterpret_cast<const u32 *>(o + bo), pw = *reinterpret_cast<const u32 *>(p + bo);
                const int e0 = (int)(__byte_perm(ow, 0u, 0x4240) - __byte_perm(pw, 0u, 0x4240));
                const int e1 = (int)(__byte_perm(ow, 0u, 0x4341) - __byte_perm(pw, 0u, 0x4341));
                if (SSD) sq = lat_sq4(ow, pw, sq);
                sum = had4_lane(q0 - e0, q1 - e1, G) + had4_lane(q0 + e0, q1 + e1, G);
            } else {
                sum = had4_lane(q0, q1, G);
            }
        }
#pragma unroll
        for (int d = 1; d < R; d <<= 1) {
            sum += __shfl_xor_sync(0xFFFFFFFFu, sum, d);
            if (SSD) sq += __shfl_xor_sync(0xFFFFFFFFu, sq, d);
        }
        sum *= 2;
        if (act && k == 0) {
            u32 v;
            if (!PAIR) v = R == 8 ? (u32)((sum + 2) >> 2) : (u32)((sum + 1) >> 1);
            else v = R == 8 ? had_scale(sum, sq128, k128) : had_scale(sum, sq32, k32);
            if (n_tiles >> lnt == n_tiles) {           // one tile per job
                s_satd[j] = v;
                if (SSD) s_ssd0[j] = sq;
            } else {
                atomicAdd(&s_satd[j], v);
                if (SSD) atomicAdd(&s_ssd0[j], sq);
            }
        }
    }
}

// Prediction table.  A sample of every mode but the plane and the bilinear one is the 4-tap filter of
// f4tap on four reference samples s[base], s[base + d], s[base + 2 d], s[base + 3 d] (d = 1 or -1; or 0,
// which copies s[base]: the horizontal, the vertical and, with the DC value kept at LAT_DC, the DC mode;
// mode 32's 3-tap filter is the 4-tap one with offset 0).  base, d and the filter offset depend on the
// shape, the mode and the sample only, so they are tabulated once per device: one path for 31 modes, where
// the mode's own arithmetic took three times the instructions and, on blocks of less than a warp's
// samples, a pass for each of the modes a warp holds.  An entry is base (16 bits, signed), d (8, signed),
// offset (8); entries are [class][mode][raster sample].  The end-of-reference clamps of the angular modes
// have no place in it: the lattice's neighbour arrays repeat their last sample past 2w / 2h.
constexpr int LAT_DC = -280;                          // where a CU's neighbour array keeps its DC value

// first entry of a class's table
__host__ __device__ constexpr int lat_table_at(int lw, int lh) { return 33 * (((1 << lw) - 4) * 124 + (1 << lw) * ((1 << lh) - 4)); }
constexpr int LAT_TABLE_ENTRIES = 33 * 124 * 124;

static __device__ u32 lat_table_entry(int w, int h, int m, int i, int j)
{
    int base = 0, d = 0, off = 0;
    if (m == 0) base = LAT_DC;
    else if (m == 12) base = 1 + i;
    else if (m == 24) base = -1 - j;
    else if (m >= 3 && m <= 11) { base = ang_ctx(m, 0, j + 1, &off) + i; d = 1; }
    else if (m >= 13 && m <= 23) {
        const int yy = j - ang_ctx(m, 1, i + 1, &off);
        if (yy <= -1) { base = i + 2 - ang_ctx(m, 0, j + 1, &off); d = -1; }
        else { base = -yy - 2; d = 1; }
    } else if (m >= 25 && m <= 31) { base = -j - ang_ctx(m, 1, i + 1, &off); d = -1; }
    else if (m == 32) {
        const int rs = min(h / 2 + w - 1, h), n = (j >> 1) + i;
        base = n >= rs ? -1 - 2 * rs : (j & 1) ? -3 - 2 * n : -2 - 2 * n;
        d = -1;
    }
    return (u32)(u16)(s16)base | (u32)(u8)(s8)d << 16 | (u32)off << 24;
}

// four prediction samples of mode m along the row from (x, y), as bytes (com_intra_pred with ipf)
template <int W, int H>
__device__ __forceinline__ u32 lat_pred4(const u32 *tab, const pel *s, const IpredBlock &B, int m, int ipf, int x, int y)
{
    constexpr int LW_ = W == 4 ? 2 : W == 8 ? 3 : W == 16 ? 4 : W == 32 ? 5 : 6, LH_ = H == 4 ? 2 : H == 8 ? 3 : H == 16 ? 4 : H == 32 ? 5 : 6;
    int v[4];
    const bool own = m == 1 || m == 2;                 // their values enter the IPF unclipped
    if (!own) {
        // (LAT_NO_MODE reads mode 32's row, not past the table)
        const uint4 e4 = __ldg(reinterpret_cast<const uint4 *>(tab + (min(m, 32) * H + y) * W + x));
        const u32 e[4] = { e4.x, e4.y, e4.z, e4.w };
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const pel *p = s + (int)(s16)(e[k] & 0xFFFF);
            const int d = (int)(s8)(u8)(e[k] >> 16), off = (int)(e[k] >> 24);
            const int p0 = p[0], p1 = p[d], p2 = p[2 * d], p3 = p[3 * d];
            v[k] = (32 * (p0 + 2 * p1 + p2) + off * (p2 + p3 - p0 - p1) + 64) >> 7;   // f4tap
        }
    } else if (m == 1) {
#pragma unroll
        for (int k = 0; k < 4; k++) v[k] = (B.pl_t + y * B.pl_c + (x + k) * B.pl_b) >> 5;
    } else {
        constexpr int lxy = LW_ + LH_ + 1, offs = 1 << (LW_ + LH_);
        const int le = s[-y - 1], dx = B.bi_a - le;
        int predx = (le << LW_) + (x + 1) * dx;
#pragma unroll
        for (int k = 0; k < 4; k++, predx += dx) {
            const int up = s[x + k + 1], refup = (up << LH_) + (y + 1) * (B.bi_b - up);
            v[k] = ((predx << LH_) + (refup << LW_) + (x + k) * y * B.bi_wt + offs) >> lxy;
        }
    }
    if (ipf) {
        const int le = s[-y - 1];
        int ih = LW_ - 2, iv = LH_ - 2, vr = H < 10 ? H : 10, hr = W < 10 ? W : 10;
        if (m >= 3 && m <= 18) vr = 0;
        if (m > 18) hr = 0;
        if (y < vr || x < hr) {
            const int ct = y < vr ? kIpfParam[iv][y] : 0;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int cl = x + k < hr ? kIpfParam[ih][x + k] : 0;
                if (y < vr || x + k < hr) v[k] = (cl * le + ct * s[1 + x + k] + (64 - cl - ct) * v[k] + 32) >> 6;
            }
        }
    }
    u32 o = 0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        if (own) v[k] = min(255, max(0, v[k]));
        o |= ((u32)v[k] & 255u) << (8 * k);            // (an IPF value may leave 0..255: stored modulo 256)
    }
    return o;
}

// Optional per-stage clocks (built with UAVS3E_LAT_STAGE_CLOCKS, off in the library): thread 0
// of each CTA adds the SM cycles between consecutive CTA barriers of a tile to
// g_lat_stage_clk[class][stage].  Stages: 0 tables and job setup, 1 org block and neighbours,
// 2 org row-pass sums and block setup, 3 prediction, 4 SATD and forward row pass, 5 forward
// column pass, then per QP 6 quantisation, 7 inverse column pass, 8 inverse row pass,
// reconstruction and SSD, 9 records.
constexpr int LAT_STAGES = 10;
#ifdef UAVS3E_LAT_STAGE_CLOCKS
__device__ unsigned long long g_lat_stage_clk[LAT_SHAPES][LAT_STAGES];
#define LAT_STAGE_BEGIN() long long lat_clk0 = clock64()
#define LAT_STAGE(k)                                                                                       \
    do {                                                                                                  \
        if (threadIdx.x == 0) {                                                                           \
            const long long t_ = clock64();                                                               \
            atomicAdd(&g_lat_stage_clk[(LW - 2) * 5 + (LH - 2)][k], (unsigned long long)(t_ - lat_clk0)); \
            lat_clk0 = t_;                                                                                \
        }                                                                                                 \
    } while (0)
#else
#define LAT_STAGE_BEGIN() do { } while (0)
#define LAT_STAGE(k) do { } while (0)
#endif

__device__ __forceinline__ LatPerm lat_perm(const LatPerm *p)
{
    const int2 v = __ldg(reinterpret_cast<const int2 *>(p));
    return { v.x, (s16)(v.y & 0xFFFF), (s16)(v.y >> 16) };
}

// entry i of a class's table image: fold_w / fold_h are the folded DCT2 matrices, scanpos the scan order
constexpr int LAT_IMAGE_BYTES = 10 * 1024;   // the largest: 9472 (64x64)
static __device__ void lat_image_fill(const s8 *fold_w, const s8 *fold_h, const u16 *scanpos, int lw, int lh, u8 *img)
{
    LatLayout L;
    lat_layout(lw, lh, 1, 1, LAT_BUDGET, L);
    const int w = L.w, h = L.h, kw = L.kw, kh = L.kh;
    for (int i = threadIdx.x; i < kw * w; i += blockDim.x) {
        const int u = i >> lw, x = i & (w - 1);
        const u8 v = (u8)fold_w[u * w + x];
        img[L.o_fw + u * L.fw_ws * 4 + x] = v;        // Fw[u][x]
        if (x < (w >> 1)) img[L.o_fwt + x * L.fwt_ws * 4 + lat_eo(u, kw)] = v;
    }
    for (int i = threadIdx.x; i < kh * h; i += blockDim.x) {
        const int v = i >> lh, y = i & (h - 1);
        const u8 c = (u8)fold_h[v * h + y];
        img[L.o_fh + v * L.fh_ws * 4 + y] = c;        // Fh[v][y]
        if (y < (h >> 1)) img[L.o_fht + y * L.fht_ws * 4 + lat_eo(v, kh)] = c;
    }
    for (int i = threadIdx.x; i < kw * kh; i += blockDim.x)
        ((u16 *)(img + L.o_scan))[i] = scanpos[(i >> L.lkw) * w + (i & (kw - 1))];
}

// One tile of shape class (LW, LH): a few whole CUs, or one CU and a chunk of its modes, as the
// class's layout says.  Called by every thread of the CTA; the tile's data lives in `sm` (the
// layout's dynamic shared memory) and `S`.
template <int LW, int LH>
__device__ __forceinline__ void lat_tile(const LatParams &P, const LatPerm *perm, int n_shape, int tile, u8 *sm,
                                         LatShared &S)
{
    IpredBlock *sB = S.B;
    u8 *s_mode = S.mode;
    u32 *s_satd = S.satd, *s_flag = S.flag;

    LatLayout L;
    LAT_STAGE_BEGIN();
    // compile-time shape: the indices and trip counts below are constants
    lat_layout(LW, LH, P.n_modes, P.n_qp, P.budget[(LW - 2) * 5 + (LH - 2)], L);
    const int w = L.w, h = L.h, lw = L.lw, lh = L.lh, kw = L.kw, lkw = L.lkw;
    const int N = w * h, lN = lw + lh;
    constexpr int W_ = 1 << LW, H_ = 1 << LH, KW_ = W_ < 32 ? W_ : 32, KH_ = H_ < 32 ? H_ : 32;
    constexpr int LKW_ = LW < 5 ? LW : 5, LKH_ = LH < 5 ? LH : 5;
    // row passes: a task is one matrix row (in registers) against RY data rows; column passes:
    // against RU data columns.  Lanes of a warp take consecutive matrix rows, so the data row
    // they read is the same (one broadcast load).
    constexpr int RY = H_ < 8 ? H_ : 8, NYC = H_ / RY;
    constexpr int RU = KW_ < 8 ? KW_ : 8, NUC = KW_ / RU;
    const int tid = threadIdx.x, lane = tid & 31, wbase = tid & ~31;

    // this tile's CUs and modes
    const int grp = tile / L.nchunk, chunk = tile % L.nchunk;
    const int cu0 = grp * L.G;
    const int Gv = min(L.G, n_shape - cu0);
    const int m0 = chunk * P.n_modes / L.nchunk;          // chunks differ by one mode at most
    const int MCv = (chunk + 1) * P.n_modes / L.nchunk - m0;
    const int J = Gv * MCv;
    if (Gv <= 0 || MCv <= 0) return;
    // j / MCv as a multiply: with m = ceil(2^16 / MCv), (j m) >> 16 = j / MCv for every
    // j * MCv < 2^16 (here j < LAT_MAX_JOBS and MCv <= 33)
    const u32 mc_magic = (65536u + (u32)MCv - 1u) / (u32)MCv;

    const u32 *fw = (const u32 *)(sm + L.o_fw), *fh = (const u32 *)(sm + L.o_fh);
    const u32 *fht = (const u32 *)(sm + L.o_fht), *fwt = (const u32 *)(sm + L.o_fwt);
    u8 *cub = sm + L.o_cu, *jobb = sm + L.o_job;

    // job j -> (CU g, mode m): j = g * MCv + (m - m0)
#define JG(j) ((int)(((u32)(j) * mc_magic) >> 16))
#define JPRED(j) (jobb + (j) * L.job_bytes + L.j_pred)
#define JT(j) ((s16 *)(jobb + (j) * L.job_bytes + L.j_t))
#define JC(j) ((s16 *)(jobb + (j) * L.job_bytes + L.j_c))
#define JDQT(j) ((s16 *)(jobb + (j) * L.job_bytes + L.j_dqt))
#define JT2(j) ((s16 *)(jobb + (j) * L.job_bytes + L.j_t2))
#define CORG(g) (cub + (g) * L.cu_bytes + L.c_org)

    // ---- matrices: rows packed 4 bytes to a word.  The inverse passes use the even/odd
    // symmetry of the folded DCT2 (row k of an N-point matrix satisfies F[k][N-1-n] =
    // (-1)^k F[k][n], as the encoder's butterflies build it): for the first half of the outputs
    // n they keep column n with the even-k entries first and the odd-k entries after them
    // (Fw^T, Fh^T in even/odd order), and each sum over k splits into an even part E and an odd
    // part O with out[n] = E + O and out[N-1-n] = E - O.
    // The class's tables come as an image of this part of shared memory, built once per device.  A CTA
    // takes its tiles from the queue in class order, so consecutive tiles mostly share the class: the
    // tables of the previous tile are kept (the layout of a class is fixed within a launch).
    constexpr int cls = (LW - 2) * 5 + (LH - 2);
    if (P.n_qp > 0 && S.tables != cls) {
        const uint4 *img = reinterpret_cast<const uint4 *>(P.images + cls * LAT_IMAGE_BYTES);
        for (int i = tid; i < L.o_cu / 16; i += LAT_THREADS) reinterpret_cast<uint4 *>(sm)[i] = __ldg(img + i);
    }
    const u16 *s_scan = (const u16 *)(sm + L.o_scan);
    if (tid < Gv) S.cu[tid] = lat_perm(perm + cu0 + tid);
    for (int j = tid; j < J; j += LAT_THREADS) {
        const int g = JG(j), mi = m0 + (j - g * MCv);
        // (a record is stored at its mode: an entry above 32 would fall into other CUs' records)
        s_mode[j] = (u8)(P.modes ? min((int)P.modes[(size_t)lat_perm(perm + cu0 + g).id * P.n_modes + mi], LAT_NO_MODE) : mi);
        s_satd[j] = 0; s_flag[j] = 0; S.ssd0[j] = 0;
        S.nz[j] = 0; S.sum[j] = 0; S.hash[j] = 0; S.last[j] = -1; S.ssd[j] = 0;
    }
    LAT_STAGE(0);

    // ---- per CU: org block, neighbours (com_intra_get_nbr with every in-picture sample
    // reconstructed).  Each thread reads its CU's position itself: no wait between that and the samples.
    // four samples per thread (CU x positions are multiples of 4): one word load where the
    // picture and its pitch are word-aligned
    for (int i = tid; i < Gv * (N >> 2); i += LAT_THREADS) {
        const int g = i >> (lN - 2), p = (i & ((N >> 2) - 1)) << 2;
        const LatPerm cu = lat_perm(perm + cu0 + g);
        const pel *src = P.org + (long long)(cu.y + (p >> lw)) * P.i_org + cu.x + (p & (w - 1));
        u32 v;
        if (P.org_words) v = __ldg(reinterpret_cast<const u32 *>(src));
        else v = (u32)src[0] | (u32)src[1] << 8 | (u32)src[2] << 16 | (u32)src[3] << 24;
        *reinterpret_cast<u32 *>(cub + g * L.cu_bytes + L.c_org + (p >> lw) * L.ps + (p & (w - 1))) = v;
    }
    const int range = max(w, h) * 4 + 4;
    for (int i = tid; i < Gv * range; i += LAT_THREADS) {
        const int g = i / range, k = i - g * range;
        const LatPerm cu = lat_perm(perm + cu0 + g);
        const int x = cu.x, y = cu.y;
        const int avail = (y > 0 ? 1 : 0) | (x > 0 ? 2 : 0);
        const int up_cnt = (y > 0) ? min(w >> 2, max(0, (P.W - (x + w)) >> 2)) : 0;
        const int le_cnt = (x > 0) ? min(h >> 2, max(0, (P.H - (y + h)) >> 2)) : 0;
        pel *nbm = cub + g * L.cu_bytes + L.c_nb + 288;
        nbm[1 + k] = (avail & 1) ? P.rec[(long long)(y - 1) * P.i_rec + x + min(k, w + 4 * up_cnt - 1)] : (pel)128;
        nbm[-1 - k] = (avail & 2) ? P.rec[(long long)(y + min(k, h + 4 * le_cnt - 1)) * P.i_rec + x - 1] : (pel)128;
        if (k == 0) {
            pel c;
            if (x > 0 && y > 0) c = P.rec[(long long)(y - 1) * P.i_rec + x - 1];
            else if (y > 0) c = P.rec[(long long)(y - 1) * P.i_rec + x];
            else if (x > 0) c = P.rec[(long long)y * P.i_rec + x - 1];
            else c = 128;
            nbm[0] = c;
        }
    }
    __syncthreads(); LAT_STAGE(1);
    if (tid == 0 && P.n_qp > 0) S.tables = cls;   // every thread has read S.tables above
    if ((tid >> 5) < Gv) {
        // a warp per CU: the sums that the DC and plane modes take from the neighbours
        const int g = tid >> 5;
        const LatPerm cu = S.cu[g];
        const int avail = (cu.y > 0 ? 1 : 0) | (cu.x > 0 ? 2 : 0) | ((cu.x > 0 && cu.y > 0) ? 4 : 0);
        pel *nbm = cub + g * L.cu_bytes + L.c_nb + 288;
        int up = 0, left = 0, ch = 0, cv = 0;
#pragma unroll
        for (int k = lane; k < w; k += 32) {
            up += nbm[k + 1];
            if (k < w / 2) ch += (k + 1) * (nbm[w / 2 + k + 1] - nbm[w / 2 - k - 1]);
        }
#pragma unroll
        for (int k = lane; k < h; k += 32) {
            left += nbm[-k - 1];
            if (k < h / 2) cv += (k + 1) * (nbm[-h / 2 - k - 1] - nbm[-h / 2 + k + 1]);
        }
        up = __reduce_add_sync(0xFFFFFFFFu, up); left = __reduce_add_sync(0xFFFFFFFFu, left);
        ch = __reduce_add_sync(0xFFFFFFFFu, ch); cv = __reduce_add_sync(0xFFFFFFFFu, cv);
        if (lane == 0) {
            ipred_block_finish(nbm, w, h, avail, 8, up, left, ch, cv, sB[g]);
            nbm[LAT_DC] = (pel)sB[g].dc;
        }
    }
    // org part of the forward row pass: Torg[y][u] = sum_x Fw[u][x] org[y][x] (no transform
    // stage runs when no QP is asked: SATD records only)
    for (int i = tid; i < (P.n_qp > 0 ? Gv * kw * h : 0); i += LAT_THREADS) {
        const int u = i & (kw - 1), y = (i >> lkw) & (h - 1), g = i >> (lkw + lh);
        const u8 *c = cub + g * L.cu_bytes;
        const u32 *o = (const u32 *)(c + L.c_org + y * L.ps), *f = fw + u * L.fw_ws;
        int acc = 0;
        #pragma unroll
        for (int k = 0; k < (w >> 2); k++) acc = dp4a_us(o[k], f[k], acc);
        ((int *)(c + L.c_torg))[y * kw + u] = acc;
    }
    __syncthreads(); LAT_STAGE(2);

    // ---- prediction, four samples a task
    for (int i = tid; i < (J << (lN - 2)); i += LAT_THREADS) {
        const int j = i >> (lN - 2), p = i & ((N >> 2) - 1);
        const int m = s_mode[j];
        const int x = (p << 2) & (w - 1), y = p >> (lw - 2), g = JG(j);
        *reinterpret_cast<u32 *>(JPRED(j) + y * L.ps + x) =
            lat_pred4<W_, H_>(P.ipred + lat_table_at(LW, LH), cub + g * L.cu_bytes + L.c_nb + 288, sB[g], m, P.ipf, x, y);
    }
    __syncthreads(); LAT_STAGE(3);

    // ---- SATD (com_had tiling) and forward row pass T[u][y] = (Torg - sum_x Fw pred + rnd) >> sh1
    {
        constexpr int TW = lat_tw(1 << LW, 1 << LH), TH = lat_th(1 << LW, 1 << LH);
        constexpr int lnt = LW + LH - (TW == 16 ? 4 : TW == 8 ? 3 : 2) - (TH == 16 ? 4 : TH == 8 ? 3 : 2);
        if (P.n_qp > 0)
            lat_satd_tiles<TW, TH, true>(J << lnt, lnt, (1 << LW) / TW, cub, L.cu_bytes, L.c_org, jobb, L.job_bytes,
                                         L.j_pred, L.ps, mc_magic, s_satd, S.ssd0, P.sq32, P.sq128, P.k32, P.k128);
        else
            lat_satd_tiles<TW, TH, false>(J << lnt, lnt, (1 << LW) / TW, cub, L.cu_bytes, L.c_org, jobb, L.job_bytes,
                                          L.j_pred, L.ps, mc_magic, s_satd, S.ssd0, P.sq32, P.sq128, P.k32, P.k128);
    }
    {
        const int sh1 = lw - 2, rnd1 = sh1 > 0 ? 1 << (sh1 - 1) : 0;
        for (int i = tid; i < (P.n_qp > 0 ? J * NYC * KW_ : 0); i += LAT_THREADS) {
            const int u = i & (KW_ - 1), yc = (i >> LKW_) % NYC, j = i / (KW_ * NYC);
            const int *torg = (const int *)(cub + JG(j) * L.cu_bytes + L.c_torg) + yc * RY * KW_ + u;
            const u8 *pr = JPRED(j) + yc * RY * L.ps;
            constexpr int XW = W_ < 16 ? W_ / 4 : 4;     // words of a row at a time
            int acc[RY];
#pragma unroll
            for (int r = 0; r < RY; r++) acc[r] = 0;
#pragma unroll 1
            for (int x = 0; x < W_ / 4; x += XW) {
                u32 f[XW];
                lat_row<XW>(fw + u * L.fw_ws + x, f);
#pragma unroll
                for (int r = 0; r < RY; r++) {
                    u32 pw[XW];
                    lat_row<XW>(pr + r * L.ps + 4 * x, pw);
#pragma unroll
                    for (int k = 0; k < XW; k++) acc[r] = dp4a_us(pw[k], f[k], acc[r]);
                }
            }
            u32 tv[RY / 2];
#pragma unroll
            for (int r = 0; r < RY; r++) acc[r] = (torg[r * KW_] - acc[r] + rnd1) >> sh1;
#pragma unroll
            for (int r = 0; r < RY / 2; r++) tv[r] = __byte_perm((u32)acc[2 * r], (u32)acc[2 * r + 1], 0x5410);
            lat_store<RY / 2>(JT(j) + u * L.ts + yc * RY, tv);
        }
    }
    __syncthreads(); LAT_STAGE(4);

    // quantisation parameters per QP
    const int odd = lN & 1, log2_size = lN >> 1;
    const int q_bits = lat_q_bits(log2_size);
    const u32 qadd = 1u << (q_bits - 1);

    // ---- forward column pass C[v][u] = (sum_y Fh[v][y] T[u][y] + rnd2) >> sh2, and the
    // quant_check flags of every QP (bit q: some |C| above that QP's all-zero threshold)
    {
        const int sh2 = lh + 5, rnd2 = 1 << (sh2 - 1);
        for (int i = tid; i < (P.n_qp > 0 ? J * NUC * KH_ : 0); i += LAT_THREADS) {
            const int v = i & (KH_ - 1), uc = (i >> LKH_) % NUC, j = i / (KH_ * NUC);
            const s16 *T = JT(j) + uc * RU * L.ts;
            int acc[RU];
#pragma unroll
            for (int r = 0; r < RU; r++) acc[r] = rnd2;
            if constexpr (H_ == 4) {
                const u32 f = fh[v * L.fh_ws];
#pragma unroll
                for (int r = 0; r < RU; r++) {
                    const uint2 t = *reinterpret_cast<const uint2 *>(T + r * L.ts);
                    acc[r] = dp2a_hi(t.y, f, dp2a_lo(t.x, f, acc[r]));
                }
            } else {
#pragma unroll 1
                for (int y = 0; y < H_; y += 8) {
                    const uint2 fv = *reinterpret_cast<const uint2 *>(fh + v * L.fh_ws + y / 4);
                    const u32 f0 = fv.x, f1 = fv.y;
#pragma unroll
                    for (int r = 0; r < RU; r++) {
                        const uint4 t = *reinterpret_cast<const uint4 *>(T + r * L.ts + y);
                        acc[r] = dp2a_hi(t.y, f0, dp2a_lo(t.x, f0, acc[r]));
                        acc[r] = dp2a_hi(t.w, f1, dp2a_lo(t.z, f1, acc[r]));
                    }
                }
            }
            u32 cv[RU / 2];
            int amax = 0;
#pragma unroll
            for (int r = 0; r < RU; r++) {
                acc[r] = (int)(s16)(acc[r] >> sh2);
                amax = max(amax, abs(acc[r]));
            }
#pragma unroll
            for (int r = 0; r < RU / 2; r++) cv[r] = __byte_perm((u32)acc[2 * r], (u32)acc[2 * r + 1], 0x5410);
            lat_store<RU / 2>(JC(j) + v * L.cs + uc * RU, cv);
            u32 fl = 0;
#pragma unroll
            for (int q = 0; q < LAT_MAX_QP; q++)
                if (q < P.n_qp && amax > P.qp[lN - 4][q].thr) fl |= 1u << q;
            if (fl) atomicOr(&s_flag[j], fl);
        }
    }
    __syncthreads(); LAT_STAGE(5);
    for (int j = tid; j < J; j += LAT_THREADS)
        if (s_mode[j] != LAT_NO_MODE) P.satd_out[(size_t)S.cu[JG(j)].id * 33 + s_mode[j]] = s_satd[j];
    if (P.n_qp == 0) return;
    // the list of the jobs that each QP codes, a warp per QP: quant_check found a coefficient above its
    // threshold, whose level is then not zero; the others keep the prediction's SSD and empty statistics.
    // The first reader, the inverse column pass, comes behind the barrier of the first quantisation.
    // (Built at the start of each QP's turn, behind a barrier of its own, the lists made calls of few modes
    // slower than no lists at all: 104 us and 96 for one mode at four QPs of 256x256.)
    if ((tid >> 5) < P.n_qp) {
        const int q = tid >> 5;
        int n = 0;
        for (int base = 0; base < J; base += 32) {
            const int j = base + lane;
            const bool own = j < J && ((s_flag[j] >> q) & 1);
            const u32 m = __ballot_sync(0xFFFFFFFFu, own);
            if (own) S.list[q][n + __popc(m & ((1u << lane) - 1))] = (u8)j;
            n += __popc(m);
        }
        if (lane == 0) S.coded[q] = n;
    }
    // levels and magnitudes of a block of at most 256 coefficients go into one word, the count from bit 23
    constexpr bool PACK = KW_ * KH_ <= 256, CHUNKS = KW_ > 8 || KH_ > 8;
    for (int q = 0; q < P.n_qp; q++) {
        const int q_value = P.qp[lN - 4][q].q_value, dq_scale = P.qp[lN - 4][q].dq_scale, dq_shift = P.qp[lN - 4][q].dq_shift;
        // first-pass levels, statistics, dequantisation (stored transposed, DQ^T[u][v], each row
        // in even/odd order of v).  The
        // level (|c| q_value + 2^(q_bits-1)) >> q_bits is exact in 32 bits: |c| <= 2^15 and
        // q_value < 2^15; it is 0 below the level threshold and, with q_value 0, for a QP that codes
        // nothing of the job.  A task is RV coefficient rows (HV apart) of a job over RU columns, 8
        // coefficients, and lanes take consecutive v: the statistics are summed in registers and reduced
        // once per task.  (16 a task: 20.57 ms for a 1080p frame at four QPs where 8 take 20.86, but 96 us
        // for one mode at four QPs of 256x256 where 8 take 87: tiles of few jobs leave most threads idle.)
        // The level hash of a record is the sum of level x weight(p) mod 2^32 over raster positions
        // p = v w + u, weight(p) = (K p + 0x7F4A7C15) | 1 with K = 0x9E3779B1: odd and spread over 32 bits, so
        // the hash changes with any single level, any sign and any exchange of two different levels.  The
        // weight is linear in p but for its lowest bit, and w and the first column are even: weight = row
        // part + constant of the column.
        {
            constexpr int RV = 8 / RU, HV = KH_ / RV;
            constexpr int TPJ = HV * NUC, SEG = TPJ < 32 ? TPJ : 32;
            for (int base = wbase; base < J * TPJ; base += LAT_THREADS) {
                const int i = base + lane;
                const bool act = i < J * TPJ;
                const int ii = act ? i : base;
                const int v = ii % HV, uc = ii / HV % NUC, j = ii / TPJ;
                const u32 on = act ? (s_flag[j] >> q) & 1 : 0u;
                if (!__any_sync(0xFFFFFFFFu, on)) continue;
                const int qv = on ? q_value : 0;
                // level of c: (|c| qv + 2^(q_bits - 1)) >> q_bits with c's sign, which is
                // (c qv + 2^(q_bits - 1) - (c < 0)) >> q_bits; two to a word (|c| <= 2^15, qv < 2^15 and
                // q_bits >= 15, so 16 bits hold one)
                int lv[RV][RU];
                u32 lp[RV][RU / 2], mask[RV], any = 0;
#pragma unroll
                for (int k = 0; k < RV; k++) {
                    u32 cp[RU / 2];
                    lat_row<RU / 2>(JC(j) + (v + k * HV) * L.cs + uc * RU, cp);
                    mask[k] = 0;
#pragma unroll
                    for (int r = 0; r < RU; r++) {
                        const int c = r & 1 ? (int)cp[r >> 1] >> 16 : (int)(s16)(cp[r >> 1] & 0xFFFF);
                        lv[k][r] = (c * qv + ((int)qadd + (c >> 31))) >> q_bits;
                    }
#pragma unroll
                    for (int r = 0; r < RU / 2; r++) {
                        lp[k][r] = __byte_perm((u32)lv[k][2 * r], (u32)lv[k][2 * r + 1], 0x5410);
                        mask[k] += __vminu2(lp[k][r], 0x00010001u) << r;   // bit r: column 2r, bit 16 + r: column 2r + 1
                    }
                    any |= mask[k];
                }
                // rows and chunks of eight columns without a level are not stored: the inverse passes
                // do not read them (a chunk with a level is stored whole)
                if (!__any_sync(0xFFFFFFFFu, any != 0)) continue;
                u32 sa = 0, hs = 0, count = 0, rows[RV];
                int own_last = -1;
#pragma unroll
                for (int k = 0; k < RV; k++) {
                    const int vk = v + k * HV;
                    s16 *dqt = JDQT(j) + uc * RU * L.ds + lat_eo(vk, KH_);
#pragma unroll
                    for (int r = 0; r < RU; r += 2) {
                        sa += (u32)abs(lv[k][r]) + (u32)abs(lv[k][r + 1]);
                        const int d0 = (lv[k][r] * dq_scale + (1 << dq_shift >> 1)) >> dq_shift;
                        const int d1 = (lv[k][r + 1] * dq_scale + (1 << dq_shift >> 1)) >> dq_shift;
                        u32 d = lat_pack16(d0, d1);
                        if (odd) d = __byte_perm((u32)(((int)(s16)(d & 0xFFFF) * 181 + 128) >> 8), (u32)((((int)d >> 16) * 181 + 128) >> 8), 0x5410);
                        if (act) {
                            dqt[r * L.ds] = (s16)(d & 0xFFFF);
                            dqt[(r + 1) * L.ds] = (s16)(d >> 16);
                        }
                    }
                    // sum of level x weight, the weight of column r being wrow + K r + (r & 1): from the
                    // sums over the pairs p of s_p = lev[2p] + lev[2p+1], of p s_p, and of the odd columns
                    int at = 0, ks = 0, odds = 0;
#pragma unroll
                    for (int r = RU / 2 - 1; r >= 0; r--) {
                        at = dp2a_lo(lp[k][r], 0x0101u, at);
                        if (r > 0) ks += at;
                        odds = dp2a_lo(lp[k][r], 0x0100u, odds);
                    }
                    const u32 wrow = (u32)(vk * w + uc * RU) * 0x9E3779B1u + 0x7F4A7C15u;
                    hs += (u32)at * wrow + (u32)ks * (2u * 0x9E3779B1u) + (u32)odds * (0x9E3779B1u + 1u);
                    count += (u32)__popc(mask[k]);
                    // along a row the scan index grows with the column
                    const int he = 31 - __clz((int)(mask[k] & 0xFFFFu)), ho = 31 - __clz((int)(mask[k] >> 16));
                    if (mask[k]) own_last = max(own_last, (int)s_scan[vk * KW_ + uc * RU + max(2 * he, 2 * ho + 1)]);
                    rows[k] = CHUNKS ? __ballot_sync(0xFFFFFFFFu, mask[k] != 0) : 0;
                }
                // the count of levels rides above the sum of their magnitudes, which is below 2^23 for a
                // segment's at most 256 levels (those are below 23053)
                const u32 both = lat_seg_sum<SEG>(sa + (count << 23), lane);
                sa = both & 0x7FFFFFu; hs = lat_seg_sum<SEG>(hs, lane);
                const u32 nz = both >> 23;
                const int last = lat_seg_max<SEG>(own_last, lane);
                if (act && (lane & (SEG - 1)) == 0 && nz) {
                    atomicAdd(&S.sum[j], PACK ? both : sa);
                    atomicAdd(&S.hash[j], hs);
                    atomicMax(&S.last[j], last);
                    if (!PACK) atomicAdd(&S.nz[j], nz);
                    if (!CHUNKS) continue;
                    // which chunks of columns and of rows hold levels (bits 16.. and 20..)
                    constexpr u32 SEG_MASK = SEG == 32 ? 0xFFFFFFFFu : (1u << (SEG & 31)) - 1;
                    u32 ch = KH_ <= 8 ? 1u << 20 : 0u, cols = 0;
#pragma unroll
                    for (int k = 0; k < RV; k++) {
                        const u32 own = (rows[k] >> lane) & SEG_MASK;
                        cols |= own;
                        if (KH_ > 8 && HV < 8 && own) ch |= 1u << (20 + k * HV / 8);
                        if (KH_ > 8 && HV >= 8) {
#pragma unroll
                            for (int g = 0; g < SEG / 8; g++)
                                if ((own >> (8 * g)) & 0xFFu) ch |= 1u << (20 + k * (HV / 8) + g % (HV >= 8 ? HV / 8 : 1));
                        }
                    }
                    constexpr u32 HV_MASK = HV == 32 ? 0xFFFFFFFFu : (1u << (HV & 31)) - 1;
#pragma unroll
                    for (int g = 0; g < SEG / HV; g++)
                        if ((cols >> (g * HV)) & HV_MASK) ch |= 1u << (16 + (uc + g) % NUC);
                    atomicOr(&S.nz[j], ch);
                }
            }
        }
        __syncthreads(); LAT_STAGE(6);
        // the inverse passes run over the coded jobs only
        const int JC_ = S.coded[q];
        const u8 *list = S.list[q];
        // inverse column pass T2[y][u] = clip16((sum_v Fh[v][y] DQ[v][u] + 16) >> 5); a task forms
        // rows y and H-1-y from the even-v and odd-v sums over CU columns u.  Chunks of columns past the
        // last level's are left out, empty ones before it are zeros.  Tiles with few
        // jobs take CU/2 columns per task so that the CTA's threads still have a task each.
        auto inv_col = [&](auto cu_tag) {
            constexpr int CU = decltype(cu_tag)::value, NCU = KW_ / CU;
            for (int i = tid; i < JC_ * NCU * (H_ / 2); i += LAT_THREADS) {
                const int y = i & (H_ / 2 - 1), uc = (i >> (LH - 1)) % NCU, k = i / ((H_ / 2) * NCU);
                const int j = list[k];
                const u32 ch = S.nz[j] >> 16;
                const int col = uc * CU >> 3;
                if (KW_ > 8 && !((ch & 15) >> col)) continue;
                int e[CU], o[CU];
                const int nv = KW_ > 8 && !((ch >> col) & 1) ? 0 : KH_ > 8 ? 32 - __clz((int)((ch >> 4) & 15)) : 1;
                if (KH_ == 4 && nv == 0) {
#pragma unroll
                    for (int r = 0; r < CU; r++) e[r] = o[r] = 0;
                } else {
                    lat_eo_sums<KH_, CU>(JDQT(j) + uc * CU * L.ds, L.ds, fht + y * L.fht_ws, nv, e, o);
                }
                s16 *t2 = JT2(j);
#pragma unroll
                for (int half = 0; half < 2; half++) {
                    int t[CU];
#pragma unroll
                    for (int r = 0; r < CU; r++) t[r] = (half ? e[r] - o[r] + 16 : e[r] + o[r] + 16) >> 5;
                    s16 *row = t2 + (half ? H_ - 1 - y : y) * L.t2s;
                    if constexpr (CU == 8) {
                        const u32 v[4] = { lat_pack16(t[0], t[2]), lat_pack16(t[4], t[6]), lat_pack16(t[1], t[3]), lat_pack16(t[5], t[7]) };
                        lat_store<4>(row + uc * 8, v);
                    } else if constexpr (KW_ == 4) {
                        const u32 v[2] = { lat_pack16(t[0], t[2]), lat_pack16(t[1], t[3]) };
                        lat_store<2>(row, v);
                    } else {
                        u32 *p = reinterpret_cast<u32 *>(row + (uc >> 1) * 8) + (uc & 1);
                        p[0] = lat_pack16(t[0], t[2]); p[2] = lat_pack16(t[1], t[3]);
                    }
                }
            }
        };
        if (RU == 8 && JC_ * NUC * (H_ / 2) < LAT_THREADS) inv_col(std::integral_constant<int, 4>{});
        else inv_col(std::integral_constant<int, RU>{});
        __syncthreads(); LAT_STAGE(7);
        // inverse row pass, reconstruction, SSD: a task is the columns x, x+1, W-2-x, W-1-x over CY
        // rows (the even-u and odd-u sums of the T2 row give two of them); CY = 2 for tiles with
        // few jobs.  The clip of the residual to -256..255 is left out: the clip of the reconstruction
        // gives the same sample without it.
        auto inv_row = [&](auto cy_tag) {
            constexpr int CY = decltype(cy_tag)::value, NCY = H_ / CY;
            constexpr int TPJ = (W_ / 4) * NCY, SEG = TPJ < 32 ? TPJ : 32;
            for (int base = wbase; base < JC_ * TPJ; base += LAT_THREADS) {
                const int i = base + lane;
                const bool act = i < JC_ * TPJ;
                const int ii = act ? i : base;
                const int x = (ii & (W_ / 4 - 1)) * 2, yc = (ii >> (LW - 2)) % NCY, k = ii / TPJ;
                const int j = list[k];
                const s16 *t2 = JT2(j) + yc * CY * L.t2s;
                const u32 *f = fwt + x * L.fwt_ws;
                // e0, o0: column x (and W-1-x); e1, o1: column x+1 (and W-2-x)
                int e0[CY], o0[CY], e1[CY], o1[CY];
                if constexpr (KW_ == 4) {
                    const u32 f0 = f[0], f1 = f[L.fwt_ws];
#pragma unroll
                    for (int r = 0; r < CY; r++) {
                        const uint2 v = *reinterpret_cast<const uint2 *>(t2 + r * L.t2s);
                        e0[r] = dp2a_lo(v.x, f0, 2048); o0[r] = dp2a_hi(v.y, f0, 0);
                        e1[r] = dp2a_lo(v.x, f1, 2048); o1[r] = dp2a_hi(v.y, f1, 0);
                    }
                } else {
#pragma unroll
                    for (int r = 0; r < CY; r++) { e0[r] = e1[r] = 2048; o0[r] = o1[r] = 0; }
                    const int nu = KW_ > 8 ? 32 - __clz((int)((S.nz[j] >> 16) & 15)) : 1;
#pragma unroll 1
                    for (int c = 0; c < nu; c++, t2 += 8, f += 2) {
                        const uint2 f0 = *reinterpret_cast<const uint2 *>(f), f1 = *reinterpret_cast<const uint2 *>(f + L.fwt_ws);
#pragma unroll
                        for (int r = 0; r < CY; r++) {
                            const uint4 v = *reinterpret_cast<const uint4 *>(t2 + r * L.t2s);
                            e0[r] = dp2a_hi(v.y, f0.x, dp2a_lo(v.x, f0.x, e0[r]));
                            o0[r] = dp2a_hi(v.w, f0.y, dp2a_lo(v.z, f0.y, o0[r]));
                            e1[r] = dp2a_hi(v.y, f1.x, dp2a_lo(v.x, f1.x, e1[r]));
                            o1[r] = dp2a_hi(v.w, f1.y, dp2a_lo(v.z, f1.y, o1[r]));
                        }
                    }
                }
                const pel *po = CORG(JG(j)) + yc * CY * L.ps, *pp = JPRED(j) + yc * CY * L.ps;
                u32 e = 0;
#pragma unroll
                for (int r = 0; r < CY; r++) {
                    const auto pair = [](const pel *p) { return (u32)*reinterpret_cast<const u16 *>(p); };
                    const u32 pl = pair(pp + r * L.ps + x), pr = pair(pp + r * L.ps + W_ - 2 - x);
                    const u32 org = pair(po + r * L.ps + x) | pair(po + r * L.ps + W_ - 2 - x) << 16;
                    const u32 rec = pack_sat_u8((int)(pl & 0xFF) + ((e0[r] + o0[r]) >> 12), (int)(pl >> 8) + ((e1[r] + o1[r]) >> 12),
                                              (int)(pr & 0xFF) + ((e1[r] - o1[r]) >> 12), (int)(pr >> 8) + ((e0[r] - o0[r]) >> 12));
                    e = lat_sq4(org, rec, e);
                }
                if (!act) e = 0;
                e = lat_seg_sum<SEG>(e, lane);
                if (act && (lane & (SEG - 1)) == 0) atomicAdd(&S.ssd[j], e);
            }
        };
        if (JC_ * (W_ / 4) * (H_ / 4) < LAT_THREADS) inv_row(std::integral_constant<int, 2>{});
        else inv_row(std::integral_constant<int, 4>{});
        __syncthreads(); LAT_STAGE(8);
        for (int j = tid; j < J; j += LAT_THREADS) {
            LatQ o;
            o.ssd = (s_flag[j] >> q) & 1 ? S.ssd[j] : S.ssd0[j];
            o.coef_hash = S.hash[j];
            o.num_nz = (u16)(PACK ? S.sum[j] >> 23 : S.nz[j] & 0xFFFFu);
            o.last_nz = (s16)S.last[j];
            o.sum_abs = PACK ? S.sum[j] & 0x7FFFFFu : S.sum[j];
            if (s_mode[j] != LAT_NO_MODE) P.q_out[((size_t)S.cu[JG(j)].id * 33 + s_mode[j]) * P.n_qp + q] = o;
            if (q + 1 < P.n_qp) { S.nz[j] = 0; S.sum[j] = 0; S.hash[j] = 0; S.last[j] = -1; S.ssd[j] = 0; }
        }
        __syncthreads(); LAT_STAGE(9);
    }
#undef JG
#undef JPRED
#undef JT
#undef JC
#undef JDQT
#undef JT2
#undef CORG
}

// the size classes in launch order, largest CUs first (their tiles are the longest): rank r
// takes class (log2 w - 2) * 5 + (log2 h - 2) = lat_order(r)
__host__ __device__ constexpr int lat_order(int r) { return (4 - r / 5) * 5 + (4 - r % 5); }

}  // namespace uc
