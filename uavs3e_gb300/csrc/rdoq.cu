// RDOQ of transform blocks for lists of blocks: quant_non_zero with flat quantisation
// (src/quant.c:315-383) -> rdoq_quant_block (:196-313), each block with the bin-cost estimates
// the encoder derived from its entropy-coder state (rdoq_init_cu_est_bits, :139-156) -- the
// levels and the count of coded coefficients bit-exact with the reference's call.
//
// Two launches with a grouping between them; a short list takes one (RQ_SHORT_PER_SM).  k_rdoq_list, a
// warp per block: zeroes the coefficients past 32 columns / rows, runs quant_check, and lists in scan
// order the positions whose first-pass level (quant_rdoq) is not zero.  The decision pass is a chain
// (each coded level selects the contexts of the next), so k_rdoq_chain walks one block per lane over its
// listed positions, the blocks ordered by their position counts (blocksort.cuh): a run of z zero levels
// adds est_run[last_b_zero][0] + (z - 1) est_run[1][0] bits at once, as the reference's per-position
// loop accumulates them.  The listing is bound by memory latency (60 us for 60,000 blocks of the 23
// shapes, 39 M coefficients), the chains by the dependent instructions of the longest block (0.30 ms
// for 860 positions, about 190 instructions each).  One launch in which a warp listed its 32 blocks one
// after the other and then walked them, whatever their lengths, took 1.10 ms.
#include "blocksort.cuh"
#include "common.cuh"
#include "quant_tables.cuh"
#include "tables.h"
#include "uavs3e_cuda_internal.h"
#include "../../include/uavs3e_cuda.h"

#include <math.h>
#include <mutex>
#include <string.h>

namespace uc {

// blocks per SM below which a list takes one launch, a warp per block (k_rdoq_short), instead of listing,
// grouping and chains.  On 152 SMs, blocks of 1024 samples and more take the same time either way at
// 760 (258 us and 265; 217 and 265 at 512, 349 and 267 at 2,048), mixed shapes at 1,024 (259 and 265);
// one 4x4 block takes 12 us and 22.
constexpr int RQ_SHORT_PER_SM = 5;
constexpr int RQ_WARPS = 2;          // blocks per CTA of the listing: they differ in size, few wait for one another

struct RdoqReq {
    u32 coef_offset; u8 log2w, log2h, qp, is_intra, ch_type, slice_type; u16 est; u32 pad; s64 lambda;
};
struct RdoqEst {
    s32 ctp[2]; s32 cbf[3][2]; s32 run[24][2]; s32 lvl[24][2]; s32 lst[2][6][12][2];
};
static_assert(sizeof(RdoqReq) == sizeof(uavs3e_cuda_rdoq_req_t), "request layout");
static_assert(sizeof(RdoqEst) == sizeof(uavs3e_cuda_rdoq_est_t), "estimate layout");

struct RdoqParams {
    const RdoqReq *reqs;
    int n, n_est;
    const RdoqEst *ests;
    s16 *coefs;
    unsigned long long n_coefs;
    s32 *num_nz;
    u32 *scratch;             // per coefficient: the listed positions of each block
    const u16 *scan[7][7];
    const u16 *scanpos[7][7];
    s32 err_scale[80][6];     // tbl_rdoq_err_scale (rdoq_init_err_scale, src/quant.c:69-83), 8-bit
};

// rate of a level (>= 1) beside the run's, rdoq_one_coef (src/quant.c:158-194): l0 / l1 = the costs of
// the first and the further bins of the level symbol
__device__ __forceinline__ s32 rq_level_rate(u32 level, int2 l0, int2 l1)
{
    const s32 mid = l0.x + l1.x * (s32)(level - 2) + l1.y;
    const s32 far = l0.x + l1.x * 7 + (((31 - __clz((int)level - 8)) << 1) + 1) * 32768;
    return level == 1 ? l0.y : (level < 9 ? mid : far);
}

// block r's samples in shared memory while its positions are listed: rows below 32 (the coded part
// of a 64-sample side), raster order
constexpr int RQ_STAGE = 32 * 64;
constexpr int RQ_UNROLL = 4;         // 32-position windows whose shared loads are in flight together

// Listing, a warp per block: zeroes the coefficients past 32 columns / rows, runs quant_check and, for
// a block that is coded, lists in scan order the positions whose first-pass level (quant_rdoq) is
// not zero (a ballot and a prefix count per 32 positions) and clears the block (the chain writes its
// levels).  Returns the positions listed.  The block is read from memory once, by 16-byte vectors where it
// starts on a 16-byte boundary.
template <bool VEC>
__device__ __forceinline__ int rq_list_block(const RdoqParams &P, const RdoqReq &q, s16 *st, int lane)
{
    const int lw = q.log2w, lh = q.log2h, w = 1 << lw, h = 1 << lh;
    s16 *coef = P.coefs + q.coef_offset;
    const int max_num = w * h, max_used = 1 << (lw + min(5, lh));
    const int odd = (lw + lh) & 1, log2_size = (lw + lh) >> 1;
    const int q_bits = 14 + (15 - 8 - log2_size);
    const int q_value = odd ? ((int)kQScale[q.qp] * 181 + 64) >> 7 : (int)kQScale[q.qp];
    const int offset = (q.slice_type == 1 ? 201 : 153) << (q_bits - 9);
    const int nz_thr = ((((1 << q_bits) - offset) << 10) / q_value - 1) >> 10;
    // rows below 32 into shared memory (columns past 32 as zeros, in memory too); quant_check
    // (rdoq_quant_block) over these first max_used coefficients
    bool above = false;
    if (VEC) {
        const int nv = max_used / 8;                  // 2 .. 256
        for (int v0 = lane; v0 < nv; v0 += 32 * RQ_UNROLL) {
            uint4 x[RQ_UNROLL];
#pragma unroll
            for (int j = 0; j < RQ_UNROLL; j++) {
                const int v = v0 + 32 * j;
                // w = 64: the vectors of a row's right half are not coded
                x[j] = v < nv && !(w > 32 && ((8 * v) & 32)) ? reinterpret_cast<const uint4 *>(coef)[v] : make_uint4(0, 0, 0, 0);
            }
#pragma unroll
            for (int j = 0; j < RQ_UNROLL; j++) {
                const int v = v0 + 32 * j;
                if (v >= nv) break;
                if (w > 32 && ((8 * v) & 32)) reinterpret_cast<uint4 *>(coef)[v] = x[j];
                reinterpret_cast<uint4 *>(st)[v] = x[j];
                const u32 xs[4] = { x[j].x, x[j].y, x[j].z, x[j].w };
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const int c0 = (int)(s16)xs[k], c1 = (int)xs[k] >> 16;
                    above |= c0 > nz_thr || c0 < -nz_thr || c1 > nz_thr || c1 < -nz_thr;
                }
            }
        }
        for (int v = max_used / 8 + lane; v < max_num / 8; v += 32)    // rows past 32
            reinterpret_cast<uint4 *>(coef)[v] = make_uint4(0, 0, 0, 0);
    } else {
        for (int p = lane; p < max_used; p += 32) {
            int c = coef[p];
            if ((p & (w - 1)) >= 32) coef[p] = (s16)(c = 0);
            st[p] = (s16)c;
            above |= c > nz_thr || c < -nz_thr;
        }
        for (int p = max_used + lane; p < max_num; p += 32) coef[p] = 0;
    }
    if (!__any_sync(0xffffffffu, above)) return 0;
    __syncwarp();
    // scan order; the positions whose first-pass level (quant_rdoq) is not zero -- exactly those
    // with |c| >= thr -- are listed in order as (position << 16 | coefficient).  The zig-zag visits
    // the anti-diagonals one after the other, so everything past the last kept coefficient's position
    // lies outside the kept 32 columns / rows.
    const u16 *scan = P.scan[lw][lh];
    const int n_scan = (int)P.scanpos[lw][lh][(min(h, 32) - 1) * w + min(w, 32) - 1] + 1;
    const int thr = ((1 << (q_bits - 1)) - 1) / q_value + 1;
    u32 *list = P.scratch + q.coef_offset;
    int cnt = 0;
    for (int base = 0; base < n_scan; base += 32 * RQ_UNROLL) {
        int c[RQ_UNROLL];
#pragma unroll
        for (int j = 0; j < RQ_UNROLL; j++) {
            const int i = base + 32 * j + lane, p = i < n_scan ? scan[i] : RQ_STAGE;
            c[j] = p < max_used ? st[p] : 0;
        }
#pragma unroll
        for (int j = 0; j < RQ_UNROLL; j++) {
            const bool mark = abs(c[j]) >= thr;
            const u32 m = __ballot_sync(0xffffffffu, mark);
            if (mark) list[cnt + __popc(m & ((1u << lane) - 1))] = ((u32)(base + 32 * j + lane) << 16) | (u16)(s16)c[j];
            cnt += __popc(m);
        }
    }
    if (VEC)
        for (int v = lane; v < max_used / 8; v += 32) reinterpret_cast<uint4 *>(coef)[v] = make_uint4(0, 0, 0, 0);
    else
        for (int p = lane; p < max_used; p += 32) coef[p] = 0;
    return cnt;
}

// the positions listed of a block, -1 for one outside the supported domain (left untouched)
__device__ __forceinline__ int rq_list(const RdoqParams &P, const RdoqReq &q, s16 *st, int lane)
{
    const int lw = q.log2w, lh = q.log2h;
    if (lw < 2 || lw > 6 || lh < 2 || lh > 6 || q.qp > 79 || q.ch_type > 2 || q.est >= P.n_est ||
        (unsigned long long)q.coef_offset + (1ull << (lw + lh)) > P.n_coefs)
        return -1;
    return (((uintptr_t)(P.coefs + q.coef_offset)) & 15) == 0 ? rq_list_block<true>(P, q, st, lane)
                                                              : rq_list_block<false>(P, q, st, lane);
}

// the listing of a grouped list: each block is counted into the grouping by its positions
__global__ void __launch_bounds__(32 * RQ_WARPS) k_rdoq_list(const RdoqParams P, BlockOrder O)
{
    __shared__ __align__(16) s16 s_stage[RQ_WARPS][RQ_STAGE];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r = blockIdx.x * RQ_WARPS + warp;
    if (r >= P.n) return;
    const RdoqReq q = P.reqs[r];
    const int cnt = rq_list(P, q, s_stage[warp], lane);
    if (lane == 0) { P.num_nz[r] = cnt; O.key[r] = bs_count(O.counts, (u32)max(cnt, 0)); }
}

// N pairs of estimates: 8 or 16 bytes at once where the estimate sets start on 16 bytes (a set is a
// multiple of 16 bytes long, a class's two run or level pairs start on 16)
template <int N, bool VEC>
__device__ __forceinline__ void rq_pairs(const s32 (*p)[2], int2 (&v)[N])
{
    if constexpr (VEC && N == 2) {
        const int4 x = *reinterpret_cast<const int4 *>(p);
        v[0] = make_int2(x.x, x.y);
        v[1] = make_int2(x.z, x.w);
    } else if constexpr (VEC) {
        v[0] = *reinterpret_cast<const int2 *>(p);
    } else {
#pragma unroll
        for (int k = 0; k < N; k++) v[k] = make_int2(p[k][0], p[k][1]);
    }
}

// the decision chain of a block, by one lane, over its cnt > 0 listed positions; returns num_nz
template <bool VEC>
__device__ __forceinline__ int rq_chain(const RdoqParams &P, const RdoqReq &q, int cnt)
{
    const int lw = q.log2w, lh = q.log2h, ch = q.ch_type, max_num = 1 << (lw + lh);
    const int odd = (lw + lh) & 1, log2_size = (lw + lh) >> 1;
    const int q_bits = 14 + (15 - 8 - log2_size);
    const int q_value = odd ? ((int)kQScale[q.qp] * 181 + 64) >> 7 : (int)kQScale[q.qp];
    s16 *coef = P.coefs + q.coef_offset;
    const u16 *scan = P.scan[lw][lh];
    const u32 *list = P.scratch + q.coef_offset;
    const RdoqEst &E = P.ests[q.est];
    const s32 err_scale = P.err_scale[q.qp][log2_size - 1];
    const s64 lambda = q.lambda;
    const u32 add = 1u << (q_bits - 1);
    s64 best_delta, curr_delta;
    if (!q.is_intra && ch == 0) { best_delta = (s64)E.ctp[1] * lambda; curr_delta = (s64)E.ctp[0] * lambda; }
    else { best_delta = (s64)E.cbf[ch][0] * lambda; curr_delta = (s64)E.cbf[ch][1] * lambda; }
    const int base = ch == 0 ? 0 : 12;
    const s32 (*lst)[2] = E.lst[ch != 0][5];
    const s32 (*est_run)[2] = E.run + 10 + base, (*est_lvl)[2] = E.lvl + 10 + base;
    u32 last_b_zero = 0;
    int k_end = -1, k_last = -1, tmp_nz = 0, num_nz = 0, prev = -1;
    // the list two entries ahead and the next entry's raster position one ahead: neither waits
    u32 next = list[0], next2 = list[min(1, cnt - 1)];
    int p_next = scan[next >> 16];
    for (int k = 0; k < cnt; k++) {
        const u32 ent = next;
        const int p = p_next;
        next = next2;
        p_next = scan[next >> 16];
        next2 = list[min(k + 2, cnt - 1)];
        const int i = (int)(ent >> 16), c = (s16)(ent & 0xffffu);
        // every estimate the position may need, loaded at once: which ones follow from the previous
        // level only
        const int lg = 31 - __clz(i + 1);
        int2 rv[2], lv[2], ev[1];
        rq_pairs<2, VEC>(est_run, rv);
        rq_pairs<2, VEC>(est_lvl, lv);
        rq_pairs<1, VEC>(lst + lg, ev);
        const int2 r0 = rv[0], r1 = rv[1], l0 = lv[0], l1 = lv[1], end = ev[0];
        // distortions: the scaled magnitude of the coefficient and of its difference from the two
        // levels tried stays below 2^31 for every block size and QP (2^30 at |c| = 2^15: the scale
        // undoes the quantiser's), so the squares are 32 x 32-bit products
        const u32 ld = (u32)abs(c) * (u32)q_value;
        const s32 e = (s32)(((s64)ld * err_scale) >> 20);
        const s64 zerr = (s64)e * e;
        const u32 lev_a = (ld + add) >> q_bits;            // >= 1: a listed position
        const s32 d_a = (s32)(ld - (lev_a << q_bits)), d_b = d_a + (s32)(1u << q_bits);
        const s32 e_a = (s32)(((s64)d_a * err_scale) >> 20), e_b = (s32)(((s64)d_b * err_scale) >> 20);
        const int z = i - prev - 1;                        // zero levels since the previous listed position
        prev = i;
        if (z > 0) {
            curr_delta += (s64)((last_b_zero ? r1.x : r0.x) + (z - 1) * r1.x) * lambda;
            last_b_zero = 1;
        }
        // rdoq_one_coef: no level, then the rounded level, then the one below it (if not 0), each kept
        // when it costs strictly less
        const int2 run = last_b_zero ? r1 : r0;
        const s32 rate0 = 32768 + (i == max_num - 1 ? 0 : run.y);
        s64 cc = zerr + (s64)run.x * lambda;
        const s64 c_a = (s64)e_a * e_a + (s64)(rate0 + rq_level_rate(lev_a, l0, l1)) * lambda;
        const s64 c_b = (s64)e_b * e_b + (s64)(rate0 + rq_level_rate(lev_a - 1, l0, l1)) * lambda;
        u32 level = 0;
        if (c_a < cc) { cc = c_a; level = lev_a; }
        if (lev_a > 1 && c_b < cc) { cc = c_b; level = lev_a - 1; }
        curr_delta += cc - zerr;
        last_b_zero = 1;
        if (level) {
            const s64 end_cost = curr_delta + (s64)end.y * lambda;
            curr_delta += (s64)end.x * lambda;
            k_last = k;
            coef[p] = (s16)(c < 0 ? -(int)level : (int)level);
            tmp_nz++;
            if (end_cost < best_delta) { best_delta = end_cost; k_end = k; num_nz += tmp_nz; tmp_nz = 0; }
            last_b_zero = 0;
            const int cls = min((int)level - 1, 5);
            est_lvl = E.lvl + (cls << 1) + base;
            est_run = E.run + (cls << 1) + base;
            lst = E.lst[ch != 0][cls];
        }
    }
    if (num_nz)
        for (int k = k_end + 1; k <= k_last; k++)  // levels after the chosen last position, back to zero
            coef[scan[list[k] >> 16]] = 0;
    return num_nz;
}

// Decision chains, a block per lane, 32 blocks with about as many listed positions per warp in the
// order of the grouping.  num_nz[r] holds the positions listed (0 or -1: the block is done).
template <bool VEC>
__global__ void __launch_bounds__(32) k_rdoq_chain(const RdoqParams P, const int *perm)
{
    const int at = blockIdx.x * 32 + threadIdx.x;
    if (at >= P.n) return;
    const int r = perm[at];
    const int cnt = P.num_nz[r];
    if (cnt <= 0) return;
    const RdoqReq q = P.reqs[r];
    P.num_nz[r] = rq_chain<VEC>(P, q, cnt);
}

// A short list, in one launch: a warp lists a block and its first lane walks the chain.
template <bool VEC>
__global__ void __launch_bounds__(32 * RQ_WARPS) k_rdoq_short(const RdoqParams P)
{
    __shared__ __align__(16) s16 s_stage[RQ_WARPS][RQ_STAGE];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r = blockIdx.x * RQ_WARPS + warp;
    if (r >= P.n) return;
    const RdoqReq q = P.reqs[r];
    const int cnt = rq_list(P, q, s_stage[warp], lane);
    __syncwarp();                                      // the list and the cleared block
    if (lane == 0) P.num_nz[r] = cnt > 0 ? rq_chain<VEC>(P, q, cnt) : cnt;
}

// rdoq_init_err_scale (src/quant.c:69-83) for 8-bit: 2^(15 - tr_shift) / q_value in 20-bit fixed
// point, computed once
struct RqErrScale {
    s32 v[80][6];
    RqErrScale()
    {
        static const u16 qs[80] = {
            16302, 15024, 13777, 12634, 11626, 10624, 9742, 8958, 8192, 7512, 6889, 6305, 5793, 5303, 4878, 4467,
            4091, 3756, 3444, 3161, 2894, 2654, 2435, 2235, 2048, 1878, 1722, 1579, 1449, 1329, 1218, 1117,
            1024, 939, 861, 790, 724, 664, 609, 558, 512, 470, 430, 395, 362, 332, 304, 279,
            256, 235, 215, 197, 181, 166, 152, 140, 128, 116, 108, 99, 91, 83, 76, 69,
            64, 59, 54, 49, 45, 41, 38, 35, 32, 30, 27, 25, 23, 21, 19, 18,
        };
        for (int qp = 0; qp < 80; qp++)
            for (int i = 0; i < 6; i++) {
                const int tr_shift = 15 - 8 - (i + 1);
                double es = pow(2.0, 15 - tr_shift);
                es = es / qs[qp] / 1;
                v[qp][i] = (s32)(es * (double)(1 << 20));
            }
    }
};

int launch_rdoq(const void *reqs, int n, const void *ests, int n_est, s16 *coefs, unsigned long long n_coefs,
                s32 *num_nz, cudaStream_t st)
{
    if (!reqs || !ests || !coefs || !num_nz || n < 0 || n_est < 1) return set_status(UC_ERR_ARG, "rdoq: null argument");
    if (n == 0) return UC_OK;
    int dev = 0;
    UC_CHECK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return set_status(UC_ERR_UNSUPPORTED, "rdoq: device index");
    const DevTables *tab = device_tables(dev);
    if (!tab) return set_status(UC_ERR_MEMORY, "rdoq: table upload failed");
    RdoqParams P;
    memset(&P, 0, sizeof(P));
    P.reqs = (const RdoqReq *)reqs; P.n = n; P.ests = (const RdoqEst *)ests; P.n_est = n_est;
    P.coefs = coefs; P.n_coefs = n_coefs; P.num_nz = num_nz;
    for (int a = 0; a < 7; a++)
        for (int b = 0; b < 7; b++) { P.scan[a][b] = tab->scan[a][b]; P.scanpos[a][b] = tab->scanpos[a][b]; }
    static const RqErrScale kErr;
    memcpy(P.err_scale, kErr.v, sizeof(P.err_scale));
    int sms = 0;
    UC_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const bool brief = n < RQ_SHORT_PER_SM * sms, vec = ((uintptr_t)ests & 15) == 0;
    // one word per coefficient (the position lists, at the coefficients' offsets) and the grouping's
    // arrays
    const size_t b_list = ((size_t)n_coefs * sizeof(u32) + 255) & ~(size_t)255;
    char *ws = nullptr;
    int rc = work_alloc((void **)&ws, b_list + (brief ? 256 : bs_bytes((size_t)n)), st);
    if (rc) return rc;
    P.scratch = (u32 *)ws;
    prof_begin(PROF_RDOQ, st);
    cudaError_t e = cudaSuccess;
    if (brief) {
        const unsigned ctas = (unsigned)((n + RQ_WARPS - 1) / RQ_WARPS);
        if (vec) k_rdoq_short<true><<<ctas, 32 * RQ_WARPS, 0, st>>>(P);
        else k_rdoq_short<false><<<ctas, 32 * RQ_WARPS, 0, st>>>(P);
        e = cudaGetLastError();
    } else if ((e = cudaMemsetAsync(bs_place(ws + b_list, (size_t)n).counts, 0, BS_CLEAR, st)) == cudaSuccess) {
        const BlockOrder O = bs_place(ws + b_list, (size_t)n);
        k_rdoq_list<<<(unsigned)((n + RQ_WARPS - 1) / RQ_WARPS), 32 * RQ_WARPS, 0, st>>>(P, O);
        k_bs_scatter<<<(unsigned)((n + BS_BUCKETS - 1) / BS_BUCKETS), BS_BUCKETS, 0, st>>>(O.key, O.counts, n, O.perm);
        if (vec) k_rdoq_chain<true><<<(unsigned)((n + 31) / 32), 32, 0, st>>>(P, O.perm);
        else k_rdoq_chain<false><<<(unsigned)((n + 31) / 32), 32, 0, st>>>(P, O.perm);
        e = cudaGetLastError();
    }
    rc = work_free(ws, st);
    UC_CHECK(e);
    if (rc) return rc;
    count_launch(brief ? 1 : 3);
    prof_end(PROF_RDOQ, st);
    return UC_OK;
}

}  // namespace uc

using namespace uc;

// per device: buffers of the host-memory entry point
// quant_non_zero's weighted branch (pic_wq_enable, src/quant.c:335-380) for lists of blocks: the
// zero-out past 32 columns / rows, then every level (s16)((|c| scale ns_scale 64 / weight + offset)
// >> shift) in 64-bit arithmetic with the weight of the sample's cell of the 4x4 (4x4 blocks) or
// 8x8 matrix (one cell per 2^(max(log2 w, log2 h) - 3) samples each way).  A warp per block.
__global__ void __launch_bounds__(128) k_quant_wq(const RdoqReq *reqs, int n, const u8 *wq4, const u8 *wq8,
                                                  s16 *coefs, unsigned long long n_coefs, s32 *num_nz)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r = blockIdx.x * 4 + warp;
    if (r >= n) return;
    const RdoqReq q = reqs[r];
    const int lw = q.log2w, lh = q.log2h, w = 1 << lw, h = 1 << lh;
    if (lw < 2 || lw > 6 || lh < 2 || lh > 6 || q.qp > 79 || q.ch_type > 2 ||
        (unsigned long long)q.coef_offset + (unsigned long long)(w * h) > n_coefs) {
        if (lane == 0) num_nz[r] = -1;       // outside the supported domain: block untouched
        return;
    }
    s16 *coef = coefs + q.coef_offset;
    const int log2_size = (lw + lh) >> 1, odd = (lw + lh) & 1;
    const int ns_shift = odd ? 7 : 0, ns_scale = odd ? 181 : 1;
    const int shift = 14 + 15 - 8 - (log2_size - ns_shift);
    const long long offset = (long long)(q.slice_type == 1 ? 171 : 85) << (shift - 9);
    const long long scale = (long long)kQScale[q.qp] * ns_scale * 64;
    const bool small = lw == 2 && lh == 2;
    const u8 *wq = small ? wq4 : wq8;
    const int idx_shift = small ? 0 : max(lw, lh) - 3, width = small ? 4 : 8;
    int nz = 0;
    for (int p = lane; p < w * h; p += 32) {
        const int i = p >> lw, j = p & (w - 1);
        const int c = (i >= 32 || j >= 32) ? 0 : coef[p];
        const int weight = wq[(i >> idx_shift) * width + (j >> idx_shift)];
        const int lev = (s16)(u16)(unsigned long long)((((long long)abs(c) * scale) / weight + offset) >> shift);
        const s16 v = (s16)(c < 0 ? -lev : lev);
        coef[p] = v;
        nz += v != 0;
    }
#pragma unroll
    for (int m = 16; m; m >>= 1) nz += __shfl_xor_sync(0xffffffffu, nz, m);
    if (lane == 0) num_nz[r] = nz;
}

int launch_quant_wq(const void *reqs, int n, const u8 *wq4, const u8 *wq8, s16 *coefs, unsigned long long n_coefs,
                    s32 *num_nz, cudaStream_t st)
{
    if (n < 0 || (n > 0 && (!reqs || !wq4 || !wq8 || !coefs || !num_nz)))
        return set_status(UC_ERR_ARG, "quant_wq: null argument");
    if (n == 0) return UC_OK;
    prof_begin(PROF_RDOQ, st);
    k_quant_wq<<<(unsigned)((n + 3) / 4), 128, 0, st>>>((const RdoqReq *)reqs, n, wq4, wq8, coefs, n_coefs, num_nz);
    UC_CHECK(cudaGetLastError());
    count_launch(1);
    prof_end(PROF_RDOQ, st);
    return UC_OK;
}

struct RdoqScratch {
    std::mutex mu;
    cudaStream_t st = nullptr;
    void *buf = nullptr;
    size_t cap = 0;
};
static RdoqScratch g_rdoq[64];

extern "C" UAVS3E_CUDA_API int uavs3e_cuda_rdoq(const uavs3e_cuda_rdoq_req_t *reqs, int n,
                                                const uavs3e_cuda_rdoq_est_t *ests, int n_est, int16_t *coefs,
                                                size_t n_coefs, int32_t *num_nz)
{
    int rc = ensure_init();
    if (rc) return rc;
    if (n < 0 || n_est < 1 || (n > 0 && (!reqs || !ests || !coefs || !num_nz)))
        return set_status(UC_ERR_ARG, "rdoq: bad argument");
    if (n == 0) return UC_OK;
    int dev = 0;
    UC_CHECK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return set_status(UC_ERR_UNSUPPORTED, "rdoq: device index");
    RdoqScratch &S = g_rdoq[dev];
    std::lock_guard<std::mutex> lk(S.mu);
    if (!S.st) UC_CHECK(cudaStreamCreateWithFlags(&S.st, cudaStreamNonBlocking));
    auto up = [](size_t b) { return (b + 255) & ~(size_t)255; };
    const size_t b_req = up((size_t)n * sizeof(*reqs)), b_est = up((size_t)n_est * sizeof(*ests));
    const size_t b_coef = up(n_coefs * sizeof(int16_t)), b_nz = up((size_t)n * sizeof(int32_t));
    const size_t need = b_req + b_est + b_coef + b_nz;
    if (S.cap < need) {
        if (S.buf) UC_CHECK(cudaFree(S.buf));
        S.buf = nullptr;
        S.cap = 0;
        UC_CHECK(cudaMalloc(&S.buf, need));
        S.cap = need;
    }
    char *b = (char *)S.buf;
    void *d_req = b, *d_est = b + b_req;
    int16_t *d_coef = (int16_t *)(b + b_req + b_est);
    int32_t *d_nz = (int32_t *)(b + b_req + b_est + b_coef);
    UC_CHECK(cudaMemcpyAsync(d_req, reqs, (size_t)n * sizeof(*reqs), cudaMemcpyHostToDevice, S.st));
    UC_CHECK(cudaMemcpyAsync(d_est, ests, (size_t)n_est * sizeof(*ests), cudaMemcpyHostToDevice, S.st));
    UC_CHECK(cudaMemcpyAsync(d_coef, coefs, n_coefs * sizeof(int16_t), cudaMemcpyHostToDevice, S.st));
    rc = launch_rdoq(d_req, n, d_est, n_est, d_coef, (unsigned long long)n_coefs, d_nz, S.st);
    if (rc) return rc;
    UC_CHECK(cudaMemcpyAsync(coefs, d_coef, n_coefs * sizeof(int16_t), cudaMemcpyDeviceToHost, S.st));
    UC_CHECK(cudaMemcpyAsync(num_nz, d_nz, (size_t)n * sizeof(int32_t), cudaMemcpyDeviceToHost, S.st));
    UC_CHECK(cudaStreamSynchronize(S.st));
    return UC_OK;
}

extern "C" UAVS3E_CUDA_API int uavs3e_cuda_rdoq_device(const uavs3e_cuda_rdoq_req_t *d_reqs, int n,
                                                       const uavs3e_cuda_rdoq_est_t *d_ests, int n_est,
                                                       int16_t *d_coefs, size_t n_coefs, int32_t *d_num_nz,
                                                       void *stream)
{
    int rc = ensure_init();
    if (rc) return rc;
    return launch_rdoq(d_reqs, n, d_ests, n_est, d_coefs, (unsigned long long)n_coefs, d_num_nz, (cudaStream_t)stream);
}

extern "C" UAVS3E_CUDA_API int uavs3e_cuda_quant_wq(const uavs3e_cuda_rdoq_req_t *reqs, int n, const uint8_t *wq4,
                                                   const uint8_t *wq8, int16_t *coefs, size_t n_coefs,
                                                   int32_t *num_nz)
{
    int rc = ensure_init();
    if (rc) return rc;
    if (n < 0 || (n > 0 && (!reqs || !wq4 || !wq8 || !coefs || !num_nz)))
        return set_status(UC_ERR_ARG, "quant_wq: bad argument");
    if (n == 0) return UC_OK;
    int dev = 0;
    UC_CHECK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return set_status(UC_ERR_UNSUPPORTED, "quant_wq: device index");
    RdoqScratch &S = g_rdoq[dev];
    std::lock_guard<std::mutex> lk(S.mu);
    if (!S.st) UC_CHECK(cudaStreamCreateWithFlags(&S.st, cudaStreamNonBlocking));
    auto up = [](size_t b) { return (b + 255) & ~(size_t)255; };
    const size_t b_req = up((size_t)n * sizeof(*reqs)), b_wq = 256;
    const size_t b_coef = up(n_coefs * sizeof(int16_t)), b_nz = up((size_t)n * sizeof(int32_t));
    const size_t need = b_req + b_wq + b_coef + b_nz;
    if (S.cap < need) {
        if (S.buf) UC_CHECK(cudaFree(S.buf));
        S.buf = nullptr;
        S.cap = 0;
        UC_CHECK(cudaMalloc(&S.buf, need));
        S.cap = need;
    }
    char *b = (char *)S.buf;
    void *d_req = b;
    u8 *d_wq = (u8 *)(b + b_req);
    int16_t *d_coef = (int16_t *)(b + b_req + b_wq);
    int32_t *d_nz = (int32_t *)(b + b_req + b_wq + b_coef);
    UC_CHECK(cudaMemcpyAsync(d_req, reqs, (size_t)n * sizeof(*reqs), cudaMemcpyHostToDevice, S.st));
    UC_CHECK(cudaMemcpyAsync(d_wq, wq4, 16, cudaMemcpyHostToDevice, S.st));
    UC_CHECK(cudaMemcpyAsync(d_wq + 16, wq8, 64, cudaMemcpyHostToDevice, S.st));
    UC_CHECK(cudaMemcpyAsync(d_coef, coefs, n_coefs * sizeof(int16_t), cudaMemcpyHostToDevice, S.st));
    rc = launch_quant_wq(d_req, n, d_wq, d_wq + 16, d_coef, (unsigned long long)n_coefs, d_nz, S.st);
    if (rc) return rc;
    UC_CHECK(cudaMemcpyAsync(coefs, d_coef, n_coefs * sizeof(int16_t), cudaMemcpyDeviceToHost, S.st));
    UC_CHECK(cudaMemcpyAsync(num_nz, d_nz, (size_t)n * sizeof(int32_t), cudaMemcpyDeviceToHost, S.st));
    UC_CHECK(cudaStreamSynchronize(S.st));
    return UC_OK;
}

extern "C" UAVS3E_CUDA_API int uavs3e_cuda_quant_wq_device(const uavs3e_cuda_rdoq_req_t *d_reqs, int n,
                                                          const uint8_t *d_wq4, const uint8_t *d_wq8,
                                                          int16_t *d_coefs, size_t n_coefs, int32_t *d_num_nz,
                                                          void *stream)
{
    int rc = ensure_init();
    if (rc) return rc;
    return launch_quant_wq(d_reqs, n, d_wq4, d_wq8, d_coefs, (unsigned long long)n_coefs, d_num_nz,
                           (cudaStream_t)stream);
}
