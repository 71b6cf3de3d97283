// Coefficient rate for lists of transform blocks: lbac_enc_run_length_cc_rdo (src/entropy.c:1688-
// 1950), the counting-mode coder the encoder's RDO runs on each candidate's levels -- per non-zero
// level in zig-zag order its run of zeros (truncated unary, cap 16, exp-Golomb escape), level - 1
// (cap 8, escape), sign and last flag (the averaged last1 / last2 pair), every bin on the context
// model it selects, the models updated as they go -- from the coder state the caller passes
// (range and the channel's run, run_rdoq, level, last1, last2 models).  Results: the bits
// counted, the range and the models after the block, bit-exact with the reference.
//
// Two launches with a grouping between them; a short list takes one (CR_SHORT_PER_SM).  A warp per block
// lists its levels in scan order (k_cr_list), the blocks are ordered by the bins they will code
// (blocksort.cuh), and a lane per block codes its chain (k_cr_code).  The chains bound the call: one lane's
// bins follow one another.  60,000 blocks of the 23 shapes (5.6 M levels, 31 M bins, up to 5,300 bins a
// block) take 67 us to list and 0.55 ms to code; one launch in which a warp listed 32 blocks in turn and
// then coded them side by side, symbol after symbol, took 2.37 ms with 4 of 32 lanes active on average.
// The model update is the rule the reference tabulates in tbl_plps / tbl_plps_ext (src/entropy.c:41),
// computed.
#include "blocksort.cuh"
#include "common.cuh"
#include "tables.h"
#include "uavs3e_cuda_internal.h"
#include "../../include/uavs3e_cuda.h"

#include <algorithm>
#include <mutex>
#include <string.h>

namespace uc {

struct CoefCtx { s16 run[12], run_rdoq[12], level[12], last1[6], last2[12]; };
struct CrReq { u32 coef_offset; u8 log2w, log2h, ch_type, pad; u16 num_sig, range; CoefCtx ctx; };
struct CrOut { u32 bits; u16 range, pad; CoefCtx ctx; };
static_assert(sizeof(CrReq) == sizeof(uavs3e_cuda_coef_rate_req_t), "coef rate request layout");
static_assert(sizeof(CrOut) == sizeof(uavs3e_cuda_coef_rate_out_t), "coef rate result layout");

struct CrParams {
    const CrReq *reqs;
    int n;
    const s16 *levels;
    unsigned long long n_levels;
    CrOut *out;
    u32 *fixed;                          // per block: bits that do not depend on the coder state, or CR_BAD
    const u16 *scan[7][7];
};

// the model after one bin: window state (bits 11-12: windows 3, 3, 4, 5), LPS probability (bits
// 1-10), MPS (bit 0); an MPS shrinks the probability by p >> w + p >> (w + 2), an LPS grows it by
// 197 / 95 / 46 (reflected about 1023 with the MPS flipped) and steps the state up.  Both outcomes
// are formed and selected: the chain waits on the select, not on a branch.
__device__ __forceinline__ u32 cr_next(u32 model, bool mps)
{
    const u32 c = (model >> 11) & 3, w = max(c + 2, 3u), p = (model >> 1) & 1023;
    const u32 pm = p - (p >> w) - (p >> (w + 2));
    const u32 m_next = (max(c, 1u) << 11) | (pm << 1) | (model & 1);
    const u32 pl = p + __byte_perm(0x2E5FC5C5u, 0u, 0x4440 + c);     // 197, 197, 95, 46
    const bool flip = pl > 1023;
    const u32 l_next = (min(c + 1, 3u) << 11) | ((flip ? 2047 - pl : pl) << 1) | ((model & 1) ^ (flip ? 1u : 0u));
    return mps ? m_next : l_next;
}

// counting-mode coding of one bin (lbac_encode_bin with no bitstream); the range after an LPS is
// formed beside the one after an MPS and selected
__device__ __forceinline__ void cr_code(u32 &range, u32 &bits, u32 lps, bool eq)
{
    u32 mps = range - lps;
    const u32 s = mps < 256 ? 1u : 0u;
    mps |= 0x100;
    const u32 l = (range << s) - mps;                // at least 1: a model's LPS range is never 0
    const u32 sh = (u32)__clz((int)l) - 23u;
    range = eq ? mps : l << sh;
    bits += s + (eq ? 0u : sh);
}

// cr_next of every model and bin, in shared memory: next[2 model + bin].  The rule takes some 17
// instructions, a look-up 3, and a chain runs 2 to 3 of them per bin.
struct CrTable { u16 next[2 * 8192]; };

__device__ __forceinline__ u32 cr_step(const CrTable &T, u32 mdl, u32 bin) { return T.next[2 * mdl + bin]; }

// what the range coder needs of a bin: the model's LPS range (8 bits) and whether the bin is the MPS
__device__ __forceinline__ u16 cr_code_of(u32 mdl, u32 bin)
{
    return (u16)(((mdl >> 3) & 255) | (bin == (mdl & 1) ? 256u : 0u));
}

// bits of the exp-Golomb escape of v >= -1 (order 0): sum of 2^k steps down to below 0
__device__ __forceinline__ u32 cr_egk(int v) { return 2u * (31u - (u32)__clz(v + 2)) + 1u; }

// blocks per SM below which a list takes one launch, a CTA per block (k_cr_short), instead of listing,
// grouping and chains: as long as two waves of CTAs hold it.  On 152 SMs, one 4x4 block takes 10.5 us and
// 22, 768 blocks of at most 64 samples 56 and 71, of 1024 samples and more 339 and 585; at 2,048 99 and 71,
// 545 and 538.
constexpr int CR_SHORT_PER_SM = 6;
constexpr int CR_LIST_WARPS = 8;     // blocks per CTA of the listing
constexpr int CR_LIST_UNROLL = 4;    // 32-position windows whose loads are in flight together
constexpr u32 CR_BAD = 0xFFFFFFFFu;  // a request outside the domain, or fewer levels than num_sig

// A listed level: its run of zeros (12 bits), min(level - 1, 7) (3), whether level - 1 >= 8 (1), the
// last2 context of its position (4), whether it is the block's last scan position (1).
__device__ __forceinline__ u32 cr_entry(int run, int sym, int pos, int n)
{
    return (u32)run | (u32)min(sym, 7) << 12 | (sym >= 8 ? 1u << 15 : 0u) | (u32)(31 - __clz(pos + 1)) << 16 |
           (pos == n - 1 ? 1u << 20 : 0u);
}

// Listing, a warp per block: checks the request and writes, in scan order, an entry for each of the
// block's first num_sig non-zero levels to list[] at the block's own level offset (a ballot and a
// prefix count per 32 positions); sums the bits the coder state has no part in (signs and escapes), or
// CR_BAD, and the bins the block will code (0 for a bad request).
struct CrListed { u32 fixed, len; };
__device__ __forceinline__ CrListed cr_list(const CrParams &P, int r, u32 *list_all, int lane)
{
    const u32 word = lane < 30 ? reinterpret_cast<const u32 *>(P.reqs + r)[lane] : 0u;
    const u32 offset = __shfl_sync(0xffffffffu, word, 0), dims = __shfl_sync(0xffffffffu, word, 1);
    const u32 sr = __shfl_sync(0xffffffffu, word, 2);
    const int lw = dims & 255, lh = (dims >> 8) & 255, ch = (dims >> 16) & 255, top = ch ? 5 : 6;
    const int num_sig = sr & 0xffff, range = sr >> 16;
    bool ok = lw >= 2 && lw <= top && lh >= 2 && lh <= top;
    const int n = ok ? 1 << (lw + lh) : 0;
    ok = ok && num_sig >= 1 && num_sig <= n && range >= 256 && range <= 511 &&
         (unsigned long long)offset + (unsigned long long)n <= P.n_levels;
    // the models, two to a word from word 3 on: a live LPS probability and 13 bits (chroma codes no
    // last2 context past 9: its last word is not looked at)
    if (lane >= 3 && lane < (ch ? 29 : 30))
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const int m = (int)(s16)(word >> (16 * k));
            ok = ok && ((m >> 1) & 1023) >= 4 && m >= 0 && m < 8192;
        }
    ok = __all_sync(0xffffffffu, ok);
    int cnt = 0;
    u32 len = 0, fixed = 0;
    if (ok) {
        const s16 *coef = P.levels + offset;
        const u16 *scan = P.scan[lw][lh];
        u32 *list = list_all + offset;
        int last = -1;                                // position of the last non-zero level before the window
        for (int base = 0; base < n && cnt < num_sig; base += 32 * CR_LIST_UNROLL) {
            int c[CR_LIST_UNROLL];
#pragma unroll
            for (int j = 0; j < CR_LIST_UNROLL; j++) {
                const int i = base + 32 * j + lane;
                c[j] = i < n ? coef[scan[i]] : 0;
            }
#pragma unroll
            for (int j = 0; j < CR_LIST_UNROLL; j++) {
                const u32 m = __ballot_sync(0xffffffffu, c[j] != 0);
                if (m == 0) continue;
                const u32 below = m & ((1u << lane) - 1);
                const int i = base + 32 * j + lane, at = cnt + __popc(below);
                if (c[j] != 0 && at < num_sig) {
                    const int prev = below ? base + 32 * j + 31 - __clz((int)below) : last;
                    const int run = i - prev - 1, sym = abs(c[j]) - 1;
                    list[at] = cr_entry(run, sym, i, n);
                    len += 3 + min(run, 15) + min(sym, 7);
                    fixed += 1 + (run >= 16 ? cr_egk(run - 17) : 0u) + (sym >= 8 ? cr_egk(sym - 9) : 0u);
                }
                cnt += __popc(m);
                last = base + 32 * j + 31 - __clz((int)m);
            }
        }
        len = __reduce_add_sync(0xffffffffu, len);
        fixed = __reduce_add_sync(0xffffffffu, fixed);
        ok = cnt >= num_sig;
    }
    return { ok ? fixed : CR_BAD, ok ? len : 0u };
}

// the listing of a grouped list: a block's bins are its chain length
__global__ void __launch_bounds__(32 * CR_LIST_WARPS) k_cr_list(const CrParams P, u32 *list_all, BlockOrder O)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r = blockIdx.x * CR_LIST_WARPS + warp;
    if (r >= P.n) return;
    const CrListed l = cr_list(P, r, list_all, lane);
    if (lane == 0) {
        O.key[r] = bs_count(O.counts, l.len);
        P.fixed[r] = l.fixed;
    }
}

// Coding, 32 chains of like length per CTA in the order of the grouping.  Neither the models nor the
// order of the bins depend on the range, so the chain splits over the CTA's five warps, lane l of each
// working on block l: warps 0 to 2 step the run, level and run_rdoq models, warp 3 the last models --
// each but warp 2 writing a code per bin (the model's LPS range and whether the bin is the MPS) to its
// place in the block's sequence of bins -- and warp 4 runs the range over the codes, one chunk behind.
// All but warp 3 take one bin per iteration, whatever symbol of the block it belongs to, so lanes wait
// for one another only at the end of a chunk.  What bounds a call is its longest chain, one dependent
// instruction after the other: a lane that codes its block alone, symbol after symbol, has to loop
// over the longest symbol of its warp each time.
//
// The 54 models of a lane's block sit in shared memory as [model][lane].
constexpr int CR_CTAS = 3;            // CTAs of 74 KB that share an SM
constexpr int CR_ROLES = 5;
constexpr int CR_CODES = 256;         // most bins of a chunk
constexpr int CR_LEVEL_CODES = 25;    // most bins of one level: run 16, level 8, last flag

struct CrShared {
    CrTable T;
    u16 mdl[54][32];                  // run, run_rdoq, level (12 each), last1 (6), last2 (12)
    u16 codes[2][CR_CODES + 4][32];
    u32 ring[CR_ROLES - 1][BS_RING][32];
    int n_codes[2][32];
    int more[2];                      // another chunk follows
    int group;
};

// where a lane stands in its block's list
struct CrWalk {
    BsWindow list;
    u32 k, num_sig;
    int t0;                           // context pair of the next level (2 min(previous level - 1, 5))
    // the next level: its entry and context pair, and its place nc in the chunk, which moves past it
    __device__ __forceinline__ u32 take(int &nc, int &at, int &t)
    {
        const u32 v = list.take(k++);
        at = nc;
        t = t0;
        const int nl = (v >> 12) & 7;
        nc += 3 + min((int)(v & 4095), 15) + nl - (int)(v >> 20);
        t0 = min(nl, 5) << 1;
        return v;
    }
};

// the run (ROLE 0), level (1) or run_rdoq (2) models of a chunk's levels, one bin per iteration: a
// truncated unary symbol is its first bin ('1' for 0) on the first model of the pair, then '0' per unit
// and the closing '1' on the second, omitted at the cap (run 16, level 8; run_rdoq has none).  A long
// run of zeros stops changing the run_rdoq model once its probability is too small to move, so its
// walk skips to the closing bin there.
template <int ROLE>
__device__ __forceinline__ int cr_models(CrShared &S, CrWalk &W, u16 (*codes)[32], int lane)
{
    int nc = 0, at = 0, t = 0, z = 0, cnt = -1, target = 0;
    for (;;) {
        if (z > cnt) {                                 // the symbol is done
            if (W.k >= W.num_sig || nc > CR_CODES - CR_LEVEL_CODES) break;
            const u32 v = W.take(nc, at, t);
            const int run = v & 4095, nr = min(run, 15), nl = (v >> 12) & 7;
            target = ROLE == 1 ? nl + (int)((v >> 15) & 1) : run;
            cnt = ROLE == 0 ? nr : ROLE == 1 ? nl : run;
            at += ROLE == 1 ? 1 + nr : 0;
            t += ROLE == 0 ? 0 : ROLE == 1 ? 24 : 12;
            z = 0;
        }
        u16 &slot = S.mdl[t + (z > 0 ? 1 : 0)][lane];
        const u32 m = slot, bin = z == target ? 1u : 0u;
        const u32 nm = cr_step(S.T, m, bin);
        if (ROLE != 2) codes[at + z][lane] = cr_code_of(m, bin);
        slot = (u16)nm;
        z = (ROLE == 2 && nm == m && z > 0 && z < target) ? target : z + 1;
    }
    return nc;
}

// the last flags of a chunk's levels, each on the averaged pair of its two models
__device__ __forceinline__ void cr_lasts(CrShared &S, CrWalk &W, u16 (*codes)[32], int lane)
{
    int nc = 0;
    while (W.k < W.num_sig && nc <= CR_CODES - CR_LEVEL_CODES) {
        int at, t;
        const u32 v = W.take(nc, at, t);
        if (v >> 20) break;                            // the last scan position has no flag
        const int i1 = 36 + (t >> 1), i2 = 42 + (int)((v >> 16) & 15);
        const u32 f1 = S.mdl[i1][lane], f2 = S.mdl[i2][lane];
        const u32 p1 = (f1 & 2047) >> 1, p2 = (f2 & 2047) >> 1, c1 = f1 & 1, c2 = f2 & 1;
        const bool first = p1 < p2;
        const u32 cm = (c1 == c2 || first) ? c1 : c2;
        const u32 pl = c1 == c2 ? (p1 + p2) >> 1 : 1023 - ((first ? p2 - p1 : p1 - p2) >> 1);
        const u32 flag = W.k == W.num_sig ? 1u : 0u;
        codes[nc - 1][lane] = (u16)((pl >> 2) | (flag == cm ? 256u : 0u));
        S.mdl[i1][lane] = (u16)cr_step(S.T, f1, flag);
        S.mdl[i2][lane] = (u16)cr_step(S.T, f2, flag);
    }
}

// cr_next of every model and bin by `threads` threads, of which this is number t
__device__ __forceinline__ void cr_fill(CrTable &T, int t, int threads)
{
    for (int k = t; k < 2 * 8192; k += threads) T.next[k] = (u16)cr_next((u32)k >> 1, (k & 1) == ((k >> 1) & 1));
}

// the chains of 32 listed blocks by the CTA's five warps, lane l working on block i (where `mine`), whose
// listing gave `fixed`; every thread of the CTA calls it, with the model table in place
__device__ __forceinline__ void cr_chains(const CrParams &P, CrShared &S, const u32 *list_all, int lane, int role, bool mine,
                                          int i, u32 fixed)
{
    // a role's models: words [w0, w1) of the request's 27 and the same words of the result
    const int w0 = role == 0 ? 0 : role == 1 ? 12 : role == 2 ? 6 : 18, w1 = role == 3 ? 27 : role == 4 ? 18 : w0 + 6;
    const u32 *qw = reinterpret_cast<const u32 *>(P.reqs + i);
    u32 *ow = reinterpret_cast<u32 *>(P.out + i);
    const u32 sr = qw[2];
    CrWalk W;
    W.k = 0;
    W.num_sig = fixed == CR_BAD ? 0u : sr & 0xffff;    // a bad request codes no level: its state stays
    W.list.open(list_all + qw[0], role < 4 ? W.num_sig : 0u, smem_addr(&S.ring[role & 3][0][lane]));
    W.t0 = 10;
    for (int k = w0; k < w1; k++) {
        const u32 x = qw[3 + k];
        S.mdl[2 * k][lane] = (u16)x;
        S.mdl[2 * k + 1][lane] = (u16)(x >> 16);
    }
    u32 range = sr >> 16, bits = fixed;
    bool fill = true;
    for (int s = 0;; s++) {
        const int b = s & 1;
        u16 (*codes)[32] = S.codes[b];
        if (fill) {
            if (role == 0) {
                const int nc = cr_models<0>(S, W, codes, lane);
                // up to a multiple of four codes: an MPS with LPS range 0 changes nothing
#pragma unroll
                for (int j = 0; j < 3; j++) codes[nc + j][lane] = 256;
                S.n_codes[b][lane] = nc;
                const int more = __any_sync(0xffffffffu, W.k < W.num_sig);
                if (lane == 0) S.more[b] = more;
            } else if (role == 1) {
                cr_models<1>(S, W, codes, lane);
            } else if (role == 2) {
                cr_models<2>(S, W, codes, lane);
            } else if (role == 3) {
                cr_lasts(S, W, codes, lane);
            }
        }
        if (role == 4 && s > 0) {
            codes = S.codes[b ^ 1];
            const int nc = S.n_codes[b ^ 1][lane];
            for (int j = 0; j < nc; j += 4) {
                u32 c[4];
#pragma unroll
                for (int q = 0; q < 4; q++) c[q] = codes[j + q][lane];
#pragma unroll
                for (int q = 0; q < 4; q++) cr_code(range, bits, c[q] & 255, c[q] >> 8);
            }
        }
        __syncthreads();
        if (!fill) break;
        fill = S.more[b] != 0;
    }
    W.list.close();
    if (mine) {
        for (int k = w0; k < w1; k++) ow[2 + k] = (u32)S.mdl[2 * k][lane] | (u32)S.mdl[2 * k + 1][lane] << 16;
        if (role == 4) {
            ow[0] = bits;                              // CR_BAD = ~0 for a bad request
            ow[1] = range;
        }
    }
}

__global__ void __launch_bounds__(32 * CR_ROLES) k_cr_code(const CrParams P, const u32 *list_all, const BlockOrder O)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    CrShared &S = *reinterpret_cast<CrShared *>(smem_raw);
    const int lane = threadIdx.x & 31, role = threadIdx.x >> 5;
    cr_fill(S.T, threadIdx.x, 32 * CR_ROLES);
    // groups of 32 chains from the work counter, the longest chains first
    for (;;) {
        if (threadIdx.x == 0) S.group = (int)atomicAdd(O.counts + BS_WORK, 1u);
        __syncthreads();
        if (S.group * 32 >= P.n) return;
        const int at = S.group * 32 + lane;
        const bool mine = at < P.n;
        const int i = mine ? O.perm[at] : 0;
        cr_chains(P, S, list_all, lane, role, mine, i, mine ? P.fixed[i] : CR_BAD);
    }
}

// A short list, in one launch: a CTA per block, whose first warp lists it while the others fill the model
// table; lane 0 of each warp then works on its chain.
__global__ void __launch_bounds__(32 * CR_ROLES) k_cr_short(const CrParams P, u32 *list_all)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    CrShared &S = *reinterpret_cast<CrShared *>(smem_raw);
    const int lane = threadIdx.x & 31, role = threadIdx.x >> 5;
    if (role == 0) {
        const CrListed l = cr_list(P, blockIdx.x, list_all, lane);
        if (lane == 0) S.group = (int)l.fixed;
    } else {
        cr_fill(S.T, threadIdx.x - 32, 32 * (CR_ROLES - 1));
    }
    __syncthreads();
    cr_chains(P, S, list_all, lane, role, lane == 0, blockIdx.x, lane == 0 ? (u32)S.group : CR_BAD);
}

int launch_coef_rate(const void *reqs, int n, const s16 *levels, unsigned long long n_levels, void *out,
                     cudaStream_t st)
{
    if (n < 0 || (n > 0 && (!reqs || !levels || !out))) return set_status(UC_ERR_ARG, "coef_rate: null argument");
    if (n == 0) return UC_OK;
    int dev = 0;
    UC_CHECK(cudaGetDevice(&dev));
    const DevTables *tab = device_tables(dev);
    if (!tab) return set_status(UC_ERR_MEMORY, "coef_rate: table upload failed");
    CrParams P;
    memset(&P, 0, sizeof(P));
    P.reqs = (const CrReq *)reqs; P.n = n; P.levels = levels; P.n_levels = n_levels; P.out = (CrOut *)out;
    for (int a = 0; a < 7; a++)
        for (int b = 0; b < 7; b++) P.scan[a][b] = tab->scan[a][b];
    int sms = 0;
    UC_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const bool brief = n < CR_SHORT_PER_SM * sms;
    // one word per level (the lists, at the levels' offsets), the grouping's arrays, a word per block
    const size_t b_list = ((size_t)n_levels * sizeof(u32) + 255) & ~(size_t)255, b_order = bs_bytes((size_t)n);
    char *ws = nullptr;
    int rc = work_alloc((void **)&ws, b_list + (brief ? 256 : b_order + (size_t)n * sizeof(u32)), st);
    if (rc) return rc;
    u32 *list = (u32 *)ws;
    const BlockOrder O = bs_place(ws + b_list, (size_t)n);
    P.fixed = (u32 *)(ws + b_list + b_order);
    cudaError_t e = cudaFuncSetAttribute(brief ? (const void *)k_cr_short : (const void *)k_cr_code,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(CrShared));
    if (e == cudaSuccess && brief) {
        k_cr_short<<<(unsigned)n, 32 * CR_ROLES, sizeof(CrShared), st>>>(P, list);
        e = cudaGetLastError();
    } else if (e == cudaSuccess && (e = cudaMemsetAsync(O.counts, 0, BS_CLEAR, st)) == cudaSuccess) {
        // persistent CTAs: each fills its model table once
        k_cr_list<<<(unsigned)((n + CR_LIST_WARPS - 1) / CR_LIST_WARPS), 32 * CR_LIST_WARPS, 0, st>>>(P, list, O);
        k_bs_scatter<<<(unsigned)((n + BS_BUCKETS - 1) / BS_BUCKETS), BS_BUCKETS, 0, st>>>(O.key, O.counts, n, O.perm);
        k_cr_code<<<(unsigned)std::min((n + 31) / 32, sms * CR_CTAS), 32 * CR_ROLES, sizeof(CrShared), st>>>(P, list, O);
        e = cudaGetLastError();
    }
    rc = work_free(ws, st);
    UC_CHECK(e);
    if (rc) return rc;
    count_launch(brief ? 1 : 3);
    return UC_OK;
}

struct CrScratch {
    std::mutex mu;
    cudaStream_t st = nullptr;
    void *buf = nullptr;
    size_t cap = 0;
};
static CrScratch g_cr[64];

}  // namespace uc

using namespace uc;

extern "C" UAVS3E_CUDA_API int uavs3e_cuda_coef_rate(const uavs3e_cuda_coef_rate_req_t *reqs, int n,
                                                    const int16_t *levels, size_t n_levels,
                                                    uavs3e_cuda_coef_rate_out_t *out)
{
    int rc = ensure_init();
    if (rc) return rc;
    if (n < 0 || (n > 0 && (!reqs || !levels || !out))) return set_status(UC_ERR_ARG, "coef_rate: bad argument");
    if (n == 0) return UC_OK;
    int dev = 0;
    UC_CHECK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return set_status(UC_ERR_UNSUPPORTED, "coef_rate: device index");
    CrScratch &S = g_cr[dev];
    std::lock_guard<std::mutex> lk(S.mu);
    if (!S.st) UC_CHECK(cudaStreamCreateWithFlags(&S.st, cudaStreamNonBlocking));
    auto up = [](size_t b) { return (b + 255) & ~(size_t)255; };
    const size_t b_req = up((size_t)n * sizeof(*reqs)), b_lev = up(n_levels * sizeof(int16_t));
    const size_t need = b_req + b_lev + up((size_t)n * sizeof(*out));
    if (S.cap < need) {
        if (S.buf) UC_CHECK(cudaFree(S.buf));
        S.buf = nullptr;
        S.cap = 0;
        UC_CHECK(cudaMalloc(&S.buf, need));
        S.cap = need;
    }
    char *b = (char *)S.buf;
    void *d_req = b, *d_out = b + b_req + b_lev;
    s16 *d_lev = (s16 *)(b + b_req);
    UC_CHECK(cudaMemcpyAsync(d_req, reqs, (size_t)n * sizeof(*reqs), cudaMemcpyHostToDevice, S.st));
    UC_CHECK(cudaMemcpyAsync(d_lev, levels, n_levels * sizeof(int16_t), cudaMemcpyHostToDevice, S.st));
    rc = launch_coef_rate(d_req, n, d_lev, (unsigned long long)n_levels, d_out, S.st);
    if (rc) return rc;
    UC_CHECK(cudaMemcpyAsync(out, d_out, (size_t)n * sizeof(*out), cudaMemcpyDeviceToHost, S.st));
    UC_CHECK(cudaStreamSynchronize(S.st));
    return UC_OK;
}

extern "C" UAVS3E_CUDA_API int uavs3e_cuda_coef_rate_device(const uavs3e_cuda_coef_rate_req_t *d_reqs, int n,
                                                           const int16_t *d_levels, size_t n_levels,
                                                           uavs3e_cuda_coef_rate_out_t *d_out, void *stream)
{
    int rc = ensure_init();
    if (rc) return rc;
    return launch_coef_rate(d_reqs, n, d_levels, (unsigned long long)n_levels, d_out, (cudaStream_t)stream);
}
