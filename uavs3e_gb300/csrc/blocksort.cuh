// Grouping of variable-length block chains: kernels that walk one sequential chain per lane (the
// coefficient rate, the RDOQ decision) take their blocks in the order of their chain lengths, the
// longest first, so that the 32 chains of a warp end together and the longest ones start first.
//
// The kernel that lists a block's chain counts the block into one of 256 buckets of its length
// (bs_bucket: 16 buckets per octave, so the chains of a bucket differ by at most 1/16) and keeps
// the block's rank in it; k_bs_scatter turns the counts into bucket offsets and writes the order.
#pragma once
#include "common.cuh"

namespace uc {

constexpr int BS_BUCKETS = 256;

// bucket of a chain of `len` steps, longer chains first; lengths of 2^19 and more share bucket 0
__device__ __forceinline__ u32 bs_bucket(u32 len)
{
    if (len < 16) return BS_BUCKETS - 1 - len;
    const int e = 31 - __clz(len);
    const u32 v = ((u32)(e - 3) << 4) + ((len >> (e - 4)) & 15u);
    return BS_BUCKETS - 1 - min(v, (u32)(BS_BUCKETS - 1));
}

// {bucket, rank in the bucket} of a block (one lane calls it); counts[] starts at 0
__device__ __forceinline__ uint2 bs_count(u32 *counts, u32 len)
{
    const u32 b = bs_bucket(len);
    return make_uint2(b, atomicAdd(counts + b, 1u));
}

// perm[offset of the bucket + rank] = block; 256 threads a CTA, one block per thread
static __global__ void __launch_bounds__(BS_BUCKETS) k_bs_scatter(const uint2 *key, const u32 *counts, int n, int *perm)
{
    __shared__ u32 s_off[BS_BUCKETS];
    __shared__ u32 s_warp[BS_BUCKETS / 32];
    const int t = threadIdx.x, lane = t & 31;
    const u32 own = counts[t];
    u32 v = own;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const u32 p = __shfl_up_sync(0xffffffffu, v, d);
        if (lane >= d) v += p;
    }
    if (lane == 31) s_warp[t >> 5] = v;
    __syncthreads();
    for (int w = 0; w < (t >> 5); w++) v += s_warp[w];
    s_off[t] = v - own;
    __syncthreads();
    const int i = blockIdx.x * BS_BUCKETS + t;
    if (i >= n) return;
    const uint2 k = key[i];
    perm[s_off[k.x] + k.y] = i;
}

// A lane's window on its chain's list of words: the chains of a warp read 32 lists at 32 places, so
// nearly every read of some lane leaves the L1; the words come through a ring of BS_RING words a lane
// in shared memory ([word][lane]), filled BS_AHEAD words ahead by asynchronous copies, one copy group
// per word.
constexpr int BS_RING = 8, BS_AHEAD = 6;
struct BsWindow {
    const u32 *list;
    u32 ring;                         // shared address of the lane's column
    u32 n;
    __device__ __forceinline__ void fetch(u32 k)
    {
        // past the list's end the last word again, so that every step has its group
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n\tcp.async.commit_group;" ::
                     "r"(ring + (k & (BS_RING - 1)) * 128), "l"(list + min(k, n - 1)) : "memory");
    }
    // list of n words (n may be 0: nothing is read); word 0 is in place afterwards
    __device__ __forceinline__ void open(const u32 *l, u32 words, u32 column)
    {
        list = l; n = words; ring = column;
        if (n == 0) return;
#pragma unroll 1
        for (u32 k = 0; k < BS_AHEAD; k++) fetch(k);
        asm volatile("cp.async.wait_group %0;" ::"n"(BS_AHEAD - 1) : "memory");
    }
    // word k, and the copy of word k + BS_AHEAD; word k + 1 is in place afterwards
    __device__ __forceinline__ u32 take(u32 k)
    {
        u32 v;
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(ring + (k & (BS_RING - 1)) * 128) : "memory");
        fetch(k + BS_AHEAD);
        asm volatile("cp.async.wait_group %0;" ::"n"(BS_AHEAD - 1) : "memory");
        return v;
    }
    // no copy of the lane is in flight afterwards
    __device__ __forceinline__ void close() { asm volatile("cp.async.wait_all;" ::: "memory"); }
};

// the arrays of one call's grouping inside a workspace: counts (and one work counter), cleared before
// the listing; then {bucket, rank}, then the order
struct BlockOrder { u32 *counts; uint2 *key; int *perm; };
constexpr int BS_WORK = BS_BUCKETS;                       // index of the work counter
constexpr size_t BS_CLEAR = (BS_BUCKETS + 1) * sizeof(u32);
constexpr size_t BS_HEAD = (BS_CLEAR + 255) & ~(size_t)255;

static inline size_t bs_bytes(size_t n)
{
    return BS_HEAD + ((n * sizeof(uint2) + 255) & ~(size_t)255) + ((n * sizeof(int) + 255) & ~(size_t)255);
}

static inline BlockOrder bs_place(void *base, size_t n)
{
    BlockOrder o;
    o.counts = (u32 *)base;
    o.key = (uint2 *)((char *)base + BS_HEAD);
    o.perm = (int *)((char *)o.key + ((n * sizeof(uint2) + 255) & ~(size_t)255));
    return o;
}

}  // namespace uc
