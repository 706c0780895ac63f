// ibf.cu -- single-level interleaved Bloom filter on the device: store, emplace/clear/widen kernels, the plain
// (one launch per call) query kernels, and their C-ABI entry points (include/hibf_gb300.h).
//
// Reference interface: seqan::hibf::interleaved_bloom_filter (include/hibf/interleaved_bloom_filter.hpp,
// src/interleaved_bloom_filter.cpp).

#include <algorithm>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/hibf_gb300_synthetic.h"
#include "archive.hpp"
#include "common.hpp"
#include "count.cuh"
#include "device.cuh"

namespace hibf_gb300
{

thread_local std::string g_last_error;

void set_last_error(std::string msg)
{
    g_last_error = std::move(msg);
}

// ---------------------------------------------------------------------------------------------------------------
// Kernels
// ---------------------------------------------------------------------------------------------------------------

// emplace (src/interleaved_bloom_filter.cpp:119-140).  One thread per value; atomicOr makes concurrent inserts
// order-independent.  The old words are not needed (an IBF that tracks occupancy inserts through emplace_exact), so
// the atomics return nothing and a warp never waits on them.
__global__ void k_emplace(uint64_t * __restrict__ words, uint64_t bin_size, uint32_t row_words, uint32_t shift,
                          uint32_t h, uint64_t const * __restrict__ values, uint64_t const * __restrict__ bins,
                          uint64_t n, uint64_t bin, uint64_t n_bins, int * bad_bin)
{
    uint64_t const stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < n; i += stride)
    {
        uint64_t const v = values[i];
        uint64_t const b = bins ? bins[i] : bin;
        if (b >= n_bins)
        {
            *bad_bin = 1; // device-supplied bin index out of range: skipped, reported by hibf_gpu_ibf_status
            continue;
        }
        uint64_t const bit = 1ull << (b & 63u);
        uint64_t const wofs = b >> 6;
        for (uint32_t k = 0; k < h; ++k)
        {
            uint64_t const r = hash_row(v, c_hash_seeds[k], shift, bin_size);
            atomicOr(reinterpret_cast<unsigned long long *>(words + r * row_words + wofs),
                     static_cast<unsigned long long>(bit));
        }
    }
}

// emplace of the synthetic single-level workload: value i of the launch is hg_ibf_bin_value of bin
// first_bin + i / vpb, generated in place instead of read (same bits as k_emplace with those values; the atomics
// return nothing).
__global__ void k_synth_emplace(uint64_t * __restrict__ words, uint64_t bin_size, uint32_t row_words, uint32_t shift,
                                uint32_t h, uint64_t seed, uint64_t vpb, uint64_t first_bin, uint64_t n)
{
    uint64_t const stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < n; i += stride)
    {
        uint64_t const b = first_bin + i / vpb;
        uint64_t const v = hg_ibf_bin_value(seed, vpb, b, i % vpb);
        uint64_t const bit = 1ull << (b & 63u);
        uint64_t const wofs = b >> 6;
        for (uint32_t k = 0; k < h; ++k)
        {
            uint64_t const r = hash_row(v, c_hash_seeds[k], shift, bin_size);
            atomicOr(reinterpret_cast<unsigned long long *>(words + r * row_words + wofs),
                     static_cast<unsigned long long>(bit));
        }
    }
}

// ---------------------------------------------------------------------------------------------------------------
// Exact occupancy.  The reference counts a value for its bin when one of its bits was not set yet, inserting one value
// after the other (src/interleaved_bloom_filter.cpp:119-140).  With concurrent atomicOr that depends on timing, so an
// IBF that tracks occupancy inserts in chunks, in two passes.  The first enters every position (row * tb + bin) that is
// still unset into a hash table and lowers the position's entry to the chunk's first value there; the second counts a
// value that is first at one of its positions and sets its bits.  Both are bound by random accesses that L2 serves (the
// table of a chunk is at most 100 MB): 530,624 values with h = 2 take 41 us; sorting the positions took 14 launches,
// 260 us, and as much again in allocations.
// ---------------------------------------------------------------------------------------------------------------
constexpr unsigned long long kFreeEntry = ~0ull;
constexpr uint32_t kIsSet = ~0u; // the entry of a position whose bit was set before the chunk, or of no position

// Value i of the chunk and its bin: from the arrays, or (SYNTH) value `first + i` of the generated bin `bin`.
template <bool SYNTH>
__device__ __forceinline__ uint64_t occ_value(uint64_t const * values, uint64_t const * bins, uint64_t seed,
                                              uint64_t vpb, uint64_t first, uint64_t i, uint64_t bin, uint64_t & b)
{
    b = !SYNTH && bins ? bins[i] : bin;
    if constexpr (SYNTH)
        return hg_ibf_bin_value(seed, vpb, bin, first + i);
    else
        return values[i];
}

// The table has mask + 1 slots (a power of two, at least 1.5 per position, so that a free one is always found): keys
// and the lowest value index per key.  entries[i * h + k]: the slot of value i's position k.  A value that repeats the
// one before it in its bin is not entered: that one has its positions and comes first.  (2^20 times one value, h = 2:
// every position queued for two addresses, 1,715 us a call, now 85.)
template <bool SYNTH>
__global__ void k_occ_enter(uint64_t const * __restrict__ words, uint64_t bin_size, uint32_t row_words, uint32_t shift,
                            uint32_t h, uint64_t const * __restrict__ values, uint64_t const * __restrict__ bins,
                            uint64_t seed, uint64_t vpb, uint64_t first, uint64_t n, uint64_t bin, uint64_t n_bins,
                            uint64_t tb, unsigned long long * keys, unsigned int * lowest, uint32_t mask,
                            uint32_t * __restrict__ entries)
{
    uint64_t const stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    uint64_t const first_i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x;
    int const lane = threadIdx.x & 31;
    for (uint64_t base = first_i - lane; base < n; base += stride) // whole warps: they compare their values
    {
        uint64_t const i = base + lane;
        uint64_t b = ~0ull, v = 0;
        if (i < n)
            v = occ_value<SYNTH>(values, bins, seed, vpb, first, i, bin, b);
        uint64_t const v_before = __shfl_up_sync(kFullMask, v, 1), b_before = __shfl_up_sync(kFullMask, b, 1);
        bool const repeats = lane > 0 && v == v_before && b == b_before;
        for (uint32_t k = 0; k < h && i < n; ++k)
        {
            uint32_t entry = kIsSet;
            if (b < n_bins && !repeats)
            {
                uint64_t const r = hash_row(v, c_hash_seeds[k], shift, bin_size);
                if (!((words[r * row_words + (b >> 6)] >> (b & 63u)) & 1u))
                {
                    unsigned long long const key = r * tb + b;
                    uint32_t slot = static_cast<uint32_t>(((key ^ (key >> 32)) * 11400714819323198485ULL) >> 32) & mask;
                    for (;;)
                    {
                        unsigned long long const old = atomicCAS(keys + slot, kFreeEntry, key);
                        if (old == kFreeEntry || old == key)
                            break;
                        slot = (slot + 1u) & mask;
                    }
                    atomicMin(lowest + slot, static_cast<unsigned int>(i));
                    entry = slot;
                }
            }
            entries[i * h + k] = entry;
        }
    }
}

template <bool SYNTH>
__global__ void k_occ_insert(uint64_t * __restrict__ words, uint64_t bin_size, uint32_t row_words, uint32_t shift,
                             uint32_t h, uint64_t const * __restrict__ values, uint64_t const * __restrict__ bins,
                             uint64_t seed, uint64_t vpb, uint64_t first, uint64_t n, uint64_t bin, uint64_t n_bins,
                             unsigned int const * __restrict__ lowest, uint32_t const * __restrict__ entries,
                             unsigned long long * __restrict__ occupancy, int * bad_bin)
{
    uint64_t const stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    uint64_t const first_i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x;
    int const lane = threadIdx.x & 31;
    for (uint64_t base = first_i - lane; base < n; base += stride) // whole warps: they add up their counts
    {
        uint64_t const i = base + lane;
        bool newly = false;
        uint64_t b = ~0ull;
        if (i < n)
        {
            uint64_t const v = occ_value<SYNTH>(values, bins, seed, vpb, first, i, bin, b);
            if (b >= n_bins)
            {
                *bad_bin = 1; // device-supplied bin index out of range: skipped, reported by hibf_gpu_ibf_status
            }
            else
            {
                unsigned long long const bit = 1ull << (b & 63u);
                for (uint32_t k = 0; k < h; ++k)
                {
                    uint32_t const entry = entries[i * h + k];
                    if (entry == kIsSet)
                        continue;
                    newly = newly || lowest[entry] == static_cast<unsigned int>(i);
                    uint64_t const r = hash_row(v, c_hash_seeds[k], shift, bin_size);
                    atomicOr(reinterpret_cast<unsigned long long *>(words + r * row_words + (b >> 6)), bit);
                }
            }
        }
        // one addition per bin and warp: a user bin's values usually come together (530,624 values of 64 bins added one
        // by one took 50 us)
        unsigned const counted = __ballot_sync(kFullMask, newly);
        if (newly)
        {
            unsigned const same = __match_any_sync(counted, b);
            if (lane == __ffs(same) - 1)
                atomicAdd(occupancy + b, static_cast<unsigned long long>(__popc(same)));
        }
    }
}

// Sets *bad (mapped host memory) when a bin index is out of range.
__global__ void k_check_bins(uint64_t const * __restrict__ bins, uint64_t n, uint64_t n_bins, int * bad)
{
    uint64_t const stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    bool mine = false;
    for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < n; i += stride)
        mine = mine || bins[i] >= n_bins;
    if (mine)
        *bad = 1;
}

// clear(bin) (src/interleaved_bloom_filter.cpp:142-148): clear one bit of every row.
__global__ void k_clear_bin(uint64_t * __restrict__ words, uint64_t bin_size, uint32_t row_words, uint64_t word,
                            uint64_t keep)
{
    uint64_t const stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    for (uint64_t r = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; r < bin_size; r += stride)
        atomicAnd(reinterpret_cast<unsigned long long *>(words + r * row_words + word), keep);
}

// clear(range) (include/hibf/interleaved_bloom_filter.hpp:283-297): per row, clear the listed bins word by word.
__global__ void k_clear_words(uint64_t * __restrict__ words, uint64_t bin_size, uint32_t row_words,
                              uint32_t const * __restrict__ widx, uint64_t const * __restrict__ keep, uint32_t nw)
{
    uint64_t const total = bin_size * nw;
    uint64_t const stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < total; i += stride)
    {
        uint64_t const r = i / nw;
        uint32_t const e = static_cast<uint32_t>(i % nw);
        atomicAnd(reinterpret_cast<unsigned long long *>(words + r * row_words + widx[e]), keep[e]);
    }
}

// increase_bin_number_to (src/interleaved_bloom_filter.cpp:163-202): old row r becomes the first words of new row r.
__global__ void k_widen(uint64_t * __restrict__ dst, uint32_t dst_row_words, uint64_t const * __restrict__ src,
                        uint32_t src_row_words, uint32_t copy_words, uint64_t bin_size)
{
    uint64_t const total = bin_size * dst_row_words;
    uint64_t const stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < total; i += stride)
    {
        uint64_t const r = i / dst_row_words;
        uint32_t const w = static_cast<uint32_t>(i % dst_row_words);
        dst[i] = w < copy_words ? src[r * src_row_words + w] : 0u;
    }
}

// bulk_contains (src/interleaved_bloom_filter.cpp:204-291) for many values with H hash functions: out[v * bin_words +
// j] = AND of word j of the h rows.  The same work mapping as the counting loop (count.cuh) -- LPV lanes per row, lanes
// hash U values each, the H row words of four sub-steps are loaded together (4 * H loads per lane in flight) -- and
// each lane stores its word of the AND.  The grid's first dimension is the slab (LPV words) of a row wider than a warp,
// so that blocks which start together read the pieces of the same rows.  A warp takes all values that it hashes at
// once, or (FEW, rows of four words and more) only those whose words it loads together.
template <int LPV, int H, typename R, bool FEW>
__global__ void __launch_bounds__(256) k_bulk_contains_h(row_params row, uint64_t const * __restrict__ values,
                                                         uint64_t n, uint64_t * __restrict__ out)
{
    uint32_t const w0 = blockIdx.x * LPV;
    row_params const rp = row_slab(row, w0, LPV);
    constexpr int G = 32 / LPV;
    constexpr int U = LPV >= 4 ? 1 : 4 / LPV;
    constexpr int STEPS = FEW ? 4 : U * LPV;
    constexpr int BLOCK = STEPS * G;
    int const lane = threadIdx.x & 31;
    int const g = lane / LPV;
    int const j = lane % LPV;
    bool const wj = static_cast<uint32_t>(j) < rp.bin_words;
    uint64_t const bw = row.bin_words;
    uint64_t const * __restrict__ words = rp.words + j;
    out += w0;
    uint64_t const warp = (blockIdx.y * static_cast<uint64_t>(blockDim.x) + threadIdx.x) >> 5;
    uint64_t const nwarps = (static_cast<uint64_t>(gridDim.y) * blockDim.x) >> 5;
    for (uint64_t base = warp * BLOCK; base < n; base += nwarps * BLOCK)
    {
        R row_of[U][H];
#pragma unroll
        for (int u = 0; u < U; ++u)
        {
            uint64_t const idx = base + static_cast<uint64_t>(u * 32 + lane);
            uint64_t const v = idx < n && (!FEW || lane < BLOCK) ? values[idx] : 0u;
#pragma unroll
            for (int i = 0; i < H; ++i)
                row_of[u][i] = hash_row_as<R>(v, c_hash_seeds[i], rp.hash_shift, rp.bin_size);
        }
#pragma unroll 1
        for (int s = 0; s < STEPS; s += 4)
        {
            uint64_t w[4][H];
            uint64_t idx[4];
            bool ok[4];
#pragma unroll
            for (int t = 0; t < 4; ++t)
            {
                int const step = s + t;
                int const u = U == 1 ? 0 : step / LPV;
                int const src = (step % LPV) * G + g;
                idx[t] = base + static_cast<uint64_t>(u * 32 + src);
                ok[t] = wj && idx[t] < n;
#pragma unroll
                for (int i = 0; i < H; ++i)
                {
                    R r = row_of[u][i];
                    if constexpr (LPV > 1)
                        r = __shfl_sync(kFullMask, r, src);
                    w[t][i] = ok[t] ? ldg_evict_first(words + static_cast<uint64_t>(r) * rp.row_words) : 0ull;
                }
            }
#pragma unroll
            for (int t = 0; t < 4; ++t)
            {
                uint64_t x = w[t][0];
#pragma unroll
                for (int i = 1; i < H; ++i)
                    x &= w[t][i];
                if (ok[t])
                    out[idx[t] * bw + j] = x;
            }
        }
    }
}

using contains_kernel_t = void (*)(row_params, uint64_t const *, uint64_t, uint64_t *);

template <int H, typename R>
contains_kernel_t contains_kernel_h(uint32_t lpv_log2, bool few)
{
    switch (lpv_log2)
    {
    case 0:
        return k_bulk_contains_h<1, H, R, false>;
    case 1:
        return k_bulk_contains_h<2, H, R, false>;
    case 2:
        return k_bulk_contains_h<4, H, R, false>;
    case 3:
        return k_bulk_contains_h<8, H, R, false>;
    case 4:
        return few ? k_bulk_contains_h<16, H, R, true> : k_bulk_contains_h<16, H, R, false>;
    default:
        return k_bulk_contains_h<32, H, R, false>;
    }
}

template <typename R>
contains_kernel_t contains_kernel(uint64_t h, uint32_t lpv_log2, bool few)
{
    switch (h)
    {
    case 1:
        return contains_kernel_h<1, R>(lpv_log2, few);
    case 2:
        return contains_kernel_h<2, R>(lpv_log2, few);
    case 3:
        return contains_kernel_h<3, R>(lpv_log2, few);
    case 4:
        return contains_kernel_h<4, R>(lpv_log2, few);
    default:
        return contains_kernel_h<5, R>(lpv_log2, few);
    }
}

// The end of a counting block: the sum of its warps' counters, in the caller's width.  A block on its own in its slab
// writes its sums, else the slab's last block (by ticket) writes the totals, and with `reset` leaves totals and ticket
// at 0 for the next call.  (Clearing before and a storing kernel after cost a read of 250 values on 64 bins 5 of its 36
// us.)
__device__ __forceinline__ void finish_counts(uint32_t const * s_counts, uint32_t n_counters, uint32_t w0,
                                              uint32_t slab_words, unsigned long long * totals, unsigned int * ticket,
                                              bool reset, uint64_t bins, int width, void * out)
{
    int const nwarps_block = blockDim.x >> 5;
    uint64_t const bin0 = 64ull * w0;
    for (uint32_t i = threadIdx.x; i < n_counters; i += blockDim.x)
    {
        uint64_t sum = 0;
        for (int w = 0; w < nwarps_block; ++w)
            sum += s_counts[w * n_counters + i];
        if (gridDim.y == 1)
        {
            if (bin0 + i < bins)
                store_count(out, width, bin0 + i, sum);
        }
        else if (sum)
        {
            atomicAdd(totals + bin0 + i, static_cast<unsigned long long>(sum));
        }
    }
    if (gridDim.y == 1)
        return;
    __shared__ bool s_last;
    __threadfence(); // this thread's additions before the block's ticket
    __syncthreads();
    if (threadIdx.x == 0)
        s_last = atomicAdd(ticket, 1u) == gridDim.y - 1u;
    __syncthreads();
    if (!s_last)
        return;
    __threadfence();
    for (uint32_t i = threadIdx.x; i < n_counters; i += blockDim.x)
    {
        if (bin0 + i < bins)
            store_count(out, width, bin0 + i, __ldcg(totals + bin0 + i));
        if (reset && i < 64u * slab_words)
            totals[bin0 + i] = 0;
    }
    if (reset && threadIdx.x == 0)
        *ticket = 0;
}

// bulk_count over n values into one counting vector: every warp counts a contiguous chunk into shared counters of its
// own (planes_flush_to, no shared-memory atomics), the block adds them up and to the 64-bit global totals.
// Four blocks per SM (64 registers) measured faster than two (1.53 vs 2.16 ms for 2^24 values on 1,024 bins, h = 3):
// more warps keep more row loads in flight.  For h of 4 and 5, whose rows fill more registers, three blocks: a million
// values on 64 bins, h = 5, took 70 us with four, which spill.
// The grid's first dimension is the slab of a row wider than a warp: a block counts LPV words of every row, a warp one
// piece of 128 or 256 bytes per value and hash function.  (Rows wider than a warp were counted one value
// at a time, every set bit by an atomic: 200,003 values on 8,192 bins, h = 2, counted and looked up took 9.43 ms; 0.21
// with this kernel, 0.20 with the asynchronous one below.)  One kernel per row width: with all six in one the loop
// spilled 156 bytes per thread at h = 3.
constexpr unsigned count_blocks_per_sm(int h)
{
    return h <= 3 ? 4 : 3;
}

template <int LPV, int H, typename R>
__global__ void __launch_bounds__(256, count_blocks_per_sm(H))
    k_bulk_count(row_params row, uint64_t const * __restrict__ values, uint64_t n, uint64_t chunk,
                 unsigned long long * totals, unsigned int * tickets, bool reset, uint64_t bins, int width,
                 void * __restrict__ out)
{
    extern __shared__ uint32_t s_counts[];
    uint32_t const w0 = blockIdx.x * LPV;
    row_params const rp = row_slab(row, w0, LPV);
    constexpr uint32_t n_counters = 64u * LPV;
    int const nwarps_block = blockDim.x >> 5;
    for (uint32_t i = threadIdx.x; i < n_counters * nwarps_block; i += blockDim.x)
        s_counts[i] = 0;
    __syncthreads();
    int const lane = threadIdx.x & 31;
    uint32_t * counts = s_counts + (threadIdx.x >> 5) * n_counters;
    uint64_t const warp = (blockIdx.y * static_cast<uint64_t>(blockDim.x) + threadIdx.x) >> 5;
    uint64_t const nwarps = (static_cast<uint64_t>(gridDim.y) * blockDim.x) >> 5;
    for (uint64_t start = warp * chunk; start < n; start += nwarps * chunk)
    {
        uint64_t const len = (n - start) < chunk ? (n - start) : chunk;
        warp_count<R, LPV, H, 7, 1, 1, true>(rp, values + start, len, counts, lane);
    }
    __syncthreads();
    finish_counts(s_counts, n_counters, w0, rp.bin_words, totals, tickets + blockIdx.x, reset, bins, width, out);
}

// The same count with one or two hash functions for rows, or slabs of rows, of 9 to 16 words (128-byte pieces) and
// calls that fill the GPU: the pieces go to shared memory by asynchronous copies, three stages of eight values ahead of
// their use, so that reads are in flight all the time and hold no registers; the loop above issues a group, waits for
// it and adds it up.  Eight lanes copy a piece (16 bytes each), 16 lanes add it up (one word each).  8,192 bins, a
// million values, h = 1: 331 -> 229 us; 2,048 bins, h = 2: 133 -> 89; 600 bins, h = 1: 69 -> 53.  With three hash
// functions and more the loop above has enough reads in flight (1,000 bins, h = 3, four million values: 254 us against
// 271 here), so they have no asynchronous form.
constexpr int kAsyncStages = 4;      // stages in the ring of a warp
constexpr int kAsyncValues = 8;      // values per stage
constexpr int kAsyncWarps = 4;       // warps per block
constexpr uint32_t kAsyncWords = 16; // words of a piece

template <int H>
constexpr uint32_t async_ring_words()
{
    return kAsyncStages * kAsyncValues * H * kAsyncWords;
}

template <int H>
constexpr size_t async_smem()
{
    return kAsyncWarps * (async_ring_words<H>() * 8u + 64u * kAsyncWords * 4u);
}

// Blocks per SM: what shared memory holds (228 KiB, 1 KiB of it per block).
template <int H>
constexpr unsigned async_blocks_per_sm()
{
    return static_cast<unsigned>(228u * 1024u / (async_smem<H>() + 1024u));
}

__device__ __forceinline__ void copy_async16(void * smem, void const * global, uint32_t bytes, uint64_t policy)
{
    asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2, %3;" ::"r"(
                     static_cast<uint32_t>(__cvta_generic_to_shared(smem))),
                 "l"(global), "r"(bytes), "l"(policy)
                 : "memory");
}

template <int H, typename R>
__global__ void __launch_bounds__(32 * kAsyncWarps, async_blocks_per_sm<H>())
    k_bulk_count_async(row_params row, uint64_t const * __restrict__ values, uint64_t n, uint64_t chunk,
                       unsigned long long * totals, unsigned int * tickets, bool reset, uint64_t bins, int width,
                       void * __restrict__ out)
{
    constexpr uint32_t n_counters = 64u * kAsyncWords;
    extern __shared__ __align__(16) uint64_t s_ring[];
    uint32_t * const s_counts = reinterpret_cast<uint32_t *>(s_ring + kAsyncWarps * async_ring_words<H>());
    uint32_t const w0 = blockIdx.x * kAsyncWords;
    row_params const rp = row_slab(row, w0, kAsyncWords);
    for (uint32_t i = threadIdx.x; i < n_counters * kAsyncWarps; i += blockDim.x)
        s_counts[i] = 0;
    __syncthreads();
    int const lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t * const counts = s_counts + w * n_counters;
    uint64_t * const ring = s_ring + w * async_ring_words<H>();
    uint64_t policy;
    asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
    // this lane copies 16 bytes (words 2c, 2c + 1) of every fourth piece; words past the row's end arrive as 0
    uint32_t const c = lane & 7;
    uint32_t const bytes = 2u * c + 2u <= rp.bin_words ? 16u : (2u * c + 1u == rp.bin_words ? 8u : 0u);
    uint64_t const * const from = rp.words + (bytes ? 2u * c : 0u);
    int const g = lane >> 4, j = lane & 15;
    uint64_t P[7];
#pragma unroll
    for (int k = 0; k < 7; ++k)
        P[k] = 0;
    int acc = 0;
    uint64_t const warp = blockIdx.y * static_cast<uint64_t>(kAsyncWarps) + w;
    uint64_t const nwarps = static_cast<uint64_t>(gridDim.y) * kAsyncWarps;
    for (uint64_t start = warp * chunk; start < n; start += nwarps * chunk)
    {
        uint64_t const len = min(chunk, n - start);
        uint64_t const * const vals = values + start;
        uint32_t const stages = static_cast<uint32_t>((len + kAsyncValues - 1) / kAsyncValues);
        R r[H];
        uint64_t nv = static_cast<uint64_t>(lane) < len ? __ldcg(vals + lane) : 0u;
        for (uint32_t t = 0; t < stages + kAsyncStages - 1u; ++t)
        {
            if (t < stages)
            {
                if (t % (32 / kAsyncValues) == 0) // the next 32 values, one per lane
                {
#pragma unroll
                    for (int k = 0; k < H; ++k)
                        r[k] = hash_row_as<R>(nv, c_hash_seeds[k], rp.hash_shift, rp.bin_size);
                    uint64_t const ahead = static_cast<uint64_t>(t) * kAsyncValues + 32u + lane;
                    nv = ahead < len ? __ldcg(vals + ahead) : 0u;
                }
                uint64_t * const stage = ring + (t % kAsyncStages) * (kAsyncValues * H * kAsyncWords);
#pragma unroll
                for (int k = 0; k < H; ++k)
#pragma unroll
                    for (int half = 0; half < 2; ++half)
                    {
                        int const v = 4 * half + (lane >> 3); // value of the stage
                        R const rv = __shfl_sync(kFullMask, r[k],
                                                 (t % (32 / kAsyncValues)) * kAsyncValues + static_cast<uint32_t>(v));
                        bool const there = static_cast<uint64_t>(t) * kAsyncValues + static_cast<uint32_t>(v) < len;
                        copy_async16(stage + (k * kAsyncValues + v) * kAsyncWords + 2u * c,
                                     from + static_cast<uint64_t>(rv) * rp.row_words, there ? bytes : 0u, policy);
                    }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            if (t + 1u < kAsyncStages)
                continue;
            asm volatile("cp.async.wait_group %0;" ::"n"(kAsyncStages - 1) : "memory");
            __syncwarp(); // the other lanes' copies of this stage
            uint64_t const * const stage =
                ring + ((t + 1u) % kAsyncStages) * (kAsyncValues * H * kAsyncWords); // stage t + 1 - kAsyncStages
            uint64_t m[4];
#pragma unroll
            for (int q = 0; q < 4; ++q)
            {
                uint64_t x = stage[(2 * q + g) * kAsyncWords + j];
#pragma unroll
                for (int k = 1; k < H; ++k)
                    x &= stage[(k * kAsyncValues + 2 * q + g) * kAsyncWords + j];
                m[q] = x;
            }
            __syncwarp(); // read by every lane before it is refilled
            planes_add4<7>(P, m[0], m[1], m[2], m[3]);
            acc += 4;
            if (acc > 127 - 4)
            {
                planes_flush_to<16, 7>(P, counts, lane, acc, rp.bin_words);
                acc = 0;
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncwarp();
    }
    if (acc)
        planes_flush_to<16, 7>(P, counts, lane, acc, rp.bin_words);
    __syncthreads();
    finish_counts(s_counts, n_counters, w0, rp.bin_words, totals, tickets + blockIdx.x, reset, bins, width, out);
}

using bulk_count_kernel_t = void (*)(row_params, uint64_t const *, uint64_t, uint64_t, unsigned long long *,
                                     unsigned int *, bool, uint64_t, int, void *);

template <int H, typename R>
bulk_count_kernel_t bulk_count_kernel_h(uint32_t lpv_log2)
{
    switch (lpv_log2)
    {
    case 0:
        return k_bulk_count<1, H, R>;
    case 1:
        return k_bulk_count<2, H, R>;
    case 2:
        return k_bulk_count<4, H, R>;
    case 3:
        return k_bulk_count<8, H, R>;
    case 4:
        return k_bulk_count<16, H, R>;
    default:
        return k_bulk_count<32, H, R>;
    }
}

template <typename R>
bulk_count_kernel_t bulk_count_kernel(uint64_t h, uint32_t lpv_log2)
{
    switch (h)
    {
    case 1:
        return bulk_count_kernel_h<1, R>(lpv_log2);
    case 2:
        return bulk_count_kernel_h<2, R>(lpv_log2);
    case 3:
        return bulk_count_kernel_h<3, R>(lpv_log2);
    case 4:
        return bulk_count_kernel_h<4, R>(lpv_log2);
    default:
        return bulk_count_kernel_h<5, R>(lpv_log2);
    }
}

// The asynchronous kernel of h hash functions, its shared memory and its blocks per SM.
struct async_count
{
    bulk_count_kernel_t kernel;
    size_t smem;
    unsigned blocks_per_sm;
};

template <int H>
async_count async_count_h(bool wide)
{
    return async_count{wide ? k_bulk_count_async<H, uint64_t> : k_bulk_count_async<H, uint32_t>, async_smem<H>(),
                       async_blocks_per_sm<H>()};
}

// Whether a call of n values over `slabs` pieces per row is large enough for the asynchronous kernel: its warps then
// have some 100 values each.  (1,000 bins, h = 2: 100,000 values 25 us against 26, 300,000 34 against 33; 2,048 bins,
// 100,000 values 31 against 27; 8,192 bins, h = 1, 10,000 values 22.3 against 21.7, 30,000 30 against 26.)
bool async_count_pays(uint64_t h, uint64_t bin_words, uint64_t n, uint32_t slabs)
{
    return h <= 2 && bin_words > kAsyncWords / 2 && n * slabs >= 200000;
}

int sm_count()
{
    static int n = []
    {
        int dev = 0, c = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&c, cudaDevAttrMultiProcessorCount, dev) !=
                                                      cudaSuccess)
            return 132;
        return c;
    }();
    return n;
}

inline unsigned grid_for(uint64_t work, unsigned block)
{
    uint64_t const want = (work + block - 1) / block;
    uint64_t const cap = static_cast<uint64_t>(sm_count()) * 16u;
    return static_cast<unsigned>(std::max<uint64_t>(1, std::min(want, cap)));
}

} // namespace hibf_gb300

using namespace hibf_gb300;

// -----------------------------------------------------------------------------------------------------------------
// Object
// -----------------------------------------------------------------------------------------------------------------
// The tables of inserts with exact occupancy, up to 122 MB each: an allocation and its release take longer than the
// insert, so the filters of a device share what is kept, which is given back with the last of them.  Every call has a
// buffer of its own while it runs; two are kept.  (With one kept by every filter a thousand filters held 122 GB.)
class scratch_pool
{
public:
    std::unique_ptr<dbuf> take(size_t bytes)
    {
        std::unique_ptr<dbuf> buf;
        {
            std::lock_guard<std::mutex> lk(mu_);
            auto better = [bytes](size_t x, size_t y) // the smallest that is large enough, else the largest
            {
                if ((x >= bytes) != (y >= bytes))
                    return x >= bytes;
                return x >= bytes ? x < y : x > y;
            };
            auto best = kept_.begin();
            for (auto it = kept_.begin(); it != kept_.end(); ++it)
                if (better((*it)->bytes, (*best)->bytes))
                    best = it;
            if (best != kept_.end())
            {
                buf = std::move(*best);
                kept_.erase(best);
            }
        }
        if (!buf)
            buf = std::make_unique<dbuf>();
        buf->ensure(bytes);
        return buf;
    }
    void give(std::unique_ptr<dbuf> buf) // nothing on the device uses it any more
    {
        std::lock_guard<std::mutex> lk(mu_);
        if (kept_.size() < 2)
            kept_.push_back(std::move(buf));
    }
    // The current device's.
    static std::shared_ptr<scratch_pool> of_device()
    {
        static std::mutex mu;
        static std::map<int, std::weak_ptr<scratch_pool>> pools;
        int dev = 0;
        HG_CUDA(cudaGetDevice(&dev));
        std::lock_guard<std::mutex> lk(mu);
        std::shared_ptr<scratch_pool> p = pools[dev].lock();
        if (!p)
            pools[dev] = p = std::make_shared<scratch_pool>();
        return p;
    }

private:
    std::mutex mu_;
    std::vector<std::unique_ptr<dbuf>> kept_;
};

// Calls on one stream run one after the other and may share their scratch; those on other streams may run at the same
// time and have another one.
struct count_scratch
{
    unsigned long long stream{}; // the stream's number, which no later stream gets
    dbuf buf;
};
constexpr uint32_t kCountStreams = 16;

struct hibf_gpu_ibf
{
    uint64_t bins{};
    uint64_t bin_size{};
    uint64_t hash_funs{};
    uint64_t bin_words{};
    uint64_t row_words{};
    uint32_t shift{};
    bool track_occupancy{};
    dbuf store;     // bin_size * row_words words
    dbuf occupancy; // technical_bins counters
    // bulk_count's scratch, technical_bins 64-bit totals and a ticket per slab: device-pointer calls clear theirs,
    // host-pointer calls, one at a time, leave host_totals at 0
    std::mutex count_mu;
    count_scratch totals[kCountStreams];
    uint32_t n_totals{};
    dbuf captured_totals; // of calls in a stream capture
    dbuf host_totals;
    hbuf h_in, h_out; // small host-pointer calls: values the kernels read in place, results they write
    dbuf io;        // staging for host-pointer calls
    dbuf io2;
    std::mutex occ_mu; // one insert with exact occupancy at a time
    std::shared_ptr<scratch_pool> occ_pool;
    dbuf flag; // device int: an emplace saw a bin index out of range
    cudaStream_t stream{};
    int status{HIBF_GPU_OK};
    std::mutex mu;

    row_params rp() const
    {
        return row_params{store.as<uint64_t>(), bin_size, static_cast<uint32_t>(row_words),
                          static_cast<uint32_t>(bin_words), shift};
    }
    bool wide_rows() const // the kernels take 64-bit row indices
    {
        return bin_size > UINT32_MAX;
    }
    // Lanes (log2) that read a row, or a slab of a row, for n values.  Rows of up to 16 words are read whole.  Wider
    // ones are counted in slabs of 16 words: with 32, whose counters leave room for three blocks per SM, 8,192 bins (h
    // = 1, a million values) took 421 us against 336, 3,000 values 24 against 18.  Only long calls on rows of 17 to 31
    // words take one slab of 32 (1,500 bins, h = 4, 300,000 values: 64 us against 71).
    uint32_t count_lanes_log2(uint64_t n) const
    {
        if (bin_words <= 16)
            return lanes_log2(static_cast<uint32_t>(bin_words));
        return bin_words < kSlabWords && n > (1u << 17) ? 5 : 4;
    }
    // bulk_contains keeps no counters, so long calls read slabs of 32 words where those leave at most half a slab idle
    // at the row's end (2,048 bins, h = 2, a million values: 119 us against 123 with slabs of 16; 3,000 values 10.3
    // against 8.4; 2,500 bins, 40 words, 238 us with slabs of 16 and 251 with 32).
    uint32_t contains_lanes_log2(uint64_t n) const
    {
        if (bin_words <= 16)
            return lanes_log2(static_cast<uint32_t>(bin_words));
        uint64_t const rest = bin_words % kSlabWords;
        return n > (1u << 16) && (rest == 0 || rest > kSlabWords / 2) ? 5 : 4;
    }
    uint32_t slabs(uint32_t lanes_log2) const
    {
        return static_cast<uint32_t>((bin_words + (1u << lanes_log2) - 1) >> lanes_log2);
    }
    uint64_t technical_bins() const
    {
        return bin_words * 64u;
    }
};

namespace
{

cudaStream_t pick(hibf_gpu_ibf * f, void * s)
{
    return s ? static_cast<cudaStream_t>(s) : f->stream;
}

// Occupancy in insertion order and the bits, chunk by chunk; chunks run one after the other, so each sees the bits of
// the chunks before it.  SYNTH: the n values are the generated values of bin `bin` (vpb per bin).  Calls on several
// streams take turns.
template <bool SYNTH>
void emplace_exact(hibf_gpu_ibf * f, uint64_t const * d_values, uint64_t const * d_bins, uint64_t n, uint64_t bin,
                   uint64_t seed, uint64_t vpb, cudaStream_t s)
{
    constexpr uint64_t kChunk = 1u << 20;
    unsigned const block = 256;
    uint32_t const h = static_cast<uint32_t>(f->hash_funs);
    uint64_t const m_max = std::min(n, kChunk) * h;
    uint64_t slots = 1024;
    while (slots < m_max + m_max / 2)
        slots *= 2;
    std::lock_guard<std::mutex> lk(f->occ_mu);
    if (!f->occ_pool)
        f->occ_pool = scratch_pool::of_device();
    std::unique_ptr<dbuf> scratch = f->occ_pool->take(slots * 12 + m_max * 4);
    auto * const keys = scratch->as<unsigned long long>();
    auto * const lowest = reinterpret_cast<unsigned int *>(keys + slots);
    auto * const entries = lowest + slots;
    uint32_t const rw = static_cast<uint32_t>(f->row_words);
    for (uint64_t c0 = 0; c0 < n; c0 += kChunk)
    {
        uint64_t const c = std::min(kChunk, n - c0);
        uint64_t const * vals = SYNTH ? nullptr : d_values + c0;
        uint64_t const * bins = (SYNTH || !d_bins) ? nullptr : d_bins + c0;
        HG_CUDA(cudaMemsetAsync(keys, 0xFF, slots * 12, s)); // free entries, no value yet
        k_occ_enter<SYNTH><<<grid_for(c, block), block, 0, s>>>(
            f->store.as<uint64_t>(), f->bin_size, rw, f->shift, h, vals, bins, seed, vpb, c0, c, bin, f->bins,
            f->technical_bins(), keys, lowest, static_cast<uint32_t>(slots - 1), entries);
        HG_CUDA(cudaGetLastError());
        k_occ_insert<SYNTH><<<grid_for(c, block), block, 0, s>>>(
            f->store.as<uint64_t>(), f->bin_size, rw, f->shift, h, vals, bins, seed, vpb, c0, c, bin, f->bins, lowest,
            entries, f->occupancy.as<unsigned long long>(), f->flag.as<int>());
        HG_CUDA(cudaGetLastError());
    }
    HG_CUDA(cudaStreamSynchronize(s));
    f->occ_pool->give(std::move(scratch));
}

void launch_emplace(hibf_gpu_ibf * f, uint64_t const * d_values, uint64_t const * d_bins, uint64_t n, uint64_t bin,
                    cudaStream_t s)
{
    if (n == 0)
        return;
    if (f->track_occupancy)
    {
        emplace_exact<false>(f, d_values, d_bins, n, bin, 0, 1, s);
        return;
    }
    unsigned const block = 256;
    k_emplace<<<grid_for(n, block), block, 0, s>>>(f->store.as<uint64_t>(), f->bin_size,
                                                   static_cast<uint32_t>(f->row_words), f->shift,
                                                   static_cast<uint32_t>(f->hash_funs), d_values, d_bins, n, bin,
                                                   f->bins, f->flag.as<int>());
    HG_CUDA(cudaGetLastError());
}

// Per-bin counters bulk_count accumulates for filter f (a multiple of 64, at least its technical bins).
uint64_t count_counters(hibf_gpu_ibf const * f)
{
    return row_counters(static_cast<uint32_t>(f->bin_words));
}

// Bytes of bulk_count's scratch for filter f: its totals and a ticket per slab (of 16 words, the narrowest).
uint64_t count_scratch_bytes(hibf_gpu_ibf const * f)
{
    return count_counters(f) * sizeof(unsigned long long) + f->slabs(4) * sizeof(unsigned int);
}

// The scratch of a call on stream s; the caller holds f->count_mu until the call is in the stream.  The first
// kCountStreams streams have one each, calls on others take and return it in the stream's order (`taken`).  A captured
// call runs on the stream its graph is launched on, so captured calls have one for themselves, which the first call
// outside a capture allocates (nothing can be allocated within one); graphs that hold counts on one filter must not
// overlap.
struct taken_scratch
{
    void * p{};
    cudaStream_t s{};
    ~taken_scratch()
    {
        if (p)
            cudaFreeAsync(p, s);
    }
};
unsigned long long * stream_scratch(hibf_gpu_ibf * f, cudaStream_t s, taken_scratch & taken)
{
    size_t const bytes = count_scratch_bytes(f);
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    HG_CUDA(cudaStreamIsCapturing(s, &capture));
    f->captured_totals.ensure(bytes);
    if (capture != cudaStreamCaptureStatusNone)
        return f->captured_totals.as<unsigned long long>();
    unsigned long long id = 0;
    HG_CUDA(cudaStreamGetId(s, &id));
    uint32_t k = 0;
    while (k < f->n_totals && f->totals[k].stream != id)
        ++k;
    if (k == kCountStreams)
    {
        taken.s = s;
        HG_CUDA(cudaMallocAsync(&taken.p, bytes, s));
        return static_cast<unsigned long long *>(taken.p);
    }
    f->totals[k].buf.ensure(bytes);
    if (k == f->n_totals)
    {
        f->totals[k].stream = id;
        ++f->n_totals;
    }
    return f->totals[k].buf.as<unsigned long long>();
}

// bulk_count of n values into `out` (device memory, or mapped host memory).  `totals` is device scratch of
// count_scratch_bytes(f); null means the stream's (grown on demand, the only allocation here).  `reset`: it is at 0 and
// is left at 0.
void launch_count(hibf_gpu_ibf * f, uint64_t const * values, uint64_t n, int width, void * out, cudaStream_t s,
                  unsigned long long * totals = nullptr, bool reset = false)
{
    if (!n)
    {
        HG_CUDA(cudaMemsetAsync(out, 0, f->bins * static_cast<uint64_t>(width), s));
        return;
    }
    std::unique_lock<std::mutex> lk(f->count_mu, std::defer_lock);
    taken_scratch taken;
    if (!totals)
    {
        lk.lock();
        totals = stream_scratch(f, s, taken);
    }
    auto * const tickets = reinterpret_cast<unsigned int *>(totals + count_counters(f));
    if (uint32_t const slabs = f->slabs(4); async_count_pays(f->hash_funs, f->bin_words, n, slabs))
    {
        async_count const a = f->hash_funs == 1 ? async_count_h<1>(f->wide_rows()) : async_count_h<2>(f->wide_rows());
        uint64_t const blocks = std::max<uint64_t>(1, static_cast<uint64_t>(sm_count()) * a.blocks_per_sm / slabs);
        uint64_t const warps = blocks * kAsyncWarps;
        uint64_t const chunk = ((n + warps - 1) / warps + kAsyncValues - 1) / kAsyncValues * kAsyncValues;
        unsigned const grid =
            static_cast<unsigned>(((n + chunk - 1) / chunk + kAsyncWarps - 1) / kAsyncWarps);
        if (grid > 1 && !reset)
            HG_CUDA(cudaMemsetAsync(totals, 0, count_scratch_bytes(f), s));
        HG_CUDA(cudaFuncSetAttribute(a.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(a.smem)));
        a.kernel<<<dim3(slabs, grid), 32 * kAsyncWarps, a.smem, s>>>(f->rp(), values, n, chunk, totals, tickets, reset,
                                                                    f->bins, width, out);
        HG_CUDA(cudaGetLastError());
        return;
    }
    unsigned const block = 256;
    // One contiguous chunk per warp of a full wave, over all slabs: as many blocks of 8 warps per SM as the kernel is
    // built for, or the 3 whose 64 KiB of counters fit where a slab is 32 words.  A chunk is at least 32 values, one
    // per lane: a call of 250 values then runs on eight warps of one block instead of one warp, one of 10,000 on 40 SMs
    // (with chunks of 512: 1,000 bins, h = 3, 10,000 values 92 us, now 18).  From 128 values on, narrow rows round it
    // to whole passes of four values per lane.
    uint32_t const lanes = f->count_lanes_log2(n);
    uint32_t const slabs = f->slabs(lanes);
    bool const full_slabs = lanes == 5;
    uint64_t const per_sm = full_slabs ? 3u : count_blocks_per_sm(static_cast<int>(f->hash_funs));
    uint64_t const blocks = std::max<uint64_t>(1, static_cast<uint64_t>(sm_count()) * per_sm / slabs);
    uint64_t const wave = blocks * 8u;
    uint64_t const even = (n + wave - 1) / wave;
    uint64_t const round = full_slabs || even <= 96 ? 32 : 128;
    uint64_t const chunk = (even + round - 1) / round * round;
    uint64_t const warps = (n + chunk - 1) / chunk;
    unsigned const grid = static_cast<unsigned>(std::max<uint64_t>(1, std::min<uint64_t>((warps + 7) / 8, blocks)));
    if (grid > 1 && !reset)
        HG_CUDA(cudaMemsetAsync(totals, 0, count_scratch_bytes(f), s));
    size_t const smem = (64u << lanes) * sizeof(uint32_t) * (block / 32);
    bulk_count_kernel_t const kernel = f->wide_rows() ? bulk_count_kernel<uint64_t>(f->hash_funs, lanes)
                                                      : bulk_count_kernel<uint32_t>(f->hash_funs, lanes);
    if (smem > 48 * 1024)
        HG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    kernel<<<dim3(slabs, grid), block, smem, s>>>(f->rp(), values, n, chunk, totals, tickets, reset, f->bins, width,
                                                  out);
    HG_CUDA(cudaGetLastError());
}

void launch_contains(hibf_gpu_ibf * f, uint64_t const * d_values, uint64_t n, uint64_t * d_out, cudaStream_t s)
{
    if (n == 0)
        return;
    uint32_t const lanes = f->contains_lanes_log2(n);
    uint32_t const slabs = f->slabs(lanes);
    // Slabs of 16 words: 8 values per warp where 32 would leave the GPU's warps mostly idle, up to one wave of warps
    // (8,192 bins, h = 3: 2,000 values 9.2 -> 5.2 us, 7,000 values 10.4 -> 9.4, 30,000 values 21.2 -> 22.7).
    uint64_t const wave = static_cast<uint64_t>(sm_count()) * 64u;
    bool const few = slabs > 1 && lanes == 4 && (n + 7) / 8 * slabs <= wave;
    contains_kernel_t const kernel = f->wide_rows() ? contains_kernel<uint64_t>(f->hash_funs, lanes, few)
                                                    : contains_kernel<uint32_t>(f->hash_funs, lanes, few);
    kernel<<<dim3(slabs, grid_for(few ? n * 4 : n, 256)), 256, 0, s>>>(f->rp(), d_values, n, d_out);
    HG_CUDA(cudaGetLastError());
}

constexpr uint64_t kDeviceCheck = 1u << 14; // host-pointer inserts of as many values check their bins on the device
constexpr uint64_t kSmallBytes = 64u << 10; // host-pointer calls of up to this many bytes in and out need no copies

// bulk_count of host values, finished on return: the counts in page-locked memory of the filter, valid until its next
// host-pointer call (the caller holds f->mu).  Few values are read in place by the kernel, others are copied; the
// kernel writes the counts to the host.
void const * count_host(hibf_gpu_ibf * f, uint64_t const * values, uint64_t n, int width)
{
    if (!f->host_totals.p || f->host_totals.bytes < count_scratch_bytes(f))
    {
        f->host_totals.ensure(count_scratch_bytes(f));
        HG_CUDA(cudaMemsetAsync(f->host_totals.p, 0, f->host_totals.bytes, f->stream));
    }
    f->h_out.ensure(std::max<uint64_t>(f->bins * static_cast<uint64_t>(width), kSmallBytes));
    if (!n)
    {
        std::memset(f->h_out.p, 0, f->bins * static_cast<uint64_t>(width));
        return f->h_out.p;
    }
    uint64_t const * in = nullptr;
    if (n * 8 <= kSmallBytes)
    {
        f->h_in.ensure(kSmallBytes);
        std::memcpy(f->h_in.p, values, n * 8);
        in = f->h_in.as<uint64_t>();
    }
    else
    {
        f->io.ensure(n * 8);
        HG_CUDA(cudaMemcpyAsync(f->io.p, values, n * 8, cudaMemcpyHostToDevice, f->stream));
        in = f->io.as<uint64_t>();
    }
    launch_count(f, in, n, width, f->h_out.p, f->stream, f->host_totals.as<unsigned long long>(), true);
    HG_CUDA(cudaStreamSynchronize(f->stream));
    return f->h_out.p;
}

int width_ok(int width)
{
    return width == 1 || width == 2 || width == 4 || width == 8;
}

// ---------------------------------------------------------------------------------------------------------------
// bulk_count without allocation.  The 64-bit per-bin totals that bulk_count accumulates live in this fixed array
// instead of a cudaMalloc'd buffer.  Every device that loads the library holds it (128 KiB) until the process exits.
// ---------------------------------------------------------------------------------------------------------------
constexpr uint64_t kNoAllocMaxCounters = HIBF_GPU_NOALLOC_MAX_BINS;
// (and a 32-bit ticket per slab of at least 16 words)
constexpr uint64_t kNoAllocTickets = kNoAllocMaxCounters / (64u * 16u);
static __device__ __align__(256) unsigned long long g_noalloc_totals[kNoAllocMaxCounters + (kNoAllocTickets + 1) / 2];

// Device address of g_noalloc_totals per device.  In host code the array's name is only a host-side stand-in, so
// the address is looked up once per device (cudaGetSymbolAddress, with that device current) and cached.
constexpr int kMaxDevices = 256;
std::mutex g_noalloc_mu;
unsigned long long * g_noalloc_addr[kMaxDevices] = {};

unsigned long long * noalloc_totals()
{
    int dev = 0;
    HG_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices)
        fail(HIBF_GPU_ERR_INVALID_ARG, "device ordinal out of range");
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (!g_noalloc_addr[dev])
    {
        void * p = nullptr;
        HG_CUDA(cudaGetSymbolAddress(&p, g_noalloc_totals));
        g_noalloc_addr[dev] = static_cast<unsigned long long *>(p);
    }
    return g_noalloc_addr[dev];
}

} // namespace

extern "C"
{

    char const * hibf_gpu_last_error(void)
    {
        return g_last_error.c_str();
    }

    int hibf_gpu_abi_version(void)
    {
        return HIBF_GPU_ABI_VERSION;
    }

    int hibf_gpu_device_count(int * count)
    {
        return guarded(
            [&]
            {
                int n = 0;
                cudaError_t e = cudaGetDeviceCount(&n);
                if (e != cudaSuccess)
                {
                    (void)cudaGetLastError();
                    n = 0;
                }
                if (count)
                    *count = n;
            });
    }

    int hibf_gpu_ibf_create(uint64_t bins, uint64_t bin_size, uint64_t hash_funs, int track_occupancy,
                            hibf_gpu_ibf ** out)
    {
        return guarded(
            [&]
            {
                if (!out)
                    fail(HIBF_GPU_ERR_INVALID_ARG, "out is null");
                *out = nullptr;
                if (bins == 0)
                    fail(HIBF_GPU_ERR_LOGIC, "The number of bins must be > 0.");
                if (hash_funs == 0 || hash_funs > 5)
                    fail(HIBF_GPU_ERR_LOGIC, "The number of hash functions must be > 0 and <= 5.");
                if (bin_size == 0)
                    fail(HIBF_GPU_ERR_LOGIC, "The size of a bin must be > 0.");
                require_device();
                auto f = new hibf_gpu_ibf{};
                try
                {
                    f->bins = bins;
                    f->bin_size = bin_size;
                    f->hash_funs = hash_funs;
                    f->bin_words = (bins + 63u) / 64u;
                    f->row_words = padded_row_words(f->bin_words);
                    f->shift = static_cast<uint32_t>(__builtin_clzll(bin_size));
                    f->track_occupancy = track_occupancy != 0;
                    HG_CUDA(cudaStreamCreateWithFlags(&f->stream, cudaStreamNonBlocking));
                    size_t const bytes = bin_size * f->row_words * sizeof(uint64_t);
                    f->store.ensure(bytes);
                    HG_CUDA(cudaMemsetAsync(f->store.p, 0, bytes, f->stream));
                    f->flag.ensure(sizeof(int));
                    HG_CUDA(cudaMemsetAsync(f->flag.p, 0, sizeof(int), f->stream));
                    f->occupancy.ensure(f->technical_bins() * sizeof(uint64_t));
                    HG_CUDA(cudaMemsetAsync(f->occupancy.p, 0, f->technical_bins() * sizeof(uint64_t), f->stream));
                    HG_CUDA(cudaStreamSynchronize(f->stream));
                }
                catch (...)
                {
                    if (f->stream)
                        cudaStreamDestroy(f->stream);
                    delete f;
                    throw;
                }
                *out = f;
            });
    }

    int hibf_gpu_ibf_destroy(hibf_gpu_ibf * f)
    {
        return guarded(
            [&]
            {
                if (!f)
                    return;
                cudaStreamSynchronize(f->stream);
                cudaStreamDestroy(f->stream);
                delete f;
            });
    }

    int hibf_gpu_ibf_info(hibf_gpu_ibf const * f, uint64_t out[5])
    {
        return guarded(
            [&]
            {
                if (!f || !out)
                    fail(HIBF_GPU_ERR_INVALID_ARG, "null argument");
                out[0] = f->bins;
                out[1] = f->bin_size;
                out[2] = f->hash_funs;
                out[3] = f->bin_words * 64u * f->bin_size;
                out[4] = f->row_words * 8u;
            });
    }

    int hibf_gpu_ibf_emplace_d(hibf_gpu_ibf * f, uint64_t const * d_values, uint64_t const * d_bins, uint64_t n,
                               uint64_t bin, void * stream)
    {
        return guarded(
            [&]
            {
                if (!f || (n && !d_values))
                    fail(HIBF_GPU_ERR_INVALID_ARG, "null argument");
                if (!d_bins && bin >= f->bins)
                    fail(HIBF_GPU_ERR_INVALID_ARG, "bin index out of range");
                launch_emplace(f, d_values, d_bins, n, bin, pick(f, stream));
            });
    }

    int hibf_gpu_synth_ibf_emplace(hibf_gpu_ibf * f, uint64_t seed, uint64_t values_per_bin, uint64_t first_bin,
                                   uint64_t n_bins, void * stream)
    {
        return guarded(
            [&]
            {
                if (!f || values_per_bin == 0)
                    fail(HIBF_GPU_ERR_INVALID_ARG, "bad argument");
                if (first_bin > f->bins || n_bins > f->bins - first_bin)
                    fail(HIBF_GPU_ERR_INVALID_ARG, "bin range out of range");
                if (n_bins && values_per_bin > UINT64_MAX / n_bins)
                    fail(HIBF_GPU_ERR_INVALID_ARG, "too many values");
                uint64_t const n = n_bins * values_per_bin;
                if (!n)
                    return;
                if (f->track_occupancy)
                {
                    for (uint64_t b = first_bin; b < first_bin + n_bins; ++b)
                        emplace_exact<true>(f, nullptr, nullptr, values_per_bin, b, seed, values_per_bin,
                                            pick(f, stream));
                    return;
                }
                unsigned const block = 256;
                k_synth_emplace<<<grid_for(n, block), block, 0, pick(f, stream)>>>(
                    f->store.as<uint64_t>(), f->bin_size, static_cast<uint32_t>(f->row_words), f->shift,
                    static_cast<uint32_t>(f->hash_funs), seed, values_per_bin, first_bin, n);
                HG_CUDA(cudaGetLastError());
            });
    }

    int hibf_gpu_ibf_emplace(hibf_gpu_ibf * f, uint64_t const * values, uint64_t n, uint64_t bin)
    {
        return guarded(
            [&]
            {
                if (!f || (n && !values))
                    fail(HIBF_GPU_ERR_INVALID_ARG, "null argument");
                if (bin >= f->bins)
                    fail(HIBF_GPU_ERR_INVALID_ARG, "bin index out of range");
                std::lock_guard<std::mutex> lk(f->mu);
                f->io.ensure(n * 8);
                HG_CUDA(cudaMemcpyAsync(f->io.p, values, n * 8, cudaMemcpyHostToDevice, f->stream));
                launch_emplace(f, f->io.as<uint64_t>(), nullptr, n, bin, f->stream);
                HG_CUDA(cudaStreamSynchronize(f->stream));
            });
    }

    int hibf_gpu_ibf_emplace_binned(hibf_gpu_ibf * f, uint64_t const * values, uint64_t const * bins, uint64_t n)
    {
        return guarded(
            [&]
            {
                if (!f || (n && (!values || !bins)))
                    fail(HIBF_GPU_ERR_INVALID_ARG, "null argument");
                // Nothing is inserted if any bin is out of range.  Many bins are checked on the device, beside the copy
                // of the values (the host reads 530,624 of them in 0.2 ms, about as long as everything else takes).
                bool const on_device = n >= kDeviceCheck;
                for (uint64_t i = 0; i < n && !on_device; ++i)
                    if (bins[i] >= f->bins)
                        fail(HIBF_GPU_ERR_INVALID_ARG, "bin index out of range");
                std::lock_guard<std::mutex> lk(f->mu);
                f->io.ensure(n * 8);
                f->io2.ensure(n * 8);
                HG_CUDA(cudaMemcpyAsync(f->io2.p, bins, n * 8, cudaMemcpyHostToDevice, f->stream));
                if (on_device)
                {
                    f->h_out.ensure(kSmallBytes);
                    *f->h_out.as<int>() = 0;
                    k_check_bins<<<grid_for(n, 256), 256, 0, f->stream>>>(f->io2.as<uint64_t>(), n, f->bins,
                                                                          f->h_out.as<int>());
                    HG_CUDA(cudaGetLastError());
                }
                HG_CUDA(cudaMemcpyAsync(f->io.p, values, n * 8, cudaMemcpyHostToDevice, f->stream));
                if (on_device)
                {
                    HG_CUDA(cudaStreamSynchronize(f->stream));
                    if (*static_cast<int volatile const *>(f->h_out.p))
                        fail(HIBF_GPU_ERR_INVALID_ARG, "bin index out of range");
                }
                launch_emplace(f, f->io.as<uint64_t>(), f->io2.as<uint64_t>(), n, 0, f->stream);
                HG_CUDA(cudaStreamSynchronize(f->stream));
            });
    }

    int hibf_gpu_ibf_clear(hibf_gpu_ibf * f, uint64_t bin)
    {
        return guarded(
            [&]
            {
                if (!f)
                    fail(HIBF_GPU_ERR_INVALID_ARG, "null argument");
                if (bin >= f->bins)
                    fail(HIBF_GPU_ERR_INVALID_ARG, "bin index out of range");
                std::lock_guard<std::mutex> lk(f->mu);
                k_clear_bin<<<grid_for(f->bin_size, 256), 256, 0, f->stream>>>(
                    f->store.as<uint64_t>(), f->bin_size, static_cast<uint32_t>(f->row_words), bin >> 6,
                    ~(1ull << (bin & 63u)));
                HG_CUDA(cudaGetLastError());
                HG_CUDA(cudaMemsetAsync(f->occupancy.as<uint64_t>() + bin, 0, sizeof(uint64_t), f->stream));
                HG_CUDA(cudaStreamSynchronize(f->stream));
            });
    }

    int hibf_gpu_ibf_clear_range(hibf_gpu_ibf * f, uint64_t const * bins, uint64_t n)
    {
        return guarded(
            [&]
            {
                if (!f || (n && !bins))
                    fail(HIBF_GPU_ERR_INVALID_ARG, "null argument");
                std::vector<uint64_t> masks(f->bin_words, 0);
                for (uint64_t i = 0; i < n; ++i)
                {
                    if (bins[i] >= f->technical_bins())
                        fail(HIBF_GPU_ERR_INVALID_ARG, "bin index out of range");
                    masks[bins[i] >> 6] |= 1ull << (bins[i] & 63u);
                }
                std::vector<uint32_t> widx;
                std::vector<uint64_t> keep;
                for (uint64_t w = 0; w < f->bin_words; ++w)
                    if (masks[w])
                    {
                        widx.push_back(static_cast<uint32_t>(w));
                        keep.push_back(~masks[w]);
                    }
                if (widx.empty())
                    return;
                std::lock_guard<std::mutex> lk(f->mu);
                f->io.ensure(widx.size() * 4);
                f->io2.ensure(keep.size() * 8);
                HG_CUDA(cudaMemcpyAsync(f->io.p, widx.data(), widx.size() * 4, cudaMemcpyHostToDevice, f->stream));
                HG_CUDA(cudaMemcpyAsync(f->io2.p, keep.data(), keep.size() * 8, cudaMemcpyHostToDevice, f->stream));
                uint32_t const nw = static_cast<uint32_t>(widx.size());
                k_clear_words<<<grid_for(f->bin_size * nw, 256), 256, 0, f->stream>>>(
                    f->store.as<uint64_t>(), f->bin_size, static_cast<uint32_t>(f->row_words), f->io.as<uint32_t>(),
                    f->io2.as<uint64_t>(), nw);
                HG_CUDA(cudaGetLastError());
                HG_CUDA(cudaStreamSynchronize(f->stream));
            });
    }

    int hibf_gpu_ibf_try_increase_bin_number_to(hibf_gpu_ibf * f, uint64_t new_bins, int * increased)
    {
        return guarded(
            [&]
            {
                if (!f || !increased)
                    fail(HIBF_GPU_ERR_INVALID_ARG, "null argument");
                uint64_t const nbw = (new_bins + 63u) / 64u;
                *increased = 0;
                if (new_bins < f->bins || nbw > f->bin_words)
                    return;
                f->bins = new_bins;
                *increased = 1;
            });
    }

    int hibf_gpu_ibf_increase_bin_number_to(hibf_gpu_ibf * f, uint64_t new_bins)
    {
        return guarded(
            [&]
            {
                if (!f)
                    fail(HIBF_GPU_ERR_INVALID_ARG, "null argument");
                if (new_bins < f->bins)
                    fail(HIBF_GPU_ERR_INVALID_ARG, "The number of new bins must be >= the current number of bins.");
                uint64_t const nbw = (new_bins + 63u) / 64u;
                if (nbw <= f->bin_words)
                {
                    f->bins = new_bins;
                    return;
                }
                std::lock_guard<std::mutex> lk(f->mu);
                uint64_t const nrw = padded_row_words(nbw);
                dbuf fresh;
                fresh.ensure(f->bin_size * nrw * 8);
                k_widen<<<grid_for(f->bin_size * nrw, 256), 256, 0, f->stream>>>(
                    fresh.as<uint64_t>(), static_cast<uint32_t>(nrw), f->store.as<uint64_t>(),
                    static_cast<uint32_t>(f->row_words), static_cast<uint32_t>(f->bin_words), f->bin_size);
                HG_CUDA(cudaGetLastError());
                dbuf occ;
                occ.ensure(nbw * 64 * 8);
                HG_CUDA(cudaMemsetAsync(occ.p, 0, nbw * 64 * 8, f->stream));
                HG_CUDA(cudaMemcpyAsync(occ.p, f->occupancy.p, f->technical_bins() * 8, cudaMemcpyDeviceToDevice,
                                        f->stream));
                HG_CUDA(cudaStreamSynchronize(f->stream));
                std::swap(f->store.p, fresh.p);
                std::swap(f->store.bytes, fresh.bytes);
                std::swap(f->occupancy.p, occ.p);
                std::swap(f->occupancy.bytes, occ.bytes);
                f->bins = new_bins;
                f->bin_words = nbw;
                f->row_words = nrw;
            });
    }

    int hibf_gpu_ibf_bulk_contains_d(hibf_gpu_ibf * f, uint64_t const * d_values, uint64_t n, uint64_t * d_out,
                                     void * stream)
    {
        return guarded(
            [&]
            {
                if (!f || (n && (!d_values || !d_out)))
                    fail(HIBF_GPU_ERR_INVALID_ARG, "null argument");
                launch_contains(f, d_values, n, d_out, pick(f, stream));
            });
    }

    int hibf_gpu_ibf_bulk_contains(hibf_gpu_ibf * f, uint64_t const * values, uint64_t n, uint64_t * out)
    {
        return guarded(
            [&]
            {
                if (!f || (n && (!values || !out)))
                    fail(HIBF_GPU_ERR_INVALID_ARG, "null argument");
                if (n == 0)
                    return;
                std::lock_guard<std::mutex> lk(f->mu);
                if (n * 8 <= kSmallBytes && n * f->bin_words * 8 <= kSmallBytes)
                {
                    f->h_in.ensure(kSmallBytes);
                    f->h_out.ensure(kSmallBytes);
                    std::memcpy(f->h_in.p, values, n * 8);
                    launch_contains(f, f->h_in.as<uint64_t>(), n, f->h_out.as<uint64_t>(), f->stream);
                    HG_CUDA(cudaStreamSynchronize(f->stream));
                    std::memcpy(out, f->h_out.p, n * f->bin_words * 8);
                    return;
                }
                f->io.ensure(n * 8);
                f->io2.ensure(n * f->bin_words * 8);
                HG_CUDA(cudaMemcpyAsync(f->io.p, values, n * 8, cudaMemcpyHostToDevice, f->stream));
                launch_contains(f, f->io.as<uint64_t>(), n, f->io2.as<uint64_t>(), f->stream);
                HG_CUDA(cudaMemcpyAsync(out, f->io2.p, n * f->bin_words * 8, cudaMemcpyDeviceToHost, f->stream));
                HG_CUDA(cudaStreamSynchronize(f->stream));
            });
    }

    int hibf_gpu_ibf_bulk_count_d(hibf_gpu_ibf * f, uint64_t const * d_values, uint64_t n, int width, void * d_out,
                                  void * stream)
    {
        return guarded(
            [&]
            {
                if (!f || (n && !d_values) || !d_out)
                    fail(HIBF_GPU_ERR_INVALID_ARG, "null argument");
                if (!width_ok(width))
                    fail(HIBF_GPU_ERR_INVALID_ARG, "width must be 1, 2, 4 or 8");
                launch_count(f, d_values, n, width, d_out, pick(f, stream));
            });
    }

    int hibf_gpu_ibf_bulk_count(hibf_gpu_ibf * f, uint64_t const * values, uint64_t n, int width, void * out)
    {
        return guarded(
            [&]
            {
                if (!f || (n && !values) || !out)
                    fail(HIBF_GPU_ERR_INVALID_ARG, "null argument");
                if (!width_ok(width))
                    fail(HIBF_GPU_ERR_INVALID_ARG, "width must be 1, 2, 4 or 8");
                std::lock_guard<std::mutex> lk(f->mu);
                std::memcpy(out, count_host(f, values, n, width), f->bins * static_cast<uint64_t>(width));
            });
    }

    int hibf_gpu_ibf_membership_for(hibf_gpu_ibf * f, uint64_t const * values, uint64_t n, uint16_t threshold,
                                    uint64_t * out_ids, uint64_t * n_out)
    {
        return guarded(
            [&]
            {
                if (!f || (n && !values) || !out_ids || !n_out)
                    fail(HIBF_GPU_ERR_INVALID_ARG, "null argument");
                std::lock_guard<std::mutex> lk(f->mu);
                uint16_t const * const counts = static_cast<uint16_t const *>(count_host(f, values, n, 2));
                uint64_t m = 0;
                for (uint64_t b = 0; b < f->bins; ++b)
                    if (counts[b] >= threshold)
                        out_ids[m++] = b;
                *n_out = m;
            });
    }

    int hibf_gpu_ibf_save(hibf_gpu_ibf * f, char const * path)
    {
        return guarded(
            [&]
            {
                if (!f || !path)
                    fail(HIBF_GPU_ERR_INVALID_ARG, "null argument");
                std::lock_guard<std::mutex> lk(f->mu);
                HG_CUDA(cudaStreamSynchronize(f->stream));
                file_writer w(path);
                write_ibf_header(w, f->bins, f->bin_size, f->hash_funs);
                write_rows(w, f->store.as<uint64_t>(), f->bin_size, f->bin_words, f->row_words, f->stream);
                uint64_t const tb = f->technical_bins();
                std::vector<uint64_t> occ(tb, 0);
                if (f->track_occupancy)
                {
                    HG_CUDA(cudaMemcpyAsync(occ.data(), f->occupancy.p, tb * 8, cudaMemcpyDeviceToHost, f->stream));
                    HG_CUDA(cudaStreamSynchronize(f->stream));
                }
                w.u64s(occ);
                w.u8(f->track_occupancy ? 1 : 0);
                w.close();
            });
    }

    int hibf_gpu_ibf_load(char const * path, hibf_gpu_ibf ** out)
    {
        return guarded(
            [&]
            {
                if (!path || !out)
                    fail(HIBF_GPU_ERR_INVALID_ARG, "null argument");
                *out = nullptr;
                file_reader r(path);
                ibf_header const h = read_ibf_header(r);
                long const words_at = r.tell();
                r.skip(h.bin_size * h.bin_words * 8);
                std::vector<uint64_t> const occ = r.u64s(h.technical_bins);
                uint8_t const track = r.u8();
                if (occ.size() != h.technical_bins || track > 1 || !r.at_end())
                    fail(HIBF_GPU_ERR_INVALID_ARG, "archive: malformed interleaved_bloom_filter");
                hibf_gpu_ibf * f = nullptr;
                int const st = hibf_gpu_ibf_create(h.bins, h.bin_size, h.hash_funs, track, &f);
                if (st != HIBF_GPU_OK)
                    fail(st, g_last_error);
                try
                {
                    r.seek(words_at);
                    read_rows(r, f->store.as<uint64_t>(), f->bin_size, f->bin_words, f->row_words, f->stream);
                    HG_CUDA(cudaMemcpyAsync(f->occupancy.p, occ.data(), occ.size() * 8, cudaMemcpyHostToDevice,
                                            f->stream));
                    HG_CUDA(cudaStreamSynchronize(f->stream));
                }
                catch (...)
                {
                    hibf_gpu_ibf_destroy(f);
                    throw;
                }
                *out = f;
            });
    }

    int hibf_gpu_ibf_upload_words(hibf_gpu_ibf * f, uint64_t const * words, uint64_t n_words)
    {
        return guarded(
            [&]
            {
                if (!f || !words)
                    fail(HIBF_GPU_ERR_INVALID_ARG, "null argument");
                if (n_words != f->bin_words * f->bin_size)
                    fail(HIBF_GPU_ERR_INVALID_ARG, "word count does not match the filter");
                std::lock_guard<std::mutex> lk(f->mu);
                HG_CUDA(cudaMemcpy2DAsync(f->store.p, f->row_words * 8, words, f->bin_words * 8, f->bin_words * 8,
                                          f->bin_size, cudaMemcpyHostToDevice, f->stream));
                HG_CUDA(cudaStreamSynchronize(f->stream));
            });
    }

    int hibf_gpu_ibf_download_words(hibf_gpu_ibf * f, uint64_t * words, uint64_t n_words)
    {
        return guarded(
            [&]
            {
                if (!f || !words)
                    fail(HIBF_GPU_ERR_INVALID_ARG, "null argument");
                if (n_words != f->bin_words * f->bin_size)
                    fail(HIBF_GPU_ERR_INVALID_ARG, "word count does not match the filter");
                std::lock_guard<std::mutex> lk(f->mu);
                if (f->row_words == f->bin_words)
                    HG_CUDA(cudaMemcpyAsync(words, f->store.p, n_words * 8, cudaMemcpyDeviceToHost, f->stream));
                else
                    HG_CUDA(cudaMemcpy2DAsync(words, f->bin_words * 8, f->store.p, f->row_words * 8, f->bin_words * 8,
                                              f->bin_size, cudaMemcpyDeviceToHost, f->stream));
                HG_CUDA(cudaStreamSynchronize(f->stream));
            });
    }

    int hibf_gpu_ibf_download_occupancy(hibf_gpu_ibf * f, uint64_t * out, uint64_t n)
    {
        return guarded(
            [&]
            {
                if (!f || !out)
                    fail(HIBF_GPU_ERR_INVALID_ARG, "null argument");
                if (n != f->technical_bins())
                    fail(HIBF_GPU_ERR_INVALID_ARG, "occupancy has technical_bins entries");
                std::lock_guard<std::mutex> lk(f->mu);
                HG_CUDA(cudaMemcpyAsync(out, f->occupancy.p, n * 8, cudaMemcpyDeviceToHost, f->stream));
                HG_CUDA(cudaStreamSynchronize(f->stream));
            });
    }

    int hibf_gpu_ibf_track_occupancy(hibf_gpu_ibf const * f, int * out)
    {
        return guarded(
            [&]
            {
                if (!f || !out)
                    fail(HIBF_GPU_ERR_INVALID_ARG, "null argument");
                *out = f->track_occupancy ? 1 : 0;
            });
    }

    int hibf_gpu_ibf_status(hibf_gpu_ibf * f)
    {
        if (!f)
            return HIBF_GPU_ERR_INVALID_ARG;
        cudaError_t const e = cudaStreamSynchronize(f->stream);
        if (e != cudaSuccess)
        {
            set_last_error(cudaGetErrorString(e));
            return HIBF_GPU_ERR_CUDA;
        }
        int bad = 0;
        if (cudaMemcpy(&bad, f->flag.p, sizeof(int), cudaMemcpyDeviceToHost) == cudaSuccess && bad)
        {
            cudaMemset(f->flag.p, 0, sizeof(int));
            set_last_error("an emplace received a bin index out of range; those values were skipped");
            return HIBF_GPU_ERR_INVALID_ARG;
        }
        return f->status;
    }

    // Same result as hibf_gpu_ibf_bulk_count_d, for callers that cannot allocate device memory.  The counting
    // scratch is the static array above, passed to the same launch as bulk_count_d: this call makes no cudaMalloc,
    // cudaFree or other allocating call.  The first call on a device looks up the array's device address and keeps it
    // for the process (issue it before any stream capture; a device reset after it is not supported); calls that
    // overlap on the GPU share the array and race; the totals are cleared at the start of every call.
    int hibf_gpu_ibf_bulk_count_noalloc_d(hibf_gpu_ibf * f, uint64_t const * d_values, uint64_t n, int width,
                                          void * d_out, void * stream)
    {
        return guarded(
            [&]
            {
                if (!f || (n && !d_values) || !d_out)
                    fail(HIBF_GPU_ERR_INVALID_ARG, "null argument");
                if (!width_ok(width))
                    fail(HIBF_GPU_ERR_INVALID_ARG, "width must be 1, 2, 4 or 8");
                if (count_counters(f) > kNoAllocMaxCounters)
                    fail(HIBF_GPU_ERR_INVALID_ARG, "hibf_gpu_ibf_bulk_count_noalloc_d supports at most " +
                                                       std::to_string(kNoAllocMaxCounters) +
                                                       " bins; use hibf_gpu_ibf_bulk_count_d");
                launch_count(f, d_values, n, width, d_out, pick(f, stream), noalloc_totals());
            });
    }

} // extern "C"
