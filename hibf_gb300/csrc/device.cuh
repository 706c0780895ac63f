// device.cuh -- device-side building blocks shared by the IBF and HIBF kernels.
//
// Layout of one IBF in HBM (the "bit store"):
//   bin_size rows; row r holds technical_bins bits (technical_bins = 64 * bin_words), LSB-first in 64-bit words,
//   starting at word r * row_words.  row_words >= bin_words pads a row so that it never straddles a 32-byte sector:
//   rows of 8/16/32 bytes stay as they are, 24 bytes become 32, longer rows are rounded up to a multiple of 32 bytes.
//   Bin b of row r is bit (b % 64) of word r * row_words + b / 64 -- the reference's bit_vector layout
//   (include/hibf/interleaved_bloom_filter.hpp:146; src/interleaved_bloom_filter.cpp:48-52) with a padded stride.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace hibf_gb300
{

constexpr unsigned kFullMask = 0xFFFFFFFFu;

// For a kernel launched beside the one before it on its stream (launch_beside): waits until that one has ended and its
// writes are visible; no-op in an ordinary launch.
__device__ __forceinline__ void wait_for_prerequisites()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
// Lets the kernel launched beside this one become resident once every block of this one has started.
__device__ __forceinline__ void launch_dependents()
{
    asm volatile("griddepcontrol.launch_dependents;");
}
constexpr uint32_t kSlabWords = 32; // words of a row that a warp reads at once, one per lane

// Lanes per value (log2) for a row, or the last slab of a row, of `words` 64-bit words (1 to kSlabWords).
__host__ __device__ constexpr uint32_t lanes_log2(uint32_t words)
{
    uint32_t l = 0;
    while ((1u << l) < words && l < 5u)
        ++l;
    return l;
}

// Counters the counting loop writes for rows of `words` words: 64 per lane of a row that one warp reads at once, 64 per
// word of a wider one.
__host__ __device__ constexpr uint32_t row_counters(uint32_t words)
{
    return words > kSlabWords ? 64u * words : 64u << lanes_log2(words);
}

// The multiplicative hashing seeds of include/hibf/interleaved_bloom_filter.hpp:172-176.  A filter's bit positions
// are defined by them, so bit-exact parity requires the same five constants.
__constant__ uint64_t c_hash_seeds[5] = {13572355802537770549ULL,
                                         13043817825332782213ULL,
                                         10650232656628343401ULL,
                                         16499269484942379435ULL,
                                         4893150838803335377ULL};

// Row selected by hash function `i` (hash_and_fit, include/hibf/interleaved_bloom_filter.hpp:185-195, divided by
// technical_bins): multiply by the seed, fold the high bits down by hash_shift = countl_zero(bin_size), multiply by
// 2^64 / golden ratio, then fastrange into [0, bin_size) with the high half of a 64x64-bit product.
__device__ __forceinline__ uint64_t hash_row(uint64_t v, uint64_t seed, uint32_t shift, uint64_t bin_size)
{
    uint64_t h = v * seed;
    h ^= h >> shift;
    h *= 11400714819323198485ULL;
    return __umul64hi(h, bin_size);
}

// The same row as a 32-bit index, for filters of fewer than 2^32 rows: hash_shift is then at least 32, so only the high
// word is folded into the low one, and the product's high half needs two 32-bit products.  About 10 instructions
// against 20, and half the registers and shuffles for the index.
__device__ __forceinline__ uint32_t hash_row32(uint64_t v, uint64_t seed, uint32_t shift, uint32_t bin_size)
{
    uint64_t const m = v * seed;
    uint32_t const hi = static_cast<uint32_t>(m >> 32);
    uint32_t const lo = static_cast<uint32_t>(m) ^ (hi >> (shift - 32u));
    uint64_t const h = ((static_cast<uint64_t>(hi) << 32) | lo) * 11400714819323198485ULL;
    uint64_t const low = __umulhi(static_cast<uint32_t>(h), bin_size);
    return static_cast<uint32_t>((static_cast<uint64_t>(static_cast<uint32_t>(h >> 32)) * bin_size + low) >> 32);
}

// R = the type of a row index: uint32_t below 2^32 rows, else uint64_t.
template <typename R>
__device__ __forceinline__ R hash_row_as(uint64_t v, uint64_t seed, uint32_t shift, uint64_t bin_size)
{
    if constexpr (sizeof(R) == 4)
        return hash_row32(v, seed, shift, static_cast<uint32_t>(bin_size));
    else
        return hash_row(v, seed, shift, bin_size);
}

__device__ __forceinline__ uint64_t ldg_nc(uint64_t const * p)
{
    uint64_t r;
    asm volatile("ld.global.nc.L1::no_allocate.u64 %0, [%1];" : "=l"(r) : "l"(p));
    return r;
}

__device__ __forceinline__ uint64_t globaltimer_ns()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Counter i of an array of `width`-byte counters: v modulo the width (the reference's counting_vector wraps).
__device__ __forceinline__ void store_count(void * out, int width, uint64_t i, uint64_t v)
{
    switch (width)
    {
    case 1:
        static_cast<uint8_t *>(out)[i] = static_cast<uint8_t>(v);
        break;
    case 2:
        static_cast<uint16_t *>(out)[i] = static_cast<uint16_t>(v);
        break;
    case 4:
        static_cast<uint32_t *>(out)[i] = static_cast<uint32_t>(v);
        break;
    default:
        static_cast<uint64_t *>(out)[i] = v;
    }
}

// ---------------------------------------------------------------------------------------------------------------
// Bit-sliced ("vertical") counters.  P[k] holds bit k of 64 independent counters, one per bin of a 64-bit row word.
// Adding four 0/1 masks costs a carry-save tree (full adder + three half adders) plus a ripple through the planes:
// about a dozen LOP3 per 32-bit half, instead of 64 per-bin adds.
// ---------------------------------------------------------------------------------------------------------------
template <int K>
__device__ __forceinline__ void planes_add4(uint64_t (&P)[K], uint64_t a, uint64_t b, uint64_t c, uint64_t d)
{
    uint64_t const u = a ^ b;
    uint64_t const s1 = u ^ c;
    uint64_t const c1 = (a & b) | (u & c); // weight 2
    uint64_t const w1 = s1 ^ d;
    uint64_t const c2 = s1 & d; // weight 2
    uint64_t const w2 = c1 ^ c2;
    uint64_t const w4 = c1 & c2;
    // plane 0 += w1
    uint64_t carry = P[0] & w1;
    P[0] ^= w1;
    // plane 1 += w2 + carry
    uint64_t t = P[1] ^ w2;
    uint64_t carry2 = (P[1] & w2) | (t & carry);
    P[1] = t ^ carry;
    // plane 2 += w4 + carry2
    t = P[2] ^ w4;
    carry = (P[2] & w4) | (t & carry2);
    P[2] = t ^ carry2;
#pragma unroll
    for (int k = 3; k < K; ++k)
    {
        uint64_t const n = P[k] & carry;
        P[k] ^= carry;
        carry = n;
    }
}

// 32x32 bit transpose across a warp: on entry lane r holds row r (bit c = A[r][c]); on exit lane c holds column c
// (bit r = A[r][c]).  Five butterfly exchanges of shrinking blocks.
__device__ __forceinline__ uint32_t warp_transpose32(uint32_t x, int lane)
{
    uint32_t constexpr masks[5] = {0x0000FFFFu, 0x00FF00FFu, 0x0F0F0F0Fu, 0x33333333u, 0x55555555u};
#pragma unroll
    for (int i = 0; i < 5; ++i)
    {
        int const s = 16 >> i;
        uint32_t const m = masks[i];
        uint32_t const y = __shfl_xor_sync(kFullMask, x, s);
        x = (lane & s) ? ((x & ~m) | ((y & ~m) >> s)) : ((x & m) | ((y & m) << s));
    }
    return x;
}

} // namespace hibf_gb300
