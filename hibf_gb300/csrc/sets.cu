// sets.cu -- the build front end's set materialisation on the device.
//
// The reference reads every user bin into a hash set (compute_kmers, src/build/compute_kmers.cpp:23-32) and sizes a
// merged max bin by the distinct count of its subtree's union (src/hierarchical_interleaved_bloom_filter.cpp:39-171,
// the favourite child's kmers).  Here both are hash tables on the device:
//   distinct_sets_device  every user bin's distinct values in first-appearance order: an entry per (user bin, value)
//                         keeps the value's first position, the values at such positions are compacted in order;
//   union_size_device     the distinct count of the union of some user bins' sets: the number of table entries.
// Bound by the table's random accesses (a 4-byte slot and the value it names, both in L2 for a few million values): the
// 64-user-bin workload, 1.47e6 values, takes 50 us of kernels; a segmented sort, a selection and a sort back took 2.1
// ms, and a dozen buffers were allocated for them.
// Only the order of split user bins' values depends on the reference's hash set (robin_hood iteration order); the
// host replays that from the first-appearance order these produce.
#include <algorithm>
#include <initializer_list>
#include <vector>

#include <cub/cub.cuh>

#include "common.hpp"

namespace hibf_gb300
{
int sm_count();

namespace
{

constexpr uint64_t kBatchValues = 1ull << 30; // values per device batch (positions and user bin bounds are ints)

constexpr uint32_t kFreeSlot = ~0u;

// The segment of position i: the last s with seg_off[s] <= i.
__device__ __forceinline__ uint32_t segment_of(int const * __restrict__ seg_off, uint32_t n_seg, uint32_t i)
{
    uint32_t lo = 0, hi = n_seg - 1u;
    while (lo < hi)
    {
        uint32_t const mid = (lo + hi + 1u) >> 1;
        if (static_cast<uint32_t>(seg_off[mid]) <= i)
            lo = mid;
        else
            hi = mid - 1u;
    }
    return lo;
}

// The first slot of (segment, value).  Each enters through a multiplication of its own: with the segment's number only
// added or xored to the value's bits, user bins of dense values (short k-mers, ids) or of ranges of ids share their
// hashes, and 1,024 bins that hold (bin << 17) + 0..2^14 took 926 probes per value.
__device__ __forceinline__ uint32_t first_slot(uint64_t v, uint32_t segment, uint32_t mask)
{
    uint64_t h = v * 0x9E3779B97F4A7C15ULL;
    h = (h ^ (h >> 32)) + segment * 0xD6E8FEB86659FD93ULL;
    return static_cast<uint32_t>((h * 0xC2B2AE3D27D4EB4FULL) >> 32) & mask;
}

// Enters every position into the table of (segment, value): a slot holds the lowest position of its pair.  mask + 1
// slots, a power of two and at least 1.5 per position, so a free one is always found.  entry[i]: position i's slot.
// Bound by random accesses to slots and values.  A slot is looked at before it is claimed, and a pair's position is
// lowered only where it is lower, so that values repeated many times read one address instead of queueing for it: 2^22
// positions of one value 8,096 -> 137 us, of 16 values 996 -> 47.  Distinct values (us, one claim and no look before
// -> now): 32 bins of 2^20 random ones 1,865 -> 1,624, 64 bins of 23,000 37 -> 47; 32 bins of all 22-bit values
// 126,179 -> 10,144, (bin << 17) + 0..2^14 145,041 -> 543.
__global__ void k_distinct_enter(uint64_t const * __restrict__ values, uint64_t n, int const * __restrict__ seg_off,
                                 uint32_t n_seg, uint32_t * slots, uint32_t mask, uint32_t * __restrict__ entry)
{
    for (uint64_t p = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; p < n;
         p += static_cast<uint64_t>(gridDim.x) * blockDim.x)
    {
        uint32_t const i = static_cast<uint32_t>(p);
        uint32_t const s = segment_of(seg_off, n_seg, i);
        uint32_t const b = static_cast<uint32_t>(seg_off[s]), e = static_cast<uint32_t>(seg_off[s + 1]);
        uint64_t const v = values[i];
        uint32_t slot = first_slot(v, s, mask);
        for (;;)
        {
            uint32_t old = __ldcg(slots + slot);
            if (old == kFreeSlot)
                old = atomicCAS(slots + slot, kFreeSlot, i);
            if (old == kFreeSlot)
                break;
            if (old >= b && old < e && values[old] == v) // a position of this segment: the same pair
            {
                if (i < old)
                    atomicMin(slots + slot, i);
                break;
            }
            slot = (slot + 1u) & mask;
        }
        entry[i] = slot;
    }
}

// flag[i] (optional): position i is its value's first in its segment; count[s]: how many are in segment s.
__global__ void k_distinct_first(uint32_t const * __restrict__ slots, uint32_t const * __restrict__ entry, uint64_t n,
                                 int const * __restrict__ seg_off, uint32_t n_seg, unsigned char * __restrict__ flag,
                                 unsigned long long * __restrict__ count)
{
    int const lane = threadIdx.x & 31;
    uint64_t const at = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x;
    for (uint64_t base = at - lane; base < n; base += static_cast<uint64_t>(gridDim.x) * blockDim.x)
    {
        uint64_t const i = base + lane; // whole warps: they add up their counts
        bool const first = i < n && slots[entry[i]] == static_cast<uint32_t>(i);
        if (flag && i < n)
            flag[i] = first ? 1 : 0;
        unsigned const counted = __ballot_sync(0xffffffffu, first);
        if (first)
        {
            uint32_t const s = segment_of(seg_off, n_seg, static_cast<uint32_t>(i));
            unsigned const same = __match_any_sync(counted, s);
            if (lane == __ffs(same) - 1)
                atomicAdd(count + s, static_cast<unsigned long long>(__popc(same)));
        }
    }
}

// Number of i with i == 0 or keys[i] != keys[i - 1] (keys sorted).
__global__ void k_count_runs(uint64_t const * __restrict__ keys, uint64_t n, unsigned long long * __restrict__ out)
{
    unsigned long long c = 0;
    for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<uint64_t>(gridDim.x) * blockDim.x)
        c += (i == 0 || keys[i - 1] != keys[i]) ? 1u : 0u;
    for (int o = 16; o > 0; o >>= 1)
        c += __shfl_down_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0 && c)
        atomicAdd(out, c);
}

unsigned grid_for(uint64_t n)
{
    return static_cast<unsigned>(std::max<uint64_t>(1, std::min<uint64_t>((n + 255) / 256, sm_count() * 8ull)));
}

uint64_t table_slots(uint64_t n)
{
    uint64_t slots = 1024;
    while (slots < n + n / 2)
        slots *= 2;
    return slots;
}

// Consecutive pieces of one allocation, each aligned for any type (an allocation and its release cost about 0.1 ms).
struct arena
{
    dbuf buf;
    size_t used{0};
    void reserve(std::initializer_list<size_t> pieces)
    {
        size_t total = 0;
        for (size_t p : pieces)
            total += (p + 255) / 256 * 256;
        buf.ensure(total);
        used = 0;
    }
    template <typename T>
    T * take(size_t bytes)
    {
        T * const p = reinterpret_cast<T *>(buf.as<char>() + used);
        used += (bytes + 255) / 256 * 256;
        return p;
    }
};

} // namespace

bool device_present()
{
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess || n == 0)
    {
        (void)cudaGetLastError();
        return false;
    }
    return true;
}

void distinct_sets_device(uint64_t const * values, std::vector<uint64_t> const & offsets,
                          std::vector<std::vector<uint64_t>> & sets)
{
    uint64_t const nub = offsets.size() - 1;
    sets.assign(nub, {});
    cudaStream_t s = nullptr;
    HG_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    struct stream_guard
    {
        cudaStream_t s;
        ~stream_guard()
        {
            cudaStreamSynchronize(s);
            cudaStreamDestroy(s);
        }
    } const guard{s};
    arena mem;
    std::vector<uint64_t> distinct;
    std::vector<unsigned long long> counts;
    for (uint64_t u0 = 0; u0 < nub;)
    {
        // a batch of whole user bins, at most kBatchValues values unless one bin alone is larger
        uint64_t u1 = u0 + 1;
        while (u1 < nub && offsets[u1 + 1] - offsets[u0] <= kBatchValues)
            ++u1;
        uint64_t const base = offsets[u0];
        uint64_t const m = offsets[u1] - base;
        if (m >= (1ull << 31))
            fail(HIBF_GPU_ERR_INVALID_ARG, "a user bin of 2^31 or more values");
        uint32_t const nseg = static_cast<uint32_t>(u1 - u0);
        if (m == 0)
        {
            u0 = u1;
            continue;
        }
        std::vector<int> off(nseg + 1);
        for (uint32_t k = 0; k <= nseg; ++k)
            off[k] = static_cast<int>(offsets[u0 + k] - base);
        uint64_t const slots = table_slots(m);
        size_t select_bytes = 0;
        HG_CUDA(cub::DeviceSelect::Flagged(nullptr, select_bytes, static_cast<uint64_t const *>(nullptr),
                                           static_cast<unsigned char const *>(nullptr), static_cast<uint64_t *>(nullptr),
                                           static_cast<unsigned long long *>(nullptr), m, s));
        size_t const off_bytes = (nseg + 1) * sizeof(int), count_bytes = nseg * sizeof(unsigned long long);
        mem.reserve({m * 8, m * 8, slots * 4, m * 4, m, off_bytes, count_bytes, 8, select_bytes});
        uint64_t * const d_in = mem.take<uint64_t>(m * 8);
        uint64_t * const d_out = mem.take<uint64_t>(m * 8);
        uint32_t * const d_slots = mem.take<uint32_t>(slots * 4);
        uint32_t * const d_entry = mem.take<uint32_t>(m * 4);
        unsigned char * const d_flag = mem.take<unsigned char>(m);
        int * const d_off = mem.take<int>(off_bytes);
        auto * const d_count = mem.take<unsigned long long>(count_bytes);
        auto * const d_nsel = mem.take<unsigned long long>(8);
        void * const d_tmp = mem.take<char>(select_bytes);
        HG_CUDA(cudaMemcpyAsync(d_in, values + base, m * 8, cudaMemcpyHostToDevice, s));
        HG_CUDA(cudaMemcpyAsync(d_off, off.data(), off_bytes, cudaMemcpyHostToDevice, s));
        HG_CUDA(cudaMemsetAsync(d_slots, 0xFF, slots * 4, s));
        HG_CUDA(cudaMemsetAsync(d_count, 0, count_bytes, s));
        k_distinct_enter<<<grid_for(m), 256, 0, s>>>(d_in, m, d_off, nseg, d_slots, static_cast<uint32_t>(slots - 1),
                                                     d_entry);
        HG_CUDA(cudaGetLastError());
        k_distinct_first<<<grid_for(m), 256, 0, s>>>(d_slots, d_entry, m, d_off, nseg, d_flag, d_count);
        HG_CUDA(cudaGetLastError());
        // positions ascending = user bins in order, each in first-appearance order
        HG_CUDA(cub::DeviceSelect::Flagged(d_tmp, select_bytes, static_cast<uint64_t const *>(d_in),
                                           static_cast<unsigned char const *>(d_flag), d_out, d_nsel, m, s));
        counts.resize(nseg);
        HG_CUDA(cudaMemcpyAsync(counts.data(), d_count, count_bytes, cudaMemcpyDeviceToHost, s));
        HG_CUDA(cudaStreamSynchronize(s));
        uint64_t total = 0;
        for (unsigned long long c : counts)
            total += c;
        distinct.resize(total);
        HG_CUDA(cudaMemcpyAsync(distinct.data(), d_out, total * 8, cudaMemcpyDeviceToHost, s));
        HG_CUDA(cudaStreamSynchronize(s));
        uint64_t at = 0;
        for (uint32_t k = 0; k < nseg; ++k)
        {
            sets[u0 + k].assign(distinct.data() + at, distinct.data() + at + counts[k]);
            at += counts[k];
        }
        u0 = u1;
    }
}

namespace
{

// The union's size by a sort, for more values than the table's 32-bit positions name.
uint64_t union_size_sorted(std::vector<std::vector<uint64_t>> const & sets, std::vector<uint64_t> const & members,
                           uint64_t n, cudaStream_t s)
{
    dbuf d_in, d_sorted, d_tmp, d_count;
    d_in.ensure(n * 8);
    d_sorted.ensure(n * 8);
    d_count.ensure(8);
    uint64_t at = 0;
    for (uint64_t u : members)
    {
        if (!sets[u].empty())
            HG_CUDA(cudaMemcpyAsync(d_in.as<uint64_t>() + at, sets[u].data(), sets[u].size() * 8,
                                    cudaMemcpyHostToDevice, s));
        at += sets[u].size();
    }
    size_t t = 0;
    HG_CUDA(cub::DeviceRadixSort::SortKeys(nullptr, t, d_in.as<uint64_t>(), d_sorted.as<uint64_t>(), n, 0, 64, s));
    d_tmp.ensure(t);
    HG_CUDA(cub::DeviceRadixSort::SortKeys(d_tmp.p, t, d_in.as<uint64_t>(), d_sorted.as<uint64_t>(), n, 0, 64, s));
    HG_CUDA(cudaMemsetAsync(d_count.p, 0, 8, s));
    k_count_runs<<<grid_for(n), 256, 0, s>>>(d_sorted.as<uint64_t>(), n, d_count.as<unsigned long long>());
    HG_CUDA(cudaGetLastError());
    unsigned long long c = 0;
    HG_CUDA(cudaMemcpyAsync(&c, d_count.p, 8, cudaMemcpyDeviceToHost, s));
    HG_CUDA(cudaStreamSynchronize(s));
    return c;
}

} // namespace

uint64_t union_size_device(std::vector<std::vector<uint64_t>> const & sets, std::vector<uint64_t> const & members)
{
    uint64_t n = 0;
    for (uint64_t u : members)
        n += sets[u].size();
    if (n == 0)
        return 0;
    cudaStream_t s = nullptr;
    HG_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    struct stream_guard
    {
        cudaStream_t s;
        ~stream_guard()
        {
            cudaStreamSynchronize(s);
            cudaStreamDestroy(s);
        }
    } const guard{s};
    if (n >= (1ull << 31))
        return union_size_sorted(sets, members, n, s);
    arena mem;
    uint64_t const slots = table_slots(n);
    mem.reserve({n * 8, slots * 4, n * 4, 8, 8});
    uint64_t * const d_in = mem.take<uint64_t>(n * 8);
    uint32_t * const d_slots = mem.take<uint32_t>(slots * 4);
    uint32_t * const d_entry = mem.take<uint32_t>(n * 4);
    int * const d_off = mem.take<int>(8);
    auto * const d_count = mem.take<unsigned long long>(8);
    uint64_t at = 0;
    for (uint64_t u : members)
    {
        if (!sets[u].empty())
            HG_CUDA(cudaMemcpyAsync(d_in + at, sets[u].data(), sets[u].size() * 8, cudaMemcpyHostToDevice, s));
        at += sets[u].size();
    }
    int const off[2] = {0, static_cast<int>(n)};
    HG_CUDA(cudaMemcpyAsync(d_off, off, 8, cudaMemcpyHostToDevice, s));
    HG_CUDA(cudaMemsetAsync(d_slots, 0xFF, slots * 4, s));
    HG_CUDA(cudaMemsetAsync(d_count, 0, 8, s));
    k_distinct_enter<<<grid_for(n), 256, 0, s>>>(d_in, n, d_off, 1, d_slots, static_cast<uint32_t>(slots - 1), d_entry);
    HG_CUDA(cudaGetLastError());
    k_distinct_first<<<grid_for(n), 256, 0, s>>>(d_slots, d_entry, n, d_off, 1, nullptr, d_count);
    HG_CUDA(cudaGetLastError());
    unsigned long long c = 0;
    HG_CUDA(cudaMemcpyAsync(&c, d_count, 8, cudaMemcpyDeviceToHost, s));
    HG_CUDA(cudaStreamSynchronize(s));
    return c;
}

} // namespace hibf_gb300
