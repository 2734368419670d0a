// Binning: prefix sum of per-block instance counts, (tile, Gaussian) instance
// emission, a stable least-significant-digit radix sort of the instance keys
// and per-tile range extraction.  All kernels are hand written (no CUB).
//
// Replaces, with identical results (same key width, same stable order, same
// uint2 ranges), the reference sequence
//   cub::DeviceScan::InclusiveSum + blocking D2H copy + create_instances_cu +
//   cub::DeviceRadixSort::SortPairs + extract_instance_ranges_cu
// (rasterization/src/hybrid_blend/inference.cu:109-165, rasterization/src/shared_kernels.cu:7-95).
//
// Differences in how the work is organised:
//  * the per-Gaussian prefix sum is never materialised: the preprocess kernel leaves one
//    count per block of 256 Gaussians, one small kernel scans those, and the emission
//    kernel rebuilds the in-block offsets in shared memory;
//  * the instance count stays on the device: emission, sort and range kernels run
//    persistent grids (a multiple of the SM count) and read the count from the frame
//    status, so the frame has no host synchronisation in the middle;
//  * a Gaussian's instances are emitted by the whole block (coalesced runs), not by one thread;
//  * digits are up to 9 bits wide, so tile keys of up to 18 bits need two passes; every
//    pass stages the locally sorted tile in shared memory so that global writes are runs.
#include "kernels.h"

#include <algorithm>
#include <cstring>

namespace htgs {

FrameGeometry make_geometry(int mode, int width, int height) {
    FrameGeometry g;
    g.width = width; g.height = height;
    g.tile_w = mode_tile_w(mode); g.tile_h = mode_tile_h(mode);
    g.grid_w = (width + g.tile_w - 1) / g.tile_w;
    g.grid_h = (height + g.tile_h - 1) / g.tile_h;
    g.n_tiles = g.grid_w * g.grid_h;
    return g;
}

static int bit_length(uint32_t v) { int b = 0; while (v) { ++b; v >>= 1; } return b; }   // rasterization/include/rasterization_utils.h:3-13

// Digits of at most kMaxRadixBits bits, about equally wide; returns how many.
static int split_digits(int bits, int* width, int* shift, int most = kMaxRadixBits) {
    const int n = (bits + most - 1) / most;
    int at = 0;
    for (int i = 0; i < n; ++i) {
        width[i] = bits / n + (i < bits % n ? 1 : 0);
        shift[i] = at;
        at += width[i];
    }
    return n;
}

SortPlan make_sort_plan(int mode, int n_tiles) {
    SortPlan p{};
    const int tile_bits = bit_length(uint32_t(n_tiles > 0 ? n_tiles - 1 : 0));
    if (mode == HTGS_MODE_ALPHA_BLEND_GLOBAL_ORDERING) { p.key_bytes = 8; p.end_bit = tile_bits + 32; }   // alpha_blend_global_ordering/inference.cu:45
    else { p.end_bit = tile_bits; p.key_bytes = tile_bits <= 16 ? 2 : 4; }                                 // hybrid_blend/inference.cu:121-129
    p.n_passes = split_digits(tile_bits, p.bits, p.shift);
    p.final_buffer = p.n_passes & 1;
    return p;
}

namespace {

inline size_t align16(size_t v) { return (v + 15) & ~size_t(15); }

constexpr int kSortThreads = 256;
constexpr int kSortItems = kSortTile / kSortThreads;   // 16
constexpr int kSortWarps = kSortThreads / 32;          // 8

__device__ __forceinline__ uint32_t warp_inclusive_scan(uint32_t v) {
    #pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31) >= o) v += t;
    }
    return v;
}

// Exclusive scan of block sums -> block offsets; publishes the instance count.  One CTA: every thread takes a run of
// consecutive values (so that the whole array is covered in ONE round: load, thread-local sums, one block scan, store)
// instead of looping over the array 1024 values at a time with four barriers per round.
constexpr int kScanThreads = 1024;
constexpr int kScanRun = 16;            // values per thread and round: 16384 block sums (4.2 M Gaussians) per round
// instances: the above.  visible (GLOBAL_ORDERING): adds up the instances, and makes the blocks' visible Gaussians, which lie where the offsets
// go, into their prefix.
enum class ScanOf { instances, visible };
template <ScanOf OF>
__global__ void __launch_bounds__(kScanThreads) scan_block_sums_kernel(const uint32_t* __restrict__ block_sums, uint32_t* block_offsets,
                                                                     uint32_t n_blocks, uint32_t capacity, FrameStatus* status) {
    grid_dependency();
    __shared__ unsigned long long warp_tot[kScanThreads / 32];
    __shared__ unsigned long long carry_s;
    [[maybe_unused]] __shared__ unsigned long long instances_s;
    if (threadIdx.x == 0) { carry_s = 0ull; instances_s = 0ull; }
    [[maybe_unused]] unsigned long long instances = 0;
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (uint32_t base = 0; base < n_blocks; base += kScanThreads * kScanRun) {
        const uint32_t first = base + threadIdx.x * kScanRun;
        uint32_t v[kScanRun];
        unsigned long long mine = 0;
        #pragma unroll
        for (int i = 0; i < kScanRun; ++i) {
            v[i] = first + i < n_blocks ? (OF == ScanOf::visible ? block_offsets : block_sums)[first + i] : 0u;
            mine += v[i];
            if constexpr (OF == ScanOf::visible) instances += first + i < n_blocks ? block_sums[first + i] : 0u;
        }
        unsigned long long inc = mine;
        #pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const unsigned long long t = __shfl_up_sync(0xffffffffu, inc, o); if (lane >= uint32_t(o)) inc += t; }
        if (lane == 31) warp_tot[warp] = inc;
        __syncthreads();
        if (warp == 0) {
            const unsigned long long t = warp_tot[lane];
            unsigned long long s = t;
            #pragma unroll
            for (int o = 1; o < 32; o <<= 1) { const unsigned long long u = __shfl_up_sync(0xffffffffu, s, o); if (lane >= uint32_t(o)) s += u; }
            warp_tot[lane] = s - t;
        }
        __syncthreads();
        unsigned long long running = carry_s + warp_tot[warp] + (inc - mine);
        #pragma unroll
        for (int i = 0; i < kScanRun; ++i) {
            if (first + i < n_blocks) block_offsets[first + i] = running > 0xffffffffull ? 0xffffffffu : uint32_t(running);
            running += v[i];
        }
        __syncthreads();
        if (threadIdx.x == kScanThreads - 1) carry_s = running;
        __syncthreads();
    }
    if constexpr (OF == ScanOf::visible) {
        #pragma unroll
        for (int o = 16; o > 0; o >>= 1) instances += __shfl_xor_sync(0xffffffffu, instances, o);
        if (lane == 0) atomicAdd(&instances_s, instances);
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        const unsigned long long total = OF == ScanOf::visible ? instances_s : carry_s;
        status->n_instances = total > 0xffffffffull ? 0xffffffffu : uint32_t(total);
        status->overflow = total > (unsigned long long)capacity ? 1u : 0u;
    }
}

// What a sort sorts: the frame's instances, or its visible Gaussians (of which there are no more than instances).  No more than the buffers hold:
// htgs_forward_finish may be given a smaller count than htgs_forward_begin counted, and its lists are cut then.  Nothing once a wait has given up:
// the output of a pass that did not finish is not a list of valid indices.
// One load: kernels of a few microseconds wait for this first (a load per member, the second only if the first was zero: list_visible_kernel 47 -> 56 us at
// 8 M Gaussians).
__device__ __forceinline__ uint32_t frame_instances(const FrameStatus* status, uint32_t capacity, bool visible = false) {
    const uint4 head = *reinterpret_cast<const uint4*>(status);        // n_instances, overflow, n_visible, error
    return (head.y | head.w) != 0 ? 0u : min(visible ? head.z : head.x, capacity);
}

// One block per 256 Gaussians (the blocks of the preprocess kernel), which writes their instances cooperatively: slot j belongs to
// the Gaussian whose exclusive offset is the last one <= j (eight steps of search); inside a Gaussian the order is row-major over
// its tile box (rasterization/src/shared_kernels.cu:21-28), so the emitted stream is identical to the reference's.  Bound by
// instructions (the search, the split in row and column by a multiplication).  7.3 M instances: 49 us, 154 M: 493 us.  A search per
// warp (five steps) where the warps have about equal work gave 51 and 504 us, always 88 and 715: one warp often has most of them.
// The kernel also clears what the sort and the range kernel count in (`clear`): one launch instead of three.
struct ClearList { uint4* begin[3]; uint64_t count[3]; uint64_t per_sort_block[3]; };   // 16-byte words: a fixed number, plus so many per sort block of the frame
__device__ __forceinline__ void clear_words(const ClearList& clear, uint32_t instances) {
    const uint64_t sort_blocks = (uint64_t(instances) + kSortTile - 1) / kSortTile;
    #pragma unroll
    for (int c = 0; c < 3; ++c) {
        const uint64_t words = clear.count[c] + clear.per_sort_block[c] * sort_blocks;
        for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < words; i += uint64_t(gridDim.x) * blockDim.x) clear.begin[c][i] = make_uint4(0u, 0u, 0u, 0u);
    }
}
// SORTED (GLOBAL_ORDERING): the blocks are those of the visible Gaussians in depth order, `list`; what has to be cleared has been by then.  A block adds up
// the blocks in front of it, of `block_sums` those of its group of 256 and of `group_sums` whole groups, which takes the place of a scan kernel.
constexpr uint32_t kSumGroup = kPreprocessBlock;
template <typename KeyT, bool SORTED>
__global__ void __launch_bounds__(kPreprocessBlock) emit_instances_kernel(
    const uint32_t* __restrict__ n_touched, const ushort4* __restrict__ bounds, const uint32_t* __restrict__ list,
    const uint32_t* __restrict__ block_sums, const uint32_t* __restrict__ block_offsets, const uint32_t* __restrict__ group_sums, KeyT* __restrict__ keys, uint32_t* __restrict__ prims,
    uint32_t n_primitives, uint32_t grid_w, uint32_t capacity, const FrameStatus* __restrict__ status, const __grid_constant__ ClearList clear)
{
    grid_dependency();
    const uint32_t frame = frame_instances(status, capacity, SORTED), n = SORTED ? frame : n_primitives;
    if constexpr (!SORTED) clear_words(clear, frame);
    if (SORTED && blockIdx.x * kPreprocessBlock >= n) return;
    const uint32_t total = block_sums[blockIdx.x];
    if (total == 0 || frame == 0) return;   // a frame that does not fit its instance buffers is skipped by every later stage
    __shared__ uint32_t excl[kPreprocessBlock];
    __shared__ uint4 box[kPreprocessBlock];          // x_min | y_min << 16, width, reciprocal of the width (2^32 / width, rounded up; 0: divide), Gaussian
    __shared__ uint32_t warp_tot[kPreprocessBlock / 32];
    [[maybe_unused]] __shared__ uint32_t warp_before[kPreprocessBlock / 32];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    if constexpr (SORTED) {
        const uint32_t group = blockIdx.x / kSumGroup, in_group = blockIdx.x % kSumGroup;
        uint32_t before = threadIdx.x < in_group ? block_sums[blockIdx.x - in_group + threadIdx.x] : 0u;
        for (uint32_t i = threadIdx.x; i < group; i += kPreprocessBlock) before += group_sums[i];
        before = __reduce_add_sync(0xffffffffu, before);
        if (lane == 0) warp_before[warp] = before;
    }
    const uint32_t first = blockIdx.x * kPreprocessBlock;
    const uint32_t at = first + threadIdx.x;
    const bool valid = at < n;
    const uint32_t idx = SORTED ? (valid ? list[at] : 0u) : at;
    const uint32_t cnt = valid ? n_touched[idx] : 0u;
    if (cnt) {
        const ushort4 b = bounds[idx];
        const uint32_t w = uint32_t(b.y) - uint32_t(b.x);
        const uint32_t rcp = w > 1 && uint64_t(cnt) * w < (1ull << 32) ? 0xffffffffu / w + 1u : 0u;
        box[threadIdx.x] = make_uint4(uint32_t(b.x) | (uint32_t(b.z) << 16), w, rcp, idx);
    }
    const uint32_t inc = warp_inclusive_scan(cnt);
    excl[threadIdx.x] = inc - cnt;
    if (lane == 31) warp_tot[warp] = inc;
    __syncthreads();
    uint32_t warp_base = 0;
    uint64_t base = SORTED ? 0u : block_offsets[blockIdx.x];
    #pragma unroll
    for (int w = 0; w < kPreprocessBlock / 32; ++w) {
        if (w < int(warp)) warp_base += warp_tot[w];
        if constexpr (SORTED) base += warp_before[w];
    }
    auto emit = [&](uint32_t slot, uint32_t local, uint32_t owner) {
        const uint4 b = box[owner];
        const uint32_t ly = b.y == 1u ? local : b.z ? __umulhi(local, b.z) : local / b.y;
        const uint32_t lx = local - ly * b.y;
        const uint32_t tile = ((b.x >> 16) + ly) * grid_w + (b.x & 0xffffu) + lx;
        const uint64_t dst = base + slot;
        if (dst < capacity) {
            keys[dst] = KeyT(tile);
            prims[dst] = b.w;
        }
    };
    __syncthreads();
    excl[threadIdx.x] += warp_base;
    __syncthreads();
    for (uint32_t j = threadIdx.x; j < total; j += kPreprocessBlock) {
        uint32_t lo = 0;
        #pragma unroll
        for (uint32_t step = kPreprocessBlock / 2; step > 0; step >>= 1) if (excl[lo + step] <= j) lo += step;
        emit(j, j - excl[lo], lo);
    }
}

template <typename KeyT>
__device__ __forceinline__ uint32_t digit_of(KeyT k, int shift, uint32_t mask) { return uint32_t(k >> shift) & mask; }

// ---- stable LSD radix sort, one kernel per pass ("onesweep") ------------------------------------------------------------
// One kernel counts the digits of EVERY pass in a single read of the keys; then each pass is ONE scatter kernel whose sort
// blocks learn where their digits start from their predecessors through tables of published counts (decoupled look-back)
// instead of a histogram kernel and a scan kernel in front of every scatter.
//
// Scratch (cleared by the emission kernel): per pass a ticket counter, the digit histogram, a word per (sort block, digit) - bit 31:
// published, below it the block's count - and a 64-bit word per (group of 32 sort blocks, digit): bits 62-63 = state (0 nothing
// yet, 1 the group's own count, 2 the count summed over the group and all groups before it), below it the count.  A block adds
// the words of the blocks of its group in front of it and walks back over groups: the blocks of the first wave, which all start
// together and find no summed count nearby, need a few round trips to L2 instead of one for every 16 blocks in front of them.
// Blocks take their number from the pass's ticket counter when they start, so a block only ever waits for blocks that are
// already running; every wait is bounded and reports through the frame status instead of spinning forever.
constexpr uint32_t kRowPublished = 1u << 31;
constexpr unsigned long long kGroupAggregate = 1ull << 62, kGroupPrefix = 2ull << 62, kGroupValue = (1ull << 62) - 1ull;
constexpr uint32_t kLookbackPolls = 1u << 20;      // about half a second of polling before a block gives up
constexpr uint32_t kGroup = 32;                    // sort blocks per group
constexpr int kLookbackBatch = 8;                  // words read per step

constexpr int kMostDepthWords = 3 << kMaxRadixBits;     // of the sort by depth: three passes of 9 bits, or four of at most 8
constexpr int kFirstDepthPass = 4;       // its place in tickets and digit_hist; there are at most four passes over the tile
struct SortScratch {
    unsigned long long* depth_groups;    // GLOBAL_ORDERING, the sort by depth: [groups][depth_words], all passes
    uint32_t* depth_rows;                // [sort_blocks_cap][row_stride]
    uint32_t* group_sums;                // instances of every kSumGroup blocks of the emission
    uint32_t* tickets;                   // [16]
    uint32_t* digit_hist;                // [8][kMaxRadixBins]
    unsigned long long* groups[8];       // per pass [ceil(sort_blocks_cap / kGroup)][1 << bits]
    uint32_t* rows[8];                   // [sort_blocks_cap][row_stride]: the passes' counts of a sort block lie behind one another
    size_t fixed_bytes, row_stride, bytes;
};
// depth_words: words per sort block that the passes over the depth take (0 in the other modes)
__host__ SortScratch carve_sort_scratch(void* base, const SortPlan& plan, uint32_t sort_blocks_cap, size_t depth_words) {
    SortScratch sc{};
    unsigned char* p = static_cast<unsigned char*>(base);
    size_t off = 0;
    sc.tickets = reinterpret_cast<uint32_t*>(p + off); off += 64;
    sc.digit_hist = reinterpret_cast<uint32_t*>(p + off); off += size_t(8) * kMaxRadixBins * sizeof(uint32_t);
    const size_t n_groups = (size_t(sort_blocks_cap) + kGroup - 1) / kGroup;
    for (int i = 0; i < plan.n_passes; ++i) {
        sc.groups[i] = reinterpret_cast<unsigned long long*>(p + off);
        off += (n_groups << plan.bits[i]) * sizeof(unsigned long long);
    }
    sc.depth_groups = reinterpret_cast<unsigned long long*>(p + off);
    off += n_groups * depth_words * sizeof(unsigned long long);
    sc.group_sums = reinterpret_cast<uint32_t*>(p + off);
    if (depth_words > 0) off += (size_t(sort_blocks_cap) * (kSortTile / kPreprocessBlock) / kSumGroup + 1) * sizeof(uint32_t);
    off = (off + 15) & ~size_t(15);
    sc.fixed_bytes = off;
    for (int i = 0; i < plan.n_passes; ++i) {
        sc.rows[i] = reinterpret_cast<uint32_t*>(p + off) + sc.row_stride;
        sc.row_stride += size_t(1) << plan.bits[i];
    }
    sc.depth_rows = reinterpret_cast<uint32_t*>(p + off) + sc.row_stride;
    sc.row_stride += depth_words;
    sc.row_stride = (sc.row_stride + 3) & ~size_t(3);
    sc.bytes = off + size_t(sort_blocks_cap) * sc.row_stride * sizeof(uint32_t);
    return sc;
}

struct PassTable { int n_passes; int shift[8]; int bits[8]; bool visible; };

// Digit histograms of all passes in one read of the keys.  A thread takes 16 bytes of consecutive keys per load and
// counts runs of equal digits before touching shared memory: a Gaussian's instances are neighbouring tiles, so the high
// digits of consecutive keys agree (one atomic per run) while the low digits differ (no two lanes on one counter).
template <typename KeyT>
__global__ void __launch_bounds__(256) radix_histogram_all_kernel(const KeyT* __restrict__ keys, uint32_t* __restrict__ digit_hist,
                                                                   const FrameStatus* status, uint32_t capacity, const __grid_constant__ PassTable passes) {
    grid_dependency();
    constexpr uint32_t kRun = 16 / sizeof(KeyT);
    __shared__ uint32_t hist[8 * kMaxRadixBins];
    const uint32_t n = frame_instances(status, capacity, passes.visible);
    for (uint32_t i = threadIdx.x; i < uint32_t(passes.n_passes) * kMaxRadixBins; i += 256) hist[i] = 0;
    __syncthreads();
    const uint32_t n_runs = (n + kRun - 1) / kRun;
    for (uint32_t r = blockIdx.x * 256 + threadIdx.x; r < n_runs; r += gridDim.x * 256) {
        const uint32_t first = r * kRun;
        KeyT k[kRun];
        uint32_t count = kRun;
        if (first + kRun <= n) {
            const uint4 raw = __ldg(reinterpret_cast<const uint4*>(keys + first));      // the key buffers are 256-byte aligned
            __builtin_memcpy(k, &raw, 16);
        } else {
            count = n - first;
            #pragma unroll
            for (uint32_t i = 0; i < kRun; ++i) k[i] = i < count ? keys[first + i] : KeyT(0);
        }
        for (int p = 0; p < passes.n_passes; ++p) {
            const int shift = passes.shift[p];
            const uint32_t mask = (1u << passes.bits[p]) - 1u;
            uint32_t run_digit = uint32_t(k[0] >> shift) & mask, run_length = 1;
            #pragma unroll
            for (uint32_t i = 1; i < kRun; ++i) {
                if (i < count) {
                    const uint32_t d = uint32_t(k[i] >> shift) & mask;
                    if (d == run_digit) ++run_length;
                    else { atomicAdd(&hist[p * kMaxRadixBins + run_digit], run_length); run_digit = d; run_length = 1; }
                }
            }
            atomicAdd(&hist[p * kMaxRadixBins + run_digit], run_length);
        }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < uint32_t(passes.n_passes) * kMaxRadixBins; i += 256) {
        const uint32_t v = hist[i];
        if (v) atomicAdd(&digit_hist[i], v);
    }
}

// Exclusive scan of up to 512 values held in shared memory by 256 threads (two per thread).
__device__ __forceinline__ void block_exclusive_scan_512(uint32_t* vals, uint32_t n_bins, uint32_t* warp_tot) {
    const uint32_t i0 = 2 * threadIdx.x, i1 = i0 + 1;
    const uint32_t a = i0 < n_bins ? vals[i0] : 0u, b = i1 < n_bins ? vals[i1] : 0u;
    const uint32_t s = a + b;
    const uint32_t inc = warp_inclusive_scan(s);
    if ((threadIdx.x & 31) == 31) warp_tot[threadIdx.x >> 5] = inc;
    __syncthreads();
    uint32_t warp_base = 0;
    #pragma unroll
    for (int w = 0; w < kSortWarps; ++w) if (w < int(threadIdx.x >> 5)) warp_base += warp_tot[w];
    const uint32_t excl = warp_base + inc - s;
    if (i0 < n_bins) vals[i0] = excl;
    if (i1 < n_bins) vals[i1] = excl + a;
    __syncthreads();
}

// One pass: stable scatter.  Warp w of a sort block owns the 512 consecutive keys [w*512, (w+1)*512) of the block's tile
// and visits them in 16 rounds of 32, so (warp, round, lane) order is input order.  A warp keeps per digit a count and a mask in
// shared memory: the lanes of a round OR themselves into the mask of their digit, read mask and count back, and the highest
// lane of each digit adds the round to the count.  That is 16 instructions for a round; a ballot per digit bit took over 100
// (225 in the whole kernel, now 138).  A scan over warps and digits turns the counts into positions in the locally sorted
// tile, which is staged in shared memory (over the masks) and written out as runs.  The Gaussian indices are requested after
// the ranking, so that they do not hold registers before.
// Bound by the latency of a block's phases and their barriers.  7.3 M keys of 16 bits, both passes: 189 -> 123 us; 154 M keys of
// 32 bits: 3.86 -> 2.78 ms.  Six blocks per SM instead of four change nothing.
template <typename KeyT> constexpr int scatter_blocks_per_sm() { return sizeof(KeyT) == 4 ? 5 : 4; }
template <typename KeyT>
__global__ void __launch_bounds__(kSortThreads, scatter_blocks_per_sm<KeyT>()) radix_scatter_kernel(
    const KeyT* __restrict__ keys_in, const uint32_t* __restrict__ prims_in, KeyT* __restrict__ keys_out, uint32_t* __restrict__ prims_out,
    const uint32_t* __restrict__ digit_hist, uint32_t* rows, uint32_t row_stride, unsigned long long* groups, uint32_t* ticket,
    FrameStatus* status, uint32_t capacity, int shift, int bits, bool visible)
{
    grid_dependency();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const uint32_t n_bins = 1u << bits, mask = n_bins - 1;
    uint32_t* block_excl = reinterpret_cast<uint32_t*>(smem_raw);                 // [n_bins]
    uint32_t* global_base = block_excl + n_bins;                                  // [n_bins]
    uint32_t* digit_base = global_base + n_bins;                                  // [n_bins]
    uint32_t* shared_region = digit_base + n_bins + (bits == 1 ? 2 : 0);          // 16-byte aligned
    uint2* table = reinterpret_cast<uint2*>(shared_region);                       // [kSortWarps][n_bins] (mask, count), then:
    uint32_t* prims_s = shared_region;                                            // [kSortTile]
    KeyT* keys_s = reinterpret_cast<KeyT*>(prims_s + kSortTile);                  // [kSortTile]
    __shared__ uint32_t warp_tot[kSortWarps];
    __shared__ uint32_t s_blk, s_failed;

    const uint32_t n = frame_instances(status, capacity, visible);
    const uint32_t n_blocks = uint32_t((uint64_t(n) + kSortTile - 1) / kSortTile);
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (n == 0) return;       // without a ticket: the others of a pass in which a wait gave up do not miss this block

    // exclusive prefix of the digit totals (same for every sort block)
    for (uint32_t d = threadIdx.x; d < n_bins; d += kSortThreads) digit_base[d] = digit_hist[d];
    if (threadIdx.x == 0) s_failed = 0;
    __syncthreads();
    block_exclusive_scan_512(digit_base, n_bins, warp_tot);

    for (;;) {
        if (threadIdx.x == 0) s_blk = atomicAdd(ticket, 1u);
        for (uint32_t i = threadIdx.x; i < kSortWarps * n_bins / 2; i += kSortThreads) reinterpret_cast<uint4*>(table)[i] = make_uint4(0u, 0u, 0u, 0u);
        __syncthreads();
        const uint32_t blk = s_blk;
        if (blk >= n_blocks) break;
        const uint32_t base = blk * kSortTile + warp * (kSortItems * 32);
        constexpr bool kPacked = sizeof(KeyT) == 2;      // 16-bit keys share a register with their rank
        KeyT key[kSortItems];
        uint32_t rank[kSortItems];
        auto key_of = [&](int r) -> KeyT { return kPacked ? KeyT(rank[r]) : key[r]; };
        #pragma unroll
        for (int r = 0; r < kSortItems; ++r) {
            const uint32_t idx = base + r * 32 + lane;
            key[r] = idx < n ? keys_in[idx] : KeyT(0);
        }
        uint2* mine = table + warp * n_bins;
        #pragma unroll
        for (int r = 0; r < kSortItems; ++r) {
            const bool valid = base + r * 32 + lane < n;
            uint2* cell = mine + digit_of(key[r], shift, mask);
            if (valid) atomicOr(&cell->x, 1u << lane);
            __syncwarp();
            uint2 seen = make_uint2(0u, 0u);
            if (valid) seen = *cell;
            rank[r] = seen.y + __popc(seen.x & lanemask_lt());
            if constexpr (kPacked) rank[r] = (rank[r] << 16) | uint32_t(key[r]);
            __syncwarp();
            if (valid && (seen.x >> lane) == 1u) *cell = make_uint2(0u, seen.y + __popc(seen.x));
            __syncwarp();
        }
        __syncthreads();
        // per digit: exclusive prefix over warps, the block's count; publish it and look back for where the digit's run starts
        for (uint32_t d = threadIdx.x; d < n_bins; d += kSortThreads) {
            uint32_t running = 0;
            #pragma unroll
            for (int w = 0; w < kSortWarps; ++w) { const uint32_t t = table[w * n_bins + d].y; table[w * n_bins + d].y = running; running += t; }
            block_excl[d] = running;
            volatile uint32_t* row = rows + d;
            row[size_t(blk) * row_stride] = kRowPublished | running;
            const uint32_t group = blk / kGroup, group_first = group * kGroup;
            const bool closes_group = blk - group_first == kGroup - 1u;
            uint32_t polls = 0;
            unsigned long long before = 0;          // instances with this digit in the preceding sort blocks
            bool failed = false;                    // gave up: report, never spin forever
            for (uint32_t p = group_first; p < blk; p += kLookbackBatch) {
                uint32_t v[kLookbackBatch];
                #pragma unroll
                for (uint32_t i = 0; i < kLookbackBatch; ++i) v[i] = row[size_t(min(p + i, blk - 1u)) * row_stride];
                #pragma unroll
                for (uint32_t i = 0; i < kLookbackBatch; ++i) {
                    if (p + i >= blk) continue;
                    while (!(v[i] & kRowPublished) && ++polls < kLookbackPolls) v[i] = row[size_t(p + i) * row_stride];
                    failed |= !(v[i] & kRowPublished);
                    before += v[i] & ~kRowPublished;
                }
            }
            volatile unsigned long long* sums = groups + d;
            if (closes_group) sums[size_t(group) << bits] = kGroupAggregate | (before + running);
            bool done = false;
            for (uint32_t p = group; p > 0 && !done;) {
                const uint32_t step = min(uint32_t(kLookbackBatch), p);
                unsigned long long v[kLookbackBatch];
                #pragma unroll
                for (uint32_t i = 0; i < kLookbackBatch; ++i) v[i] = sums[size_t(p - 1u - (i < step ? i : 0u)) << bits];
                #pragma unroll
                for (uint32_t i = 0; i < kLookbackBatch; ++i) {
                    if (done || i >= step) continue;
                    while ((v[i] >> 62) == 0ull && ++polls < kLookbackPolls) v[i] = sums[size_t(p - 1u - i) << bits];
                    if ((v[i] >> 62) == 0ull) { failed = true; done = true; continue; }
                    before += v[i] & kGroupValue;
                    if (v[i] & kGroupPrefix) done = true;
                }
                p -= step;
            }
            if (closes_group) sums[size_t(group) << bits] = kGroupPrefix | ((before + running) & kGroupValue);
            if (failed) s_failed = 1;
            global_base[d] = digit_base[d] + uint32_t(before);
        }
        __syncthreads();
        uint32_t prim[kSortItems];
        #pragma unroll
        for (int r = 0; r < kSortItems; ++r) {
            const uint32_t idx = base + r * 32 + lane;
            prim[r] = idx < n ? __ldg(prims_in + idx) : 0u;
        }
        block_exclusive_scan_512(block_excl, n_bins, warp_tot);
        const bool failed = s_failed != 0;
        // local stable placement
        #pragma unroll
        for (int r = 0; r < kSortItems; ++r) {
            const uint32_t d = digit_of(key_of(r), shift, mask);
            rank[r] += (block_excl[d] + mine[d].y) << (kPacked ? 16 : 0);
        }
        __syncthreads();                  // the masks and counts are no longer needed
        for (uint32_t d = threadIdx.x; d < n_bins; d += kSortThreads) global_base[d] -= block_excl[d];
        #pragma unroll
        for (int r = 0; r < kSortItems; ++r) {
            if (base + r * 32 + lane < n) {
                const uint32_t at = kPacked ? rank[r] >> 16 : rank[r];
                keys_s[at] = key_of(r);
                prims_s[at] = prim[r];
            }
        }
        __syncthreads();
        const uint32_t in_block = min(uint32_t(kSortTile), n - blk * kSortTile);
        if (!failed) {
            #pragma unroll
            for (int i = 0; i < kSortItems; ++i) {
                const uint32_t j = i * kSortThreads + threadIdx.x;
                if (j < in_block) {
                    const KeyT k = keys_s[j];
                    const uint32_t dst = global_base[digit_of(k, shift, mask)] + j;
                    keys_out[dst] = k;
                    prims_out[dst] = prims_s[j];
                }
            }
        }
        __syncthreads();
    }
    if (threadIdx.x == 0 && s_failed) atomicOr(&status->error, 2u);
}

template <typename KeyT> constexpr size_t scatter_smem_bytes(int bits = kMaxRadixBits) {
    const size_t n_bins = size_t(1) << bits, table = kSortWarps * n_bins * sizeof(uint2), staging = kSortTile * (sizeof(uint32_t) + sizeof(KeyT));
    return (3 * n_bins + (bits == 1 ? 2 : 0)) * sizeof(uint32_t) + (table > staging ? table : staging);
}

// Tiles by the length of their lists, longest first, in half-octave classes: blocks start in this order, so that the long lists do
// not end up as the tail of a launch.  Inside a class the order is that of the image up to a few thousand tiles, which keeps
// tiles that share Gaussians together in time.  Run by one block of 1024 threads.
constexpr int kOrderThreads = 1024;
__device__ __forceinline__ void order_tiles(const uint2* ranges, uint32_t* order, uint32_t n_tiles) {
    __shared__ uint32_t start[kOrderClasses];
    constexpr int kUnroll = 4;
    if (threadIdx.x < kOrderClasses) start[threadIdx.x] = 0;
    __syncthreads();
    #pragma unroll
    for (int pass = 0; pass < 2; ++pass) {
        for (uint32_t base = 0; base < n_tiles; base += kOrderThreads * kUnroll) {
            uint2 r[kUnroll];
            #pragma unroll
            for (int i = 0; i < kUnroll; ++i) {
                const uint32_t t = base + i * kOrderThreads + threadIdx.x;
                r[i] = t < n_tiles ? __ldcg(ranges + t) : make_uint2(0u, 0u);
            }
            #pragma unroll
            for (int i = 0; i < kUnroll; ++i) {
                const uint32_t t = base + i * kOrderThreads + threadIdx.x;
                const bool valid = t < n_tiles;
                const uint32_t c = order_class(r[i].y - r[i].x);
                // one shared-memory atomic per class and warp
                const uint32_t same = __match_any_sync(0xffffffffu, valid ? c : 0xffffffffu);
                const int leader = __ffs(same) - 1;
                uint32_t at = 0;
                if (valid && int(threadIdx.x & 31u) == leader) at = atomicAdd(&start[c], uint32_t(__popc(same)));
                at = __shfl_sync(0xffffffffu, at, leader) + __popc(same & lanemask_lt());
                if (pass == 1 && valid) order[at] = t;
            }
        }
        __syncthreads();
        if (pass == 0) {
            if (threadIdx.x < 32) {
                const uint32_t a = start[2 * threadIdx.x], b = start[2 * threadIdx.x + 1];
                const uint32_t inc = warp_inclusive_scan(a + b);
                start[2 * threadIdx.x] = inc - a - b;
                start[2 * threadIdx.x + 1] = inc - b;
            }
            __syncthreads();
        }
    }
}

// Tile ranges from the sorted keys (rasterization/src/shared_kernels.cu:56-95); ranges were zeroed before.
// A thread takes kRangeRun consecutive keys with one 16-byte load (plus the key in front of them), so the sorted keys
// are read once, in full sectors, and a thread has all its loads in flight before its first comparison.
template <typename KeyT>
__global__ void __launch_bounds__(kOrderThreads) tile_ranges_kernel(const KeyT* __restrict__ keys, uint2* __restrict__ ranges, uint32_t* __restrict__ order,
                                                                    FrameStatus* status, uint32_t capacity, uint32_t n_tiles) {
    grid_dependency();
    constexpr uint32_t kRangeRun = 16 / sizeof(KeyT);            // 8 or 4 keys per 16-byte load
    const uint32_t n = frame_instances(status, capacity);
    const uint32_t n_runs = (n + kRangeRun - 1) / kRangeRun;
    for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < n_runs; r += gridDim.x * blockDim.x) {
        const uint32_t first = r * kRangeRun;
        KeyT k[kRangeRun];
        if (first + kRangeRun <= n) {
            const uint4 raw = __ldg(reinterpret_cast<const uint4*>(keys + first));      // the key buffers are 256-byte aligned
            __builtin_memcpy(k, &raw, 16);
        } else {
            #pragma unroll
            for (uint32_t i = 0; i < kRangeRun; ++i) k[i] = first + i < n ? keys[first + i] : KeyT(0);
        }
        uint32_t prev = first ? uint32_t(keys[first - 1]) : 0xffffffffu;
        #pragma unroll
        for (uint32_t i = 0; i < kRangeRun; ++i) {
            const uint32_t at = first + i;
            if (at < n) {
                const uint32_t tile = uint32_t(k[i]);
                if (at == 0) ranges[tile].x = 0;
                else if (prev != tile) { ranges[prev].y = at; ranges[tile].x = at; }
                if (at == n - 1) ranges[tile].y = n;
                prev = tile;
            }
        }
    }
    __shared__ bool is_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) is_last = atomicAdd(&status->range_blocks_done, 1u) == gridDim.x - 1u;
    __syncthreads();
    if (is_last) {
        __threadfence();
        order_tiles(ranges, order, n_tiles);
        if (threadIdx.x == 0) status->range_blocks_done = 0;      // htgs_forward_finish may be called again on this status
    }
}

// Visible Gaussians of a GLOBAL_ORDERING frame in index order, with the bits of their depth as keys: the input of the sort by depth.
__global__ void __launch_bounds__(kPreprocessBlock) list_visible_kernel(const uint32_t* __restrict__ n_touched, const EvalRecord* __restrict__ eval, const uint32_t* __restrict__ visible_offsets,
                                                                        uint32_t* __restrict__ keys, uint32_t* __restrict__ prims, uint32_t n_primitives, uint32_t lowest_key,
                                                                        uint32_t capacity, const FrameStatus* __restrict__ status, const __grid_constant__ ClearList clear) {
    grid_dependency();
    const uint32_t idx = blockIdx.x * kPreprocessBlock + threadIdx.x, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const bool visible = idx < n_primitives && n_touched[idx] != 0;
    const uint32_t instances = frame_instances(status, capacity);
    clear_words(clear, instances);
    if (instances == 0) return;
    __shared__ uint32_t warp_tot[kPreprocessBlock / 32];
    const uint32_t ballot = __ballot_sync(0xffffffffu, visible);
    if (lane == 0) warp_tot[warp] = __popc(ballot);
    __syncthreads();
    if (!visible) return;
    uint32_t at = visible_offsets[blockIdx.x] + __popc(ballot & lanemask_lt());
    #pragma unroll
    for (int w = 0; w < kPreprocessBlock / 32; ++w) if (w < int(warp)) at += warp_tot[w];
    if (at >= capacity) return;
    keys[at] = __float_as_uint(eval[idx].mt3.w) - lowest_key;
    prims[at] = idx;
}

// Instances of every 256 of them, once they are in depth order, and of every 256 such blocks.
__global__ void __launch_bounds__(kPreprocessBlock) sum_sorted_kernel(const uint32_t* __restrict__ list, const uint32_t* __restrict__ n_touched, uint32_t* __restrict__ block_sums,
                                                                      uint32_t* __restrict__ group_sums, uint32_t capacity, const FrameStatus* __restrict__ status) {
    grid_dependency();
    const uint32_t n = frame_instances(status, capacity, true), i = blockIdx.x * kPreprocessBlock + threadIdx.x;
    if (blockIdx.x * kPreprocessBlock >= n) return;
    __shared__ uint32_t warp_tot[kPreprocessBlock / 32];
    const uint32_t sum = __reduce_add_sync(0xffffffffu, i < n ? n_touched[list[i]] : 0u);
    if ((threadIdx.x & 31u) == 0) warp_tot[threadIdx.x >> 5] = sum;
    __syncthreads();
    if (threadIdx.x != 0) return;
    uint32_t total = 0;
    #pragma unroll
    for (int w = 0; w < kPreprocessBlock / 32; ++w) total += warp_tot[w];
    block_sums[blockIdx.x] = total;
    atomicAdd(group_sums + blockIdx.x / kSumGroup, total);
}

__global__ void __launch_bounds__(256) global_keys_kernel(const uint2* __restrict__ ranges, const uint32_t* __restrict__ prims, const EvalRecord* __restrict__ eval,
                                                          unsigned long long* __restrict__ keys, const FrameStatus* __restrict__ status) {
    if (status->overflow || status->error) return;
    const uint2 range = ranges[blockIdx.x];
    for (uint32_t i = range.x + threadIdx.x; i < range.y; i += 256) keys[i] = (static_cast<unsigned long long>(blockIdx.x) << 32) | __float_as_uint(eval[prims[i]].mt3.w);
}

// The passes over `passes`: histogram, then one scatter each, from buffer 0 to buffer n_passes & 1.
template <typename KeyT>
cudaError_t launch_radix_sort(const PassTable& passes, KeyT* const (&keys)[2], uint32_t* const (&prims)[2], uint32_t* digit_hist, uint32_t* const* rows, uint32_t row_stride,
                              unsigned long long* const* groups, uint32_t* tickets, const InstBuffers& inst, uint32_t most_sort_blocks, FrameStatus* status, int sm_count,
                              cudaStream_t stream, uint32_t* launches) {
    static PerDeviceOnce configured;
    const cudaError_t err = configured.run([] { return cudaFuncSetAttribute(radix_scatter_kernel<KeyT>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(scatter_smem_bytes<KeyT>())); });
    if (err != cudaSuccess || passes.n_passes == 0) return err;
    const uint32_t hist_grid = std::min<uint32_t>(std::max(most_sort_blocks, 1u), uint32_t(sm_count) * 8u);
    launch_after(radix_histogram_all_kernel<KeyT>, hist_grid, 256, 0, stream, keys[0], digit_hist, status, inst.capacity, passes);
    for (int p = 0; p < passes.n_passes; ++p) {
        const size_t smem = scatter_smem_bytes<KeyT>(passes.bits[p]);
        const uint32_t resident = uint32_t(std::min<size_t>(scatter_blocks_per_sm<KeyT>(), (227 * 1024) / (smem + 1024)));
        const uint32_t scatter_grid = std::min<uint32_t>(std::max(most_sort_blocks, 1u), uint32_t(sm_count) * resident);
        launch_after(radix_scatter_kernel<KeyT>, scatter_grid, kSortThreads, smem, stream, keys[p & 1], prims[p & 1], keys[(p & 1) ^ 1], prims[(p & 1) ^ 1], digit_hist + size_t(p) * kMaxRadixBins,
                     rows[p], row_stride, groups[p], tickets + p, status, inst.capacity, passes.shift[p], passes.bits[p], passes.visible);
    }
    if (launches) *launches += 1u + uint32_t(passes.n_passes);
    return cudaSuccess;
}

PassTable tile_passes(const SortPlan& plan) {
    PassTable t{};
    t.n_passes = plan.n_passes;
    for (int p = 0; p < plan.n_passes; ++p) { t.shift[p] = plan.shift[p]; t.bits[p] = plan.bits[p]; }
    return t;
}

ClearList clear_list(const SortScratch& sc, const FrameGeometry& geo, uint2* tile_ranges) {
    ClearList clear{};      // the buffers are 256-byte aligned and padded to 256 bytes
    clear.begin[0] = reinterpret_cast<uint4*>(tile_ranges); clear.count[0] = (uint64_t(geo.n_tiles) + 1) / 2;
    if (sc.row_stride > 0) {
        clear.begin[1] = reinterpret_cast<uint4*>(sc.tickets); clear.count[1] = sc.fixed_bytes / 16;
        clear.begin[2] = reinterpret_cast<uint4*>(reinterpret_cast<unsigned char*>(sc.tickets) + sc.fixed_bytes); clear.per_sort_block[2] = sc.row_stride / 4;
    }
    return clear;
}

// A frame without Gaussians or without room for instances.
template <typename KeyT>
cudaError_t empty_ranges(const FrameGeometry& geo, const InstBuffers& inst, uint2* tile_ranges, uint32_t* tile_order, FrameStatus* status, cudaStream_t stream, cudaEvent_t* ev, uint32_t* launches) {
    const cudaError_t err = cudaMemsetAsync(tile_ranges, 0, sizeof(uint2) * size_t(geo.n_tiles), stream);
    if (err != cudaSuccess) return err;
    if (ev) { cudaEventRecord(ev[0], stream); cudaEventRecord(ev[1], stream); }
    launch_after(tile_ranges_kernel<KeyT>, 1, kOrderThreads, 0, stream, static_cast<const KeyT*>(inst.keys[0]), tile_ranges, tile_order, status, 0u, uint32_t(geo.n_tiles));
    if (ev) cudaEventRecord(ev[2], stream);
    if (launches) *launches += 1;
    return cudaGetLastError();
}

template <typename KeyT>
cudaError_t emit_sort_ranges_t(const HtgsScene& scene, const FrameGeometry& geo, const SortPlan& plan, const PrimBuffers& prim, const InstBuffers& inst,
                               uint2* tile_ranges, uint32_t* tile_order, FrameStatus* status, int sm_count, cudaStream_t stream, cudaEvent_t* ev, uint32_t* launches) {
    const uint32_t n = uint32_t(scene.n_primitives);
    const uint32_t prim_blocks = (n + kPreprocessBlock - 1) / kPreprocessBlock;
    if (prim_blocks == 0 || inst.capacity == 0) return empty_ranges<KeyT>(geo, inst, tile_ranges, tile_order, status, stream, ev, launches);
    const SortScratch sc = carve_sort_scratch(inst.sort_scratch, plan, inst.sort_blocks_cap, 0);
    KeyT* const keys[2] = {static_cast<KeyT*>(inst.keys[0]), static_cast<KeyT*>(inst.keys[1])};
    launch_after(emit_instances_kernel<KeyT, false>, prim_blocks, kPreprocessBlock, 0, stream,
        prim.n_touched, prim.bounds, nullptr, prim.block_sums, prim.block_offsets, nullptr, keys[0], inst.prims[0], n,
        uint32_t(geo.grid_w), inst.capacity, status, clear_list(sc, geo, tile_ranges));
    if (ev) cudaEventRecord(ev[0], stream);
    if (launches) *launches += 1;
    const cudaError_t err = launch_radix_sort<KeyT>(tile_passes(plan), keys, inst.prims, sc.digit_hist, sc.rows, uint32_t(sc.row_stride), sc.groups, sc.tickets, inst, inst.sort_blocks_cap,
                                                    status, sm_count, stream, launches);
    if (err != cudaSuccess) return err;
    if (ev) cudaEventRecord(ev[1], stream);
    launch_after(tile_ranges_kernel<KeyT>, uint32_t(sm_count), kOrderThreads, 0, stream, keys[plan.final_buffer], tile_ranges, tile_order, status, inst.capacity, uint32_t(geo.n_tiles));
    if (ev) cudaEventRecord(ev[2], stream);
    if (launches) *launches += 1;
    return cudaGetLastError();
}

// GLOBAL_ORDERING: the lists are in order of depth, Gaussians of equal depth in order of their index.  The reference sorts the instances by 64-bit keys
// of tile and depth (alpha_blend_global_ordering/inference.cu:40-110); a Gaussian's instances share its depth, so here the visible Gaussians are
// sorted by depth, then their instances are emitted in that order and sorted by tile alone.  Both sorts are stable, so the lists are the same:
// four passes over a third of the Gaussians and two over 16-bit keys take the place of five or six over 64-bit keys.
// 1.5 M Gaussians, 980 x 545, 2.8 M instances, scan to ranges: 259 -> 189 us (four passes of 7 bits; three of 9: 195).
//
// The key buffers (8 bytes an instance, of which the sorts by tile need 2 or 4) hold everything in turn: keys[0] and keys[1] the depth keys and, in
// their second halves, the Gaussians; the sorted list stays in one of them, with the sums over its blocks in the first half, and the tile keys take both
// halves of the other.  What the scan left in the per-Gaussian buffers is only read: htgs_forward_finish may be called again on them.
template <typename KeyT>
cudaError_t emit_sort_ranges_global(const HtgsScene& scene, const HtgsView& view, const FrameGeometry& geo, const SortPlan& plan, const PrimBuffers& prim, const InstBuffers& inst,
                                    uint2* tile_ranges, uint32_t* tile_order, FrameStatus* status, int sm_count, cudaStream_t stream, cudaEvent_t* ev, uint32_t* launches) {
    const uint32_t n = uint32_t(scene.n_primitives);
    const uint32_t prim_blocks = (n + kPreprocessBlock - 1) / kPreprocessBlock;
    if (prim_blocks == 0 || inst.capacity == 0) return empty_ranges<KeyT>(geo, inst, tile_ranges, tile_order, status, stream, ev, launches);
    // The centres of visible Gaussians lie between the planes (preprocess.cu), so with a positive near plane the distance of their bits from those of
    // the near plane is all that has to be sorted: 27 bits for 0.2 to 1000.  Otherwise all 32 bits, as the unsigned numbers that the reference's keys hold.
    int32_t near_bits, far_bits;
    std::memcpy(&near_bits, &view.near_plane, 4);
    std::memcpy(&far_bits, &view.far_plane, 4);
    const bool window = near_bits > 0 && far_bits >= near_bits && far_bits <= 0x7f800000;
    PassTable depth{};
    const int depth_bits = window ? std::max(bit_length(uint32_t(far_bits - near_bits)), 1) : 32;
    // Digits: the fewest passes while a pass is mostly latency, shorter digits, whose look-back and ranking are cheaper per sort block, once the sort
    // blocks fill the GPU.  27 bits, three passes of 9 against four of 7 (kernels alone): 16 k Gaussians 31 us against 37, 400 k 42 / 47, 1 M (166 k visible) 51 / 54,
    // 3 M 74 / 74, 1.5 M (628 k visible) 114 / 103, 8 M 95 / 83.  How many are visible the host does not know.
    const uint32_t most_visible = std::min(n, inst.capacity), visible_blocks = (most_visible + kPreprocessBlock - 1) / kPreprocessBlock;
    depth.n_passes = split_digits(depth_bits, depth.bits, depth.shift, most_visible <= (1u << 19) ? kMaxRadixBits : depth_bits <= 28 ? 7 : 8);
    depth.visible = true;
    size_t depth_words = 0;
    for (int p = 0; p < depth.n_passes; ++p) depth_words += size_t(1) << depth.bits[p];
    const SortScratch sc = carve_sort_scratch(inst.sort_scratch, plan, inst.sort_blocks_cap, depth_words);
    uint32_t* depth_rows[4];
    unsigned long long* depth_groups[4];
    const size_t n_groups = (size_t(inst.sort_blocks_cap) + kGroup - 1) / kGroup;
    for (int p = 0, at = 0; p < depth.n_passes; at += 1 << depth.bits[p], ++p) { depth_rows[p] = sc.depth_rows + at; depth_groups[p] = sc.depth_groups + n_groups * size_t(at); }
    uint32_t* const depth_keys[2] = {static_cast<uint32_t*>(inst.keys[0]), static_cast<uint32_t*>(inst.keys[1])};
    uint32_t* const depth_prims[2] = {depth_keys[0] + inst.capacity + 4, depth_keys[1] + inst.capacity + 4};
    launch_after(list_visible_kernel, prim_blocks, kPreprocessBlock, 0, stream, prim.n_touched, prim.eval, prim.block_offsets, depth_keys[0], depth_prims[0], n,
                 window ? uint32_t(near_bits) : 0u, inst.capacity, status, clear_list(sc, geo, tile_ranges));
    cudaError_t err = launch_radix_sort<uint32_t>(depth, depth_keys, depth_prims, sc.digit_hist + size_t(kFirstDepthPass) * kMaxRadixBins, depth_rows, uint32_t(sc.row_stride), depth_groups,
                                                  sc.tickets + kFirstDepthPass, inst, (most_visible + kSortTile - 1) / kSortTile, status, sm_count, stream, launches);
    if (err != cudaSuccess) return err;
    const uint32_t* list = depth_prims[depth.n_passes & 1];
    uint32_t* const sorted_sums = depth_keys[depth.n_passes & 1];       // the sorted depths have done their work: capacity + 4 words for one per 256 visible Gaussians
    unsigned char* free_buffer = static_cast<unsigned char*>(inst.keys[(depth.n_passes & 1) ^ 1]);
    KeyT* const keys[2] = {reinterpret_cast<KeyT*>(free_buffer), reinterpret_cast<KeyT*>(free_buffer + align16(size_t(inst.capacity) * 4))};
    launch_after(sum_sorted_kernel, visible_blocks, kPreprocessBlock, 0, stream, list, prim.n_touched, sorted_sums, sc.group_sums, inst.capacity, status);
    launch_after(emit_instances_kernel<KeyT, true>, visible_blocks, kPreprocessBlock, 0, stream, prim.n_touched, prim.bounds, list, sorted_sums, nullptr, sc.group_sums, keys[0], inst.prims[0], n,
                 uint32_t(geo.grid_w), inst.capacity, status, ClearList{});
    if (launches) *launches += 3;
    if (ev) cudaEventRecord(ev[0], stream);
    if ((err = launch_radix_sort<KeyT>(tile_passes(plan), keys, inst.prims, sc.digit_hist, sc.rows, uint32_t(sc.row_stride), sc.groups, sc.tickets, inst, inst.sort_blocks_cap,
                                       status, sm_count, stream, launches)) != cudaSuccess) return err;
    if (ev) cudaEventRecord(ev[1], stream);
    launch_after(tile_ranges_kernel<KeyT>, uint32_t(sm_count), kOrderThreads, 0, stream, keys[plan.final_buffer], tile_ranges, tile_order, status, inst.capacity, uint32_t(geo.n_tiles));
    if (ev) cudaEventRecord(ev[2], stream);
    if (launches) *launches += 1;
    return cudaGetLastError();
}

}  // namespace

size_t sort_scratch_bytes(const SortPlan& plan, uint32_t sort_blocks_cap) { return carve_sort_scratch(nullptr, plan, sort_blocks_cap, plan.key_bytes == 8 ? kMostDepthWords : 0).bytes; }

cudaError_t launch_scan_only(int mode, const HtgsScene& scene, const PrimBuffers& prim, uint32_t capacity, FrameStatus* status, cudaStream_t stream) {
    const uint32_t n = uint32_t(scene.n_primitives);
    const uint32_t prim_blocks = (n + kPreprocessBlock - 1) / kPreprocessBlock;
    const auto kernel = mode == HTGS_MODE_ALPHA_BLEND_GLOBAL_ORDERING ? scan_block_sums_kernel<ScanOf::visible> : scan_block_sums_kernel<ScanOf::instances>;
    launch_after(kernel, 1, kScanThreads, 0, stream, prim.block_sums, prim.block_offsets, prim_blocks, capacity, status);
    return cudaGetLastError();
}

cudaError_t launch_emit_sort_ranges(const HtgsScene& scene, const HtgsView& view, const FrameGeometry& geo, const SortPlan& plan, const PrimBuffers& prim,
                                    const InstBuffers& inst, uint2* tile_ranges, uint32_t* tile_order, FrameStatus* status, int sm_count, cudaStream_t stream,
                                    cudaEvent_t* stage_events, uint32_t* launches) {
    switch (plan.key_bytes) {
        case 2: return emit_sort_ranges_t<uint16_t>(scene, geo, plan, prim, inst, tile_ranges, tile_order, status, sm_count, stream, stage_events, launches);
        case 4: return emit_sort_ranges_t<uint32_t>(scene, geo, plan, prim, inst, tile_ranges, tile_order, status, sm_count, stream, stage_events, launches);
        case 8:
            return plan.end_bit <= 32 + 16 ? emit_sort_ranges_global<uint16_t>(scene, view, geo, plan, prim, inst, tile_ranges, tile_order, status, sm_count, stream, stage_events, launches)
                                           : emit_sort_ranges_global<uint32_t>(scene, view, geo, plan, prim, inst, tile_ranges, tile_order, status, sm_count, stream, stage_events, launches);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_global_keys(const FrameGeometry& geo, const SortPlan& plan, const PrimBuffers& prim, const InstBuffers& inst, const uint2* tile_ranges, const FrameStatus* status,
                               cudaStream_t stream) {
    global_keys_kernel<<<uint32_t(geo.n_tiles), 256, 0, stream>>>(tile_ranges, inst.prims[plan.final_buffer], prim.eval, static_cast<unsigned long long*>(inst.keys[0]), status);
    return cudaGetLastError();
}

}  // namespace htgs
