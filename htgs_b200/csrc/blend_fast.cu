// Relaxed-precision inference for HYBRID_BLEND, ALPHA_BLEND_FIRST_K and OIT_BLEND: the kernels behind fast_rasterize.
//
// Replaces blend_cu of rasterization/include/{hybrid_blend,alpha_blend_first_k,oit_blend}/kernels/fast_inference.cuh
// (the reference's fast-math build; HYBRID keeps a half-precision K-buffer; RGB only, no depth output).  Results agree with that kernel to
// about 1e-3 per channel, not bit for bit: this path trades the operation-for-operation evaluation of the
// exact kernel (blend.cu) for fewer instructions per fragment.
//
//  * The organisation is that of the exact kernel (blend.cu): a warp per 8 x 4 pixels filters its tile's list, keeps a window of two
//    halves of 16 records that its lanes walk independently, and long lists start first.  Against a CTA per 8 x 8 tile with
//    masks by ballots and a barrier every 64 instances: 944 -> 820 us at 3 M Gaussians, 1297 x 840, K = 16.
//  * Per fragment, rho^2 and depth are ratios of quadratics in (pixel - projected centre) whose coefficients the
//    preprocess stored per Gaussian (FastRecord): 6 shared-memory loads, 20 multiply-adds, one approximate
//    reciprocal and one approximate exp2 instead of two plane constructions, two cross products, an IEEE divide
//    and expf.  The rho^2 cutoff test is implied by the alpha test (opacity <= 1) and dropped.
//  * K-buffer.  The K nearest core fragments of a pixel are kept UNSORTED in shared memory: one key per entry (the
//    fragment depth with its low log2(K) mantissa bits replaced by the entry's position, so the largest key names
//    the entry to evict) and a half-precision premultiplied RGBA payload (as the reference's fast path stores it).
//    An insertion overwrites the entry of the largest key, re-reads the one row of four keys that changed and
//    updates the per-row maxima it keeps in registers: about 20 ALU-pipe instructions and 9 shared-memory wavefronts
//    instead of 5 instructions per level of a sorted chain.
//    Entries are sorted once per pixel when the tile is composited.  Fragments of exactly equal depth are ordered by
//    position instead of by arrival.  FIRST_K uses the same buffer with (alpha, Gaussian index) payloads and no tail;
//    OIT has no buffer at all and skips the depth polynomial.
#include "kernels.h"

#include <cuda_fp16.h>


namespace htgs {

namespace {

constexpr int kFastThreads = 32;     // 8 x 4 pixels, one thread per pixel
constexpr int kFastHalf = 16;        // records per half of the window
constexpr int kFastQueue = 64;       // survivors of the filter that wait for a place
// pixels of 32 from which on a record is evaluated by all lanes together.  12: 1030 us, 16: 1022, 20: 1015, 24: 1012, 28: 1017 (3 M Gaussians, 1297 x 840, K = 16; 0.5 M, 3127 x
// 1880: 1745, 1748, 1740, 1726, 1733): lanes that walk their own records read each one's rows again, all together they also evaluate where it does not reach.
constexpr int kFastDense = 20;

// HYBRID: candidates that a lane evaluates per trip.  3 M Gaussians, 1297 x 840, and 4 M in dense clusters, 1920 x 1080, two and three: K = 4 221 and 221 us, 3.79 and 3.80 ms;
// K = 8 250 and 252, 4.13 and 4.15; K = 16 317 and 301, 5.03 and 4.70 (four: 307, 4.71); K = 32 455 and 481, 6.61 and 6.89.  K = 32 stays with three all the same: how far a lane
// is ahead decides between entries whose keys agree but for the depth bits that the position takes, so with two some pixels differ by up to 1e-3, also under
// htgs_set_fast_deterministic.
constexpr int kFastPerTrip = 3;

template <int MODE, int K> struct FastSmem {
    static constexpr bool has_kbuffer = MODE != HTGS_MODE_OIT_BLEND;
    static constexpr bool has_prim = MODE == HTGS_MODE_ALPHA_BLEND_FIRST_K;
    static constexpr size_t rec_off = 0;
    static constexpr size_t keys_off = rec_off + 2 * kFastHalf * sizeof(FastRecord);
    static constexpr size_t keys_bytes = has_kbuffer ? size_t(K) * kFastThreads * 4 : 0;     // uint4 [K/4][threads]
    static constexpr size_t pay_off = keys_off + keys_bytes;
    static constexpr size_t pay_bytes = has_kbuffer ? size_t(K) * kFastThreads * 8 : 0;      // 8-byte payload [K][threads]
    static constexpr size_t ctr_off = pay_off + pay_bytes;                                   // float2 per record: projected centre relative to the tile's origin
    static constexpr size_t prim_off = ctr_off + 2 * kFastHalf * 8;                          // Gaussian index of every record (FIRST_K)
    static constexpr size_t queue_ctr_off = prim_off + (has_prim ? 2 * kFastHalf * 4 : 0);
    static constexpr size_t queue_prim_off = queue_ctr_off + kFastQueue * 8;
    static constexpr size_t queue_mask_off = queue_prim_off + kFastQueue * 4;
    // the same for dense records: staged, and waiting
    static constexpr size_t dense_rec_off = queue_mask_off + kFastQueue * 4;
    static constexpr size_t dense_ctr_off = dense_rec_off + kFastHalf * sizeof(FastRecord);
    static constexpr size_t dense_mask_off = dense_ctr_off + kFastHalf * 8;
    static constexpr size_t dense_prim_off = dense_mask_off + kFastHalf * 4;
    static constexpr size_t dense_queue_ctr_off = dense_prim_off + (has_prim ? kFastHalf * 4 : 0);
    static constexpr size_t dense_queue_prim_off = dense_queue_ctr_off + kFastQueue * 8;
    static constexpr size_t dense_queue_mask_off = dense_queue_prim_off + kFastQueue * 4;
    static constexpr size_t bar_off = dense_queue_mask_off + kFastQueue * 4;
    static constexpr size_t total = bar_off + 3 * 8;
    static_assert(bar_off % 8 == 0 && keys_off % 16 == 0 && dense_rec_off % 16 == 0, "shared-memory sections must stay 16-byte aligned");
};

__device__ __forceinline__ float rcp_approx(float x) { float y; asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
__device__ __forceinline__ float exp2_approx(float x) { float y; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }

// maximum of N keys as a tree of three-input max
template <int N>
__device__ __forceinline__ uint32_t reduce_max(const uint32_t (&v)[N]) {
    if constexpr (N == 1) return v[0];
    else if constexpr (N == 2) return max(v[0], v[1]);
    else {
        constexpr int M = N / 3 + N % 3;
        uint32_t r[M];
        #pragma unroll
        for (int i = 0; i < N / 3; ++i) r[i] = __vimax3_u32(v[3 * i], v[3 * i + 1], v[3 * i + 2]);
        #pragma unroll
        for (int i = 0; i < N % 3; ++i) r[N / 3 + i] = v[3 * (N / 3) + i];
        return reduce_max<M>(r);
    }
}

// Core keys: 32-bit unsigned, ordered like the depth, carrying the entry's position in the low log2(K) bits.
// The depth keeps its full 23-bit mantissa; the exponent is re-based to a window of 2^(9 - log2 K) binades starting
// at 2^kMinExp (K = 16: [2^-12, 2^20), K = 32: [2^-4, 2^12)); depths outside the window (or negative) saturate, which
// only loses the order among fragments that all lie outside it.
template <int K> struct KeyCodec {
    static constexpr int pos_bits = K == 4 ? 2 : K == 8 ? 3 : K == 16 ? 4 : 5;
    static constexpr int exp_bits = 9 - pos_bits;
    static constexpr int min_exp = K == 32 ? -4 : -12;
    static constexpr int32_t base = int32_t(127 + min_exp) << 23;
    static constexpr int32_t limit = int32_t((1u << (23 + exp_bits)) - 1u);
    static __device__ __forceinline__ uint32_t encode(float depth, uint32_t pos) {
        const int32_t rel = min(max(__float_as_int(depth) - base, 0), limit);
        return uint32_t(rel) * uint32_t(K) + pos;
    }
    static __device__ __forceinline__ float decode(uint32_t key) { return __int_as_float(int32_t(key >> pos_bits) + base); }
    static constexpr uint32_t empty = 0xffffffffu & ~uint32_t(K - 1);
};

__device__ __forceinline__ uint2 pack_half4(float x, float y, float z, float w) {
    const __half2 a = __floats2half2_rn(x, y), b = __floats2half2_rn(z, w);
    return make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
}
__device__ __forceinline__ float4 unpack_half4(uint2 p) {
    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&p.x));
    const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&p.y));
    return make_float4(a.x, a.y, b.x, b.y);
}

// Replace the entry with the largest key by (depth, payload); returns the payload that fell out (zeros for an
// entry that was still empty).  Entry c keeps its key in component (c & 3) of uint4 row (c >> 2).  Registers hold
// the maximum of every row (`row_max`), so that only the row that changed is read back: one vector load instead
// of K/4 (shared-memory bandwidth is what bounds this kernel).
template <int K>
__device__ __forceinline__ uint2 core_replace(uint32_t* keys, uint2* pay, uint32_t tid, float depth, uint2 payload, uint32_t (&row_max)[K / 4],
                                              uint32_t& kmax) {
    const uint32_t c = kmax & uint32_t(K - 1);
    uint2* slot = pay + c * kFastThreads + tid;
    const uint2 evicted = *slot;
    *slot = payload;
    const uint32_t q = c >> 2;
    uint4* row_ptr = reinterpret_cast<uint4*>(keys) + q * kFastThreads + tid;
    reinterpret_cast<uint32_t*>(row_ptr)[c & 3u] = KeyCodec<K>::encode(depth, c);
    const uint4 row = *row_ptr;
    const uint32_t m = max(__vimax3_u32(row.x, row.y, row.z), row.w);
    #pragma unroll
    for (int i = 0; i < K / 4; ++i) row_max[i] = (q == uint32_t(i)) ? m : row_max[i];
    kmax = reduce_max<K / 4>(row_max);
    return evicted;
}

template <int MODE, int K>
__global__ void __launch_bounds__(kFastThreads) blend_fast_kernel(
    const uint2* __restrict__ tile_ranges, const uint32_t* __restrict__ tile_order, const uint32_t* __restrict__ prims_sorted, const FastRecord* __restrict__ records,
    const CullRecord* __restrict__ cull, float* __restrict__ image, uint32_t width, uint32_t height, uint32_t grid_w, bool to_chw,
    FrameStatus* status)
{
    cudaGridDependencySynchronize();      // no launch_after kernel follows
    using SL = FastSmem<MODE, K>;
    using MT = ModeTraits<MODE>;
    constexpr bool kHybrid = MODE == HTGS_MODE_HYBRID_BLEND;
    constexpr bool kFirstK = MODE == HTGS_MODE_ALPHA_BLEND_FIRST_K;
    constexpr bool kOit = MODE == HTGS_MODE_OIT_BLEND;
    static_assert(kHybrid || kFirstK || kOit, "no relaxed-precision kernel for this mode");
    extern __shared__ __align__(128) unsigned char smem[];
    FastRecord* s_rec = reinterpret_cast<FastRecord*>(smem + SL::rec_off);
    float2* s_ctr = reinterpret_cast<float2*>(smem + SL::ctr_off);
    [[maybe_unused]] uint32_t* s_prim = reinterpret_cast<uint32_t*>(smem + SL::prim_off);
    float2* s_queue_ctr = reinterpret_cast<float2*>(smem + SL::queue_ctr_off);
    uint32_t* s_queue_prim = reinterpret_cast<uint32_t*>(smem + SL::queue_prim_off);
    uint32_t* s_queue_mask = reinterpret_cast<uint32_t*>(smem + SL::queue_mask_off);
    uint64_t* s_bar = reinterpret_cast<uint64_t*>(smem + SL::bar_off);
    [[maybe_unused]] uint32_t* keys = reinterpret_cast<uint32_t*>(smem + SL::keys_off);
    [[maybe_unused]] uint2* pay = reinterpret_cast<uint2*>(smem + SL::pay_off);

    const uint32_t tid = threadIdx.x, lane = tid;
    const uint32_t tile = __ldg(tile_order + blockIdx.x / 2), part = blockIdx.x % 2;
    const uint32_t tile_x = tile % grid_w, block_y = (tile / grid_w) * 2 + part;
    if (block_y * 4 >= height) return;
    const uint32_t px_i = tile_x * 8 + (tid & 7);
    const uint32_t py_i = block_y * 4 + (tid >> 3);
    const bool inside = px_i < width && py_i < height;
    // fragments are measured from the tile's origin (not the block's), so that both blocks of a tile round alike
    const float local_x = float(tid & 7), local_y = float((tid >> 3) + 4 * part), tile_y0 = float((tile / grid_w) * 8);
    const float block_x0 = float(tile_x * 8), block_y0 = float(block_y * 4);

    FastRecord* s_dense = reinterpret_cast<FastRecord*>(smem + SL::dense_rec_off);
    float2* s_dense_ctr = reinterpret_cast<float2*>(smem + SL::dense_ctr_off);
    uint32_t* s_dense_mask = reinterpret_cast<uint32_t*>(smem + SL::dense_mask_off);
    [[maybe_unused]] uint32_t* s_dense_prim = reinterpret_cast<uint32_t*>(smem + SL::dense_prim_off);
    if (lane < 3) mbar_init(s_bar + lane, 1);
    mbar_fence_init();

    // empty core: the largest keys, carrying their position; zero payloads (FIRST_K: alpha 0, no Gaussian)
    if constexpr (SL::has_kbuffer) {
        #pragma unroll
        for (int c = 0; c < K; ++c) {
            keys[((c >> 2) * kFastThreads + tid) * 4 + (c & 3)] = KeyCodec<K>::empty | uint32_t(c);
            pay[c * kFastThreads + tid] = make_uint2(0u, kFirstK ? 0xffffffffu : 0u);
        }
    }
    [[maybe_unused]] uint32_t row_max[K / 4];
    #pragma unroll
    for (int q = 0; q < K / 4; ++q) row_max[q] = KeyCodec<K>::empty | uint32_t(4 * q + 3);
    [[maybe_unused]] uint32_t kmax = 0xffffffffu;            // position K-1
    [[maybe_unused]] float depth_max = __int_as_float(0x7f800000);   // depth a fragment has to beat to enter the core
    float4 tail = make_float4(0.0f, 0.0f, 0.0f, 0.0f);       // HYBRID tail / OIT sums: premultiplied rgb, alpha sum
    float transmittance_tail = 1.0f;

    const uint2 range = tile_ranges[tile];
    bool wait_failed = false;

    uint32_t next = range.x + lane;                      // the instance this lane tests next
    uint32_t g_here = 0, g_ahead = 0;
    float4 c0 = make_float4(0.0f, 0.0f, 0.0f, 0.0f), c1 = c0;      // outline; c, cx_lo, cy_lo
    auto request_outline = [&](uint32_t g) {
        c0 = ldg4(reinterpret_cast<const float*>(cull + g));
        c1 = ldg4(reinterpret_cast<const float*>(cull + g) + 4);
    };
    if (next < range.y) { g_here = __ldg(prims_sorted + next); request_outline(g_here); }
    if (next + 32 < range.y) g_ahead = __ldg(prims_sorted + next + 32);
    // Survivors of the filter wait in two queues: those that touch many of the 32 pixels and the others.
    uint32_t sparse_head = 0, sparse = 0, dense_head = 0, dense = 0;
    auto filter = [&]() {
        uint32_t mask = 0;
        if (next < range.y) mask = outline_mask(c0, c1.x, block_x0, block_y0);
        const bool is_dense = __popc(mask) >= kFastDense;
        const uint32_t sparse_lanes = __ballot_sync(0xffffffffu, mask != 0 && !is_dense), dense_lanes = __ballot_sync(0xffffffffu, is_dense);
        if (mask != 0) {
            const uint32_t at = (is_dense ? dense_head + dense + __popc(dense_lanes & lanemask_lt()) : sparse_head + sparse + __popc(sparse_lanes & lanemask_lt())) & uint32_t(kFastQueue - 1);
            unsigned char* queue = smem + (is_dense ? SL::dense_queue_ctr_off : SL::queue_ctr_off);     // centres, indices, masks
            reinterpret_cast<float2*>(queue)[at] = make_float2((block_x0 - c0.x) - c1.y, (tile_y0 - c0.y) - c1.z);
            reinterpret_cast<uint32_t*>(queue + kFastQueue * 8)[at] = g_here;
            reinterpret_cast<uint32_t*>(queue + kFastQueue * 12)[at] = mask;
        }
        sparse += __popc(sparse_lanes);
        dense += __popc(dense_lanes);
        next += 32;
        g_here = g_ahead;
        if (next < range.y) request_outline(g_here);
        if (next + 32 < range.y) g_ahead = __ldg(prims_sorted + next + 32);
    };
    auto fill_queues = [&]() {
        while (sparse < kFastHalf && dense < kFastHalf && next - lane < range.y) filter();
        __syncwarp();
    };
    // The next `count` (<= kFastHalf) records of a queue into slots first - lane: index, centre and a copy under way.  Returns the lane's mask.
    auto stage = [&](size_t queue_off, uint32_t head, uint32_t count, uint32_t slot, FastRecord* rec, float2* ctr, uint32_t* prim, uint64_t* bar) -> uint32_t {
        uint32_t g = 0, mask = 0;
        if (lane < count) {
            const unsigned char* queue = smem + queue_off;
            const uint32_t at = (head + lane) & uint32_t(kFastQueue - 1);
            ctr[slot] = reinterpret_cast<const float2*>(queue)[at];
            g = reinterpret_cast<const uint32_t*>(queue + kFastQueue * 8)[at];
            mask = reinterpret_cast<const uint32_t*>(queue + kFastQueue * 12)[at];
            if constexpr (SL::has_prim) prim[slot] = g;
        }
        if (lane == 0) mbar_arrive_expect_tx(bar, count * uint32_t(sizeof(FastRecord)));
        __syncwarp();
        if (lane < count) bulk_copy_g2s(rec + slot, records + g, uint32_t(sizeof(FastRecord)), bar);
        return mask;
    };

    uint32_t window = 0;                                 // this pixel's candidates: bits 31..16 the older half, 15..0 the newer half
    uint32_t phases = 0;                                 // parity of each barrier
    uint32_t half = 0;
    fill_queues();
    for (;;) {
        const bool more = next - lane < range.y;
        const uint32_t n_dense = dense >= kFastHalf || !more ? min(dense, uint32_t(kFastHalf)) : 0u;
        const uint32_t n_sparse = sparse >= kFastHalf || !more ? min(sparse, uint32_t(kFastHalf)) : 0u;
        const bool step = n_sparse != 0 || (!more && __any_sync(0xffffffffu, window != 0));
        if (n_dense == 0 && !step) break;                // only with nothing left: otherwise a queue is full
        if (n_dense != 0) {
            const uint32_t mask = stage(SL::dense_queue_ctr_off, dense_head, n_dense, lane, s_dense, s_dense_ctr, s_dense_prim, s_bar + 2);
            if (lane < n_dense) s_dense_mask[lane] = mask;
            dense_head += n_dense;
            dense -= n_dense;
        }
        if (n_sparse != 0) {
            const uint32_t slot = half * kFastHalf + (uint32_t(kFastHalf) - 1u - (lane & uint32_t(kFastHalf - 1)));
            const uint32_t mine = transpose_masks(stage(SL::queue_ctr_off, sparse_head, n_sparse, slot, s_rec, s_ctr, s_prim, s_bar + half), lane);
            sparse_head += n_sparse;
            sparse -= n_sparse;
            if (inside) window |= mine;
        }
        fill_queues();
        if (n_sparse != 0) {
            if (!mbar_wait_bounded(s_bar + half, (phases >> half) & 1u)) wait_failed = true;
            phases ^= 1u << half;
            __syncwarp();
        }
        const uint32_t flip = half * kFastHalf;          // bit j of the window is record j ^ flip
        auto pop_candidate = [&](bool& valid) -> uint32_t {
            valid = window != 0;
            const uint32_t j = uint32_t(31 - __clz(int(window | 1u)));
            window &= ~(1u << j);
            return j ^ flip;
        };
        auto evaluate = [&](const FastRecord* record, float2 ctr, float& depth, float4& frag) {
            const float4* rec = reinterpret_cast<const float4*>(record);
            const float4 r0 = rec[0], r1 = rec[1], r3 = rec[3], r4 = rec[4];
            const float dx = local_x + ctr.x, dy = local_y + ctr.y;
            const float xx = dx * dx, xy = dx * dy, yy = dy * dy;
            const float e = fmaf(r0.x, xx, fmaf(r0.y, xy, r0.z * yy));
            const float den = fmaf(r0.w, dx, fmaf(r1.y, xx, 1.0f)) + fmaf(r1.x, dy, fmaf(r1.z, xy, r1.w * yy));
            const float den_rcp = rcp_approx(den);
            const float alpha = fminf(exp2_approx(fmaf(e, den_rcp, r3.z)), kMaxFragmentAlpha);
            if constexpr (kOit) {
                depth = 0.0f;   // the RGB-only OIT result does not depend on depth
            } else {
                const float4 r2 = rec[2];
                const float num_z = fmaf(r2.x, dx, fmaf(r2.z, xx, r2.w * xy)) + fmaf(r2.y, dy, r3.x * yy);
                depth = fmaf(num_z, den_rcp, r3.y);
            }
            if constexpr (kFirstK) frag = make_float4(0.0f, 0.0f, 0.0f, alpha);   // the colour is fetched when the tile is composited
            else frag = make_float4(r3.w * alpha, r4.x * alpha, r4.y * alpha, alpha);
        };
        auto commit = [&](uint32_t prim, float depth, float4 frag) {
            if constexpr (kHybrid) {
                if (depth < depth_max && frag.w >= MT::min_alpha_core) {
                    frag = unpack_half4(core_replace<K>(keys, pay, tid, depth, pack_half4(frag.x, frag.y, frag.z, frag.w), row_max, kmax));
                    depth_max = KeyCodec<K>::decode(kmax);
                }
                tail += frag;
                transmittance_tail *= 1.0f - frag.w;
            } else if constexpr (kFirstK) {
                if (depth < depth_max) {   // whatever falls out of the buffer is dropped (alpha_blend_first_k/kernels/fast_inference.cuh:147-160)
                    core_replace<K>(keys, pay, tid, depth, make_uint2(__float_as_uint(frag.w), prim), row_max, kmax);
                    depth_max = KeyCodec<K>::decode(kmax);
                }
            } else {   // oit_blend/kernels/fast_inference.cuh:138-141
                tail += frag;
                transmittance_tail *= 1.0f - frag.w;
            }
        };
        auto prim_of = [&](const uint32_t* prims, uint32_t j) -> uint32_t { return SL::has_prim ? prims[j] : 0u; };
        if (step) {        // until no lane has a candidate of the older half left
            // HYBRID: as in the exact kernel one candidate of a lane enters the buffer per trip, and a second one, with what comes behind it,
            // goes back into the window (3 M Gaussians, 1297 x 840, K = 16: an insertion per candidate 623 us; candidates per trip two 617, three
            // 580, four 595; K = 32 at 1 M: 576, -, 537, 540).  A shorter insertion into empty places, as there, does not pay here (582).
            if constexpr (kHybrid) {
                while (__any_sync(0xffffffffu, window >= 0x10000u)) {
                    const uint32_t before = window;
                    uint32_t bit[kFastPerTrip];
                    float depth[kFastPerTrip];
                    float4 frag[kFastPerTrip];
                    bool counts[kFastPerTrip];
                    #pragma unroll
                    for (int i = 0; i < kFastPerTrip; ++i) {
                        bool valid;
                        const uint32_t j = pop_candidate(valid);
                        bit[i] = j ^ flip;
                        evaluate(s_rec + j, s_ctr[j], depth[i], frag[i]);
                        counts[i] = valid && !(frag[i].w < MT::min_alpha);
                    }
                    bool enters = false, stopped = false;
                    float in_depth = 0.0f;
                    float4 in_frag = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    uint32_t stop_bit = 0;
                    #pragma unroll
                    for (int i = 0; i < kFastPerTrip; ++i) {
                        const bool nearer = counts[i] && depth[i] < depth_max && frag[i].w >= MT::min_alpha_core;
                        if (nearer && enters && !stopped) { stopped = true; stop_bit = bit[i]; }
                        if (nearer && !enters) { in_depth = depth[i]; in_frag = frag[i]; }
                        enters |= nearer;
                        if (counts[i] && !nearer && !stopped) { tail += frag[i]; transmittance_tail *= 1.0f - frag[i].w; }
                    }
                    if (stopped) window = before & ((2u << stop_bit) - 1u);
                    if (enters) {
                        const float4 out = unpack_half4(core_replace<K>(keys, pay, tid, in_depth, pack_half4(in_frag.x, in_frag.y, in_frag.z, in_frag.w), row_max, kmax));
                        depth_max = KeyCodec<K>::decode(kmax);
                        tail += out;
                        transmittance_tail *= 1.0f - out.w;
                    }
                }
            } else {
                while (__any_sync(0xffffffffu, window >= 0x10000u)) {
                    bool v0, v1;
                    const uint32_t j0 = pop_candidate(v0);
                    const uint32_t j1 = pop_candidate(v1);
                    float depth0, depth1;
                    float4 frag0, frag1;
                    evaluate(s_rec + j0, s_ctr[j0], depth0, frag0);
                    evaluate(s_rec + j1, s_ctr[j1], depth1, frag1);
                    if (v0 && !(frag0.w < MT::min_alpha)) commit(prim_of(s_prim, j0), depth0, frag0);
                    if (v1 && !(frag1.w < MT::min_alpha)) commit(prim_of(s_prim, j1), depth1, frag1);
                }
            }
            window <<= 16;
            half ^= 1u;
        }
        if (n_dense != 0) {
            if (!mbar_wait_bounded(s_bar + 2, (phases >> 2) & 1u)) wait_failed = true;
            phases ^= 4u;
            __syncwarp();
            for (uint32_t j = 0; j < n_dense; j += 2) {
                const uint32_t k = min(j + 1, n_dense - 1);
                const bool v0 = inside && ((s_dense_mask[j] >> lane) & 1u), v1 = inside && j + 1 < n_dense && ((s_dense_mask[k] >> lane) & 1u);
                float depth0, depth1;
                float4 frag0, frag1;
                evaluate(s_dense + j, s_dense_ctr[j], depth0, frag0);
                evaluate(s_dense + k, s_dense_ctr[k], depth1, frag1);
                if (v0 && !(frag0.w < MT::min_alpha)) commit(prim_of(s_dense_prim, j), depth0, frag0);
                if (v1 && !(frag1.w < MT::min_alpha)) commit(prim_of(s_dense_prim, k), depth1, frag1);
            }
            __syncwarp();
        }
    }

    if (wait_failed) atomicOr(&status->error, 1u);
    if (!inside) return;

    float3 rgb_pixel = make_float3(0.0f, 0.0f, 0.0f);
    if constexpr (SL::has_kbuffer) {
        // ---- composite: sort the core entries by key, blend front to back (hybrid_blend/kernels/fast_inference.cuh:193-216,
        // alpha_blend_first_k/kernels/fast_inference.cuh:166-180)
        uint32_t v[K];
        {
            const uint4* rows = reinterpret_cast<const uint4*>(keys) + tid;
            #pragma unroll
            for (int q = 0; q < K / 4; ++q) {
                const uint4 row = rows[q * kFastThreads];
                v[4 * q] = row.x; v[4 * q + 1] = row.y; v[4 * q + 2] = row.z; v[4 * q + 3] = row.w;
            }
        }
        #pragma unroll
        for (int k = 2; k <= K; k <<= 1) {
            #pragma unroll
            for (int j = k >> 1; j > 0; j >>= 1) {
                #pragma unroll
                for (int i = 0; i < K; ++i) {
                    const int l = i ^ j;
                    if (l > i) {
                        const uint32_t lo = min(v[i], v[l]), hi = max(v[i], v[l]);
                        if ((i & k) == 0) { v[i] = lo; v[l] = hi; } else { v[i] = hi; v[l] = lo; }
                    }
                }
            }
        }
        float transmittance_core = 1.0f;
        #pragma unroll
        for (int k = 0; k < K; ++k) {
            if (transmittance_core >= kTransmittanceThreshold) {
                const uint32_t c = v[k] & uint32_t(K - 1);
                const uint2 cell = pay[c * kFastThreads + tid];
                if constexpr (kHybrid) {
                    const float4 rgba = unpack_half4(cell);
                    rgb_pixel += transmittance_core * f3(rgba);
                    transmittance_core *= 1.0f - rgba.w;
                } else {
                    if (cell.y == 0xffffffffu) { transmittance_core = 0.0f; continue; }   // empty entries sort last: nothing follows
                    const float alpha = __uint_as_float(cell.x);
                    const float* rec = reinterpret_cast<const float*>(records + cell.y);
                    const float3 rgb = make_float3(__ldg(rec + 15), __ldg(rec + 16), __ldg(rec + 17));   // FastRecord::r, g, b
                    rgb_pixel += (transmittance_core * alpha) * rgb;
                    transmittance_core *= 1.0f - alpha;
                }
            }
        }
        if constexpr (kHybrid) {
            if (transmittance_core >= kTransmittanceThreshold && tail.w >= MT::min_alpha) {
                const float weight_tail = transmittance_core * (1.0f - transmittance_tail);
                rgb_pixel += weight_tail * (1.0f / tail.w) * f3(tail);
            }
        }
    } else {
        // oit_blend/kernels/fast_inference.cuh:147-152
        if (tail.w >= MT::min_alpha) rgb_pixel = ((1.0f - transmittance_tail) * (1.0f / tail.w)) * f3(tail);
    }
    const uint32_t pixel_idx = width * py_i + px_i;
    if (to_chw) {
        const uint32_t n_pixels = width * height;
        image[pixel_idx] = __saturatef(rgb_pixel.x);
        image[n_pixels + pixel_idx] = __saturatef(rgb_pixel.y);
        image[2 * n_pixels + pixel_idx] = __saturatef(rgb_pixel.z);
    } else {
        image[3 * pixel_idx] = __saturatef(rgb_pixel.x);
        image[3 * pixel_idx + 1] = __saturatef(rgb_pixel.y);
        image[3 * pixel_idx + 2] = __saturatef(rgb_pixel.z);
    }
}

template <int MODE, int K>
cudaError_t launch_fast_k(const FrameGeometry& geo, const PrimBuffers& prim, const uint32_t* prims_sorted, const uint2* tile_ranges, const uint32_t* tile_order, float* image,
                          bool to_chw, FrameStatus* status, cudaStream_t stream) {
    using SL = FastSmem<MODE, K>;
    static_assert(SL::total <= 48 * 1024, "no opt-in for more shared memory needed");
    if (geo.n_tiles == 0) return cudaSuccess;
    launch_after(blend_fast_kernel<MODE, K>, uint32_t(geo.n_tiles) * 2u, kFastThreads, SL::total, stream,
        tile_ranges, tile_order, prims_sorted, reinterpret_cast<const FastRecord*>(prim.eval), prim.cull, image, uint32_t(geo.width), uint32_t(geo.height),
        uint32_t(geo.grid_w), to_chw, status);
    return cudaGetLastError();
}

template <int MODE>
cudaError_t launch_fast_mode(int K, const FrameGeometry& geo, const PrimBuffers& prim, const uint32_t* prims_sorted, const uint2* tile_ranges, const uint32_t* tile_order,
                             float* image, bool to_chw, FrameStatus* status, cudaStream_t stream) {
    switch (effective_k(MODE, K)) {
        case 4: return launch_fast_k<MODE, 4>(geo, prim, prims_sorted, tile_ranges, tile_order, image, to_chw, status, stream);
        case 8: return launch_fast_k<MODE, 8>(geo, prim, prims_sorted, tile_ranges, tile_order, image, to_chw, status, stream);
        case 16: return launch_fast_k<MODE, 16>(geo, prim, prims_sorted, tile_ranges, tile_order, image, to_chw, status, stream);
        case 32: return launch_fast_k<MODE, 32>(geo, prim, prims_sorted, tile_ranges, tile_order, image, to_chw, status, stream);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace

bool blend_fast_supports(int mode, int K) {
    if (mode == HTGS_MODE_OIT_BLEND) return true;
    if (mode != HTGS_MODE_HYBRID_BLEND && mode != HTGS_MODE_ALPHA_BLEND_FIRST_K) return false;
    const int k = effective_k(mode, K);
    return k == 4 || k == 8 || k == 16 || k == 32;
}

cudaError_t launch_blend_fast(int mode, int K, const FrameGeometry& geo, const PrimBuffers& prim, const uint32_t* prims_sorted, const uint2* tile_ranges, const uint32_t* tile_order,
                              float* image, bool to_chw, FrameStatus* status, cudaStream_t stream) {
    switch (mode) {
        case HTGS_MODE_HYBRID_BLEND: return launch_fast_mode<HTGS_MODE_HYBRID_BLEND>(K, geo, prim, prims_sorted, tile_ranges, tile_order, image, to_chw, status, stream);
        case HTGS_MODE_ALPHA_BLEND_FIRST_K: return launch_fast_mode<HTGS_MODE_ALPHA_BLEND_FIRST_K>(K, geo, prim, prims_sorted, tile_ranges, tile_order, image, to_chw, status, stream);
        case HTGS_MODE_OIT_BLEND: return launch_fast_k<HTGS_MODE_OIT_BLEND, 4>(geo, prim, prims_sorted, tile_ranges, tile_order, image, to_chw, status, stream);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace htgs
