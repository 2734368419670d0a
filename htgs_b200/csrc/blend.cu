// Per-tile blend kernels (inference) for the four blend modes.
//
// Replaces blend_cu of the reference
//   HYBRID_BLEND               rasterization/include/hybrid_blend/kernels/inference.cuh:78-216
//   ALPHA_BLEND_FIRST_K        rasterization/include/alpha_blend_first_k/kernels/inference.cuh:79-208
//   ALPHA_BLEND_GLOBAL_ORDERING rasterization/include/alpha_blend_global_ordering/kernels/inference.cuh:78-176
//   OIT_BLEND                  rasterization/include/oit_blend/kernels/inference.cuh:78-177
// The per-fragment arithmetic (planes through the pixel ray, rho^2, G, alpha, depth of the point
// of maximum contribution) and every threshold decision are kept operation for operation, and each
// pixel still sees its tile's instances in list order, so results match the reference bit for bit.
// How the work is organised is different.  A CTA is ONE warp and blends 8 x 4 pixels, half of a tile (an eighth of
// GLOBAL_ORDERING's 16 x 16 tile, whose lists have to be the reference's; its pixels share no state).  Nothing is shared
// between warps, so there is no block barrier, a short list frees its resources at once, and the warp runs this pipeline
// over its tile's list:
//
//  1. Filter.  Lane = instance: 32 instances at a time, the conservative outline of the Gaussian (an ellipse) is cut with the
//     four pixel rows, which gives a 32-bit mask of the pixels it can touch.  Instances that touch none (half of a list:
//     lists come from tile boxes) are dropped, the others wait in a queue, in list order.
//  2. Window.  Records are staged in two halves of 16; each lane's 80-byte bulk asynchronous copy (TMA, cp.async.bulk)
//     brings one, an mbarrier per half tracks them, and the next instances are filtered while they fly.  The masks of a
//     half are transposed (16 x 32 bits, shuffles), so that lane = pixel holds the bits of its own candidates: the
//     older half in the upper 16 bits of a word, the newer one below.
//  3. Exact pass.  Every lane walks the bits of its own word from the top, two or three candidates per trip; almost every one is
//     an accepted fragment.  A half is replaced when no lane has a bit of it left; lanes that are ahead work on the newer half
//     meanwhile, so lanes wait for the pixel with the most fragments only over a tile, not over every batch of 64 (lanes busy
//     per step: 0.92 instead of 0.83 at 1297 x 840, 3 M Gaussians).
//  4. K-buffer (core_buffer.cuh).  The K nearest core fragments lie unsorted in shared memory, 12 bytes each; an insertion
//     overwrites the one that falls out and costs the same for every K, or takes the next empty place, which costs a quarter of that.
//     The colour of the entry that will fall out next is fetched from its record right after the insertion before, so that it has
//     arrived when it is needed.
//
// Blocks start in the order of `tile_order`, long lists first: the last blocks of a launch are short ones.
//
// What bounds it: instruction issue (77 % of the issue slots at 1 M Gaussians, 1297 x 840, K = 16; a fifth of the instructions are
// insertions, a quarter filter, window and compositing), at the 22 warps per SM that the K-buffers leave (K = 32: 14).  3 M
// Gaussians, 1297 x 840, K = 16: 788 us; 8 M, 4K, K = 32: 27.8 ms.
#include <algorithm>
#include <type_traits>

#include "core_buffer.cuh"
#include "kernels.h"

namespace htgs {

namespace {

constexpr int kBlockW = 8, kBlockH = 4;          // pixels of a warp
constexpr int kHalf = 16;                        // records per half of the window
constexpr int kQueue = 64;                       // survivors of the filter that wait for a place: fewer than kHalf before a step of 32

// The unsorted buffer from four entries on, where the depth range allows it (core_key_window); the chain otherwise.
// `dividing` is the chain in a kernel that divides where the others take reciprocal_rn: every blend is launched in that form too, and
// FrameStatus::divide tells which of the two launches has to do with the frame.  The other one returns at once: 1184 CTAs (all 34230 of a
// frame of 1297 x 840 took 22 us).
// A branch in the loop instead cost the frame 2 to 4 %, two copies of the loop 1 to 2 %.
enum class Buffer { chain, keys, keys_and_colours, dividing };
template <int K, Buffer BUFFER> struct CoreOf { using type = SortedCore<K, 32>; };
template <int K> struct CoreOf<K, Buffer::keys> { using type = UnsortedCore<K, 32, false>; };
template <int K> struct CoreOf<K, Buffer::keys_and_colours> { using type = UnsortedCore<K, 32, true>; };
// HYBRID_BLEND with the unsorted buffer: candidates that a lane evaluates per trip, of which one may enter the buffer.  With K = 32 the 14 warps
// that shared memory leaves have registers for a third one, which hides more latency than its repeated evaluations cost where lists are long and opaque: 4 M
// Gaussians in dense clusters, 1920 x 1080, two 9.79 ms, three 9.27 (elsewhere two are up to 4 % faster: 3 M, 1297 x 840, 622 and 647 us).  A training forward,
// which writes what lies in the buffer, is faster with two (step at 1 M 1181 and 1261 us), and so are smaller buffers: three cost 5 % at K = 4 and 8 and 7 at 16.
constexpr int candidates_per_trip(int K, bool train) { return K >= 32 && !train ? 3 : 2; }
// Whether one insertion serves a trip.  With four entries in long lists, of which few candidates enter, what a trip decides costs more than the insertions (blend at 4 M as
// above: 6.09 ms with an insertion per candidate, 6.35 with one per trip; 3 M, 1297 x 840: 346 and 342 us).  A training step is faster with one per trip there too (400 k, 980 x
// 545: 626 and 615 us).  With eight entries, 6.93 and 6.73 ms, 401 and 383 us.
template <typename SL> constexpr bool merges_insertions(int K, bool train) { return SL::Core::unsorted && (K >= 8 || train || SL::Core::keeps_colour); }
// Whether entries are appended while there are empty places: its branch costs smaller buffers more than the shorter insertion saves (K = 8, as above: 6.82 ms and
// 387 us with it, 6.73 and 383 without; K = 16: 7.25 and 414 with it, 7.28 and 424 without), but not where a grid is resident at once (256 x 256: 166 and 170 us).
template <typename SL> constexpr bool appends_to_empty_places(int K) { return K >= 16 || SL::Core::keeps_colour; }
struct NoCore { static constexpr bool keeps_colour = false, unsorted = false; static constexpr size_t smem_bytes = 0; };

template <int MODE, int K, Buffer BUFFER, BlendTask TASK> struct SmemLayout {
    static constexpr bool has_kbuffer = (MODE == HTGS_MODE_HYBRID_BLEND || MODE == HTGS_MODE_ALPHA_BLEND_FIRST_K);
    using Core = typename std::conditional<has_kbuffer, typename CoreOf<K, BUFFER>::type, NoCore>::type;
    static constexpr size_t record_off = 0;
    static constexpr size_t core_off = record_off + 2 * kHalf * sizeof(EvalRecord);
    static constexpr size_t queue_prim_off = core_off + Core::smem_bytes;
    static constexpr size_t queue_mask_off = queue_prim_off + kQueue * 4;
    static constexpr size_t queue_pos_off = queue_mask_off + kQueue * 4;
    static constexpr bool has_pos = has_kbuffer && TASK == BlendTask::training;
    static constexpr bool has_word = has_kbuffer || TASK == BlendTask::max_weights;
    static constexpr size_t word_off = queue_pos_off + (has_pos ? kQueue * 4 : 0);       // what a K-buffer entry is filed under, per staged record
    static constexpr size_t bar_off = word_off + (has_word ? 2 * kHalf * 4 : 0);
    static constexpr size_t total = bar_off + 2 * 8;
};

// The shared per-fragment front end (hybrid_blend/kernels/inference.cuh:137-148).
struct FragmentFront {
    float3 m, d;
    float numerator_rho2, denominator;
};
__device__ __forceinline__ FragmentFront fragment_front(const float4& VPMT1, const float4& VPMT2, const float4& VPMT4, float pixel_x, float pixel_y) {
    FragmentFront f;
    const float4 plane_x_diag = VPMT1 - VPMT4 * pixel_x;
    const float4 plane_y_diag = VPMT2 - VPMT4 * pixel_y;
    const float3 plane_x_diag_normal = f3(plane_x_diag);
    const float3 plane_y_diag_normal = f3(plane_y_diag);
    f.m = plane_x_diag.w * plane_y_diag_normal - plane_x_diag_normal * plane_y_diag.w;
    f.d = cross(plane_x_diag_normal, plane_y_diag_normal);
    f.numerator_rho2 = dot(f.m, f.m);
    f.denominator = dot(f.d, f.d);
    return f;
}

// One block of 8 x 4 pixels.  `phases`: the parities of the two halves' barriers, which the caller has initialised.  False if a wait gave up.
template <int MODE, int K, Buffer BUFFER, BlendTask TASK>
__device__ __forceinline__ bool blend_block(
    uint32_t block, uint32_t& phases, unsigned char* smem, const uint2* __restrict__ tile_ranges, const uint32_t* __restrict__ tile_order, const uint32_t* __restrict__ prims_sorted, const EvalRecord* __restrict__ eval,
    const CullRecord* __restrict__ cull, float* __restrict__ image, float* __restrict__ depth_out, float* __restrict__ alpha_out,
    unsigned int* __restrict__ max_weights, float weight_threshold, TrainPixelBuffers tout, uint32_t width, uint32_t height, uint32_t grid_w, bool to_chw,
    bool use_median_depth, int32_t key_base, FrameStatus* status)
{
    constexpr bool kDivide = BUFFER == Buffer::dividing;
    using MT = ModeTraits<MODE>;
    using SL = SmemLayout<MODE, K, BUFFER, TASK>;
    constexpr bool TRAIN = TASK == BlendTask::training, STATS = TASK == BlendTask::image_with_statistics, WEIGHTS = TASK == BlendTask::max_weights;
    constexpr bool kHybrid = MODE == HTGS_MODE_HYBRID_BLEND;
    constexpr bool kFirstK = MODE == HTGS_MODE_ALPHA_BLEND_FIRST_K;
    constexpr bool kGlobal = MODE == HTGS_MODE_ALPHA_BLEND_GLOBAL_ORDERING;
    constexpr bool kMerged = kHybrid && merges_insertions<SL>(K, TRAIN);
    constexpr bool kAppends = appends_to_empty_places<SL>(K);
    constexpr int kPerTrip = candidates_per_trip(K, TRAIN);
    constexpr uint32_t kTileX = MT::tile_w / kBlockW, kTileY = MT::tile_h / kBlockH;     // blocks per binning tile
    EvalRecord* s_record = reinterpret_cast<EvalRecord*>(smem + SL::record_off);
    uint32_t* s_queue_prim = reinterpret_cast<uint32_t*>(smem + SL::queue_prim_off);
    uint32_t* s_queue_mask = reinterpret_cast<uint32_t*>(smem + SL::queue_mask_off);
    [[maybe_unused]] uint32_t* s_queue_pos = reinterpret_cast<uint32_t*>(smem + SL::queue_pos_off);
    [[maybe_unused]] uint32_t* s_word = reinterpret_cast<uint32_t*>(smem + SL::word_off);
    uint64_t* s_bar = reinterpret_cast<uint64_t*>(smem + SL::bar_off);

    const uint32_t lane = threadIdx.x;
    const uint32_t tile = __ldg(tile_order + block / (kTileX * kTileY)), part = block % (kTileX * kTileY);
    const uint32_t block_x = (tile % grid_w) * kTileX + part % kTileX, block_y = (tile / grid_w) * kTileY + part / kTileX;
    if (block_x * kBlockW >= width || block_y * kBlockH >= height) return true;       // a ragged edge leaves blocks without pixels
    const uint32_t px_i = block_x * kBlockW + (lane & 7u);
    const uint32_t py_i = block_y * kBlockH + (lane >> 3);
    const bool inside = px_i < width && py_i < height;
    const float pixel_x = __uint2float_rn(px_i);
    const float pixel_y = __uint2float_rn(py_i);
    const float block_x0 = float(block_x * kBlockW), block_y0 = float(block_y * kBlockH);

    // ---- per-pixel state -------------------------------------------------------------------
    [[maybe_unused]] typename SL::Core core;
    // what is known of the entry that falls out of the buffer next: payload and colour, zero for an empty entry
    [[maybe_unused]] uint2 last = make_uint2(0u, kNoEntry);
    [[maybe_unused]] float3 last_rgb = make_float3(0.0f, 0.0f, 0.0f);
    if constexpr (SL::has_kbuffer) core.init(smem + SL::core_off, lane, key_base);
    // HYBRID tail / OIT accumulators / GLOBAL_ORDERING running blend
    float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);   // HB: premultiplied tail rgba; OIT: alpha-weighted rgb,depth; GO: rgb, depth
    float acc_depth = 0.0f;                              // HB: depth * alpha of the tail; OIT: alpha sum
    float transmittance = 1.0f;                          // HB: tail; OIT / GO: pixel
    bool done = !inside;

    const uint2 range = tile_ranges[tile];
    // colour of the Gaussian that a payload's word names: its index, or (training) its position in the tile's list
    [[maybe_unused]] auto colour_of = [&](uint32_t word) -> float3 {
        const uint32_t g = TRAIN ? __ldg(prims_sorted + range.x + word) : word;
        const float4 second = ldg4(reinterpret_cast<const float*>(cull + g) + 4);
        return make_float3(second.y, second.z, second.w);
    };
    bool wait_failed = false;
    [[maybe_unused]] uint32_t stat_candidates = 0, stat_accepted = 0, stat_trips = 0, stat_trips_inserting = 0, stat_insertions = 0;

    // ---- 1. filter: the 32 instances from `next` on; their outlines and the indices of the 32 behind them are on their way ----
    uint32_t next = range.x + lane;                      // the instance this lane tests next
    uint32_t g_here = 0, g_ahead = 0;
    float4 outline = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float outline_c = 0.0f;
    auto request_outline = [&](uint32_t g) {
        outline = ldg4(reinterpret_cast<const float*>(cull + g));
        outline_c = __ldg(reinterpret_cast<const float*>(cull + g) + 4);
    };
    if (next < range.y) { g_here = __ldg(prims_sorted + next); request_outline(g_here); }
    if (next + 32 < range.y) g_ahead = __ldg(prims_sorted + next + 32);
    uint32_t queue_head = 0, queued = 0;
    auto filter = [&]() {
        uint32_t mask = 0;
        if (next < range.y) mask = outline_mask(outline, outline_c, block_x0, block_y0);
        const uint32_t survivors = __ballot_sync(0xffffffffu, mask != 0);
        if (mask != 0) {
            const uint32_t at = (queue_head + queued + __popc(survivors & lanemask_lt())) & uint32_t(kQueue - 1);
            s_queue_prim[at] = g_here;
            s_queue_mask[at] = mask;
            if constexpr (SL::has_pos) s_queue_pos[at] = next - range.x;
        }
        queued += __popc(survivors);
        next += 32;
        g_here = g_ahead;
        if (next < range.y) request_outline(g_here);
        if (next + 32 < range.y) g_ahead = __ldg(prims_sorted + next + 32);
    };
    while (queued < kHalf && next - lane < range.y) filter();
    __syncwarp();

    uint32_t window = 0;                                 // this pixel's candidates: bits 31..16 the older half, 15..0 the newer half
    for (uint32_t half = 0;; half ^= 1u) {
        // ---- 2. replace the half that no lane needs any more ----------------------------------------------------------
        const uint32_t count = min(queued, uint32_t(kHalf));
        if (count != 0) {
            uint32_t g = 0, mask = 0;
            const uint32_t slot = half * kHalf + (uint32_t(kHalf) - 1u - (lane & uint32_t(kHalf - 1)));
            if (lane < count) {
                const uint32_t at = (queue_head + lane) & uint32_t(kQueue - 1);
                g = s_queue_prim[at];
                mask = s_queue_mask[at];
                if constexpr (SL::has_word) s_word[slot] = TRAIN ? s_queue_pos[at] : g;
            }
            if (lane == 0) mbar_arrive_expect_tx(s_bar + half, count * uint32_t(sizeof(EvalRecord)));
            __syncwarp();
            if (lane < count) bulk_copy_g2s(s_record + slot, eval + g, uint32_t(sizeof(EvalRecord)), s_bar + half);
            queue_head += count;
            queued -= count;
            const uint32_t mine = transpose_masks(mask, lane);
            if (!done) window |= mine;
            if constexpr (STATS) stat_candidates += __popc(done ? 0u : mine);
            while (queued < kHalf && next - lane < range.y) filter();
            if (!mbar_wait_bounded(s_bar + half, (phases >> half) & 1u)) wait_failed = true;
            phases ^= 1u << half;
            __syncwarp();
        } else if (!__any_sync(0xffffffffu, window != 0)) {
            break;
        }
        // ---- 3. exact pass: until no lane has a candidate of the older half left ---------------------------------------
        const uint32_t flip = half * kHalf;              // bit j of the window is record j ^ flip
        auto pop_candidate = [&](bool& valid) -> uint32_t {
            valid = window != 0;
            const uint32_t j = uint32_t(31 - __clz(int(window | 1u)));
            window &= ~(1u << j);
            return j ^ flip;
        };
        [[maybe_unused]] auto evaluate = [&](bool valid, uint32_t j, float& depth, float& alpha) -> bool {       // HYBRID
            const float4* rec = reinterpret_cast<const float4*>(s_record + j);
            const FragmentFront fr = fragment_front(rec[0], rec[1], rec[2], pixel_x, pixel_y);
            const float numerator_rho2 = fr.numerator_rho2;
            const float denominator = fr.denominator;
            const bool inside_cutoff = !(numerator_rho2 > MT::max_cutoff_sq * denominator);
            const float denominator_rcp = kDivide ? 1.0f / denominator : reciprocal_rn(denominator);
            const float G = expf(-0.5f * numerator_rho2 * denominator_rcp);
            alpha = fminf(rec[4].w * G, kMaxFragmentAlpha);
            const float3 eval_point_diag = cross(fr.d, fr.m) * denominator_rcp;
            const float4 MT3 = rec[3];
            depth = dot(f3(MT3), eval_point_diag) + MT3.w;
            return valid && inside_cutoff && !(alpha < MT::min_alpha);
        };
        [[maybe_unused]] auto add_to_tail = [&](float depth, const float4& frag) {
            if constexpr (STATS) ++stat_accepted;
            if constexpr (TRAIN) {
                acc += make_float4(frag.x * frag.w, frag.y * frag.w, frag.z * frag.w, frag.w);
            } else {       // premultiplied colours are rounded before they are summed (inference.cuh:158)
                acc += make_float4(__fmul_rn(frag.x, frag.w), __fmul_rn(frag.y, frag.w), __fmul_rn(frag.z, frag.w), frag.w);
                if (!use_median_depth) acc_depth += depth * frag.w;
            }
            transmittance *= 1.0f - frag.w;
        };
        while (__any_sync(0xffffffffu, window >= 0x10000u)) {
            if constexpr (kMerged) {
                // A lane takes kPerTrip candidates; their evaluations are independent instruction streams.  One of them may enter the buffer: the
                // warp runs an insertion (a third of a trip's instructions) whenever one lane has one to do, and with one insertion per
                // candidate (9 lanes of 32 at a time) that was four times for every five candidates.  A second one of a lane, and what comes
                // behind it, goes back into the window.  The tail's sums stay in list order: what falls out takes the place of what entered.
                // 3 M Gaussians, 1297 x 840, K = 16: 866 -> 787 us, training forward 1026 -> 894; 4K, K = 32: 33.7 -> 27.8 ms.  (FIRST_K, where
                // every candidate enters until the buffer is full, gets slower: 262 -> 292 us.)
                const uint32_t before = window;
                uint32_t j[kPerTrip], bit[kPerTrip];
                float depth[kPerTrip], alpha[kPerTrip];
                bool counts[kPerTrip];
                #pragma unroll
                for (int i = 0; i < kPerTrip; ++i) {
                    bool valid;
                    j[i] = pop_candidate(valid);
                    bit[i] = j[i] ^ flip;
                    counts[i] = evaluate(valid, j[i], depth[i], alpha[i]);
                }
                const float limit = core.limit();
                bool enters = false, stopped = false, is_entering[kPerTrip];
                float in_depth = 0.0f, in_alpha = 0.0f;
                uint32_t in_j = 0, stop_bit = 0;
                #pragma unroll
                for (int i = 0; i < kPerTrip; ++i) {
                    const bool nearer = counts[i] && depth[i] < limit && alpha[i] >= MT::min_alpha_core;
                    is_entering[i] = nearer && !enters;
                    if (is_entering[i]) { in_depth = depth[i]; in_alpha = alpha[i]; in_j = j[i]; }
                    if (nearer && enters && !stopped) { stopped = true; stop_bit = bit[i]; }
                    enters |= nearer;
                    counts[i] = counts[i] && !stopped;
                }
                if (stopped) window = before & ((2u << stop_bit) - 1u);
                if constexpr (STATS) { stat_trips += 1; stat_trips_inserting += __any_sync(0xffffffffu, enters) ? 1 : 0; stat_insertions += enters ? 1 : 0; }
                float4 evicted = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (enters) {
                    const uint2 payload = make_uint2(__float_as_uint(in_alpha), s_word[in_j]);   // training: what the backward pass looks up
                    // what falls out is a fragment, or nothing (alpha 0; its colour does not matter)
                    if constexpr (SL::Core::keeps_colour) {
                        float3 rgb = f3(reinterpret_cast<const float4*>(s_record + in_j)[4]);
                        core.template insert<kAppends>(in_depth, payload, last, rgb);
                        evicted = make_float4(rgb.x, rgb.y, rgb.z, __uint_as_float(last.x));
                    } else {
                        if (!core.template insert<kAppends>(in_depth, payload, last, last_rgb)) last_rgb = colour_of(last.y);
                        evicted = make_float4(last_rgb.x, last_rgb.y, last_rgb.z, __uint_as_float(last.x));
                        if (!(kAppends && core.filling()) && core.last(last)) last_rgb = colour_of(last.y);
                    }
                }
                #pragma unroll
                for (int i = 0; i < kPerTrip; ++i) {
                    if (counts[i]) {
                        const float4 rgba = reinterpret_cast<const float4*>(s_record + j[i])[4];
                        add_to_tail(is_entering[i] ? limit : depth[i], is_entering[i] ? evicted : make_float4(rgba.x, rgba.y, rgba.z, alpha[i]));
                    }
                }
            } else if constexpr (kHybrid) {
                // Two candidates per trip, as above; the buffer and tail updates happen strictly in list order.  The colour is loaded ahead where registers
                // allow (K = 4: 6.17 -> 6.09 ms in dense clusters; K = 2, whose chain is in registers, 303 -> 313 us).
                constexpr bool kColourAhead = SL::Core::unsorted;
                auto colour_at = [&](uint32_t j) { return reinterpret_cast<const float4*>(s_record + j)[4]; };
                auto commit = [&](float depth, float alpha, uint32_t j, float4 rgba) {
                    if constexpr (!kColourAhead) rgba = colour_at(j);
                    float4 frag = make_float4(rgba.x, rgba.y, rgba.z, alpha);
                    if (depth < core.limit() && alpha >= MT::min_alpha_core) {
                        const float limit = core.limit();
                        if (!core.replace(depth, make_uint2(__float_as_uint(alpha), s_word[j]), last, last_rgb)) last_rgb = colour_of(last.y);
                        frag = make_float4(last_rgb.x, last_rgb.y, last_rgb.z, __uint_as_float(last.x));
                        if (core.last(last)) last_rgb = colour_of(last.y);
                        depth = limit;
                    }
                    add_to_tail(depth, frag);
                };
                bool v0, v1;
                const uint32_t j0 = pop_candidate(v0);
                const uint32_t j1 = pop_candidate(v1);
                float depth0, depth1, alpha0, alpha1;
                const bool ok0 = evaluate(v0, j0, depth0, alpha0);
                const bool ok1 = evaluate(v1, j1, depth1, alpha1);
                float4 rgba0 = make_float4(0.0f, 0.0f, 0.0f, 0.0f), rgba1 = rgba0;
                if constexpr (kColourAhead) { rgba0 = colour_at(j0); rgba1 = colour_at(j1); }
                if constexpr (STATS) {   // how often a lane of the warp inserts
                    const bool in0 = ok0 && depth0 < core.limit() && alpha0 >= MT::min_alpha_core;
                    stat_trips += 1; stat_trips_inserting += __any_sync(0xffffffffu, in0) ? 1 : 0; stat_insertions += in0 ? 1 : 0;
                }
                if (ok0) commit(depth0, alpha0, j0, rgba0);
                if constexpr (STATS) {
                    const bool in1 = ok1 && depth1 < core.limit() && alpha1 >= MT::min_alpha_core;
                    stat_trips += 1; stat_trips_inserting += __any_sync(0xffffffffu, in1) ? 1 : 0; stat_insertions += in1 ? 1 : 0;
                }
                if (ok1) commit(depth1, alpha1, j1, rgba1);
            } else {
                // The other three modes use the same two-candidates-per-trip shape: both evaluations (divide, expf, depth) are
                // independent instruction streams; the state updates happen in list order.  A fragment counts iff it passes
                // the cutoff, the alpha threshold and (FIRST_K) the depth test against the buffer - conditions that do not
                // depend on the order in which they are checked (alpha_blend_first_k/kernels/inference.cuh:147-160,
                // alpha_blend_global_ordering/kernels/inference.cuh:139-160, oit_blend/kernels/inference.cuh:139-160).
                constexpr bool kNeedsPointDepth = kFirstK || (!kGlobal && !TRAIN);
                auto evaluate = [&](bool valid, uint32_t j, float& alpha, float& depth, float4& rgba_in) -> bool {
                    const float4* rec = reinterpret_cast<const float4*>(s_record + j);
                    const FragmentFront fr = fragment_front(rec[0], rec[1], rec[2], pixel_x, pixel_y);
                    const float numerator_rho2 = fr.numerator_rho2;
                    const float denominator = fr.denominator;
                    const bool inside_cutoff = !(numerator_rho2 > MT::max_cutoff_sq * denominator);
                    const float denominator_rcp = kDivide ? 1.0f / denominator : reciprocal_rn(denominator);
                    rgba_in = rec[4];
                    const float G = expf(-0.5f * numerator_rho2 * denominator_rcp);
                    alpha = fminf(rgba_in.w * G, kMaxFragmentAlpha);
                    const float4 MT3 = rec[3];
                    if constexpr (kNeedsPointDepth) {
                        const float3 eval_point_diag = cross(fr.d, fr.m) * denominator_rcp;
                        depth = dot(f3(MT3), eval_point_diag) + MT3.w;
                    } else {
                        depth = MT3.w;
                    }
                    return valid && inside_cutoff && !(alpha < MT::min_alpha);
                };
                auto commit = [&](uint32_t j, float alpha, float depth, const float4& rgba_in) {
                    if constexpr (kFirstK) {
                        if (depth >= core.limit()) return;
                        if constexpr (STATS) ++stat_accepted;
                        const uint2 payload = make_uint2(__float_as_uint(alpha), s_word[j]);
                        if constexpr (SL::Core::unsorted) {
                            if (core.filling()) { core.append(depth, payload, last_rgb); return; }
                        }
                        core.last(last);
                        core.replace(depth, payload, last, last_rgb);   // what falls out is dropped
                    } else if constexpr (kGlobal) {
                        if (done) return;
                        if constexpr (STATS) ++stat_accepted;
                        const float blending_weight = transmittance * alpha;
                        if constexpr (WEIGHTS) { if (!(blending_weight < weight_threshold)) raise_weight(max_weights, s_word[j], blending_weight); }
                        acc.x += blending_weight * rgba_in.x; acc.y += blending_weight * rgba_in.y; acc.z += blending_weight * rgba_in.z;
                        if constexpr (!TRAIN) {
                            if (use_median_depth) acc.w = (transmittance > 0.5f) ? depth : acc.w;
                            else acc.w += blending_weight * depth;
                        }
                        transmittance *= 1.0f - alpha;
                        if (transmittance < kTransmittanceThreshold) { done = true; window = 0; }
                    } else {   // OIT_BLEND
                        if constexpr (STATS) ++stat_accepted;
                        if constexpr (TRAIN) {
                            acc.x += alpha * rgba_in.x; acc.y += alpha * rgba_in.y; acc.z += alpha * rgba_in.z;
                        } else {
                            acc += alpha * make_float4(rgba_in.x, rgba_in.y, rgba_in.z, depth);
                        }
                        acc_depth += alpha;
                        transmittance *= 1.0f - alpha;
                    }
                };
                bool v0, v1;
                const uint32_t j0 = pop_candidate(v0);
                const uint32_t j1 = pop_candidate(v1);
                float alpha0, alpha1, depth0, depth1;
                float4 rgba0, rgba1;
                const bool ok0 = evaluate(v0, j0, alpha0, depth0, rgba0);
                const bool ok1 = evaluate(v1, j1, alpha1, depth1, rgba1);
                if (ok0) commit(j0, alpha0, depth0, rgba0);
                if (ok1) commit(j1, alpha1, depth1, rgba1);
            }
        }
        if constexpr (kGlobal) { if (__all_sync(0xffffffffu, done)) break; }
        window <<= 16;
    }

    if (wait_failed) atomicOr(&status->error, 1u);
    if constexpr (STATS) {
        const uint32_t c = __reduce_add_sync(0xffffffffu, stat_candidates), a = __reduce_add_sync(0xffffffffu, stat_accepted);
        if (lane == 0) { atomicAdd(&status->candidate_pairs, (unsigned long long)c); atomicAdd(&status->accepted_fragments, (unsigned long long)a); }
        const uint32_t ins = __reduce_add_sync(0xffffffffu, stat_insertions);
        if (lane == 0 && stat_trips) {
            atomicAdd(&status->warp_trips, (unsigned long long)stat_trips); atomicAdd(&status->warp_trips_inserting, (unsigned long long)stat_trips_inserting);
            atomicAdd(&status->lane_insertions, (unsigned long long)ins);
        }
    }
    if (!inside) return !wait_failed;
    if constexpr (SL::has_kbuffer) core.finish();

    const uint32_t pixel_idx = width * py_i + px_i;
    const uint32_t n_pixels = width * height;

    if constexpr (WEIGHTS) {
        // ---- largest weights (alpha_blend_first_k/kernels/update_max_weights.cuh; GLOBAL_ORDERING raises them on the way) ----
        if constexpr (kFirstK) {
            float t = 1.0f;
            #pragma unroll
            for (int k = 0; k < K; ++k) {
                float depth;
                uint2 payload;
                const bool stored = core.entry(k, depth, payload);
                const float alpha = __uint_as_float(payload.x);
                const float blending_weight = t * alpha;
                t *= 1.0f - alpha;
                if (t < kTransmittanceThreshold) t = 0.0f;
                if (stored && !(blending_weight < weight_threshold)) raise_weight(max_weights, payload.y, blending_weight);
            }
        }
    } else if constexpr (TRAIN) {
        // ---- training forward: unclamped CHW image + what the backward pass needs per pixel ------------
        const uint32_t slot_base = tile * 64u + part * 32u + lane;   // tile-major pixel slot (modes with 8 x 8 tiles)
        const uint32_t PP = tout.padded_pixels;
        float3 rgb_pixel = make_float3(0.0f, 0.0f, 0.0f);
        if constexpr (kHybrid) {
            // hybrid_blend/kernels/forward.cuh:176-233
            float transmittance_core = 1.0f;
            #pragma unroll
            for (int k = 0; k < K; ++k) {
                float depth;
                uint2 payload;
                const bool stored = core.entry(k, depth, payload);
                if (transmittance_core >= kTransmittanceThreshold && stored) {
                    const float alpha = __uint_as_float(payload.x);
                    const float blending_weight = transmittance_core * alpha;
                    rgb_pixel += blending_weight * colour_of(payload.y);
                    transmittance_core *= 1.0f - alpha;
                    if (transmittance_core < kTransmittanceThreshold) transmittance_core = 0.0f;
                }
            }
            float3 weighted_rgb_tail = make_float3(0.0f, 0.0f, 0.0f);
            float tail_info[6] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};   // the reference leaves these unwritten without tail mass; zeros make the backward terms vanish
            if (acc.w >= MT::min_alpha) {
                const float alpha_sum_tail_rcp = 1.0f / acc.w;
                const float3 rgb_tail = f3(acc);
                weighted_rgb_tail = transmittance_core * (1.0f - transmittance) * alpha_sum_tail_rcp * rgb_tail;
                tail_info[0] = rgb_tail.x; tail_info[1] = rgb_tail.y; tail_info[2] = rgb_tail.z;
                tail_info[3] = alpha_sum_tail_rcp; tail_info[4] = transmittance; tail_info[5] = transmittance_core;
            }
            #pragma unroll
            for (int c = 0; c < 6; ++c) tout.info_tail[c * PP + slot_base] = tail_info[c];
            float3 rgb_pixel_new = make_float3(0.0f, 0.0f, 0.0f);
            transmittance_core = 1.0f;
            #pragma unroll
            for (int k = 0; k < K; ++k) {
                float depth;
                uint2 payload;
                const bool skip = !core.entry(k, depth, payload) || transmittance_core < kTransmittanceThreshold;
                tout.idx_core[k * PP + slot_base] = skip ? kNoEntry : payload.y;
                if (!skip) {
                    const float3 rgb = colour_of(payload.y);
                    const float4 rgba = make_float4(rgb.x, rgb.y, rgb.z, __uint_as_float(payload.x));
                    const float blending_weight = transmittance_core * rgba.w;
                    rgb_pixel_new += blending_weight * f3(rgba);
                    const float one_minus_alpha = 1.0f - rgba.w;
                    const float one_minus_alpha_rcp = 1.0f / fmaxf(one_minus_alpha, kOneMinusAlphaEps);
                    tout.info_core[k * PP + slot_base] = make_float4(
                        rgba.x * transmittance_core - (rgb_pixel.x - rgb_pixel_new.x + weighted_rgb_tail.x) * one_minus_alpha_rcp,
                        rgba.y * transmittance_core - (rgb_pixel.y - rgb_pixel_new.y + weighted_rgb_tail.y) * one_minus_alpha_rcp,
                        rgba.z * transmittance_core - (rgb_pixel.z - rgb_pixel_new.z + weighted_rgb_tail.z) * one_minus_alpha_rcp,
                        blending_weight);
                    transmittance_core *= one_minus_alpha;
                }
            }
            rgb_pixel += weighted_rgb_tail;
        } else if constexpr (kFirstK) {
            // alpha_blend_first_k/kernels/forward.cuh:167-213
            float t = 1.0f;
            bool stop = false;
            #pragma unroll
            for (int k = 0; k < K; ++k) {
                if (!stop && t >= kTransmittanceThreshold) {
                    float depth;
                    uint2 payload;
                    if (!core.entry(k, depth, payload)) stop = true;
                    else {
                        const float alpha = __uint_as_float(payload.x);
                        const float blending_weight = t * alpha;
                        rgb_pixel += blending_weight * colour_of(payload.y);
                        t *= 1.0f - alpha;
                    }
                }
            }
            float3 rgb_pixel_new = make_float3(0.0f, 0.0f, 0.0f);
            t = 1.0f;
            #pragma unroll
            for (int k = 0; k < K; ++k) {
                float depth;
                uint2 payload;
                const bool skip = !core.entry(k, depth, payload) || t < kTransmittanceThreshold;
                tout.idx_core[k * PP + slot_base] = skip ? kNoEntry : payload.y;
                if (!skip) {
                    const float alpha = __uint_as_float(payload.x);
                    const float3 rgb = colour_of(payload.y);
                    const float blending_weight = t * alpha;
                    rgb_pixel_new += blending_weight * rgb;
                    const float one_minus_alpha = 1.0f - alpha;
                    const float one_minus_alpha_rcp = 1.0f / fmaxf(one_minus_alpha, kOneMinusAlphaEps);
                    tout.info_core[k * PP + slot_base] = make_float4(
                        rgb.x * t - (rgb_pixel.x - rgb_pixel_new.x) * one_minus_alpha_rcp,
                        rgb.y * t - (rgb_pixel.y - rgb_pixel_new.y) * one_minus_alpha_rcp,
                        rgb.z * t - (rgb_pixel.z - rgb_pixel_new.z) * one_minus_alpha_rcp,
                        blending_weight);
                    t *= one_minus_alpha;
                }
            }
        } else if constexpr (kGlobal) {
            rgb_pixel = f3(acc);
        } else {
            // oit_blend/kernels/forward.cuh:143-163
            float info[5] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
            if (acc_depth >= MT::min_alpha) {
                const float alpha_sum_rcp = 1.0f / acc_depth;
                rgb_pixel = (1.0f - transmittance) * alpha_sum_rcp * f3(acc);
                info[0] = acc.x; info[1] = acc.y; info[2] = acc.z; info[3] = alpha_sum_rcp; info[4] = transmittance;
            }
            #pragma unroll
            for (int c = 0; c < 5; ++c) tout.info_tail[c * PP + slot_base] = info[c];
        }
        image[pixel_idx] = rgb_pixel.x;
        image[n_pixels + pixel_idx] = rgb_pixel.y;
        image[2 * n_pixels + pixel_idx] = rgb_pixel.z;
        return !wait_failed;
    } else {
    // ---- inference compositing ----------------------------------------------------------------------
    float3 rgb_pixel = make_float3(0.0f, 0.0f, 0.0f);
    float depth_pixel = 0.0f;
    float alpha_pixel = 0.0f;
    if constexpr (kHybrid) {
        // hybrid_blend/kernels/inference.cuh:174-199
        float transmittance_core = 1.0f;
        #pragma unroll
        for (int k = 0; k < K; ++k) {
            float depth;
            uint2 payload;
            const bool stored = core.entry(k, depth, payload);
            if (transmittance_core >= kTransmittanceThreshold && stored) {
                const float alpha = __uint_as_float(payload.x);
                const float3 rgb = colour_of(payload.y);
                rgb_pixel += transmittance_core * make_float3(__fmul_rn(rgb.x, alpha), __fmul_rn(rgb.y, alpha), __fmul_rn(rgb.z, alpha));
                if (use_median_depth) depth_pixel = transmittance_core > 0.5f ? depth : depth_pixel;
                else depth_pixel += transmittance_core * alpha * depth;
                transmittance_core *= 1.0f - alpha;
            }
        }
        float total_alpha = 1.0f - transmittance_core;
        if (transmittance_core >= kTransmittanceThreshold && acc.w >= MT::min_alpha) {
            const float weight_tail = transmittance_core * (1.0f - transmittance);
            rgb_pixel += weight_tail * (1.0f / acc.w) * f3(acc);
            if (!use_median_depth) depth_pixel += weight_tail * (1.0f / acc.w) * acc_depth;
            total_alpha += weight_tail;
        }
        if (!use_median_depth) depth_pixel = (total_alpha > 0.0f) ? depth_pixel / total_alpha : 0.0f;
        alpha_pixel = total_alpha;
    } else if constexpr (kFirstK) {
        // alpha_blend_first_k/kernels/inference.cuh:172-191
        float t = 1.0f;
        bool stop = false;
        #pragma unroll
        for (int k = 0; k < K; ++k) {
            if (!stop && t >= kTransmittanceThreshold) {
                float depth;
                uint2 payload;
                if (!core.entry(k, depth, payload)) { stop = true; }
                else {
                    const float alpha = __uint_as_float(payload.x);
                    const float blending_weight = t * alpha;
                    rgb_pixel += blending_weight * colour_of(payload.y);
                    if (use_median_depth) depth_pixel = (t > 0.5f) ? depth : depth_pixel;
                    else depth_pixel += blending_weight * depth;
                    t *= 1.0f - alpha;
                }
            }
        }
        if (!use_median_depth) depth_pixel = (t < 1.0f) ? depth_pixel / (1.0f - t) : 0.0f;
        alpha_pixel = 1.0f - t;
    } else if constexpr (kGlobal) {
        rgb_pixel = f3(acc);
        depth_pixel = acc.w;
        if (!use_median_depth) depth_pixel = (transmittance < 1.0f) ? depth_pixel / (1.0f - transmittance) : 0.0f;
        alpha_pixel = 1.0f - transmittance;
    } else {
        // oit_blend/kernels/inference.cuh:150-160
        float4 rgbd_pixel = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (acc_depth >= MT::min_alpha) {
            const float alpha = 1.0f - transmittance;
            rgbd_pixel = alpha * (1.0f / acc_depth) * acc;
            rgbd_pixel.w = rgbd_pixel.w / alpha;
            alpha_pixel = alpha;
        }
        rgb_pixel = f3(rgbd_pixel);
        depth_pixel = rgbd_pixel.w;
    }
    if (to_chw) {
        image[pixel_idx] = __saturatef(rgb_pixel.x);
        image[n_pixels + pixel_idx] = __saturatef(rgb_pixel.y);
        image[2 * n_pixels + pixel_idx] = __saturatef(rgb_pixel.z);
    } else {
        const uint32_t base_idx = 3 * pixel_idx;
        image[base_idx] = __saturatef(rgb_pixel.x);
        image[base_idx + 1] = __saturatef(rgb_pixel.y);
        image[base_idx + 2] = __saturatef(rgb_pixel.z);
    }
    if (depth_out) depth_out[pixel_idx] = depth_pixel;
    if (alpha_out) alpha_out[pixel_idx] = alpha_pixel;
    }
    return !wait_failed;
}

// Warps per SM that forms with unsorted keys leave registers for: those that shared memory admits (K = 16: 22, K = 32: 14), fewer where that
// would spill (K = 8: 31).  Without a bound the calls of the tie handling make the compiler spend 93 to 96 registers on some and spill others to 64 or 72.
constexpr int blend_min_blocks(int mode, int K, Buffer buffer) {
    if ((buffer != Buffer::keys && buffer != Buffer::keys_and_colours) || K < 8) return 0;
    return mode == HTGS_MODE_HYBRID_BLEND ? (K >= 32 ? 20 : 24) : K >= 32 ? 14 : K >= 16 ? 22 : 28;
}

template <int MODE, int K, Buffer BUFFER, BlendTask TASK>
__global__ void __launch_bounds__(32, blend_min_blocks(MODE, K, BUFFER)) blend_kernel(
    const uint2* __restrict__ tile_ranges, const uint32_t* __restrict__ tile_order, const uint32_t* __restrict__ prims_sorted, const EvalRecord* __restrict__ eval,
    const CullRecord* __restrict__ cull, float* __restrict__ image, float* __restrict__ depth_out, float* __restrict__ alpha_out,
    unsigned int* __restrict__ max_weights, float weight_threshold, TrainPixelBuffers tout, uint32_t width, uint32_t height, uint32_t grid_w, bool to_chw,
    bool use_median_depth, int32_t key_base, FrameStatus* status, uint32_t n_blocks)
{
    cudaGridDependencySynchronize();
    if ((__ldg(&status->divide) != 0) != (BUFFER == Buffer::dividing)) return;
    extern __shared__ __align__(128) unsigned char smem[];
    uint64_t* s_bar = reinterpret_cast<uint64_t*>(smem + SmemLayout<MODE, K, BUFFER, TASK>::bar_off);
    if (threadIdx.x < 2) mbar_init(s_bar + threadIdx.x, 1);
    mbar_fence_init();
    uint32_t phases = 0;
    auto one = [&](uint32_t block) {
        return blend_block<MODE, K, BUFFER, TASK>(block, phases, smem, tile_ranges, tile_order, prims_sorted, eval, cull, image, depth_out, alpha_out, max_weights, weight_threshold,
                                                  tout, width, height, grid_w, to_chw, use_median_depth, key_base, status);
    };
    if constexpr (BUFFER != Buffer::dividing) {
        one(blockIdx.x);
    } else {       // a small grid, since it mostly has nothing to do
        for (uint32_t block = blockIdx.x; block < n_blocks; block += gridDim.x) {
            if (!__all_sync(0xffffffffu, one(block))) return;      // the barriers' state is not known any more; the status has the error
            __syncwarp();
        }
    }
}

struct BlendLaunch {
    FrameGeometry geo;
    PrimBuffers prim;
    const uint32_t* prims_sorted;
    const uint2* tile_ranges;
    const uint32_t* tile_order;
    BlendOutputs out;
    TrainPixelBuffers tout;
    FrameStatus* status;
    cudaStream_t stream;
};

template <int MODE, int K, Buffer BUFFER, BlendTask TASK>
cudaError_t launch_task(const BlendLaunch& l, int32_t key_base) {
    using SL = SmemLayout<MODE, K, BUFFER, TASK>;
    using MT = ModeTraits<MODE>;
    auto kernel = blend_kernel<MODE, K, BUFFER, TASK>;
    if constexpr (SL::total > 48 * 1024) {
        static PerDeviceOnce configured;
        const cudaError_t err = configured.run([&] { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(SL::total)); });
        if (err != cudaSuccess) return err;
    }
    const uint32_t blocks = uint32_t(l.geo.n_tiles) * uint32_t((MT::tile_w / kBlockW) * (MT::tile_h / kBlockH));
    const uint32_t grid = BUFFER == Buffer::dividing ? std::min(blocks, uint32_t(sm_count_of_current_device()) * 8u) : blocks;
    const cudaError_t err = launch_after(kernel, grid, 32, SL::total, l.stream, l.tile_ranges, l.tile_order, l.prims_sorted, l.prim.eval, l.prim.cull, l.out.image, l.out.depth, l.out.alpha,
                                              reinterpret_cast<unsigned int*>(l.out.max_weights), l.out.weight_threshold, l.tout, uint32_t(l.geo.width),
                                              uint32_t(l.geo.height), uint32_t(l.geo.grid_w), l.out.to_chw, l.out.use_median_depth, key_base, l.status, blocks);
    if constexpr (BUFFER == Buffer::dividing) return err;
    else return err != cudaSuccess ? err : launch_task<MODE, K, Buffer::dividing, TASK>(l, 0);
}

template <int MODE, int K, Buffer BUFFER>
cudaError_t launch_buffer(const BlendLaunch& l, BlendTask task, int32_t key_base) {
    switch (task) {
        case BlendTask::image: return launch_task<MODE, K, BUFFER, BlendTask::image>(l, key_base);
        case BlendTask::image_with_statistics: return launch_task<MODE, K, BUFFER, BlendTask::image_with_statistics>(l, key_base);
        case BlendTask::training: return launch_task<MODE, K, BUFFER, BlendTask::training>(l, key_base);
        case BlendTask::max_weights:
            if constexpr (MODE == HTGS_MODE_ALPHA_BLEND_FIRST_K || MODE == HTGS_MODE_ALPHA_BLEND_GLOBAL_ORDERING)
                return launch_task<MODE, K, BUFFER, BlendTask::max_weights>(l, key_base);
    }
    return cudaErrorInvalidValue;
}

// K is rounded down to a power of two <= 32 (hybrid_blend/inference.cu:15-28).  Below four entries the chain is shorter than a row
// update; it also serves depth ranges that the keys do not cover.
template <int MODE, int K>
cudaError_t launch_k(const BlendLaunch& l, BlendTask task, const HtgsView& view) {
    if constexpr (K < 4) {
        return launch_buffer<MODE, K, Buffer::chain>(l, task, 0);
    } else {
        const CoreKeyWindow window = core_key_window(K, view.near_plane, view.far_plane);
        if (!window.covers) return launch_buffer<MODE, K, Buffer::chain>(l, task, 0);
        // A grid that is resident at once leaves shared memory unused, and its time is that of its longest list: there the buffer
        // keeps the colours too (24 bytes an entry), so that an insertion does not wait for one (256 x 256, 16384 Gaussians:
        // 232 -> 197 us; at 1297 x 840 it costs occupancy: 1181 -> 1333 us).
        if constexpr (MODE == HTGS_MODE_HYBRID_BLEND) {
            constexpr size_t smem = SmemLayout<MODE, K, Buffer::keys_and_colours, BlendTask::image>::total;
            constexpr int per_sm = int((227 * 1024) / (smem + 1024)) < 32 ? int((227 * 1024) / (smem + 1024)) : 32;
            // With four entries the colours cost little shared memory, and one insertion per trip pays until lists are long: up to four times the resident grid
            // (blend with the colours and without: 500 x 400, 60 k 53 and 64 us; 800 x 600, 200 k 104 and 113; 980 x 545, 400 k 167 and 180; 1297 x 840, 400 k 147 and 141).
            constexpr int grids = K == 4 ? 4 : 1;
            if (task == BlendTask::image && l.geo.n_tiles * 2 <= grids * per_sm * sm_count_of_current_device())
                return launch_task<MODE, K, Buffer::keys_and_colours, BlendTask::image>(l, window.base);
        }
        return launch_buffer<MODE, K, Buffer::keys>(l, task, window.base);
    }
}

template <int MODE>
cudaError_t launch_mode(const BlendLaunch& l, BlendTask task, const HtgsView& view) {
    switch (effective_k(MODE, view.K)) {
        case 32: return launch_k<MODE, 32>(l, task, view);
        case 16: return launch_k<MODE, 16>(l, task, view);
        case 8: return launch_k<MODE, 8>(l, task, view);
        case 4: return launch_k<MODE, 4>(l, task, view);
        case 2: return launch_k<MODE, 2>(l, task, view);
        default: return launch_k<MODE, 1>(l, task, view);
    }
}

}  // namespace

int effective_k(int mode, int K) {
    if (mode != HTGS_MODE_HYBRID_BLEND && mode != HTGS_MODE_ALPHA_BLEND_FIRST_K) return 1;
    return K >= 32 ? 32 : K >= 16 ? 16 : K >= 8 ? 8 : K >= 4 ? 4 : K >= 2 ? 2 : 1;
}

cudaError_t launch_blend(int mode, BlendTask task, const HtgsView& view, const FrameGeometry& geo, const PrimBuffers& prim, const uint32_t* prims_sorted,
                         const uint2* tile_ranges, const uint32_t* tile_order, const BlendOutputs& out, const TrainPixelBuffers& tout, FrameStatus* status,
                         cudaStream_t stream) {
    const BlendLaunch l{geo, prim, prims_sorted, tile_ranges, tile_order, out, tout, status, stream};
    switch (mode) {
        case HTGS_MODE_HYBRID_BLEND: return launch_mode<HTGS_MODE_HYBRID_BLEND>(l, task, view);
        case HTGS_MODE_ALPHA_BLEND_FIRST_K: return launch_mode<HTGS_MODE_ALPHA_BLEND_FIRST_K>(l, task, view);
        case HTGS_MODE_ALPHA_BLEND_GLOBAL_ORDERING: return launch_buffer<HTGS_MODE_ALPHA_BLEND_GLOBAL_ORDERING, 1, Buffer::chain>(l, task, 0);
        case HTGS_MODE_OIT_BLEND: return launch_buffer<HTGS_MODE_OIT_BLEND, 1, Buffer::chain>(l, task, 0);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace htgs
