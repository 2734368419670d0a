// Backward pass of the rasterizer.
//
// Replaces the backward blend_cu / preprocess_cu pairs of the reference
//   HYBRID_BLEND                rasterization/include/hybrid_blend/kernels/backward.cuh:10-331
//   ALPHA_BLEND_FIRST_K         rasterization/include/alpha_blend_first_k/kernels/backward.cuh:10-206
//   ALPHA_BLEND_GLOBAL_ORDERING rasterization/include/alpha_blend_global_ordering/kernels/backward.cuh:10-251
//   OIT_BLEND                   rasterization/include/oit_blend/kernels/backward.cuh:10-290
// and the helpers convert_quaternion_to_rotation_matrix_backward / convert_sh_to_rgb_backward
// (rasterization/include/kernel_utils.cuh:44-61, 190-281).
//
// The chain rule is the reference's: gradients flow through alpha = opacity * G and the colour only
// (not through depth, thresholds, the min(.,1) clamp or the bounds).  The organisation is new:
//  * every mode accumulates the same per-Gaussian record of five float4 with 16-byte vector reductions
//    (red.global.add.v4.f32) instead of 15-17 scalar atomics: 12 moments that stand for dL/dVPMT1, dL/dVPMT2, dL/dVPMT4 (below),
//    (dL/drgb, dL/dopacity) and sum |dL/dposition|.  One per-Gaussian kernel turns the record into the six output gradients
//    (the reference repeats the scale / rotation chain rule per fragment in two of its modes);
//  * HYBRID / FIRST_K / OIT: the (Gaussian, pixel) candidates of a batch are cut into segments of at most 16 pixels of one
//    Gaussian, one segment per lane.  The forward pass saves core entries as positions in the tile's list, so which pairs
//    are core entries is a table filled once per batch, not a search per pair;
//  * GLOBAL_ORDERING needs the running transmittance per pixel: one warp per 8x4 pixels walks the Gaussians that reach them, lane =
//    pixel, and leaves what only the pixel knows of a pair in a table; then lane = Gaussian sums the pairs of the table and
//    adds a record per Gaussian and warp.
#include "kernels.h"

#include <algorithm>

namespace htgs {

namespace {

__device__ __forceinline__ void red_add_v4(float4* addr, const float4& v) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}

// The backward pass is not bit-identical to the reference's in any case (its sums are atomic), so where a value only
// scales a gradient term it uses the hardware approximations (1 ulp reciprocal, 2 ulp exp2) instead of the IEEE sequences:
// about 25 of the ~160 instructions per pair.
__device__ __forceinline__ float rcp_approx(float x) { float y; asm("rcp.approx.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
__device__ __forceinline__ float exp_approx(float x) { float y; asm("ex2.approx.f32 %0, %1;" : "=f"(y) : "f"(x * 1.4426950408889634f)); return y; }

// The gradient of rho^2 = N / D, N = |m|^2, D = |d|^2, w.r.t. the rows VPMT1, VPMT2, VPMT4 (hybrid_blend/kernels/backward.cuh:258-285), in moments.
// Along a Gaussian's pixels m and d are affine and N and D quadratic in (x, y) = pixel - centre, a point that the
// preprocess chose (make_moment_centre; PairRecord has the coefficients), and as well in (s, y) with the sheared s = x + shear * y:  m = M0 + s Ms + y My,  d = D0 + s Ds + y Dy  (AffinePlanes).
// The shear makes Ms and My orthogonal: however long and slanted the ellipse, the terms of m do not cancel.  The rows' gradients
// are quadratic in (s, y) too, with coefficients that are the Gaussian's alone, so a pair only adds
//     u = dL/drho^2 / D  (times D at the centre, which the record divides by)  and  v = u N / D,  each times  1, s, y, ss, sy, yy
// to the Gaussian's record, and rows_from_moments applies the coefficients once per Gaussian.  Of the sum of v, which the rows of a scale
// all but cancel against the second moments of u, only v - u N is added up, which vanishes with the perspective: u N follows from the
// moments of u (a third to a half of the rounding of grad_scales).  That is 13 instructions per pair
// instead of 54 for the rows themselves, and offsets from the centre keep the sums well conditioned, where the rows' sums hold products with
// pixel coordinates that cancel later.
struct AffinePlanes { float3 M0, Ms, My, D0, Ds, Dy; float4 A, B; float shear; };     // A = VPMT1 - cx VPMT4, B = VPMT2 - cy VPMT4
// In double where sums are turned into rows: for a Gaussian a hundred times as long as thick the sheared My is a hundredth of its terms
// (in float32 the gradients of rotations lost 1e-5 of their norm by it).
template <typename Real>
__device__ __forceinline__ AffinePlanes affine_planes(const float4& T1, const float4& T2, const float4& T4, float cx, float cy, float shear) {
    struct R3 { Real x, y, z; };
    auto comb = [](Real p, const R3& a, Real q, const R3& b) { return R3{p * a.x + q * b.x, p * a.y + q * b.y, p * a.z + q * b.z}; };
    auto cross3 = [](const R3& a, const R3& b) { return R3{a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x}; };
    auto narrow = [](const R3& a) { return make_float3(float(a.x), float(a.y), float(a.z)); };
    const Real x = cx, y = cy, w = T4.w, sh = shear;
    const R3 n{T4.x, T4.y, T4.z}, a{T1.x - x * n.x, T1.y - x * n.y, T1.z - x * n.z}, b{T2.x - y * n.x, T2.y - y * n.y, T2.z - y * n.z};
    const Real aw = T1.w - x * w, bw = T2.w - y * w;
    const R3 ms = comb(bw, n, -w, b), ds = cross3(b, n);
    AffinePlanes p;
    p.A = make_float4(float(a.x), float(a.y), float(a.z), float(aw));
    p.B = make_float4(float(b.x), float(b.y), float(b.z), float(bw));
    p.M0 = narrow(comb(aw, b, -bw, a));
    p.D0 = narrow(cross3(a, b));
    p.Ms = narrow(ms);
    p.Ds = narrow(ds);
    p.My = narrow(comb(Real(1), comb(w, a, -aw, n), -sh, ms));
    p.Dy = narrow(comb(Real(1), cross3(n, a), -sh, ds));
    p.shear = shear;
    return p;
}

// N and D of a PairRecord at (s, y), side by side in one register pair: q0 = coefficients of 1 and s, q1 = of y and ss, q2 = of sy and yy.
// They are brought side by side when a record is staged.  Stored so, N takes the chain rule three loads per Gaussian instead of two (3 M Gaussians: 219 -> 225 us),
// and the pair loops gain nothing.
struct PairForm { float4 q0, q1, q2; };
__device__ __forceinline__ PairForm side_by_side(const float4& n0, const float4& n1, const float4& d1) {
    return {make_float4(n0.x, n1.z, n0.y, n1.w), make_float4(n0.z, d1.x, n0.w, d1.y), make_float4(n1.x, d1.z, n1.y, d1.w)};
}
__device__ __forceinline__ f32x2 low2(const float4& v) { return pack2(v.x, v.y); }
__device__ __forceinline__ f32x2 high2(const float4& v) { return pack2(v.z, v.w); }
__device__ __forceinline__ void evaluate_pair(const PairForm& f, float s, float y, float& numerator, float& denominator) {
    const f32x2 s2 = pack2(s, s), y2 = pack2(y, y);
    const float2 v = unpack2(fma2(high2(f.q2), mul2(y2, y2), fma2(low2(f.q2), mul2(s2, y2), fma2(high2(f.q1), mul2(s2, s2), fma2(low2(f.q1), y2, fma2(high2(f.q0), s2, low2(f.q0)))))));
    numerator = v.x;
    denominator = v.y;
}

// Whether the forward pass accepts a fragment is settled by rho^2 unless it lies within kLevelBand of the level where alpha meets
// its threshold (or rho^2 the cutoff); then the forward's own arithmetic is repeated.  The band is far wider than the
// difference between the quadratics and the forward's planes (a few 1e-6 of rho^2).
constexpr float kLevelBand = 5e-5f;
__device__ __forceinline__ float upper_level(float lower) { return fmaf(lower, 3.0f * kLevelBand, lower) + 4e-6f; }      // beyond it a fragment is certainly rejected
template <typename MT>
__device__ __forceinline__ float acceptance_level(float opacity) { return fminf(MT::max_cutoff_sq, 2.0f * __logf(opacity * MT::min_alpha_rcp)); }
template <typename MT>
__device__ __noinline__ bool accepted_by_forward(const EvalRecord* rec, float pixel_x, float pixel_y) {
    const float* r = reinterpret_cast<const float*>(rec);
    const float4 T1 = ldg4(r), T2 = ldg4(r + 4), T4 = ldg4(r + 8);
    const float opacity = __ldg(r + 19);
    const float4 plane_x_diag = T1 - T4 * pixel_x;
    const float4 plane_y_diag = T2 - T4 * pixel_y;
    const float3 m = plane_x_diag.w * f3(plane_y_diag) - f3(plane_x_diag) * plane_y_diag.w;
    const float3 d = cross(f3(plane_x_diag), f3(plane_y_diag));
    const float numerator_rho2 = dot(m, m), denominator = dot(d, d);
    const float G = expf(-0.5f * numerator_rho2 * (1.0f / denominator));
    return !(numerator_rho2 > MT::max_cutoff_sq * denominator) && !(fminf(opacity * G, kMaxFragmentAlpha) < MT::min_alpha);
}

// Sums over pairs, as pairs of registers: a pair of pixel offsets (s, y) serves both factors of a product.  13 instructions (single ones: 19).
struct PairMoments {
    f32x2 uv;                       // u, v - u N
    f32x2 u1, u2, v1, v2;           // us, uy | uss, uyy | vs, vy | vss, vyy
    float usy, vsy;
    __device__ __forceinline__ float4 row(int i) const {      // as they lie in the Gaussian's record
        const float2 a = unpack2(i == 0 ? uv : i == 1 ? u2 : v2), b = i == 2 ? make_float2(usy, vsy) : unpack2(i == 0 ? u1 : v1);
        return make_float4(a.x, a.y, b.x, b.y);
    }
};
__device__ __forceinline__ void add_moments(PairMoments& a, float u, float v, float uN, float s, float y) {
    const f32x2 sy = pack2(s, y), us_uy = mul2(pack2(u, u), sy), vs_vy = mul2(pack2(v, v), sy);
    a.uv = add2(a.uv, pack2(u, v - uN));
    a.u1 = add2(a.u1, us_uy);
    a.u2 = fma2(us_uy, sy, a.u2);
    a.v1 = add2(a.v1, vs_vy);
    a.v2 = fma2(vs_vy, sy, a.v2);
    a.usy = fmaf(unpack2(us_uy).x, y, a.usy);
    a.vsy = fmaf(unpack2(vs_vy).x, y, a.vsy);
}

// dL/dVPMT1 = sum dX, dL/dVPMT2 = sum dY, and E = sum (x dX + y dY), so that dL/dVPMT4 = -(cx sum dX + cy sum dY + E).  With
// X = A - x VPMT4, Y = B - y VPMT4, dm = 2 u m and dd = -2 v d:
//     dX = (Y x dd - Y.w dm, Y . dm),   dY = (X.w dm - X x dd, -X . dm)
// and the cubic terms of E cancel: x dX + y dY = ((x B - y A) x dd - (x B.w - y A.w) dm, (x B - y A) . dm).
struct RowGradients { float4 dX, dY, E; };
__device__ __forceinline__ RowGradients rows_from_moments(const AffinePlanes& p, const float4& T4, const float4& n0, const float4& n1, const float4& r0, const float4& r1, const float4& r2) {
    const float3 A = f3(p.A), B = f3(p.B), n = f3(T4);
    const float u = r0.x, us = r0.z, uy = r0.w, uss = r1.x, uyy = r1.y, usy = r2.z;      // PairMoments::row
    // the sum of v from that of v - u N; n0, n1: N as the pairs saw it
    const float v = r0.y + fmaf(n1.y, uyy, fmaf(n1.x, usy, fmaf(n0.w, uss, fmaf(n0.z, uy, fmaf(n0.y, us, n0.x * u))))), vs = r1.z, vy = r1.w, vss = r2.x, vsy = r2.w, vyy = r2.y;
    // sums of u m and v d, and of these times y and x = s - shear * y
    const float3 m1 = u * p.M0 + us * p.Ms + uy * p.My, my = uy * p.M0 + usy * p.Ms + uyy * p.My;
    const float3 d1 = v * p.D0 + vs * p.Ds + vy * p.Dy, dy = vy * p.D0 + vsy * p.Ds + vyy * p.Dy;
    const float3 mx = us * p.M0 + uss * p.Ms + usy * p.My - p.shear * my, dx = vs * p.D0 + vss * p.Ds + vsy * p.Dy - p.shear * dy;
    RowGradients g;
    const float3 gx = -(p.B.w * m1 - T4.w * my) - (cross(B, d1) - cross(n, dy));
    const float3 gy = (p.A.w * m1 - T4.w * mx) + (cross(A, d1) - cross(n, dx));
    const float3 ge = -(p.B.w * mx - p.A.w * my) - (cross(B, dx) - cross(A, dy));
    g.dX = make_float4(2.0f * gx.x, 2.0f * gx.y, 2.0f * gx.z, 2.0f * (dot(B, m1) - dot(n, my)));
    g.dY = make_float4(2.0f * gy.x, 2.0f * gy.y, 2.0f * gy.z, -2.0f * (dot(A, m1) - dot(n, mx)));
    g.E = make_float4(2.0f * ge.x, 2.0f * ge.y, 2.0f * ge.z, 2.0f * (dot(B, mx) - dot(A, my)));
    return g;
}

// sum |dL/dposition| needs every pair's own fourth column (dL/dVPMT1.w, dL/dVPMT2.w, dL/dVPMT4.w) = (Y . dm, -X . dm, ...)
struct CameraCols { float3 c1, c2, c3; };   // columns 1..3 of rows (1,2,4) of VPM
__device__ __forceinline__ CameraCols load_camera_cols(const float* __restrict__ VPM) {
    const float4 r1 = ldg4(VPM), r2 = ldg4(VPM + 4), r4 = ldg4(VPM + 12);
    return {make_float3(r1.x, r2.x, r4.x), make_float3(r1.y, r2.y, r4.y), make_float3(r1.z, r2.z, r4.z)};
}
// Y . m and X . m (3-vectors) as quadratics about the centre; the fourth columns of a pair are 2u times these.
struct AbsForm { float4 y0, x0, y1x1; };      // Y . m: 1, s, y, sy | X . m: 1, s, y, ss | Y . m: yy, X . m: sy, yy
__device__ __forceinline__ AbsForm abs_form(const EvalRecord* rec, const float4& centre_shear_scale) {
    const float* r = reinterpret_cast<const float*>(rec);
    const float4 T4 = ldg4(r + 8);
    const AffinePlanes p = affine_planes<float>(ldg4(r), ldg4(r + 4), T4, centre_shear_scale.x, centre_shear_scale.y, centre_shear_scale.z);
    const float3 a = f3(p.A), b = f3(p.B), n = f3(T4);
    const float scale = centre_shear_scale.w;
    const float nm0 = dot(n, p.M0), nms = dot(n, p.Ms), nmy = dot(n, p.My);
    return {scale * make_float4(dot(b, p.M0), dot(b, p.Ms), dot(b, p.My) - nm0, -nms), scale * make_float4(dot(a, p.M0), dot(a, p.Ms) - nm0, fmaf(p.shear, nm0, dot(a, p.My)), -nms),
            scale * make_float4(-nmy, fmaf(p.shear, nms, -nmy), p.shear * nmy, 0.0f)};
}
__device__ __forceinline__ float abs_position_gradient(const AbsForm& f, float u, float s, float y, float pixel_x, float pixel_y, const CameraCols& cam) {
    const float sy = s * y, yy = y * y;
    const float wx = 2.0f * u * fmaf(f.y1x1.x, yy, fmaf(f.y0.w, sy, fmaf(f.y0.z, y, fmaf(f.y0.y, s, f.y0.x))));
    const float wy = -2.0f * u * fmaf(f.y1x1.z, yy, fmaf(f.y1x1.y, sy, fmaf(f.x0.w, s * s, fmaf(f.x0.z, y, fmaf(f.x0.y, s, f.x0.x)))));
    const float wz = -pixel_x * wx - pixel_y * wy;
    const float3 c4 = make_float3(wx, wy, wz);
    return fabsf(dot(cam.c1, c4)) + fabsf(dot(cam.c2, c4)) + fabsf(dot(cam.c3, c4));
}

__device__ __forceinline__ float small_int_to_float(uint32_t i) { return __uint_as_float(0x4b000000u | i) - 8388608.0f; }      // i < 2^23; off the pipe of the conversions

constexpr int kBwdThreads = 128;       // threads per tile: one staged instance each
constexpr int kBwdSegments = 4 * kBwdThreads;      // of a batch, at most
constexpr int kBwdCoreRow = 68;        // bytes per staged instance: 64 pixels, and an odd number of words against bank conflicts
template <int MODE, int K, bool ABS_GRAD> struct BwdSmem {
    static constexpr bool has_core = (MODE == HTGS_MODE_HYBRID_BLEND || MODE == HTGS_MODE_ALPHA_BLEND_FIRST_K);
    static constexpr bool has_tail = (MODE == HTGS_MODE_HYBRID_BLEND || MODE == HTGS_MODE_OIT_BLEND);
    static constexpr int core_rows = has_core ? K : 0;
    static constexpr size_t cg_off = 0;
    static constexpr size_t cg_bytes = has_core ? size_t(K) * 64 * 16 : 0;
    static constexpr size_t tc_off = cg_off + cg_bytes;
    static constexpr size_t tc_bytes = has_tail ? 64 * 16 : 0;
    static constexpr size_t ta_off = tc_off + tc_bytes;
    static constexpr size_t ta_bytes = has_tail ? 64 * 4 : 0;
    static constexpr size_t zero_off = ta_off + ta_bytes;      // 16 bytes of zeros: the terms of a pair that is not accepted
    static constexpr size_t stage_off = zero_off + 16;
    static constexpr size_t stage_bytes = kBwdThreads * ((ABS_GRAD ? 8 : 5) * 16 + 4 + (MODE == HTGS_MODE_ALPHA_BLEND_FIRST_K ? 8 : 0)) + kBwdSegments * (4 + 1);
    static constexpr size_t core_off = (stage_off + stage_bytes + 15) & ~size_t(15);     // [NT][kBwdCoreRow] core entry of each (staged instance, pixel) pair
    static constexpr size_t core_bytes = has_core ? size_t(kBwdThreads) * kBwdCoreRow : 0;
    static constexpr size_t total = core_off + core_bytes;
    // Five spill the pair loop, which pays only for OIT_BLEND, whose loop reads no buffer (1297 x 840, 1 and 3 M Gaussians: four blocks 291 and 428 us, five 280
    // and 424; five with one pair per trip 283 and 430, four with one 300 and 444).  The bound of four spills up to 32 bytes in HYBRID_BLEND
    // with absolute gradients and 20 with K = 32; one pair per trip, which spilled 4 and none, was slower in all of them (1 M Gaussians, absolute gradients, K = 2, 4,
    // 8, 16, 32: 431, 422, 432, 444, 581 -> 396, 401, 399, 409, 501; K = 32 without: 478 -> 441).
    static constexpr int max_blocks = MODE == HTGS_MODE_OIT_BLEND && !ABS_GRAD ? 5 : 4;
    static constexpr int min_blocks = int((227 * 1024) / (total + 1024)) < max_blocks ? int((227 * 1024) / (total + 1024)) : max_blocks;   // what the register budget is held to
};

// HYBRID_BLEND / ALPHA_BLEND_FIRST_K / OIT_BLEND: one CTA per 8x8 tile (long lists first), one thread per Gaussian of a batch of kBwdThreads.
template <int MODE, int K, bool ABS_GRAD>
__global__ void __launch_bounds__(kBwdThreads, (BwdSmem<MODE, K, ABS_GRAD>::min_blocks)) backward_tile_kernel(
    const uint2* __restrict__ tile_ranges, const uint32_t* __restrict__ tile_order, const uint32_t* __restrict__ prims_sorted, const EvalRecord* __restrict__ eval,
    const CullRecord* __restrict__ cull, const PairRecord* __restrict__ pair, TrainPixelBuffers tin, const float* __restrict__ grad_image, const float* __restrict__ VPM,
    float4* __restrict__ accum, uint32_t width, uint32_t height, uint32_t grid_w, uint32_t g_first, uint32_t g_end)
{
    using MT = ModeTraits<MODE>;
    using SM = BwdSmem<MODE, K, ABS_GRAD>;
    constexpr bool kHybrid = MODE == HTGS_MODE_HYBRID_BLEND;
    constexpr bool kFirstK = MODE == HTGS_MODE_ALPHA_BLEND_FIRST_K;
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr uint32_t kNotCore = kFirstK ? 0xffu : uint32_t(SM::core_rows);      // in s_core: not a core entry
    [[maybe_unused]] unsigned char* s_core = smem + SM::core_off;
    float4* s_terms = reinterpret_cast<float4*>(smem + SM::cg_off);                        // [K][64] (W * grad_pixel, A . grad_pixel), then s_tc
    [[maybe_unused]] float4* s_tc = reinterpret_cast<float4*>(smem + SM::tc_off);          // [64] (full_weight * grad_pixel, common term)
    [[maybe_unused]] float* s_ta = reinterpret_cast<float*>(smem + SM::ta_off);            // [64] term divided by (1 - alpha)

    const uint32_t tid = threadIdx.x;
    const uint32_t tile = __ldg(tile_order + blockIdx.x);
    const uint32_t tile_x = tile % grid_w, tile_y = tile / grid_w;
    const uint2 tile_range = tile_ranges[tile];
    uint2 range = tile_range;
    // A pass over the Gaussians [g_first, g_end) only: a tile's list is ascending in Gaussian index for these modes (instances
    // are emitted in index order and the tile sort is stable), so the pass walks one contiguous piece of it.
    if (g_first != 0u || g_end != 0xffffffffu) {
        auto lower_bound = [&](uint32_t lo, uint32_t hi, uint32_t g) {
            while (lo < hi) { const uint32_t mid = (lo + hi) >> 1; if (__ldg(prims_sorted + mid) < g) lo = mid + 1; else hi = mid; }
            return lo;
        };
        range.x = lower_bound(tile_range.x, tile_range.y, g_first);
        range.y = lower_bound(range.x, tile_range.y, g_end);
    }
    if (range.x >= range.y) return;
    const uint32_t n_pixels = width * height;
    const uint32_t PP = tin.padded_pixels;
    constexpr uint32_t NT = kBwdThreads, kParts = NT / 64;
    const uint32_t pix = tid & 63, part = tid >> 6;          // the per-pixel terms are set up by kParts threads per pixel
    const uint32_t slot = tile * 64 + pix;
    const float x0 = float(tile_x * 8), y0 = float(tile_y * 8);
    // pixels of the tile that exist in the image, as a 64-bit mask (bit = row * 8 + column)
    uint64_t inside_mask = 0;
    {
        const uint32_t cols = min(8u, width - tile_x * 8), rows = min(8u, height - tile_y * 8);
        const uint64_t row_bits = (1ull << cols) - 1ull;
        for (uint32_t r = 0; r < rows; ++r) inside_mask |= row_bits << (8 * r);
    }

    // Software pipeline of the staging loads.  While batch b is processed, the outlines of batch b + 1 (requested one batch earlier)
    // give the pixel masks, the records of those instances that touch a pixel (six in ten) are requested, then the outlines of
    // batch b + 2 and the indices of batch b + 3.
    uint32_t g_rec = 0, g_out = 0, g_idx = 0;
    float4 rN0 = make_float4(0, 0, 0, 0), rN1 = rN0, rD1 = rN0, rC = rN0, rRGBA = rN0, outline = rN0;     // rC: centre, shear, 1 / D at the centre
    float outline_c = 0.0f;
    uint64_t mask_rec = 0;
    auto load_index = [&](uint32_t inst) { return inst < range.y ? __ldg(prims_sorted + inst) : 0u; };
    auto request_outline = [&](uint32_t inst) {
        if (inst >= range.y) return;
        outline = ldg4(reinterpret_cast<const float*>(cull + g_out));
        outline_c = __ldg(reinterpret_cast<const float*>(cull + g_out) + 4);
    };
    auto request_record = [&](uint32_t inst) {              // of the instance whose outline has arrived
        mask_rec = 0;
        if (inst < range.y) mask_rec = (uint64_t(outline_mask(outline, outline_c, x0, y0)) | (uint64_t(outline_mask(outline, outline_c, x0, y0 + 4.0f)) << 32)) & inside_mask;
        if (mask_rec == 0) return;
        g_rec = g_out;
        const float* rec = reinterpret_cast<const float*>(pair + g_rec);
        rN0 = ldg4(rec); rN1 = ldg4(rec + 4); rD1 = ldg4(rec + 8); rC = ldg4(rec + 12);
        rRGBA = ldg4(reinterpret_cast<const float*>(eval + g_rec) + 16);
    };
    g_out = load_index(range.x + tid);
    g_idx = load_index(range.x + NT + tid);
    request_outline(range.x + tid);
    // ---- per-pixel terms of this tile (hybrid_blend/kernels/backward.cuh:137-176, oit_blend/kernels/backward.cuh:131-156)
    // core_pos: this thread's share of the pixel's core entries, as positions in the tile's list
    [[maybe_unused]] uint32_t core_pos[SM::has_core ? (K + kParts - 1) / kParts : 1];
    {
        const uint32_t px_i = tile_x * 8 + (pix & 7), py_i = tile_y * 8 + (pix >> 3);
        const bool inside = px_i < width && py_i < height;
        float3 grad_pixel = make_float3(0.0f, 0.0f, 0.0f);
        if (inside) {
            const uint32_t pixel_idx = width * py_i + px_i;
            grad_pixel = make_float3(__ldg(grad_image + pixel_idx), __ldg(grad_image + n_pixels + pixel_idx), __ldg(grad_image + 2 * n_pixels + pixel_idx));
        }
        if constexpr (SM::has_core) {
            // All loads of a group are in flight together; entries that do not exist are read (their slots do) and dropped.
            constexpr int kShare = (K + int(kParts) - 1) / int(kParts), kGroup = kShare < 8 ? kShare : 8;
            #pragma unroll
            for (int i0 = 0; i0 < kShare; i0 += kGroup) {
                float4 info[kGroup];
                #pragma unroll
                for (int i = 0; i < kGroup; ++i) {
                    const int k = min((i0 + i) * int(kParts) + int(part), K - 1);
                    core_pos[i0 + i] = __ldg(tin.idx_core + k * PP + slot);
                    info[i] = __ldg(tin.info_core + k * PP + slot);
                }
                #pragma unroll
                for (int i = 0; i < kGroup; ++i) {
                    const int k = (i0 + i) * int(kParts) + int(part);
                    if (k >= K || !inside) core_pos[i0 + i] = 0xffffffffu;
                    const float3 drgb = info[i].w * grad_pixel;
                    if (k < K) s_terms[k * 64 + pix] = make_float4(drgb.x, drgb.y, drgb.z, dot(f3(info[i]), grad_pixel));
                }
            }
        }
        if constexpr (SM::has_tail) {
            if (part == 0) {
                float4 tc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                float ta = 0.0f;
                if (inside) {
                    const float3 rgb_tail = make_float3(tin.info_tail[slot], tin.info_tail[PP + slot], tin.info_tail[2 * PP + slot]);
                    const float alpha_sum_rcp = tin.info_tail[3 * PP + slot];
                    const float transmittance_tail = tin.info_tail[4 * PP + slot];
                    const float transmittance_core = kHybrid ? tin.info_tail[5 * PP + slot] : 1.0f;
                    const float weight_tail = transmittance_core * alpha_sum_rcp;
                    const float full_weight_tail = weight_tail * (1.0f - transmittance_tail);
                    const float rgb_dot_grad = dot(rgb_tail, grad_pixel);
                    const float3 part = full_weight_tail * grad_pixel;
                    tc = make_float4(part.x, part.y, part.z, -full_weight_tail * alpha_sum_rcp * rgb_dot_grad);
                    ta = weight_tail * transmittance_tail * rgb_dot_grad;
                }
                s_tc[pix] = tc;
                s_ta[pix] = ta;
            }
        }
    }
    if (tid == 0) s_terms[SM::zero_off / 16] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    [[maybe_unused]] CameraCols cam;
    if constexpr (ABS_GRAD) cam = load_camera_cols(VPM);
    request_record(range.x + tid);
    g_out = g_idx;
    request_outline(range.x + NT + tid);
    g_idx = load_index(range.x + 2 * NT + tid);

    // ---- batches of NT instances.  A Gaussian's pixels are cut into segments of at most 16 (two rows; four rows if they hold no
    //      more); a lane takes one segment, sums its record in registers and adds it to the Gaussian's.  All lanes of a warp change
    //      Gaussians at the same time: with the pairs split evenly over the lanes instead, some lane changed in almost every step,
    //      and the warp spent a third of its instructions on that (1450 -> 1290 us at 3 M Gaussians, 1297 x 840, K = 16).
    float4* s_q0 = reinterpret_cast<float4*>(smem + SM::stage_off);
    float4* s_q1 = s_q0 + NT;
    float4* s_q2 = s_q1 + NT;
    float4* s_rgba = s_q2 + NT;
    float4* s_pos = s_rgba + NT;         // tile origin - centre, rho^2 below which a fragment is certainly accepted, shear
    [[maybe_unused]] float4* s_abs = s_pos + NT;    // ABS_GRAD: [3][NT]
    [[maybe_unused]] unsigned long long* s_mask = reinterpret_cast<unsigned long long*>(s_pos + NT * (ABS_GRAD ? 4 : 1));      // FIRST_K
    uint32_t* s_g = reinterpret_cast<uint32_t*>(s_mask + (kFirstK ? NT : 0));
    uint32_t* s_segment = s_g + NT;      // pixels of a segment, 32 of the tile's 64
    unsigned char* s_owner = reinterpret_cast<unsigned char*>(s_segment + kBwdSegments);      // staged instance * 2 + which 32 pixels
    __shared__ uint32_t s_warp_total[NT / 32];
    const uint32_t lane = tid & 31, warp = tid >> 5;
    // The training forward saved, per pixel and core entry, the POSITION of the entry's Gaussian in the tile's list, so the
    // entries that belong to a batch are those within NT of its start, and position - start is the staged slot.
    // FIRST_K gives gradient to stored fragments only: there the entries also set the pixel masks of the staged instances.
    // `limit`: staged instances of the batch (entries further down the list belong to a later batch, or - in a pass over a
    // range of Gaussians - to Gaussians beyond the range, whose slots in this batch hold nothing).
    [[maybe_unused]] auto scatter_core_entries = [&](uint32_t batch_pos, uint32_t limit) {
        #pragma unroll
        for (int i = 0; i < int((K + kParts - 1) / kParts); ++i) {
            const uint32_t j = core_pos[i] - batch_pos;
            if (j < limit) {
                s_core[j * kBwdCoreRow + pix] = (unsigned char)(i * int(kParts) + int(part));
                if constexpr (kFirstK) atomicOr(reinterpret_cast<uint32_t*>(s_mask + j) + (pix >> 5), 1u << (pix & 31));
            }
        }
    };
    for (uint32_t batch_begin = range.x; batch_begin < range.y; batch_begin += NT) {
        __syncthreads();                  // previous batch fully consumed
        const uint32_t inst = batch_begin + tid;
        uint64_t my_mask = mask_rec;
        if (my_mask != 0) {
            const PairForm form = side_by_side(rN0, rN1, rD1);
            s_q0[tid] = form.q0; s_q1[tid] = form.q1; s_q2[tid] = form.q2; s_rgba[tid] = rRGBA;
            float level = 0.0f;
            if constexpr (!kFirstK) level = acceptance_level<MT>(rRGBA.w);
            const float band = kLevelBand * level + 1e-6f;
            s_pos[tid] = make_float4(x0 - rC.x, y0 - rC.y, level - band, rC.z);
            if constexpr (ABS_GRAD) {
                const AbsForm af = abs_form(eval + g_rec, rC);
                s_abs[tid] = af.y0; s_abs[NT + tid] = af.x0; s_abs[2 * NT + tid] = af.y1x1;
            }
            s_g[tid] = g_rec;
            if constexpr (SM::has_core) {      // no pair of my instance is a core entry until the scatter below says so
                uint32_t* row = reinterpret_cast<uint32_t*>(s_core + tid * kBwdCoreRow);
                #pragma unroll
                for (int i = 0; i < 16; ++i) row[i] = kNotCore * 0x01010101u;
            }
        }
        request_record(inst + NT);
        g_out = g_idx;
        request_outline(inst + 2 * NT);
        g_idx = load_index(inst + 3 * NT);
        if constexpr (kFirstK) {
            s_mask[tid] = 0;
            __syncthreads();
            scatter_core_entries(batch_begin - tile_range.x, min(NT, range.y - batch_begin));   // the forward's stored core positions count from the start of the tile's list
            __syncthreads();
            my_mask = s_mask[tid];
        }
        // segments with more than 8 pixels come first, so that the lanes of a warp have about equally many steps
        const uint32_t halves[2] = {uint32_t(my_mask), uint32_t(my_mask >> 32)};
        uint32_t segments[4], cnt = 0;                   // low half word: long segments, high half word: short ones
        #pragma unroll
        for (int h = 0; h < 2; ++h) {
            const bool split = __popc(halves[h]) > 16;
            segments[2 * h] = split ? halves[h] & 0xffffu : halves[h];
            segments[2 * h + 1] = split ? halves[h] & 0xffff0000u : 0u;
        }
        #pragma unroll
        for (int i = 0; i < 4; ++i) cnt += segments[i] == 0 ? 0u : __popc(segments[i]) > 8 ? 1u : 0x10000u;
        uint32_t inc = cnt;
        #pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o); if (lane >= uint32_t(o)) inc += t; }
        if (lane == 31) s_warp_total[warp] = inc;
        __syncthreads();
        uint32_t at = inc - cnt, total = 0;
        #pragma unroll
        for (uint32_t w = 0; w < NT / 32; ++w) {
            const uint32_t t = s_warp_total[w];
            if (w < warp) at += t;
            total += t;
        }
        const uint32_t n_long = total & 0xffffu, n_segments = n_long + (total >> 16);
        uint32_t at_long = at & 0xffffu, at_short = n_long + (at >> 16);
        #pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (segments[i] == 0) continue;
            const uint32_t slot_at = __popc(segments[i]) > 8 ? at_long++ : at_short++;
            s_segment[slot_at] = segments[i];
            s_owner[slot_at] = (unsigned char)(2 * tid + i / 2);
        }
        if constexpr (SM::has_core && !kFirstK) scatter_core_entries(batch_begin - tile_range.x, min(NT, range.y - batch_begin));   // the forward's stored core positions count from the start of the tile's list
        __syncthreads();
        for (uint32_t first = warp * 32; first < n_segments; first += NT) {
            const bool has_segment = first + lane < n_segments;
            uint32_t pixels = has_segment ? s_segment[first + lane] : 0u;
            const uint32_t owner = s_owner[min(first + lane, n_segments - 1u)], j = owner >> 1;
            const float row0 = float((owner & 1u) * 4u);
            const PairForm form{s_q0[j], s_q1[j], s_q2[j]};
            const float4 rgba = s_rgba[j], pos = s_pos[j];
            PairMoments moments{};
            f32x2 aC_rg = pack2(0.0f, 0.0f);                // dL/drgb and dL/dopacity
            float aC_b = 0.0f, aC_opacity = 0.0f;
            [[maybe_unused]] float abs_grad = 0.0f;
            bool touched = false;
            const uint32_t first_pixel = (owner & 1u) * 32u;
            // Two pairs per trip, without a branch behind the test: independent instruction streams, which the 14 warps of an SM that registers
            // and shared memory leave need (they issue on half of the cycles).  3 M Gaussians, 1297 x 840, K = 16: one pair with single
            // instructions and branches for core and tail 980 us; packed, one row of terms for both 917; two pairs 873; without the branch 865.
            // OIT 233 -> 226, FIRST_K 123 -> 111 (0.5 M, 800 x 600).
            struct Pair { float s, y, rho2, numerator, denominator_rcp, column, row; uint32_t terms, p; bool ok; };
            auto look = [&](uint32_t bit, bool valid) -> Pair {
                Pair r;
                r.p = bit + first_pixel;
                r.column = small_int_to_float(bit & 7u); r.row = row0 + small_int_to_float(bit >> 3);
                r.y = pos.y + r.row; r.s = fmaf(pos.w, r.y, pos.x + r.column);
                float denominator;
                evaluate_pair(form, r.s, r.y, r.numerator, denominator);
                // the row of the pixel's terms: a core entry's, or that of the tail behind them
                r.terms = 0;
                if constexpr (SM::has_core) r.terms = s_core[j * kBwdCoreRow + r.p];
                r.denominator_rcp = rcp_approx(denominator);
                r.rho2 = r.numerator * r.denominator_rcp;
                if constexpr (kFirstK) {
                    r.ok = valid && r.terms != kNotCore;           // only stored fragments carry gradient (first_k backward.cuh:84-87)
                } else {
                    r.ok = valid && r.rho2 < pos.z;
                    if (valid && !r.ok && !(r.rho2 > upper_level(pos.z))) r.ok = accepted_by_forward<MT>(eval + s_g[j], x0 + r.column, y0 + r.row);
                }
                return r;
            };
            // Of a pair that is not accepted only zeros, read as such: its pixel's gradient may be an infinity or a NaN, which times zero is a NaN.
            auto add = [&](Pair r) {
                if (!r.ok) r.rho2 = r.numerator = r.denominator_rcp = 0.0f;
                const float G = exp_approx(-0.5f * r.rho2);
                const float alpha = fminf(rgba.w * G, kMaxFragmentAlpha);
                const float4 term = s_terms[r.ok ? r.terms * 64 + r.p : uint32_t(SM::zero_off / 16)];
                float dL_dalpha = term.w, scale = 1.0f;
                if constexpr (SM::has_tail) {            // both, since in almost every step some lanes have the one and some the other
                    const float tail_dL_dalpha = term.w + dot(f3(rgba), f3(term)) + s_ta[r.p] * rcp_approx(fmaxf(1.0f - alpha, kOneMinusAlphaEps));
                    const bool core = !r.ok || r.terms < uint32_t(SM::core_rows);
                    scale = core ? 1.0f : alpha;
                    dL_dalpha = core ? dL_dalpha : tail_dL_dalpha;
                }
                aC_rg = fma2(low2(term), pack2(scale, scale), aC_rg);
                aC_b = fmaf(term.z, scale, aC_b);
                aC_opacity = fmaf(dL_dalpha, G, aC_opacity);
                touched |= r.ok;
                const float u = -0.5f * dL_dalpha * rgba.w * G * r.denominator_rcp;      // dL/drho^2 / D, times D at the centre
                add_moments(moments, u, u * r.rho2, u * r.numerator, r.s, r.y);
                if constexpr (ABS_GRAD)
                    abs_grad += abs_position_gradient(AbsForm{s_abs[j], s_abs[NT + j], s_abs[2 * NT + j]}, u, r.s, r.y, x0 + r.column, y0 + r.row, cam);
            };
            while (pixels != 0) {
                const uint32_t bit0 = uint32_t(__ffs(int(pixels)) - 1);
                pixels &= pixels - 1;
                const bool second = pixels != 0;
                const uint32_t bit1 = second ? uint32_t(__ffs(int(pixels)) - 1) : bit0;
                pixels &= pixels - 1;
                const Pair a = look(bit0, true), b = look(bit1, second);
                add(a);
                add(b);
            }
            // The segments of a Gaussian (at most four) lie side by side, but for the border between long and short ones: they are added up
            // before they go out, since it is the number of additions to a record that its rounding grows with.
            const uint32_t key = has_segment ? j : ~lane;
            const bool join_1 = __shfl_down_sync(0xffffffffu, key, 1) == key && lane < 31;
            const uint32_t joined_1 = __ballot_sync(0xffffffffu, join_1), joined_2 = joined_1 & (joined_1 >> 1);      // with the next lane, with the next but one
            auto join = [&](float& x, int o, bool take) { const float t = __shfl_down_sync(0xffffffffu, x, o); if (take) x += t; };
            auto join2 = [&](f32x2& x, int o, bool take) { const f32x2 t = __shfl_down_sync(0xffffffffu, x, o); if (take) x = add2(x, t); };
            auto join_all = [&](int o, bool take) {
                join2(moments.uv, o, take); join2(moments.u1, o, take); join2(moments.u2, o, take); join2(moments.v1, o, take); join2(moments.v2, o, take);
                join(moments.usy, o, take); join(moments.vsy, o, take);
                join2(aC_rg, o, take); join(aC_b, o, take); join(aC_opacity, o, take);
                if constexpr (ABS_GRAD) join(abs_grad, o, take);
            };
            uint32_t out = __ballot_sync(0xffffffffu, touched);
            if (joined_1 != 0) {
                join_all(1, join_1);
                out |= joined_1 & (out >> 1);
            }
            if (joined_2 != 0) {
                join_all(2, (joined_2 >> lane) & 1u);
                out |= joined_2 & (out >> 2);
            }
            if (((out & ~(joined_1 << 1)) >> lane) & 1u) {
                float4* rec = accum + size_t(s_g[j]) * 5;
                red_add_v4(rec, moments.row(0)); red_add_v4(rec + 1, moments.row(1)); red_add_v4(rec + 2, moments.row(2));
                red_add_v4(rec + 3, make_float4(unpack2(aC_rg).x, unpack2(aC_rg).y, aC_b, aC_opacity));
                if constexpr (ABS_GRAD) red_add_v4(rec + 4, make_float4(abs_grad, 0.0f, 0.0f, 0.0f));
            }
        }
    }
}

// ALPHA_BLEND_GLOBAL_ORDERING: front to back in key order, using the final pixel colour so that
// "colour behind" = rgb_pixel - rgb_pixel_new (alpha_blend_global_ordering/kernels/backward.cuh:104-161).
// One warp per 8x4 pixels (an eighth of a binning tile; a pixel shares no state with its neighbours), long lists first; it stops
// when its pixels are opaque.  The list is filtered against the block as in the forward pass and taken in chunks of 16 survivors:
//  1. lane = survivor: its record becomes the quadratics of N and D (PairForm) in shared memory; the masks are transposed;
//  2. lane = pixel: walks its own candidates in order and leaves per pair what only the pixel knows - blending weight, dL/dG / opacity,
//     rho^2, 1 / D - in a table, and a bit for every accepted pair;
//  3. lane = (survivor, half of the pixels): walks the accepted pairs of its survivor and sums the moments in registers; the
//     two halves are added and the record goes out with vector reductions.
// The warp never reduces over pixels (which took 64 instructions per Gaussian and warp, whether one pixel or 32 contributed).
constexpr int kGoChunk = 16;
constexpr int kGoQueue = 64;
template <bool ABS_GRAD>
__global__ void __launch_bounds__(32) backward_global_kernel(
    const uint2* __restrict__ tile_ranges, const uint32_t* __restrict__ tile_order, const uint32_t* __restrict__ prims_sorted, const EvalRecord* __restrict__ eval,
    const CullRecord* __restrict__ cull, const PairRecord* __restrict__ pair, const float* __restrict__ grad_image, const float* __restrict__ image, const float* __restrict__ VPM,
    float4* __restrict__ accum, uint32_t width, uint32_t height, uint32_t grid_w)
{
    using MT = ModeTraits<HTGS_MODE_ALPHA_BLEND_GLOBAL_ORDERING>;
    constexpr uint32_t kTileX = MT::tile_w / 8, kTileY = MT::tile_h / 4;
    __shared__ float4 s_pair[kGoChunk][33];              // [survivor][pixel]: weight, dL/dalpha * G, rho^2, 1 / D; zeros in the column behind the pixels
    __shared__ float4 s_q0[kGoChunk], s_q1[kGoChunk], s_q2[kGoChunk], s_rgba[kGoChunk], s_pos[kGoChunk];
    __shared__ float4 s_grad[33];                        // dL/dpixel, and zeros
    __shared__ uint32_t s_g[kGoChunk], s_queue_prim[kGoQueue], s_queue_mask[kGoQueue];
    const uint32_t lane = threadIdx.x;
    const uint32_t tile = __ldg(tile_order + blockIdx.x / (kTileX * kTileY)), part = blockIdx.x % (kTileX * kTileY);
    const uint32_t block_x = (tile % grid_w) * kTileX + part % kTileX, block_y = (tile / grid_w) * kTileY + part / kTileX;
    if (block_x * 8 >= width || block_y * 4 >= height) return;
    const uint32_t px_i = block_x * 8 + (lane & 7u), py_i = block_y * 4 + (lane >> 3);
    const bool inside = px_i < width && py_i < height;
    const float x0 = float(block_x * 8), y0 = float(block_y * 4);
    const float local_x = float(lane & 7u), local_y = float(lane >> 3);
    const uint32_t n_pixels = width * height;
    float3 grad_pixel = make_float3(0, 0, 0), rgb_pixel = make_float3(0, 0, 0);
    if (inside) {
        const uint32_t pixel_idx = width * py_i + px_i;
        grad_pixel = make_float3(__ldg(grad_image + pixel_idx), __ldg(grad_image + n_pixels + pixel_idx), __ldg(grad_image + 2 * n_pixels + pixel_idx));
        rgb_pixel = make_float3(__ldg(image + pixel_idx), __ldg(image + n_pixels + pixel_idx), __ldg(image + 2 * n_pixels + pixel_idx));
    }
    s_grad[lane] = make_float4(grad_pixel.x, grad_pixel.y, grad_pixel.z, 0.0f);
    if (lane < kGoChunk) s_pair[lane][32] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (lane == 0) s_grad[32] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    [[maybe_unused]] CameraCols cam;
    if constexpr (ABS_GRAD) cam = load_camera_cols(VPM);
    float3 rgb_pixel_new = make_float3(0, 0, 0);
    float transmittance = 1.0f;
    bool done = !inside;

    const uint2 range = tile_ranges[tile];
    uint32_t next = range.x + lane;
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
        if (next < range.y) mask = outline_mask(outline, outline_c, x0, y0);
        const uint32_t survivors = __ballot_sync(0xffffffffu, mask != 0);
        if (mask != 0) {
            const uint32_t at = (queue_head + queued + __popc(survivors & lanemask_lt())) & uint32_t(kGoQueue - 1);
            s_queue_prim[at] = g_here;
            s_queue_mask[at] = mask;
        }
        queued += __popc(survivors);
        next += 32;
        g_here = g_ahead;
        if (next < range.y) request_outline(g_here);
        if (next + 32 < range.y) g_ahead = __ldg(prims_sorted + next + 32);
    };
    // the record of the survivor this lane stages (both half warps hold the same 16)
    const uint32_t mine = lane & uint32_t(kGoChunk - 1);
    uint32_t g_mine = 0, mask_mine = 0, count = 0;
    float4 rN0 = make_float4(0, 0, 0, 0), rN1 = rN0, rD1 = rN0, rC = rN0, rRGBA = rN0;
    auto take = [&]() {                                  // the next chunk: indices, masks, and requests for its records
        while (queued < kGoChunk && next - lane < range.y) filter();
        __syncwarp();
        count = min(queued, uint32_t(kGoChunk));
        mask_mine = 0;
        if (mine < count) {
            const uint32_t at = (queue_head + mine) & uint32_t(kGoQueue - 1);
            g_mine = s_queue_prim[at];
            mask_mine = s_queue_mask[at];
            const float* rec = reinterpret_cast<const float*>(pair + g_mine);
            rN0 = ldg4(rec); rN1 = ldg4(rec + 4); rD1 = ldg4(rec + 8); rC = ldg4(rec + 12);
            rRGBA = ldg4(reinterpret_cast<const float*>(eval + g_mine) + 16);
        }
        queue_head += count;
        queued -= count;
        __syncwarp();
    };
    take();
    while (count != 0) {
        const uint32_t g = g_mine;
        // ---- 1. lane = survivor ------------------------------------------------------------------------------------
        [[maybe_unused]] AbsForm af{};
        if (mine < count) {
            if (lane < kGoChunk) {
                const PairForm form = side_by_side(rN0, rN1, rD1);
                s_q0[mine] = form.q0; s_q1[mine] = form.q1; s_q2[mine] = form.q2; s_rgba[mine] = rRGBA;
                const float level = acceptance_level<MT>(rRGBA.w);
                const float band = kLevelBand * level + 1e-6f;
                s_pos[mine] = make_float4(x0 - rC.x, y0 - rC.y, level - band, rC.z);
                s_g[mine] = g;
            }
            if constexpr (ABS_GRAD) af = abs_form(eval + g, rC);
        }
        const float opacity = rRGBA.w;
        const float offset_x = x0 - rC.x, offset_y = y0 - rC.y, shear = rC.z;
        uint32_t candidates = transpose_masks(lane < kGoChunk ? mask_mine : 0u, lane);      // bit 15 - i: survivor i
        if (done) candidates = 0;
        __syncwarp();
        take();                                          // the records of the next chunk fly while this one is worked on
        // ---- 2. lane = pixel ------------------------------------------------------------------------------------------
        uint32_t accepted = 0;
        // What does not depend on the transmittance can be evaluated for two candidates side by side.  1.5 M Gaussians, 980 x 545: with absolute gradients
        // 692 us with one per trip, 662 with two; without them 579 and 604.  (Before, with one pair per trip in part 3 too: 717 and 593.)
        struct Seen { float rho2, denominator_rcp, G, alpha; uint32_t bit; bool ok; };
        auto look = [&]() -> Seen {
            Seen r;
            const bool valid = candidates != 0;
            r.bit = uint32_t(31 - __clz(int(candidates | 1u)));
            candidates &= ~(1u << r.bit);
            const uint32_t j = uint32_t(kGoChunk - 1) - r.bit;
            const float4 pos = s_pos[j];
            const float y = pos.y + local_y, s = fmaf(pos.w, y, pos.x + local_x);
            float numerator_rho2, denominator;
            evaluate_pair(PairForm{s_q0[j], s_q1[j], s_q2[j]}, s, y, numerator_rho2, denominator);
            r.denominator_rcp = rcp_approx(denominator);
            r.rho2 = numerator_rho2 * r.denominator_rcp;
            r.ok = valid && r.rho2 < pos.z;
            if (valid && !r.ok && !(r.rho2 > upper_level(pos.z))) r.ok = accepted_by_forward<MT>(eval + s_g[j], x0 + local_x, y0 + local_y);
            r.G = exp_approx(-0.5f * r.rho2);
            r.alpha = fminf(s_rgba[j].w * r.G, kMaxFragmentAlpha);
            return r;
        };
        auto blend = [&](const Seen& r) {
            if (!r.ok || done) return;
            const uint32_t j = uint32_t(kGoChunk - 1) - r.bit;
            const float3 rgb = f3(s_rgba[j]);
            const float blending_weight = transmittance * r.alpha;
            rgb_pixel_new += blending_weight * rgb;
            const float one_minus_alpha = 1.0f - r.alpha;
            const float one_minus_alpha_rcp = rcp_approx(fmaxf(one_minus_alpha, kOneMinusAlphaEps));
            const float dL_dalpha = dot(transmittance * rgb - (rgb_pixel - rgb_pixel_new) * one_minus_alpha_rcp, grad_pixel);
            s_pair[j][lane] = make_float4(blending_weight, dL_dalpha * r.G, r.rho2, r.denominator_rcp);
            accepted |= 1u << r.bit;
            transmittance *= one_minus_alpha;
            if (transmittance < kTransmittanceThreshold) { done = true; candidates = 0; }
        };
        while (__any_sync(0xffffffffu, candidates != 0)) {
            const Seen first = look();
            if constexpr (ABS_GRAD) {
                const Seen second = look();
                blend(first);
                blend(second);
            } else {
                blend(first);
            }
        }
        // ---- 3. lane = (survivor, half of the pixels) -----------------------------------------------------------------------
        // transposing back: bit 15 - i of lane p -> bit p of survivor i, this lane's 16 pixels in the low bits
        uint32_t pixels = transpose_half(accepted, lane);
        const uint32_t halves = __ballot_sync(0xffffffffu, pixels != 0), any = halves | (halves >> 16) | (halves << 16);     // survivors with an accepted pair
        __syncwarp();
        PairMoments moments{};
        float4 aC = make_float4(0, 0, 0, 0);
        [[maybe_unused]] float abs_grad = 0.0f;
        const uint32_t first_pixel = lane & 16u;
        auto add = [&](uint32_t p) {
            const float4 pair = s_pair[mine][p];
            const float4 grad = s_grad[p];
            const float y = offset_y + small_int_to_float(p >> 3), s = fmaf(shear, y, offset_x + small_int_to_float(p & 7u));
            aC.x = fmaf(pair.x, grad.x, aC.x); aC.y = fmaf(pair.x, grad.y, aC.y); aC.z = fmaf(pair.x, grad.z, aC.z);
            aC.w += pair.y;
            const float dL_drho2 = -0.5f * opacity * pair.y, u = dL_drho2 * pair.w;
            add_moments(moments, u, u * pair.z, dL_drho2 * pair.z, s, y);
            if constexpr (ABS_GRAD) abs_grad += abs_position_gradient(af, u, s, y, x0 + small_int_to_float(p & 7u), y0 + small_int_to_float(p >> 3), cam);
        };
        while (pixels != 0) {
            const uint32_t p0 = first_pixel + uint32_t(__ffs(int(pixels)) - 1);
            pixels &= pixels - 1;
            const uint32_t p1 = pixels != 0 ? first_pixel + uint32_t(__ffs(int(pixels)) - 1) : 32u;
            pixels &= pixels - 1;
            add(p0);
            add(p1);
        }
        __syncwarp();
        auto both_halves = [](float4& v) {
            v.x += __shfl_xor_sync(0xffffffffu, v.x, 16); v.y += __shfl_xor_sync(0xffffffffu, v.y, 16);
            v.z += __shfl_xor_sync(0xffffffffu, v.z, 16); v.w += __shfl_xor_sync(0xffffffffu, v.w, 16);
        };
        auto both_halves2 = [](f32x2& v) { v = add2(v, __shfl_xor_sync(0xffffffffu, v, 16)); };
        both_halves2(moments.uv); both_halves2(moments.u1); both_halves2(moments.u2); both_halves2(moments.v1); both_halves2(moments.v2); both_halves(aC);
        moments.usy += __shfl_xor_sync(0xffffffffu, moments.usy, 16);
        moments.vsy += __shfl_xor_sync(0xffffffffu, moments.vsy, 16);
        if constexpr (ABS_GRAD) abs_grad += __shfl_xor_sync(0xffffffffu, abs_grad, 16);
        if ((any >> lane) & 1u) {                        // the two half warps share the four or five reductions of a record
            float4* rec = accum + size_t(g) * 5;
            if (lane < kGoChunk) { red_add_v4(rec, moments.row(0)); red_add_v4(rec + 1, moments.row(1)); }
            else { red_add_v4(rec + 2, moments.row(2)); red_add_v4(rec + 3, aC); }
            if constexpr (ABS_GRAD) { if (lane < kGoChunk) red_add_v4(rec + 4, make_float4(abs_grad, 0.0f, 0.0f, 0.0f)); }
        }
        if (__all_sync(0xffffffffu, done)) break;
        __syncwarp();
    }
}

// kernel_utils.cuh:44-61
__device__ __forceinline__ float4 quat_backward(const float4& q, const float (&dR)[9]) {
    const float r = q.x, x = q.y, y = q.z, z = q.w;
    const float r21_sub_r12 = dR[3] - dR[1], r21_add_r12 = dR[3] + dR[1];
    const float r13_sub_r31 = dR[2] - dR[6], r13_add_r31 = dR[2] + dR[6];
    const float r32_sub_r23 = dR[7] - dR[5], r32_add_r23 = dR[7] + dR[5];
    return make_float4(
        2.0f * (x * r32_sub_r23 + y * r13_sub_r31 + z * r21_sub_r12),
        2.0f * (r * r32_sub_r23 - 2.0f * x * (dR[4] + dR[8]) + y * r21_add_r12 + z * r13_add_r31),
        2.0f * (r * r13_sub_r31 + x * r21_add_r12 - 2.0f * y * (dR[0] + dR[8]) + z * r32_add_r23),
        2.0f * (r * r21_sub_r12 + x * r13_add_r31 + y * r32_add_r23 - 2.0f * z * (dR[0] + dR[4])));
}

// Per-Gaussian chain rule: accumulated record -> the six output gradients
// (hybrid_blend/kernels/backward.cuh:10-102; SH part kernel_utils.cuh:190-281).  Every output element is
// defined after the call: the rows of Gaussians that the view culled are written as zeros.  What bounds it is the store of the rows
// (236 bytes per Gaussian at SH degree 3): a warp collects its 32 rows of grad_sh_rest in shared memory and stores them as
// one block of 16-byte words.  3 M Gaussians: 248 us, against 219 us for rows stored in place after 0.7 GB of memsets, which
// ran beside the per-tile kernel and slowed it down.
//
// COMPACT: instead of the six dense rows (59 floats at SH degree 3) the kernel appends one 64-byte record per Gaussian the view
// kept to `out.compact_rows` (common.cuh: compact gradient rows): the gradients of position, scale, rotation and opacity and the
// clamp-masked colour gradient.  The rows of grad_sh_0 / grad_sh_rest are (basis function of the view direction) x (colour
// gradient), so whoever knows the camera position can rebuild them (sh_rest_gradient_rows, exchange.cu); this is what
// the ranks of a multi-GPU trainer send one another instead of the dense rows.
constexpr int kChainThreads = 128;
template <bool COMPACT>
__global__ void __launch_bounds__(kChainThreads, 7) preprocess_backward_kernel(
    const float* __restrict__ positions, const float* __restrict__ scales, const float* __restrict__ rotations, const float* __restrict__ sh_rest,
    const float* __restrict__ M, const float* __restrict__ VPM, const float* __restrict__ cam_position_ptr,
    const uint32_t* __restrict__ n_touched, const EvalRecord* __restrict__ eval, const PairRecord* __restrict__ pair, const uint8_t* __restrict__ clamp,
    const float4* __restrict__ accum, BackwardOutputs out,
    uint32_t n_primitives, int active_sh_bases, int total_sh_bases, uint32_t g_first, uint32_t g_end)
{
    extern __shared__ __align__(16) float s_rows[];      // dense: [warps][32][3 * total_sh_bases] where that is at most 45 wide
    const uint32_t idx = g_first + blockIdx.x * kChainThreads + threadIdx.x;
    if constexpr (COMPACT) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {      // header: the camera the receivers need (its first word, the row count, was cleared by the launcher)
            CompactGradientHeader* header = reinterpret_cast<CompactGradientHeader*>(out.compact_rows);
            header->cam_x = __ldg(cam_position_ptr); header->cam_y = __ldg(cam_position_ptr + 1); header->cam_z = __ldg(cam_position_ptr + 2);
            header->active_sh_bases = uint32_t(active_sh_bases);
        }
    }
    const bool kept = idx < g_end && n_touched[idx] != 0;
    [[maybe_unused]] const int row_width = 3 * min(total_sh_bases, 15);
    [[maybe_unused]] float* my_row = s_rows + size_t(threadIdx.x) * row_width;
    [[maybe_unused]] int rows_set = 0;                 // of my_row
    float3 grad_scale = make_float3(0, 0, 0), grad_rgb = make_float3(0, 0, 0), dL_dposition = make_float3(0, 0, 0);
    float4 grad_rotation = make_float4(0, 0, 0, 0);
    float grad_opacity = 0.0f;
    if (kept) {
    const float4 dC = accum[size_t(idx) * 5 + 3];
    const float4 T4 = ldg4(reinterpret_cast<const float*>(eval + idx) + 8);
    const float4 centre = ldg4(&pair[idx].cx);       // and shear, 1 / D at the centre
    const RowGradients rows = rows_from_moments(affine_planes<double>(ldg4(reinterpret_cast<const float*>(eval + idx)), ldg4(reinterpret_cast<const float*>(eval + idx) + 4), T4,
                                                              centre.x, centre.y, centre.z), T4, ldg4(&pair[idx].n0.x), ldg4(&pair[idx].n1.x), centre.w * accum[size_t(idx) * 5], centre.w * accum[size_t(idx) * 5 + 1], centre.w * accum[size_t(idx) * 5 + 2]);
    // dL/dVPMT4 = -(cx dL/dVPMT1 + cy dL/dVPMT2 + E): the products with the centre are moved to the rows of VPM, where they cancel
    const float4 dT1 = rows.dX, dT2 = rows.dY, dT4 = make_float4(-rows.E.x, -rows.E.y, -rows.E.z, -rows.E.w);
    const float3 c1 = make_float3(dT1.x, dT2.x, dT4.x), c2 = make_float3(dT1.y, dT2.y, dT4.y), c3 = make_float3(dT1.z, dT2.z, dT4.z);
    const float3 c4 = make_float3(dT1.w, dT2.w, dT4.w);
    const float4 r4 = ldg4(VPM + 12), r1 = ldg4(VPM) - centre.x * r4, r2 = ldg4(VPM + 4) - centre.y * r4;
    const float3 VPM1 = f3(r1), VPM2 = f3(r2), VPM4 = f3(r4);
    const float3 VPM_c1 = make_float3(r1.x, r2.x, r4.x), VPM_c2 = make_float3(r1.y, r2.y, r4.y), VPM_c3 = make_float3(r1.z, r2.z, r4.z);

    const float3 scale = make_float3(scales[3 * size_t(idx)], scales[3 * size_t(idx) + 1], scales[3 * size_t(idx) + 2]);
    const float4 q = ldg4(rotations + 4 * size_t(idx));
    const float r = q.x, x = q.y, y = q.z, z = q.w;
    const float xx = x * x, yy = y * y, zz = z * z, xy = x * y, xz = x * z, yz = y * z, rx = r * x, ry = r * y, rz = r * z;
    const float3 R_c1 = make_float3(1.0f - 2.0f * (yy + zz), 2.0f * (xy + rz), 2.0f * (xz - ry));
    const float3 R_c2 = make_float3(2.0f * (xy - rz), 1.0f - 2.0f * (xx + zz), 2.0f * (yz + rx));
    const float3 R_c3 = make_float3(2.0f * (xz + ry), 2.0f * (yz - rx), 1.0f - 2.0f * (xx + yy));
    grad_scale = make_float3(
        dot(make_float3(dot(VPM1, R_c1), dot(VPM2, R_c1), dot(VPM4, R_c1)), c1),
        dot(make_float3(dot(VPM1, R_c2), dot(VPM2, R_c2), dot(VPM4, R_c2)), c2),
        dot(make_float3(dot(VPM1, R_c3), dot(VPM2, R_c3), dot(VPM4, R_c3)), c3));
    const float dR[9] = {
        dot(VPM_c1, c1) * scale.x, dot(VPM_c1, c2) * scale.y, dot(VPM_c1, c3) * scale.z,
        dot(VPM_c2, c1) * scale.x, dot(VPM_c2, c2) * scale.y, dot(VPM_c2, c3) * scale.z,
        dot(VPM_c3, c1) * scale.x, dot(VPM_c3, c2) * scale.y, dot(VPM_c3, c3) * scale.z};
    grad_rotation = quat_backward(q, dR);
    grad_opacity = dC.w;

    // colour: undo the clamp at 0, then SH backward
    const uint8_t cl = clamp[idx];
    grad_rgb = make_float3((cl & 1) ? 0.0f : dC.x, (cl & 2) ? 0.0f : dC.y, (cl & 4) ? 0.0f : dC.z);
    const float3 position = make_float3(positions[3 * size_t(idx)], positions[3 * size_t(idx) + 1], positions[3 * size_t(idx) + 2]);
    float3 drgb_dposition = make_float3(0, 0, 0);
    if (active_sh_bases > 1) {
        const float3* co = reinterpret_cast<const float3*>(sh_rest) + size_t(idx) * total_sh_bases;
        const float3 cam_position = make_float3(__ldg(cam_position_ptr), __ldg(cam_position_ptr + 1), __ldg(cam_position_ptr + 2));
        const float3 raw = position - cam_position;
        const float3 dir = normalize(raw);
        const float dx = dir.x, dy = dir.y, dz = dir.z;
        float3 gdx = -0.48860251190291987f * co[2];
        float3 gdy = -0.48860251190291987f * co[0];
        float3 gdz = 0.48860251190291987f * co[1];
        if (active_sh_bases > 4) {
            const float sxx = dx * dx, syy = dy * dy, szz = dz * dz, sxy = dx * dy, sxz = dx * dz, syz = dy * dz;
            gdx = gdx + (1.0925484305920792f * dy) * co[3] + (-1.0925484305920792f * dz) * co[6] + (1.0925484305920792f * dx) * co[7];
            gdy = gdy + (1.0925484305920792f * dx) * co[3] + (-1.0925484305920792f * dz) * co[4] + (-1.0925484305920792f * dy) * co[7];
            gdz = gdz + (-1.0925484305920792f * dy) * co[4] + (1.8923493915151202f * dz) * co[5] + (-1.0925484305920792f * dx) * co[6];
            if (active_sh_bases > 9) {
                gdx = gdx + (-3.5402615395598609f * sxy) * co[8] + (2.8906114426405538f * syz) * co[9]
                          + (0.45704579946446572f - 2.2852289973223288f * szz) * co[12] + (2.8906114426405538f * sxz) * co[13]
                          + (-1.7701307697799304f * sxx + 1.7701307697799304f * syy) * co[14];
                gdy = gdy + (-1.7701307697799304f * sxx + 1.7701307697799304f * syy) * co[8] + (2.8906114426405538f * sxz) * co[9]
                          + (0.45704579946446572f - 2.2852289973223288f * szz) * co[10] + (-2.8906114426405538f * syz) * co[13]
                          + (3.5402615395598609f * sxy) * co[14];
                gdz = gdz + (2.8906114426405538f * sxy) * co[9] + (-4.5704579946446566f * syz) * co[10]
                          + (5.597644988851731f * szz - 1.1195289977703462f) * co[11] + (-4.5704579946446566f * sxz) * co[12]
                          + (1.4453057213202769f * sxx - 1.4453057213202769f * syy) * co[13];
            }
        }
        const float3 gdir = make_float3(dot(gdx, grad_rgb), dot(gdy, grad_rgb), dot(gdz, grad_rgb));
        const float xr = raw.x, yr = raw.y, zr = raw.z;
        const float xxr = xr * xr, yyr = yr * yr, zzr = zr * zr, xyr = xr * yr, xzr = xr * zr, yzr = yr * zr;
        const float norm_sq = xxr + yyr + zzr;
        drgb_dposition = make_float3(
            (yyr + zzr) * gdir.x - xyr * gdir.y - xzr * gdir.z,
            -xyr * gdir.x + (xxr + zzr) * gdir.y - yzr * gdir.z,
            -xzr * gdir.x - yzr * gdir.y + (xxr + yyr) * gdir.z) * rsqrtf(norm_sq * norm_sq * norm_sq);
        if constexpr (!COMPACT) {
            float3 rows[15];
            rows_set = sh_rest_gradient_rows(dir, grad_rgb, active_sh_bases, rows);
            #pragma unroll
            for (int i = 0; i < 15; ++i)
                if (i < rows_set) { my_row[3 * i] = rows[i].x; my_row[3 * i + 1] = rows[i].y; my_row[3 * i + 2] = rows[i].z; }
        }
    }
    dL_dposition = make_float3(dot(VPM_c1, c4), dot(VPM_c2, c4), dot(VPM_c3, c4)) + drgb_dposition;
    if (out.densification_info != nullptr) {     // hybrid_blend/kernels/backward.cuh:85-98
        float z_scale = 1.0f;
        if (out.use_distance_scaling) {
            const float4 M3 = ldg4(M + 8);
            z_scale = (dot(f3(M3), position) + M3.w) * 0.5f;
        }
        float* info = out.densification_info;
        info[idx] += 1.0f;
        info[size_t(n_primitives) + idx] += length(dL_dposition * z_scale);
        if (out.densification_rows == 3) info[2 * size_t(n_primitives) + idx] += z_scale * accum[size_t(idx) * 5 + 4].x;
    }
    }   // kept
    if constexpr (!COMPACT) {
        if (idx < g_end) {
            reinterpret_cast<float3*>(out.grad_scales)[idx] = grad_scale;
            reinterpret_cast<float4*>(out.grad_rotations)[idx] = grad_rotation;
            out.grad_opacities[idx] = grad_opacity;
            reinterpret_cast<float3*>(out.grad_sh_0)[idx] = kShBand0 * grad_rgb;
            reinterpret_cast<float3*>(out.grad_positions)[idx] = dL_dposition;
        }
        if (total_sh_bases > 0) {
            const uint32_t lane = threadIdx.x & 31u, warp_first = idx - lane;
            if (warp_first >= g_end) return;
            const bool any = __any_sync(0xffffffffu, rows_set > 0);
            if (any) {
                for (int i = 3 * rows_set; i < row_width; ++i) my_row[i] = 0.0f;
                __syncwarp();
            }
            const float* block = s_rows + size_t(threadIdx.x - lane) * row_width;
            const uint32_t width = 3u * uint32_t(total_sh_bases), floats = min(32u, g_end - warp_first) * width;
            float* dst = out.grad_sh_rest + size_t(warp_first) * width;
            if (total_sh_bases <= 15 && (reinterpret_cast<uintptr_t>(dst) & 15u) == 0) {
                for (uint32_t i = lane; i < floats / 4; i += 32)
                    reinterpret_cast<float4*>(dst)[i] = any ? reinterpret_cast<const float4*>(block)[i] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                const uint32_t rest = floats & ~3u;
                if (rest + lane < floats) dst[rest + lane] = any ? block[rest + lane] : 0.0f;
            } else {
                for (uint32_t i = lane; i < floats; i += 32) {
                    const uint32_t row = i / width, column = i - row * width;
                    dst[i] = any && column < uint32_t(row_width) ? block[row * row_width + column] : 0.0f;
                }
            }
        }
    } else {
        // one slot per kept Gaussian: a warp takes its slots with one atomic (the order of the rows carries no meaning)
        const uint32_t kept_mask = __ballot_sync(0xffffffffu, kept);
        if (kept_mask == 0) return;
        const uint32_t lane = threadIdx.x & 31u;
        uint32_t base = 0;
        if (lane == uint32_t(__ffs(kept_mask) - 1)) base = atomicAdd(reinterpret_cast<uint32_t*>(out.compact_rows), uint32_t(__popc(kept_mask)));
        base = __shfl_sync(0xffffffffu, base, __ffs(kept_mask) - 1);
        const uint32_t slot = base + uint32_t(__popc(kept_mask & ((1u << lane) - 1u)));
        if (kept && slot < out.compact_capacity) {      // rows beyond the capacity are dropped; the count tells the reader
            float4* row = out.compact_rows + 4 * (size_t(slot) + 1);
            row[0] = make_float4(__uint_as_float(idx), dL_dposition.x, dL_dposition.y, dL_dposition.z);
            row[1] = make_float4(grad_scale.x, grad_scale.y, grad_scale.z, grad_opacity);
            row[2] = grad_rotation;
            row[3] = make_float4(grad_rgb.x, grad_rgb.y, grad_rgb.z, 0.0f);
        }
    }
}

template <int MODE, int K>
cudaError_t launch_tile_backward(bool abs_grad, const FrameGeometry& geo, const PrimBuffers& prim, const uint32_t* prims_sorted, const uint2* tile_ranges, const uint32_t* tile_order,
                                 const TrainPixelBuffers& tin, const float* grad_image, const float* VPM, float4* accum, uint32_t g_first, uint32_t g_end,
                                 cudaStream_t stream) {
    auto launch = [&](auto kernel, size_t smem) -> cudaError_t {
        // both instantiations have the same function-pointer type, so this lambda (and a static in it) is shared by them
        static PerDeviceOnce configured[2];
        if (smem > 48 * 1024) {
            const cudaError_t err = configured[abs_grad ? 1 : 0].run([&] { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)); });
            if (err != cudaSuccess) return err;
        }
        kernel<<<uint32_t(geo.n_tiles), kBwdThreads, smem, stream>>>(tile_ranges, tile_order, prims_sorted, prim.eval, prim.cull, prim.pair, tin, grad_image, VPM, accum,
                                                uint32_t(geo.width), uint32_t(geo.height), uint32_t(geo.grid_w), g_first, g_end);
        return cudaGetLastError();
    };
    return abs_grad ? launch(backward_tile_kernel<MODE, K, true>, BwdSmem<MODE, K, true>::total) : launch(backward_tile_kernel<MODE, K, false>, BwdSmem<MODE, K, false>::total);
}

template <int MODE>
cudaError_t launch_tile_backward_k(int K, bool abs_grad, const FrameGeometry& geo, const PrimBuffers& prim, const uint32_t* prims_sorted,
                                   const uint2* tile_ranges, const uint32_t* tile_order, const TrainPixelBuffers& tin, const float* grad_image, const float* VPM, float4* accum,
                                   uint32_t g_first, uint32_t g_end, cudaStream_t stream) {
    switch (K) {
        case 32: return launch_tile_backward<MODE, 32>(abs_grad, geo, prim, prims_sorted, tile_ranges, tile_order, tin, grad_image, VPM, accum, g_first, g_end, stream);
        case 16: return launch_tile_backward<MODE, 16>(abs_grad, geo, prim, prims_sorted, tile_ranges, tile_order, tin, grad_image, VPM, accum, g_first, g_end, stream);
        case 8: return launch_tile_backward<MODE, 8>(abs_grad, geo, prim, prims_sorted, tile_ranges, tile_order, tin, grad_image, VPM, accum, g_first, g_end, stream);
        case 4: return launch_tile_backward<MODE, 4>(abs_grad, geo, prim, prims_sorted, tile_ranges, tile_order, tin, grad_image, VPM, accum, g_first, g_end, stream);
        case 2: return launch_tile_backward<MODE, 2>(abs_grad, geo, prim, prims_sorted, tile_ranges, tile_order, tin, grad_image, VPM, accum, g_first, g_end, stream);
        default: return launch_tile_backward<MODE, 1>(abs_grad, geo, prim, prims_sorted, tile_ranges, tile_order, tin, grad_image, VPM, accum, g_first, g_end, stream);
    }
}

}  // namespace

namespace {
__global__ void __launch_bounds__(256) visibility_kernel(const uint32_t* __restrict__ n_touched, uint8_t* __restrict__ visible, uint32_t n) {
    const uint32_t i = blockIdx.x * 256 + threadIdx.x;
    if (i < n) visible[i] = n_touched[i] != 0;
}
}  // namespace

cudaError_t launch_visibility(const uint32_t* n_touched, uint8_t* visible, uint32_t n, cudaStream_t stream) {
    if (n == 0) return cudaSuccess;
    visibility_kernel<<<(n + 255) / 256, 256, 0, stream>>>(n_touched, visible, n);
    return cudaGetLastError();
}

cudaError_t clear_backward_outputs(const HtgsScene& scene, const BackwardOutputs& out, uint32_t first, uint32_t count, cudaStream_t stream) {
    const size_t n = size_t(count), at = size_t(first), B = size_t(scene.total_sh_bases);
    if (n == 0) return cudaSuccess;
    cudaError_t err;
    if ((err = cudaMemsetAsync(out.grad_positions + at * 3, 0, n * 3 * 4, stream)) != cudaSuccess) return err;
    if ((err = cudaMemsetAsync(out.grad_scales + at * 3, 0, n * 3 * 4, stream)) != cudaSuccess) return err;
    if ((err = cudaMemsetAsync(out.grad_rotations + at * 4, 0, n * 4 * 4, stream)) != cudaSuccess) return err;
    if ((err = cudaMemsetAsync(out.grad_opacities + at, 0, n * 4, stream)) != cudaSuccess) return err;
    if ((err = cudaMemsetAsync(out.grad_sh_0 + at * 3, 0, n * 3 * 4, stream)) != cudaSuccess) return err;
    if (B && (err = cudaMemsetAsync(out.grad_sh_rest + at * B * 3, 0, n * B * 3 * 4, stream)) != cudaSuccess) return err;
    return cudaSuccess;
}

namespace {
__global__ void __launch_bounds__(256) clear_records_kernel(float4* __restrict__ accum, const uint32_t* __restrict__ visible_list, const FrameStatus* __restrict__ status) {
    const uint64_t words = uint64_t(status->n_visible) * 5;
    for (uint64_t i = blockIdx.x * 256u + threadIdx.x; i < words; i += gridDim.x * 256u)
        accum[size_t(__ldg(visible_list + i / 5)) * 5 + i % 5] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
}

cudaError_t launch_chain_rule(const HtgsScene& scene, const HtgsView& view, const PrimBuffers& prim, const GradAccumBuffers& acc, const BackwardOutputs& out,
                              uint32_t n, uint32_t first, uint32_t count, cudaStream_t stream) {
    const uint32_t grid = (count + kChainThreads - 1) / kChainThreads;
    if (out.compact_rows != nullptr) {
        const cudaError_t err = cudaMemsetAsync(out.compact_rows, 0, sizeof(CompactGradientHeader), stream);
        if (err != cudaSuccess) return err;
        preprocess_backward_kernel<true><<<grid, kChainThreads, 0, stream>>>(scene.positions, scene.scales, scene.rotations, scene.sh_rest, view.M, view.VPM,
                                                                             view.cam_position, prim.n_touched, prim.eval, prim.pair, prim.clamp, acc.accum, out, n,
                                                                             view.active_sh_bases, scene.total_sh_bases, first, first + count);
    } else {
        const size_t smem = size_t(kChainThreads) * 3 * size_t(scene.total_sh_bases < 15 ? scene.total_sh_bases : 15) * sizeof(float);
        preprocess_backward_kernel<false><<<grid, kChainThreads, smem, stream>>>(scene.positions, scene.scales, scene.rotations, scene.sh_rest, view.M, view.VPM,
                                                                                 view.cam_position, prim.n_touched, prim.eval, prim.pair, prim.clamp, acc.accum, out, n,
                                                                                 view.active_sh_bases, scene.total_sh_bases, first, first + count);
    }
    return cudaGetLastError();
}
}  // namespace

cudaError_t launch_backward(int mode, int K, const HtgsScene& scene, const HtgsView& view, const FrameGeometry& geo, const PrimBuffers& prim,
                            const uint32_t* prims_sorted, const uint2* tile_ranges, const uint32_t* tile_order, const TrainPixelBuffers& tin, const float* grad_image,
                            const float* image, const GradAccumBuffers& acc, const BackwardOutputs& out, const FrameStatus* status, int sm_count,
                            uint32_t first, uint32_t count, int stages, cudaStream_t stream) {
    const uint32_t n = uint32_t(scene.n_primitives);
    if (n == 0 || count == 0) return out.compact_rows ? cudaMemsetAsync(out.compact_rows, 0, sizeof(CompactGradientHeader), stream) : cudaSuccess;
    const bool whole = first == 0 && count == n;
    if (!(stages & kBackwardAccumulate)) {      // the per-Gaussian chain rule alone, over records an earlier call accumulated
        return launch_chain_rule(scene, view, prim, acc, out, n, first, count, stream);
    }
    // the pixel-parallel GLOBAL_ORDERING pass needs every fragment in front of a fragment: it cannot run over a part of the Gaussians
    if (!whole && mode == HTGS_MODE_ALPHA_BLEND_GLOBAL_ORDERING) return cudaErrorNotSupported;
    const uint32_t g_first = whole ? 0u : first, g_end = whole ? 0xffffffffu : first + count;
    cudaError_t err = cudaSuccess;
    if (whole) {       // only the records of Gaussians that the view kept are ever added to or read (one in six: 35 us at 3 M, a memset of all 45)
        clear_records_kernel<<<std::min<uint32_t>((n + 63) / 64, uint32_t(sm_count) * 8u), 256, 0, stream>>>(acc.accum, prim.visible_list, status);
        err = cudaGetLastError();
    } else {
        err = cudaMemsetAsync(acc.accum + size_t(first) * 5, 0, size_t(count) * 5 * sizeof(float4), stream);
    }
    if (err != cudaSuccess) return err;
    // rows that the caller adds to (the kernels of the exchange) have to start at zero
    if (out.compact_rows != nullptr && out.grad_positions != nullptr && (err = clear_backward_outputs(scene, out, first, count, stream)) != cudaSuccess) return err;
    const bool abs_grad = out.densification_info != nullptr && out.densification_rows == 3;
    const int k = effective_k(mode, K);
    switch (mode) {
        case HTGS_MODE_HYBRID_BLEND:
            err = launch_tile_backward_k<HTGS_MODE_HYBRID_BLEND>(k, abs_grad, geo, prim, prims_sorted, tile_ranges, tile_order, tin, grad_image, view.VPM, acc.accum, g_first, g_end, stream); break;
        case HTGS_MODE_ALPHA_BLEND_FIRST_K:
            err = launch_tile_backward_k<HTGS_MODE_ALPHA_BLEND_FIRST_K>(k, abs_grad, geo, prim, prims_sorted, tile_ranges, tile_order, tin, grad_image, view.VPM, acc.accum, g_first, g_end, stream); break;
        case HTGS_MODE_OIT_BLEND:
            err = launch_tile_backward<HTGS_MODE_OIT_BLEND, 1>(abs_grad, geo, prim, prims_sorted, tile_ranges, tile_order, tin, grad_image, view.VPM, acc.accum, g_first, g_end, stream); break;
        case HTGS_MODE_ALPHA_BLEND_GLOBAL_ORDERING: {
            const auto kernel = abs_grad ? backward_global_kernel<true> : backward_global_kernel<false>;
            kernel<<<uint32_t(geo.n_tiles) * 8u, 32, 0, stream>>>(tile_ranges, tile_order, prims_sorted, prim.eval, prim.cull, prim.pair, grad_image, image, view.VPM, acc.accum,
                                                                  uint32_t(geo.width), uint32_t(geo.height), uint32_t(geo.grid_w));
            err = cudaGetLastError();
            break;
        }
        default: return cudaErrorInvalidValue;
    }
    if (err != cudaSuccess) return err;
    if (!(stages & kBackwardChainRule)) return cudaSuccess;
    return launch_chain_rule(scene, view, prim, acc, out, n, first, count, stream);
}

}  // namespace htgs
