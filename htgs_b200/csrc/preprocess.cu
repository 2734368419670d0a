// Per-Gaussian preprocess: exact perspective-correct screen bounds, ray-evaluation
// setup, SH -> RGB, view depth, plus two things the reference does not have:
// the per-block instance count (which replaces a separate prefix-sum pass over
// all Gaussians) and a conservative screen-space ellipse used by the blend
// kernels to skip (pixel, Gaussian) pairs the exact test would reject.
//
// Two kernels: a cull pass over all Gaussians and a finish pass over the list of visible ones (typically one in
// six), so that the expensive half (SH evaluation, float64 outline) runs in full warps.
//
// Replaces the sixteen preprocess_cu variants of the reference
// (rasterization/include/*/kernels/{forward,inference}.cuh:10-76) and the device helpers
// transform_and_cull / convert_sh_to_rgb (rasterization/include/kernel_utils.cuh:63-188).
// The float expression shapes of the bounds computation are kept as in the reference so
// that tile boxes are bit-identical; everything around them is new.
#include "kernels.h"

namespace htgs {

namespace {

struct Mat3 { float r11, r12, r13, r21, r22, r23, r31, r32, r33; };

// rasterization/include/kernel_utils.cuh:30-42.  The multiply-add contraction of every entry is
// written out with intrinsics: it is the rounding the reference build (nvcc 12.9, sm_100a, default
// -fmad) was measured to produce for each entry, and the compiler cannot re-associate intrinsics.
__device__ __forceinline__ Mat3 quat_to_mat(const float4& q) {
    const float r = q.x, x = q.y, y = q.z, z = q.w;
    const float yy_zz = __fadd_rn(__fmul_rn(y, y), __fmul_rn(z, z));
    const float xx_zz = __fmaf_rn(x, x, __fmul_rn(z, z));
    const float xx_yy = __fmaf_rn(x, x, __fmul_rn(y, y));
    const float rz = __fmul_rn(r, z), rx = __fmul_rn(r, x), xz = __fmul_rn(x, z);
    return {__fmaf_rn(-2.0f, yy_zz, 1.0f), __fmul_rn(2.0f, __fmaf_rn(x, y, -rz)), __fmul_rn(2.0f, __fmaf_rn(r, y, xz)),
            __fmul_rn(2.0f, __fmaf_rn(x, y, rz)), __fmaf_rn(-2.0f, xx_zz, 1.0f), __fmul_rn(2.0f, __fmaf_rn(y, z, -rx)),
            __fmul_rn(2.0f, __fmaf_rn(-r, y, xz)), __fmul_rn(2.0f, __fmaf_rn(y, z, rx)), __fmaf_rn(-2.0f, xx_yy, 1.0f)};
}

// Rows of (VP*M*T) and (M*T): kernel_utils.cuh:102,111,119,123 and hybrid_blend/kernels/inference.cuh:61.
// As for the rotation matrix, the contraction of each dot product is pinned to what the reference build
// was measured to round like: x*x' fused into y*y', then z*z' fused on top - except the first component
// of the rows built from VPM row 4 and M row 3, where y*y' is fused into x*x'.
__device__ __forceinline__ float dot3_pinned(const float3& a, const float3& b) {
    return __fmaf_rn(a.z, b.z, __fmaf_rn(a.x, b.x, __fmul_rn(a.y, b.y)));
}
__device__ __forceinline__ float dot3_pinned_alt(const float3& a, const float3& b) {
    return __fmaf_rn(a.z, b.z, __fmaf_rn(a.y, b.y, __fmul_rn(a.x, b.x)));
}
template <bool ALT_FIRST>
__device__ __forceinline__ float4 row_times_T(const float4& row, const float3& u, const float3& v, const float3& w, const float3& p) {
    const float3 r = f3(row);
    return make_float4(ALT_FIRST ? dot3_pinned_alt(r, u) : dot3_pinned(r, u), dot3_pinned(r, v), dot3_pinned(r, w), __fadd_rn(dot3_pinned(r, p), row.w));
}

// rasterization/include/kernel_utils.cuh:140-188
// `c`: the Gaussian's coefficients beyond the first band, in shared memory.
template <bool TRAIN>
__device__ __forceinline__ float3 sh_to_rgb(const float3& dc, const float* c, const float3& position, const float3& cam_position, int active_sh_bases,
                                            uint8_t* clamp_bits) {
    float3 result = 0.5f + 0.28209479177387814f * dc;
    if (active_sh_bases > 1) {
        auto coef = [&](int i) { return make_float3(c[3 * i], c[3 * i + 1], c[3 * i + 2]); };
        const float3 dir = normalize(position - cam_position);
        const float x = dir.x, y = dir.y, z = dir.z;
        result = result + (-0.48860251190291987f * y) * coef(0)
                        + (0.48860251190291987f * z) * coef(1)
                        + (-0.48860251190291987f * x) * coef(2);
        if (active_sh_bases > 4) {
            const float xx = x * x, yy = y * y, zz = z * z;
            const float xy = x * y, xz = x * z, yz = y * z;
            result = result + (1.0925484305920792f * xy) * coef(3)
                            + (-1.0925484305920792f * yz) * coef(4)
                            + (0.94617469575755997f * zz - 0.31539156525251999f) * coef(5)
                            + (-1.0925484305920792f * xz) * coef(6)
                            + (0.54627421529603959f * xx - 0.54627421529603959f * yy) * coef(7);
            if (active_sh_bases > 9) {
                result = result + (0.59004358992664352f * y * (-3.0f * xx + yy)) * coef(8)
                                + (2.8906114426405538f * xy * z) * coef(9)
                                + (0.45704579946446572f * y * (1.0f - 5.0f * zz)) * coef(10)
                                + (0.3731763325901154f * z * (5.0f * zz - 3.0f)) * coef(11)
                                + (0.45704579946446572f * x * (1.0f - 5.0f * zz)) * coef(12)
                                + (1.4453057213202769f * z * (xx - yy)) * coef(13)
                                + (0.59004358992664352f * x * (-xx + 3.0f * yy)) * coef(14);
            }
        }
    }
    if constexpr (TRAIN) {
        *clamp_bits = uint8_t((result.x < 0 ? 1 : 0) | (result.y < 0 ? 2 : 0) | (result.z < 0 ? 4 : 0));
    }
    return make_float3(fmaxf(0.0f, result.x), fmaxf(0.0f, result.y), fmaxf(0.0f, result.z));
}

struct OutlineThresholds { float max_cutoff_sq, min_alpha_rcp; };
OutlineThresholds outline_thresholds(int mode) {
    if (mode == HTGS_MODE_ALPHA_BLEND_FIRST_K) return {ModeTraits<HTGS_MODE_ALPHA_BLEND_FIRST_K>::max_cutoff_sq, ModeTraits<HTGS_MODE_ALPHA_BLEND_FIRST_K>::min_alpha_rcp};
    return {ModeTraits<HTGS_MODE_HYBRID_BLEND>::max_cutoff_sq, ModeTraits<HTGS_MODE_HYBRID_BLEND>::min_alpha_rcp};      // the other three share them
}

// Conservative outline of { pixel : the exact per-fragment test can accept }.
//
// A fragment is accepted only if rho^2 <= max_cutoff_sq and opacity * exp(-rho^2 / 2) >= min_alpha, i.e.
// rho^2 <= L with L = min(max_cutoff_sq, 2 ln(opacity / min_alpha)).  rho^2(pixel) is the squared distance
// (in the Gaussian's unit frame) of the pixel ray to the centre, so the accepted set is the projected outline
// of the ellipsoid |q|^2 <= L: an ellipse whose dual conic is C_ab = L * sum_i T_a[i] T_b[i] - T_a[3] T_b[3]
// (rows a,b of VP*M*T).  Centre and shape are evaluated in float64 from the float32 rows the blend kernels use;
// the shape matrix is inflated by (0.3 px)^2 and the quadratic form relaxed by 2% to cover the float32
// rounding of the exact per-fragment evaluation.  An outline that is not a proper ellipse disables culling
// for the Gaussian ("accept everything"), and L <= 0 rejects everything.
__device__ __forceinline__ CullRecord make_cull_record(const float4& t1, const float4& t2, const float4& t4, float opacity, const OutlineThresholds& thresholds) {
    CullRecord rec = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};   // a = b2 = c = 0: every pixel passes
    const double level = fmin(double(thresholds.max_cutoff_sq), 2.0 * log(double(opacity) * double(thresholds.min_alpha_rcp))) * 1.001 + 1e-4;
    if (!(level > 0.0)) { rec.cx = __int_as_float(0x7f800000); return rec; }   // +inf: every comparison fails, nothing passes
    auto conic = [&](const float4& a, const float4& b) {
        return level * (double(a.x) * double(b.x) + double(a.y) * double(b.y) + double(a.z) * double(b.z)) - double(a.w) * double(b.w);
    };
    const double c44 = conic(t4, t4);
    if (c44 == 0.0) return rec;
    const double inv = 1.0 / c44;
    const double cx = conic(t1, t4) * inv, cy = conic(t2, t4) * inv;
    double sxx = cx * cx - conic(t1, t1) * inv;
    double syy = cy * cy - conic(t2, t2) * inv;
    const double sxy = cx * cy - conic(t1, t2) * inv;
    if (!(sxx > 0.0) || !(syy > 0.0)) return rec;
    const double det0 = sxx * syy - sxy * sxy;
    if (!(det0 > 0.0)) return rec;
    const double inflate = 0.09 + 1e-6 * (cx * cx + cy * cy);
    sxx += inflate; syy += inflate;
    const double det = sxx * syy - sxy * sxy;
    const double relax = 1.0 / 1.02;
    const double a = syy / det * relax, b2 = -2.0 * sxy / det * relax, c = sxx / det * relax;
    if (!isfinite(a) || !isfinite(b2) || !isfinite(c) || !isfinite(cx) || !isfinite(cy)) return rec;
    if (fabs(cx) > 1e6 || fabs(cy) > 1e6) return rec;   // float32 pixel offsets would lose the sub-pixel part
    rec.cx = float(cx); rec.cy = float(cy);
    rec.a = float(a); rec.b2 = float(b2); rec.c = float(c);
    return rec;
}

// Coefficients of the relaxed-precision record (see FastRecord): float64 from the float32 rows the exact path uses.
// `centre` receives the projected centre (pixels), which the quadratics are expanded around.
__device__ __forceinline__ void make_fast_record(const float4& t1, const float4& t2, const float4& t4, const float4& mt3, const float3& rgb,
                                                 float opacity, float4* dst, double (&centre)[2]) {
    struct D3 { double x, y, z; };
    auto cross3 = [](const D3& a, const D3& b) { return D3{a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x}; };
    auto dot3 = [](const D3& a, const D3& b) { return a.x * b.x + a.y * b.y + a.z * b.z; };
    const double w4 = double(t4.w);
    const double cx = double(t1.w) / w4, cy = double(t2.w) / w4;
    const D3 n4{double(t4.x), double(t4.y), double(t4.z)};
    const D3 a{double(t1.x) - n4.x * cx, double(t1.y) - n4.y * cx, double(t1.z) - n4.z * cx};
    const D3 b{double(t2.x) - n4.x * cy, double(t2.y) - n4.y * cy, double(t2.z) - n4.z * cy};
    const D3 d0 = cross3(a, b), dX = cross3(b, n4), dY = cross3(n4, a);
    const double inv = 1.0 / dot3(d0, d0);
    const double e_scale = -0.5 * 1.4426950408889634 * w4 * w4 * inv;
    const D3 m3{double(mt3.x), double(mt3.y), double(mt3.z)};
    const double z_scale = w4 * inv;
    const D3 dXa = cross3(dX, a), dYb = cross3(dY, b);
    float v[20] = {
        float(e_scale * dot3(b, b)), float(-2.0 * e_scale * dot3(a, b)), float(e_scale * dot3(a, a)), float(2.0 * inv * dot3(d0, dX)),
        float(2.0 * inv * dot3(d0, dY)), float(inv * dot3(dX, dX)), float(2.0 * inv * dot3(dX, dY)), float(inv * dot3(dY, dY)),
        float(-z_scale * dot3(m3, cross3(d0, b))), float(z_scale * dot3(m3, cross3(d0, a))), float(-z_scale * dot3(m3, cross3(dX, b))),
        float(z_scale * dot3(m3, D3{dXa.x - dYb.x, dXa.y - dYb.y, dXa.z - dYb.z})),
        float(z_scale * dot3(m3, cross3(dY, a))), mt3.w, log2f(opacity), rgb.x,
        rgb.y, rgb.z, 0.0f, 0.0f};
    bool finite = isfinite(cx) && isfinite(cy);
    #pragma unroll
    for (int i = 0; i < 20; ++i) finite = finite && isfinite(v[i]);
    if (!finite) {   // degenerate Gaussian: contributes nothing
        #pragma unroll
        for (int i = 0; i < 20; ++i) v[i] = 0.0f;
        v[14] = -__int_as_float(0x7f800000);
        centre[0] = centre[1] = 0.0;
    } else {
        centre[0] = cx; centre[1] = cy;
    }
    #pragma unroll
    for (int i = 0; i < 5; ++i) dst[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
}

// The point from which the backward pass measures the pixels of a Gaussian: its projected centre, where m = 0 and its weight is largest, or,
// where that lies outside the tile box (long or near Gaussians), the point of the box where |m|^2, with its slopes at the projected
// centre, is smallest.  From a point off the weight the moments of train.cu cancel (from the centre of the outline, which perspective
// moves away from the projected centre: up to 3e-5 of the position gradient of a Gaussian of 2000 tiles, from here 1e-6).
template <int MODE>
__device__ __forceinline__ float2 make_moment_centre(const float4& t1, const float4& t2, const float4& t4, const ushort4& box) {
    using MT = ModeTraits<MODE>;
    const float x0 = float(box.x) * MT::tile_w, x1 = float(box.y) * MT::tile_w - 1.0f, y0 = float(box.z) * MT::tile_h, y1 = float(box.w) * MT::tile_h - 1.0f;
    const float cx = t1.w / t4.w, cy = t2.w / t4.w;
    if (cx >= x0 && cx <= x1 && cy >= y0 && cy <= y1) return make_float2(cx, cy);
    // m = (y - cy) a - (x - cx) b there, up to the depth: |m|^2 = xx dx^2 + xy dx dy + yy dy^2
    const float3 a = f3(t1) - cx * f3(t4), b = f3(t2) - cy * f3(t4);
    const float xx = dot(b, b), xy = -2.0f * dot(a, b), yy = dot(a, a);
    float2 best = make_float2(0.5f * (x0 + x1), 0.5f * (y0 + y1));
    float smallest = FLT_MAX;
    auto consider = [&](float x, float y) {
        const float dx = x - cx, dy = y - cy, q = dx * (xx * dx + xy * dy) + yy * dy * dy;
        if (q < smallest) { smallest = q; best = make_float2(x, y); }
    };
    const float along_y = -0.5f * xy / yy, along_x = -0.5f * xy / xx;      // where the form is smallest along an edge, per unit of the other coordinate
    consider(x0, fminf(fmaxf(fmaf(along_y, x0 - cx, cy), y0), y1));
    consider(x1, fminf(fmaxf(fmaf(along_y, x1 - cx, cy), y0), y1));
    consider(fminf(fmaxf(fmaf(along_x, y0 - cy, cx), x0), x1), y0);
    consider(fminf(fmaxf(fmaf(along_x, y1 - cy, cx), x0), x1), y1);
    return best;
}

// m = M0 + x Mx + y My and d = D0 + x Dx + y Dy about the centre (train.cu: AffinePlanes); the shear makes the two slopes of m orthogonal.
__device__ __forceinline__ PairRecord make_pair_record(const float4& t1, const float4& t2, const float4& t4, const float2& centre) {
    struct D3 { double x, y, z; };
    auto cross3 = [](const D3& a, const D3& b) { return D3{a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x}; };
    auto dot3 = [](const D3& a, const D3& b) { return a.x * b.x + a.y * b.y + a.z * b.z; };
    auto comb = [](double p, const D3& a, double q, const D3& b) { return D3{p * a.x + q * b.x, p * a.y + q * b.y, p * a.z + q * b.z}; };
    const double cx = double(centre.x), cy = double(centre.y), w = double(t4.w);
    const D3 n{double(t4.x), double(t4.y), double(t4.z)};
    const D3 a{double(t1.x) - cx * n.x, double(t1.y) - cx * n.y, double(t1.z) - cx * n.z};
    const D3 b{double(t2.x) - cy * n.x, double(t2.y) - cy * n.y, double(t2.z) - cy * n.z};
    const double aw = double(t1.w) - cx * w, bw = double(t2.w) - cy * w;
    const D3 m0 = comb(aw, b, -bw, a), ms = comb(bw, n, -w, b);
    D3 my = comb(w, a, -aw, n);
    const D3 d0 = cross3(a, b), ds = cross3(b, n);
    D3 dy = cross3(n, a);
    const double ms_sq = dot3(ms, ms);
    float shear = ms_sq > 0.0 ? float(dot3(ms, my) / ms_sq) : 0.0f;
    if (!(fabsf(shear) < 1e6f)) shear = 0.0f;
    my = comb(1.0, my, -double(shear), ms);
    dy = comb(1.0, dy, -double(shear), ds);
    // N and D grow with the fourth power of sizes in pixels: both are divided by D0
    const double scale = 1.0 / fmax(dot3(d0, d0), 1e-300);
    PairRecord r;
    r.n0 = make_float4(float(scale * dot3(m0, m0)), float(2.0 * scale * dot3(m0, ms)), float(2.0 * scale * dot3(m0, my)), float(scale * dot3(ms, ms)));
    r.n1 = make_float4(float(2.0 * scale * dot3(ms, my)), float(scale * dot3(my, my)), float(scale * dot3(d0, d0)), float(2.0 * scale * dot3(d0, ds)));
    r.d1 = make_float4(float(2.0 * scale * dot3(d0, dy)), float(scale * dot3(ds, ds)), float(2.0 * scale * dot3(ds, dy)), float(scale * dot3(dy, dy)));
    r.cx = centre.x; r.cy = centre.y; r.shear = shear; r.scale = float(scale);
    return r;
}

// Pass 1, one thread per Gaussian: culling, tile box, and the rows VPMT1, VPMT2, VPMT4, MT3 (written where the
// evaluation record lives).  The visible Gaussians of a block are appended to `visible_list` (the order of the list
// depends on the order in which blocks finish; nothing downstream depends on it).
template <int MODE, bool TRAIN>
__global__ void __launch_bounds__(kPreprocessBlock) preprocess_cull_kernel(
    const float* __restrict__ positions, const float* __restrict__ scales, const float* __restrict__ rotations,
    const float* __restrict__ opacities, const float* __restrict__ M, const float* __restrict__ VPM,
    PrimBuffers out, FrameStatus* status, uint32_t n_primitives, uint32_t grid_w, uint32_t grid_h,
    float near_plane, float far_plane, float scale_modifier_arg)
{
    using MT = ModeTraits<MODE>;
    __shared__ uint32_t warp_sum[kPreprocessBlock / 32];
    __shared__ uint32_t warp_vis[kPreprocessBlock / 32];
    __shared__ uint32_t list_base;

    const uint32_t idx = blockIdx.x * kPreprocessBlock + threadIdx.x;
    const uint32_t warp = threadIdx.x >> 5;
    uint32_t n_touched = 0;

    if (idx < n_primitives) {
        const float4 M3 = ldg4(M + 8);
        const float3 position = make_float3(__ldg(positions + 3 * size_t(idx)), __ldg(positions + 3 * size_t(idx) + 1), __ldg(positions + 3 * size_t(idx) + 2));
        const float opacity = __ldg(opacities + idx);
        // near/far culling of the centre (kernel_utils.cuh:88-90)
        const float z = __fadd_rn(dot3_pinned(f3(M3), position), M3.w);
        if (!(z < near_plane || z > far_plane)) {
            const float scale_modifier = TRAIN ? 1.0f : scale_modifier_arg;
            const float3 scale = make_float3(__ldg(scales + 3 * size_t(idx)), __ldg(scales + 3 * size_t(idx) + 1), __ldg(scales + 3 * size_t(idx) + 2));
            const float4 q = ldg4(rotations + 4 * size_t(idx));
            const Mat3 R = quat_to_mat(q);
            const float3 u = make_float3(R.r11 * scale.x, R.r21 * scale.x, R.r31 * scale.x) * scale_modifier;
            const float3 v = make_float3(R.r12 * scale.y, R.r22 * scale.y, R.r32 * scale.y) * scale_modifier;
            const float3 w = make_float3(R.r13 * scale.z, R.r23 * scale.z, R.r33 * scale.z) * scale_modifier;
            const float4 VPM4 = ldg4(VPM + 12);
            const float4 T4 = row_times_T<true>(VPM4, u, v, w, position);
            // tight cutoff for the opacity threshold of the mode (kernel_utils.cuh:104-108)
            const float rho_cutoff = 2.0f * logf(opacity * MT::min_alpha_rcp);
            const float4 d = make_float4(rho_cutoff, rho_cutoff, rho_cutoff, -1.0f);
            const float s = dot(d, T4 * T4);
            if (s != 0.0f) {
                const float4 f = (1.0f / s) * d;
                // exact near/far culling by the screen-space z extent (kernel_utils.cuh:110-116)
                const float4 VPM3 = ldg4(VPM + 8);
                const float4 T3 = row_times_T<false>(VPM3, u, v, w, position);
                const float center_z = dot(f, T3 * T4);
                const float extent_z = sqrtf(fmaxf(center_z * center_z - dot(f, T3 * T3), 0.0f));
                const float z_min = center_z - extent_z;
                const float z_max = center_z + extent_z;
                if (!(z_min < -1.0f || z_max > 1.0f)) {
                    const float4 VPM1 = ldg4(VPM);
                    const float4 T1 = row_times_T<false>(VPM1, u, v, w, position);
                    const float center_x = dot(f, T1 * T4);
                    const float extent_x = sqrtf(fmaxf(center_x * center_x - dot(f, T1 * T1), 0.0f));
                    const float4 VPM2 = ldg4(VPM + 4);
                    const float4 T2 = row_times_T<false>(VPM2, u, v, w, position);
                    const float center_y = dot(f, T2 * T4);
                    const float extent_y = sqrtf(fmaxf(center_y * center_y - dot(f, T2 * T2), 0.0f));
                    // tile box (+0.5: pixel centres sit at integer coordinates; kernel_utils.cuh:126-137)
                    const float tw = float(MT::tile_w), th = float(MT::tile_h);
                    const uint32_t x_min = min(grid_w, static_cast<uint32_t>(max(0, __float2int_rd((center_x - extent_x + 0.5f) / tw))));
                    const uint32_t x_max = min(grid_w, static_cast<uint32_t>(max(0, __float2int_ru((center_x + extent_x + 0.5f) / tw))));
                    const uint32_t y_min = min(grid_h, static_cast<uint32_t>(max(0, __float2int_rd((center_y - extent_y + 0.5f) / th))));
                    const uint32_t y_max = min(grid_h, static_cast<uint32_t>(max(0, __float2int_ru((center_y + extent_y + 0.5f) / th))));
                    n_touched = (x_max - x_min) * (y_max - y_min);
                    if (n_touched != 0) {
                        out.bounds[idx] = make_ushort4((unsigned short)x_min, (unsigned short)x_max, (unsigned short)y_min, (unsigned short)y_max);
                        float4* dst = reinterpret_cast<float4*>(out.eval + idx);
                        dst[0] = T1; dst[1] = T2; dst[2] = T4;
                        if constexpr (MODE == HTGS_MODE_ALPHA_BLEND_GLOBAL_ORDERING) dst[3] = make_float4(0.0f, 0.0f, 0.0f, z);
                        else dst[3] = make_float4(dot3_pinned_alt(f3(M3), u), dot3_pinned(f3(M3), v), dot3_pinned(f3(M3), w), z);
                        dst[4] = make_float4(position.x, position.y, position.z, opacity);      // until the finish pass puts the colour there
                    }
                }
            }
        }
        out.n_touched[idx] = n_touched;
    }

    // per-block totals (instances, visible Gaussians) and the block's slice of the list of visible Gaussians
    const bool visible = n_touched != 0;
    const uint32_t ballot = __ballot_sync(0xffffffffu, visible);
    uint32_t sum = n_touched;
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if ((threadIdx.x & 31) == 0) { warp_sum[warp] = sum; warp_vis[warp] = __popc(ballot); }
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t total = 0, total_vis = 0;
        #pragma unroll
        for (int i = 0; i < kPreprocessBlock / 32; ++i) { total += warp_sum[i]; total_vis += warp_vis[i]; }
        out.block_sums[blockIdx.x] = total;
        if constexpr (MODE == HTGS_MODE_ALPHA_BLEND_GLOBAL_ORDERING) out.block_offsets[blockIdx.x] = total_vis;      // the scan's input for this mode
        list_base = total_vis ? atomicAdd(&status->n_visible, total_vis) : 0u;
    }
    __syncthreads();
    if (visible) {
        uint32_t slot = list_base + __popc(ballot & lanemask_lt());
        #pragma unroll
        for (int i = 0; i < kPreprocessBlock / 32; ++i)
            if (i < int(warp)) slot += warp_vis[i];
        out.visible_list[slot] = idx;
    }
}

// Whether |d|^2 = |(T1 - x T4) x (T2 - y T4)|^2 stays between 2^-100 and 2^100 at every pixel of the box.  d is the cofactor matrix of the rows
// times (x, y, 1), so |d| is at least the product of the two smaller singular values of the rows, |det| over the largest one.  Holds for
// Gaussians of 1e-9 to 1e5 units at a focal length of 1000 pixels; whatever overflows, underflows or is not a number does not hold.
template <int MODE>
__device__ __forceinline__ bool denominator_in_range(const float4& t1, const float4& t2, const float4& t4, const ushort4& box) {
    using MT = ModeTraits<MODE>;
    const float3 a = f3(t1), b = f3(t2), n = f3(t4);
    const float aa = dot(a, a), bb = dot(b, b), nn = dot(n, n), det = dot(n, cross(a, b));
    const float x = float(box.y) * MT::tile_w, y = float(box.w) * MT::tile_h;
    const float largest = (sqrtf(aa) + x * sqrtf(nn)) * (sqrtf(bb) + y * sqrtf(nn));      // >= |d|
    return det * det > 0x1p-100f * (aa + bb + nn) && largest < 0x1p50f;
}

// Pass 2, one lane per VISIBLE Gaussian (grid-stride over the list, a warp at a time): colour from the SH coefficients, the
// remaining parts of the evaluation record, the conservative outline.  Runs with full warps whatever the
// fraction of Gaussians that survived culling.
//
// The visible Gaussians are scattered, so a lane's inputs share no cache line with its neighbours', and a warp's load of one float
// costs the L1 a look-up per lane, for 45 coefficients, 16 floats of the rows, position and opacity.  So each lane fetches its
// inputs with two bulk copies, the record (in which the cull pass left position and opacity too) and the 16-byte aligned window around
// its row of coefficients, and reads them from shared memory; strides of 80 and, at degree 3, 208 bytes spread the lanes over the
// banks.  What bounds it now is DRAM (40 to 47 % of its throughput at 600 bytes in 64-byte pieces per Gaussian) and the latency of the float64 chains.
// Where no coefficients are wanted (degree 0, importance weights) a lane loads its record itself: the copies' round trip through the mbarrier costs more than
// five loads (16 k Gaussians: 5.5 us, by copies 6.4; 1 M 8.2 and 8.7, importance weights 7.6 and 8.2; 3 M 20.1 and 20.3).
// Loads by lane -> copies, 3 M Gaussians, 1297 x 840: 88 -> 73 us, training 107 -> 88, relaxed precision 94 -> 79, 1.5 M in GLOBAL_ORDERING 82 -> 65.
constexpr int kFinishBlock = 128;
constexpr int kFinishWarps = kFinishBlock / 32;
struct FinishLayout {               // of a warp's part of shared memory: 32 windows, 32 records
    uint32_t window_bytes;          // copied around a row of coefficients (0: degree 0, or no colour wanted)
    uint32_t window_stride;
};
inline FinishLayout finish_layout(int active_sh_bases, bool colour) {
    if (!colour || active_sh_bases <= 1) return {0, 0};
    const uint32_t bytes = (12u * uint32_t(active_sh_bases - 1) + 12u + 15u) & ~15u;      // a row starts up to 12 bytes behind a 16-byte boundary
    return {bytes, (bytes / 16u) % 2u ? bytes : bytes + 16u};                             // an odd number of 16-byte words
}
// Relaxed precision: five blocks spill 28 bytes, four none; both passes of the preprocess at four, five and six blocks: 1 M Gaussians 36.6, 37.6 and 39.5 us, 3 M 93, 92 and
// 95, 8 M 224, 227 and 233, 4 M in dense clusters, 1920 x 1080, 274, 279 and 288 (loads by lane, without a bound: 39, 100, 247, 314).
constexpr int finish_blocks_per_sm(bool train, bool fast) { return train || fast ? 5 : 6; }
template <int MODE, bool TRAIN, bool FAST>
__global__ void __launch_bounds__(kFinishBlock, finish_blocks_per_sm(TRAIN, FAST)) preprocess_finish_kernel(
    const float* __restrict__ sh_0, const float* __restrict__ sh_rest, const float* __restrict__ cam_position_ptr, PrimBuffers out, FrameStatus* status,
    uint32_t n_primitives, int active_sh_bases, int total_sh_bases, OutlineThresholds thresholds, FinishLayout layout)
{
    grid_dependency();
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ uint64_t s_bar[kFinishWarps];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint64_t* bar = s_bar + warp;
    if (lane == 0) mbar_init(bar, 1);
    mbar_fence_init();
    __syncwarp();
    unsigned char* my_window = smem + warp * (32u * (layout.window_stride + sizeof(EvalRecord))) + lane * layout.window_stride;
    float4* my_record = reinterpret_cast<float4*>(smem + warp * (32u * (layout.window_stride + sizeof(EvalRecord))) + 32u * layout.window_stride) + lane * 5u;
    const bool staged = layout.window_bytes != 0;
    const uint32_t n_visible = status->n_visible;
    const float3 cam_position = make_float3(__ldg(cam_position_ptr), __ldg(cam_position_ptr + 1), __ldg(cam_position_ptr + 2));
    const size_t row_bytes = size_t(total_sh_bases) * 12u;
    const uintptr_t sh_begin = reinterpret_cast<uintptr_t>(sh_rest), sh_end = sh_begin + size_t(n_primitives) * row_bytes;
    const uint32_t step = gridDim.x * kFinishBlock;
    uint32_t i = blockIdx.x * kFinishBlock + threadIdx.x;
    uint32_t gi_next = i < n_visible ? out.visible_list[i] : 0u;
    for (uint32_t parity = 0; i - lane < n_visible; i += step, parity ^= 1u) {
        const bool valid = i < n_visible;
        const uint32_t gi = gi_next;
        float4* dst = reinterpret_cast<float4*>(out.eval + gi);
        // the window may reach beyond the ends of the tensor: at the first and last row, if these do not lie on 16-byte boundaries
        const uintptr_t row = sh_begin + size_t(gi) * row_bytes, window = row & ~uintptr_t(15);
        const bool whole = valid && staged && window >= sh_begin && window + layout.window_bytes <= sh_end;
        float4 t1 = make_float4(0.0f, 0.0f, 0.0f, 0.0f), t2 = t1, t4 = t1, m3 = t1, centre_opacity = t1;
        if (staged) {
            const uint32_t n_valid = __popc(__ballot_sync(0xffffffffu, valid)), n_whole = __popc(__ballot_sync(0xffffffffu, whole));
            if (lane == 0) mbar_arrive_expect_tx(bar, n_valid * uint32_t(sizeof(EvalRecord)) + n_whole * layout.window_bytes);
            __syncwarp();
            if (valid) bulk_copy_g2s(my_record, dst, uint32_t(sizeof(EvalRecord)), bar);
            if (whole) bulk_copy_g2s(my_window, reinterpret_cast<const void*>(window), layout.window_bytes, bar);
        } else if (valid) {
            t1 = dst[0]; t2 = dst[1]; t4 = dst[2]; m3 = dst[3]; centre_opacity = dst[4];
        }
        float* coefficients = reinterpret_cast<float*>(my_window + (row & 15u));
        if (valid && !whole && staged) {
            const float* from = sh_rest + size_t(gi) * size_t(total_sh_bases) * 3;
            for (int c = 0; c < 3 * (active_sh_bases - 1); ++c) coefficients[c] = __ldg(from + c);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // in front of the copy that the next round puts here
        }
        float3 dc = make_float3(0.0f, 0.0f, 0.0f);
        ushort4 box = make_ushort4(0, 0, 0, 0);
        if (valid) {
            if (sh_0) dc = make_float3(__ldg(sh_0 + 3 * size_t(gi)), __ldg(sh_0 + 3 * size_t(gi) + 1), __ldg(sh_0 + 3 * size_t(gi) + 2));
            if constexpr (!FAST) box = out.bounds[gi];
        }
        gi_next = i + step < n_visible ? out.visible_list[i + step] : 0u;
        if (staged) {
            if (!mbar_wait_bounded(bar, parity)) {
                atomicOr(&status->error, 1u);
                return;
            }
            if (valid) { t1 = my_record[0]; t2 = my_record[1]; t4 = my_record[2]; m3 = my_record[3]; centre_opacity = my_record[4]; }
        }
        if (valid) {
            const float3 position = f3(centre_opacity);
            const float opacity = centre_opacity.w;
            uint8_t clamp_bits = 0;
            const float3 rgb = sh_0 ? sh_to_rgb<TRAIN>(dc, coefficients, position, cam_position, active_sh_bases, &clamp_bits)
                                    : make_float3(0.0f, 0.0f, 0.0f);   // colour-less callers (update_max_weights)
            [[maybe_unused]] double centre[2] = {0.0, 0.0};
            if constexpr (FAST) make_fast_record(t1, t2, t4, m3, rgb, opacity, dst, centre);
            else dst[4] = make_float4(rgb.x, rgb.y, rgb.z, opacity);
            if constexpr (!FAST) { if (!denominator_in_range<MODE>(t1, t2, t4, box)) atomicOr(&status->divide, 1u); }
            CullRecord cr = make_cull_record(t1, t2, t4, opacity, thresholds);
            if constexpr (TRAIN) {
                out.clamp[gi] = clamp_bits;
                const PairRecord pair = make_pair_record(t1, t2, t4, make_moment_centre<MODE>(t1, t2, t4, box));
                float4* pdst = reinterpret_cast<float4*>(out.pair + gi);
                pdst[0] = pair.n0; pdst[1] = pair.n1; pdst[2] = pair.d1; pdst[3] = make_float4(pair.cx, pair.cy, pair.shear, pair.scale);
            }
            if constexpr (FAST) {
                // The fragment evaluation measures from the projected centre, the outline test from the centre of
                // the outline: the record carries the (small) difference, so that outline centre + difference
                // gives the projected centre to better than float32 resolution at the pixel's magnitude.
                cr.r = float(centre[0] - double(cr.cx));
                cr.g = float(centre[1] - double(cr.cy));
            } else {
                cr.r = rgb.x; cr.g = rgb.y; cr.b = rgb.z;
            }
            float4* cdst = reinterpret_cast<float4*>(out.cull + gi);
            cdst[0] = make_float4(cr.cx, cr.cy, cr.a, cr.b2);
            cdst[1] = make_float4(cr.c, cr.r, cr.g, cr.b);
        }
        __syncwarp();
    }
}

template <int MODE, bool TRAIN, bool FAST>
cudaError_t launch_t(const HtgsScene& scene, const HtgsView& view, const FrameGeometry& geo, const PrimBuffers& prim, FrameStatus* status, int outline_mode, cudaStream_t stream) {
    const uint32_t n = uint32_t(scene.n_primitives);
    const uint32_t blocks = (n + kPreprocessBlock - 1) / kPreprocessBlock;
    if (blocks == 0) return cudaSuccess;
    preprocess_cull_kernel<MODE, TRAIN><<<blocks, kPreprocessBlock, 0, stream>>>(
        scene.positions, scene.scales, scene.rotations, scene.opacities, view.M, view.VPM, prim, status, n, uint32_t(geo.grid_w),
        uint32_t(geo.grid_h), view.near_plane, view.far_plane, view.scale_modifier);
    cudaError_t err = cudaGetLastError();
    if (err != cudaSuccess) return err;
    const FinishLayout layout = finish_layout(view.active_sh_bases, scene.sh_0 != nullptr);
    const uint32_t finish_blocks = min((n + kFinishBlock - 1) / kFinishBlock, uint32_t(sm_count_of_current_device()) * uint32_t(finish_blocks_per_sm(TRAIN, FAST)));
    launch_after(preprocess_finish_kernel<MODE, TRAIN, FAST>, finish_blocks, kFinishBlock, layout.window_bytes != 0 ? size_t(kFinishBlock) * (layout.window_stride + sizeof(EvalRecord)) : 0, stream,
        scene.sh_0, scene.sh_rest, view.cam_position, prim, status, n, view.active_sh_bases, scene.total_sh_bases, outline_thresholds(outline_mode), layout);
    return cudaGetLastError();
}

}  // namespace

int sm_count_of_current_device() {
    static std::atomic<int> cached[64] = {};
    int device = 0;
    cudaGetDevice(&device);
    if (device < 0 || device >= 64) return 148;
    int n = cached[device].load(std::memory_order_relaxed);
    if (!n) {
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || n <= 0) n = 148;
        cached[device].store(n, std::memory_order_relaxed);
    }
    return n;
}

cudaError_t launch_preprocess(int mode, bool train, const HtgsScene& scene, const HtgsView& view, const FrameGeometry& geo,
                              const PrimBuffers& prim, FrameStatus* status, cudaStream_t stream, int outline_mode, bool fast_records) {
    if (fast_records) {
        if (train) return cudaErrorInvalidValue;
        switch (mode) {
            case HTGS_MODE_HYBRID_BLEND: return launch_t<HTGS_MODE_HYBRID_BLEND, false, true>(scene, view, geo, prim, status, outline_mode, stream);
            case HTGS_MODE_ALPHA_BLEND_FIRST_K: return launch_t<HTGS_MODE_ALPHA_BLEND_FIRST_K, false, true>(scene, view, geo, prim, status, outline_mode, stream);
            case HTGS_MODE_OIT_BLEND: return launch_t<HTGS_MODE_OIT_BLEND, false, true>(scene, view, geo, prim, status, outline_mode, stream);
            default: return cudaErrorInvalidValue;
        }
    }
    switch (mode) {
#define HTGS_CASE(M) case M: return train ? launch_t<M, true, false>(scene, view, geo, prim, status, outline_mode, stream) : launch_t<M, false, false>(scene, view, geo, prim, status, outline_mode, stream);
        HTGS_CASE(HTGS_MODE_HYBRID_BLEND)
        HTGS_CASE(HTGS_MODE_ALPHA_BLEND_FIRST_K)
        HTGS_CASE(HTGS_MODE_ALPHA_BLEND_GLOBAL_ORDERING)
        HTGS_CASE(HTGS_MODE_OIT_BLEND)
#undef HTGS_CASE
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace htgs
