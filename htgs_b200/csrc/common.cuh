// Shared declarations of the sm_100a rasterizer core: per-mode constants, the
// device-side data layout, small vector algebra and PTX wrappers.
#pragma once

#include <cuda_runtime.h>
#include <cstdint>
#include <cfloat>

#include "../../include/htgs_b200.h"

namespace htgs {

// ---------------------------------------------------------------------------
// per-mode numerical constants; they are part of the numerical contract with
// the reference (rasterization/include/*/config.h:15-29)
// ---------------------------------------------------------------------------
constexpr float kTransmittanceThreshold = 1e-4f;
constexpr float kMaxFragmentAlpha = 1.0f;
constexpr float kOneMinusAlphaEps = 1e-8f;

template <int MODE> struct ModeTraits;
template <> struct ModeTraits<HTGS_MODE_HYBRID_BLEND> {
    static constexpr int tile_w = 8, tile_h = 8;
    static constexpr float min_alpha_rcp = 255.0f;
    static constexpr float min_alpha = 1.0f / 255.0f;
    static constexpr float max_cutoff_sq = 11.0825270903f;
    static constexpr float min_alpha_core = 1.0f / 20.0f;
};
template <> struct ModeTraits<HTGS_MODE_ALPHA_BLEND_FIRST_K> {
    static constexpr int tile_w = 8, tile_h = 8;
    static constexpr float min_alpha_rcp = 20.0f;
    static constexpr float min_alpha = 1.0f / 20.0f;
    static constexpr float max_cutoff_sq = 5.99146454711f;
    static constexpr float min_alpha_core = 0.0f;
};
template <> struct ModeTraits<HTGS_MODE_ALPHA_BLEND_GLOBAL_ORDERING> {
    static constexpr int tile_w = 16, tile_h = 16;
    static constexpr float min_alpha_rcp = 255.0f;
    static constexpr float min_alpha = 1.0f / 255.0f;
    static constexpr float max_cutoff_sq = 11.0825270903f;
    static constexpr float min_alpha_core = 0.0f;
};
template <> struct ModeTraits<HTGS_MODE_OIT_BLEND> {
    static constexpr int tile_w = 8, tile_h = 8;
    static constexpr float min_alpha_rcp = 255.0f;
    static constexpr float min_alpha = 1.0f / 255.0f;
    static constexpr float max_cutoff_sq = 11.0825270903f;
    static constexpr float min_alpha_core = 0.0f;
};

inline int mode_tile_w(int mode) { return mode == HTGS_MODE_ALPHA_BLEND_GLOBAL_ORDERING ? 16 : 8; }
inline int mode_tile_h(int mode) { return mode == HTGS_MODE_ALPHA_BLEND_GLOBAL_ORDERING ? 16 : 8; }

// ---------------------------------------------------------------------------
// data layout in HBM
// ---------------------------------------------------------------------------
// What the blend kernels need to evaluate one Gaussian at a pixel: 80 bytes,
// 16-byte aligned, so one record moves to shared memory with a single bulk
// asynchronous copy.  Rows of the 3x4 matrices (VP*M*T) and (M*T) of the
// reference (kernel_utils.cuh:98-123, hybrid_blend/kernels/inference.cuh:57-74).
struct __align__(16) EvalRecord {
    float4 vpmt1;
    float4 vpmt2;
    float4 vpmt4;
    float4 mt3;    // .w = view-space depth of the centre
    float4 rgba;   // view-dependent colour (clamped at 0), opacity
};
static_assert(sizeof(EvalRecord) == 80, "EvalRecord must be 80 bytes");

// Conservative screen-space outline of the fragment-acceptance region
// { pixel : alpha(pixel) >= min_alpha }, an ellipse
//   a*dx^2 + b2*dx*dy + c*dy^2 <= 1,  (dx,dy) = pixel - (cx,cy),
// computed in float64, inflated by a safety margin (see preprocess.cu).  It
// has no counterpart in the reference; it only removes (pixel, Gaussian)
// pairs that the exact per-fragment test would reject anyway.
struct __align__(16) CullRecord {
    float cx, cy;
    float a, b2;
    float c;
    // Exact path: the Gaussian's colour.  The blend kernels look it up when a fragment leaves the K-buffer and when a pixel is
    // composited; here it shares the 32-byte sector that the outline test has read (the evaluation records do not stay in L2).
    // Relaxed-precision path: (projected centre of the Gaussian - (cx, cy)), 0.
    float r, g, b;
};
static_assert(sizeof(CullRecord) == 32, "CullRecord must be 32 bytes");

// Relaxed-precision evaluation record (fast_rasterize path, HYBRID_BLEND), same size and place as EvalRecord.
// With (dx, dy) = pixel - (cx, cy), where (cx, cy) is the projected centre of the Gaussian, the two planes through
// the pixel ray (hybrid_blend/kernels/fast_inference.cuh:150-156) give m = w4 * (dy * a - dx * b) and
// d = d0 + dx * dX + dy * dY, so rho^2 = (m.m)/(d.d) and depth = MT3.(d x m)/(d.d) + MT3.w are ratios of
// quadratics in (dx, dy) whose coefficients are fixed per Gaussian (float64 in the preprocess, divided by d0.d0):
//   e     = q1xx dx^2 + q1xy dx dy + q1yy dy^2           = -0.5 * log2(e) * (m.m) / (d0.d0)
//   den   = 1 + q2x dx + q2y dy + q2xx dx^2 + q2xy dx dy + q2yy dy^2  = (d.d) / (d0.d0)
//   num_z = q3x dx + q3y dy + q3xx dx^2 + q3xy dx dy + q3yy dy^2       = MT3.(d x m) / (d0.d0)
//   alpha = min(exp2(e / den + log2_opacity), 1),   depth = num_z / den + depth_centre
// The centre travels with the outline record (CullRecord: outline centre cx, cy plus the difference cx_lo, cy_lo to the
// projected centre): a single float32 centre costs 6e-5 px at x ~ 1000, the dominant error of alpha for Gaussians of
// sub-pixel extent.  The staging thread turns it into a tile-relative offset, dx = x_in_tile + dx0.
struct __align__(16) FastRecord {
    float q1xx, q1xy, q1yy, q2x;
    float q2y, q2xx, q2xy, q2yy;
    float q3x, q3y, q3xx, q3xy;
    float q3yy, depth_centre, log2_opacity, r;
    float g, b, pad0, pad1;
};
static_assert(sizeof(FastRecord) == sizeof(EvalRecord), "FastRecord shares the storage of EvalRecord");

// What the backward pass evaluates a pair with (training only).  rho^2 = N / D (both up to a factor that cancels), N = |m|^2 and D = |d|^2
// quadratic in (s, y): y = pixel_y - cy, s = pixel_x - cx + shear * y.  Computed in float64: a rounding of a coefficient is the
// same at every pixel and does not average out in a gradient that sums thousands of them.
struct __align__(16) PairRecord {
    float4 n0, n1, d1;        // n0 = N: 1, s, y, ss   n1 = N: sy, yy, D: 1, s   d1 = D: y, ss, sy, yy   (N first: the chain rule reads only that)
    float cx, cy, shear, scale;     // scale: what N and D were multiplied by (1 / D at the centre)
};
static_assert(sizeof(PairRecord) == 64, "PairRecord must be 64 bytes");

// Device-resident frame status, copied to the host at the end of a call.
struct __align__(16) FrameStatus {      // its first four words are read with one load
    unsigned int n_instances;     // total (tile, Gaussian) instances of the frame
    unsigned int overflow;        // 1 if n_instances exceeded the instance capacity of the workspace
    unsigned int n_visible;       // Gaussians that survived culling
    unsigned int error;           // bounded waits that gave up, bad arguments seen on the device, ...
    unsigned long long candidate_pairs;     // statistics mode of the blend kernels
    unsigned long long accepted_fragments;  // statistics mode of the blend kernels
    unsigned long long warp_trips;          // statistics mode, HYBRID_BLEND: times a warp came to the insertion, behind two or three candidates per lane (K < 8 or a wide depth range: one)
    unsigned long long warp_trips_inserting;// ... and at least one lane inserted into its K-buffer
    unsigned long long lane_insertions;     // ... and the lanes that inserted
    unsigned int range_blocks_done;         // blocks of the tile-range kernel that have finished; the last one orders the tiles
    unsigned int divide;                    // 1 if a visible Gaussian's |d|^2 may lie outside the range of reciprocal_rn
};

// ---------------------------------------------------------------------------
// vector algebra.  The expression shapes (association order of sums of
// products) follow the helper the reference uses (utils/helper_math.h: dot
// 1267-1274, cross 1451-1454, normalize 1328-1332), so that the compiler's
// multiply-add contraction yields the same rounding as the reference build.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float3 f3(const float4& a) { return make_float3(a.x, a.y, a.z); }
__device__ __forceinline__ float dot(const float3& a, const float3& b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ float dot(const float4& a, const float4& b) { return a.x * b.x + a.y * b.y + a.z * b.z + a.w * b.w; }
__device__ __forceinline__ float3 cross(const float3& a, const float3& b) {
    return make_float3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}
__device__ __forceinline__ float3 operator*(const float3& a, float s) { return make_float3(a.x * s, a.y * s, a.z * s); }
__device__ __forceinline__ float3 operator*(float s, const float3& a) { return make_float3(s * a.x, s * a.y, s * a.z); }
__device__ __forceinline__ float3 operator*(const float3& a, const float3& b) { return make_float3(a.x * b.x, a.y * b.y, a.z * b.z); }
__device__ __forceinline__ float3 operator+(const float3& a, const float3& b) { return make_float3(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ float3 operator-(const float3& a, const float3& b) { return make_float3(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ float3 operator+(float s, const float3& a) { return make_float3(s + a.x, s + a.y, s + a.z); }
__device__ __forceinline__ float3 operator-(const float3& a) { return make_float3(-a.x, -a.y, -a.z); }
__device__ __forceinline__ void operator+=(float3& a, const float3& b) { a.x += b.x; a.y += b.y; a.z += b.z; }
__device__ __forceinline__ float4 operator*(const float4& a, const float4& b) { return make_float4(a.x * b.x, a.y * b.y, a.z * b.z, a.w * b.w); }
__device__ __forceinline__ float4 operator*(const float4& a, float s) { return make_float4(a.x * s, a.y * s, a.z * s, a.w * s); }
__device__ __forceinline__ float4 operator*(float s, const float4& a) { return make_float4(s * a.x, s * a.y, s * a.z, s * a.w); }
__device__ __forceinline__ float4 operator-(const float4& a, const float4& b) { return make_float4(a.x - b.x, a.y - b.y, a.z - b.z, a.w - b.w); }
__device__ __forceinline__ float4 operator+(const float4& a, const float4& b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
__device__ __forceinline__ void operator+=(float4& a, const float4& b) { a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w; }
__device__ __forceinline__ float3 normalize(const float3& v) { const float inv_len = rsqrtf(dot(v, v)); return v * inv_len; }
__device__ __forceinline__ float length(const float3& v) { return sqrtf(dot(v, v)); }

// 1 / x rounded to nearest: the hardware approximation (within one unit in the last place) and one Newton step with the residual in a
// fused multiply-add (Markstein, IBM J. Res. Dev. 34(1), 1990).  Equal to 1.0f / x for 2^-126 <= x <= 2^126, where x and 1 / x are
// normal numbers (tests/test_gpu_reciprocal.py compares all of them), and not for other x: frames that hold a Gaussian whose
// denominators may be such a number divide instead (FrameStatus::divide).  The compiler's quotient takes a branch, which keeps two
// evaluations from being interleaved; without it the blend kernels run 10 % faster.
__device__ __forceinline__ float reciprocal_rn(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return __fmaf_rn(y, __fmaf_rn(-x, y, 1.0f), y);
}

// Two floats in one register pair: one instruction for two rounded operations (two of them take the FMA pipe as long as four single ones would, but half
// the issue slots).
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) { f32x2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi)); return r; }
__device__ __forceinline__ float2 unpack2(f32x2 v) { float2 r; asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v)); return r; }
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) { f32x2 r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) { f32x2 r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) { f32x2 r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }


__device__ __forceinline__ float4 ldg4(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }

__device__ __forceinline__ float sqrt_approx(float x) { float y; asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }

// Pixels of the 8 x 4 block at (x0, y0) that the outline a dx^2 + b2 dx dy + c dy^2 <= 1 about (cx, cy) can touch: bit
// (row * 8 + column).  A row is cut in an interval; 0.01 pixel is added at both ends, far more than the roundings here and
// far less than the 0.3 pixel by which the outline was inflated.  Lengths along the row are in units of the block's width, so that the clamp to
// the block is the additions' saturation; a row that the outline does not reach has the root of a negative number, which the
// saturation turns into 0 at both ends.  The ends are rounded to whole pixels by adding 1.5 * 2^23, whose low bits then are the
// shift counts.  About 70 instructions, five of them on the pipe for roots and conversions (rounding by conversions: 100 and 13).  3 M Gaussians, 1297 x
// 840: max_weights 449 -> 438 us, backward tiles 995 -> 980, blend 866 -> 856; 1.5 M in GLOBAL_ORDERING: blend 268 -> 257.
__device__ __forceinline__ uint32_t outline_mask(const float4& c0, float cc, float x0, float y0) {
    float a_rcp;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(a_rcp) : "f"(c0.z));
    const float slope = (-0.0625f * c0.w) * a_rcp;                             // centre of the interval per unit of dy
    const float width = 0.015625f * a_rcp;
    const float shrink = fmaf(slope, slope, -cc * width);                      // half width^2 = 1/a + shrink * dy^2
    const float middle = fmaf(c0.x - x0, 0.125f, 0.0625f), dy0 = y0 - c0.y;    // half a pixel further, for the rounding
    uint32_t mask = 0;
    #pragma unroll
    for (int r = 3; r >= 0; --r) {
        const float dy = dy0 + float(r);
        const float half = sqrt_approx(fmaf(shrink * dy, dy, width)) + 0.00125f;
        const float mid = fmaf(slope, dy, middle);
        const float begin = fmaf(__saturatef(mid - half), 8.0f, 12582912.0f), end = fmaf(__saturatef(mid + half), 8.0f, 12582912.0f);
        // bits begin .. end - 1 (the shifts take their count modulo 32)
        const uint32_t row = __funnelshift_l(0u, 1u, __float_as_uint(end)) - __funnelshift_l(0u, 1u, __float_as_uint(begin));
        mask = mask * 256u + row;
    }
    if (c0.z == 0.0f) mask = c0.x > 1e30f ? 0u : 0xffffffffu;   // nothing can be accepted / no proper ellipse: every pixel is a candidate
    return mask;
}

// 16 x 16 bits per half warp: row r in the low half word of lane r -> column r.
__device__ __forceinline__ uint32_t transpose_16x16(uint32_t x, uint32_t lane) {
    #pragma unroll
    for (int d = 8; d > 0; d >>= 1) {
        const uint32_t low = d == 8 ? 0x00ffu : d == 4 ? 0x0f0fu : d == 2 ? 0x3333u : 0x5555u;
        const bool up = lane & uint32_t(d);
        const uint32_t y = __shfl_xor_sync(0xffffffffu, x, d);
        const uint32_t t = __funnelshift_l(y, y, up ? 32u - d : d);
        const uint32_t keep = up ? ~low : low;
        x = (x & keep) | (t & ~keep);
    }
    return x & 0xffffu;
}
// Lane i < 16 holds the pixel mask of survivor i; the result has, in lane = pixel, bit 15 - i set if survivor i can touch it.
__device__ __forceinline__ uint32_t transpose_masks(uint32_t mask, uint32_t lane) {
    return transpose_16x16(__shfl_sync(0xffffffffu, mask, 15u - (lane & 15u)) >> (lane & 16u), lane);
}
// The way back: lane = pixel holds bits 15 - i; the result has, in lanes i and i + 16, survivor i's pixels 0..15 and 16..31.
__device__ __forceinline__ uint32_t transpose_half(uint32_t bits, uint32_t lane) {
    return __shfl_sync(0xffffffffu, transpose_16x16(bits & 0xffffu, lane), (lane & 16u) | (15u - (lane & 15u)));
}

// update_max_weights: the largest weight of a Gaussian, as the bits of a non-negative float
__device__ __forceinline__ void raise_weight(unsigned int* max_weights, uint32_t primitive_idx, float weight) {
    const unsigned int bits = __float_as_uint(weight);
    if (max_weights[primitive_idx] < bits) atomicMax(&max_weights[primitive_idx], bits);
}

// ---------------------------------------------------------------------------
// PTX wrappers: mbarrier + bulk asynchronous copy (TMA, non-tensor, single-CTA destination)
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return ok != 0;
}
// Bounded wait: gives up after `limit` polls and reports failure instead of spinning forever.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, uint32_t limit = (1u << 22)) {
    for (uint32_t i = 0; i < limit; ++i)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}
// global -> shared bulk copy; src/dst 16-byte aligned, bytes a multiple of 16; completion is
// signalled on the mbarrier as transferred bytes.
__device__ __forceinline__ void bulk_copy_g2s(void* dst_smem, const void* src_gmem, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_u32(dst_smem)), "l"(src_gmem), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}

// First statement of a kernel that is launched with launch_after: waits until the previous kernel of the stream has finished and its writes
// are visible, then lets the next one take its place on the SMs as soon as this one has no block left to start.  In this
// order a kernel never starts beside the last but one, which may still be reading (and caching) what the last one overwrites.
__device__ __forceinline__ void grid_dependency() {
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
}

__device__ __forceinline__ unsigned int lanemask_lt() { unsigned int m; asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m)); return m; }

// ---------------------------------------------------------------------------
// Compact gradient rows (multi-GPU gradient exchange).  A buffer is one 64-byte header followed by 64-byte rows,
// one per Gaussian the view kept, in no particular order:
//     float4 0: Gaussian index (bits), dL/dposition          float4 2: dL/drotation (r, x, y, z)
//     float4 1: dL/dscale, dL/dopacity                       float4 3: dL/drgb after the clamp mask, 0
// The rows of grad_sh_0 and grad_sh_rest are products of dL/drgb with functions of the view direction
// (kernel_utils.cuh:190-281 of the reference), so a reader that has the camera position rebuilds them.
// ---------------------------------------------------------------------------
struct CompactGradientHeader {
    unsigned int count;            // rows appended (may exceed the capacity: rows beyond it were dropped)
    float cam_x, cam_y, cam_z;     // camera position of the view the rows were computed for
    unsigned int active_sh_bases;  // 1, 4, 9 or 16
    unsigned int reserved[11];
};
static_assert(sizeof(CompactGradientHeader) == 64, "the header takes one row");
constexpr int kCompactRowFloat4s = 4;
constexpr float kShBand0 = 0.28209479177387814f;

// dL/dsh_rest of one Gaussian: rows[i] = (basis function i + 1 of `dir`) * grad_rgb for the active bases; returns how many
// rows were written (0, 3, 8 or 15).  One definition for the kernel that writes dense gradients and for the kernels that
// rebuild them from compact rows, so that both produce the same bits.
__device__ __forceinline__ int sh_rest_gradient_rows(const float3& dir, const float3& grad_rgb, int active_sh_bases, float3 (&rows)[15]) {
    if (active_sh_bases <= 1) return 0;
    const float dx = dir.x, dy = dir.y, dz = dir.z;
    rows[0] = (-0.48860251190291987f * dy) * grad_rgb;
    rows[1] = (0.48860251190291987f * dz) * grad_rgb;
    rows[2] = (-0.48860251190291987f * dx) * grad_rgb;
    if (active_sh_bases <= 4) return 3;
    const float sxx = dx * dx, syy = dy * dy, szz = dz * dz, sxy = dx * dy, sxz = dx * dz, syz = dy * dz;
    rows[3] = (1.0925484305920792f * sxy) * grad_rgb;
    rows[4] = (-1.0925484305920792f * syz) * grad_rgb;
    rows[5] = (0.94617469575755997f * szz - 0.31539156525251999f) * grad_rgb;
    rows[6] = (-1.0925484305920792f * sxz) * grad_rgb;
    rows[7] = (0.54627421529603959f * sxx - 0.54627421529603959f * syy) * grad_rgb;
    if (active_sh_bases <= 9) return 8;
    rows[8] = (0.59004358992664352f * dy * (-3.0f * sxx + syy)) * grad_rgb;
    rows[9] = (2.8906114426405538f * sxy * dz) * grad_rgb;
    rows[10] = (0.45704579946446572f * dy * (1.0f - 5.0f * szz)) * grad_rgb;
    rows[11] = (0.3731763325901154f * dz * (5.0f * szz - 3.0f)) * grad_rgb;
    rows[12] = (0.45704579946446572f * dx * (1.0f - 5.0f * szz)) * grad_rgb;
    rows[13] = (1.4453057213202769f * dz * (sxx - syy)) * grad_rgb;
    rows[14] = (0.59004358992664352f * dx * (-sxx + 3.0f * syy)) * grad_rgb;
    return 15;
}

}  // namespace htgs
