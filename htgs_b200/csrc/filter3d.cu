// 3D smoothing-filter update (Mip-Splatting style): for every point inside the (tolerance-widened) frustum of a view,
// filter_3d = min(filter_3d, distance2filter * z) and the point is marked visible.
// Replaces update_3d_filter_cu / update_3d_filter_wrapper of the reference
// (filter3d/src/filter3d_kernels.cu:6-35, filter3d/src/filter3d_api.cu:6-47).  HBM-bound streaming kernel:
// 12 bytes read per point, 5 bytes read-modify-written for the points in view.
#include <algorithm>
#include <cmath>
#include <limits>
#include <string>

#include "kernels.h"


using namespace htgs;

namespace {

__global__ void __launch_bounds__(256) update_3d_filter_kernel(const float* __restrict__ positions, const float* __restrict__ w2c, float* __restrict__ filter_3d,
                                                                 uint8_t* __restrict__ visibility_mask, uint32_t n_points, float left, float right, float top,
                                                                 float bottom, float near_plane, float distance2filter) {
    using namespace htgs;
    const float4 r1 = ldg4(w2c), r2 = ldg4(w2c + 4), r3 = ldg4(w2c + 8);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n_points; i += gridDim.x * blockDim.x) {
        const float3 p = make_float3(__ldg(positions + 3 * size_t(i)), __ldg(positions + 3 * size_t(i) + 1), __ldg(positions + 3 * size_t(i) + 2));
        const float z = dot(f3(r3), p) + r3.w;
        if (z < near_plane) continue;
        const float x_clip = dot(f3(r1), p) + r1.w;
        if (x_clip < left * z || x_clip > right * z) continue;
        const float y_clip = dot(f3(r2), p) + r2.w;
        if (y_clip < top * z || y_clip > bottom * z) continue;
        const float filter_3d_new = distance2filter * z;
        if (filter_3d[i] < filter_3d_new) continue;
        filter_3d[i] = filter_3d_new;
        visibility_mask[i] = 1;
    }
}

// Several views in one pass over the points.  What a sequence of single-view calls leaves is the smallest distance2filter * z of
// the views that see the point (or the old value, if that is smaller), whatever the order of the views, and rounding is
// monotone; so it is enough to find the smallest z of those views, z being the very value update_3d_filter_kernel computes.
//
// What bounds it is instruction issue (600 M tests for 3 M points and 200 views against 51 MB of memory traffic).  The host
// scales the x and y rows of a view so that its frustum is |x| <= z, |y| <= z: a test is then ten packed multiply-adds for two
// points, and a comparison of max(|x|, |y|) with z, without a branch.  Where the two lie closer than the roundings of this form
// (`slack`, about one test in 10^5) the arithmetic of update_3d_filter_kernel decides.  Points or views that are not
// finite numbers go through the sequence itself.  A thread takes several points, so that a view is fetched from shared memory
// once for all of them: six, or two where six would leave SMs without a full set of threads.  200 views, 3 M points: 1040 us (the
// sequence, one point per thread) -> 440 us; 100 k points 68 -> 44 us.
struct __align__(16) FilterView {
    float r3[4], x[4], y[4];                        // depth row as given, scaled rows
    float r1[4], r2[4], left, right, top, bottom;   // as given
    float near_plane, pad[3];
};
template <int VIEWS> struct FilterViewBatch { FilterView view[VIEWS]; float largest_entry, largest_offset; };   // by value: up to 28 KB of kernel parameters
// Sizes of the kernel's parameter block: 3.6 KB, 5.4 KB and 29 KB.  A launch costs more the larger it is, most of all beyond 4 KB; 40 views take 36 us
// with room for 48 and 47 us with room for 256 (16 k points; 300 k: 37 and 51, 3 M: 123 and 126).
constexpr int kFewestViews = 32, kFewViews = 48, kManyViews = 256;

__device__ __forceinline__ float view_depth(const FilterView& v, const float3& p) { return htgs::dot(make_float3(v.r3[0], v.r3[1], v.r3[2]), p) + v.r3[3]; }
__device__ __forceinline__ bool in_view(const FilterView& v, const float3& p, float z) {      // as update_3d_filter_kernel tests it
    if (z < v.near_plane) return false;
    const float x_clip = htgs::dot(make_float3(v.r1[0], v.r1[1], v.r1[2]), p) + v.r1[3];
    if (x_clip < v.left * z || x_clip > v.right * z) return false;
    const float y_clip = htgs::dot(make_float3(v.r2[0], v.r2[1], v.r2[2]), p) + v.r2[3];
    return !(y_clip < v.top * z || y_clip > v.bottom * z);
}

template <int VIEWS, int PAIRS>
__global__ void __launch_bounds__(256) update_3d_filter_views_kernel(const float* __restrict__ positions, float* __restrict__ filter_3d,
                                                                       uint8_t* __restrict__ visibility_mask, uint32_t n_points,
                                                                       const __grid_constant__ FilterViewBatch<VIEWS> batch, int n_views, float distance2filter) {
    constexpr int kPoints = 2 * PAIRS;
    __shared__ float4 s_rows[VIEWS][6];             // r3, x, y with every number twice
    __shared__ float s_near[VIEWS];
    for (int k = threadIdx.x; k < n_views * 3; k += 256) {
        const int v = k / 3, row = k - 3 * v;
        const float4 q = reinterpret_cast<const float4*>(&batch.view[v])[row];
        s_rows[v][2 * row] = make_float4(q.x, q.x, q.y, q.y);
        s_rows[v][2 * row + 1] = make_float4(q.z, q.z, q.w, q.w);
        if (row == 0) s_near[v] = batch.view[v].near_plane;
    }
    __syncthreads();
    const uint32_t base = blockIdx.x * (256 * kPoints) + threadIdx.x;
    auto point_at = [&](int k) -> float3 {
        const uint32_t i = min(base + k * 256, n_points - 1);
        return make_float3(__ldg(positions + 3 * size_t(i)), __ldg(positions + 3 * size_t(i) + 1), __ldg(positions + 3 * size_t(i) + 2));
    };
    f32x2 px[PAIRS], py[PAIRS], pz[PAIRS];
    float slack[kPoints], z_min[kPoints];
    #pragma unroll
    for (int k = 0; k < kPoints; k += 2) {
        const float3 a = point_at(k), b = point_at(k + 1);
        px[k / 2] = pack2(a.x, b.x); py[k / 2] = pack2(a.y, b.y); pz[k / 2] = pack2(a.z, b.z);
        slack[k] = 2e-6f * fmaf(batch.largest_entry, fabsf(a.x) + fabsf(a.y) + fabsf(a.z), batch.largest_offset);
        slack[k + 1] = 2e-6f * fmaf(batch.largest_entry, fabsf(b.x) + fabsf(b.y) + fabsf(b.z), batch.largest_offset);
        z_min[k] = z_min[k + 1] = __int_as_float(0x7f800000);
    }
    for (int v = 0; v < n_views; ++v) {
        const ulonglong2* row = reinterpret_cast<const ulonglong2*>(s_rows[v]);
        const ulonglong2 z01 = row[0], z23 = row[1], x01 = row[2], x23 = row[3], y01 = row[4], y23 = row[5];
        const float near_plane = s_near[v];
        bool unsure = false;
        float z[kPoints];
        #pragma unroll
        for (int k = 0; k < PAIRS; ++k) {
            // z: as nvcc contracts r3.x * p.x + r3.y * p.y + r3.z * p.z, + r3.w
            const float2 zz = unpack2(add2(fma2(z23.x, pz[k], fma2(z01.x, px[k], mul2(z01.y, py[k]))), z23.y));
            const float2 xx = unpack2(fma2(x23.x, pz[k], fma2(x01.y, py[k], fma2(x01.x, px[k], x23.y))));
            const float2 yy = unpack2(fma2(y23.x, pz[k], fma2(y01.y, py[k], fma2(y01.x, px[k], y23.y))));
            #pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int i = 2 * k + h;
                z[i] = h ? zz.y : zz.x;
                const float beyond = fmaxf(fabsf(h ? xx.y : xx.x), fabsf(h ? yy.y : yy.x)) - z[i];
                if (beyond < -slack[i] && z[i] >= near_plane) z_min[i] = fminf(z_min[i], z[i]);
                unsure |= fabsf(beyond) <= slack[i];
            }
        }
        if (unsure) {
            #pragma unroll
            for (int i = 0; i < kPoints; ++i)
                if (z[i] < z_min[i] && in_view(batch.view[v], point_at(i), z[i])) z_min[i] = z[i];
        }
    }
    #pragma unroll
    for (int k = 0; k < kPoints; ++k) {
        const uint32_t i = base + k * 256;
        if (i >= n_points) break;
        const float before = filter_3d[i];
        if (slack[k] < 1e30f) {
            const float after = distance2filter * z_min[k];
            if (z_min[k] < __int_as_float(0x7f800000) && !(before < after)) { filter_3d[i] = after; visibility_mask[i] = 1; }
        } else {
            float current = before;
            bool updated = false;
            const float3 p = point_at(k);
            for (int v = 0; v < n_views; ++v) {
                const float depth = view_depth(batch.view[v], p);
                if (!in_view(batch.view[v], p, depth) || current < distance2filter * depth) continue;
                current = distance2filter * depth;
                updated = true;
            }
            if (updated) { filter_3d[i] = current; visibility_mask[i] = 1; }
        }
    }
}

void frustum_bounds(int32_t width, int32_t height, float focal_x, float focal_y, float center_x, float center_y, float clipping_tolerance,
                    float& left, float& right, float& top, float& bottom) {
    // frustum bounds in normalised camera coordinates (filter3d_api.cu:23-33)
    const float bounds_factor = clipping_tolerance + 0.5f;
    const float width_f = static_cast<float>(width), height_f = static_cast<float>(height);
    const float max_x_shifted = bounds_factor * width_f, max_y_shifted = bounds_factor * height_f;
    const float principal_offset_x = center_x - 0.5f * width_f, principal_offset_y = center_y - 0.5f * height_f;
    left = (-max_x_shifted - principal_offset_x) / focal_x; right = (max_x_shifted - principal_offset_x) / focal_x;
    top = (-max_y_shifted - principal_offset_y) / focal_y; bottom = (max_y_shifted - principal_offset_y) / focal_y;
}

template <int VIEWS, int PAIRS>
cudaError_t launch_views(const float* positions, const HtgsFilterView* views, int count, float* filter_3d, uint8_t* visibility_mask, uint32_t n_points,
                         float clipping_tolerance, float distance2filter, cudaStream_t stream) {
    FilterViewBatch<VIEWS> batch;
    batch.largest_entry = batch.largest_offset = 0.0f;
    bool finite = distance2filter >= 0.0f;
    for (int v = 0; v < count; ++v) {
        const HtgsFilterView& in = views[v];
        FilterView& out = batch.view[v];
        for (int c = 0; c < 4; ++c) { out.r1[c] = in.w2c[c]; out.r2[c] = in.w2c[4 + c]; out.r3[c] = in.w2c[8 + c]; }
        frustum_bounds(in.width, in.height, in.focal_x, in.focal_y, in.center_x, in.center_y, clipping_tolerance, out.left, out.right, out.top, out.bottom);
        out.near_plane = in.near_plane;
        out.pad[0] = out.pad[1] = out.pad[2] = 0.0f;
        // left z <= x_clip <= right z  is  |x_clip - middle z| / half <= z
        const double half_x = 0.5 * (double(out.right) - out.left), middle_x = 0.5 * (double(out.right) + out.left);
        const double half_y = 0.5 * (double(out.bottom) - out.top), middle_y = 0.5 * (double(out.bottom) + out.top);
        finite = finite && half_x > 0.0 && half_y > 0.0 && std::isfinite(out.near_plane);
        for (int c = 0; c < 4; ++c) {
            out.x[c] = float((out.r1[c] - middle_x * out.r3[c]) / half_x);
            out.y[c] = float((out.r2[c] - middle_y * out.r3[c]) / half_y);
            // bounds the terms of the scaled rows, and those of the given rows' own roundings on the same scale
            const double x_terms = (std::fabs(out.r1[c]) + std::fabs(middle_x * out.r3[c])) / half_x, y_terms = (std::fabs(out.r2[c]) + std::fabs(middle_y * out.r3[c])) / half_y;
            const double largest = std::max(double(std::fabs(out.r3[c])), std::max(x_terms, y_terms));
            finite = finite && std::isfinite(largest) && largest < 1e30;
            float& bound = c < 3 ? batch.largest_entry : batch.largest_offset;
            bound = std::max(bound, float(largest));
        }
    }
    if (!finite) batch.largest_offset = std::numeric_limits<float>::infinity();      // every point takes the sequence
    const uint32_t blocks = (n_points + 512 * PAIRS - 1) / (512 * PAIRS);
    update_3d_filter_views_kernel<VIEWS, PAIRS><<<blocks, 256, 0, stream>>>(positions, filter_3d, visibility_mask, n_points, batch, count, distance2filter);
    return cudaGetLastError();
}

}  // namespace

extern "C" int htgs_update_3d_filter_views(const float* positions, const HtgsFilterView* views, int32_t n_views, float* filter_3d,
                                           uint8_t* visibility_mask, int32_t n_points, float clipping_tolerance, float distance2filter, void* stream) {
    if (n_points < 0 || n_views < 0 || (n_points > 0 && n_views > 0 && (!positions || !views || !filter_3d || !visibility_mask))) {
        htgs::set_last_error("htgs_update_3d_filter_views: null pointer or negative size");
        return HTGS_ERR_INVALID_ARGUMENT;
    }
    if (n_points == 0) return HTGS_OK;
    // two points to a thread where more would leave SMs without a full set of threads
    const bool many_points = n_views > kFewViews && uint32_t(n_points) >= uint32_t(htgs::sm_count_of_current_device()) * 4096u;
    for (int32_t first = 0; first < n_views;) {
        const int32_t left = n_views - first, count = std::min<int32_t>(left, left > kFewViews ? kManyViews : kFewViews);
        const auto launch = count <= kFewestViews ? launch_views<kFewestViews, 1> : count <= kFewViews ? launch_views<kFewViews, 1> : many_points ? launch_views<kManyViews, 3> : launch_views<kManyViews, 1>;
        const cudaError_t err = launch(positions, views + first, count, filter_3d, visibility_mask, uint32_t(n_points), clipping_tolerance, distance2filter,
                                       static_cast<cudaStream_t>(stream));
        if (err != cudaSuccess) {
            htgs::set_last_error((std::string("htgs_update_3d_filter_views: ") + cudaGetErrorString(err)).c_str());
            return HTGS_ERR_CUDA;
        }
        first += count;
    }
    return HTGS_OK;
}

extern "C" int htgs_update_3d_filter(const float* positions, const float* w2c, float* filter_3d, uint8_t* visibility_mask, int32_t n_points,
                                     int32_t width, int32_t height, float focal_x, float focal_y, float center_x, float center_y, float near_plane,
                                     float clipping_tolerance, float distance2filter, void* stream) {
    if (n_points < 0 || (n_points > 0 && (!positions || !w2c || !filter_3d || !visibility_mask))) {
        htgs::set_last_error("htgs_update_3d_filter: null pointer or negative size");
        return HTGS_ERR_INVALID_ARGUMENT;
    }
    if (n_points == 0) return HTGS_OK;
    float left, right, top, bottom;
    frustum_bounds(width, height, focal_x, focal_y, center_x, center_y, clipping_tolerance, left, right, top, bottom);
    const uint32_t blocks = uint32_t(std::min<int64_t>((int64_t(n_points) + 255) / 256, int64_t(htgs::sm_count_of_current_device()) * 8));
    update_3d_filter_kernel<<<blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(positions, w2c, filter_3d, visibility_mask, uint32_t(n_points), left, right, top,
                                                                                  bottom, near_plane, distance2filter);
    const cudaError_t err = cudaGetLastError();
    if (err != cudaSuccess) {
        htgs::set_last_error((std::string("htgs_update_3d_filter: ") + cudaGetErrorString(err)).c_str());
        return HTGS_ERR_CUDA;
    }
    return HTGS_OK;
}
