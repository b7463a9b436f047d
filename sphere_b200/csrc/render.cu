// Ray-traced image of the particles: the reference's renderer
// (src/raytracer.cuh: imageInit, rayInitPerspective, rayIntersectSpheres,
// rayIntersectSpheresColormap, DEM::cameraInit, DEM::render;
// src/colorbar.h) as one kernel that writes a host RGBA buffer; the caller
// writes the PPM (DEM::writePPM, src/file_io.cpp:734-757).
//
// Every pixel casts one ray from the eye and keeps the nearest hit, the first
// in original order among equally near ones.  The reference tests every
// sphere for every pixel; here a block renders a tile of 16 x 16 pixels and
// tests only the spheres whose projection can reach it: each sphere gets a
// rectangle of pixels (k_render_prep), 32 spheres adjacent in the cell sort
// share the rectangle around theirs, and a tile first walks those.  The hit
// test's own FP32 arithmetic is the reference's in its order (this file is
// compiled with -fmad=false; vector lengths and normalisation use IEEE sqrtf
// and division), and the rectangles cover its rounding, so the pixels equal a
// host restatement of the same formulas.  800 x 800 pixels of 100,000 spheres, a
// whole call on a B200: 50.6 ms with every ray against every sphere, 0.57 ms so
// (the camera's extent is reduced on the device too, and the scratch is kept).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "engine_internal.h"
#include "dem_launch.h"

namespace sphb {

namespace {

constexpr int kRtTile = 16;                        // pixels per side of a block's tile
constexpr int kRtThreads = kRtTile * kRtTile;
constexpr unsigned kRtList = 2 * kRtThreads;       // spheres staged per pass over the pixels

struct F3 {
    float x, y, z;
};
__host__ __device__ inline F3 f3(float x, float y, float z) { return F3{x, y, z}; }
__host__ __device__ inline F3 operator+(F3 a, F3 b) { return f3(a.x + b.x, a.y + b.y, a.z + b.z); }
__host__ __device__ inline F3 operator-(F3 a, F3 b) { return f3(a.x - b.x, a.y - b.y, a.z - b.z); }
__host__ __device__ inline F3 operator-(F3 a) { return f3(-a.x, -a.y, -a.z); }
__host__ __device__ inline F3 operator*(float s, F3 a) { return f3(s * a.x, s * a.y, s * a.z); }
__host__ __device__ inline F3 operator*(F3 a, float s) { return f3(a.x * s, a.y * s, a.z * s); }
__host__ __device__ inline F3 operator*(F3 a, F3 b) { return f3(a.x * b.x, a.y * b.y, a.z * b.z); }
__host__ __device__ inline F3 operator/(F3 a, float s) { return f3(a.x / s, a.y / s, a.z / s); }
__host__ __device__ inline float dot(F3 a, F3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__host__ __device__ inline F3 cross(F3 a, F3 b)
{
    return f3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}
__host__ __device__ inline float length(F3 v) { return sqrtf(dot(v, v)); }
__host__ __device__ inline F3 normalize(F3 v) { return v * (1.0f / sqrtf(dot(v, v))); }

// the blue-white-red colour map of src/colorbar.h
__device__ inline float cm_red(float r) { return fminf(1.0f, 0.209f * r * r * r - 2.49f * r * r + 3.0f * r + 0.0109f); }
__device__ inline float cm_green(float r) { return fminf(1.0f, -2.44f * r * r + 2.15f * r + 0.369f); }
__device__ inline float cm_blue(float r) { return fminf(1.0f, -2.21f * r * r + 1.61f * r + 0.573f); }

struct Camera {
    F3 u, v, w, eye, light;
    float d;
    float plane[4];   // image plane extent (x0, x1, y0, y1)
    unsigned width, height;
};

// Largest coordinates of the particles (from 0), as bit patterns of
// non-negative doubles, which order like integers.
__global__ void __launch_bounds__(256) k_render_extent(DevParams P, DevState S, unsigned long long *out)
{
    unsigned long long m[3] = {0, 0, 0};
    for (unsigned k = blockIdx.x * blockDim.x + threadIdx.x; k < P.np; k += gridDim.x * blockDim.x) {
        const double4 x = S.x[k];
        const double c[3] = {x.x, x.y, x.z};
        for (int d = 0; d < 3; ++d)
            if (c[d] > 0.0) m[d] = max(m[d], (unsigned long long)__double_as_longlong(c[d]));
    }
    for (int d = 0; d < 3; ++d) {
        for (int o = 16; o > 0; o >>= 1) m[d] = max(m[d], __shfl_xor_sync(0xffffffffu, m[d], o));
        if ((threadIdx.x & 31) == 0) atomicMax(&out[d], m[d]);
    }
}

// DEM::render + DEM::cameraInit: the reference's eye and look-at points
__global__ void k_render_camera(DevParams P, const unsigned long long *extent, unsigned width, unsigned height,
                                Camera *out)
{
    Camera C;
    C.width = width;
    C.height = height;
    const float imgw = (float)(P.L[0] * 1.35f);
    const F3 lookat = f3((float)__longlong_as_double((long long)extent[0]),
                         (float)__longlong_as_double((long long)extent[1]),
                         (float)__longlong_as_double((long long)extent[2])) / 2.0f;
    const F3 eye = f3((float)(P.L[0] * 2.3f), (float)(P.L[1] * -5.0f), (float)(P.L[2] * 1.3f));
    const float hw_ratio = (float)(height / width);   // integer division, as the reference
    C.plane[0] = -0.5f * imgw;
    C.plane[1] = 0.5f * imgw;
    C.plane[2] = -0.5f * imgw * hw_ratio;
    C.plane[3] = 0.5f * imgw * hw_ratio;
    const F3 view = eye - lookat;
    const F3 up = f3(0.0f, 0.0f, 1.0f);
    C.w = -view / length(view);
    C.u = cross(up, C.w) / length(cross(up, C.w));
    C.v = cross(C.w, C.u);
    C.eye = eye;
    C.d = length(view) * 0.8f;
    C.light = normalize(-1.0f * eye * f3(1.0f, 0.2f, 0.6f));
    *out = C;
}

// Range of q for which the line from the origin through (q, D) passes within
// r of the point (a, b), both ways along the line; the whole axis where the
// point is too near to the origin or the line could turn through the plane.
__device__ void line_range(double a, double b, double r, double D, double &lo, double &hi)
{
    lo = -1e300;
    hi = 1e300;
    const double n = sqrt(a * a + b * b);
    if (!(r < 0.999 * n)) return;
    const double s = b < 0.0 ? -1.0 : 1.0;
    const double t = atan2(s * a, s * b), w = asin(r / n), edge = 1.5707;
    if (t - w < -edge || t + w > edge) return;
    lo = D * tan(t - w);
    hi = D * tan(t + w);
}

// Per-particle render data in sorted order: position and radius in FP32, the
// colour-map value (FP64) and the fixvel flag, and the rectangle of pixels
// (columns x..z, rows y..w) outside which the hit test fails; the rectangle
// around 32 of them.
//
// The test is Delta = (2 d.ec)^2 - 4 d.d (ec.ec - R^2) > 0 in FP32.  With unit
// roundoff u the two products differ from their exact values by less than
// 36 u and 48 u times |d|^2 (|ec|^2 + R^2) (dot products of three terms on
// differences of FP32 coordinates, two multiplications each), so a positive
// Delta means a distance from the line below sqrt(R^2 + 21 u (|ec|^2 + R^2)).
// 32 u are allowed here, 1e-5 |ec| for the rounding of d and of the camera's
// axes, and a pixel to each side for the rounding of the image coordinates.
__global__ void k_render_prep(DevParams P, DevState S, int method, float lower_cutoff, const Camera *cam,
                              float4 *xr, double *val, float *fixvel, float4 *rect, float4 *grect)
{
    const unsigned k = blockIdx.x * blockDim.x + threadIdx.x;
    float4 box = make_float4(1e30f, 1e30f, -1e30f, -1e30f);   // empty
    if (k < P.np) {
        const double4 x = S.x[k];
        const float4 c = make_float4((float)x.x, (float)x.y, (float)x.z, (float)x.w);
        xr[k] = c;
        const double4 v = S.vel[k];
        fixvel[k] = (float)v.w;
        double a = 0.0;
        if (method == 1) {
            a = S.p[k];
        } else if (method == 2) {
            a = sqrt(v.x * v.x + v.y * v.y + v.z * v.z);
        } else if (method == 3) {
            const double4 w = S.angvel[k];
            a = sqrt(w.x * w.x + w.y * w.y + w.z * w.z);
        } else if (method == 4) {
            a = S.xyzsum[k].x;
        } else if (method == 5) {
            const double4 r = S.angpos[k];
            a = sqrt(r.x * r.x + r.y * r.y + r.z * r.z);
        }
        val[k] = a;
        const bool shown = method == 0 || !(lower_cutoff > 0.0) ||
                           ((float)a > lower_cutoff && (float)v.w == 0.f);
        if (shown) {
            const Camera C = *cam;
            const double sx = (double)c.x - C.eye.x, sy = (double)c.y - C.eye.y, sz = (double)c.z - C.eye.z;
            const double l2 = sx * sx + sy * sy + sz * sz, R2 = (double)c.w * c.w;
            box = make_float4(-1e30f, -1e30f, 1e30f, 1e30f);
            if (l2 < 1e15 && R2 < 1e15) {
                const double Rc = sqrt(R2 + 32.0 * 0x1p-24 * (l2 + R2)) + 1e-5 * sqrt(l2);
                const double fu = sx * C.u.x + sy * C.u.y + sz * C.u.z;
                const double fv = sx * C.v.x + sy * C.v.y + sz * C.v.z;
                const double fw = -(sx * C.w.x + sy * C.w.y + sz * C.w.z);
                double lo, hi;
                if (C.plane[1] > C.plane[0]) {
                    line_range(fu, fw, Rc, C.d, lo, hi);
                    const double px = C.width / ((double)C.plane[1] - C.plane[0]);
                    box.x = (float)fmax(-1e30, (lo - C.plane[0]) * px - 1.5);
                    box.z = (float)fmin(1e30, (hi - C.plane[0]) * px + 0.5);
                }
                if (C.plane[3] > C.plane[2]) {
                    line_range(fv, fw, Rc, C.d, lo, hi);
                    const double px = C.height / ((double)C.plane[3] - C.plane[2]);
                    box.y = (float)fmax(-1e30, (lo - C.plane[2]) * px - 1.5);
                    box.w = (float)fmin(1e30, (hi - C.plane[2]) * px + 0.5);
                }
            }
        }
        rect[k] = box;
    }
    for (int o = 16; o > 0; o >>= 1) {
        box.x = fminf(box.x, __shfl_xor_sync(0xffffffffu, box.x, o));
        box.y = fminf(box.y, __shfl_xor_sync(0xffffffffu, box.y, o));
        box.z = fmaxf(box.z, __shfl_xor_sync(0xffffffffu, box.z, o));
        box.w = fmaxf(box.w, __shfl_xor_sync(0xffffffffu, box.w, o));
    }
    if ((threadIdx.x & 31) == 0 && k < P.np) grect[k >> 5] = box;
}

// One pixel per thread, a tile of 16 x 16 per block.  method 0: Lambertian
// shading; 1..5: the colour map of val / max_val (fixed particles grey).
__global__ void __launch_bounds__(kRtThreads) k_render(const Camera *cam, const float4 *xr, const double *val,
                                                     const float *fixvel, const float4 *rect,
                                                     const float4 *grect, const uint32_t *orig_of, unsigned np,
                                                     int method, float max_val, uchar4 *img)
{
    __shared__ float4 sx[kRtList];
    __shared__ unsigned sk[kRtList];
    __shared__ unsigned sg[kRtThreads];
    __shared__ unsigned count, groups;
    __shared__ unsigned jlo, jhi;
    const Camera C = *cam;
    const unsigned t = threadIdx.x, lane = t & 31u, wid = t >> 5;
    const unsigned tiles_x = (C.width + kRtTile - 1) / kRtTile;
    const unsigned i0 = (blockIdx.x % tiles_x) * kRtTile, r0 = (blockIdx.x / tiles_x) * kRtTile;
    const unsigned col = i0 + t % kRtTile, row = r0 + t / kRtTile;
    const bool active = col < C.width && row < C.height;
    const unsigned mempos = active ? row * C.width + col : 0u;
    // rayInitPerspective
    const unsigned i = active ? mempos % C.width : 0u;
    const unsigned j = active ? (unsigned)(int)floorf((float)mempos / C.width) % C.width : 0u;
    if (t == 0) {
        jlo = 0xffffffffu;
        jhi = 0u;
        count = 0u;
    }
    __syncthreads();
    if (active) {
        atomicMin(&jlo, j);
        atomicMax(&jhi, j);
    }
    const float p_u = C.plane[0] + (C.plane[1] - C.plane[0]) * (i + 0.5f) / C.width;
    const float p_v = C.plane[2] + (C.plane[3] - C.plane[2]) * (j + 0.5f) / C.height;
    const F3 e = C.eye;
    const F3 d = (-C.d) * C.w + p_u * C.u + p_v * C.v;
    __syncthreads();
    const float bx0 = (float)i0, bx1 = (float)(i0 + kRtTile - 1), by0 = (float)jlo, by1 = (float)jhi;
    auto reaches = [&](float4 b) { return b.x <= bx1 && b.z >= bx0 && b.y <= by1 && b.w >= by0; };
    float tdist = 1e10f, thit = 0.f;
    unsigned hit = 0xffffffffu, hito = 0xffffffffu;   // sorted position and original index
    // spheres in the list, as the block barrier counts them: the same number in
    // every thread, while `count` may already be growing with the next turn
    unsigned staged = 0;
    // the spheres in the list against this thread's pixel
    auto trace = [&]() {
        if (active)
            for (unsigned q = 0; q < staged; ++q) {
                const float4 x = sx[q];
                const F3 c = f3(x.x, x.y, x.z);
                const float R = x.w;
                const F3 ec = e - c;
                const float Delta = (2.0f * dot(d, ec)) * (2.0f * dot(d, ec)) -
                                    4.0f * dot(d, d) * (dot(ec, ec) - R * R);
                if (!(Delta > 0.0f)) continue;
                const float t_minus =
                    (dot(-d, ec) - sqrtf(dot(d, ec) * dot(d, ec) - dot(d, d) * (dot(ec, ec) - R * R))) /
                    dot(d, d);
                const float a = fabsf(t_minus);
                if (a > tdist || !(a < 1e10f)) continue;
                const unsigned k = sk[q], o = orig_of[k];
                if (a < tdist || o < hito) {
                    tdist = a;
                    thit = t_minus;
                    hit = k;
                    hito = o;
                }
            }
    };
    const unsigned ngroups = (np + 31u) / 32u;
    for (unsigned base = 0; base < ngroups; base += kRtThreads) {
        if (t == 0) groups = 0u;
        __syncthreads();
        const unsigned g = base + t;
        const bool in = g < ngroups && reaches(grect[g]);
        const unsigned found = __ballot_sync(0xffffffffu, in);
        unsigned at = 0;
        if (lane == 0 && found) at = atomicAdd(&groups, (unsigned)__popc(found));
        at = __shfl_sync(0xffffffffu, at, 0);
        if (in) sg[at + __popc(found & ((1u << lane) - 1u))] = g;
        __syncthreads();
        // a warp per group; at most kRtThreads spheres join the list per turn
        for (unsigned q0 = 0; q0 < groups; q0 += kRtThreads / 32) {
            const unsigned q = q0 + wid;
            const unsigned k = q < groups ? sg[q] * 32u + lane : np;
            const bool take = k < np && reaches(rect[k]);
            const unsigned mask = __ballot_sync(0xffffffffu, take);
            unsigned pos = 0;
            if (lane == 0 && mask) pos = atomicAdd(&count, (unsigned)__popc(mask));
            pos = __shfl_sync(0xffffffffu, pos, 0) + __popc(mask & ((1u << lane) - 1u));
            if (take) {
                sx[pos] = xr[k];
                sk[pos] = k;
            }
            staged += (unsigned)__syncthreads_count(take);
            if (staged > kRtList - kRtThreads) {
                trace();
                __syncthreads();
                staged = 0u;
                if (t == 0) count = 0u;
                __syncthreads();
            }
        }
        __syncthreads();
    }
    trace();
    if (!active) return;
    uchar4 out = make_uchar4(255, 255, 255, 255);   // imageInit: white background
    if (tdist < 1e10f) {
        const float4 x = xr[hit];
        const F3 p = e + thit * d;
        const F3 n = normalize(2.0f * (p - f3(x.x, x.y, x.z)));
        const float dotprod = fmaxf(0.0f, dot(n, C.light));
        const float I_d = 40.0f, k_d = 5.0f, k_a = 10.0f, I_a = 5.0f;
        const float shade = k_d * I_d * dotprod + k_a * I_a;
        if (method == 0) {
            out.x = (unsigned char)(shade * 0.48f);
            out.y = (unsigned char)(shade * 0.41f);
            out.z = (unsigned char)(shade * 0.27f);
        } else {
            float ratio = (float)(val[hit] / (double)max_val);
            if (ratio < 0.01f) ratio = 0.01f;
            if (ratio > 0.99f) ratio = 0.99f;
            float r = cm_red(ratio), g = cm_green(ratio), b = cm_blue(ratio);
            if (fixvel[hit] > 0.f) r = g = b = 0.5f;
            out.x = (unsigned char)(shade * r);
            out.y = (unsigned char)(shade * g);
            out.z = (unsigned char)(shade * b);
        }
    }
    img[mempos] = out;
}

}  // namespace

int Engine::render(int method, float max_val, float lower_cutoff, unsigned width, unsigned height,
                   unsigned char *rgba)
{
    if (!rgba || width == 0 || height == 0 || method < 0 || method > 5)
        return fail(ST_ARG, "render: bad arguments");
    if ((size_t)width * height > (1u << 26)) return fail(ST_ARG, "render: image too large");
    int rc = poll_errors("render");
    if (rc < 0 && rc != ST_OUTSIDE && rc != ST_CAPACITY) return rc;
    const size_t n = hs.np, pixels = (size_t)width * height, ngroups = (n + 31) / 32;
    // the engine keeps the scratch between images of one size or smaller
    size_t off = 0;
    auto carve = [&](size_t bytes) {
        const size_t at = off;
        off += (bytes + 255) & ~(size_t)255;
        return at;
    };
    const size_t o_ext = carve(3 * 8), o_cam = carve(sizeof(Camera)), o_xr = carve(n * 16),
                 o_val = carve(n * 8), o_fix = carve(n * 4), o_rect = carve(n * 16),
                 o_grect = carve(ngroups * 16), o_img = carve(pixels * 4);
    unsigned char *ws = query_scratch(off);
    if (!ws) return fail(ST_CUDA, "render: out of device memory");
    auto *ext = (unsigned long long *)(ws + o_ext);
    Camera *cam = (Camera *)(ws + o_cam);
    float4 *xr = (float4 *)(ws + o_xr), *rect = (float4 *)(ws + o_rect), *grect = (float4 *)(ws + o_grect);
    double *val = (double *)(ws + o_val);
    float *fixv = (float *)(ws + o_fix);
    uchar4 *img = (uchar4 *)(ws + o_img);
    cudaError_t e = cudaMemsetAsync(ext, 0, 3 * 8, stream);
    if (e != cudaSuccess) return cuda_fail(e, "render");
    if (n) k_render_extent<<<(unsigned)std::min<size_t>((n + 255) / 256, 592), 256, 0, stream>>>(P, S, ext);
    k_render_camera<<<1, 1, 0, stream>>>(P, ext, width, height, cam);
    if (n)
        k_render_prep<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(P, S, method, lower_cutoff, cam, xr, val,
                                                                       fixv, rect, grect);
    const size_t tiles = (size_t)((width + kRtTile - 1) / kRtTile) * ((height + kRtTile - 1) / kRtTile);
    k_render<<<(unsigned)tiles, kRtThreads, 0, stream>>>(cam, xr, val, fixv, rect, grect, S.orig_of, (unsigned)n,
                                                         method, max_val, img);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(rgba, img, pixels * 4, cudaMemcpyDeviceToHost, stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    if (e != cudaSuccess) return cuda_fail(e, "render");
    return ST_OK;
}

}  // namespace sphb
