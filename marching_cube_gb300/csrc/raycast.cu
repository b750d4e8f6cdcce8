// Ray casting of a short2 TSDF volume into depth and normal maps on sm_103a.
//
// Replaces d_voxel_extract_depth_and_normal_map and its host set-up
// (cu_kinect_fusion_v1.cu:786-986, with the trilinear sampler :551-657 and
// the surface normal :3146-3233).  One thread per pixel marches its ray as
// the reference does: entry and exit over the six faces of the volume shrunk
// by one voxel, steps of 1 voxel, backing off and stepping 0.25 inside the
// truncation band, the zero crossing placed by linear interpolation of the
// last two samples (eq. 15), a back-face crossing ends the ray.
//
// The camera set-up (K, M = K R^T, M^-1, camera centre) is computed on the
// device by one thread per CTA in the reference's binary32 operation order,
// so host compilers' contraction rules play no part in the results.  A
// singular M writes nothing, as the reference launches nothing then.
//
// Arithmetic: the reference's expressions in IEEE binary32, source order, no
// contraction (--fmad=false).
#include <cuda_runtime.h>
#include <float.h>
#include <stdint.h>

#include "mc_common.cuh"

namespace mcg {
namespace {

struct RayCamera {
    float IM[3][3];  // (K R^T)^-1, columns IM[j]
    float cc[3];     // camera centre in voxel units
    int ok;
};

struct RayParams {
    const short2 *vol;
    int nx, ny, nz;
    float grid_s;
    float fx, fy, cx, cy;
    float r[9], t[3];  // camera -> global, rotation column-major
    int w, h;
    float *depth;
    float *normal;
};

// _cu_voxel_extract_depth_and_normal_map (:965-986): K (cu_geometry_functions.h:248-255),
// matrix33_mt, float33_inv (cu_vector_functions.h:555-575), float3_div_c
__device__ void ray_camera(const RayParams &p, RayCamera &c) {
    const float K[3][3] = {{p.fx, 0.0f, 0.0f}, {0.0f, p.fy, 0.0f}, {p.cx, p.cy, 1.0f}};
    float M[3][3];
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int i = 0; i < 3; ++i)
            M[j][i] = K[0][i] * p.r[j] + K[1][i] * p.r[3 + j] + K[2][i] * p.r[6 + j];
    const float A = M[2][2] * M[1][1] - M[2][1] * M[1][2];
    const float B = M[0][2] * M[2][1] - M[0][1] * M[2][2];
    const float C = M[0][1] * M[1][2] - M[0][2] * M[1][1];
    const float det = M[0][0] * A + M[1][0] * B + M[2][0] * C;
    c.ok = !(det > -FLT_EPSILON && det < FLT_EPSILON);
    float I[3][3];
    I[0][0] = A;
    I[0][1] = B;
    I[0][2] = C;
    I[1][0] = M[1][2] * M[2][0] - M[1][0] * M[2][2];
    I[1][1] = M[0][0] * M[2][2] - M[0][2] * M[2][0];
    I[1][2] = M[0][2] * M[1][0] - M[0][0] * M[1][2];
    I[2][0] = M[1][0] * M[2][1] - M[1][1] * M[2][0];
    I[2][1] = M[0][1] * M[2][0] - M[0][0] * M[2][1];
    I[2][2] = M[0][0] * M[1][1] - M[0][1] * M[1][0];
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int i = 0; i < 3; ++i) c.IM[j][i] = I[j][i] / det;
#pragma unroll
    for (int i = 0; i < 3; ++i) c.cc[i] = p.t[i] / p.grid_s;
}

// Index of voxels: 32-bit, and coordinates below 2^22, for SMALL volumes.
template <bool SMALL>
struct RayIndex {
    using I = long long;
    static __device__ __forceinline__ int whole(float p) { return (int)p; }
};
template <>
struct RayIndex<true> {
    using I = unsigned int;
    // trunc(p) for 0 <= p < 2^22: in binade [2^23, 2^24) a float is an integer,
    // so the sum rounded down holds floor(p) in its low bits
    static __device__ __forceinline__ int whole(float p) {
        return (int)(__float_as_uint(__fadd_rd(p, 8388608.0f)) & 0x7fffffu);
    }
};

struct RayPos {
    float x, y, z;
    bool in;  // inside [0, hi) on every axis
};

__device__ __forceinline__ RayPos ray_at(const float *rd, const float *cc, const float *hi, float t) {
    RayPos q;
    q.x = rd[0] * t + cc[0];
    q.y = rd[1] * t + cc[1];
    q.z = rd[2] * t + cc[2];
    q.in = !(q.x < 0.0f || q.y < 0.0f || q.z < 0.0f || q.x >= hi[0] || q.y >= hi[1] || q.z >= hi[2]);
    return q;
}

// The tsdf of voxel *v, loaded where this stands: a plain load would be moved
// down to where its value is first tested, behind the test of the one before
// it, and the loads of a batch would run one after another.
__device__ __forceinline__ short ray_voxel(const short2 *v) {
    short t;
    asm volatile("ld.global.nc.s16 %0, [%1];" : "=h"(t) : "l"(v));
    return t;
}

__device__ __forceinline__ bool at_bound(short t) { return t == (short)kMaxTsdf || t == (short)-kMaxTsdf; }

// d_voxel_extract_trilinear_interpolated_sdf (:551-657): the corners in the
// reference's order V000, V100, V010, V001, V101, V011, V110, V111, fetched
// together; the first +-32766 among them gives +-1, else
// float_interpolation_trilinear (cu_math_functions.h:107-111)
template <bool SMALL>
__device__ __forceinline__ float trilinear_sdf(const RayParams &p, const RayPos &q) {
    using RI = RayIndex<SMALL>;
    using I = typename RI::I;
    const int ix = RI::whole(q.x), iy = RI::whole(q.y), iz = RI::whole(q.z);
    const I sy = (I)p.nx, sz = (I)p.nx * (I)p.ny;
    const I base = (I)iz * sz + (I)iy * sy + (I)ix;
    // a row's second corner by the address of its first, which the load adds
    // to (a 32-bit index of its own takes an address of its own)
    const short2 *r0 = p.vol + base, *ry = p.vol + (I)(base + sy), *rz = p.vol + (I)(base + sz),
                 *ryz = p.vol + (I)(base + sy + sz);
    const short2 *const at[8] = {r0, r0 + 1, ry, rz, rz + 1, ryz, ry + 1, ryz + 1};
    short t[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) t[k] = ray_voxel(at[k]);
    bool any = false;
#pragma unroll
    for (int k = 0; k < 8; ++k) any = any || abs((int)t[k]) == kMaxTsdf;
    if (any) {
        float bound = 0.0f;
#pragma unroll
        for (int k = 7; k >= 0; --k)
            if (at_bound(t[k])) bound = t[k] > 0 ? 1.0f : -1.0f;
        return bound;
    }
    float s[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) s[k] = mcg_unpack_tsdf(t[k]);
    const float x = q.x - (float)ix, y = q.y - (float)iy, z = q.z - (float)iz;
    const float a = 1.0f - x, b = 1.0f - y, c = 1.0f - z;
    return s[0] * a * b * c + s[1] * x * b * c + s[2] * a * y * c + s[3] * a * b * z + s[4] * x * b * z +
           s[5] * a * y * z + s[6] * x * y * c + s[7] * x * y * z;
}

// The surface normal at q (grid units, kf.cu:3146-3233): normal_global with the
// 8 samples fetched together.
__device__ __forceinline__ float3 ray_normal(const RayParams &p, float qx, float qy, float qz) {
    const int ix = (int)qx, iy = (int)qy, iz = (int)qz;
    const long long xy = (long long)p.nx * p.ny, N = xy * p.nz;
    const long long base = (long long)iz * xy + (long long)iy * p.nx + ix;
    const long long off[8] = {0, 1, 1 + (long long)p.nx, p.nx, xy, xy + 1, xy + 1 + p.nx, xy + p.nx};
    if (base < 0 || base + off[6] >= N) return make_float3(0.f, 0.f, 0.f);  // the offsets are >= 0, off[6] the largest
    short t[8];
    bool bound = false;
#pragma unroll
    for (int k = 0; k < 8; ++k) t[k] = ray_voxel(p.vol + base + off[k]);
    float s[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        bound = bound || at_bound(t[k]);
        put_slot(s, k, mcg_unpack_tsdf(t[k]));
    }
    if (bound) return make_float3(0.f, 0.f, 0.f);
    return normal_from_samples(s, qx - (float)ix, qy - (float)iy, qz - (float)iz);
}

// The march.  A sample's place does not depend on the sample before it as long
// as the step stays the same, so outside the truncation band (steps of 1),
// where nearly every first corner is at a bound and decides its sample alone,
// a ray fetches the first corners of its next RC_FAR samples together and goes
// on to the first that is not at a bound, which needs all its corners.  A
// coordinate rd t + cc is monotonic in t in binary32 too, so a batch whose
// first and last samples lie inside the volume lies inside it.  A crossing is
// only noted and worked out after the march: the rays of a warp meet theirs at
// different samples, and each would hold up the others.
//
// What bounds the launch is the longest rays' chains (600 samples outside the
// band and up to 400 inside at 512^3, 1100 cycles for one inside) and, below
// that, the instructions of a sample.  640x480 rays of a 512^3 volume: one
// sample after another, each corner waiting for the one before it, 647 us;
// this 467.  Batches of 2, 4 and 16: 480, 466 and 538 us; several lanes a ray
// 610 us and more; whole samples two and four at a time 516 and 588 us;
// prefetches a voxel ahead inside the band 516 us.  Where rays fill the chip
// the instructions are all of it: 1920x1080 rays of a 256^3 volume that is all
// band took 7.6 ms one sample after another and 8.9 with eight 32-bit corner
// indices, eight tests for which bound, and 64-bit counts of samples; 7.3 now.
constexpr int RC_FAR = 8;
constexpr int RC_BX = 8, RC_BY = 16;  // pixels per CTA: a warp's rays are 8 x 4 neighbours

template <bool SMALL>
__global__ void __launch_bounds__(RC_BX * RC_BY) raycast_kernel(RayParams p) {
    __shared__ RayCamera cam;
    if (threadIdx.x == 0 && threadIdx.y == 0) ray_camera(p, cam);
    __syncthreads();
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= p.w || y >= p.h || !cam.ok) return;
    const long long idx = (long long)y * p.w + x;
    p.depth[idx] = 0.0f;
    if (p.normal) {
        p.normal[3 * idx] = 0.0f;
        p.normal[3 * idx + 1] = 0.0f;
        p.normal[3 * idx + 2] = 0.0f;
    }
    const float margin = 1.0f;
    const float hi[3] = {(float)p.nx - margin, (float)p.ny - margin, (float)p.nz - margin};
    const float dt_max = 1.0f, dt_min = 0.25f;
    float dt = dt_max;
    bool dt_status = false;
    const float fx = (float)x, fy = (float)y;
    // float33_mv_2 (cu_vector_functions.h:623-626), then float3_unit
    float rd[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) rd[i] = cam.IM[0][i] * fx + cam.IM[1][i] * fy + cam.IM[2][i];
    {
        const float norm = sqrtf(rd[0] * rd[0] + rd[1] * rd[1] + rd[2] * rd[2]);
        if (norm > FLT_EPSILON || norm < -FLT_EPSILON) {
#pragma unroll
            for (int i = 0; i < 3; ++i) rd[i] = rd[i] / norm;
        }
    }
#pragma unroll
    for (int i = 0; i < 3; ++i)
        if (rd[i] == 0.0f) rd[i] = (float)1e-15;
    const float *cc = cam.cc;
    // entry and exit over the faces c = margin and c = c_max of each axis
    float t_min = FLT_MAX, t_max = 0.0f;
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
        const int a1 = ax == 0 ? 1 : 0, a2 = ax == 2 ? 1 : 2;
#pragma unroll
        for (int side = 0; side < 2; ++side) {
            const float t = ((side == 0 ? margin : hi[ax]) - cc[ax]) / rd[ax];
            if (t > 0.0f) {
                const float u1 = rd[a1] * t + cc[a1];
                const float u2 = rd[a2] * t + cc[a2];
                if (u1 > margin && u1 < hi[a1] && u2 > margin && u2 < hi[a2]) {
                    if (t < t_min) t_min = t;
                    if (t > t_max) t_max = t;
                }
            }
        }
    }
    if (t_min == FLT_MAX && t_max == 0.0f) return;
    if (t_min == t_max) t_min = dt * margin;
    // the reference's march cannot run longer than this; the bound only guards
    // inputs (non-finite poses) on which it would not end
    const float span = t_max - t_min;
    const int cap = span < 1.0e7f ? (int)(span * 8.0f) + 4096 : 0;
    float t1 = 0.0f, sdf1 = 1.0f;
    int steps = 0;
    float t = t_min, t2 = 0.0f;
    bool hit = false;
    // what a sample does: false ends the ray.  On return t is the sample's
    // place (or where the march backs off to), dt the next step.  A crossing
    // is only noted: the rays of a warp meet theirs at different samples, and
    // each would hold up the others while it is worked out.
    auto step = [&](float sdf) -> bool {
        if (sdf < 0.0f && sdf > -1.0f && sdf1 >= 0.0f && sdf1 < 1.0f) {
            t2 = t1 - dt * sdf1 / (sdf - sdf1);  // eq. (15)
            hit = true;
            return false;
        }
        if (sdf1 <= 0.0f && sdf1 > -1.0f && sdf >= 0.0f && sdf < 1.0f) return false;  // back face
        if (sdf > -1.0f && sdf < 1.0f) {
            if (!dt_status) {
                t -= dt;
                dt_status = true;
                dt = dt_min;
                return true;
            }
        } else if (dt_status) {
            dt_status = false;
            dt = dt_max;
        }
        t1 = t;
        sdf1 = sdf;
        return true;
    };
    bool go = t < t_max && steps < cap;
    bool batch = false;  // the first sample goes by itself: a ray that enters at the surface ends there
    while (go) {
        if (batch && !dt_status) {
            float at[RC_FAR];
            at[0] = t;
#pragma unroll
            for (int k = 1; k < RC_FAR; ++k) at[k] = at[k - 1] + dt;
            const RayPos q0 = ray_at(rd, cc, hi, t), q1 = ray_at(rd, cc, hi, at[RC_FAR - 1]);
            if (at[RC_FAR - 1] < t_max && q0.in && q1.in && steps + RC_FAR <= cap) {
                using RI = RayIndex<SMALL>;
                using I = typename RI::I;
                short first[RC_FAR];
#pragma unroll
                for (int k = 0; k < RC_FAR; ++k) {
                    const float px = rd[0] * at[k] + cc[0], py = rd[1] * at[k] + cc[1], pz = rd[2] * at[k] + cc[2];
                    const I i = ((I)RI::whole(pz) * (I)p.ny + (I)RI::whole(py)) * (I)p.nx + (I)RI::whole(px);
                    first[k] = ray_voxel(p.vol + i);
                }
                bool open = true;  // every sample so far at a bound: +-1, neither a crossing nor in the band
                int n = 0;
                t = at[RC_FAR - 1];
#pragma unroll
                for (int k = 0; k < RC_FAR; ++k) {
                    const bool bound = at_bound(first[k]);
                    if (open && !bound) t = at[k];
                    open = open && bound;
                    if (open) {
                        t1 = at[k];
                        sdf1 = first[k] > 0 ? 1.0f : -1.0f;
                        n = k + 1;
                    }
                }
                steps += n;
                if (open) {
                    t += dt;
                    go = t < t_max && steps < cap;
                    continue;
                }
            }
        }
        const RayPos q = ray_at(rd, cc, hi, t);
        if (q.in) go = step(trilinear_sdf<SMALL>(p, q));
        batch = true;
        if (go) {
            t += dt;
            ++steps;
            go = t < t_max && steps < cap;
        }
    }
    if (hit) {
        const float n0 = rd[0] * t2, n1 = rd[1] * t2, n2 = rd[2] * t2;
        const float q0 = n0 + cc[0], q1 = n1 + cc[1], q2 = n2 + cc[2];
        // float_camera_intrinsic_unproject_2 (cu_geometry_functions.h:237-240)
        const float ux = (fx - p.cx) / p.fx, uy = (fy - p.cy) / p.fy;
        p.depth[idx] = sqrtf(n0 * n0 + n1 * n1 + n2 * n2) / sqrtf(ux * ux + uy * uy + 1.0f) * p.grid_s;
        if (p.normal) {
            // the surface normal at the hit (grid units), then float33_tv: R^T n
            const float3 sn = ray_normal(p, q0, q1, q2);
#pragma unroll
            for (int i = 0; i < 3; ++i)
                p.normal[3 * idx + i] = p.r[3 * i] * sn.x + p.r[3 * i + 1] * sn.y + p.r[3 * i + 2] * sn.z;
        }
    }
}

}  // namespace
}  // namespace mcg

using namespace mcg;

extern "C" mcg_status mcg_raycast(mcg_context *ctx, const void *vol, int32_t nx, int32_t ny, int32_t nz,
                                  float grid_s, const mcg_intrinsic *k, const mcg_extrinsic *e, int32_t w, int32_t h,
                                  float *depth, float *normal, mcg_stream_t stream) {
    if (!ctx || !vol || !k || !e || !depth || nx < 2 || ny < 2 || nz < 2 || w <= 0 || h <= 0) return MCG_ERR_INVALID_ARG;
    if (!(grid_s > 0.0f)) return MCG_ERR_INVALID_ARG;
    cudaError_t err = cudaSetDevice(ctx->device);
    if (err != cudaSuccess) return mcg_cuda_fail(ctx, err);
    RayParams p;
    p.vol = static_cast<const short2 *>(vol);
    p.nx = nx;
    p.ny = ny;
    p.nz = nz;
    p.grid_s = grid_s;
    p.fx = k->fx;
    p.fy = k->fy;
    p.cx = k->cx;
    p.cy = k->cy;
    for (int i = 0; i < 9; ++i) p.r[i] = e->r[i];
    for (int i = 0; i < 3; ++i) p.t[i] = e->t[i];
    p.w = w;
    p.h = h;
    p.depth = depth;
    p.normal = normal;
    const dim3 block(RC_BX, RC_BY), grid((w + RC_BX - 1) / RC_BX, (h + RC_BY - 1) / RC_BY);
    const long long voxels = (long long)nx * ny * nz;
    const bool small = voxels < (1ll << 32) && nx < (1 << 22) && ny < (1 << 22) && nz < (1 << 22);
    if (small) raycast_kernel<true><<<grid, block, 0, (cudaStream_t)stream>>>(p);
    else raycast_kernel<false><<<grid, block, 0, (cudaStream_t)stream>>>(p);
    err = cudaGetLastError();
    return err == cudaSuccess ? MCG_OK : mcg_cuda_fail(ctx, err);
}
