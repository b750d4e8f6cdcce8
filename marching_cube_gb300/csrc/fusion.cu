// KinectFusion-side kernels on sm_103a: voxel init, depth -> metre / vertex /
// normal maps, and the projective TSDF integrate step.
//
// Replaces (cu_kinect_fusion_v1.cu, all inside the reference's `#if 0`):
//   d_voxel_initialize            (:364-379)  -> voxel_init_kernel
//   d_kinect_depth_to_meter       (:99-113)   \
//   d_img_meter_to_vertex         (:116-127)   > depth_maps_kernel (fused)
//   d_img_vertex_to_normal        (:130-151)  /
//   d_voxel_volumetric_depth_scaling (:416-425) -> depth_scale_kernel
//   d_voxel_volumetric_integration (:427-532) -> integrate_blocks_kernel, integrate_kernel
//
// The reference walks x inside each thread (one thread per (y, z) row), every
// voxel of the volume in turn.  Here a first launch lists the blocks of 8^3
// voxels that the frame can update, and a second takes the voxels of those,
// each lane 16 bytes along x with one load and store, and only when at least
// one of its voxels is updated.
//
// Arithmetic: the reference's expressions in IEEE binary32, source order, no
// contraction (--fmad=false), __float2int_rn for the pixel coordinates.
#include <cuda_runtime.h>
#include <float.h>
#include <stdint.h>

#include <algorithm>

#include "mcg_internal.h"
#include "unpack.h"

namespace mcg {
namespace {

// ---- voxel init -------------------------------------------------------------
__global__ void voxel_init_kernel(uint4 *__restrict__ v4, long long n4, unsigned int word0,
                                  unsigned int word1, int words_per_voxel) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long stride = (long long)gridDim.x * blockDim.x;
    uint4 val;
    if (words_per_voxel == 1) val = make_uint4(word0, word0, word0, word0);
    else val = make_uint4(word0, word1, word0, word1);
    for (long long k = i; k < n4; k += stride) v4[k] = val;
}

__global__ void voxel_init_tail_kernel(unsigned int *__restrict__ w, long long first_word,
                                       long long n_words, unsigned int word0, unsigned int word1,
                                       int words_per_voxel) {
    const long long i = first_word + (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_words) return;
    w[i] = (words_per_voxel == 1 || (i & 1) == 0) ? word0 : word1;
}

// ---- depth maps ---------------------------------------------------------------
struct Intr {
    float fx, fy, cx, cy;
};

// d_kinect_depth_to_meter, OpenNI branch (:105, :112): invalid -> 0
__device__ __forceinline__ float meter_of(uint16_t d, float dmin, float dmax) {
    float m = (float)d / 1000.0f;
    if (m < dmin || m > dmax) m = 0.0f;
    return m;
}

// float_camera_intrinsic_unproject_3 (cu_geometry_functions.h:237-246)
__device__ __forceinline__ float3 unproject(const Intr &k, int j, int i, float m) {
    if (m == 0.0f) return make_float3(0.f, 0.f, 0.f);
    const float px = ((float)j - k.cx) / k.fx;
    const float py = ((float)i - k.cy) / k.fy;
    return make_float3(px * m, py * m, m);
}

__device__ __forceinline__ bool vvalid(float3 v) { return !(v.x == 0.f && v.y == 0.f && v.z == 0.f); }

// float3_unit (cu_vector_functions.h:258-264)
__device__ __forceinline__ float3 unit3(float3 n) {
    const float norm = sqrtf(n.x * n.x + n.y * n.y + n.z * n.z);
    if (norm > FLT_EPSILON || norm < -FLT_EPSILON) {
        n.x = n.x / norm;
        n.y = n.y / norm;
        n.z = n.z / norm;
    }
    return n;
}

// d_img_vertex_to_normal (:130-151) for one pixel given its three vertices
__device__ __forceinline__ float3 normal_of(float3 vc, float3 vx, float3 vy) {
    if (!(vvalid(vc) && vvalid(vx) && vvalid(vy))) return make_float3(0.f, 0.f, 0.f);
    const float3 tx = make_float3(vx.x - vc.x, vx.y - vc.y, vx.z - vc.z);
    const float3 ty = make_float3(vc.x - vy.x, vc.y - vy.y, vc.z - vy.z);
    float3 n;
    n.x = tx.y * ty.z - tx.z * ty.y;
    n.y = tx.z * ty.x - tx.x * ty.z;
    n.z = tx.x * ty.y - tx.y * ty.x;
    return unit3(n);
}

// one thread per pixel; the right and lower neighbours' vertices are
// recomputed from depth instead of being exchanged
__global__ void depth_maps_kernel(Intr k, int w, int h, const uint16_t *__restrict__ depth,
                                  float dmin, float dmax, float *__restrict__ meter,
                                  float3 *__restrict__ vertex, float3 *__restrict__ normal) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= h || j >= w) return;
    const long long idx = (long long)i * w + j;
    const float m = meter_of(depth[idx], dmin, dmax);
    const float3 vc = unproject(k, j, i, m);
    if (meter) meter[idx] = m;
    if (vertex) vertex[idx] = vc;
    if (normal) {
        float3 n = make_float3(0.f, 0.f, 0.f);
        if (i < h - 1 && j < w - 1) {
            const float3 vx = unproject(k, j + 1, i, meter_of(depth[idx + 1], dmin, dmax));
            const float3 vy = unproject(k, j, i + 1, meter_of(depth[idx + w], dmin, dmax));
            n = normal_of(vc, vx, vy);
        }
        normal[idx] = n;
    }
}

__global__ void meter_to_vertex_kernel(Intr k, int w, int h, const float *__restrict__ meter,
                                       float3 *__restrict__ vertex) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= h || j >= w) return;
    const long long idx = (long long)i * w + j;
    vertex[idx] = unproject(k, j, i, meter[idx]);
}

__global__ void vertex_to_normal_kernel(int w, int h, const float3 *__restrict__ vertex,
                                        float3 *__restrict__ normal) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= h || j >= w) return;
    const long long idx = (long long)i * w + j;
    float3 n = make_float3(0.f, 0.f, 0.f);
    if (i < h - 1 && j < w - 1) n = normal_of(vertex[idx], vertex[idx + 1], vertex[idx + w]);
    normal[idx] = n;
}

// ---- integrate ------------------------------------------------------------------
// d_voxel_volumetric_depth_scaling (:416-425): z-depth -> distance along the
// ray; also, for the block culling below, the largest valid one of every tile
// of TILE_W x TILE_H pixels (0: none; a pixel is valid as the integration
// tests it, > FLT_MIN), and the block counter set to zero.  One frame per
// blockIdx.z.
constexpr int TILE_W = 16, TILE_H = 8;

__global__ void __launch_bounds__(256) depth_scale_kernel(Intr k, int w, int h, const float *__restrict__ depth,
                                                          float *__restrict__ scaled, float *__restrict__ tiles,
                                                          unsigned int *__restrict__ count) {
    __shared__ unsigned int s_max[TILE_H][2];
    depth += (long long)blockIdx.z * w * h;
    scaled += (long long)blockIdx.z * w * h;
    tiles += (long long)blockIdx.z * (2 * gridDim.x) * gridDim.y;
    const int x = blockIdx.x * 32 + threadIdx.x;
    const int y = blockIdx.y * TILE_H + threadIdx.y;
    float z = 0.0f;
    if (x < w && y < h) {
        const float px = ((float)x - k.cx) / k.fx;
        const float py = ((float)y - k.cy) / k.fy;
        const long long i = (long long)y * w + x;
        const float d = depth[i] * sqrtf(px * px + py * py + 1.0f);
        scaled[i] = d;
        if (d > FLT_MIN) z = d;
    }
    // positive floats order as their bits
    const bool left = threadIdx.x < TILE_W;
    const unsigned int zl = __reduce_max_sync(0xffffffffu, left ? __float_as_uint(z) : 0u);
    const unsigned int zr = __reduce_max_sync(0xffffffffu, left ? 0u : __float_as_uint(z));
    if (threadIdx.x < 2) s_max[threadIdx.y][threadIdx.x] = threadIdx.x ? zr : zl;
    __syncthreads();
    if (threadIdx.y == 0 && threadIdx.x < 2) {
        unsigned int m = 0;
#pragma unroll
        for (int i = 0; i < TILE_H; ++i) m = max(m, s_max[i][threadIdx.x]);
        tiles[(long long)blockIdx.y * (2 * gridDim.x) + 2 * blockIdx.x + threadIdx.x] = __uint_as_float(m);
    }
    if (blockIdx.x + blockIdx.y + blockIdx.z + threadIdx.x + threadIdx.y == 0) *count = 0;
}

struct IntegParams {
    int nx, ny, nz;
    float min_t, max_t, grid_s;
    Intr k;
    float r[9], t[3];
    int w, h;
    const float *ds;        // ray-length depth
    const float3 *normals;  // optional normal map
    const float *ray_x;     // accumulated x coordinate per voxel column
    const float *pose_dev;  // if set: r[9], t[3] read from device memory (graph replay)
    int is_dynamic;
    const float *tiles;     // largest valid ray-length depth per tile of pixels, tiles_x per tile row
    int tiles_x;
    int nbx, nby;           // blocks of IB^3 voxels per axis
    unsigned int nblocks;
    unsigned int *list;     // blocks that can hold an updated voxel, or null: all
    unsigned int *count;    // how many of them
    // several frames at once: how many (pose_dev, ds, normals and tiles hold
    // them one after another), and per listed block which of them (bits)
    int n_frames;
    unsigned int *masks;
};

constexpr int FRAMES = 32;  // frames taken at once

// pose from device memory into the block's copy of the parameters
__device__ __forceinline__ void load_pose(IntegParams &p) {
    __shared__ float pose[12];
    if (p.pose_dev) {
        if (threadIdx.x < 12) pose[threadIdx.x] = p.pose_dev[threadIdx.x];
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 9; ++i) p.r[i] = pose[i];
#pragma unroll
        for (int i = 0; i < 3; ++i) p.t[i] = pose[9 + i];
    }
}

// d_pack_tsdf / d_pack_weight / d_unpack_weight (cu_kinect_fusion_v1.h:152-171)
__device__ __forceinline__ short pack_tsdf(float f) { return (short)(int)(f * (float)kMaxTsdf); }
__device__ __forceinline__ unsigned short pack_weight(float w) {
    w = (w < kUbW) ? w / kUbW : 1.0f;
    return (unsigned short)(w * (float)kMaxW + 0.5f);
}
__device__ __forceinline__ float unpack_weight(unsigned short w) { return (float)w / (float)kMaxW * kUbW; }

// One observation of a voxel: truncated sdf, weight before the dynamic term,
// ray-length depth at the pixel, ds/dz (0 where the sdf is clamped at 1),
// the pixel's ray scale and the pixel index.
struct Obs {
    float s, w0, z, dsdz, c;
    long long pix;
};

// Per-voxel part of :442-529 up to the update.  Returns false when the voxel
// is not updated.  zat(u, v, pix, c) gives the ray-length depth at the pixel
// (and its ray scale c).
template <class ZAt>
__device__ __forceinline__ bool observe_core(const float *r, const float *t, const Intr &k, int w, int h,
                                             float min_t, float max_t, const float3 *normals, ZAt zat,
                                             float px, float py, float pz, Obs &o) {
    // float_camera_extrinsic_backward (cu_geometry_functions.h:125-129), matrix33_tv
    const float v0 = px - t[0], v1 = py - t[1], v2 = pz - t[2];
    const float q0 = r[0] * v0 + r[1] * v1 + r[2] * v2;
    const float q1 = r[3] * v0 + r[4] * v1 + r[5] * v2;
    const float q2 = r[6] * v0 + r[7] * v1 + r[8] * v2;
    if (q2 < FLT_MIN) return false;
    // float_camera_intrinsic_project_3 (cu_geometry_functions.h:232-235)
    const float uf = k.fx * (q0 / q2) + k.cx;
    const float vf = k.fy * (q1 / q2) + k.cy;
    const int u = __float2int_rn(uf), v = __float2int_rn(vf);
    if (u < 0 || v < 0 || u >= (w - 2) || v >= (h - 2)) return false;
    const long long pix = (long long)v * w + u;
    float c = 1.0f;
    const float z_val = zat(u, v, pix, c);
    if (!(z_val > FLT_MIN)) return false;
    const float qn = sqrtf(q0 * q0 + q1 * q1 + q2 * q2);
    float s = z_val - qn;
    if (!(s >= -min_t)) return false;
    float dsdz;
    if (s > 0.0f) {
        s = s / max_t;
        dsdz = 1.0f / max_t;
        if (s > 1.0f) {
            s = 1.0f;
            dsdz = 0.0f;
        }
    } else {
        s = s / min_t;
        dsdz = 1.0f / min_t;
    }
    float wgt = 1.0f;
    if (normals) {
        const float3 n = normals[pix];
        if (!vvalid(n)) return false;
        wgt = -(n.x * (q0 / qn) + n.y * (q1 / qn) + n.z * (q2 / qn));
        if (wgt < FLT_MIN) return false;
    }
    o.w0 = wgt / z_val;
    o.s = s;
    o.z = z_val;
    o.dsdz = dsdz;
    o.c = c;
    o.pix = pix;
    return true;
}

__device__ __forceinline__ bool observe(const IntegParams &p, float px, float py, float pz,
                                        float &sdf, float &weight) {
    Obs o;
    const float *ds = p.ds;
    if (!observe_core(p.r, p.t, p.k, p.w, p.h, p.min_t, p.max_t, p.normals,
                      [ds](int, int, long long pix, float &) { return ds[pix]; }, px, py, pz, o))
        return false;
    sdf = o.s;
    weight = o.w0;
    return true;
}

// :509-529 weighted running average (FP32 path)
__device__ __forceinline__ void fuse_core(int is_dynamic, float sdf, float weight, float sdf1, float w1,
                                          float &sdf2, float &w2) {
    if (is_dynamic) {
        const float d = fabsf(sdf - sdf1);
        weight = weight * (1.0f + d * d * 10.0f);
    }
    w2 = w1 + weight;
    sdf2 = (w1 * sdf1 + weight * sdf) / w2;
}

__device__ __forceinline__ void fuse(const IntegParams &p, float sdf, float weight, float sdf1,
                                     float w1, float &sdf2, float &w2) {
    fuse_core(p.is_dynamic, sdf, weight, sdf1, w1, sdf2, w2);
}

// Block culling.  A block of IB^3 voxels is an affine image of a box in the
// camera's frame (centre q, half axes e): every linear form L of its voxels is
// at most L(q) + sum |L(e_i)|, every |voxel| at least |q| less the longest half
// diagonal, and where all of it lies before the camera its pixels lie inside
// the bounds of its corners' projections.  A voxel is updated only if q_z > 0,
// its pixel (after rounding) lies in u [0, w-3], v [0, h-3], and that pixel is
// valid with |q| <= depth + min_t; so a block is left out when one of the five
// half-spaces of the view misses it, or when no valid pixel inside its bounds
// is as far as the block's near side.  Each bound is widened by what the
// binary32 error of the per-voxel arithmetic and of these tests can move it;
// the exact per-voxel tests still decide inside the blocks kept.  NaN and
// infinite intermediate values fail the comparisons and keep the block.
//
// Why blocks: at 512^3 and 640x480 about 20 M voxels lie in the view and no
// deeper than the frame, 0.7 M are updated, and about 2 M lie in the blocks
// kept.  Testing the view's voxels one by one behind a per-row interval took
// 267 us (33 M threads, two IEEE divisions for each of the 20 M); one thread
// per block here, then one warp per 128 voxels of the blocks kept (below).
// Depth maps + integration of a 640x480 frame into 512^3: 305 -> 58 us (94
// with blocks next to the camera searched, see below); one 320x240 frame into
// 256^3 float2: 72 -> 20 us.
constexpr int IB = 8;
// A volume of so few blocks takes them all: listing them costs a launch and its
// latency (64^3 and 640x480 23 us, 13 without; 128^3 20-25 and 14-18; 160^3, 8000
// blocks, 17-19 and 18-25).
constexpr long long IB_ALL = 4096;

__device__ __forceinline__ bool integ_block_kept(const IntegParams &p, const float *R, const float *t,
                                                 const float *tiles, int x0, int y0, int z0) {
    const int x1 = x0 + min(IB, p.nx - x0) - 1, y1 = y0 + min(IB, p.ny - y0) - 1, z1 = z0 + min(IB, p.nz - z0) - 1;
    const float lo[3] = {p.ray_x[x0], (float)y0 * p.grid_s, (float)z0 * p.grid_s};
    const float hi[3] = {p.ray_x[x1], (float)y1 * p.grid_s, (float)z1 * p.grid_s};
    float c[3], hf[3], mag[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        hf[i] = 0.5f * (hi[i] - lo[i]);
        mag[i] = fmaxf(fabsf(lo[i]), fabsf(hi[i])) + fabsf(t[i]);
        c[i] = 0.5f * (hi[i] + lo[i]) - t[i];
    }
    float q[3], e[3][3], sz[3];  // e[axis][component]
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        const float *r = R + 3 * j;
        q[j] = r[0] * c[0] + r[1] * c[1] + r[2] * c[2];
        sz[j] = fabsf(r[0]) * mag[0] + fabsf(r[1]) * mag[1] + fabsf(r[2]) * mag[2];
#pragma unroll
        for (int i = 0; i < 3; ++i) e[i][j] = r[i] * hf[i];
    }
    // the five half-spaces, as linear forms (a0, a1, a2): one pixel wider each
    const float ul = p.k.cx + 2.0f, uh = (float)p.w - 1.0f - p.k.cx;
    const float vl = p.k.cy + 2.0f, vh = (float)p.h - 1.0f - p.k.cy;
    const float form[5][3] = {{0.0f, 0.0f, 1.0f}, {p.k.fx, 0.0f, ul}, {-p.k.fx, 0.0f, uh}, {0.0f, p.k.fy, vl},
                              {0.0f, -p.k.fy, vh}};
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        float top = form[k][0] * q[0] + form[k][1] * q[1] + form[k][2] * q[2];
#pragma unroll
        for (int i = 0; i < 3; ++i)
            top += fabsf(form[k][0] * e[i][0] + form[k][1] * e[i][1] + form[k][2] * e[i][2]);
        const float err = 1e-5f * (fabsf(form[k][0]) * sz[0] + fabsf(form[k][1]) * sz[1] + fabsf(form[k][2]) * sz[2]);
        if (top < -(err + 1e-3f)) return false;
    }
    const float size = sz[0] + sz[1] + sz[2];
    const float near_z = q[2] - fabsf(e[0][2]) - fabsf(e[1][2]) - fabsf(e[2][2]);
    if (!(near_z > 1e-3f * size)) return true;  // at the camera's plane: no bound on the pixels
    // pixel bounds: with q_z above a thousandth of the terms' size the
    // projection is good to 1e-3 (|f| + |c| + extent) pixels on either side
    float u0 = FLT_MAX, u1 = -FLT_MAX, v0 = FLT_MAX, v1 = -FLT_MAX, half = 0.0f;
    bool finite = true;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float sx = i & 1 ? 1.0f : -1.0f, sy = i & 2 ? 1.0f : -1.0f, s2 = i & 4 ? 1.0f : -1.0f;
        float d[3];
#pragma unroll
        for (int j = 0; j < 3; ++j) d[j] = sx * e[0][j] + sy * e[1][j] + s2 * e[2][j];
        const float iz = 1.0f / (q[2] + d[2]);
        const float u = p.k.fx * (q[0] + d[0]) * iz + p.k.cx, v = p.k.fy * (q[1] + d[1]) * iz + p.k.cy;
        finite = finite && isfinite(u) && isfinite(v);
        u0 = fminf(u0, u);
        u1 = fmaxf(u1, u);
        v0 = fminf(v0, v);
        v1 = fmaxf(v1, v);
        if (i < 4) half = fmaxf(half, d[0] * d[0] + d[1] * d[1] + d[2] * d[2]);
    }
    if (!finite) return true;
    const float mu = 1.0f + 2e-3f * (fabsf(p.k.fx) + fabsf(p.k.cx) + (float)p.w);
    const float mv = 1.0f + 2e-3f * (fabsf(p.k.fy) + fabsf(p.k.cy) + (float)p.h);
    const int pu0 = (int)fmaxf(floorf(u0 - mu), 0.0f), pu1 = (int)fminf(ceilf(u1 + mu), (float)(p.w - 3));
    const int pv0 = (int)fmaxf(floorf(v0 - mv), 0.0f), pv1 = (int)fminf(ceilf(v1 + mv), (float)(p.h - 3));
    if (pu1 < pu0 || pv1 < pv0) return false;
    // a block close to the camera covers up to the whole image, and nearly
    // all of those hold updates: not searched (the one thread's search of some
    // hundred tiles was most of this launch, 27 us at 512^3)
    const int tu0 = pu0 / TILE_W, tu1 = pu1 / TILE_W, tv0 = pv0 / TILE_H, tv1 = pv1 / TILE_H;
    if ((tu1 - tu0 + 1) * (tv1 - tv0 + 1) > 64) return true;
    // TILES loads at a time, also across rows (a row's few tiles at a time, one
    // after another: 160^3 and 640x480 29 us where the view is full, 19 so)
    constexpr int TILES = 4;
    float zt = 0.0f;
    const int n = (tu1 - tu0 + 1) * (tv1 - tv0 + 1);
    int tx = tu0;
    const float *row = tiles + (long long)tv0 * p.tiles_x;
    for (int i = 0; i < n; i += TILES) {
        float z[TILES];
#pragma unroll
        for (int k = 0; k < TILES; ++k) {
            z[k] = i + k < n ? row[tx] : 0.0f;
            if (++tx > tu1) {
                tx = tu0;
                row += p.tiles_x;
            }
        }
#pragma unroll
        for (int k = 0; k < TILES; ++k) zt = fmaxf(zt, z[k]);
    }
    if (zt == 0.0f) return false;  // no valid pixel
    const float near = sqrtf(q[0] * q[0] + q[1] * q[1] + q[2] * q[2]) - sqrtf(half);
    return !(near > zt + p.min_t + 1e-5f * (size + zt + p.min_t));
}

__global__ void __launch_bounds__(256) integrate_blocks_kernel(IntegParams p) {
    load_pose(p);
    const unsigned int b = blockIdx.x * 256u + threadIdx.x;
    bool keep = false;
    if (b < p.nblocks) {
        const unsigned int row = b / (unsigned int)p.nbx;
        keep = integ_block_kept(p, p.r, p.t, p.tiles, (int)(b - row * (unsigned int)p.nbx) * IB,
                                (int)(row % (unsigned int)p.nby) * IB, (int)(row / (unsigned int)p.nby) * IB);
    }
    const unsigned int m = __ballot_sync(0xffffffffu, keep);
    if (m == 0) return;
    const int lane = threadIdx.x & 31, leader = __ffs(m) - 1;
    unsigned int at = 0;
    if (lane == leader) at = atomicAdd(p.count, (unsigned int)__popc(m));
    at = __shfl_sync(0xffffffffu, at, leader);
    if (keep) p.list[at + __popc(m & ((1u << lane) - 1u))] = b;
}

__device__ __forceinline__ short2 fused_voxel(const IntegParams &p, short2 v, float sdf, float wt) {
    float s2, w2;
    // mcg_unpack_tsdf: (float)tsdf / 32766, exact
    fuse(p, sdf, wt, mcg_unpack_tsdf(v.x), unpack_weight((unsigned short)v.y), s2, w2);
    return make_short2(pack_tsdf(s2), (short)pack_weight(w2));
}

__device__ __forceinline__ float2 fused_voxel(const IntegParams &p, float2 v, float sdf, float wt) {
    float s2, w2;
    fuse(p, sdf, wt, v.x, v.y, s2, w2);
    return make_float2(s2, w2);
}

// The voxels of the blocks kept: a warp takes 32 x 16 bytes of one block at a
// time (short2: 16 of its 64 rows, 4 voxels a lane; float2: 8 rows, 2 voxels a
// lane), so that a frame whose surface lies in a few thousand blocks still
// fills the SMs.  A lane's voxels move with one 16-byte load and store where
// the rows allow it (vec), and only when one of them is updated.
template <class T>
__global__ void __launch_bounds__(256) integrate_kernel(IntegParams p, T *__restrict__ vol, int vec) {
    constexpr int VPL = 16 / (int)sizeof(T);    // voxels per lane
    constexpr int LPR = IB / VPL;               // lanes per row
    constexpr int RPP = 32 / LPR;               // rows per pass
    constexpr int PASSES = IB * IB / RPP;       // passes per block
    load_pose(p);
    const int lane = threadIdx.x & 31;
    // (64-bit: a volume can have 2^30 blocks)
    const unsigned long long items = (unsigned long long)(p.list ? *p.count : p.nblocks) * PASSES;
    const unsigned int warps = gridDim.x * 8u;
    for (unsigned long long it = blockIdx.x * 8u + (threadIdx.x >> 5); it < items; it += warps) {
        const unsigned int b = p.list ? p.list[it / PASSES] : (unsigned int)(it / PASSES);
        const unsigned int brow = b / (unsigned int)p.nbx;
        const int r = (int)(it % PASSES) * RPP + lane / LPR;  // row of the block, y fastest
        const int x0 = (int)(b - brow * (unsigned int)p.nbx) * IB + (lane % LPR) * VPL;
        const int y = (int)(brow % (unsigned int)p.nby) * IB + r % IB;
        const int z = (int)(brow / (unsigned int)p.nby) * IB + r / IB;
        if (x0 >= p.nx || y >= p.ny || z >= p.nz) continue;
        const float py = (float)y * p.grid_s, pz = (float)z * p.grid_s;
        float sdf[VPL], wt[VPL];
        unsigned int upd = 0;
#pragma unroll
        for (int i = 0; i < VPL; ++i) {
            const int x = x0 + i;
            if (x < p.nx && observe(p, p.ray_x[x], py, pz, sdf[i], wt[i])) upd |= 1u << i;
        }
        if (!upd) continue;
        T *at = vol + ((long long)z * p.ny + y) * p.nx + x0;
        T cur[VPL];
        if (vec) {
            *reinterpret_cast<uint4 *>(cur) = *reinterpret_cast<const uint4 *>(at);
        } else {
#pragma unroll
            for (int i = 0; i < VPL; ++i)
                if (upd & (1u << i)) cur[i] = at[i];
        }
#pragma unroll
        for (int i = 0; i < VPL; ++i)
            if (upd & (1u << i)) cur[i] = fused_voxel(p, cur[i], sdf[i], wt[i]);
        if (vec) {
            *reinterpret_cast<uint4 *>(at) = *reinterpret_cast<const uint4 *>(cur);
        } else {
#pragma unroll
            for (int i = 0; i < VPL; ++i)
                if (upd & (1u << i)) at[i] = cur[i];
        }
    }
}

// Several frames in one pass over the volume: per block the frames that can
// update it, and each voxel of the blocks listed goes through those in order,
// read and written once.  Ten 320x240 frames into 256^3 float2: 222 us on the
// device in thirty launches one frame at a time, 136 in three (depths 6, block
// list 15, voxels 115: instruction issue, the voxels' projections).
__global__ void __launch_bounds__(256) integrate_blocks_frames_kernel(IntegParams p) {
    __shared__ float pose[12 * FRAMES];
    __shared__ unsigned int s_mask[32];
    if (threadIdx.x < 32) s_mask[threadIdx.x] = 0;
    for (int i = threadIdx.x; i < 12 * p.n_frames; i += 256) pose[i] = p.pose_dev[i];
    __syncthreads();
    // 32 blocks a CTA, a warp for every eighth frame
    const int lane = threadIdx.x & 31;
    const unsigned int b = blockIdx.x * 32u + lane;
    unsigned int mask = 0;
    if (b < p.nblocks) {
        const unsigned int row = b / (unsigned int)p.nbx;
        const int x0 = (int)(b - row * (unsigned int)p.nbx) * IB, y0 = (int)(row % (unsigned int)p.nby) * IB,
                  z0 = (int)(row / (unsigned int)p.nby) * IB;
        const long long ntiles = (long long)p.tiles_x * ((p.h + TILE_H - 1) / TILE_H);
        for (int f = threadIdx.x >> 5; f < p.n_frames; f += 8)
            if (integ_block_kept(p, pose + 12 * f, pose + 12 * f + 9, p.tiles + f * ntiles, x0, y0, z0)) mask |= 1u << f;
    }
    if (mask) atomicOr(&s_mask[lane], mask);
    __syncthreads();
    if (threadIdx.x >= 32) return;
    mask = s_mask[lane];
    const unsigned int m = __ballot_sync(0xffffffffu, mask != 0);
    if (m == 0) return;
    const int leader = __ffs(m) - 1;
    unsigned int at = 0;
    if (lane == leader) at = atomicAdd(p.count, (unsigned int)__popc(m));
    at = __shfl_sync(0xffffffffu, at, leader) + __popc(m & ((1u << lane) - 1u));
    if (mask) {
        p.list[at] = b;
        p.masks[at] = mask;
    }
}

template <class T>
__global__ void __launch_bounds__(256) integrate_frames_kernel(IntegParams p, T *__restrict__ vol, int vec) {
    constexpr int VPL = 16 / (int)sizeof(T), LPR = IB / VPL, RPP = 32 / LPR, PASSES = IB * IB / RPP;
    __shared__ float pose[12 * FRAMES];
    for (int i = threadIdx.x; i < 12 * p.n_frames; i += 256) pose[i] = p.pose_dev[i];
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const unsigned int items = *p.count * PASSES;
    const unsigned int warps = gridDim.x * 8u;
    const long long plane = (long long)p.w * p.h;
    for (unsigned int it = blockIdx.x * 8u + (threadIdx.x >> 5); it < items; it += warps) {
        const unsigned int b = p.list[it / PASSES];
        const unsigned int brow = b / (unsigned int)p.nbx;
        const int r = (int)(it % PASSES) * RPP + lane / LPR;
        const int x0 = (int)(b - brow * (unsigned int)p.nbx) * IB + (lane % LPR) * VPL;
        const int y = (int)(brow % (unsigned int)p.nby) * IB + r % IB;
        const int z = (int)(brow / (unsigned int)p.nby) * IB + r / IB;
        if (x0 >= p.nx || y >= p.ny || z >= p.nz) continue;
        const float py = (float)y * p.grid_s, pz = (float)z * p.grid_s;
        T *at = vol + ((long long)z * p.ny + y) * p.nx + x0;
        T cur[VPL];
        unsigned int got = 0, changed = 0;  // voxels read, updated
        for (unsigned int m = p.masks[it / PASSES]; m; m &= m - 1) {
            const int f = __ffs(m) - 1;
            const float *ds = p.ds + f * plane;
#pragma unroll
            for (int i = 0; i < VPL; ++i) {
                const int x = x0 + i;
                Obs o;
                if (x >= p.nx ||
                    !observe_core(pose + 12 * f, pose + 12 * f + 9, p.k, p.w, p.h, p.min_t, p.max_t,
                                  p.normals ? p.normals + f * plane : nullptr,
                                  [ds](int, int, long long pix, float &) { return ds[pix]; }, p.ray_x[x], py, pz, o))
                    continue;
                if (vec && !got) {
                    *reinterpret_cast<uint4 *>(cur) = *reinterpret_cast<const uint4 *>(at);
                    got = ~0u;
                } else if (!(got & (1u << i))) {
                    cur[i] = at[i];
                    got |= 1u << i;
                }
                cur[i] = fused_voxel(p, cur[i], o.s, o.w0);
                changed |= 1u << i;
            }
        }
        if (!changed) continue;
        if (vec) {
            *reinterpret_cast<uint4 *>(at) = *reinterpret_cast<const uint4 *>(cur);
        } else {
#pragma unroll
            for (int i = 0; i < VPL; ++i)
                if (changed & (1u << i)) at[i] = cur[i];
        }
    }
}

// ---- integrate adjoint ----------------------------------------------------------
// Reverse of a sequence of float2 integrate steps (no counterpart in the
// reference).  Per voxel, step k (observation s, weight w) maps
//   W' = W + w,  F' = (W F + w s) / W'
// so, holding the discrete choices (pixel, truncation, clamp) fixed,
//   dF'/dF = W/W',  dF'/dW = (F - F')/W',  dF'/ds = w/W',  dF'/dw = (s - F')/W'
// and s = (c d - |q|)/m (m = max_t or min_t, ds/dz = 0 where clamped),
// w = wgt / (c d) (dw/dd = -w c / z) with d the pixel's z-depth and c its
// ray scale.  The dynamic term multiplies w by 1 + 10 (s - F)^2.  Normal maps
// are held constant.
constexpr int BW_SEG = 16;                    // frames whose (F, W) one thread keeps while reversing
constexpr int BW_MAX_FRAMES = BW_SEG * 32;    // frames per call (checkpoint every BW_SEG)

struct IntegBwParams {
    int nx, ny, nz;
    float min_t, max_t, grid_s;
    Intr k;
    int w, h, n_frames;
    const float *poses;    // n_frames x (r[9] column-major, t[3])
    const float *depth;    // n_frames x h x w metres (z-depth)
    const float3 *normals; // n_frames x h x w, or null
    const float *ray_x;
    int is_dynamic;
    const float2 *vol0;    // volume before the first frame, or null: (-1, 0)
    const float *grad_f;   // dL/dF after the last frame, voxel i's at i * grad_step
    const float *grad_w;   // dL/dW after the last frame, or null: 0
    int grad_step;
    float *grad_depth;     // n_frames x h x w, accumulated
    float *grad_f0;        // dL/dF before the first frame, or null
    float *grad_w0;
};

__device__ __forceinline__ bool bw_observe(const IntegBwParams &p, const float *pose, int f, float px,
                                           float py, float pz, Obs &o) {
    const long long plane = (long long)p.w * p.h;
    const float *dep = p.depth + f * plane;
    const Intr k = p.k;
    return observe_core(pose, pose + 9, k, p.w, p.h, p.min_t, p.max_t, p.normals ? p.normals + f * plane : nullptr,
                        [dep, k](int u, int v, long long pix, float &c) {
                            // d_voxel_volumetric_depth_scaling (:416-425) for one pixel
                            const float cx = ((float)u - k.cx) / k.fx;
                            const float cy = ((float)v - k.cy) / k.fy;
                            c = sqrtf(cx * cx + cy * cy + 1.0f);
                            return dep[pix] * c;
                        },
                        px, py, pz, o);
}

// One voxel with a gradient: dL/dF, dL/dW of the volume before the first frame
// in gF, gW on return.
__device__ __forceinline__ void backward_voxel(const IntegBwParams &p, const float *s_pose, long long i, float &gF,
                                               float &gW) {
    const int nseg = (p.n_frames + BW_SEG - 1) / BW_SEG;
    const int x = (int)(i % p.nx);
    const long long row = i / p.nx;
    const int y = (int)(row % p.ny), z = (int)(row / p.ny);
    const float px = p.ray_x[x], py = (float)y * p.grid_s, pz = (float)z * p.grid_s;
    float F = p.vol0 ? p.vol0[i].x : -1.0f;
    float W = p.vol0 ? p.vol0[i].y : 0.0f;
    // forward sweep: (F, W) at the start of every segment
    float ckF[BW_MAX_FRAMES / BW_SEG], ckW[BW_MAX_FRAMES / BW_SEG];
    ckF[0] = F;
    ckW[0] = W;
    for (int f = 0; f < (nseg - 1) * BW_SEG; ++f) {
        Obs o;
        if (bw_observe(p, s_pose + 12 * f, f, px, py, pz, o)) fuse_core(p.is_dynamic, o.s, o.w0, F, W, F, W);
        if ((f + 1) % BW_SEG == 0) {
            ckF[(f + 1) / BW_SEG] = F;
            ckW[(f + 1) / BW_SEG] = W;
        }
    }
    for (int sg = nseg - 1; sg >= 0; --sg) {
        const int f0 = sg * BW_SEG;
        const int f1 = min(p.n_frames, f0 + BW_SEG);
        // the segment forward, its observations and (F, W) before each kept
        float sF[BW_SEG], sW[BW_SEG];
        Obs ob[BW_SEG];
        int seen = 0;
        float cF = ckF[sg], cW = ckW[sg];
        for (int f = f0; f < f1; ++f) {
            Obs o;
            if (!bw_observe(p, s_pose + 12 * f, f, px, py, pz, o)) continue;
            o.pix += f * ((long long)p.w * p.h);
            sF[seen] = cF;
            sW[seen] = cW;
            ob[seen++] = o;
            fuse_core(p.is_dynamic, o.s, o.w0, cF, cW, cF, cW);
        }
        // (a warp's lanes at the same place of their arrays, which are interleaved
        // lane by lane)
        for (int k = f1 - f0 - 1; k >= 0; --k) {
            if (k >= seen) continue;
            const Obs o = ob[k];
            const float Fp = sF[k], Wp = sW[k];
            float wv = o.w0, mult = 1.0f, d = 0.0f;
            if (p.is_dynamic) {
                d = o.s - Fp;
                mult = 1.0f + d * d * 10.0f;
                wv = wv * mult;
            }
            const float Wn = Wp + wv;
            const float Fn = (Wp * Fp + wv * o.s) / Wn;
            float gs = gF * wv / Wn;
            const float gw = gF * (o.s - Fn) / Wn + gW;
            float gFp = gF * Wp / Wn;
            const float gWp = gF * (Fp - Fn) / Wn + gW;
            float gw0 = gw;
            if (p.is_dynamic) {
                const float t = gw * o.w0 * 20.0f * d;
                gs += t;
                gFp -= t;
                gw0 = gw * mult;
            }
            const float gz = gs * o.dsdz - gw0 * o.w0 / o.z;
            atomicAdd(p.grad_depth + o.pix, gz * o.c);
            gF = gFp;
            gW = gWp;
        }
    }
}

// Few voxels have a gradient (the band around the surface that the mesh
// touches), spread thinly over the volume's rows: a CTA collects those of
// ROUNDS voxels a thread at a time and works them out BW_THREADS together.
// Bound: the work on those voxels (an observation is two divisions and a
// gather).  256^3 and ten 320x240 frames, gradients at the mesh's voxels: one
// thread a voxel and three observations a frame 526 us, this 83; at every voxel
// 3.1 and 1.6 ms.  With observations kept by frame and each lane going back over
// its own these took 94 us and 2.8 ms, and 128^3 with 40 frames 7.5 ms where one
// thread a voxel takes 1.7 and this 1.3; with all lanes on the same frame 97 us
// and 1.7 ms.  Four rounds where they leave a CTA for every place, else one: 64^3
// with 40 frames 379 us with four, 199 with one (240 with a thread a voxel); 256^3
// at the mesh's voxels 96 and 126.
constexpr int BW_THREADS = 128;

template <int ROUNDS>
__global__ void __launch_bounds__(BW_THREADS) integrate_backward_kernel(IntegBwParams p) {
    constexpr int BW_SCAN = ROUNDS * BW_THREADS;
    extern __shared__ float s_pose[];
    __shared__ long long s_at[BW_THREADS + BW_SCAN];
    __shared__ float2 s_g[BW_THREADS + BW_SCAN];
    __shared__ int s_n;
    const int tid = threadIdx.x, lane = tid & 31;
    for (int i = tid; i < p.n_frames * 12; i += BW_THREADS) s_pose[i] = p.poses[i];
    if (tid == 0) s_n = 0;
    __syncthreads();
    const long long n = (long long)p.nx * p.ny * p.nz;
    auto work = [&](int k) {
        const long long i = s_at[k];
        float gF = s_g[k].x, gW = s_g[k].y;
        backward_voxel(p, s_pose, i, gF, gW);
        if (p.grad_f0) p.grad_f0[i] = gF;
        if (p.grad_w0) p.grad_w0[i] = gW;
    };
    for (long long base = (long long)blockIdx.x * BW_SCAN; base < n; base += (long long)gridDim.x * BW_SCAN) {
        float gF[ROUNDS], gW[ROUNDS];
#pragma unroll
        for (int k = 0; k < ROUNDS; ++k) {
            const long long i = base + k * BW_THREADS + tid;
            gF[k] = i < n ? p.grad_f[i * p.grad_step] : 0.0f;
            gW[k] = i < n && p.grad_w ? p.grad_w[i * p.grad_step] : 0.0f;
        }
#pragma unroll
        for (int k = 0; k < ROUNDS; ++k) {
            const long long i = base + k * BW_THREADS + tid;
            const bool has = gF[k] != 0.0f || gW[k] != 0.0f;
            const unsigned int m = __ballot_sync(0xffffffffu, has);
            if (m) {
                int at = 0;
                if (lane == 0) at = atomicAdd(&s_n, __popc(m));
                at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & ((1u << lane) - 1u));
                if (has) {
                    s_at[at] = i;
                    s_g[at] = make_float2(gF[k], gW[k]);
                }
            }
            if (!has && i < n) {
                if (p.grad_f0) p.grad_f0[i] = gF[k];
                if (p.grad_w0) p.grad_w0[i] = gW[k];
            }
        }
        __syncthreads();
        int left = s_n;
        while (left >= BW_THREADS) {  // uniform
            left -= BW_THREADS;
            work(left + tid);
        }
        __syncthreads();
        if (tid == 0) s_n = left;
        __syncthreads();
    }
    if (tid < s_n) work(tid);
}

long long blocks_of(int n) { return ((long long)n + IB - 1) / IB; }

Intr intr_of(const mcg_intrinsic *k) { return Intr{k->fx, k->fy, k->cx, k->cy}; }

// Room for the depth tiles of any image of so many pixels (one column of
// pixels has most: two tiles for eight), so that a stream capture needs an
// earlier call of as many pixels only, as for the depths themselves.
size_t tile_room(long long pixels) { return (size_t)(pixels / 4 + 2); }

// ensure() for integrate's scratch: what a captured graph may refer to is not freed
template <class T>
bool ensure_integ(mcg_context *ctx, T **ptr, size_t *cap, size_t n) {
    if (*cap < n && *ptr && ctx->integ_captured) {
        ctx->integ_old.push_back(*ptr);
        *ptr = nullptr;
    }
    return ensure(ptr, cap, n);
}

}  // namespace
}  // namespace mcg

using namespace mcg;

extern "C" {

mcg_status mcg_voxel_init(mcg_context *ctx, void *vol, int32_t voxel_type, int64_t n_voxels,
                          mcg_stream_t stream) {
    if (!ctx || (n_voxels > 0 && !vol) || n_voxels < 0) return MCG_ERR_INVALID_ARG;
    if (voxel_type != MCG_VOXEL_SHORT2 && voxel_type != MCG_VOXEL_FLOAT2) return MCG_ERR_INVALID_ARG;
    if (n_voxels == 0) return MCG_OK;
    cudaError_t e = cudaSetDevice(ctx->device);
    if (e != cudaSuccess) return mcg_cuda_fail(ctx, e);
    cudaStream_t s = (cudaStream_t)stream;
    unsigned int w0, w1;
    int wpv;
    if (voxel_type == MCG_VOXEL_SHORT2) {
        // {tsdf = -32766, w = 0}
        w0 = (unsigned int)(unsigned short)(short)(-kMaxTsdf);
        w1 = 0;
        wpv = 1;
    } else {
        const float m1 = -1.0f;
        w0 = *reinterpret_cast<const unsigned int *>(&m1);
        w1 = 0;
        wpv = 2;
    }
    const long long n_words = (long long)n_voxels * wpv;
    long long n4 = 0;
    if (((uintptr_t)vol & 15) == 0) n4 = n_words / 4;
    if (n4 > 0) {
        long long grid = (n4 + 255) / 256;
        const long long cap = (long long)ctx->num_sms * 16;
        if (grid > cap) grid = cap;
        voxel_init_kernel<<<(int)grid, 256, 0, s>>>((uint4 *)vol, n4, w0, w1, wpv);
    }
    const long long first = n4 * 4;
    if (first < n_words) {
        const long long rem = n_words - first;
        voxel_init_tail_kernel<<<(unsigned int)((rem + 255) / 256), 256, 0, s>>>(
            (unsigned int *)vol, first, n_words, w0, w1, wpv);
    }
    e = cudaGetLastError();
    return e == cudaSuccess ? MCG_OK : mcg_cuda_fail(ctx, e);
}

mcg_status mcg_depth_to_maps(mcg_context *ctx, const mcg_intrinsic *k, int32_t w, int32_t h,
                             const uint16_t *depth_mm, float depth_min, float depth_max,
                             float *meter, float *vertex, float *normal, mcg_stream_t stream) {
    if (!ctx || !k || !depth_mm || w <= 0 || h <= 0) return MCG_ERR_INVALID_ARG;
    if (!meter && !vertex && !normal) return MCG_OK;
    cudaError_t e = cudaSetDevice(ctx->device);
    if (e != cudaSuccess) return mcg_cuda_fail(ctx, e);
    const dim3 block(32, 8), grid((w + 31) / 32, (h + 7) / 8);
    depth_maps_kernel<<<grid, block, 0, (cudaStream_t)stream>>>(intr_of(k), w, h, depth_mm, depth_min,
                                                                depth_max, meter, (float3 *)vertex,
                                                                (float3 *)normal);
    e = cudaGetLastError();
    return e == cudaSuccess ? MCG_OK : mcg_cuda_fail(ctx, e);
}

mcg_status mcg_meter_to_vertex(mcg_context *ctx, const mcg_intrinsic *k, int32_t w, int32_t h,
                               const float *meter, float *vertex, mcg_stream_t stream) {
    if (!ctx || !k || !meter || !vertex || w <= 0 || h <= 0) return MCG_ERR_INVALID_ARG;
    cudaError_t e = cudaSetDevice(ctx->device);
    if (e != cudaSuccess) return mcg_cuda_fail(ctx, e);
    const dim3 block(32, 8), grid((w + 31) / 32, (h + 7) / 8);
    meter_to_vertex_kernel<<<grid, block, 0, (cudaStream_t)stream>>>(intr_of(k), w, h, meter, (float3 *)vertex);
    e = cudaGetLastError();
    return e == cudaSuccess ? MCG_OK : mcg_cuda_fail(ctx, e);
}

mcg_status mcg_vertex_to_normal(mcg_context *ctx, int32_t w, int32_t h, const float *vertex,
                                float *normal, mcg_stream_t stream) {
    if (!ctx || !vertex || !normal || w <= 0 || h <= 0) return MCG_ERR_INVALID_ARG;
    cudaError_t e = cudaSetDevice(ctx->device);
    if (e != cudaSuccess) return mcg_cuda_fail(ctx, e);
    const dim3 block(32, 8), grid((w + 31) / 32, (h + 7) / 8);
    vertex_to_normal_kernel<<<grid, block, 0, (cudaStream_t)stream>>>(w, h, (const float3 *)vertex, (float3 *)normal);
    e = cudaGetLastError();
    return e == cudaSuccess ? MCG_OK : mcg_cuda_fail(ctx, e);
}

// x coordinate table, accumulated exactly as :434/:444 do
// x coordinate of voxel column x as kf.cu:434-444 accumulates it: p.x starts
// at 0 and grows by grid_s per voxel, in FP32, one addition after another
__global__ void ray_x_kernel(float *__restrict__ out, int nx, float g) {
    float px = -g;
    for (int x = 0; x < nx; ++x) {
        px = __fadd_rn(px, g);
        out[x] = px;
    }
}

// the context's table for (nx, grid_s), built by one thread on stream s the
// first time (and waited for); inside a stream capture a missing table is MCG_ERR_STATE (an
// earlier call with this volume shape outside the capture builds it)
static mcg_status ray_x_table(mcg_context *ctx, int32_t nx, float grid_s, cudaStream_t s, const float **out) {
    for (const auto &r : ctx->ray_x)
        if (r.nx == nx && __builtin_memcmp(&r.g, &grid_s, sizeof(float)) == 0) {
            *out = r.d;
            return MCG_OK;
        }
    if (mcg_capturing(s)) return MCG_ERR_STATE;
    float *d = nullptr;
    if (cudaMalloc((void **)&d, sizeof(float) * (size_t)nx) != cudaSuccess)
        return mcg_cuda_fail(ctx, cudaErrorMemoryAllocation);
    ray_x_kernel<<<1, 1, 0, s>>>(d, nx, grid_s);
    // once per shape: complete before a call on another stream can use it
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
        cudaFree(d);
        return mcg_cuda_fail(ctx, e);
    }
    ctx->ray_x.push_back({nx, grid_s, d});
    *out = d;
    return MCG_OK;
}

static mcg_status integrate_impl(mcg_context *ctx, void *vol, int32_t voxel_type, int32_t nx, int32_t ny,
                                 int32_t nz, float min_t, float max_t, float grid_s, const mcg_intrinsic *k,
                                 const mcg_extrinsic *ext, const float *pose_dev, int32_t w, int32_t h,
                                 const float *depth_m, const float *normals, int32_t is_dynamic,
                                 mcg_stream_t stream) {
    if (!ctx || !vol || !k || (!ext && !pose_dev) || !depth_m || nx <= 0 || ny <= 0 || nz <= 0 || w <= 0 || h <= 0)
        return MCG_ERR_INVALID_ARG;
    if (voxel_type != MCG_VOXEL_SHORT2 && voxel_type != MCG_VOXEL_FLOAT2) return MCG_ERR_INVALID_ARG;
    if (!(min_t > 0.0f) || !(max_t > 0.0f) || !(grid_s > 0.0f)) return MCG_ERR_INVALID_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    cudaError_t e = cudaSetDevice(ctx->device);
    if (e != cudaSuccess) return mcg_cuda_fail(ctx, e);
    const long long nbx = blocks_of(nx), nby = blocks_of(ny), nbz = blocks_of(nz);
    const long long nblocks = nbx * nby * nbz;
    if (nblocks > (long long)UINT32_MAX) return MCG_ERR_TOO_LARGE;  // (a terabyte of voxels at least)
    const dim3 b2(32, TILE_H), g2((w + 31) / 32, (h + TILE_H - 1) / TILE_H);
    const size_t ntiles = tile_room((long long)w * h);
    // inside a stream capture nothing may be allocated: an earlier call of
    // the same shapes outside the capture has sized every buffer
    if (mcg_capturing(s)) {
        if (ctx->depth_scaled_cap < (size_t)w * h || ctx->integ_blocks_cap < (size_t)nblocks ||
            ctx->integ_tiles_cap < ntiles || ctx->integ_count_cap < 1)
            return MCG_ERR_STATE;
        ctx->integ_captured = true;
    }
    if (!ensure_integ(ctx, &ctx->depth_scaled, &ctx->depth_scaled_cap, (size_t)w * h))
        return mcg_cuda_fail(ctx, cudaErrorMemoryAllocation);
    const float *ray_x = nullptr;
    {
        const mcg_status st = ray_x_table(ctx, nx, grid_s, s, &ray_x);
        if (st != MCG_OK) return st;
    }
    IntegParams p = {};
    p.nx = nx; p.ny = ny; p.nz = nz;
    p.min_t = min_t; p.max_t = max_t; p.grid_s = grid_s;
    p.k = intr_of(k);
    for (int i = 0; i < 9; ++i) p.r[i] = ext ? ext->r[i] : 0.0f;
    for (int i = 0; i < 3; ++i) p.t[i] = ext ? ext->t[i] : 0.0f;
    p.pose_dev = ext ? nullptr : pose_dev;
    p.w = w; p.h = h;
    p.ds = ctx->depth_scaled;
    p.normals = (const float3 *)normals;
    p.ray_x = ray_x;
    p.is_dynamic = is_dynamic ? 1 : 0;
    if (!ensure_integ(ctx, &ctx->integ_blocks, &ctx->integ_blocks_cap, (size_t)nblocks) ||
        !ensure_integ(ctx, &ctx->integ_tiles, &ctx->integ_tiles_cap, ntiles) ||
        !ensure(&ctx->integ_count, &ctx->integ_count_cap, (size_t)1))
        return mcg_cuda_fail(ctx, cudaErrorMemoryAllocation);
    p.tiles = ctx->integ_tiles;
    p.tiles_x = 2 * (int)g2.x;
    p.nbx = (int)nbx;
    p.nby = (int)nby;
    p.nblocks = (unsigned int)nblocks;
    p.list = ctx->integ_blocks;
    p.count = ctx->integ_count;
    depth_scale_kernel<<<g2, b2, 0, s>>>(p.k, w, h, depth_m, ctx->depth_scaled, ctx->integ_tiles, ctx->integ_count);
    if (nblocks > IB_ALL) integrate_blocks_kernel<<<(unsigned int)((nblocks + 255) / 256), 256, 0, s>>>(p);
    else p.list = nullptr;
    // one warp per item; the grid holds what the SMs can and strides over more
    const long long most = (long long)ctx->num_sms * 8;
    if (voxel_type == MCG_VOXEL_SHORT2) {
        const int vec = (nx % 4 == 0) && (((uintptr_t)vol & 15) == 0);
        const unsigned int grid = (unsigned int)std::min(most, (nblocks * 4 + 7) / 8);
        integrate_kernel<short2><<<grid, 256, 0, s>>>(p, (short2 *)vol, vec);
    } else {
        const int vec = (nx % 2 == 0) && (((uintptr_t)vol & 15) == 0);
        const unsigned int grid = (unsigned int)std::min(most, nblocks);
        integrate_kernel<float2><<<grid, 256, 0, s>>>(p, (float2 *)vol, vec);
    }
    e = cudaGetLastError();
    return e == cudaSuccess ? MCG_OK : mcg_cuda_fail(ctx, e);
}

// n_frames frames of at most FRAMES in one pass; the caller has checked the
// arguments and the scratch
static mcg_status integrate_pass(mcg_context *ctx, void *vol, int32_t voxel_type, int32_t nx, int32_t ny, int32_t nz,
                                 float min_t, float max_t, float grid_s, const mcg_intrinsic *k, int n_frames,
                                 const float *poses_dev, int32_t w, int32_t h, const float *depth_m,
                                 const float *normals, int32_t is_dynamic, const float *ray_x, cudaStream_t s) {
    const dim3 b2(32, TILE_H), g2((w + 31) / 32, (h + TILE_H - 1) / TILE_H, n_frames);
    IntegParams p = {};
    p.nx = nx; p.ny = ny; p.nz = nz;
    p.min_t = min_t; p.max_t = max_t; p.grid_s = grid_s;
    p.k = intr_of(k);
    p.pose_dev = poses_dev;
    p.w = w; p.h = h;
    p.ds = ctx->depth_scaled;
    p.normals = (const float3 *)normals;
    p.ray_x = ray_x;
    p.is_dynamic = is_dynamic ? 1 : 0;
    p.tiles = ctx->integ_tiles;
    p.tiles_x = 2 * (int)g2.x;
    p.nbx = (int)blocks_of(nx);
    p.nby = (int)blocks_of(ny);
    const long long nblocks = p.nbx * (p.nby * blocks_of(nz));
    p.nblocks = (unsigned int)nblocks;
    p.list = ctx->integ_blocks;
    p.count = ctx->integ_count;
    p.n_frames = n_frames;
    p.masks = ctx->integ_masks;
    depth_scale_kernel<<<g2, b2, 0, s>>>(p.k, w, h, depth_m, ctx->depth_scaled, ctx->integ_tiles, ctx->integ_count);
    integrate_blocks_frames_kernel<<<(unsigned int)((nblocks + 31) / 32), 256, 0, s>>>(p);
    const long long most = (long long)ctx->num_sms * 8;
    if (voxel_type == MCG_VOXEL_SHORT2) {
        const int vec = (nx % 4 == 0) && (((uintptr_t)vol & 15) == 0);
        integrate_frames_kernel<short2>
            <<<(unsigned int)std::min(most, (nblocks * 4 + 7) / 8), 256, 0, s>>>(p, (short2 *)vol, vec);
    } else {
        const int vec = (nx % 2 == 0) && (((uintptr_t)vol & 15) == 0);
        integrate_frames_kernel<float2><<<(unsigned int)std::min(most, nblocks), 256, 0, s>>>(p, (float2 *)vol, vec);
    }
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? MCG_OK : mcg_cuda_fail(ctx, e);
}

mcg_status mcg_integrate_frames(mcg_context *ctx, void *vol, int32_t voxel_type, int32_t nx, int32_t ny, int32_t nz,
                                float min_t, float max_t, float grid_s, const mcg_intrinsic *k, int32_t n_frames,
                                const float *poses_dev, int32_t w, int32_t h, const float *depth_m,
                                const float *normals, int32_t is_dynamic, mcg_stream_t stream) {
    if (!ctx || !vol || !k || n_frames < 0 || (n_frames > 0 && (!poses_dev || !depth_m)) || nx <= 0 || ny <= 0 ||
        nz <= 0 || w <= 0 || h <= 0)
        return MCG_ERR_INVALID_ARG;
    if (voxel_type != MCG_VOXEL_SHORT2 && voxel_type != MCG_VOXEL_FLOAT2) return MCG_ERR_INVALID_ARG;
    if (!(min_t > 0.0f) || !(max_t > 0.0f) || !(grid_s > 0.0f)) return MCG_ERR_INVALID_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    const long long pixels = (long long)w * h;
    const size_t nblocks = (size_t)(blocks_of(nx) * blocks_of(ny) * blocks_of(nz));
    const size_t ntiles = tile_room(pixels);
    // frames a pass: 256 MB of ray-length depth at most
    const int most = (int)std::min<long long>({n_frames, FRAMES, std::max(1ll, (64ll << 20) / pixels)});
    // One frame, or scratch that cannot be had (no memory; inside a stream
    // capture, not sized by an earlier call of the same shapes): frame by frame.
    bool together = most > 1 && nblocks <= (size_t)(UINT32_MAX / 16);
    const cudaError_t e = cudaSetDevice(ctx->device);
    if (e != cudaSuccess) return mcg_cuda_fail(ctx, e);
    if (together && mcg_capturing(s)) {
        together = ctx->depth_scaled_cap >= (size_t)pixels * most && ctx->integ_tiles_cap >= ntiles * most &&
                   ctx->integ_blocks_cap >= nblocks && ctx->integ_masks_cap >= nblocks && ctx->integ_count_cap >= 1;
        ctx->integ_captured = ctx->integ_captured || together;
    } else if (together) {
        together = ensure_integ(ctx, &ctx->depth_scaled, &ctx->depth_scaled_cap, (size_t)pixels * most) &&
                   ensure_integ(ctx, &ctx->integ_tiles, &ctx->integ_tiles_cap, ntiles * most) &&
                   ensure_integ(ctx, &ctx->integ_blocks, &ctx->integ_blocks_cap, nblocks) &&
                   ensure_integ(ctx, &ctx->integ_masks, &ctx->integ_masks_cap, nblocks) &&
                   ensure(&ctx->integ_count, &ctx->integ_count_cap, (size_t)1);
        if (!together) cudaGetLastError();
    }
    for (int f = 0; f < n_frames;) {
        const float *d = depth_m + f * pixels, *n = normals ? normals + 3 * f * pixels : nullptr;
        const int nf = together ? std::min(n_frames - f, most) : 1;
        mcg_status st;
        if (nf > 1) {
            const float *ray_x = nullptr;
            st = ray_x_table(ctx, nx, grid_s, s, &ray_x);
            if (st == MCG_OK)
                st = integrate_pass(ctx, vol, voxel_type, nx, ny, nz, min_t, max_t, grid_s, k, nf, poses_dev + 12 * f, w,
                                    h, d, n, is_dynamic, ray_x, s);
        } else {
            st = integrate_impl(ctx, vol, voxel_type, nx, ny, nz, min_t, max_t, grid_s, k, nullptr, poses_dev + 12 * f,
                                w, h, d, n, is_dynamic, stream);
        }
        if (st != MCG_OK) return st;
        f += nf;
    }
    return MCG_OK;
}

mcg_status mcg_integrate(mcg_context *ctx, void *vol, int32_t voxel_type, int32_t nx, int32_t ny,
                         int32_t nz, float min_t, float max_t, float grid_s,
                         const mcg_intrinsic *k, const mcg_extrinsic *ext, int32_t w, int32_t h,
                         const float *depth_m, const float *normals, int32_t is_dynamic,
                         mcg_stream_t stream) {
    if (!ext) return MCG_ERR_INVALID_ARG;
    return integrate_impl(ctx, vol, voxel_type, nx, ny, nz, min_t, max_t, grid_s, k, ext, nullptr, w, h, depth_m,
                          normals, is_dynamic, stream);
}

mcg_status mcg_integrate_device_pose(mcg_context *ctx, void *vol, int32_t voxel_type, int32_t nx, int32_t ny,
                                     int32_t nz, float min_t, float max_t, float grid_s, const mcg_intrinsic *k,
                                     const float *pose_dev, int32_t w, int32_t h, const float *depth_m,
                                     const float *normals, int32_t is_dynamic, mcg_stream_t stream) {
    if (!pose_dev) return MCG_ERR_INVALID_ARG;
    return integrate_impl(ctx, vol, voxel_type, nx, ny, nz, min_t, max_t, grid_s, k, nullptr, pose_dev, w, h,
                          depth_m, normals, is_dynamic, stream);
}


static mcg_status integrate_backward_impl(mcg_context *ctx, const void *vol0, int32_t nx, int32_t ny, int32_t nz,
                                          float min_t, float max_t, float grid_s, const mcg_intrinsic *k,
                                          int32_t n_frames, const float *poses_dev, int32_t w, int32_t h,
                                          const float *depth_m, const float *normals, int32_t is_dynamic,
                                          const float *grad_f, const float *grad_w, int grad_step, float *grad_depth,
                                          float *grad_f0, float *grad_w0, mcg_stream_t stream) {
    if (!ctx || !k || !poses_dev || !depth_m || !grad_f || !grad_depth || nx <= 0 || ny <= 0 || nz <= 0 ||
        w <= 0 || h <= 0 || n_frames <= 0)
        return MCG_ERR_INVALID_ARG;
    if (!(min_t > 0.0f) || !(max_t > 0.0f) || !(grid_s > 0.0f)) return MCG_ERR_INVALID_ARG;
    if (n_frames > BW_MAX_FRAMES) return MCG_ERR_TOO_LARGE;
    cudaStream_t s = (cudaStream_t)stream;
    cudaError_t e = cudaSetDevice(ctx->device);
    if (e != cudaSuccess) return mcg_cuda_fail(ctx, e);
    const float *ray_x = nullptr;
    const mcg_status st = ray_x_table(ctx, nx, grid_s, s, &ray_x);
    if (st != MCG_OK) return st;
    IntegBwParams p;
    p.nx = nx; p.ny = ny; p.nz = nz;
    p.min_t = min_t; p.max_t = max_t; p.grid_s = grid_s;
    p.k = intr_of(k);
    p.w = w; p.h = h; p.n_frames = n_frames;
    p.poses = poses_dev;
    p.depth = depth_m;
    p.normals = (const float3 *)normals;
    p.ray_x = ray_x;
    p.is_dynamic = is_dynamic ? 1 : 0;
    p.vol0 = (const float2 *)vol0;
    p.grad_f = grad_f;
    p.grad_w = grad_w;
    p.grad_step = grad_step;
    p.grad_depth = grad_depth;
    p.grad_f0 = grad_f0;
    p.grad_w0 = grad_w0;
    const long long n = (long long)nx * ny * nz;
    const long long most = (long long)ctx->num_sms * 8;
    const size_t poses = sizeof(float) * 12 * n_frames;
    if (n >= most * 4 * BW_THREADS)
        integrate_backward_kernel<4><<<(unsigned int)most, BW_THREADS, poses, s>>>(p);
    else
        integrate_backward_kernel<1>
            <<<(unsigned int)std::min(most, (n + BW_THREADS - 1) / BW_THREADS), BW_THREADS, poses, s>>>(p);
    e = cudaGetLastError();
    return e == cudaSuccess ? MCG_OK : mcg_cuda_fail(ctx, e);
}

mcg_status mcg_integrate_backward(mcg_context *ctx, const void *vol0, int32_t nx, int32_t ny, int32_t nz,
                                  float min_t, float max_t, float grid_s, const mcg_intrinsic *k, int32_t n_frames,
                                  const float *poses_dev, int32_t w, int32_t h, const float *depth_m,
                                  const float *normals, int32_t is_dynamic, const float *grad_f,
                                  const float *grad_w, float *grad_depth, float *grad_f0, float *grad_w0,
                                  mcg_stream_t stream) {
    return integrate_backward_impl(ctx, vol0, nx, ny, nz, min_t, max_t, grid_s, k, n_frames, poses_dev, w, h, depth_m,
                                   normals, is_dynamic, grad_f, grad_w, 1, grad_depth, grad_f0, grad_w0, stream);
}

mcg_status mcg_integrate_backward_volume(mcg_context *ctx, const void *vol0, int32_t nx, int32_t ny, int32_t nz,
                                         float min_t, float max_t, float grid_s, const mcg_intrinsic *k,
                                         int32_t n_frames, const float *poses_dev, int32_t w, int32_t h,
                                         const float *depth_m, const float *normals, int32_t is_dynamic,
                                         const float *grad_vol, float *grad_depth, float *grad_f0, float *grad_w0,
                                         mcg_stream_t stream) {
    return integrate_backward_impl(ctx, vol0, nx, ny, nz, min_t, max_t, grid_s, k, n_frames, poses_dev, w, h, depth_m,
                                   normals, is_dynamic, grad_vol, grad_vol ? grad_vol + 1 : nullptr, 2, grad_depth,
                                   grad_f0, grad_w0, stream);
}

}  // extern "C"
