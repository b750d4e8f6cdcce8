// Depth pyramid and projective point-to-plane ICP on sm_103a
// (cu_kinect_fusion_v1.cu:66-80, 226-261, 988-1301).
//
// The reference runs, per ICP iteration, a correspondence kernel, a kernel
// writing the 6 columns of A and b, then 27 pairs of nppsMul_32f +
// thrust::inclusive_scan for the normal equations, copies them to the host
// and solves there.  Here one cooperative launch (icp_loop) runs all
// iterations of a level: per pixel the correspondence (nearest pixel, step 1,
// or bilinear, step 4), the row of A and b (step 2) and the inlier flag (step
// 3); the 27 products A_i A_j and A_i b are formed in binary32 as nppsMul_32f
// forms them and summed in binary64 in a fixed order; then Cholesky, the
// determinant and 1-norm condition tests, the increment, its bounds, exp([w]x)
// (Rodrigues), compose and the stopping rule of kf.cu:1177-1262.  The host
// reads the outcome once.  Per-pixel arithmetic is the reference's binary32 in
// source order (--fmad=false).
#include <cuda_runtime.h>
#include <float.h>
#include <math.h>
#include <stdint.h>

#include "mcg_internal.h"

namespace mcg {
namespace {

constexpr int IC_THREADS = 256;

// the outcome of a loop
struct IcpState {
    float r[9], t[3];  // pose_rel: rotation column-major, translation
    int rt;            // succeeded
    int iters;         // iterations run
    int late;          // a wait at the grid barrier ran out
    unsigned int arrived;  // the barrier's counter
};

struct IcpArgs {
    float nt, dt;
    float fx, fy, cx, cy;
    int w1, h1, w2, h2;
    const float3 *v1, *n1, *v2, *n2;
};

__device__ __forceinline__ bool ic_nz(float3 n) { return n.x != 0.0f || n.y != 0.0f || n.z != 0.0f; }
__device__ __forceinline__ float3 ic_rot(const float *r, float3 p) {  // float33_mv
    return make_float3(r[0] * p.x + r[3] * p.y + r[6] * p.z, r[1] * p.x + r[4] * p.y + r[7] * p.z,
                       r[2] * p.x + r[5] * p.y + r[8] * p.z);
}
__device__ __forceinline__ float3 ic_fwd(const float *r, const float *t, float3 p) {  // extrinsic_forward
    const float3 q = ic_rot(r, p);
    return make_float3(q.x + t[0], q.y + t[1], q.z + t[2]);
}
__device__ __forceinline__ float3 ic_bwd(const float *r, const float *t, float3 p) {  // extrinsic_backward
    const float dx = p.x - t[0], dy = p.y - t[1], dz = p.z - t[2];
    return make_float3(r[0] * dx + r[1] * dy + r[2] * dz, r[3] * dx + r[4] * dy + r[5] * dz,
                       r[6] * dx + r[7] * dy + r[8] * dz);
}
__device__ __forceinline__ float ic_dist(float3 a, float3 b) {  // float3_distance
    float d = a.x - b.x, s = d * d;
    d = a.y - b.y;
    s += d * d;
    d = a.z - b.z;
    s += d * d;
    return sqrtf(s);
}
__device__ __forceinline__ float3 ic_bilerp(const float3 *v, float x, float y) {  // vector3_interpolation_bilinear
    const float a = 1.0f - x, b = 1.0f - y;
    const float ab = a * b, xb = x * b, ay = a * y, xy = x * y;
    return make_float3(v[0].x * ab + v[1].x * xb + v[2].x * ay + v[3].x * xy,
                       v[0].y * ab + v[1].y * xb + v[2].y * ay + v[3].y * xy,
                       v[0].z * ab + v[1].z * xb + v[2].z * ay + v[3].z * xy);
}

// steps 1 / 4 for pixel idx of map 1: the transformed match in *out
template <bool BILINEAR>
__device__ __forceinline__ bool ic_match(const IcpArgs &a, const float *r, const float *t, long long idx,
                                         float3 *v1o, float3 *n1o, float3 *out) {
    const float3 p1 = a.v1[idx], m1 = a.n1[idx];
    *v1o = p1;
    *n1o = m1;
    if (!ic_nz(m1)) return false;
    const float3 p3 = ic_bwd(r, t, p1);
    const float px = a.fx * (p3.x / p3.z) + a.cx, py = a.fy * (p3.y / p3.z) + a.cy;
    if (!BILINEAR) {
        const int ix = __float2int_rn(px), iy = __float2int_rn(py);
        if (ix < 0 || iy < 0 || ix >= a.w2 || iy >= a.h2) return false;
        const long long j = (long long)iy * a.w2 + ix;
        float3 m2 = a.n2[j];
        if (!ic_nz(m2)) return false;
        m2 = ic_rot(r, m2);
        if (!(m1.x * m2.x + m1.y * m2.y + m1.z * m2.z > a.nt)) return false;
        const float3 p2 = ic_fwd(r, t, a.v2[j]);
        if (!(ic_dist(p1, p2) < a.dt)) return false;
        *out = p2;
        return true;
    } else {
        const int ix = (int)px, iy = (int)py;
        if (ix < 0 || iy < 0 || ix >= a.w2 - 1 || iy >= a.h2 - 1) return false;
        const long long j = (long long)iy * a.w2 + ix;
        float3 nn[4] = {a.n2[j], a.n2[j + 1], a.n2[j + a.w2], a.n2[j + a.w2 + 1]};
        if (!(ic_nz(nn[0]) && ic_nz(nn[1]) && ic_nz(nn[2]) && ic_nz(nn[3]))) return false;
        const float du = px - ix, dv = py - iy;
        const float3 m2 = ic_rot(r, ic_bilerp(nn, du, dv));
        if (!(m1.x * m2.x + m1.y * m2.y + m1.z * m2.z > a.nt)) return false;
        nn[0] = a.v2[j];
        nn[1] = a.v2[j + 1];
        nn[2] = a.v2[j + a.w2];
        nn[3] = a.v2[j + a.w2 + 1];
        const float3 p2 = ic_fwd(r, t, ic_bilerp(nn, du, dv));
        if (!(ic_dist(p1, p2) < a.dt)) return false;
        *out = p2;
        return true;
    }
}

// step 2: the row of A and b of a match
__device__ __forceinline__ void ic_row(float3 p1, float3 m1, float3 o, float A[6], float *b) {
    A[0] = m1.z * o.y - m1.y * o.z;
    A[1] = m1.x * o.z - m1.z * o.x;
    A[2] = m1.y * o.x - m1.x * o.y;
    A[3] = m1.x;
    A[4] = m1.y;
    A[5] = m1.z;
    *b = m1.x * p1.x + m1.y * p1.y + m1.z * p1.z - m1.x * o.x - m1.y * o.y - m1.z * o.z;
}

// one correspondence pass with all per-pixel outputs (for checking and for
// callers that want the rows): v21 (x = FLT_MAX and y = z = 0 when none),
// A column-major (n rows per column), b, inlier flags
template <bool BILINEAR>
__global__ void __launch_bounds__(IC_THREADS) icp_correspond_kernel(IcpArgs a, const float *__restrict__ pose,
                                                                    float3 *__restrict__ v21, float *__restrict__ A,
                                                                    float *__restrict__ bv, uint8_t *__restrict__ inl) {
    const long long n = (long long)a.w1 * a.h1;
    for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < n;
         idx += (long long)gridDim.x * blockDim.x) {
        float3 p1, m1, o = make_float3(FLT_MAX, 0.0f, 0.0f);
        const bool found = ic_match<BILINEAR>(a, pose, pose + 9, idx, &p1, &m1, &o);
        if (v21) v21[idx] = found ? o : make_float3(FLT_MAX, 0.0f, 0.0f);
        if (inl) inl[idx] = found ? 0xff : 0;
        if (A) {
            float row[6] = {0, 0, 0, 0, 0, 0}, b = 0.0f;
            if (found) ic_row(p1, m1, o, row, &b);
#pragma unroll
            for (int c = 0; c < 6; ++c) A[c * n + idx] = row[c];
            bv[idx] = b;
        }
    }
}

// ---- the loop ------------------------------------------------------------------
// One cooperative launch runs a level's whole loop.  Per iteration every CTA
// adds up the products of its pixels (27 sums: 21 of A_i A_j, i <= j, row-major
// upper triangle, 6 of A_i b; the products in binary32 as nppsMul_32f forms
// them, the sums in binary64) and stores them, one grid barrier makes them
// visible, and every CTA then adds the CTAs' sums in the same order and solves
// for itself, so that no second barrier has to bring the pose back.  Partial
// sums alternate between two buffers: a CTA can be at most one barrier ahead
// of another that still reads.
//
// What bounds it: the binary64 units (two sums a clock and SM).  A warp
// reduces its 27 sums by halving (each step a lane keeps half of the values
// and adds the other lane's: 31 sums and shuffles, against 135 for a tree per
// value), the solve spreads over lanes (rows of the factorisation, columns of
// the inverse beside the right-hand side).  Before, an iteration was two
// launches, the second one warp adding 304 CTAs' sums one after another and
// one thread solving, 76 us; the launches after the loop's end cost 4 us each.
// Tracking a 640x480 frame (pyramid, maps, three levels): 1286 -> 633 us, of
// which the loops 810 -> 261 us.
constexpr int IL_THREADS = 512;
constexpr int IL_WARPS = IL_THREADS / 32;
constexpr int IL_SUMS = 27;
constexpr unsigned long long IL_LIMIT_NS = 2000000000ull;  // longest wait at the grid barrier

struct IcpShared {
    double red[IL_WARPS][32];
    double sum[IL_SUMS];
    double x[6], md, prev_md;
    float pose[12];
    float inc[12];
    int it, rt, done, iters, late;
};

__device__ __forceinline__ unsigned long long ic_now() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// all CTAs of the launch (one cooperative launch: they run together); false
// when the wait ran out
__device__ __forceinline__ bool ic_grid_barrier(IcpShared &S, unsigned int *arrived, unsigned int target) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(arrived, 1u);
        const unsigned long long t0 = ic_now();
        for (;;) {
            unsigned int v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(arrived) : "memory");
            if (v >= target) break;
            if (ic_now() - t0 > IL_LIMIT_NS) {
                S.late = 1;
                break;
            }
        }
    }
    __syncthreads();
    return S.late == 0;
}

// warp-wide sums of 32 values per lane: lane k returns the sum of value k
__device__ __forceinline__ double ic_warp_sums(double (&v)[32]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int k = 0; k < o; ++k) {
            const double keep = up ? v[k + o] : v[k], send = up ? v[k] : v[k + o];
            v[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    return v[0];
}

// Cholesky solve with the reference's tests by one warp.  A lane holds a row of
// six values and the factorisation runs over the rows of AtA (lanes 0-5), the
// right-hand side (lane 6) and the unit vectors (lanes 8-13) alike: what it
// leaves in a row v is the solution of L y = v, so the forward substitutions
// come with the factor.  The back substitutions then give the increment (lane
// 6) and the columns of the inverse for the condition number.  Updates run
// ahead (right-looking) and the diagonal enters as its reciprocal square root,
// because a chain of dependent binary64 operations is what this takes: the
// same solve by substitution with divisions took about 20 us, this 4.
// Fills S.x and S.md; returns false (on every lane) to stop the loop.
__device__ bool ic_solve(IcpShared &S) {
    const unsigned int full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    double v[6], anorm = 0.0;
    bool off = false;
#pragma unroll
    for (int j = 0; j < 6; ++j) {
        v[j] = lane == 8 + j ? 1.0 : 0.0;
        if (lane < 6) {
            const int lo = min(lane, j), hi = max(lane, j);
            v[j] = S.sum[lo * 6 - lo * (lo - 1) / 2 + hi - lo];
            anorm += fabs(v[j]);  // column `lane` (AtA is symmetric)
            if (j < lane && v[j] != 0.0) off = true;
        }
        if (lane == 6) v[j] = S.sum[21 + j];
    }
    if (!__any_sync(full, off)) return false;  // empty
    double det = 1.0, rinv[6];
#pragma unroll
    for (int j = 0; j < 6; ++j) {
        const double d = __shfl_sync(full, v[j], j);
        if (!(d > 0.0)) return false;  // not positive definite
        rinv[j] = rsqrt(d);
        v[j] *= rinv[j];
        det *= d;
#pragma unroll
        for (int k = j + 1; k < 6; ++k) v[k] = fma(-v[j], __shfl_sync(full, v[j], k), v[k]);
    }
    if (!(fabs(det) > 1e-15)) return false;  // null space
    double z[6], inorm = 0.0;
#pragma unroll
    for (int r = 0; r < 6; ++r) z[r] = v[r];
#pragma unroll
    for (int p = 5; p >= 0; --p) {
        z[p] *= rinv[p];
        inorm += fabs(z[p]);
#pragma unroll
        for (int r = 0; r < 6; ++r)
            if (r < p) z[r] = fma(-__shfl_sync(full, v[r], p), z[p], z[r]);
    }
    if (lane < 8 || lane > 13) inorm = 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        anorm = fmax(anorm, __shfl_xor_sync(full, anorm, o));
        inorm = fmax(inorm, __shfl_xor_sync(full, inorm, o));
    }
    if (!(1.0 > 5e-5 * (anorm * inorm))) return false;  // ill-conditioned
    if (lane == 6) {
        double m = 0.0;
#pragma unroll
        for (int r = 0; r < 6; ++r) {
            S.x[r] = z[r];
            m = fma(S.sum[21 + r], z[r], m);
        }
        S.md = m;
    }
    __syncwarp();
    return true;
}

// sin(th) / th and (1 - cos(th)) / th^2 from th^2: their power series, to
// 1e-19 below half a radian (th2^8 / 17!)
__device__ __forceinline__ void ic_rodrigues(double th2, double &ca, double &cb) {
    if (th2 < 0.25) {
        double a = -1.0 / 1307674368000.0, b = -1.0 / 20922789888000.0;  // 1 / 15!, 1 / 16!
        const double ka[7] = {1.0, 6.0, 120.0, 5040.0, 362880.0, 39916800.0, 6227020800.0};
        const double kb[7] = {2.0, 24.0, 720.0, 40320.0, 3628800.0, 479001600.0, 87178291200.0};
#pragma unroll
        for (int k = 6; k >= 0; --k) {
            const double sg = k & 1 ? -1.0 : 1.0;
            a = fma(a, th2, sg / ka[k]);
            b = fma(b, th2, sg / kb[k]);
        }
        ca = a;
        cb = b;
    } else {
        const double th = sqrt(th2);
        ca = sin(th) / th;
        cb = (1.0 - cos(th)) / th2;
    }
}

// one step of the loop after the sums, by warp 0: the increment, its bounds,
// exp([w]x) by Rodrigues' formula, compose, the stopping rule (kf.cu:1177-1262)
__device__ void ic_step(IcpShared &S, float rtb, float ttb) {
    const int lane = threadIdx.x & 31;
    bool rt = ic_solve(S);
    if (rt) {
        const double x0 = S.x[0], x1 = S.x[1], x2 = S.x[2];
        if (fabs(x0) > rtb || fabs(x1) > rtb || fabs(x2) > rtb || fabs(S.x[3]) > ttb || fabs(S.x[4]) > ttb ||
            fabs(S.x[5]) > ttb) {
            rt = false;  // out of bound
        } else {
            double ca, cb;
            ic_rodrigues(x0 * x0 + x1 * x1 + x2 * x2, ca, cb);
            const int c = min(lane / 3, 2), r = lane % 3;
            if (lane < 9) {
                const double K[3][3] = {{0.0, -x2, x1}, {x2, 0.0, -x0}, {-x1, x0, 0.0}};
                double kk = 0.0, kr = 0.0;
#pragma unroll
                for (int p = 0; p < 3; ++p) {
                    const double krp = r == 0 ? K[0][p] : r == 1 ? K[1][p] : K[2][p];
                    const double kpc = c == 0 ? K[p][0] : c == 1 ? K[p][1] : K[p][2];
                    kk += krp * kpc;
                    if (p == c) kr = krp;
                }
                S.inc[lane] = (float)((r == c ? 1.0 : 0.0) + ca * kr + cb * kk);  // column-major
            } else if (lane < 12) {
                S.inc[lane] = (float)S.x[lane - 6];
            }
            __syncwarp();
            // float_camera_extrinsic_compose(pose, inc): R = Ri R, t = Ri t + ti (binary32)
            float v = 0.0f;
            if (lane < 9)
                v = S.inc[r] * S.pose[3 * c] + S.inc[3 + r] * S.pose[3 * c + 1] + S.inc[6 + r] * S.pose[3 * c + 2];
            else if (lane < 12)
                v = S.inc[r] * S.pose[9] + S.inc[3 + r] * S.pose[10] + S.inc[6 + r] * S.pose[11] + S.inc[lane];
            __syncwarp();
            if (lane < 12) S.pose[lane] = v;
        }
    }
    __syncwarp();
    if (lane == 0) {
        S.iters += 1;
        if (rt) {
            const double md = S.md;
            if (md > S.prev_md || md < 1e-5) S.it = 1;
            S.prev_md = md;
        }
        S.rt = rt ? 1 : 0;
        S.it -= 1;
        S.done = S.it == 0 || !rt;
    }
}

struct IcpInit {
    float pose[12];
    int it_max;
    float rt, tt;
};

template <bool BILINEAR>
__global__ void __launch_bounds__(IL_THREADS, 1)
    icp_loop(IcpArgs a, IcpInit in, IcpState *__restrict__ st, double *partial, unsigned int *arrived,
             uint8_t *__restrict__ flags, uint8_t *__restrict__ inl) {
    __shared__ IcpShared S;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int G = (int)gridDim.x;
    if (tid < 12) S.pose[tid] = in.pose[tid];
    if (tid == 0) {
        S.it = in.it_max;
        S.rt = 1;
        S.done = S.iters = S.late = 0;
        S.prev_md = (double)FLT_MAX;
    }
    __syncthreads();
    const long long n = (long long)a.w1 * a.h1;
    for (int pass = 0;; ++pass) {
        double acc[32];
#pragma unroll
        for (int k = 0; k < 32; ++k) acc[k] = 0.0;
        for (long long idx = (long long)blockIdx.x * IL_THREADS + tid; idx < n; idx += (long long)G * IL_THREADS) {
            float3 p1, m1, o;
            const bool found = ic_match<BILINEAR>(a, S.pose, S.pose + 9, idx, &p1, &m1, &o);
            if (flags) flags[idx] = found ? 0xff : 0;
            if (found) {
                float row[6], b;
                ic_row(p1, m1, o, row, &b);
                int k = 0;
#pragma unroll
                for (int i = 0; i < 6; ++i) {
#pragma unroll
                    for (int j = i; j < 6; ++j) acc[k++] += (double)(row[i] * row[j]);
                }
#pragma unroll
                for (int i = 0; i < 6; ++i) acc[21 + i] += (double)(row[i] * b);
            }
        }
        S.red[warp][lane] = ic_warp_sums(acc);
        __syncthreads();
        double *buf = partial + (long long)(pass & 1) * G * IL_SUMS;
        if (tid < IL_SUMS) {
            double v = 0.0;
#pragma unroll
            for (int w = 0; w < IL_WARPS; ++w) v += S.red[w][tid];
            __stcg(buf + (long long)blockIdx.x * IL_SUMS + tid, v);
        }
        if (!ic_grid_barrier(S, arrived, (unsigned int)(pass + 1) * (unsigned int)G)) break;
        // warp w adds the sums of CTAs w, w + IL_WARPS, ...; then the warps' in order
        if (lane < IL_SUMS) {
            double v = 0.0;
            for (int c = warp; c < G; c += IL_WARPS) v += __ldcg(buf + (long long)c * IL_SUMS + lane);
            S.red[warp][lane] = v;
        }
        __syncthreads();
        if (warp == 0) {
            if (lane < IL_SUMS) {
                double v = 0.0;
#pragma unroll
                for (int w = 0; w < IL_WARPS; ++w) v += S.red[w][lane];
                S.sum[lane] = v;
            }
            __syncwarp();
            ic_step(S, in.rt, in.tt);
        }
        __syncthreads();
        if (S.done) break;
    }
    // the caller's map receives the last pass's flags only when the loop
    // succeeds (kf.cu:1285-1292); each thread copies what it wrote
    if (inl && S.rt && !S.late)
        for (long long idx = (long long)blockIdx.x * IL_THREADS + tid; idx < n; idx += (long long)G * IL_THREADS)
            inl[idx] = flags[idx];
    if (tid == 0 && S.late) st->late = 1;
    if (blockIdx.x == 0) {
        if (tid < 12) (tid < 9 ? st->r[tid] : st->t[tid - 9]) = S.pose[tid];
        if (tid == 0) {
            st->rt = S.rt;
            st->iters = S.iters;
        }
    }
}

// kf.cu:226-261
__global__ void pyramid_down_kernel(int sw, int sh, int dw, int dh, const float *__restrict__ s,
                                    const uint8_t *__restrict__ sm, float *__restrict__ d, uint8_t *__restrict__ dm,
                                    float sigma) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= dw || y >= dh) return;
    const int D = 5, H = D >> 1;
    int si = (y << 1) * sw + (x << 1);
    const int di = y * dw + x;
    dm[di] = 0;
    if (!sm[si]) return;
    const float center = s[si];
    const int tx = min((x << 1) - H + D, sw - 1), ty = min((y << 1) - H + D, sh - 1);
    float sum = 0.0f;
    int count = 0;
    for (int cy = max(0, (y << 1) - H); cy < ty; ++cy)
        for (int cx = max(0, (x << 1) - H); cx < tx; ++cx) {
            si = cy * sw + cx;
            if (sm[si]) {
                const float val = s[si];
                if (fabsf(val - center) < sigma) {
                    sum += val;
                    ++count;
                }
            }
        }
    if (count) {
        d[di] = sum / count;
        dm[di] = 0xff;
    }
}

// kf.cu:66-72 (to_mask = 1), 74-80 (to_mask = 0)
__global__ void mask_kernel(long long n, int to_mask, float *__restrict__ data, uint8_t *__restrict__ mask) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        if (to_mask)
            mask[i] = data[i] != 0.0f ? 0xff : 0;
        else if (mask[i] == 0)
            data[i] = 0.0f;
    }
}

IcpArgs make_args(const mcg_icp_params *p, const mcg_intrinsic *k, int w1, int h1, int w2, int h2, const float *v1,
                  const float *n1, const float *v2, const float *n2) {
    IcpArgs a;
    a.nt = p->nt;
    a.dt = p->dt;
    a.fx = k->fx;
    a.fy = k->fy;
    a.cx = k->cx;
    a.cy = k->cy;
    a.w1 = w1;
    a.h1 = h1;
    a.w2 = w2;
    a.h2 = h2;
    a.v1 = reinterpret_cast<const float3 *>(v1);
    a.n1 = reinterpret_cast<const float3 *>(n1);
    a.v2 = reinterpret_cast<const float3 *>(v2);
    a.n2 = reinterpret_cast<const float3 *>(n2);
    return a;
}

bool icp_args_ok(const mcg_icp_params *p, const mcg_intrinsic *k, int w1, int h1, int w2, int h2, const void *v1,
                 const void *n1, const void *v2, const void *n2) {
    return p && k && v1 && n1 && v2 && n2 && w1 > 0 && h1 > 0 && w2 > 0 && h2 > 0 && p->it_max > 0;
}

}  // namespace
}  // namespace mcg

using namespace mcg;

extern "C" mcg_status mcg_pyramid_down(mcg_context *ctx, int32_t sw, int32_t sh, int32_t dw, int32_t dh,
                                       const float *src, const uint8_t *src_mask, float *dst, uint8_t *dst_mask,
                                       float sigma, mcg_stream_t stream) {
    if (!ctx || !src || !src_mask || !dst || !dst_mask || sw <= 0 || sh <= 0 || dw <= 0 || dh <= 0 ||
        2 * (dw - 1) >= sw || 2 * (dh - 1) >= sh)
        return MCG_ERR_INVALID_ARG;
    cudaError_t e = cudaSetDevice(ctx->device);
    if (e != cudaSuccess) return mcg_cuda_fail(ctx, e);
    const dim3 block(16, 16), grid((dw + 15) / 16, (dh + 15) / 16);
    pyramid_down_kernel<<<grid, block, 0, (cudaStream_t)stream>>>(sw, sh, dw, dh, src, src_mask, dst, dst_mask, sigma);
    e = cudaGetLastError();
    return e == cudaSuccess ? MCG_OK : mcg_cuda_fail(ctx, e);
}

extern "C" mcg_status mcg_depth_mask(mcg_context *ctx, int64_t n, float *data, uint8_t *mask, int32_t to_mask,
                                     mcg_stream_t stream) {
    if (!ctx || !data || !mask || n < 0) return MCG_ERR_INVALID_ARG;
    cudaError_t e = cudaSetDevice(ctx->device);
    if (e != cudaSuccess) return mcg_cuda_fail(ctx, e);
    if (n == 0) return MCG_OK;
    const int blocks = (int)std::min<long long>((n + 255) / 256, (long long)ctx->num_sms * 8);
    mask_kernel<<<blocks, 256, 0, (cudaStream_t)stream>>>(n, to_mask ? 1 : 0, data, mask);
    e = cudaGetLastError();
    return e == cudaSuccess ? MCG_OK : mcg_cuda_fail(ctx, e);
}

extern "C" mcg_status mcg_icp_correspond(mcg_context *ctx, const mcg_icp_params *p, const mcg_intrinsic *k2,
                                         const mcg_extrinsic *pose_rel, int32_t w1, int32_t h1, int32_t w2, int32_t h2,
                                         const float *v1, const float *n1, const float *v2, const float *n2,
                                         float *v21, float *A, float *b, uint8_t *inlier, mcg_stream_t stream) {
    if (!ctx || !pose_rel || !icp_args_ok(p, k2, w1, h1, w2, h2, v1, n1, v2, n2) || (A && !b) || (!A && b))
        return MCG_ERR_INVALID_ARG;
    cudaError_t e = cudaSetDevice(ctx->device);
    if (e != cudaSuccess) return mcg_cuda_fail(ctx, e);
    const cudaStream_t s = (cudaStream_t)stream;
    if (!ensure(&ctx->icp_pose, &ctx->icp_pose_cap, 12)) return mcg_cuda_fail(ctx, cudaErrorMemoryAllocation);
    float hp[12];
    for (int i = 0; i < 9; ++i) hp[i] = pose_rel->r[i];
    for (int i = 0; i < 3; ++i) hp[9 + i] = pose_rel->t[i];
    if ((e = cudaMemcpyAsync(ctx->icp_pose, hp, sizeof(hp), cudaMemcpyHostToDevice, s)) != cudaSuccess)
        return mcg_cuda_fail(ctx, e);
    const IcpArgs a = make_args(p, k2, w1, h1, w2, h2, v1, n1, v2, n2);
    const long long n = (long long)w1 * h1;
    const int blocks = (int)std::min<long long>((n + IC_THREADS - 1) / IC_THREADS, (long long)ctx->num_sms * 8);
    if (p->bilinear)
        icp_correspond_kernel<true><<<blocks, IC_THREADS, 0, s>>>(a, ctx->icp_pose, reinterpret_cast<float3 *>(v21), A,
                                                                   b, inlier);
    else
        icp_correspond_kernel<false><<<blocks, IC_THREADS, 0, s>>>(a, ctx->icp_pose, reinterpret_cast<float3 *>(v21),
                                                                    A, b, inlier);
    if ((e = cudaGetLastError()) != cudaSuccess || (e = cudaStreamSynchronize(s)) != cudaSuccess)  // hp is on the stack
        return mcg_cuda_fail(ctx, e);
    return MCG_OK;
}

extern "C" mcg_status mcg_icp(mcg_context *ctx, const mcg_icp_params *p, const mcg_intrinsic *k2,
                              mcg_extrinsic *pose_rel, int32_t w1, int32_t h1, int32_t w2, int32_t h2, const float *v1,
                              const float *n1, const float *v2, const float *n2, uint8_t *inlier, int32_t *ok,
                              int32_t *iterations, mcg_stream_t stream) {
    if (!ctx || !pose_rel || !ok || !icp_args_ok(p, k2, w1, h1, w2, h2, v1, n1, v2, n2)) return MCG_ERR_INVALID_ARG;
    cudaError_t e = cudaSetDevice(ctx->device);
    if (e != cudaSuccess) return mcg_cuda_fail(ctx, e);
    const cudaStream_t s = (cudaStream_t)stream;
    const long long npx = (long long)w1 * h1;
    // one CTA per SM at most: the launch is cooperative and its CTAs wait for each other
    int G = (int)std::min<long long>((npx + IL_THREADS - 1) / IL_THREADS, (long long)ctx->num_sms);
    if (!ensure(&ctx->icp_state, &ctx->icp_state_cap, sizeof(IcpState)) ||
        !ensure(&ctx->icp_partial, &ctx->icp_partial_cap, (size_t)2 * ctx->num_sms * IL_SUMS))
        return mcg_cuda_fail(ctx, cudaErrorMemoryAllocation);
    if (!ctx->h_icp_state && cudaMallocHost((void **)&ctx->h_icp_state, sizeof(IcpState)) != cudaSuccess) {
        ctx->h_icp_state = nullptr;
        return mcg_cuda_fail(ctx, cudaErrorMemoryAllocation);
    }
    IcpState *hs = reinterpret_cast<IcpState *>(ctx->h_icp_state);
    IcpState *ds = reinterpret_cast<IcpState *>(ctx->icp_state);
    IcpInit in;
    for (int i = 0; i < 9; ++i) in.pose[i] = pose_rel->r[i];
    for (int i = 0; i < 3; ++i) in.pose[9 + i] = pose_rel->t[i];
    in.it_max = p->it_max;
    in.rt = p->rt;
    in.tt = p->tt;
    if ((e = cudaMemsetAsync(ds, 0, sizeof(IcpState), s)) != cudaSuccess) return mcg_cuda_fail(ctx, e);
    uint8_t *flags = nullptr;
    if (inlier) {
        if (!ensure(&ctx->icp_inlier, &ctx->icp_inlier_cap, (size_t)npx))
            return mcg_cuda_fail(ctx, cudaErrorMemoryAllocation);
        flags = ctx->icp_inlier;
    }
    IcpArgs a = make_args(p, k2, w1, h1, w2, h2, v1, n1, v2, n2);
    unsigned int *arrived = &ds->arrived;
    void *args[] = {&a, &in, &ds, &ctx->icp_partial, &arrived, &flags, &inlier};
    const void *fn = p->bilinear ? (const void *)icp_loop<true> : (const void *)icp_loop<false>;
    if ((e = cudaLaunchCooperativeKernel(fn, dim3(G), dim3(IL_THREADS), args, 0, s)) != cudaSuccess ||
        (e = cudaMemcpyAsync(hs, ds, sizeof(IcpState), cudaMemcpyDeviceToHost, s)) != cudaSuccess ||
        (e = cudaStreamSynchronize(s)) != cudaSuccess)
        return mcg_cuda_fail(ctx, e);
    if (hs->late) return MCG_ERR_TIMEOUT;
    *ok = hs->rt;
    if (iterations) *iterations = hs->iters;
    if (hs->rt) {
        for (int i = 0; i < 9; ++i) pose_rel->r[i] = hs->r[i];
        for (int i = 0; i < 3; ++i) pose_rel->t[i] = hs->t[i];
    }
    return MCG_OK;
}
