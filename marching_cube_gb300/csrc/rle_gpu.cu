// Run-length encoding of a device volume on the GPU (the file format of
// cu_kinect_fusion_v1.cu:1303-1600, described in rle.cpp).
//
// The reference encodes slice after slice on one host thread
// (cu_voxel_run_length_encode_slice, :1367-1417).  The format:
//   - voxel i of a slice starts a run when i = 0 or it differs from voxel i-1
//     (tsdf only in the reference format, the whole voxel in the lossless one);
//   - a record starts at every run start and every 16383 voxels into a run
//     (the 14-bit count), as the sequential encoder splits long runs;
//   - a record is 2 bytes (kinds 1/2: +-32766 with, in the lossless format,
//     w = 0) or 6 bytes (kind 3: header + the record's first voxel).
// Here every chunk of 4096 voxels of a slice is encoded on its own:
//   1. rle_mark: one pass over the volume; a bit per voxel that starts a run,
//      and per chunk the bytes of those records and the first and last of them;
//   2. rle_place: one CTA per slice; the run in force at each chunk's start,
//      hence the chunk's split (a run that reaches into a chunk has at most one
//      there: chunks are shorter than 16383), byte offset and the record that
//      follows it;  rle_slices: the slices' offsets and the image's size;
//   3. rle_emit: per chunk with records, from its bits, the voxels at record
//      starts only; the bytes are laid out in shared memory and leave coalesced.
// The image then crosses to the host in one copy.  Scratch is a bit per voxel
// (each slice's rounded up to words) and 24 bytes per chunk, of as many slices
// as fit RSCRATCH, or memory; with more slices, passes 1 and 2 run once more
// before pass 3.
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>

#include "mcg_internal.h"

namespace mcg {
namespace {

constexpr int RT = 256;            // threads per CTA
constexpr int RCHUNK = 4096;       // voxels per chunk
constexpr int RWORDS = RCHUNK / 32;
constexpr int RWARPS = RT / 32;
constexpr long long RSCRATCH = 288ll << 20;  // bytes of run-start bits and chunk records at a time: 2^31 voxels'
// Most bytes of an image (at 6 a voxel) whose records are written before its size
// has been read: encoding 32^3 voxels takes 67 us so, 79 with the wait between the
// launches; 96^3 146 and 151.
constexpr long long RAHEAD = 8ll << 20;
constexpr int kMaxRun = 0x3fff;

// record kind of a record whose first voxel is v (put_run in rle.cpp)
__device__ __forceinline__ unsigned record_kind(uint32_t v, bool lossless) {
    const int16_t t = (int16_t)(v & 0xffffu);
    const bool w0 = (v >> 16) == 0u;
    if (t == (int16_t)kMaxTsdf && (!lossless || w0)) return 1u;
    if (t == (int16_t)-kMaxTsdf && (!lossless || w0)) return 2u;
    return 3u;
}

// a chunk's record starts: the run starts it holds, then what rle_place adds
struct RleChunk {
    int first, last;  // slice index of the first and last run start; first = INT32_MAX, last = -1: none
    int bytes;        // bytes of the records at run starts
    int split;        // slice index of the record that splits a run from before the chunk, or -1
    int off;          // byte offset of the chunk's first record in the slice's records
    int next;         // slice index of the first record after the chunk (the slice's end if none)
};

// Pass 1.  A warp reads 512 consecutive voxels, 16 bytes a lane at a time, all
// loads ahead of their use.  Bound: HBM (the volume once: 79 us for 512^3
// voxels).  One CTA sweeping a slice, a block scan per chunk, took 311 us for
// these just to count and 563 us more to write (26 MB); the passes here take
// 101, 5, 2 and 53 us.  This one took 138 us with the run starts' kinds and
// words worked out for every 128 voxels, also where no run starts.
__global__ void __launch_bounds__(RT) rle_mark(const uint32_t *__restrict__ vol, int xy, int nchunks, int lossless_i,
                                               RleChunk *__restrict__ chunks, uint32_t *__restrict__ marks, int cwords,
                                               int vec) {
    constexpr int Q = RCHUNK / RT / 4;  // 16-byte words per lane
    __shared__ int s_first[RWARPS], s_last[RWARPS], s_bytes[RWARPS];
    const bool lossless = lossless_i != 0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long c = blockIdx.x;
    const int z = (int)(c / nchunks), c0 = (int)(c - (long long)z * nchunks) * RCHUNK;
    const uint32_t *sl = vol + (long long)z * xy;
    const int w0 = c0 + warp * 128 * Q;  // the warp's voxels w0 .. w0 + 128 Q - 1
    uint4 v[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const int i = w0 + 128 * q + 4 * lane;
        if (vec && i < xy) {  // xy is a multiple of 4
            v[q] = __ldg(reinterpret_cast<const uint4 *>(sl + i));
        } else {
            v[q].x = i < xy ? __ldg(sl + i) : 0u;
            v[q].y = i + 1 < xy ? __ldg(sl + i + 1) : 0u;
            v[q].z = i + 2 < xy ? __ldg(sl + i + 2) : 0u;
            v[q].w = i + 3 < xy ? __ldg(sl + i + 3) : 0u;
        }
    }
    uint32_t before = w0 > 0 && w0 <= xy ? __ldg(sl + w0 - 1) : 0u;
    const uint32_t differ = lossless ? 0xffffffffu : 0xffffu;
    int bytes = 0, first = INT32_MAX, last = -1;
    const int word0 = warp * 4 * Q;  // cwords of a chunk's words are kept (those of a slice shorter than a chunk)
    uint32_t *out = marks + c * cwords;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const int i = w0 + 128 * q + 4 * lane;
        uint32_t left = __shfl_up_sync(0xffffffffu, v[q].w, 1);
        if (lane == 0) left = before;
        before = __shfl_sync(0xffffffffu, v[q].w, 31);
        const uint32_t x[5] = {left, v[q].x, v[q].y, v[q].z, v[q].w};
        uint32_t bits = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if ((x[k + 1] ^ x[k]) & differ) bits |= 1u << k;
        if (i == 0) bits |= 1u;  // a slice starts a run
        if (i + 4 > xy) bits &= i < xy ? (1u << (xy - i)) - 1u : 0u;
        uint32_t word = 0;
        if (__any_sync(0xffffffffu, bits)) {
            // most 128 voxels have no run start
            if (bits) {
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (bits & (1u << k)) bytes += record_kind(x[k + 1], lossless) == 3u ? 6 : 2;
                first = min(first, i + __ffs(bits) - 1);
                last = i + 31 - __clz(bits);
            }
            // eight lanes' bits make a word
            word = bits << (4 * (lane & 7));
            word |= __shfl_xor_sync(0xffffffffu, word, 1);
            word |= __shfl_xor_sync(0xffffffffu, word, 2);
            word |= __shfl_xor_sync(0xffffffffu, word, 4);
        }
        const int at = word0 + 4 * q + (lane >> 3);
        if ((lane & 7) == 0 && at < cwords) out[at] = word;
    }
    bytes = __reduce_add_sync(0xffffffffu, bytes);
    first = __reduce_min_sync(0xffffffffu, first);
    last = __reduce_max_sync(0xffffffffu, last);
    if (lane == 0) {
        s_first[warp] = first;
        s_last[warp] = last;
        s_bytes[warp] = bytes;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        RleChunk r{INT32_MAX, -1, 0, -1, 0, 0};
#pragma unroll
        for (int w = 0; w < RWARPS; ++w) {
            r.first = min(r.first, s_first[w]);
            r.last = max(r.last, s_last[w]);
            r.bytes += s_bytes[w];
        }
        chunks[c] = r;
    }
}

// Pass 2.  One warp per slice, 32 chunks at a time: forward for the run in
// force, the split and the offsets, then backward for the record after each.
__global__ void __launch_bounds__(32) rle_place(const uint32_t *__restrict__ vol, int xy, int nchunks, int lossless_i,
                                                RleChunk *__restrict__ chunks,
                                                unsigned long long *__restrict__ slice_bytes) {
    const unsigned int full = 0xffffffffu;
    const int z = blockIdx.x, lane = threadIdx.x;
    RleChunk *ch = chunks + (long long)z * nchunks;
    const uint32_t *sl = vol + (long long)z * xy;
    int run = 0;                  // start of the run in force at the first of the 32 chunks
    unsigned long long off = 0;   // bytes before it
    for (int k0 = 0; k0 < nchunks; k0 += 32) {
        const int k = k0 + lane, c0 = k * RCHUNK, c1 = min(c0 + RCHUNK, xy);
        RleChunk r{INT32_MAX, -1, 0, -1, 0, 0};
        if (k < nchunks) r = ch[k];
        int m = r.last;  // run starts ascend: the last one so far
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(full, m, o);
            if (lane >= o) m = max(m, u);
        }
        int in = __shfl_up_sync(full, m, 1);
        if (lane == 0) in = -1;
        in = max(in, run);
        int split = -1, bytes = r.bytes;
        if (k < nchunks) {
            // the first record past c0 - 1 that a run from before the chunk would start
            const int s = in + (c0 - in + kMaxRun - 1) / kMaxRun * kMaxRun;
            if (in < c0 && s < min(c1, r.first)) {
                split = s;
                bytes += record_kind(__ldg(sl + s), lossless_i != 0) == 3u ? 6 : 2;
            }
        }
        unsigned int sum = (unsigned int)bytes;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned int u = __shfl_up_sync(full, sum, o);
            if (lane >= o) sum += u;
        }
        if (k < nchunks) {
            ch[k].split = split;
            ch[k].off = (int)(off + sum - (unsigned int)bytes);
            ch[k].bytes = bytes;
        }
        run = max(run, __shfl_sync(full, m, 31));
        off += __shfl_sync(full, sum, 31);
    }
    if (lane == 0) slice_bytes[z] = off;
    __syncwarp();
    int after = xy;  // first record after the 32 chunks
    for (int k0 = (nchunks - 1) / 32 * 32; k0 >= 0; k0 -= 32) {
        const int k = k0 + lane;
        int f = INT32_MAX;
        if (k < nchunks) f = ch[k].split >= 0 ? ch[k].split : ch[k].first;
        int m = f;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_down_sync(full, m, o);
            if (lane + o < 32) m = min(m, u);
        }
        int next = __shfl_down_sync(full, m, 1);
        if (lane == 31) next = INT32_MAX;
        if (k < nchunks) ch[k].next = min(next, after);
        after = min(after, __shfl_sync(full, m, 0));
    }
}

// The slices' offsets in the image (after the 40-byte header, each with its
// 4-byte count) and, behind them, the image's size.  One CTA.
__global__ void __launch_bounds__(RT) rle_slices(const unsigned long long *__restrict__ bytes, int nz,
                                                 unsigned long long *__restrict__ off) {
    __shared__ unsigned long long s_w[RWARPS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned long long at = 40;
    for (int z0 = 0; z0 < nz; z0 += RT) {
        const int z = z0 + (int)threadIdx.x;
        const unsigned long long own = z < nz ? 4 + bytes[z] : 0;
        unsigned long long sum = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long u = __shfl_up_sync(0xffffffffu, sum, o);
            if (lane >= o) sum += u;
        }
        if (lane == 31) s_w[warp] = sum;
        __syncthreads();
        unsigned long long pre = 0, all = 0;
#pragma unroll
        for (int w = 0; w < RWARPS; ++w) {
            if (w < warp) pre += s_w[w];
            all += s_w[w];
        }
        __syncthreads();
        if (z < nz) off[z] = at + pre + sum - own;
        at += all;
    }
    if (threadIdx.x == 0) off[nz] = at;
}

// Pass 3.  Bound: the chain of loads and scans of a chunk, so as many chunks in
// flight as an SM has threads for: 128 us with 256 threads and room for all of
// a chunk's records (41 KB), 53 with 128 threads and 9 KB.
constexpr int ET = RWORDS, EWARPS = ET / 32;  // a thread for each word of marks

struct RleEmit {
    uint16_t pos[RCHUNK + 1];  // record starts, then the record after the chunk, from the chunk's first voxel
    uint16_t img[3 * ET];      // ET records at a time
    int wn[EWARPS], wb[EWARPS];
};

__global__ void __launch_bounds__(ET) rle_emit(const uint32_t *__restrict__ vol, int xy, int nchunks, int lossless_i,
                                               const RleChunk *__restrict__ chunks, const uint32_t *__restrict__ marks,
                                               int cwords, const unsigned long long *__restrict__ slice_bytes,
                                               const unsigned long long *__restrict__ slice_off,
                                               uint8_t *__restrict__ img) {
    __shared__ RleEmit S;
    const bool lossless = lossless_i != 0;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long long c = blockIdx.x;
    const int z = (int)(c / nchunks), c0 = (int)(c - (long long)z * nchunks) * RCHUNK;
    const uint32_t word = tid < cwords ? marks[c * cwords + tid] : 0u;
    const RleChunk r = chunks[c];
    const unsigned long long so = slice_off[z];  // even: 40, then 4 and even record bytes a slice
    if (c0 == 0 && tid < 2) reinterpret_cast<uint16_t *>(img + so)[tid] = (uint16_t)(slice_bytes[z] >> (16 * tid));
    if (r.bytes == 0) return;  // no record starts here
    // record starts in order: the split, then the marked voxels
    int n = __popc(word), incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
    }
    if (lane == 31) S.wn[warp] = incl;
    __syncthreads();
    const int extra = r.split >= 0 ? 1 : 0;
    int at = extra + incl - n, total = extra;
#pragma unroll
    for (int w = 0; w < EWARPS; ++w) {
        if (w < warp) at += S.wn[w];
        total += S.wn[w];
    }
    for (uint32_t m = word; m; m &= m - 1) S.pos[at++] = (uint16_t)(32 * tid + __ffs(m) - 1);
    if (tid == 0) {
        if (extra) S.pos[0] = (uint16_t)(r.split - c0);
        S.pos[total] = (uint16_t)(r.next - c0);  // at most a record's voxels past the chunk
    }
    __syncthreads();
    const uint32_t *sl = vol + (long long)z * xy + c0;
    uint16_t *out = reinterpret_cast<uint16_t *>(img + so + 4 + (unsigned int)r.off);
    for (int j0 = 0; j0 < total; j0 += ET) {
        const int j = j0 + tid;
        uint32_t v = 0;
        int halves = 0, count = 0;
        unsigned kind = 0;
        if (j < total) {
            const int p = S.pos[j];
            v = __ldg(sl + p);
            count = S.pos[j + 1] - p;
            kind = record_kind(v, lossless);
            halves = kind == 3u ? 3 : 1;
        }
        int sum = halves;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, sum, o);
            if (lane >= o) sum += u;
        }
        if (lane == 31) S.wb[warp] = sum;
        __syncthreads();
        int pre = 0, all = 0;
#pragma unroll
        for (int w = 0; w < EWARPS; ++w) {
            if (w < warp) pre += S.wb[w];
            all += S.wb[w];
        }
        const int h = pre + sum - halves;
        if (halves) {
            S.img[h] = (uint16_t)((unsigned)count | (kind << 14));
            if (halves == 3) {
                S.img[h + 1] = (uint16_t)(v & 0xffffu);
                S.img[h + 2] = (uint16_t)(v >> 16);
            }
        }
        __syncthreads();
        for (int i = tid; i < all; i += ET) out[i] = S.img[i];
        out += all;
    }
}

const char kTagRef[16] = "VOLUME_TSDF_RGB";
const char kTagLossless[16] = "VOLUME_TSDF_W32";

}  // namespace
}  // namespace mcg

using namespace mcg;

extern "C" mcg_status mcg_rle_encode(mcg_context *ctx, const void *vol, int32_t nx, int32_t ny, int32_t nz,
                                         float min_t, float max_t, float grid_s, int32_t lossless, uint8_t *image,
                                         int64_t capacity, int64_t *size, mcg_stream_t stream) {
    // image == NULL with capacity == 0 asks for the image size only
    const bool query = !image && capacity == 0;
    if (!ctx || !vol || (!image && !query) || !size || nx <= 0 || ny <= 0 || nz <= 0) return MCG_ERR_INVALID_ARG;
    *size = 0;
    const long long xy = (long long)nx * ny;
    // record counts are 14-bit and slice byte counts 32-bit (the file format)
    if (6 * xy > 0xffffffffll) return MCG_ERR_TOO_LARGE;
    cudaStream_t s = (cudaStream_t)stream;
    cudaError_t e = cudaSetDevice(ctx->device);
    if (e != cudaSuccess) return mcg_cuda_fail(ctx, e);
    const long long nchunks = (xy + RCHUNK - 1) / RCHUNK;
    const int cwords = nchunks == 1 ? (int)((xy + 31) / 32) : RWORDS;  // words of marks per chunk
    const long long slice_scratch = nchunks * (long long)(sizeof(RleChunk) + 4 * cwords);
    long long per = std::min<long long>(nz, std::max(1ll, RSCRATCH / slice_scratch));  // slices at a time
    if (!ensure(&ctx->rle_slices, &ctx->rle_slices_cap, (size_t)2 * nz + 1))
        return mcg_cuda_fail(ctx, cudaErrorMemoryAllocation);
    auto scratch = [&]() {  // for `per` slices, fewer where that cannot be had
        while (!ensure(&ctx->rle_chunks, &ctx->rle_chunks_cap, (size_t)(per * nchunks) * sizeof(RleChunk)) ||
               !ensure(&ctx->rle_marks, &ctx->rle_marks_cap, (size_t)(per * nchunks * cwords))) {
            cudaGetLastError();
            if (per == 1) return false;
            per = (per + 1) / 2;
        }
        return true;
    };
    if (!scratch()) return mcg_cuda_fail(ctx, cudaErrorMemoryAllocation);
    unsigned long long *d_bytes = ctx->rle_slices, *d_off = ctx->rle_slices + nz;
    const uint32_t *v = static_cast<const uint32_t *>(vol);
    const int vec = ((reinterpret_cast<uintptr_t>(vol) & 15u) == 0 && xy % 4 == 0) ? 1 : 0;
    const int ll = lossless ? 1 : 0;
    // passes 1 and 2 of the slices from z on
    auto mark = [&](long long z, long long n) {
        RleChunk *chunks = reinterpret_cast<RleChunk *>(ctx->rle_chunks);
        rle_mark<<<(unsigned int)(n * nchunks), RT, 0, s>>>(v + z * xy, (int)xy, (int)nchunks, ll, chunks, ctx->rle_marks,
                                                            cwords, vec);
        rle_place<<<(unsigned int)n, 32, 0, s>>>(v + z * xy, (int)xy, (int)nchunks, ll, chunks, d_bytes + z);
    };
    for (long long z = 0; z < nz; z += per) mark(z, std::min(per, nz - z));
    rle_slices<<<1, RT, 0, s>>>(d_bytes, nz, d_off);
    e = cudaGetLastError();
    if (e != cudaSuccess) return mcg_cuda_fail(ctx, e);
    bool again = false;  // the marks are not there any more
    auto emit = [&]() {
        for (long long z = 0; z < nz; z += per) {
            const long long n = std::min(per, nz - z);
            if (again || per < nz) mark(z, n);
            rle_emit<<<(unsigned int)(n * nchunks), ET, 0, s>>>(v + z * xy, (int)xy, (int)nchunks, ll,
                                                                reinterpret_cast<RleChunk *>(ctx->rle_chunks),
                                                                ctx->rle_marks, cwords, d_bytes + z, d_off + z,
                                                                ctx->rle_image);
        }
    };
    // a small volume's records are written before its size is known
    bool ahead = !query && per == nz && mcg_rle_bound(nx, ny, nz) <= RAHEAD;
    if (ahead && !ensure(&ctx->rle_image, &ctx->rle_image_cap, (size_t)mcg_rle_bound(nx, ny, nz))) {
        cudaGetLastError();
        ahead = false;
    }
    if (ahead) {
        emit();
        e = cudaGetLastError();
        if (e != cudaSuccess) return mcg_cuda_fail(ctx, e);
    }
    unsigned long long o = 0;
    e = cudaMemcpyAsync(&o, d_off + nz, sizeof(o), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return mcg_cuda_fail(ctx, e);
    if (query || (long long)o > capacity) {
        *size = (int64_t)o;
        return query ? MCG_OK : MCG_ERR_CAPACITY;
    }
    if (!ahead) {
        if (!ensure(&ctx->rle_image, &ctx->rle_image_cap, (size_t)o)) {
            // the image before the scratch, then what is left for that
            cudaGetLastError();
            cudaFree(ctx->rle_chunks);
            cudaFree(ctx->rle_marks);
            ctx->rle_chunks = nullptr;
            ctx->rle_marks = nullptr;
            ctx->rle_chunks_cap = ctx->rle_marks_cap = 0;
            if (!ensure(&ctx->rle_image, &ctx->rle_image_cap, (size_t)o) || !scratch())
                return mcg_cuda_fail(ctx, cudaErrorMemoryAllocation);
            again = true;
        }
        emit();
        e = cudaGetLastError();
        if (e != cudaSuccess) return mcg_cuda_fail(ctx, e);
    }
    // header (:1303-1310), then the slices
    memcpy(image, lossless ? kTagLossless : kTagRef, 16);
    const int32_t dims[3] = {nx, ny, nz};
    memcpy(image + 16, dims, 12);
    memcpy(image + 28, &min_t, 4);
    memcpy(image + 32, &max_t, 4);
    memcpy(image + 36, &grid_s, 4);
    e = cudaMemcpyAsync(image + 40, ctx->rle_image + 40, o - 40, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return mcg_cuda_fail(ctx, e);
    *size = (int64_t)o;
    return MCG_OK;
}
