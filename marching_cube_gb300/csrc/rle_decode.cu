// Run-length volume decoder on sm_103a (cu_kinect_fusion_v1.cu:1419-1447 per
// slice, :1533-1600 per file).
//
// Only the compressed image crosses the host link: it is copied to the
// device in slabs of whole slices on a copy stream while earlier slabs
// expand (from a file: pieces read by host threads into pinned buffers while
// the GPU copies and expands the pieces before).  One CTA expands 4096 16-bit
// words of a z-slice (and further ones what is beyond each RD_PART voxels):
//  * every word is a record header, or the first or second word of a
//    literal; which one follows from the words before it through a
//    three-state machine (header -> header, or -> literal 1 for kinds 0 and
//    3; literal 1 -> literal 2 -> header).  Each thread composes the state
//    maps of its 16 words and a block scan of the compositions, from the
//    chunk's entry state (rle_summarize, rle_slice_scan), gives every word its
//    state;
//  * a block scan of the run lengths of the headers places each run in the
//    slice; runs go to shared memory as (start, voxel);
//  * the chunk's voxels are written by all threads, 16 bytes at a time, each
//    voxel's run found by counting the run starts up to it.
// The slice is full once its voxels are placed; records after that are
// ignored.  A record that is needed and has length 0, runs past the slice
// or lacks its literal, or a stream that ends early, is an error
// (MCG_ERR_FORMAT), exactly the checks of the host decoder.
#include <cuda_runtime.h>
#include <errno.h>
#include <fcntl.h>
#include <stdint.h>
#include <string.h>
#include <sys/stat.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <thread>
#include <vector>

#include "mcg_internal.h"

namespace mcg {
namespace {

constexpr int RD_THREADS = 256;
constexpr int RD_WPT = 16;                     // words per thread
constexpr int RD_CHUNK = RD_THREADS * RD_WPT;  // words per chunk
constexpr unsigned RD_ID = 0u | (1u << 2) | (2u << 4);  // identity state map

// state maps: 2 bits per entry state (0 header, 1 literal word 1, 2 literal word 2)
__device__ __forceinline__ unsigned rd_apply(unsigned f, unsigned s) { return (f >> (2 * s)) & 3u; }
__device__ __forceinline__ unsigned rd_then(unsigned a, unsigned b) {  // a, then b
    return rd_apply(b, rd_apply(a, 0)) | (rd_apply(b, rd_apply(a, 1)) << 2) | (rd_apply(b, rd_apply(a, 2)) << 4);
}
__device__ __forceinline__ unsigned rd_word_map(unsigned w) {
    const unsigned kind = w >> 14;
    return ((kind == 0u || kind == 3u) ? 1u : 0u) | (2u << 2);  // header -> literal 1 / header; 1 -> 2; 2 -> 0
}

// exclusive block scan of a value under an associative op; returns the
// exclusive prefix, *total the block total
template <class T, class Op>
__device__ __forceinline__ T rd_block_scan(T v, T id, Op op, T *s_w, T *total) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    T inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const T u = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc = op(u, inc);
    }
    T ex = __shfl_up_sync(0xffffffffu, inc, 1);
    if (lane == 0) ex = id;
    if (lane == 31) s_w[wid] = inc;
    __syncthreads();
    T pre = id, all = id;
#pragma unroll
    for (int i = 0; i < RD_THREADS / 32; ++i) {
        if (i < wid) pre = op(pre, s_w[i]);
        all = op(all, s_w[i]);
    }
    __syncthreads();
    *total = all;
    return op(pre, ex);
}

__device__ __forceinline__ uint32_t rd_pack(unsigned tsdf16, unsigned w16) { return (tsdf16 & 0xffffu) | (w16 << 16); }

// ---- chunk-parallel expansion ---------------------------------------------
// A chunk is RD_CHUNK words of one slice.  Its summary holds, for each state
// the chunk may be entered in, the state it leaves in (the map f) and the
// voxels its headers emit; summaries compose associatively, so a scan along
// the slice gives every chunk its entry state and first voxel.

struct Sum {
    unsigned f;
    long long v[3];
};

__device__ __forceinline__ long long sum_pick(const Sum &x, unsigned e) {  // x.v[e] without local memory
    return e == 0u ? x.v[0] : (e == 1u ? x.v[1] : x.v[2]);
}

__device__ __forceinline__ Sum sum_then(const Sum &a, const Sum &b) {
    Sum r;
    r.f = rd_then(a.f, b.f);
#pragma unroll
    for (int e = 0; e < 3; ++e) r.v[e] = a.v[e] + sum_pick(b, rd_apply(a.f, (unsigned)e));
    return r;
}

__device__ __forceinline__ Sum sum_shfl_up(const Sum &x, int o) {
    Sum r;
    r.f = __shfl_up_sync(0xffffffffu, x.f, o);
#pragma unroll
    for (int e = 0; e < 3; ++e) r.v[e] = __shfl_up_sync(0xffffffffu, x.v[e], o);
    return r;
}

// exclusive block scan of summaries; *total the block's composition
__device__ __forceinline__ Sum sum_block_scan(const Sum &x, Sum *s_w, Sum *total) {
    const Sum id{RD_ID, {0, 0, 0}};
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    Sum inc = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const Sum u = sum_shfl_up(inc, o);
        if (lane >= o) inc = sum_then(u, inc);
    }
    Sum ex = sum_shfl_up(inc, 1);
    if (lane == 0) ex = id;
    if (lane == 31) s_w[wid] = inc;
    __syncthreads();
    Sum pre = id, all = id;
#pragma unroll
    for (int i = 0; i < RD_THREADS / 32; ++i) {
        if (i < wid) pre = sum_then(pre, s_w[i]);
        all = sum_then(all, s_w[i]);
    }
    __syncthreads();
    *total = all;
    return sum_then(pre, ex);
}

struct Dir {
    const long long *off, *len;  // byte range of each slice's records in the image
    const long long *cbase;      // first chunk of each slice (one entry more than slices)
    int z0, z1;                  // the slab: only its entries, and cbase[z1], are there yet
};

// slice of chunk c of the slab, and its words [c0, c0 + cw) of nw
__device__ __forceinline__ void rd_chunk(const Dir &d, long long c, int *z, long long *c0, int *cw, long long *nw) {
    // the slab's last slice with cbase <= c (cbase[z0] <= c): 32 probes a step.
    // Entries past the slab may be another image's (a file's directory comes
    // piece by piece), so they are not looked at.
    const int lane = threadIdx.x & 31;
    int lo = d.z0, n = d.z1 - d.z0;
    while (n > 1) {
        const int step = (n + 31) / 32, i = lane * step;
        const unsigned m = __ballot_sync(0xffffffffu, i < n && d.cbase[lo + i] <= c);
        const int at = (31 - __clz(m)) * step;
        lo += at;
        n = min(step, n - at);
    }
    *z = lo;
    *nw = d.len[lo] / 2;
    *c0 = (c - d.cbase[lo]) * RD_CHUNK;
    *cw = (int)min((long long)RD_CHUNK, *nw - *c0);
}

// the chunk's words (+2 past its end for a literal that straddles it) into W,
// zeros after them.  The chunk starts at any byte: 16-byte pieces are read
// from the aligned address below it and shifted into place; only pieces
// holding kept words are read, which stay within 32 bytes past the slice's
// bytes (the image buffer has 64 bytes of slack after the image).
__device__ __forceinline__ void rd_load(const uint8_t *__restrict__ img, const Dir &d, int z, long long c0, int cw,
                                        long long nw, uint16_t *W) {
    const uint8_t *first = img + d.off[z] + 2 * c0;
    const uint4 *p = reinterpret_cast<const uint4 *>((uintptr_t)first & ~(uintptr_t)15);
    const unsigned sh = (unsigned)((uintptr_t)first & 15);
    const unsigned q = sh >> 2, r = 8u * (sh & 3u);
    const long long lim = min((long long)cw + 2, nw - c0);  // words to keep
    constexpr int PIECES = (RD_CHUNK + 8) / 8;                // 8 words per piece
    const long long loaded = (lim + 7) / 8;                   // pieces holding kept words
    for (int j = threadIdx.x; j < PIECES; j += RD_THREADS) {
        if (j >= loaded) {  // nothing to keep: no read past the slice's bytes
            reinterpret_cast<uint4 *>(W)[j] = make_uint4(0, 0, 0, 0);
            continue;
        }
        const uint4 lo = __ldg(p + j), hi = __ldg(p + j + 1);
        const unsigned x[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
        unsigned o[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            // words k+q and k+q+1 of x without a dynamic register index
            const unsigned a = q == 0 ? x[k] : q == 1 ? x[k + 1] : q == 2 ? x[k + 2] : x[k + 3];
            const unsigned b = q == 0 ? x[k + 1] : q == 1 ? x[k + 2] : q == 2 ? x[k + 3] : x[k + 4];
            o[k] = __funnelshift_r(a, b, r);
        }
        const long long w0 = 8ll * j;  // first word of the piece
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (w0 + 2 * k >= lim) o[k] = 0;
            else if (w0 + 2 * k + 1 >= lim) o[k] &= 0xffffu;
        }
        reinterpret_cast<uint4 *>(W)[j] = make_uint4(o[0], o[1], o[2], o[3]);
    }
    __syncthreads();
}

// this thread's 16 words and the 2 after them, from shared memory into
// registers with two 16-byte loads (conflict-free) and one 4-byte load
__device__ __forceinline__ void rd_words(const uint16_t *W, int b, unsigned w[RD_WPT + 2]) {
    const uint4 *p = reinterpret_cast<const uint4 *>(W + b);
#pragma unroll
    for (int i = 0; i < RD_WPT / 8; ++i) {
        const uint4 a = p[i];
        const unsigned x[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            w[8 * i + 2 * k] = x[k] & 0xffffu;
            w[8 * i + 2 * k + 1] = x[k] >> 16;
        }
    }
    const unsigned t = *reinterpret_cast<const unsigned *>(W + b + RD_WPT);
    w[RD_WPT] = t & 0xffffu;
    w[RD_WPT + 1] = t >> 16;
}

// A thread's words (nk of them), entered in each state: the state it leaves
// in, its headers and their voxels, as state | headers << 2 | voxels << 8.
// From the last word to the first (walking each of the three entry states for
// itself, with 64-bit voxel counts, rle_summarize took 51 us for 26 MB; now 27):
// a header's walk is that of the word after
// its record and its own, and entry state 1 (two literal words left) starts at
// word 2, state 2 at word 1.
__device__ __forceinline__ void rd_walk(const unsigned *w, int nk, unsigned t[3]) {
    // words past the end: 0, 1 or 2 literal words of the next thread's left
    unsigned f[RD_WPT + 3];
#pragma unroll
    for (int k = RD_WPT + 2; k >= 0; --k) {
        if (k < RD_WPT && k < nk) {
            const unsigned kind = w[k] >> 14;
            f[k] = (kind == 0u || kind == 3u ? f[k + 3] : f[k + 1]) + ((w[k] & 0x3fffu) << 8 | 4u);
        } else {
            f[k] = k == nk ? 0u : k == nk + 1 ? 2u : 1u;
        }
    }
    t[0] = f[0];
    t[1] = f[2];
    t[2] = f[1];
}

// pass 1: summaries of chunks c0 + blockIdx.x
__global__ void __launch_bounds__(RD_THREADS) rle_summarize(const uint8_t *__restrict__ img, Dir d, long long cfirst,
                                                            Sum *__restrict__ sums) {
    __shared__ __align__(16) uint16_t W[RD_CHUNK + 8];
    __shared__ Sum s_w[RD_THREADS / 32];
    const long long c = cfirst + blockIdx.x;
    int z, cw;
    long long c0, nw;
    rd_chunk(d, c, &z, &c0, &cw, &nw);
    rd_load(img, d, z, c0, cw, nw, W);
    const int b = threadIdx.x * RD_WPT, nk = max(0, min(cw, b + RD_WPT) - b);
    unsigned w[RD_WPT + 2];
    rd_words(W, b, w);
    unsigned wk[3], f = 0, v[3];
    rd_walk(w, nk, wk);
#pragma unroll
    for (int e = 0; e < 3; ++e) {
        f |= (wk[e] & 3u) << (2 * e);
        v[e] = wk[e] >> 8;
    }
    // composed in order over the warp, then over the warps (a chunk's voxels fit 32 bits)
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned fb = __shfl_down_sync(0xffffffffu, f, o), v0 = __shfl_down_sync(0xffffffffu, v[0], o),
                       v1 = __shfl_down_sync(0xffffffffu, v[1], o), v2 = __shfl_down_sync(0xffffffffu, v[2], o);
#pragma unroll
        for (int e = 0; e < 3; ++e) {
            const unsigned at = rd_apply(f, (unsigned)e);
            v[e] += at == 0u ? v0 : at == 1u ? v1 : v2;
        }
        f = rd_then(f, fb);
    }
    if (lane == 0) s_w[wid] = Sum{f, {(long long)v[0], (long long)v[1], (long long)v[2]}};
    __syncthreads();
    if (threadIdx.x == 0) {
        Sum total = s_w[0];
#pragma unroll
        for (int i = 1; i < RD_THREADS / 32; ++i) total = sum_then(total, s_w[i]);
        sums[c] = total;
    }
}

// A chunk of few records can hold a slice of voxels (16383 a record; 512^3
// voxels of a scene: 3517 chunks of 38162 voxels on average, 254 of 262144),
// so a chunk's voxels beyond the first RD_PART are expanded by CTAs of their
// own, RD_PART each.  A slice has room for (xy - 1) / RD_PART of these: one
// that would start at voxel s is entry s / RD_PART - 1, its own since those of
// a chunk start RD_PART apart and the next chunk's begin at least RD_PART
// after the chunk's end.  rle_expand there: 163 us without, 144 with parts of
// 65536, 158 with parts of 32768 (the steps before a part's voxels are repeated).
constexpr int RD_PART = 65536;

// pass 2: one CTA per slice z0 + blockIdx.x: entry state and first voxel of
// each of its chunks, and its parts (chunk << 16 | part, or -1); a slice whose records end before it is full is an error
__global__ void __launch_bounds__(RD_THREADS) rle_slice_scan(Dir d, int z0, long long xy,
                                                             const Sum *__restrict__ sums,
                                                             unsigned char *__restrict__ entry,
                                                             long long *__restrict__ first,
                                                             long long *__restrict__ parts, int *__restrict__ err) {
    __shared__ Sum s_w[RD_THREADS / 32];
    const int z = z0 + blockIdx.x;
    const long long cb = d.cbase[z], ce = d.cbase[z + 1];
    unsigned state = 0;
    long long out = 0;
    const long long np = (xy - 1) / RD_PART;
    parts += z * np;
    for (long long i = threadIdx.x; i < np; i += RD_THREADS) parts[i] = -1;
    for (long long k = cb; k < ce; k += RD_THREADS) {
        const long long c = k + threadIdx.x;
        const Sum x = c < ce ? sums[c] : Sum{RD_ID, {0, 0, 0}};
        Sum total;
        const Sum pre = sum_block_scan(x, s_w, &total);  // (a barrier between parts[] = -1 and its entries)
        if (c < ce) {
            const unsigned en = rd_apply(pre.f, state);
            const long long a = out + sum_pick(pre, state), b = min(xy, a + sum_pick(x, en));
            entry[c] = (unsigned char)en;
            first[c] = a;
            for (long long s = a + RD_PART, p = 1; s < b; s += RD_PART, ++p) parts[s / RD_PART - 1] = c << 16 | p;
        }
        out += sum_pick(total, state);
        state = rd_apply(total.f, state);
    }
    if (threadIdx.x == 0 && out < xy) atomicOr(err, 1);
}

// Voxels [out, end) of a slice from the chunk's runs (rs: starts counted from
// `out`, rv: voxels from rv[1] on, n of them), RD_TILE voxels at a time: a bit is set where a
// run starts, the set bits before each 32-bit word are counted, and a voxel's
// run is the number of bits up to its own.  Each lane writes four consecutive
// voxels, 16 bytes.  Bound: the instructions of this, then writing the volume.
// Expanding 512^3 voxels from 26 MB: a binary search over the chunk's runs for
// each voxel took 967 us, for each four voxels between those of a warp's ends
// 431 us; this 171 us, 144 with long chunks in parts, 135 with the words and
// bits of a full tile's voxels at fixed places and one look-up where no run
// starts inside the four, 132 with six CTAs per SM instead of five.
constexpr int RD_TILE = 16384;

struct RunTile {
    uint32_t start[RD_TILE / 32];  // bit: a run starts at this voxel
    int before[RD_TILE / 32];      // runs that start before the word's first voxel
    int w[RD_THREADS / 32];
};

__device__ __forceinline__ void rd_write_runs(RunTile &S, uint32_t *__restrict__ slice, long long out, long long end,
                                              const int *rs, const uint32_t *rv, int n, int part) {
    constexpr int WPT = RD_TILE / 32 / RD_THREADS;  // words per thread
    const int tid = threadIdx.x;
    const int total = (int)(end - out);
    // tiles start on 16-byte boundaries: the first one at or below `out`
    const int lead = (int)((reinterpret_cast<uintptr_t>(slice + out) >> 2) & 3u);
    // this part's voxels; the last one takes what is left
    const int first = part * RD_PART - lead;
    const int last = (part + 1) * (long long)RD_PART < total ? first + RD_PART : total;
    int base = 0;  // runs that start before the tile
    if (part) {
        int c = 0;
        for (int r = tid; r < n; r += RD_THREADS) c += rs[r] < first;
        rd_block_scan<int>(c, 0, [](int a, int b) { return a + b; }, S.w, &base);
    }
    for (int t0 = first; t0 < last; t0 += RD_TILE) {
        for (int i = tid; i < RD_TILE / 32; i += RD_THREADS) S.start[i] = 0u;
        __syncthreads();
        for (int r = tid; r < n; r += RD_THREADS) {
            const unsigned int p = (unsigned int)(rs[r] - t0);
            if (p < (unsigned int)RD_TILE) atomicOr(&S.start[p >> 5], 1u << (p & 31));
        }
        __syncthreads();
        int c[WPT], sum = 0;
#pragma unroll
        for (int i = 0; i < WPT; ++i) {
            c[i] = sum;
            sum += __popc(S.start[tid * WPT + i]);
        }
        int all;
        const int ex = base + rd_block_scan<int>(sum, 0, [](int a, int b) { return a + b; }, S.w, &all);
#pragma unroll
        for (int i = 0; i < WPT; ++i) S.before[tid * WPT + i] = ex + c[i];
        base += all;
        __syncthreads();
        const int stop = min(RD_TILE, last - t0);
        // four voxels a thread and step, at the same bits of their words every time
        const int bit = (4 * tid) & 31;
        const uint32_t below = (1u << bit) - 1u;
        auto four = [&](int p) -> uint4 {
            const uint32_t word = S.start[p >> 5], f = word >> bit;
            const uint32_t *v = rv + S.before[p >> 5] + __popc(word & below);
            if (f & 1u) ++v;
            uint4 q;
            q.x = q.y = q.z = q.w = v[0];
            if (f & 14u) {
                if (f & 2u) ++v;
                q.y = v[0];
                if (f & 4u) ++v;
                q.z = v[0];
                if (f & 8u) ++v;
                q.w = v[0];
            }
            return q;
        };
        uint32_t *dst = slice + out + t0;  // (not below the slice's buffer where it is written)
        if (t0 >= 0 && stop == RD_TILE) {
#pragma unroll 4
            for (int i = 0; i < RD_TILE / (4 * RD_THREADS); ++i) {
                const int p = 4 * tid + 4 * RD_THREADS * i;
                *reinterpret_cast<uint4 *>(dst + p) = four(p);
            }
        } else {
            for (int p = 4 * tid; p < stop; p += 4 * RD_THREADS) {
                const uint4 q = four(p);
                const uint32_t w[4] = {q.x, q.y, q.z, q.w};
                const int v = t0 + p;
                if (v >= 0 && v + 4 <= total) {
                    *reinterpret_cast<uint4 *>(dst + p) = q;
                } else {
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (v + k >= 0 && v + k < total) dst[p + k] = w[k];
                }
            }
        }
        __syncthreads();
    }
}

// pass 3: expand chunks cfirst + blockIdx.x, and the parts after them
__global__ void __launch_bounds__(RD_THREADS, 6) rle_expand(const uint8_t *__restrict__ img, Dir d, long long cfirst,
                                                         long long xy, const unsigned char *__restrict__ entry_of,
                                                         const long long *__restrict__ first_of,
                                                         const long long *__restrict__ parts, long long nc,
                                                         uint32_t *__restrict__ vol, int *__restrict__ err) {
    __shared__ union {
        __align__(16) uint16_t W[RD_CHUNK + 8];  // until every thread has its words
        int rs[RD_CHUNK];
    } U;
    uint16_t *const W = U.W;
    int *const rs = U.rs;
    __shared__ uint32_t rv[RD_CHUNK + 1];  // run r's voxel at r + 1; 0: voxels below `out`, not written
    __shared__ RunTile S;
    __shared__ unsigned s_f[RD_THREADS / 32];
    __shared__ unsigned long long s_l[RD_THREADS / 32];
    long long c = cfirst + blockIdx.x;
    int part = 0;
    if (blockIdx.x >= nc) {
        const long long i = parts[blockIdx.x - nc];
        if (i < 0) return;
        c = i >> 16;
        part = (int)(i & 0xffff);
    }
    const long long out = first_of[c], n = xy;
    if (out >= n) return;  // records after a full slice are ignored
    int z, cw;
    long long c0, nw;
    rd_chunk(d, c, &z, &c0, &cw, &nw);
    rd_load(img, d, z, c0, cw, nw, W);
    const unsigned state = entry_of[c];
    uint32_t *out_slice = vol + (long long)z * xy;
    bool bad = false;
    const int b = threadIdx.x * RD_WPT, nk = max(0, min(cw, b + RD_WPT) - b);
    unsigned w[RD_WPT + 2];
    rd_words(W, b, w);
    unsigned wk3[3];
    rd_walk(w, nk, wk3);
    unsigned fall;
    const unsigned fpre = rd_block_scan<unsigned>((wk3[0] & 3u) | (wk3[1] & 3u) << 2 | (wk3[2] & 3u) << 4, RD_ID,
                                                  [](unsigned a, unsigned c2) { return rd_then(a, c2); }, s_f, &fall);
    const unsigned entry = rd_apply(fpre, state);
    const unsigned own = entry == 0u ? wk3[0] : entry == 1u ? wk3[1] : wk3[2];
    // records and voxels before this thread's, in one scan
    unsigned long long tot;
    const unsigned long long pre = rd_block_scan<unsigned long long>(
        (unsigned long long)(own >> 8) << 32 | ((own >> 2) & 63u), 0ull,
        [](unsigned long long a, unsigned long long c2) { return a + c2; }, s_l, &tot);
    const int rtot = (int)(unsigned int)tot;
    const long long vtot = (long long)(tot >> 32);
    unsigned s = entry;
    int r = (int)(unsigned int)pre;
    long long o = (long long)(pre >> 32);
#pragma unroll
    for (int k = 0; k < RD_WPT; ++k) {
        if (k < nk) {
            const unsigned wk = w[k];
            if (s == 0u) {
                const unsigned cnt = wk & 0x3fff, kind = wk >> 14;
                uint32_t val;
                bool lit_ok = true;
                if (kind == 1u) {
                    val = rd_pack((unsigned)kMaxTsdf, 0u);
                } else if (kind == 2u) {
                    val = rd_pack((unsigned)(-kMaxTsdf), 0u);
                } else {
                    lit_ok = c0 + b + k + 2 < nw;
                    val = rd_pack(w[k + 1], w[k + 2]);
                }
                const long long start = out + o;
                if (start < n && (cnt == 0u || start + (long long)cnt > n || !lit_ok)) bad = true;
                rs[r] = (int)min(o, (long long)INT32_MAX);
                rv[r + 1] = val;
                ++r;
                o += cnt;
            }
            s = rd_apply(rd_word_map(wk), s);
        }
    }
    if (threadIdx.x == 0) rv[0] = 0u;
    __syncthreads();
    const long long end = min(n, out + vtot);
    rd_write_runs(S, out_slice, out, end, rs, rv, rtot, part);
    if (bad) atomicOr(err, 1);
}

struct Slab {
    int z0, z1;      // slices
    int64_t b0, b1;  // image bytes that hold them (b0 = end of the previous slab)
};

// The three passes over slices [z0, z1), once the stream s has their bytes
// and their directory entries (offsets, lengths, chunk bases).
cudaError_t launch_expand(mcg_context *ctx, const Slab &sl, const long long *cbase_host, int64_t xy, void *vol,
                          cudaStream_t s) {
    if (sl.z1 <= sl.z0) return cudaSuccess;
    const int nz = ctx->rd_dir_n;
    const Dir d{ctx->rd_dir, ctx->rd_dir + nz, ctx->rd_dir + 2 * nz, sl.z0, sl.z1};
    const long long cf = cbase_host[sl.z0], nc = cbase_host[sl.z1] - cf;
    Sum *sums = reinterpret_cast<Sum *>(ctx->rd_sum);
    unsigned char *entry = ctx->rd_entry;
    const long long np = (xy - 1) / RD_PART;  // parts a slice
    if (nc > 0) rle_summarize<<<(unsigned)nc, RD_THREADS, 0, s>>>(ctx->rle_image, d, cf, sums);
    rle_slice_scan<<<sl.z1 - sl.z0, RD_THREADS, 0, s>>>(d, sl.z0, xy, sums, entry, ctx->rd_first, ctx->rd_parts,
                                                         ctx->rd_err);
    if (nc > 0)
        rle_expand<<<(unsigned)(nc + (sl.z1 - sl.z0) * np), RD_THREADS, 0, s>>>(
            ctx->rle_image, d, cf, xy, entry, ctx->rd_first, ctx->rd_parts + sl.z0 * np, nc,
            static_cast<uint32_t *>(vol), ctx->rd_err);
    return cudaGetLastError();
}

constexpr int64_t RD_SLAB = (int64_t)64 << 20;  // image bytes per copy

// device buffers for an image of `size` bytes and nz slices: the image, the
// directory (offsets, lengths, chunk bases) and the per-chunk arrays; xy >= 1
mcg_status prepare(mcg_context *ctx, int64_t xy, int nz, int64_t size) {
    const size_t chunks = (size_t)(size / (2 * RD_CHUNK)) + (size_t)nz + 1;  // bounds the chunks of any image
    if (!ensure(&ctx->rle_image, &ctx->rle_image_cap, (size_t)size + 64) ||
        !ensure(&ctx->rd_dir, &ctx->rd_dir_cap, 3 * (size_t)nz + 1) || !ensure(&ctx->rd_err, &ctx->rd_err_cap, 1) ||
        !ensure(&ctx->rd_sum, &ctx->rd_sum_cap, chunks * sizeof(Sum)) ||
        !ensure(&ctx->rd_first, &ctx->rd_first_cap, chunks) ||
        !ensure(&ctx->rd_parts, &ctx->rd_parts_cap, (size_t)((xy - 1) / RD_PART) * nz) ||
        !ensure(&ctx->rd_entry, &ctx->rd_entry_cap, chunks))
        return mcg_cuda_fail(ctx, cudaErrorMemoryAllocation);
    ctx->rd_dir_n = nz;
    return MCG_OK;
}

// chunks of a slice of len record bytes
inline long long slice_chunks(long long len) { return (len / 2 + RD_CHUNK - 1) / RD_CHUNK; }

mcg_status finish(mcg_context *ctx, cudaStream_t s) {
    int h_err = 0;
    cudaError_t e = cudaMemcpyAsync(&h_err, ctx->rd_err, sizeof(int), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return mcg_cuda_fail(ctx, e);
    return h_err ? MCG_ERR_FORMAT : MCG_OK;
}

bool pread_full(int fd, uint8_t *dst, int64_t n, int64_t off) {
    while (n > 0) {
        const ssize_t r = pread(fd, dst, (size_t)std::min<int64_t>(n, (int64_t)1 << 30), (off_t)off);
        if (r <= 0) {
            if (r < 0 && errno == EINTR) continue;
            return false;
        }
        dst += r;
        off += r;
        n -= r;
    }
    return true;
}

}  // namespace
}  // namespace mcg

using namespace mcg;

extern "C" mcg_status mcg_rle_decode(mcg_context *ctx, const uint8_t *image, int64_t size, void *vol,
                                     int64_t capacity_voxels, mcg_stream_t stream) {
    if (!ctx || !image || !vol) return MCG_ERR_INVALID_ARG;
    int32_t dims[3];
    float params[3];
    mcg_status st = mcg_rle_header(image, size, dims, params);
    if (st != MCG_OK) return st;
    const int64_t xy = (int64_t)dims[0] * dims[1];
    if (xy * dims[2] > capacity_voxels) return MCG_ERR_CAPACITY;
    if (xy > INT32_MAX / 2) return MCG_ERR_TOO_LARGE;
    const int nz = dims[2];
    std::vector<long long> dir(3 * (size_t)nz + 1);  // offsets, lengths, chunk bases
    long long *cbase = dir.data() + 2 * (size_t)nz;
    int64_t p = 40;
    cbase[0] = 0;
    for (int z = 0; z < nz; ++z) {
        if (p + 4 > size) return MCG_ERR_FORMAT;
        uint32_t s32;
        memcpy(&s32, image + p, 4);
        p += 4;
        if (p + (int64_t)s32 > size) return MCG_ERR_FORMAT;
        dir[z] = p;
        dir[nz + z] = s32;
        cbase[z + 1] = cbase[z] + slice_chunks(s32);
        p += s32;
    }
    cudaError_t e = cudaSetDevice(ctx->device);
    if (e != cudaSuccess) return mcg_cuda_fail(ctx, e);
    if ((st = prepare(ctx, xy, nz, p)) != MCG_OK) return st;
    const cudaStream_t s = (cudaStream_t)stream;
    if ((e = cudaMemsetAsync(ctx->rd_err, 0, sizeof(int), s)) != cudaSuccess ||
        (e = cudaMemcpyAsync(ctx->rd_dir, dir.data(), dir.size() * sizeof(long long), cudaMemcpyHostToDevice, s)) !=
            cudaSuccess)
        return mcg_cuda_fail(ctx, e);
    // slabs of whole slices: each copied on a copy stream, then expanded on
    // s while the next slab copies
    cudaStream_t cs = nullptr;
    std::vector<cudaEvent_t> evs;
    auto done = [&](mcg_status r) {
        if (cs) cudaStreamSynchronize(cs);
        cudaStreamSynchronize(s);  // the directory copy reads dir
        for (auto ev : evs) cudaEventDestroy(ev);
        if (cs) cudaStreamDestroy(cs);
        return r;
    };
    cudaEvent_t ev = nullptr;
    if ((e = cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking)) != cudaSuccess) {
        cs = nullptr;
        return done(mcg_cuda_fail(ctx, e));
    }
    auto new_event = [&]() -> cudaError_t {
        const cudaError_t r = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
        if (r == cudaSuccess) evs.push_back(ev);
        return r;
    };
    // the copies wait for earlier work on s (an earlier decode reads the image buffer)
    if ((e = new_event()) != cudaSuccess || (e = cudaEventRecord(ev, s)) != cudaSuccess ||
        (e = cudaStreamWaitEvent(cs, ev, 0)) != cudaSuccess)
        return done(mcg_cuda_fail(ctx, e));
    Slab sl{0, 0, 0, 0};
    while (sl.z1 < nz) {
        sl.z0 = sl.z1;
        sl.b0 = sl.b1;
        while (sl.z1 < nz && (sl.z1 == sl.z0 || dir[sl.z1] + dir[nz + sl.z1] - sl.b0 <= RD_SLAB)) ++sl.z1;
        sl.b1 = dir[sl.z1 - 1] + dir[nz + sl.z1 - 1];
        if ((e = cudaMemcpyAsync(ctx->rle_image + sl.b0, image + sl.b0, (size_t)(sl.b1 - sl.b0),
                                 cudaMemcpyHostToDevice, cs)) != cudaSuccess ||
            (e = new_event()) != cudaSuccess || (e = cudaEventRecord(ev, cs)) != cudaSuccess ||
            (e = cudaStreamWaitEvent(s, ev, 0)) != cudaSuccess ||
            (e = launch_expand(ctx, sl, cbase, xy, vol, s)) != cudaSuccess)
            return done(mcg_cuda_fail(ctx, e));
    }
    return done(finish(ctx, s));
}

extern "C" mcg_status mcg_rle_decode_file(mcg_context *ctx, const char *path, void *vol, int64_t capacity_voxels,
                                          int32_t dims[3], float params[3], mcg_stream_t stream) {
    if (!ctx || !path || !vol || !dims || !params) return MCG_ERR_INVALID_ARG;
    const int fd = open(path, O_RDONLY);
    if (fd < 0) return MCG_ERR_IO;
    struct stat sb;
    uint8_t head[40];
    if (fstat(fd, &sb) != 0 || !pread_full(fd, head, std::min<int64_t>(40, (int64_t)sb.st_size), 0)) {
        close(fd);
        return MCG_ERR_IO;
    }
    const int64_t size = (int64_t)sb.st_size;
    mcg_status st = mcg_rle_header(head, size, dims, params);
    const int64_t xy = (int64_t)dims[0] * dims[1];
    if (st == MCG_OK && xy * dims[2] > capacity_voxels) st = MCG_ERR_CAPACITY;
    if (st == MCG_OK && xy > INT32_MAX / 2) st = MCG_ERR_TOO_LARGE;
    cudaError_t e = cudaSuccess;
    if (st == MCG_OK && (e = cudaSetDevice(ctx->device)) != cudaSuccess) st = mcg_cuda_fail(ctx, e);
    const int nz = dims[2];
    if (st == MCG_OK) st = prepare(ctx, xy, nz, size);
    if (st == MCG_OK && !ctx->h_rd_stage) {
        if (cudaMallocHost((void **)&ctx->h_rd_stage, 2 * (size_t)RD_SLAB) != cudaSuccess) {
            ctx->h_rd_stage = nullptr;
            st = mcg_cuda_fail(ctx, cudaErrorMemoryAllocation);
        }
    }
    if (st != MCG_OK) {
        close(fd);
        return st;
    }
    const cudaStream_t s = (cudaStream_t)stream;
    cudaEvent_t copied[2] = {nullptr, nullptr};
    std::vector<long long> dir(3 * (size_t)nz + 1, 0);  // offsets, lengths, chunk bases
    long long *cbase = dir.data() + 2 * (size_t)nz;
    for (int b = 0; b < 2 && st == MCG_OK; ++b)
        if ((e = cudaEventCreateWithFlags(&copied[b], cudaEventDisableTiming)) != cudaSuccess) st = mcg_cuda_fail(ctx, e);
    if (st == MCG_OK && (e = cudaMemsetAsync(ctx->rd_err, 0, sizeof(int), s)) != cudaSuccess) st = mcg_cuda_fail(ctx, e);
    // Pieces of RD_SLAB bytes are read by host threads into two pinned
    // buffers and copied on s; the directory is walked in the host copy as
    // pieces arrive, and the slices that end inside the resident bytes are
    // expanded after each piece.
    int z_walk = 0, z_done = 0;
    int64_t p = 40;          // next slice byte count
    uint8_t cnt_buf[4];      // a count split across two pieces
    int cnt_have = 0;
    const int hw = (int)std::max(1u, std::thread::hardware_concurrency());
    for (int64_t b0 = 0, piece = 0; st == MCG_OK && b0 < size; b0 += RD_SLAB, ++piece) {
        const int64_t n = std::min<int64_t>(RD_SLAB, size - b0);
        uint8_t *buf = ctx->h_rd_stage + (size_t)(piece & 1) * RD_SLAB;
        if (piece >= 2 && (e = cudaEventSynchronize(copied[piece & 1])) != cudaSuccess) {
            st = mcg_cuda_fail(ctx, e);
            break;
        }
        const int nt = (int)std::min<int64_t>(std::min(16, hw), (n + (1 << 20) - 1) >> 20);
        std::atomic<int> ok{1};
        std::vector<std::thread> pool;
        const int64_t part = (n + nt - 1) / nt;
        for (int t = 0; t < nt; ++t) {
            const int64_t a = t * part, c = std::min(n, a + part);
            if (a >= c) break;
            pool.emplace_back([&, a, c]() {
                if (!pread_full(fd, buf + a, c - a, b0 + a)) ok.store(0);
            });
        }
        for (auto &th : pool) th.join();
        if (!ok.load()) {
            st = MCG_ERR_IO;
            break;
        }
        if ((e = cudaMemcpyAsync(ctx->rle_image + b0, buf, (size_t)n, cudaMemcpyHostToDevice, s)) != cudaSuccess ||
            (e = cudaEventRecord(copied[piece & 1], s)) != cudaSuccess) {
            st = mcg_cuda_fail(ctx, e);
            break;
        }
        // walk the directory through this piece
        const int64_t b1 = b0 + n;
        while (z_walk < nz && p < b1) {
            while (cnt_have < 4 && p + cnt_have < b1) {
                cnt_buf[cnt_have] = buf[p + cnt_have - b0];
                ++cnt_have;
            }
            if (cnt_have < 4) break;  // the count continues in the next piece
            uint32_t s32;
            memcpy(&s32, cnt_buf, 4);
            cnt_have = 0;
            p += 4;
            if (p + (int64_t)s32 > size) {
                st = MCG_ERR_FORMAT;
                break;
            }
            dir[z_walk] = p;
            dir[nz + z_walk] = s32;
            cbase[z_walk + 1] = cbase[z_walk] + slice_chunks(s32);
            p += s32;
            ++z_walk;
        }
        if (st != MCG_OK) break;
        // slices complete in [0, b1): those walked whose bytes end by b1
        int z_ready = z_done;
        while (z_ready < z_walk && dir[z_ready] + dir[nz + z_ready] <= b1) ++z_ready;
        if (z_ready > z_done) {
            if ((e = cudaMemcpyAsync(ctx->rd_dir + z_done, dir.data() + z_done, (size_t)(z_ready - z_done) * 8,
                                     cudaMemcpyHostToDevice, s)) != cudaSuccess ||
                (e = cudaMemcpyAsync(ctx->rd_dir + nz + z_done, dir.data() + nz + z_done,
                                     (size_t)(z_ready - z_done) * 8, cudaMemcpyHostToDevice, s)) != cudaSuccess ||
                (e = cudaMemcpyAsync(ctx->rd_dir + 2 * nz + z_done, cbase + z_done, (size_t)(z_ready - z_done + 1) * 8,
                                     cudaMemcpyHostToDevice, s)) != cudaSuccess) {
                st = mcg_cuda_fail(ctx, e);
                break;
            }
            const Slab sl{z_done, z_ready, 0, 0};
            if ((e = launch_expand(ctx, sl, cbase, xy, vol, s)) != cudaSuccess) {
                st = mcg_cuda_fail(ctx, e);
                break;
            }
            z_done = z_ready;
        }
    }
    if (st == MCG_OK && z_walk < nz) st = MCG_ERR_FORMAT;  // the file ends inside the directory
    mcg_status fin = finish(ctx, s);
    if (st == MCG_OK) st = fin;
    for (int b = 0; b < 2; ++b)
        if (copied[b]) cudaEventDestroy(copied[b]);
    close(fd);
    return st;
}
