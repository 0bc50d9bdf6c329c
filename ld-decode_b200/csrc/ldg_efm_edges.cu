// Zero crossings of the demodulator's EFM output on the GPU: the edges that
// EFM_PLL.process (lddecode/efm_pll.py:124-167) detects one sample at a
// time and feeds to its PLL.  A crossing is a sample whose sign differs
// from the sample before it (negative against not negative); each is kept
// as its position and the two sample values, from which the PLL's
// interpolated fraction -prev / (cur - prev) follows exactly.  With the
// crossings on the host, ldg_efm_pll_process_edges runs the PLL without
// the samples: an EFM stream then crosses PCIe as ~8 bytes per crossing
// (one every ~25 samples of band-limited EFM) instead of 2 bytes per
// sample.
//
// Two streaming launches over the same contiguous chunks, one per resident
// CTA: the first counts each chunk's crossings, the second adds up the counts
// before its chunk and writes its crossings, from the chunk's end to its
// start, whose samples the first left in L2 last.  Bound: HBM, 2 bytes read
// per sample and 8 written per crossing.  80 M samples, B200: 197 us as
// counts, a scan and a second pass with 2-byte loads; 68 us so (2.7 TB/s
// of the 182 MB it has to move).  One pass with decoupled look-back took 80
// us at best: the CTAs of a wave all wait for the wave's slowest load.
#include <stdint.h>

#include <string>

#include "ldg_copy.cuh"
#include "ldgpu.h"

namespace ldg {
int api_fail(int code, const std::string& msg);
}

namespace {

// 128 threads and 16 CTAs per SM: 68 us; 256 and 8: 72, 512 and 4: 77, 1024 and
// 2: 84 (the more CTAs, the less a barrier holds up).
constexpr int kThreads = 128;
constexpr int kTile = 32 * kThreads;    // samples: one 32-bit word of sign flags per thread
constexpr int kMaxChunks = 148 * 16;    // the resident CTAs
// Crossings of a tile above which a warp writes them word by word, not each
// thread its own word's: 80 M samples with a crossing every 4 take 153 us for 194,
// white noise 180 for 537, a crossing every 8 the other way round 146 for 116.
constexpr int kDense = kTile / 6;

size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

// Sample i sits at position i + mis of the tiles, mis the samples x lies past
// a 16-byte boundary, so that any x takes 16-byte loads.

// Eight samples from i on (0 outside [0, n), where In is false), two per word.
template <bool In>
__device__ __forceinline__ uint4 load8(const int16_t* __restrict__ x, long long n, long long i) {
    if (In || (i >= 0 && i + 8 <= n)) return __ldg(reinterpret_cast<const uint4*>(x + i));
    unsigned w[4] = {0, 0, 0, 0};
    for (int k = 0; k < 8; ++k)
        if (i + k >= 0 && i + k < n) w[k >> 1] |= (unsigned)(uint16_t)x[i + k] << (16 * (k & 1));
    return make_uint4(w[0], w[1], w[2], w[3]);
}

constexpr unsigned kSigns = 0x80008000u;

// Sign changes among eight samples, given the word that ends with the sample
// before them.
__device__ __forceinline__ int changes8(uint4 v, unsigned before) {
    const unsigned a = (v.x ^ __funnelshift_l(before, v.x, 16)) & kSigns;
    const unsigned b = (v.y ^ __funnelshift_l(v.x, v.y, 16)) & kSigns;
    const unsigned c = (v.z ^ __funnelshift_l(v.y, v.z, 16)) & kSigns;
    const unsigned d = (v.w ^ __funnelshift_l(v.z, v.w, 16)) & kSigns;
    return __popc(a | (b >> 1) | (c >> 2) | (d >> 3));
}

// Their sign bits, the first sample's in bit 7.
__device__ __forceinline__ unsigned signs8(uint4 v) {
    const unsigned s = (v.x & kSigns) | ((v.y & kSigns) >> 2) | ((v.z & kSigns) >> 4) | ((v.w & kSigns) >> 6);
    return ((s & 0xffffu) | (s >> 17)) >> 8;
}

// Crossings among the tile samples c .. c + 31 (c the tile's, i = t0 + c the
// array's index) from their signs and the sign of the sample before: none
// outside [0, n), and sample 0 against x[-1] (has_before) or against 0.
template <bool In>
__device__ __forceinline__ unsigned crossings32(unsigned f, unsigned before, const int16_t* __restrict__ x, long long n,
                                                long long i, int has_before) {
    unsigned prev = (f << 1) | before;
    if (In) return f ^ prev;
    if (i <= 0 && i + 32 > 0) {
        const unsigned first = 1u << (int)(-i);
        prev = (prev & ~first) | (has_before && x[-1] < 0 ? first : 0u);
    }
    unsigned e = f ^ prev;
    if (i < 0) e &= i <= -32 ? 0u : 0xffffffffu << (int)(-i);
    if (i + 32 > n) e &= i >= n ? 0u : 0xffffffffu >> (int)(i + 32 - n);
    return e;
}

// A chunk's crossings.  A tile whose samples, and the one before, all exist
// compares neighbouring words; the array's first and last tiles go sample by
// sample.
__global__ void __launch_bounds__(kThreads) efm_count_kernel(const int16_t* __restrict__ x, long long n, int mis,
                                                             int has_before, long long ntiles,
                                                             long long* __restrict__ counts) {
    __shared__ int warp_sum[kThreads / 32];
    const int t = threadIdx.x, lane = t & 31;
    const long long g0 = ntiles * blockIdx.x / gridDim.x, g1 = ntiles * (blockIdx.x + 1) / gridDim.x;
    int c = 0;
#pragma unroll 1
    for (long long tile = g0; tile < g1; ++tile) {
        const long long t0 = tile * kTile - mis;
        if (t0 > 0 && t0 + kTile <= n) {
            const int16_t* xt = x + t0 + 8 * t;
            uint4 v[4];
            unsigned ahead[4];  // the word that ends with the sample before the warp's 256
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = __ldg(reinterpret_cast<const uint4*>(xt + 8 * j * kThreads));
            if (lane == 0) {
#pragma unroll
                for (int j = 0; j < 4; ++j) ahead[j] = (unsigned)(uint16_t)__ldg(xt + 8 * j * kThreads - 1) << 16;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const unsigned up = __shfl_up_sync(0xffffffffu, v[j].w, 1);
                c += changes8(v[j], lane ? up : ahead[j]);
            }
        } else {
            for (int k = t; k < kTile; k += kThreads) {
                const long long i = t0 + k;
                if (i < 0 || i >= n) continue;
                const int prev = i > 0 || has_before ? x[i - 1] : 0;
                c += (prev ^ x[i]) < 0;
            }
        }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if (lane == 0) warp_sum[t >> 5] = c;
    __syncthreads();
    if (t == 0) {
        int s = 0;
        for (int w = 0; w < kThreads / 32; ++w) s += warp_sum[w];
        counts[blockIdx.x] = s;
    }
}

// Writes one tile's crossings, the last of them at edges[end - 1]; returns
// their number.  The signs make a shared bitmap; thread t owns the 32 samples
// of word t.  All threads; ends with every read of the shared arrays done
// but warp_tot's.
template <bool In>
__device__ __forceinline__ int write_tile(const int16_t* __restrict__ x, long long n, long long t0, int has_before,
                                          unsigned* bm, int* warp_tot, ldg_efm_edge* __restrict__ edges,
                                          long long cap, long long pos_offset, long long end) {
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    uint8_t* bytes = reinterpret_cast<uint8_t*>(bm);
    uint4 v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = load8<In>(x, n, t0 + 8 * (j * kThreads + t));
#pragma unroll
    for (int j = 0; j < 4; ++j) bytes[j * kThreads + t] = (uint8_t)signs8(v[j]);
    unsigned before = 0;
    if (t == 0) before = In || (t0 > 0 && t0 <= n) ? (unsigned)(x[t0 - 1] < 0) : 0u;
    __syncthreads();
    if (t > 0) before = (bm[t - 1] >> 24) & 1u;
    // byte order to sample order: the word's first sample in bit 0
    const unsigned f = __brev(__byte_perm(bm[t], 0, 0x0123));
    unsigned e = crossings32<In>(f, before, x, n, t0 + 32 * t, has_before);
    const int cnt = __popc(e);
    int inc = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    if (lane == 31) warp_tot[warp] = inc;
    __syncthreads();
    int total = 0, ahead = 0;  // crossings of the tile, of the warps before this one
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) {
        const int q = warp_tot[w];
        ahead += w < warp ? q : 0;
        total += q;
    }
    long long k = end - total + ahead + inc - cnt;
    const int16_t* xt = x + t0 + 32 * t;
    const unsigned pos = (unsigned)(pos_offset + t0 + 32 * t);
    const bool whole = In && end <= cap && (reinterpret_cast<uintptr_t>(edges) & 7) == 0;
    if (whole && total > kDense) {
        // lane l takes sample l of the warp's words in turn, so that a store's lanes write side by side
        uint2* out = reinterpret_cast<uint2*>(edges + (end - total + ahead));
        const int16_t* xw = x + t0 + 1024 * warp + lane;
        const unsigned pw = (unsigned)(pos_offset + t0 + 1024 * warp + lane);
        const int at = inc - cnt;
#pragma unroll 4
        for (int s = 0; s < 32; ++s) {
            const unsigned es = __shfl_sync(0xffffffffu, e, s);
            const int o = __shfl_sync(0xffffffffu, at, s);
            if ((es >> lane) & 1u)
                out[o + __popc(es & ((1u << lane) - 1u))] =
                    make_uint2(pw + 32 * s, (unsigned)(uint16_t)xw[32 * s - 1] | ((unsigned)(uint16_t)xw[32 * s] << 16));
        }
        return total;
    }
    if (whole) {
        uint2* out = reinterpret_cast<uint2*>(edges + k);
        while (e) {
            const int c = __ffs(e) - 1;
            e &= e - 1;
            *out++ = make_uint2(pos + c, (unsigned)(uint16_t)xt[c - 1] | ((unsigned)(uint16_t)xt[c] << 16));
        }
        return total;
    }
    while (e) {
        const int c = __ffs(e) - 1;
        e &= e - 1;
        if (k < cap) {
            ldg_efm_edge r;
            r.pos = (int32_t)(pos + c);
            r.prev = t0 + 32 * t + c > 0 || has_before ? xt[c - 1] : (int16_t)0;
            r.cur = xt[c];
            edges[k] = r;
        }
        ++k;
    }
    return total;
}

__global__ void __launch_bounds__(kThreads) efm_write_kernel(const int16_t* __restrict__ x, long long n, int mis,
                                                             int has_before, long long ntiles,
                                                             const long long* __restrict__ counts,
                                                             ldg_efm_edge* __restrict__ edges, long long cap,
                                                             long long pos_offset, long long* count_out) {
    __shared__ unsigned bm[2][kThreads];
    __shared__ int warp_tot[2][kThreads / 32];
    __shared__ long long s_sum[kThreads / 32];
    const int t = threadIdx.x;
    const long long g0 = ntiles * blockIdx.x / gridDim.x, g1 = ntiles * (blockIdx.x + 1) / gridDim.x;
    // the crossings up to this chunk's end
    long long s = 0;
    for (int g = t; g <= (int)blockIdx.x; g += kThreads) s += counts[g];
#pragma unroll
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((t & 31) == 0) s_sum[t >> 5] = s;
    __syncthreads();
    long long end = 0;
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) end += s_sum[w];
    if (t == 0 && count_out && blockIdx.x == gridDim.x - 1) *count_out = end;
    // the shared arrays alternate: a tile's barriers order the reads of the
    // tile before it against the writes of the tile after
#pragma unroll 1
    for (long long tile = g1 - 1; tile >= g0; --tile) {
        const long long t0 = tile * kTile - mis;
        const int b = (int)(tile & 1);
        if (t0 > 0 && t0 + kTile <= n) {
            end -= write_tile<true>(x, n, t0, has_before, bm[b], warp_tot[b], edges, cap, pos_offset, end);
        } else {
            end -= write_tile<false>(x, n, t0, has_before, bm[b], warp_tot[b], edges, cap, pos_offset, end);
        }
    }
}

}  // namespace

extern "C" {

int64_t ldg_efm_edges_scratch_bytes(int64_t n) {
    if (n < 0) return -1;
    return (int64_t)align256(kMaxChunks * sizeof(long long));  // a count per chunk
}

int ldg_efm_edges(const int16_t* efm, int64_t n, int32_t has_before, int64_t pos_offset, ldg_efm_edge* edges,
                  int64_t cap, int64_t* count, void* scratch, void* stream) {
    if (!efm || !edges || !scratch || n < 0 || cap < 0)
        return ldg::api_fail(LDG_ERR_ARG, "ldg_efm_edges: NULL buffer or negative size");
    if (pos_offset < 0 || pos_offset + n > (int64_t)INT32_MAX)
        return ldg::api_fail(LDG_ERR_RANGE, "ldg_efm_edges: positions must fit int32 (pos_offset + n)");
    long long* dcount = nullptr;
    if (count) {
        dcount = static_cast<long long*>(ldg::device_view(count));
        if (!dcount)
            return ldg::api_fail(LDG_ERR_ARG, "ldg_efm_edges: count must be device memory or pinned host memory");
    }
    cudaStream_t st = (cudaStream_t)stream;
    if (n > 0) {
        const int mis = (int)((reinterpret_cast<uintptr_t>(efm) & 15) / sizeof(int16_t));
        const long long ntiles = (n + mis + kTile - 1) / kTile;
        long long* counts = static_cast<long long*>(scratch);
        const unsigned grid = (unsigned)(ntiles < kMaxChunks ? ntiles : kMaxChunks);
        efm_count_kernel<<<grid, kThreads, 0, st>>>(efm, n, mis, has_before, ntiles, counts);
        efm_write_kernel<<<grid, kThreads, 0, st>>>(efm, n, mis, has_before, ntiles, counts, edges, cap, pos_offset,
                                                    dcount);
    } else if (dcount) {
        if (cudaMemsetAsync(dcount, 0, sizeof(long long), st) != cudaSuccess) cudaGetLastError();
    }
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return ldg::api_fail(LDG_ERR_CUDA, std::string("ldg_efm_edges: ") + cudaGetErrorString(e));
    return LDG_OK;
}

}  // extern "C"

namespace {

// one thread per field: its EFM slice [startloc + int(ll[1]), startloc +
// int(ll[end_line])) and the samples at both ends
__global__ void efm_slices_kernel(const long long* __restrict__ startloc, const unsigned long long* __restrict__ llp,
                                  const int* __restrict__ end_line, int n, const int16_t* __restrict__ efm,
                                  long long efm_len, long long* bounds, int16_t* samples) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double* ll = reinterpret_cast<const double*>(llp[i]);
    const long long lo = startloc[i] + (long long)ll[1];  // truncation, as int() of the location
    const long long hi = startloc[i] + (long long)ll[end_line[i]];
    bounds[2 * i] = lo;
    bounds[2 * i + 1] = hi;
    samples[2 * i] = lo >= 0 && lo < efm_len ? efm[lo] : (int16_t)0;
    samples[2 * i + 1] = hi - 1 >= 0 && hi - 1 < efm_len ? efm[hi - 1] : (int16_t)0;
}

}  // namespace

extern "C" int ldg_efm_field_slices(const int64_t* startloc, const uint64_t* linelocs, const int32_t* end_line,
                                    int32_t n, const int16_t* efm, int64_t efm_len, int64_t* bounds,
                                    int16_t* samples, void* stream) {
    if (n < 0 || (n > 0 && (!startloc || !linelocs || !end_line || !efm || !bounds || !samples)))
        return ldg::api_fail(LDG_ERR_ARG, "ldg_efm_field_slices: NULL buffer or negative count");
    if (n == 0) return LDG_OK;
    const void* p[5] = {startloc, linelocs, end_line, bounds, samples};
    void* d[5];
    for (int k = 0; k < 5; ++k) {
        d[k] = ldg::device_view(p[k]);
        if (!d[k])
            return ldg::api_fail(LDG_ERR_ARG, "ldg_efm_field_slices: arrays must be device memory or pinned host memory");
    }
    efm_slices_kernel<<<(n + 127) / 128, 128, 0, (cudaStream_t)stream>>>(
        static_cast<const long long*>(d[0]), static_cast<const unsigned long long*>(d[1]),
        static_cast<const int*>(d[2]), n, efm, efm_len, static_cast<long long*>(d[3]), static_cast<int16_t*>(d[4]));
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess)
        return ldg::api_fail(LDG_ERR_CUDA, std::string("ldg_efm_field_slices: ") + cudaGetErrorString(e));
    return LDG_OK;
}
