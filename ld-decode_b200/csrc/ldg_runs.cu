// Sync-pulse runs on the GPU.
//
// ldg_sync_runs: runs of demod_05 at or below the sync threshold over a
// whole capture-wide output array -- the pulses findpulses
// (lddecode/utils.py:1101-1157) finds, for every field read window at once --
// and the mean level inside the long ones (getpulses' VSYNC level check,
// core.py:2242-2322).
//
// Two launches over the same contiguous chunks, one per resident CTA.
// runs_flags_kernel reads the samples once, leaves one below-threshold flag
// bit per sample and, per chunk, the number of runs that start in it and its
// first clear sample; runs_write_kernel adds up the starts before its chunk,
// walks the chunk's flags (1/32 of the samples' bytes, in L2) and writes its
// runs, with the long ones' means, straight into the caller's pinned
// buffers.  A run that leaves its chunk ends at the first clear sample of
// the chunks after it.  Bound: HBM, 4 bytes per sample.
//
// The whole call on a B200, wait included: 78 us at 60 M samples (24 k runs)
// and 37 us at 5.8 M; one pass with decoupled look-back and a pairing launch
// took 139 and 63, as the look-back and a warp's long runs, one after
// another, are serial chains.
#include <climits>
#include <cmath>
#include <cstdint>
#include <mutex>
#include <string>

#include "ldg_copy.cuh"
#include "ldgpu.h"

struct ldg_ctx;

namespace ldg {
int lines_fail(int code, const std::string& msg);
int ctx_device(const ldg_ctx* c);
std::mutex& ctx_mutex(ldg_ctx* c);
int ctx_lines_scratch(ldg_ctx* c, size_t need, void** out);
int ctx_host_word(ldg_ctx* c, long long** host, long long** dev);
}  // namespace ldg

namespace {

constexpr int kThreads = 128;
constexpr int kWarps = kThreads / 32;
constexpr int kSteps = 4;                       // 128-sample steps of a warp per tile
constexpr int kWarpSpan = 128 * kSteps;         // contiguous samples of a warp
constexpr int kTile = kWarps * kWarpSpan;       // samples
constexpr int kTileGroups = kTile / 128;        // flag groups of a tile
constexpr int kMaxChunks = 148 * 8;             // all resident; 148 * 16 took 80 us for 78 at 60 M samples
constexpr int kAhead = 16;                       // loads in flight per lane of a long run's mean
constexpr long long kNone = LLONG_MAX;

size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

// Sample i sits at position i + mis, mis the samples x lies past a 16-byte
// boundary, so that any x takes 16-byte loads.  The flags of the positions
// 128 g .. 128 g + 127 are one group: bit l of word k belongs to position
// 128 g + 4 l + k (the ballots of a warp's float4 loads).

__device__ __forceinline__ long long min_all(long long v) {
#pragma unroll
    for (int o = 16; o; o >>= 1) v = min(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

__device__ __forceinline__ long long sum_all(long long v) {
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__global__ void __launch_bounds__(kThreads) runs_flags_kernel(const float* __restrict__ x, long long n, int mis,
                                                              float thr, long long ntiles, uint4* __restrict__ flags,
                                                              int* __restrict__ starts,
                                                              long long* __restrict__ first_clear) {
    __shared__ int s_count[kWarps];
    __shared__ long long s_clear[kWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long g0 = ntiles * blockIdx.x / gridDim.x, g1 = ntiles * (blockIdx.x + 1) / gridDim.x;
    int count = 0;           // the same in every lane
    long long clear = kNone;  // likewise
#pragma unroll 1
    for (long long tile = g0; tile < g1; ++tile) {
        const long long w0 = tile * kTile - mis + kWarpSpan * warp;
        float4 v[kSteps];
        if (w0 > 0 && w0 + kWarpSpan <= n) {
#pragma unroll
            for (int j = 0; j < kSteps; ++j) v[j] = __ldcs(reinterpret_cast<const float4*>(x + w0 + 128 * j) + lane);
        } else {
#pragma unroll
            for (int j = 0; j < kSteps; ++j) {
                const long long i = w0 + 128 * j + 4 * lane;
                const float out = nanf("");  // never at or below a threshold
                v[j].x = i >= 0 && i < n ? x[i] : out;
                v[j].y = i + 1 >= 0 && i + 1 < n ? x[i + 1] : out;
                v[j].z = i + 2 >= 0 && i + 2 < n ? x[i + 2] : out;
                v[j].w = i + 3 >= 0 && i + 3 < n ? x[i + 3] : out;
            }
        }
        unsigned before = w0 > 0 && w0 <= n && x[w0 - 1] <= thr ? 1u : 0u;  // the flag of the sample before
        uint4* out = flags + tile * kTileGroups + kSteps * warp;
#pragma unroll
        for (int j = 0; j < kSteps; ++j) {
            const unsigned b0 = __ballot_sync(0xffffffffu, v[j].x <= thr), b1 = __ballot_sync(0xffffffffu, v[j].y <= thr);
            const unsigned b2 = __ballot_sync(0xffffffffu, v[j].z <= thr), b3 = __ballot_sync(0xffffffffu, v[j].w <= thr);
            const unsigned s0 = b0 & ~((b3 << 1) | before), s1 = b1 & ~b0, s2 = b2 & ~b1, s3 = b3 & ~b2;
            if (s0 | s1 | s2 | s3) count += __popc(s0) + __popc(s1) + __popc(s2) + __popc(s3);
            before = b3 >> 31;
            const unsigned all = b0 & b1 & b2 & b3;
            if (clear == kNone && ~all) {
                const int l = __ffs(~all) - 1;
                const int k = !((b0 >> l) & 1u) ? 0 : !((b1 >> l) & 1u) ? 1 : !((b2 >> l) & 1u) ? 2 : 3;
                clear = w0 + 128 * j + 4 * l + k;
            }
            if (lane == j) out[j] = make_uint4(b0, b1, b2, b3);
        }
    }
    if (lane == 0) {
        s_count[warp] = count;
        s_clear[warp] = clear;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int c = 0;
        long long m = kNone;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            c += s_count[w];
            m = min(m, s_clear[w]);
        }
        starts[blockIdx.x] = c;
        first_clear[blockIdx.x] = m;
    }
}

// rs, rl, rm: the caller's arrays of `cap` runs (host-mapped, or device
// memory that is copied back); from, to: device copies of the runs' bounds.
// A thread owns 128 samples' flags; runs are handed to the CTA's threads for
// output, the long ones to its warps in turn (lane l sums every 32nd sample).
__global__ void __launch_bounds__(kThreads) runs_write_kernel(
    const float* __restrict__ x, long long n, int mis, long long ntiles, const uint4* __restrict__ flags,
    const int* __restrict__ starts, const long long* __restrict__ first_clear, long long min_long, long long trim_lo,
    long long trim_hi, long long* from, long long* to, long long cap, long long* rs, long long* rl, double* rm,
    long long* count_out) {
    __shared__ long long s_part[kWarps], s_from[kThreads], s_len[kThreads];
    __shared__ double s_mean[kThreads];
    __shared__ int s_tot[kWarps];
    __shared__ unsigned s_long[kWarps];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int chunk = blockIdx.x, nchunks = gridDim.x;
    const long long g0 = kTileGroups * (ntiles * chunk / nchunks), g1 = kTileGroups * (ntiles * (chunk + 1) / nchunks);

    long long sum = 0;
    for (int c = 4 * t; c < chunk; c += 4 * kThreads) {  // starts holds a multiple of four
        const int4 v = *reinterpret_cast<const int4*>(starts + c);
        sum += v.x;
        if (c + 1 < chunk) sum += v.y;
        if (c + 2 < chunk) sum += v.z;
        if (c + 3 < chunk) sum += v.w;
    }
    sum = sum_all(sum);
    if (lane == 0) s_part[warp] = sum;
    __syncthreads();
    long long first = 0;  // the chunk's first run
#pragma unroll
    for (int w = 0; w < kWarps; ++w) first += s_part[w];

    long long run = first;
#pragma unroll 1
    for (long long gt = g0; gt < g1; gt += kThreads) {
        const long long g = gt + t;
        uint4 b = make_uint4(0, 0, 0, 0);
        unsigned before = 0;
        if (g < g1) {
            b = flags[g];
            before = g > 0 ? flags[g - 1].w >> 31 : 0u;
        }
        const uint4 p = make_uint4((b.w << 1) | before, b.x, b.y, b.z);  // the flags of the samples before
        const int cnt = __popc(b.x & ~p.x) + __popc(b.y & ~p.y) + __popc(b.z & ~p.z) + __popc(b.w & ~p.w);
        int inc = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += y;
        }
        __syncthreads();  // the last round's reads of s_tot
        if (lane == 31) s_tot[warp] = inc;
        __syncthreads();
        long long k = run + inc - cnt;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            k += w < warp ? s_tot[w] : 0;
            run += s_tot[w];
        }
        const unsigned e0 = b.x ^ p.x, e1 = b.y ^ p.y, e2 = b.z ^ p.z, e3 = b.w ^ p.w;
        const long long i0 = 128 * g - mis;
        if (g < g1) {
            for (unsigned any = e0 | e1 | e2 | e3; any; any &= any - 1) {
                const int l = __ffs(any) - 1;
                const unsigned e = ((e0 >> l) & 1u) | ((e1 >> l) & 1u) << 1 | ((e2 >> l) & 1u) << 2 | ((e3 >> l) & 1u) << 3;
                const unsigned f = ((b.x >> l) & 1u) | ((b.y >> l) & 1u) << 1 | ((b.z >> l) & 1u) << 2 | ((b.w >> l) & 1u) << 3;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (!((e >> j) & 1u)) continue;
                    const long long i = i0 + 4 * l + j;
                    if ((f >> j) & 1u) {
                        if (k < cap) from[k] = i;
                        ++k;
                    } else if (k > first && k <= cap) {  // an earlier chunk's run is ended there
                        to[k - 1] = i;
                    }
                }
            }
        }
    }
    // the run that leaves the chunk
    if (warp == 0 && run > first && run <= cap && (flags[g1 - 1].w >> 31)) {
        long long end = kNone;
        for (int c0 = chunk + 1; c0 < nchunks && end == kNone; c0 += 32)
            end = min_all(c0 + lane < nchunks ? first_clear[c0 + lane] : kNone);
        if (lane == 0) to[run - 1] = end;
    }
    __syncthreads();

    const long long last = min(run, cap);
#pragma unroll 1
    for (long long r0 = first; r0 < last; r0 += kThreads) {
        const long long r = r0 + t;
        long long s = 0, len = 0;
        bool whole = false;  // a run open at the end of the array is not one
        if (r < last) {
            const long long e = to[r];
            s = from[r];
            len = e - s;
            whole = e < n;
        }
        const unsigned longs = __ballot_sync(0xffffffffu, whole && len > min_long);
        s_from[t] = s;
        s_len[t] = len;
        s_mean[t] = nan("");
        if (lane == 0) s_long[warp] = longs;
        __syncthreads();
        int turn = 0;
#pragma unroll 1
        for (int w = 0; w < kWarps; ++w) {
            for (unsigned m = s_long[w]; m; m &= m - 1, ++turn) {
                if (turn % kWarps != warp) continue;
                const int q = 32 * w + __ffs(m) - 1;
                const long long lo = s_from[q] + trim_lo, hi = s_from[q] + s_len[q] - trim_hi;
                double acc = 0;
                long long i = lo + lane;
                for (; i + 32 * (kAhead - 1) < hi; i += 32 * kAhead) {
                    float v[kAhead];
#pragma unroll
                    for (int j = 0; j < kAhead; ++j) v[j] = x[i + 32 * j];
#pragma unroll
                    for (int j = 0; j < kAhead; ++j) acc += (double)v[j];
                }
                for (; i < hi; i += 32) acc += (double)x[i];
#pragma unroll
                for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
                if (lane == 0 && hi > lo) s_mean[q] = acc / (double)(hi - lo);
            }
        }
        __syncthreads();
        if (whole) {
            rs[r] = s;
            rl[r] = len;
            rm[r] = s_mean[t];
        }
        __syncthreads();
    }
    if (chunk == nchunks - 1 && t == 0) {
        const long long p = n - 1 + mis;
        const uint4 b = flags[p >> 7];
        const unsigned word = (p & 3) == 0 ? b.x : (p & 3) == 1 ? b.y : (p & 3) == 2 ? b.z : b.w;
        *count_out = run - ((word >> ((p & 127) >> 2)) & 1u);
    }
}

}  // namespace

extern "C" int ldg_sync_runs(ldg_ctx* c, const float* d05, int64_t n, double threshold, int64_t min_long,
                             int64_t trim_lo, int64_t trim_hi, int64_t* run_start, int64_t* run_len, double* run_mean,
                             int64_t cap, int64_t* nruns, void* stream) {
    if (!c || !d05 || !run_start || !run_len || !run_mean || !nruns)
        return ldg::lines_fail(LDG_ERR_ARG, "ldg_sync_runs: NULL argument");
    if (n < 2 || cap < 1 || trim_lo < 0 || trim_hi < 0) return ldg::lines_fail(LDG_ERR_ARG, "ldg_sync_runs: bad size");
    std::lock_guard<std::mutex> lk(ldg::ctx_mutex(c));
    int prev = -1;
    cudaGetDevice(&prev);
    cudaSetDevice(ldg::ctx_device(c));
    cudaStream_t st = (cudaStream_t)stream;
    const int mis = (int)((reinterpret_cast<uintptr_t>(d05) & 15) / sizeof(float));
    const long long ntiles = (n + mis + kTile - 1) / kTile;
    const int nchunks = (int)(ntiles < kMaxChunks ? ntiles : kMaxChunks);
    const size_t b_flags = align256((size_t)ntiles * kTileGroups * sizeof(uint4));
    const size_t b_starts = align256(kMaxChunks * sizeof(int)), b_clear = align256(kMaxChunks * sizeof(long long));
    const size_t b_runs = align256(cap * sizeof(long long));
    const size_t need = b_flags + b_starts + b_clear + 4 * b_runs + align256(cap * sizeof(double));
    void* scratch = nullptr;
    auto done = [&](int rc) {
        if (prev >= 0) cudaSetDevice(prev);
        return rc;
    };
    if (ldg::ctx_lines_scratch(c, need, &scratch) != LDG_OK) return done(LDG_ERR_CUDA);
    char* p = static_cast<char*>(scratch);
    uint4* flags = reinterpret_cast<uint4*>(p);
    int* starts = reinterpret_cast<int*>(p + b_flags);
    long long* clear = reinterpret_cast<long long*>(p + b_flags + b_starts);
    long long* from = reinterpret_cast<long long*>(p + b_flags + b_starts + b_clear);
    long long* to = from + b_runs / sizeof(long long);
    long long* rs = to + b_runs / sizeof(long long);
    long long* rl = rs + b_runs / sizeof(long long);
    double* rm = reinterpret_cast<double*>(rl + b_runs / sizeof(long long));
    auto cuda_fail = [&](const char* what) {
        return done(ldg::lines_fail(LDG_ERR_CUDA, std::string("ldg_sync_runs: ") + what + ": " +
                                                      cudaGetErrorString(cudaGetLastError())));
    };
    long long *hw = nullptr, *dw = nullptr;  // the run count, host-mapped
    if (ldg::ctx_host_word(c, &hw, &dw) != LDG_OK) return cuda_fail("host word");
    volatile long long* vhw = hw;
    vhw[0] = -1;
    // a float32 sample is at or below `threshold` when it is at or below the
    // greatest float32 that is
    float thr = (float)threshold;
    if ((double)thr > threshold) thr = std::nextafterf(thr, -INFINITY);
    runs_flags_kernel<<<nchunks, kThreads, 0, st>>>(d05, n, mis, thr, ntiles, flags, starts, clear);
    // runs straight into the caller's pinned (mapped) buffers when they are:
    // the host then waits for the stream only (no copy-engine transfer, which
    // would queue behind bulk copies of an end-to-end pipeline)
    void* drs = ldg::device_view(run_start);
    void* drl = ldg::device_view(run_len);
    void* drm = ldg::device_view(run_mean);
    const bool mapped = drs && drl && drm;
    runs_write_kernel<<<nchunks, kThreads, 0, st>>>(
        d05, n, mis, ntiles, flags, starts, clear, min_long, trim_lo, trim_hi, from, to, cap,
        mapped ? static_cast<long long*>(drs) : rs, mapped ? static_cast<long long*>(drl) : rl,
        mapped ? static_cast<double*>(drm) : rm, dw);
    if (cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(st) != cudaSuccess) return cuda_fail("scan");
    const long long nr = vhw[0];
    if (nr < 0) return cuda_fail("run count not written");
    *nruns = nr;
    if (nr > cap) return done(ldg::lines_fail(LDG_ERR_RANGE, "ldg_sync_runs: more runs than cap"));
    if (!mapped && nr > 0) {
        if (cudaMemcpyAsync(run_start, rs, nr * sizeof(long long), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
            cudaMemcpyAsync(run_len, rl, nr * sizeof(long long), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
            cudaMemcpyAsync(run_mean, rm, nr * sizeof(double), cudaMemcpyDeviceToHost, st) != cudaSuccess)
            return cuda_fail("D2H");
        if (cudaStreamSynchronize(st) != cudaSuccess) return cuda_fail("run copy");
    }
    return done(LDG_OK);
}
