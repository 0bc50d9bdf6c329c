// AC3-RF front end on the GPU and the symbol-timing DPLL on the host.
//
// Restates lddecode/ac3rf.py: Ac3RfDemodulator.demodulate_to_symbols
// (ac3rf.py:372-396) -- two real half-band /2 stages (ac3rf.py:99-151), a
// 2.88 MHz mix with a 14-bit phase-accumulator NCO (ac3rf.py:352-357,
// 382-392), two complex half-band /2 stages and a root-raised-cosine matched
// filter (ac3rf.py:154-167, 343-349) -- and AC3_DPLL.reclock_symbols
// (ac3rf.py:232-299).
//
// The reference streams blocks through FIR stages that carry their history
// (zeros at the start) and decimation phase; every stage is a causal FIR, so
// output j of a stage is sum_k h[k] u[phi + D j - k] over its whole input
// history with u[i < 0] = 0, independent of how the input was chunked.  The
// GPU computes each stage that way over shared-memory tiles: one CTA makes
// kTile final (fs/16) samples from the input window it depends on.
#include <cmath>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "ldg_ac3.h"
#include "ldg_attr.cuh"

namespace ldg {

namespace {

constexpr int kTile = 512;      // final samples per CTA
constexpr int kAc3Threads = 256;

struct Ac3Params {
    const void* in;             // absolute samples [in_first, in_first + nsamples)
    int in_kind;                // 0 int16, 1 float32
    long long in_first;
    long long nsamples;
    long long out_first;
    long long out_count;
    float* out_i;
    float* out_q;
    Ac3Taps taps;
};

__device__ __forceinline__ float tap_sum(const float* u, long long ulo, long long pos, const float* val,
                                         const int* off, int n) {
    // sum_k val[k] * u[pos - off[k]] in the reference's order; u[i] = 0 for i < 0
    float acc = 0.0f;
    for (int k = 0; k < n; ++k) {
        const long long i = pos - off[k];
        const float x = i < 0 ? 0.0f : u[i - ulo];
        acc = (k == 0) ? val[0] * x : fmaf(val[k], x, acc);
    }
    return acc;
}

__global__ void __launch_bounds__(kAc3Threads) ac3_frontend_kernel(const __grid_constant__ Ac3Params p) {
    extern __shared__ float sm[];
    const Ac3Taps& t = p.taps;
    const long long J = p.out_first + (long long)blockIdx.x * kTile;
    const long long Jend = min(J + (long long)kTile, p.out_first + p.out_count);
    if (J >= Jend) return;
    // index ranges of every stage this tile needs (inclusive lo, exclusive hi)
    const long long lo5 = J, hi5 = Jend;
    const long long lo4 = lo5 - (t.n_rrc - 1), hi4 = hi5;
    const long long lo3 = 2 * lo4 - (t.n_hb23 - 1), hi3 = 2 * (hi4 - 1) + 1;
    const long long lo2 = 2 * lo3 - (t.n_hb19 - 1), hi2 = 2 * (hi3 - 1) + 1;
    const long long lo1 = 2 * lo2 - (t.n_hb19 - 1), hi1 = 2 * (hi2 - 1) + 1;
    const long long lo0 = 2 * lo1 - (t.n_hb19 - 1), hi0 = 2 * (hi1 - 1) + 1;
    const int n0 = (int)(hi0 - lo0), n1 = (int)(hi1 - lo1), n2 = (int)(hi2 - lo2);
    const int n3 = (int)(hi3 - lo3), n4 = (int)(hi4 - lo4);
    float* u0 = sm;                 // input
    float* u1 = u0 + n0;            // stage 1
    float* u2 = u1 + n1;            // stage 2 (real), then mixed I in place
    float* q2 = u2 + n2;            // mixed Q
    float* i3 = q2 + n2;
    float* q3 = i3 + n3;
    float* i4 = q3 + n3;
    float* q4 = i4 + n4;
    for (int k = threadIdx.x; k < n0; k += blockDim.x) {
        const long long gi = lo0 + k - p.in_first;  // the host checked gi >= 0 wherever lo0 + k >= 0
        float v = 0.0f;
        if (lo0 + k >= 0 && gi >= 0 && gi < p.nsamples)
            v = p.in_kind == 0 ? (float)static_cast<const int16_t*>(p.in)[gi] : static_cast<const float*>(p.in)[gi];
        u0[k] = v;
    }
    __syncthreads();
    for (int k = threadIdx.x; k < n1; k += blockDim.x) {
        const long long j = lo1 + k;
        u1[k] = j < 0 ? 0.0f : tap_sum(u0, lo0, 2 * j, t.hb19_val, t.hb19_off, t.n_hb19_nz);
    }
    __syncthreads();
    for (int k = threadIdx.x; k < n2; k += blockDim.x) {
        const long long j = lo2 + k;
        float v = j < 0 ? 0.0f : tap_sum(u1, lo1, 2 * j, t.hb19_val, t.hb19_off, t.n_hb19_nz);
        // NCO: phase = (step * j) mod 2^bits, cos/sin tables
        const unsigned mask = (1u << t.lut_bits) - 1u;
        const unsigned ph = j < 0 ? 0u : (unsigned)(((unsigned long long)(j & mask) * (unsigned)t.phase_step) & mask);
        u2[k] = v * t.cos_lut[ph];
        q2[k] = v * t.sin_lut[ph];
    }
    __syncthreads();
    for (int k = threadIdx.x; k < n3; k += blockDim.x) {
        const long long j = lo3 + k;
        i3[k] = j < 0 ? 0.0f : tap_sum(u2, lo2, 2 * j, t.hb19_val, t.hb19_off, t.n_hb19_nz);
        q3[k] = j < 0 ? 0.0f : tap_sum(q2, lo2, 2 * j, t.hb19_val, t.hb19_off, t.n_hb19_nz);
    }
    __syncthreads();
    for (int k = threadIdx.x; k < n4; k += blockDim.x) {
        const long long j = lo4 + k;
        i4[k] = j < 0 ? 0.0f : tap_sum(i3, lo3, 2 * j, t.hb23_val, t.hb23_off, t.n_hb23_nz);
        q4[k] = j < 0 ? 0.0f : tap_sum(q3, lo3, 2 * j, t.hb23_val, t.hb23_off, t.n_hb23_nz);
    }
    __syncthreads();
    for (int k = threadIdx.x; k < (int)(hi5 - lo5); k += blockDim.x) {
        const long long j = lo5 + k;
        p.out_i[j - p.out_first] = tap_sum(i4, lo4, j, t.rrc_val, t.rrc_off, t.n_rrc_nz);
        p.out_q[j - p.out_first] = tap_sum(q4, lo4, j, t.rrc_val, t.rrc_off, t.n_rrc_nz);
    }
}

// ---- the reference's own filter shapes (half-band 19 / 23 taps, a dense
// root-raised cosine): every stage register-blocked over split-phase tiles
//
// Bound: shared-memory load bandwidth, then FP32 issue (320 multiply-adds per
// 16 input samples).  A half-band /2 stage reads one phase of its input at
// every tap but the centre one, so a stage's output is kept as its even and
// its odd samples: output k then takes E[k .. k + taps / 2] and one O, all at
// unit stride, and a thread's kR consecutive outputs share their loads (16
// bytes each).  The tile is chosen so that the eight-output stages fill 512
// threads exactly (8192, 4096 and 2 x 2048 values) for any matched filter; two
// buffers serve the five stages in turn (110 KB, two CTAs per SM).  The
// mixer's table is stored in the order the phase accumulator visits it, so
// its reads are contiguous.  Taps come from the kernel's parameters
// (constant operands).  Each output is the same chain of multiply-adds as the
// general kernel's, so the results are equal bit for bit.
// 2 s of int16 samples (80 M), B200: 2058 us by the general kernel, 172 us by this
// one (1.2 TB/s of the 200 MB it has to move); 197 us with the mixer's entries read
// one by one and the matched filter's last taps by scalar loads.

constexpr int kFastThreads = 512;
constexpr int kHb19Nz = 11, kHb23Nz = 13, kMaxRrc = kMaxAc3Rrc;
constexpr int kN4 = 1006, kN3 = 2 * kN4 - 1 + 22, kN2 = 2 * kN3 - 1 + 18, kN1 = 2 * kN2 - 1 + 18,
              kN0 = 2 * kN1 - 1 + 18;  // samples of every stage a tile holds
static_assert(kN0 == 16383 && kN1 <= 2 * 8 * kFastThreads && kN2 <= 8 * kFastThreads, "one or two rounds of eight");
static_assert(kN3 <= 8 * (kFastThreads / 2) && kN4 <= 4 * (kFastThreads / 2), "one round per channel");

// Padded index of the arrays read eight outputs (32 bytes) per thread apart: four
// words per 32 keep a quarter warp's 16-byte reads on different banks.
__host__ __device__ constexpr int pad8(int i) { return i + 4 * (i >> 5); }
constexpr int kHalf0 = pad8(8192 + 32), kHalf1 = pad8(4096 + 32), kHalf2 = pad8(2048 + 32), kHalf3 = 1024 + 32;
constexpr int kXLen = 1024;  // a channel's stage-4 samples, shifted by up to three
constexpr int kBufA = 2 * kHalf0, kBufB = 2 * kHalf1;
static_assert(4 * kHalf2 <= kBufA && 4 * kHalf3 <= kBufB && 2 * kXLen + 4 <= kBufA, "stages share two buffers");

struct Ac3FastParams {
    const void* in;
    int in_kind;
    long long in_first;
    long long nsamples;
    long long out_first;
    long long out_count;
    float* out_i;
    float* out_q;
    const float2* mix;          // (cos, sin) of sample j's phase at j mod 2^lut_bits
    int mix_mask;
    int n_rrc;
    float hb19[kHb19Nz], hb23[kHb23Nz], rrc[kMaxRrc];
};

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float a, float b, float c, float d) {
    *reinterpret_cast<float4*>(p) = make_float4(a, b, c, d);
}

// Eight outputs k0 .. k0 + 7 of the 19-tap half-band stage over split-phase
// input (padded halves E, O): taps 0, 2, .., 8, then the centre, then 10, .., 18.
__device__ __forceinline__ void hb19x8(const float* E, const float* O, int k0, const float* h, float (&acc)[8]) {
    float e[20], o[8];
#pragma unroll
    for (int c = 0; c < 5; ++c) {
        const float4 v = ld4(E + pad8(k0 + 4 * c));
        e[4 * c] = v.x;
        e[4 * c + 1] = v.y;
        e[4 * c + 2] = v.z;
        e[4 * c + 3] = v.w;
    }
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        const float4 v = ld4(O + pad8(k0 + 4 + 4 * c));
        o[4 * c] = v.x;
        o[4 * c + 1] = v.y;
        o[4 * c + 2] = v.z;
        o[4 * c + 3] = v.w;
    }
#pragma unroll
    for (int r = 0; r < 8; ++r) acc[r] = h[0] * e[r + 9];
#pragma unroll
    for (int m = 1; m < 5; ++m)
#pragma unroll
        for (int r = 0; r < 8; ++r) acc[r] = fmaf(h[m], e[r + 9 - m], acc[r]);
#pragma unroll
    for (int r = 0; r < 8; ++r) acc[r] = fmaf(h[5], o[r], acc[r]);
#pragma unroll
    for (int m = 5; m < 10; ++m)
#pragma unroll
        for (int r = 0; r < 8; ++r) acc[r] = fmaf(h[m + 1], e[r + 9 - m], acc[r]);
}

__global__ void __launch_bounds__(kFastThreads, 2) ac3_frontend_fast_kernel(const __grid_constant__ Ac3FastParams p) {
    extern __shared__ float sm[];
    float* A = sm;
    float* B = sm + kBufA;
    const int t = threadIdx.x;
    const int tile = kN4 - (p.n_rrc - 1);  // final samples per CTA
    const long long J = p.out_first + (long long)blockIdx.x * tile;
    const int nout = (int)min((long long)tile, p.out_first + p.out_count - J);
    const long long lo2 = 4 * (J - (p.n_rrc - 1)) - 2 * 22 - 18;  // stage-2 index of local sample 0
    const long long lo0 = 4 * lo2 - 2 * 18 - 18;                  // raw index of local sample 0

    // raw samples, split by parity: pairs as one load where the address allows
    {
        float* E = A;
        float* O = A + kHalf0;
        const long long g0 = lo0 - p.in_first;
        const bool inside = lo0 >= 0 && g0 >= 0 && g0 + 2 * 8192 <= p.nsamples;
        if (p.in_kind == 0) {
            const int16_t* x = static_cast<const int16_t*>(p.in);
            if (inside && (reinterpret_cast<uintptr_t>(x + g0) & 3) == 0) {
                const int* x2 = reinterpret_cast<const int*>(x + g0);
#pragma unroll 8
                for (int i = t; i < 8192; i += kFastThreads) {
                    const int w = __ldcs(x2 + i);
                    E[pad8(i)] = (float)(int16_t)(w & 0xffff);
                    O[pad8(i)] = (float)(int16_t)(((unsigned)w) >> 16);
                }
            } else {
                for (int i = t; i < 2 * 8192; i += kFastThreads) {
                    const long long gi = g0 + i;
                    const float v = lo0 + i >= 0 && gi >= 0 && gi < p.nsamples ? (float)x[gi] : 0.0f;
                    ((i & 1) ? O : E)[pad8(i >> 1)] = v;
                }
            }
        } else {
            const float* x = static_cast<const float*>(p.in);
            if (inside && (reinterpret_cast<uintptr_t>(x + g0) & 7) == 0) {
                const float2* x2 = reinterpret_cast<const float2*>(x + g0);
#pragma unroll 8
                for (int i = t; i < 8192; i += kFastThreads) {
                    const float2 w = __ldcs(x2 + i);
                    E[pad8(i)] = w.x;
                    O[pad8(i)] = w.y;
                }
            } else {
                for (int i = t; i < 2 * 8192; i += kFastThreads) {
                    const long long gi = g0 + i;
                    const float v = lo0 + i >= 0 && gi >= 0 && gi < p.nsamples ? x[gi] : 0.0f;
                    ((i & 1) ? O : E)[pad8(i >> 1)] = v;
                }
            }
        }
        // the stages' last threads read (and discard) a little past the tile
        if (t < 32) {
            E[pad8(8192 + t)] = 0.0f;
            O[pad8(8192 + t)] = 0.0f;
            B[pad8(4096 + t)] = 0.0f;
            B[kHalf1 + pad8(4096 + t)] = 0.0f;
        }
    }
    __syncthreads();
    // stage 1: A -> B
#pragma unroll 1
    for (int k0 = 8 * t; k0 < 8192; k0 += 8 * kFastThreads) {
        float y[8];
        hb19x8(A, A + kHalf0, k0, p.hb19, y);
        st4(B + pad8(k0 >> 1), y[0], y[2], y[4], y[6]);
        st4(B + kHalf1 + pad8(k0 >> 1), y[1], y[3], y[5], y[7]);
    }
    __syncthreads();
    // stage 2 and the mixer: B -> A (I even, I odd, Q even, Q odd)
    {
        const int k0 = 8 * t;
        float y[8], q[8];
        hb19x8(B, B + kHalf1, k0, p.hb19, y);
        // two table entries per load (lo2 and k0 are even, the table's length too)
#pragma unroll
        for (int r = 0; r < 8; r += 2) {
            const float4 cs = __ldg(reinterpret_cast<const float4*>(p.mix + (int)((lo2 + k0 + r) & p.mix_mask)));
            q[r] = y[r] * cs.y;
            y[r] = y[r] * cs.x;
            q[r + 1] = y[r + 1] * cs.w;
            y[r + 1] = y[r + 1] * cs.z;
        }
        st4(A + pad8(k0 >> 1), y[0], y[2], y[4], y[6]);
        st4(A + kHalf2 + pad8(k0 >> 1), y[1], y[3], y[5], y[7]);
        st4(A + 2 * kHalf2 + pad8(k0 >> 1), q[0], q[2], q[4], q[6]);
        st4(A + 3 * kHalf2 + pad8(k0 >> 1), q[1], q[3], q[5], q[7]);
        if (t < 32) {
#pragma unroll
            for (int c = 0; c < 4; ++c) A[c * kHalf2 + pad8(2048 + t)] = 0.0f;
        }
    }
    __syncthreads();
    const int ch = t >> 8, tc = t & 255;  // half of the threads per channel from here
    // stage 3: A -> B
    {
        const int k0 = 8 * tc;
        float y[8];
        hb19x8(A + 2 * ch * kHalf2, A + (2 * ch + 1) * kHalf2, k0, p.hb19, y);
        float* E = B + 2 * ch * kHalf3;
        st4(E + (k0 >> 1), y[0], y[2], y[4], y[6]);
        st4(E + kHalf3 + (k0 >> 1), y[1], y[3], y[5], y[7]);
        if (tc < 32) {
            E[1024 + tc] = 0.0f;
            E[kHalf3 + 1024 + tc] = 0.0f;
        }
    }
    __syncthreads();
    // stage 4 (23 taps): B -> A, shifted so that the matched filter's reads
    // of four taps start on 16 bytes
    const int shift = (4 - p.n_rrc) & 3;
    float* X = A + 4 + ch * kXLen;  // (four words of room before the first sample)
    {
        const int k0 = 4 * tc;
        const float* E = B + 2 * ch * kHalf3;
        const float* O = E + kHalf3;
        float e[16], o[8], y[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const float4 v = ld4(E + k0 + 4 * c);
            e[4 * c] = v.x;
            e[4 * c + 1] = v.y;
            e[4 * c + 2] = v.z;
            e[4 * c + 3] = v.w;
        }
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const float4 v = ld4(O + k0 + 4 + 4 * c);
            o[4 * c] = v.x;
            o[4 * c + 1] = v.y;
            o[4 * c + 2] = v.z;
            o[4 * c + 3] = v.w;
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            float acc = p.hb23[0] * e[r + 11];
#pragma unroll
            for (int m = 1; m < 6; ++m) acc = fmaf(p.hb23[m], e[r + 11 - m], acc);
            acc = fmaf(p.hb23[6], o[r + 1], acc);
#pragma unroll
            for (int m = 6; m < 12; ++m) acc = fmaf(p.hb23[m + 1], e[r + 11 - m], acc);
            y[r] = acc;
        }
        if (k0 < kN4) {
#pragma unroll
            for (int r = 0; r < 4; ++r) X[k0 + r + shift] = y[r];
        }
    }
    __syncthreads();
    // matched filter: four outputs per thread over a window of eight samples
    // that slides down four taps at a time
    {
        const int k0 = 4 * tc;
        if (k0 >= nout) return;
        const float* w0 = X + shift + k0 + p.n_rrc - 1;  // sample of output k0 at tap 0
        float acc[4] = {-0.0f, -0.0f, -0.0f, -0.0f};     // h * x + -0 is h * x
        float4 hi = ld4(w0 + 1);                         // samples of tap -1 .. -4 (outputs 1 .. 3 at tap 0 use three)
        float4 lo = ld4(w0 - 3);
        const int groups = p.n_rrc >> 2;
#pragma unroll 1
        for (int g = 0; g < groups; ++g) {
            const float x[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                const float h = p.rrc[4 * g + m];
#pragma unroll
                for (int r = 0; r < 4; ++r)
                    acc[r] = fmaf(h, x[3 + r - m], acc[r]);
            }
            hi = lo;
            lo = ld4(w0 - 3 - 4 * (g + 1));  // (at the last group X[k0 ..] when taps remain, else discarded)
        }
        const int rest = p.n_rrc & 3;
        const float x[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            if (m < rest) {
                const float h = p.rrc[4 * groups + m];
#pragma unroll
                for (int r = 0; r < 4; ++r) acc[r] = fmaf(h, x[3 + r - m], acc[r]);
            }
        }
        float* out = (ch ? p.out_q : p.out_i) + (J - p.out_first) + k0;
#pragma unroll
        for (int r = 0; r < 4; ++r)
            if (k0 + r < nout) out[r] = acc[r];
    }
}

size_t tile_smem(const Ac3Taps& t) {
    const long long n4 = kTile + t.n_rrc - 1;
    const long long n3 = 2 * n4 - 1 + t.n_hb23 - 1;
    const long long n2 = 2 * n3 - 1 + t.n_hb19 - 1;
    const long long n1 = 2 * n2 - 1 + t.n_hb19 - 1;
    const long long n0 = 2 * n1 - 1 + t.n_hb19 - 1;
    return (size_t)(n0 + n1 + 2 * n2 + 2 * n3 + 2 * n4) * sizeof(float);
}

}  // namespace

long long ac3_history(const Ac3Taps& t) {
    // input samples before 16 * j that final output j depends on
    return 16LL * (t.n_rrc - 1) + 8LL * (t.n_hb23 - 1) + 7LL * (t.n_hb19 - 1);
}

cudaError_t launch_ac3_frontend(const void* in, int in_kind, long long in_first, long long nsamples,
                                long long out_first, long long out_count, float* out_i, float* out_q,
                                const Ac3Taps& taps, cudaStream_t stream) {
    if (out_count <= 0) return cudaSuccess;
    if (taps.fast) {
        Ac3FastParams f;
        f.in = in;
        f.in_kind = in_kind;
        f.in_first = in_first;
        f.nsamples = nsamples;
        f.out_first = out_first;
        f.out_count = out_count;
        f.out_i = out_i;
        f.out_q = out_q;
        f.mix = taps.mix;
        f.mix_mask = (1 << taps.lut_bits) - 1;
        f.n_rrc = taps.n_rrc;
        memcpy(f.hb19, taps.h_hb19, sizeof(f.hb19));
        memcpy(f.hb23, taps.h_hb23, sizeof(f.hb23));
        memcpy(f.rrc, taps.h_rrc, sizeof(f.rrc));
        constexpr size_t bytes = (size_t)(kBufA + kBufB) * sizeof(float);
        static SmemAttr fast_attr;
        cudaError_t e = fast_attr.ensure(ac3_frontend_fast_kernel, bytes);
        if (e != cudaSuccess) return e;
        const int tile = kN4 - (taps.n_rrc - 1);
        ac3_frontend_fast_kernel<<<(unsigned)((out_count + tile - 1) / tile), kFastThreads, bytes, stream>>>(f);
        return cudaGetLastError();
    }
    Ac3Params p;
    p.in = in;
    p.in_kind = in_kind;
    p.in_first = in_first;
    p.nsamples = nsamples;
    p.out_first = out_first;
    p.out_count = out_count;
    p.out_i = out_i;
    p.out_q = out_q;
    p.taps = taps;
    const size_t smem = tile_smem(taps);
    static SmemAttr attr;
    cudaError_t e = attr.ensure(ac3_frontend_kernel, smem);
    if (e != cudaSuccess) return e;
    const unsigned grid = (unsigned)((out_count + kTile - 1) / kTile);
    ac3_frontend_kernel<<<grid, kAc3Threads, smem, stream>>>(p);
    return cudaGetLastError();
}

size_t ac3_tile_smem(const Ac3Taps& t) { return tile_smem(t); }

// ---- symbol-timing DPLL (host, ac3rf.py:200-299)

Ac3Dpll::Ac3Dpll(double fs) {
    symbol_distance = (int)std::nearbyint(fs / kSymbolRate);
    nominal_add = (int)((double)(1 << kCounterBits) * kSymbolRate / fs);
    prev_i.assign(symbol_distance, 0.0f);
    prev_q.assign(symbol_distance, 0.0f);
    const double pi = 3.14159265358979323846;
    const double omega = 2 * pi * 1800, zeta = 0.6, ts = 1.0 / kSymbolRate, gain = 0.3;
    g1 = (1 - std::exp(-2 * zeta * omega * ts)) / gain;
    g2 = (1 + std::exp(-2 * omega * zeta * ts) -
          2 * std::exp(-omega * zeta * ts) * std::cos(omega * ts * std::sqrt(1 - zeta * zeta))) /
         gain;
}

long long Ac3Dpll::reclock(const float* in_i, const float* in_q, long long n, uint8_t* out) {
    const int mask = (1 << kCounterBits) - 1;
    const int sd = symbol_distance;
    long long count = 0;
    for (long long i = 0; i < n; ++i) {
        float di, dq;
        if (i >= sd) {
            di = in_i[i - sd];
            dq = in_q[i - sd];
        } else {
            di = prev_i[i];
            dq = prev_q[i];
        }
        const float re = in_i[i] * di + in_q[i] * dq;
        const float im = in_q[i] * di - in_i[i] * dq;
        int cur;
        if (std::fabs(re) >= std::fabs(im))
            cur = re >= 0 ? 0 : 3;
        else
            cur = im >= 0 ? 1 : 2;
        if (cur != prev_symbol) {
            toggle_position = clk_counter;
            number_of_toggles += 1;
        }
        prev_symbol = cur;
        const int new_counter = (clk_counter + nominal_add + filter_out) & mask;
        filter_out = 0;
        if (new_counter < clk_counter) {
            out[count++] = (uint8_t)prev_symbol;
            const int error = number_of_toggles == 1 ? -(toggle_position - (1 << (kCounterBits - 1))) : 0;
            int es = (error_sum + error) & ((1 << kErrorSumBits) - 1);
            if (es >= (1 << (kErrorSumBits - 1))) es -= 1 << kErrorSumBits;
            error_sum = es;
            filter_out = (int)(error * g1 + error_sum * g2);  // truncation toward zero, as int()
            number_of_toggles = 0;
        }
        clk_counter = new_counter;
    }
    // keep the last symbol_distance samples (of previous tail + this input) for the next call
    if (n >= sd) {
        for (int k = 0; k < sd; ++k) {
            prev_i[k] = in_i[n - sd + k];
            prev_q[k] = in_q[n - sd + k];
        }
    } else {
        std::vector<float> ti(prev_i.begin() + n, prev_i.end()), tq(prev_q.begin() + n, prev_q.end());
        ti.insert(ti.end(), in_i, in_i + n);
        tq.insert(tq.end(), in_q, in_q + n);
        prev_i.swap(ti);
        prev_q.swap(tq);
    }
    return count;
}

}  // namespace ldg

// ---- C ABI

#include "ldgpu.h"

namespace {
thread_local std::string g_ac3_err;
int ac3_fail(int code, const std::string& m) {
    g_ac3_err = m;
    return code;
}
}  // namespace

struct ldg_ac3 {
    int device = 0;
    ldg::Ac3Taps taps{};
    std::vector<void*> allocs;
    std::mutex mu;
};

struct ldg_ac3_dpll {
    ldg::Ac3Dpll d;
    explicit ldg_ac3_dpll(double fs) : d(fs) {}
};

extern "C" {

const char* ldg_ac3_last_error(void) { return g_ac3_err.c_str(); }

void ldg_ac3_destroy(ldg_ac3* a) {
    if (!a) return;
    int prev = -1;
    cudaGetDevice(&prev);
    cudaSetDevice(a->device);
    for (void* p : a->allocs) cudaFree(p);
    if (prev >= 0) cudaSetDevice(prev);
    delete a;
}

int ldg_ac3_create(ldg_ac3** out, int32_t device, const float* hb19, int32_t n19, const float* hb23, int32_t n23,
                   const float* rrc, int32_t nrrc, int32_t lut_bits, const float* cos_lut, const float* sin_lut,
                   int32_t phase_step) {
    if (!out || !hb19 || !hb23 || !rrc || !cos_lut || !sin_lut) return ac3_fail(LDG_ERR_ARG, "ldg_ac3_create: NULL argument");
    *out = nullptr;
    if (n19 < 3 || n23 < 3 || nrrc < 1 || n19 > 255 || n23 > 255 || nrrc > 1023 || lut_bits < 4 || lut_bits > 20)
        return ac3_fail(LDG_ERR_ARG, "ldg_ac3_create: bad filter length or NCO table size");
    int prev = -1;
    cudaGetDevice(&prev);
    if (cudaSetDevice(device) != cudaSuccess) {
        cudaGetLastError();
        return ac3_fail(LDG_ERR_CUDA, "ldg_ac3_create: bad device");
    }
    ldg_ac3* a = new ldg_ac3();
    a->device = device;
    auto upload = [&](const void* src, size_t bytes) -> void* {
        void* d = nullptr;
        if (cudaMalloc(&d, bytes) != cudaSuccess) return nullptr;
        a->allocs.push_back(d);
        if (cudaMemcpy(d, src, bytes, cudaMemcpyHostToDevice) != cudaSuccess) return nullptr;
        return d;
    };
    bool ok = true;
    auto nz = [&](const float* h, int n, const float** val, const int** off, int* nnz) {
        std::vector<float> v;
        std::vector<int> o;
        for (int k = 0; k < n; ++k)
            if (h[k] != 0.0f) {
                v.push_back(h[k]);
                o.push_back(k);
            }
        *nnz = (int)v.size();
        *val = static_cast<const float*>(upload(v.data(), v.size() * sizeof(float)));
        *off = static_cast<const int*>(upload(o.data(), o.size() * sizeof(int)));
        ok = ok && *val && *off && *nnz > 0;
    };
    ldg::Ac3Taps& t = a->taps;
    t.n_hb19 = n19;
    t.n_hb23 = n23;
    t.n_rrc = nrrc;
    nz(hb19, n19, &t.hb19_val, &t.hb19_off, &t.n_hb19_nz);
    nz(hb23, n23, &t.hb23_val, &t.hb23_off, &t.n_hb23_nz);
    nz(rrc, nrrc, &t.rrc_val, &t.rrc_off, &t.n_rrc_nz);
    const size_t lut_bytes = (size_t(1) << lut_bits) * sizeof(float);
    t.cos_lut = static_cast<const float*>(upload(cos_lut, lut_bytes));
    t.sin_lut = static_cast<const float*>(upload(sin_lut, lut_bytes));
    t.lut_bits = lut_bits;
    t.phase_step = phase_step;
    ok = ok && t.cos_lut && t.sin_lut;
    // the reference's filter shapes take the register-blocked kernel: half-band
    // taps where it expects them, a matched filter without zero taps
    auto halfband = [](const float* h, int n) {
        for (int k = 0; k < n; ++k)
            if ((h[k] != 0.0f) != (k % 2 == 0 || k == n / 2)) return false;
        return true;
    };
    t.fast = n19 == 19 && n23 == 23 && nrrc >= 4 && nrrc <= ldg::kMaxAc3Rrc && t.n_rrc_nz == nrrc && halfband(hb19, 19) &&
             halfband(hb23, 23);
    if (t.fast) {
        for (int k = 0, j = 0; k < n19; ++k)
            if (hb19[k] != 0.0f) t.h_hb19[j++] = hb19[k];
        for (int k = 0, j = 0; k < n23; ++k)
            if (hb23[k] != 0.0f) t.h_hb23[j++] = hb23[k];
        for (int k = 0; k < ldg::kMaxAc3Rrc; ++k) t.h_rrc[k] = k < nrrc ? rrc[k] : 0.0f;
        const unsigned mask = (1u << lut_bits) - 1u;
        std::vector<float2> mix(size_t(1) << lut_bits);
        for (unsigned j = 0; j <= mask; ++j) {
            const unsigned ph = (unsigned)(((unsigned long long)j * (unsigned)phase_step) & mask);
            mix[j] = make_float2(cos_lut[ph], sin_lut[ph]);
        }
        t.mix = static_cast<const float2*>(upload(mix.data(), mix.size() * sizeof(float2)));
        ok = ok && t.mix;
    }
    if (prev >= 0) cudaSetDevice(prev);
    if (!ok || ldg::ac3_tile_smem(t) > 227 * 1024) {
        const std::string msg = cudaGetErrorString(cudaGetLastError());
        ldg_ac3_destroy(a);
        return ac3_fail(LDG_ERR_CUDA, "ldg_ac3_create: " + msg);
    }
    *out = a;
    return LDG_OK;
}

int ldg_ac3_frontend(ldg_ac3* a, const void* in, int32_t in_kind, int64_t in_first, int64_t nsamples,
                     int64_t out_first, int64_t out_count, float* out_i, float* out_q, void* stream) {
    if (!a || !in || !out_i || !out_q) return ac3_fail(LDG_ERR_ARG, "ldg_ac3_frontend: NULL argument");
    if (in_kind != LDG_IN_INT16 && in_kind != LDG_IN_FLOAT32) return ac3_fail(LDG_ERR_ARG, "ldg_ac3_frontend: bad in_kind");
    if (nsamples < 0 || in_first < 0 || out_first < 0 || out_count < 0)
        return ac3_fail(LDG_ERR_ARG, "ldg_ac3_frontend: negative size");
    // after n inputs the reference has produced ceil(n/16) outputs
    const long long avail = (in_first + nsamples + 15) / 16;
    if (out_first + out_count > avail)
        return ac3_fail(LDG_ERR_ARG, "ldg_ac3_frontend: outputs beyond the input (at most ceil(end/16))");
    if (out_count && in_first > 0 && 16 * out_first - ldg::ac3_history(a->taps) < in_first)
        return ac3_fail(LDG_ERR_ARG, "ldg_ac3_frontend: the input window does not cover the filters' history");
    if (out_count == 0) return LDG_OK;
    std::lock_guard<std::mutex> lk(a->mu);
    int prev = -1;
    cudaGetDevice(&prev);
    cudaSetDevice(a->device);
    auto is_dev = [](const void* p) {
        cudaPointerAttributes at;
        if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        return at.type == cudaMemoryTypeDevice || at.type == cudaMemoryTypeManaged;
    };
    const size_t esz = in_kind == LDG_IN_INT16 ? 2 : 4;
    const bool hin = !is_dev(in), hi = !is_dev(out_i), hq = !is_dev(out_q);
    cudaStream_t st = (cudaStream_t)stream;
    void *din = const_cast<void*>(in), *dio = out_i, *dqo = out_q;
    std::vector<void*> tmp;
    auto fail_cuda = [&](const char* what) {
        for (void* p : tmp) cudaFree(p);
        if (prev >= 0) cudaSetDevice(prev);
        return ac3_fail(LDG_ERR_CUDA, std::string("ldg_ac3_frontend: ") + what + ": " +
                                          cudaGetErrorString(cudaGetLastError()));
    };
    if (hin) {
        if (cudaMalloc(&din, nsamples * esz) != cudaSuccess) return fail_cuda("cudaMalloc");
        tmp.push_back(din);
        if (cudaMemcpyAsync(din, in, nsamples * esz, cudaMemcpyHostToDevice, st) != cudaSuccess) return fail_cuda("H2D");
    }
    if (hi) {
        if (cudaMalloc(&dio, out_count * 4) != cudaSuccess) return fail_cuda("cudaMalloc");
        tmp.push_back(dio);
    }
    if (hq) {
        if (cudaMalloc(&dqo, out_count * 4) != cudaSuccess) return fail_cuda("cudaMalloc");
        tmp.push_back(dqo);
    }
    if (ldg::launch_ac3_frontend(din, in_kind, in_first, nsamples, out_first, out_count, (float*)dio, (float*)dqo,
                                 a->taps, st) != cudaSuccess)
        return fail_cuda("launch");
    if (hi && cudaMemcpyAsync(out_i, dio, out_count * 4, cudaMemcpyDeviceToHost, st) != cudaSuccess) return fail_cuda("D2H");
    if (hq && cudaMemcpyAsync(out_q, dqo, out_count * 4, cudaMemcpyDeviceToHost, st) != cudaSuccess) return fail_cuda("D2H");
    if (!tmp.empty()) {
        if (cudaStreamSynchronize(st) != cudaSuccess) return fail_cuda("sync");
        for (void* p : tmp) cudaFree(p);
    }
    if (prev >= 0) cudaSetDevice(prev);
    return LDG_OK;
}

int ldg_ac3_dpll_create(ldg_ac3_dpll** out, double final_fs) {
    if (!out) return ac3_fail(LDG_ERR_ARG, "ldg_ac3_dpll_create: NULL argument");
    if (!(final_fs >= 2 * ldg::kSymbolRate) || final_fs > 1e9)
        return ac3_fail(LDG_ERR_ARG, "ldg_ac3_dpll_create: sample rate must be >= 2 x 288 kHz");
    *out = new ldg_ac3_dpll(final_fs);
    return LDG_OK;
}

void ldg_ac3_dpll_destroy(ldg_ac3_dpll* d) { delete d; }

int ldg_ac3_dpll_reclock(ldg_ac3_dpll* d, const float* in_i, const float* in_q, int64_t n, uint8_t* out,
                         int64_t* nout) {
    if (!d || (!in_i && n) || (!in_q && n) || (!out && n) || !nout)
        return ac3_fail(LDG_ERR_ARG, "ldg_ac3_dpll_reclock: NULL argument");
    if (n < 0) return ac3_fail(LDG_ERR_ARG, "ldg_ac3_dpll_reclock: negative length");
    *nout = d->d.reclock(in_i, in_q, n, out);
    return LDG_OK;
}

}  // extern "C"
