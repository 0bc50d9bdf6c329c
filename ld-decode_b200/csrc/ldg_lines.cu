// Per-line refinement of line locations on the GPU.
//
// ldg_lines_refine: the per-line refinement of Field.process() for all
// fields of a capture (pulse-level line locations from the host chain):
//   lines_hsync_kernel   one warp per line: refine_linelocs_hsync
//                        (core.py:2483-2551)
//   lines_burst_kernel   NTSC, one warp per line: compute_deriv_error
//                        (2553-2564), the colour-burst zero crossings of
//                        compute_line_bursts (2998-3047, clb_findbursts
//                        utils.py:1339-1368)
//   lines_pal_kernel     PAL, one CTA per field: compute_deriv_error,
//                        refine_linelocs_pilot twice (3054-3093) and
//                        fix_badlines (2566-2589) -> final line locations;
//                        the burst levels and line 7-19 burst crossings
//                        of determine_field_number (3095-3203).
//   pal_sequence_kernel  PAL, one CTA walking the fields in order: the
//                        8-field sequence (field phase IDs).
//   burst_round_kernel   NTSC, one CTA per field, twice, and
//   burst_verify_kernel  one CTA walking the fields in order: the burst
//                        phase of every line starts from the previous
//                        field's phase_adjust_median (compute_burst_offsets,
//                        core.py:3360-3388), two passes of the phase
//                        update, the field's median and its field-1/4 flag;
//                        speculated in parallel, verified in order.
//   burst_apply_kernel   NTSC, one CTA per field: refine_linelocs_burst
//                        (3390-3440), fix_badlines with linelocs2 as backup,
//                        the 117.25-degree subcarrier shift (3493-3495).
// Positions, fits and phases are FP64; samples are the float32 outputs.
#include <cmath>
#include <cstdint>
#include <mutex>
#include <string>

#include "ldg_attr.cuh"
#include "ldgpu.h"

struct ldg_ctx;

namespace ldg {
int lines_fail(int code, const std::string& msg);
int ctx_device(const ldg_ctx* c);
std::mutex& ctx_mutex(ldg_ctx* c);
}  // namespace ldg

namespace {

constexpr int kMaxL = LDG_CHAIN_MAX_LINES;
constexpr int kBurstLines = 266;    // compute_burst_offsets covers lines 0..265
constexpr int kPilotLines = 323;    // refine_linelocs_pilot covers lines 0..322
constexpr int kZc = 16;             // clb_findbursts' fixed zero-crossing slots
constexpr int kBurstThreads = 288;  // >= kBurstLines, whole warps
constexpr int kHsWin = 512;         // samples of a line's H-sync window in shared memory (40 MSPS needs ~480)

// --------------------------------------------------------- per-line helpers

// A line's window of a sample array staged in shared memory: x[i] from the
// window when i lies in [base, end), else from global memory.
struct WinView {
    const float* g;
    const float* s;
    long long base, end;
    __device__ __forceinline__ float operator[](long long i) const { return (i >= base && i < end) ? s[i - base] : g[i]; }
};

// np.median of a float32 slice (even length: float32 mean of the middle two)
template <class X>
__device__ double median_f32(const X& x, long long lo, long long hi, long long n) {
    lo = max(lo, 0LL);
    hi = min(hi, n);
    float v[128];
    int m = 0;
    for (long long i = lo; i < hi && m < 128; ++i) {
        const float t = x[i];
        int k = m++;
        while (k > 0 && v[k - 1] > t) {
            v[k] = v[k - 1];
            --k;
        }
        v[k] = t;
    }
    if (m == 0) return nan("");
    if (m & 1) return (double)v[m / 2];
    return (double)((v[m / 2 - 1] + v[m / 2]) * 0.5f);
}

// Warp-cooperative forms (every lane returns the same result).

// calczc (utils.py:812-841) over x[0, n): first crossing of `target` within
// count+1 samples from int(start); edge 0 decides rising/falling from
// x[int(start)].  Comparisons and the interpolation in FP64; 32 samples
// tested per step and the first crossing by ballot.
template <class X>
__device__ bool warp_calczc(const X& x, long long n, double start_offset, double target, int edge, double count,
                            double& out) {
    const int lane = threadIdx.x & 31;
    const long long s = (long long)start_offset;
    if (s < 0 || s >= n) return false;
    const long long icount = (long long)(count + 1);
    if (edge == 0) edge = (double)x[s] < target ? 1 : -1;
    const long long end = min(s + icount, n);
    for (long long c0 = s + 1; c0 < end; c0 += 32) {
        const long long i = c0 + lane;
        bool hit = false;
        if (i < end) {
            const double a = (double)x[i - 1], b = (double)x[i];
            hit = edge == 1 ? (a < target && b >= target) : (a > target && b <= target);
        }
        const unsigned m = __ballot_sync(0xffffffffu, hit);
        if (m) {
            const long long loc = c0 + __ffs(m) - 1;
            const double a = (double)x[loc - 1] - target, b = (double)x[loc] - target;
            out = (double)(loc - 1) + ((b - a != 0) ? -a / (-a + b) : 0.0);
            return true;
        }
    }
    return false;
}

template <class X>
__device__ void warp_minmax(const X& x, long long lo, long long hi, long long n, float& mn, float& mx) {
    const int lane = threadIdx.x & 31;
    lo = max(lo, 0LL);
    hi = min(hi, n);
    mn = INFINITY;
    mx = -INFINITY;
    for (long long i = lo + lane; i < hi; i += 32) {
        const float v = x[i];
        mn = fminf(mn, v);
        mx = fmaxf(mx, v);
    }
    for (int o = 16; o; o >>= 1) {
        mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
}

// np.median of a float32 slice of up to 64 samples: the warp sorts them
// (bitonic network over elements e = lane and e = lane + 32, unused ones
// +inf) and reads the middle one or two; longer slices fall back to one
// lane.  The middle values do not depend on how ties are ordered.
template <class X>
__device__ double warp_median_f32(const X& x, long long lo, long long hi, long long n) {
    const int lane = threadIdx.x & 31;
    lo = max(lo, 0LL);
    hi = min(hi, n);
    const int m = (int)max(hi - lo, 0LL);
    if (m == 0) return nan("");
    if (m > 64) {
        double r = 0;
        if (lane == 0) r = median_f32(x, lo, hi, n);
        return __shfl_sync(0xffffffffu, r, 0);
    }
    float v0 = lane < m ? x[lo + lane] : INFINITY;
    float v1 = lane + 32 < m ? x[lo + 32 + lane] : INFINITY;
#pragma unroll
    for (int k = 2; k <= 64; k <<= 1) {
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            if (j == 32) {
                // partners lane and lane + 32 in the same lane; ascending (k = 64)
                const float a = fminf(v0, v1), b = fmaxf(v0, v1);
                v0 = a;
                v1 = b;
            } else {
                const float p0 = __shfl_xor_sync(0xffffffffu, v0, j);
                const float p1 = __shfl_xor_sync(0xffffffffu, v1, j);
                const bool lower = (lane & j) == 0;  // this element is the pair's first
                const bool up0 = (lane & k) == 0, up1 = ((lane + 32) & k) == 0;
                v0 = (lower == up0) ? fminf(v0, p0) : fmaxf(v0, p0);
                v1 = (lower == up1) ? fminf(v1, p1) : fmaxf(v1, p1);
            }
        }
    }
    auto at = [&](int e) {
        const float a = __shfl_sync(0xffffffffu, v0, e & 31);
        const float b = __shfl_sync(0xffffffffu, v1, e & 31);
        return e < 32 ? a : b;
    };
    const float va = at((m - 1) / 2), vb = at(m / 2);
    if (m & 1) return (double)va;
    return (double)((va + vb) * 0.5f);
}

// get_linelen (core.py:1655-1672) with linecount + lineoffset = lc
__device__ double line_len(const double* ll, int line, int lc, double linelen) {
    double length;
    if (line >= lc) length = ll[line] - ll[line - 1];
    else if (line > 0) length = (ll[line + 1] - ll[line - 1]) / 2;
    else length = ll[line + 1] - ll[line];
    return length <= 0 ? linelen : length;
}

// second differences above 4 samples mark both later lines bad
__device__ void deriv_error_block(const double* ll, unsigned char* bad, int nl) {
    const int j = threadIdx.x;
    bool b1 = false;
    if (j + 2 < nl) b1 = fabs((ll[j + 2] - ll[j + 1]) - (ll[j + 1] - ll[j])) > 4;
    __syncthreads();
    if (b1) {
        bad[j + 1] = 1;
        bad[j + 2] = 1;
    }
    __syncthreads();
}

// fix_badlines' interpolation over good neighbours; reads ll, writes out
__device__ void fix_badlines_block(const double* ll, const unsigned char* bad, double* out, int nl, int firstcheck) {
    const int l = threadIdx.x;
    if (l < nl) {
        double v = ll[l];
        if (bad[l]) {
            int pg = l - 1;
            while (pg >= 0 && bad[pg]) --pg;
            int ng = l + 1;
            while (ng < nl && bad[ng]) ++ng;
            if (pg >= firstcheck && ng < nl) {
                const double gap = (ll[ng] - ll[pg]) / (double)(ng - pg);
                v = (gap * (double)(l - pg)) + ll[pg];
            }
        }
        out[l] = v;
    }
    __syncthreads();
}

// (key, index) pairs in a strict total order
__device__ __forceinline__ bool pair_less(double ka, int ia, double kb, int ib) {
    return ka < kb || (ka == kb && ia < ib);
}

// ascending bitonic sort of one (key, index) pair per lane across a warp
__device__ __forceinline__ void warp_sort_pairs(double& key, int& idx) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 2; k <= 32; k <<= 1) {
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            const double ok = __shfl_xor_sync(0xffffffffu, key, j);
            const int oi = __shfl_xor_sync(0xffffffffu, idx, j);
            const bool up = (lane & k) == 0;
            const bool lower = (lane & j) == 0;
            const bool partner_less = pair_less(ok, oi, key, idx);
            // ascending block: the lower lane keeps the smaller pair
            const bool take = lower == up ? partner_less : !partner_less;
            if (take) {
                key = ok;
                idx = oi;
            }
        }
    }
}

// number of pairs in a sorted run of 32 that order before (key, idx)
__device__ __forceinline__ int run_rank(const double* rk, const int* ri, double key, int idx) {
    int lo = 0;
#pragma unroll
    for (int step = 16; step > 0; step >>= 1)
        if (pair_less(rk[lo + step - 1], ri[lo + step - 1], key, idx)) lo += step;
    return lo + (pair_less(rk[lo], ri[lo], key, idx) ? 1 : 0);
}

struct LineParams {
    ldg_lines_args a;
    int system;
    double freq, linelen, linefreq0, samplesperline;
    double half_sync, lo_ok, hi_ok, hz_ire, fsc_mhz, pilot_mhz;
    struct BurstRec* rec;  // nfields x kBurstLines
    double* ll2;           // nfields x kMaxL (NTSC linelocs2)
    double* adjs;          // nfields x kBurstLines (NaN: none)
    int* field14;          // per field
};

// One line's colour-burst zero crossings as clb_findbursts uses them: the
// seed-independent part of zc_cycles, (bstart + zcs - s_rem) / zcburstdiv,
// for all 16 slots (unused slots hold zcs = 0), and the rising flags.
struct BurstRec {
    double cyc[kZc];
    int count, rising, valid, pad;
};

constexpr int kBurstWin = 128;  // samples of a line's colour burst

// The first set bit at or after j of a 128-bit mask, 128 when none.
__device__ __forceinline__ int next_bit(const unsigned (&m)[4], int j) {
#pragma unroll
    for (int w = 0; w < 4; ++w) {
        const int o = j - 32 * w;
        const unsigned v = o <= 0 ? m[w] : o >= 32 ? 0u : m[w] & (0xffffffffu << o);
        if (v) return 32 * w + __ffs(v) - 1;
    }
    return kBurstWin;
}

// compute_line_bursts up to the phase update: the zero crossings of the
// line's colour burst (they do not depend on the phase seed).  One warp: the
// burst's samples staged in shared memory, the sums in the samples' order by
// every lane (the two means side by side), and the search for crossings on
// bit masks of the samples.  The staged values are FP64, converted by one
// lane each: converted at every use, the conversions (16 per clock and SM)
// were the bound: 103 us for 89 fields, now 79 (ncu).
struct BurstWin {
    double b[kBurstWin + 1], d[kBurstWin];  // the two sums' reads on different banks
};

__device__ void warp_burst_record(const LineParams& P, const double* ll, int line, int lc, const float* burst,
                                  const float* demod, long long n, BurstWin& win, BurstRec* r) {
    const int lane = threadIdx.x & 31;
    const double l0 = ll[line];
    const long long s = (long long)l0;
    const double s_rem = l0 - (double)s;
    const double lfreq = P.samplesperline * line_len(ll, line, lc, P.linelen);
    const double fsc_inv = 1 / P.fsc_mhz;
    const long long bstart = (long long)(21 * fsc_inv * lfreq);
    const long long bend = (long long)(28 * fsc_inv * lfreq);
    const long long lo = s + bstart, hi = min(s + bend, n);
    if (lane == 0) {
        r->valid = 0;
        r->count = 0;
        r->rising = 0;
    }
    if (lo < 0 || hi <= lo) return;
    const int m = (int)min(hi - lo, (long long)kBurstWin);
    float vb[4], vd[4];  // this lane's samples
    __syncwarp();
#pragma unroll
    for (int w = 0; w < 4; ++w) {
        const int k = 32 * w + lane;
        vb[w] = k < m ? burst[lo + k] : 0.0f;
        vd[w] = k < m ? demod[lo + k] : 0.0f;
    }
#pragma unroll
    for (int w = 0; w < 4; ++w) {
        if (32 * w + lane < m) {
            win.b[32 * w + lane] = (double)vb[w];
            win.d[32 * w + lane] = (double)vd[w];
        }
    }
    __syncwarp();
    // odd lanes the demodulated video's sum, even lanes the burst's
    const double* src = (lane & 1) ? win.d : win.b;
    double acc = 0;
#pragma unroll 8
    for (int k = 0; k < m; ++k) acc += src[k];
    const float mean = (float)(acc / m);
    const float mean_f = __shfl_sync(0xffffffffu, mean, 0), mean_d = __shfl_sync(0xffffffffu, mean, 1);
    float mx = 0;
    __syncwarp();
#pragma unroll
    for (int w = 0; w < 4; ++w) {
        const int k = 32 * w + lane;
        if (k < m) {
            mx = fmaxf(mx, fabsf(vd[w] - mean_d));
            vb[w] = vb[w] - mean_f;
            win.b[k] = (double)vb[w];
        }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    __syncwarp();
    if ((double)mx > 30 * P.hz_ire) return;
    double m2 = 0;
#pragma unroll 8
    for (int k = 0; k < m; ++k) m2 += win.b[k];
    m2 /= m;
    double ss = 0;
#pragma unroll 8
    for (int k = 0; k < m; ++k) {
        const double d = win.b[k] - m2;
        ss += d * d;
    }
    const double threshold = sqrt(ss / m);
    // per sample: above the threshold, negative, a rising / falling crossing
    unsigned above[4], neg[4], up[4], down[4];
#pragma unroll
    for (int w = 0; w < 4; ++w) {
        const int k = 32 * w + lane;
        const float v = k < m ? vb[w] : 0.0f;
        float u = __shfl_up_sync(0xffffffffu, v, 1);  // the sample before
        const float last = w ? __shfl_sync(0xffffffffu, vb[w ? w - 1 : 0], 31) : 0.0f;
        if (lane == 0) u = last;
        above[w] = __ballot_sync(0xffffffffu, k < m && (double)fabsf(v) > threshold);
        neg[w] = __ballot_sync(0xffffffffu, v < 0);
        up[w] = __ballot_sync(0xffffffffu, k > 0 && k < m && u < 0 && v >= 0);
        down[w] = __ballot_sync(0xffffffffu, k > 0 && k < m && u > 0 && v <= 0);
    }
    const double zcburstdiv = (lfreq * fsc_inv) / 2;
    float mine = 0.0f;  // lane k: slot k's crossing
    int c = 0, rising = 0, j = 0;
    while (c < kZc) {
        j = next_bit(above, j);
        if (j >= m - 1) break;
        const unsigned nw = j < 64 ? (j < 32 ? neg[0] : neg[1]) : (j < 96 ? neg[2] : neg[3]);
        const bool is_neg = (nw >> (j & 31)) & 1u;
        // calczc from j: the first crossing of its sign within 16 samples
        const unsigned cross[4] = {is_neg ? up[0] : down[0], is_neg ? up[1] : down[1], is_neg ? up[2] : down[2],
                                   is_neg ? up[3] : down[3]};
        const int loc = next_bit(cross, j + 1);
        if (loc >= min(j + 17, m)) break;
        const double a = win.b[loc - 1], b = win.b[loc];
        const double zc = (double)(loc - 1) + ((b - a != 0) ? -a / (-a + b) : 0.0);
        if (is_neg) rising |= 1 << c;
        if (lane == c) mine = (float)zc;
        ++c;
        j = (int)zc + 1;
    }
    if (lane < kZc) r->cyc[lane] = ((double)bstart + (double)mine - s_rem) / zcburstdiv;
    if (lane == 0) {
        r->valid = 1;
        r->count = c;
        r->rising = rising;
    }
}

// FieldPAL.get_burstlevel (core.py:3095-3104, numpy slice semantics at
// the window's end): the RMS of demod over 2.4 us from 5.5 us into line
// l_adj, less its mean, times sqrt(2); NaN for the reference's None (a
// sample above 30 IRE) or an empty slice.  lc = linecount + lineoffset of
// the moment (get_linelen's last-line rule).
struct LevelWindow {
    long long lo, hi;  // samples [lo, hi); empty when hi <= lo
};

__device__ __forceinline__ LevelWindow pal_level_window(const LineParams& P, const double* ll, int l_adj, int lc,
                                                        long long n) {
    const double begin = ll[l_adj] + 5.5 * (P.samplesperline * line_len(ll, l_adj, lc, P.linelen));
    const double length = 2.4 * (P.samplesperline * P.linelen);
    LevelWindow w{(long long)begin, min((long long)(begin + length + 1.0), n)};
    if (w.lo < 0) w.hi = w.lo;
    return w;
}

__device__ double pal_burstlevel(const float* x, int m, double hz_ire) {
    if (m <= 0) return nan("");
    double acc = 0;  // float32 samples near 7 MHz: this double sum is exact
#pragma unroll 4
    for (int k = 0; k < m; ++k) acc += (double)x[k];
    const float mean_f = (float)(acc / (double)m);
    float mx = -INFINITY;
    double s1 = 0;
#pragma unroll 4
    for (int k = 0; k < m; ++k) {
        const float v = x[k] - mean_f;
        mx = fmaxf(mx, v);
        s1 += (double)v;
    }
    if ((double)mx > 30 * hz_ire) return nan("");
    const double mu = s1 / (double)m;
    double ss = 0;
#pragma unroll 4
    for (int k = 0; k < m; ++k) {
        const double d = (double)(x[k] - mean_f) - mu;
        ss += d * d;
    }
    return sqrt(ss / (double)m) * 1.4142135623730951;
}

// _angle_mean_phase / phase_distance helpers (core.py:3085-3093)
__device__ __forceinline__ double phase_distance(double x, double c) {
    double d = (x - floor(x)) - c;
    if (d < -0.5) d += 1;
    else if (d > 0.5) d -= 1;
    return d;
}

constexpr int kRefineWarps = 8;      // lines per CTA of the per-line kernels
constexpr int kPalThreads = 1024;    // one CTA per PAL field
constexpr int kLevelLines = 303;     // lines 11 .. 312 and line 6 of the sequence
constexpr int kLevelWarps = (kLevelLines + 31) / 32;
constexpr int kStage = 3;            // lines of a warp whose levels' samples are loaded at once
constexpr int kLevelWin = 99;        // samples of a burst level (odd: lanes on different banks; 40 MSPS needs 98)
static_assert(kMaxL <= kPalThreads && kLevelWarps <= kPalThreads / 32 - 4, "one thread per line");
static_assert(kLevelLines <= kPilotLines && kLevelWin <= 128, "the levels' windows");

// For each of the first `count` threads the largest v of the threads up to and
// including it.  All threads of the CTA; wsum: 32 ints.
__device__ __forceinline__ int block_max_scan(int v, int* wsum) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v = max(v, y);
    }
    if (lane == 31) wsum[warp] = v;
    __syncthreads();
    for (int w = 0; w < warp; ++w) v = max(v, wsum[w]);
    __syncthreads();
    return v;
}

// A pilot pass's windows and crossings.
struct PilotWin {
    long long st[kPilotLines];              // the line's samples: pilot[st, st + m)
    int m[kPilotLines];
    int loc[kPilotLines];                   // the crossing lies between loc - 1 and loc (st's offset); 0: none
    float a[kPilotLines], b[kPilotLines];   // those two samples
    double mean;                            // the mean phase
};

constexpr int kPilotLoads = 8;  // loads in flight per line and lane (40 MSPS needs 241 samples)

// One refine_linelocs_pilot pass over ll (shared), in place: a thread per line
// computes its window, a warp per two lines finds their pilots' peaks and the
// crossings after them, a thread per line the rest.  The line's FP64 work --
// four divisions -- is done once per line, not by every lane of its warp: the
// FP64 unit issues one warp's instruction per clock and SM, and bounded the
// pass so.  What is left is mostly latency: the ordered sums of 323 terms, the
// sines and cosines, the arctangent.
__device__ void pilot_pass(const LineParams& P, double* ll, const float* pilot, long long n, PilotWin& W, double* zcs,
                           double* red, int* wsum) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int l = threadIdx.x;
    double pl = 0, lsoffset = 0;
    if (l < kPilotLines) {
        double adjfreq = P.freq;
        if (l > 1) adjfreq /= (ll[l] - ll[l - 1]) / P.linelen;
        pl = (adjfreq / P.pilot_mhz) / 2;
        const double b0 = ll[l];
        const long long st = (long long)(b0 + 0.0);
        long long sp = (long long)(b0 + 6 * P.linefreq0 + 0.0 + 1);
        sp = min(sp, n);
        lsoffset = b0 - (double)st;
        const bool some = st >= 0 && sp > st;
        W.st[l] = some ? st : 0;
        W.m[l] = some ? (int)(sp - st) : 0;
    }
    __syncthreads();
    for (int l0 = warp; l0 < kPilotLines; l0 += 2 * (kPalThreads / 32)) {
        float v[2][kPilotLoads];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int line = l0 + q * (kPalThreads / 32);
            const int m = line < kPilotLines ? W.m[line] : 0;
            const float* seg = pilot + (line < kPilotLines ? W.st[line] : 0);
#pragma unroll
            for (int j = 0; j < kPilotLoads; ++j) v[q][j] = lane + 32 * j < m ? seg[lane + 32 * j] : -0.0f;
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int line = l0 + q * (kPalThreads / 32);
            if (line >= kPilotLines) break;
            const int m = W.m[line];
            const float* seg = pilot + W.st[line];
            // the first of the largest magnitudes: magnitudes as integers, one
            // up, so that 0 stands for none (a NaN is not larger than anything)
            unsigned best = 0;
            int peak = 0x7fffffff;
            auto look = [&](float x, int k) {
                const unsigned key = k < m && fabsf(x) >= 0.0f ? __float_as_uint(fabsf(x)) + 1u : 0u;
                if (key > best) {
                    best = key;
                    peak = k;
                }
            };
#pragma unroll
            for (int j = 0; j < kPilotLoads; ++j) look(v[q][j], lane + 32 * j);
            for (int k = lane + 32 * kPilotLoads; k < m; k += 32) look(seg[k], k);
            const unsigned most = __reduce_max_sync(0xffffffffu, best);
            peak = (int)__reduce_min_sync(0xffffffffu, best == most ? (unsigned)peak : 0x7fffffffu);
            if (peak == 0x7fffffff) peak = 0;
            // calczc from the peak to 0 within 16 samples
            const float x0 = lane <= 16 && peak + lane < m ? seg[peak + lane] : 0.0f;
            const float x1 = __shfl_down_sync(0xffffffffu, x0, 1);
            const float xp = __shfl_sync(0xffffffffu, x0, 0);
            const bool hit = lane < 16 && peak + 1 + lane < m && (xp < 0 ? x0 < 0 && x1 >= 0 : x0 > 0 && x1 <= 0);
            const unsigned hits = __ballot_sync(0xffffffffu, hit);
            const int first = __ffs(hits) - 1;
            if (hits ? lane == first : lane == 0) {
                W.loc[line] = hits ? peak + 1 + first : 0;
                W.a[line] = x0;
                W.b[line] = x1;
            }
        }
    }
    __syncthreads();
    bool good = false;
    if (l < kPilotLines) {
        const int loc = W.loc[l];
        good = loc > 0;
        if (good) {
            const double a = (double)W.a[l], b = (double)W.b[l];
            const double zb = (double)(loc - 1) + ((b - a != 0) ? -a / (-a + b) : 0.0);
            zcs[l] = (zb - lsoffset) / pl;
        }
    }
    // a line without a crossing repeats the previous line's value (0 before any)
    const int from = block_max_scan(good ? l : -1, wsum);
    const double z = l < kPilotLines && from >= 0 ? zcs[from] : 0.0;
    // mean phase of the fractional parts
    if (l < kPilotLines) {
        const double x2 = z - (double)(int)z;
        const double th = x2 * 3.14159265358979323846 * 2;
        red[l] = cos(th);
        red[kMaxL + 1 + l] = sin(th);
    }
    __syncthreads();
    if (warp == 0) {  // the two sums in line order, side by side (on different banks)
        const double* v = red + (lane & 1 ? kMaxL + 1 : 0);
        double a = 0;
#pragma unroll 8
        for (int k = 0; k < kPilotLines; ++k) a += v[k];
        const double c = __shfl_sync(0xffffffffu, a, 0), s = __shfl_sync(0xffffffffu, a, 1);
        double am = atan2(s / kPilotLines, c / kPilotLines) / (3.14159265358979323846 * 2);
        if (am < 0) am = 1 + am;
        if (lane == 0) W.mean = am;
    }
    __syncthreads();
    if (l < kPilotLines) ll[l] += phase_distance(z, W.mean) * pl;
    __syncthreads();
}

// refine_linelocs_hsync, one warp per line: the line location into P.ll2, its
// flag into linebad.  Each line's samples (from just before its search start
// to past its porch) are staged in shared memory by one burst of independent
// loads, so the searches below do not wait on one global load after another.
// Bound: latency, one line's chain of searches.  Lines of a field are
// independent, so they spread over the chip.  With one CTA walking a field's
// lines, and one thread per line on the bursts or pilots after it, this stage
// took 220 us for one NTSC field and 355 us for 15 PAL ones; with a warp per
// line (ncu) 7 + 15 us and, PAL, 14 us here (the rest: lines_pal_kernel).
__global__ void __launch_bounds__(32 * kRefineWarps) lines_hsync_kernel(const __grid_constant__ LineParams P) {
    const int f = P.a.first_field + blockIdx.y;
    const ldg_lines_args& a = P.a;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int li = blockIdx.x * kRefineWarps + warp;
    if (li >= a.proclines) return;
    const long long base = a.startloc[f];
    const long long n = min((long long)a.wlen[f], (long long)(a.capture_len - base));
    const float* d05 = a.d05 + base;
    __shared__ float win[kRefineWarps][kHsWin];
    const double start = a.linelocs1[(long long)f * kMaxL + li];
    bool b = a.linebad1[(long long)f * kMaxL + li];
    double v2 = start;
    if ((li >= 3 && li <= 6) || (P.system == 1 && li >= 1 && li <= 2)) {
        b = true;
    } else {
        const double l1 = start - P.freq;
        const long long wb = max((long long)l1 - 64, 0LL);
        const long long we = min(wb + kHsWin, n);
        float* w = win[warp];
        for (long long i = wb + lane; i < we; i += 32) w[i - wb] = d05[i];
        __syncwarp();
        const WinView x{d05, w, wb, we};
        double zc;
        if (warp_calczc(x, n, l1, P.half_sync, 0, P.freq * 2, zc) && !b) {
            v2 = zc;
            float mn, mx;
            warp_minmax(x, (long long)(zc - (P.freq * 0.75)), (long long)(zc + (P.freq * 8)), n, mn, mx);
            if ((double)mn < P.lo_ok || (double)mx > P.hi_ok) {
                b = true;
            } else {
                const double porch =
                    warp_median_f32(x, (long long)(zc + (P.freq * 8)), (long long)(zc + (P.freq * 9)), n);
                const double sync =
                    warp_median_f32(x, (long long)(zc + (P.freq * 1)), (long long)(zc + (P.freq * 2.5)), n);
                double zc2;
                if (warp_calczc(x, n, l1, (porch + sync) / 2, 0, 400, zc2) && fabs(zc2 - zc) < (P.freq / 2))
                    v2 = zc2;
                else
                    b = true;
            }
        } else {
            b = true;
        }
    }
    if (lane == 0) {
        P.ll2[(long long)f * kMaxL + li] = b ? start : v2;
        a.linebad[(long long)f * kMaxL + li] = b;
    }
}

// NTSC, one warp per line: the second differences' bad-line flags (a line's
// flag depends on the two lines before it and the one after), linelocs2 out,
// the line's burst zero crossings.
__global__ void __launch_bounds__(32 * kRefineWarps) lines_burst_kernel(const __grid_constant__ LineParams P) {
    const int f = P.a.first_field + blockIdx.y;
    const ldg_lines_args& a = P.a;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int l = blockIdx.x * kRefineWarps + warp, nl = a.proclines;
    if (l >= nl) return;
    const double* ll = P.ll2 + (long long)f * kMaxL;
    if (lane == 0) {
        bool bad = false;
        if (l >= 1 && l + 1 < nl) bad |= fabs((ll[l + 1] - ll[l]) - (ll[l] - ll[l - 1])) > 4;
        if (l >= 2) bad |= fabs((ll[l] - ll[l - 1]) - (ll[l - 1] - ll[l - 2])) > 4;
        if (bad) a.linebad[(long long)f * kMaxL + l] = 1;
        if (a.linelocs2) a.linelocs2[(long long)f * kMaxL + l] = ll[l];
    }
    if (l >= kBurstLines) return;
    const long long base = a.startloc[f];
    const long long n = min((long long)a.wlen[f], (long long)(a.capture_len - base));
    __shared__ BurstWin win[kRefineWarps];
    warp_burst_record(P, ll, l, a.linecount[f], a.burst + base, a.demod + base, n, win[warp],
                      P.rec + (long long)f * kBurstLines + l);
}

// PAL, one CTA per field: second differences, two pilot passes, fix_badlines
// (no backup, lines from 0), the inputs of the 8-field sequence.  Bound: one
// field's chain of stages.  15 fields (ncu): 105 us with every lane dividing
// for its warp's line, one line's loads in flight per warp, the bursts after the
// levels and the levels' median by a block-wide sort; 51 us so.
__global__ void __launch_bounds__(kPalThreads) lines_pal_kernel(const __grid_constant__ LineParams P) {
    extern __shared__ float lev[];  // kLevelLines x kLevelWin
    const int f = P.a.first_field + blockIdx.x;
    const ldg_lines_args& a = P.a;
    const long long base = a.startloc[f];
    const long long n = min((long long)a.wlen[f], (long long)(a.capture_len - base));
    const int nl = a.proclines;
    __shared__ double ll[kMaxL], tmp[kMaxL], red[2 * kMaxL + 1], mid[2];
    __shared__ unsigned char bad[kMaxL];
    __shared__ int wsum[32], runs[kLevelWarps][32];
    __shared__ PilotWin pw;
    __shared__ BurstWin win[4];
    static_assert(2 * kMaxL + 1 >= kLevelWarps * 32, "the levels' sorted runs");
    const int i = threadIdx.x, lane = i & 31, warp = i >> 5;
    if (i < nl) {
        ll[i] = P.ll2[(long long)f * kMaxL + i];
        bad[i] = a.linebad[(long long)f * kMaxL + i];
    }
    __syncthreads();
    deriv_error_block(ll, bad, nl);
    pilot_pass(P, ll, a.pilot + base, n, pw, tmp, red, wsum);
    pilot_pass(P, ll, a.pilot + base, n, pw, tmp, red, wsum);
    deriv_error_block(ll, bad, nl);
    fix_badlines_block(ll, bad, tmp, nl, 0);
    if (i < nl) {
        a.linelocs[(long long)f * kMaxL + i] = tmp[i];
        a.linebad[(long long)f * kMaxL + i] = bad[i];
    }
    __syncthreads();
    // inputs of the 8-field sequence (FieldPAL.process, core.py:3212-3236):
    // calc_burstmedian runs while the field's line count and offset are still
    // compute_linelocs' (263 / 262 and 0), determine_field_number after they
    // become 312 / 313 and 2 / 3
    const bool isf = a.isfirst[f] != 0;
    const int lc_med = isf ? 263 : 262;
    const int off = isf ? 2 : 3;
    const int lc_seq = (isf ? 312 : 313) + off;
    const float* demod = a.demod + base;
    // the levels' samples staged a warp per line, kStage lines' loads in
    // flight, then a thread per line sums them in order; beside it the last
    // four warps take the burst crossings of lines 7-19
    const LevelWindow lw = i >= kLevelLines       ? LevelWindow{0, 0}
                           : i < kLevelLines - 1 ? pal_level_window(P, tmp, 11 + i, lc_med, n)
                                                 : pal_level_window(P, tmp, 6 + off, lc_seq, n);
    const int lm = (int)max(lw.hi - lw.lo, 0LL);
    if (i < kLevelLines) {
        pw.st[i] = lm ? lw.lo : 0;
        pw.m[i] = lm <= kLevelWin ? lm : 0;
    }
    __syncthreads();
    for (int e0 = warp; e0 < kLevelLines; e0 += kStage * (kPalThreads / 32)) {
        float v[kStage][4];
#pragma unroll
        for (int q = 0; q < kStage; ++q) {
            const int e = e0 + q * (kPalThreads / 32);
            const int m = e < kLevelLines ? pw.m[e] : 0;
            const float* x = demod + (e < kLevelLines ? pw.st[e] : 0);
#pragma unroll
            for (int j = 0; j < 4; ++j) v[q][j] = lane + 32 * j < m ? x[lane + 32 * j] : 0.0f;
        }
#pragma unroll
        for (int q = 0; q < kStage; ++q) {
            const int e = e0 + q * (kPalThreads / 32);
            const int m = e < kLevelLines ? pw.m[e] : 0;
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (lane + 32 * j < m) lev[e * kLevelWin + lane + 32 * j] = v[q][j];
        }
    }
    __syncthreads();
    double lvl = INFINITY;
    if (i < kLevelLines) {
        const double b = pal_burstlevel(lm <= kLevelWin ? lev + i * kLevelWin : demod + lw.lo, lm, P.hz_ire);
        if (i == kLevelLines - 1) P.adjs[(long long)f * kBurstLines] = b;
        else if (!isnan(b)) lvl = b;
    } else if (warp >= kPalThreads / 32 - 4) {
        const int j = warp - (kPalThreads / 32 - 4);
        warp_burst_record(P, tmp, 7 + 4 * j + off, lc_seq, a.burst + base, demod, n, win[j],
                          P.rec + (long long)f * kBurstLines + j);
    }
    // their median: a level's rank is the sum of its positions in the warps' sorted runs
    const bool level = lvl != INFINITY;
    if (warp < kLevelWarps) {
        double key = lvl;
        int idx = i;
        warp_sort_pairs(key, idx);
        red[i] = key;
        runs[warp][lane] = idx;
    }
    const int cnt = __syncthreads_count(level);
    if (level) {
        int r = 0;
#pragma unroll
        for (int w = 0; w < kLevelWarps; ++w) r += run_rank(red + 32 * w, runs[w], lvl, i);
        if (r == (cnt - 1) / 2) mid[0] = lvl;
        if (r == cnt / 2) mid[1] = lvl;
    }
    __syncthreads();
    if (i == 0) {
        const double med = cnt & 1 ? mid[1] : (mid[0] + mid[1]) / 2.0;
        P.adjs[(long long)f * kBurstLines + 1] = cnt ? med / P.hz_ire : 0.0;
    }
}

// np.median of 16 doubles (mean of the two middle ones): Batcher's
// odd-even merge sort network (63 compare-exchanges, the values stay in
// registers)
#define LDG_CS(a, b)                 \
    {                                \
        const double x_ = v[a];      \
        const double y_ = v[b];      \
        if (x_ > y_) {               \
            v[a] = y_;               \
            v[b] = x_;               \
        }                            \
    }
__device__ __forceinline__ double median16(double* v) {
    LDG_CS(0, 1) LDG_CS(2, 3) LDG_CS(4, 5) LDG_CS(6, 7)
    LDG_CS(8, 9) LDG_CS(10, 11) LDG_CS(12, 13) LDG_CS(14, 15)
    LDG_CS(0, 2) LDG_CS(1, 3) LDG_CS(4, 6) LDG_CS(5, 7)
    LDG_CS(8, 10) LDG_CS(9, 11) LDG_CS(12, 14) LDG_CS(13, 15)
    LDG_CS(1, 2) LDG_CS(5, 6) LDG_CS(9, 10) LDG_CS(13, 14)
    LDG_CS(0, 4) LDG_CS(1, 5) LDG_CS(2, 6) LDG_CS(3, 7)
    LDG_CS(8, 12) LDG_CS(9, 13) LDG_CS(10, 14) LDG_CS(11, 15)
    LDG_CS(2, 4) LDG_CS(3, 5) LDG_CS(10, 12) LDG_CS(11, 13)
    LDG_CS(1, 2) LDG_CS(3, 4) LDG_CS(5, 6) LDG_CS(9, 10)
    LDG_CS(11, 12) LDG_CS(13, 14) LDG_CS(0, 8) LDG_CS(1, 9)
    LDG_CS(2, 10) LDG_CS(3, 11) LDG_CS(4, 12) LDG_CS(5, 13)
    LDG_CS(6, 14) LDG_CS(7, 15) LDG_CS(4, 8) LDG_CS(5, 9)
    LDG_CS(6, 10) LDG_CS(7, 11) LDG_CS(2, 4) LDG_CS(3, 5)
    LDG_CS(6, 8) LDG_CS(7, 9) LDG_CS(10, 12) LDG_CS(11, 13)
    LDG_CS(1, 2) LDG_CS(3, 4) LDG_CS(5, 6) LDG_CS(7, 8)
    LDG_CS(9, 10) LDG_CS(11, 12) LDG_CS(13, 14)
    return (v[kZc / 2 - 1] + v[kZc / 2]) / 2.0;
}
#undef LDG_CS

// ---- NTSC burst phase of every field (compute_burst_offsets, core.py:3360-3388)
//
// Each field's lines start clb_findbursts' phase update from the previous
// field's phase_adjust_median, so the fields form a chain.  The seed enters
// only through the first pass's rounding int(cyc + .5) of every slot: for
// all seeds that leave those roundings as they are, the first pass ends at
// the same phase (the median of the rounded deviations, which moves with
// the seed), so the second pass, the line's adjustment, its rising count
// and the field's median are the same up to the last bits of the FP64
// arithmetic.  So the chain runs as
//   round 1  every field of the range at once, seeded with 0 (the range's
//            first field with its true seed): its median;
//   rounds 2 .. kBurstRounds  every field at once seeded with the round
//            before's median of the field before it (each round carries the
//            true seeds at least one field further, and a seed a few
//            thousandths of a cycle off already decides most fields); the
//            last round keeps adjustments, field-1/4 flag, median, and the
//            interval of seeds that gives the same roundings (with a
//            margin of 1e-9 cycles, also around the second pass's
//            roundings); a field with a valid line without zero crossings
//            (its adjustment is the seed itself) has none;
//   verify   one CTA walking the range in order with the true seeds: a
//            field whose true seed is the last round's seed or lies in its
//            interval keeps that round's results, any other is computed
//            again from its true seed.
// The integer results (rising counts, field-1/4 flags) are those of the
// fields in order; the adjustments and medians agree with them to the
// last bits (kept within 1e-9 of the host restatement by the tests).

constexpr int kBurstWarps = kBurstThreads / 32;
constexpr double kBurstMargin = 1e-9;

struct BurstSmem {
    double rkey[kBurstWarps][32];
    int ridx[kBurstWarps][32];
    double med2[2];
    double lo[kBurstWarps], hi[kBurstWarps];
    double pam, flo, fhi, seed;
    int xonly, next;
};

// The cell of x that int(x + .5) (truncation toward zero) maps to rnd:
// [r - .5, r + .5) for r >= 1, (-1.5, .5) for r = 0, (r - 1.5, r - .5] for r <= -1.
__device__ __forceinline__ void round_cell(int rnd, double& lo, double& hi) {
    lo = rnd >= 1 ? rnd - .5 : rnd - 1.5;
    hi = rnd >= 1 ? rnd + .5 : (rnd == 0 ? .5 : rnd - .5);
}

// One field's burst phase update from seed `prev` (the previous field's
// phase_adjust_median; 0 without one), lines in parallel: two passes of
// clb_findbursts' phase update per line, the field's median from per-warp
// sorted runs (a value's rank is the sum of its positions in the runs), its
// rising count.  All kBurstThreads threads call it; `cur` is the calling
// thread's line record.  Writes the lines' adjustments to adjs_f (NaN: none)
// and the field-1/4 flag to *field14_f when given; leaves the median times 2
// in sm.pam and, with `interval`, the seeds giving the same roundings in
// (sm.flo, sm.fhi) and sm.xonly set when the result depends on the seed
// otherwise.  Ends with the CTA in step.
__device__ void burst_field(const BurstRec& cur, double prev, double* adjs_f, int* field14_f, bool interval,
                            BurstSmem& sm) {
    const int l = threadIdx.x, lane = l & 31, warp = l >> 5;
    const bool line = l < kBurstLines;
    double adj = INFINITY;
    bool ok = false, rising = false, xo = false;
    double plo = -INFINITY, phi = INFINITY;
    if (line && cur.valid) {
        double pa = -prev;
        int rising_count = 0;
        for (int pass = 0; pass < 2; ++pass) {
            rising_count = 0;
            if (cur.count) {
                double dev[kZc];
                int odd = 0;
#pragma unroll
                for (int k = 0; k < kZc; ++k) {
                    const double cyc = cur.cyc[k] + pa;
                    const int rnd = (int)(cyc + .5);
                    if (rnd % 2 != 0) odd |= 1 << k;
                    dev[k] = (double)rnd - cyc;
                    if (interval) {
                        double clo, chi;
                        round_cell(rnd, clo, chi);
                        if (pass == 0) {
                            // seeds s with cur.cyc[k] - s in the cell
                            plo = fmax(plo, cur.cyc[k] - chi);
                            phi = fmin(phi, cur.cyc[k] - clo);
                        } else if (!(fmin(cyc - clo, chi - cyc) > kBurstMargin)) {
                            xo = true;
                        }
                    }
                }
                pa += median16(dev);
                rising_count = __popc((unsigned)(cur.rising ^ odd) & 0xffffu);
            } else {
                xo = true;  // no crossings: the line's adjustment is the seed itself
            }
        }
        rising = (double)rising_count > ((double)cur.count / 2);
        adj = (-pa) / 2;
        ok = true;
    }
    if (line && adjs_f) adjs_f[l] = ok ? adj : nan("");
    double sk = adj;
    int si = l;
    warp_sort_pairs(sk, si);
    sm.rkey[warp][lane] = sk;
    sm.ridx[warp][lane] = si;
    if (interval) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            plo = fmax(plo, __shfl_xor_sync(0xffffffffu, plo, o));
            phi = fmin(phi, __shfl_xor_sync(0xffffffffu, phi, o));
        }
        if (lane == 0) {
            sm.lo[warp] = plo;
            sm.hi[warp] = phi;
        }
    }
    const int cnt = __syncthreads_count(ok);
    const int rsum = __syncthreads_count(ok && !(l % 2) && rising);
    const int xany = __syncthreads_or(xo);
    if (ok) {
        int r = 0;
#pragma unroll
        for (int w = 0; w < kBurstWarps; ++w) r += run_rank(sm.rkey[w], sm.ridx[w], adj, l);
        if (cnt & 1) {
            if (r == cnt / 2) sm.med2[0] = sm.med2[1] = adj;
        } else {
            if (r == cnt / 2 - 1) sm.med2[0] = adj;
            if (r == cnt / 2) sm.med2[1] = adj;
        }
    }
    __syncthreads();
    if (l == 0) {
        // np.median of an empty list is NaN, which the reference then carries forward
        const double med = cnt ? (sm.med2[0] + sm.med2[1]) / 2.0 : nan("");
        sm.pam = med * 2;
        if (field14_f) *field14_f = rsum > (cnt / 4);
        if (interval) {
            double a = -INFINITY, b = INFINITY;
            for (int w = 0; w < kBurstWarps; ++w) {
                a = fmax(a, sm.lo[w]);
                b = fmin(b, sm.hi[w]);
            }
            sm.flo = a;
            sm.fhi = b;
            sm.xonly = xany || isnan(prev);
        }
    }
    __syncthreads();
}

// The true seed of the range's first field: the field before it (a later
// range continues from the previous range's output) or the caller's.
__device__ __forceinline__ double range_seed(const LineParams& P) {
    const ldg_lines_args& a = P.a;
    return a.first_field > 0 ? a.phase_adjust[a.first_field - 1]
                             : (a.prev_phase_adjust_dev ? *a.prev_phase_adjust_dev : a.prev_phase_adjust);
}

constexpr int kBurstRounds = 4;  // rounds before the verification walk

struct BurstSpec {
    double* out1;   // the medians x 2 per field of the odd rounds
    double* out2;   // ... of the even rounds
    double* seed2;  // the last round's seed per field
    double* lo;     // the last round's interval of seeds with the same roundings
    double* hi;
    int* xonly;     // the last round's result depends on the seed otherwise
};

// Round `round` (1 .. kBurstRounds): one CTA per field of the range, seeded
// with 0 (round 1) or with the previous round's median of the field before.
__global__ void __launch_bounds__(kBurstThreads) burst_round_kernel(const __grid_constant__ LineParams P, int round, const __grid_constant__ BurstSpec B) {
    __shared__ BurstSmem sm;
    const ldg_lines_args& a = P.a;
    const int f = a.first_field + blockIdx.x;
    double seed = 0.0;
    if (a.has_prev[f]) {
        if (f == a.first_field) seed = range_seed(P);
        else if (round > 1) seed = (round & 1 ? B.out2 : B.out1)[f - 1];
    }
    BurstRec cur;
    cur.valid = 0;
    if (threadIdx.x < kBurstLines) cur = P.rec[(long long)f * kBurstLines + threadIdx.x];
    if (round < kBurstRounds) {
        burst_field(cur, seed, nullptr, nullptr, false, sm);
        if (threadIdx.x == 0) (round & 1 ? B.out1 : B.out2)[f] = sm.pam;
    } else {
        burst_field(cur, seed, P.adjs + (long long)f * kBurstLines, P.field14 + f, true, sm);
        if (threadIdx.x == 0) {
            a.phase_adjust[f] = sm.pam;
            B.seed2[f] = seed;
            B.lo[f] = sm.flo;
            B.hi[f] = sm.fhi;
            B.xonly[f] = sm.xonly;
        }
    }
}

// The fields of the range in order with their true seeds: the CTA stages
// the last round's seeds, intervals, flags and medians of up to kBurstScan
// fields in shared memory, thread 0 walks over the fields that round got
// right; a field it did not is computed again by the whole CTA.
constexpr int kBurstScan = 512;

__global__ void __launch_bounds__(kBurstThreads) burst_verify_kernel(const __grid_constant__ LineParams P, const __grid_constant__ BurstSpec B) {
    __shared__ BurstSmem sm;
    __shared__ double s_seed2[kBurstScan], s_lo[kBurstScan], s_hi[kBurstScan], s_pam[kBurstScan];
    __shared__ unsigned char s_flags[kBurstScan];  // bit 0: has a previous field; bit 1: no interval
    const ldg_lines_args& a = P.a;
    const int f1 = a.first_field + a.count;
    if (threadIdx.x == 0) sm.seed = range_seed(P);  // the result of the field before the range
    int f = a.first_field;
    while (f < f1) {
        const int n = min(kBurstScan, f1 - f);
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            s_seed2[i] = B.seed2[f + i];
            s_lo[i] = B.lo[f + i];
            s_hi[i] = B.hi[f + i];
            s_pam[i] = a.phase_adjust[f + i];
            s_flags[i] = (unsigned char)((a.has_prev[f + i] ? 1 : 0) | (B.xonly[f + i] ? 2 : 0));
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            double prev = sm.seed;  // the result of field f - 1
            int g = 0;
            for (; g < n; ++g) {
                const double p = (s_flags[g] & 1) ? prev : 0.0;
                const bool same = __double_as_longlong(p) == __double_as_longlong(s_seed2[g]);
                const bool inside = !(s_flags[g] & 2) && p > s_lo[g] + kBurstMargin && p < s_hi[g] - kBurstMargin;
                if (!same && !inside) {
                    prev = p;  // field g's seed
                    break;
                }
                prev = s_pam[g];
            }
            sm.next = f + g;
            sm.seed = prev;
        }
        __syncthreads();
        const int g = sm.next;
        if (g < f + n) {
            BurstRec cur;
            cur.valid = 0;
            if (threadIdx.x < kBurstLines) cur = P.rec[(long long)g * kBurstLines + threadIdx.x];
            burst_field(cur, sm.seed, P.adjs + (long long)g * kBurstLines, P.field14 + g, false, sm);
            if (threadIdx.x == 0) {
                a.phase_adjust[g] = sm.pam;
                sm.seed = sm.pam;
            }
            f = g + 1;
        } else {
            f = g;
        }
        __syncthreads();
    }
}

// PAL 8-field sequence (determine_field_number, core.py:3128-3203), fields in
// order.  Sixteen lanes, one per zero-crossing slot, follow line 7 + 4j: its
// burst phase starts from the previous field's (0 when there is none, when
// that line had no result or when that field decided its ID before measuring
// phases), two passes of clb_findbursts' phase update, rising or not.  The
// field's ID comes from line 6's burst level against the field's median
// (present / absent / out of both ranges) and the majority of rising lines,
// or is the previous ID + 1 when that evidence is missing or split.  Bound: a
// field's chain of FP64 latencies, since the next field starts from its
// phases; the next field's inputs are loaded meanwhile and the slots' median
// is found by rank.  15 fields, one lane per line sorting its slots: 43 us; so
// 17 us (ncu).
constexpr int kSeqThreads = 4 * kZc;

__global__ void __launch_bounds__(kSeqThreads) pal_sequence_kernel(const __grid_constant__ LineParams P) {
    const ldg_lines_args& a = P.a;
    const int f0 = a.first_field, f1 = a.first_field + a.count;
    const int j = threadIdx.x / kZc, slot = threadIdx.x % kZc, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __shared__ int votes[2][2];  // [turn][warp]: lines | rising lines << 8
    int turn = 0;  // the other turn's barrier lies between a vote's reads and the next writes
    double seed;
    int prev_id;
    if (f0 > 0) {
        seed = a.phase_adjust[(long long)(f0 - 1) * 4 + j];
        prev_id = a.field_phase[f0 - 1];
    } else {
        seed = a.prev_pal_adjust_dev ? a.prev_pal_adjust_dev[j] : a.prev_pal_adjust[j];
        prev_id = a.prev_field_phase_dev ? *a.prev_field_phase_dev : a.prev_field_phase;
    }
    struct Inputs {
        double cyc, b6, bm;
        int count, rising, valid, has_prev, isfirst;
    };
    auto inputs = [&](int f) {
        const BurstRec& r = P.rec[(long long)f * kBurstLines + j];
        const double* lev = P.adjs + (long long)f * kBurstLines;
        return Inputs{r.cyc[slot], lev[0], lev[1], r.count, r.rising, r.valid, a.has_prev[f], a.isfirst[f]};
    };
    Inputs next{};
    if (f0 < f1) next = inputs(f0);
    for (int f = f0; f < f1; ++f) {
        const Inputs in = next;
        if (f + 1 < f1) next = inputs(f + 1);
        const bool has_prev = in.has_prev != 0;
        const int following = has_prev ? (prev_id + 1 == 9 ? 1 : prev_id + 1) : 1;
        int hasburst = -1;
        if (!isnan(in.b6)) {
            const double b = in.b6 / P.hz_ire;
            if (b >= in.bm * 0.8 && b <= in.bm * 1.2) hasburst = 1;
            else if (b < in.bm * 0.2) hasburst = 0;
        }
        double out = nan("");
        int id = following;
        if (hasburst >= 0) {  // the same for all threads
            const bool isf = in.isfirst != 0;
            const int m4 = isf ? (hasburst ? 3 : 1) : (hasburst ? 2 : 4);
            double pa = -((has_prev && !isnan(seed)) ? seed : 0.0);
            int rising_count = 0;
#pragma unroll
            for (int pass = 0; pass < 2; ++pass) {
                const double cyc = in.cyc + pa;
                const int rnd = (int)(cyc + .5);
                const double dev = (double)rnd - cyc;
                const unsigned odd = __ballot_sync(0xffffffffu, rnd % 2 != 0) >> (lane & kZc);
                // np.median of the line's 16 slots (mean of the two middle ones)
                int r = 0;
#pragma unroll
                for (int k = 0; k < kZc; ++k) {
                    const double o = __shfl_sync(0xffffffffu, dev, k, kZc);
                    r += pair_less(o, k, dev, slot);
                }
                const int group = lane & kZc;
                const unsigned m0 = (__ballot_sync(0xffffffffu, r == kZc / 2 - 1) >> group) & 0xffffu;
                const unsigned m1 = (__ballot_sync(0xffffffffu, r == kZc / 2) >> group) & 0xffffu;
                const double v0 = __shfl_sync(0xffffffffu, dev, (__ffs(m0) - 1) & (kZc - 1), kZc);
                const double v1 = __shfl_sync(0xffffffffu, dev, (__ffs(m1) - 1) & (kZc - 1), kZc);
                if (in.count) {
                    pa += (v0 + v1) / 2.0;
                    rising_count = __popc((unsigned)(in.rising ^ odd) & 0xffffu);
                }
            }
            const bool valid = in.valid != 0;
            const bool rising = (double)rising_count > ((double)in.count / 2);
            if (valid) out = -pa;
            const int lines = __popc(__ballot_sync(0xffffffffu, slot == 0 && valid));
            const int rlines = __popc(__ballot_sync(0xffffffffu, slot == 0 && valid && rising));
            turn ^= 1;
            if (lane == 0) votes[turn][warp] = lines | rlines << 8;
            __syncthreads();
            const int both = votes[turn][0] + votes[turn][1];
            const int count = both & 255, rcount = both >> 8;
            if (count != 0 && rcount * 2 != count) {
                bool firstfour = rcount * 2 > count;
                if (m4 == 2) firstfour = !firstfour;
                id = m4 + (firstfour ? 0 : 4);
            }
        }
        if (slot == 0) a.phase_adjust[(long long)f * 4 + j] = out;
        if (threadIdx.x == 0) a.field_phase[f] = id;
        seed = out;
        prev_id = id;
    }
}

// NTSC: refine_linelocs_burst's application, fix_badlines, subcarrier shift
__global__ void __launch_bounds__(512) burst_apply_kernel(const __grid_constant__ LineParams P, double shift) {
    const int f = P.a.first_field + blockIdx.x;
    const ldg_lines_args& a = P.a;
    const int nl = a.proclines;
    const int lc = a.linecount[f];
    __shared__ double ll2[kMaxL], adj_ll[kMaxL], out[kMaxL], adjs[kBurstLines];
    __shared__ unsigned char bad[kMaxL], has[kBurstLines];
    __shared__ double keys[512], mid[2];
    __shared__ int nadj, wsum[32];
    const int l = threadIdx.x;
    if (l == 0) nadj = 0;
    if (l < nl) {
        ll2[l] = P.ll2[(long long)f * kMaxL + l];
        bad[l] = a.linebad[(long long)f * kMaxL + l];
    }
    double an = nan("");
    if (l < kBurstLines) an = P.adjs[(long long)f * kBurstLines + l];
    __syncthreads();
    if (l >= 1 && l < kBurstLines && l < nl && isnan(an)) bad[l] = 1;
    __syncthreads();
    double adj = nan("");
    if (l < kBurstLines && l < nl) {
        has[l] = 0;
        if (!(isnan(ll2[l]) || bad[l]) && !isnan(an)) {
            const double lfreq = P.samplesperline * line_len(ll2, l, lc, P.linelen);
            adj = an * lfreq * (1 / P.fsc_mhz);
            has[l] = 1;
            atomicAdd(&nadj, 1);
        }
        adjs[l] = adj;
    }
    keys[l] = isnan(adj) ? INFINITY : adj;
    if (l < nl) adj_ll[l] = ll2[l];
    __syncthreads();
    const int cnt = nadj;  // the same for all threads
    if (cnt) {
        // the adjustments' median: every line counts those below and equal to its own
        if (l < kBurstLines && l < nl && has[l]) {
            const double mine = keys[l];
            int less = 0, same = 0;
#pragma unroll 4
            for (int k = 0; k < kBurstLines; ++k) {
                less += keys[k] < mine;
                same += keys[k] == mine;
            }
            const int r1 = cnt & 1 ? cnt / 2 : cnt / 2 - 1, r2 = cnt / 2;
            if (less <= r1 && r1 < less + same) mid[0] = mine;
            if (less <= r2 && r2 < less + same) mid[1] = mine;
        }
        __syncthreads();
        const double med = cnt & 1 ? mid[1] : (mid[0] + mid[1]) / 2.0;
        // a line without a valid adjustment takes the last valid one before it (the median before any)
        const bool valid = l < kBurstLines && l < nl && has[l] && adj - med >= -2 && adj - med <= 2;
        const int from = block_max_scan(valid ? l : -1, wsum);
        if (l < kBurstLines && l < nl) adj_ll[l] += from >= 0 ? adjs[from] : med;
    }
    if (l == 0) {
        const bool first = a.isfirst[f] != 0, f14 = cnt && P.field14[f] != 0;
        a.field_phase[f] = cnt ? (first ? (f14 ? 1 : 3) : (f14 ? 4 : 2)) : 1;
    }
    __syncthreads();
    // fix_badlines(linelocs3, linelocs2): deriv error, NaN from backup, interpolate (from line 1)
    deriv_error_block(adj_ll, bad, nl);
    if (l < nl && isnan(adj_ll[l])) adj_ll[l] = ll2[l];
    __syncthreads();
    fix_badlines_block(adj_ll, bad, out, nl, 1);
    if (l < nl) {
        a.linelocs[(long long)f * kMaxL + l] = out[l] - shift;
        a.linebad[(long long)f * kMaxL + l] = bad[l];
    }
}

size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

}  // namespace

extern "C" {

int64_t ldg_lines_scratch_bytes(int32_t nfields) {
    if (nfields < 0) return -1;
    return (int64_t)(align256((size_t)nfields * kBurstLines * sizeof(BurstRec)) +
                     align256((size_t)nfields * kMaxL * sizeof(double)) +
                     align256((size_t)nfields * kBurstLines * sizeof(double)) +
                     align256((size_t)nfields * sizeof(int)) + 5 * align256((size_t)nfields * sizeof(double)) +
                     align256((size_t)nfields * sizeof(int)));
}

}  // extern "C"

extern "C" int ldg_lines_refine(ldg_ctx* c, const ldg_lines_args* a) {
    if (!c || !a) return ldg::lines_fail(LDG_ERR_ARG, "ldg_lines_refine: NULL argument");
    if (a->nfields < 0 || a->proclines < 8 || a->proclines > kMaxL || (a->k.system != 0 && a->k.system != 1))
        return ldg::lines_fail(LDG_ERR_ARG, "ldg_lines_refine: bad size or system");
    if (a->nfields == 0) return LDG_OK;
    if (!a->d05 || !a->startloc || !a->wlen || !a->isfirst || !a->linecount || !a->has_prev || !a->linelocs1 ||
        !a->linebad1 || !a->linelocs || !a->linebad || !a->scratch ||
        !a->demod || !a->burst || !a->phase_adjust || !a->field_phase || (a->k.system == 1 && !a->pilot))
        return ldg::lines_fail(LDG_ERR_ARG, "ldg_lines_refine: NULL buffer");
    if (a->k.system == 0 && a->proclines < kBurstLines)
        return ldg::lines_fail(LDG_ERR_ARG, "ldg_lines_refine: NTSC needs proclines >= 266");
    if (a->k.system == 1 && a->proclines < kPilotLines)
        return ldg::lines_fail(LDG_ERR_ARG, "ldg_lines_refine: PAL needs proclines >= 323");
    if (a->first_field < 0 || a->first_field >= a->nfields || a->count < 0 ||
        a->first_field + a->count > a->nfields || a->stages < 0 || a->stages > 7)
        return ldg::lines_fail(LDG_ERR_ARG, "ldg_lines_refine: bad field range or stages");
    LineParams P;
    P.a = *a;
    if (P.a.count == 0) P.a.count = a->nfields - a->first_field;
    P.system = a->k.system;
    P.freq = a->k.freq;
    P.linelen = a->k.linelen;
    P.linefreq0 = a->k.linefreq0;
    P.samplesperline = a->k.samplesperline;
    P.half_sync = a->k.half_sync;
    P.lo_ok = a->k.lo_ok;
    P.hi_ok = a->k.hi_ok;
    P.hz_ire = a->k.hz_ire;
    P.fsc_mhz = a->k.fsc_mhz;
    P.pilot_mhz = a->k.pilot_mhz;
    char* s = static_cast<char*>(a->scratch);
    const size_t nf = (size_t)a->nfields;
    P.rec = reinterpret_cast<BurstRec*>(s);
    s += align256(nf * kBurstLines * sizeof(BurstRec));
    P.ll2 = reinterpret_cast<double*>(s);
    s += align256(nf * kMaxL * sizeof(double));
    P.adjs = reinterpret_cast<double*>(s);
    s += align256(nf * kBurstLines * sizeof(double));
    P.field14 = reinterpret_cast<int*>(s);
    s += align256(nf * sizeof(int));
    BurstSpec B;
    B.out1 = reinterpret_cast<double*>(s);
    s += align256(nf * sizeof(double));
    B.out2 = reinterpret_cast<double*>(s);
    s += align256(nf * sizeof(double));
    B.seed2 = reinterpret_cast<double*>(s);
    s += align256(nf * sizeof(double));
    B.lo = reinterpret_cast<double*>(s);
    s += align256(nf * sizeof(double));
    B.hi = reinterpret_cast<double*>(s);
    s += align256(nf * sizeof(double));
    B.xonly = reinterpret_cast<int*>(s);
    int prev = -1;
    cudaGetDevice(&prev);
    cudaSetDevice(ldg::ctx_device(c));
    cudaStream_t st = (cudaStream_t)a->stream;
    const int stages = a->stages ? a->stages : 7;
    if (stages & 1) {
        const unsigned per_field = (unsigned)((a->proclines + kRefineWarps - 1) / kRefineWarps);
        if (P.system == 1) {
            constexpr size_t bytes = (size_t)kLevelLines * kLevelWin * sizeof(float);
            static ldg::SmemAttr attr;
            if (attr.ensure(lines_pal_kernel, bytes) != cudaSuccess) {
                if (prev >= 0) cudaSetDevice(prev);
                return ldg::lines_fail(LDG_ERR_CUDA, std::string("ldg_lines_refine: ") +
                                                         cudaGetErrorString(cudaGetLastError()));
            }
        }
        for (int lo = 0; lo < P.a.count; lo += 65535) {  // grid.y limit
            LineParams Q = P;
            Q.a.first_field = P.a.first_field + lo;
            const unsigned nfl = (unsigned)(P.a.count - lo < 65535 ? P.a.count - lo : 65535);
            lines_hsync_kernel<<<dim3(per_field, nfl), 32 * kRefineWarps, 0, st>>>(Q);
            if (P.system == 0) lines_burst_kernel<<<dim3(per_field, nfl), 32 * kRefineWarps, 0, st>>>(Q);
        }
        if (P.system == 1)
            lines_pal_kernel<<<P.a.count, kPalThreads, (size_t)kLevelLines * kLevelWin * sizeof(float), st>>>(P);
    }
    if (P.system == 1 && (stages & 2)) pal_sequence_kernel<<<1, kSeqThreads, 0, st>>>(P);
    if (P.system == 0) {
        if (stages & 2) {
            for (int r = 1; r <= kBurstRounds; ++r)
                burst_round_kernel<<<P.a.count, kBurstThreads, 0, st>>>(P, r, B);
            burst_verify_kernel<<<1, kBurstThreads, 0, st>>>(P, B);
        }
        const double shift = (117.25 / 360) / P.fsc_mhz * P.freq;
        if (stages & 4) burst_apply_kernel<<<P.a.count, 512, 0, st>>>(P, shift);
    }
    cudaError_t e = cudaGetLastError();
    if (prev >= 0) cudaSetDevice(prev);
    if (e != cudaSuccess) return ldg::lines_fail(LDG_ERR_CUDA, std::string("ldg_lines_refine: ") + cudaGetErrorString(e));
    return LDG_OK;
}
