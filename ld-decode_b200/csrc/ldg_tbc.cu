// Time-base correction: resample demodulated fields onto the 4fsc output
// grid (restates Field.computewow_scaled, lddecode/core.py:2591-2623,
// scale_field, lddecode/utils.py:127-183, and hz_to_output_array,
// lddecode/utils.py:1061-1075).
//
// Two kernels per batch of fields:
//   wow_levels_kernel  one CTA per field: the per-line-segment wow factors
//                      (slopes of the expected->actual line-location spline),
//                      their pixel-weighted median and 15*MAD outlier rule ->
//                      one level-adjust factor per segment.
//   spline_*           (quadratic / cubic wow interpolation only) the spline's
//                      pieces, the exact median and MAD of the per-pixel wow
//                      factors, and with level smoothing the IIR's state
//                      every 32 pixels.
//   tbc_gather_kernel  one thread per output pixels: FP64 spline coordinate,
//                      optional float32 rounding (the reference's own cast),
//                      16-tap windowed-sinc gather with linear interpolation
//                      between LUT phases, level adjust, uint16 conversion.
#include <algorithm>
#include <climits>

#include "ldg_tbc.cuh"

namespace ldg {

namespace {

constexpr int kWowThreads = 512;
constexpr int kMaxSeg = kWowThreads;  // segments (lines - 1) per field handled

__device__ __forceinline__ long long first_pixel_at(double xk, double outscale) {
    // smallest i >= 0 with i * outscale >= xk (same FP product as the gather)
    long long i = (long long)ceil(xk / outscale);
    if (i < 0) i = 0;
    while (i > 0 && __dmul_rn((double)(i - 1), outscale) >= xk) --i;  // one or two steps
    while (__dmul_rn((double)i, outscale) < xk) ++i;
    return i;
}

// Bitonic sort of (key, weight) pairs, ascending by key, n = kWowThreads.
__device__ void bitonic_sort(double* key, long long* wt) {
    const int t = threadIdx.x;
    for (int k = 2; k <= kWowThreads; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
            const int ixj = t ^ j;
            if (ixj > t) {
                const bool up = (t & k) == 0;
                const double a = key[t], b = key[ixj];
                if ((a > b) == up) {
                    key[t] = b;
                    key[ixj] = a;
                    const long long w = wt[t];
                    wt[t] = wt[ixj];
                    wt[ixj] = w;
                }
            }
            __syncthreads();
        }
    }
}

// Weighted median (numpy convention: mean of the two middle elements for an
// even count) of the sorted (key, wt) list, total count n.  Block-wide
// inclusive scan of the weights (warp shuffles + one shared pass).
__device__ double weighted_median(const double* key, const long long* wt, long long* csum,
                                  long long n) {
    __shared__ long long warp_tot[kWowThreads / 32];
    __shared__ double res[2];
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    long long x = wt[t];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const long long y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_tot[w] = x;
    __syncthreads();
    if (w == 0) {
        long long y = lane < kWowThreads / 32 ? warp_tot[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const long long z = __shfl_up_sync(0xffffffffu, y, o);
            if (lane >= o) y += z;
        }
        if (lane < kWowThreads / 32) warp_tot[lane] = y;
    }
    __syncthreads();
    const long long incl = x + (w ? warp_tot[w - 1] : 0);
    csum[t] = incl;
    const long long r1 = (n & 1) ? n / 2 : n / 2 - 1;
    const long long r2 = n / 2;
    const long long lo = incl - wt[t];
    if (wt[t] > 0) {
        if (r1 >= lo && r1 < incl) res[0] = key[t];
        if (r2 >= lo && r2 < incl) res[1] = key[t];
    }
    __syncthreads();
    const double r = (n & 1) ? res[1] : (res[0] + res[1]) / 2;
    __syncthreads();
    return r;
}

}  // namespace

__global__ void __launch_bounds__(kWowThreads) wow_levels_kernel(const TbcField* fields,
                                                                 double threshold_mult) {
    const TbcField& f = fields[blockIdx.x];
    if (f.spline_k >= 2) return;  // the spline kernels' field
    __shared__ double key[kWowThreads];
    __shared__ long long wt[kWowThreads];
    __shared__ long long csum[kWowThreads];
    __shared__ double slope_s[kMaxSeg];
    const int nseg = f.nlines - 1;
    const int t = threadIdx.x;
    if (nseg < 1 || nseg > kMaxSeg) {
        if (t == 0) f.status[0] = LDG_TBC_BAD_LINES;
        return;
    }
    const double inl = f.inlinelen;
    double slope = 0.0;
    long long cnt = 0;
    if (t < nseg) {
        const double y0 = f.linelocs[t], y1 = f.linelocs[t + 1];
        const double w = 1.0 / ((double)(t + 1) * inl - (double)t * inl);
        slope = __dadd_rn(__dmul_rn(y0, -w), __dmul_rn(y1, w));
        // pixels of the wow array [0, nwow) falling in this segment
        const long long lo = (t == 0) ? 0 : first_pixel_at((double)t * inl, f.outscale);
        const long long hi = (t == nseg - 1) ? f.nwow : first_pixel_at((double)(t + 1) * inl, f.outscale);
        const long long a = min(lo, f.nwow), b = min(hi, f.nwow);
        cnt = b > a ? b - a : 0;
        slope_s[t] = slope;
        f.seg_lo[t] = a;
    }
    key[t] = (t < nseg) ? slope : 1.0e300;
    wt[t] = cnt;
    __syncthreads();
    bitonic_sort(key, wt);
    const double med = weighted_median(key, wt, csum, f.nwow);
    // MAD over the same weighted set
    if (t < nseg) {
        key[t] = fabs(slope_s[t] - med);
        wt[t] = cnt;
    } else {
        key[t] = 1.0e300;
        wt[t] = 0;
    }
    __syncthreads();
    bitonic_sort(key, wt);
    const double mad = weighted_median(key, wt, csum, f.nwow);
    const double thr = mad > 0 ? threshold_mult * mad : 0.001;
    if (t < nseg) {
        const double s = slope_s[t];
        f.seg_level[t] = (fabs(s - med) > thr) ? med : s;
    }
    if (f.smooth_b > 0) {
        // level-adjust IIR (utils.py:141-149), y[0] = la[0], y[i] = a la[i] +
        // b y[i-1]: over segment j (constant level c_j) it is c_j + (y_before
        // - c_j) b^(i - lo_j + 1); the value entering each segment is carried
        // from segment to segment by one thread
        __syncthreads();
        if (t == 0) {
            double y = f.seg_level[0];
            for (int j = 0; j < nseg; ++j) {
                const double c = f.seg_level[j];
                f.seg_start[j] = y;
                const long long hi = (j + 1 < nseg) ? f.seg_lo[j + 1] : f.nwow;
                const long long len = hi - f.seg_lo[j];
                if (len > 0) y = c + (y - c) * pow(f.smooth_b, (double)len);
            }
        }
    }
}


// ---- quadratic / cubic wow interpolation (core.py:2602-2621) --------------
//
// The reference builds scipy's make_interp_spline through the points
// (i * inlinelen, linelocs[i]): k = 2 with scipy's default knots for even
// degree (the data points' midpoints, the first and last omitted), k = 3
// with natural end conditions (knots at the data points, s'' = 0 at both
// ends).  Here each spline is built directly as piecewise polynomials:
//   cubic      the classic second-derivative form, one tridiagonal system
//              for M_1 .. M_{n-2} (M_0 = M_{n-1} = 0);
//   quadratic  the derivative s' is piecewise linear and continuous over the
//              breakpoints x_0, (x_j + x_{j+1})/2 for j = 1 .. n-3, x_{n-1};
//              its values D_0 .. D_{n-2} at the breakpoints solve one
//              tridiagonal system whose row i states that the integral of s'
//              over [x_i, x_{i+1}] is y_{i+1} - y_i (the trapezoid rule is
//              exact for the linear pieces of s').
// Both systems are diagonally dominant and solved by the Thomas algorithm in
// FP64.  Outside the data range the first and last pieces extend, as scipy's
// BSpline extrapolates.

constexpr int kSplThreads = 1024;
constexpr int kSplMaxLines = 513;
constexpr int kHistBins = 2048;

// Coordinate and wow factor at x from a field's piece table pc (kSplStride
// doubles per piece: left edge, anchor, c0..c3; value c0 + c1 t + c2 t^2 +
// c3 t^3 at t = x - anchor).  The piece is guessed from x / inlinelen (shift
// 0: cubic pieces start at data points; 0.5: quadratic ones at midpoints)
// and fixed by exact comparisons with the left edges.  Every operation is
// an explicitly rounded intrinsic so that the statistics kernel and the
// gather get the same values.
__device__ __forceinline__ void spline_eval(const double* pc, int np, double x, double inv_inl, double shift,
                                            double& coord, double& wow) {
    int p = (int)floor(__dadd_rn(__dmul_rn(x, inv_inl), -shift));
    p = min(max(p, 0), np - 1);
    while (p > 0 && x < pc[p * kSplStride]) --p;
    while (p + 1 < np && x >= pc[(p + 1) * kSplStride]) ++p;
    const double* c = pc + p * kSplStride;
    const double t = __dadd_rn(x, -c[1]);
    coord = __fma_rn(t, __fma_rn(t, __fma_rn(t, c[5], c[4]), c[3]), c[2]);
    wow = __fma_rn(t, __fma_rn(t, __dmul_rn(3.0, c[5]), __dmul_rn(2.0, c[4])), c[3]);
}

// Order-preserving map of a double onto an unsigned 64-bit key.
__device__ __forceinline__ unsigned long long order_key(double v) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(v);
    return (u >> 63) ? ~u : (u | 0x8000000000000000ull);
}

__device__ __forceinline__ double key_value(unsigned long long k) {
    const unsigned long long u = (k >> 63) ? (k & 0x7fffffffffffffffull) : ~k;
    return __longlong_as_double((long long)u);
}

// The wow factors of pixels i0 .. i1-1 in order (one thread's chunk):
// body(i, wow).  The pixel position i * outscale comes from an exact double
// counter, the piece advances when the position passes the next piece's
// left edge (positions only grow), and the current piece's coefficients
// stay in registers -- the same position, piece and rounded operations as
// spline_eval, so the same wow factor as the gather's, at a fraction of the
// instructions of a search per pixel.
struct WowWalk {
    const double* pc;
    int np;
    double outscale, inv_inl, shift;
    template <class Body>
    __device__ __forceinline__ void operator()(long long i0, long long i1, Body body) const {
        if (i0 >= i1) return;
        double xi = (double)i0;
        double x = __dmul_rn(xi, outscale);
        int p = (int)floor(__dadd_rn(__dmul_rn(x, inv_inl), -shift));
        p = min(max(p, 0), np - 1);
        while (p > 0 && x < pc[p * kSplStride]) --p;
        while (p + 1 < np && x >= pc[(p + 1) * kSplStride]) ++p;
        double next, anc, c3, c4x2, c5x3;
        auto load = [&]() {
            const double* c = pc + p * kSplStride;
            next = p + 1 < np ? pc[(p + 1) * kSplStride] : INFINITY;
            anc = c[1];
            c3 = c[3];
            c4x2 = __dmul_rn(2.0, c[4]);
            c5x3 = __dmul_rn(3.0, c[5]);
        };
        load();
        for (long long i = i0; i < i1; ++i) {
            if (x >= next) {
                while (p + 1 < np && x >= pc[(p + 1) * kSplStride]) ++p;
                load();
            }
            const double t = __dadd_rn(x, -anc);
            body(i, __fma_rn(t, __fma_rn(t, c5x3, c4x2), c3));
            xi = __dadd_rn(xi, 1.0);
            x = __dmul_rn(xi, outscale);
        }
    }
};

constexpr int kCollect = kHistBins / 2;  // keys ranked in shared memory (the histogram's space)

struct SelectShared {
    unsigned warp_sum[32];
    unsigned long long prefix;  // key bits fixed so far
    long long krem;             // wanted rank among the keys that share them
    long long below;            // keys below that set
    unsigned eq;                // keys sharing the prefix (after the last pass: equal to the result)
    unsigned long long wmin[32];
    int ncoll, has_next;        // collected keys; the next key in rank order was among them
    long long cless;            // collected keys below the result
    unsigned long long next;    // that next key
};

// k-th smallest (0-based) of key(i), i in [0, n): most-significant-digit
// radix selection in up to six passes (digits of 11, 11, 11, 11, 11 and 9
// bits) over a shared histogram; the keys are recomputed on every pass.
// Once at most kCollect keys share the digits found so far, one more pass
// collects them into shared memory and the result is found among them by
// exact ranking (each thread counts the keys below and equal to its own),
// which also gives the next key in rank order when it is among them.  Each
// thread walks its own contiguous chunk of pixels and adds runs of equal
// digits at once; the 32 lanes of a warp look at pixels ~n/1024 apart,
// whose digits mostly differ where the runs are short.  On
// return sh.prefix is the key, sh.below the number of keys below it, sh.eq
// the number equal to it.
template <class Visit>
__device__ void radix_select(Visit visit, long long n, long long k, unsigned* hist, SelectShared& sh) {
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    if (t == 0) {
        sh.prefix = 0;
        sh.krem = k;
        sh.below = 0;
        sh.eq = 0;
        sh.has_next = 0;
    }
    unsigned long long mask = 0;
    const long long chunk = (n + kSplThreads - 1) / kSplThreads;
    const long long i0 = (long long)t * chunk, i1 = min(n, i0 + chunk);
    for (int pass = 0; pass < 6; ++pass) {
        const int shift = pass < 5 ? 53 - 11 * pass : 0;
        const unsigned dmask = pass < 5 ? 0x7ffu : 0x1ffu;
        for (int b = t; b < kHistBins; b += kSplThreads) hist[b] = 0;
        __syncthreads();
        const unsigned long long prefix = sh.prefix;
        // runs of one digit (the rule in the high passes, where a whole
        // chunk shares its sign and exponent) are counted in a register
        unsigned run_d = 0xffffffffu, run_n = 0;
        visit(i0, i1, [&](long long, unsigned long long kk) {
            if ((kk & mask) != prefix) return;
            const unsigned d = (unsigned)(kk >> shift) & dmask;
            if (d != run_d) {
                if (run_n) atomicAdd(&hist[run_d], run_n);
                run_d = d;
                run_n = 0;
            }
            ++run_n;
        });
        if (run_n) atomicAdd(&hist[run_d], run_n);
        __syncthreads();
        // the bin holding rank krem: block scan over bin pairs
        const unsigned h0 = hist[2 * t], h1 = hist[2 * t + 1];
        const unsigned s = h0 + h1;
        unsigned incl = s;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) sh.warp_sum[w] = incl;
        __syncthreads();
        if (w == 0) {
            unsigned y = sh.warp_sum[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned z = __shfl_up_sync(0xffffffffu, y, o);
                if (lane >= o) y += z;
            }
            sh.warp_sum[lane] = y;
        }
        __syncthreads();
        const long long excl = (long long)(incl - s) + (w ? (long long)sh.warp_sum[w - 1] : 0);
        const long long kr = sh.krem;
        __syncthreads();
        if (s > 0 && kr >= excl && kr < excl + s) {
            const bool first = kr < excl + h0;
            const long long bel = excl + (first ? 0 : h0);
            sh.prefix = prefix | ((unsigned long long)(2 * t + (first ? 0 : 1)) << shift);
            sh.krem = kr - bel;
            sh.below += bel;
            sh.eq = first ? h0 : h1;
        }
        mask |= (unsigned long long)dmask << shift;
        __syncthreads();
        if (pass < 5 && sh.eq <= (unsigned)kCollect) {  // uniform: a shared value after a barrier
            unsigned long long* coll = reinterpret_cast<unsigned long long*>(hist);
            const unsigned long long pre = sh.prefix;
            if (t == 0) sh.ncoll = 0;
            __syncthreads();
            visit(i0, i1, [&](long long, unsigned long long kk) {
                if ((kk & mask) == pre) {
                    const int pos = atomicAdd(&sh.ncoll, 1);
                    if (pos < kCollect) coll[pos] = kk;
                }
            });
            __syncthreads();
            const int nc = min(sh.ncoll, kCollect);
            const long long kr = sh.krem;
            __syncthreads();
            if (t < nc) {
                const unsigned long long mine = coll[t];
                int less = 0, same = 0;
                for (int q = 0; q < nc; ++q) {
                    const unsigned long long o = coll[q];
                    less += o < mine;
                    same += o == mine;
                }
                // threads holding equal keys store equal values
                if (less <= kr && kr < less + same) {
                    sh.prefix = mine;
                    sh.cless = less;
                    sh.eq = (unsigned)same;
                }
                if (kr + 1 < nc && less <= kr + 1 && kr + 1 < less + same) {
                    sh.next = mine;
                    sh.has_next = 1;
                }
            }
            __syncthreads();
            if (t == 0) sh.below += sh.cless;
            __syncthreads();
            return;
        }
    }
}

// Smallest key(i) above `above` (all ones when there is none).
template <class Visit>
__device__ unsigned long long min_key_above(Visit visit, long long n, unsigned long long above, SelectShared& sh) {
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    unsigned long long m = ~0ull;
    const long long chunk = (n + kSplThreads - 1) / kSplThreads;
    visit((long long)t * chunk, min(n, (long long)t * chunk + chunk), [&](long long, unsigned long long kk) {
        if (kk > above && kk < m) m = kk;
    });
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long y = __shfl_xor_sync(0xffffffffu, m, o);
        m = y < m ? y : m;
    }
    if (lane == 0) sh.wmin[w] = m;
    __syncthreads();
    m = sh.wmin[lane];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long y = __shfl_xor_sync(0xffffffffu, m, o);
        m = y < m ? y : m;
    }
    __syncthreads();
    return m;
}

// Of key(i), i in [0, n): the value of rank r1, or with `two` the mean of that
// and the next in order (numpy's median of the whole set when r1 is its
// middle rank).
template <class Visit>
__device__ double select_mean(Visit visit, long long n, long long r1, bool two, unsigned* hist, SelectShared& sh) {
    radix_select(visit, n, r1, hist, sh);
    const unsigned long long k1 = sh.prefix;
    const long long upto = sh.below + sh.eq;  // keys <= k1
    const bool has_next = sh.has_next != 0;
    const unsigned long long kn = sh.next;
    __syncthreads();
    const double v1 = key_value(k1);
    if (!two) return v1;
    const double v2 = has_next ? key_value(kn) : (upto >= r1 + 2 ? v1 : key_value(min_key_above(visit, n, k1, sh)));
    return __dadd_rn(v1, v2) / 2;
}

// The wow factors' median and MAD of a field, and with level smoothing the
// IIR's state every 32 pixels, in kernels of one CTA per field that decide
// and kernels of kSplSlices CTAs per field that walk its pixels:
//   spline_build    the pieces; a bracket for the median from kSplSamples
//                   pixels at even steps
//   spline_pass     counts the wow factors up to the bracket's low end, keeps
//                   those between its ends
//   spline_median   the median, exactly, from those (their number below tells
//                   which rank to take, or that it is an end); a bracket for the MAD
//   spline_pass     the same for |wow - median|
//   spline_mad      the MAD
//   spline_maps / spline_levels / spline_maps   (smoothing) the IIR over each
//                   chunk of pixels as a map, the maps' scan, the states
// A bracket's ranks lie kSplMargin samples either side of the median's: the
// factors are smooth along a line, so an evenly stepped sample misjudges a
// rank by about one sample per crossing and square root of the crossings, ~10
// of 4096.  Evenly spaced lines make most factors equal, and such a value is
// an end of its bracket: not kept, and where the median is an end the CTA counts
// the factors beyond it in one more walk (60 evenly spaced NTSC fields, cubic,
// smoothing: 660 us the whole call; 1204 by one CTA per field, 1320 with every
// such value kept until none fitted).  Where a bracket fails all the same (or
// keeps too many), the CTA selects from all pixels by radix passes.
// Bound: instruction issue of the walks (FP64 pipe next).  As one CTA per
// field walking all pixels up to ten times: 672 us for 60 NTSC fields (cubic,
// smoothing; as long for one); the eight launches together 250 us (ncu: build
// 67, passes 33 and 32, median 31, MAD 12, maps 44 and 26, levels 8; the build
// is one thread's chain of divisions and two rank selections).
constexpr int kSplSlices = 16;
constexpr int kSplPassThreads = 256;
constexpr int kSplMapThreads = 64;
constexpr int kSplSamples = 4096;
constexpr int kSplMargin = 48;
static_assert(sizeof(SplCtl) <= kSplCtlDoubles * sizeof(double), "the control block's place");

// Ranks of the median: r1, and r1 + 1 when the count is even.
__device__ __forceinline__ long long median_rank(long long n) { return (n & 1) ? n / 2 : n / 2 - 1; }

// The bracket [lo, hi] for the median of value(i), i in [0, L).
template <class Value>
__device__ void find_bracket(Value value, long long L, double* samp, unsigned* hist, SelectShared& sh, SplCtl* ctl) {
    const int t = threadIdx.x;
    double lo = -INFINITY, hi = INFINITY;
    if (L > kSplKeep) {
        for (int s = t; s < kSplSamples; s += kSplThreads)
            samp[s] = value((long long)(((double)s + 0.5) * ((double)L / kSplSamples)));
        __syncthreads();
        auto visit = [&](long long a0, long long a1, auto body) {
            for (long long i = a0; i < a1; ++i) body(i, order_key(samp[i]));
        };
        const double at = (double)median_rank(L) * ((double)kSplSamples / (double)L);
        const long long rl = (long long)at - kSplMargin, rh = (long long)at + 1 + kSplMargin;
        if (rl >= 0) {
            radix_select(visit, kSplSamples, rl, hist, sh);
            lo = key_value(sh.prefix);
            __syncthreads();
        }
        if (rh < kSplSamples) {
            radix_select(visit, kSplSamples, rh, hist, sh);
            hi = key_value(sh.prefix);
            __syncthreads();
        }
    }
    if (t == 0) {
        ctl->lo = lo;
        ctl->hi = hi;
        ctl->low = 0;
        ctl->kept = 0;
    }
}

// Of key(i), i in [0, n): how many lie below `lo`, and how many up to `hi`.
template <class Visit>
__device__ void count_keys(Visit visit, long long n, unsigned long long lo, unsigned long long hi, SelectShared& sh,
                           long long& below, long long& upto) {
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const long long chunk = (n + kSplThreads - 1) / kSplThreads;
    unsigned long long both = 0;  // counts in 32 bits each
    visit((long long)t * chunk, min(n, (long long)t * chunk + chunk), [&](long long, unsigned long long kk) {
        both += (unsigned long long)(kk <= hi) << 32 | (unsigned long long)(kk < lo);
    });
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) both += __shfl_xor_sync(0xffffffffu, both, o);
    if (lane == 0) sh.wmin[w] = both;
    __syncthreads();
    both = sh.wmin[lane];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) both += __shfl_xor_sync(0xffffffffu, both, o);
    __syncthreads();
    below = (long long)(both & 0xffffffffu);
    upto = (long long)(both >> 32);
}

// The median of all L values from what the pass counted and kept, all(i0, i1, body)
// visiting them in order: one that was kept, an end of the bracket (whose ranks
// one more walk tells), or (kept too many, or the median outside the bracket)
// selected from all.  `signs`: zeros of both signs occur, which a bracket's end
// does not tell apart.
template <class All>
__device__ double bracket_median(const TbcField& f, All all, long long L, bool signs, unsigned* hist, SelectShared& sh) {
    const SplCtl* ctl = spline_ctl(f);
    const bool two = !(L & 1);
    const long long r1 = median_rank(L), r2 = L / 2;
    const double lo = ctl->lo, hi = ctl->hi;
    const long long n1 = ctl->low, kept = ctl->kept, n2 = n1 + kept;  // ranks up to the low end, of what was kept
    bool usable = lo <= hi && kept <= kSplKeep && !(signs && (lo == 0 || hi == 0));
    __syncthreads();
    const bool in1 = r1 >= n1 && r1 < n2, in2 = r2 >= n1 && r2 < n2;
    if (usable && !(in1 && in2)) {
        long long below, upto;
        count_keys(all, L, order_key(lo), order_key(hi), sh, below, upto);
        usable = r1 >= below && r2 < upto;
    }
    if (!usable) return select_mean(all, L, r1, two, hist, sh);
    double v = 0.0;
    if (in1 || in2) {
        const double* k = spline_kept(f);
        v = select_mean(
            [&](long long a0, long long a1, auto body) {
                for (long long i = a0; i < a1; ++i) body(i, order_key(k[i]));
            },
            kept, (in1 ? r1 : r2) - n1, in1 && in2 && two, hist, sh);
        if (in1 && in2) return v;
    }
    const double v1 = in1 ? v : r1 < n1 ? lo : hi;
    const double v2 = in2 ? v : r2 < n1 ? lo : hi;
    return two ? __dadd_rn(v1, v2) / 2 : v1;
}

__device__ __forceinline__ WowWalk field_walk(const TbcField& f) {
    return WowWalk{f.spl, f.npieces, f.outscale, f.inv_inl, f.spline_k == 3 ? 0.0 : 0.5};
}

__device__ __forceinline__ double wow_at(const TbcField& f, long long i) {
    double c, w;
    spline_eval(f.spl, f.npieces, __dmul_rn((double)i, f.outscale), f.inv_inl, f.spline_k == 3 ? 0.0 : 0.5, c, w);
    return w;
}

// The tridiagonal system's rows in parallel, solved by thread 0 (Thomas), the
// pieces in parallel.
__global__ void __launch_bounds__(kSplThreads) spline_build_kernel(const TbcField* fields) {
    const TbcField& f = fields[blockIdx.x];
    if (f.spline_k < 2) return;
    __shared__ double mem[kSplSamples];  // the rows while solving, then the samples
    __shared__ unsigned long long hist_mem[kHistBins / 2];  // 8-byte aligned: also the collected keys
    __shared__ SelectShared sh;
    double* ra = mem;
    double* rb = ra + kSplMaxLines;
    double* rc = rb + kSplMaxLines;
    double* rd = rc + kSplMaxLines;
    double* cp = rd + kSplMaxLines;
    double* dp = cp + kSplMaxLines;
    static_assert(6 * kSplMaxLines <= kSplSamples, "the rows' place");
    const int t = threadIdx.x;
    const int n = f.nlines;
    const bool cubic = f.spline_k == 3;
    SplCtl* ctl = spline_ctl(f);
    if (n < 4 || n > kSplMaxLines) {
        if (t == 0) {
            f.status[0] = LDG_TBC_BAD_LINES;
            ctl->bad = 1;
        }
        return;
    }
    if (t == 0) ctl->bad = 0;
    const double inl = f.inlinelen;
    const double* y = f.linelocs;
    auto X = [&](int i) { return (double)i * inl; };
    // quadratic breakpoints
    auto BK = [&](int j) {
        return j == 0 ? X(0) : (j == n - 2 ? X(n - 1) : __dmul_rn(__dadd_rn(X(j), X(j + 1)), 0.5));
    };
    const int m = n - 2 + (cubic ? 0 : 1);  // unknowns
    for (int r = t; r < m; r += kSplThreads) {
        double a = 0, b = 0, c = 0, d = 0;
        if (cubic) {
            const int i = r + 1;
            const double h0 = X(i) - X(i - 1), h1 = X(i + 1) - X(i);
            a = h0;
            b = 2.0 * (h0 + h1);
            c = h1;
            d = 6.0 * ((y[i + 1] - y[i]) / h1 - (y[i] - y[i - 1]) / h0);
        } else {
            // integral of s' over [x_r, x_{r+1}], split at breakpoint r when it lies inside
            auto add = [&](double p, double q, int j, double& cj, double& cj1) {
                const double b0 = BK(j), wj = BK(j + 1) - b0;
                const double rp = (p - b0) / wj, rq = (q - b0) / wj;
                const double hw = (q - p) / 2;
                cj += hw * ((1.0 - rp) + (1.0 - rq));
                cj1 += hw * (rp + rq);
            };
            if (r == 0) {
                add(X(0), X(1), 0, b, c);
            } else if (r == n - 2) {
                add(X(n - 2), X(n - 1), n - 3, a, b);
            } else {
                add(X(r), BK(r), r - 1, a, b);
                add(BK(r), X(r + 1), r, b, c);
            }
            d = y[r + 1] - y[r];
        }
        ra[r] = a;
        rb[r] = b;
        rc[r] = c;
        rd[r] = d;
    }
    __syncthreads();
    if (t == 0) {
        double cq = rc[0] / rb[0], dq = rd[0] / rb[0];
        cp[0] = cq;
        dp[0] = dq;
        for (int r = 1; r < m; ++r) {
            const double a = ra[r];
            const double den = rb[r] - a * cq;
            cq = rc[r] / den;
            dq = (rd[r] - a * dq) / den;
            cp[r] = cq;
            dp[r] = dq;
        }
        for (int r = m - 2; r >= 0; --r) dp[r] = dp[r] - cp[r] * dp[r + 1];
    }
    __syncthreads();
    const int np = f.npieces;
    for (int p = t; p < np; p += kSplThreads) {
        double e[kSplStride];
        if (cubic) {
            auto M = [&](int i) { return (i == 0 || i == n - 1) ? 0.0 : dp[i - 1]; };
            const double h = X(p + 1) - X(p);
            const double m0 = M(p), m1 = M(p + 1);
            e[0] = X(p);
            e[1] = X(p);
            e[2] = y[p];
            e[3] = (y[p + 1] - y[p]) / h - h * (2.0 * m0 + m1) / 6.0;
            e[4] = m0 / 2.0;
            e[5] = (m1 - m0) / (6.0 * h);
        } else {
            const double left = BK(p), wp = BK(p + 1) - left;
            const int a = p == 0 ? 0 : (p == n - 3 ? n - 1 : p + 1);
            const double dd = dp[p + 1] - dp[p];
            e[0] = left;
            e[1] = X(a);
            e[2] = y[a];
            e[3] = dp[p] + dd * (X(a) - left) / wp;
            e[4] = dd / (2.0 * wp);
            e[5] = 0.0;
        }
#pragma unroll
        for (int q = 0; q < kSplStride; ++q) f.spl[p * kSplStride + q] = e[q];
    }
    __syncthreads();
    find_bracket([&](long long i) { return wow_at(f, i); }, f.nwow, mem, reinterpret_cast<unsigned*>(hist_mem), sh, ctl);
}

// One slice of a field's pixels against the bracket: how many lie up to its low
// end, and the values between its ends (in no order).
template <bool Mad>
__global__ void __launch_bounds__(kSplPassThreads) spline_pass_kernel(const TbcField* fields) {
    const TbcField& f = fields[blockIdx.y];
    if (f.spline_k < 2) return;
    SplCtl* ctl = spline_ctl(f);
    if (ctl->bad) return;
    constexpr int kHold = 2048;
    __shared__ double held[kHold];
    __shared__ int s_n, s_at;
    __shared__ volatile int s_full;  // more kept than the field's scratch holds: the bracket is of no use
    const int t = threadIdx.x;
    if (t == 0) s_n = s_full = 0;
    __syncthreads();
    const double lo = ctl->lo, hi = ctl->hi, med = Mad ? f.stat[0] : 0.0;
    double* kept = spline_kept(f);
    const long long L = f.nwow;
    const long long per = (L + kSplSlices * kSplPassThreads - 1) / (kSplSlices * kSplPassThreads);
    const long long i0 = ((long long)blockIdx.x * kSplPassThreads + t) * per, i1 = min(L, i0 + per);
    int low = 0;
    field_walk(f)(i0, i1, [&](long long, double w) {
        const double v = Mad ? fabs(__dadd_rn(w, -med)) : w;
        low += v <= lo;
        if (v > lo && v < hi) {
            const int at = atomicAdd(&s_n, 1);
            if (at < kHold) {
                held[at] = v;
            } else if (!s_full) {
                const int g = atomicAdd(&ctl->kept, 1);
                if (g < kSplKeep) kept[g] = v; else s_full = 1;
            }
        }
    });
#pragma unroll
    for (int o = 16; o; o >>= 1) low += __shfl_xor_sync(0xffffffffu, low, o);
    if ((t & 31) == 0 && low) atomicAdd(&ctl->low, low);
    __syncthreads();
    const int n = min(s_n, kHold);
    if (t == 0) s_at = n ? atomicAdd(&ctl->kept, n) : 0;
    __syncthreads();
    for (int i = t; i < n; i += kSplPassThreads)
        if (s_at + i < kSplKeep) kept[s_at + i] = held[i];
}

__global__ void __launch_bounds__(kSplThreads) spline_median_kernel(const TbcField* fields) {
    const TbcField& f = fields[blockIdx.x];
    if (f.spline_k < 2 || spline_ctl(f)->bad) return;
    __shared__ double samp[kSplSamples];
    __shared__ unsigned long long hist_mem[kHistBins / 2];
    __shared__ SelectShared sh;
    unsigned* hist = reinterpret_cast<unsigned*>(hist_mem);
    const WowWalk walk = field_walk(f);
    const double med = bracket_median(
        f,
        [&](long long a0, long long a1, auto body) {
            walk(a0, a1, [&](long long i, double w) { body(i, order_key(w)); });
        },
        f.nwow, true, hist, sh);
    if (threadIdx.x == 0) f.stat[0] = med;
    __syncthreads();
    find_bracket([&](long long i) { return fabs(__dadd_rn(wow_at(f, i), -med)); }, f.nwow, samp, hist, sh,
                 spline_ctl(f));
}

__global__ void __launch_bounds__(kSplThreads) spline_mad_kernel(const TbcField* fields, double threshold_mult) {
    const TbcField& f = fields[blockIdx.x];
    if (f.spline_k < 2 || spline_ctl(f)->bad) return;
    __shared__ unsigned long long hist_mem[kHistBins / 2];
    __shared__ SelectShared sh;
    const WowWalk walk = field_walk(f);
    const double med = f.stat[0];
    const double mad = bracket_median(
        f,
        [&](long long a0, long long a1, auto body) {
            walk(a0, a1, [&](long long i, double w) { body(i, order_key(fabs(__dadd_rn(w, -med)))); });
        },
        f.nwow, false, reinterpret_cast<unsigned*>(hist_mem), sh);
    if (threadIdx.x == 0) f.stat[1] = mad > 0 ? threshold_mult * mad : 0.001;
}

// Level-adjust IIR (utils.py:141-149), y[0] = la[0], y[i] = a la[i] + b y[i-1]:
// kSplChunks contiguous chunks of a field's pixels, one thread each.  The first
// launch finds each chunk's map y -> A y + B, spline_levels each chunk's y
// before its first pixel, the second the levels where the gather's warps begin.
// The chunks and the order of the scan decide the levels' last bits.
template <class Body>
__device__ __forceinline__ void walk_levels(const TbcField& f, int chunk, Body body) {
    const double med = f.stat[0], thr = f.stat[1];
    const long long C = (f.nwow + kSplChunks - 1) / kSplChunks;
    const long long i0 = chunk * C;
    field_walk(f)(i0, min(f.nwow, i0 + C), [&](long long i, double wv) {
        const double la = fabs(__dadd_rn(wv, -med)) > thr ? med : wv;
        body(i, __dmul_rn(f.smooth_a, la), la);
    });
}

template <bool Record>
__global__ void __launch_bounds__(kSplMapThreads) spline_maps_kernel(const TbcField* fields) {
    const TbcField& f = fields[blockIdx.y];
    if (f.spline_k < 2 || !(f.smooth_b > 0) || spline_ctl(f)->bad) return;
    const int chunk = blockIdx.x * kSplMapThreads + threadIdx.x;
    const double b = f.smooth_b;
    double* maps = spline_maps(f);
    if (!Record) {
        double B = 0.0;
        walk_levels(f, chunk, [&](long long i, double ala, double la) {
            B = i == 0 ? la : __dadd_rn(ala, __dmul_rn(b, B));
        });
        maps[chunk] = B;
    } else {
        // the level just before output pixel 32 m (wow index igbase + 32 m)
        const long long igbase = (long long)f.outwidth * (f.lineoffset + 1);
        const long long nyb = ((long long)f.linesout * f.outwidth + 31) / 32;
        const long long i0 = chunk * ((f.nwow + kSplChunks - 1) / kSplChunks);
        long long m = i0 + 1 - igbase <= 0 ? 0 : (i0 + 1 - igbase + 31) / 32;
        double y = maps[kSplChunks + chunk];
        walk_levels(f, chunk, [&](long long i, double ala, double la) {
            y = i == 0 ? la : __dadd_rn(ala, __dmul_rn(b, y));
            if (m < nyb && i + 1 == igbase + 32 * m) {
                f.ybefore[m] = y;
                ++m;
            }
        });
    }
}

__global__ void __launch_bounds__(kSplChunks) spline_levels_kernel(const TbcField* fields) {
    const TbcField& f = fields[blockIdx.x];
    if (f.spline_k < 2 || !(f.smooth_b > 0) || spline_ctl(f)->bad) return;
    __shared__ double wA[32], wB[32], wy[32];
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    double* maps = spline_maps(f);
    // the chunk's A: b times itself for each pixel, 0 when the first is among them
    const long long C = (f.nwow + kSplChunks - 1) / kSplChunks;
    const int pixels = (int)max(min(f.nwow - t * C, C), 0LL);
    double A = t == 0 && pixels ? 0.0 : 1.0, B = maps[t];
    for (int k = 0; k < pixels; ++k) A = __dmul_rn(f.smooth_b, A);
    // inclusive scan of the maps over the warp, then over the warps
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double Ap = __shfl_up_sync(0xffffffffu, A, o), Bp = __shfl_up_sync(0xffffffffu, B, o);
        if (lane >= o) {
            B = __fma_rn(A, Bp, B);
            A = __dmul_rn(A, Ap);
        }
    }
    if (lane == 31) {
        wA[w] = A;
        wB[w] = B;
    }
    __syncthreads();
    if (t == 0) {
        double yy = 0.0;
        for (int q = 0; q < 32; ++q) {
            wy[q] = yy;
            yy = __fma_rn(wA[q], yy, wB[q]);
        }
    }
    __syncthreads();
    const double Ae = __shfl_up_sync(0xffffffffu, A, 1), Be = __shfl_up_sync(0xffffffffu, B, 1);
    maps[kSplChunks + t] = lane == 0 ? wy[w] : __fma_rn(Ae, wy[w], Be);
}

constexpr int kGatherThreads = 128;  // 16 CTAs per SM (256 and 8: 1 % slower, 512 and 4: 4 %)

// What the gather reads of a field, in the launch's parameters: from the
// constant bank a warp gets a value without the load pipe, which bounds the
// kernel (read from the descriptors in memory they were some 20 of its ~145
// wavefronts per warp: 50 PAL fields 352 us, so 311 us, 60 NTSC ones 334 and
// 299 us; ncu).
struct GatherField {
    const float* buf;
    const double* linelocs;
    const double* seg_level;
    const double* seg_start;
    const long long* seg_lo;
    int* status;
    float* out_f32;
    uint16_t* out_u16;
    const double* spl;
    const double* stat;
    const double* ybefore;
    double inlinelen, outscale, inv_inl, u16_scale, u16_offset, smooth_a, smooth_b;
    long long buf_len, igbase, nout;
    int nseg, npieces, spline_k, coord_f32;
};

template <int N>
struct GatherBatch {
    GatherField f[N];
};
constexpr int kGatherBatch = 160;  // fields of a launch (29 KB of parameters of at most 32)
static_assert(sizeof(GatherBatch<kGatherBatch>) <= 32000, "kernel parameters");

// Input coordinate (FP64) of output pixel ig, optionally rounded to float32
// as the reference does; the spline segment j is also returned.  The
// segment is found from x * (1/inlinelen) and then fixed by exact
// comparisons with the integer knots; w = 1/(x1 - x0) = 1/inlinelen is
// precomputed with the same rounding.
__device__ __forceinline__ double pixel_coord(const GatherField& f, long long ig, int nseg, int& j) {
    const double inl = f.inlinelen;
    const double x = __dmul_rn((double)ig, f.outscale);
    j = (int)(x * f.inv_inl);
    j = min(max(j, 0), nseg - 1);
    if (j > 0 && (double)j * inl > x) --j;
    if (j < nseg - 1 && (double)(j + 1) * inl <= x) ++j;
    const double x0 = (double)j * inl, x1 = (double)(j + 1) * inl;
    const double y0 = __ldg(f.linelocs + j), y1 = __ldg(f.linelocs + j + 1);
    const double w = f.inv_inl;
    double c = __dadd_rn(__dmul_rn(y0, __dmul_rn(w, x1 - x)), __dmul_rn(y1, __dmul_rn(w, x - x0)));
    if (f.coord_f32) c = (double)__double2float_rn(c);
    return c;
}

// One warp per 32 consecutive output pixels of one field; blockIdx.y is the
// field.  Each lane computes its own pixel's FP64 coordinate; then groups of
// 8 lanes gather one pixel at a time (at step p group g takes pixel 4p + g,
// so a step's four pixels are adjacent): lane k of a group reads taps 2k, 2k+1
// of the input and one float4 of the interleaved LUT (the two taps of phase
// ps and their differences to phase ps + 1), so a pixel's 64-byte input
// span and its 128 bytes of LUT are each one contiguous access; the 8
// partial sums meet in a transposing reduction (lane k of group g ends with
// pixel 4k + g) and one shuffle takes each pixel's sum to its own lane.
// One lane's share of a pixel: taps in[0] and in[1], weights from the row
// (the interleaved float4 of w and the next-phase difference of the pixel's LUT
// phase) at fraction alpha; float32 products, FP64 sum.
__device__ __forceinline__ double two_taps(const float* in, const float4* row, float alpha) {
    const float4 q = __ldg(row);
    const float x0 = __ldg(in), x1 = __ldg(in + 1);
    const float w0 = fmaf(alpha, q.z, q.x), w1 = fmaf(alpha, q.w, q.y);
    return (double)(x0 * w0) + (double)(x1 * w1);
}

// Sum over a group's 8 lanes of their shares of the group's 8 pixels
// (share(p): this lane's share of pixel p), as a transposing reduction: at
// each level a lane keeps half of its pixels and adds the partner's shares
// of them, so lane k ends with the whole sum of pixel k.  The shares are
// formed in the order the reduction consumes them (pixels j and j + 4, for
// j = 0, 2, 1, 3), so at most two partial sums are live beside them.
template <class S>
__device__ __forceinline__ double group_sum(int k, S&& share) {
    const bool h4 = (k & 4) != 0, h2 = (k & 2) != 0, h1 = (k & 1) != 0;
    double b2[2];
#pragma unroll
    for (int jj = 0; jj < 2; ++jj) {
        double b4[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int j = jj + 2 * h;
            const double a = share(j), c = share(j + 4);
            b4[h] = (h4 ? c : a) + __shfl_xor_sync(0xffffffffu, h4 ? a : c, 4);
        }
        b2[jj] = (h2 ? b4[1] : b4[0]) + __shfl_xor_sync(0xffffffffu, h2 ? b4[0] : b4[1], 2);
    }
    return (h1 ? b2[1] : b2[0]) + __shfl_xor_sync(0xffffffffu, h1 ? b2[0] : b2[1], 1);
}

// The group sum with each pixel's first tap and phase in separate shuffles
// (phase -1: a pixel left at 0), for warps whose first taps do not fit
// 16-bit offsets.
__device__ __noinline__ double gather_unpacked(const float* buf, const float* lut, int sti, int psi, float alpha,
                                               int grp, int k) {
    return group_sum(k, [&](int p) {
        const int src = 4 * p + grp;
        const int pst = __shfl_sync(0xffffffffu, sti, src);
        const int pps = __shfl_sync(0xffffffffu, psi, src);
        const float pal = __shfl_sync(0xffffffffu, alpha, src);
        return pps >= 0 ? two_taps(buf + pst + 2 * k, reinterpret_cast<const float4*>(lut) + (size_t)pps * 8 + k, pal) : 0.0;
    });
}

template <int N>
__global__ void __launch_bounds__(kGatherThreads, 16) tbc_gather_kernel(const __grid_constant__ GatherBatch<N> batch,
                                                                    const float* lut) {
    const GatherField& f = batch.f[blockIdx.y];
    const long long nout = f.nout;
    const long long wbase = (long long)blockIdx.x * kGatherThreads + (threadIdx.x & ~31);
    if (wbase >= nout) return;  // whole warps leave together
    const int lane = threadIdx.x & 31, grp = lane >> 3, k = lane & 7;
    const long long i = wbase + lane;
    const int nseg = f.nseg;
    const long long igbase = f.igbase;
    int jj = 0;
    double cc, wv = 0.0;
    if (f.spline_k >= 2) {
        const double x = __dmul_rn((double)(igbase + (i < nout ? i : 0)), f.outscale);
        spline_eval(f.spl, f.npieces, x, f.inv_inl, f.spline_k == 2 ? 0.5 : 0.0, cc, wv);
        if (f.coord_f32) cc = (double)__double2float_rn(cc);
    } else {
        cc = pixel_coord(f, igbase + (i < nout ? i : 0), nseg, jj);
    }
    const long long ci = (long long)cc;
    const double ph = __dmul_rn(cc - (double)ci, 65536.0);
    const int ps = (int)ph;
    const float alpha = __double2float_rn(ph - (double)ps);
    const long long st = ci - 7;
    const bool ok = i < nout && st >= 0 && st + 16 <= f.buf_len && ps >= 0 && ps < 65536;
    if (i < nout && !ok && f.status) atomicOr(f.status, LDG_TBC_OUT_OF_RANGE);
    // first tap as a 32-bit offset (buf_len < 2^31); phase -1 marks a pixel left at 0
    const int sti = ok ? (int)st : 0;
    const int psi = ok ? ps : -1;
    // The 32 pixels' first taps lie within a few hundred samples of each
    // other: as offsets from the warp's lowest one they fit 16 bits, and each
    // pixel's offset, phase and fraction travel through shared memory in one
    // read (by shuffles, two per pixel: 312 against 298 us for 50 PAL fields;
    // they share the load pipe's writeback with the tap loads).  A pixel left
    // at 0 takes the lowest one's taps and is set to 0 after the sum (a test
    // at every pixel, and full addresses formed there: 298 against 260 us).
    const int low = __reduce_min_sync(0xffffffffu, ok ? sti : INT_MAX);
    const bool packed = __all_sync(0xffffffffu, !ok || sti - low <= 0xffff);
    double held = 0.0;  // after the group sum: the whole sum of pixel 4 k + grp
    if (low == INT_MAX) {
        // no pixel of the warp has its taps inside the buffer
    } else if (packed) {
        __shared__ uint2 s_px[kGatherThreads];
        uint2* px = s_px + (threadIdx.x & ~31);
        px[lane] = make_uint2(ok ? ((unsigned)(sti - low) << 16) | (unsigned)ps : 0u, __float_as_uint(alpha));
        __syncwarp();
        const float* in = f.buf + low + 2 * k;
        const float4* row = reinterpret_cast<const float4*>(lut) + k;
        const uint2* mine = px + grp;
        held = group_sum(k, [&](int p) {
            // the group's p-th pixel: at each step the four groups take four
            // adjacent pixels, whose 16-tap windows overlap (fewer cache lines
            // per tap load)
            const uint2 v = mine[4 * p];
            return two_taps(in + (v.x >> 16), row + (size_t)(v.x & 0xffffu) * 8, __uint_as_float(v.y));
        });
    } else {
        // first taps too far apart for 16-bit offsets (wild line locations): rare
        held = gather_unpacked(f.buf, lut, sti, psi, alpha, grp, k);
    }
    // pixel `lane` is at lane 8 (lane % 4) + lane / 4
    double mine = __shfl_sync(0xffffffffu, held, 8 * (lane & 3) + (lane >> 2));
    if (!ok) mine = 0.0;
    double level;
    if (f.spline_k >= 2) {
        const double med = f.stat[0];
        level = fabs(__dadd_rn(wv, -med)) > f.stat[1] ? med : wv;
        if (f.smooth_b > 0) {
            // the IIR over this warp's 32 pixels as a scan of affine maps,
            // started from the level just before the warp's first pixel
            double A = f.smooth_b, B = __dmul_rn(f.smooth_a, level);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const double Ap = __shfl_up_sync(0xffffffffu, A, o), Bp = __shfl_up_sync(0xffffffffu, B, o);
                if (lane >= o) {
                    B = __fma_rn(A, Bp, B);
                    A = __dmul_rn(A, Ap);
                }
            }
            level = __fma_rn(A, f.ybefore[wbase >> 5], B);
        }
    } else {
        level = 0.0;
    }
    if (i >= nout) return;
    if (f.spline_k < 2) {
        level = f.seg_level[jj];
        if (f.smooth_b > 0) {
            const long long ig = igbase + i;  // index into the wow array
            level = level + (f.seg_start[jj] - level) * pow(f.smooth_b, (double)(ig - f.seg_lo[jj] + 1));
        }
    }
    const float out = (float)(level * mine);
    if (f.out_f32) f.out_f32[i] = out;
    if (f.out_u16) {
        double v = (double)out * f.u16_scale + f.u16_offset + 0.5;
        v = fmin(fmax(v, 0.0), 65535.0);
        f.out_u16[i] = (uint16_t)(unsigned)v;
    }
}

template <int N>
static cudaError_t launch_gather(const TbcField* fields, int n, long long max_nout, const float* lut,
                                 cudaStream_t stream) {
    GatherBatch<N> batch;
    for (int i = 0; i < n; ++i) {
        const TbcField& f = fields[i];
        batch.f[i] = {f.buf, f.linelocs, f.seg_level, f.seg_start, f.seg_lo, f.status, f.out_f32, f.out_u16, f.spl, f.stat,
                      f.ybefore, f.inlinelen, f.outscale, f.inv_inl, f.u16_scale, f.u16_offset, f.smooth_a, f.smooth_b,
                      f.buf_len, (long long)f.outwidth * (f.lineoffset + 1), (long long)f.linesout * f.outwidth,
                      f.nlines - 1, f.npieces, f.spline_k, f.coord_f32};
    }
    const unsigned gx = (unsigned)((max_nout + kGatherThreads - 1) / kGatherThreads);
    tbc_gather_kernel<N><<<dim3(gx, (unsigned)n), kGatherThreads, 0, stream>>>(batch, lut);
    return cudaGetLastError();
}

cudaError_t launch_tbc(const TbcField* dfields, const TbcField* hfields, int nfields, long long max_nout,
                       const float* lut, double threshold_mult, bool any_spline, bool any_smooth, cudaStream_t stream) {
    if (nfields <= 0) return cudaSuccess;
    wow_levels_kernel<<<nfields, kWowThreads, 0, stream>>>(dfields, threshold_mult);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    if (any_spline) {
        spline_build_kernel<<<nfields, kSplThreads, 0, stream>>>(dfields);
        for (int pass = 0; pass < 2; ++pass) {
            for (int off = 0; off < nfields; off += 65535) {  // grid.y limit
                const unsigned n = (unsigned)(nfields - off < 65535 ? nfields - off : 65535);
                if (pass) spline_pass_kernel<true><<<dim3(kSplSlices, n), kSplPassThreads, 0, stream>>>(dfields + off);
                else spline_pass_kernel<false><<<dim3(kSplSlices, n), kSplPassThreads, 0, stream>>>(dfields + off);
            }
            if (pass) spline_mad_kernel<<<nfields, kSplThreads, 0, stream>>>(dfields, threshold_mult);
            else spline_median_kernel<<<nfields, kSplThreads, 0, stream>>>(dfields);
        }
        if (any_smooth) {
            for (int off = 0; off < nfields; off += 65535) {
                const unsigned n = (unsigned)(nfields - off < 65535 ? nfields - off : 65535);
                spline_maps_kernel<false><<<dim3(kSplChunks / kSplMapThreads, n), kSplMapThreads, 0, stream>>>(dfields + off);
            }
            spline_levels_kernel<<<nfields, kSplChunks, 0, stream>>>(dfields);
            for (int off = 0; off < nfields; off += 65535) {
                const unsigned n = (unsigned)(nfields - off < 65535 ? nfields - off : 65535);
                spline_maps_kernel<true><<<dim3(kSplChunks / kSplMapThreads, n), kSplMapThreads, 0, stream>>>(dfields + off);
            }
        }
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    for (int off = 0; off < nfields && e == cudaSuccess; off += kGatherBatch) {
        const int n = nfields - off < kGatherBatch ? nfields - off : kGatherBatch;
        // no more parameters than the batch needs
        e = n <= 4 ? launch_gather<4>(hfields + off, n, max_nout, lut, stream)
                   : n <= 32 ? launch_gather<32>(hfields + off, n, max_nout, lut, stream)
                             : launch_gather<kGatherBatch>(hfields + off, n, max_nout, lut, stream);
    }
    return e;
}

// RF TBC (Field.rf_tbc, lddecode/core.py:2724-2752): each output line l is
// the cubic scaler (utils.py:37-70) over the raw input between linelocs[l]
// and linelocs[l + 1], both moved back by the video delay, rounded half to
// even and stored as int16.  The arithmetic is the reference's FP64
// expression term by term with every product and sum rounded on its own
// (no fused multiply-adds), so the output is bit-identical.  One CTA per
// (line, field).
//
// Bound: the FP64 pipe (about one warp instruction per clock and SM;
// conversions between integers and FP64 half that).  The polynomial's
// coefficients are sums of 16-bit samples, exact in integers, and numbers
// cross between int and double by an addition to 2^52 (and 2^51 or 2^31),
// whose low word then is the integer: 17 FP64 operations per sample instead of
// 21 and 8 conversions.  Five samples per thread are in flight, and one CTA
// takes up to four lines.  50 PAL fields (40 M samples), B200 (ncu): 128 us
// before, 88 us so.
constexpr int kRfThreads = 256, kRfPer = 5, kRfMaxLines = 4;
constexpr double kIntMagic = 6755399441055744.0;  // 2^52 + 2^51

__device__ __forceinline__ double int_to_double(int k) {  // exact, |k| < 2^31
    return __dsub_rn(__hiloint2double(0x43300000, k ^ (int)0x80000000), 4503601774854144.0);  // 2^52 + 2^31
}

// One output line: begin and scale of its input, the samples' output.
struct RfLine {
    double begin, sf;
    int16_t* out;
    int inside;  // every tap of the line lies inside the read
};

__global__ void __launch_bounds__(kRfThreads) rf_tbc_kernel(const RfTbcField* fields, int lines_per_cta) {
    __shared__ RfLine s_line[kRfMaxLines];
    const RfTbcField& f = fields[blockIdx.y];
    const int line0 = blockIdx.x * lines_per_cta;
    const int nlines = min(lines_per_cta, f.nout - line0);
    if (nlines <= 0) return;
    const int n = f.linelen;
    const int16_t* in = f.in;
    const double limit = (double)(f.len - 2);
    // one thread per line: what the whole line shares
    if (threadIdx.x < nlines) {
        const int line = line0 + threadIdx.x, l = f.startline + line;
        RfLine q;
        q.begin = __dsub_rn(f.ll[l], f.delay);
        const double end = __dsub_rn(f.ll[l + 1], f.delay);
        q.sf = __ddiv_rn(__dsub_rn(end, q.begin), (double)n);
        q.out = f.out + (long long)line * n;
        // taps int(coord) - 1 .. int(coord) + 2 inside the read: 1 <= coord < len - 2.
        // The rounded coordinate never turns back along a line, so its ends tell for all of it
        const double last = __dadd_rn(__dmul_rn((double)(n - 1), q.sf), q.begin);
        q.inside = f.len < (1ll << 31) && q.begin >= 1.0 && q.begin < limit && last >= 1.0 && last < limit;
        s_line[threadIdx.x] = q;
    }
    __syncthreads();
    for (int k = 0; k < nlines; ++k) {
        const double begin = s_line[k].begin, sf = s_line[k].sf;
        int16_t* out = s_line[k].out;
        if (s_line[k].inside) {
            double xi = (double)threadIdx.x;
            for (int i0 = threadIdx.x; i0 < n; i0 += kRfPer * kRfThreads) {
                // kRfPer samples at a time, their loads in flight together
                double x[kRfPer];
                int p0[kRfPer], p1[kRfPer], p2[kRfPer], p3[kRfPer];
#pragma unroll
                for (int j = 0; j < kRfPer; ++j) {
                    // past the line's end: its last sample again
                    const double xj = i0 + j * kRfThreads < n ? xi : (double)(n - 1);
                    const double coord = __dadd_rn(__dmul_rn(xj, sf), begin);
                    // floor: the sum with 2^52 rounded down
                    const double fl = __dadd_rd(coord, 4503599627370496.0);
                    const int16_t* q = in + (__double2loint(fl) - 1);
                    p0[j] = __ldg(q);
                    p1[j] = __ldg(q + 1);
                    p2[j] = __ldg(q + 2);
                    p3[j] = __ldg(q + 3);
                    x[j] = __dsub_rn(coord, __dsub_rn(fl, 4503599627370496.0));
                    xi = __dadd_rn(xi, (double)kRfThreads);
                }
#pragma unroll
                for (int j = 0; j < kRfPer; ++j) {
                    // p1 + 0.5 x (p2 - p0 + x (2 p0 - 5 p1 + 4 p2 - p3 + x (3 (p1 - p2) + p3 - p0)))
                    const double c = int_to_double(3 * (p1[j] - p2[j]) + p3[j] - p0[j]);
                    const double b =
                        __dadd_rn(int_to_double(2 * p0[j] - 5 * p1[j] + 4 * p2[j] - p3[j]), __dmul_rn(x[j], c));
                    const double a = __dadd_rn(int_to_double(p2[j] - p0[j]), __dmul_rn(x[j], b));
                    // half of x a is exact, so this rounds as (0.5 x) a and then p1 + that do
                    const double v = __fma_rn(0.5, __dmul_rn(x[j], a), int_to_double(p1[j]));
                    if (i0 + j * kRfThreads < n)
                        out[i0 + j * kRfThreads] = (int16_t)__double2loint(__dadd_rn(v, kIntMagic));  // half to even
                }
            }
            continue;
        }
        for (int i = threadIdx.x; i < n; i += kRfThreads) {
            const double coord = __dadd_rn(__dmul_rn((double)i, sf), begin);
            if (!(coord >= 1.0 && coord < limit)) {
                atomicOr(f.status, LDG_TBC_OUT_OF_RANGE);
                out[i] = 0;
                continue;
            }
            const long long ic = (long long)coord;
            const int16_t* q = in + (ic - 1);
            const double p0 = q[0], p1 = q[1], p2 = q[2], p3 = q[3];
            const double x = __dsub_rn(coord, (double)ic);
            const double c = __dsub_rn(__dadd_rn(__dmul_rn(3.0, __dsub_rn(p1, p2)), p3), p0);
            const double b = __dadd_rn(
                __dsub_rn(__dadd_rn(__dsub_rn(__dmul_rn(2.0, p0), __dmul_rn(5.0, p1)), __dmul_rn(4.0, p2)), p3),
                __dmul_rn(x, c));
            const double a = __dadd_rn(__dsub_rn(p2, p0), __dmul_rn(x, b));
            const double v = __dadd_rn(p1, __dmul_rn(__dmul_rn(0.5, x), a));
            out[i] = (int16_t)(int)rint(v);
        }
    }
}

cudaError_t launch_rf_tbc(const RfTbcField* dfields, int nfields, int max_lines, cudaStream_t stream) {
    if (nfields <= 0 || max_lines <= 0) return cudaSuccess;
    // several lines per CTA once there are CTAs enough for every SM: what a line
    // shares (its descriptor, its locations, a division) is a chain of latencies
    const int per = std::min(kRfMaxLines, (int)std::max(1ll, (long long)max_lines * nfields / (148 * 8)));
    const unsigned gx = (unsigned)((max_lines + per - 1) / per);
    for (int off = 0; off < nfields; off += 65535) {
        const int n = nfields - off < 65535 ? nfields - off : 65535;
        rf_tbc_kernel<<<dim3(gx, (unsigned)n), kRfThreads, 0, stream>>>(dfields + off, per);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace ldg
