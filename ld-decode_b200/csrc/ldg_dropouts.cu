// Dropout detection of a batch of fields: Field.dropout_detect
// (lddecode/core.py:2962-2983), in four launches over all fields.
//
//  1. dropout_std_kernel   one CTA per 4096 samples: sum and squared
//     deviations of rfhpf (nb_std, core.py:2836) about the CTA's own mean,
//     FP64, merged by dropout_merge_kernel with the pairwise update of Chan,
//     Golub and LeVeque (the mean squared deviation numba forms in another
//     order; its error measured 7.6e-17, 1.1e-16 before); one more CTA per field
//     for the sync areas of every line l >= 1 (core.py:2867-2873): whole
//     lines for the vertical-sync lines,
//     otherwise the first hsync_len samples; Python slice bounds, then a
//     prefix maximum of the area ends so that "inside any area" is one
//     search.
//  2. dropout_mask_kernel  one CTA per 8192 samples: the error mask
//     (core.py:2837-2887) over the field's lines, one bit per sample.
//  3. dropout_place_kernel one CTA per field: the error samples merged into
//     spans (build_errlist, core.py:2889-2908) and the spans placed on TBC
//     lines (dropout_errlist_to_tbc, core.py:2910-2960), in the reference's
//     FP64 arithmetic (or integers that decide the same).
//
// Bound: HBM, 20 bytes per sample of the field's lines.  One CTA doing all of
// a field took 1.07 ms for one field and 1.36 ms for 60 (a span merge sample
// by sample on one thread, and 16 conversions to FP64 per clock and SM);
// the four kernels 58 us and 240 us (ncu; 68, 8, 128 and 36 us for 60 fields,
// the mask at 5.0 TB/s).  The whole call by the errors in one NTSC field: none
// 0.69 and 0.05 ms, 200 bursts of 100 samples 3.0 and 0.08, 1 % of the samples 2.8
// and 0.55, every 40th 6.7 and 2.6, every third 26.7 and 0.53.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <climits>

#include "ldg_attr.cuh"
#include "ldg_dropouts.cuh"

namespace ldg {

namespace {

constexpr int kStdThreads = 256, kStdPer = kDropStdTile / kStdThreads;
constexpr int kMaskThreads = 256, kMaskPer = kDropMaskTile / kMaskThreads;
constexpr int kPlaceThreads = 1024;
constexpr int kPlaceWords = 26112;  // mask words of a field held in shared memory, with its spans' starts (204 KB)
constexpr int kListWords = 2 * (2 * kPlaceThreads + 2);  // pairs: a word's fresh errors, at most two per thread, and an end

__device__ __forceinline__ long long py_index(long long x, long long n) {
    // a slice bound as Python normalises it
    if (x < 0) {
        x += n;
        return x < 0 ? 0 : x;
    }
    return x > n ? n : x;
}

__device__ __forceinline__ bool is_vsync_line(int l, int system, int isfirst) {
    // Field.get_vsync_lines (core.py:2814-2827)
    if (l >= 1 && l < (isfirst ? 10 : 9)) return true;
    return system == 1 && l >= (isfirst ? 311 : 310) && l < 318;
}

// Sum of v over the CTA, the same for every thread.
template <int Threads>
__device__ double block_sum(double v, double* red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    double r = 0;
    for (int w = 0; w < Threads / 32; ++w) r += red[w];
    __syncthreads();
    return r;
}

// The field's rfhpf standard deviation from its tiles' sums and squared
// deviations; one warp, the same result in every lane.
__device__ double merge_std(const double2* part, long long n) {
    const int lane = threadIdx.x & 31;
    const int tiles = (int)((n + kDropStdTile - 1) / kDropStdTile);
    double s = 0;
    for (int i = lane; i < tiles; i += 32) s += part[i].x;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    const double mean = s / (double)n;
    double m2 = 0;
    for (int i = lane; i < tiles; i += 32) {
        const double cnt = (double)min((long long)kDropStdTile, n - (long long)i * kDropStdTile);
        const double d = part[i].x / cnt - mean;
        m2 += fma(cnt * d, d, part[i].y);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m2 += __shfl_xor_sync(0xffffffffu, m2, o);
    return sqrt(m2 / (double)n);
}

// The largest float not above x (for x > limit with a float x).
__device__ __forceinline__ float float_down(double x) {
    const float f = (float)x;
    return (double)f > x ? nextafterf(f, -INFINITY) : f;
}

struct Emitter {
    int* out;
    int cap;
    int n;
    bool over;
    __device__ void put(int line, long long a, long long b) {
        if (n < cap) {
            out[3 * n] = line;
            out[3 * n + 1] = (int)a;
            out[3 * n + 2] = (int)b;
        } else {
            over = true;
        }
        ++n;
    }
};

// A span [c0, c1) that starts in line `line` (of line locations a, b at its ends)
// as TBC line ranges (core.py:2910-2960).
__device__ __forceinline__ void emit_span(Emitter& em, int line, int lineoffset, double a, double b, double c0, double c1,
                                          double outlinelen) {
    const double span = b - a;
    const long long start = (long long)(((c0 - a) / span) * outlinelen);
    const long long end = (long long)rint(((c1 - a) / span) * outlinelen);
    const int first = line + 1 - lineoffset;
    const long long ol = (long long)outlinelen;
    if (end > ol) {
        const long long k = end / ol;
        em.put(first - 1, start, ol);
        for (long long j = 0; j < k - 1; ++j) em.put((int)(first + j + 1) - 1, 0, ol);
        em.put((int)(first + k) - 1, 0, end % ol);
    } else {
        em.put(first - 1, start, end);
    }
}

// Exclusive scan of v over the CTA; *total its sum.
__device__ int block_scan(int v, int* wsum, int* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    if (lane == 31) wsum[warp] = inc;
    __syncthreads();
    int before = 0, all = 0;
    for (int w = 0; w < kPlaceThreads / 32; ++w) {
        const int q = wsum[w];
        before += w < warp ? q : 0;
        all += q;
    }
    __syncthreads();
    *total = all;
    return before + inc - v;
}

// ---- spans (build_errlist's merge)
//
// A span that starts with error sample c0 ends, after each error sample e that
// joins it, at c0 + min(1.7 (e - c0), cap); the next one joins if it lies up
// to 20 samples past that end, else it starts the next span.  So a span reaches
// c0 + cap + 20 at most, and short of that a sample with an error among the 20
// before it always joins: only the others, the fresh ones, are tested.

struct SpanRule {
    double cap;
    int reach;   // samples past c0 that a span can reach
    bool plain;  // ... for every c0, and the test below in integers
    int gap;     // no sample more than this past the last one joins

    __device__ explicit SpanRule(double c) : cap(c) {
        // c0 + cap + 20 is rounded twice, by 5e-7 at most (samples fit 31 bits)
        const double part = cap - floor(cap);
        plain = cap < 1e6 && (part == 0 || (part > 1e-6 && part < 1 - 1e-6));
        reach = plain ? (int)cap + 20 : 0;
        // up to 20 + min(0.7 d, cap - d) samples past a span of d samples: at most at d = cap / 1.7
        gap = (int)fmin(cap * (0.7 / 1.7) + 22.0, 1.0e9);
    }
    __device__ int last_reached(int c0) const {
        return plain && c0 < 0x7fffffff - reach ? c0 + reach : (int)fmin(floor(((double)c0 + cap) + 20.0), 2147483646.0);
    }
    // the end of a span of error samples c0 .. last
    __device__ double end(int c0, int last) const {
        double pad = (double)(last - c0) * 1.7;
        if (cap < pad) pad = cap;
        return (double)c0 + pad;
    }
    // does error sample e, the next after `last` and within the span's reach, join it?  (1.7 d is a whole
    // number, and then exact in FP64 too, or a tenth away from one)
    __device__ bool joins(int c0, int last, int e) const {
        return plain ? 10 * (e - c0 - 20) <= 17 * (last - c0) : (double)e <= end(c0, last) + 20.0;
    }
    // is error sample e, the next after `prev` (-1: none), the first of a segment?  Its spans do not
    // depend on what came before.  (Only a mask word's first error: a word then belongs to one segment.)
    __device__ bool heads(int e, int prev) const { return prev < 0 || (e - prev > gap && e >> 5 != prev >> 5); }
};

// The error samples of word m with none among the 20 before them; pm: the word before.
__device__ __forceinline__ unsigned fresh_errors(unsigned m, unsigned pm) {
    const unsigned long long both = (unsigned long long)m << 32 | pm;
    unsigned long long x = both << 1;
    x |= x << 1;
    x |= x << 2;
    x |= x << 4;
    x |= x << 8;
    x |= x << 4;
    return m & ~(unsigned)(x >> 32);
}

// The spans of the segment that starts with the first error of word w, in order:
// span(its first error sample, its last).  words[w], w < wend: the errors, fresh[w]
// the fresh ones.  A step for every word and every error tested; returns what is
// left of `steps`, less than 0 when they did not do.
template <class Span>
__device__ __forceinline__ int walk_segment(const SpanRule& rule, const unsigned* words, const unsigned* fresh, int w,
                                            int wend, int steps, Span&& span) {
    unsigned m = words[w];
    int c0 = 32 * w + __ffs(m) - 1, far = rule.last_reached(c0);
    unsigned todo = fresh[w] & (m - 1);  // (the first error is fresh)
    int last = c0;                       // the last error of the words before, then of this one
    for (;;) {
        const int base = 32 * w;
        // the word's errors past the reach, and its fresh ones, in order
        if (todo != 0 || far < base + 31) {
            for (;; --steps) {
                const unsigned over = far < base ? m : far - base < 31 ? m & (0xfffffffeu << (far - base)) : 0u;
                const unsigned any = over | todo;
                if (!any) break;
                const unsigned bit = any & (0u - any), low = m & (bit - 1u);
                todo &= ~bit;
                const int e = base + __ffs(any) - 1, prev = low ? base + 31 - __clz(low) : last;
                if (!(over & bit) && rule.joins(c0, prev, e)) continue;
                span(c0, prev);
                c0 = e;
                far = rule.last_reached(c0);
            }
        }
        last = base + 31 - __clz(m);
        // on to the next word with errors, if they still belong to the segment
        bool on = true;
        do {
            if (++w >= wend || 32 * w - last > rule.gap) {
                on = false;
                break;
            }
            m = words[w];
        } while (!m);
        if (--steps < 0) return steps;
        if (!on || rule.heads(32 * w + __ffs(m) - 1, last)) {
            span(c0, last);
            return steps;
        }
        todo = fresh[w];
    }
}

// The starts of the field's spans among its error words [w0, wend), to marks, by
// the CTA, a window of a word per thread at a time (plain rules only).  A fresh
// error f, the next after p, joins the span from c0 on if c0 <= T, by the rule
// p - (10 (f - p) - 200) / 7: the threads list the window's pairs (f, T), and one of
// them steps through the list: a comparison per fresh error, a search per span
// that ends at its reach.  marks holds the fresh errors before.
__device__ __forceinline__ void walk_windows(const SpanRule& rule, const unsigned* words, unsigned* marks, int w0, int wend,
                                             int2* list, int* wsum) {
    const int t = threadIdx.x;
    int c0 = INT_MAX, far = INT_MAX;  // (before any span)
    for (int wb = w0; wb < wend; wb += kPlaceThreads) {
        const int w = wb + t, wtop = min(wend, wb + kPlaceThreads), we = (int)min(32ll * wtop, 0x7fffffffll);
        const unsigned m = w < wend ? words[w] : 0u;
        if (!__syncthreads_or(m != 0)) continue;  // (its marks are 0)
        unsigned fresh = m ? marks[w] : 0u;
        int n;
        int at = block_scan(__popc(fresh), wsum, &n);
        if (t == 0) list[n] = make_int2(INT_MAX, 0);
        for (; fresh; fresh &= fresh - 1) {
            const int f = 32 * w + __ffs(fresh) - 1;
            const unsigned low = m & ((fresh & (0u - fresh)) - 1u);
            int p = -1;
            if (low) {
                p = 32 * w + 31 - __clz(low);
            } else {  // none within `gap`: a new segment
                for (int u = w - 1; u >= w0 && f - 32 * u <= rule.gap + 31; --u) {
                    const unsigned v = words[u];
                    if (v) {
                        p = 32 * u + 31 - __clz(v);
                        break;
                    }
                }
            }
            list[at++] = make_int2(f, p < 0 ? -1 : p - (10 * (f - p) - 194) / 7);
        }
        if (m) marks[w] = 0;
        __syncthreads();
        if (t == 0) {
            int2 r = list[0];
            for (int i = 0;;) {
                if (r.x <= far) {
                    if (r.x == INT_MAX) break;  // (only before any span)
                    const int2 next = list[++i];
                    const bool starts = c0 > r.y;
                    if (starts) {
                        c0 = r.x;
                        far = rule.last_reached(c0);
                        atomicOr(marks + (c0 >> 5), 1u << (c0 & 31));
                    }
                    r = next;
                } else {
                    // the first error past the reach: one of the next 20 samples, or a fresh one
                    int x = far + 1;
                    if (x >= we) break;
                    const unsigned after = (x >> 5) + 1 < wtop ? words[(x >> 5) + 1] : 0u;
                    const unsigned v = __funnelshift_r(words[x >> 5], after, x & 31) & 0xfffffu;
                    x = v ? x + __ffs(v) - 1 : r.x;
                    if (x >= we) break;
                    if (x == r.x) r = list[++i];
                    c0 = x;
                    far = rule.last_reached(c0);
                    atomicOr(marks + (c0 >> 5), 1u << (c0 & 31));
                }
            }
        }
        __syncthreads();
    }
}

constexpr int kHeld = 4;    // spans a thread keeps from counting its dropouts
constexpr int kSteps = 256;  // of a thread's walk before the field goes by windows

}  // namespace

__global__ void __launch_bounds__(kStdThreads, 5) dropout_std_kernel(const DropField* fields, const DropConsts k,
                                                                  const DropScratch sc) {
    __shared__ double red[kStdThreads / 32];
    const DropField f = fields[blockIdx.y];
    const long long n = f.len;
    const int t = threadIdx.x;
    if (blockIdx.x < gridDim.x - 1) {
        const long long i0 = (long long)blockIdx.x * kDropStdTile;
        if (i0 >= n) return;
        const int cnt = (int)min((long long)kDropStdTile, n - i0);
        float v[kStdPer];
#pragma unroll
        for (int j = 0; j < kStdPer; ++j) v[j] = t + j * kStdThreads < cnt ? __ldg(f.rfhpf + i0 + t + j * kStdThreads) : 0.0f;
        double s = 0;
#pragma unroll
        for (int j = 0; j < kStdPer; ++j) s += (double)v[j];
        s = block_sum<kStdThreads>(s, red);
        const double mean = s / (double)cnt;
        double m2 = 0;
#pragma unroll
        for (int j = 0; j < kStdPer; ++j) {
            const double d = t + j * kStdThreads < cnt ? (double)v[j] - mean : 0.0;
            m2 = fma(d, d, m2);
        }
        m2 = block_sum<kStdThreads>(m2, red);
        if (t == 0) sc.part[f.tile0 + blockIdx.x] = make_double2(s, m2);
        return;
    }
    // the sync areas
    __shared__ int rs[kMaxDropRegions], pm[2][kMaxDropRegions];
    __shared__ int s_bad;
    if (t == 0) s_bad = 0;
    __syncthreads();
    const int nreg = f.nlines - 1;
    for (int r = t; r < nreg; r += kStdThreads) {
        const int l = r + 1;
        const long long a = (long long)f.ll[l];
        long long b;
        if (is_vsync_line(l, k.system, f.isfirst)) {
            if (l + 1 >= f.nlines) {
                atomicOr(&s_bad, 2);
                b = a;
            } else {
                b = (long long)f.ll[l + 1];
            }
        } else {
            b = a + f.hsync_len;
        }
        rs[r] = (int)py_index(a, n);
        pm[0][r] = (int)py_index(b, n);
    }
    __syncthreads();
    int cur = 0;
    for (int o = 1; o < nreg; o <<= 1, cur ^= 1) {
        for (int r = t; r < nreg; r += kStdThreads)
            pm[cur ^ 1][r] = r >= o ? max(pm[cur][r], pm[cur][r - o]) : pm[cur][r];
        __syncthreads();
    }
    int2* area = sc.areas + (size_t)blockIdx.y * kMaxDropRegions;
    for (int r = t; r < nreg; r += kStdThreads) {
        if (r > 0 && rs[r] < rs[r - 1]) atomicOr(&s_bad, 1);
        area[r] = make_int2(rs[r], pm[cur][r]);
    }
    __syncthreads();
    if (t == 0) sc.bad[blockIdx.y] = s_bad;
}

// One warp per field.
__global__ void __launch_bounds__(128) dropout_merge_kernel(const DropField* fields, int nfields, const DropScratch sc,
                                                            double* rfstd_out) {
    const int f = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (f >= nfields) return;
    const double sd = merge_std(sc.part + fields[f].tile0, fields[f].len);
    if ((threadIdx.x & 31) == 0) {
        sc.rf_hi[f] = float_down(sd * 3.0);
        if (rfstd_out) rfstd_out[f] = sd;
    }
}

__device__ __forceinline__ void mask_range(const DropField& f, long long& lo, long long& hi) {
    lo = py_index((long long)f.ll[f.lineoffset + 1], f.len);
    hi = py_index((long long)f.ll[f.lineoffset + f.linecount + 1], f.len);
}

// Thread t takes samples t, t + 256, .. of the tile, so every load of a warp
// is one line and its 32 error flags one word; a sample's sync area is the
// walk from the sample 256 before.
__global__ void __launch_bounds__(kMaskThreads) dropout_mask_kernel(const DropField* fields, const DropConsts k,
                                                                    const DropScratch sc) {
    __shared__ int rs[kMaxDropRegions], pm[kMaxDropRegions];
    const DropField f = fields[blockIdx.y];
    long long lo, hi;
    mask_range(f, lo, hi);
    const long long i0 = (long long)blockIdx.x * kDropMaskTile;
    if (i0 + kDropMaskTile <= lo || i0 >= hi || sc.bad[blockIdx.y]) return;
    const int t = threadIdx.x, nreg = f.nlines - 1;
    const int2* area = sc.areas + (size_t)blockIdx.y * kMaxDropRegions;
    for (int r = t; r < nreg; r += kMaskThreads) {
        const int2 q = area[r];
        rs[r] = q.x;
        pm[r] = q.y;
    }
    __syncthreads();
    const float rf_hi = sc.rf_hi[blockIdx.y], fhalf = float_down(k.fhalf);
    // 32-bit offsets from the tile's first sample: [from, to) the ones in the field's lines
    const int from = (int)max(lo - i0, 0ll), to = (int)min(hi - i0, (long long)kDropMaskTile);
    const int base = (int)i0, rot = (int)min((long long)k.video_rot - i0, (long long)kDropMaskTile);
    const float* hp = f.rfhpf + i0 - k.video_rot;
    const float* raw = f.raw + i0;
    const float* dm = f.demod + i0;
    const float* d5 = f.d05 + i0;
    // last area starting at or before this thread's first sample
    int idx = -1;
    {
        const int i = base + t;
        int a = 0, b = nreg - 1;
        while (a <= b) {
            const int mid = (a + b) >> 1;
            if (rs[mid] <= i) {
                idx = mid;
                a = mid + 1;
            } else {
                b = mid - 1;
            }
        }
    }
    // the area's end and the next one's start, as offsets
    int end = idx >= 0 ? pm[idx] - base : INT_MIN;
    int next = idx + 1 < nreg ? rs[idx + 1] - base : INT_MAX;
    unsigned* words = sc.words + f.word0 + (i0 >> 5);
    constexpr int kBatch = 8;  // samples whose loads are in flight together
#pragma unroll 1
    for (int j0 = 0; j0 < kMaskPer; j0 += kBatch) {
        float h[kBatch], r[kBatch], d[kBatch], q[kBatch];
        const int o0 = t + j0 * kMaskThreads;
#pragma unroll
        for (int j = 0; j < kBatch; ++j) {
            const int o = o0 + j * kMaskThreads;
            const bool in = o >= from && o < to;
            h[j] = in && o >= rot ? __ldcs(hp + o) : 0.0f;
            r[j] = in ? __ldcs(raw + o) : 0.0f;
            d[j] = in ? __ldcs(dm + o) : 0.0f;
            q[j] = in ? __ldcs(d5 + o) : 0.0f;
        }
#pragma unroll
        for (int j = 0; j < kBatch; ++j) {
            const int o = o0 + j * kMaskThreads;
            while (o >= next) {
                ++idx;
                end = pm[idx] - base;
                next = idx + 1 < nreg ? rs[idx + 1] - base : INT_MAX;
            }
            const bool sync = o < end;
            bool e = o >= rot && (h[j] > rf_hi || h[j] < -rf_hi);
            e |= r[j] > fhalf;
            e |= (d[j] < (sync ? k.smin : k.vmin)) || (d[j] > k.vmax);
            e |= (q[j] < (sync ? k.smin05 : k.vmin05)) || (q[j] > k.vmax05);
            const unsigned m = __ballot_sync(0xffffffffu, e && o >= from && o < to);
            if ((t & 31) == 0) words[o >> 5] = m;
        }
    }
}

// Threads own consecutive words of the mask.  An error sample further from the
// one before it than any span lets one join starts a segment: the thread that
// owns it walks the segment's spans (past its words where it runs on), keeps
// them and counts their dropouts, which it writes after a scan (walking again
// when there are more than it keeps).  Noise (a carrier lost for lines on end) is
// one segment of thousands of spans; there the whole field is walked by windows,
// which mark the spans' starts for all threads to place, and so is a field whose
// line locations turn back, where a span's line hangs on the span before: one
// thread finds the lines and all place (one NTSC field, every 40th sample: 4.9 ms, 9.7 when
// that thread placed them too).  Bound: a thread's chain of instructions.
__global__ void __launch_bounds__(kPlaceThreads) dropout_place_kernel(const DropField* fields, const DropConsts k,
                                                                      const DropScratch sc, int* drops, int* counts) {
    extern __shared__ unsigned swords[];  // the list of walk_windows, 2 * place_words words
    int2* list = reinterpret_cast<int2*>(swords);
    __shared__ int wsum[32], wmax[32];
    __shared__ int s_down;
    __shared__ double ll[kMaxDropRegions + 1];  // the line locations (the placement searches them)
    const DropField f = fields[blockIdx.x];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    for (int l = t; l < f.nlines; l += kPlaceThreads) ll[l] = f.ll[l];
    const int bad = sc.bad[blockIdx.x];
    if (bad) {
        if (t == 0) {
            counts[2 * blockIdx.x] = (bad & 2) ? -3 : -2;
            counts[2 * blockIdx.x + 1] = 0;
        }
        return;
    }
    if (t == 0) s_down = 0;
    __syncthreads();
    long long lo, hi;
    mask_range(f, lo, hi);
    const double ll0 = ll[f.lineoffset];
    const int from = (int)min(max(lo, (long long)ceil(ll0)), hi);  // the errors before line `lineoffset` start no span
    // samples fit 31 bits, and words and bits are counted in int
    const int w0 = (int)(lo >> 5), nw = hi > lo ? (int)((hi + 31) >> 5) - w0 : 0, wend = w0 + nw;
    // the mask from `from` on and the spans' starts, in shared memory when they fit (a field of 0.83 M samples does)
    unsigned* const gwords = sc.words + f.word0;
    const bool held = nw <= sc.place_words;
    int n = 0;  // errors of the field
#pragma unroll 8
    for (int w = w0 + t; w < wend; w += kPlaceThreads) {
        unsigned m = gwords[w];
        n += __popc(m);
        if (w <= from >> 5) m = w < from >> 5 ? 0u : m & (0xffffffffu << (from & 31));
        if (held) swords[kListWords + w - w0] = m;
        else gwords[w] = m;
    }
    int nerr;
    block_scan(n, wsum, &nerr);
    if (t == 0) counts[2 * blockIdx.x + 1] = nerr > k.err_cap ? -1 : nerr;
    if (nerr > k.err_cap) {
        if (t == 0) counts[2 * blockIdx.x] = 0;
        return;
    }
    // are the line locations in order?
    for (int l = f.lineoffset + t; l < f.lineoffset + f.linecount; l += kPlaceThreads)
        if (!(ll[l] <= ll[l + 1])) s_down = 1;
    const int per = (nw + kPlaceThreads - 1) / kPlaceThreads;
    const int wa = w0 + min(nw, t * per), wb = w0 + min(nw, (t + 1) * per);
    const SpanRule rule(k.freq_mhz * 12.0);
    // a span as the placement gets it: 8 samples ahead and 4 behind, but the last one as it is
    auto start_of = [](int c0, bool is_last) { return (double)(is_last ? c0 : c0 - 8); };

    auto place_field = [&](const unsigned* words, unsigned* marks) {
        // the last error of the words before this thread's, and of the field
        int before = -1, top = -1;
        for (int w = wa; w < wb; ++w) {
            const unsigned m = words[w];
            if (m) before = 32 * w + 31 - __clz(m);
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, before, o);
            if (lane >= o) before = max(before, y);
        }
        if (lane == 31) wmax[warp] = before;
        before = __shfl_up_sync(0xffffffffu, before, 1);
        if (lane == 0) before = -1;
        for (int w = w0 + t; w < wend; w += kPlaceThreads) {
            const unsigned m = words[w];
            marks[w] = m ? fresh_errors(m, w > w0 ? words[w - 1] : 0u) : 0u;
        }
        __syncthreads();
        for (int w = 0; w < 32; ++w) {
            if (w < warp) before = max(before, wmax[w]);
            top = max(top, wmax[w]);
        }
        if (top < 0 || !((double)top > ll0)) {  // no error, or none past ll0 (the last one decides whether there are spans)
            if (t == 0) counts[2 * blockIdx.x] = 0;
            return;
        }
        Emitter em{drops + (size_t)blockIdx.x * k.out_cap * 3, k.out_cap, 0, false}, dry{nullptr, 0, 0, false};
        const int line0 = f.lineoffset, line1 = f.lineoffset + f.linecount;
        // the line of a span: the first one it starts in, -1 for none or a span that is skipped
        auto skipped = [&](double s0, bool is_last) { return s0 < ll0 && !is_last; };  // a later span exists
        auto line_of = [&](int c0, int end) {
            const bool is_last = end >= top;
            const double s0 = start_of(c0, is_last);
            if (skipped(s0, is_last)) return -1;
            int x = line0, y = line1;  // first line with s0 <= its end
            while (x < y) {
                const int mid = (x + y) >> 1;
                if (ll[mid + 1] >= s0) y = mid; else x = mid + 1;
            }
            return x < line1 && s0 >= ll[x] ? x : -1;
        };
        auto place_in = [&](Emitter& out, int c0, int end, int line) {
            if (line < 0) return;
            const bool is_last = end >= top;
            const double c1 = rule.end(c0, end);
            emit_span(out, line, line0, ll[line], ll[line + 1], start_of(c0, is_last), is_last ? c1 : c1 + 4.0,
                      (double)k.outlinelen);
        };
        auto place = [&](Emitter& out, int c0, int end) { place_in(out, c0, end, line_of(c0, end)); };
        // the spans of the segments that start in this thread's words, in order
        auto segments = [&](int steps, auto&& span) {
            int prev = before;
            for (int w = wa; w < wb && steps >= 0; ++w) {
                const unsigned m = words[w];
                if (!m) continue;
                if (rule.heads(32 * w + __ffs(m) - 1, prev)) steps = walk_segment(rule, words, marks, w, wend, steps, span);
                prev = 32 * w + 31 - __clz(m);
            }
            return steps;
        };
        int nspans = 0, held0[kHeld], held1[kHeld], total;
        const int left = s_down ? -1 : segments(rule.plain ? kSteps : INT_MAX, [&](int c0, int end) {
            if (nspans < kHeld) {
                held0[nspans] = c0;
                held1[nspans] = end;
            }
            ++nspans;
            place(dry, c0, end);
        });
        if (!__syncthreads_or(left < 0)) {
            em.n = block_scan(dry.n, wsum, &total);
            if (nspans <= kHeld) {
                for (int q = 0; q < nspans; ++q) place(em, held0[q], held1[q]);
            } else {
                segments(INT_MAX, [&](int c0, int end) { place(em, c0, end); });
            }
            if (t == 0) counts[2 * blockIdx.x] = total > k.out_cap ? -1 : total;
            return;
        }
        const bool marked = rule.plain;
        if (marked) walk_windows(rule, words, marks, w0, wend, list, wsum);
        // the spans that start in this thread's words (or in the segments that do), in order
        auto spans = [&](auto&& body) {
            if (!marked) {
                segments(INT_MAX, body);
                return;
            }
            for (int w = wa; w < wb; ++w) {
                for (unsigned m = marks[w]; m; m &= m - 1) {
                    // every error up to the next span's start, and short of the reach, is this one's
                    const int c0 = 32 * w + __ffs(m) - 1, far = rule.last_reached(c0);
                    unsigned above = m & (m - 1), from_c0 = 0u - (m & (0u - m));
                    int end = c0;
                    for (int u = w; u < wend && 32 * u <= far; from_c0 = 0xffffffffu, above = ++u < wend ? marks[u] : 0u) {
                        unsigned e = words[u] & from_c0;
                        if (above) e &= (above & (0u - above)) - 1u;
                        if (far - 32 * u < 31) e &= ~(0xfffffffeu << (far - 32 * u));
                        if (e) end = 32 * u + 31 - __clz(e);
                        if (above) break;
                    }
                    body(c0, end);
                }
            }
        };
        // a span per thread at a time; with line locations out of order a span's line depends on the one of
        // the span before, and one thread finds the lines
        nspans = 0;
        spans([&](int, int) { ++nspans; });
        const int base = block_scan(nspans, wsum, &total);
        int written = 0, line = line0;
        for (int batch = 0; batch < total; batch += kPlaceThreads) {
            if (base < batch + kPlaceThreads && base + nspans > batch) {
                int i = base - batch;
                spans([&](int c0, int end) {
                    if (i >= 0 && i < kPlaceThreads) list[i] = make_int2(c0, end);
                    ++i;
                });
            }
            __syncthreads();
            const int n = min(total - batch, kPlaceThreads);
            int* lines = reinterpret_cast<int*>(list + kPlaceThreads);
            if (s_down && t == 0) {
                for (int i = 0; i < n; ++i) {
                    const int2 q = list[i];
                    const bool is_last = q.y >= top;
                    const double s0 = start_of(q.x, is_last);
                    lines[i] = -1;
                    if (skipped(s0, is_last)) continue;
                    while (line < line1 && !(s0 >= ll[line] && s0 <= ll[line + 1])) ++line;
                    if (line < line1) lines[i] = line;
                }
            }
            if (s_down) __syncthreads();
            int c0 = 0, end = 0, at = -1;
            if (t < n) {
                c0 = list[t].x;
                end = list[t].y;
                at = s_down ? lines[t] : line_of(c0, end);
            }
            dry.n = 0;
            place_in(dry, c0, end, at);
            int made;
            em.n = written + block_scan(dry.n, wsum, &made);
            place_in(em, c0, end, at);
            written += made;
        }
        if (t == 0) counts[2 * blockIdx.x] = written > k.out_cap ? -1 : written;
    };
    // (each form's pointers into one address space)
    if (held) place_field(swords + kListWords - w0, swords + kListWords + sc.place_words - w0);
    else place_field(gwords, sc.starts + f.word0);
}

size_t dropout_scratch(DropField* fields, int nfields, char* base, DropScratch* sc) {
    const size_t nf = (size_t)nfields;
    size_t tiles = 0, words = 0;
    for (int i = 0; i < nfields; ++i) {
        fields[i].tile0 = (long long)tiles;
        fields[i].word0 = (long long)words;
        tiles += (size_t)((fields[i].len + kDropStdTile - 1) / kDropStdTile);
        // whole mask tiles (32 words beyond a field's last sample are not written)
        words += (size_t)((fields[i].len + kDropMaskTile - 1) / kDropMaskTile) * (kDropMaskTile / 32);
    }
    DropScratch q;
    char* p = base;
    auto take = [&](size_t bytes) {
        char* r = p;
        p += (bytes + 255) & ~(size_t)255;
        return r;
    };
    q.part = reinterpret_cast<double2*>(take(tiles * sizeof(double2)));
    q.areas = reinterpret_cast<int2*>(take(nf * kMaxDropRegions * sizeof(int2)));
    q.bad = reinterpret_cast<int*>(take(nf * sizeof(int)));
    q.rf_hi = reinterpret_cast<float*>(take(nf * sizeof(float)));
    q.words = reinterpret_cast<unsigned*>(take(words * sizeof(unsigned)));
    q.starts = reinterpret_cast<unsigned*>(take(words * sizeof(unsigned)));
    q.place_words = 0;
    if (sc) *sc = q;
    return (size_t)(p - base);
}

cudaError_t launch_dropouts(const DropField* fields, int nfields, long long max_len, const DropConsts& k,
                            DropScratch sc, int* drops, int* counts, double* rfstd, cudaStream_t stream) {
    if (nfields <= 0) return cudaSuccess;
    sc.place_words = (int)std::min((long long)kPlaceWords, max_len / 32 + 2);
    const unsigned std_tiles = (unsigned)((max_len + kDropStdTile - 1) / kDropStdTile);
    const unsigned mask_tiles = (unsigned)((max_len + kDropMaskTile - 1) / kDropMaskTile);
    for (int lo = 0; lo < nfields; lo += 65535) {  // grid.y limit
        const unsigned n = (unsigned)(nfields - lo < 65535 ? nfields - lo : 65535);
        DropScratch q = sc;
        q.areas += (size_t)lo * kMaxDropRegions;
        q.bad += lo;
        q.rf_hi += lo;
        dropout_std_kernel<<<dim3(std_tiles + 1, n), kStdThreads, 0, stream>>>(fields + lo, k, q);
        dropout_merge_kernel<<<(n + 3) / 4, 128, 0, stream>>>(fields + lo, (int)n, q, rfstd ? rfstd + lo : nullptr);
        dropout_mask_kernel<<<dim3(mask_tiles, n), kMaskThreads, 0, stream>>>(fields + lo, k, q);
    }
    // no more shared memory than the longest mask and the list need
    const size_t bytes = ((size_t)kListWords + 2 * sc.place_words) * sizeof(unsigned);
    static SmemAttr attr;
    const cudaError_t e = attr.ensure(dropout_place_kernel, bytes);
    if (e != cudaSuccess) return e;
    dropout_place_kernel<<<nfields, kPlaceThreads, bytes, stream>>>(fields, k, sc, drops, counts);
    return cudaGetLastError();
}

}  // namespace ldg
