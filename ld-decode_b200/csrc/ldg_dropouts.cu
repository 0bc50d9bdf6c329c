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
//     FP64 arithmetic.
//
// Bound: HBM, 20 bytes per sample of the field's lines.  One CTA doing all of
// a field took 1.07 ms for one field and 1.36 ms for 60 (a span merge sample
// by sample on one thread, and 16 conversions to FP64 per clock and SM);
// the four kernels 58 us and 240 us (ncu; 68, 8, 128 and 36 us for 60 fields,
// the mask at 5.0 TB/s).
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
constexpr int kPlaceWords = 48 * 1024;  // mask words of a field held in shared memory (192 KB)

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

// Spans to TBC lines (core.py:2910-2960), fed one span at a time in order.
struct LinePlacer {
    const double* ll;
    int line, end_line, lineoffset;
    double outlinelen;
    double ll0;
    bool placing;          // past the reference's initial skip of spans before line `lineoffset`
    bool have_pending;
    double p0, p1;
    Emitter* em;

    __device__ void place(double c0, double c1) {
        while (line < end_line) {
            const double a = ll[line], b = ll[line + 1];
            if (c0 >= a && c0 <= b) {
                const double span = b - a;
                const long long start = (long long)(((c0 - a) / span) * outlinelen);
                const long long end = (long long)rint(((c1 - a) / span) * outlinelen);
                const int first = line + 1 - lineoffset;
                const long long ol = (long long)outlinelen;
                if (end > ol) {
                    const long long k = end / ol;
                    em->put(first - 1, start, ol);
                    for (long long j = 0; j < k - 1; ++j) em->put((int)(first + j + 1) - 1, 0, ol);
                    em->put((int)(first + k) - 1, 0, end % ol);
                } else {
                    em->put(first - 1, start, end);
                }
                return;
            }
            ++line;
        }
    }
    __device__ void feed(double s0, double s1) {
        if (!placing) {
            if (!have_pending) {
                p0 = s0;
                p1 = s1;
                have_pending = true;
                return;
            }
            if (p0 < ll0) {  // a later span exists: the reference pops on
                p0 = s0;
                p1 = s1;
                return;
            }
            placing = true;
            place(p0, p1);
        }
        place(s0, s1);
    }
    __device__ void finish() {
        if (!placing && have_pending) {
            placing = true;
            place(p0, p1);
        }
    }
};

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

// The error samples of a field as bits, those before `end` (samples fit 31 bits).
struct ErrorBits {
    const unsigned* words;
    int end;
    // the first error sample at or after i, `end` when there is none before `limit`
    __device__ int next(int i, int limit) const {
        limit = min(limit, end);
        while (i < limit) {
            const unsigned m = words[i >> 5] >> (i & 31);
            if (m) {
                i += __ffs(m) - 1;
                return i < limit ? i : end;
            }
            i = (i | 31) + 1;
        }
        return end;
    }
    // the last sample of the run of error samples that i is in
    __device__ int run_end(int i) const {
        for (;;) {
            const unsigned m = ~(words[i >> 5] >> (i & 31));  // zeros shifted in count as no error
            const int k = m ? __ffs(m) - 1 : 32;
            i += k;
            if ((i & 31) != 0 || i >= end || !(words[i >> 5] & 1u)) return min(i, end) - 1;
        }
    }
};

// build_errlist's merge from error sample `e` on, which starts a span.  Within
// a run of errors every sample extends the span until the span's cap (12 us,
// and 20 samples) is behind it, so a run takes one step per cap.  Stops at the
// first error more than `gap` samples after the last (no span reaches
// that far: it starts a new one whatever came before) and returns the last
// error sample before it; span(c0, c1, last) gets each span, `last` for the
// one that ends with the field's last error sample, `top`.
template <class Span>
__device__ int merge_segment(const ErrorBits& bits, int e, int gap, double cap, int top, Span&& span) {
    int c0 = e, b;
    double c1 = (double)e;
    for (;;) {
        b = bits.run_end(e);
        while (e <= b) {
            if (e > c0 && (double)e <= c1 + 20.0) {
                const int last = (int)min((double)b, floor(((double)c0 + cap) + 20.0));
                e = max(e, last);
                double pad = (double)(e - c0) * 1.7;
                if (cap < pad) pad = cap;
                c1 = (double)c0 + pad;
            } else if (e > c0) {
                span(c0, c1, false);
                c0 = e;
                c1 = (double)e;
            }
            ++e;
        }
        e = b + 1 > bits.end - gap ? bits.next(b + 1, bits.end) : bits.next(b + 1, b + 1 + gap);
        if (e >= bits.end) break;
    }
    span(c0, c1, b >= top);
    return b;
}

constexpr int kHeld = 4;  // spans a thread keeps from the first merge of its segments

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

// Threads own consecutive words of the mask.  An error sample more than a
// span's reach after the one before it starts a segment, whose merge
// does not depend on what came before: the thread that owns it merges the
// segment (past its words where it runs on) and keeps its spans; their
// dropouts are counted, then written.  (More spans than it keeps: the
// merge runs again for each of the two.)
__global__ void __launch_bounds__(kPlaceThreads) dropout_place_kernel(const DropField* fields, const DropConsts k,
                                                                      const DropScratch sc, int* drops, int* counts) {
    extern __shared__ unsigned swords[];  // kPlaceWords
    __shared__ int wsum[32];
    __shared__ int s_first, s_down;
    __shared__ double ll[kMaxDropRegions + 1];  // the line locations (the placement searches them)
    const DropField f = fields[blockIdx.x];
    const int t = threadIdx.x;
    for (int l = t; l < f.nlines; l += kPlaceThreads) ll[l] = f.ll[l];
    const int bad = sc.bad[blockIdx.x];
    if (bad) {
        if (t == 0) {
            counts[2 * blockIdx.x] = (bad & 2) ? -3 : -2;
            counts[2 * blockIdx.x + 1] = 0;
        }
        return;
    }
    if (t == 0) {
        s_first = 0x7fffffff;
        s_down = 0;
    }
    __syncthreads();
    long long lo, hi;
    mask_range(f, lo, hi);
    const double ll0 = ll[f.lineoffset];
    const int from = (int)min(max(lo, (long long)ceil(ll0)), hi);  // the errors before line `lineoffset` start no span
    const long long w0 = lo >> 5, nw = hi > lo ? ((hi + 31) >> 5) - w0 : 0;
    // the mask in shared memory when it fits (a field of 1.5 M samples does):
    // the searches below are chains of single-word reads
    ErrorBits bits{sc.words + f.word0, (int)hi};
    if (nw <= sc.place_words) {
#pragma unroll 8
        for (int w = t; w < (int)nw; w += kPlaceThreads) swords[w] = bits.words[w0 + w];
        bits.words = swords - w0;
    }
    __syncthreads();
    const long long per = (nw + kPlaceThreads - 1) / kPlaceThreads;
    // this thread's samples
    const int a = (int)min(max((long long)from, (w0 + t * per) << 5), hi);
    const int b = (int)min(hi, (w0 + (t + 1) * per) << 5);
    // errors of the field; this thread's last one, and the last one before its words
    int n = 0;
    long long last = -1;
    for (long long w = w0 + t * per; w < min(w0 + nw, w0 + (t + 1) * per); ++w) {
        const unsigned m = bits.words[w];
        n += __popc(m);
        if (m) last = 32 * w + 31 - __clz(m);
    }
    int nerr;
    block_scan(n, wsum, &nerr);
    if (t == 0) counts[2 * blockIdx.x + 1] = nerr > k.err_cap ? -1 : nerr;
    if (nerr > k.err_cap) {
        if (t == 0) counts[2 * blockIdx.x] = 0;
        return;
    }
    if (last < from) last = -1;  // (the last error alone decides whether there are spans: it must lie past ll0)
    __shared__ int wmax[32];
    int before = (int)last;
    const int lane = t & 31, warp = t >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, before, o);
        if (lane >= o) before = max(before, y);
    }
    if (lane == 31) wmax[warp] = before;
    before = __shfl_up_sync(0xffffffffu, before, 1);
    if (lane == 0) before = -1;
    // are the line locations in order?
    for (int l = f.lineoffset + t; l < f.lineoffset + f.linecount; l += kPlaceThreads)
        if (!(ll[l] <= ll[l + 1])) s_down = 1;
    __syncthreads();
    int top = -1;
    for (int w = 0; w < 32; ++w) {
        if (w < warp) before = max(before, wmax[w]);
        top = max(top, wmax[w]);
    }
    if (top < 0 || !((double)top > ll0)) {  // no error, or none past ll0
        if (t == 0) counts[2 * blockIdx.x] = 0;
        return;
    }
    const double cap = k.freq_mhz * 12.0;
    const int gap = (int)min(cap + 21.0, 1.0e9);
    // every segment that starts among this thread's samples, in order
    auto segments = [&](auto&& span) {
        int prev = before;
        for (int e = bits.next(a, b); e < bits.end;) {
            if (prev < 0 || e - prev > gap) {
                prev = merge_segment(bits, e, gap, cap, top, span);
            } else {
                prev = bits.run_end(e);
            }
            e = bits.next(prev + 1, b);
        }
    };
    // a span as the placement gets it: 8 samples ahead and 4 behind, but the last one as it is
    auto start_of = [](int c0, bool is_last) { return (double)(is_last ? c0 : c0 - 8); };
    Emitter em{drops + (size_t)blockIdx.x * k.out_cap * 3, k.out_cap, 0, false};
    if (s_down) {
        // line locations out of order: the placement's search depends on the spans before
        if (t == 0) {
            LinePlacer lp{ll, f.lineoffset, f.lineoffset + f.linecount, f.lineoffset, (double)k.outlinelen, ll0,
                          false, false, 0.0, 0.0, &em};
            int e = bits.next(from, bits.end);
            while (e < bits.end) {
                const int l = merge_segment(bits, e, gap, cap, top, [&](int c0, double c1, bool is_last) {
                    lp.feed(start_of(c0, is_last), is_last ? c1 : c1 + 4.0);
                });
                e = bits.next(l + 1, bits.end);
            }
            lp.finish();
            counts[2 * blockIdx.x] = em.over ? -1 : em.n;
        }
        return;
    }
    // the first span the placement keeps: the first from ll0 on, else the last
    int nspans = 0, first = 0x7fffffff;
    int held0[kHeld];
    double held1[kHeld];
    bool ends = false;  // the last span is the field's last
    segments([&](int c0, double c1, bool is_last) {
        if (nspans < kHeld) {
            held0[nspans] = c0;
            held1[nspans] = c1;
        }
        ends = is_last;
        if (first == 0x7fffffff && start_of(c0, is_last) >= ll0) first = nspans;
        ++nspans;
    });
    int total;
    const int base = block_scan(nspans, wsum, &total);
    if (first != 0x7fffffff) atomicMin(&s_first, base + first);
    __syncthreads();
    const int keep = min(s_first, total - 1);
    // the line of a span: the first one it starts in
    auto line_of = [&](double c0) {
        int x = f.lineoffset, y = f.lineoffset + f.linecount;  // first line with c0 <= its end
        while (x < y) {
            const int mid = (x + y) >> 1;
            if (ll[mid + 1] >= c0) y = mid; else x = mid + 1;
        }
        return x < f.lineoffset + f.linecount && c0 >= ll[x] ? x : -1;
    };
    auto place = [&](Emitter& out) {
        int i = base;
        auto one = [&](int c0, double c1, bool is_last) {
            if (i++ < keep) return;
            const double s0 = start_of(c0, is_last);
            const int line = line_of(s0);
            if (line < 0) return;
            LinePlacer lp{ll, line, line + 1, f.lineoffset, (double)k.outlinelen, ll0, true, false, 0.0, 0.0, &out};
            lp.place(s0, is_last ? c1 : c1 + 4.0);
        };
        if (nspans <= kHeld) {
            for (int q = 0; q < nspans; ++q) one(held0[q], held1[q], ends && q == nspans - 1);
        } else {
            segments(one);
        }
    };
    Emitter dry{nullptr, 0, 0, false};
    place(dry);
    const int at = block_scan(dry.n, wsum, &total);
    em.n = at;
    place(em);
    if (t == 0) counts[2 * blockIdx.x] = total > k.out_cap ? -1 : total;
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
    // no more shared memory than the longest mask needs
    const size_t bytes = (size_t)sc.place_words * sizeof(unsigned);
    static SmemAttr attr;
    const cudaError_t e = attr.ensure(dropout_place_kernel, bytes);
    if (e != cudaSuccess) return e;
    dropout_place_kernel<<<nfields, kPlaceThreads, bytes, stream>>>(fields, k, sc, drops, counts);
    return cudaGetLastError();
}

}  // namespace ldg
