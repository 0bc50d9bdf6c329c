// Fused per-block RF demodulator: one 1024-thread CTA per 32768-sample
// overlap-save block, persistent over blocks.
//
// Per block, in shared memory (a 16384-point complex working set S):
//   X = R2C(x)                         input spectrum, bins 0..N/2 (first FFT
//                                      pass reads the int16 block directly)
//   rfhpf  = C2R(X * Frfhpf)           -> float32 (last pass stores directly)
//   efm    = C2R(X * Fefm/2)           -> int16 (truncated)
//   audio  = 2 x (1024-bin sub-band * filt1 -> iFFT -> FM discriminator)
//   z      = analytic signal of X * RFVideo * MTF^m, as its even and odd
//            samples: two 16384-point inverse FFTs whose first pass reads
//            X * G (resp. X * G * W^-k) from the parked spectrum
//   demod_raw = arg(z[n] conj z[n-1]) * fs / 2pi, in [0, fs)
//   D      = R2C(clip(demod_raw, 1.5 MHz, 0.75 fs))
//   demod / demod_05 / demod_burst [/ demod_pilot] = C2R(D * F) with rolls
// The real-FFT pre/post-processing is fused with parking the spectrum and
// with the filter products; spectra and the even half of z are parked in a
// per-CTA global scratch (256 KB per CTA, L2 resident).  This restates
// RFDecode.demodblock_cpu (lddecode/core.py:755-879) and unwrap_hilbert
// (lddecode/utils.py:898-926).
//
// This file: the device code of a block, shared by the kernels that give a
// block to one CTA (ldg_demod.cu) and to a cluster (ldg_demod_split.cu).  The
// two are compiled apart: with both in one unit the compiler inlined less
// into the first (1671 against 1661 us per 2368 NTSC blocks in place, 1968 against 1928
// us per 2368 PAL blocks Stockham).
#pragma once
#include "ldg_attr.cuh"
#include "ldg_demod.cuh"
#include "ldg_fft.cuh"
#include "ldg_fft_ip.cuh"

namespace ldg {

namespace {

constexpr float kTwoPi = 6.28318530717958647692f;
constexpr float kInvM = 1.0f / kM;

// arctan t for t in [0, 1]: the minimax polynomial of Abramowitz & Stegun,
// Handbook of Mathematical Functions, 4.4.49 (after Hastings): arctan t / t
// = 1 + a2 t^2 + ... + a16 t^16 with |error| <= 2e-8; in float32 Horner
// form within 1.6 ulp of arctan.
__device__ __forceinline__ float atan01(float t) {
    const float t2 = t * t;
    float p = 0.0028662257f;
    p = fmaf(p, t2, -0.0161657367f);
    p = fmaf(p, t2, 0.0429096138f);
    p = fmaf(p, t2, -0.0752896400f);
    p = fmaf(p, t2, 0.1065626393f);
    p = fmaf(p, t2, -0.1420889944f);
    p = fmaf(p, t2, 0.1999355085f);
    p = fmaf(p, t2, -0.3333314528f);
    p = fmaf(p, t2, 1.0f);
    return t * p;
}

// arg(re + i im) in [0, 2 pi): the octant's arctan of min/max, reflected
__device__ __forceinline__ float arg_2pi(float im, float re) {
    constexpr float kPi = 3.14159265358979323846f, kHalfPi = 1.57079632679489661923f;
    const float ax = fabsf(re), ay = fabsf(im);
    const float mx = fmaxf(ax, ay), mn = fminf(ax, ay);
    float r = atan01(mx > 0.0f ? mn / mx : 0.0f);
    if (ay > ax) r = kHalfPi - r;
    if (re < 0.0f) r = kPi - r;
    return im < 0.0f ? kTwoPi - r : r;
}

__device__ __forceinline__ float fm_disc(float2 a, float2 b, float k) {
    // arg(a * conj(b)) wrapped to [0, 2pi), times k = rate / 2pi
    const float re = fmaf(a.x, b.x, a.y * b.y);
    const float im = fmaf(a.y, b.x, -a.x * b.y);
    return arg_2pi(im, re) * k;
}

// ---- first-pass loaders

struct InLoader16 {  // x[2m], x[2m+1] from int16 samples
    const int16_t* x;
    __device__ float2 operator()(int, int m) const {
        const int w = __ldcs(reinterpret_cast<const int*>(x) + m);  // read once: streaming
        return make_float2((float)(int16_t)(w & 0xffff), (float)(int16_t)(((unsigned)w) >> 16));
    }
};

struct InLoader32 {  // float32 samples
    const float* x;
    __device__ float2 operator()(int, int m) const { return __ldg(reinterpret_cast<const float2*>(x) + m); }
};

struct ParkLoader {
    const float2* p;
    __device__ float2 operator()(int, int m) const { return p[m]; }
};

// X[k] * G[k] from the parked spectrum (X[0], X[M] packed in element 0);
// `odd` selects the odd-sample spectrum (G * W^-k, and X0 G0 - XM GM at 0).
struct AnalyticLoader {
    const float2* X;
    const float2* G;
    const float2* Godd;
    bool odd;
    __device__ float2 operator()(int, int k) const {
        const float2 x = X[k];
        if (k == 0) {
            const float2 a = cscale(__ldg(G), x.x);
            const float2 b = cscale(__ldg(G + kM), x.y);
            return odd ? csub(a, b) : cadd(a, b);
        }
        return cmul(x, __ldg((odd ? Godd : G) + k));
    }
};

// ---- last-pass storers (z[m] = M * (x[2m] + i x[2m+1]))

// Real output: sample n of the block goes to out[i], i = (n - off) mod N, if i < len
// (off = start + roll).  Streaming stores: outputs are not re-read here, keep
// L2 for the parked spectra.  PairStorer for outputs whose sample pairs stay
// pairs (pairs_kept), RealStorer for the others (rfhpf starts at an odd
// sample): the choice is one branch per transform.  Testing alignment and both
// bounds at every pair instead: 1745 against 1685 us per 2368 NTSC blocks (in
// place), 1978 against 1931 us per 2368 PAL blocks (Stockham), B200.
struct PairStorer {
    float* out;
    int off, len;
    __device__ void operator()(int, int m, float2 v) const {
        const int i0 = (2 * m - off) & (kN - 1);
        if (i0 < len) __stcs(reinterpret_cast<float2*>(out + i0), make_float2(v.x * kInvM, v.y * kInvM));
    }
};

struct RealStorer {
    float* out;
    int off, len;
    __device__ void operator()(int, int m, float2 v) const {
        const int i0 = (2 * m - off) & (kN - 1);
        const int i1 = (i0 + 1) & (kN - 1);
        if (i0 < len) __stcs(out + i0, v.x * kInvM);
        if (i1 < len) __stcs(out + i1, v.y * kInvM);
    }
};

// Do the pairs (2m, 2m + 1) of a block land on aligned pairs of out, both inside or both outside?
template <class T>
__device__ __forceinline__ bool pairs_kept(const T* out, int off, int len) {
    return ((off | len) & 1) == 0 && (reinterpret_cast<uintptr_t>(out) & (2 * sizeof(T) - 1)) == 0;
}

__device__ __forceinline__ int16_t to_efm(float x) {
    x = fminf(fmaxf(x * kInvM, -32768.0f), 32767.0f);
    return (int16_t)__float2int_rz(x);
}

struct EfmPairStorer {
    int16_t* out;
    int off, len;
    __device__ void operator()(int, int m, float2 v) const {
        const int i0 = (2 * m - off) & (kN - 1);
        // both samples in one aligned 32-bit store (little-endian: v.x first)
        if (i0 < len)
            __stcs(reinterpret_cast<int*>(out + i0),
                   (int)__byte_perm((unsigned)(int)to_efm(v.x), (unsigned)(int)to_efm(v.y), 0x5410));
    }
};

struct EfmStorer {
    int16_t* out;
    int off, len;
    __device__ void operator()(int, int m, float2 v) const {
        const int i0 = (2 * m - off) & (kN - 1);
        const int i1 = (i0 + 1) & (kN - 1);
        if (i0 < len) __stcs(reinterpret_cast<short*>(out) + i0, (short)to_efm(v.x));
        if (i1 < len) __stcs(reinterpret_cast<short*>(out) + i1, (short)to_efm(v.y));
    }
};

struct ParkStorer {
    float2* p;
    __device__ void operator()(int, int m, float2 v) const { p[m] = v; }
};

// ---- real-FFT pre/post-processing, fused with parking and filter products

// C2R pre-processing of the pair (H[k], H[M-k]) into the M-point complex
// spectrum whose inverse FFT is M * (x[2m] + i x[2m+1]).
__device__ __forceinline__ void c2r_pair(float2* S, int k, float2 hk, float2 hm, float2 wk) {
    const float2 e = make_float2(0.5f * (hk.x + hm.x), 0.5f * (hk.y - hm.y));
    const float2 d = make_float2(0.5f * (hk.x - hm.x), 0.5f * (hk.y + hm.y));
    const float2 o = cmul(d, cconj(wk));
    S[pad(k)] = make_float2(e.x - o.y, e.y + o.x);
    if (k != kM / 2) S[pad(kM - k)] = make_float2(e.x + o.y, o.x - e.y);
}

__device__ __forceinline__ void c2r_dc(float2* S, float x0, float xm, const float2* F) {
    const float h0 = x0 * __ldg(&F[0].x), hm = xm * __ldg(&F[kM].x);
    S[0] = make_float2(0.5f * (h0 + hm), 0.5f * (h0 - hm));
}

struct AudioTaps {
    float2* A;             // two padded 1024-point sets
    int lowbin[2];
    const float2* filt1[2];
};

// Post-processing of one bin pair (k, M-k), 0 < k <= M/2, from Z[k], Z[M-k]
// (S), the real-FFT twiddle wk and, if F is given, the filter bins.
__device__ __forceinline__ void post_pair(float2* S, float2* park, const AudioTaps* au, int k, float2 zk, float2 zm,
                                          float2 wk, const float2* F, float2 fk, float2 fm) {
    const float2 e = make_float2(0.5f * (zk.x + zm.x), 0.5f * (zk.y - zm.y));
    const float2 o = make_float2(0.5f * (zk.y + zm.y), -0.5f * (zk.x - zm.x));
    const float2 tt = cmul(wk, o);
    const float2 xk = cadd(e, tt);
    const float2 xm = cconj(csub(e, tt));
    park[k] = xk;
    if (k != kM / 2) park[kM - k] = xm;
    if (au) {
#pragma unroll
        for (int ch = 0; ch < 2; ++ch) {
            const int rel = k - au->lowbin[ch];
            if (rel >= 0 && rel <= 512) {
                const float2 xb = rel < 512 ? xk : cconj(xk);
                au->A[ch * padded(1024) + pad(rel)] = cmul(xb, __ldg(au->filt1[ch] + rel));
            }
        }
    }
    if (F) c2r_pair(S, k, cmul(xk, fk), cmul(xm, fm), wk);
}

// S holds Z = FFT_M(x[2m] + i x[2m+1]).  Computes X[k] for k = 0..M, parks
// it, taps the audio sub-bands and, if F is given, leaves the C2R input of
// X * F in S.  Thread t handles k = t + kThreads i; two bins per step with all
// their loads issued before the arithmetic (latency of the global twiddle
// and filter loads overlapped).
__device__ void post_r2c(float2* S, const Tables& t, float2* park, const float2* F, const AudioTaps* au) {
    const int t0 = threadIdx.x;
    const float2 zero = make_float2(0.f, 0.f);
#pragma unroll 1
    for (int i = 0; i < kM / 2 / kThreads; i += 2) {
        const int ka = t0 + i * kThreads, kb = ka + kThreads;  // kb > 0; ka == 0 only for thread 0
        const float2 zka = S[pad(ka)];
        const float2 zma = ka ? S[pad(kM - ka)] : zero;
        const float2 zkb = S[pad(kb)], zmb = S[pad(kM - kb)];
        const float2 wa = __ldg(t.t32 + ka), wb = __ldg(t.t32 + kb);
        float2 fka = zero, fma = zero, fkb = zero, fmb = zero;
        if (F) {
            fka = __ldg(F + ka);
            fma = __ldg(F + kM - ka);
            fkb = __ldg(F + kb);
            fmb = __ldg(F + kM - kb);
        }
        if (ka == 0) {
            const float x0 = zka.x + zka.y, xm = zka.x - zka.y;
            park[0] = make_float2(x0, xm);
            if (F) c2r_dc(S, x0, xm, F);
        } else {
            post_pair(S, park, au, ka, zka, zma, wa, F, fka, fma);
        }
        post_pair(S, park, au, kb, zkb, zmb, wb, F, fkb, fmb);
    }
    if (t0 == 0) {  // k = M/2
        const int k = kM / 2;
        const float2 z = S[pad(k)];
        post_pair(S, park, au, k, z, z, __ldg(t.t32 + k), F, F ? __ldg(F + k) : zero, F ? __ldg(F + k) : zero);
    }
}

// Is the bin pair (k, M - k) inside the band [klo, khi] where the filter's
// float32 bins are not zero?  (Outside it X * F is zero and so is the C2R
// input; for a band-limited filter such as the EFM one most pairs are.)
__device__ __forceinline__ bool pair_live(int k, int klo, int khi) {
    const int m = k == 0 ? kM : kM - k;
    return (k >= klo && k <= khi) || (m >= klo && m <= khi);
}

// C2R input of X * F in S, X from the parked spectrum; two bins per step,
// loads first.  Pairs outside F's band [klo, khi] are written as zeros
// without their loads.
__device__ void pre_c2r(float2* S, const Tables& t, const float2* park, const float2* F, int klo = 0,
                        int khi = kM) {
    const int t0 = threadIdx.x;
    const float2 zero = make_float2(0.f, 0.f);
#pragma unroll 1
    for (int i = 0; i < kM / 2 / kThreads; i += 2) {
        const int ka = t0 + i * kThreads, kb = ka + kThreads;
        if (!pair_live(ka, klo, khi) && !pair_live(kb, klo, khi)) {
            S[pad(ka)] = zero;
            if (ka) S[pad(kM - ka)] = zero;
            S[pad(kb)] = zero;
            S[pad(kM - kb)] = zero;
            continue;
        }
        const float2 xka = park[ka], xkb = park[kb], xmb = park[kM - kb];
        const float2 xma = ka ? park[kM - ka] : xka;
        const float2 fka = __ldg(F + ka), fma = __ldg(F + kM - ka), fkb = __ldg(F + kb), fmb = __ldg(F + kM - kb);
        const float2 wa = __ldg(t.t32 + ka), wb = __ldg(t.t32 + kb);
        if (ka == 0) {
            c2r_dc(S, xka.x, xka.y, F);
        } else {
            c2r_pair(S, ka, cmul(xka, fka), cmul(xma, fma), wa);
        }
        c2r_pair(S, kb, cmul(xkb, fkb), cmul(xmb, fmb), wb);
    }
    if (t0 == 0) {
        const int k = kM / 2;
        if (pair_live(k, klo, khi)) {
            const float2 x = park[k];
            c2r_pair(S, k, cmul(x, __ldg(F + k)), cmul(x, __ldg(F + k)), __ldg(t.t32 + k));
        } else {
            S[pad(k)] = zero;
        }
    }
}

__device__ void audio_stage(const DemodParams& p, float2* A, const Tables& t, int blk) {
    constexpr int stride = padded(1024);
    fft1k_x2<true>(A, t);
    const float kk = p.a_rate / kTwoPi;
    for (int idx = threadIdx.x; idx < 2 * 1024; idx += kThreads) {
        const int ch = idx >> 10, n = idx & 1023;
        const int i = n - p.s_audio.start;
        float* oa = ch ? p.o_audio[1] : p.o_audio[0];
        if (i < 0 || i >= p.s_audio.len || oa == nullptr) continue;
        const float2* Ab = A + ch * stride;
        const float d = (n == 0) ? 0.0f : fm_disc(Ab[pad(n)], Ab[pad(n - 1)], kk);
        __stcs(oa + (long long)blk * p.s_audio.len + i, d + (ch ? p.a_low[1] : p.a_low[0]));
    }
}

// PAL_V4300D_NotchFilter (lddecode/core.py:774-798) on the parked input
// spectrum: in bins [lo, hi), every bin whose magnitude exceeds the band's
// mean + 3 std (FP64, population std) is zeroed with its two neighbours; the
// mirrored negative-frequency bins are implicit in the half spectrum.  One
// warp; the decisions use the magnitudes before any bin is zeroed.  At most
// 1024 bins (checked on the host).
__device__ void notch_park(float2* park, int lo, int hi) {
    if (threadIdx.x >= 32) return;
    const int lane = threadIdx.x;
    const int n = hi - lo;
    auto mag = [&](int i) {
        const float2 x = park[lo + i];
        return sqrt((double)x.x * (double)x.x + (double)x.y * (double)x.y);
    };
    double s = 0.0;
    for (int i = lane; i < n; i += 32) s += mag(i);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    const double mean = s / (double)n;
    double q = 0.0;
    for (int i = lane; i < n; i += 32) {
        const double d = mag(i) - mean;
        q += d * d;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
    const double m = mean + sqrt(q / (double)n) * 3.0;
    unsigned flags = 0;
    for (int i = lane, j = 0; i < n; i += 32, ++j)
        if (mag(i) > m) flags |= 1u << j;
    __syncwarp();
    for (int i = lane, j = 0; i < n; i += 32, ++j) {
        if ((flags >> j) & 1u) {
            const float2 z = make_float2(0.f, 0.f);
            park[lo + i - 1] = z;
            park[lo + i] = z;
            park[lo + i + 1] = z;
        }
    }
}

// Invalidate this CTA's scratch (parkX and parkZ, kScratchPerCta bytes,
// 128-byte aligned) in L2 without write-back: discard.global.L2 per 128-byte
// line.  Every thread of the CTA is past its last scratch access.
__device__ __forceinline__ void discard_scratch(float2* base) {
    char* b = reinterpret_cast<char*>(base);
    constexpr int kLines = (int)(kScratchPerCta / 128);
    for (int l = threadIdx.x; l < kLines; l += kThreads)
        asm volatile("discard.global.L2 [%0], 128;" ::"l"(b + (size_t)l * 128) : "memory");
}

// FM discriminator: demod[2m] from (z_e[m], z_o[m-1]), demod[2m+1] from
// (z_o[m], z_e[m]) -- the even samples parked (parkZ), the odd ones in S,
// both in natural order; the clipped pairs replace X in the parking slot.
__device__ __forceinline__ void discriminate(const DemodParams& p, int blk, const float2* S, float2* parkX,
                                             const float2* parkZ) {
    {
        const float kfs = p.fs_hz / kTwoPi;
        const float clip_hi = p.fs_hz * 0.75f;
        float* oraw = p.o_raw ? p.o_raw + (long long)blk * p.s_video.len : nullptr;
        const int vs = p.s_video.start, vl = p.s_video.len;
        const bool pairs = oraw && pairs_kept(oraw, vs, vl);
        auto disc_store = [&](int m, float de, float dodd) {
            if (oraw) {
                const int i0 = 2 * m - vs;
                if (pairs) {
                    if ((unsigned)i0 < (unsigned)vl) __stcs(reinterpret_cast<float2*>(oraw + i0), make_float2(de, dodd));
                } else {
                    if (i0 >= 0 && i0 < vl) __stcs(oraw + i0, de);
                    if (i0 + 1 >= 0 && i0 + 1 < vl) __stcs(oraw + i0 + 1, dodd);
                }
            }
            parkX[m] = make_float2(fminf(fmaxf(de, 1500000.0f), clip_hi), fminf(fmaxf(dodd, 1500000.0f), clip_hi));
        };
        // two samples per step, the parked (L2) loads first
#pragma unroll 2
        for (int m = threadIdx.x; m < kM; m += 2 * kThreads) {
            const int mb = m + kThreads;
            const float2 zea = parkZ[m], zeb = parkZ[mb];
            const float2 zoa = S[pad(m)], zob = S[pad(mb)];
            const float2 zpa = m ? S[pad(m - 1)] : zoa, zpb = S[pad(mb - 1)];
            const float dea = (m == 0) ? 0.0f : fm_disc(zea, zpa, kfs);
            const float doa = fm_disc(zoa, zea, kfs);
            const float deb = fm_disc(zeb, zpb, kfs);
            const float dob = fm_disc(zob, zeb, kfs);
            disc_store(m, dea, doa);
            disc_store(mb, deb, dob);
        }
    }
}

// Inverse transform of S (either decomposition: pass tables or stage tables)
// with its real output stored at out.
__device__ __forceinline__ void inverse_out(float2* S, const Tables& t, float* out, int off, int len) {
    if (pairs_kept(out, off, len)) fft16k<true>(S, t, SmemIO(), PairStorer{out, off, len});
    else fft16k<true>(S, t, SmemIO(), RealStorer{out, off, len});
}
__device__ __forceinline__ void inverse_out(float2* S, const Tables& t, int16_t* out, int off, int len) {
    if (pairs_kept(out, off, len)) fft16k<true>(S, t, SmemIO(), EfmPairStorer{out, off, len});
    else fft16k<true>(S, t, SmemIO(), EfmStorer{out, off, len});
}
__device__ __forceinline__ void inverse_out(float2* S, const ip::Twiddles& tw, float* out, int off, int len) {
    if (pairs_kept(out, off, len)) ip::fft16k_inv(S, tw, SmemIO(), PairStorer{out, off, len});
    else ip::fft16k_inv(S, tw, SmemIO(), RealStorer{out, off, len});
}
__device__ __forceinline__ void inverse_out(float2* S, const ip::Twiddles& tw, int16_t* out, int off, int len) {
    if (pairs_kept(out, off, len)) ip::fft16k_inv(S, tw, SmemIO(), EfmPairStorer{out, off, len});
    else ip::fft16k_inv(S, tw, SmemIO(), EfmStorer{out, off, len});
}

// One block: every requested output of block `blk` of p.  parkX/parkZ: this
// CTA's scratch (kScratchPerCta).  Ends with the CTA's threads in step.
__device__ __forceinline__ void demod_block(const DemodParams& p, int blk, float2* S, float2* A, const Tables& t,
                                            float2* parkX, float2* parkZ) {
    // ---- input spectrum X (first pass reads the block), parked; audio taps; rfhpf input
    if (p.in_kind == 0) {
        fft16k<false>(S, t, InLoader16{static_cast<const int16_t*>(p.in) + (long long)blk * p.in_stride});
    } else {
        fft16k<false>(S, t, InLoader32{static_cast<const float*>(p.in) + (long long)blk * p.in_stride});
    }
    if (p.audio) {
        for (int idx = threadIdx.x; idx < 2 * 511; idx += kThreads) {
            const int ch = idx / 511, k = 513 + idx % 511;
            A[ch * padded(1024) + pad(k)] = make_float2(0.f, 0.f);
        }
    }
    {
        AudioTaps au{A, {p.a_lowbin[0], p.a_lowbin[1]}, {p.a_filt1[0], p.a_filt1[1]}};
        post_r2c(S, t, parkX, p.o_rfhpf ? p.f_rfhpf : nullptr, p.audio ? &au : nullptr);
    }
    __syncthreads();
    // rfhpf (already in S) and the audio taps use the spectrum before the
    // notch, as the reference does (its notch band lies far from the audio bands)
    if (p.notch_hi > p.notch_lo) {
        notch_park(parkX, p.notch_lo, p.notch_hi);
        __syncthreads();
    }
    if (p.audio) audio_stage(p, A, t, blk);

    // ---- rfhpf
    if (p.o_rfhpf) {
        inverse_out(S, t, p.o_rfhpf + (long long)blk * p.s_rfhpf.len, p.s_rfhpf.start, p.s_rfhpf.len);
    }

    // ---- EFM
    if (p.o_efm) {
        pre_c2r(S, t, parkX, p.f_efm, p.efm_klo, p.efm_khi);
        __syncthreads();
        inverse_out(S, t, p.o_efm + (long long)blk * p.s_efm.len, p.s_efm.start, p.s_efm.len);
    }

    // ---- analytic signal: even samples (parked), then odd samples (in S)
    fft16k<true>(S, t, AnalyticLoader{parkX, p.f_g, p.f_godd, false}, ParkStorer{parkZ});
    fft16k<true>(S, t, AnalyticLoader{parkX, p.f_g, p.f_godd, true});

    discriminate(p, blk, S, parkX, parkZ);
    __syncthreads();

    // ---- spectrum D of the clipped demod, then the video outputs
    fft16k<false>(S, t, ParkLoader{parkX});
    int first = -1;
#pragma unroll
    for (int o = 0; o < OUT_NVIDEO; ++o)
        if (first < 0 && p.o_video[o]) first = o;
    post_r2c(S, t, parkX, first >= 0 ? p.f_video[first] : nullptr, nullptr);
    __syncthreads();
#pragma unroll
    for (int o = 0; o < OUT_NVIDEO; ++o) {
        if (p.o_video[o] == nullptr) continue;
        if (o != first) {
            pre_c2r(S, t, parkX, p.f_video[o]);
            __syncthreads();
        }
        inverse_out(S, t, p.o_video[o] + (long long)blk * p.s_video.len, p.s_video.start + p.roll[o], p.s_video.len);
    }
    __syncthreads();
    // the parked spectra are dead: drop their L2 lines without writing them
    // back (the next block on this scratch writes before it reads)
    discard_scratch(parkX);
}

struct CtaSmem {
    float2* S;
    float2* A;
    Tables t;       // Stockham pass tables (t.s3 / t.s4 only for the Stockham variant) and the 1024-point ones
    ip::Twiddles tw;  // in-place stage tables (in-place variant)
};

// Carves the dynamic shared memory -- working set, audio bands, 1024-point
// tables, then the 16384-point tables of the variant -- and loads the tables.
template <int V>
__device__ __forceinline__ CtaSmem cta_setup(float2* smem, const float2* tw16, const float2* tw32) {
    CtaSmem c;
    c.S = smem;
    c.A = smem + padded(kM);
    float2* s2 = c.A + 2 * padded(1024);
    float2* s4a = s2 + kS2;
    float2* rest = s4a + kS4a;
    load_1k_tables(s2, s4a, tw16);
    c.t.t16 = tw16;
    c.t.t32 = tw32;
    c.t.s2 = s2;
    c.t.s4a = s4a;
    if (V == kVariantStockham) {
        float2* s3 = rest;
        float2* s4 = s3 + kS3;
        load_pass_tables(s3, s4, tw16);
        c.t.s3 = s3;
        c.t.s4 = s4;
        c.tw = {nullptr, nullptr, nullptr};
    } else {
        float2* t1 = rest;
        float2* t2 = t1 + ip::kT1;
        float2* t3 = t2 + ip::kT2;
        ip::load_stage_tables(t1, t2, t3, tw16);
        c.tw = {t1, t2, t3};
        c.t.s3 = nullptr;
        c.t.s4 = nullptr;
    }
    __syncthreads();
    return c;
}

// ---- the in-place variant: spectra in position order (ldg_fft_ip.cuh)

// X[k] * G[k] at positions p .. p+3 (k = bin_of(p)) from the parked spectrum
// (position order, X[0] and X[M] packed at position 0) and G at positions;
// `odd` as AnalyticLoader.
struct AnalyticLoaderIp {
    const float2* X;
    const float2* Gpos;
    const float2* G;  // natural order: G[0], G[M]
    bool odd;
    __device__ void quad(int p, float2 (&v)[4]) const {
        const float4 x01 = *reinterpret_cast<const float4*>(X + p);
        const float4 x23 = *reinterpret_cast<const float4*>(X + p + 2);
        const float4 g01 = __ldg(reinterpret_cast<const float4*>(Gpos + p));
        const float4 g23 = __ldg(reinterpret_cast<const float4*>(Gpos + p + 2));
        v[0] = cmul(make_float2(x01.x, x01.y), make_float2(g01.x, g01.y));
        v[1] = cmul(make_float2(x01.z, x01.w), make_float2(g01.z, g01.w));
        v[2] = cmul(make_float2(x23.x, x23.y), make_float2(g23.x, g23.y));
        v[3] = cmul(make_float2(x23.z, x23.w), make_float2(g23.z, g23.w));
        if (p == 0) {
            const float2 a = cscale(__ldg(G), x01.x);
            const float2 b = cscale(__ldg(G + kM), x01.y);
            v[0] = odd ? csub(a, b) : cadd(a, b);
        }
    }
};

// A bin pair of the table p.tw_pair: W_N^k, the positions p (bin k) and q
// (bin M - k) of its two bins and their padded indices in the working set.
// Taken from the table (16 contiguous bytes per thread) the indices cost no
// arithmetic; formed from u by digit reversal: 1685 against 1663 us per 2368
// NTSC blocks, B200.
struct Pair {
    float2 w;
    int p, q;    // positions (parked spectrum)
    int sp, sq;  // pad(p), pad(q)
};

__device__ __forceinline__ Pair load_pair(const float4* t) {
    const float4 v = __ldg(t);
    const unsigned pads = __float_as_uint(v.z), at = __float_as_uint(v.w);
    return {make_float2(v.x, v.y), (int)(at & 0xffff), (int)(at >> 16), (int)(pads & 0xffff), (int)(pads >> 16)};
}

// C2R pre-processing of one bin pair (c2r_pair in position order; p == q for
// k = M/2, where both values are the same).
__device__ __forceinline__ void c2r_pair_ip(float2* S, const Pair& u, float2 hk, float2 hm) {
    const float2 e = make_float2(0.5f * (hk.x + hm.x), 0.5f * (hk.y - hm.y));
    const float2 d = make_float2(0.5f * (hk.x - hm.x), 0.5f * (hk.y + hm.y));
    const float2 o = cmul(d, cconj(u.w));
    S[u.sp] = make_float2(e.x - o.y, e.y + o.x);
    if (u.q != u.p) S[u.sq] = make_float2(e.x + o.y, o.x - e.y);
}

// post_pair in position order: X[k], X[M-k] of the pair from Z[k] = S[p],
// Z[M-k] = S[q]; parked at p and q; with F, the C2R input of X * F left at p, q.
__device__ __forceinline__ void post_pair_ip(float2* S, float2* park, const Pair& u, float2 zk, float2 zm, bool hasF,
                                             float4 f) {
    const float2 e = make_float2(0.5f * (zk.x + zm.x), 0.5f * (zk.y - zm.y));
    const float2 o = make_float2(0.5f * (zk.y + zm.y), -0.5f * (zk.x - zm.x));
    const float2 tt = cmul(u.w, o);
    const float2 xk = cadd(e, tt);
    const float2 xm = cconj(csub(e, tt));
    park[u.p] = xk;
    if (u.q != u.p) park[u.q] = xm;
    if (hasF) c2r_pair_ip(S, u, cmul(xk, make_float2(f.x, f.y)), cmul(xm, make_float2(f.z, f.w)));
}

// post_r2c in position order: S holds Z at positions; parks X (position
// order) and, with FP, leaves the C2R input of X * F in S.  Thread t takes
// pairs u = t + kThreads i, two per step, loads first.
__device__ void post_r2c_ip(float2* S, const float4* twp, float2* park, const float4* FP) {
    const int t0 = threadIdx.x;
    const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
    for (int i = 0; i < 8; i += 2) {
        const int ua = t0 + i * kThreads, ub = ua + kThreads;
        const Pair a = load_pair(twp + ua), b = load_pair(twp + ub);
        float4 fa = zero4, fb = zero4;
        if (FP) {
            fa = __ldg(FP + ua);
            fb = __ldg(FP + ub);
        }
        const float2 zka = S[a.sp], zma = S[a.sq];
        const float2 zkb = S[b.sp], zmb = S[b.sq];
        post_pair_ip(S, park, a, zka, zma, FP != nullptr, fa);  // ua < 7680: never the pair of bins 0 and M
        if (b.p != 0) {
            post_pair_ip(S, park, b, zkb, zmb, FP != nullptr, fb);
        } else {  // bins 0 and M
            const float x0 = zkb.x + zkb.y, xm = zkb.x - zkb.y;
            park[0] = make_float2(x0, xm);
            if (FP) {
                const float h0 = x0 * fb.x, hm = xm * fb.z;
                S[0] = make_float2(0.5f * (h0 + hm), 0.5f * (h0 - hm));
            }
        }
    }
    if (t0 == 0) {  // u = M/2: position 2, bin M/2, its own partner
        const int u = kM / 2;
        const Pair c = load_pair(twp + u);
        const float2 z = S[c.sp];
        post_pair_ip(S, park, c, z, z, FP != nullptr, FP ? __ldg(FP + u) : zero4);
    }
}

// pre_c2r in position order: the C2R input of X * F in S, X from the parked
// spectrum (position order).  Band: pairs outside F's band [klo, khi] are
// written as zeros without their loads.
template <bool Band>
__device__ void pre_c2r_ip(float2* S, const float4* twp, const float2* park, const float4* FP, int klo = 0,
                           int khi = kM) {
    const int t0 = threadIdx.x;
    const float2 zero = make_float2(0.f, 0.f);
#pragma unroll 1
    for (int i = 0; i < 8; i += 2) {
        const int ua = t0 + i * kThreads, ub = ua + kThreads;
        const Pair a = load_pair(twp + ua), b = load_pair(twp + ub);
        if (Band && !pair_live(ip::bin_of(a.p), klo, khi) && !pair_live(ip::bin_of(b.p), klo, khi)) {
            // a is never the pair of bins 0 and M (ua < 7680); b may be
            S[a.sp] = zero;
            S[a.sq] = zero;
            S[b.sp] = zero;
            if (b.p != 0) S[b.sq] = zero;
            continue;
        }
        const float4 fa = __ldg(FP + ua), fb = __ldg(FP + ub);
        const float2 xka = park[a.p], xma = park[a.q], xkb = park[b.p], xmb = park[b.q];
        c2r_pair_ip(S, a, cmul(xka, make_float2(fa.x, fa.y)), cmul(xma, make_float2(fa.z, fa.w)));
        if (b.p != 0) {
            c2r_pair_ip(S, b, cmul(xkb, make_float2(fb.x, fb.y)), cmul(xmb, make_float2(fb.z, fb.w)));
        } else {
            const float h0 = xkb.x * fb.x, hm = xkb.y * fb.z;
            S[0] = make_float2(0.5f * (h0 + hm), 0.5f * (h0 - hm));
        }
    }
    if (t0 == 0) {
        const int u = kM / 2;
        const Pair c = load_pair(twp + u);
        if (!Band || pair_live(kM / 2, klo, khi)) {
            const float2 x = park[c.p];
            const float4 f = __ldg(FP + u);
            c2r_pair_ip(S, c, cmul(x, make_float2(f.x, f.y)), cmul(x, make_float2(f.z, f.w)));
        } else {
            S[c.sp] = zero;
        }
    }
}

// notch_park on the position-order parked spectrum.
__device__ void notch_park_ip(float2* park, int lo, int hi) {
    if (threadIdx.x >= 32) return;
    const int lane = threadIdx.x;
    const int n = hi - lo;
    auto mag = [&](int i) {
        const float2 x = park[ip::pos_of(lo + i)];
        return sqrt((double)x.x * (double)x.x + (double)x.y * (double)x.y);
    };
    double s = 0.0;
    for (int i = lane; i < n; i += 32) s += mag(i);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    const double mean = s / (double)n;
    double q = 0.0;
    for (int i = lane; i < n; i += 32) {
        const double d = mag(i) - mean;
        q += d * d;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
    const double m = mean + sqrt(q / (double)n) * 3.0;
    unsigned flags = 0;
    for (int i = lane, j = 0; i < n; i += 32, ++j)
        if (mag(i) > m) flags |= 1u << j;
    __syncwarp();
    for (int i = lane, j = 0; i < n; i += 32, ++j) {
        if ((flags >> j) & 1u) {
            const float2 z = make_float2(0.f, 0.f);
            park[ip::pos_of(lo + i - 1)] = z;
            park[ip::pos_of(lo + i)] = z;
            park[ip::pos_of(lo + i + 1)] = z;
        }
    }
}

// The audio bands' bins from the parked spectrum (position order), filtered.
__device__ __forceinline__ void gather_audio_ip(const DemodParams& p, float2* A, const float2* parkX) {
    for (int idx = threadIdx.x; idx < 2 * 513; idx += kThreads) {
        const int ch = idx >= 513, rel = idx - 513 * ch;
        const float2 x = parkX[ip::pos_of(p.a_lowbin[ch] + rel)];
        A[ch * padded(1024) + pad(rel)] = cmul(rel < 512 ? x : cconj(x), __ldg(p.a_filt1[ch] + rel));
    }
}

// demod_block with the in-place transforms: the same outputs from the same
// steps, spectra in position order.
__device__ __forceinline__ void demod_block_ip(const DemodParams& p, int blk, float2* S, float2* A, const Tables& t,
                                               const ip::Twiddles& tw, float2* parkX, float2* parkZ) {
    if (p.in_kind == 0) {
        ip::fft16k_fwd(S, tw, InLoader16{static_cast<const int16_t*>(p.in) + (long long)blk * p.in_stride});
    } else {
        ip::fft16k_fwd(S, tw, InLoader32{static_cast<const float*>(p.in) + (long long)blk * p.in_stride});
    }
    if (p.audio) {
        for (int idx = threadIdx.x; idx < 2 * 511; idx += kThreads) {
            const int ch = idx / 511, k = 513 + idx % 511;
            A[ch * padded(1024) + pad(k)] = make_float2(0.f, 0.f);
        }
    }
    post_r2c_ip(S, p.tw_pair, parkX, p.o_rfhpf ? p.fp_rfhpf : nullptr);
    __syncthreads();
    if (p.audio) {
        // the audio bands' bins, gathered from the parked spectrum (before the
        // notch, as the taps in post_r2c of the Stockham form): one L2 load per
        // thread instead of a band test in every bin pair's post-processing
        gather_audio_ip(p, A, parkX);
        __syncthreads();
    }
    if (p.notch_hi > p.notch_lo) {
        notch_park_ip(parkX, p.notch_lo, p.notch_hi);
        __syncthreads();
    }
    if (p.audio) audio_stage(p, A, t, blk);

    if (p.o_rfhpf) {
        inverse_out(S, tw, p.o_rfhpf + (long long)blk * p.s_rfhpf.len, p.s_rfhpf.start, p.s_rfhpf.len);
    }
    if (p.o_efm) {
        pre_c2r_ip<true>(S, p.tw_pair, parkX, p.fp_efm, p.efm_klo, p.efm_khi);
        __syncthreads();
        inverse_out(S, tw, p.o_efm + (long long)blk * p.s_efm.len, p.s_efm.start, p.s_efm.len);
    }

    ip::fft16k_inv(S, tw, AnalyticLoaderIp{parkX, p.g_pos, p.f_g, false}, ParkStorer{parkZ});
    ip::fft16k_inv(S, tw, AnalyticLoaderIp{parkX, p.godd_pos, p.f_g, true});

    discriminate(p, blk, S, parkX, parkZ);
    __syncthreads();

    ip::fft16k_fwd(S, tw, ParkLoader{parkX});
    int first = -1;
#pragma unroll
    for (int o = 0; o < OUT_NVIDEO; ++o)
        if (first < 0 && p.o_video[o]) first = o;
    post_r2c_ip(S, p.tw_pair, parkX, first >= 0 ? p.fp_video[first] : nullptr);
    __syncthreads();
#pragma unroll
    for (int o = 0; o < OUT_NVIDEO; ++o) {
        if (p.o_video[o] == nullptr) continue;
        if (o != first) {
            pre_c2r_ip<false>(S, p.tw_pair, parkX, p.fp_video[o]);
            __syncthreads();
        }
        inverse_out(S, tw, p.o_video[o] + (long long)blk * p.s_video.len, p.s_video.start + p.roll[o], p.s_video.len);
    }
    __syncthreads();
    discard_scratch(parkX);
}

template <int V>
__device__ __forceinline__ void run_block(const DemodParams& p, int blk, const CtaSmem& c, float2* parkX,
                                          float2* parkZ) {
    if (V == kVariantStockham) {
        demod_block(p, blk, c.S, c.A, c.t, parkX, parkZ);
    } else {
        demod_block_ip(p, blk, c.S, c.A, c.t, c.tw, parkX, parkZ);
    }
}

}  // namespace

}  // namespace ldg
