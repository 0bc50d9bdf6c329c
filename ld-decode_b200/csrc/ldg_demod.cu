// Launches of the fused per-block demodulator (ldg_demod_block.cuh): one CTA
// per block, persistent CTAs over a work queue; and the transforms beside it
// (analog audio stage 2, blocks from spectra).
#include "ldg_demod_block.cuh"

namespace ldg {

namespace {

template <int V>
__device__ __forceinline__ void demod_body(const DemodParams& p, float2* smem) {
    const CtaSmem c = cta_setup<V>(smem, p.tw16, p.tw32);

    __shared__ int s_got;
    const bool per_block = p.slot_lock != nullptr;
    const int slot = per_block ? (int)(blockIdx.x % (unsigned)p.nslots) : (int)blockIdx.x;
    if (per_block) {
        if (threadIdx.x == 0) {
            int got = 0;
            for (int tries = 0; tries < (1 << 22); ++tries) {
                if (atomicCAS(p.slot_lock + slot, 0, 1) == 0) {
                    got = 1;
                    break;
                }
                __nanosleep(256);
            }
            if (!got) atomicOr(p.error, kDemodErrSlotWait);
            __threadfence();
            s_got = got;
        }
        __syncthreads();
        if (!s_got) return;
    }
    int blk = per_block ? (int)blockIdx.x * p.blocks_per_cta : (int)blockIdx.x;
    const int blk_end = per_block ? min(blk + p.blocks_per_cta, p.nblocks) : p.nblocks;
    const int blk_step = per_block ? 1 : (int)gridDim.x;
    float2* parkX = p.scratch + (size_t)slot * 2 * kM;
    float2* parkZ = parkX + kM;
    for (; blk < blk_end; blk += blk_step) run_block<V>(p, blk, c, parkX, parkZ);
    if (per_block) {
        // every thread is done with the slot's scratch before it is handed on
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            atomicExch(p.slot_lock + slot, 0);
        }
    }
}

// Persistent CTAs over a device work queue of blocks of many captures: each
// CTA pops `grab` consecutive global block indices at a time from *head,
// finds the capture that holds each (binary search over first_block), keeps
// that capture's parameters in shared memory, and demodulates the block.
template <int V>
__device__ __forceinline__ void queue_body(const QueueParams& q, float2* smem) {
    const CtaSmem c = cta_setup<V>(smem, q.tw16, q.tw32);
    __shared__ DemodParams sp;
    __shared__ long long s_pop;
    __shared__ int s_item;
    float2* parkX = q.scratch + (size_t)blockIdx.x * 2 * kM;
    float2* parkZ = parkX + kM;
    int cur = -1;
    for (;;) {
        if (threadIdx.x == 0) s_pop = (long long)atomicAdd(q.head, (unsigned long long)q.grab);
        __syncthreads();
        const long long g0 = s_pop;
        if (g0 >= q.total) break;
        const long long g1 = min(g0 + (long long)q.grab, q.total);
        for (long long g = g0; g < g1; ++g) {
            if (threadIdx.x == 0) {
                int lo = 0, hi = q.nitems - 1;  // last item whose first block is <= g
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (q.first_block[mid] <= g) lo = mid; else hi = mid - 1;
                }
                s_item = lo;
            }
            __syncthreads();
            const int it = s_item;
            if (it != cur) {
                const int* src = reinterpret_cast<const int*>(q.items + it);
                int* dst = reinterpret_cast<int*>(&sp);
                for (int w = threadIdx.x; w < (int)(sizeof(DemodParams) / sizeof(int)); w += kThreads) dst[w] = src[w];
                cur = it;
                __syncthreads();
            }
            run_block<V>(sp, (int)(g - q.first_block[it]), c, parkX, parkZ);
        }
    }
}

}  // namespace

// The demodulator with the Stockham transforms (natural-order spectra).
__global__ void __launch_bounds__(kThreads, 1) demod_kernel(const __grid_constant__ DemodParams p) {
    extern __shared__ float2 smem[];
    demod_body<kVariantStockham>(p, smem);
}

// The demodulator with the in-place transforms (position-order spectra).
__global__ void __launch_bounds__(kThreads, 1) demod_ip_kernel(const __grid_constant__ DemodParams p) {
    extern __shared__ float2 smem[];
    demod_body<kVariantInPlace>(p, smem);
}

__global__ void __launch_bounds__(kThreads, 1) demod_queue_kernel(const __grid_constant__ QueueParams q) {
    extern __shared__ float2 smem[];
    queue_body<kVariantStockham>(q, smem);
}

__global__ void __launch_bounds__(kThreads, 1) demod_queue_ip_kernel(const __grid_constant__ QueueParams q) {
    extern __shared__ float2 smem[];
    queue_body<kVariantInPlace>(q, smem);
}

// ---- analog audio stage 2 (RFDecode.runfilter_audio_phase2, core.py:884-915)

namespace {

// raw[j] = x[j] - carrier (float32), zero where a left-channel spike is
// within 8 samples or beyond the segment (the transform's zero padding)
struct Audio2Loader {
    const float* x;
    float cf;
    int n;
    const unsigned* mask;
    __device__ float val(int j) const {
        if (j >= n || ((mask[j >> 5] >> (j & 31)) & 1u)) return 0.0f;
        return __ldg(x + j) - cf;
    }
    __device__ float2 operator()(int, int m) const { return make_float2(val(2 * m), val(2 * m + 1)); }
};

struct Audio2Storer {
    float* out;
    double cf;
    int n;
    __device__ void operator()(int, int m, float2 v) const {
        const int j = 2 * m;
        if (j < n) out[j] = (float)((double)(v.x * kInvM) + cf);
        if (j + 1 < n) out[j + 1] = (float)((double)(v.y * kInvM) + cf);
    }
};

// Input spectrum from Z (as post_r2c), times the filter, into the C2R input
// (no parking).
__device__ void audio2_filter(float2* S, const Tables& t, const float2* F) {
    for (int k = threadIdx.x; k <= kM / 2; k += kThreads) {
        if (k == 0) {
            const float2 z = S[0];
            c2r_dc(S, z.x + z.y, z.x - z.y, F);
            continue;
        }
        const float2 zk = S[pad(k)], zm = S[pad(kM - k)];
        const float2 e = make_float2(0.5f * (zk.x + zm.x), 0.5f * (zk.y - zm.y));
        const float2 o = make_float2(0.5f * (zk.y + zm.y), -0.5f * (zk.x - zm.x));
        const float2 wk = __ldg(t.t32 + k);
        const float2 tt = cmul(wk, o);
        const float2 xk = cadd(e, tt);
        const float2 xm = cconj(csub(e, tt));
        c2r_pair(S, k, cmul(xk, __ldg(F + k)), cmul(xm, __ldg(F + kM - k)), wk);
    }
}

}  // namespace

// One CTA per (segment, channel): the left channel's spikes (findpeaks,
// utils.py:1207-1216: samples above 500 kHz from the carrier rising above
// the segment's last value) mark +-8 samples that are zeroed in both
// channels; then R2C, the stage-2 filter, C2R, carrier added back.
__global__ void __launch_bounds__(kThreads, 1) audio2_kernel(const __grid_constant__ Audio2Params p) {
    extern __shared__ float2 smem[];
    const CtaSmem c = cta_setup<kVariantStockham>(smem, p.tw16, p.tw32);
    const Audio2Seg sg = p.segs[blockIdx.x];
    const int ch = blockIdx.y;
    const int n = sg.len;
    unsigned* mask = reinterpret_cast<unsigned*>(c.A);  // kN bits in the audio-band area
    for (int w = threadIdx.x; w < kN / 32; w += kThreads) mask[w] = 0u;
    __syncthreads();
    const float cfl = p.cf32[0];
    auto a2 = [&](int i) {
        const float v = __ldg(sg.left + i) - cfl;
        return v < 500000.0f ? 0.0f : v;
    };
    const float last = a2(n - 1);
    for (int i = threadIdx.x; i < n - 1; i += kThreads) {
        const float ai = a2(i);
        if (ai > last && a2(i + 1) > ai) {
            const int l = i - 1;
            const int lo = max(0, l - 8), hi = min(l + 8, n);
            for (int j = lo; j < hi; ++j) atomicOr(mask + (j >> 5), 1u << (j & 31));
        }
    }
    __syncthreads();
    const float* x = ch ? sg.right : sg.left;
    fft16k<false>(c.S, c.t, Audio2Loader{x, p.cf32[ch], n, mask});
    audio2_filter(c.S, c.t, p.filt[ch]);
    __syncthreads();
    fft16k<true>(c.S, c.t, SmemIO(), Audio2Storer{ch ? sg.out_right : sg.out_left, p.cf[ch], n});
}

// ---- demodblock's fftdata (RFDecode.demodblock_cpu, core.py:758-761)

// The real block ifft(X).real of a full N-bin spectrum (complex128), one CTA
// per block: its Hermitian part (X[k] + conj(X[N-k])) / 2 on the
// non-negative bins, the C2R pre-processing and one inverse 16384-point
// transform.
__global__ void __launch_bounds__(kThreads, 1) spectrum_block_kernel(const __grid_constant__ SpectrumParams p) {
    extern __shared__ float2 smem[];
    const CtaSmem c = cta_setup<kVariantStockham>(smem, p.tw16, p.tw32);
    const double2* X = p.spectra + (long long)blockIdx.x * kN;
    auto herm = [&](int k) {  // bins 0 < k < N/2
        const double2 a = X[k], b = X[kN - k];
        return make_float2((float)(0.5 * (a.x + b.x)), (float)(0.5 * (a.y - b.y)));
    };
    for (int k = threadIdx.x; k <= kM / 2; k += kThreads) {
        if (k == 0) {
            // bins 0 and N/2: their real parts (the imaginary parts leave ifft(X).real alone)
            const double h0 = X[0].x, hm = X[kM].x;
            c.S[0] = make_float2((float)(0.5 * (h0 + hm)), (float)(0.5 * (h0 - hm)));
            continue;
        }
        c2r_pair(c.S, k, herm(k), herm(kM - k), __ldg(c.t.t32 + k));
    }
    __syncthreads();
    fft16k<true>(c.S, c.t, SmemIO(), PairStorer{p.out + (long long)blockIdx.x * kN, 0, kN});
}

cudaError_t launch_spectrum_blocks(const SpectrumParams& p, int nblocks, cudaStream_t stream) {
    static SmemAttr attr;
    cudaError_t e = attr.ensure(spectrum_block_kernel, kSmemBytes);
    if (e != cudaSuccess) return e;
    if (nblocks <= 0) return cudaSuccess;
    spectrum_block_kernel<<<nblocks, kThreads, kSmemBytes, stream>>>(p);
    return cudaGetLastError();
}

cudaError_t launch_audio2(const Audio2Params& p, int nsegs, cudaStream_t stream) {
    static SmemAttr attr;
    cudaError_t e = attr.ensure(audio2_kernel, kSmemBytes);
    if (e != cudaSuccess) return e;
    if (nsegs <= 0) return cudaSuccess;
    audio2_kernel<<<dim3((unsigned)nsegs, 2), kThreads, kSmemBytes, stream>>>(p);
    return cudaGetLastError();
}

cudaError_t prepare_demod_queue() {
    static SmemAttr attr, attr_ip;
    cudaError_t e = attr.ensure(demod_queue_kernel, kSmemBytes);
    if (e != cudaSuccess) return e;
    return attr_ip.ensure(demod_queue_ip_kernel, kSmemBytesIp);
}

cudaError_t launch_demod_queue(const QueueParams& q, int grid, cudaStream_t stream) {
    cudaError_t e = prepare_demod_queue();
    if (e != cudaSuccess) return e;
    if (q.total <= 0 || grid <= 0) return cudaSuccess;
    if (q.variant == kVariantInPlace) {
        demod_queue_ip_kernel<<<grid, kThreads, kSmemBytesIp, stream>>>(q);
    } else {
        demod_queue_kernel<<<grid, kThreads, kSmemBytes, stream>>>(q);
    }
    return cudaGetLastError();
}

cudaError_t launch_demod(const DemodParams& p, int grid, cudaStream_t stream) {
    static SmemAttr attr, attr_ip;
    cudaError_t e = attr.ensure(demod_kernel, kSmemBytes);
    if (e != cudaSuccess) return e;
    e = attr_ip.ensure(demod_ip_kernel, kSmemBytesIp);
    if (e != cudaSuccess) return e;
    if (p.nblocks <= 0) return cudaSuccess;
    if (p.variant == kVariantInPlace) {
        if (!p.tw_pair || !p.g_pos || !p.godd_pos) return cudaErrorInvalidValue;
        demod_ip_kernel<<<grid, kThreads, kSmemBytesIp, stream>>>(p);
    } else {
        demod_kernel<<<grid, kThreads, kSmemBytes, stream>>>(p);
    }
    return cudaGetLastError();
}

}  // namespace ldg
