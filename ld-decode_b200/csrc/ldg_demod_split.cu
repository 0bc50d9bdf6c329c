// Small batches: one block on a cluster of C CTAs.
//
// A block is a chain of ten transforms on one SM (~117 us in place, ~128 us
// Stockham), so a batch with fewer blocks than SMs takes as long as one
// block however few it has.  Here the C CTAs of a cluster share a block: each
// transforms the input itself (cheaper than handing the spectrum round),
// then the transforms that depend only on it go to different CTAs --
//   C = 4: even analytic samples | odd ones, audio | rfhpf | EFM
//   C = 2: rfhpf, even analytic samples | audio, EFM, odd analytic samples
// -- the analytic signal meets in global scratch, every CTA discriminates its
// share of the samples, and after a second exchange each CTA transforms the
// demodulated signal and makes its share of the video outputs.  The same
// functions in the same order per value: outputs are bit-identical to the
// other kernels'.

#include <mutex>

#include "ldg_demod_block.cuh"

namespace ldg {

namespace {

// FM discriminator of samples 2 m, 2 m + 1 for m in [m0, m1): demod[2m] from
// (z_e[m], z_o[m-1]), demod[2m+1] from (z_o[m], z_e[m]), both in natural
// order; the clipped pairs go to clip.
template <class ZE, class ZO>
__device__ __forceinline__ void discriminate(const DemodParams& p, int blk, int m0, int m1, ZE ze, ZO zo,
                                             float2* clip) {
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
        clip[m] = make_float2(fminf(fmaxf(de, 1500000.0f), clip_hi), fminf(fmaxf(dodd, 1500000.0f), clip_hi));
    };
    // two samples per step, the parked (L2) loads first
#pragma unroll 2
    for (int m = m0 + threadIdx.x; m < m1; m += 2 * kThreads) {
        const int mb = m + kThreads;
        const float2 zea = ze(m), zeb = ze(mb);
        const float2 zoa = zo(m), zob = zo(mb);
        const float2 zpa = m ? zo(m - 1) : zoa, zpb = zo(mb - 1);
        const float dea = (m == 0) ? 0.0f : fm_disc(zea, zpa, kfs);
        const float doa = fm_disc(zoa, zea, kfs);
        const float deb = fm_disc(zeb, zpb, kfs);
        const float dob = fm_disc(zob, zeb, kfs);
        disc_store(m, dea, doa);
        disc_store(mb, deb, dob);
    }
}

// Between CTAs of a cluster: global writes before are seen after.
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Samples written by the cluster's other CTAs (read at L2).
struct SharedLoader {
    const float2* p;
    __device__ float2 operator()(int, int m) const { return __ldcg(p + m); }
};

template <int V, class LD>
__device__ __forceinline__ void forward_from(const CtaSmem& c, const LD& ld) {
    if constexpr (V == kVariantStockham) fft16k<false>(c.S, c.t, ld);
    else ip::fft16k_fwd(c.S, c.tw, ld);
}

template <int V, class T>
__device__ __forceinline__ void inverse_to(const CtaSmem& c, T* out, int off, int len) {
    if constexpr (V == kVariantStockham) inverse_out(c.S, c.t, out, off, len);
    else inverse_out(c.S, c.tw, out, off, len);
}

template <int V, int C>
__device__ __forceinline__ void demod_block_split(const DemodParams& p, int blk, int rank, const CtaSmem& c,
                                                  float2* base) {
    constexpr bool st = V == kVariantStockham;
    const bool hp = p.o_rfhpf && rank == (C == 4 ? 2 : 0);
    const bool efm = p.o_efm && rank == (C == 4 ? 3 : 1);
    const bool audio = p.audio && rank == 1;
    float2* parkX = base + (size_t)rank * kM;
    float2* ze = base + (size_t)C * kM;  // even samples of the analytic signal, odd ones, clipped demod
    float2* zo = ze + kM;
    float2* clip = zo + kM;

    if (p.in_kind == 0) {
        forward_from<V>(c, InLoader16{static_cast<const int16_t*>(p.in) + (long long)blk * p.in_stride});
    } else {
        forward_from<V>(c, InLoader32{static_cast<const float*>(p.in) + (long long)blk * p.in_stride});
    }
    if (audio) {
        for (int idx = threadIdx.x; idx < 2 * 511; idx += kThreads) {
            const int ch = idx / 511, k = 513 + idx % 511;
            c.A[ch * padded(1024) + pad(k)] = make_float2(0.f, 0.f);
        }
    }
    if constexpr (st) {
        AudioTaps au{c.A, {p.a_lowbin[0], p.a_lowbin[1]}, {p.a_filt1[0], p.a_filt1[1]}};
        post_r2c(c.S, c.t, parkX, hp ? p.f_rfhpf : nullptr, audio ? &au : nullptr);
        __syncthreads();
    } else {
        post_r2c_ip(c.S, p.tw_pair, parkX, hp ? p.fp_rfhpf : nullptr);
        __syncthreads();
        if (audio) {
            gather_audio_ip(p, c.A, parkX);
            __syncthreads();
        }
    }
    if (p.notch_hi > p.notch_lo) {
        if constexpr (st) notch_park(parkX, p.notch_lo, p.notch_hi);
        else notch_park_ip(parkX, p.notch_lo, p.notch_hi);
        __syncthreads();
    }
    if (audio) audio_stage(p, c.A, c.t, blk);
    if (hp) inverse_to<V>(c, p.o_rfhpf + (long long)blk * p.s_rfhpf.len, p.s_rfhpf.start, p.s_rfhpf.len);
    if (efm) {
        if constexpr (st) pre_c2r(c.S, c.t, parkX, p.f_efm, p.efm_klo, p.efm_khi);
        else pre_c2r_ip<true>(c.S, p.tw_pair, parkX, p.fp_efm, p.efm_klo, p.efm_khi);
        __syncthreads();
        inverse_to<V>(c, p.o_efm + (long long)blk * p.s_efm.len, p.s_efm.start, p.s_efm.len);
    }
    if (rank < 2) {
        const bool odd = rank == 1;
        if constexpr (st) {
            fft16k<true>(c.S, c.t, AnalyticLoader{parkX, p.f_g, p.f_godd, odd}, ParkStorer{odd ? zo : ze});
        } else {
            ip::fft16k_inv(c.S, c.tw, AnalyticLoaderIp{parkX, odd ? p.godd_pos : p.g_pos, p.f_g, odd},
                           ParkStorer{odd ? zo : ze});
        }
    }
    cluster_sync();
    discriminate(p, blk, rank * (kM / C), (rank + 1) * (kM / C), [&](int m) { return __ldcg(ze + m); },
                 [&](int m) { return __ldcg(zo + m); }, clip);
    cluster_sync();

    // this CTA's video outputs: every C-th of those asked for
    int mine = -1, nth = 0;
#pragma unroll
    for (int o = 0; o < OUT_NVIDEO; ++o)
        if (p.o_video[o] && nth++ % C == rank && mine < 0) mine = o;
    if (mine < 0) return;
    forward_from<V>(c, SharedLoader{clip});
    if constexpr (st) post_r2c(c.S, c.t, parkX, p.f_video[mine], nullptr);
    else post_r2c_ip(c.S, p.tw_pair, parkX, p.fp_video[mine]);
    __syncthreads();
    nth = 0;
#pragma unroll
    for (int o = 0; o < OUT_NVIDEO; ++o) {
        if (p.o_video[o] == nullptr || nth++ % C != rank) continue;
        if (o != mine) {
            if constexpr (st) pre_c2r(c.S, c.t, parkX, p.f_video[o]);
            else pre_c2r_ip<false>(c.S, p.tw_pair, parkX, p.fp_video[o]);
            __syncthreads();
        }
        inverse_to<V>(c, p.o_video[o] + (long long)blk * p.s_video.len, p.s_video.start + p.roll[o], p.s_video.len);
    }
}

}  // namespace

template <int V, int C>
__global__ void __cluster_dims__(C, 1, 1) __launch_bounds__(kThreads, 1)
    demod_split_kernel(const __grid_constant__ DemodParams p) {
    extern __shared__ float2 smem[];
    const CtaSmem c = cta_setup<V>(smem, p.tw16, p.tw32);
    const int blk = blockIdx.x / C, rank = blockIdx.x % C;
    demod_block_split<V, C>(p, blk, rank, c, p.scratch + (size_t)blk * (C + 3) * kM);
}

namespace {

template <int V, int C>
constexpr size_t split_smem() { return V == kVariantStockham ? kSmemBytes : kSmemBytesIp; }

template <int V, int C>
SmemAttr& split_attr() {
    static SmemAttr attr;
    return attr;
}

template <int V, int C>
cudaError_t launch_split(const DemodParams& p, cudaStream_t stream) {
    const cudaError_t e = split_attr<V, C>().ensure(demod_split_kernel<V, C>, split_smem<V, C>());
    if (e != cudaSuccess) return e;
    demod_split_kernel<V, C><<<p.nblocks * C, kThreads, split_smem<V, C>(), stream>>>(p);
    return cudaGetLastError();
}

// Clusters of C that the current device holds at once (0: none, or an error).
template <int V, int C>
int resident_clusters() {
    static std::mutex mu;
    static int known[SmemAttr::kMaxDevices] = {};  // + 1
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= SmemAttr::kMaxDevices) return 0;
    std::lock_guard<std::mutex> lk(mu);
    if (known[dev] == 0) {
        int n = 0;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(C);
        cfg.blockDim = dim3(kThreads);
        cfg.dynamicSmemBytes = split_smem<V, C>();
        cudaLaunchAttribute at = {};
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = C;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        if (split_attr<V, C>().ensure(demod_split_kernel<V, C>, split_smem<V, C>()) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&n, demod_split_kernel<V, C>, &cfg) != cudaSuccess) {
            cudaGetLastError();
            n = 0;
        }
        known[dev] = n + 1;
    }
    return known[dev] - 1;
}

size_t split_scratch(long long nblocks, int c) { return (size_t)nblocks * (c + 3) * kM * sizeof(float2); }

}  // namespace

// As many CTAs per block as still run all at once: PAL blocks (Stockham) take
// 55 us on four CTAs, 81 us on two and 130 us on one, NTSC (in place) 52, 78
// and 112 us, with any number of blocks up to the resident clusters (33 of
// four, 74 of two on a B200); a second wave of clusters of four takes 105 us,
// of two 158 us.
int demod_split(int variant, long long nblocks, size_t scratch_bytes) {
    const bool st = variant == kVariantStockham;
    const int r4 = st ? resident_clusters<kVariantStockham, 4>() : resident_clusters<kVariantInPlace, 4>();
    if (nblocks <= r4 && split_scratch(nblocks, 4) <= scratch_bytes) return 4;
    const int r2 = st ? resident_clusters<kVariantStockham, 2>() : resident_clusters<kVariantInPlace, 2>();
    return nblocks <= r2 && split_scratch(nblocks, 2) <= scratch_bytes ? 2 : 1;
}

cudaError_t launch_demod_split(const DemodParams& p, int c, cudaStream_t stream) {
    if (p.nblocks <= 0) return cudaSuccess;
    if (p.variant == kVariantInPlace) {
        if (!p.tw_pair || !p.g_pos || !p.godd_pos) return cudaErrorInvalidValue;
        return c == 4 ? launch_split<kVariantInPlace, 4>(p, stream) : launch_split<kVariantInPlace, 2>(p, stream);
    }
    return c == 4 ? launch_split<kVariantStockham, 4>(p, stream) : launch_split<kVariantStockham, 2>(p, stream);
}

}  // namespace ldg
