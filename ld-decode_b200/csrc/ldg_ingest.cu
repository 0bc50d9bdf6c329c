// .lds ingest: DomesdayDuplicator 10-bit packed samples (4 samples in 5
// bytes, most significant bits first) to the signed 16-bit samples the
// reference's loader returns (unpack_data_4_40, lddecode/utils.py:371-391):
// value v of a sample -> (v - 512) << 6.
//
// Each CTA stages a contiguous run of packed bytes in shared memory with
// 16-byte loads; each thread then takes eight samples, 80 bits, out of four
// words with funnel shifts and writes them as 16 bytes.  Any first sample
// works the same way: the ten bits of a sample are found by their bit
// position.  Bound: HBM, 1.25 bytes read and 2 written per sample: 60 M
// samples (195 MB) take 39 us on a B200 (41 with 256 threads); four samples
// per thread from five byte loads took 63.
#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

#include "ldg_noalloc.h"
#include "ldgpu.h"

namespace {

constexpr int kThreads = 128;
constexpr int kRounds = 4;
constexpr int kSamples = 8 * kThreads * kRounds;        // samples of a CTA
constexpr int kVecs = (kSamples / 4 * 5 + 16 + 8) / 16 + 1;  // 16-byte vectors that cover them from any bit on

__device__ __forceinline__ uint32_t big_endian(uint32_t v) { return __byte_perm(v, 0, 0x0123); }

// two samples whose ten bits are on top of `a` and `b`
__device__ __forceinline__ uint32_t two(uint32_t a, uint32_t b) {
    return (__byte_perm(a, b, 0x7632) & 0xFFC0FFC0u) ^ 0x80008000u;  // (v - 512) << 6
}

// CTA c writes out[8 i - skew .. + 7] for the threads' i, skew (0 or 4) the
// samples `out` lies past a 16-byte boundary; what lies outside [0, n) is
// neither read past the buffer nor written.
__global__ void __launch_bounds__(kThreads) lds_unpack_kernel(const uint8_t* __restrict__ packed, long long nbytes,
                                                              long long first, long long n, int skew,
                                                              int16_t* __restrict__ out) {
    __shared__ __align__(16) uint32_t words[4 * kVecs + 4];
    const long long o0 = (long long)blockIdx.x * kSamples - skew;
    const long long bit0 = 10 * (first + o0);
    const long long at0 = (bit0 >> 3) - (long long)((reinterpret_cast<uintptr_t>(packed) + (bit0 >> 3)) & 15);
    for (int v = threadIdx.x; v < kVecs; v += kThreads) {
        const long long at = at0 + 16LL * v;
        uint4 q;
        if (at >= 0 && at + 16 <= nbytes) {
            q = __ldcs(reinterpret_cast<const uint4*>(packed + at));
        } else {
            uint32_t w[4] = {0, 0, 0, 0};
            for (int j = 0; j < 16; ++j)
                if (at + j >= 0 && at + j < nbytes) w[j >> 2] |= (uint32_t)packed[at + j] << (8 * (j & 3));
            q = make_uint4(w[0], w[1], w[2], w[3]);
        }
        reinterpret_cast<uint4*>(words)[v] = q;
    }
    __syncthreads();
    const int lead = (int)(bit0 - 8 * at0);  // 0 .. 127
#pragma unroll
    for (int r = 0; r < kRounds; ++r) {
        const int i = r * kThreads + threadIdx.x;
        const long long o = o0 + 8 * i;
        if (o >= n) break;
        const int bit = lead + 80 * i, sh = bit & 31;
        const uint32_t* w = words + (bit >> 5);
        const uint32_t b0 = big_endian(w[0]), b1 = big_endian(w[1]), b2 = big_endian(w[2]), b3 = big_endian(w[3]);
        const uint32_t x0 = __funnelshift_l(b1, b0, sh), x1 = __funnelshift_l(b2, b1, sh), x2 = __funnelshift_l(b3, b2, sh);
        const uint4 s = make_uint4(two(x0, x0 << 10), two(x0 << 20, __funnelshift_l(x1, x0, 30)),
                                   two(x1 << 8, x1 << 18), two(__funnelshift_l(x2, x1, 28), x2 << 6));
        if (o >= 0 && o + 8 <= n) {
            __stcs(reinterpret_cast<uint4*>(out + o), s);
        } else {
            const uint32_t h[4] = {s.x, s.y, s.z, s.w};
            for (int j = 0; j < 8; ++j)
                if (o + j >= 0 && o + j < n) out[o + j] = (int16_t)(h[j >> 1] >> (16 * (j & 1)));
        }
    }
}

}  // namespace

extern "C" int ldg_unpack_lds(const uint8_t* packed, int64_t nbytes, int64_t first, int64_t n, int16_t* out,
                              void* stream) {
    using ldg::api_fail;
    if (!packed || !out) return api_fail(LDG_ERR_ARG, "ldg_unpack_lds: NULL buffer");
    if (first < 0 || n < 0 || nbytes < 0) return api_fail(LDG_ERR_ARG, "ldg_unpack_lds: negative size");
    if (n == 0) return LDG_OK;
    const long long last_group = (first + n - 1) / 4;
    if ((last_group + 1) * 5 > nbytes)
        return api_fail(LDG_ERR_RANGE, "ldg_unpack_lds: the packed buffer ends before the last sample");
    if ((reinterpret_cast<uintptr_t>(packed) & 3) != 0 || (reinterpret_cast<uintptr_t>(out) & 7) != 0)
        return api_fail(LDG_ERR_ARG, "ldg_unpack_lds: packed must be 4-byte and out 8-byte aligned");
    const int skew = (int)((reinterpret_cast<uintptr_t>(out) & 15) / sizeof(int16_t));
    const long long grid = (n + skew + kSamples - 1) / kSamples;
    if (grid > 0x7fffffffLL) return api_fail(LDG_ERR_ARG, "ldg_unpack_lds: too many samples");
    lds_unpack_kernel<<<(unsigned)grid, kThreads, 0, (cudaStream_t)stream>>>(packed, nbytes, first, n, skew, out);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return api_fail(LDG_ERR_CUDA, std::string("ldg_unpack_lds: ") + cudaGetErrorString(e));
    return LDG_OK;
}
