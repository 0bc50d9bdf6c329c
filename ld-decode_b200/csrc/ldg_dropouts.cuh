// Dropout detection kernel (Field.dropout_detect, lddecode/core.py:2829-2983).
#pragma once
#include <cuda_runtime.h>

namespace ldg {

constexpr int kDropStdTile = 4096;   // samples per CTA of the standard deviation
constexpr int kDropMaskTile = 8192;  // samples per CTA of the error mask
constexpr int kMaxDropRegions = 512;  // sync areas: lines 1 .. nlines-1, nlines <= 513

struct DropField {
    const float* demod;
    const float* d05;
    const float* raw;
    const float* rfhpf;
    long long len;
    const double* ll;
    int nlines, lineoffset, linecount, isfirst, hsync_len;
    long long tile0, word0;  // its first entries of DropScratch.part and .words
};

struct DropConsts {
    int system, video_rot, outlinelen, err_cap, out_cap;
    double freq_mhz, fhalf;
    float vmin, vmax, vmin05, vmax05, smin, smin05;  // float32 limits (Hz)
};

// Device scratch of a call, per field: tiles' rfhpf sums and squared
// deviations, sync areas (start, prefix maximum of the ends), a flag for areas
// that cannot be built, the error mask.  Tiles and mask words follow each
// field's own length (one long read among short ones costs its own).
struct DropScratch {
    double2* part;
    int2* areas;
    int* bad;
    float* rf_hi;       // the error limit of rfhpf (3 standard deviations)
    unsigned* words;
    unsigned* starts;   // the spans' first error samples
    int place_words;    // mask words the placement's shared memory holds
};

// Bytes of scratch for these fields, setting their tile0 and word0; with sc, its layout at base.
size_t dropout_scratch(DropField* fields, int nfields, char* base, DropScratch* sc);

// scratch: as dropout_scratch laid it out; max_len: the longest field's samples.
cudaError_t launch_dropouts(const DropField* fields, int nfields, long long max_len, const DropConsts& k,
                            DropScratch sc, int* drops, int* counts, double* rfstd, cudaStream_t stream);

}  // namespace ldg
