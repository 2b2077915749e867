// field_fft.h -- the FAST E/B field as a convolution over the LOD bins (field_fft.cu).
#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

namespace ion {

struct DevLbm;

// FftField::direct: a word per component, known before the sums, and the word that the last kernel sets
constexpr uint32_t FFT_LATE = 4;

// What one domain keeps for the convolution (device memory, laid out once per grid shape):
// the spectra of R/|R|^3 for every distinct offset of a cell inside its bin.
struct FftField {
    float2* G = nullptr;       // [uz][uy][ux][kx = 0..nd][component][kz][ky]
    float2* S = nullptr;       // [kx = 0..nd][q, q vx, q vy, q vz][kz][ky], of the present step
    float* out = nullptr;      // [6][oz of a chunk][oy][ox][Ix][Iz][Iy]: the sums, before they go to the cells
    uint32_t* direct = nullptr;  // [FFT_LATE + 1], one non-zero: the sources ask for the direct sum
    float* noise = nullptr;    // [4], from [1]: rounding of a concentrated current (0: it is spread out)
    uint32_t ux = 0, uy = 0, uz = 0;  // distinct offsets per axis: bin edge / 2 + 1
    uint32_t chunk = 0;        // in-bin z offsets whose sums fit in `out`
    float spread = 0.0f;       // how spread out the sources have to be (field_fft.cu, concentrated)
    float kappa = 0.0f;        // root of the mean of 1/|R|^4 on the padded lattice
};

// bytes of the sums that are held at once (a few in-bin z offsets of a large grid)
constexpr size_t FFT_OUT_BYTES = 48ull << 20;

// whether a domain's FAST field runs as the convolution, and its sizes in bytes
bool fft_field_fits(const DevLbm& L);
void fft_field_sizes(const DevLbm& L, FftField& F, size_t* g_bytes, size_t* s_bytes, size_t* out_bytes);
void fft_field_spread(const DevLbm& L, FftField& F);
cudaError_t launch_fft_plan(const DevLbm& L, const FftField& F, cudaStream_t s);
// sources -> spectra, sums of every cell, E/B; returns the number of launches.  F.direct is
// left with a non-zero word when the direct sum has to run instead, over all of E and B.  gate: null, or
// nothing runs while *gate is 0.
uint32_t launch_fft_field(const DevLbm& L, const FftField& F, const uint32_t* gate, cudaStream_t s);

// blocks of the three kernels; the sums of a large grid go in passes of F.chunk z offsets
uint32_t fft_passes(const DevLbm& L, const FftField& F);
uint32_t fft_src_blocks(const DevLbm& L);
uint32_t fft_sum_blocks(const DevLbm& L, const FftField& F, uint32_t pass);
uint32_t fft_put_blocks(const DevLbm& L, const FftField& F, uint32_t pass);

// many domains of one bin count at once: views on the device, prefix sums of the blocks
// per domain (of one pass)
struct FftBatch {
    const DevLbm* doms;
    const uint32_t* index;     // [n] an entry's domain
    const FftField* fields;    // [n]
    const uint32_t *src_off, *sum_off, *put_off;  // [n+1]
    uint32_t n, nd, src_blocks, sum_blocks, put_blocks;
};
uint32_t launch_fft_batch(const FftBatch* passes, uint32_t n, cudaStream_t s);

}  // namespace ion
