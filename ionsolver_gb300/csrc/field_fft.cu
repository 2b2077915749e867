// field_fft.cu -- the FAST E/B field of a whole domain as convolutions over the LOD bins.
//
// A cell c = I b + o (bin I, offset o inside the bin, bin edge b per axis) sums
// w_J R/|R|^3 over the bins J != I, R = b (I - J) + (o - b/2): for one offset o this
// is a convolution over the bin lattice with a kernel that depends on o and I - J only,
// zero at I = J (the own bin).  With the lattice padded to twice its edge (nd -> M = 2 nd)
// the convolution is a product of spectra, so the domain's field is, per offset, three
// transforms for E and three for B instead of 8^D terms per cell: at nd = 16 about 600
// operations per cell where the direct sum (field_kernels.cuh, eb_tile) takes 56,000.
// The sources are the direct sum's: bins [first_src, 8^D), (q, q v) with q v rounded first.
//
//   k_fft_plan  once per grid shape: spectra of R/|R|^3.  An offset o and its mirror image b - o have spectra
//               that differ by the sign of a wave number and of a component, so
//               (b/2 + 1) of b offsets per axis are kept.
//   k_fft_src   spectra of the sources, 4 (nd + 1) blocks; the four of kx = 0 also look at the
//               range and the spread of the sources (see below).
//   k_fft_sum   one block per offset and component of E or B: product of spectra, then the
//               inverse transforms along z, y and x in registers, passed on through
//               shared memory.
//   k_fft_put   the sums to the cells, x-rows at a time: E_stat + KE e, B_stat + KMU b.
//
// Rounding: the field's error against 64 bits is 1.6e-7 to 2.2e-7 of its norm from 8^3 to 256^3
// cells (the direct 32-bit sums: 2.6e-7 to 8.6e-7).  The transforms spread it evenly over the
// lattice, where the direct sum's is relative to a cell's own terms: with the charge in a few
// bins the weakest cells would be up to 1e-4 of their field off (one bin 1.3e-5, the direct sum
// 4.5e-7).  So k_fft_src compares the two (see `concentrated`), and where the convolution's error would
// be the larger one, `direct` is set and k_update_e_b_gated runs instead.  It also runs for
// sources that are infinite, where the convolution would leave NaN and the direct sum keeps the
// sign, or whose largest value lies outside [1e-28, 1e25], where sums could over- or underflow (a
// NaN charge leaves NaN in every cell either way).
#include <algorithm>
#include <cmath>

#include "field_fft.h"
#include "fft_regs.cuh"
#include "ion_device.cuh"
#include "ion_launch.h"

namespace ion {

namespace {

__host__ __device__ constexpr uint32_t slot_elems(uint32_t nd) { return nd * nd; }  // one kx plane, [z][y]
// kx planes transformed together: PL M = 64 lines, two lanes each
__host__ __device__ constexpr uint32_t planes(uint32_t nd) { return 32u / nd; }
__host__ __device__ constexpr uint32_t stage_elems(uint32_t nd) { return planes(nd) * nd * (2u * nd + 1u); }
// the staged planes overlay the slots that are not written yet
__host__ __device__ constexpr uint32_t sum_smem(uint32_t nd) { return ((nd - planes(nd)) * slot_elems(nd) + stage_elems(nd)) * 8u; }
static_assert(planes(16) * slot_elems(16) <= stage_elems(16) && planes(8) * slot_elems(8) <= stage_elems(8),
              "the last planes' slots lie inside the staging area");
constexpr uint32_t SUM_THREADS = 128, SRC_THREADS = 512, PUT_THREADS = 256, PUT_X = 128;
// k_fft_sum's blocks per SM: 96 registers at nd = 16 (with six it spills, 111 -> 148 us at 128^3),
// half the line at nd = 8
__host__ __device__ constexpr int sum_blocks(int nd) { return nd == 16 ? 5 : 8; }

#define ION_TW(j) {(float)cos32(j), (float)sin32(j)}
__constant__ float2 c_tw[32] = {  // exp(2 pi i j / 32)
    ION_TW(0),  ION_TW(1),  ION_TW(2),  ION_TW(3),  ION_TW(4),  ION_TW(5),  ION_TW(6),  ION_TW(7),
    ION_TW(8),  ION_TW(9),  ION_TW(10), ION_TW(11), ION_TW(12), ION_TW(13), ION_TW(14), ION_TW(15),
    ION_TW(16), ION_TW(17), ION_TW(18), ION_TW(19), ION_TW(20), ION_TW(21), ION_TW(22), ION_TW(23),
    ION_TW(24), ION_TW(25), ION_TW(26), ION_TW(27), ION_TW(28), ION_TW(29), ION_TW(30), ION_TW(31)};
#undef ION_TW

// ---------------------------------------------------------------------------
// spectra of R/|R|^3: one block per distinct offset and kx.  In 32 bits: |2 R|^2 is exact, and
// the transforms' error adds to that of the step's (together 2e-7 of the field's norm).  A
// 256^3 grid's plan takes 0.58 ms; in 64 bits, at 1/64 of the rate, it took 21 ms
// ---------------------------------------------------------------------------
template <int ND>
__global__ void __launch_bounds__(256) k_fft_plan(const DevLbm L, const FftField F) {
    constexpr int M = 2 * ND, ROW = M + 1;
    __shared__ C2 a[3 * M * ROW];  // [component][mz][my], rows of M + 1
    __shared__ C2 tw[M];
    const uint32_t kx = blockIdx.x % (ND + 1u), u = blockIdx.x / (ND + 1u);
    const uint32_t ox = u % F.ux, oy = (u / F.ux) % F.uy, oz = u / (F.ux * F.uy);
    if (threadIdx.x < M) {
        const float2 w = c_tw[((threadIdx.x * kx) % M) * (32 / M)];
        tw[threadIdx.x] = {w.x, -w.y};
    }
    __syncthreads();
    const float bx = L.bsx, by = L.bsy, bz = L.bsz;
    const float sx = ox - 0.5f * bx, sy = oy - 0.5f * by, sz = oz - 0.5f * bz;
    for (int t = threadIdx.x; t < M * M; t += blockDim.x) {
        const int my = t % M, mz = t / M;
        C2 g[3] = {{0.0f, 0.0f}, {0.0f, 0.0f}, {0.0f, 0.0f}};
        if (my != ND && mz != ND) {
            const float ry = by * (my < ND ? my : my - M) + sy, rz = bz * (mz < ND ? mz : mz - M) + sz;
            for (int mx = 0; mx < M; mx++) {
                if (mx == ND || (mx | my | mz) == 0) continue;  // outside the bin lattice, the own bin
                const float rx = bx * (mx < ND ? mx : mx - M) + sx;
                const float r2 = fmaf(rx, rx, fmaf(ry, ry, rz * rz));
                const float i3 = 1.0f / (r2 * sqrtf(r2));
                const C2 w = tw[mx];
                const float vx = rx * i3, vy = ry * i3, vz = rz * i3;
                g[0] = {fmaf(vx, w.x, g[0].x), fmaf(vx, w.y, g[0].y)};
                g[1] = {fmaf(vy, w.x, g[1].x), fmaf(vy, w.y, g[1].y)};
                g[2] = {fmaf(vz, w.x, g[2].x), fmaf(vz, w.y, g[2].y)};
            }
        }
        for (int c = 0; c < 3; c++) a[(c * M + mz) * ROW + my] = g[c];
    }
    __syncthreads();
    if (threadIdx.x < 3u * M) {  // along y, a row per thread
        C2* row = a + threadIdx.x * ROW;
        C2 v[M];
#pragma unroll
        for (int k = 0; k < M; k++) v[k] = row[k];
        fft_regs<M, -1>(v);
#pragma unroll
        for (int k = 0; k < M; k++) row[k] = v[k];
    }
    __syncthreads();
    if (threadIdx.x < 3u * M) {  // along z, a column per thread
        const int c = threadIdx.x / M, ky = threadIdx.x % M;
        C2 v[M];
#pragma unroll
        for (int k = 0; k < M; k++) v[k] = a[(c * M + k) * ROW + ky];
        fft_regs<M, -1>(v);
        float2* out = F.G + ((((size_t)u * (ND + 1u) + kx) * 3u + c) * M) * M + ky;
#pragma unroll
        for (int k = 0; k < M; k++) out[k * M] = make_float2(v[k].x, v[k].y);
    }
}

// ---------------------------------------------------------------------------
// spectra of the sources: block = component + 4 kx
// ---------------------------------------------------------------------------

// Whether a component w_J of the sources (s, scaled by a power of two to below 1) is too
// concentrated for the convolution.  Its error is about the same in every cell, of the size
// |w| kappa: |w|^2 = sum w_J^2, kappa^2 = the mean of 1/|R|^4 over the padded lattice.  The direct
// sum's is relative to the cell's own sum of |w_J|/|R|^2, least far from the sources: estimated over
// 4^3 groups of bins, each at the distance of its centre and half a group an axis (within 15% of
// the cells' least sum on boxes of even edges).  Both errors against 64 bits, per cell relative
// to that sum, root mean square, 2,800 distributions in 22 box shapes: with the least sum above
// 4 |w| kappa at nd = 16 and 2.75 |w| kappa at nd = 8 the convolution's is at most 0.88 and 1.08 of the
// direct sum's; at half the line of nd = 16 it reaches 2.  Charges and currents spread over the box, as in
// all the configurations, lie at 5 to 10 and at 3 to 5 (one charged bin: 0.1).  Bins twice as
// long as wide lie lower, eight times as long below the line.  F.spread holds the square of the
// line times kappa.  (All of it in fixed order: a batch decides as its domains do alone.)
template <int ND>
__device__ __forceinline__ bool concentrated(const DevLbm& L, const FftField& F, const float* s, const float scale, float& norm) {
    constexpr uint32_t G = ND / 4;  // bins a group and axis
    __shared__ float s_sum[64], s_sq[64], s_inv[64];
    __shared__ uint32_t s_min;
    const uint32_t g = threadIdx.x / 8u, sub = threadIdx.x % 8u;  // eight lanes a group
    static_assert(SRC_THREADS == 512u, "64 groups of eight lanes");
    float sum = 0.0f, sq = 0.0f;
#pragma unroll
    for (uint32_t k = sub; k < G * G * G; k += 8u) {
        const uint32_t x = g % 4u * G + k % G, y = g / 4u % 4u * G + k / G % G, z = g / 16u * G + k / (G * G);
        const float v = fabsf(s[(z * ND + y) * (ND + 1) + x]) * scale;
        sum = sum + v;
        sq = fmaf(v, v, sq);
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
        sum = sum + __shfl_xor_sync(0xFFFFFFFFu, sum, o);
        sq = sq + __shfl_xor_sync(0xFFFFFFFFu, sq, o);
    }
    if (sub == 0u) { s_sum[g] = sum; s_sq[g] = sq; }
    if (threadIdx.x < 64u) {  // 1/|R|^2 of groups (x, y, z) apart
        const float rx = ((threadIdx.x % 4u) + 0.5f) * (float)(G * L.bsx), ry = ((threadIdx.x / 4u % 4u) + 0.5f) * (float)(G * L.bsy),
                    rz = ((threadIdx.x / 16u) + 0.5f) * (float)(G * L.bsz);
        s_inv[threadIdx.x] = 1.0f / fmaf(rx, rx, fmaf(ry, ry, rz * rz));
    }
    if (threadIdx.x == 0u) s_min = 0x7F800000u;
    __syncthreads();
    float a = 0.0f, q = 0.0f;
#pragma unroll
    for (uint32_t j = sub; j < 64u; j += 8u) {
        const uint32_t dx = abs((int)(j % 4u) - (int)(g % 4u)), dy = abs((int)(j / 4u % 4u) - (int)(g / 4u % 4u)),
                       dz = abs((int)(j / 16u) - (int)(g / 16u));
        a = fmaf(s_sum[j], s_inv[dx + 4u * dy + 16u * dz], a);
        q = q + s_sq[j];
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
        a = a + __shfl_xor_sync(0xFFFFFFFFu, a, o);
        q = q + __shfl_xor_sync(0xFFFFFFFFu, q, o);
    }
    if (sub == 0u) atomicMin(&s_min, __float_as_uint(a));  // (in any order; a >= 0)
    __syncthreads();
    const float least = __uint_as_float(s_min);
    norm = sqrtf(q);
    return least * least < F.spread * q;
}

template <int ND>
__device__ __forceinline__ void fft_src(const DevLbm& L, const FftField& F, const uint32_t block) {
    constexpr uint32_t M = 2u * ND, NB = ND * ND * ND;
    __shared__ float s[ND * ND * (ND + 1)];  // [z][y][x], rows of ND + 1
    __shared__ float2 a[ND][ND], b[ND][M], tw[M];
    __shared__ uint32_t s_max[2];
    const uint32_t c = block % 4u, kx = block / 4u;
    const uint32_t first = L.first_src, last = min(L.n_lod_own, L.n_bins);
    if (threadIdx.x < 2u) s_max[threadIdx.x] = 0u;
    if (threadIdx.x < M) tw[threadIdx.x] = c_tw[threadIdx.x * (32u / M)];  // the lanes index it apart
    __syncthreads();
    uint32_t m[2] = {0u, 0u};  // the largest charge and value of the component: NaN > Inf > finite
#pragma unroll
    for (uint32_t d = threadIdx.x; d < NB; d += SRC_THREADS) {
        const float4 v = d >= first && d < last ? reinterpret_cast<const float4*>(L.qu_lod)[d] : make_float4(0.f, 0.f, 0.f, 0.f);
        const float w = c == 0u ? v.x : c == 1u ? v.x * v.y : c == 2u ? v.x * v.z : v.x * v.w;
        s[d / ND * (ND + 1) + d % ND] = w;
        m[0] = max(m[0], __float_as_uint(v.x) & 0x7FFFFFFFu);
        m[1] = max(m[1], __float_as_uint(w) & 0x7FFFFFFFu);
    }
    if (kx == 0u) {
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const uint32_t v = __reduce_max_sync(0xFFFFFFFFu, m[k]);
            if ((threadIdx.x & 31u) == 0u) atomicMax(&s_max[k], v);
        }
    }
    __syncthreads();
    if (kx == 0u) {  // the component's block decides for it
        const uint32_t v = s_max[1];
        const float scale = __uint_as_float(0x7E800000u - (v & 0x7F800000u));
        bool bad = false, few = false;
        float norm = 0.0f;
        if (s_max[0] <= 0x7F800000u && v != 0u) {  // a NaN charge makes every cell's E and B NaN either way
            bad = !(v >= __float_as_uint(1e-28f) && v <= __float_as_uint(1e25f));
            if (!bad) few = concentrated<ND>(L, F, s, scale, norm);
        }
        if (threadIdx.x == 0u) {
            F.direct[c] = bad || (few && c == 0u);
            if (c == 0u) F.direct[FFT_LATE] = 0u;
            else F.noise[c] = few ? F.kappa * (norm / scale) : 0.0f;
        }
    }
    // along x at this kx
    for (uint32_t t = threadIdx.x; t < ND * ND; t += SRC_THREADS) {
        float2 acc = make_float2(0.0f, 0.0f);
#pragma unroll
        for (uint32_t x = 0; x < ND; x++) {
            const float v = s[t * (ND + 1) + x];
            const float2 w = tw[(kx * x) % M];
            acc.x = fmaf(v, w.x, acc.x);
            acc.y = fmaf(-v, w.y, acc.y);
        }
        a[t / ND][t % ND] = acc;
    }
    __syncthreads();
    // along y, then along z
    for (uint32_t t = threadIdx.x; t < ND * M; t += SRC_THREADS) {
        const uint32_t ky = t % M, z = t / M;
        float2 acc = make_float2(0.0f, 0.0f);
#pragma unroll
        for (uint32_t y = 0; y < ND; y++) {
            const float2 v = a[z][y], w = tw[(ky * y) % M];
            acc.x = fmaf(v.x, w.x, fmaf(v.y, w.y, acc.x));
            acc.y = fmaf(v.y, w.x, fmaf(-v.x, w.y, acc.y));
        }
        b[z][ky] = acc;
    }
    __syncthreads();
    float2* out = F.S + (size_t)(kx * 4u + c) * M * M;
    for (uint32_t t = threadIdx.x; t < M * M; t += SRC_THREADS) {
        const uint32_t ky = t % M, kz = t / M;
        float2 acc = make_float2(0.0f, 0.0f);
#pragma unroll
        for (uint32_t z = 0; z < ND; z++) {
            const float2 v = b[z][ky], w = tw[(kz * z) % M];
            acc.x = fmaf(v.x, w.x, fmaf(v.y, w.y, acc.x));
            acc.y = fmaf(v.y, w.x, fmaf(-v.x, w.y, acc.y));
        }
        out[t] = acc;
    }
}

// ---------------------------------------------------------------------------
// the sums of one offset: block = (((oz - oz0) bsy + oy) bsx + ox) 6 + (0..2: E, 3..5: B)
// ---------------------------------------------------------------------------
__device__ __forceinline__ C2 cmul(const float2 a, const float2 b) {
    return {fmaf(a.x, b.x, -(a.y * b.y)), fmaf(a.x, b.y, a.y * b.x)};
}
__device__ __forceinline__ C2 cmul_sub(const C2 s, const float2 a, const float2 b) {
    return {fmaf(-a.x, b.x, fmaf(a.y, b.y, s.x)), fmaf(-a.x, b.y, fmaf(-a.y, b.x, s.y))};
}

// Lines of M points are transformed by two lanes, 16 apart, as the N-point transforms of their
// even and odd points (N = nd).  Of the first N outputs the lower lane gets the first half, the
// upper lane the second; the upper lane's transform comes half a turn on, so that both keep
// the lower half of their registers and pass on the upper half.  The turn w^n comes after the
// exchange, fused into the additions of half as many points (k_fft_sum at 128^3 121 -> 111 us
// against turning the upper lane's points before it, which leaves the lower lane waiting).
template <int N>
__device__ __forceinline__ void fft_pair(C2 (&v)[N], const bool upper) {
    fft_regs<N, 1, true>(v, upper ? -1.0f : 1.0f);
#pragma unroll
    for (int n = 0; n < N / 2; n++) {  // even + w^n odd; w^(N/2) = i
        const C2 own = v[n], got = {__shfl_xor_sync(0xFFFFFFFFu, v[n + N / 2].x, 16),
                                           __shfl_xor_sync(0xFFFFFFFFu, v[n + N / 2].y, 16)};
        const C2 even = {upper ? got.x : own.x, upper ? got.y : own.y};
        const C2 odd = {upper ? -own.y : got.x, upper ? own.x : got.y};
        v[n] = add_twist<1>(even, odd, n * (16 / N));
    }
}

template <int ND>
__device__ __forceinline__ void fft_sum(const DevLbm& L, const FftField& F, const uint32_t block, const uint32_t oz0,
                                        float2* sm) {
    constexpr uint32_t M = 2u * ND, PL = planes(ND), SLOT = slot_elems(ND), ROW = M + 1u;
    const uint32_t field = block % 6u, o = block / 6u, f = field % 3u;
    const uint32_t ox = o % L.bsx, oy = (o / L.bsx) % L.bsy, oz = oz0 + o / (L.bsx * L.bsy);
    // the offset's spectra, or its mirror image's: R_a changes sign with the wave number k_a
    const bool fx = ox >= F.ux, fy = oy >= F.uy, fz = oz >= F.uz;
    const uint32_t u = (fx ? L.bsx - ox : ox) + ((fy ? L.bsy - oy : oy) + (fz ? L.bsz - oz : oz) * F.uy) * F.ux;
    auto negative = [&](uint32_t c) { return c == 0u ? fx : c == 1u ? fy : fz; };
    // component of the product: E_f = G_f q; B_f = (q v)_i G_j - (q v)_j G_i, (f, i, j) cyclic
    const uint32_t i = f == 2u ? 0u : f + 1u, j = f == 0u ? 2u : f - 1u;
    // G(-kx, ky, kz) = conj G(kx, -ky, -kz): kx stays in 0..nd
    const bool ry = fx != fy, rz = fx != fz;
    const uint32_t t = threadIdx.x, par = (t >> 4) & 1u;  // even or odd points of the line
    const uint32_t id = (t >> 5) * 16u + (t & 15u);       // line along z: (plane, ky)
    const uint32_t ky = id % M, pl = id / M, gy = ry ? (M - ky) % M : ky;
    const uint32_t conj = fx ? 0x80000000u : 0u, differ = negative(i) != negative(j) ? 0x80000000u : 0u;
    const float2* const G = F.G + (size_t)u * (ND + 1u) * 3u * M * M + gy;
    const float2* const S = F.S + par * M + ky;
    auto flip = [](float v, uint32_t m) { return __uint_as_float(__float_as_uint(v) ^ m); };
    auto gather = [&](uint32_t kx, C2(&v)[ND], auto&& put) {
        const float2* g = G + (size_t)kx * 3u * M * M;
        const float2* s = S + (size_t)kx * 4u * M * M;
        // kz = 2 k + par, or M - kz; the row's address is formed at each load (an opaque step:
        // kept in registers from plane to plane the addresses spill)
        const int start = (int)(rz ? M * M - par * M : par * M);
        int step = rz ? -(int)(2u * M) : (int)(2u * M);
        asm volatile("" : "+r"(step));
        if (field < 3u) {
#pragma unroll
            for (uint32_t k = 0; k < (uint32_t)ND; k++) {
                const int gz = k == 0u ? start & (int)(M * M - 1u) : start + (int)k * step;
                float2 a = __ldg(g + f * M * M + gz);
                a.y = flip(a.y, conj);
                put(v[k], cmul(a, __ldg(s + 2u * k * M)));
            }
        } else {
#pragma unroll
            for (uint32_t k = 0; k < (uint32_t)ND; k++) {
                const int gz = k == 0u ? start & (int)(M * M - 1u) : start + (int)k * step;
                float2 a = __ldg(g + j * M * M + gz), b = __ldg(g + i * M * M + gz);
                a.y = flip(a.y, conj);
                b.x = flip(b.x, differ);
                b.y = flip(b.y, conj ^ differ);
                put(v[k], cmul_sub(cmul(__ldg(s + (1u + i) * M * M + 2u * k * M), a),
                                   __ldg(s + (1u + j) * M * M + 2u * k * M), b));
            }
        }
    };
#pragma unroll 1
    for (uint32_t p0 = 0; p0 < (uint32_t)ND; p0 += PL) {
        float2* stage = sm + p0 * SLOT;  // [plane][z][ky], rows of M + 1
        C2 v[ND];
        gather(p0 + pl, v, [](C2& d, const C2 p) { d = p; });
        // the transforms of kx = 0 and kx = nd are real: one complex line holds both
        if (p0 + pl == 0u) gather(ND, v, [](C2& d, const C2 p) { d = {d.x - p.y, d.y + p.x}; });
        fft_pair<ND>(v, par != 0u);
        float2* w = stage + (pl * ND + par * (ND / 2u)) * ROW + ky;
#pragma unroll
        for (uint32_t n = 0; n < (uint32_t)ND / 2u; n++) w[n * ROW] = make_float2(v[n].x, v[n].y);
        __syncthreads();
        const bool on = id < PL * ND;  // line along y: (plane, z)
        if (on) {
            const float2* r = stage + id * ROW + par;
#pragma unroll
            for (uint32_t k = 0; k < (uint32_t)ND; k++) v[k] = {r[2u * k].x, r[2u * k].y};
            fft_pair<ND>(v, par != 0u);
        }
        __syncthreads();  // the staged lines are read: the slots below them may be written
        if (on) {
            // slot [z][(y + z) mod nd]: rows of nd without bank conflicts
            const uint32_t z = id % ND;
            float2* q = sm + (p0 + id / ND) * SLOT + z * ND;
#pragma unroll
            for (uint32_t n = 0; n < (uint32_t)ND / 2u; n++)
                q[(n + par * (ND / 2u) + z) % ND] = make_float2(v[n].x, v[n].y);
        }
    }
    __syncthreads();
    // along x, real outputs: with X_k the line's transform and h = nd, z_k = (X_k + conj X_{h-k})
    // + i w^k (X_k - conj X_{h-k}) transforms to (x_0 + i x_1, x_2 + i x_3, ...)
    for (uint32_t line = t; line < SLOT; line += SUM_THREADS) {
        const uint32_t y = line % ND, z = line / ND;
        const float2* r = sm + z * ND + (y + z) % ND;
        C2 v[ND];
        v[0] = {r[0].x + r[0].y, r[0].x - r[0].y};
#pragma unroll
        for (uint32_t k = 1; k <= (uint32_t)ND / 2u; k++) {
            const float2 p = r[k * SLOT], q = r[(ND - k) * SLOT];
            const C2 sum = {p.x + q.x, p.y - q.y}, dif = {p.x - q.x, p.y + q.y};
            const C2 a = twist<1>(dif, k * (16 / ND) + 8);  // i w^k dif
            v[k] = {sum.x + a.x, sum.y + a.y};
            // k -> h - k: sum -> conj sum, dif -> -conj dif, i w^k -> conj (i w^k)
            if (2u * k < (uint32_t)ND) v[ND - k] = {sum.x - a.x, a.y - sum.y};
        }
        fft_regs<ND, 1>(v);
        constexpr float scale = 1.0f / (float)(M * M * M);  // a power of two: exact
        const float w = negative(field < 3u ? f : j) ? -scale : scale;
        float* out = F.out + (((size_t)field * F.chunk * L.bsy * L.bsx + o) * ND * ND + z) * ND + y;
#pragma unroll
        for (uint32_t n = 0; n < (uint32_t)ND / 2u; n++) {
            out[(2u * n) * ND * ND] = v[n].x * w;
            out[(2u * n + 1u) * ND * ND] = v[n].y * w;
        }
    }
}

// ---------------------------------------------------------------------------
// the sums to the cells: block = (0: E, 1: B) + 2 (tile + tiles (Iz + nd (oz - oz0))); a block
// transposes PUT_X neighbouring (oy, x) of nd rows each (y = Iy bsy + oy), three components,
// through shared memory.  A thread's loads are all in flight before the first is used, and the
// components share its indices (one component a block, loads one after another: 55 us at
// 128^3; tiles of one oy leave lanes idle on rows below PUT_X cells)
// ---------------------------------------------------------------------------
template <int ND>
__device__ __forceinline__ void fft_put(const DevLbm& L, const FftField& F, uint32_t block, const uint32_t oz0) {
    __shared__ float s[3][ND][PUT_X + 1];
    const uint32_t plane_xy = L.bsy * L.nx, tiles = (plane_xy + PUT_X - 1u) / PUT_X;
    const bool B = block & 1u;
    block >>= 1;
    const uint32_t e0 = block % tiles * PUT_X;
    block /= tiles;
    const uint32_t Iz = block % ND, ozl = block / ND;
    const size_t N = L.n, plane = (size_t)F.chunk * L.bsy * L.bsx * (ND * ND * ND);
    const float* in = F.out + (B ? 3u : 0u) * plane + (size_t)ozl * L.bsy * L.bsx * (ND * ND * ND) + Iz * ND;
    const uint32_t Iy = threadIdx.x % ND;
    constexpr uint32_t XS = PUT_THREADS / ND, GET = PUT_X / XS;  // cells apart, cells per thread
    float v[3][GET];
#pragma unroll
    for (uint32_t k = 0; k < GET; k++) {
        const uint32_t e = e0 + threadIdx.x / ND + k * XS;
        const uint32_t oy = L.dx.div(e), x = e - oy * L.nx, Ix = x / L.bsx, ox = x - Ix * L.bsx;
        const float* p = in + (size_t)((oy * L.bsx + ox) * ND + Ix) * (ND * ND) + Iy;
#pragma unroll
        for (uint32_t c = 0; c < 3; c++) v[c][k] = e < plane_xy ? __ldcs(p + c * plane) : 0.0f;
    }
    const uint32_t z = Iz * L.bsz + oz0 + ozl;
    constexpr uint32_t PUT = PUT_X * ND / PUT_THREADS, YS = PUT_THREADS / PUT_X;
    const uint32_t xl = threadIdx.x % PUT_X, y0 = threadIdx.x / PUT_X, e = e0 + xl;
    const uint32_t oy = L.dx.div(e), x = e - oy * L.nx;
    const uint32_t n0 = x + (oy + y0 * L.bsy + z * L.ny) * L.nx, row = YS * L.bsy * L.nx;
    const float* const stat = B ? L.b_stat : L.e_stat;
    float* const dyn = B ? L.b_dyn : L.e_dyn;
    const float scale = B ? L.kmu : L.ke;
    const float noise = B ? F.noise[1] + F.noise[2] + F.noise[3] : 0.0f;
    const float least = 256.0f * fabsf(L.kmu) * noise;
    uint32_t small = noise > 0.0f ? (1u << PUT) - 1u : 0u;  // bit k: cell k's B is not above that so far
    bool on[PUT];
#pragma unroll
    for (uint32_t k = 0; k < PUT; k++) on[k] = e < plane_xy && (L.flags[n0 + k * row] & F_BO) != F_S;
#pragma unroll
    for (uint32_t c = 0; c < 3; c++)
#pragma unroll
        for (uint32_t k = 0; k < GET; k++) s[c][Iy][threadIdx.x / ND + k * XS] = v[c][k];
    __syncthreads();
#pragma unroll
    for (uint32_t c = 0; c < 3; c++) {
        float st[PUT];
#pragma unroll
        for (uint32_t k = 0; k < PUT; k++) st[k] = on[k] ? stat[c * N + n0 + k * row] : 0.0f;
#pragma unroll
        for (uint32_t k = 0; k < PUT; k++)
            if (on[k]) {
                const float r = st[k] + scale * s[c][y0 + k * YS][xl];
                dyn[c * N + n0 + k * row] = r;
                if (fabsf(r) > least) small &= ~(1u << k);
            } else {
                small &= ~(1u << k);
            }
    }
    if (small) atomicOr(F.direct + FFT_LATE, 1u);
}

// gate: null, or the kernels run only when *gate != 0.  Then resident blocks walk the work, so
// that a closed gate costs little; without a gate the grid has a block for each.
template <int ND>
__global__ void __launch_bounds__(SRC_THREADS) k_fft_src(const DevLbm L, const FftField F, const uint32_t* gate) {
    if (gate && *gate == 0u) return;
    fft_src<ND>(L, F, blockIdx.x);
}
template <int ND>
__global__ void __launch_bounds__(SUM_THREADS, sum_blocks(ND)) k_fft_sum(const DevLbm L, const FftField F, const uint32_t oz0,
                                                                     const uint32_t* gate, const uint32_t blocks) {
    extern __shared__ __align__(16) float2 sum_sm[];
    if ((gate && *gate == 0u) || any_of(F.direct)) return;
    for (uint32_t b = blockIdx.x; b < blocks; b += gridDim.x) {
        fft_sum<ND>(L, F, b, oz0, sum_sm);
        if (gate) __syncthreads();
    }
}
template <int ND>
__global__ void __launch_bounds__(PUT_THREADS) k_fft_put(const DevLbm L, const FftField F, const uint32_t oz0,
                                                         const uint32_t* gate, const uint32_t blocks) {
    if ((gate && *gate == 0u) || any_of(F.direct)) return;
    for (uint32_t b = blockIdx.x; b < blocks; b += gridDim.x) {
        fft_put<ND>(L, F, b, oz0);
        if (gate) __syncthreads();
    }
}

// the same blocks over many domains (FftBatch): a block's domain by its prefix sums
__device__ __forceinline__ uint32_t batch_entry(const FftBatch& B, const uint32_t* off, DevLbm& sL, FftField& sF,
                                                uint32_t& s_e) {
    if (threadIdx.x == 0) {
        uint32_t lo = 0, hi = B.n;  // off[lo] <= block < off[hi]
        while (hi - lo > 1u) {
            const uint32_t mid = (lo + hi) >> 1;
            if (off[mid] <= blockIdx.x) lo = mid;
            else hi = mid;
        }
        s_e = lo;
    }
    __syncthreads();
    const uint32_t e = s_e;
    static_assert(sizeof(DevLbm) % 4 == 0 && sizeof(FftField) % 4 == 0, "copied in words");
    const uint32_t* l = reinterpret_cast<const uint32_t*>(B.doms + B.index[e]);
    const uint32_t* f = reinterpret_cast<const uint32_t*>(B.fields + e);
    for (uint32_t i = threadIdx.x; i < sizeof(DevLbm) / 4; i += blockDim.x) reinterpret_cast<uint32_t*>(&sL)[i] = l[i];
    for (uint32_t i = threadIdx.x; i < sizeof(FftField) / 4; i += blockDim.x) reinterpret_cast<uint32_t*>(&sF)[i] = f[i];
    __syncthreads();
    return blockIdx.x - off[e];
}
template <int ND>
__global__ void __launch_bounds__(SRC_THREADS) k_fft_src_batch(const FftBatch B) {
    __shared__ DevLbm L;
    __shared__ FftField F;
    __shared__ uint32_t e;
    const uint32_t block = batch_entry(B, B.src_off, L, F, e);
    fft_src<ND>(L, F, block);
}
template <int ND>
__global__ void __launch_bounds__(SUM_THREADS, sum_blocks(ND)) k_fft_sum_batch(const FftBatch B, const uint32_t pass) {
    extern __shared__ __align__(16) float2 sum_sm[];
    __shared__ DevLbm L;
    __shared__ FftField F;
    __shared__ uint32_t e;
    const uint32_t block = batch_entry(B, B.sum_off, L, F, e);
    if (any_of(F.direct)) return;
    fft_sum<ND>(L, F, block, pass * F.chunk, sum_sm);
}
template <int ND>
__global__ void __launch_bounds__(PUT_THREADS) k_fft_put_batch(const FftBatch B, const uint32_t pass) {
    __shared__ DevLbm L;
    __shared__ FftField F;
    __shared__ uint32_t e;
    const uint32_t block = batch_entry(B, B.put_off, L, F, e);
    if (any_of(F.direct)) return;
    fft_put<ND>(L, F, block, pass * F.chunk);
}

template <int ND>
cudaError_t prepare_kernels() {
    cudaError_t e = cudaFuncSetAttribute(k_fft_sum<ND>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sum_smem(ND));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_fft_sum_batch<ND>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sum_smem(ND));
    return e;
}

uint32_t chunk_len(const DevLbm& L, const FftField& F, uint32_t pass) {
    const uint32_t oz = pass * F.chunk;
    return oz >= L.bsz ? 0u : F.chunk < L.bsz - oz ? F.chunk : L.bsz - oz;
}

template <int ND>
uint32_t launch_field_nd(const DevLbm& L, const FftField& F, const uint32_t* gate, cudaStream_t s) {
    uint32_t resident = 0xFFFFFFFFu;
    if (gate) {
        int dev = 0, sms = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        resident = (uint32_t)sum_blocks(ND) * (uint32_t)(sms > 0 ? sms : 1);
    }
    k_fft_src<ND><<<fft_src_blocks(L), SRC_THREADS, 0, s>>>(L, F, gate);
    for (uint32_t p = 0; p < fft_passes(L, F); p++) {
        const uint32_t sum = fft_sum_blocks(L, F, p), put = fft_put_blocks(L, F, p), oz = p * F.chunk;
        k_fft_sum<ND><<<sum < resident ? sum : resident, SUM_THREADS, sum_smem(ND), s>>>(L, F, oz, gate, sum);
        k_fft_put<ND><<<put < resident ? put : resident, PUT_THREADS, 0, s>>>(L, F, oz, gate, put);
    }
    return 1u + 2u * fft_passes(L, F);
}

template <int ND>
uint32_t launch_batch_nd(const FftBatch* B, uint32_t passes, cudaStream_t s) {
    k_fft_src_batch<ND><<<B->src_blocks, SRC_THREADS, 0, s>>>(*B);
    for (uint32_t p = 0; p < passes; p++) {
        k_fft_sum_batch<ND><<<B[p].sum_blocks, SUM_THREADS, sum_smem(ND), s>>>(B[p], p);
        k_fft_put_batch<ND><<<B[p].put_blocks, PUT_THREADS, 0, s>>>(B[p], p);
    }
    return 1u + 2u * passes;
}

}  // namespace

// Depths 3 and 4 (at depth 2 the direct sum has 64 terms, of which the near box are most),
// without cells of the reference's near field.  Grid sizes beyond 2^16 cells an edge keep the direct sum:
// its coordinates and block counts stay in 32 bits here.
bool fft_field_fits(const DevLbm& L) {
    return (L.nd == 8u || L.nd == 16u) && L.near_x == 1u && L.near_y == 1u && L.near_z == 1u && L.nx <= 65536u &&
           L.ny <= 65536u && L.nz <= 65536u;
}

void fft_field_sizes(const DevLbm& L, FftField& F, size_t* g_bytes, size_t* s_bytes, size_t* out_bytes) {
    F.ux = L.bsx / 2u + 1u;
    F.uy = L.bsy / 2u + 1u;
    F.uz = L.bsz / 2u + 1u;
    if (F.ux > L.bsx) F.ux = L.bsx;  // an edge of one cell has the offset 0 only
    if (F.uy > L.bsy) F.uy = L.bsy;
    if (F.uz > L.bsz) F.uz = L.bsz;
    const size_t M = 2u * L.nd, plane = M * M * sizeof(float2);
    *g_bytes = (size_t)F.ux * F.uy * F.uz * (L.nd + 1u) * 3u * plane;
    *s_bytes = (L.nd + 1u) * 4u * plane;
    const size_t per = 6u * sizeof(float) * (size_t)(L.n / L.bsz);  // one in-bin z offset
    const uint32_t fit = (uint32_t)std::min<size_t>(std::max<size_t>(FFT_OUT_BYTES / per, 1), L.bsz);
    F.chunk = (L.bsz + (L.bsz + fit - 1u) / fit - 1u) / ((L.bsz + fit - 1u) / fit);  // passes of about equal length
    *out_bytes = per * F.chunk;
}

// The line of `concentrated`: (4 kappa)^2 or (2.75 kappa)^2.  kappa^2 is taken over the bins up to
// four apart (1/|R|^4 falls fast) and up to four offsets an axis.
void fft_field_spread(const DevLbm& L, FftField& F) {
    const uint32_t bs[3] = {L.bsx, L.bsy, L.bsz};
    double r2[3][4][9], sum = 0.0;  // squares along an axis, [offset][difference of the bins]
    for (int a = 0; a < 3; a++)
        for (uint32_t i = 0; i < 4; i++)
            for (int d = -4; d <= 4; d++) {
                const double r = (double)bs[a] * d + (2u * i + 1u) * bs[a] / 8u - 0.5 * bs[a];
                r2[a][i][d + 4] = r * r;
            }
    for (int o = 0; o < 64; o++)
        for (int d = 0; d < 729; d++) {
            if (d == 364) continue;  // the own bin
            const double r = r2[0][o % 4][d % 9] + r2[1][o / 4 % 4][d / 9 % 9] + r2[2][o / 16][d / 81];
            sum += 1.0 / (r * r);
        }
    const double M = 2.0 * L.nd, line = L.nd == 16u ? 4.0 : 2.75, k2 = sum / (64.0 * M * M * M);
    F.kappa = (float)std::sqrt(k2);
    F.spread = (float)(line * line * k2);
}

cudaError_t launch_fft_plan(const DevLbm& L, const FftField& F, cudaStream_t s) {
    const cudaError_t e = L.nd == 16u ? prepare_kernels<16>() : prepare_kernels<8>();
    if (e != cudaSuccess) return e;
    const uint32_t blocks = F.ux * F.uy * F.uz * (L.nd + 1u);
    if (L.nd == 16u) k_fft_plan<16><<<blocks, 256, 0, s>>>(L, F);
    else k_fft_plan<8><<<blocks, 256, 0, s>>>(L, F);
    return cudaGetLastError();
}

uint32_t fft_passes(const DevLbm& L, const FftField& F) { return (L.bsz + F.chunk - 1u) / F.chunk; }
uint32_t fft_src_blocks(const DevLbm& L) { return 4u * (L.nd + 1u); }
uint32_t fft_sum_blocks(const DevLbm& L, const FftField& F, uint32_t pass) {
    return 6u * chunk_len(L, F, pass) * L.bsy * L.bsx;
}
uint32_t fft_put_blocks(const DevLbm& L, const FftField& F, uint32_t pass) {
    return 2u * ((L.bsy * L.nx + PUT_X - 1u) / PUT_X) * L.nd * chunk_len(L, F, pass);
}

uint32_t launch_fft_batch(const FftBatch* B, uint32_t passes, cudaStream_t s) {
    return B->nd == 16u ? launch_batch_nd<16>(B, passes, s) : launch_batch_nd<8>(B, passes, s);
}

uint32_t launch_fft_field(const DevLbm& L, const FftField& F, const uint32_t* gate, cudaStream_t s) {
    return L.nd == 16u ? launch_field_nd<16>(L, F, gate, s) : launch_field_nd<8>(L, F, gate, s);
}

}  // namespace ion
