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
//   k_fft_plan  once per grid shape: spectra of R/|R|^3 (64-bit sums and transforms,
//               rounded to 32 bits).  An offset o and its mirror image b - o have spectra
//               that differ by the sign of a wave number and of a component, so
//               (b/2 + 1) of b offsets per axis are kept.
//   k_fft_src   spectra of the sources, 4 (nd + 1) blocks; block 0 also looks at the range
//               of the sources (see below).
//   k_fft_sum   one block per offset and field (E or B): product of spectra, then the
//               inverse transforms along z, y and x in registers, passed on through
//               shared memory.
//   k_fft_put   the sums to the cells, x-rows at a time: E_stat + KE e, B_stat + KMU b.
//
// Rounding: a 32-bit transform's error is about 1.5e-7 of the field's norm (the direct
// 32-bit sums: 1.1e-6), spread evenly over the lattice.  An infinite bin would leave NaN
// where the direct sum keeps the sign, and sums near the ends of the exponent range would
// over- or underflow at other places; so for sources that are not finite, or whose largest
// value lies outside [1e-28, 1e25], `direct` is set and k_update_e_b_gated runs instead.
#include "field_fft.h"
#include "fft_regs.cuh"
#include "ion_device.cuh"
#include "ion_launch.h"

namespace ion {

namespace {

__host__ __device__ constexpr uint32_t slot_elems(uint32_t nd) { return 3u * nd * nd; }  // one kx plane, 3 components, [z][y]
// kx planes transformed together: 3 PL M = 192 threads
__host__ __device__ constexpr uint32_t planes(uint32_t nd) { return 32u / nd; }
__host__ __device__ constexpr uint32_t stage_elems(uint32_t nd) { return planes(nd) * 3u * nd * (2u * nd + 1u); }
// the staged planes overlay the slots that are not written yet
__host__ __device__ constexpr uint32_t sum_smem(uint32_t nd) { return ((nd - planes(nd)) * slot_elems(nd) + stage_elems(nd)) * 8u; }
static_assert(planes(16) * slot_elems(16) <= stage_elems(16) && planes(8) * slot_elems(8) <= stage_elems(8),
              "the last planes' slots lie inside the staging area");
constexpr uint32_t SUM_THREADS = 192, SRC_THREADS = 256, PUT_THREADS = 256, PUT_X = 128;

#define ION_TW(j) {(float)cos32(j), (float)sin32(j)}
__constant__ float2 c_tw[32] = {  // exp(2 pi i j / 32)
    ION_TW(0),  ION_TW(1),  ION_TW(2),  ION_TW(3),  ION_TW(4),  ION_TW(5),  ION_TW(6),  ION_TW(7),
    ION_TW(8),  ION_TW(9),  ION_TW(10), ION_TW(11), ION_TW(12), ION_TW(13), ION_TW(14), ION_TW(15),
    ION_TW(16), ION_TW(17), ION_TW(18), ION_TW(19), ION_TW(20), ION_TW(21), ION_TW(22), ION_TW(23),
    ION_TW(24), ION_TW(25), ION_TW(26), ION_TW(27), ION_TW(28), ION_TW(29), ION_TW(30), ION_TW(31)};
#undef ION_TW

// ---------------------------------------------------------------------------
// spectra of R/|R|^3: one block per distinct offset and kx
// ---------------------------------------------------------------------------
template <int ND>
__global__ void __launch_bounds__(256) k_fft_plan(const DevLbm L, const FftField F) {
    constexpr int M = 2 * ND;
    extern __shared__ __align__(16) uint8_t plan_smem[];
    C2<double>* a = reinterpret_cast<C2<double>*>(plan_smem);  // [component][mz][my], rows of M + 1
    __shared__ C2<double> tw[M];
    constexpr int ROW = M + 1;
    const uint32_t kx = blockIdx.x % (ND + 1u), u = blockIdx.x / (ND + 1u);
    const uint32_t ox = u % F.ux, oy = (u / F.ux) % F.uy, oz = u / (F.ux * F.uy);
    if (threadIdx.x < M) {
        const int j = (int)((threadIdx.x * kx) % M) * (32 / M);
        tw[threadIdx.x] = {cospi(j / 16.0), -sinpi(j / 16.0)};
    }
    __syncthreads();
    const double bx = L.bsx, by = L.bsy, bz = L.bsz;
    const double sx = ox - 0.5 * bx, sy = oy - 0.5 * by, sz = oz - 0.5 * bz;
    for (int t = threadIdx.x; t < M * M; t += blockDim.x) {
        const int my = t % M, mz = t / M;
        C2<double> g[3] = {{0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}};
        if (my != ND && mz != ND) {
            const double ry = by * (my < ND ? my : my - M) + sy, rz = bz * (mz < ND ? mz : mz - M) + sz;
            for (int mx = 0; mx < M; mx++) {
                if (mx == ND || (mx | my | mz) == 0) continue;  // outside the bin lattice, the own bin
                const double rx = bx * (mx < ND ? mx : mx - M) + sx;
                const double r2 = rx * rx + ry * ry + rz * rz;
                // 1/sqrt(r2): two Newton steps double the digits of the 32-bit value twice
                double y = (double)rsqrtf((float)r2);
                y = y * fma(-0.5 * r2 * y, y, 1.5);
                y = y * fma(-0.5 * r2 * y, y, 1.5);
                const double i3 = y * y * y;
                const C2<double> w = tw[mx];
                const double vx = rx * i3, vy = ry * i3, vz = rz * i3;
                g[0] = {fma(vx, w.x, g[0].x), fma(vx, w.y, g[0].y)};
                g[1] = {fma(vy, w.x, g[1].x), fma(vy, w.y, g[1].y)};
                g[2] = {fma(vz, w.x, g[2].x), fma(vz, w.y, g[2].y)};
            }
        }
        for (int c = 0; c < 3; c++) a[(c * M + mz) * ROW + my] = g[c];
    }
    __syncthreads();
    if (threadIdx.x < 3u * M) {  // along y, a row per thread
        C2<double>* row = a + threadIdx.x * ROW;
        C2<double> v[M];
#pragma unroll
        for (int k = 0; k < M; k++) v[k] = row[k];
        fft_regs<M, -1>(v);
#pragma unroll
        for (int k = 0; k < M; k++) row[k] = v[k];
    }
    __syncthreads();
    if (threadIdx.x < 3u * M) {  // along z, a column per thread
        const int c = threadIdx.x / M, ky = threadIdx.x % M;
        C2<double> v[M];
#pragma unroll
        for (int k = 0; k < M; k++) v[k] = a[(c * M + k) * ROW + ky];
        fft_regs<M, -1>(v);
        float2* out = F.G + ((((size_t)u * (ND + 1u) + kx) * 3u + c) * M) * M + ky;
#pragma unroll
        for (int k = 0; k < M; k++) out[k * M] = make_float2((float)v[k].x, (float)v[k].y);
    }
}

// ---------------------------------------------------------------------------
// spectra of the sources: block = component + 4 kx
// ---------------------------------------------------------------------------
template <int ND>
__device__ __forceinline__ void fft_src(const DevLbm& L, const FftField& F, const uint32_t block) {
    constexpr uint32_t M = 2u * ND, NB = ND * ND * ND;
    __shared__ float s[ND * ND * (ND + 1)];  // [z][y][x], rows of ND + 1
    __shared__ float2 a[ND][ND], b[ND][M];
    __shared__ uint32_t s_max[4], s_bad;
    const uint32_t c = block % 4u, kx = block / 4u;
    const uint32_t first = L.first_src, last = min(L.n_lod_own, L.n_bins);
    if (threadIdx.x < 4u) s_max[threadIdx.x] = 0u;
    if (threadIdx.x == 0u) s_bad = 0u;
    __syncthreads();
    uint32_t m[4] = {0u, 0u, 0u, 0u};
    for (uint32_t d = threadIdx.x; d < NB; d += SRC_THREADS) {
        const float4 v = d >= first && d < last ? reinterpret_cast<const float4*>(L.qu_lod)[d] : make_float4(0.f, 0.f, 0.f, 0.f);
        const float w[4] = {v.x, v.x * v.y, v.x * v.z, v.x * v.w};
        s[d / ND * (ND + 1) + d % ND] = c == 0u ? w[0] : c == 1u ? w[1] : c == 2u ? w[2] : w[3];
        if (block == 0u) {
#pragma unroll
            for (int k = 0; k < 4; k++) m[k] = max(m[k], __float_as_uint(w[k]) & 0x7FFFFFFFu);  // NaN > Inf > finite
        }
    }
    if (block == 0u) {
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint32_t v = __reduce_max_sync(0xFFFFFFFFu, m[k]);
            if ((threadIdx.x & 31u) == 0u) atomicMax(&s_max[k], v);
        }
    }
    __syncthreads();
    if (block == 0u && threadIdx.x < 4u) {
        const uint32_t v = s_max[threadIdx.x];
        if (v != 0u && !(v >= __float_as_uint(1e-28f) && v <= __float_as_uint(1e25f))) atomicExch(&s_bad, 1u);
    }
    // along x at this kx
    for (uint32_t t = threadIdx.x; t < ND * ND; t += SRC_THREADS) {
        float2 acc = make_float2(0.0f, 0.0f);
#pragma unroll
        for (uint32_t x = 0; x < ND; x++) {
            const float v = s[t * (ND + 1) + x];
            const float2 w = c_tw[((kx * x) % M) * (32u / M)];
            acc.x = fmaf(v, w.x, acc.x);
            acc.y = fmaf(-v, w.y, acc.y);
        }
        a[t / ND][t % ND] = acc;
    }
    __syncthreads();
    if (block == 0u && threadIdx.x == 0u) *F.direct = s_bad;
    // along y, then along z
    for (uint32_t t = threadIdx.x; t < ND * M; t += SRC_THREADS) {
        const uint32_t ky = t % M, z = t / M;
        float2 acc = make_float2(0.0f, 0.0f);
#pragma unroll
        for (uint32_t y = 0; y < ND; y++) {
            const float2 v = a[z][y], w = c_tw[((ky * y) % M) * (32u / M)];
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
            const float2 v = b[z][ky], w = c_tw[((kz * z) % M) * (32u / M)];
            acc.x = fmaf(v.x, w.x, fmaf(v.y, w.y, acc.x));
            acc.y = fmaf(v.y, w.x, fmaf(-v.x, w.y, acc.y));
        }
        out[t] = acc;
    }
}

// ---------------------------------------------------------------------------
// the sums of one offset: block = (((oz - oz0) bsy + oy) bsx + ox) 2 + (0: E, 1: B)
// ---------------------------------------------------------------------------
__device__ __forceinline__ C2<float> cmul(const float2 a, const float2 b) {
    return {fmaf(a.x, b.x, -(a.y * b.y)), fmaf(a.x, b.y, a.y * b.x)};
}
__device__ __forceinline__ C2<float> cmul_sub(const C2<float> s, const float2 a, const float2 b) {
    return {fmaf(-a.x, b.x, fmaf(a.y, b.y, s.x)), fmaf(-a.x, b.y, fmaf(-a.y, b.x, s.y))};
}

template <int ND>
__device__ __forceinline__ void fft_sum(const DevLbm& L, const FftField& F, const uint32_t block, const uint32_t oz0,
                                        float2* sm) {
    constexpr uint32_t M = 2u * ND, PL = planes(ND), SLOT = slot_elems(ND), ROW = M + 1u;
    const uint32_t group = block & 1u, o = block >> 1;
    const uint32_t ox = o % L.bsx, oy = (o / L.bsx) % L.bsy, oz = oz0 + o / (L.bsx * L.bsy);
    // the offset's spectra, or its mirror image's: R_a changes sign with the wave number k_a
    const bool fx = ox >= F.ux, fy = oy >= F.uy, fz = oz >= F.uz;
    const uint32_t u = (fx ? L.bsx - ox : ox) + ((fy ? L.bsy - oy : oy) + (fz ? L.bsz - oz : oz) * F.uy) * F.ux;
    const float2* G = F.G + (size_t)u * (ND + 1u) * 3u * M * M;
    // G(-kx, ky, kz) = conj G(kx, -ky, -kz): kx stays in 0..nd
    const bool ry = fx != fy, rz = fx != fz;
    const uint32_t t = threadIdx.x;
    const uint32_t f = (t / M) % 3u, pl = t / (3u * M), ky = t % M;  // this thread's line along z
    const uint32_t gy = ry ? (M - ky) % M : ky;
    // components of the product: E_f = G_f q; B_f = (q v)_i G_j - (q v)_j G_i, (f, i, j) cyclic
    const uint32_t i = f == 2u ? 0u : f + 1u, j = f == 0u ? 2u : f - 1u;
    auto flipped = [&](uint32_t c) { return c == 0u ? fx : c == 1u ? fy : fz; };
    const bool nf = flipped(f), ni = flipped(i), nj = flipped(j);
    auto product = [&](uint32_t kx, uint32_t kz) -> C2<float> {
        const uint32_t gz = rz ? (M - kz) % M : kz;
        const float2* g = G + (size_t)kx * 3u * M * M + gz * M + gy;
        const float2* s = F.S + (size_t)kx * 4u * M * M + kz * M + ky;
        auto load_g = [&](uint32_t c, bool neg) {
            float2 v = __ldg(g + c * M * M);
            if (fx) v.y = -v.y;
            if (neg) { v.x = -v.x; v.y = -v.y; }
            return v;
        };
        if (group == 0u) return cmul(load_g(f, nf), __ldg(s));
        const float2 si = __ldg(s + (1u + i) * M * M), sj = __ldg(s + (1u + j) * M * M);
        return cmul_sub(cmul(si, load_g(j, nj)), sj, load_g(i, ni));
    };
#pragma unroll 1
    for (uint32_t p0 = 0; p0 < (uint32_t)ND; p0 += PL) {
        float2* stage = sm + p0 * SLOT;  // [plane][component][z][ky], rows of M + 1
        {
            const uint32_t kx = p0 + pl;
            auto half_line = [&](uint32_t par, C2<float>(&v)[ND]) {  // kz = par, par + 2, ...
#pragma unroll
                for (uint32_t k = 0; k < (uint32_t)ND; k++) v[k] = product(kx, 2u * k + par);
                if (kx == 0u) {  // the transforms of kx = 0 and kx = nd are real: one complex line holds both
#pragma unroll
                    for (uint32_t k = 0; k < (uint32_t)ND; k++) {
                        const C2<float> a = product(ND, 2u * k + par);
                        v[k] = {v[k].x - a.y, v[k].y + a.x};
                    }
                }
                fft_regs<ND, 1>(v);
            };
            C2<float> e[ND], d[ND];
            half_line(0u, e);
            half_line(1u, d);
            fft_join<ND, 1>(e, d);
            float2* w = stage + (pl * 3u + f) * ND * ROW + ky;
#pragma unroll
            for (uint32_t z = 0; z < (uint32_t)ND; z++) w[z * ROW] = make_float2(e[z].x, e[z].y);
        }
        __syncthreads();
        C2<float> e[ND], d[ND];
        const uint32_t line = t;  // (plane, component, z)
        const uint32_t z = line % ND;
        if (line < PL * 3u * ND) {
            const float2* r = stage + line * ROW;
#pragma unroll
            for (uint32_t k = 0; k < (uint32_t)ND; k++) {
                const float2 a = r[2u * k], b = r[2u * k + 1u];
                e[k] = {a.x, a.y};
                d[k] = {b.x, b.y};
            }
            fft_half<ND, 1>(e, d);
        }
        __syncthreads();  // the staged lines are read: the slots below them may be written
        if (line < PL * 3u * ND) {
            // slot [component][z][(y + z) mod nd]: rows of nd without bank conflicts
            float2* w = sm + (p0 + line / (3u * ND)) * SLOT + (line / ND % 3u * ND + z) * ND;
#pragma unroll
            for (uint32_t y = 0; y < (uint32_t)ND; y++) w[(y + z) % ND] = make_float2(e[y].x, e[y].y);
        }
    }
    __syncthreads();
    // along x, real outputs: with X_k the line's transform and h = nd, z_k = (X_k + conj X_{h-k})
    // + i w^k (X_k - conj X_{h-k}) transforms to (x_0 + i x_1, x_2 + i x_3, ...)
    const uint32_t noz = F.chunk;
    for (uint32_t line = t; line < SLOT; line += SUM_THREADS) {
        const uint32_t y = line % ND, z = line / ND % ND, c = line / (ND * ND);
        const float2* r = sm + (c * ND + z) * ND + (y + z) % ND;
        C2<float> v[ND];
        const float2 r0 = r[0];
        v[0] = {r0.x + r0.y, r0.x - r0.y};
        float2 X[ND];
#pragma unroll
        for (uint32_t k = 1; k < (uint32_t)ND; k++) X[k] = r[k * SLOT];
#pragma unroll
        for (uint32_t k = 1; k < (uint32_t)ND; k++) {
            const float2 p = X[k], q = X[ND - k];
            const C2<float> dif = twist<1>(C2<float>{p.x - q.x, p.y + q.y}, k * (16 / ND) + 8);  // times i w^k
            v[k] = {(p.x + q.x) + dif.x, (p.y - q.y) + dif.y};
        }
        fft_regs<ND, 1>(v);
        constexpr float scale = 1.0f / (float)(M * M * M);  // a power of two: exact
        float* out = F.out + (((((size_t)(group * 3u + c) * noz * L.bsy * L.bsx) + o) * ND) * ND + z) * ND + y;
#pragma unroll
        for (uint32_t n = 0; n < (uint32_t)ND / 2u; n++) {
            out[(2u * n) * ND * ND] = v[n].x * scale;
            out[(2u * n + 1u) * ND * ND] = v[n].y * scale;
        }
    }
}

// ---------------------------------------------------------------------------
// the sums to the cells: block = component + 6 (x tile + tiles (Iz + nd (oy + bsy (oz - oz0))));
// a block transposes nd rows (y = Iy bsy + oy) of up to PUT_X cells through shared memory
// ---------------------------------------------------------------------------
template <int ND>
__device__ __forceinline__ void fft_put(const DevLbm& L, const FftField& F, uint32_t block, const uint32_t oz0) {
    __shared__ float s[ND][PUT_X + 1];
    const uint32_t tiles = (L.nx + PUT_X - 1u) / PUT_X;
    const uint32_t c = block % 6u;
    block /= 6u;
    const uint32_t x0 = block % tiles * PUT_X;
    block /= tiles;
    const uint32_t Iz = block % ND, oy = block / ND % L.bsy, ozl = block / (ND * L.bsy);
    const uint32_t cnt = min(PUT_X, L.nx - x0);
    const float* in = F.out + (((size_t)(c * F.chunk + ozl) * L.bsy + oy) * L.bsx) * (ND * ND * ND) + Iz * ND;
    for (uint32_t t = threadIdx.x; t < cnt * ND; t += PUT_THREADS) {
        const uint32_t Iy = t % ND, xl = t / ND, x = x0 + xl, Ix = x / L.bsx, ox = x - Ix * L.bsx;
        s[Iy][xl] = in[(size_t)(ox * ND + Ix) * (ND * ND) + Iy];
    }
    __syncthreads();
    const uint32_t z = Iz * L.bsz + oz0 + ozl;
    const size_t N = L.n;
    const uint32_t k = c < 3u ? c : c - 3u;
    const float* stat = (c < 3u ? L.e_stat : L.b_stat) + k * N;
    float* dyn = (c < 3u ? L.e_dyn : L.b_dyn) + k * N;
    const float scale = c < 3u ? L.ke : L.kmu;
    for (uint32_t t = threadIdx.x; t < PUT_X * ND; t += PUT_THREADS) {
        const uint32_t xl = t % PUT_X, Iy = t / PUT_X;
        if (xl >= cnt) continue;
        const uint32_t n = x0 + xl + ((Iy * L.bsy + oy) + z * L.ny) * L.nx;
        if ((L.flags[n] & F_BO) != F_S) dyn[n] = stat[n] + scale * s[Iy][xl];
    }
}

template <int ND>
__global__ void __launch_bounds__(SRC_THREADS) k_fft_src(const DevLbm L, const FftField F) {
    fft_src<ND>(L, F, blockIdx.x);
}
template <int ND>
__global__ void __launch_bounds__(SUM_THREADS, 2) k_fft_sum(const DevLbm L, const FftField F, const uint32_t oz0) {
    extern __shared__ __align__(16) float2 sum_sm[];
    if (*F.direct) return;
    fft_sum<ND>(L, F, blockIdx.x, oz0, sum_sm);
}
template <int ND>
__global__ void __launch_bounds__(PUT_THREADS) k_fft_put(const DevLbm L, const FftField F, const uint32_t oz0) {
    if (*F.direct) return;
    fft_put<ND>(L, F, blockIdx.x, oz0);
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
__global__ void __launch_bounds__(SUM_THREADS, 2) k_fft_sum_batch(const FftBatch B, const uint32_t pass) {
    extern __shared__ __align__(16) float2 sum_sm[];
    __shared__ DevLbm L;
    __shared__ FftField F;
    __shared__ uint32_t e;
    const uint32_t block = batch_entry(B, B.sum_off, L, F, e);
    if (*F.direct) return;
    fft_sum<ND>(L, F, block, pass * F.chunk, sum_sm);
}
template <int ND>
__global__ void __launch_bounds__(PUT_THREADS) k_fft_put_batch(const FftBatch B, const uint32_t pass) {
    __shared__ DevLbm L;
    __shared__ FftField F;
    __shared__ uint32_t e;
    const uint32_t block = batch_entry(B, B.put_off, L, F, e);
    if (*F.direct) return;
    fft_put<ND>(L, F, block, pass * F.chunk);
}

template <int ND>
cudaError_t prepare_kernels() {
    const int plan = 3 * 2 * ND * (2 * ND + 1) * 16;
    cudaError_t e = cudaFuncSetAttribute(k_fft_sum<ND>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sum_smem(ND));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_fft_sum_batch<ND>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sum_smem(ND));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_fft_plan<ND>, cudaFuncAttributeMaxDynamicSharedMemorySize, plan);
    return e;
}

uint32_t chunk_len(const DevLbm& L, const FftField& F, uint32_t pass) {
    const uint32_t oz = pass * F.chunk;
    return oz >= L.bsz ? 0u : F.chunk < L.bsz - oz ? F.chunk : L.bsz - oz;
}

template <int ND>
uint32_t launch_field_nd(const DevLbm& L, const FftField& F, cudaStream_t s) {
    k_fft_src<ND><<<fft_src_blocks(L), SRC_THREADS, 0, s>>>(L, F);
    for (uint32_t p = 0; p < fft_passes(L, F); p++) {
        k_fft_sum<ND><<<fft_sum_blocks(L, F, p), SUM_THREADS, sum_smem(ND), s>>>(L, F, p * F.chunk);
        k_fft_put<ND><<<fft_put_blocks(L, F, p), PUT_THREADS, 0, s>>>(L, F, p * F.chunk);
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
    const size_t fit = FFT_OUT_BYTES / per;
    F.chunk = fit < 1 ? 1u : fit < L.bsz ? (uint32_t)fit : L.bsz;
    *out_bytes = per * F.chunk;
}

cudaError_t launch_fft_plan(const DevLbm& L, const FftField& F, cudaStream_t s) {
    const cudaError_t e = L.nd == 16u ? prepare_kernels<16>() : prepare_kernels<8>();
    if (e != cudaSuccess) return e;
    const uint32_t blocks = F.ux * F.uy * F.uz * (L.nd + 1u);
    if (L.nd == 16u) k_fft_plan<16><<<blocks, 256, 3 * 32 * 33 * 16, s>>>(L, F);
    else k_fft_plan<8><<<blocks, 256, 3 * 16 * 17 * 16, s>>>(L, F);
    return cudaGetLastError();
}

uint32_t fft_passes(const DevLbm& L, const FftField& F) { return (L.bsz + F.chunk - 1u) / F.chunk; }
uint32_t fft_src_blocks(const DevLbm& L) { return 4u * (L.nd + 1u); }
uint32_t fft_sum_blocks(const DevLbm& L, const FftField& F, uint32_t pass) {
    return 2u * chunk_len(L, F, pass) * L.bsy * L.bsx;
}
uint32_t fft_put_blocks(const DevLbm& L, const FftField& F, uint32_t pass) {
    return 6u * ((L.nx + PUT_X - 1u) / PUT_X) * L.nd * L.bsy * chunk_len(L, F, pass);
}

uint32_t launch_fft_batch(const FftBatch* B, uint32_t passes, cudaStream_t s) {
    return B->nd == 16u ? launch_batch_nd<16>(B, passes, s) : launch_batch_nd<8>(B, passes, s);
}

uint32_t launch_fft_field(const DevLbm& L, const FftField& F, cudaStream_t s) {
    return L.nd == 16u ? launch_field_nd<16>(L, F, s) : launch_field_nd<8>(L, F, s);
}

}  // namespace ion
