// setup_kernels.cu -- geometry and static-field kernels, FP64 reductions.
//
//   voxelize  : IonSolver src/kernels/sim_kernels.cl:1150-1231 (one thread
//               or warp per bounding-box column, Moeller-Trumbore in both ray
//               directions, 16-bit hit distances, parity with correction).
//   psi / B   : sim_kernels.cl:1234-1276.  The reference loops over all N
//               cells for each of the (N+2)^3 potential points and tests the
//               magnet flag; here the magnet cells are first compacted into an
//               ascending index list (same summation order, ~N/N_magnet less
//               work) and staged through shared memory.
//   static E  : sim_kernels.cl:1278-1300, same compaction over charged cells.
//   FP64 sums : deterministic two-pass tree reductions of decoded DDFs.
#include <algorithm>
#include <cmath>

#include "ion_device.cuh"
#include "ion_launch.h"
#include "reduce_f64.cuh"

namespace ion {

// ---------------------------------------------------------------------------
// voxelisation
// ---------------------------------------------------------------------------
struct V3 { float x, y, z; };
__device__ __forceinline__ V3 vsub(V3 a, V3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ V3 vcross(V3 a, V3 b) { return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x}; }
__device__ __forceinline__ float vdot(V3 a, V3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ int iclamp(int x, int lo, int hi) { return x < lo ? lo : (x > hi ? hi : x); }

constexpr uint32_t VOX_WARPS = 4, VOX_THREADS = 128, VOX_HITS = 64;

// a thread per column
__global__ void __launch_bounds__(VOX_THREADS) k_voxelize(const DevLbm L, VoxArgs A) {
    const uint32_t a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= A.columns) return;
    const int nx = (int)L.nx, ny = (int)L.ny, nz = (int)L.nz;
    const int dir = A.direction;
    uint32_t c[3];
    if (dir == 0) { c[0] = (uint32_t)iclamp((int)A.x0, 0, nx - 1); c[1] = a % L.ny; c[2] = a / L.ny; }
    else if (dir == 1) { c[0] = a / L.nz; c[1] = (uint32_t)iclamp((int)A.y0, 0, ny - 1); c[2] = a % L.nz; }
    else { c[0] = a % L.nx; c[1] = a / L.nx; c[2] = (uint32_t)iclamp((int)A.z0, 0, nz - 1); }
    const V3 org = {(((float)c[0] + 0.5f) - 0.5f * (float)nx) + (0.5f * (float)nx - 0.5f),
                    (((float)c[1] + 0.5f) - 0.5f * (float)ny) + (0.5f * (float)ny - 0.5f),
                    (((float)c[2] + 0.5f) - 0.5f * (float)nz) + (0.5f * (float)nz - 0.5f)};
    bool outside;
    if (dir == 0) outside = org.y < A.y0 || org.z < A.z0 || org.y >= A.y1 || org.z >= A.z1;
    else if (dir == 1) outside = org.x < A.x0 || org.z < A.z0 || org.x >= A.x1 || org.z >= A.z1;
    else outside = org.x < A.x0 || org.y < A.y0 || org.x >= A.x1 || org.y >= A.y1;
    if (outside) return;
    const V3 rdir = {(float)(dir == 0), (float)(dir == 1), (float)(dir == 2)};
    uint16_t dist[64];
    for (int i = 0; i < 64; i++) dist[i] = 0;
    uint32_t hits = 0, back = 0;
    for (uint32_t i = 0; i < A.ntri; i++) {
        const V3 P0 = {A.p0[3 * i], A.p0[3 * i + 1], A.p0[3 * i + 2]};
        const V3 P1 = {A.p1[3 * i], A.p1[3 * i + 1], A.p1[3 * i + 2]};
        const V3 P2 = {A.p2[3 * i], A.p2[3 * i + 1], A.p2[3 * i + 2]};
        const V3 e1 = vsub(P1, P0), e2 = vsub(P2, P0), s0 = vsub(org, P0);
        const V3 pv = vcross(rdir, e2), qv = vcross(s0, e1);
        const float inv = 1.0f / vdot(e1, pv);
        const float su = inv * vdot(s0, pv), sv = inv * vdot(rdir, qv), sd = inv * vdot(e2, qv);
        if (su >= 0.0f && su < 1.0f && sv >= 0.0f && su + sv < 1.0f) {
            if (sd > 0.0f) {
                if (hits < 64u && sd < 65536.0f) dist[hits] = (uint16_t)sd;
                hits++;
            } else {
                back++;
            }
        }
    }
    const uint32_t ns = hits < 64u ? hits : 64u;
    for (uint32_t i = 1; i < ns; i++) {
        const uint16_t key = dist[i];
        int k = (int)i - 1;
        while (k >= 0 && dist[k] > key) { dist[k + 1] = dist[k]; k--; }
        dist[k + 1] = key;
    }
    bool inside = (hits % 2u) && (back % 2u);
    uint32_t next = (hits % 2u) != (back % 2u);
    const uint32_t h0 = c[dir];
    const uint32_t hmax = dir == 0 ? (uint32_t)iclamp((int)A.x1, 0, nx) : dir == 1 ? (uint32_t)iclamp((int)A.y1, 0, ny)
                                                                                  : (uint32_t)iclamp((int)A.z1, 0, nz);
    const uint32_t last = hits - 1u < 63u ? hits - 1u : 63u;
    const uint32_t hmesh = h0 + (uint32_t)dist[last];
    const size_t N = L.n;
    for (uint32_t hh = h0; hh < hmax; hh++) {
        while (next < hits && hh > h0 + (uint32_t)dist[next < 63u ? next : 63u]) { inside = !inside; next++; }
        inside = inside && (next < hits && hh < hmesh);
        uint32_t cc[3] = {c[0], c[1], c[2]};
        cc[dir] = hh;
        const uint32_t n = cc[0] + (cc[1] + cc[2] * L.ny) * L.nx;
        if (inside) {
            L.flags[n] = (uint8_t)((L.flags[n] & ~F_BO) | A.flag);
            if (L.ext_mhd) {
                if (A.flag & F_M) { L.b_dyn[n] = A.mx; L.b_dyn[N + n] = A.my; L.b_dyn[2 * N + n] = A.mz; }
                else if ((A.flag & F_F) || (A.flag & F_C)) L.b_dyn[n] = A.mx;
            }
        }
    }
}

// a warp per column: the lanes take the triangles side by side and file their hits in triangle
// order
__global__ void __launch_bounds__(VOX_WARPS * 32) k_voxelize_warp(const DevLbm L, VoxArgs A) {
    __shared__ uint16_t s_dist[VOX_WARPS][VOX_HITS], s_sorted[VOX_WARPS][VOX_HITS];
    const uint32_t wid = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t a = blockIdx.x * VOX_WARPS + wid;
    if (a >= A.columns) return;
    const int nx = (int)L.nx, ny = (int)L.ny, nz = (int)L.nz;
    const int dir = A.direction;
    uint32_t c[3];
    if (dir == 0) { c[0] = (uint32_t)iclamp((int)A.x0, 0, nx - 1); c[1] = a % L.ny; c[2] = a / L.ny; }
    else if (dir == 1) { c[0] = a / L.nz; c[1] = (uint32_t)iclamp((int)A.y0, 0, ny - 1); c[2] = a % L.nz; }
    else { c[0] = a % L.nx; c[1] = a / L.nx; c[2] = (uint32_t)iclamp((int)A.z0, 0, nz - 1); }
    const V3 org = {(((float)c[0] + 0.5f) - 0.5f * (float)nx) + (0.5f * (float)nx - 0.5f),
                    (((float)c[1] + 0.5f) - 0.5f * (float)ny) + (0.5f * (float)ny - 0.5f),
                    (((float)c[2] + 0.5f) - 0.5f * (float)nz) + (0.5f * (float)nz - 0.5f)};
    bool outside;
    if (dir == 0) outside = org.y < A.y0 || org.z < A.z0 || org.y >= A.y1 || org.z >= A.z1;
    else if (dir == 1) outside = org.x < A.x0 || org.z < A.z0 || org.x >= A.x1 || org.z >= A.z1;
    else outside = org.x < A.x0 || org.y < A.y0 || org.x >= A.x1 || org.y >= A.y1;
    if (outside) return;
    const V3 rdir = {(float)(dir == 0), (float)(dir == 1), (float)(dir == 2)};
    uint16_t* const dist = s_dist[wid];
    uint16_t* const sorted = s_sorted[wid];
    for (uint32_t i = lane; i < VOX_HITS; i += 32u) dist[i] = sorted[i] = 0;
    __syncwarp();
    uint32_t hits = 0, back = 0;
    for (uint32_t base = 0; base < A.ntri; base += 32u) {
        const uint32_t i = base + lane;
        bool hit = false;
        float sd = 0.0f;
        if (i < A.ntri) {
            const V3 P0 = {A.p0[3 * i], A.p0[3 * i + 1], A.p0[3 * i + 2]};
            const V3 P1 = {A.p1[3 * i], A.p1[3 * i + 1], A.p1[3 * i + 2]};
            const V3 P2 = {A.p2[3 * i], A.p2[3 * i + 1], A.p2[3 * i + 2]};
            const V3 e1 = vsub(P1, P0), e2 = vsub(P2, P0), s0 = vsub(org, P0);
            const V3 pv = vcross(rdir, e2), qv = vcross(s0, e1);
            const float inv = 1.0f / vdot(e1, pv);
            const float su = inv * vdot(s0, pv), sv = inv * vdot(rdir, qv);
            sd = inv * vdot(e2, qv);
            hit = su >= 0.0f && su < 1.0f && sv >= 0.0f && su + sv < 1.0f;
        }
        const uint32_t ahead = __ballot_sync(0xFFFFFFFFu, hit && sd > 0.0f);
        back += __popc(__ballot_sync(0xFFFFFFFFu, hit && !(sd > 0.0f)));
        const uint32_t at = hits + __popc(ahead & ((1u << lane) - 1u));
        if (hit && sd > 0.0f && at < VOX_HITS && sd < 65536.0f) dist[at] = (uint16_t)sd;
        hits += __popc(ahead);
    }
    __syncwarp();
    const uint32_t ns = hits < VOX_HITS ? hits : VOX_HITS;
    for (uint32_t i = lane; i < ns; i += 32u) {  // ascending, by rank
        const uint16_t key = dist[i];
        uint32_t rank = 0;
        for (uint32_t k = 0; k < ns; k++) rank += dist[k] < key || (dist[k] == key && k < i);
        sorted[rank] = key;
    }
    __syncwarp();
    bool inside = (hits % 2u) && (back % 2u);
    uint32_t next = (hits % 2u) != (back % 2u);
    const uint32_t h0 = c[dir];
    const uint32_t hmax = dir == 0 ? (uint32_t)iclamp((int)A.x1, 0, nx) : dir == 1 ? (uint32_t)iclamp((int)A.y1, 0, ny)
                                                                                  : (uint32_t)iclamp((int)A.z1, 0, nz);
    const uint32_t last = hits - 1u < VOX_HITS - 1u ? hits - 1u : VOX_HITS - 1u;
    const uint32_t hmesh = h0 + (uint32_t)sorted[last];
    const size_t N = L.n;
    for (uint32_t base = h0; base < hmax; base += 32u) {
        uint32_t in = 0u;  // the next 32 cells of the column: every lane follows the crossings, then writes its cell
        for (uint32_t k = 0; k < 32u && base + k < hmax; k++) {
            const uint32_t hh = base + k;
            while (next < hits && hh > h0 + (uint32_t)sorted[next < VOX_HITS - 1u ? next : VOX_HITS - 1u]) { inside = !inside; next++; }
            inside = inside && (next < hits && hh < hmesh);
            in |= (uint32_t)inside << k;
        }
        if (!((in >> lane) & 1u)) continue;
        uint32_t cc[3] = {c[0], c[1], c[2]};
        cc[dir] = base + lane;
        const uint32_t n = cc[0] + (cc[1] + cc[2] * L.ny) * L.nx;
        L.flags[n] = (uint8_t)((L.flags[n] & ~F_BO) | A.flag);
        if (L.ext_mhd) {
            if (A.flag & F_M) { L.b_dyn[n] = A.mx; L.b_dyn[N + n] = A.my; L.b_dyn[2 * N + n] = A.mz; }
            else if ((A.flag & F_F) || (A.flag & F_C)) L.b_dyn[n] = A.mx;
        }
    }
}

// A thread per column leaves most SMs with a few warps, each waiting on one triangle's divide
// after another, until there are many columns; a warp per column repeats the walk in every lane.
// us a call, thread / warp: 64^3 with 48 triangles 39 / 20, 128^3 with 224 on 14,209 columns
// 110 / 77, 192^3 with 12 on 10,000 columns 37 / 52, 512^3 with 12 on 216,039 columns 299 /
// 3,440 and with 3,968 3,766 / 5,199.  The forms cross near 9,000 columns at 12 triangles,
// 22,000 at 224, 45,000 at 960 and 85,000 at 3,968: a square root of the triangles.
static bool voxelize_by_warps(uint64_t columns, uint32_t ntri) {
    return columns <= 8192u || columns * columns <= 1800000ull * ntri;
}

void launch_voxelize(const DevLbm& L, const VoxArgs& A, cudaStream_t s) {
    const uint32_t edge[3] = {L.nx, L.ny, L.nz};
    const float lo[3] = {A.x0, A.y0, A.z0}, hi[3] = {A.x1, A.y1, A.z1};
    uint64_t columns = 1;  // inside the mesh's bounds
    for (int a = 0; a < 3; a++)
        if (a != A.direction)
            columns *= (uint64_t)std::max(0.0, std::min((double)edge[a], std::ceil((double)hi[a])) - std::max(0.0, std::ceil((double)lo[a])));
    if (voxelize_by_warps(columns, A.ntri)) k_voxelize_warp<<<grid_for(A.columns, VOX_WARPS), VOX_WARPS * 32, 0, s>>>(L, A);
    else k_voxelize<<<grid_for(A.columns, VOX_THREADS), VOX_THREADS, 0, s>>>(L, A);
}

// ---------------------------------------------------------------------------
// order-preserving compaction of cells whose flags match a mask
// (count per 1024-cell tile -> exclusive scan of tile counts -> scatter)
// ---------------------------------------------------------------------------
constexpr uint32_t CT = 1024;

__global__ void __launch_bounds__(CT) k_compact_count(const uint8_t* flags, uint32_t n, uint8_t mask, uint32_t* tiles) {
    const uint32_t i = blockIdx.x * CT + threadIdx.x;
    const int hit = i < n && (flags[i] & mask) != 0;
    const int c = __syncthreads_count(hit);
    if (threadIdx.x == 0) tiles[blockIdx.x] = (uint32_t)c;
}

__global__ void __launch_bounds__(CT) k_compact_scan(uint32_t* tiles, uint32_t ntiles, uint32_t* total) {
    __shared__ uint32_t part[CT];
    const uint32_t per = (ntiles + CT - 1) / CT;
    const uint32_t b = threadIdx.x * per, e = min(b + per, ntiles);
    uint32_t s = 0;
    for (uint32_t i = b; i < e; i++) s += tiles[i];
    part[threadIdx.x] = s;
    __syncthreads();
    for (uint32_t off = 1; off < CT; off <<= 1) {  // inclusive Hillis-Steele scan
        const uint32_t v = threadIdx.x >= off ? part[threadIdx.x - off] : 0u;
        __syncthreads();
        part[threadIdx.x] += v;
        __syncthreads();
    }
    uint32_t run = threadIdx.x ? part[threadIdx.x - 1] : 0u;
    for (uint32_t i = b; i < e; i++) { const uint32_t c = tiles[i]; tiles[i] = run; run += c; }
    if (threadIdx.x == CT - 1) *total = part[CT - 1];
}

__global__ void __launch_bounds__(CT) k_compact_scatter(const uint8_t* flags, uint32_t n, uint8_t mask,
                                                        const uint32_t* tiles, uint32_t* out) {
    __shared__ uint32_t warp_count[CT / 32];
    const uint32_t i = blockIdx.x * CT + threadIdx.x;
    const bool hit = i < n && (flags[i] & mask) != 0;
    const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    const uint32_t ball = __ballot_sync(0xFFFFFFFFu, hit);
    if (lane == 0) warp_count[wid] = __popc(ball);
    __syncthreads();
    uint32_t off = tiles[blockIdx.x];
    for (uint32_t w = 0; w < wid; w++) off += warp_count[w];
    if (hit) out[off + __popc(ball & ((1u << lane) - 1u))] = i;
}

void launch_compact(const DevLbm& L, uint8_t mask, uint32_t* tiles, uint32_t* list, uint32_t* total, cudaStream_t s) {
    const uint32_t ntiles = (L.n + CT - 1) / CT;
    k_compact_count<<<ntiles, CT, 0, s>>>(L.flags, L.n, mask, tiles);
    k_compact_scan<<<1, CT, 0, s>>>(tiles, ntiles, total);
    k_compact_scatter<<<ntiles, CT, 0, s>>>(L.flags, L.n, mask, tiles, list);
}

// ---------------------------------------------------------------------------
// magnetic scalar potential on the padded grid, stored in E_dyn
// ---------------------------------------------------------------------------
constexpr uint32_t MAG_TILE = 256;

// On few points k_psi and k_static_b are launched for lists of fewer than `below` cells before the host
// knows the length, which k_static_b reports.
__global__ void __launch_bounds__(256) k_psi(const DevLbm L, const uint32_t* mags, const uint32_t* count, const uint32_t below,
                                             float* psi) {
    __shared__ float4 s_p[MAG_TILE];  // (x+1, y+1, z+1) as float
    __shared__ float4 s_m[MAG_TILE];  // magnetisation
    const uint32_t l0 = L.nx + 2, l1 = L.ny + 2;
    const uint32_t np = (l0 * l1) * (L.nz + 2);
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t t = i % (l0 * l1);
    const float cx = (float)(t % l0), cy = (float)(t / l0), cz = (float)(i / (l0 * l1));
    const uint32_t nm = *count;
    if (nm >= below) return;
    const size_t N = L.n;
    float acc = 0.0f;
    for (uint32_t base = 0; base < nm; base += MAG_TILE) {
        __syncthreads();
        for (uint32_t k = threadIdx.x; k < MAG_TILE && base + k < nm; k += blockDim.x) {
            const uint32_t m = mags[base + k];
            uint32_t x, y, z;
            cell_xyz(L, m, x, y, z);
            s_p[k] = make_float4((float)(x + 1u), (float)(y + 1u), (float)(z + 1u), 0.0f);
            s_m[k] = make_float4(L.b_dyn[m], L.b_dyn[N + m], L.b_dyn[2 * N + m], 0.0f);
        }
        __syncthreads();
        const uint32_t cnt = min(MAG_TILE, nm - base);
        if (i < np) {
            for (uint32_t k = 0; k < cnt; k++) {
                const float4 p = s_p[k], m = s_m[k];
                const float dx = cx - p.x, dy = cy - p.y, dz = cz - p.z;
                const float l = sqrtf((dx * dx + dy * dy) + dz * dz);
                if (!(l == 0.0f)) acc = acc + ((dx * m.x + dy * m.y) + dz * m.z) / ((l * l) * l);
            }
        }
    }
    if (i < np) psi[i] = (float)((double)acc / (4.0 * 3.14159265358979323846));
}

__global__ void __launch_bounds__(256) k_static_b(const DevLbm L, const uint32_t* count, const uint32_t below, PsiInfo* info,
                                                  const float* psi) {
    const uint32_t n = blockIdx.x * blockDim.x + threadIdx.x;
    if (info && n == 0u) info->count = *count;
    if (*count >= below || n >= L.n || (L.flags[n] & F_S) == F_S) return;
    uint32_t x, y, z;
    cell_xyz(L, n, x, y, z);
    const uint32_t l0 = L.nx + 2, l1 = L.ny + 2;
    const size_t c = (x + 1u) + ((size_t)(y + 1u) + (size_t)(z + 1u) * l1) * l0;
    const size_t zo = (size_t)l0 * l1;
    const float gx = (psi[c + 1] - psi[c - 1]) / 2.0f, gy = (psi[c + l0] - psi[c - l0]) / 2.0f,
                gz = (psi[c + zo] - psi[c - zo]) / 2.0f;
    const float m = -L.kmu0;
    const size_t N = L.n;
    L.b_stat[n] = L.b_stat[n] + m * gx;
    L.b_stat[N + n] = L.b_stat[N + n] + m * gy;
    L.b_stat[2 * N + n] = L.b_stat[2 * N + n] + m * gz;
}

// ---------------------------------------------------------------------------
// the potential from tabulated terms.  A term ((d . M) / |d|^3, d = point - magnet cell) depends
// on d and M only, so for a list with few distinct magnetisations the terms of every d are
// computed once (k_psi's operations, k_psi_terms) and a point's sum is one addition per magnet
// cell, in list order as before: bit-identical.  (+0 stands in where k_psi skips d = 0: a sum
// that starts at +0 is never -0, so adding it changes nothing.)
//
// The list is cut into runs of cells that follow each other along x with one M (k_psi_runs).  A
// thread sums PSI_R points in x: a step along a run takes one new term for PSI_R additions.
// Lanes are neighbouring (y, z), and the table is laid out [z][x][y] so that they load
// consecutive terms; rows that follow each other in y find most of their terms in L1.  Bound by
// the additions: at 128^3 and 6,800 cells 0.63 ms (immediate load offsets; 0.76 ms with computed
// addresses, 0.69 ms with two rows in packed additions at half the warps), k_psi 15.9 ms.
// ---------------------------------------------------------------------------
constexpr uint32_t PSI_R = 16, PSI_THREADS = 256, RUN_THREADS = 1024;

// one block, the list in tiles: distinct magnetisations, bounds and runs, in list order (of a list
// of fewer than `from` cells the length only).
// runs[r] = (first list entry, its cell | magnetisation << 30), runs[number of runs] = (list length, 0)
__global__ void __launch_bounds__(RUN_THREADS) k_psi_runs(const DevLbm L, const uint32_t* list, const uint32_t* count,
                                                          uint2* runs, const uint32_t max_runs, const uint32_t from,
                                                          PsiInfo* info) {
    __shared__ uint32_t s_m[PSI_KINDS][3], s_kinds, s_first, s_warp[RUN_THREADS / 32], s_lo[3], s_hi[3];
    const uint32_t nm = *count, t = threadIdx.x, lane = t & 31u;
    const size_t N = L.n;
    if (nm < from) {
        if (t == 0) info->count = nm;
        return;
    }
    if (t == 0) s_kinds = 0u;
    if (t < 3) { s_lo[t] = 0xFFFFFFFFu; s_hi[t] = 0u; }
    uint32_t nruns = 0;
    auto mag = [&](uint32_t n, int c) { return __float_as_uint(L.b_dyn[c * N + n]); };
    for (uint32_t base = 0; base < nm; base += RUN_THREADS) {
        const uint32_t i = base + t;
        const bool in = i < nm;
        uint32_t n = 0, x = 0, y = 0, z = 0, m[3] = {0u, 0u, 0u}, kind = 0;
        bool start = false;
        if (in) {
            n = list[i];
            cell_xyz(L, n, x, y, z);
            for (int c = 0; c < 3; c++) m[c] = mag(n, c);
            const uint32_t before = i ? list[i - 1] : 0u;
            start = i == 0 || n != before + 1u || x == 0u || mag(before, 0) != m[0] || mag(before, 1) != m[1] ||
                    mag(before, 2) != m[2];
        }
        for (;;) {  // the first entry of a magnetisation that is not known yet adds it
            __syncthreads();
            if (t == 0) s_first = 0xFFFFFFFFu;
            __syncthreads();
            bool known = !in;
            for (uint32_t k = 0; k < s_kinds; k++)
                if (in && s_m[k][0] == m[0] && s_m[k][1] == m[1] && s_m[k][2] == m[2]) { known = true; kind = k; }
            if (!known) atomicMin(&s_first, t);
            __syncthreads();
            const uint32_t f = s_first;
            if (f == 0xFFFFFFFFu) break;
            if (s_kinds == PSI_KINDS) {  // too many: the host takes k_psi
                if (t == 0) { info->count = nm; info->kinds = PSI_KINDS + 1u; }
                return;
            }
            __syncthreads();
            if (t == f) {
                for (int c = 0; c < 3; c++) s_m[s_kinds][c] = m[c];
                s_kinds++;
            }
        }
        if (in) {
            const uint32_t p[3] = {x, y, z};
            for (int c = 0; c < 3; c++) { atomicMin(&s_lo[c], p[c]); atomicMax(&s_hi[c], p[c]); }
        }
        const uint32_t ball = __ballot_sync(0xFFFFFFFFu, start);
        if (lane == 0) s_warp[t >> 5] = __popc(ball);
        __syncthreads();
        uint32_t at = nruns;
        for (uint32_t w = 0; w < RUN_THREADS / 32; w++) {
            if (w < (t >> 5)) at += s_warp[w];
            nruns += s_warp[w];
        }
        if (nruns >= max_runs) {  // no room (nor much use): the host takes k_psi
            if (t == 0) { info->count = nm; info->kinds = PSI_KINDS + 1u; }
            return;
        }
        if (start) runs[at + __popc(ball & ((1u << lane) - 1u))] = make_uint2(i, n | kind << 30);
        __syncthreads();
    }
    if (t == 0) {
        runs[nruns] = make_uint2(nm, 0u);
        info->count = nm;
        info->runs = nruns;
        info->kinds = s_kinds;
    }
    if (t < 3) { info->lo[t] = s_lo[t]; info->hi[t] = s_hi[t]; }
    if (t < 3u * PSI_KINDS) (&info->m[0][0])[t] = __uint_as_float((&s_m[0][0])[t]);
}

// terms T[kind][z][x][y] of the differences point - cell, from (x0, y0, z0) on
__global__ void __launch_bounds__(256) k_psi_terms(const PsiTable P) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x, x = i / P.ny, y = i % P.ny;
    const uint32_t k = blockIdx.y / P.tz, z = blockIdx.y % P.tz;
    if (x >= P.tx) return;
    const float dx = (float)(P.x0 + (int)x), dy = (float)(P.y0 + (int)y), dz = (float)(P.z0 + (int)z);
    const float* m = P.m[k];
    const float l = sqrtf((dx * dx + dy * dy) + dz * dz);
    float v = 0.0f;
    if (!(l == 0.0f)) v = ((dx * m[0] + dy * m[1]) + dz * m[2]) / ((l * l) * l);
    P.T[(((size_t)k * P.tz + z) * P.tx + x) * P.ty + y] = v;
}

// PITCH: the table's row length in elements (0: P.ty), a constant so that a step's load is an
// immediate offset
template <uint32_t PITCH>
__global__ void __launch_bounds__(PSI_THREADS, 4) k_psi_runs_sum(const DevLbm L, const PsiTable P, float* psi) {
    constexpr int R = (int)PSI_R;
    const uint32_t l0 = L.nx + 2, l1 = L.ny + 2, l2 = L.nz + 2;
    const uint32_t nxb = (l0 + PSI_R - 1u) / PSI_R, rows = l1 * l2;
    const int64_t ty = PITCH ? PITCH : P.ty;
    // warps of a block: the x blocks of the same 32 rows first
    const uint32_t w = blockIdx.x * (PSI_THREADS / 32u) + (threadIdx.x >> 5);
    const uint32_t xb = w % nxb, row = w / nxb * 32u + (threadIdx.x & 31u);
    if (w / nxb * 32u >= rows) return;  // whole warps
    const bool valid = row < rows;
    const uint32_t cy = (valid ? row : 0u) % l1, cz = (valid ? row : 0u) / l1;
    // the term of point (PSI_R xb, cy, cz) and a cell whose run offset is 0
    const float* const origin = P.T + ((int64_t)((int)cz - P.z0) * P.tx + ((int)(xb * PSI_R) - P.x0)) * ty + ((int)cy - P.y0);
    float acc[R];
#pragma unroll
    for (int i = 0; i < R; i++) acc[i] = 0.0f;
    uint2 run = P.runs[0];
    for (uint32_t r = 0; r < P.nruns; r++) {
        const uint2 next = P.runs[r + 1u];
        uint32_t x, y, z;
        cell_xyz(L, run.y & 0x3FFFFFFFu, x, y, z);
        const int64_t kind = (int64_t)(run.y >> 30) * P.tz;
        // points are the padded grid's: the cell lies at (x + 1, y + 1, z + 1)
        const float* p = origin + ((kind - (int64_t)(z + 1u)) * P.tx - (int64_t)(x + 1u)) * ty - (int64_t)(y + 1u);
        uint32_t left = next.x - run.x;
        run = next;
        // up to R steps along the run: `above` holds the terms of the points at its position,
        // `below` gets the R terms before them
        auto steps = [&](const float (&above)[R], float (&below)[R]) {
            if (left >= PSI_R) {
#pragma unroll
                for (int k = 1; k <= R; k++) below[R - k] = __ldg(p - k * ty);
#pragma unroll
                for (int k = 0; k < R; k++)
#pragma unroll
                    for (int i = 0; i < R; i++) acc[i] = acc[i] + (i >= k ? above[i - k] : below[R + i - k]);
                p -= R * ty;
                left -= PSI_R;
            } else {
#pragma unroll
                for (int k = 0; k < R - 1; k++) {
                    if (k >= (int)left) break;
                    if (k > 0) below[R - k] = __ldg(p - k * ty);
#pragma unroll
                    for (int i = 0; i < R; i++) acc[i] = acc[i] + (i >= k ? above[i - k] : below[R + i - k]);
                }
                left = 0u;
            }
        };
        float a[R], b[R];
#pragma unroll
        for (int i = 0; i < R; i++) a[i] = __ldg(p + i * ty);
        for (;;) {
            steps(a, b);
            if (!left) break;
            steps(b, a);
            if (!left) break;
        }
    }
    if (!valid) return;
#pragma unroll
    for (uint32_t i = 0; i < PSI_R; i++) {
        const uint32_t cx = xb * PSI_R + i;
        if (cx < l0) psi[cx + (size_t)row * l0] = (float)((double)acc[i] / (4.0 * 3.14159265358979323846));
    }
}

void launch_psi_runs(const DevLbm& L, const uint32_t* list, const uint32_t* count, uint2* runs, uint32_t max_runs, uint32_t from,
                     PsiInfo* info, cudaStream_t s) {
    k_psi_runs<<<1, RUN_THREADS, 0, s>>>(L, list, count, runs, max_runs, from, info);
}

// Estimates in us, from calls on 16^3 to 256^3 cells with 1 to 2,000 magnet cells, scattered or
// in a block; both forms take 42 us besides.  A cell costs the direct sum a divide per point (or
// its latency, on few points); the table costs a host read-back and a term per entry, then
// per point an addition a cell and some seven a run.  The lines are crossed near 460 cells at 32^3, 130 at 64^3 and
// 40 at 128^3 (in one block): direct / table, us, 32^3 with 100 scattered cells 53 / 106, in a
// block 55 / 82; 128^3 with 64 scattered 232 / 470, in a block 234 / 163.
static double psi_points(const DevLbm& L) { return (double)(L.nx + 2u) * (L.ny + 2u) * (L.nz + 2u); }
static double psi_direct_us(const DevLbm& L, double cells) { return cells * std::max(0.13, 0.07 + 1.2e-6 * psi_points(L)); }
uint32_t psi_table_from(const DevLbm& L) {
    if (L.n >= 1u << 30) return 0xFFFFFFFFu;  // a run keeps its magnetisation in the index's top bits
    const double np = psi_points(L);
    return (uint32_t)(((np < PSI_FEW_POINTS ? 60.0 : 45.0) + 2.5e-5 * np) / psi_direct_us(L, 1.0));
}
bool psi_table_pays(const DevLbm& L, const PsiInfo& I, size_t entries) {
    const double np = psi_points(L);
    return psi_direct_us(L, I.count) >
           20.0 + 1.6e-5 * (double)entries + I.runs * std::max(0.12, 3.2e-7 * np) + I.count * std::max(0.05, 2.6e-8 * np);
}

size_t psi_table_size(const DevLbm& L, const PsiInfo& I, PsiTable& P) {
    const uint32_t nxb = (L.nx + 2u + PSI_R - 1u) / PSI_R;
    // x: a thread's points reach PSI_R nxb - 1, its loads run up to PSI_R past the end of a run
    P.x0 = -(int)(I.hi[0] + 1u) - (int)(2u * PSI_R);
    P.y0 = -(int)(I.hi[1] + 1u);
    P.z0 = -(int)(I.hi[2] + 1u);
    P.tx = nxb * PSI_R + (I.hi[0] - I.lo[0]) + 2u * PSI_R;
    P.ty = L.ny + 2u + (I.hi[1] - I.lo[1]);
    P.ny = P.ty;
    if (P.ty <= 256u) P.ty = (P.ty + 63u) / 64u * 64u;  // the constant pitches
    P.tz = L.nz + 2u + (I.hi[2] - I.lo[2]);
    P.nruns = I.runs;
    for (uint32_t k = 0; k < PSI_KINDS; k++)
        for (int c = 0; c < 3; c++) P.m[k][c] = I.m[k][c];
    return (size_t)I.kinds * P.tz * P.tx * P.ty * sizeof(float);
}

void launch_psi_table_static_b(const DevLbm& L, const PsiTable& P, uint32_t kinds, const uint32_t* count, cudaStream_t s) {
    k_psi_terms<<<dim3((P.tx * P.ny + 255u) / 256u, P.tz * kinds), 256, 0, s>>>(P);
    const uint64_t rows = (uint64_t)(L.ny + 2) * (L.nz + 2), nxb = (L.nx + 2u + PSI_R - 1u) / PSI_R;
    const unsigned grid = grid_for((rows + 31u) / 32u * nxb * 32u, PSI_THREADS);
    if (P.ty == 64u) k_psi_runs_sum<64><<<grid, PSI_THREADS, 0, s>>>(L, P, L.e_dyn);
    else if (P.ty == 128u) k_psi_runs_sum<128><<<grid, PSI_THREADS, 0, s>>>(L, P, L.e_dyn);
    else if (P.ty == 192u) k_psi_runs_sum<192><<<grid, PSI_THREADS, 0, s>>>(L, P, L.e_dyn);
    else if (P.ty == 256u) k_psi_runs_sum<256><<<grid, PSI_THREADS, 0, s>>>(L, P, L.e_dyn);
    else k_psi_runs_sum<0><<<grid, PSI_THREADS, 0, s>>>(L, P, L.e_dyn);
    k_static_b<<<grid_for(L.n, 256), 256, 0, s>>>(L, count, 0xFFFFFFFFu, nullptr, L.e_dyn);
}

void launch_psi_static_b(const DevLbm& L, const uint32_t* mags, const uint32_t* count, uint32_t below, PsiInfo* info, cudaStream_t s) {
    const uint64_t np = (uint64_t)(L.nx + 2) * (L.ny + 2) * (L.nz + 2);
    k_psi<<<grid_for(np, 256), 256, 0, s>>>(L, mags, count, below, L.e_dyn);
    k_static_b<<<grid_for(L.n, 256), 256, 0, s>>>(L, count, below, info, L.e_dyn);
}

// static E from charged solids (charge per cell held in B_dyn.x by the voxeliser) into E:
// E_stat (static_e_from_mesh) or E_var (precompute_E_ECR, the same kernel)
__global__ void __launch_bounds__(256) k_static_e(const DevLbm L, const uint32_t* list, const uint32_t* count, float* E) {
    __shared__ float4 s_c[MAG_TILE];
    const uint32_t n = blockIdx.x * blockDim.x + threadIdx.x;
    const bool active = n < L.n && (L.flags[n] & F_S) != F_S;
    uint32_t x = 0, y = 0, z = 0;
    if (n < L.n) cell_xyz(L, n, x, y, z);
    const uint32_t nc = *count;
    float ex = 0.0f, ey = 0.0f, ez = 0.0f;
    for (uint32_t base = 0; base < nc; base += MAG_TILE) {
        __syncthreads();
        for (uint32_t k = threadIdx.x; k < MAG_TILE && base + k < nc; k += blockDim.x) {
            const uint32_t m = list[base + k];
            uint32_t a, b, c;
            cell_xyz(L, m, a, b, c);
            s_c[k] = make_float4((float)a, (float)b, (float)c, L.b_dyn[m]);
        }
        __syncthreads();
        if (active) {
            const uint32_t cnt = min(MAG_TILE, nc - base);
            for (uint32_t k = 0; k < cnt; k++) {
                const float4 p = s_c[k];
                const float dx = (float)x - p.x, dy = (float)y - p.y, dz = (float)z - p.z;
                const float l = sqrtf((dx * dx + dy * dy) + dz * dz);
                if (l == 0.0f) continue;
                const float l3 = (l * l) * l;
                ex = ex + (dx * p.w) / l3; ey = ey + (dy * p.w) / l3; ez = ez + (dz * p.w) / l3;
            }
        }
    }
    if (active) {
        const size_t N = L.n;
        E[n] = E[n] + ex * L.ke;
        E[N + n] = E[N + n] + ey * L.ke;
        E[2 * N + n] = E[2 * N + n] + ez * L.ke;
    }
}

void launch_static_e(const DevLbm& L, const uint32_t* list, const uint32_t* count, float* E, cudaStream_t s) {
    k_static_e<<<grid_for(L.n, 256), 256, 0, s>>>(L, list, count, E);
}

void launch_sum_f64(const void* x, int ft, uint64_t count, double* partials, uint32_t nparts, double* out,
                    cudaStream_t s) {
    // nparts blocks of ceil(count / nparts) values (reduce_f64.cuh)
    launch_sum_two_pass(x, ft, count, (count + nparts - 1) / nparts, nparts, partials, out, s);
}

// ---------------------------------------------------------------------------
// storage-codec round trip (used to check the device codecs exhaustively)
// ---------------------------------------------------------------------------
__global__ void k_codec(int ft, const float* in, uint16_t* enc, float* dec, const uint16_t* raw, float* raw_dec,
                        uint64_t n) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (ft == ION_FP16S) {
        Ddf<ION_FP16S>::st(enc, i, in[i]);
        dec[i] = Ddf<ION_FP16S>::ld(enc, i);
        raw_dec[i] = Ddf<ION_FP16S>::ld(raw, i);
    } else {
        enc[i] = fp16c_encode(in[i]);  // any NaN, where Ddf's takes results of arithmetic
        dec[i] = Ddf<ION_FP16C>::ld(enc, i);
        raw_dec[i] = Ddf<ION_FP16C>::ld(raw, i);
    }
}

void launch_codec(int ft, const float* in, uint16_t* enc, float* dec, const uint16_t* raw, float* raw_dec, uint64_t n,
                  cudaStream_t s) {
    k_codec<<<grid_for(n, 256), 256, 0, s>>>(ft, in, enc, dec, raw, raw_dec, n);
}

// ---------------------------------------------------------------------------
// FP32 FMA throughput probe: 8 independent FMA chains per thread, enough
// warps to fill every SM; the denominator of the field kernel's roofline.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_fma_probe(float* out, int iters, float a, float b) {
    float r[8];
#pragma unroll
    for (int k = 0; k < 8; k++) r[k] = (float)(threadIdx.x + k) * 1e-3f;
    for (int i = 0; i < iters; i++) {
#pragma unroll
        for (int k = 0; k < 8; k++) r[k] = fmaf(r[k], a, b);
    }
    float s = 0.0f;
#pragma unroll
    for (int k = 0; k < 8; k++) s += r[k];
    if (s == 123.456f) out[threadIdx.x] = s;  // keeps the chains alive
}

// ---------------------------------------------------------------------------
// Self-test of div_rn_shared against the IEEE division, bit for bit, on
// pseudo-random quotients over the ranges the E/B sums produce: numerators
// |x| in [2^-1, 2^13) and exact small integers and halves, denominators
// b = (s s) s with s = sqrt(r2), r2 in [2^-2, 2^27), and b drawn directly in
// [2^-3, 2^40).
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint64_t mix64(uint64_t z) {
    z += 0x9e3779b97f4a7c15ull;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}
__device__ __forceinline__ float unit(uint64_t v) { return (float)(v >> 40) * (1.0f / 16777216.0f); }  // [0, 1)

__global__ void __launch_bounds__(256) k_div_check(uint64_t samples, uint64_t seed, unsigned long long* bad,
                                                   float* first_bad) {
    unsigned long long local = 0;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < samples;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t h1 = mix64(seed ^ (i * 3 + 0)), h2 = mix64(seed ^ (i * 3 + 1)), h3 = mix64(seed ^ (i * 3 + 2));
        float x;
        if ((h1 & 7u) == 0) x = (float)((int)(h1 >> 40) % 16385 - 8192) * 0.5f;  // small integers and halves
        else x = exp2f(-1.0f + 14.0f * unit(h1)) * ((h1 & 8u) ? -1.0f : 1.0f);
        float b;
        if (h2 & 1u) {
            const float s = sqrtf(exp2f(-2.0f + 29.0f * unit(h2)));
            b = (s * s) * s;
        } else {
            b = exp2f(-3.0f + 43.0f * unit(h2));
        }
        b = __uint_as_float(__float_as_uint(b) ^ ((uint32_t)h3 & 0x7u));  // vary the low mantissa bits
        const float want = __fdiv_rn(x, b);
        const float got = div_rn_shared(x, b, __frcp_rn(b));
        if (__float_as_uint(want) != __float_as_uint(got)) {
            if (atomicAdd(bad, 1ull) == 0ull) { first_bad[0] = x; first_bad[1] = b; }
            local++;
        }
    }
    (void)local;
}

void launch_div_check(uint64_t samples, uint64_t seed, unsigned long long* bad, float* first_bad, cudaStream_t s) {
    k_div_check<<<152 * 8, 256, 0, s>>>(samples, seed, bad, first_bad);
}

void launch_fma_probe(float* out, int blocks, int iters, cudaStream_t s) {
    k_fma_probe<<<blocks, 256, 0, s>>>(out, iters, 0.999999f, 1e-6f);
}

}  // namespace ion
