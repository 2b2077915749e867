// field_table.cu -- the BITWISE E/B field with R/|R|^3 from a table.
//
// Cell and bin coordinates are integers and halves, so R of a cell and a bin is exact and
// depends only on the bins' difference and the cell's offset in its bin, and so do the three
// quotients R/|R|^3 (IEEE sqrt and divides) that are most of eb_tile<false>'s work: 36 of its
// 57 operations per term.  Here they are computed once per grid shape, of |2 R| with the
// operations of add_src<false> (a sign passes through all of them unchanged).  A term's other 21
// operations and the order of the sums are those of eb_tile<false>: the field is bit-identical.
//
// The table lies [difference of the bins][in-bin offset] (in_bins), about 128 bytes per cell.
// Grids above 2^25 cells, 4 GB of it, keep one entry per |2 R|, [z][y][x], 16 bytes per cell: a
// load then touches a line for every (y, z) of its lanes' offsets, and each entry costs its
// index and three signs.  Same blocks, us a step, [z][y][x] against in_bins: 32^3 146 / 111,
// 64^3 671 / 615, 96^3 2,230 / 2,043, 256^3 41,941 / 38,089; depth 3 at 192^3 2,940 / 2,635.
//
// A thread holds the cells of one in-bin offset in R neighbouring bins along x.  Along a row
// of source bins every step needs one new table entry, the others move on by a cell: R + nd - 1
// entries per row of nd sources and R cells.  Lanes are neighbouring offsets (coalesced table
// rows, one broadcast source), the warps of a block the R-groups of the same offsets, whose
// entries overlap in L1.  Bound by FP32 issue: 22.6 instructions per term, of which 21 are its operations (R = 4).
#include "field_table.h"
#include "ion_device.cuh"
#include "ion_launch.h"

namespace ion {

namespace {

// |2 R| along an axis has the parity of the bin edge: entry a >> 1 holds a = |2 R|
__global__ void __launch_bounds__(256) k_field_table(const DevLbm L, const FieldTable F) {
    const uint32_t x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y, z = blockIdx.z;
    if (x >= F.tx) return;
    const float rx = 0.5f * (float)(2u * x + (L.bsx & 1u)), ry = 0.5f * (float)(2u * y + (L.bsy & 1u)),
                rz = 0.5f * (float)(2u * z + (L.bsz & 1u));
    float4 p = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (rx != 0.0f || ry != 0.0f || rz != 0.0f) {  // R = 0 only in the own bin, which is skipped
        const float s = sqrtf((rx * rx + ry * ry) + rz * rz);
        const float c3 = (s * s) * s;
        const float r = __frcp_rn(c3);
        p = make_float4(div_rn_shared(rx, c3, r), div_rn_shared(ry, c3, r), div_rn_shared(rz, c3, r), 0.0f);
    }
    F.T[((size_t)z * F.ty + y) * F.tx + x] = p;
}

// in_bins: 2 R = b (2 D) + 2 offset - b for D = 1 - nd .. nd - 1; the quotients of |2 R| with R's signs
__global__ void __launch_bounds__(256) k_field_table_bins(const DevLbm L, const FieldTable F) {
    const uint32_t no = L.bsx * L.bsy * L.bsz, k = blockIdx.x * blockDim.x + threadIdx.x;  // at most 2^28
    if (k >= F.tx * F.ty * F.tz * no) return;
    const uint32_t o = k % no, d = k / no;
    const int m = (int)L.nd - 1;
    const int ax = (int)L.bsx * (2 * ((int)(d % F.tx) - m) - 1) + 2 * (int)(o % L.bsx),
              ay = (int)L.bsy * (2 * ((int)(d / F.tx % F.ty) - m) - 1) + 2 * (int)(o / L.bsx % L.bsy),
              az = (int)L.bsz * (2 * ((int)(d / (F.tx * F.ty)) - m) - 1) + 2 * (int)(o / (L.bsx * L.bsy));
    const float rx = 0.5f * (float)abs(ax), ry = 0.5f * (float)abs(ay), rz = 0.5f * (float)abs(az);
    float4 p = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (ax != 0 || ay != 0 || az != 0) {
        const float s = sqrtf((rx * rx + ry * ry) + rz * rz);
        const float c3 = (s * s) * s;
        const float r = __frcp_rn(c3);
        const float qx = div_rn_shared(rx, c3, r), qy = div_rn_shared(ry, c3, r), qz = div_rn_shared(rz, c3, r);
        p = make_float4(ax < 0 ? -qx : qx, ay < 0 ? -qy : qy, az < 0 ? -qz : qz, 0.0f);
    }
    F.T[k] = p;
}

struct P3 { float x, y, z; };

__device__ __forceinline__ void add_term(const P3& p, const float4& v, float (&e)[3], float (&b)[3]) {
    e[0] = e[0] + v.x * p.x; e[1] = e[1] + v.x * p.y; e[2] = e[2] + v.x * p.z;
    const float bx = v.z * p.z - v.w * p.y, by = v.w * p.x - v.y * p.z, bz = v.y * p.y - v.z * p.x;
    b[0] = b[0] + v.x * bx; b[1] = b[1] + v.x * by; b[2] = b[2] + v.x * bz;
}

// What a thread sums: the R neighbouring bins i0.. along x of one in-bin offset, in bin row (iy, iz)
struct TableItem {
    bool valid;
    uint32_t i0, ox, oy, oz, iy, iz;
    int x0, step;  // cell 0 and source 0, and a bin's step: 2 R_x, or (BINS) the index in the table row
};
template <int ND, int R, int EB, bool BINS>
__device__ __forceinline__ TableItem table_item(const DevLbm& L) {
    TableItem t;
    const uint32_t no = L.bsx * L.bsy * L.bsz;
    const uint32_t item = blockIdx.x * EB + threadIdx.x % EB;
    t.valid = item < no * (ND * ND);
    t.i0 = threadIdx.x / EB * R;
    // (EB offsets, Iz, Iy, offset), then the no % EB last ones likewise: the bins of the same
    // offsets run side by side and find their table rows in L2
    uint32_t o, I = t.valid ? item : 0u, m = EB;
    if (I < no / EB * EB * (ND * ND)) {
        o = I / (EB * ND * ND) * EB;
        I %= EB * ND * ND;
    } else {
        m = no % EB;
        o = no - m;
        I -= o * (ND * ND);
    }
    o += I % m;
    I /= m;
    t.iy = I % ND;
    t.iz = I / ND;
    t.ox = o % L.bsx;
    t.oy = o / L.bsx % L.bsy;
    t.oz = o / (L.bsx * L.bsy);
    t.x0 = BINS ? (int)((t.i0 + ND - 1u) * no + o) : (int)(2u * (L.bsx * t.i0 + t.ox)) - (int)L.bsx;
    t.step = BINS ? (int)no : 2 * (int)L.bsx;
    return t;
}
// the table row of source row (jy, jz), and the signs of its entries
template <int ND, bool BINS>
struct TableRow {
    const float4* row;
    uint32_t sy = 0, sz = 0;
    __device__ __forceinline__ TableRow(const DevLbm& L, const FieldTable& F, const TableItem& t, int jy, int jz) {
        if constexpr (BINS) {
            row = F.T + (((int)t.iz - jz + ND - 1) * (2 * ND - 1) + ((int)t.iy - jy + ND - 1)) * (2 * ND - 1) * t.step;
        } else {
            const int ay = (int)(2u * (L.bsy * t.iy + t.oy)) - (int)L.bsy - 2 * (int)L.bsy * jy;
            const int az = (int)(2u * (L.bsz * t.iz + t.oz)) - (int)L.bsz - 2 * (int)L.bsz * jz;
            sy = (uint32_t)ay & 0x80000000u;
            sz = (uint32_t)az & 0x80000000u;
            row = F.T + ((size_t)((uint32_t)abs(az) >> 1) * F.ty + ((uint32_t)abs(ay) >> 1)) * F.tx;
        }
    }
    __device__ __forceinline__ P3 entry(int x) const {
        if constexpr (BINS) {
            const float4 t = __ldg(row + x);
            return {t.x, t.y, t.z};
        } else {
            const float4 t = __ldg(row + ((uint32_t)abs(x) >> 1));
            return {__uint_as_float(__float_as_uint(t.x) ^ ((uint32_t)x & 0x80000000u)),
                    __uint_as_float(__float_as_uint(t.y) ^ sy), __uint_as_float(__float_as_uint(t.z) ^ sz)};
        }
    }
};
// a row that holds a lane's own bin, or starts or ends inside the sources
template <int ND, int R, bool BINS>
__device__ __forceinline__ void table_edge_row(const TableRow<ND, BINS>& w, const TableItem& t, const float4* src, int d0, int first,
                                               int last, bool own_row, int step, float (&e)[R][3], float (&b)[R][3]) {
#pragma unroll 1
    for (int j = max(first - d0, 0); j < min(last - d0, ND); j++) {
        const float4 v = src[j];
#pragma unroll
        for (int i = 0; i < R; i++)
            if (!own_row || (int)t.i0 + i != j) add_term(w.entry(t.x0 + (i - j) * step), v, e[i], b[i]);
    }
}
template <int R>
__device__ __forceinline__ void table_store(const DevLbm& L, const TableItem& t, const float (&e)[R][3], const float (&b)[R][3]) {
    if (!t.valid) return;
    const size_t N = L.n;
#pragma unroll
    for (int i = 0; i < R; i++) {
        const uint32_t n = (t.i0 + i) * L.bsx + t.ox + ((t.iy * L.bsy + t.oy) + (t.iz * L.bsz + t.oz) * L.ny) * L.nx;
        if ((L.flags[n] & F_BO) == F_S) continue;
#pragma unroll
        for (int c = 0; c < 3; c++) {
            L.e_dyn[c * N + n] = L.e_stat[c * N + n] + L.ke * e[i][c];
            L.b_dyn[c * N + n] = L.b_stat[c * N + n] + L.kmu * b[i][c];
        }
    }
}

template <int ND, int R, int EB, bool BINS>
__global__ void __launch_bounds__(EB * (ND / R), 512 / (EB * (ND / R))) k_update_e_b_table(const DevLbm L, const FieldTable F) {
    constexpr uint32_t THREADS = EB * (ND / R);
    __shared__ float4 src[ND * ND];  // one z plane of sources: (q, vx, vy, vz)
    const TableItem t = table_item<ND, R, EB, BINS>(L);
    const int first = (int)L.first_src, last = (int)min(L.n_lod_own, L.n_bins);
    float e[R][3] = {}, b[R][3] = {};
    for (int jz = first / (ND * ND); jz < ND; jz++) {
        __syncthreads();
        for (uint32_t k = threadIdx.x; k < ND * ND; k += THREADS)
            src[k] = reinterpret_cast<const float4*>(L.qu_lod)[jz * (ND * ND) + k];
        __syncthreads();
#pragma unroll 1
        for (int jy = 0; jy < ND; jy++) {
            const int d0 = (jz * ND + jy) * ND;
            if (d0 + ND <= first || d0 >= last) continue;
            const TableRow<ND, BINS> w(L, F, t, jy, jz);
            int step = t.step;
            asm volatile("" : "+r"(step));  // the entries' indices are formed per row, not kept
            const bool own_row = (uint32_t)jy == t.iy && (uint32_t)jz == t.iz;
            if (d0 >= first && d0 + ND <= last && !__any_sync(0xFFFFFFFFu, own_row)) {
                P3 p[R + ND - 1];  // entry k: bins R - 1 - k apart
#pragma unroll
                for (int k = 0; k < R - 1; k++) p[k] = w.entry(t.x0 + (R - 1 - k) * step);
#pragma unroll
                for (int j = 0; j < ND; j++) {
                    p[R - 1 + j] = w.entry(t.x0 - j * step);
                    const float4 v = src[jy * ND + j];
#pragma unroll
                    for (int i = 0; i < R; i++) add_term(p[R - 1 - i + j], v, e[i], b[i]);
                }
            } else {
                table_edge_row<ND, R, BINS>(w, t, src + jy * ND, d0, first, last, own_row, step, e, b);
            }
        }
    }
    table_store<R>(L, t, e, b);
}

template <int ND, int R, int EB, bool BINS>
cudaError_t launch(const DevLbm& L, const FieldTable& F, cudaStream_t s) {
    const unsigned items = L.n / ND;  // cells over the bins along x
    k_update_e_b_table<ND, R, EB, BINS><<<(items + EB - 1) / EB, EB * (ND / R), 0, s>>>(L, F);
    return cudaGetLastError();
}

}  // namespace

// Depths 3 and 4 without cells of the reference's near field; edges below 2^16 cells keep 2 R
// in 32 bits and every coordinate exact.
bool field_table_fits(const DevLbm& L) {
    return (L.nd == 8u || L.nd == 16u) && L.near_x == 1u && L.near_y == 1u && L.near_z == 1u && L.nx < 65536u &&
           L.ny < 65536u && L.nz < 65536u;
}

size_t field_table_size(const DevLbm& L, FieldTable& F) {
    F.in_bins = L.n <= 1u << 25;
    if (F.in_bins) {
        F.tx = F.ty = F.tz = 2u * L.nd - 1u;
        return (size_t)F.tx * F.ty * F.tz * (L.bsx * L.bsy * L.bsz) * sizeof(float4);
    }
    F.tx = (2u * L.nx - L.bsx) / 2u + 1u;  // the largest |2 R| is 2 n - b
    F.ty = (2u * L.ny - L.bsy) / 2u + 1u;
    F.tz = (2u * L.nz - L.bsz) / 2u + 1u;
    return (size_t)F.tx * F.ty * F.tz * sizeof(float4);
}

cudaError_t launch_field_table(const DevLbm& L, const FieldTable& F, cudaStream_t s) {
    if (F.in_bins) {
        const uint32_t entries = F.tx * F.ty * F.tz * (L.bsx * L.bsy * L.bsz);
        k_field_table_bins<<<(entries + 255u) / 256u, 256, 0, s>>>(L, F);
        return cudaGetLastError();
    }
    k_field_table<<<dim3((F.tx + 255u) / 256u, F.ty, F.tz), 256, 0, s>>>(L, F);
    return cudaGetLastError();
}

// Four cells a thread amortise the table entries and the source best (22 against 23 instructions
// a term); small boxes fill the schedulers better with two.  Two against four, us a step with
// three domains in turn: depth 4 32^3 111 / 144, 48^3 280 / 281, 64^3 651 / 614; depth 3 48^3
// 56 / 61, 64^3 118 / 108.  The line lies between 48^3 and 64^3.
cudaError_t launch_update_e_b_table(const DevLbm& L, const FieldTable& F, cudaStream_t s) {
    const bool wide = L.n >= 3u << 16;
    if (!F.in_bins) return L.nd == 16u ? launch<16, 4, 32, false>(L, F, s) : launch<8, 4, 64, false>(L, F, s);
    if (L.nd == 16u) return wide ? launch<16, 4, 32, true>(L, F, s) : launch<16, 2, 16, true>(L, F, s);
    return wide ? launch<8, 4, 64, true>(L, F, s) : launch<8, 2, 32, true>(L, F, s);
}

}  // namespace ion
