// ion_launch.h -- host-side launchers of the sm_103a kernels.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace ion {

struct DevLbm;

inline unsigned grid_for(uint64_t n, unsigned block) {
    const uint64_t g = (n + block - 1) / block;
    return (unsigned)(g ? g : 1);
}

// voxelize_mesh arguments (IonSolver src/mesh.rs:281-343)
struct VoxArgs {
    const float *p0, *p1, *p2;  // device, [ntri][3]
    uint32_t ntri;
    int direction;
    uint32_t columns;
    float x0, y0, z0, x1, y1, z1;  // bounding box +-2
    uint8_t flag;
    float mx, my, mz;
};

// a list of magnet cells as runs along x (setup_kernels.cu, k_psi_runs)
constexpr uint32_t PSI_KINDS = 4;  // distinct magnetisations with a table of their own
// On fewer points a wait costs a short list more than two launches for nothing a long one: the direct
// sum of short lists is launched before the host knows the length (32^3 without cells 41 us; with a look at the
// list 57).
constexpr uint32_t PSI_FEW_POINTS = 1u << 18;
struct PsiInfo {
    uint32_t count, runs, kinds;   // kinds > PSI_KINDS: not tabulated
    uint32_t lo[3], hi[3];         // bounds of the cells
    float m[PSI_KINDS][3];
};
struct PsiTable {
    float* T;
    const uint2* runs;
    uint32_t nruns, tx, ty, tz;    // T is [kind][z][x][y], of ty the first ny are used
    uint32_t ny;
    int x0, y0, z0;                // the first differences
    float m[PSI_KINDS][3];
};

constexpr unsigned RED_BLOCK = 256;

// Cells per thread of the E/B update: each staged source is applied to
// EB_CPT cells held in registers.
constexpr uint32_t EB_CPT = 4;
// The E/B update walks a domain in aligned bricks of EB_BX x EB_BY x EB_CPT
// cells (1024 = 256 threads x EB_CPT); thread t of a 256-thread block holds
// the cells (t % EB_BX, t / EB_BX, 0..EB_CPT-1) of its brick, a 128-thread
// block one half of a brick (sub = 0, 1 in y).  FAST coordinates are taken
// relative to the brick's centre, which depends only on the cell.
constexpr uint32_t EB_BX = 16, EB_BY = 16;
// LOD bins summed together by one block, neighbours along x: eight of 16^3 bins, fewer of the
// coarser levels, whose 512 or 64 bins would leave most SMs without a block (128^3 at depth 3:
// 49 us with eight, 23 us with two)
__host__ __device__ constexpr uint32_t lod_bins_per_block(uint32_t nd) { return nd >= 16u ? 8u : nd == 8u ? 2u : 1u; }
inline uint32_t lod_blocks(uint32_t nd) { return nd / lod_bins_per_block(nd) * nd * nd; }
inline uint32_t eb_bricks(uint32_t nx, uint32_t ny, uint32_t nz) {
    return ((nx + EB_BX - 1) / EB_BX) * ((ny + EB_BY - 1) / EB_BY) * ((nz + EB_CPT - 1) / EB_CPT);
}

// device view of a batch of domains (batch_kernels.cu)
struct BatchDev {
    const DevLbm* doms;
    uint32_t ndom;
    const uint32_t* tile_off;  // [ndom+1] prefix sums of ceil(n / (EB_CPT * blockDim)) (stream_collide tiles)
    uint32_t total_tiles;
    const uint32_t* brick_off;  // [ndom+1] prefix sums of bricks x (256 / blockDim) (E/B tiles)
    uint32_t total_bricks;
    const uint32_t* bin_off;   // [ndom+1] prefix sums of lod_blocks (LOD bin groups; 1 at depth 0)
    uint32_t total_bins;
    uint32_t* err;
    const uint32_t* row_off;   // [ndom+1] prefix sums of the groups of rows (the row-staged stencil), or null
    uint32_t total_rows;       // 0: the stencil runs in tiles of cells with global loads
};
// threads per block of the batch's stencil kernel (its tiles: BATCH_SC_THREADS * EB_CPT cells;
// row-staged: BATCH_SC_THREADS - 32 compute threads, so rows of up to BATCH_ROW_MAX cells,
// staged at a row stride of BATCH_ROW_STRIDE elements: 96 x 4 bytes keeps every stream
// 16-byte aligned, and the smaller buffers fit five CTAs per SM in FP32 MHD)
constexpr uint32_t BATCH_SC_THREADS = 128;
constexpr uint32_t BATCH_ROW_MAX = BATCH_SC_THREADS - 32, BATCH_ROW_STRIDE = BATCH_ROW_MAX;
static_assert(BATCH_ROW_STRIDE % 16 == 0, "row streams of 16-byte multiples in shared memory");
int batch_max_blocks_per_sm(int ft, bool mhd, bool fast, bool rows, int block);
cudaError_t launch_batch_step(const BatchDev& B, int ft, bool mhd, bool fast, uint32_t grid, uint32_t block,
                              uint64_t t, cudaStream_t s);

// the direct field sum of the domains (256-thread bricks) whose gate is set
cudaError_t launch_batch_gated(const BatchDev& B, const uint32_t* const* gates, uint32_t grid, cudaStream_t s);

// per velocity set (lbm_q19.cu, lbm_q15.cu, lbm_q9.cu)
#define ION_DECLARE_LBM_DISPATCH(NAME)                                                                    \
    void NAME##_stream_collide(const DevLbm& L, int ft, int mode, bool trt, uint64_t t, uint32_t* err,       \
                               cudaStream_t s);                                                            \
    void NAME##_initialize(const DevLbm& L, int ft, int mode, cudaStream_t s);                            \
    void NAME##_update_fields(const DevLbm& L, int ft, uint64_t t, cudaStream_t s);
ION_DECLARE_LBM_DISPATCH(q19)
ION_DECLARE_LBM_DISPATCH(q15)
ION_DECLARE_LBM_DISPATCH(q9)

void launch_lod_bins(const DevLbm& L, cudaStream_t s);
void launch_update_e_b(const DevLbm& L, bool fast, uint32_t* err, cudaStream_t s);
void launch_div_check(uint64_t samples, uint64_t seed, unsigned long long* bad, float* first_bad, cudaStream_t s);
// gate: null, or nothing runs while *gate is 0; direct: null, or FftField::direct, nothing runs while
// all its words are 0
void launch_update_e_b_gated(const DevLbm& L, uint32_t* err, const uint32_t* gate, const uint32_t* direct, cudaStream_t s);
void launch_voxelize(const DevLbm& L, const VoxArgs& A, cudaStream_t s);
void launch_compact(const DevLbm& L, uint8_t mask, uint32_t* tiles, uint32_t* list, uint32_t* total, cudaStream_t s);
// the potential summed directly and the static field, of a list of fewer than `below` cells; its length to
// info->count (where given)
void launch_psi_static_b(const DevLbm& L, const uint32_t* mags, const uint32_t* count, uint32_t below, PsiInfo* info,
                         cudaStream_t s);
// runs of the list; the table's size for them; the table, the potential and the static field
void launch_psi_runs(const DevLbm& L, const uint32_t* list, const uint32_t* count, uint2* runs, uint32_t max_runs,
                     uint32_t from, PsiInfo* info, cudaStream_t s);
// the length from which a list's runs are worth a look, and whether they pay for the table (of `entries` terms)
uint32_t psi_table_from(const DevLbm& L);
bool psi_table_pays(const DevLbm& L, const PsiInfo& I, size_t entries);
size_t psi_table_size(const DevLbm& L, const PsiInfo& I, PsiTable& P);
void launch_psi_table_static_b(const DevLbm& L, const PsiTable& P, uint32_t kinds, const uint32_t* count, cudaStream_t s);
void launch_static_e(const DevLbm& L, const uint32_t* list, const uint32_t* count, float* E, cudaStream_t s);
void launch_sum_f64(const void* x, int ft, uint64_t count, double* partials, uint32_t nparts, double* out,
                    cudaStream_t s);
void launch_fma_probe(float* out, int blocks, int iters, cudaStream_t s);
void launch_codec(int ft, const float* in, uint16_t* enc, float* dec, const uint16_t* raw, float* raw_dec, uint64_t n,
                  cudaStream_t s);

}  // namespace ion

namespace ion {
// error reporting and launch accounting of the C ABI (ion_api.cu)
int api_fail(int code, const char* message);
void api_count_launches(uint64_t n);
}  // namespace ion
