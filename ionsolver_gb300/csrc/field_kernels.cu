// field_kernels.cu -- launchers of the LOD-bin and E/B kernels (field_kernels.cuh).
#include "field_kernels.cuh"

namespace ion {

void launch_lod_bins(const DevLbm& L, cudaStream_t s) {
    k_lod_bins<<<lod_blocks(L.nd), LB_THREADS, 0, s>>>(L);
}

void launch_update_e_b_gated(const DevLbm& L, uint32_t* err, const uint32_t* gate, const uint32_t* direct, cudaStream_t s) {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const uint32_t bricks = eb_bricks(L.nx, L.ny, L.nz), resident = 2u * (uint32_t)(sms > 0 ? sms : 1);
    k_update_e_b_gated<<<bricks < resident ? bricks : resident, 256, 0, s>>>(L, err, gate, direct, bricks);
}

void launch_update_e_b(const DevLbm& L, bool fast, uint32_t* err, cudaStream_t s) {
    const unsigned g = eb_bricks(L.nx, L.ny, L.nz);
    if (fast) k_update_e_b_fast<<<g, 256, 0, s>>>(L, err);
    else k_update_e_b_exact<<<g, 256, 0, s>>>(L, err);
}

}  // namespace ion
