// field_table.h -- the BITWISE E/B field from tabulated R/|R|^3 (field_table.cu).
#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

namespace ion {

struct DevLbm;

// R/|R|^3 between cells and bin centres, (x, y, z, 0): of every distance |2 R|, [z][y][x]; or, in
// bins, of every difference D of two bins and in-bin offset, [Dz][Dy][Dx][offset]
struct FieldTable {
    float4* T = nullptr;
    uint32_t tx = 0, ty = 0, tz = 0;
    bool in_bins = false;
};

bool field_table_fits(const DevLbm& L);
size_t field_table_size(const DevLbm& L, FieldTable& F);
cudaError_t launch_field_table(const DevLbm& L, const FieldTable& F, cudaStream_t s);
cudaError_t launch_update_e_b_table(const DevLbm& L, const FieldTable& F, cudaStream_t s);

}  // namespace ion
