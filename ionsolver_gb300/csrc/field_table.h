// field_table.h -- the BITWISE E/B field from tabulated R/|R|^3 (field_table.cu).
#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

namespace ion {

struct DevLbm;

// R/|R|^3 of every distance |2 R| between a cell and a bin centre: [z][y][x], (x, y, z, 0)
struct FieldTable {
    float4* T = nullptr;
    uint32_t tx = 0, ty = 0, tz = 0;
};

bool field_table_fits(const DevLbm& L);
size_t field_table_size(const DevLbm& L, FieldTable& F);
cudaError_t launch_field_table(const DevLbm& L, const FieldTable& F, cudaStream_t s);
cudaError_t launch_update_e_b_table(const DevLbm& L, const FieldTable& F, cudaStream_t s);

}  // namespace ion
