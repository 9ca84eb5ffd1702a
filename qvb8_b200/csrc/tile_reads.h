// How many bytes of a packed row a copy may take: host arithmetic that the kernels use as it stands (no CUDA in here, so a
// test compiles it for the host).
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define QV_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define QV_HOST_DEVICE inline
#endif

namespace qv {

// 16-byte vectors of a row of nb-bit ids (16-byte aligned) in its next stage of at most `stage` columns, `left` columns from
// the row's end; both are multiples of 128, so the vectors end where the columns do.
QV_HOST_DEVICE constexpr int row_stage_vecs(int left, int stage, int nb) { return (left < stage ? left : stage) / 128 * nb; }

constexpr bool row_stage_vecs_fit(int stage) {
    for (int nb = 3; nb <= 8; ++nb)
        for (int left = 128; left <= 2 * stage; left += 128) {
            const int v = row_stage_vecs(left, stage, nb), columns = left < stage ? left : stage;
            if (v * 128 != columns * nb) return false;                 // exactly the columns' bytes: none beyond the row
        }
    return true;
}

}  // namespace qv
