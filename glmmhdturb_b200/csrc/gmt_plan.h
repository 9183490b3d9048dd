// gmt_plan.h -- how a step is cut up for its grid: rules of sizes only, plain C++ without CUDA.
#pragma once
#include <algorithm>
#include <cstddef>

namespace gmt {

// --- the FP64 step's passes (gmt_passes.cuh) -----------------------------------------------------
constexpr int PASS_TX = 16, PASS_TY = 8;   // columns per block of the flux pass
constexpr size_t PASS_SCRATCH_BYTES = (size_t)1 << 30;   // of a context, or of all lanes of an ensemble
constexpr int GRID_YZ = 65535;             // largest gridDim.y and gridDim.z

// scratch of a slab of S planes: primitives of S + 4 planes, predictors of S + 2, PPM's flags
inline size_t passes_scratch_bytes(int nx, int ny, int S) {
    return (size_t)nx * ny * ((size_t)9 * (2 * S + 6) * sizeof(double) + (S + 2));
}

// planes per slab of the FP64 step's passes: slabs of equal thickness whose scratch stays within `budget`,
// cut down to three or four planes; 0, the tile march, where even those exceed it (1 GB: cross sections
// above about 1029^2).  A slab repeats the primitives of four planes and the predictors of two, so
// thick ones: 256^3 8.60 ms within 1 GB, 8.94 ms within 256 MB, 10.7 ms within 64 MB (4 planes), which L2
// would hold; the march takes 14.1 ms.
// The passes put a slab's planes, and the flux pass its rows of tiles, in gridDim.y: a narrow box of many
// planes has more slabs than its scratch asks for, and one of too many rows none.
inline int pass_slab(int nx, int ny, int nz, size_t budget) {
    if (((long)ny + PASS_TY - 1) / PASS_TY > GRID_YZ) return 0;
    long slabs = 1;
    auto planes = [&] { return (int)((nz + slabs - 1) / slabs); };
    auto over = [&] { return passes_scratch_bytes(nx, ny, planes()) > budget; };
    while (planes() > GRID_YZ - 4 || (planes() > 4 && over())) ++slabs;
    return over() ? 0 : planes();
}

}  // namespace gmt
