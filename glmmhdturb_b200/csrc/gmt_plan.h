// gmt_plan.h -- how a step is cut up for its grid: rules of sizes only, plain C++ without CUDA.
#pragma once
#include <algorithm>
#include <cmath>
#include <cstddef>

namespace gmt {

// --- the FP64 step's passes (gmt_passes.cuh) -----------------------------------------------------
constexpr int PASS_TX = 16, PASS_TY = 8;   // columns per block of the flux pass
constexpr int PASS_MINB = 4;               // its blocks on an SM
constexpr size_t PASS_SCRATCH_BYTES = (size_t)1 << 30;   // of a context, or of all lanes of an ensemble
constexpr size_t PASS_OVERLAP_ZONES = (size_t)40 * 40 * 40;   // boxes below: steps on several streams overlap
constexpr int GRID_YZ = 65535;             // largest gridDim.y and gridDim.z

// scratch of a slab of S planes: primitives of S + 4 planes, predictors of S + 2, PPM's flags
inline size_t passes_scratch_bytes(int nx, int ny, int S) {
    return (size_t)nx * ny * ((size_t)9 * (2 * S + 6) * sizeof(double) + (S + 2));
}

// planes per slab of the FP64 step's passes: slabs of equal thickness whose scratch stays within `budget`,
// cut down to three or four planes; 0, the tile march, where even those exceed it (1 GB: cross sections
// above about 1029^2).  A slab repeats the primitives of four planes and the predictors of two, so
// thick ones: 256^3 7.99 ms within 1 GB, 8.29 ms within 256 MB, 9.91 ms within 64 MB (4 planes), which L2
// would hold; the march takes 13.7 ms.
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

// Lanes (streams with scratch of their own) of an FP64 ensemble: four, or two where a fourth of the budget
// would cut a box of the mean size into slabs.  ms a step with 1, 2, 4, 8, 16 lanes: 16 boxes of 32^3 1.59, 0.86,
// 0.52, 0.40, 0.39; 8 of 96^3 3.80, 3.49, 3.54, 3.55, 3.56; cut into slabs from four lanes on, 6 of 128^3 6.57,
// 6.09, 6.32, 6.33, 6.34, and 4 of 192^3 13.96, 13.58, 14.07, 14.08, 14.09 (two slabs with two lanes).  Small
// boxes beside large ones need the four: 60 of 32^3 and 4 of 128^3 7.28 with two, 5.98 with four.
inline int pass_lanes(int units, size_t mean_zones) {
    const int n = (int)std::cbrt((double)mean_zones), lanes = std::min(units, 4);
    return passes_scratch_bytes(n, n, n) <= PASS_SCRATCH_BYTES / lanes ? lanes : std::min(units, 2);
}

// planes per block of the flux pass over a slab of S planes: the extra z face of a chunk costs a third of a
// plane, so long chunks, but enough blocks for several rounds of PASS_MINB blocks on every SM
inline int pass_flux_planes(int nx, int ny, int S) {
    const long bx = (nx + PASS_TX - 1) / PASS_TX, by = (ny + PASS_TY - 1) / PASS_TY;
    int lz = S;
    while (lz > 4 && bx * by * ((S + lz - 1) / lz) < 148L * PASS_MINB * 3) lz = (lz + 1) / 2;
    return lz;
}

// --- ensembles -----------------------------------------------------------------------------------
// How many of `count` boxes of n^3 one launch takes: small boxes by the dozen finish sooner than a launch, a tick
// and a table for each of them can be started (us a step, own launches -> together, and a persistent kernel
// over a queue of all boxes' tiles: FP32 512 of 16^3 1297 -> 413, 713; 64 and 256 of 32^3 342 -> 280, 286, and 1231
// -> 888, 1068; FP64 256 of 16^3 6075 -> 1017, 1439).
// FP32: 16^3 and 32^3, in ensembles whose mean box is below 40^3.  Among larger boxes the small ones fill gaps
// better one by one (mean box 79k zones 132 -> 141, 132k 506 -> 550; 73k 441 -> 417; 64 uneven boxes of 642k 15.67 -> 15.99 ms).
// FP64: 16^3, more of them than lanes (4 of them 99 -> 149, 16 372 -> 152); one by one they run as passes, together
// as the tile march, whose bits are the same, and 32^3 boxes are faster as passes.
constexpr int BATCH_BOXES = 64;
inline int ens_batch(int esize, int n, int count, size_t mean_zones) {
    const bool small = esize == 8 ? n <= 16 && count > 4 : n <= 32 && mean_zones < (size_t)40 * 40 * 40;
    return small ? std::min(count, BATCH_BOXES) : 1;
}

// --- z chunks of the tile marches ----------------------------------------------------------------
// Planes per block of `threads` columns in reals of `esize` bytes, `cols` tiles wide: the z chunk that fills the
// chip best.
//
// A tile whose block fills an SM (FP32 above 256 threads, of 128 registers; FP64 from 128 threads, by its
// shared memory; the automatic tiles are all of this kind): the number of rounds of blocks over the 148 SMs
// times the length of a block.  Short chunks repeat the fixed part, long ones leave SMs idle in the last round;
// with more than one round a share of a block's time is added, because blocks do not end together.
// The constants are fitted to the FP32 MC + HLLD step and to FP64 sweeps of the march and CT.  FP32 PPM, minmod, the march
// and CT use them unfitted: 8^3 to 256^3 they take 0.55 to 1.01 of their times with a rule that asked for eight rounds.
// (FP32 MC + HLLD, chunk -> us: 64^3 4 -> 41, 8 -> 66; 96^3 12 -> 92, 6 -> 105; 192^3 32 -> 694,
// 6 -> 833; 256^3 32 -> 1549, 16 -> 1623; 512^3 128 -> 11.59 ms, 64 and 256 -> 11.70 ms; the second
// figures of the first four are the chunks of a rule that only asked for eight rounds of blocks.)
//
// Of smaller tiles, which a caller may choose, several blocks share an SM and hide one another's start, and
// one block for each SM leaves most of it idle: halved until there are eight rounds of blocks, or 8 planes.
// (FP32 MC + HLLD, us, that rule -> one block for each SM: 16x8 at 128^3 342 -> 729, 8x8 at 64^3 76 -> 204,
// 32x4 at 128^3 368 -> 747, 16x16 at 256^3 1454 -> 1531; FP64 8x8 at 128x64x96 975 -> 2792.)
inline int choose_chunk(long cols, int nz, int esize, int threads) {
    if (esize == 8 ? threads < 128 : threads <= 256) {
        long lz = nz;
        while (lz > 8 && cols * ((nz + lz - 1) / lz) < 148L * 8) lz = (lz + 1) / 2;
        return (int)lz;
    }
    // a block takes lz planes and 2.8 planes' time for its start and for the first and last planes, which
    // only reconstruct (FP32, 64^3, chunk 4 -> 64: 41 -> 401 us, 6.05 us a plane).  In FP64 a plane is mostly
    // its Riemann solves, which those planes do without: 0.4 to 1.2 planes (chunk sweeps of the march and CT, MC
    // and PPM, 64^3 to 160^3), and no share for the last round.  At 2.8 planes 128^3 got chunks of half the box
    // or all of it where 8 and 16 planes are faster: march PPM 2733 -> 2554 us, CT PPM 5802 -> 5306 us.
    // Four planes at least, which is not the best for a small box that has the chip to itself (32^3: 21 us at 1, 31
    // at 3, 37 at 4; 48^3: 29 at 2, 40 at 4).  The one reason is a test that holds
    // a loop over single boxes to half of the ensemble's rate: at 1 or 2 planes the loop's small boxes reach 5.65
    // against 11.2 Gzone/s, now 5.2.
    const double start = esize == 8 ? 0.8 : 2.8, tail = esize == 8 ? 0.0 : 0.2;
    double best = 1e300;
    int last = 0, choice = nz;
    for (int nch = 1; nch <= std::min(nz, 4096); ++nch) {
        const int lz = (nz + nch - 1) / nch;
        if (lz == last || (lz < 4 && nch > 1)) continue;
        last = lz;
        const long rounds = (cols * (((long)nz + lz - 1) / lz) + 147) / 148;
        const double cost = ((double)rounds + (rounds > 1 ? tail : 0.0)) * (lz + start);
        if (cost < best) { best = cost; choice = lz; }
    }
    return choice;
}

}  // namespace gmt
