// Prints what the rules of gmt_plan.h choose.  One query per line of standard input, one answer per line:
//   slab nx ny nz lanes -> planes per slab of the FP64 passes of one of `lanes` lanes, bytes of their scratch
//   lanes units mean_zones -> lanes of an FP64 ensemble
//   batch esize n count mean_zones -> boxes of n^3 in one launch of an ensemble
//   chunk cols nz esize threads -> planes per block of a tile march
#include <cstdio>
#include <cstring>

#include "../../glmmhdturb_b200/csrc/gmt_plan.h"

int main() {
    char what[32];
    while (std::scanf("%31s", what) == 1) {
        if (!std::strcmp(what, "slab")) {
            int nx, ny, nz, lanes;
            if (std::scanf("%d %d %d %d", &nx, &ny, &nz, &lanes) != 4) return 1;
            const int S = gmt::pass_slab(nx, ny, nz, gmt::PASS_SCRATCH_BYTES / lanes);
            std::printf("%d %zu\n", S, S > 0 ? gmt::passes_scratch_bytes(nx, ny, S) : (size_t)0);
        } else if (!std::strcmp(what, "lanes")) {
            int units;
            size_t zones;
            if (std::scanf("%d %zu", &units, &zones) != 2) return 1;
            std::printf("%d\n", gmt::pass_lanes(units, zones));
        } else if (!std::strcmp(what, "batch")) {
            int esize, n, count;
            size_t zones;
            if (std::scanf("%d %d %d %zu", &esize, &n, &count, &zones) != 4) return 1;
            std::printf("%d\n", gmt::ens_batch(esize, n, count, zones));
        } else if (!std::strcmp(what, "chunk")) {
            long cols;
            int nz, esize, threads;
            if (std::scanf("%ld %d %d %d", &cols, &nz, &esize, &threads) != 4) return 1;
            std::printf("%d\n", gmt::choose_chunk(cols, nz, esize, threads));
        } else {
            return 1;
        }
    }
    return 0;
}
