// Host-side check of the resident solve's classes (ariel_b200/csrc/pcg.cuh): res_class_mask() has
// the class of every FLUID count that a grid of this size allows and that a block can hold, and no
// other, so that a handle loads and launches what its scenes can reach.  Runs on the CPU only;
// prints "ok" and exits 0 when all hold.
#include <cstdio>

#include "pcg.cuh"

using namespace ariel;

int main() {
    for (int n : {2, 8, 13, 20, 32, 53, 54, 64, 66, 67, 77, 85, 86, 97, 107, 128, 160, 256}) {
        const long long cells = (long long)n * n * n;
        for (int mode : {kRef32, kFp64, kMixed})
            for (int scenes : {1, 2, 128}) {
                int want = 0;
                for (long long nf = 0; nf <= cells; ++nf) {
                    const int cs = chunk_size(nf), chunks = (int)((nf + cs - 1) / cs);
                    if (mode == kRef32 || (mode == kFp64 && scenes > 1)) continue;
                    if (res_max_cpb(mode, scenes, cs, chunks) > 0) want |= 1 << res_class(scenes, cs, chunks);
                }
                const int got = res_class_mask(mode, scenes, cells);
                if (got != want || (mode == kFp64 && (got & ~(1 | 8)))) {
                    std::printf("%d^3, mode %d, %d scenes: classes %x, reached %x\n", n, mode, scenes, got, want);
                    return 1;
                }
            }
    }
    std::printf("ok\n");
    return 0;
}
