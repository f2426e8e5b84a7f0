// Misuse that cuda_emul.h has to report. Test infrastructure only.
#include "cuda_emul.h"

// What is wrong with a CTA of two warps that hand something to and fro (null:
// nothing); kind: the mistake in it.
extern "C" const char* emul_check(int kind, uint64_t seed) {
    const bool ok = emul::run(64, seed, [&] {
        const uint32_t t = threadIdx.x;
        for (uint32_t i = 0; i < 3; ++i) {
            if (t < 32) {
                cdb::bar_arrive(1, 64);
                if (kind == 1 && i == 1) continue;  // overtakes a late second warp
                cdb::bar_sync(2, 64);
            } else {
                cdb::bar_sync(1, kind == 2 && i == 2 ? 96 : 64);
                if (kind == 1 && i == 1) continue;
                if (kind == 3 && i == 2) break;
                cdb::bar_arrive(2, 64);
            }
        }
        if (kind == 4 && t % 2) __syncwarp();
        else (void)__shfl_sync(0xffffffffu, t, 0);
    });
    return ok ? nullptr : emul::cta()->bad;
}
