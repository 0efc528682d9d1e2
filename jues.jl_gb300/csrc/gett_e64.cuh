// FP64 tensor contraction on the tcgen05 tensor cores (gett_e64.cu).
#pragma once
#include "common.cuh"

namespace jues {

// C = alpha A.B + beta C as gett_f64, on the tensor cores; false (nothing done) when the sizes or
// the memory left do not suit it and the FP64 pipe should run the contraction
bool gett_e64(Ctx *ctx, const GettArgs &a, const char *name);

// gett_f64.cu: recompute the listed output tiles on the FP64 pipe.  list[0] = count, then tile
// numbers t: rows [128 (t % mtiles), + 128), columns [32 (t / mtiles), + 32) of g's output.
void gett_f64_tiles(Ctx *ctx, const GettArgs &g, const int *list, long long mtiles, const char *name);

}  // namespace jues
