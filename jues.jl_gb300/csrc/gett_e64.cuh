// FP64 tensor contraction on the tcgen05 tensor cores (gett_e64.cu).
#pragma once
#include <cuda_fp16.h>

#include "common.cuh"
#include "gett_f64.cuh"

namespace jues {

// C = alpha A.B + beta C as gett_f64, on the tensor cores; false (nothing done) when the sizes or
// the memory left do not suit it and the FP64 pipe should run the contraction
bool gett_e64(Ctx *ctx, const GettArgs &a, const char *name);

// where and how the results of one contraction are stored
struct E64Out {
    double alpha, beta;
    double *C;
    const double *Cin;
    int *list;                  // tiles left to the FP64 pipe: count, then (problem, tile) pairs
    long long row0;             // first row of the panel in the whole output
    long long mtiles_all;       // row tiles of the whole output (tile numbers in the list)
    long long N;                // columns
    int alpha_pow2, alpha_k, alpha_neg;
    int beta_mode;              // 0: C = v; 1: C += v in place; 2: C = Cin + v; 3: C = beta Cin + v
};
// one contraction as the kernels see it
struct E64Args : E64Out {
    long long M;                // rows of this launch's panel
    int rowA, rowB;             // first operand rows in the planes
    int item0;                  // first work item of a grouped launch's problem
    int k16;                    // K steps of 16
    int mtiles, ntiles;         // of this launch
    const int *expA, *expB;     // biased exponent of each row's largest element (0: zero row)
    Mode mC, nC;
    unsigned *flags;
    int ksplit, kper;           // K parts of kper chunks each
    longlong2 *part;            // ksplit > 1: [part][tile][BN][BM] pairs of 64-bit sums
    float *pmag;                // and their sums of magnitudes
};

// digit planes and the magnitude plane, [np + 1][rows][Kpad], of one operand (or of several with the same K, rows
// concatenated)
struct E64Planes {
    DBuf<__half> planes;
    DBuf<int> exps;
    long long rows = 0, K = 0, Kpad = 0;
    int np = 0;
};
// np = 7 digit planes (FP64) or 3 (27 bits: split precision)
void e64_alloc(Ctx *ctx, E64Planes &P, long long rows, long long K, int np);
void e64_pack(Ctx *ctx, E64Planes &P, const double *src, const Mode &rm, const Mode &km, long long R);
// C[mC(m) + nC(n)] = alpha sum_k A[rowA + m, k] B[rowB + n, k] + beta C, beta 0 or 1; item0: the items of
// the problems before it in the launch (e64_tiles each)
E64Args e64_problem(Ctx *ctx, const E64Planes &A, const E64Planes &B, long long K, long long rowA, long long M,
                    long long rowB, long long N, double alpha, double beta, double *C, const Mode &mC, const Mode &nC, int item0,
                    int *list);
inline long long e64_tiles(long long M, long long N) { return ((M + 127) / 128) * ((N + 31) / 32); }
// one launch over n problems (device tables: probs, and f64 the same contractions for the FP64 pipe);
// list holds 4 items + 1 ints
void e64_group_run(Ctx *ctx, const E64Planes &A, const E64Planes &B, const E64Args *probs, const GroupProblem *f64,
                   int n, long long items, int *list, const char *name);

// A stage of a batch (K <= 128 throughout).  Stages run one after another, so their operands go through one
// set of planes: reserve sizes it for the largest of the stages that suit it and fit the memory left; build gives
// null for the others
struct E64Group;
struct E64Shared {
    DBuf<__half> planes[2];
    DBuf<int> exps[2], list;
};
void e64_shared_reserve(Ctx *ctx, E64Shared &sh, const std::vector<const std::vector<GettArgs> *> &stages);
E64Group *e64_group_build(Ctx *ctx, const std::vector<GettArgs> &probs, const E64Shared &sh, const char *name);
void e64_group_exec(Ctx *ctx, E64Group *g);
void e64_group_destroy(E64Group *g);

// gett_f64.cu: recompute the listed output tiles on the FP64 pipe.  list[0] = count, then pairs
// (problem, tile t): rows [128 (t % mt), + 128), columns [16 (t / mt), + 16) of the problem's output, mt =
// its 128-row tiles; the problem is *one, or probs[problem] (device)
void gett_f64_tiles(Ctx *ctx, const GettArgs *one, const GroupProblem *probs, const int *list, const char *name);

}  // namespace jues
