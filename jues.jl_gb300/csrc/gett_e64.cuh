// FP64 tensor contraction on the tcgen05 tensor cores (gett_e64.cu).
#pragma once
#include <cuda_fp16.h>

#include "common.cuh"
#include "gett_f64.cuh"

namespace jues {

// C = alpha A.B + beta C as gett_f64, on the tensor cores; false (nothing done) when the sizes or
// the memory left do not suit it and the FP64 pipe should run the contraction
bool gett_e64(Ctx *ctx, const GettArgs &a, const char *name);

// Results left to the FP64 pipe, in ints: the counts of whole half tiles (128 x 16) and of half tiles with few
// elements left out, (problem, tile) pairs of the first, then E64_FINE_INTS for each of the second: problem, tile,
// count of pieces, and the pieces, a row's eight columns each: row | column group << 7 | left-out columns << 8
constexpr int E64_FINE = 64, E64_FINE_INTS = 3 + E64_FINE / 2;
inline size_t e64_list_ints(long long tiles) { return 2 + 2 * (size_t)tiles * (2 + E64_FINE_INTS); }   // of 128 x 32

// where and how the results of one contraction are stored
struct E64Out {
    double alpha, beta;
    double *C;
    const double *Cin;
    int *list, *fine;           // results left to the FP64 pipe; the half tiles with few of them
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
                    int *list, long long list_tiles);
inline long long e64_tiles(long long M, long long N) { return ((M + 127) / 128) * ((N + 31) / 32); }
// one launch over n problems (device tables: probs, and f64 the same contractions for the FP64 pipe);
// list has room for list_tiles >= items tiles (as the problems were told)
void e64_group_run(Ctx *ctx, const E64Planes &A, const E64Planes &B, const E64Args *probs, const GroupProblem *f64,
                   int n, long long items, int *list, long long list_tiles, const char *name);

// A stage of a batch (K <= 128 throughout).  Stages run one after another, so their operands go through one
// set of planes: reserve sizes it for the largest of the stages that suit it and fit the memory left; build gives
// null for the others
struct E64Group;
struct E64Shared {
    DBuf<__half> planes[2];
    DBuf<int> exps[2], list;
    long long list_tiles = 0;
};
void e64_shared_reserve(Ctx *ctx, E64Shared &sh, const std::vector<const std::vector<GettArgs> *> &stages);
E64Group *e64_group_build(Ctx *ctx, const std::vector<GettArgs> &probs, const E64Shared &sh, const char *name);
void e64_group_exec(Ctx *ctx, E64Group *g);
void e64_group_destroy(E64Group *g);

// gett_f64.cu: recompute the listed results on the FP64 pipe.  Tile t of a problem is its rows
// [128 (t % mt), + 128), columns [16 (t / mt), + 16), mt = its 128-row tiles; the problem is *one, or probs[problem]
// (device)
void gett_f64_tiles(Ctx *ctx, const GettArgs *one, const GroupProblem *probs, const int *list, long long list_tiles,
                    const char *name);

}  // namespace jues
