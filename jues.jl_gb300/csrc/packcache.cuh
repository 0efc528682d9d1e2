// Packed-operand cache of a context (gett_tc.cu, gett_e64.cu): scratch planes for transient
// operands, persistent planes for operands declared constant (integrals), dropped explicitly.
#pragma once
#include <cuda_fp16.h>

#include "common.cuh"

namespace jues {

constexpr int E64_NP = 7;   // digit planes of gett_e64.cu

struct PackEntry {
    const double *src;
    Mode r, k;
    long long R, K, Rpad, Kpad;
    int np;              // operand planes: 2, 3 (gett_tc.cu) or E64_NP (gett_e64.cu)
    DBuf<__half> buf;
    DBuf<int> exps;
};
struct PackCache {
    bool busy = false;   // inside a cache operation: frees of the cache's own buffers are not lookups
    // a digit product being set up: its kept operands, and whether the transient planes are its own
    const PackEntry *in_use[2] = {nullptr, nullptr};
    bool e64_active = false;
    std::vector<std::unique_ptr<PackEntry>> cached;
    DBuf<__half> scratch[2];
    DBuf<int> scratch_exp[2];
    // buffers of dropped entries, reused by later entries (no cudaFree/cudaMalloc per sweep)
    std::vector<DBuf<__half>> free_planes;
    std::vector<DBuf<int>> free_exps;
    // FP64 digit planes (gett_e64.cu): transient operands, their row exponents, the list of output
    // tiles left to the FP64 pipe
    DBuf<__half> e64_planes[2];
    DBuf<int> e64_exps[2], e64_list;
};

inline bool same_mode(const Mode &a, const Mode &b) {
    return a.d0 == b.d0 && a.d1 == b.d1 && a.s0 == b.s0 && a.s1 == b.s1 && a.s2 == b.s2;
}

template <class T>
inline DBuf<T> take_buffer(Ctx *ctx, std::vector<DBuf<T>> &pool, size_t need) {
    int best = -1;
    for (int i = 0; i < (int)pool.size(); ++i)
        if (pool[i].n >= need && (best < 0 || pool[i].n < pool[best].n)) best = i;
    if (best >= 0 && pool[best].n <= 2 * need) {
        DBuf<T> b = std::move(pool[best]);
        pool.erase(pool.begin() + best);
        return b;
    }
    return DBuf<T>(ctx, need);
}

}  // namespace jues
