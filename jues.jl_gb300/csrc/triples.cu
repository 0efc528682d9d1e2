// Closed-shell (T) energy correction (src/CoupledCluster/PerturbativeTriples.jl:35-138).
//
// The reference loops over occupied triples i >= j >= k and builds W[a,b,c] (v^3) from twelve
// small contractions per triple.  They are six orderings (p,x),(q,y),(r,u) of (i,a),(j,b),(k,c) of one
// function,
//     F_pqr[x,y,u] = sum_d (yd|xp) T2[r,q,u,d] - sum_l (ur|ql) T2[p,l,x,y],
// a single contraction over the stacked index (d | l) with the rows R[(x,y,p)] = [(yd|xp) | -T2[p,l,x,y]] and
// the columns Q[(u,r,q)] = [T2[r,q,u,d] | (ur|ql)].  Both are formed and cut into digit planes once
// (gett_e64.cu: seven planes for FP64, three for the split forms); every contraction is then a range of
// their rows, so the six of many (i, j) pairs with all k <= j run as six grouped launches that add into
// W[a,b,c,k] through the output modes, and one kernel forms V = W + the three (vo|vo) T1 terms on the
// fly and sums the reference's weighted energy expression over a >= b >= c (:117-131).  The twelve
// contractions per pair took 48 launches with their packs; at o = 12, v = 48 the call took 31 ms.
// A row of R and a column of Q each hold integrals beside amplitudes under one scale of the digits, so the
// amplitudes enter both as sigma T2, sigma the power of two that brings their largest element to the integrals'
// (a factor of sigma on W, taken off with alpha): with amplitudes far smaller than the integrals the digits of
// half of each row would else be lost and its contractions redone on the FP64 pipe (T2 2^-10 of the size that it
// has beside these integrals, o = 12, v = 48: 34 ms, with sigma 4.0).
// Partial sums go to fixed per-block slots that are added in a fixed order, and the six additions
// to W are ordered by their launches, so the result is deterministic.
#include <algorithm>
#include <cmath>
#include <memory>
#include <vector>

#include "gett_e64.cuh"
#include "triples.cuh"

namespace jues {

namespace {

constexpr int PT_THREADS = 256;
constexpr int PT_BLOCKS = 152 * 4;
constexpr int PT_T = 8, PT_P1 = 9, PT_P2 = 73;   // tile edge; pitches of a tile cube (free of bank conflicts)

// one (i, j, k): W[a,b,c] at w0
struct PtItem {
    int i, j, k;
    long long w0;
};

__device__ __forceinline__ double pt_warp_sum(double x) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) x += __shfl_down_sync(0xffffffffu, x, d);
    return x;
}

// Work item: one (i, j, k) and one triple of 8-wide virtual tiles A >= B >= C.  The six orderings of
// the tile triple are loaded as 8^3 cubes (64-byte runs of W's unit-stride index; a gather of the six
// orderings per thread read 32-byte sectors for 8 bytes), so W is read once.  FP64 issue bounds it (about 70
// operations a point), so tile triples on a diagonal go through lists of their a >= b >= c, which fill the
// warps: 288 of 512 points with two equal tiles, 120 with three (o = 12, v = 48: 1.28 -> 0.97 ms).
__global__ void __launch_bounds__(PT_THREADS) pt_energy_kernel(const double *__restrict__ W,
                                                               const PtItem *__restrict__ items, int nitems,
                                                               const int *__restrict__ tiles, int ntiles,
                                                               const double *__restrict__ T1, View4 Vvovo,
                                                               const double *__restrict__ fo,
                                                               const double *__restrict__ fv, int o, int v,
                                                               double *slots) {
    __shared__ double cube[6][PT_T * PT_P2], vo[3][6][PT_T * PT_T], t1s[3][3][PT_T], fvs[3][PT_T];
    const long long v2 = (long long)v * v;
    const long long *S = Vvovo.s;
    const int tid = threadIdx.x;
    const long long total = (long long)nitems * ntiles;
    double acc = 0.0;
    // the points a + 8 b + 64 c of tile triples A = B > C, A > B = C and A = B = C
    constexpr int PAIR = PT_T * (PT_T + 1) / 2, CUBE = PT_T * (PT_T + 1) * (PT_T + 2) / 6;
    __shared__ unsigned short points[2 * PT_T * PAIR + CUBE];
    for (int e = tid; e < PT_T * PT_T * PT_T; e += PT_THREADS) {
        const int a = e & 7, b = (e >> 3) & 7, c = e >> 6;
        if (a >= b) points[c * PAIR + a * (a + 1) / 2 + b] = (unsigned short)e;
        if (b >= c) points[PT_T * PAIR + (b * (b + 1) / 2 + c) * PT_T + a] = (unsigned short)e;
        if (a >= b && b >= c) points[2 * PT_T * PAIR + a * (a + 1) * (a + 2) / 6 + b * (b + 1) / 2 + c] = (unsigned short)e;
    }
    for (long long w = blockIdx.x; w < total; w += gridDim.x) {
        const PtItem it = items[w / ntiles];
        const int pk = tiles[w % ntiles];
        const int org[3] = {(pk & 1023) * PT_T, (pk >> 10 & 1023) * PT_T, (pk >> 20) * PT_T};
        const int occ[3] = {it.i, it.j, it.k};
        const double *Wk = W + it.w0;
        __syncthreads();   // the previous item is done with the tiles
        // orderings abc, acb, bac, bca, cab, cba
        constexpr int P0[6] = {0, 0, 1, 1, 2, 2}, P1[6] = {1, 2, 0, 2, 0, 1}, P2[6] = {2, 1, 2, 0, 1, 0};
#pragma unroll
        for (int n = 0; n < 12; ++n) {
            const int p = n >> 1, e = tid + 256 * (n & 1);
            const int x = e & 7, y = (e >> 3) & 7, z = e >> 6;
            const int gx = org[P0[p]] + x, gy = org[P1[p]] + y, gz = org[P2[p]] + z;
            cube[p][x + PT_P1 * y + PT_P2 * z] =
                (gx < v && gy < v && gz < v) ? Wk[gx + (long long)v * gy + v2 * gz] : 0.0;
        }
        // (vo|vo) tiles of the ordered tile pairs ab, ac, ba, bc, ca, cb: [x,j,y,k], [x,i,y,k], [x,i,y,j]
        constexpr int Q0[6] = {0, 0, 1, 1, 2, 2}, Q1[6] = {1, 2, 0, 2, 0, 1}, M0[3] = {1, 0, 0}, M1[3] = {2, 2, 1};
        for (int n = tid; n < 18 * 64; n += PT_THREADS) {
            const int m = n / 384, p = (n >> 6) % 6, x = n & 7, y = (n >> 3) & 7;
            const int gx = org[Q0[p]] + x, gy = org[Q1[p]] + y;
            vo[m][p][x + 8 * y] =
                (gx < v && gy < v) ? Vvovo.p[gx * S[0] + occ[M0[m]] * S[1] + gy * S[2] + occ[M1[m]] * S[3]] : 0.0;
        }
        if (tid < 72) {
            const int m = tid / 24, p = (tid / 8) % 3, gx = org[p] + (tid & 7);
            t1s[m][p][tid & 7] = gx < v ? T1[occ[m] + (long long)o * gx] : 0.0;
            if (m == 0) fvs[p][tid & 7] = gx < v ? fv[gx] : 0.0;
        }
        __syncthreads();
        const double dij = fo[it.i] + fo[it.j] + fo[it.k], num = 2.0 - (it.i == it.j) - (it.j == it.k);
        const bool ab = org[0] == org[1], bc = org[1] == org[2];
        const int count = ab && bc ? CUBE : ab || bc ? PT_T * PAIR : PT_T * PT_T * PT_T;
        const unsigned short *list = points + (ab && bc ? 2 * PT_T * PAIR : bc ? PT_T * PAIR : 0);
        for (int q = tid; q < count; q += PT_THREADS) {
            const int e = ab || bc ? list[q] : q;
            const int a = e & 7, b = (e >> 3) & 7, c = e >> 6;
            const int ga = org[0] + a, gb = org[1] + b, gc = org[2] + c;
            if (ga >= v) continue;   // a >= b >= c by the lists
            const int loc[3] = {a, b, c};
            double wv[6], vv[6];
#pragma unroll
            for (int p = 0; p < 6; ++p) {
                const int x = loc[P0[p]], y = loc[P1[p]], z = loc[P2[p]];
                wv[p] = cube[p][x + PT_P1 * y + PT_P2 * z];
                // V[p,q,r] = W[p,q,r] + Vvovo[q,j,r,k] T1[i,p] + Vvovo[p,i,r,k] T1[j,q] + Vvovo[p,i,q,j] T1[k,r]  (:113)
                auto pair = [&](int s, int t) { return 2 * s + (t > s ? t - 1 : t); };   // index of (s, t) in Q0, Q1
                vv[p] = wv[p] + vo[0][pair(P1[p], P2[p])][y + 8 * z] * t1s[0][P0[p]][x] +
                        vo[1][pair(P0[p], P2[p])][x + 8 * z] * t1s[1][P1[p]][y] +
                        vo[2][pair(P0[p], P1[p])][x + 8 * y] * t1s[2][P2[p]][z];
            }
            // 0 abc, 1 acb, 2 bac, 3 bca, 4 cab, 5 cba
            double X = 0.0;
#pragma unroll
            for (int p = 0; p < 6; ++p) X = fma(wv[p], vv[p], X);
            const double Y = vv[0] + vv[3] + vv[4];
            const double Z = vv[1] + vv[2] + vv[5];
            const double E = (Y - 2.0 * Z) * (wv[0] + wv[3] + wv[4]) + (Z - 2.0 * Y) * (wv[1] + wv[2] + wv[5]) + 3.0 * X;
            const double den = (dij - fvs[0][a] - fvs[1][b] - fvs[2][c]) * (1.0 + (ga == gb) + (gb == gc));
            acc += E * num / den;
        }
    }
    __syncthreads();
    double *sh = &cube[0][0];
    acc = pt_warp_sum(acc);
    if ((tid & 31) == 0) sh[tid >> 5] = acc;
    __syncthreads();
    if (tid < 32) {
        double x = tid < PT_THREADS / 32 ? sh[tid] : 0.0;
        x = pt_warp_sum(x);
        if (tid == 0) slots[blockIdx.x] += x;   // one block per slot, launches in stream order
    }
}

__global__ void pt_sum_slots(const double *slots, int n, double *out) {
    __shared__ double sh[32];
    double x = 0.0;
    for (int s = threadIdx.x; s < n; s += blockDim.x) x += slots[s];
    x = pt_warp_sum(x);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = x;
    __syncthreads();
    if (threadIdx.x < 32) {
        x = threadIdx.x < (int)(blockDim.x >> 5) ? sh[threadIdx.x] : 0.0;
        x = pt_warp_sum(x);
        if (threadIdx.x == 0) *out = x;
    }
}

__global__ void pt_zero(double *p, int n) {
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x) p[s] = 0.0;
}

// one W term: W[(rows),(cols)] (+)= alpha sum_x A[(rows),x] B[x,(cols)]
// A operands that are the same slice for every pair sharing i (or j) are kept packed
// (a_const) and dropped at the end
void term(Ctx *ctx, int prec, long long M, long long N, long long K, double alpha, const double *A, Mode mA, Mode kA,
          const double *B, Mode kB, Mode nB, double beta, double *W, Mode mC, Mode nC, const char *name,
          bool a_const = false) {
    GettArgs g;
    g.M = M; g.N = N; g.K = K;
    g.alpha = alpha; g.beta = beta;
    g.A = A; g.mA = mA; g.kA = kA;
    g.B = B; g.kB = kB; g.nB = nB;
    g.C = W; g.mC = mC; g.nC = nC;
    g.a_const = a_const;
    gett(ctx, prec, g, name);
}

}  // namespace

double pT_flops(int o, int v) {
    const double tr = (double)o * (o + 1) * (o + 2) / 6.0;
    return tr * 12.0 * (double)v * v * v * (double)(v + o);
}

namespace {

// the energy sum of nitems (i, j, k) whose W is formed
void energy(Ctx *ctx, const double *W, const PtItem *items, long long nitems, const DBuf<int> &tiles, const double *T1,
            const View4 &Vvovo, const double *fo, const double *fv, int o, int v, double *slots) {
    Ctx::Scope s(ctx, "pt_energy");
    const long long work = nitems * (long long)tiles.n;
    pt_energy_kernel<<<(unsigned)std::min<long long>(work, PT_BLOCKS), PT_THREADS, 0, ctx->stream>>>(
        W, items, (int)nitems, tiles.p, (int)tiles.n, T1, Vvovo, fo, fv, o, v, slots);
    JUES_CHECK_CUDA(cudaGetLastError());
}

// W of one (i, j) pair and all k <= j by twelve contractions read from the arrays themselves: the form that
// needs no memory beyond W (used when the stacked operands do not fit)
void pair_w(Ctx *ctx, int prec, int i, int j, const double *T2, const View4 &Vv, const View4 &Vo, int o, int v,
            double *w) {
    const long long oo = (long long)o * o, oov = oo * v;
    const long long v2 = (long long)v * v, v3 = v2 * v;
    const long long *V0 = Vv.s, *O0 = Vo.s;
    const long long nk = j + 1;
    const double *Vi = Vv.p + i * V0[3], *Vj = Vv.p + j * V0[3];
    // output modes of the five index groupings of W[a,b,c,k]
    const Mode ab = mode2(v, 1, v), ck = mode2(v, v2, v3);
    const Mode ac = mode2(v, 1, v2), bk = mode2(v, v, v3);
    const Mode ack = mode3(v, v, 1, v2, v3), bck = mode3(v, v, v, v2, v3);
    const Mode bc = mode2(v, v, v2), ak = mode2(v, 1, v3);
    // PerturbativeTriples.jl:104-111; each line below is one term (ijk, ikj, kij, kji, jki, jik)
    // Vvvvo[b,d,a,i] T2[k,j,c,d] -> rows (a,b), cols (c,k)
    term(ctx, prec, v2, v * nk, v, 1.0, Vi, mode2(v, V0[2], V0[0]), plain(V0[1]), T2 + (long long)o * j,
         plain(oov), mode2(v, oo, 1), 0.0, w, ab, ck, "pt_w", true);
    // - Vvooo[c,k,j,l] T2[i,l,a,b] -> rows (a,b), cols (c,k)
    term(ctx, prec, v2, v * nk, o, -1.0, T2 + i, mode2(v, oo, oov), plain(o), Vo.p + j * O0[2],
         plain(O0[3]), mode2(v, O0[0], O0[1]), 1.0, w, ab, ck, "pt_w", true);
    // Vvvvo[c,d,a,i] T2[j,k,b,d] -> rows (a,c), cols (b,k)
    term(ctx, prec, v2, v * nk, v, 1.0, Vi, mode2(v, V0[2], V0[0]), plain(V0[1]), T2 + j, plain(oov),
         mode2(v, oo, o), 1.0, w, ac, bk, "pt_w", true);
    // - Vvooo[b,j,k,l] T2[i,l,a,c] -> rows (a,c), cols (b,k)
    term(ctx, prec, v2, v * nk, o, -1.0, T2 + i, mode2(v, oo, oov), plain(o), Vo.p + j * O0[1],
         plain(O0[3]), mode2(v, O0[0], O0[2]), 1.0, w, ac, bk, "pt_w", true);
    // Vvvvo[a,d,c,k] T2[j,i,b,d] -> rows (a,c,k), cols b
    term(ctx, prec, v2 * nk, v, v, 1.0, Vv.p, mode3(v, v, V0[0], V0[2], V0[3]), plain(V0[1]),
         T2 + j + (long long)o * i, plain(oov), plain(oo), 1.0, w, ack, plain(v), "pt_w");
    // - Vvooo[b,j,i,l] T2[k,l,c,a] -> rows (a,c,k), cols b
    term(ctx, prec, v2 * nk, v, o, -1.0, T2, mode3(v, v, oov, oo, 1), plain(o), Vo.p + j * O0[1] + i * O0[2],
         plain(O0[3]), plain(O0[0]), 1.0, w, ack, plain(v), "pt_w");
    // Vvvvo[b,d,c,k] T2[i,j,a,d] -> rows (b,c,k), cols a
    term(ctx, prec, v2 * nk, v, v, 1.0, Vv.p, mode3(v, v, V0[0], V0[2], V0[3]), plain(V0[1]),
         T2 + i + (long long)o * j, plain(oov), plain(oo), 1.0, w, bck, plain(1), "pt_w");
    // - Vvooo[a,i,j,l] T2[k,l,c,b] -> rows (b,c,k), cols a
    term(ctx, prec, v2 * nk, v, o, -1.0, T2, mode3(v, v, oov, oo, 1), plain(o), Vo.p + i * O0[1] + j * O0[2],
         plain(O0[3]), plain(O0[0]), 1.0, w, bck, plain(1), "pt_w");
    // Vvvvo[c,d,b,j] T2[i,k,a,d] -> rows (b,c), cols (a,k)
    term(ctx, prec, v2, v * nk, v, 1.0, Vj, mode2(v, V0[2], V0[0]), plain(V0[1]), T2 + i, plain(oov),
         mode2(v, oo, o), 1.0, w, bc, ak, "pt_w", true);
    // - Vvooo[a,i,k,l] T2[j,l,b,c] -> rows (b,c), cols (a,k)
    term(ctx, prec, v2, v * nk, o, -1.0, T2 + j, mode2(v, oo, oov), plain(o), Vo.p + i * O0[1],
         plain(O0[3]), mode2(v, O0[0], O0[2]), 1.0, w, bc, ak, "pt_w", true);
    // Vvvvo[a,d,b,j] T2[k,i,c,d] -> rows (a,b), cols (c,k)
    term(ctx, prec, v2, v * nk, v, 1.0, Vj, mode2(v, V0[0], V0[2]), plain(V0[1]), T2 + (long long)o * i,
         plain(oov), mode2(v, oo, 1), 1.0, w, ab, ck, "pt_w", true);
    // - Vvooo[c,k,i,l] T2[j,l,b,a] -> rows (a,b), cols (c,k)
    term(ctx, prec, v2, v * nk, o, -1.0, T2 + j, mode2(v, oov, oo), plain(o), Vo.p + i * O0[2],
         plain(O0[3]), mode2(v, O0[0], O0[1]), 1.0, w, ab, ck, "pt_w", true);
}

// out = max(out, bits of |x|) over the four-index array a of extents d0..d3
__global__ void __launch_bounds__(256) pt_absmax_kernel(View4 a, int d0, int d1, int d2, long long n,
                                                        unsigned long long *out) {
    unsigned long long m = 0;
    for (long long t = blockIdx.x * 256LL + threadIdx.x; t < n; t += 256LL * gridDim.x) {
        const long long t1 = t / d0, t2 = t1 / d1;
        const double x = a.p[t % d0 * a.s[0] + t1 % d1 * a.s[1] + t2 % d2 * a.s[2] + t2 / d2 * a.s[3]];
        m = max(m, (unsigned long long)__double_as_longlong(fabs(x)));
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, d));
    if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

// log2 of sigma: the power of two nearest sqrt(max|Vvvvo| max|Vvooo|) / max|T2|; 0 where one of them is zero or
// not finite
int amplitude_scale(Ctx *ctx, const double *T2, const View4 &Vv, const View4 &Vo, int o, int v) {
    auto *bits = reinterpret_cast<unsigned long long *>(ctx->d_red);
    JUES_CHECK_CUDA(cudaMemsetAsync(bits, 0, 3 * sizeof(*bits), ctx->stream));
    {
        Ctx::Scope s(ctx, "pt_absmax");
        auto run = [&](const View4 &a, int d0, int d1, int d2, int d3, int k) {
            const long long n = (long long)d0 * d1 * d2 * d3;
            pt_absmax_kernel<<<(unsigned)std::min<long long>((n + 1023) / 1024, 152 * 8), 256, 0, ctx->stream>>>(
                a, d0, d1, d2, n, bits + k);
            JUES_CHECK_CUDA(cudaGetLastError());
        };
        run(col_major(T2, o, o, v), o, o, v, v, 0);
        run(Vv, v, v, v, o, 1);
        run(Vo, v, o, o, o, 2);
        ctx->count_launch();
        ctx->count_launch();
    }
    double x[3];
    JUES_CHECK_CUDA(cudaMemcpyAsync(x, bits, sizeof(x), cudaMemcpyDeviceToHost, ctx->stream));
    ctx->sync();
    for (double y : x)
        if (!(y > 0.0) || !std::isfinite(y)) return 0;
    const double l = 0.5 * (std::log2(x[1]) + std::log2(x[2])) - std::log2(x[0]);
    return (int)std::lrint(std::max(-90.0, std::min(90.0, l)));
}

// rows R and columns Q, dense and as digit planes; throws JUES_ENOMEM where they do not fit
struct PtStacks {
    DBuf<double> R, Q;
    E64Planes pr, pq;
    long long rowsR, rowsQ, K;
    double unscale;   // 1 / sigma
    PtStacks(Ctx *ctx, int np, const double *T2, const View4 &Vv, const View4 &Vo, int o, int v) {
        const long long oo = (long long)o * o, oov = oo * v, v2 = (long long)v * v;
        K = v + o;
        rowsR = v2 * o;
        rowsQ = 2 * v * oo;   // (u,r,q) with r fast, then with q fast
        R = DBuf<double>(ctx, (size_t)(rowsR * K));
        Q = DBuf<double>(ctx, (size_t)(rowsQ * K));
        e64_alloc(ctx, pr, rowsR, K, np);
        e64_alloc(ctx, pq, rowsQ, K, np);
        const int ls = amplitude_scale(ctx, T2, Vv, Vo, o, v);
        const double sigma = std::ldexp(1.0, ls);
        unscale = std::ldexp(1.0, -ls);
        const long long *V0 = Vv.s, *O0 = Vo.s;
        // R[x + v y + v^2 p, d] = Vvvvo[y,d,x,p];  R[.., v + l] = -sigma T2[p,l,x,y]
        permute4(ctx, Perm4{{v, v, o, v}, {V0[2], V0[0], V0[3], V0[1]}, {1, v, v2, rowsR}}, 1.0, Vv.p, 0.0, R.p);
        permute4(ctx, Perm4{{v, v, o, o}, {oo, oov, 1, o}, {1, v, v2, rowsR}}, -sigma, T2, 0.0, R.p + rowsR * v);
        for (int h = 0; h < 2; ++h) {
            // Q[u + v r + v o q, d] = sigma T2[r,q,u,d];  Q[.., v + l] = Vvooo[u,r,q,l]; second half: r and q traded
            double *q = Q.p + h * v * oo;
            const long long sr = h ? (long long)v * o : v, sq = h ? v : (long long)v * o;
            permute4(ctx, Perm4{{v, o, o, v}, {oo, 1, o, oov}, {1, sr, sq, rowsQ}}, sigma, T2, 0.0, q);
            permute4(ctx, Perm4{{v, o, o, o}, {O0[0], O0[1], O0[2], O0[3]}, {1, sr, sq, rowsQ}}, 1.0, Vo.p, 0.0,
                     q + rowsQ * v);
        }
        e64_pack(ctx, pr, R.p, plain(1), plain(rowsR), rowsR);
        e64_pack(ctx, pq, Q.p, plain(1), plain(rowsQ), rowsQ);
    }
};

// the six contractions of one pair (PerturbativeTriples.jl:104-111), term t: rows of R, columns of Q and
// the place of (x, y, p | u, r or q) in W[a,b,c,k]
struct PtTerm {
    long long rowA, M, rowB, N;
    Mode mC, nC;
};
PtTerm pt_term(int t, int i, int j, int o, int v) {
    const long long v2 = (long long)v * v, v3 = v2 * v, nk = j + 1, half = (long long)v * o * o, vo = (long long)v * o;
    const long long single = (long long)v * (t == 4 ? j : i) + vo * (t == 4 ? i : j);   // (r, q) of the last two
    switch (t) {
        case 0: return {v2 * i, v2, vo * j, v * nk, mode2(v, 1, v), mode2(v, v2, v3)};           // ijk: (a,b), (c,k)
        case 1: return {v2 * i, v2, half + vo * j, v * nk, mode2(v, 1, v2), mode2(v, v, v3)};    // ikj: (a,c), (b,k)
        case 2: return {v2 * j, v2, vo * i, v * nk, mode2(v, v, 1), mode2(v, v2, v3)};           // jik: (b,a), (c,k)
        case 3: return {v2 * j, v2, half + vo * i, v * nk, mode2(v, v, v2), mode2(v, 1, v3)};    // jki: (b,c), (a,k)
        case 4: return {0, v2 * nk, single, v, mode3(v, v, v2, 1, v3), plain(v)};                // kij: (c,a,k), b
        default: return {0, v2 * nk, single, v, mode3(v, v, v2, v, v3), plain(1)};               // kji: (c,b,k), a
    }
}

}  // namespace

double pT_energy(Ctx *ctx, int prec, const double *T1, const double *T2, const View4 &Vv, const View4 &Vo,
                 const View4 &Vvovo, const double *fo, const double *fv, int o, int v) {
    JUES_REQUIRE(o > 0 && v > 0, "need o > 0 and v > 0");
    JUES_REQUIRE(v < 1024, "the (T) energy kernel packs virtual indices in 10 bits (v < 1024)");
    const long long v3 = (long long)v * v * v;
    // triples of virtual tiles A >= B >= C, packed
    std::vector<int> htiles;
    const int nt = (v + PT_T - 1) / PT_T;
    for (int a = 0; a < nt; ++a)
        for (int b = 0; b <= a; ++b)
            for (int c = 0; c <= b; ++c) htiles.push_back(a | b << 10 | c << 20);
    DBuf<int> tiles(ctx, htiles.size());
    JUES_CHECK_CUDA(cudaMemcpyAsync(tiles.p, htiles.data(), htiles.size() * sizeof(int), cudaMemcpyHostToDevice,
                                    ctx->stream));
    DBuf<double> slots(ctx, PT_BLOCKS + 1);
    pt_zero<<<4, 256, 0, ctx->stream>>>(slots.p, PT_BLOCKS + 1);
    JUES_CHECK_CUDA(cudaGetLastError());
    // pairs (i >= j) in batches whose W stays in L2 (96 MB, at least one pair)
    const long long most = std::max<long long>(o, (96LL << 20) / (8 * v3));
    std::vector<PtItem> hitems;
    struct Batch {
        int i0, j0, npair;
        long long item0, nitems;
    };
    std::vector<Batch> batches;
    for (int i = 0; i < o; ++i)
        for (int j = 0; j <= i; ++j) {
            if (batches.empty() || batches.back().nitems + j + 1 > most)
                batches.push_back({i, j, 0, (long long)hitems.size(), 0});
            Batch &b = batches.back();
            for (int k = 0; k <= j; ++k) hitems.push_back({i, j, k, v3 * (b.nitems + k)});
            b.npair += 1;
            b.nitems += j + 1;
        }
    long long wmax = 0;
    for (const Batch &b : batches) wmax = std::max(wmax, b.nitems);
    DBuf<PtItem> items(ctx, hitems.size());
    JUES_CHECK_CUDA(cudaMemcpyAsync(items.p, hitems.data(), hitems.size() * sizeof(PtItem), cudaMemcpyHostToDevice,
                                    ctx->stream));
    DBuf<double> W;
    // the stacked form needs its operands' planes; the pair-by-pair form only W of one pair
    std::unique_ptr<PtStacks> st;
    DBuf<E64Args> dargs;
    DBuf<GroupProblem> dprobs;
    DBuf<int> list;
    std::vector<E64Args> args;
    std::vector<GroupProblem> probs;
    std::vector<long long> nitem;   // GEMM items of each launch
    long long most_items = 0;
    try {
        W = DBuf<double>(ctx, (size_t)(v3 * wmax));
        const int np = prec == JUES_PREC_SPLIT || prec == JUES_PREC_SPLIT2 ? 3 : 7;
        st.reset(new PtStacks(ctx, np, T2, Vv, Vo, o, v));
        auto build = [&](int *lp, long long lt) {
            args.clear();
            probs.clear();
            nitem.clear();
            for (const Batch &b : batches)
                for (int t = 0; t < 6; ++t) {
                    long long n = 0;
                    int i = b.i0, j = b.j0;
                    long long w0 = 0;
                    for (int p = 0; p < b.npair; ++p) {
                        const PtTerm m = pt_term(t, i, j, o, v);
                        args.push_back(e64_problem(ctx, st->pr, st->pq, st->K, m.rowA, m.M, m.rowB, m.N, st->unscale, t ? 1.0 : 0.0,
                                                   W.p + w0, m.mC, m.nC, (int)n, lp, lt));
                        GettArgs g;
                        g.M = m.M; g.N = m.N; g.K = st->K;
                        g.alpha = st->unscale; g.beta = t ? 1.0 : 0.0;
                        g.A = st->R.p + m.rowA; g.mA = plain(1); g.kA = plain(st->rowsR);
                        g.B = st->Q.p + m.rowB; g.kB = plain(st->rowsQ); g.nB = plain(1);
                        g.C = W.p + w0; g.mC = m.mC; g.nC = m.nC;
                        probs.push_back(to_problem(g));
                        n += e64_tiles(m.M, m.N);
                        w0 += v3 * (j + 1);
                        if (++j > i) { ++i; j = 0; }
                    }
                    nitem.push_back(n);
                    most_items = std::max(most_items, n);
                }
        };
        build(nullptr, 0);
        list = DBuf<int>(ctx, e64_list_ints(most_items));
        build(list.p, most_items);
        dargs = DBuf<E64Args>(ctx, args.size());
        dprobs = DBuf<GroupProblem>(ctx, probs.size());
        JUES_CHECK_CUDA(cudaMemcpyAsync(dargs.p, args.data(), args.size() * sizeof(E64Args), cudaMemcpyHostToDevice,
                                        ctx->stream));
        JUES_CHECK_CUDA(cudaMemcpyAsync(dprobs.p, probs.data(), probs.size() * sizeof(GroupProblem),
                                        cudaMemcpyHostToDevice, ctx->stream));
    } catch (const Error &e) {
        if (e.code != JUES_ENOMEM) throw;
        st.reset();
        list.reset();
        dargs.reset();
        dprobs.reset();
        W.reset();
    }
    if (st) {
        size_t at = 0, launch = 0;
        for (const Batch &b : batches) {
            for (int t = 0; t < 6; ++t, ++launch) {
                e64_group_run(ctx, st->pr, st->pq, dargs.p + at, dprobs.p + at, b.npair, nitem[launch], list.p, most_items,
                              "pt_w");
                at += (size_t)b.npair;
            }
            energy(ctx, W.p, items.p + b.item0, b.nitems, tiles, T1, Vvovo, fo, fv, o, v, slots.p);
        }
    } else {
        W = DBuf<double>(ctx, (size_t)(v3 * o));
        // the items of a pair with W at the buffer's start: the pairs' k run in order, so pair (i, j)'s items
        // differ from the batches' in w0 alone
        for (auto &x : hitems) x.w0 = v3 * x.k;
        JUES_CHECK_CUDA(cudaMemcpyAsync(items.p, hitems.data(), hitems.size() * sizeof(PtItem), cudaMemcpyHostToDevice,
                                        ctx->stream));
        std::vector<std::unique_ptr<PackScope>> kept;   // the slices of the operands that pair_w declares constant
        for (int i = 0; i < o; ++i)
            for (const double *p : {Vv.p + i * Vv.s[3], T2 + i}) kept.emplace_back(new PackScope(ctx, p));
        long long at = 0;
        for (int i = 0; i < o; ++i)
            for (int j = 0; j <= i; ++j) {
                pair_w(ctx, prec, i, j, T2, Vv, Vo, o, v, W.p);
                energy(ctx, W.p, items.p + at, j + 1, tiles, T1, Vvovo, fo, fv, o, v, slots.p);
                at += j + 1;
            }
    }
    pt_sum_slots<<<1, 1024, 0, ctx->stream>>>(slots.p, PT_BLOCKS, slots.p + PT_BLOCKS);
    JUES_CHECK_CUDA(cudaGetLastError());
    double et = 0.0;
    JUES_CHECK_CUDA(cudaMemcpyAsync(&et, slots.p + PT_BLOCKS, sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    JUES_CHECK_CUDA(cudaStreamSynchronize(ctx->stream));
    ctx->check_flags();
    return et;
}

}  // namespace jues
