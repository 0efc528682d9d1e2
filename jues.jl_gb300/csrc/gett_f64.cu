// FP64 tensor contraction as a GEMM over composite tensor modes (the plain, drop-in form).
//
// GB300 executes FP64 on its CUDA cores only (there is no FP64 kind for tcgen05), so this
// kernel is DFMA-issue bound: BM x BN output tiles, (BM/16) x (BN/16) register blocking per
// thread, operand tiles staged in shared memory with the per-row / per-column element offsets
// of the composite modes precomputed once per tile.  The same tile routine serves single
// problems and the grouped (batched) form, whose persistent CTAs walk a tile list that spans
// many independent problems.
#include <algorithm>
#include <string>

#include "common.cuh"
#include "convert.cuh"
#include "gett_e64.cuh"
#include "gett_f64.cuh"

namespace jues {

namespace {

constexpr int BK = 16, NT = 256;

template <int BM, int BN>
struct TileSmem {
    double As[BK][BM + 1];
    double Bs[BK][BN + 1];
    long long offA[BM], offB[BN], offCm[BM], offCn[BN];
    long long koA[BK], koB[BK];
};

template <int BM, int BN>
__device__ __forceinline__ void gett_tile(const GroupProblem &g, long long tile, TileSmem<BM, BN> &sm,
                                          long long kbeg, long long kend) {
    constexpr int TM = BM / 16, TN = BN / 16;
    const int tid = threadIdx.x;
    const long long m0 = (tile % g.mtiles) * BM;
    const long long n0 = (tile / g.mtiles) * BN;
    const int a_mfast = (g.mA.s0 == 1 && g.mA.d0 > 1);
    const int b_nfast = (g.nB.s0 == 1 && g.nB.d0 > 1);
    const int c_mfast = (g.mC.s0 == 1 && g.mC.d0 > 1);
    __syncthreads();   // the previous tile of a persistent CTA is done with the tables
    for (int r = tid; r < BM; r += NT) {
        const long long m = m0 + r;
        sm.offA[r] = m < g.M ? mode_off(g.mA, m) : -1;
        sm.offCm[r] = m < g.M ? mode_off(g.mC, m) : -1;
    }
    for (int c = tid; c < BN; c += NT) {
        const long long n = n0 + c;
        sm.offB[c] = n < g.N ? mode_off(g.nB, n) : -1;
        sm.offCn[c] = n < g.N ? mode_off(g.nC, n) : -1;
    }
    const int tr = c_mfast ? (tid & 15) : (tid >> 4);
    const int tc = c_mfast ? (tid >> 4) : (tid & 15);
    double acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.0;

    for (long long k0 = kbeg; k0 < kend; k0 += BK) {
        __syncthreads();
        if (tid < BK) {
            const long long k = k0 + tid;
            sm.koA[tid] = k < kend ? mode_off(g.kA, k) : -1;
        } else if (tid >= 32 && tid < 32 + BK) {
            const long long k = k0 + tid - 32;
            sm.koB[tid - 32] = k < kend ? mode_off(g.kB, k) : -1;
        }
        __syncthreads();
        for (int e = tid; e < BM * BK; e += NT) {
            const int m = a_mfast ? (e % BM) : (e / BK);
            const int k = a_mfast ? (e / BM) : (e % BK);
            const long long om = sm.offA[m], ok = sm.koA[k];
            sm.As[k][m] = (om >= 0 && ok >= 0) ? __ldg(g.A + om + ok) : 0.0;
        }
        for (int e = tid; e < BN * BK; e += NT) {
            const int n = b_nfast ? (e % BN) : (e / BK);
            const int k = b_nfast ? (e / BN) : (e % BK);
            const long long on = sm.offB[n], ok = sm.koB[k];
            sm.Bs[k][n] = (on >= 0 && ok >= 0) ? __ldg(g.B + on + ok) : 0.0;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            double a[TM], b[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = sm.As[kk][tr + 16 * i];
#pragma unroll
            for (int j = 0; j < TN; ++j) b[j] = sm.Bs[kk][tc + 16 * j];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
        }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const long long om = sm.offCm[tr + 16 * i];
        if (om < 0) continue;
        // a row's inputs are loaded before any of its outputs is stored (each element is this
        // thread's alone; C and Cin may alias), so those loads are in flight together
        double cin[TN];
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const long long on = sm.offCn[tc + 16 * j];
            cin[j] = (g.beta != 0.0 && on >= 0) ? g.Cin[om + on] : 0.0;
        }
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const long long on = sm.offCn[tc + 16 * j];
            if (on < 0) continue;
            double v = g.alpha * acc[i][j];
            if (g.beta != 0.0) v = fma(g.beta, cin[j], v);
            g.C[om + on] = v;
        }
    }
}

template <int BM, int BN>
__global__ void __launch_bounds__(NT) gett_f64_kernel(GroupProblem g) {
    __shared__ TileSmem<BM, BN> sm;
    gett_tile<BM, BN>(g, blockIdx.x, sm, 0, g.K);
}

// split-K form: CTA b contracts K range [s kper, min(K, (s+1) kper)), s = b / tiles, of tile
// b % tiles into the plain column-major partial ws[s] (M x N; g's output modes describe it)
template <int BM, int BN>
__global__ void __launch_bounds__(NT) gett_f64_splitk(GroupProblem g, long long tiles, long long kper) {
    __shared__ TileSmem<BM, BN> sm;
    const long long s = blockIdx.x / tiles;
    g.C += s * g.M * g.N;
    g.Cin = g.C;
    gett_tile<BM, BN>(g, blockIdx.x % tiles, sm, s * kper, min(g.K, (s + 1) * kper));
}

template <class T>
__global__ void splitk_reduce_kernel(const T *__restrict__ ws, int ks, long long sstride, long long ld, long long M,
                                     long long N, double alpha, double beta, double *C, const double *Cin, Mode mC,
                                     Mode nC) {
    // GB300 runs FP64 at about two operations per clock per SM: the FP32 partials convert on the
    // integer pipes, and alpha = 1 and beta = 0 cost nothing
    const long long total = M * N;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        long long m, n;
        divmod_ll(i, M, n, m);
        const T *p = ws + n * ld + m;
        // eight partials loaded ahead of their (in-order) sum, so the loads overlap
        double acc = 0.0;
        int s = 0;
        for (; s + 8 <= ks; s += 8) {
            T v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = p[(long long)(s + u) * sstride];
#pragma unroll
            for (int u = 0; u < 8; ++u) acc += to_f64(v[u]);
        }
        for (; s < ks; ++s) acc += to_f64(p[(long long)s * sstride]);
        const long long off = mode_off(mC, m) + mode_off(nC, n);
        double v = alpha == 1.0 ? acc : alpha * acc;
        if (beta != 0.0) v = fma(beta, Cin[off], v);
        C[off] = v;
    }
}

template <class T>
void splitk_reduce_t(Ctx *ctx, const T *ws, int ks, long long sstride, long long ld, long long M, long long N,
                     double alpha, double beta, double *C, const double *Cin, const Mode &mC, const Mode &nC,
                     const char *name) {
    const long long total = M * N;
    const long long blocks = std::min<long long>((total + 255) / 256, 152LL * 8);
    const std::string nm = std::string(name) + ".reduce";
    Ctx::Scope sc(ctx, nm.c_str());
    splitk_reduce_kernel<T><<<(unsigned)blocks, 256, 0, ctx->stream>>>(ws, ks, sstride, ld, M, N, alpha, beta, C,
                                                                      Cin ? Cin : C, mC, nC);
    JUES_CHECK_CUDA(cudaGetLastError());
}

// persistent grouped form: problem p owns tiles [tile_start[p], tile_start[p+1])
template <int BM, int BN>
__global__ void __launch_bounds__(NT) gett_f64_grouped(const GroupProblem *__restrict__ probs, int nprob,
                                                       long long total) {
    __shared__ TileSmem<BM, BN> sm;
    for (long long t = blockIdx.x; t < total; t += gridDim.x) {
        int lo = 0, hi = nprob - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (probs[mid].tile_start <= t) lo = mid; else hi = mid - 1;
        }
        gett_tile<BM, BN>(probs[lo], t - probs[lo].tile_start, sm, 0, probs[lo].K);
    }
}

// Offset of a mode index that advances by a fixed step: the division-free successor of
// mode_off (the carries replace the divisions), so a K loop costs a few integer adds per
// element instead of 32- or 64-bit divisions.
struct ModeIter {
    int i0, i1;          // the mode's first two sub-indices (unused for a single-stride mode)
    long long off;
    __device__ __forceinline__ void init(const Mode &m, long long r) {
        if (m.d0 == MODE_BIG) {
            i0 = i1 = 0;
            off = r * m.s0;
            return;
        }
        long long q, r0;
        divmod_ll(r, m.d0, q, r0);
        i0 = (int)r0;
        if (m.d1 == MODE_BIG) {
            i1 = 0;
            off = r0 * m.s0 + q * m.s1;
            return;
        }
        long long q2, r1;
        divmod_ll(q, m.d1, q2, r1);
        i1 = (int)r1;
        off = r0 * m.s0 + r1 * m.s1 + q2 * m.s2;
    }
    __device__ __forceinline__ void step(const Mode &m, int by) {
        if (m.d0 == MODE_BIG) {
            off += by * m.s0;
            return;
        }
        i0 += by;
        off += by * m.s0;
        while (i0 >= m.d0) {
            i0 -= (int)m.d0;
            off += m.s1 - m.d0 * m.s0;
            if (m.d1 != MODE_BIG && ++i1 >= m.d1) {
                i1 = 0;
                off += m.s2 - m.d1 * m.s1;
            }
        }
    }
};

// What the tensor-core form left out (gett_e64.cu).  Half tiles with few elements left out: a block each (several
// where there are few of them), four lanes to an element.  An element costs 2.3 times what it does in a whole tile,
// so half tiles go this way up to a quarter of their pieces (MP2 of s functions on a chain, nbf = 96, first quarter:
// 4.21 -> 2.95 ms).  Whole ones, 128 x 16 of one problem: a long list runs as 64 x 16 tiles, a shorter one as
// 16 x 16, and one of up to 16 entries with a warp to two outputs: FP64 issue bounds a block's 16 x 16 K
// products, and eight such blocks leave the other SMs idle (K = 3240, one, four and sixteen entries: 455, 450 and 467
// us as 16 x 16, now 82, 147 and 299).  Both lists are nearly always empty.
__global__ void __launch_bounds__(NT) gett_f64_tiles_kernel(const GroupProblem one,
                                                            const GroupProblem *__restrict__ probs,
                                                            const int *__restrict__ list,
                                                            const int *__restrict__ fine) {
    __shared__ TileSmem<64, 16> sm;
    const int n = list[0], nf = list[1];
    // a block each, or as many as there are blocks for
    const int shares = nf ? max(1, min(32, (int)gridDim.x / nf)) : 1;
    for (long long x = blockIdx.x; x < (long long)nf * shares; x += gridDim.x) {
        const long long d = x / shares;
        const int share = (int)(x % shares);
        __shared__ unsigned short elem[8 * E64_FINE];   // row | column << 7
        __shared__ int sums[NT / 32];
        const int *f = fine + d * E64_FINE_INTS;
        const GroupProblem &g = probs ? probs[f[0]] : one;
        const long long mt128 = (g.M + 127) / 128, m0 = f[1] % mt128 * 128, n0 = f[1] / mt128 * 16;
        const int tid = threadIdx.x, lane = tid & 31;
        __syncthreads();
        // the pieces' elements, in the order of the list (every block that shares it takes others of them)
        const unsigned piece = tid < f[2] ? reinterpret_cast<const unsigned short *>(f + 3)[tid] : 0u;
        int at = __popc(piece >> 8), ne = 0;
#pragma unroll
        for (int i = 1; i < 32; i <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, at, i);
            if (lane >= i) at += y;
        }
        if (lane == 31) sums[tid >> 5] = at;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < NT / 32; ++i) {
            if (i == tid >> 5) at += ne;
            ne += sums[i];
        }
        at -= __popc(piece >> 8);
        for (int j = 0; j < 8; ++j)
            if (piece >> (8 + j) & 1) elem[at++] = (unsigned short)((piece & 127) | ((piece >> 7 & 1) * 8 + j) << 7);
        __syncthreads();
        for (int e0 = share * (NT / 4) + (tid >> 5) * 8; e0 < ne; e0 += shares * (NT / 4)) {
            const int e = min(e0 + (lane & 7), ne - 1), part = lane >> 3;
            const long long m = m0 + (elem[e] & 127), c = n0 + (elem[e] >> 7);
            const bool in = m < g.M && c < g.N;
            double acc = 0.0;
            if (in) {
                const double *pa = g.A + mode_off(g.mA, m), *pb = g.B + mode_off(g.nB, c);
                ModeIter ia, ib;
                ia.init(g.kA, part);
                ib.init(g.kB, part);
#pragma unroll 4
                for (long long k = part; k < g.K; k += 4) {
                    acc = fma(__ldg(pa + ia.off), __ldg(pb + ib.off), acc);
                    ia.step(g.kA, 4);
                    ib.step(g.kB, 4);
                }
            }
            __syncwarp();
            acc += __shfl_xor_sync(0xffffffffu, acc, 8);
            acc += __shfl_xor_sync(0xffffffffu, acc, 16);
            if (part == 0 && in && e0 + lane < ne) {
                const long long off = mode_off(g.mC, m) + mode_off(g.nC, c);
                double v = g.alpha * acc;
                if (g.beta != 0.0) v = fma(g.beta, g.Cin[off], v);
                g.C[off] = v;
            }
        }
    }
    if (n <= 16) {
        const int lane = threadIdx.x & 31;
        for (int w = (blockIdx.x * NT + threadIdx.x) >> 5; w < n * 1024; w += gridDim.x * (NT / 32)) {
            const int e = w >> 10;
            const GroupProblem &g = probs ? probs[list[2 + 2 * e]] : one;
            const long long t = list[3 + 2 * e], mt128 = (g.M + 127) / 128;
            const long long m = t % mt128 * 128 + (w & 127), n0 = t / mt128 * 16 + 2 * (w >> 7 & 7);
            if (m >= g.M || n0 >= g.N) continue;
            const long long n1 = n0 + 1 < g.N ? n0 + 1 : n0;
            const double *pa = g.A + mode_off(g.mA, m);
            const double *p0 = g.B + mode_off(g.nB, n0), *p1 = g.B + mode_off(g.nB, n1);
            ModeIter ia, ib;
            ia.init(g.kA, lane);
            ib.init(g.kB, lane);
            double acc0 = 0.0, acc1 = 0.0;
#pragma unroll 4
            for (long long k = lane; k < g.K; k += 32) {
                const double x = __ldg(pa + ia.off);
                acc0 = fma(x, __ldg(p0 + ib.off), acc0);
                acc1 = fma(x, __ldg(p1 + ib.off), acc1);
                ia.step(g.kA, 32);
                ib.step(g.kB, 32);
            }
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) {
                acc0 += __shfl_xor_sync(0xffffffffu, acc0, d);
                acc1 += __shfl_xor_sync(0xffffffffu, acc1, d);
            }
            if (lane > 1 || (lane == 1 && n1 == n0)) continue;
            const long long off = mode_off(g.mC, m) + mode_off(g.nC, lane ? n1 : n0);
            double v = g.alpha * (lane ? acc1 : acc0);
            if (g.beta != 0.0) v = fma(g.beta, g.Cin[off], v);
            g.C[off] = v;
        }
        return;
    }
    const int sub = n <= 512 ? 8 : 2, rows = 128 / sub;
    for (int x = blockIdx.x; x < n * sub; x += gridDim.x) {
        const int e = x / sub;
        GroupProblem g = probs ? probs[list[2 + 2 * e]] : one;
        const long long t = list[3 + 2 * e], mt128 = (g.M + 127) / 128;
        const long long mt = sub * (t % mt128) + x % sub;
        g.mtiles = (g.M + rows - 1) / rows;
        if (mt >= g.mtiles) continue;
        if (sub == 8)
            gett_tile<16, 16>(g, mt + g.mtiles * (t / mt128), reinterpret_cast<TileSmem<16, 16> &>(sm), 0, g.K);
        else
            gett_tile<64, 16>(g, mt + g.mtiles * (t / mt128), sm, 0, g.K);
    }
}

// skinny GEMM (N <= NN <= 8): one warp per output row, lanes split K
template <int NN>
__global__ void __launch_bounds__(256, NN == 1 ? 3 : 2) gett_f64_skinny(GroupProblem g) {
    const long long warp = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (warp >= g.M) return;
    const long long m = warp;
    const long long om = mode_off(g.mA, m);
    double acc[NN];
#pragma unroll
    for (int j = 0; j < NN; ++j) acc[j] = 0.0;
    long long onb[NN];
#pragma unroll
    for (int j = 0; j < NN; ++j) onb[j] = j < g.N ? mode_off(g.nB, j) : 0;
    // four independent K positions per lane (k, k + 32, k + 64, k + 96): their loads are in
    // flight together instead of one load latency per element
    constexpr int U = 4;
    ModeIter ia[U], ib[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        ia[u].init(g.kA, lane + 32 * u);
        ib[u].init(g.kB, lane + 32 * u);
    }
    for (long long k = lane; k < g.K; k += 32 * U) {
        double a[U];
#pragma unroll
        for (int u = 0; u < U; ++u) a[u] = k + 32 * u < g.K ? __ldg(g.A + om + ia[u].off) : 0.0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (k + 32 * u < g.K) {
                const long long ok = ib[u].off;
#pragma unroll
                for (int j = 0; j < NN; ++j)
                    if (j < g.N) acc[j] = fma(a[u], __ldg(g.B + ok + onb[j]), acc[j]);
            }
            ia[u].step(g.kA, 32 * U);
            ib[u].step(g.kB, 32 * U);
        }
    }
    const long long oc = mode_off(g.mC, m);
#pragma unroll
    for (int j = 0; j < NN; ++j) {
        if (j >= g.N) break;
        double v = acc[j];
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) v += __shfl_down_sync(0xffffffffu, v, d);
        if (lane == 0) {
            const long long off = oc + mode_off(g.nC, j);
            double r = g.alpha * v;
            if (g.beta != 0.0) r = fma(g.beta, g.Cin[off], r);
            g.C[off] = r;
        }
    }
}

// skinny GEMM (N <= NN <= 8) whose rows, not K, are the unit-stride index of A: one thread per
// output row, so a warp's loads of one K position are 32 consecutive doubles; blockIdx.y takes
// K positions [y kper, (y + 1) kper) (four independent positions in flight per thread) and writes
// its partial sums to part[y][n][m] for the split-K reduction (kper = K: one part)
template <int NN>
__global__ void __launch_bounds__(256) gett_f64_rows(GroupProblem g, long long kper, double *__restrict__ part) {
    const long long m = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (m >= g.M) return;
    const long long k0 = blockIdx.y * kper, k1 = min(g.K, k0 + kper);
    const long long om = mode_off(g.mA, m);
    long long onb[NN];
#pragma unroll
    for (int j = 0; j < NN; ++j) onb[j] = j < g.N ? mode_off(g.nB, j) : 0;
    double acc[NN];
#pragma unroll
    for (int j = 0; j < NN; ++j) acc[j] = 0.0;
    constexpr int U = 4;
    ModeIter ia[U], ib[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        ia[u].init(g.kA, k0 + u);
        ib[u].init(g.kB, k0 + u);
    }
    for (long long k = k0; k < k1; k += U) {
        double a[U];
#pragma unroll
        for (int u = 0; u < U; ++u) a[u] = k + u < k1 ? __ldg(g.A + om + ia[u].off) : 0.0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (k + u < k1) {
                const long long ok = ib[u].off;
#pragma unroll
                for (int j = 0; j < NN; ++j)
                    if (j < g.N) acc[j] = fma(a[u], __ldg(g.B + ok + onb[j]), acc[j]);
            }
            ia[u].step(g.kA, U);
            ib[u].step(g.kB, U);
        }
    }
#pragma unroll
    for (int j = 0; j < NN; ++j)
        if (j < g.N) part[(blockIdx.y * g.N + j) * g.M + m] = acc[j];
}

// Smallest GEMMs (M N <= 4096 outputs, K <= 8192): one warp per output element, its lanes over K, so that
// even a single-tile problem spreads over the whole GPU instead of one CTA.  Latency bounds it.
__global__ void __launch_bounds__(256) gett_f64_dots(GroupProblem g) {
    const long long w = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (w >= g.M * g.N) return;
    const long long m = w % g.M, n = w / g.M;
    const long long oa = mode_off(g.mA, m), ob = mode_off(g.nB, n);
    ModeIter ia, ib;
    ia.init(g.kA, lane);
    ib.init(g.kB, lane);
    double acc = 0.0;
    for (long long k = lane; k < g.K; k += 32) {
        acc = fma(__ldg(g.A + oa + ia.off), __ldg(g.B + ob + ib.off), acc);
        ia.step(g.kA, 32);
        ib.step(g.kB, 32);
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, d);
    if (lane == 0) {
        const long long off = mode_off(g.mC, m) + mode_off(g.nC, n);
        double r = g.alpha * acc;
        if (g.beta != 0.0) r = fma(g.beta, g.Cin[off], r);
        g.C[off] = r;
    }
}

// Small GEMM: 2^ll threads share two neighbouring outputs of a row and split K; ll is chosen for about
// 40,000 threads in all.  FP64 issue and latency bound it, so the lanes' tree sums are kept short: with a
// warp per output, a K = 16 product of 256 x 256 spends more on the five additions and shuffles of each
// output than on its products (44 us, here 12).  The K offsets of both operands are tabulated once per
// block.  kfast: neighbouring threads take neighbouring K positions of one row (A's K is its unit-stride
// index), else neighbouring rows.  MP2 with nbf = 25 (quarter transforms with five columns): 213 -> 127 us;
// RCCD with nbf = 25, twelve sweeps: 3.80 -> 3.20 ms.
constexpr int SMALL_K = 512;
__global__ void __launch_bounds__(256) gett_f64_small(GroupProblem g, int ll, int kfast) {
    __shared__ long long ka[SMALL_K], kb[SMALL_K];
    const int tid = threadIdx.x, lane = tid & 31, L = 1 << ll;
    const long long t = blockIdx.x * 256LL + tid;
    const int kl = kfast ? lane & (L - 1) : lane >> (5 - ll);
    const long long task = kfast ? t >> ll : (t >> 5) * (32 >> ll) + (lane & ((32 >> ll) - 1));
    const bool live = task < g.M * ((g.N + 1) / 2);
    long long nb, m;
    divmod_ll(live ? task : 0, g.M, nb, m);
    const long long n0 = 2 * nb, n1 = n0 + 1 < g.N ? n0 + 1 : n0;
    const double *pa = g.A + mode_off(g.mA, m);
    const double *p0 = g.B + mode_off(g.nB, n0), *p1 = g.B + mode_off(g.nB, n1);
    double acc0 = 0.0, acc1 = 0.0;
    for (long long k0 = 0; k0 < g.K; k0 += SMALL_K) {
        const int kn = (int)min((long long)SMALL_K, g.K - k0);
        __syncthreads();
        for (int k = tid; k < kn; k += 256) {
            ka[k] = mode_off(g.kA, k0 + k);
            kb[k] = mode_off(g.kB, k0 + k);
        }
        __syncthreads();
        if (live) {
#pragma unroll 4
            for (int k = kl; k < kn; k += L) {
                const double x = __ldg(pa + ka[k]);
                acc0 = fma(x, __ldg(p0 + kb[k]), acc0);
                acc1 = fma(x, __ldg(p1 + kb[k]), acc1);
            }
        }
    }
    for (int d = kfast ? 1 : 32 >> ll; d < (kfast ? L : 32); d <<= 1) {
        acc0 += __shfl_xor_sync(0xffffffffu, acc0, d);
        acc1 += __shfl_xor_sync(0xffffffffu, acc1, d);
    }
    if (!live || kl > 1 || (kl == 1 && n1 == n0)) return;
    const long long om = mode_off(g.mC, m);
    auto put = [&](long long n, double v) {
        const long long off = om + mode_off(g.nC, n);
        double r = g.alpha * v;
        if (g.beta != 0.0) r = fma(g.beta, g.Cin[off], r);
        g.C[off] = r;
    };
    // lanes 0 and 1 store one output each; a single lane stores both
    if (kl == 0) put(n0, acc0);
    if ((L > 1 ? kl == 1 : true) && n1 != n0) put(n1, acc1);
}

// Small GEMM in tiles: a block stages tm rows of A and tn columns of B in shared memory, K in chunks of kc,
// its tm tn outputs (<= 128) times groups of threads over K.  Latency and the operands' uncoalesced loads bound
// such a product: a thread per part of an output loads every element of A once per column from L1 (100^3:
// 38 loads a thread; here 7).
constexpr int TILE_NT = 512, TILE_WORDS = 5120, TILE_KC = 384, TILE_SIDE = 16;
__global__ void __launch_bounds__(TILE_NT) gett_f64_tile(GroupProblem g, int tm, int tn, int kc, int kfastA, int kfastB) {
    __shared__ double buf[TILE_WORDS];
    __shared__ long long ka[TILE_KC], kb[TILE_KC], ra[TILE_SIDE], rb[TILE_SIDE], rc[TILE_SIDE], cc[TILE_SIDE];
    const int tid = threadIdx.x;
    const int mt = (int)((g.M + tm - 1) / tm);
    const long long m0 = (long long)(blockIdx.x % mt) * tm, n0 = (long long)(blockIdx.x / mt) * tn;
    // rows and columns past the edge read the last one and are not stored
    if (tid < tm) {
        const long long m = min(m0 + tid, g.M - 1);
        ra[tid] = mode_off(g.mA, m);
        rc[tid] = mode_off(g.mC, m);
    } else if (tid >= 32 && tid < 32 + tn) {
        const long long n = min(n0 + tid - 32, g.N - 1);
        rb[tid - 32] = mode_off(g.nB, n);
        cc[tid - 32] = mode_off(g.nC, n);
    }
    const int P = tm * tn, G = TILE_NT / P, kg = tid / P, q = tid - kg * P, r = q % tm, c = q / tm;
    double acc = 0.0;
    for (long long k0 = 0; k0 < g.K; k0 += kc) {
        const int kn = (int)min((long long)kc, g.K - k0);
        __syncthreads();
        for (int k = tid; k < kn; k += TILE_NT) {
            ka[k] = mode_off(g.kA, k0 + k);
            kb[k] = mode_off(g.kB, k0 + k);
        }
        __syncthreads();
        double *As = buf, *Bs = buf + tm * kn;   // [k][row], [k][column]
        const int na = tm * kn, nb = tn * kn;
#pragma unroll 4
        for (int e = tid; e < na; e += TILE_NT) {
            const int k = kfastA ? e % kn : e / tm, i = kfastA ? e / kn : e % tm;
            As[k * tm + i] = __ldg(g.A + ra[i] + ka[k]);
        }
#pragma unroll 4
        for (int e = tid; e < nb; e += TILE_NT) {
            const int k = kfastB ? e % kn : e / tn, i = kfastB ? e / kn : e % tn;
            Bs[k * tn + i] = __ldg(g.B + rb[i] + kb[k]);
        }
        __syncthreads();
        if (kg < G) {
#pragma unroll 4
            for (int k = kg; k < kn; k += G) acc = fma(As[k * tm + r], Bs[k * tn + c], acc);
        }
    }
    __syncthreads();
    for (int w = G; w > 1;) {
        const int h = (w + 1) / 2;
        if (kg >= h && kg < w) buf[tid] = acc;
        __syncthreads();
        if (kg + h < w) acc += buf[tid + h * P];
        w = h;
    }
    if (tid >= P || m0 + r >= g.M || n0 + c >= g.N) return;
    const long long off = rc[r] + cc[c];
    double v = g.alpha * acc;
    if (g.beta != 0.0) v = fma(g.beta, g.Cin[off], v);
    g.C[off] = v;
}

// tile of a small GEMM: the least rounds of 152 blocks times the clocks of one (FP64 issue, its loads, the
// latency of a chunk of K)
void small_tile(long long M, long long N, long long K, int &tm, int &tn, int &kc) {
    constexpr int SIDES[] = {2, 4, 5, 6, 7, 8, 10, 12, 14, 16};
    double best = 1e300;
    for (int x : SIDES)
        for (int y : SIDES) {
            const int P = x * y, G = TILE_NT / P;
            if (P > 128 || P < 16) continue;
            const long long tiles = ((M + x - 1) / x) * ((N + y - 1) / y);
            const int ch = (int)std::min<long long>(std::min(TILE_KC, TILE_WORDS / (x + y)), K);
            const double clk = 0.47 * TILE_NT * (double)((K + G - 1) / G) + 0.75 * (x + y) * (double)K +
                               1500.0 * (double)((K + ch - 1) / ch) + 1500.0;
            const double t = (double)((tiles + 151) / 152) * clk;
            if (t < best) { best = t; tm = x; tn = y; kc = ch; }
        }
}

}  // namespace

GroupProblem to_problem(const GettArgs &a) {
    GroupProblem g;
    g.M = a.M; g.N = a.N; g.K = a.K;
    g.alpha = a.alpha; g.beta = a.beta;
    g.A = a.A; g.mA = a.mA; g.kA = a.kA;
    g.B = a.B; g.kB = a.kB; g.nB = a.nB;
    g.C = a.C; g.mC = a.mC; g.nC = a.nC;
    g.Cin = a.Cin ? a.Cin : a.C;
    g.mtiles = 1;
    g.tile_start = 0;
    return g;
}

void gett_f64_tiles(Ctx *ctx, const GettArgs *one, const GroupProblem *probs, const int *list, long long list_tiles,
                    const char *name) {
    GroupProblem g{};
    if (one) g = to_problem(*one);
    const std::string nm = std::string(name) + ".rest";
    Ctx::Scope s(ctx, nm.c_str());
    gett_f64_tiles_kernel<<<152 * 4, NT, 0, ctx->stream>>>(g, probs, list, list + 2 + 4 * list_tiles);
    JUES_CHECK_CUDA(cudaGetLastError());
}

void gett_f64(Ctx *ctx, const GettArgs &a, const char *name) {
    if (a.M <= 0 || a.N <= 0) return;
    if (gett_e64(ctx, a, name)) return;
    GroupProblem g = to_problem(a);
    // A warp per output up to 4096 outputs: its 32 lanes are needed to fill the GPU (us against the kernel
    // with two outputs to a task: 9 x 9 x 9 6.0 / 7.7; 60 x 60 x 2000 32 / 38; 40 x 40 x 6000 92 / 93).
    if (a.N > 8 && a.M * a.N <= 4096 && a.K <= 8192) {
        Ctx::Scope s(ctx, name);
        gett_f64_dots<<<(unsigned)((a.M * a.N * 32 + 255) / 256), 256, 0, ctx->stream>>>(g);
        JUES_CHECK_CUDA(cudaGetLastError());
        return;
    }
    // Tiles beyond that up to 32768 outputs (us against two outputs to a task: 100 x 100 x 100 13.9 / 11.5; 25 x
    // 400 x 400 30 / 26; 150 x 150 x 150 24.5 / 18.4; 25 x 400 x 25 10.7 / 9.1); more outputs fill the GPU either
    // way (250 x 250 x 100 27 / 25, 250 x 250 x 16 11.5 / 14).
    if (a.N > 8 && a.M * a.N <= (1LL << 15) && a.K >= 16 && a.K <= 8192) {
        int tm = 8, tn = 8, kc = 1;
        small_tile(a.M, a.N, a.K, tm, tn, kc);
        const long long tiles = ((a.M + tm - 1) / tm) * ((a.N + tn - 1) / tn);
        Ctx::Scope s(ctx, name);
        gett_f64_tile<<<(unsigned)tiles, TILE_NT, 0, ctx->stream>>>(g, tm, tn, kc, a.kA.s0 == 1 && a.kA.d0 > 1,
                                                                   a.kB.s0 == 1 && a.kB.d0 > 1);
        JUES_CHECK_CUDA(cudaGetLastError());
        return;
    }
    // Two outputs to a task beyond that (100 x 100 x 100 16 -> 14 us; 25 x 400 x 25 13 -> 10; 25 x 400 x 400
    // 33 / 33), and for few columns with a short K at any M, where the kernels below lose more to their tree
    // sums and to rows that share no loads (us, M x N x K; A's K, then A's rows at unit stride: 15625 x 5 x 25
    // 66 -> 19 and 34 -> 20; 250000 x 8 x 25 1240 -> 113 and 128 -> 113).  K = 128 is where the sides meet:
    // 62500 x 8 x 128 160 / 155 and 250000 x 8 x 128 1260 / 1273 with A's rows at unit stride.
    if ((a.N > 8 && a.M * a.N <= (1LL << 16) && a.K <= 8192) || (a.N > 1 && a.N <= 8 && a.K <= 128)) {
        const long long tasks = a.M * ((a.N + 1) / 2);
        int ll = 0;
        while (ll < 5 && (tasks << ll) < 40000 && (2LL << ll) <= a.K) ++ll;
        const long long blocks = ((tasks << ll) + 255) / 256;
        JUES_REQUIRE(blocks < (1LL << 31), "GEMM too large for one launch");
        Ctx::Scope s(ctx, name);
        gett_f64_small<<<(unsigned)blocks, 256, 0, ctx->stream>>>(g, ll, a.kA.s0 == 1 && a.kA.d0 > 1);
        JUES_CHECK_CUDA(cudaGetLastError());
        return;
    }
    const bool k_unit = a.kA.s0 == 1 && a.kA.d0 > 1, rows_unit = a.mA.s0 == 1 && a.mA.d0 > 1;
    if (a.N <= 8 && rows_unit && !k_unit && a.M >= 256) {
        // thread per row, K split over blockIdx.y so that about eight blocks run per SM
        const long long rb = (a.M + 255) / 256;
        long long ks = std::max<long long>(1, std::min<long long>((152LL * 8 + rb - 1) / rb, a.K / 64));
        ks = std::min<long long>(ks, 65535);
        long long kper = (a.K + ks - 1) / ks;
        kper = (kper + 3) / 4 * 4;
        ks = (a.K + kper - 1) / kper;
        JUES_REQUIRE(rb < (1LL << 31), "GEMM too large for one launch");
        double *ws = static_cast<double *>(ctx->splitk_scratch((size_t)(ks * a.M * a.N) * sizeof(double)));
        {
            Ctx::Scope s(ctx, name);
            const dim3 grid((unsigned)rb, (unsigned)ks);
            if (a.N == 1)
                gett_f64_rows<1><<<grid, 256, 0, ctx->stream>>>(g, kper, ws);
            else
                gett_f64_rows<8><<<grid, 256, 0, ctx->stream>>>(g, kper, ws);
            JUES_CHECK_CUDA(cudaGetLastError());
        }
        splitk_reduce(ctx, ws, (int)ks, a.M * a.N, a.M, a.M, a.N, a.alpha, a.beta, a.C, g.Cin, a.mC, a.nC, name);
        return;
    }
    if (a.N <= 8) {
        long long blocks = (a.M * 32 + 255) / 256;
        JUES_REQUIRE(blocks < (1LL << 31), "GEMM too large for one launch");
        Ctx::Scope s(ctx, name);
        if (a.N == 1)
            gett_f64_skinny<1><<<(unsigned)blocks, 256, 0, ctx->stream>>>(g);
        else
            gett_f64_skinny<8><<<(unsigned)blocks, 256, 0, ctx->stream>>>(g);
        JUES_CHECK_CUDA(cudaGetLastError());
        return;
    }
    g.mtiles = (a.M + 63) / 64;
    const long long tiles = g.mtiles * ((a.N + 63) / 64);
    JUES_REQUIRE(tiles < (1LL << 31), "GEMM too large for one launch");
    // A grid below four CTAs per SM with a long K splits K (at least 512 per split); the
    // partials are reduced in FP64 in split order.
    constexpr long long kTarget = 152LL * 4;
    if (tiles < kTarget && a.K >= 1024) {
        const long long want = std::min<long long>((kTarget + tiles - 1) / tiles, a.K / 512);
        long long kper = (a.K + want - 1) / want;
        kper = (kper + BK - 1) / BK * BK;
        const long long ks = (a.K + kper - 1) / kper;
        if (ks > 1) {
            double *ws = static_cast<double *>(ctx->splitk_scratch((size_t)(ks * a.M * a.N) * sizeof(double)));
            GroupProblem p = g;
            p.C = ws;
            p.Cin = ws;
            p.mC = plain(1);
            p.nC = plain(a.M);
            p.alpha = 1.0;
            p.beta = 0.0;
            {
                Ctx::Scope s(ctx, name);
                gett_f64_splitk<64, 64><<<(unsigned)(tiles * ks), NT, 0, ctx->stream>>>(p, tiles, kper);
                JUES_CHECK_CUDA(cudaGetLastError());
            }
            splitk_reduce(ctx, ws, (int)ks, a.M * a.N, a.M, a.M, a.N, a.alpha, a.beta, a.C, g.Cin, a.mC, a.nC, name);
            return;
        }
    }
    Ctx::Scope s(ctx, name);
    gett_f64_kernel<64, 64><<<(unsigned)tiles, NT, 0, ctx->stream>>>(g);
    JUES_CHECK_CUDA(cudaGetLastError());
}

void splitk_reduce(Ctx *ctx, const float *ws, int ks, long long sstride, long long ld, long long M, long long N,
                   double alpha, double beta, double *C, const double *Cin, const Mode &mC, const Mode &nC,
                   const char *name) {
    splitk_reduce_t(ctx, ws, ks, sstride, ld, M, N, alpha, beta, C, Cin, mC, nC, name);
}
void splitk_reduce(Ctx *ctx, const double *ws, int ks, long long sstride, long long ld, long long M, long long N,
                   double alpha, double beta, double *C, const double *Cin, const Mode &mC, const Mode &nC,
                   const char *name) {
    splitk_reduce_t(ctx, ws, ks, sstride, ld, M, N, alpha, beta, C, Cin, mC, nC, name);
}

const TileShape kTileShapes[kNumTileShapes] = {{64, 64}, {32, 64}, {64, 32}, {32, 32}};

long long grouped_tiles(std::vector<GroupProblem> &probs, int shape) {
    const int BM = kTileShapes[shape].bm, BN = kTileShapes[shape].bn;
    long long start = 0;
    for (auto &p : probs) {
        p.mtiles = (p.M + BM - 1) / BM;
        p.tile_start = start;
        start += (p.M > 0 && p.N > 0) ? p.mtiles * ((p.N + BN - 1) / BN) : 0;
    }
    return start;
}

void gett_f64_grouped_launch(Ctx *ctx, const GroupProblem *d_probs, int nprob, long long total, int shape,
                             const char *name) {
    if (total <= 0) return;
    const long long grid = std::min<long long>(total, 152LL * 4);   // persistent: 4 CTAs per SM
    Ctx::Scope s(ctx, name);
    switch (shape) {
        case 0: gett_f64_grouped<64, 64><<<(unsigned)grid, NT, 0, ctx->stream>>>(d_probs, nprob, total); break;
        case 1: gett_f64_grouped<32, 64><<<(unsigned)grid, NT, 0, ctx->stream>>>(d_probs, nprob, total); break;
        case 2: gett_f64_grouped<64, 32><<<(unsigned)grid, NT, 0, ctx->stream>>>(d_probs, nprob, total); break;
        default: gett_f64_grouped<32, 32><<<(unsigned)grid, NT, 0, ctx->stream>>>(d_probs, nprob, total); break;
    }
    JUES_CHECK_CUDA(cudaGetLastError());
}

void gett(Ctx *ctx, int precision, const GettArgs &g, const char *name) {
    if (precision == JUES_PREC_SPLIT || precision == JUES_PREC_SPLIT2)
        gett_tc(ctx, g, name, 2);
    else if (precision == JUES_PREC_SPLIT3)
        gett_tc(ctx, g, name, 3);
    else
        gett_f64(ctx, g, name);
}

}  // namespace jues
