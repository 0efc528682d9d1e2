// FP64 tensor contraction on the sm_103a tensor cores, at FP64 accuracy.
//
// GB300 issues about two FP64 operations per clock per SM (1.25 TFLOP/s in all) and has no FP64
// tensor kind, but kind::f16 multiplies small integers exactly.  Every operand row (a row of A or a
// column of B, running over the whole K) gets one power-of-two scale 2^e with max |x| < 2^e, and an
// element becomes a 63-bit fixed-point number q = rint(x 2^(62-e)) cut into seven balanced 9-bit
// digits, q = sum_p d_p 2^(9 (6-p)), d_p in [-256, 256], each exact in FP16.  Then
//     sum_k a_k b_k = 2^(ea + eb - 70) sum_j S_j 2^(9 (6-j)),   S_j = sum_k sum_{p+q=j} d_p(a_k) d_q(b_k)
// with the products of j >= 7 left out (2^-63 of max|a| max|b| each).  One tcgen05.mma with plane p
// of A against the stacked planes 0..6-p of B adds to the accumulators j = p..6, so 28 products run
// as seven instructions per K = 16 step.  Over a chunk of 64 K values |S_j| <= (j+1) 64 2^16 <= 2^24
// for j <= 3, so the FP32 accumulators hold these sums exactly whatever the data; S_4, S_5 and S_6
// (2^-36 to 2^-54 of the product) could pass 2^24 only for a chunk of equal-signed maximal digits and
// then lose one unit in 2^24.  After each chunk the sums are added into 64-bit integers (S_0..S_2 and
// S_3..S_6 combined), so the accumulation over K is exact.  Cutting operands into slices whose products are
// exact is the method of Ozaki, Ogita, Oishi and Rump (Numer. Algorithms 59, 2012).
//
// Error: rounding the inputs to 2^-63 of their row's maximum and the six products of j = 7 left out are at most
// 8.1 x 2^-63 max|a| max|b| for each k whose a_k and b_k are both nonzero, and the result is rounded once.  That is far
// below an FMA loop's K 2^-53 sum |a_k b_k| unless the large elements of a row meet only small ones (or zeros) of
// the column.  So every element is judged by the magnitude it is made of: a further plane holds |x| cut to E5M2,
// whose products, a narrow 8-bit MMA for every 32 K values, sum to P <= sum |a_k b_k|; an element is taken only
// where P >= 2^-7 max|a| max|b| (and 1/16 more), which bounds its error by K 2^-53 sum |a_k b_k| + 2^-53 |a.b|
// whatever the operands are.  Elements below that, and those of rows and columns that hold a non-finite,
// subnormal-only or extreme (beyond 2^+-400) maximum, are not stored but listed, and gett_f64_tiles recomputes them
// on the FP64 pipe, with the same special values as ever: one by one where up to a quarter of the pieces (eight
// columns of a row) of a half tile have any, else the half tile (16 columns).
// Cancellation alone lists nothing, and neither do zeros of symmetry: P = 0 where a row and a column have no
// nonzero element in common, and the result is exactly 0.  Against exact products, relative Frobenius error for normal entries:
// 4.7e-17 at every size, the FMA kernels 1.3e-16 (K = 100) to 8.4e-16 (640^3).
//
// Speed (packs included): 6400^3 10.8 ms = 49 TFLOP/s against 420 ms on the FP64 pipe, 1600^3 0.26 against
// 8.1 ms, 500000 x 100 x 100 0.82 against 11.8 ms.  The magnitudes cost 4 to 7 % of that at long K: they come with B,
// so the MMA loop has one wait for both (in the ring of A planes they cost 8 to 12 %, as an FP16 plane 15 %), and
// a tile whose elements all have enough after two chunks loads no more of them (else 7 to 9 %).  At K <= 128 a tile's
// epilogue (integer issue of the sixteen drain warps, about 8000 clocks a tile) bounds it.
//
// The tile is 128 x 32: TMEM holds two buffers of 8 x 32 FP32 columns (seven digit sums and the magnitudes), so
// the drain of one chunk overlaps the MMAs of the next; a wider tile would need TMEM that is not there.  At long K
// moving the operands paces: 140 KB a chunk from L2 (13.7 TB/s over all SMs), and shared memory, of which the chunk's
// MMAs read 240 KB (with N = 32 per plane an instruction takes 4 KB of A and 1 to 7 KB of B for 16 to 112 clocks)
// while TMA writes those 140, 2990 clocks at 128 bytes a clock against 1820 of MMA at the dense rate.  A's planes
// arrive one by one (64 K values x 128 rows, 16 KB, 128-byte swizzle) in a ring of eight, B's together with the
// magnitudes of both (64-byte swizzle).
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include <cudaTypedefs.h>

#include "gett_e64.cuh"
#include "packcache.cuh"
#include "tcgen05.cuh"

namespace jues {

namespace {

constexpr int NP = E64_NP;            // digit planes of the FP64 form (the kernels take 3 too)
constexpr int BM = 128, BN = 32;      // output tile
constexpr int CK = 64;                // K per chunk: 128 bytes of FP16, one swizzle row
constexpr int SLOTS = 8;              // ring of A planes
constexpr int A_BYTES = BM * CK * 2;  // one A plane, 16 KB
// all of B and the magnitudes of both: 28 + 2 + 8 KB for seven digits
constexpr int b_bytes(int np) { return np * BN * CK * 2 + (BN + BM) * CK; }
// an operand's planes in FP16 words: np digits for each of its rows x kpad elements, then the magnitudes, bytes in
// rows of whole 32-byte sectors
constexpr long long mag_pitch(long long kpad) { return (kpad + 31) / 32 * 32; }
constexpr size_t plane_halves(int np, long long rows, long long kpad) {
    return (size_t)np * rows * kpad + (size_t)rows * mag_pitch(kpad) / 2;
}
constexpr int ring_bytes(int np) { return SLOTS * A_BYTES + 2 * b_bytes(np); }
constexpr uint32_t TMEM_COLS = 512;   // two chunk buffers of (np + 1) x 32 columns
// sixteen drain warps: the drain and the epilogue are chains of short integer operations, and with
// two warps per scheduler (eight in all) they issued one instruction in three clocks
constexpr int THREADS = 576, DRAIN = 512;
constexpr int HB = BN / 4;            // columns per drain thread
constexpr int VN = BN / 2;            // columns of a vote: eight drain warps
constexpr int BAR_BYTES = 512, ITEMS = 8;
// chunks of an item that load magnitudes whatever they are: the drain warps look at them once, after the second,
// which they have left when the loads of the sixth begin
constexpr int MAG_CHUNKS = 5;
// what the drain warps of one half need of a tile
struct Tables {
    long long rowoff[BM], coloff[VN];
    E64Out g;   // grouped: the problem's
    short rowE[BM], colE[VN];
};
constexpr int smem_bytes(int np) { return ring_bytes(np) + BAR_BYTES + ITEMS * 16 + 6 * (int)sizeof(Tables) + 1024; }
constexpr int E_MIN = 1023 - 400, E_MAX = 1023 + 400;   // biased exponents of regular row maxima
// least sum of magnitudes of a stored result: 17/16 2^-7 of max|a| max|b|, the codes' products being in units of 2^-30
constexpr float MAG_MIN = 8912896.0f;

// instruction descriptor: FP32 accumulate, FP16 A and B, both K-major, M = 128, N = n
__host__ __device__ constexpr uint32_t idesc(int n) {
    return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
}

// the magnitudes': E5M2 A and B, N = 32
__host__ __device__ constexpr uint32_t idesc_mag() { return idesc(BN) | (1u << 7) | (1u << 10); }

__host__ __device__ __forceinline__ long long e64_items(const E64Args &g) {
    return (long long)g.mtiles * g.ntiles * g.ksplit;
}

// tile -> (m0, n0): groups of 16 row tiles, rows fastest within a group, so that resident CTAs share
// a few row tiles' planes in L2
__device__ __forceinline__ void e64_origin(int mtiles, int ntiles, int tile, int &m0, int &n0) {
    const int G = min(mtiles, 16), span = G * ntiles;
    const int grp = tile / span, in = tile - grp * span;
    const int gm = min(G, mtiles - grp * G);
    m0 = (grp * G + in % gm) * BM;
    n0 = (in / gm) * BN;
}

// The sums of one element, V = hi 2^36 + lo with hi = S_0 2^18 + S_1 2^9 + S_2 (|hi| < 1.01 K 2^34) and
// lo = S_3 2^27 + S_4 2^18 + S_5 2^9 + S_6, as T = V 2^(up - 36) in 64 bits: up shifts hi's leading bit to bit 61
// (at most by 30: then |hi| < 2^32), the bits of lo that fit follow.  The conversion of T is the one
// rounding; 500000 x 100 x 100 takes 0.58 ms with the conversion instruction, 0.61 ms with the same done in
// integer operations (about 25 on the half-rate integer pipe) and 0.71 ms with two FP64 additions.
__device__ __forceinline__ long long e64_join(long long hi, long long lo, int &up) {
    hi += lo >> 36;
    const unsigned r = (unsigned)(((unsigned long long)lo << 28) >> 32);   // lo mod 2^36, its top 32 bits
    const unsigned h0 = (unsigned)hi;
    const int h1 = (int)(hi >> 32);
    up = min(30, __clz(h1 ^ (h1 >> 31)) - 2);
    const unsigned t1 = __funnelshift_l(h0, (unsigned)h1, up), t0 = __funnelshift_l(r, h0, up);
    return (long long)((unsigned long long)t1 << 32 | t0);
}

// One thread's row of a tile (8 columns): its sums become FP64 values (hi[j] is overwritten with
// the bits), and the checks above run.  mag: the elements' sums of magnitudes; ea: the row's biased exponent (0
// outside M or a zero row); colE: the columns' (shared memory).  Returns the columns left to the FP64 pipe.
template <bool LOW, class E>
__device__ __forceinline__ unsigned e64_finish(const E64Out &g, long long (&hi)[HB], const long long (&lo)[HB],
                                           const float (&mag)[HB], int ea, const E *colE) {
    const bool live = ea != 0;
    unsigned left = live && (ea < E_MIN || ea > E_MAX) ? (1u << HB) - 1 : 0u;
    const int neg = g.alpha_neg ? (int)0x80000000 : 0;
    const int sc0 = ea - 2 * 1022 - 70 + 36 + g.alpha_k;
#pragma unroll
    for (int j = 0; j < HB; ++j) {
        const int eb = colE[j];
        if (eb != 0 && ((unsigned)(eb - E_MIN) > (unsigned)(E_MAX - E_MIN) ||
                        (live && mag[j] > 0.0f && mag[j] < MAG_MIN)))
            left |= 1u << j;
        int up = 0;
        const double v = __ll2double_rn(LOW ? e64_join(hi[j], lo[j], up) : hi[j]);   // 0 for a zero row or column
        const int vh = __double2hiint(v);
        const int sc = (vh & 0x7FFFFFFF) ? (sc0 + eb - up) << 20 : 0;
        hi[j] = __double_as_longlong(__hiloint2double((vh + sc) ^ neg, __double2loint(v)));
    }
    if (!g.alpha_pow2) {
#pragma unroll
        for (int j = 0; j < HB; ++j) hi[j] = __double_as_longlong(g.alpha * __longlong_as_double(hi[j]));
    }
    return left;
}

// store one thread's row through the output modes (co: column offsets, -1 past N), without the columns left out
template <bool LEFT>
__device__ __forceinline__ void e64_store(const E64Out &g, const long long (&val)[HB], const long long *co,
                                          long long rowoff, unsigned left) {
    double *out = g.C + rowoff;
    if constexpr (LEFT) {
        for (int j = 0; j < HB; ++j) {
            if (co[j] < 0 || (left >> j & 1)) continue;
            long long x = val[0];   // no dynamic index into registers
#pragma unroll
            for (int i = 1; i < HB; ++i) x = i == j ? val[i] : x;
            const double v = __longlong_as_double(x);
            if (g.beta_mode == 0)
                out[co[j]] = v;
            else if (g.beta_mode == 1)
                red_add_f64(out + co[j], v);
            else
                out[co[j]] = g.beta_mode == 2 ? g.Cin[rowoff + co[j]] + v : fma(g.beta, g.Cin[rowoff + co[j]], v);
        }
        return;
    }
    if (g.beta_mode == 0) {
#pragma unroll
        for (int j = 0; j < HB; ++j)
            if (co[j] >= 0) out[co[j]] = __longlong_as_double(val[j]);
    } else if (g.beta_mode == 1) {
        // one owner per element: the L2's FP64 add gives the same sum as a load, add and store
#pragma unroll
        for (int j = 0; j < HB; ++j)
            if (co[j] >= 0) red_add_f64(out + co[j], __longlong_as_double(val[j]));
    } else {
        const double *in = g.Cin + rowoff;
        double cin[HB];
#pragma unroll
        for (int j = 0; j < HB; ++j) cin[j] = co[j] >= 0 ? __ldcs(in + co[j]) : 0.0;
#pragma unroll
        for (int j = 0; j < HB; ++j) {
            if (co[j] < 0) continue;
            const double v = __longlong_as_double(val[j]);
            out[co[j]] = g.beta_mode == 2 ? cin[j] + v : fma(g.beta, cin[j], v);
        }
    }
}

// barrier over the 256 drain threads of one half (named barrier 1 or 2) that counts, or ORs, a predicate over them
__device__ __forceinline__ unsigned vote_count(int half, bool pred) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "bar.red.popc.u32 %0, %3, %2, p;\n\t}"
        : "=r"(r)
        : "r"((uint32_t)pred), "n"(DRAIN / 2), "r"(half + 1)
        : "memory");
    return r;
}
__device__ __forceinline__ bool vote_any(int half, bool pred) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "bar.red.or.pred q, %3, %2, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(r)
        : "r"((uint32_t)pred), "n"(DRAIN / 2), "r"(half + 1)
        : "memory");
    return r != 0;
}

// A half tile (16 columns, the unit of a vote) of which n > 0 threads left columns out: listed whole, or where they
// are few, piece by piece; the caller stores the rest of a half tile listed by pieces (true).  lost: a thread's
// sums are not there (a failed wait): nothing of the half tile is listed or stored, the host reports the time-out.
// slot: two ints of shared memory of the half's own, free again at its next vote.
__device__ __forceinline__ bool e64_list_half(const E64Out &g, int prob, int m0, int n0, int half, unsigned n, unsigned left,
                                              bool lost, int row, int group, bool first, int *slot) {
    const int t = (int)((g.row0 + m0) / BM + g.mtiles_all * (n0 / VN));
    if (n > E64_FINE) {
        if (!vote_any(half, lost) && first && n0 < g.N) {
            const int at = atomicAdd(g.list, 1);
            g.list[2 + 2 * (long long)at] = prob;
            g.list[3 + 2 * (long long)at] = t;
        }
        return false;
    }
    if (first) {
        slot[0] = atomicAdd(g.list + 1, 1);
        slot[1] = 0;
    }
    __syncwarp();
    const bool none = vote_any(half, lost);
    int *f = g.fine + (long long)slot[0] * E64_FINE_INTS;
    if (first) {
        f[0] = prob;
        f[1] = t;
        f[2] = none ? 0 : (int)n;
    }
    __syncwarp();
    if (none) return false;
    const unsigned who = __ballot_sync(0xffffffffu, left != 0);
    if (who) {
        const int lane = threadIdx.x & 31, lead = __ffs(who) - 1;
        int at = 0;
        if (lane == lead) at = atomicAdd(slot + 1, __popc(who));
        at = __shfl_sync(0xffffffffu, at, lead) + __popc(who & ((1u << lane) - 1));
        if (left) reinterpret_cast<uint16_t *>(f + 3)[at] = (uint16_t)(row | group << 7 | left << 8);
    }
    return true;
}

// acc += integer(x) 2^sh, x the bits of an integer-valued FP32 sum
template <int SH>
__device__ __forceinline__ void add_sum(long long &acc, uint32_t x) {
    asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(acc) : "r"(__float2int_rn(__uint_as_float(x))), "n"(1 << SH));
}

// Persistent: CTA b takes work items b, b + gridDim.x, ... (an item is one tile over one K part).
// Warp 0 issues TMA, warp 1 owns TMEM and issues the MMAs, warps 2-17 drain (four per 32-lane TMEM
// quarter, 8 columns each).  Every wait is bounded; on expiry the CTA raises FLAG_TIMEOUT, skips its
// stores, waits for its own copies, frees TMEM and returns.
// GROUPED: the launch covers ngp problems (gp, in order of item0) whose operand rows lie in shared planes;
// item w belongs to the last problem with item0 <= w.  PL digit planes: 7 (FP64), or 3 = 27 bits with the six
// products of j < 3 (split precision); plane PL holds the magnitudes.
template <int PL, bool GROUPED>
__global__ void __launch_bounds__(THREADS, 1)
    gett_e64_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB,
                    const __grid_constant__ CUtensorMap magA, const __grid_constant__ CUtensorMap magB,
                    const __grid_constant__ E64Args g0, const E64Args *__restrict__ gp, int ngp, int nitems) {
    constexpr int B_BYTES = b_bytes(PL), RING_BYTES = ring_bytes(PL), BUF_COLS = (PL + 1) * BN;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t *ringB = smem + SLOTS * A_BYTES;
    uint64_t *afull = reinterpret_cast<uint64_t *>(smem + RING_BYTES);
    uint64_t *aempty = afull + SLOTS;
    uint64_t *bfull = aempty + SLOTS;    // [2]
    uint64_t *bempty = bfull + 2;
    uint64_t *cfull = bempty + 2;        // [2] chunk accumulated in TMEM buffer
    uint64_t *cempty = cfull + 2;        // [2] chunk drained
    uint64_t *fin = cempty + 2;          // the MMA thread's last commit
    uint64_t *ifull = fin + 1;           // [ITEMS] an item's place is in the queue
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(ifull + ITEMS);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    int *slots = reinterpret_cast<int *>(tmem_slot + 2);   // two ints per half (e64_list_half)
    int *judged = slots + 4;                               // [ITEMS] drain warps whose elements have enough magnitude
    int4 *queue = reinterpret_cast<int4 *>(smem + RING_BYTES + BAR_BYTES);   // [ITEMS] m0, n0, chunks, problem | part
    Tables *tabs = reinterpret_cast<Tables *>(queue + ITEMS);                // three sets per half

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // the problem of item w, cur running on from the item before; what the loops need of it in registers
    struct Shape {
        int mtiles, ntiles, item0, k16, kper, rowA, rowB;
    };
    auto load_shape = [](const E64Args &g) {
        return Shape{g.mtiles, g.ntiles, g.item0, g.k16, g.kper, g.rowA, g.rowB};
    };
    auto locate = [&](int w, int &cur, Shape &h) {
        if constexpr (GROUPED) {
            bool moved = false;
            while (cur + 1 < ngp && gp[cur + 1].item0 <= w) {
                ++cur;
                moved = true;
            }
            if (moved) h = load_shape(gp[cur]);
        }
    };
    auto first_shape = [&]() { return load_shape(GROUPED ? gp[0] : g0); };
    unsigned *const flags = g0.flags;

    if (threadIdx.x == 0) {
        for (int s = 0; s < SLOTS; ++s) {
            mbar_init(&afull[s], 1);
            mbar_init(&aempty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&bfull[b], 1);
            mbar_init(&bempty[b], 1);
            mbar_init(&cfull[b], 1);
            mbar_init(&cempty[b], DRAIN);
        }
        for (int i = 0; i < ITEMS; ++i) mbar_init(&ifull[i], 1);
        mbar_init(fin, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            // TMA: per chunk B's planes, then A's one by one; it counts A planes, gc chunks
            unsigned it = 0, gc = 0;
            int cur = 0;
            Shape g = first_shape();
            bool stop = false;
            auto wait = [&](uint64_t *bar, unsigned parity) {
                if (mbar_wait(bar, parity, abort_flag, flags)) return true;
                *abort_flag = 1;
                stop = true;
                return false;
            };
            unsigned ni = 0;
            for (int w = blockIdx.x; w < nitems && !stop; w += gridDim.x, ++ni) {
                locate(w, cur, g);
                const int tiles = g.mtiles * g.ntiles, x = w - g.item0;
                const int tile = x % tiles, part = x / tiles;
                int m0, n0;
                e64_origin(g.mtiles, g.ntiles, tile, m0, n0);
                const int c0 = part * g.kper, c1 = min((g.k16 + 3) / 4, c0 + g.kper);
                // the item's place for the drain warps.  Entry ni - 8 is read by then: B's buffer of item ni is
                // free once the MMAs of item ni - 2 are done, whose accumulators item ni - 4 has left.
                if (!wait(&bempty[gc & 1u], ((gc >> 1) & 1u) ^ 1u)) break;
                queue[ni % ITEMS] = make_int4(m0, n0, c1 - c0, GROUPED ? cur : part * tiles + tile);
                judged[ni % ITEMS] = 0;
                bool mags = true;
                mbar_arrive(&ifull[ni % ITEMS]);
                m0 += g.rowA;
                n0 += g.rowB;
                for (int c = c0; c < c1 && !stop; ++c, ++gc) {
                    const unsigned b = gc & 1u;
                    if (c > c0 && !wait(&bempty[b], ((gc >> 1) & 1u) ^ 1u)) break;
                    // Where every element of the tile has enough magnitude the item's further chunks load no more (a
                    // grouped launch's items are too short): their MMAs add those of an earlier chunk, which
                    // change nothing.  Read without an order: it decides about time alone.
                    if (!GROUPED && c == c0 + MAG_CHUNKS) mags = *(volatile int *)&judged[ni % ITEMS] < DRAIN / 32;
                    uint8_t *const bb = ringB + b * B_BYTES, *const mb = bb + PL * BN * CK * 2;
                    mbar_expect_tx(&bfull[b], mags ? B_BYTES : PL * BN * CK * 2);
                    tma_load_3d(bb, &mapB, &bfull[b], c * CK, n0, 0);
                    if (mags) {
                        tma_load_3d(mb, &magB, &bfull[b], c * CK, n0, 0);
                        tma_load_3d(mb + BN * CK, &magA, &bfull[b], c * CK, m0, 0);
                    }
                    for (int p = 0; p < PL; ++p, ++it) {
                        const unsigned s = it % SLOTS;
                        if (!wait(&aempty[s], ((it / SLOTS) & 1u) ^ 1u)) break;
                        mbar_expect_tx(&afull[s], A_BYTES);
                        tma_load_3d(smem + s * A_BYTES, &mapA, &afull[s], c * CK, m0, p);
                    }
                }
            }
            // the last copy into each buffer has landed (immediate unless an abort cut the MMA
            // thread short), so none is in flight when the CTA exits
            for (unsigned s = 0; s < SLOTS; ++s)
                if (it > s) mbar_wait_quiet(&afull[s], ((s + (it - 1 - s) / SLOTS * SLOTS) / SLOTS) & 1u);
            for (unsigned b = 0; b < 2; ++b)
                if (gc > b) mbar_wait_quiet(&bfull[b], ((b + (gc - 1 - b) / 2 * 2) >> 1) & 1u);
        }
    } else if (warp == 1) {
        // The whole warp walks the loops in step (see umma_warp)
        const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
        unsigned s = 0, ph = 0, gc = 0;   // ring slot and its phase, chunks
        int cur = 0;
        Shape g = first_shape();
        bool stop = false;
        for (int w = blockIdx.x; w < nitems && !stop; w += gridDim.x) {
            locate(w, cur, g);
            const int part = (w - g.item0) / (g.mtiles * g.ntiles);
            int k16 = g.k16, c0 = part * g.kper, c1 = min((k16 + 3) / 4, c0 + g.kper);
            if constexpr (GROUPED) {   // read from memory: warp-uniform by construction
                k16 = __shfl_sync(0xffffffffu, k16, 0);
                c0 = __shfl_sync(0xffffffffu, c0, 0);
                c1 = __shfl_sync(0xffffffffu, c1, 0);
            }
            for (int c = c0; c < c1; ++c, ++gc) {
                const unsigned b = gc & 1u;
                if ((gc >= 2 && !mbar_wait_warp(&cempty[b], ((gc >> 1) - 1u) & 1u, abort_flag, flags)) ||
                    !mbar_wait_warp(&bfull[b], (gc >> 1) & 1u, abort_flag, flags)) {
                    stop = true;
                    break;
                }
                const uint32_t b0 = sw128_lo(ringB + b * B_BYTES);
                const uint32_t dbuf = tm + b * BUF_COLS;
                const int steps = min(4, k16 - 4 * c);
#pragma unroll
                for (int p = 0; p < PL; ++p) {
                    if (!mbar_wait_warp(&afull[s], ph, abort_flag, flags)) {
                        stop = true;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t a0 = sw128_lo(smem + s * A_BYTES);
                    if (steps == 4) {
                        umma_warp_x4(dbuf + (uint32_t)(p * BN), a0, b0, idesc((PL - p) * BN), p == 0 ? 0u : 1u);
                    } else {
                        for (int kk = 0; kk < steps; ++kk)   // 32 bytes per K = 16 step
                            umma_warp(dbuf + (uint32_t)(p * BN), a0 + 2 * kk, b0 + 2 * kk, idesc((PL - p) * BN),
                                      (p == 0 && kk == 0) ? 0u : 1u);
                    }
                    umma_commit_warp(&aempty[s]);
                    if (++s == SLOTS) {
                        s = 0;
                        ph ^= 1u;
                    }
                }
                if (stop) break;
                // the magnitudes: 32 bytes per K = 32 step
                const uint32_t bm = b0 + (PL * BN * CK * 2 >> 4), am = bm + (BN * CK >> 4);
                umma_warp_f8(dbuf + (uint32_t)(PL * BN), am, bm, idesc_mag(), 0u);
                if (steps > 2) umma_warp_f8(dbuf + (uint32_t)(PL * BN), am + 2, bm + 2, idesc_mag(), 1u);
                umma_commit_warp(&bempty[b]);
                umma_commit_warp(&cfull[b]);
            }
        }
        if (stop) *abort_flag = 1;
        __syncwarp();
        // every MMA this warp issued has completed before TMEM is freed
        umma_commit_warp(fin);
        mbar_wait_quiet(fin, 0u);
    } else {
        // Per tile: add the chunks up, read the next tile's place and make its tables (their latency overlaps
        // the conversion), finish, vote, store.  Each half of the tile's columns belongs to eight warps
        // that vote and list by themselves, so that the halves drift apart and one's conversions overlap
        // the other's waits.  The vote is the only barrier: the tables of tile w + 1 are written before the
        // vote of tile w, and a thread still storing tile w - 1 reads others (three sets).  A failed wait
        // makes the warp skip TMEM from then on but keep voting (its tiles are not stored), so no thread is
        // left waiting at a barrier.
        const int quarter = warp & 3, eighth = (warp - 2) >> 2, half = eighth >> 1, sub = (eighth & 1) * HB;
        const int dt = (threadIdx.x - 64) & 255;   // within the half: warps 2-9 are half 0, 10-17 half 1
        unsigned gc = 0, ni = 0, nd = 0;   // chunks, items opened and drained
        int set = 0;
        bool bad = false;
        Tables *const mine = tabs + 3 * half;
        // the next item's place (m0, n0, chunks, problem or part's tile), its tables into set tb
        auto open = [&](int tb) -> int4 {
            if (!bad) {
                const bool got = mbar_wait(&ifull[ni % ITEMS], (ni / ITEMS) & 1u, abort_flag, flags);
                if (!__all_sync(0xffffffffu, got)) {
                    *abort_flag = 1;
                    bad = true;
                }
            }
            if (bad) return make_int4(0, 0, 0, 0);
            const int4 I = queue[ni % ITEMS];
            ++ni;
            const E64Args &g = GROUPED ? gp[I.w] : g0;
            Tables &T = mine[tb];
            if constexpr (GROUPED) {
                if (dt >= 160 && dt - 160 < (int)(sizeof(E64Out) / 8))
                    reinterpret_cast<long long *>(&T.g)[dt - 160] =
                        reinterpret_cast<const long long *>(static_cast<const E64Out *>(&g))[dt - 160];
            }
            if (GROUPED || g.ksplit == 1) {
                if (dt < BM) {
                    const long long m = (long long)I.x + dt;
                    T.rowoff[dt] = m < g.M ? mode_off(g.mC, g.row0 + m) : -1;
                    T.rowE[dt] = (short)(m < g.M ? __ldg(g.expA + m) : 0);
                } else if (dt < BM + VN) {
                    const int c = dt - BM;
                    const long long n = (long long)I.y + half * VN + c;
                    T.coloff[c] = n < g.N ? mode_off(g.nC, n) : -1;
                    T.colE[c] = (short)(n < g.N ? __ldg(g.expB + n) : 0);
                }
            }
            return I;
        };
        int4 I = make_int4(0, 0, 0, 0);
        if ((int)blockIdx.x < nitems) I = open(0);
        vote_any(half, false);
        const int row = quarter * 32 + lane;
        for (int w = blockIdx.x; w < nitems; w += gridDim.x, ++nd) {
            const Tables &T = mine[set];
            const E64Out &g = GROUPED ? T.g : static_cast<const E64Out &>(g0);
            long long hi[HB], lo[HB];
            float mag[HB];
#pragma unroll
            for (int j = 0; j < HB; ++j) {
                hi[j] = lo[j] = 0;
                mag[j] = 0.0f;
            }
            for (int c = 0; c < I.z; ++c, ++gc) {
                const unsigned buf = gc & 1u;
                if (!bad) {
                    const bool got = mbar_wait(&cfull[buf], (gc >> 1) & 1u, abort_flag, flags);
                    if (!__all_sync(0xffffffffu, got)) {
                        *abort_flag = 1;
                        bad = true;   // the whole warp
                    }
                }
                if (bad) continue;
                __syncwarp();
                tc_fence_after();
                const uint32_t base =
                    tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * BUF_COLS + eighth * HB);
                uint32_t r0[HB], r1[HB], r2[HB], rm[HB];
                tmem_ld8(base, r0);
                tmem_ld8(base + BN, r1);
                tmem_ld8(base + 2 * BN, r2);
                tmem_ld8(base + PL * BN, rm);
                tmem_ld_wait();
                if constexpr (PL == 3) {
                    tc_fence_before();
                    mbar_arrive(&cempty[buf]);
                }
#pragma unroll
                for (int j = 0; j < HB; ++j) {
                    add_sum<18>(hi[j], r0[j]);
                    add_sum<9>(hi[j], r1[j]);
                    add_sum<0>(hi[j], r2[j]);
                    mag[j] += __uint_as_float(rm[j]);
                }
                if constexpr (PL > 3) {
                    uint32_t r3[HB];
                    tmem_ld8(base + 3 * BN, r0);
                    tmem_ld8(base + 4 * BN, r1);
                    tmem_ld8(base + 5 * BN, r2);
                    tmem_ld8(base + 6 * BN, r3);
                    tmem_ld_wait();
                    tc_fence_before();
                    mbar_arrive(&cempty[buf]);
#pragma unroll
                    for (int j = 0; j < HB; ++j) {
                        add_sum<27>(lo[j], r0[j]);
                        add_sum<18>(lo[j], r1[j]);
                        add_sum<9>(lo[j], r2[j]);
                        add_sum<0>(lo[j], r3[j]);
                    }
                }
                if (!GROUPED && c == 1 && I.z > MAG_CHUNKS) {
                    // does an element still lack magnitude?  Rows and columns of zeros or past the edge need none (K
                    // parts have no tables: all do)
                    const bool tables = g0.ksplit == 1;
                    bool lacks = false;
#pragma unroll
                    for (int j = 0; j < HB; ++j) lacks |= mag[j] < MAG_MIN && (!tables || T.colE[sub + j] != 0);
                    lacks = lacks && (!tables || T.rowE[row] != 0);
                    if (!__any_sync(0xffffffffu, lacks) && lane == 0) atomicAdd(&judged[nd % ITEMS], 1);
                }
            }
            const int m0 = I.x, n0 = I.y + half * VN, at = I.w;
            set = set == 2 ? 0 : set + 1;
            if (w + (int)gridDim.x < nitems) I = open(set);
            if (!GROUPED && g0.ksplit > 1) {
                const long long at0 = ((long long)at * BN + eighth * HB) * BM + row;
#pragma unroll
                for (int j = 0; j < HB; ++j) {
                    g0.part[at0 + j * BM] = make_longlong2(hi[j], lo[j]);
                    g0.pmag[at0 + j * BM] = mag[j];
                }
                continue;
            }
            const unsigned left = e64_finish<(PL > 3)>(g, hi, lo, mag, T.rowE[row], T.colE + sub);
            const unsigned n = vote_count(half, left || bad);
            if (n == 0) {
                if (T.rowoff[row] >= 0) e64_store<false>(g, hi, T.coloff + sub, T.rowoff[row], 0u);
            } else if (e64_list_half(g, GROUPED ? at : 0, m0, n0, half, n, left, bad, row, sub / HB, dt == 0,
                                     slots + 2 * half) &&
                       T.rowoff[row] >= 0) {
                e64_store<true>(g, hi, T.coloff + sub, T.rowoff[row], left);
            }
        }
        const bool ok = !bad;
        if (!ok && lane == 0) atomicOr(flags, FLAG_TIMEOUT);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, TMEM_COLS);
    }
}

// K parts, many of them: adds each group of PART_FOLD parts into its first one, an element a thread.  Latency
// bounds the parts' pass: a tile's block took 1 us for each of up to 64 parts (100 x 50 x 4000, two tiles: 66
// us, with this launch 16).
constexpr int PART_FOLD = 8;
__global__ void __launch_bounds__(256) e64_fold_kernel(longlong2 *__restrict__ part, float *__restrict__ pmag,
                                                       int ksplit, long long n) {
    const long long i = blockIdx.x * 256LL + threadIdx.x;
    const int s0 = blockIdx.y * PART_FOLD;
    if (i >= n) return;
    longlong2 x[PART_FOLD];
    float m[PART_FOLD];
#pragma unroll
    for (int s = 0; s < PART_FOLD; ++s) {
        x[s] = s0 + s < ksplit ? part[(s0 + s) * n + i] : make_longlong2(0, 0);
        m[s] = s0 + s < ksplit ? pmag[(s0 + s) * n + i] : 0.0f;
    }
#pragma unroll
    for (int s = 1; s < PART_FOLD; ++s) {
        x[0].x += x[s].x;
        x[0].y += x[s].y;
        m[0] += m[s];
    }
    part[s0 * n + i] = x[0];
    pmag[s0 * n + i] = m[0];
}

// K parts: one block per tile adds every step-th part's 64-bit sums (exact, so their number does not matter)
// and finishes the tile as the main kernel does
__global__ void __launch_bounds__(DRAIN) e64_parts_kernel(const E64Args g, int step) {
    __shared__ long long coloff[BN];
    __shared__ int colE[BN], slots[4];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int quarter = warp & 3, eighth = warp >> 2, half = eighth >> 1;
    const int tile = blockIdx.x, tiles = g.mtiles * g.ntiles;
    int m0, n0;
    e64_origin(g.mtiles, g.ntiles, tile, m0, n0);
    if (threadIdx.x < BN) {
        const long long n = (long long)n0 + threadIdx.x;
        coloff[threadIdx.x] = n < g.N ? mode_off(g.nC, n) : -1;
        colE[threadIdx.x] = n < g.N ? __ldg(g.expB + n) : 0;
    }
    const long long mrow = (long long)m0 + quarter * 32 + lane;
    const int ea = mrow < g.M ? __ldg(g.expA + mrow) : 0;
    long long hi[HB], lo[HB];
    float mag[HB];
#pragma unroll
    for (int j = 0; j < HB; ++j) {
        hi[j] = lo[j] = 0;
        mag[j] = 0.0f;
    }
#pragma unroll 2
    for (int s = 0; s < g.ksplit; s += step) {
        const long long at = (((long long)s * tiles + tile) * BN + eighth * HB) * BM + quarter * 32 + lane;
#pragma unroll
        for (int j = 0; j < HB; ++j) {
            const longlong2 p = g.part[at + j * BM];
            hi[j] += p.x;
            lo[j] += p.y;
            mag[j] += g.pmag[at + j * BM];
        }
    }
    __syncthreads();
    const unsigned left = e64_finish<true>(g, hi, lo, mag, ea, colE + eighth * HB);
    const unsigned n = vote_count(half, left != 0);
    if (n == 0) {
        if (mrow < g.M) e64_store<false>(g, hi, coloff + eighth * HB, mode_off(g.mC, g.row0 + mrow), 0u);
    } else if (e64_list_half(g, 0, m0, n0 + half * VN, half, n, left, false, quarter * 32 + lane, eighth & 1,
                             (threadIdx.x & 255) == 0, slots + 2 * half) &&
               mrow < g.M) {
        e64_store<true>(g, hi, coloff + eighth * HB, mode_off(g.mC, g.row0 + mrow), left);
    }
}

// ---------------------------------------------------------------------------------------------
// operand digits
// ---------------------------------------------------------------------------------------------
// pack block: 2048 elements, 32 rows x 64 K where K <= 64 and 16 rows x 128 K above
constexpr int PK = 128;
constexpr int pack_rows(long long kpad) { return kpad <= 64 ? 32 : 16; }
constexpr int pack_k(long long kpad) { return kpad <= 64 ? 64 : 128; }

// one operand of a pack launch: rows [row0, row0 + R) of src into digit planes [NP][Rpad][Kpad], magnitudes
// [Rpad][mag_pitch] and the rows' exponents
struct PackArgs {
    const double *src;
    Mode rm, km;
    long long row0, R, K, Rpad, Kpad;
    int *exps;
    __half *dst;
    uint8_t *mag;
    unsigned blocks;   // of this operand in the launch
    int kfast;         // K (else the row index) is the source's unit-stride index
    int kseg;          // row-maximum pass: K chunks per block
};

// row maxima are taken over the magnitudes' high words, with a low bit set where the low word is not zero;
// the biased exponent of such a maximum is 1 for subnormals, which mark a row the tensor cores do not take
__device__ __forceinline__ unsigned mag_of(double x) {
    return ((unsigned)__double2hiint(x) & 0x7FFFFFFFu) | min((unsigned)__double2loint(x), 1u);
}
__device__ __forceinline__ int exp_of(unsigned mag) { return mag >> 20 ? (int)(mag >> 20) : (mag ? 1 : 0); }

// x in units of 2^-(9 PL - 1) of its row's power of two, rounded with ties away from zero, with the offset
// that makes its 9-bit fields the balanced digits + 256 (0..512).  base is shift_base() of the row
template <int PL>
__device__ __forceinline__ int shift_base(int E) {
    return (E ? E : 2000) + 9 * (E64_NP - PL);   // a row of zeros: everything is shifted out
}
template <int PL>
__device__ __forceinline__ unsigned long long fixed_point(double x, int base) {
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    // m 2^(9 PL - 54) >> (E - e): t = m 2^10 >> sh, then (t + 1) >> 1; below zero (-t) >> 1 = (~t + 1) >> 1
    const unsigned long long m = (((unsigned long long)((hi & 0xFFFFFu) | 0x100000u) << 32) | lo) << 10;
    const long long neg = (long long)((int)hi >> 31);
    const long long t = (long long)(m >> min(base - (int)(hi >> 20 & 0x7FFu), 63)) ^ neg;
    unsigned long long OFF = 0;
#pragma unroll
    for (int p = 0; p < PL; ++p) OFF += 256ull << (9 * p);
    return (unsigned long long)((t + 1) >> 1) + OFF;
}

// digits p of two numbers as a pair of FP16 integers: 0x6400 | u is 1024 + u (the first digit, up to 512,
// takes ten bits of its own)
template <int PL>
__device__ __forceinline__ uint32_t digit_pair(unsigned long long s0, unsigned long long s1, int p) {
    const int sh = 9 * (PL - 1 - p);
    const uint32_t w = (__byte_perm((uint32_t)(s0 >> sh), (uint32_t)(s1 >> sh), 0x5410) &
                        (p ? 0x01FF01FFu : 0x03FF03FFu)) | 0x64006400u;
    const uint32_t b = 0x65006500u;   // 1280
    const __half2 h = __hsub2(*reinterpret_cast<const __half2 *>(&w), *reinterpret_cast<const __half2 *>(&b));
    return *reinterpret_cast<const uint32_t *>(&h);
}

// |x| in units of 2^-15 of its row's power of two as E5M2: the exponent field is 29 for elements of the maximum's
// binade, the mantissa's two leading bits follow.  Smaller nonzero elements count as 2^-29 of it (the least
// normal code), so that a sum of magnitudes is zero only where no two nonzero elements meet; over 2^16 K values
// that adds less than 1/64 of MAG_MIN.
__device__ __forceinline__ uint32_t mag_code(double x, int E) {
    const unsigned h = (unsigned)__double2hiint(x) & 0x7FFFFFFFu;
    const int c = max((int)(h >> 18) - ((E - 29) << 2), 4);
    return h | (unsigned)__double2loint(x) ? (uint32_t)c : 0u;
}

template <int PL, int KW>
struct PackSmem {
    static constexpr int PR = 2048 / KW;
    uint32_t outp[PL][PR][KW / 2 + 4];   // pitch: 16-byte pieces, the pair stores of both layouts free of conflicts
    uint16_t mag[PR][KW / 2 + 4];        // pairs of magnitudes, 8-byte pieces
    long long roff[PR], koff[KW];
    unsigned rowE[PR];                   // the rows' exponents; LOCALMAX: their largest magnitudes
};

// LOCALMAX: the block sees whole rows (K <= KW) and writes their exponents; else they are read.  Integer issue
// and the block's three phases bound it: 23 bytes an element (8 read, 15 written) at 3.6 to 4.1 TB/s of 6.7.
// The digits stay one 64-bit number until two of them are put into an FP16 pair, padded K is skipped, and a
// thread writes one 16-byte piece of each plane (500000 x 100: 345 -> 305 us; 6400^2: 352 -> 306).
template <int PL, int KW, bool KFAST, bool LOCALMAX>
__device__ __forceinline__ void e64_pack_block(const PackArgs &a, long long r0, long long k0, PackSmem<PL, KW> &sm) {
    constexpr int PR = 2048 / KW, PAIRS = KW / 2;
    const int tid = threadIdx.x, lane = tid & 31;
    if (tid < PR) {
        const long long r = r0 + tid;
        sm.roff[tid] = r < a.R ? mode_off(a.rm, a.row0 + r) : -1;
        sm.rowE[tid] = LOCALMAX ? 0 : (r < a.R ? a.exps[r] : 0);
    } else if (tid >= 64 && tid < 64 + KW) {
        const long long k = k0 + tid - 64;
        sm.koff[tid - 64] = k < a.K ? mode_off(a.km, k) : -1;
    }
    __syncthreads();
    // KFAST: a warp's lanes along K; else eight rows x four pairs of K
    constexpr int RB = PR / 8;
    const int warp = tid >> 5;
    auto row_of = [&](int i) { return KFAST ? tid / PAIRS + (256 / PAIRS) * i : (lane & 7) + 8 * (warp % RB); };
    auto pair_of = [&](int i) { return KFAST ? tid & (PAIRS - 1) : (lane >> 3) + 4 * (warp / RB) + (32 / RB) * i; };
    const int pairs = (int)min((long long)KW, a.Kpad - k0) / 2;
    double x[4][2];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const long long ro = sm.roff[row_of(i)], ko = sm.koff[2 * pair_of(i) + h];
            x[i][h] = (ro >= 0 && ko >= 0) ? __ldg(a.src + ro + ko) : 0.0;
        }
    if constexpr (LOCALMAX) {
        if constexpr (KFAST) {
            // a warp's lanes share each of its four rows
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const unsigned m = __reduce_max_sync(0xffffffffu, max(mag_of(x[i][0]), mag_of(x[i][1])));
                if (lane == 0) atomicMax(&sm.rowE[row_of(i)], m);
            }
        } else {
            unsigned m = 0;
#pragma unroll
            for (int i = 0; i < 4; ++i) m = max(m, max(mag_of(x[i][0]), mag_of(x[i][1])));
            m = max(m, __shfl_xor_sync(0xffffffffu, m, 8));
            m = max(m, __shfl_xor_sync(0xffffffffu, m, 16));
            if (lane < 8) atomicMax(&sm.rowE[row_of(0)], m);
        }
        __syncthreads();
        if (tid < PR) a.exps[r0 + tid] = exp_of(sm.rowE[tid]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = row_of(i), c = pair_of(i);
        if (c >= pairs) continue;
        const int E = LOCALMAX ? exp_of(sm.rowE[r]) : (int)sm.rowE[r], base = shift_base<PL>(E);
        const unsigned long long s0 = fixed_point<PL>(x[i][0], base), s1 = fixed_point<PL>(x[i][1], base);
#pragma unroll
        for (int p = 0; p < PL; ++p) sm.outp[p][r][c] = digit_pair<PL>(s0, s1, p);
        sm.mag[r][c] = (uint16_t)(E ? mag_code(x[i][0], E) | mag_code(x[i][1], E) << 8 : 0u);
    }
    __syncthreads();
    // one piece of eight halves of each plane to a thread
    const int seg = tid & (KW / 8 - 1), row = tid / (KW / 8);
    if (4 * seg >= pairs) return;
    __half *dst = a.dst + (size_t)(r0 + row) * a.Kpad + k0 + 8 * seg;
    const size_t plane = (size_t)a.Rpad * a.Kpad;
#pragma unroll
    for (int p = 0; p < PL; ++p, dst += plane)
        *reinterpret_cast<uint4 *>(dst) = *reinterpret_cast<const uint4 *>(&sm.outp[p][row][4 * seg]);
    *reinterpret_cast<uint2 *>(a.mag + (size_t)(r0 + row) * mag_pitch(a.Kpad) + k0 + 8 * seg) =
        *reinterpret_cast<const uint2 *>(&sm.mag[row][4 * seg]);
}

// both operands of a GEMM in one launch: blocks [0, a.blocks) pack a, the rest b
template <int PL, int KW, bool LOCALMAX>
__global__ void __launch_bounds__(256, 5) e64_pack_kernel(const __grid_constant__ PackArgs a,
                                                          const __grid_constant__ PackArgs b) {
    __shared__ __align__(16) PackSmem<PL, KW> sm;
    const bool second = blockIdx.x >= a.blocks;
    const PackArgs &P = second ? b : a;
    const unsigned blk = second ? blockIdx.x - a.blocks : blockIdx.x;
    const unsigned kb = (unsigned)((P.Kpad + KW - 1) / KW), rb = (unsigned)(P.Rpad / (2048 / KW));
    if (P.kfast)
        e64_pack_block<PL, KW, true, LOCALMAX>(P, (long long)(blk / kb) * (2048 / KW), (long long)(blk % kb) * KW, sm);
    else
        e64_pack_block<PL, KW, false, LOCALMAX>(P, (long long)(blk % rb) * (2048 / KW), (long long)(blk / rb) * KW, sm);
}

// many operands with K <= KW (a batch): block b packs the rows of the last operand with first[] <= b; Rpad is
// the rows of the shared planes, dst and exps start at the operand's own rows
template <int PL, int KW>
__global__ void __launch_bounds__(256, 5) e64_pack_grouped_kernel(const PackArgs *__restrict__ ops,
                                                                  const unsigned *__restrict__ first, int nops) {
    __shared__ __align__(16) PackSmem<PL, KW> sm;
    int lo = 0, hi = nops - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (first[mid] <= blockIdx.x) lo = mid; else hi = mid - 1;
    }
    const PackArgs P = ops[lo];
    const long long r0 = (long long)(blockIdx.x - first[lo]) * (2048 / KW);
    if (P.kfast)
        e64_pack_block<PL, KW, true, true>(P, r0, 0, sm);
    else
        e64_pack_block<PL, KW, false, true>(P, r0, 0, sm);
}

// the rows' largest biased exponents for K > 128 (exps cleared before): a block covers 16 rows x kseg
// chunks of 128 K
constexpr int PR = 16;
template <bool KFAST>
__device__ __forceinline__ void e64_rowmax_block(const PackArgs &a, long long r0, long long k0) {
    __shared__ long long roff[PR], koff[PK];
    __shared__ unsigned rowE[PR];
    const int tid = threadIdx.x, lane = tid & 31;
    if (tid < PR) {
        const long long r = r0 + tid;
        roff[tid] = r < a.R ? mode_off(a.rm, a.row0 + r) : -1;
        rowE[tid] = 0;
    }
    unsigned m[4] = {0, 0, 0, 0};
    for (int c = 0; c < a.kseg && k0 + (long long)c * PK < a.K; ++c) {
        __syncthreads();
        if (tid >= 64 && tid < 64 + PK) {
            const long long k = k0 + (long long)c * PK + tid - 64;
            koff[tid - 64] = k < a.K ? mode_off(a.km, k) : -1;
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int row = KFAST ? (tid >> 6) + 4 * i : (tid & 15);
            const int k = KFAST ? (tid & 63) : (tid >> 4) + 16 * i;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const long long ro = roff[row], ko = koff[k + 64 * h];
                if (ro >= 0 && ko >= 0) m[i] = max(m[i], mag_of(__ldg(a.src + ro + ko)));
            }
        }
    }
    __syncthreads();
    if constexpr (KFAST) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const unsigned x = __reduce_max_sync(0xffffffffu, m[i]);
            if (lane == 0) atomicMax(&rowE[(tid >> 6) + 4 * i], x);
        }
    } else {
        unsigned x = max(max(m[0], m[1]), max(m[2], m[3]));
        x = max(x, __shfl_xor_sync(0xffffffffu, x, 16));
        if (lane < 16) atomicMax(&rowE[lane], x);
    }
    __syncthreads();
    if (tid < PR && r0 + tid < a.R && rowE[tid]) atomicMax(&a.exps[r0 + tid], exp_of(rowE[tid]));
}

__global__ void __launch_bounds__(256) e64_rowmax_kernel(const __grid_constant__ PackArgs a,
                                                         const __grid_constant__ PackArgs b) {
    const unsigned na = (unsigned)(a.blocks ? (a.Rpad / PR) * ((a.K + PK * a.kseg - 1) / (PK * a.kseg)) : 0);
    const bool second = blockIdx.x >= na;
    const PackArgs &P = second ? b : a;
    const unsigned blk = second ? blockIdx.x - na : blockIdx.x;
    const unsigned rb = (unsigned)(P.Rpad / PR), ks = (unsigned)((P.K + PK * P.kseg - 1) / (PK * P.kseg));
    if (P.kfast)
        e64_rowmax_block<true>(P, (long long)(blk / ks) * PR, (long long)(blk % ks) * PK * P.kseg);
    else
        e64_rowmax_block<false>(P, (long long)(blk % rb) * PR, (long long)(blk / rb) * PK * P.kseg);
}

long long roundup(long long x, long long m) { return (x + m - 1) / m * m; }

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
    static std::atomic<void *> fn{nullptr};
    void *p = fn.load();
    if (!p) {
        cudaDriverEntryPointQueryResult q;
        JUES_CHECK_CUDA(cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q));
        if (q != cudaDriverEntryPointSuccess || !p)
            throw Error(JUES_ECUDA, "cuTensorMapEncodeTiled is not available from the driver");
        fn.store(p);
    }
    return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
}

// [np][rows][kpad] elements, rows pitch bytes apart
CUtensorMap tensor_map(CUtensorMapDataType type, CUtensorMapSwizzle swizzle, long long pitch, const void *base,
                       long long kpad, long long rows, int np, int box_rows, int box_planes) {
    CUtensorMap m;
    std::memset(&m, 0, sizeof(m));
    cuuint64_t dims[3] = {(cuuint64_t)kpad, (cuuint64_t)rows, (cuuint64_t)np};
    cuuint64_t strides[2] = {(cuuint64_t)pitch, (cuuint64_t)(rows * pitch)};
    cuuint32_t box[3] = {(cuuint32_t)CK, (cuuint32_t)box_rows, (cuuint32_t)box_planes};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = encode_fn()(&m, type, 3, const_cast<void *>(base), dims, strides, box, estr,
                             CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) throw Error(JUES_ECUDA, "cuTensorMapEncodeTiled failed: " + std::to_string((int)r));
    return m;
}
// digit planes [np][rows][kpad]; one box = 64 K values (past kpad: zeros) x box_rows rows x box_planes
CUtensorMap plane_map(const __half *planes, long long rows, long long kpad, int np, int box_rows, int box_planes) {
    return tensor_map(CU_TENSOR_MAP_DATA_TYPE_FLOAT16, CU_TENSOR_MAP_SWIZZLE_128B, 2 * kpad, planes, kpad, rows, np, box_rows,
                      box_planes);
}
// the magnitudes behind them, [rows][mag_pitch] bytes
uint8_t *mag_at(const __half *planes, int np, long long rows, long long kpad) {
    return reinterpret_cast<uint8_t *>(const_cast<__half *>(planes) + (size_t)np * rows * kpad);
}
CUtensorMap mag_map(const __half *planes, long long rows, long long kpad, int np, int box_rows) {
    return tensor_map(CU_TENSOR_MAP_DATA_TYPE_UINT8, CU_TENSOR_MAP_SWIZZLE_64B, mag_pitch(kpad),
                      mag_at(planes, np, rows, kpad), kpad, rows, 1, box_rows, 1);
}

PackArgs pack_args(const double *src, const Mode &rm, const Mode &km, long long row0, long long R, long long K,
                   long long Rpad, long long Kpad, int *exps, __half *dst, uint8_t *mag) {
    PackArgs p;
    p.src = src; p.rm = rm; p.km = km;
    p.row0 = row0; p.R = R; p.K = K; p.Rpad = Rpad; p.Kpad = Kpad;
    p.exps = exps; p.dst = dst; p.mag = mag;
    p.blocks = (unsigned)((Rpad / pack_rows(Kpad)) * ((Kpad + pack_k(Kpad) - 1) / pack_k(Kpad)));
    p.kfast = km.s0 == 1 && km.d0 > 1;
    // about 16 blocks per SM in the row-maximum pass, at most 16 chunks a block
    const long long chunks = (K + PK - 1) / PK;
    p.kseg = (int)std::max<long long>(1, std::min<long long>(16, (Rpad / PR) * chunks / (152 * 16)));
    return p;
}

// digits of up to two operands (b may be null)
template <int PL>
void run_pack(Ctx *ctx, const PackArgs &a, const PackArgs *b) {
    PackArgs none{};
    const PackArgs &B = b ? *b : none;
    if (a.K <= PK) {
        Ctx::Scope s(ctx, "pack_e64");
        if (a.Kpad <= 64)
            e64_pack_kernel<PL, 64, true><<<a.blocks + B.blocks, 256, 0, ctx->stream>>>(a, B);
        else
            e64_pack_kernel<PL, 128, true><<<a.blocks + B.blocks, 256, 0, ctx->stream>>>(a, B);
        JUES_CHECK_CUDA(cudaGetLastError());
        return;
    }
    JUES_CHECK_CUDA(cudaMemsetAsync(a.exps, 0, (size_t)a.Rpad * sizeof(int), ctx->stream));
    if (b) JUES_CHECK_CUDA(cudaMemsetAsync(b->exps, 0, (size_t)b->Rpad * sizeof(int), ctx->stream));
    auto rblocks = [](const PackArgs &p) {
        return p.blocks ? (unsigned)((p.Rpad / PR) * ((p.K + PK * p.kseg - 1) / (PK * p.kseg))) : 0u;
    };
    {
        Ctx::Scope s(ctx, "pack_e64");
        e64_rowmax_kernel<<<rblocks(a) + rblocks(B), 256, 0, ctx->stream>>>(a, B);
        JUES_CHECK_CUDA(cudaGetLastError());
    }
    Ctx::Scope s(ctx, "pack_e64");
    e64_pack_kernel<PL, 128, false><<<a.blocks + B.blocks, 256, 0, ctx->stream>>>(a, B);
    JUES_CHECK_CUDA(cudaGetLastError());
}

// Whether the tensor cores take a contraction.  Measured through jues_gemm (packs, GEMM and the listed
// tiles' launch against the FP64 pipe, us): 640^3 51 against 763; 400^3 45 / 475; 200^3 (2^16 outputs or
// fewer; the FP64 side with a warp per output) 38 / 45; 150^3 35 / 25; 2304 x 48 x 48 (tiles on the
// FP64 pipe) 30 / 63; 4000 x 16 x 25 31 / 41.  The line lies where the sides meet.  A side of 8 or
// less has kernels of its own on the FP64 pipe; 9 to 15 pad the tile but gain all the same (13 x 50 x 8450
// 37 to 60 / 640; CCSD with 13 occupied of 63 orbitals, six sweeps: 22.2 -> 10.3 ms).  K <= 2^16 keeps the 64-bit
// sums far from overflow (|lo| < K 2^46).
bool wanted(long long M, long long N, long long K) {
    if (std::min(M, N) <= 8 || K < 8 || K > (1 << 16)) return false;
    const double flops = 2.0 * (double)M * (double)N * (double)K;
    return flops >= (M * N <= (1LL << 16) && K <= 8192 ? 1.6e7 : 3e6);
}

// the shared-memory limit is a per-device attribute of each kernel
template <int PL, bool GROUPED>
void allow_smem(Ctx *ctx) {
    static std::atomic<unsigned long long> set{0};
    const unsigned long long bit = ctx->device >= 0 && ctx->device < 64 ? 1ull << ctx->device : 0ull;
    if (bit && (set.load() & bit)) return;
    JUES_CHECK_CUDA(cudaFuncSetAttribute(gett_e64_kernel<PL, GROUPED>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         smem_bytes(PL)));
    set.fetch_or(bit);
}

void set_scaling(E64Args &g, double alpha, double beta, bool in_place) {
    g.alpha = alpha; g.beta = beta;
    int ak = 0;
    // operands within 2^+-400 and sums from 2^-70 on: with 2^+-100 more a result is still a normal number
    g.alpha_pow2 = std::frexp(std::fabs(alpha), &ak) == 0.5 && ak - 1 >= -100 && ak - 1 <= 100;
    g.alpha_k = g.alpha_pow2 ? ak - 1 : 0;
    g.alpha_neg = g.alpha_pow2 && alpha < 0;
    g.beta_mode = beta == 0.0 ? 0 : (beta == 1.0 ? (in_place ? 1 : 2) : 3);
}

// the allocations of one product: its planes are not reclaimed for one another
struct Busy {
    PackCache &c;
    Busy(PackCache &x, const PackEntry *a, const PackEntry *b) : c(x) {
        c.busy = c.e64_active = true;
        c.in_use[0] = a;
        c.in_use[1] = b;
    }
    ~Busy() {
        c.busy = c.e64_active = false;
        c.in_use[0] = c.in_use[1] = nullptr;
    }
};

PackEntry *find_entry(PackCache &pc, const double *src, const Mode &rm, const Mode &km, long long R, long long K,
                      long long Rpad, long long Kpad) {
    for (auto &e : pc.cached)
        if (e->np == NP && e->src == src && e->R == R && e->K == K && e->Rpad == Rpad && e->Kpad == Kpad &&
            same_mode(e->r, rm) && same_mode(e->k, km))
            return e.get();
    return nullptr;
}

// the output's unit-stride mode on the TMEM-lane side (coalesced stores) unless padding says otherwise
// (rows pad to 128, columns to 32)
GettArgs orient(const GettArgs &a0) {
    GettArgs a = a0;
    const bool m_unit = a.mC.s0 == 1 && a.mC.d0 > 1, n_unit = a.nC.s0 == 1 && a.nC.d0 > 1;
    auto cost = [](long long M, long long N, bool unit) {
        return (double)roundup(M, BM) * (double)roundup(N, BN) * (unit ? 1.0 : 1.2);
    };
    if (cost(a.N, a.M, n_unit) < cost(a.M, a.N, m_unit)) {
        std::swap(a.M, a.N);
        std::swap(a.A, a.B);
        std::swap(a.mA, a.nB);
        std::swap(a.kA, a.kB);
        std::swap(a.mC, a.nC);
        std::swap(a.a_const, a.b_const);
    }
    return a;
}

template <class T>
void grow(Ctx *ctx, DBuf<T> &b, size_t need) {
    if (b.n >= need) return;
    b.reset();
    b = DBuf<T>(ctx, need);
}

// a whole operand's digits are kept between calls when the caller declares it constant; a short-K
// one (an integral transform's) only while it is small, since reading the source again moves
// fewer bytes than its planes
bool keep_planes(bool is_const, long long K, size_t halves) {
    if (!is_const) return false;
    return K > 512 || halves * 2 <= (size_t(128) << 20);
}
// Transient planes go through panels of up to 1 GB, in halves down to 128 MB where memory is short.  Each
// panel costs two launches and a last round of tiles, which outweighs keeping its planes in L2 (packs and GEMM
// of 500000 x 16 x 100 with panels of 32, 64, 128, 256, 512 and 1024 MB: 880, 639, 560, 486, 461 and 439 us;
// 20000 x 40 x 2000: 1098, 708, 566, 471, 439 and 416 us).  The results do not depend on it.
constexpr size_t PANEL_MAX = size_t(512) << 20, PANEL_MIN = size_t(64) << 20;   // halves

}  // namespace

bool gett_e64(Ctx *ctx, const GettArgs &a0, const char *name) {
    if (!wanted(a0.M, a0.N, a0.K)) return false;
    GettArgs a = orient(a0);
    const long long Kpad = roundup(a.K, 16);   // rows of planes start on 32 bytes
    const long long Mall = roundup(a.M, BM), Nall = roundup(a.N, BM);
    if (Mall >= (1LL << 31) || Nall >= (1LL << 31) || Kpad >= (1LL << 30)) return false;
    const long long mtiles_all = Mall / BM, ntiles = roundup(a.N, BN) / BN;
    if (mtiles_all * ntiles >= (1LL << 30) || (Nall / PR) * ((Kpad + PK - 1) / PK) >= (1LL << 31)) return false;
    if (!ctx->pack) ctx->pack = new PackCache();
    PackCache &pc = *ctx->pack;
    const size_t hA = plane_halves(NP, Mall, Kpad), hB = plane_halves(NP, Nall, Kpad);
    bool keepA = keep_planes(a.a_const, a.K, hA), keepB = keep_planes(a.b_const, a.K, hB);
    PackEntry *eA = keepA ? find_entry(pc, a.A, a.mA, a.kA, a.M, a.K, Mall, Kpad) : nullptr;
    PackEntry *eB = keepB ? find_entry(pc, a.B, a.nB, a.kB, a.N, a.K, Nall, Kpad) : nullptr;
    std::unique_ptr<PackEntry> newA, newB;
    const int k16 = (int)((a.K + 15) / 16), chunks = (k16 + 3) / 4;
    long long prow = Mall;   // rows per panel of A
    int ksplit = 1, kper = chunks;
    longlong2 *part = nullptr;
    for (size_t panel = PANEL_MAX;; panel /= 2) {
        if (!keepA && hA > panel)
            prow = std::max<long long>(BM, (long long)(panel / plane_halves(NP, 2, Kpad) * 2) / BM * BM);
        if ((prow / PR) * ((Kpad + PK - 1) / PK) >= (1LL << 31)) return false;
        // K parts of a grid too small for the GPU (chunks of 64 K); exact whatever their number
        const long long panel_tiles = prow / BM * ntiles;
        // rounds of the 152 SMs times (chunks a part + about two for the tile's epilogue), plus the
        // parts' own pass (its time in chunks of 1.45 us)
        auto time = [&](int ks) {
            const long long rounds = (panel_tiles * ks + 151) / 152;
            return (double)rounds * ((chunks + ks - 1) / ks + 2) + (ks > 1 ? 4.0 + 0.02 * (double)(panel_tiles * ks) / 152 : 0.0);
        };
        ksplit = 1;
        for (int ks = 2; ks <= 64 && ks <= chunks; ++ks)
            if (panel_tiles * ks <= 152LL * 8 && time(ks) < 0.9 * time(ksplit)) ksplit = ks;
        kper = (chunks + ksplit - 1) / ksplit;
        ksplit = (chunks + kper - 1) / kper;
        try {
            Busy busy(pc, eA, eB);
            if (keepA && !eA && !newA)
                newA.reset(new PackEntry{a.A, a.mA, a.kA, a.M, a.K, Mall, Kpad, NP, take_buffer(ctx, pc.free_planes, hA),
                                         take_buffer(ctx, pc.free_exps, (size_t)Mall)});
            if (keepB && !eB && !newB)
                newB.reset(new PackEntry{a.B, a.nB, a.kB, a.N, a.K, Nall, Kpad, NP, take_buffer(ctx, pc.free_planes, hB),
                                         take_buffer(ctx, pc.free_exps, (size_t)Nall)});
            if (!keepA) {
                grow(ctx, pc.e64_planes[0], plane_halves(NP, prow, Kpad));
                grow(ctx, pc.e64_exps[0], (size_t)prow);
            }
            if (!keepB) {
                grow(ctx, pc.e64_planes[1], hB);
                grow(ctx, pc.e64_exps[1], (size_t)Nall);
            }
            grow(ctx, pc.e64_list, e64_list_ints(mtiles_all * ntiles));
            if (ksplit > 1)   // the parts' sums, then their magnitudes
                part = static_cast<longlong2 *>(ctx->splitk_scratch((size_t)ksplit * panel_tiles * BM * BN *
                                                                    (sizeof(longlong2) + sizeof(float))));
            break;
        } catch (const Error &e) {
            if (e.code != JUES_ENOMEM) throw;
            if ((keepA && !eA) || (keepB && !eB)) {   // no room to keep new planes: transient ones, in panels
                newA.reset();
                newB.reset();
                keepA = eA != nullptr;
                keepB = eB != nullptr;
                panel = 2 * PANEL_MAX;
                continue;
            }
            if (keepA || hA <= PANEL_MIN || panel <= PANEL_MIN) return false;   // the FP64 pipe needs no planes
        }
    }
    allow_smem<NP, false>(ctx);
    // C = Cin + alpha AB into a dense column-major C: copy Cin over and add in place, off the FP64 pipe
    const double *Cin = a.Cin ? a.Cin : a.C;
    const bool disjoint = Cin + a.M * a.N <= a.C || a.C + a.M * a.N <= Cin;
    if (a.beta == 1.0 && Cin != a.C && disjoint && a.mC.d0 == MODE_BIG && a.mC.s0 == 1 && a.nC.d0 == MODE_BIG &&
        a.nC.s0 == a.M) {
        JUES_CHECK_CUDA(cudaMemcpyAsync(a.C, Cin, (size_t)(a.M * a.N) * sizeof(double), cudaMemcpyDeviceToDevice,
                                        ctx->stream));
        Cin = a.C;
    }
    a.Cin = Cin;

    __half *planesB = eB ? eB->buf.p : newB ? newB->buf.p : pc.e64_planes[1].p;
    int *expsB = eB ? eB->exps.p : newB ? newB->exps.p : pc.e64_exps[1].p;
    JUES_CHECK_CUDA(cudaMemsetAsync(pc.e64_list.p, 0, 2 * sizeof(int), ctx->stream));
    for (long long r0 = 0; r0 < a.M; r0 += prow) {
        const long long R = std::min(prow, a.M - r0), Rpad = roundup(R, BM);
        __half *planesA = eA ? eA->buf.p : newA ? newA->buf.p : pc.e64_planes[0].p;
        int *expsA = eA ? eA->exps.p : newA ? newA->exps.p : pc.e64_exps[0].p;
        const bool packB = r0 == 0 && !eB;
        const PackArgs pb = pack_args(a.B, a.nB, a.kB, 0, a.N, a.K, Nall, Kpad, expsB, planesB,
                                      mag_at(planesB, NP, Nall, Kpad));
        if (!eA)
            run_pack<NP>(ctx, pack_args(a.A, a.mA, a.kA, r0, R, a.K, Rpad, Kpad, expsA, planesA, mag_at(planesA, NP, Rpad, Kpad)),
                         packB ? &pb : nullptr);
        else if (packB)
            run_pack<NP>(ctx, pb, nullptr);
        E64Args g;
        g.rowA = g.rowB = g.item0 = 0;
        g.M = R; g.N = a.N; g.row0 = r0;
        g.k16 = k16;
        g.mtiles = (int)(Rpad / BM); g.ntiles = (int)ntiles;
        g.mtiles_all = mtiles_all;
        g.expA = expsA; g.expB = expsB;
        set_scaling(g, a.alpha, a.beta, Cin == a.C);
        g.C = a.C; g.Cin = Cin; g.mC = a.mC; g.nC = a.nC;
        g.flags = ctx->d_flags;
        g.ksplit = ksplit; g.kper = kper;
        g.part = part;
        g.pmag = reinterpret_cast<float *>(part + (size_t)ksplit * g.mtiles * g.ntiles * BM * BN);
        g.list = pc.e64_list.p;
        g.fine = g.list + 2 + 4 * mtiles_all * ntiles;
        const CUtensorMap ma = plane_map(planesA, Rpad, Kpad, NP, BM, 1), mb = plane_map(planesB, Nall, Kpad, NP, BN, NP),
                          xa = mag_map(planesA, Rpad, Kpad, NP, BM), xb = mag_map(planesB, Nall, Kpad, NP, BN);
        const long long items = e64_items(g);
        {
            Ctx::Scope s(ctx, name);
            gett_e64_kernel<NP, false><<<(unsigned)std::min<long long>(items, 152), THREADS, smem_bytes(NP),
                                         ctx->stream>>>(ma, mb, xa, xb, g, nullptr, 0, (int)items);
            JUES_CHECK_CUDA(cudaGetLastError());
        }
        if (ksplit > 1) {
            const std::string nm = std::string(name) + ".reduce";
            Ctx::Scope s(ctx, nm.c_str());
            const long long n = (long long)g.mtiles * g.ntiles * BM * BN;
            int step = 1;
            if (ksplit > PART_FOLD) {
                step = PART_FOLD;
                e64_fold_kernel<<<dim3((unsigned)(n / 256), (unsigned)((ksplit + step - 1) / step)), 256, 0,
                                  ctx->stream>>>(part, g.pmag, ksplit, n);
                ctx->count_launch();
                JUES_CHECK_CUDA(cudaGetLastError());
            }
            e64_parts_kernel<<<(unsigned)(g.mtiles * g.ntiles), DRAIN, 0, ctx->stream>>>(g, step);
            JUES_CHECK_CUDA(cudaGetLastError());
        }
    }
    if (newA) pc.cached.push_back(std::move(newA));
    if (newB) pc.cached.push_back(std::move(newB));
    gett_f64_tiles(ctx, &a, nullptr, pc.e64_list.p, mtiles_all * ntiles, name);
    return true;
}

// ---------------------------------------------------------------------------------------------
// Grouped form: many contractions over row ranges of two sets of shared planes, one launch
// ---------------------------------------------------------------------------------------------
void e64_alloc(Ctx *ctx, E64Planes &P, long long rows, long long K, int np) {
    JUES_REQUIRE(np == 3 || np == E64_NP, "digit planes must be 3 or 7");
    JUES_REQUIRE(K >= 1 && K <= (1 << 16), "K out of range for the digit planes");
    P.np = np;
    P.rows = roundup(rows, BM);
    P.K = K;
    P.Kpad = roundup(K, 16);
    JUES_REQUIRE(P.rows < (1LL << 31) && (P.rows / PR) * ((P.Kpad + PK - 1) / PK) < (1LL << 31), "too many operand rows");
    P.planes = DBuf<__half>(ctx, plane_halves(np, P.rows, P.Kpad));
    P.exps = DBuf<int>(ctx, (size_t)P.rows);
}

void e64_pack(Ctx *ctx, E64Planes &P, const double *src, const Mode &rm, const Mode &km, long long R) {
    JUES_REQUIRE(R <= P.rows, "operand does not fit its planes");
    const PackArgs a = pack_args(src, rm, km, 0, R, P.K, P.rows, P.Kpad, P.exps.p, P.planes.p,
                                 mag_at(P.planes.p, P.np, P.rows, P.Kpad));
    if (P.np == 3)
        run_pack<3>(ctx, a, nullptr);
    else
        run_pack<NP>(ctx, a, nullptr);
}

E64Args e64_problem(Ctx *ctx, const E64Planes &A, const E64Planes &B, long long K, long long rowA, long long M,
                    long long rowB, long long N, double alpha, double beta, double *C, const Mode &mC, const Mode &nC, int item0,
                    int *list, long long list_tiles) {
    E64Args g{};
    g.M = M; g.N = N; g.row0 = 0;
    g.rowA = (int)rowA; g.rowB = (int)rowB; g.item0 = item0;
    g.k16 = (int)((K + 15) / 16);
    g.mtiles = (int)(roundup(M, BM) / BM); g.ntiles = (int)(roundup(N, BN) / BN);
    g.mtiles_all = g.mtiles;
    g.expA = A.exps.p + rowA; g.expB = B.exps.p + rowB;
    set_scaling(g, alpha, beta, true);
    g.C = C; g.Cin = C; g.mC = mC; g.nC = nC;
    g.flags = ctx->d_flags;
    g.ksplit = 1; g.kper = (g.k16 + 3) / 4;
    g.part = nullptr;
    g.pmag = nullptr;
    g.list = list;
    g.fine = list ? list + 2 + 4 * list_tiles : nullptr;
    return g;
}

void e64_group_run(Ctx *ctx, const E64Planes &A, const E64Planes &B, const E64Args *probs, const GroupProblem *f64,
                   int n, long long items, int *list, long long list_tiles, const char *name) {
    if (n <= 0 || items <= 0) return;
    JUES_REQUIRE(A.np == B.np && A.Kpad == B.Kpad && items < (1LL << 31), "mismatched planes");
    const CUtensorMap ma = plane_map(A.planes.p, A.rows, A.Kpad, A.np, BM, 1),
                      mb = plane_map(B.planes.p, B.rows, B.Kpad, B.np, BN, B.np),
                      xa = mag_map(A.planes.p, A.rows, A.Kpad, A.np, BM),
                      xb = mag_map(B.planes.p, B.rows, B.Kpad, B.np, BN);
    JUES_CHECK_CUDA(cudaMemsetAsync(list, 0, 2 * sizeof(int), ctx->stream));
    E64Args g{};
    g.flags = ctx->d_flags;
    const unsigned grid = (unsigned)std::min<long long>(items, 152);
    {
        Ctx::Scope s(ctx, name);
        if (A.np == 3) {
            allow_smem<3, true>(ctx);
            gett_e64_kernel<3, true><<<grid, THREADS, smem_bytes(3), ctx->stream>>>(ma, mb, xa, xb, g, probs, n, (int)items);
        } else {
            allow_smem<NP, true>(ctx);
            gett_e64_kernel<NP, true><<<grid, THREADS, smem_bytes(NP), ctx->stream>>>(ma, mb, xa, xb, g, probs, n, (int)items);
        }
        JUES_CHECK_CUDA(cudaGetLastError());
    }
    gett_f64_tiles(ctx, nullptr, f64, list, list_tiles, name);
}

// ---------------------------------------------------------------------------------------------
// One stage of a batch: many contractions with K <= 128, their operands' rows side by side in two sets of
// planes; one pack launch, one GEMM launch and the listed tiles' launch, which a CUDA graph can capture
// ---------------------------------------------------------------------------------------------
struct E64Group {
    std::string name;
    E64Planes A, B;             // views of the shared planes
    DBuf<E64Args> args;
    DBuf<GroupProblem> f64;
    DBuf<PackArgs> ops;
    DBuf<unsigned> first;
    int *list = nullptr;
    long long list_tiles = 0;
    int nprob = 0, nops = 0;
    unsigned blocks = 0;
    long long items = 0;
};

namespace {

// the stage's contractions as the kernels take them, and the planes that they need
struct StageShape {
    std::vector<GettArgs> ps;
    long long kmax = 0, kpad = 0, pr = 0, rows[2] = {0, 0}, items = 0;
    size_t halves(int side) const { return plane_halves(NP, rows[side], kpad); }
    size_t bytes() const {
        return (halves(0) + halves(1)) * sizeof(__half) +
               ((size_t)(rows[0] + rows[1]) + e64_list_ints(items)) * sizeof(int);
    }
};

// A stage below 1e8 flop in all costs its four launches more than the FP64 tiles take (24 systems of nbf 10 to
// 60: the eleven K <= 64 stages took 22 ms on the FP64 tiles and take 3 ms here).
bool stage_shape(const std::vector<GettArgs> &in, StageShape &s) {
    double flops = 0.0;
    for (const GettArgs &a : in) {
        if (a.M <= 0 || a.N <= 0) continue;
        if (a.K < 1 || a.K > PK || (a.beta != 0.0 && a.beta != 1.0) || (a.beta == 1.0 && a.Cin && a.Cin != a.C))
            return false;
        flops += 2.0 * (double)a.M * (double)a.N * (double)a.K;
        s.kmax = std::max(s.kmax, a.K);
        s.ps.push_back(orient(a));
        s.items += e64_tiles(s.ps.back().M, s.ps.back().N);
    }
    if (flops < 1e8) return false;
    s.kpad = roundup(s.kmax, 16);
    s.pr = pack_rows(s.kpad);
    for (const GettArgs &a : s.ps) {
        s.rows[0] += roundup(a.M, s.pr);
        s.rows[1] += roundup(a.N, s.pr);
    }
    for (long long &r : s.rows) r = roundup(r, BM);
    return s.rows[0] < (1LL << 30) && s.rows[1] < (1LL << 30) && s.items < (1LL << 28);
}

template <class T>
DBuf<T> view_of(const DBuf<T> &b) {
    DBuf<T> v;   // no context: never freed through it
    v.p = b.p;
    v.n = b.n;
    return v;
}

}  // namespace

void e64_shared_reserve(Ctx *ctx, E64Shared &sh, const std::vector<const std::vector<GettArgs> *> &stages) {
    std::vector<StageShape> fit;
    for (const std::vector<GettArgs> *st : stages) {
        StageShape s;
        if (stage_shape(*st, s)) fit.push_back(std::move(s));
    }
    std::sort(fit.begin(), fit.end(), [](const StageShape &a, const StageShape &b) { return a.bytes() < b.bytes(); });
    for (; !fit.empty(); fit.pop_back()) {   // without its largest stage where that does not fit
        size_t halves[2] = {0, 0}, rows[2] = {0, 0};
        long long items = 0;
        for (const StageShape &s : fit) {
            for (int k = 0; k < 2; ++k) {
                halves[k] = std::max(halves[k], s.halves(k));
                rows[k] = std::max(rows[k], (size_t)s.rows[k]);
            }
            items = std::max(items, s.items);
        }
        try {
            for (int k = 0; k < 2; ++k) {
                grow(ctx, sh.planes[k], halves[k]);
                grow(ctx, sh.exps[k], rows[k]);
            }
            grow(ctx, sh.list, e64_list_ints(items));
            sh.list_tiles = items;
            return;
        } catch (const Error &e) {
            if (e.code != JUES_ENOMEM) throw;   // the FP64 tiles need no planes
            sh = E64Shared();
        }
    }
}

E64Group *e64_group_build(Ctx *ctx, const std::vector<GettArgs> &in, const E64Shared &sh, const char *name) {
    StageShape s;
    if (!stage_shape(in, s)) return nullptr;
    for (int k = 0; k < 2; ++k)
        if (sh.planes[k].n < s.halves(k) || sh.exps[k].n < (size_t)s.rows[k]) return nullptr;
    if (sh.list_tiles < s.items) return nullptr;
    try {
        std::unique_ptr<E64Group> g(new E64Group());
        g->name = name;
        g->items = s.items;
        g->list = sh.list.p;
        g->list_tiles = sh.list_tiles;
        const long long pr = s.pr;
        for (int k = 0; k < 2; ++k) {
            E64Planes &P = k ? g->B : g->A;
            P.np = NP;
            P.rows = s.rows[k];
            P.K = s.kmax;
            P.Kpad = s.kpad;
            P.planes = view_of(sh.planes[k]);
            P.exps = view_of(sh.exps[k]);
        }
        std::vector<E64Args> args;
        std::vector<GroupProblem> f64;
        std::vector<PackArgs> ops;
        std::vector<unsigned> first;
        long long ra = 0, rb = 0, at = 0;
        auto pack = [&](const E64Planes &P, long long row, const double *src, const Mode &rm, const Mode &km, long long R,
                        long long K) {
            PackArgs p = pack_args(src, rm, km, 0, R, K, P.rows, P.Kpad, P.exps.p + row, P.planes.p + row * P.Kpad,
                                   mag_at(P.planes.p, P.np, P.rows, P.Kpad) + row * mag_pitch(P.Kpad));
            first.push_back(g->blocks);
            g->blocks += (unsigned)(roundup(R, pr) / pr);
            ops.push_back(p);
        };
        for (const GettArgs &a : s.ps) {
            pack(g->A, ra, a.A, a.mA, a.kA, a.M, a.K);
            pack(g->B, rb, a.B, a.nB, a.kB, a.N, a.K);
            args.push_back(e64_problem(ctx, g->A, g->B, a.K, ra, a.M, rb, a.N, a.alpha, a.beta, a.C, a.mC, a.nC, (int)at,
                                       g->list, g->list_tiles));
            f64.push_back(to_problem(a));
            ra += roundup(a.M, pr);
            rb += roundup(a.N, pr);
            at += e64_tiles(a.M, a.N);
        }
        g->nprob = (int)args.size();
        g->nops = (int)ops.size();
        g->args = DBuf<E64Args>(ctx, args.size());
        g->f64 = DBuf<GroupProblem>(ctx, f64.size());
        g->ops = DBuf<PackArgs>(ctx, ops.size());
        g->first = DBuf<unsigned>(ctx, first.size());
        auto up = [&](void *d, const void *h, size_t bytes) {
            JUES_CHECK_CUDA(cudaMemcpyAsync(d, h, bytes, cudaMemcpyHostToDevice, ctx->stream));
        };
        up(g->args.p, args.data(), args.size() * sizeof(E64Args));
        up(g->f64.p, f64.data(), f64.size() * sizeof(GroupProblem));
        up(g->ops.p, ops.data(), ops.size() * sizeof(PackArgs));
        up(g->first.p, first.data(), first.size() * sizeof(unsigned));
        ctx->sync();   // the host tables stay valid until then
        return g.release();
    } catch (const Error &e) {
        if (e.code != JUES_ENOMEM) throw;
        return nullptr;   // the FP64 tiles need no planes
    }
}

void e64_group_exec(Ctx *ctx, E64Group *g) {
    {
        Ctx::Scope s(ctx, "pack_e64");
        if (g->A.Kpad <= 64)
            e64_pack_grouped_kernel<NP, 64><<<g->blocks, 256, 0, ctx->stream>>>(g->ops.p, g->first.p, g->nops);
        else
            e64_pack_grouped_kernel<NP, 128><<<g->blocks, 256, 0, ctx->stream>>>(g->ops.p, g->first.p, g->nops);
        JUES_CHECK_CUDA(cudaGetLastError());
    }
    e64_group_run(ctx, g->A, g->B, g->args.p, g->f64.p, g->nprob, g->items, g->list, g->list_tiles, g->name.c_str());
}

void e64_group_destroy(E64Group *g) { delete g; }

}  // namespace jues
