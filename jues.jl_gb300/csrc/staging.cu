// Host<->device copies of many caller arrays through a page-locked staging ring.
//
// A copy from pageable memory is staged by the driver through its own bounce buffers with one
// host thread (a few GB/s on GB300's Grace host), and page-locking the caller's arrays instead
// costs about a millisecond per registration call, which dominates for hundreds of small
// arrays.  Here host threads move the data between the caller's arrays and 64 MB page-locked
// slots while the link drains or fills the neighbouring slot.
#include <algorithm>
#include <condition_variable>
#include <cstring>
#include <functional>
#include <mutex>
#include <system_error>
#include <thread>

#include "staging.cuh"

namespace jues {

namespace {

// A fixed set of worker threads running one parallel loop at a time; the caller takes tasks too.
class WorkerPool {
  public:
    explicit WorkerPool(int workers) {
        try {
            for (int i = 0; i < workers; ++i) threads_.emplace_back([this] { run(); });
        } catch (const std::system_error &) {
            // fewer threads, or the caller alone, do the same work
        }
    }
    ~WorkerPool() {
        {
            std::lock_guard<std::mutex> l(m_);
            stop_ = true;
        }
        cv_.notify_all();
        for (auto &t : threads_) t.join();
    }
    // fn(k) for every k in [0, n); returns when all have finished
    void parallel_for(int n, const std::function<void(int)> &fn) {
        if (n <= 0) return;
        {
            std::lock_guard<std::mutex> l(m_);
            fn_ = &fn;
            n_ = n;
            next_ = 0;
            done_ = 0;
            ++gen_;
        }
        cv_.notify_all();
        work();
        std::unique_lock<std::mutex> l(m_);
        done_cv_.wait(l, [&] { return done_ == n_; });
        fn_ = nullptr;
    }

  private:
    void work() {
        for (;;) {
            int k;
            const std::function<void(int)> *fn;
            {
                std::lock_guard<std::mutex> l(m_);
                if (!fn_ || next_ >= n_) return;
                k = next_++;
                fn = fn_;
            }
            (*fn)(k);
            std::lock_guard<std::mutex> l(m_);
            if (++done_ == n_) done_cv_.notify_all();
        }
    }
    void run() {
        unsigned long long seen = 0;
        for (;;) {
            {
                std::unique_lock<std::mutex> l(m_);
                cv_.wait(l, [&] { return stop_ || gen_ != seen; });
                if (stop_) return;
                seen = gen_;
            }
            work();
        }
    }
    std::vector<std::thread> threads_;
    std::mutex m_;
    std::condition_variable cv_, done_cv_;
    const std::function<void(int)> *fn_ = nullptr;
    int n_ = 0, next_ = 0, done_ = 0;
    unsigned long long gen_ = 0;
    bool stop_ = false;
};

constexpr size_t kSlot = size_t(64) << 20;
constexpr int kSlots = 3;
// Page-locking a slot takes about 15 ms, and results alone need two buffers in turn: until an upload has made the
// slots, results go through a pair of 16 MB (RCCD nbf=200 from device integrals, 328 MB of amplitudes, a context's
// first call: 190 ms through the slots, 173 here).  Results of 512 MB and more keep the
// slots: the MP2 gradient at nbf=120, 1.66 GB, takes 46.8 ms a call with them and 48.7 with the pair.
constexpr size_t kSmall = size_t(16) << 20;
constexpr int kSmalls = 2;
constexpr size_t kLarge = size_t(512) << 20;
constexpr size_t kTask = size_t(1) << 20;   // host copy granule

// one slot's worth of ranges: stage[i] in the slot <-> host[i] / dev[i]
struct Fill {
    struct Piece {
        size_t at;   // offset in the slot
        const char *src;
        char *dst;
        size_t bytes;
    };
    std::vector<Piece> pcs;
    size_t used = 0;
};

// cut the ranges into fills of at most cap bytes, in order
std::vector<Fill> plan_fills(const std::vector<HostSeg> &segs, size_t cap) {
    std::vector<Fill> fills(1);
    for (const HostSeg &s : segs) {
        size_t off = 0;
        while (off < s.bytes) {
            if (fills.back().used == cap) fills.emplace_back();
            Fill &f = fills.back();
            const size_t take = std::min(s.bytes - off, cap - f.used);
            f.pcs.push_back({f.used, static_cast<const char *>(s.src) + off, static_cast<char *>(s.dst) + off, take});
            f.used += take;
            off += take;
        }
    }
    if (fills.back().used == 0) fills.pop_back();
    return fills;
}

}  // namespace

struct Staging {
    char *host[kSlots] = {};     // kSlot bytes each, page-locked when first used
    char *small[kSmalls] = {};   // kSmall bytes each, likewise
    cudaEvent_t done[kSlots] = {};
    bool busy[kSlots] = {};
    WorkerPool *pool = nullptr;
};

static Staging *staging_of(Ctx *ctx) {
    if (ctx->staging) return ctx->staging;
    Staging *st = new Staging;
    ctx->staging = st;   // released by staging_destroy, also when a step below fails
    for (int k = 0; k < kSlots; ++k) JUES_CHECK_CUDA(cudaEventCreateWithFlags(&st->done[k], cudaEventDisableTiming));
    const unsigned hw = std::thread::hardware_concurrency();
    st->pool = new WorkerPool((int)std::min(15u, hw > 1 ? hw - 1 : 0u));
    return st;
}

// a slot's memory, null where page-locked memory is refused
static char *locked(char *&p, size_t bytes) {
    if (!p && cudaHostAlloc(reinterpret_cast<void **>(&p), bytes, cudaHostAllocDefault) != cudaSuccess) {
        cudaGetLastError();
        p = nullptr;
    }
    return p;
}
static char *slot_of(Staging *st, int k) {
    char *p = locked(st->host[k], kSlot);
    if (!p) throw Error(JUES_ECUDA, "page-locked memory for the upload ring was refused");
    return p;
}

// host side of one fill: copy the pieces' bytes between the slot and the caller's arrays in tasks of
// 1 MB (256 KB in a fill of 16 MB or less) over the workers (to_slot: caller -> slot)
static void host_copy(Staging *st, const Fill &f, char *slot, bool to_slot) {
    const size_t task = f.used > kSmall ? kTask : kTask / 4;
    const int ntask = (int)((f.used + task - 1) / task);
    st->pool->parallel_for(ntask, [&](int k) {
        const size_t lo = (size_t)k * task, hi = std::min(f.used, lo + task);
        // pieces are in slot order: start at the last one beginning at or before lo
        auto it = std::upper_bound(f.pcs.begin(), f.pcs.end(), lo,
                                   [](size_t x, const Fill::Piece &p) { return x < p.at; });
        for (--it; it != f.pcs.end() && it->at < hi; ++it) {
            const size_t a = std::max(lo, it->at), b = std::min(hi, it->at + it->bytes);
            if (a >= b) continue;
            if (to_slot)
                std::memcpy(slot + a, it->src + (a - it->at), b - a);
            else
                std::memcpy(it->dst + (a - it->at), slot + a, b - a);
        }
    });
}

void staged_h2d(Ctx *ctx, const std::vector<HostSeg> &segs) {
    const std::vector<Fill> fills = plan_fills(segs, kSlot);
    if (fills.empty()) return;
    Staging *st = staging_of(ctx);
    for (size_t i = 0; i < fills.size(); ++i) {
        const int k = (int)(i % kSlots);
        if (st->busy[k]) JUES_CHECK_CUDA(cudaEventSynchronize(st->done[k]));   // its last copy has left
        char *slot = slot_of(st, k);
        host_copy(st, fills[i], slot, true);
        for (const Fill::Piece &p : fills[i].pcs)
            JUES_CHECK_CUDA(cudaMemcpyAsync(p.dst, slot + p.at, p.bytes, cudaMemcpyHostToDevice, ctx->stream));
        JUES_CHECK_CUDA(cudaEventRecord(st->done[k], ctx->stream));
        st->busy[k] = true;
    }
}

void staged_d2h(Ctx *ctx, const std::vector<HostSeg> &segs) {
    Staging *st = staging_of(ctx);
    size_t bytes = 0;
    for (const HostSeg &s : segs) bytes += s.bytes;
    const bool small = !st->host[0] && bytes < kLarge;   // slot 0 is the first that an upload takes
    const std::vector<Fill> fills = plan_fills(segs, small ? kSmall : kSlot);
    if (fills.empty()) return;
    auto slot_at = [&](int k) { return small ? locked(st->small[k], kSmall) : locked(st->host[k], kSlot); };
    // two buffers in turn are enough; without them the driver copies into the caller's arrays
    const int most = (int)std::min<size_t>(small ? kSmalls : kSlots, fills.size());
    int slots = 0;
    while (slots < most && slot_at(slots)) ++slots;
    if (slots < std::min(most, 2)) {
        for (const HostSeg &s : segs)
            JUES_CHECK_CUDA(cudaMemcpyAsync(s.dst, s.src, s.bytes, cudaMemcpyDeviceToHost, ctx->stream));
        ctx->sync();
        return;
    }
    // the link fills slot i + 1 while the host empties slot i
    auto issue = [&](size_t i) {
        const int k = (int)(i % slots);
        if (st->busy[k]) JUES_CHECK_CUDA(cudaEventSynchronize(st->done[k]));
        char *slot = slot_at(k);
        for (const Fill::Piece &p : fills[i].pcs)
            JUES_CHECK_CUDA(cudaMemcpyAsync(slot + p.at, p.src, p.bytes, cudaMemcpyDeviceToHost, ctx->stream));
        JUES_CHECK_CUDA(cudaEventRecord(st->done[k], ctx->stream));
        st->busy[k] = true;
    };
    issue(0);
    for (size_t i = 0; i < fills.size(); ++i) {
        if (i + 1 < fills.size()) issue(i + 1);
        const int k = (int)(i % slots);
        JUES_CHECK_CUDA(cudaEventSynchronize(st->done[k]));
        host_copy(st, fills[i], slot_at(k), false);
    }
}

// Device -> host into a caller's array, complete at return.  A copy into pageable memory of 16 MB and more
// goes through the ring: the driver's own staging writes it with one host thread, page faults included
// (the MP2 gradient at nbf=120, 1.66 GB into fresh arrays: 82 ms a call, 50 ms through the ring).  Smaller
// copies and page-locked arrays are copied directly.
void copy_out(Ctx *ctx, double *h, const double *d, size_t n) {
    const size_t bytes = n * sizeof(double);
    bool staged = bytes >= (size_t(16) << 20);
    if (staged) {
        cudaPointerAttributes at;
        if (cudaPointerGetAttributes(&at, h) != cudaSuccess) {
            cudaGetLastError();
            at.type = cudaMemoryTypeUnregistered;
        }
        staged = at.type == cudaMemoryTypeUnregistered;
    }
    if (staged)
        staged_d2h(ctx, {HostSeg{h, d, bytes}});
    else if (n)
        JUES_CHECK_CUDA(cudaMemcpyAsync(h, d, bytes, cudaMemcpyDeviceToHost, ctx->stream));
    ctx->sync();
}

void staging_destroy(Staging *st) {
    if (!st) return;
    for (int k = 0; k < kSlots; ++k)
        if (st->done[k]) {
            cudaEventSynchronize(st->done[k]);
            cudaEventDestroy(st->done[k]);
        }
    for (char *h : st->host)
        if (h) cudaFreeHost(h);
    for (char *h : st->small)
        if (h) cudaFreeHost(h);
    delete st->pool;
    delete st;
}

}  // namespace jues
