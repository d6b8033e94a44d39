// Host model of the key-row streams of csrc/key_stream.cuh: the barriers are
// simulated, one chosen row's copy never lands, and the streams are driven as
// the kernels drive them, one host thread per group (or half, or warp) of
// consumers.  A bounded wait runs out when every thread waits.  Faults that a
// GPU would not forgive are counted: a barrier armed or arrived at beyond its
// count, a copy into a slot whose last copy is still out, a stream that ends
// with a copy out and not waited for.
#include <condition_variable>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <functional>
#include <map>
#include <mutex>
#include <set>
#include <string>
#include <thread>
#include <vector>

#define __device__
#define __forceinline__ inline

namespace tfhe_gb300 {

template <typename R>
struct cpx {
    R x, y;
};

struct Bar {
    int count = 1, pending = 1, phase = 0;
    long tx = 0;
    void settle() {
        if (pending == 0 && tx == 0) {
            pending = count;
            ++phase;
        }
    }
};

static std::mutex g_lock;
static std::condition_variable g_change;
static int g_threads, g_bounded;  // running; of them in a wait that can run out
static std::set<const std::function<bool()>*> g_waiting;  // what the waiting ones wait for
static bool g_run_out;                       // one bounded wait may give up
static std::map<const uint64_t*, Bar> g_bars;
static std::map<const void*, const uint64_t*> g_out;  // slot -> barrier of a copy that has not landed
static std::set<const uint64_t*> g_drained;           // barriers waited for without the abort flag
static std::set<std::string> g_faults;
static const char* g_base;
static long g_lost = -1, g_copies = 0;
static size_t g_row_bytes;
static std::vector<long> g_rows;  // copied, in order
static void fault(const char* what) { g_faults.insert(what); }
static bool passed(const uint64_t* bar, uint32_t parity) { return ((uint32_t)g_bars[bar].phase & 1) != parity; }

// Every thread waits for something that no thread will do: one bounded wait runs out.
static void all_waiting() {
    if (g_waiting.size() != (size_t)g_threads) return;
    for (const auto* done : g_waiting)
        if ((*done)()) return;
    if (g_bounded > 0) {
        g_run_out = true;
        g_change.notify_all();
    }
}
// Wait for done(); false when the wait ran out.
static bool wait_until(std::unique_lock<std::mutex>& lk, bool bounded, const std::function<bool()>& done) {
    if (done()) return true;
    g_waiting.insert(&done);
    g_bounded += bounded;
    bool ok;
    while (!(ok = done())) {
        all_waiting();
        if (bounded && g_run_out) {
            g_run_out = false;
            break;
        }
        g_change.wait(lk);
    }
    g_waiting.erase(&done);
    g_bounded -= bounded;
    return ok;
}

static void arrive(uint64_t* bar, long bytes) {
    std::unique_lock<std::mutex> lk(g_lock);
    Bar& b = g_bars[bar];
    if (b.pending == 0) fault("barrier armed or arrived at beyond its count");
    else --b.pending;
    b.tx += bytes;
    b.settle();
    g_change.notify_all();
}
inline void mbar_arrive(uint64_t* bar) { arrive(bar, 0); }
inline void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) { arrive(bar, bytes); }
inline void bulk_copy_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    std::unique_lock<std::mutex> lk(g_lock);
    if (g_out.count(dst)) fault("copy into a slot whose last copy has not landed");
    const long row = (static_cast<const char*>(src) - g_base) / (long)g_row_bytes;
    ++g_copies;
    g_rows.push_back(row);
    if (row == g_lost) {
        g_out[dst] = bar;
        g_drained.erase(bar);
        return;
    }
    Bar& b = g_bars[bar];
    b.tx -= bytes;
    b.settle();
    g_change.notify_all();
}
inline bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    std::unique_lock<std::mutex> lk(g_lock);
    return passed(bar, parity);
}
inline bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, const volatile int* abort) {
    std::unique_lock<std::mutex> lk(g_lock);
    return wait_until(lk, true, [&] { return passed(bar, parity) || *abort; }) && passed(bar, parity);
}
inline bool mbar_wait_bounded(uint64_t* bar, uint32_t parity) {
    std::unique_lock<std::mutex> lk(g_lock);
    g_drained.insert(bar);
    return wait_until(lk, true, [&] { return passed(bar, parity); });
}
inline int atomicExch(int32_t* p, int32_t v) {
    std::unique_lock<std::mutex> lk(g_lock);
    const int old = *p;
    *p = v;
    g_change.notify_all();
    return old;
}
inline void group_sync(int) {}
inline void __syncwarp() {}
struct Dim {
    unsigned x;
};
static thread_local Dim threadIdx{0};

}  // namespace tfhe_gb300

#include "key_stream.cuh"

using namespace tfhe_gb300;

static void reset(long lost, size_t row_bytes, const char* base) {
    g_bars.clear();
    g_out.clear();
    g_drained.clear();
    g_copies = 0;
    g_rows.clear();
    g_lost = lost;
    g_row_bytes = row_bytes;
    g_base = base;
    g_threads = 1;
}
static void finish(long lost, long rows, int32_t err) {
    for (const auto& o : g_out)
        if (!g_drained.count(o.second)) fault("a copy is out and nobody waits for it");
    if ((err != 0) != (lost >= 0)) fault("status word");
    if (lost < 0 && g_copies != rows) fault("rows streamed");
}
static void run(const std::vector<std::function<void()>>& bodies) {
    g_threads = (int)bodies.size();
    std::vector<std::thread> ts;
    for (const auto& body : bodies)
        ts.emplace_back([&body] {
            body();
            std::unique_lock<std::mutex> lk(g_lock);
            --g_threads;
            all_waiting();
        });
    for (auto& t : ts) t.join();
}

// A group of two threads over `items` items, blocks of two rows and one as the
// product kernel takes them; items with rotation 0 use no rows.
template <int L, bool ROT>
static void products(std::vector<int32_t> rot, long lost) {
    using Keys = ItemKeys<L, ROT>;
    static uint64_t full[Keys::S];
    static cpx<float> ring[Keys::S * Keys::kRow];
    static char key[64];
    const char* src = key;
    reset(lost, Keys::kRowBytes, src);
    int32_t err = 0;
    volatile int abort = 0;
    const int items = (int)rot.size();
    std::vector<Keys> k;
    for (int t = 0; t < 2; ++t)
        k.push_back(Keys{ring, full, &err, &abort, src, 2 * L * Keys::kRowBytes, rot.data(), 1, items, t, 0, 0, 0, 0, 0});
    k[0].start(false);
    const auto block = [&](int rows) {
        for (int u = 1; u >= 0; --u)
            for (int b = 0; b < rows; ++b) k[u].wait(k[u].used + b);
        for (int u = 0; u < 2; ++u) k[u].release(rows, 1);
    };
    std::vector<long> want;
    for (int it = 0; it < items; ++it) {
        if (ROT && rot[it] == 0) continue;
        for (int r = 0; r < 2 * L; ++r) want.push_back(2L * L * it + r);
        for (int jp = 0; jp < 2; ++jp) {
            block(2);
            if (L == 3) block(1);
        }
    }
    k[0].drain();
    if (lost < 0 && g_rows != want) fault("rows of the items that use them, in order");
    finish(lost, (long)want.size(), err);
}

static const int kS = 4, kL = 3;
static uint64_t g_full[kS], g_empty[kS];

template <typename Keys>
static void rings(long lost, int consumers, int steps, bool warp_producer,
                  const std::function<void(Keys&, int)>& body) {
    static cpx<float> ring[kS * Keys::kRow];
    static char key[64];
    reset(lost, Keys::kRowBytes, key);
    for (auto& e : g_empty) g_bars[&e].count = g_bars[&e].pending = consumers;
    int32_t err = 0;
    volatile int abort = 0;
    const uint32_t rows = (uint32_t)steps * 2 * kL;
    std::vector<std::function<void()>> bodies;
    const auto make = [&](bool producer) {
        Keys k{};
        k.ring = ring;
        k.full = g_full;
        k.empty = g_empty;
        k.err = &err;
        k.abort = &abort;
        k.producer = producer;
        k.src = key;
        k.total = rows;
        return k;
    };
    for (int c = 0; c < consumers; ++c)
        bodies.push_back([&, c] {
            Keys k = make(c == 0 && !warp_producer);
            body(k, c);
            if (k.producer) k.drain();
        });
    if (warp_producer)
        bodies.push_back([&] {
            Keys k = make(false);
            k.issue_through(rows - 1);
            k.drain();
        });
    run(bodies);
    finish(lost, rows, err);
}

template <bool WATCH>
static void ring(long lost, bool warp_producer, int steps) {
    using Keys = RingKeys<float, 2, kS, WATCH>;
    rings<Keys>(lost, 3, steps, warp_producer, [&](Keys& k, int) {
        for (int i = 0; i < steps; ++i) {
            k.row0 = (uint32_t)i * 2 * kL;
            for (int p = 0; p < 2 * kL; ++p) {
                k.acquire(p);
                k.release(p);
            }
        }
    });
}

static void polled(long lost, int steps) {
    using Keys = PolledRingKeys<float, 2, kS>;
    rings<Keys>(lost, 3, steps, false, [&](Keys& k, int) {
        for (int i = 0; i < steps; ++i) {
            k.row0 = (uint32_t)i * 2 * kL;
            for (int p = 0; p < 2 * kL;) {
                const int nb = p % kL == 0 ? 2 : 1;
                bool landed[2] = {};
                for (int b = 0; b < nb; ++b) landed[b] = k.poll(p + b);
                for (int b = 0; b < nb; ++b) {
                    k.acquire_polled(p + b, landed[b]);
                    k.release(p + b);
                }
                p += nb;
            }
        }
    });
}

// two halves of one ciphertext: each reads one polynomial's rows, half 0 streams
static void pair(long lost, int steps) {
    using Keys = RingKeys<float, 2, kS>;
    static int met[2];
    met[0] = met[1] = 0;
    const auto pair_sync = [&](int h) {
        std::unique_lock<std::mutex> lk(g_lock);
        const int n = ++met[h];
        g_change.notify_all();
        wait_until(lk, false, [&] { return met[1 - h] >= n; });
    };
    const std::function<void(Keys&, int)> body = [&](Keys& k, int h) {
        for (int i = 0; i < steps; ++i) {
            k.row0 = (uint32_t)i * 2 * kL;
            for (int lev = 0; lev < kL; ++lev) {
                k.acquire(h * kL + lev);
                k.release(h * kL + lev);
            }
            if (k.producer) k.issue_through(k.row0 + 2 * kL - 1);
            pair_sync(h);
            pair_sync(h);
            if (k.producer) {
                k.stop_if(*k.abort);
                k.issue_upto(k.row0 + 2 * kL - 1);
            }
        }
        if (k.producer) k.issue_through(k.total - 1);
    };
    // a row is read by one half
    static cpx<float> slots[kS * Keys::kRow];
    static char key[64];
    reset(lost, Keys::kRowBytes, key);
    int32_t err = 0;
    volatile int abort = 0;
    const uint32_t rows = (uint32_t)steps * 2 * kL;
    std::vector<std::function<void()>> bodies;
    for (int h = 0; h < 2; ++h)
        bodies.push_back([&, h] {
            Keys k{slots, g_full, g_empty, 0, &err, &abort, h == 0, key, rows, 0};
            body(k, h);
            if (k.producer) k.drain();
        });
    run(bodies);
    finish(lost, rows, err);
}

int main(int, char** argv) {
    const std::string what = argv[1];
    const long lost = std::atol(argv[2]);
    if (what == "products2") products<2, false>({0, 0, 0}, lost);
    else if (what == "products3") products<3, false>({0, 0, 0}, lost);
    else if (what == "rotations2") products<2, true>({0, 7, 0, 0, 2047, 1, 0}, lost);  // items 1, 4, 5: rows 4, 16, 20 on
    else if (what == "rotations3") products<3, true>({5, 0, 1, 0}, lost);               // items 0, 2: rows 0, 12 on
    else if (what == "no_rotation") products<3, true>({0, 0, 0, 0, 0}, lost);
    else if (what == "no_items") products<3, true>({}, lost);
    else if (what == "ring") ring<false>(lost, false, 3);
    else if (what == "producer_warp") ring<true>(lost, true, 3);
    else if (what == "lane_pairs") polled(lost, 3);
    else if (what == "pair") pair(lost, 3);
    else return 2;
    for (const auto& f : g_faults) std::printf("%s\n", f.c_str());
    return g_faults.empty() ? 0 : 1;
}
