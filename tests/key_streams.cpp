// Host model of the key-row streams of csrc/key_stream.cuh: the barriers are
// simulated, one chosen row's copy never lands, and the streams are driven as
// the kernels drive them.  Faults that a GPU would not forgive are counted: a
// barrier armed twice in a phase, a copy into a slot whose last copy is still
// out, a stream that ends with a copy out and not waited for.
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <set>
#include <string>

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

static std::map<const uint64_t*, Bar> g_bars;
static std::map<const void*, const uint64_t*> g_out;  // slot -> barrier of a copy that has not landed
static std::set<const uint64_t*> g_drained;           // barriers waited for without the abort flag
static std::set<std::string> g_faults;
static const char* g_base;
static long g_lost = -1, g_copies = 0;
static size_t g_row_bytes;
static void fault(const char* what) { g_faults.insert(what); }

static void arrive(uint64_t* bar, long bytes) {
    Bar& b = g_bars[bar];
    if (b.pending == 0) fault("barrier armed or arrived at more than its count");
    else --b.pending;
    b.tx += bytes;
    b.settle();
}
inline void mbar_arrive(uint64_t* bar) { arrive(bar, 0); }
inline void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) { arrive(bar, bytes); }
inline void bulk_copy_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    if (g_out.count(dst)) fault("copy into a slot whose last copy has not landed");
    const long row = (static_cast<const char*>(src) - g_base) / (long)g_row_bytes;
    ++g_copies;
    if (row == g_lost) {
        g_out[dst] = bar;
        g_drained.erase(bar);
        return;
    }
    Bar& b = g_bars[bar];
    b.tx -= bytes;
    b.settle();
}
inline bool mbar_try_wait(uint64_t* bar, uint32_t parity) { return ((uint32_t)g_bars[bar].phase & 1) != parity; }
inline bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, const volatile int*) { return mbar_try_wait(bar, parity); }
inline bool mbar_wait_bounded(uint64_t* bar, uint32_t parity) {
    g_drained.insert(bar);
    return mbar_try_wait(bar, parity);
}
inline int atomicExch(int32_t* p, int32_t v) {
    const int old = *p;
    *p = v;
    return old;
}
inline void group_sync(int) {}
inline void __syncwarp() {}
struct Dim {
    unsigned x;
};
static Dim threadIdx{0};

}  // namespace tfhe_gb300

#include "key_stream.cuh"

using namespace tfhe_gb300;

static void reset(long lost, size_t row_bytes, const char* base) {
    g_bars.clear();
    g_out.clear();
    g_drained.clear();
    g_copies = 0;
    g_lost = lost;
    g_row_bytes = row_bytes;
    g_base = base;
}
static void finish(long lost, long rows, int32_t err) {
    for (const auto& o : g_out)
        if (!g_drained.count(o.second)) fault("a copy is out and nobody waits for it");
    if ((err != 0) != (lost >= 0)) fault("status word");
    if (lost < 0 && g_copies != rows) fault("rows streamed");
}

// A group of two threads over `items` items, blocks of two rows and one as the
// product kernel takes them.
template <int L>
static void products(int items, long lost) {
    using Keys = ItemKeys<L>;
    static uint64_t full[Keys::S];
    static cpx<float> ring[Keys::S * Keys::kRow];
    static char key[64];
    const char* src = key;
    reset(lost, Keys::kRowBytes, src);
    int32_t err = 0;
    volatile int abort = 0;
    Keys k[2] = {{ring, full, &err, &abort, src, 2 * L * Keys::kRowBytes, (uint32_t)items * 2 * L, 0, 0, 0},
                 {ring, full, &err, &abort, src, 2 * L * Keys::kRowBytes, (uint32_t)items * 2 * L, 0, 0, 1}};
    k[0].issue();
    const auto block = [&](int rows) {
        for (int u = 1; u >= 0; --u)
            for (int b = 0; b < rows; ++b) k[u].wait(k[u].used + b);
        for (int u = 0; u < 2; ++u) k[u].release(rows, 1);
    };
    for (int it = 0; it < items; ++it)
        for (int jp = 0; jp < 2; ++jp) {
            block(2);
            if (L == 3) block(1);
        }
    k[0].drain();
    finish(lost, (long)items * 2 * L, err);
}

int main(int argc, char** argv) {
    const std::string what = argv[1];
    const long lost = std::atol(argv[2]);
    if (what == "products2") products<2>(3, lost);
    else if (what == "products3") products<3>(3, lost);
    else return 2;
    for (const auto& f : g_faults) std::printf("%s\n", f.c_str());
    return g_faults.empty() ? 0 : 1;
}
