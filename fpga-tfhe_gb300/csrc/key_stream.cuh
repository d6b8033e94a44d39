// key_stream.cuh -- the streams of key rows from global into shared memory:
// which row goes into which slot, when a slot may be filled again, and how a
// stream ends after a bounded wait has given up.
//
// Only bookkeeping over the primitives of async_copy.cuh and group_sync of
// fft512.cuh, included before this file, so that the protocol can also be
// compiled for the host and run against a model of the barriers
// (tests/test_key_streams.py).
#pragma once
#include <stddef.h>
#include <stdint.h>

namespace tfhe_gb300 {

// Row stream of one group of 64 threads of k_products_stream: row r is row
// r % 2l of the group's item r / 2l.  A slot is refilled as soon as both warps
// of the group have used it.
//
// A wait that gives up ends the stream: its slot's copy has not landed, so the
// slot may not be armed or filled again.  drain() then waits for the copies
// that are out, so that none is in flight when the CTA ends.
template <int L>
struct ItemKeys {
    static constexpr int S = 2;  // row slots per group
    static constexpr size_t kRow = (size_t)2 * 2 * 512;
    static constexpr size_t kRowBytes = kRow * sizeof(cpx<float>);
    cpx<float>* ring;
    uint64_t* full;
    int32_t* err;
    volatile int* abort;
    const char* src;     // first item
    size_t item_stride;  // bytes from one item of the group to the next
    uint32_t total, next, used;  // total: rows of the stream; next: rows issued
    int t;

    // thread 0: rows up to used + S - 1 (all earlier uses of their slots are over)
    __device__ __forceinline__ void issue() {
        for (; next < total && next < used + S; ++next) {
            const uint32_t slot = next % S, item = next / (2 * L), row = next - item * (2 * L);
            mbar_arrive_expect_tx(&full[slot], (uint32_t)kRowBytes);
            bulk_copy_g2s(reinterpret_cast<char*>(ring) + slot * kRowBytes,
                          src + item * item_stride + row * kRowBytes, (uint32_t)kRowBytes, &full[slot]);
        }
    }
    __device__ __forceinline__ const cpx<float>* wait(uint32_t r) {
        if (!mbar_wait_bounded(&full[r % S], (r / S) & 1, abort)) {
            *abort = 1;
            atomicExch(err, 3);
            total = next;
        }
        __syncwarp();
        return ring + (r % S) * kRow;
    }
    // the group is done with its next `rows` rows
    __device__ __forceinline__ void release(int rows, int bar_id) {
        used += rows;
        group_sync(bar_id);
        if (t == 0) issue();
        __syncwarp();
    }
    // thread 0, at the end: every copy issued has landed (at once, unless a wait gave up)
    __device__ __forceinline__ void drain() {
        for (uint32_t r = next > S ? next - S : 0; r < next; ++r)
            if (!mbar_wait_bounded(&full[r % S], (r / S) & 1)) atomicExch(err, 3);
    }
};

}  // namespace tfhe_gb300
