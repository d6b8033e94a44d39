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

// Row stream of one group of 64 threads of k_products_stream: the 2l rows of
// each of the group's items in turn; with ROT only of those whose rotation is
// not 0, which are the ones that use them.  A slot is refilled as soon as both
// warps of the group have used it.
//
// A wait that gives up ends the stream: its slot's copy has not landed, so the
// slot may not be armed or filled again.  drain() then waits for the copies
// that are out, so that none is in flight when the CTA ends.
template <int L, bool ROT>
struct ItemKeys {
    static constexpr int S = 2;  // row slots per group
    static constexpr size_t kRow = (size_t)2 * 2 * 512;
    static constexpr size_t kRowBytes = kRow * sizeof(cpx<float>);
    static constexpr uint32_t kStopped = 1u << 31;
    cpx<float>* ring;
    uint64_t* full;
    int32_t* err;
    volatile int* abort;
    const char* src;     // first item
    size_t item_stride;  // bytes from one item of the group to the next
    const int32_t* rot;  // rotation of the first item, rot_stride apart
    int rot_stride;
    int items, t;
    uint32_t next, used;  // rows issued (+ kStopped once the stream has stopped), rows read
    // thread 0: the row to issue, and the rotation of the item after its own
    int item, row, ahead;

    // thread 0, once: the first rows.  stall: self-test of the waits, the slots
    // are armed and no copy is started.
    __device__ __forceinline__ void start(bool stall) {
        if (stall) {
            for (; items > 0 && next < S; ++next) mbar_arrive_expect_tx(&full[next], (uint32_t)kRowBytes);
            item = items;
            return;
        }
        item = -1;
        if (ROT && items > 0) ahead = rot[0];
        next_item();
        issue();
    }
    __device__ __forceinline__ void next_item() {
        row = 0;
        int a;
        do {
            ++item;
            a = ahead;
            if (ROT && item + 1 < items) ahead = rot[(size_t)(item + 1) * rot_stride];
        } while (ROT && item < items && a == 0);
    }
    // thread 0: rows up to used + S - 1 (all earlier uses of their slots are over)
    __device__ __forceinline__ void issue() {
        while (item < items && next < used + S) {
            const uint32_t slot = next % S;
            mbar_arrive_expect_tx(&full[slot], (uint32_t)kRowBytes);
            bulk_copy_g2s(reinterpret_cast<char*>(ring) + slot * kRowBytes,
                          src + item * item_stride + row * kRowBytes, (uint32_t)kRowBytes, &full[slot]);
            ++next;
            if (++row == 2 * L) next_item();
        }
    }
    __device__ __forceinline__ const cpx<float>* wait(uint32_t r) {
        if (!mbar_wait_bounded(&full[r % S], (r / S) & 1, abort)) {
            *abort = 1;
            atomicExch(err, 3);
            next |= kStopped;
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
    // thread 0, at the end: every copy issued has landed.  Without a wait that
    // gave up the group has waited for each of them.
    __device__ __forceinline__ void drain() {
        if (!(next & kStopped)) return;
        const uint32_t end = next & ~kStopped;
        for (uint32_t r = end > S ? end - S : 0; r < end; ++r)
            if (!mbar_wait_bounded(&full[r % S], (r / S) & 1)) atomicExch(err, 3);
    }
};

// Rows of the shared-memory ring (see k_blind_rotate_ring): row r lies in slot
// r % S.  Consumers go on after a wait has given up, releasing rows that never
// came, so a stream that has met one issues nothing more: the slot's copy may
// still be out.  A producer that reads every row itself notices by its own
// waits.  A producer warp looks at the abort flag before it fills a slot again
// (WATCH), the pair kernel's half once a step, when the other half has read its
// rows.  (A stopped stream is marked in next_issue: a total that changes costs
// the lane-pair kernel 3 %, the flag read for every row the pair kernel 8 %.)
template <typename R, int PARTS, int S, bool WATCH = false>
struct RingKeys {
    static constexpr size_t kRow = (size_t)2 * PARTS * 512;
    static constexpr size_t kRowBytes = kRow * sizeof(cpx<R>);
    static constexpr bool kShared = true;
    cpx<R>* ring;
    uint64_t* full;
    uint64_t* empty;
    uint32_t row0;
    int32_t* err;
    volatile int* abort;   // CTA-wide: set by the first wait that gives up
    // In-line producer (one thread of the CTA when there is no producer
    // warp): before taking row r it issues rows up to r + S - 1, waiting only
    // for rows it needs itself (<= r) and skipping ahead rows whose slot is
    // still held.
    bool producer;
    const char* src;       // key rows in global memory
    uint32_t total;        // rows to stream
    uint32_t next_issue;   // first row not issued yet; + kStopped once the stream has stopped
    static constexpr uint32_t kStopped = 1u << 31;

    __device__ __forceinline__ void give_up() {
        *abort = 1;
        atomicExch(err, 3);
        next_issue |= kStopped;
    }
    __device__ __forceinline__ void stop_if(int flag) { next_issue |= flag ? kStopped : 0u; }
    __device__ __forceinline__ bool stopped() {
        if (!WATCH || !*abort) return false;
        next_issue |= kStopped;
        return true;
    }
    __device__ __forceinline__ void issue_one() {
        const uint32_t slot = next_issue % S;
        mbar_arrive_expect_tx(&full[slot], (uint32_t)kRowBytes);
        bulk_copy_g2s(reinterpret_cast<char*>(ring) + slot * kRowBytes,
                      src + (size_t)next_issue * kRowBytes, (uint32_t)kRowBytes, &full[slot]);
        ++next_issue;
    }
    __device__ __forceinline__ void issue_upto(uint32_t r) {
        while (next_issue < total && next_issue < r + S) {
            const uint32_t slot = next_issue % S;
            if (next_issue >= S) {
                const uint32_t parity = ((next_issue / S) - 1) & 1;
                if (next_issue <= r) {
                    if (!mbar_wait_bounded(&empty[slot], parity, abort)) {
                        give_up();
                        return;
                    }
                } else if (!mbar_try_wait(&empty[slot], parity)) {
                    return;
                }
            }
            issue_one();
        }
    }
    // Issue rows up to r + S - 1 whose slots are free, without waiting.
    __device__ __forceinline__ void issue_ready(uint32_t r) {
        while (next_issue < total && next_issue < r + S) {
            if (next_issue >= S && !mbar_try_wait(&empty[next_issue % S], ((next_issue / S) - 1) & 1)) return;
            issue_one();
        }
    }
    // Issue every row up to `last` (inclusive), waiting for their slots: used
    // before the producer blocks on another group, for rows that group needs.
    // Deadlock-free as long as the rows whose slots are reused (<= last - S)
    // are released by consumers that need only rows already issued.
    __device__ __forceinline__ void issue_through(uint32_t last) {
        while (next_issue < total && next_issue <= last) {
            if (next_issue >= S) {
                if (!mbar_wait_bounded(&empty[next_issue % S], ((next_issue / S) - 1) & 1, abort)) {
                    give_up();
                    return;
                }
                if (stopped()) return;
            }
            issue_one();
        }
    }
    // wait until every issued copy has landed (end of kernel)
    __device__ __forceinline__ void drain() {
        const uint32_t end = next_issue & ~kStopped;
        for (uint32_t r = end > S ? end - S : 0; r < end; ++r)
            if (!mbar_wait_bounded(&full[r % S], (r / S) & 1)) atomicExch(err, 3);
    }
    __device__ __forceinline__ void prefetch(int, int, int) const {}
    __device__ __forceinline__ const cpx<R>* acquire(int p) {
        const uint32_t r = row0 + (uint32_t)p;
        if (producer) issue_upto(r);
        const uint32_t slot = r % S;
        if (!mbar_wait_bounded(&full[slot], (r / S) & 1, abort)) give_up();
        return ring + slot * kRow;
    }
    __device__ __forceinline__ void release(int p) const { mbar_arrive(&empty[(row0 + (uint32_t)p) % S]); }
};

// The lane-pair kernel's way to the rows: acquire() in two parts, so that the
// arrival test's round trip overlaps other work -- poll() issues rows whose
// slots are free (producer, without waiting) and tests once whether row p has
// landed, acquire_polled() issues and waits (bounded) only if it had not --
// and one lane releases a slot for its whole warp (the slot's count is the
// number of consumer warps).
template <typename R, int PARTS, int S>
struct PolledRingKeys : RingKeys<R, PARTS, S> {
    using Base = RingKeys<R, PARTS, S>;
    __device__ __forceinline__ bool poll(int p) {
        const uint32_t r = this->row0 + (uint32_t)p;
        if (this->producer) this->issue_ready(r);
        __syncwarp();
        return mbar_try_wait(&this->full[r % S], (r / S) & 1);
    }
    __device__ __forceinline__ const cpx<R>* acquire_polled(int p, bool landed) {
        const uint32_t r = this->row0 + (uint32_t)p;
        const uint32_t slot = r % S;
        if (!landed) {
            if (this->producer) this->issue_upto(r);
            if (!mbar_wait_bounded(&this->full[slot], (r / S) & 1, this->abort)) this->give_up();
        }
        __syncwarp();
        return this->ring + slot * Base::kRow;
    }
    __device__ __forceinline__ void release(int p) const {
        __syncwarp();
        if ((threadIdx.x & 31) == 0) mbar_arrive(&this->empty[(this->row0 + (uint32_t)p) % S]);
    }
};

}  // namespace tfhe_gb300
