// keyswitch_mma.cu -- batched LWE key switching as an exact matrix product on
// the tensor cores (tcgen05), for base 4 and t = 8.
//
// lweKeySwitch (kernel/src/lwe-keyswitch-functions.cpp:114-129, 228-241)
// subtracts, for every input coefficient i and digit level j, the table row
// KS[i][j][h] that the digit h selects (none for h = 0): a product of a 0/1
// matrix (one row per ciphertext, one column per (i, h, j), at most one 1 per
// (i, j)) with the table.  Torus32 sums are mod 2^32, so each table word is
// split into three signed 11-, 11- and 10-bit pieces, v = c0 + 2^11 c1 +
// 2^22 c2 mod 2^32, which FP16 holds exactly; a sum of at most 8,192 pieces
// of at most 1,024 stays within 2^23, where FP32 accumulation is exact in
// any order.  The three sums are put together in integers: the result is
// lweKeySwitch's, bit for bit.
//
// Against the gather kernel (keyswitch.cu), which is bound by the integer
// instructions that pick each ciphertext's row (2.9 ms for 4,096 key
// switches), the whole product is 2 x 4,096 x 24,576 x 1,920 FLOP, 0.2 ms at
// this part's tensor rate; a small batch is bound by streaming the table once
// (94 MB of pieces, 14 us).  Measured, gather kernel and this one: 4,096 key
// switches 2.88 and 0.246 ms (1.55 PFLOP/s, 0.80 of the cuBLAS BF16 rate),
// 517 0.391 and 0.067 ms, 64 87 and 31 us, one 29 and 27 us.
//
// One CTA computes 256 ciphertexts x 80 output words (N = 240: the three
// pieces of each) over a span of coefficients: accumulators of two M = 128
// halves in TMEM, 240 columns each.  The table lies in memory in the order
// the tensor core reads it (K-major core matrices of 8 rows x 16 bytes,
// [tile][i][h][n][8 levels]), so a stage of two coefficients is one
// contiguous 23 KB bulk copy.  Eight warps make the 0/1 matrix, one
// ciphertext a thread: the eight levels of one (i, h) are 16 bytes, made from
// the coefficient's packed digits with a few bit operations.  One thread
// issues the matrix instructions, one warp the copies; four stages.  Small
// batches split the coefficients over enough CTAs to fill the SMs, and the
// parts add into the zeroed output with integer atomics (exact in any order).
#include <cuda_fp16.h>

#include "async_copy.cuh"
#include "engine.h"

namespace tfhe_gb300 {

namespace {

constexpr int kTileM = 256;      // ciphertexts per CTA
constexpr int kTileC = 80;       // output words per CTA
constexpr int kPieces = 3;
constexpr int kTileN = kPieces * kTileC;
constexpr int kLevels = 8;       // t
constexpr int kStageCoefs = 2;   // input coefficients per stage
constexpr int kChunks = 3 * kStageCoefs;                 // 16-byte K chunks (8 levels of one digit value) per stage
constexpr int kStages = 4;
constexpr int kGroupStages = 4;  // spans are multiples of 8 coefficients
constexpr uint32_t kAChunk = kTileM * 16, kBChunk = kTileN * 16;
constexpr uint32_t kABytes = kChunks * kAChunk, kBBytes = kChunks * kBChunk;
constexpr uint32_t kStageBytes = kABytes + kBBytes;
constexpr size_t kBarOff = (size_t)kStages * kStageBytes;
constexpr size_t kSmem = kBarOff + (3 * kStages + 1) * sizeof(uint64_t) + 16;
constexpr int kMakers = 8;                       // warps that make the 0/1 matrix and, at the end, read the sums
constexpr int kThreads = (kMakers + 2) * 32;
constexpr uint32_t kTmemCols = 512;              // two accumulators, 256 columns apart
static_assert(kStageBytes % 16 == 0 && kABytes % 16 == 0, "bulk copies");

// Shared-memory operand descriptor, K-major without swizzle: core matrices
// (8 rows x 16 bytes) 128 bytes apart along M/N, `k_stride` along K.
__device__ __forceinline__ uint64_t operand_desc(uint32_t addr, uint32_t k_stride) {
    return (uint64_t)((addr & 0x3ffff) >> 4) | ((uint64_t)(k_stride >> 4) << 16) | ((uint64_t)(128 >> 4) << 32) |
           ((uint64_t)1 << 46);
}

// kind::f16: FP16 operands, both K-major, FP32 accumulator, M = 128
constexpr uint32_t kInstr = (1u << 4) | ((uint32_t)(kTileN >> 3) << 17) | ((128u >> 4) << 24);

__device__ __forceinline__ void mma_f16(uint32_t d, uint64_t a, uint64_t b, bool accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a), "l"(b), "r"(kInstr), "r"((uint32_t)accumulate)
        : "memory");
}

__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void tmem_load16(uint32_t addr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(addr));
}

// The 16 bytes of digit value h: FP16 1.0 at place p where level 7 - p's
// digit is h.  u: the eight digits, level 0 in the top two of 16 bits.
__device__ __forceinline__ uint4 one_hot(uint32_t u, uint32_t h) {
    const uint32_t m = ~(u ^ (h * 0x5555u));
    const uint32_t e = m & (m >> 1) & 0x5555u;  // bit 2(7 - j): level j's digit is h
    const uint32_t y = e | (e << 14);           // bits 4w and 4w + 2 of e, 16 apart from bit 4w on
    return make_uint4((y & 0x10001u) * 0x3c00u, ((y >> 4) & 0x10001u) * 0x3c00u, ((y >> 8) & 0x10001u) * 0x3c00u,
                      ((y >> 12) & 0x10001u) * 0x3c00u);
}

__global__ void __launch_bounds__(kThreads, 1)
    k_keyswitch_mma(const void* __restrict__ tiles, const int32_t* __restrict__ in, int32_t* __restrict__ out, int count,
                    int n, int n_in, int parts, int32_t* err, int stall) {
    extern __shared__ __align__(128) char smem[];
    uint64_t* full_a = reinterpret_cast<uint64_t*>(smem + kBarOff);
    uint64_t* full_b = full_a + kStages;
    uint64_t* empty = full_b + kStages;
    uint64_t* done = empty + kStages;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
    volatile int* abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const int ntiles = (n + kTileC) / kTileC;  // n + 1 output words
    const int part = blockIdx.x % parts, tile = (blockIdx.x / parts) % ntiles;
    const int c0 = (int)(blockIdx.x / (parts * ntiles)) * kTileM;
    // this part's stages
    const int groups = n_in / (kStageCoefs * kGroupStages);
    const int s0 = (int)((long long)groups * part / parts) * kGroupStages;
    const int s1 = (int)((long long)groups * (part + 1) / parts) * kGroupStages;
    const int stages = s1 - s0;
    const bool two = count - c0 > 128;  // the second half has ciphertexts
    const int warp = threadIdx.x >> 5;

    if (threadIdx.x == 0) {
        for (int i = 0; i < kStages; ++i) {
            mbar_init(&full_a[i], kMakers);
            mbar_init(&full_b[i], 1);
            mbar_init(&empty[i], 1);
        }
        mbar_init(done, 1);
        *abort = 0;
        fence_mbar_init();
    }
    if (warp == kMakers) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(tmem_slot);
    const auto gave_up = [&]() {
        *abort = 1;
        atomicExch(err, 3);
    };

    if (warp < kMakers) {
        // the 0/1 matrix, one ciphertext a thread
        const int c = c0 + threadIdx.x;
        const bool live = c < count;
        const int32_t* src = in + (size_t)(live ? c : c0) * (n_in + 1) + s0 * kStageCoefs;
        const uint32_t prec_offset = 1u << (32 - (1 + 2 * kLevels));
        const bool work = threadIdx.x < 128 || two;
        constexpr int kAhead = kStageCoefs * kGroupStages;
        uint32_t next[kAhead];
#pragma unroll
        for (int k = 0; k < kAhead; ++k) next[k] = (uint32_t)src[k];
#pragma unroll 1
        for (int g = 0; g < stages; g += kGroupStages) {
            uint32_t cur[kAhead];
#pragma unroll
            for (int k = 0; k < kAhead; ++k) cur[k] = (next[k] + prec_offset) >> 16;
            src += kAhead;
            if (g + kGroupStages < stages) {
#pragma unroll
                for (int k = 0; k < kAhead; ++k) next[k] = (uint32_t)src[k];
            }
#pragma unroll
            for (int q = 0; q < kGroupStages; ++q) {
                const int it = g + q;
                if (it >= kStages && !mbar_wait_bounded(&empty[q], ((it / kStages) - 1) & 1, abort)) gave_up();
                __syncwarp();
                if (work) {
                    char* a = smem + q * kStageBytes + threadIdx.x * 16;
#pragma unroll
                    for (int e = 0; e < kStageCoefs; ++e)
#pragma unroll
                        for (uint32_t h = 1; h < 4; ++h)
                            *reinterpret_cast<uint4*>(a + (3 * e + (h - 1)) * kAChunk) =
                                one_hot(cur[kStageCoefs * q + e], h);
                }
                fence_proxy_async();
                __syncwarp();
                if ((threadIdx.x & 31) == 0) mbar_arrive(&full_a[q]);
            }
        }
        // without the abort flag: `done` completes after the last matrix
        // instruction that was issued, also when a wait has given up
        bool summed = mbar_wait_bounded(done, 0);
        if (!summed) gave_up();
        summed = __all_sync(0xffffffffu, summed);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // row 32 (warp % 4) + lane of half warp / 4, 16 output words at a time
        const int half = warp >> 2;
        const uint32_t taddr = tmem + ((uint32_t)(warp & 3) << 21) + (uint32_t)half * 256;
        if (summed && (half == 0 || two)) {
            const int col0 = tile * kTileC;
            const uint32_t body = live && part == 0 ? (uint32_t)in[(size_t)c * (n_in + 1) + n_in] : 0u;
            int32_t* o = out + (size_t)(live ? c : c0) * (n + 1) + col0;
#pragma unroll 1
            for (int k = 0; k < kTileC / 16; ++k) {
                uint32_t p0[16], p1[16], p2[16];
                tmem_load16(taddr + 16 * k, p0);
                tmem_load16(taddr + kTileC + 16 * k, p1);
                tmem_load16(taddr + 2 * kTileC + 16 * k, p2);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    const int col = 16 * k + e;
                    if (!live || col0 + col > n) continue;
                    const uint32_t sum = (uint32_t)__float2int_rn(__uint_as_float(p0[e])) +
                                         ((uint32_t)__float2int_rn(__uint_as_float(p1[e])) << 11) +
                                         ((uint32_t)__float2int_rn(__uint_as_float(p2[e])) << 22);
                    const uint32_t val = (col0 + col == n ? body : 0u) - sum;
                    if (parts == 1) o[col] = (int32_t)val;
                    else atomicAdd(reinterpret_cast<unsigned*>(o + col), val);
                }
                __syncwarp();
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    } else if (warp == kMakers) {
        if ((threadIdx.x & 31) == 0) {
#pragma unroll 1
            for (int it = 0; it < stages; ++it) {
                const int q = it % kStages;
                if (!mbar_wait_bounded(&full_b[q], (it / kStages) & 1, abort) ||
                    !mbar_wait_bounded(&full_a[q], (it / kStages) & 1, abort)) {
                    gave_up();
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t a = smem_u32(smem + q * kStageBytes), b = a + kABytes;
#pragma unroll
                for (int k = 0; k < kChunks / 2; ++k) {
                    const uint64_t bd = operand_desc(b + 2 * k * kBChunk, kBChunk);
                    mma_f16(tmem, operand_desc(a + 2 * k * kAChunk, kAChunk), bd, it > 0 || k > 0);
                    if (two) mma_f16(tmem + 256, operand_desc(a + 2 * k * kAChunk + 128 * 16, kAChunk), bd, it > 0 || k > 0);
                }
                mma_commit(&empty[q]);
            }
            mma_commit(done);
            // the accumulators are freed below, with no matrix instruction in flight
            if (!mbar_wait_bounded(done, 0)) atomicExch(err, 3);
        }
        __syncwarp();
    } else {
        if ((threadIdx.x & 31) == 0) {
            const char* src = reinterpret_cast<const char*>(tiles) +
                              ((size_t)tile * n_in + (size_t)s0 * kStageCoefs) * (3 * kBChunk);
            int issued = 0;
#pragma unroll 1
            for (int it = 0; it < (stall ? min(stages, 1) : stages); ++it, ++issued) {
                const int q = it % kStages;
                if (it >= kStages && !mbar_wait_bounded(&empty[q], ((it / kStages) - 1) & 1, abort)) {
                    gave_up();
                    break;
                }
                mbar_arrive_expect_tx(&full_b[q], kBBytes);
                bulk_copy_g2s(smem + q * kStageBytes + kABytes, src + (size_t)it * kBBytes, kBBytes, &full_b[q]);
            }
            // no copy in flight at the end of the kernel
            for (int it = issued > kStages ? issued - kStages : 0; it < issued; ++it)
                if (!mbar_wait_bounded(&full_b[it % kStages], (it / kStages) & 1)) atomicExch(err, 3);
        }
        __syncwarp();
    }
    __syncthreads();
    if (warp == kMakers) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
    }
}

// The table in the order k_keyswitch_mma reads it: [tile][i][h][piece * 80 +
// word][place], place p holding level 7 - p (one thread per 16 bytes).
__global__ void k_keyswitch_tiles(const int32_t* __restrict__ ks, int row_stride, int n, int n_in, uint4* __restrict__ tiles,
                                  size_t total) {
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= total) return;
    const int nn = (int)(idx % kTileN);
    const size_t row = idx / kTileN;  // (tile, i, h)
    const int h = (int)(row % 3) + 1, i = (int)((row / 3) % n_in), tile = (int)(row / 3 / n_in);
    const int piece = nn / kTileC, col = tile * kTileC + nn % kTileC;
    uint32_t w[4];
#pragma unroll
    for (int p = 0; p < 8; p += 2) {
        uint32_t half[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int j = 7 - (p + e);
            const uint32_t v = col <= n ? (uint32_t)ks[((size_t)(i * kLevels + j) * 4 + h) * row_stride + col] : 0u;
            const int32_t b0 = (int32_t)((v + 1024u) & 2047u) - 1024;
            const uint32_t v1 = (v - (uint32_t)b0) >> 11;
            const int32_t b1 = (int32_t)((v1 + 1024u) & 2047u) - 1024;
            const uint32_t v2 = (v - (uint32_t)b0) - ((uint32_t)b1 << 11);
            const int32_t b2 = (int32_t)v2 >> 22;
            const int32_t val = piece == 0 ? b0 : piece == 1 ? b1 : b2;
            half[e] = __half_as_ushort(__int2half_rn(val));
        }
        w[p / 2] = half[0] | (half[1] << 16);
    }
    tiles[idx] = make_uint4(w[0], w[1], w[2], w[3]);
}

size_t tile_units(const DevParams& P) {
    const size_t ntiles = (size_t)(P.n + kTileC) / kTileC;
    return ntiles * (size_t)(P.k * P.N) * 3 * kTileN;
}

}  // namespace

size_t keyswitch_tile_bytes(const DevParams& P) {
    // n up to 639, as in the gather kernel
    if (P.ks_basebit != 2 || P.ks_t != kLevels || P.n > 639 || (P.k * P.N) % (kStageCoefs * kGroupStages)) return 0;
    return tile_units(P) * sizeof(uint4);
}

cudaError_t launch_keyswitch_tiles(const DevParams& P, const int32_t* ks, int32_t row_stride, void* tiles,
                                   cudaStream_t st) {
    const size_t total = tile_units(P);
    k_keyswitch_tiles<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(ks, row_stride, P.n, P.k * P.N,
                                                                       reinterpret_cast<uint4*>(tiles), total);
    return cudaGetLastError();
}

cudaError_t launch_keyswitch_mma(const DevParams& P, const void* tiles, const int32_t* in, int32_t* out, int count,
                                 int32_t* err, cudaStream_t st, bool stall) {
    if (count <= 0) return cudaSuccess;
    const int n_in = P.k * P.N;
    const int blocks = ((count + kTileM - 1) / kTileM) * ((P.n + kTileC) / kTileC);
    // as many parts as fill the SMs once
    int parts = kSmCount / blocks;
    if (parts < 1) parts = 1;
    if (parts > 32) parts = 32;
    cudaError_t e = cudaFuncSetAttribute(k_keyswitch_mma, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
    if (e != cudaSuccess) return e;
    if (parts > 1) {
        e = cudaMemsetAsync(out, 0, (size_t)count * (P.n + 1) * sizeof(int32_t), st);
        if (e != cudaSuccess) return e;
    }
    k_keyswitch_mma<<<blocks * parts, kThreads, kSmem, st>>>(tiles, in, out, count, P.n, n_in, parts, err, stall);
    return cudaGetLastError();
}

}  // namespace tfhe_gb300
