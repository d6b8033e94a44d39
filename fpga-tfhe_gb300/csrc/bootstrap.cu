// bootstrap.cu -- FFT-domain kernels of the GB300 TFHE engine:
//   * key conversion (TGSW time domain -> engine FFT layout, both forms)
//   * the external product, MuxRotate and the blind-rotation loop, one
//     kernel template (EpMode) built on a fused step:
//       rotate (X^a - 1) -> gadget digits -> twisted FFT-512 -> MAC against
//       the key -> inverse FFT-512 -> Torus32 -> accumulate
//   * bootstrap front end (modulus switch, rotated test vector) and sample
//     extraction, fused into the blind-rotation kernel
//   * small kernels: gate combination, X^a - 1 rotation, extraction
//   * the Lagrange processor (polynomial <-> Lagrange half-complex form in
//     the reference's layout)
//
// Reference call stack restated here (paths inside shreks99/fpga-tfhe):
//   tfhe_blindRotate_FFT         kernel/src/tfhe_blindRotate_FFT/tfhe_blindRotate_FFT.cpp:61-147
//   tfhe_MuxRotate_FFT_FPGA      .../tfhe_MuxRotate_FFT.cpp:56-85
//   tLweMulByXaiMinusOne_FPGA    .../tfhe_MuxRotate_FFT.cpp:5-33
//   tGswFFTExternMulToTLwe_FPGA  .../tGswFFTExternMulToTLwe.cpp:203-247
//   decompose                    .../tGswFFTExternMulToTLwe.cpp:76-95
//   ifft (Int -> Lagrange)       .../tGswFFTExternMulToTLwe.cpp:97-130
//   MAC                          .../tGswFFTExternMulToTLwe.cpp:166-197
//   TorusPolynomial_fft          .../TorusPolynomial_fft.cpp:4-43
//   modulus switch / test vector kernel/src/tfhe_bootstrap_woKS_FFT/tfhe_bootstrap_woKS_FFT.cpp:3-10,57-66
//   X^{2N-b} rotation            kernel/src/tfhe_blindRotateAndExtract/mulByXaiOrCopy.cpp:25-41
#include <cooperative_groups.h>
#include <math.h>

#include <algorithm>

#include "async_copy.cuh"
#include "engine.h"
#include "fft512.cuh"
#include "key_stream.cuh"

namespace tfhe_gb300 {

namespace {

constexpr int kN = 1024;
constexpr int kHalf = 512;
// Table layout (complex entries): W^(tq) as [q][t] (512), W^(8jq) as [q][j]
// (64), psi^t W^(tq) as [q][t] (512), then psi^x (512).  The blind-rotation
// and external-product kernels keep only the "hot" part [kTabB, kTabB +
// kHotSize) in shared memory: W^(8jq) at 0, psi^t W^(tq) at 64.
constexpr int kTabA = 0;
constexpr int kTabB = 512;
constexpr int kTabT = 576;
constexpr int kTabPsi = 1088;
constexpr int kTabSize = 1600;
constexpr int kHotSize = 576;

// ----------------------------------------------------------------------
// helpers
// ----------------------------------------------------------------------
template <typename R>
__device__ __forceinline__ const cpx<R>* table_ptr(const Tables& T);
template <>
__device__ __forceinline__ const cpx<float>* table_ptr<float>(const Tables& T) {
    return reinterpret_cast<const cpx<float>*>(T.tw32);
}
template <>
__device__ __forceinline__ const cpx<double>* table_ptr<double>(const Tables& T) {
    return reinterpret_cast<const cpx<double>*>(T.tw64);
}

__device__ __forceinline__ int32_t mod_switch_2n(int32_t phase) {
    // numeric-functions.cpp:59-65 with Msize = 2N = 2048
    const uint64_t interv = ((UINT64_C(1) << 63) / 2048u) * 2;
    const uint64_t half_interval = interv / 2;
    const uint64_t phase64 = ((uint64_t)(int64_t)phase << 32) + half_interval;
    return (int32_t)(phase64 / interv);
}

// (X^a * p)[x] for a in [0, 2N): s = (x - a) mod 2N; +p[s] or -p[s - N].
__device__ __forceinline__ int32_t rot_coef(const int32_t* p, int x, int a) {
    const int s = (x - a) & (2 * kN - 1);
    const int32_t v = p[s & (kN - 1)];
    return s < kN ? v : (int32_t)(0u - (uint32_t)v);
}

// Coefficient i of X^{2N - barb} tv: the rotated test vector the blind
// rotation starts from.  tv = nullptr is the constant mu of the gate
// bootstrap (tfhe_bootstrap_woKS_FFT.cpp:63-66, mulByXaiOrCopy.cpp:25-41),
// else the polynomial of item c (programmable bootstrap).
__device__ __forceinline__ int32_t test_vector_coef(const EpArgs& a, int c, int barb, int i) {
    if (!a.tv) return (((i + barb) & (2 * kN - 1)) < kN) ? a.mu : -a.mu;
    return rot_coef(a.tv + (size_t)c * a.tv_stride, i, (2 * kN - barb) & (2 * kN - 1));
}

// Rounding the inverse transform's FP32 output to Torus32 without a float ->
// int64 conversion (on this part that conversion issues to the narrow FP64
// pipe).  M = 1.5 * 2^23: for |y| < 2^22 the sum y + M rounds y to the
// nearest integer, whose two's complement is then the low bits of the sum's
// encoding.
constexpr float kRoundMagic = 12582912.0f;
constexpr int32_t kRoundMagicBits = 0x4B400000;

// round(v / 512) mod 2^32 for |v / 512| < 2^22 (the high key part's product:
// about 2^18 typical, the exactness limit of FP32 is 2^24): one FMA and one
// integer add; both halves of a packed pair at once.
__device__ __forceinline__ void round_small_pair(cpx<float> z, uint32_t& a0, uint32_t& a1) {
    const float2 r = __ffma2_rn(pk(z), bc(0x1p-9f), bc(kRoundMagic));
    a0 = (uint32_t)(__float_as_int(r.x) - kRoundMagicBits);
    a1 = (uint32_t)(__float_as_int(r.y) - kRoundMagicBits);
}

// round(v / 512) mod 2^32 for any |v / 512| < 2^53 (the low key part's
// product, up to about 2^36): the multiple of 2^32 is removed exactly in
// FP32 (q = rint(v / 2^41), a = v - q 2^41 exact, |a| <= 2^40), and the
// remainder (|a / 512| <= 2^31) goes through a float -> int32 conversion,
// which does not use the FP64 pipe.  (A remainder of exactly +2^31
// saturates one unit short: an error of one unit in the low part.)
__device__ __forceinline__ void round_wrap_pair(cpx<float> z, uint32_t& a0, uint32_t& a1) {
    const float2 q = __fadd2_rn(__ffma2_rn(pk(z), bc(0x1p-41f), bc(kRoundMagic)), bc(-kRoundMagic));
    const float2 a = __ffma2_rn(make_float2(-q.x, -q.y), bc(0x1p41f), pk(z));
    const float2 sc = __fmul2_rn(a, bc(0x1p-9f));
    a0 = (uint32_t)__float2int_rn(sc.x);
    a1 = (uint32_t)__float2int_rn(sc.y);
}

// FP64 conversions by integer operations.  The FP64 unit of this part takes
// 19 clocks per warp instruction and SM (64 for a warp alone), and conversions
// to and from double 16, so the integer pipe does them: a normal float (or
// +0) widened by its bits, and the truncation of the inverse transform's
// output, whose division by 512 is part of the shift.  Exact, so the same
// values as (double)f and (int64_t)(z / 512) mod 2^32 for |z / 512| < 2^63.
// FP64 layer of 456 on the 3-per-CTA kernel: 92.6 -> 87.0 ms.
__device__ __forceinline__ double widen_float(float f) {
    const uint32_t b = (uint32_t)__float_as_int(f);
    const uint32_t hi = (b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + ((1023u - 127u) << 20));
    return b ? __hiloint2double((int)hi, (int)(b << 29)) : 0.0;
}
__device__ __forceinline__ uint32_t trunc_div512(double z) {
    const uint32_t hi = (uint32_t)__double2hiint(z), lo = (uint32_t)__double2loint(z);
    const int e = (int)((hi >> 20) & 0x7ffu) - 1023 - 9;  // exponent of z / 512
    const uint64_t m = ((uint64_t)((hi & 0xfffffu) | 0x100000u) << 32) | lo;
    const uint32_t v = (uint32_t)(e <= 52 ? m >> (52 - max(e, -1)) : m << min(e - 52, 63));
    return hi >> 31 ? 0u - v : v;
}

// Gadget digit of u at `decal` as a transform input: ((u >> decal) & mask) -
// halfBg.  FP32: the masked digit m < 2^22 ORed into the encoding of the
// magic constant is the float M + m, and one subtraction of M + halfBg
// gives m - halfBg exactly.
template <typename R>
__device__ __forceinline__ R digit_value(uint32_t u, int decal, uint32_t mask, int halfBg) {
    if constexpr (sizeof(R) == 4) {
        return __int_as_float((int32_t)(((u >> decal) & mask) | (uint32_t)kRoundMagicBits)) -
               (kRoundMagic + (float)halfBg);
    } else {
        return (R)widen_float(digit_value<float>(u, decal, mask, halfBg));
    }
}

// Both digits of a folded point (coefficients x and x + 512) as one
// complex transform input; FP32: one packed subtraction.
template <typename R>
__device__ __forceinline__ cpx<R> digit_pair(uint32_t u0, uint32_t u1, int decal, uint32_t mask, int halfBg) {
    if constexpr (sizeof(R) == 4) {
        const float f0 = __int_as_float((int32_t)(((u0 >> decal) & mask) | (uint32_t)kRoundMagicBits));
        const float f1 = __int_as_float((int32_t)(((u1 >> decal) & mask) | (uint32_t)kRoundMagicBits));
        return unpk(__fadd2_rn(make_float2(f0, f1), bc(-(kRoundMagic + (float)halfBg))));
    } else {
        return {digit_value<R>(u0, decal, mask, halfBg), digit_value<R>(u1, decal, mask, halfBg)};
    }
}

// ----------------------------------------------------------------------
// shared-memory plan of the FFT kernels
//   [tables: kTabSize cpx<R>] then per 64-thread group:
//   [acc: 2 x 1024 int32][NB x 2 exchange buffers of 576 cpx<R>]
// NB = number of transforms run together (max of L and the parts).
// ----------------------------------------------------------------------
template <typename R, int NB>
struct SmemPlan {
    static constexpr size_t tables = kHotSize * sizeof(cpx<R>);
    static constexpr size_t acc = 2 * kN * sizeof(int32_t);
    static constexpr size_t scratch = NB * 2 * kScratchStride * sizeof(cpx<R>);
    static constexpr size_t group = acc + scratch;
    static size_t total(int groups) { return tables + groups * group; }
};

template <typename R>
__device__ __forceinline__ FftScratch<R> scratch_at(char* base) {
    cpx<R>* s = reinterpret_cast<cpx<R>*>(base);
    return {s, s + kScratchStride};
}

template <typename R>
__device__ __forceinline__ void load_tables(cpx<R>* dst, const Tables& T) {
    const cpx<R>* src = table_ptr<R>(T);
    for (int i = threadIdx.x; i < kTabSize; i += blockDim.x) dst[i] = src[i];
}

template <typename R>
__device__ __forceinline__ FftTwiddles<R> twiddles_at(const cpx<R>* tables) {
    return {tables + kTabA, tables + kTabB};
}

// the hot tables (twist-folded pass-A twiddles, pass-B twiddles)
template <typename R>
__device__ __forceinline__ void load_hot_tables(cpx<R>* dst, const Tables& T) {
    const cpx<R>* src = table_ptr<R>(T) + kTabB;
    for (int i = threadIdx.x; i < kHotSize; i += blockDim.x) dst[i] = src[i];
}

template <typename R>
__device__ __forceinline__ FftTwiddles<R> hot_twiddles(const cpx<R>* hot) {
    return {hot + (kTabT - kTabB), hot};
}

// ----------------------------------------------------------------------
// the fused step: out = EP(ROT ? (X^a - 1) acc : acc);
//                 acc = (ROT ? acc : 0) + out
// A key row p of a TGSW in engine layout is [2 outputs][PARTS][512
// key_index order] complex values; `Keys` says where rows come from:
//   GlobalKeys -- straight from global memory (L2), 16-byte loads, with an
//                 L1 prefetch of the rows ahead of the transform;
//   RingKeys   -- from a shared-memory ring filled by a producer warp with
//                 bulk copies (see k_blind_rotate_ring).
// The l digit polynomials of an input polynomial are transformed together
// (fft512_forward_tw_multi), and IB parts of an output polynomial are
// transformed back together.
// ----------------------------------------------------------------------
template <typename R, int PARTS, int NB, typename Bar = int>
struct StepCtx {
    FftTwiddles<R> tw;  // smem twiddles: a = psi^t W^(tq) (twist folded), b = W^(8jq)
    FftIdx ix;          // this thread's exchange slots
    FftScratch<R> s[NB];
    int32_t* acc;       // smem 2 x N
    int t;
    Bar bar_id;
    int Bgbit, split;
    uint32_t offset;
};

template <typename R, int PARTS>
struct GlobalKeys {
    static constexpr size_t kRow = (size_t)2 * PARTS * kHalf;
    const cpx<R>* gsw;
    __device__ __forceinline__ void prefetch(int p0, int np, int t) const {
        const int lines = (int)(np * kRow * sizeof(cpx<R>) / 128);
        const char* gb = reinterpret_cast<const char*>(gsw + (size_t)p0 * kRow);
        for (int ln = t; ln < lines; ln += 64)
            asm volatile("prefetch.global.L1 [%0];" ::"l"(gb + (size_t)ln * 128));
    }
    __device__ __forceinline__ const cpx<R>* acquire(int p) const { return gsw + (size_t)p * kRow; }
    __device__ __forceinline__ void release(int) const {}
    static constexpr bool kShared = false;
};

template <bool SHARED>
__device__ __forceinline__ float4 key_load4(const float4* p) {
    if constexpr (SHARED) return *p;
    else return __ldg(p);
}

template <typename R, int PARTS, bool SHARED>
__device__ __forceinline__ void mac_row(cpx<R> (&out)[2][PARTS][8], const cpx<R> (&v)[8],
                                        const cpx<R>* __restrict__ g, int t) {
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int pt = 0; pt < PARTS; ++pt) {
            const cpx<R>* gk = g + (j * PARTS + pt) * kHalf;
            if constexpr (sizeof(R) == 4) {
                const float4* g4 = reinterpret_cast<const float4*>(gk);
#pragma unroll
                for (int qq = 0; qq < 4; ++qq) {
                    const float4 w = key_load4<SHARED>(g4 + qq * 64 + t);
                    const cpx<R> k0 = {(R)w.x, (R)w.y}, k1 = {(R)w.z, (R)w.w};
                    out[j][pt][2 * qq] = cmac(out[j][pt][2 * qq], v[2 * qq], k0);
                    out[j][pt][2 * qq + 1] = cmac(out[j][pt][2 * qq + 1], v[2 * qq + 1], k1);
                }
            } else {
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const cpx<R> k0 = gk[key_index<R>(t, q)];
                    out[j][pt][q] = cmac(out[j][pt][q], v[q], k0);
                }
            }
        }
}

// The L levels of input polynomial jp: digits, forward transforms run
// together, and their key rows multiply-accumulated.
template <int L, typename R, int PARTS, int NB, typename Bar, typename Keys>
__device__ __forceinline__ void forward_levels(const StepCtx<R, PARTS, NB, Bar>& S, Keys& keys,
                                               cpx<R> (&out)[2][PARTS][8], const uint32_t (&r0)[8],
                                               const uint32_t (&r1)[8], int p0, uint32_t mask, int halfBg) {
    const int t = S.t;
    cpx<R> v[L][8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
#pragma unroll
        for (int b = 0; b < L; ++b) v[b][r] = digit_pair<R>(r0[r], r1[r], 32 - (b + 1) * S.Bgbit, mask, halfBg);
    }
    fft512_forward_tw_multi<L>(v, *reinterpret_cast<const FftScratch<R>(*)[L]>(S.s), S.tw, S.ix, t, S.bar_id);
#pragma unroll
    for (int b = 0; b < L; ++b) {
        mac_row<R, PARTS, Keys::kShared>(out, v[b], keys.acquire(p0 + b), t);
        keys.release(p0 + b);
    }
}

template <typename R, int PARTS, bool ROT, int L, int IB, int NB, typename Bar, typename Keys>
__device__ __forceinline__ void ep_step(const StepCtx<R, PARTS, NB, Bar>& S, Keys& keys, int a) {
    static_assert(PARTS % IB == 0 && L <= NB && IB <= NB, "batch sizes");
    const int t = S.t;
    const int halfBg = 1 << (S.Bgbit - 1);
    const uint32_t mask = (1u << S.Bgbit) - 1;

    cpx<R> out[2][PARTS][8];
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int pt = 0; pt < PARTS; ++pt)
#pragma unroll
            for (int q = 0; q < 8; ++q) out[j][pt][q] = {(R)0, (R)0};

#pragma unroll 1
    for (int jp = 0; jp < 2; ++jp) {
        keys.prefetch(jp * L, L, t);
        const int32_t* src = S.acc + jp * kN;
        uint32_t r0[8], r1[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const int x0 = t + 64 * r;
            if (ROT) {
                r0[r] = (uint32_t)rot_coef(src, x0, a) - (uint32_t)src[x0];
                r1[r] = (uint32_t)rot_coef(src, x0 + kHalf, a) - (uint32_t)src[x0 + kHalf];
            } else {
                r0[r] = (uint32_t)src[x0];
                r1[r] = (uint32_t)src[x0 + kHalf];
            }
            r0[r] += S.offset;
            r1[r] += S.offset;
        }
        forward_levels<L>(S, keys, out, r0, r1, jp * L, mask, halfBg);
    }

    // back to the coefficient domain (j unrolled: out[j] must stay in registers)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        uint32_t c0[8], c1[8];
#pragma unroll
        for (int pt0 = 0; pt0 < PARTS; pt0 += IB) {
            cpx<R> v[IB][8];
#pragma unroll
            for (int b = 0; b < IB; ++b)
#pragma unroll
                for (int q = 0; q < 8; ++q) v[b][q] = out[j][pt0 + b][q];
            fft512_inverse_tw_multi<IB>(v, *reinterpret_cast<const FftScratch<R>(*)[IB]>(S.s), S.tw, S.ix, t,
                                        S.bar_id);
#pragma unroll
            for (int q = 0; q < 8; ++q) {
#pragma unroll
                for (int b = 0; b < IB; ++b) {
                    const int pt = pt0 + b;
                    const cpx<R> z = v[b][q];
                    uint32_t a0, a1;
                    if constexpr (sizeof(R) == 4) {
                        if (PARTS == 2 && pt == 0) round_small_pair(z, a0, a1);
                        else round_wrap_pair(z, a0, a1);
                    } else {
                        a0 = trunc_div512(z.x);  // truncates like the reference (TorusPolynomial_fft.cpp:40)
                        a1 = trunc_div512(z.y);
                    }
                    if (PARTS == 1) {
                        c0[q] = a0;
                        c1[q] = a1;
                    } else if (pt == 0) {  // high part, scaled by 2^split
                        c0[q] = a0 << S.split;
                        c1[q] = a1 << S.split;
                    } else {
                        c0[q] += a0;
                        c1[q] += a1;
                    }
                }
            }
        }
        int32_t* dst = S.acc + j * kN;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int x0 = t + 64 * q;
            if (ROT) {
                dst[x0] = (int32_t)((uint32_t)dst[x0] + c0[q]);
                dst[x0 + kHalf] = (int32_t)((uint32_t)dst[x0 + kHalf] + c1[q]);
            } else {
                dst[x0] = (int32_t)c0[q];
                dst[x0 + kHalf] = (int32_t)c1[q];
            }
        }
    }
    group_sync(S.bar_id);
}

// Rounding of one transformed-back polynomial part into c0/c1 (the 16
// coefficients x0 = t + 64q and x0 + 512 of this thread): FP32 parts --
// the high part (pt = 0) rounded and shifted by the split, the low part
// (pt = 1) added; FP64 -- the reference's truncating conversion.
template <typename R, int PARTS>
__device__ __forceinline__ void round_part(const cpx<R> (&v)[8], int pt, int split, uint32_t (&c0)[8],
                                           uint32_t (&c1)[8]) {
    if constexpr (sizeof(R) == 4) {
        if (PARTS == 2 && pt == 0) {
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                uint32_t a0, a1;
                round_small_pair(v[q], a0, a1);
                c0[q] = a0 << split;
                c1[q] = a1 << split;
            }
        } else if (PARTS == 2) {
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                uint32_t a0, a1;
                round_wrap_pair(v[q], a0, a1);
                c0[q] += a0;
                c1[q] += a1;
            }
        } else {
#pragma unroll
            for (int q = 0; q < 8; ++q) round_wrap_pair(v[q], c0[q], c1[q]);
        }
    } else {
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            c0[q] = trunc_div512(v[q].x);
            c1[q] = trunc_div512(v[q].y);
        }
    }
}

// out[j][pt] into v, (j, pt) uniform at run time, indices compile-time so
// that out stays in registers.
template <typename R, int PARTS>
__device__ __forceinline__ void pick_part(cpx<R> (&v)[8], const cpx<R> (&out)[2][PARTS][8], int j, int pt) {
#pragma unroll
    for (int jj = 0; jj < 2; ++jj)
#pragma unroll
        for (int pp = 0; pp < PARTS; ++pp)
            if (jj == j && pp == pt) {
#pragma unroll
                for (int q = 0; q < 8; ++q) v[q] = out[jj][pp][q];
            }
}

// out[j][pt] += w, (j, pt) uniform at run time.
template <typename R, int PARTS>
__device__ __forceinline__ void add_part(cpx<R> (&out)[2][PARTS][8], const cpx<R> (&w)[8], int j, int pt) {
#pragma unroll
    for (int jj = 0; jj < 2; ++jj)
#pragma unroll
        for (int pp = 0; pp < PARTS; ++pp)
            if (jj == j && pp == pt) {
#pragma unroll
                for (int q = 0; q < 8; ++q) out[jj][pp][q] = cadd(out[jj][pp][q], w[q]);
            }
}

// The fused step of the shared-ring kernel, with one copy of each transform
// in the code: the levels and the (output, part) pairs are run-time loops
// (a fully unrolled step overflows the instruction cache).  In-place
// transforms, alternating the two exchange buffers.
template <typename R, int PARTS, int L, typename Keys>
__device__ __forceinline__ void ep_step_lean(const StepCtx<R, PARTS, 1>& S, Keys& keys, int a) {
    const int t = S.t;
    const int halfBg = 1 << (S.Bgbit - 1);
    const uint32_t mask = (1u << S.Bgbit) - 1;
    int which = 0;  // the exchange buffer of the next transform

    cpx<R> out[2][PARTS][8];
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int pt = 0; pt < PARTS; ++pt)
#pragma unroll
            for (int q = 0; q < 8; ++q) out[j][pt][q] = {(R)0, (R)0};

#pragma unroll 1
    for (int jp = 0; jp < 2; ++jp) {
        const int32_t* src = S.acc + jp * kN;
        uint32_t r0[8], r1[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const int x0 = t + 64 * r;
            r0[r] = (uint32_t)rot_coef(src, x0, a) - (uint32_t)src[x0] + S.offset;
            r1[r] = (uint32_t)rot_coef(src, x0 + kHalf, a) - (uint32_t)src[x0 + kHalf] + S.offset;
        }
#pragma unroll 1
        for (int lev = 0; lev < L; ++lev) {
            const int decal = 32 - (lev + 1) * S.Bgbit;
            cpx<R> v[8];
#pragma unroll
            for (int r = 0; r < 8; ++r)
                v[r] = digit_pair<R>(r0[r], r1[r], decal, mask, halfBg);
            fft512_forward_ip1(v, which ? S.s[0].b1 : S.s[0].b0, S.tw, S.ix, t, S.bar_id);
            which ^= 1;
            const int p = jp * L + lev;
            mac_row<R, PARTS, Keys::kShared>(out, v, keys.acquire(p), t);
            keys.release(p);
        }
    }

    uint32_t c0[8], c1[8];
#pragma unroll 1
    for (int u = 0; u < 2 * PARTS; ++u) {
        const int j = u / PARTS, pt = u % PARTS;
        cpx<R> v[8];
        pick_part<R, PARTS>(v, out, j, pt);
        fft512_inverse_ip1(v, which ? S.s[0].b1 : S.s[0].b0, S.tw, S.ix, t, S.bar_id);
        which ^= 1;
        round_part<R, PARTS>(v, pt, S.split, c0, c1);
        if (pt == PARTS - 1) {
            int32_t* dst = S.acc + j * kN;
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int x0 = t + 64 * q;
                dst[x0] = (int32_t)((uint32_t)dst[x0] + c0[q]);
                dst[x0 + kHalf] = (int32_t)((uint32_t)dst[x0 + kHalf] + c1[q]);
            }
        }
    }
    group_sync(S.bar_id);
}

// The low-latency kernels (spread, cluster) load the word that gives step
// i + 1's rotation during step i and convert it only at step i + 1: a
// conversion beside the load waits for L2 in every step (cluster kernel, one
// ciphertext: 1.291 ms with it there, 1.185 ms without).  The throughput
// kernels hide that wait and convert early (a ring wave with the late
// conversion: 6.50 against 6.41 ms).
struct KParams {
    int n, Bgbit, split;
    uint32_t offset;
};

template <typename R, int PARTS, int MODE, int GROUPS, int L>
__global__ void __launch_bounds__(64 * GROUPS, 1) k_external_product(KParams kp, Tables T, EpArgs a) {
    constexpr int NB = L > PARTS ? L : PARTS;
    using Ctx = StepCtx<R, PARTS, NB, ConvergedBarrier>;
    using Plan = SmemPlan<R, NB>;
    extern __shared__ __align__(128) char smem[];
    cpx<R>* tables = reinterpret_cast<cpx<R>*>(smem);
    load_hot_tables<R>(tables, T);
    __syncthreads();

    const int g = threadIdx.x >> 6;
    const int t = threadIdx.x & 63;
    // one-step products (FP64; the split-FP32 ones run on k_products_stream):
    // a persistent grid, neighbouring items on different SMs, so that every SM
    // has the same number of them (to one) whatever the count (1,024 FP64
    // products 465 -> 377 us, 64 of them 154 -> 90 us)
    const int c = MODE == kEpBlindRotate ? blockIdx.x * GROUPS + g : (int)(blockIdx.x + gridDim.x * g);
    if (c >= a.count) return;

    char* gbase = smem + Plan::tables + (size_t)g * Plan::group;
    Ctx S;
    S.tw = hot_twiddles<R>(tables);
    S.ix = make_fft_idx(t);
    S.acc = reinterpret_cast<int32_t*>(gbase);
#pragma unroll
    for (int b = 0; b < NB; ++b)
        S.s[b] = scratch_at<R>(gbase + Plan::acc + (size_t)b * 2 * kScratchStride * sizeof(cpx<R>));
    S.t = t;
    S.bar_id = {1 + g};
    S.Bgbit = kp.Bgbit;
    S.split = kp.split;
    S.offset = kp.offset;

    const size_t gsw_elems = (size_t)2 * L * 2 * PARTS * kHalf;
    const cpx<R>* gsw_base = reinterpret_cast<const cpx<R>*>(a.gsw);

    if (MODE == kEpBlindRotate) {
        const int n = kp.n;
        if (a.acc_in) {
            const int32_t* src = a.acc_in + (size_t)c * 2 * kN;
            for (int i = t; i < 2 * kN; i += 64) S.acc[i] = src[i];
        } else {
            // test vector mu * sum X^j rotated by X^{2N - barb}: the sign of
            // coefficient x is + when (x + barb) mod 2N < N
            const int32_t* xs = a.x + (size_t)c * (n + 1);
            const int barb = mod_switch_2n(xs[n]);
            for (int i = t; i < kN; i += 64) {
                S.acc[i] = 0;
                S.acc[kN + i] = test_vector_coef(a, c, barb, i);
            }
        }
        group_sync(S.bar_id);
        const int32_t* bara = a.bara ? a.bara + (size_t)c * n : nullptr;
        const int32_t* xs = a.x ? a.x + (size_t)c * (n + 1) : nullptr;
        // the rotation amount of step i + 1 is loaded during step i
        int a_next = bara ? bara[0] : mod_switch_2n(xs[0]);
#pragma unroll 1
        for (int i = 0; i < n; ++i) {
            const int ai = a_next;
            if (i + 1 < n) a_next = bara ? bara[i + 1] : mod_switch_2n(xs[i + 1]);
            if (ai == 0) continue;  // tfhe_blindRotate_FFT.cpp:114
            GlobalKeys<R, PARTS> keys{gsw_base + (size_t)i * gsw_elems};
            ep_step<R, PARTS, true, L, PARTS, NB>(S, keys, ai);
        }
        if (a.acc_out) {
            int32_t* dst = a.acc_out + (size_t)c * 2 * kN;
            for (int i = t; i < 2 * kN; i += 64) dst[i] = S.acc[i];
        }
        if (a.lwe_out) {
            // tLweExtractLweSample: a'_0 = a_0, a'_j = -a_{N-j}, b' = b_0
            int32_t* dst = a.lwe_out + (size_t)c * (kN + 1);
            for (int i = t; i < kN; i += 64)
                dst[i] = i == 0 ? S.acc[0] : (int32_t)(0u - (uint32_t)S.acc[kN - i]);
            if (t == 0) dst[kN] = S.acc[kN];
        }
    } else {
        const int stride = (int)gridDim.x * GROUPS;
        const char* gsw = reinterpret_cast<const char*>(a.gsw);
#pragma unroll 1
        for (int item = c; item < a.count; item += stride) {
            const int32_t* src = a.acc_in + (size_t)item * 2 * kN;
            for (int i = t; i < 2 * kN; i += 64) S.acc[i] = src[i];
            group_sync(S.bar_id);
            GlobalKeys<R, PARTS> keys{reinterpret_cast<const cpx<R>*>(gsw + a.gsw_stride * (size_t)item)};
            if (MODE == kEpPlain) {
                ep_step<R, PARTS, false, L, PARTS, NB>(S, keys, 0);
            } else {
                const int ai = a.bara[item];
                if (ai != 0) ep_step<R, PARTS, true, L, PARTS, NB>(S, keys, ai);
            }
            int32_t* dst = a.acc_out + (size_t)item * 2 * kN;
            for (int i = t; i < 2 * kN; i += 64) dst[i] = S.acc[i];
            group_sync(S.bar_id);  // the accumulator is free for the next item
        }
    }
}

// ----------------------------------------------------------------------
// One-step products (external product, MuxRotate) with one TGSW per item,
// split-FP32.  HBM bounds them (98,304 bytes of key for 16,384 of sample), so
// the point is to keep key rows in flight: a persistent grid of four groups
// of 64 threads per SM, each group streaming its own items' rows, 16 KB
// apiece, into two slots of its own by bulk copies that run on across items.
// A slot is refilled as soon as both warps of the group have used it, one
// block of transforms before it is needed.  Samples go straight between
// global memory and registers (the rotation is an index).  Neighbouring
// items go to different SMs, so every SM has the same number (to one)
// whatever the count.
// Measured against four groups per CTA in waves, with L1-prefetched row loads
// through registers: 34.1 -> 27.1 us for 1,024 products of the default set
// (4.3 TB/s), 83.4 -> 59.7 us for 3,000 (5.8 TB/s), 14.5 -> 10.4 us for 300.
// What is left at 1,024 is the last round of 2.7 groups per SM.
// A MuxRotate item with rotation 0 is a copy of its sample and streams no row
// (3,000 of them 54 -> 10.5 us; with all rows 96 KB each).
// The arithmetic is ep_step's, bit for bit.
// ----------------------------------------------------------------------
template <int L>
struct ProductPlan {
    static constexpr int kGroups = 4;
    static constexpr int S = ItemKeys<L, false>::S;
    static constexpr size_t kRowBytes = ItemKeys<L, false>::kRowBytes;
    static constexpr size_t ring_off = (kHotSize * sizeof(cpx<float>) + 127) & ~(size_t)127;
    static constexpr size_t x_off = ring_off + kGroups * S * kRowBytes;
    static constexpr size_t x_group = 4 * kScratchStride * sizeof(cpx<float>);  // two transforms, two buffers each
    static constexpr size_t bar_off = x_off + kGroups * x_group;
    static constexpr size_t flag_off = bar_off + kGroups * S * sizeof(uint64_t);
    static constexpr size_t total = flag_off + 16;
};

template <int NBK, int L, bool ROT>
__device__ __forceinline__ void product_levels(ItemKeys<L, ROT>& keys, cpx<float> (&out)[2][2][8], const uint32_t (&r0)[8],
                                               const uint32_t (&r1)[8], cpx<float>* x0, const FftTwiddles<float>& tw,
                                               const FftIdx& ix, int t, int bar_id, int Bgbit, int lev0) {
    const uint32_t mask = (1u << Bgbit) - 1;
    const int halfBg = 1 << (Bgbit - 1);
    cpx<float> v[NBK][8];
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int b = 0; b < NBK; ++b)
            v[b][r] = digit_pair<float>(r0[r], r1[r], 32 - (lev0 + b + 1) * Bgbit, mask, halfBg);
    cpx<float>* x[NBK];
#pragma unroll
    for (int b = 0; b < NBK; ++b) x[b] = x0 + b * kScratchStride;
    fft512_forward_ip<NBK>(v, x, tw, ix, t, bar_id);
#pragma unroll
    for (int b = 0; b < NBK; ++b) mac_row<float, 2, true>(out, v[b], keys.wait(keys.used + b), t);
    keys.release(NBK, bar_id);  // its barrier also frees the exchange buffers for the next transform
}

template <int MODE, int L>
__global__ void __launch_bounds__(64 * ProductPlan<L>::kGroups, 1)
    k_products_stream(KParams kp, Tables T, EpArgs a) {
    using Plan = ProductPlan<L>;
    constexpr bool ROT = MODE == kEpMuxRotate;
    extern __shared__ __align__(128) char smem[];
    cpx<float>* tables = reinterpret_cast<cpx<float>*>(smem);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + Plan::bar_off);
    volatile int* abort = reinterpret_cast<volatile int*>(smem + Plan::flag_off);
    if (threadIdx.x == 0) {
        for (int i = 0; i < Plan::kGroups * Plan::S; ++i) mbar_init(&full[i], 1);
        *abort = 0;
        fence_mbar_init();
    }
    __syncthreads();
    const int g = threadIdx.x >> 6, t = threadIdx.x & 63;
    const int stride = (int)gridDim.x * Plan::kGroups;
    const int first = (int)(blockIdx.x + gridDim.x * g);
    const int items = first < a.count ? (a.count - 1 - first) / stride + 1 : 0;
    ItemKeys<L, ROT> keys{reinterpret_cast<cpx<float>*>(smem + Plan::ring_off + g * Plan::S * Plan::kRowBytes),
                          full + g * Plan::S, a.err, abort,
                          reinterpret_cast<const char*>(a.gsw) + (size_t)first * a.gsw_stride,
                          (size_t)stride * a.gsw_stride, a.bara + first, stride, items, t, 0, 0, 0, 0, 0};
    int a_next = 0;
    if (ROT && items > 0) {
        // a rotated read waits for its rotation, so the sample travels before it is read
        a_next = a.bara[first];
        asm volatile("prefetch.global.L1 [%0];" ::"l"(a.acc_in + (size_t)first * 2 * kN + 32 * t));
    }
    if (t == 0) keys.start(a.stall_keys);  // the first rows travel while the tables load
    load_hot_tables<float>(tables, T);
    __syncthreads();
    if (items == 0) return;

    const FftTwiddles<float> tw = hot_twiddles<float>(tables);
    const FftIdx ix = make_fft_idx(t);
    const int bar_id = 1 + g;
    cpx<float>* x0 = reinterpret_cast<cpx<float>*>(smem + Plan::x_off + g * Plan::x_group);
#pragma unroll 1
    for (int it = 0; it < items; ++it) {
        const int item = first + it * stride;
        const int32_t* acc = a.acc_in + (size_t)item * 2 * kN;
        int32_t* res = a.acc_out + (size_t)item * 2 * kN;
        const int ai = a_next;
        if (it + 1 < items) {  // the next item's sample into L2, 128 bytes a thread
            asm volatile("prefetch.global.L2 [%0];" ::"l"(acc + (size_t)stride * 2 * kN + 32 * t));
            if (ROT) a_next = a.bara[item + stride];
        }
        if (ROT && ai == 0) {  // tfhe_blindRotate_FFT.cpp:114 -- the sample as it is, without its rows
            int32_t keep[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) keep[i] = acc[t + 64 * i];
#pragma unroll
            for (int i = 0; i < 32; ++i) res[t + 64 * i] = keep[i];
            continue;
        }
        cpx<float> out[2][2][8];
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int pt = 0; pt < 2; ++pt)
#pragma unroll
                for (int q = 0; q < 8; ++q) out[j][pt][q] = {0.f, 0.f};
#pragma unroll 1
        for (int jp = 0; jp < 2; ++jp) {
            const int32_t* src = acc + jp * kN;
            uint32_t r0[8], r1[8];
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                const int x = t + 64 * r;
                r0[r] = kp.offset + (ROT ? (uint32_t)rot_coef(src, x, ai) - (uint32_t)src[x] : (uint32_t)src[x]);
                r1[r] = kp.offset + (ROT ? (uint32_t)rot_coef(src, x + kHalf, ai) - (uint32_t)src[x + kHalf]
                                         : (uint32_t)src[x + kHalf]);
            }
            product_levels<2, L>(keys, out, r0, r1, x0, tw, ix, t, bar_id, kp.Bgbit, 0);
            if constexpr (L == 3) product_levels<1, L>(keys, out, r0, r1, x0, tw, ix, t, bar_id, kp.Bgbit, 2);
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            // the two outputs' transforms follow each other without a barrier: one buffer pair each
            cpx<float>* const x[2] = {x0 + 2 * j * kScratchStride, x0 + (2 * j + 1) * kScratchStride};
            fft512_inverse_ip<2>(out[j], x, tw, ix, t, bar_id);
            const int32_t* old = acc + j * kN;
            int32_t* dst = res + j * kN;
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                uint32_t h0, h1, l0, l1;
                round_small_pair(out[j][0][q], h0, h1);
                round_wrap_pair(out[j][1][q], l0, l1);
                const int x = t + 64 * q;
                dst[x] = (int32_t)((h0 << kp.split) + l0 + (ROT ? (uint32_t)old[x] : 0u));
                dst[x + kHalf] = (int32_t)((h1 << kp.split) + l1 + (ROT ? (uint32_t)old[x + kHalf] : 0u));
            }
        }
        group_sync(bar_id);  // the exchange buffers are free for the next item
    }
    if (t == 0) keys.drain();
}

// ----------------------------------------------------------------------
// Blind rotation with the bootstrapping key streamed through shared memory.
//
// A CTA runs GROUPS ciphertexts (64 threads each) plus one producer warp.
// Every ciphertext of the CTA walks the same key rows in the same order
// (row r = step i * 2l + p), so the producer streams each 16 KB row once per
// CTA with a bulk copy into a ring of S slots, and all groups read it from
// shared memory: one key read per CTA instead of one per ciphertext, and no
// L2 latency on the multiply-accumulate.  Slot hand-off uses two mbarriers
// per slot: full (the copy's byte count landed) and empty (every consumer
// thread has read the row).  A group that skips a step (a_i = 0) still waits
// and releases its rows, so the ring stays in step (RingKeys).  Every wait is
// bounded; a timeout sets *err (TFHE_GPU_TIMEOUT for the host) and the kernel
// runs to its end without further waiting on the ring.
// ----------------------------------------------------------------------
template <typename R, int PARTS, int GROUPS, int L, int S, int NB = 1>
struct RingPlan {
    static constexpr size_t kRowBytes = (size_t)2 * PARTS * kHalf * sizeof(cpx<R>);
    static constexpr size_t tables = kHotSize * sizeof(cpx<R>);
    static constexpr size_t ring_off = (tables + 127) & ~(size_t)127;
    static constexpr size_t bar_off = ring_off + S * kRowBytes;
    static constexpr size_t flag_off = bar_off + 2 * S * sizeof(uint64_t);
    static constexpr size_t group_off = (flag_off + sizeof(int) + 127) & ~(size_t)127;
    static constexpr size_t acc = 2 * kN * sizeof(int32_t);
    static constexpr size_t group = acc + NB * 2 * kScratchStride * sizeof(cpx<R>);
    static constexpr size_t total = group_off + GROUPS * group;
};

// NB = 1: one transform at a time (ep_step_lean).  NB = l > 1: the l forward
// and the PARTS inverse transforms of a step run together (ep_step), which
// needs NB exchange buffer pairs per group and about 250 registers, so at
// most four groups per CTA.
template <typename R, int PARTS, int GROUPS, int L, int S, bool INLINE, int NB = 1>
__global__ void __launch_bounds__(64 * GROUPS + (INLINE ? 0 : 32), 1)
    k_blind_rotate_ring(KParams kp, Tables T, EpArgs a) {
    using Plan = RingPlan<R, PARTS, GROUPS, L, S, NB>;
    constexpr int kpl = 2 * L;
    extern __shared__ __align__(128) char smem[];
    cpx<R>* tables = reinterpret_cast<cpx<R>*>(smem);
    cpx<R>* ring = reinterpret_cast<cpx<R>*>(smem + Plan::ring_off);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + Plan::bar_off);
    uint64_t* empty = full + S;
    volatile int* abort = reinterpret_cast<volatile int*>(smem + Plan::flag_off);
    const int active = min(GROUPS, a.count - (int)blockIdx.x * GROUPS);
    if (threadIdx.x == 0) {
        for (int i = 0; i < S; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 64 * active);
        }
        *abort = 0;
        fence_mbar_init();
    }
    load_hot_tables<R>(tables, T);
    __syncthreads();

    const int warp = threadIdx.x >> 5;
    const int n = kp.n;
    const uint32_t total_rows = (uint32_t)n * kpl;
    RingKeys<R, PARTS, S, !INLINE> keys{ring, full, empty, 0, a.err, abort, false,
                               reinterpret_cast<const char*>(a.gsw), total_rows, 0};
    if (!INLINE && warp == 2 * GROUPS) {
        // producer warp: one lane streams all n * 2l key rows in order
        if ((threadIdx.x & 31) == 0 && !a.stall_keys) {
            keys.issue_through(total_rows - 1);
            keys.drain();
        }
        return;
    }

    const int g = threadIdx.x >> 6;
    const int t = threadIdx.x & 63;
    const int c = blockIdx.x * GROUPS + g;
    if (g >= active) return;
    keys.producer = INLINE && threadIdx.x == 0 && !a.stall_keys;

    char* gbase = smem + Plan::group_off + (size_t)g * Plan::group;
    StepCtx<R, PARTS, NB> St;
    St.tw = hot_twiddles<R>(tables);
    St.ix = make_fft_idx(t);
    St.acc = reinterpret_cast<int32_t*>(gbase);
#pragma unroll
    for (int b = 0; b < NB; ++b)
        St.s[b] = scratch_at<R>(gbase + Plan::acc + (size_t)b * 2 * kScratchStride * sizeof(cpx<R>));
    St.t = t;
    St.bar_id = 1 + g;
    St.Bgbit = kp.Bgbit;
    St.split = kp.split;
    St.offset = kp.offset;

    if (a.acc_in) {
        const int32_t* src = a.acc_in + (size_t)c * 2 * kN;
        for (int i = t; i < 2 * kN; i += 64) St.acc[i] = src[i];
    } else {
        const int32_t* xs = a.x + (size_t)c * (n + 1);
        const int barb = mod_switch_2n(xs[n]);
        for (int i = t; i < kN; i += 64) {
            St.acc[i] = 0;
            St.acc[kN + i] = test_vector_coef(a, c, barb, i);
        }
    }
    group_sync(St.bar_id);
    const int32_t* bara = a.bara ? a.bara + (size_t)c * n : nullptr;
    const int32_t* xs = a.x ? a.x + (size_t)c * (n + 1) : nullptr;
    int a_next = bara ? bara[0] : mod_switch_2n(xs[0]);
#pragma unroll 1
    for (int i = 0; i < n; ++i) {
        const int ai = a_next;
        if (i + 1 < n) a_next = bara ? bara[i + 1] : mod_switch_2n(xs[i + 1]);
        keys.row0 = (uint32_t)i * kpl;
        if (ai == 0) {  // tfhe_blindRotate_FFT.cpp:114 -- rows still pass through
            for (int p = 0; p < kpl; ++p) {
                keys.acquire(p);
                keys.release(p);
            }
            continue;
        }
        if constexpr (NB == 1) ep_step_lean<R, PARTS, L>(St, keys, ai);
        else ep_step<R, PARTS, true, L, PARTS, NB>(St, keys, ai);
    }
    if (keys.producer) keys.drain();
    if (a.acc_out) {
        int32_t* dst = a.acc_out + (size_t)c * 2 * kN;
        for (int i = t; i < 2 * kN; i += 64) dst[i] = St.acc[i];
    }
    if (a.lwe_out) {
        int32_t* dst = a.lwe_out + (size_t)c * (kN + 1);
        for (int i = t; i < kN; i += 64)
            dst[i] = i == 0 ? St.acc[0] : (int32_t)(0u - (uint32_t)St.acc[kN - i]);
        if (t == 0) dst[kN] = St.acc[kN];
    }
}

// ----------------------------------------------------------------------
// The throughput kernel: the shared key ring with ciphertexts in lane pairs.
//
// A set of 128 threads runs two ciphertexts: lanes 2t' and 2t'+1 hold the
// same transform points of the two (fft512_forward_duo), so their twiddle and
// key-row loads share addresses within a lane pair and take half the
// shared-memory wavefronts.  FB levels are transformed together, then the
// remaining l % FB, and the two key parts of an output together.
//
// Accumulators of a set lie as [polynomial][x < 512][ct] pairs of words
// (coefficients x and x + 512): a thread's rotated read of a folded point is
// one 64-bit load, whose pair of words the rotation by a leaves together
// (swapped when (x - a) mod 1024 >= 512), and two ciphertexts with different
// a fall on different banks (even and odd 64-bit units).
//
// A step that neither ciphertext of a set takes (a_i = 0) only lets its rows
// pass (912 noiseless constants 6.23 -> 1.11 ms; l = 2 3.88 -> 0.60 ms).  With
// one a_i = 0 that ciphertext's half of the step runs as an exact no-op (every
// digit is 0), so the set's barrier and the ring stay in step.  In a set with
// one ciphertext left the other lane of each pair repeats it and stores
// nothing.
//
// What bounds it: the FP32 pipe and the register file's operand reads
// together with the latency of 12 warps per SM (FMA pipe 54 %, issue 55 %,
// shared-memory pipe 67 %).  Against one ciphertext per 64 threads, which was
// at 80 % of the shared-memory pipe (key rows and twiddles 1,130 of 2,750
// wavefronts per ciphertext and step): 6.41 -> 6.12 ms for 912 ciphertexts of
// the default set, 4.03 -> 3.84 ms for l = 2.  Eight per SM with transforms
// one at a time took 8.5 ms for 1,216; unrolling over the two input
// polynomials 10.5 ms (the code no longer fits the instruction cache).
// ----------------------------------------------------------------------
template <int SETS, int L, int S, int NB>
struct DuoPlan {
    static constexpr size_t kRowBytes = (size_t)2 * 2 * kHalf * sizeof(cpx<float>);
    static constexpr size_t ring_off = (kHotSize * sizeof(cpx<float>) + 127) & ~(size_t)127;
    static constexpr size_t bar_off = ring_off + S * kRowBytes;
    static constexpr size_t flag_off = bar_off + 2 * S * sizeof(uint64_t);
    static constexpr size_t set_off = (flag_off + sizeof(int) + 127) & ~(size_t)127;
    static constexpr size_t acc = 2 * 2 * kN * sizeof(int32_t);
    static constexpr size_t set = acc + NB * 2 * kDuoSlots * sizeof(cpx<float>);
    static constexpr size_t total = set_off + SETS * set;
};

// word of coefficient x of polynomial j of ciphertext ct of a set
__device__ __forceinline__ int duo_word(int j, int x, int ct) {
    return j * 2 * kN + (((x & (kHalf - 1)) << 1) + ct) * 2 + (x >> 9);
}

struct DuoCtx {
    TwTable<float> tw;
    DuoIdx ix;
    cpx<float>* s;  // exchange buffers, two per transform of a block
    int32_t* acc;
    int t, ct, bar_id;
    int Bgbit, split;
    uint32_t offset;
};

// out[j][pt] += v * key row, point by point so that the four products of one
// point come one after another: v[q] is then the same register operand of
// eight packed FMAs in a row.  A packed FMA with three different register
// pairs takes 3 clocks (operand reads), with one reused 2.1 to 2.4; this
// order is 0.11 ms of a 912-ciphertext wave.
__device__ __forceinline__ void duo_mac_row(cpx<float> (&out)[2][2][8], const cpx<float> (&v)[8],
                                            const cpx<float>* __restrict__ g, int t) {
    const float4* g4 = reinterpret_cast<const float4*>(g) + t;
#pragma unroll
    for (int qq = 0; qq < 4; ++qq) {
        float4 w[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) w[u] = g4[u * (kHalf / 2) + qq * 64];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int q = 2 * qq + e;
            float2 o[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                o[u] = __ffma2_rn(pk(v[q]), bc(e ? w[u].z : w[u].x), pk(out[u >> 1][u & 1][q]));
#pragma unroll
            for (int u = 0; u < 4; ++u)
                out[u >> 1][u & 1][q] = unpk(__ffma2_rn(times_i(v[q]), bc(e ? w[u].w : w[u].y), o[u]));
        }
    }
}

template <int NBK, typename Keys>
__device__ __forceinline__ void duo_levels(const DuoCtx& S, Keys& keys, cpx<float> (&out)[2][2][8],
                                           const uint32_t (&r0)[8], const uint32_t (&r1)[8], int p0, int lev0,
                                           int which) {
    const uint32_t mask = (1u << S.Bgbit) - 1;
    const int halfBg = 1 << (S.Bgbit - 1);
    bool landed[NBK];
#pragma unroll
    for (int b = 0; b < NBK; ++b) landed[b] = keys.poll(p0 + lev0 + b);
    cpx<float> v[NBK][8];
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int b = 0; b < NBK; ++b)
            v[b][r] = digit_pair<float>(r0[r], r1[r], 32 - (lev0 + b + 1) * S.Bgbit, mask, halfBg);
    cpx<float>* x[NBK];
#pragma unroll
    for (int b = 0; b < NBK; ++b) x[b] = S.s + (2 * b + which) * kDuoSlots;
    fft512_forward_duo<NBK>(v, x, S.tw, S.ix, S.bar_id);
#pragma unroll
    for (int b = 0; b < NBK; ++b) {
        const int p = p0 + lev0 + b;
        duo_mac_row(out, v[b], keys.acquire_polled(p, landed[b]), S.t);
        keys.release(p);
    }
}

template <int L, int FB, typename Keys>
__device__ __forceinline__ void duo_step(const DuoCtx& S, Keys& keys, int a) {
    const int t = S.t;
    cpx<float> out[2][2][8];
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int pt = 0; pt < 2; ++pt)
#pragma unroll
            for (int q = 0; q < 8; ++q) out[j][pt][q] = {0.f, 0.f};
    int which = 0;  // the exchange buffers of the next transforms (in-place form: alternating)

#pragma unroll 1
    for (int jp = 0; jp < 2; ++jp) {
        const int2* src = reinterpret_cast<const int2*>(S.acc + jp * 2 * kN) + S.ct;
        uint32_t r0[8], r1[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const int s = t + 64 * r - a;
            const int2 w = src[(s & (kHalf - 1)) * 2];
            const int2 p = src[(t + 64 * r) * 2];
            // coefficient x reads s mod 1024, negated when s mod 2048 >= 1024; x + 512 reads s + 512
            const uint32_t w0 = (uint32_t)(s & kHalf ? w.y : w.x), w1 = (uint32_t)(s & kHalf ? w.x : w.y);
            r0[r] = S.offset - (uint32_t)p.x + (s & kN ? 0u - w0 : w0);
            r1[r] = S.offset - (uint32_t)p.y + ((s + kHalf) & kN ? 0u - w1 : w1);
        }
#pragma unroll
        for (int lev0 = 0; lev0 + FB <= L; lev0 += FB) {
            duo_levels<FB>(S, keys, out, r0, r1, jp * L, lev0, which);
            which ^= 1;
        }
        if constexpr (L % FB != 0) {
            duo_levels<L % FB>(S, keys, out, r0, r1, jp * L, L - L % FB, which);
            which ^= 1;
        }
    }

#pragma unroll
    for (int j = 0; j < 2; ++j) {
        cpx<float>* const x[2] = {S.s + which * kDuoSlots, S.s + (2 + which) * kDuoSlots};
        fft512_inverse_duo<2>(out[j], x, S.tw, S.ix, S.bar_id);
        which ^= 1;
        int2* dst = reinterpret_cast<int2*>(S.acc + j * 2 * kN) + S.ct;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            uint32_t h0, h1, l0, l1;
            round_small_pair(out[j][0][q], h0, h1);
            round_wrap_pair(out[j][1][q], l0, l1);
            int2 w = dst[(t + 64 * q) * 2];
            w.x = (int32_t)((uint32_t)w.x + (h0 << S.split) + l0);
            w.y = (int32_t)((uint32_t)w.y + (h1 << S.split) + l1);
            dst[(t + 64 * q) * 2] = w;
        }
    }
    duo_sync(S.bar_id);
}

template <int SETS, int L, int S, int FB>
__global__ void __launch_bounds__(kDuoThreads * SETS, 1) k_blind_rotate_duo(KParams kp, Tables T, EpArgs a) {
    constexpr int NB = 2;
    static_assert(FB <= NB && FB <= L, "buffers for the forward block and both parts");
    using Plan = DuoPlan<SETS, L, S, NB>;
    constexpr int kpl = 2 * L;
    extern __shared__ __align__(128) char smem[];
    cpx<float>* tables = reinterpret_cast<cpx<float>*>(smem);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + Plan::bar_off);
    uint64_t* empty = full + S;
    volatile int* abort = reinterpret_cast<volatile int*>(smem + Plan::flag_off);
    const int left = a.count - (int)blockIdx.x * 2 * SETS;  // ciphertexts from this CTA on
    const int active = min(SETS, (left + 1) >> 1);
    if (threadIdx.x == 0) {
        for (int i = 0; i < S; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 4 * active);  // one release per consumer warp
        }
        *abort = 0;
        fence_mbar_init();
    }
    load_hot_tables<float>(tables, T);
    __syncthreads();

    const int set = threadIdx.x >> 7;
    if (set >= active) return;
    const int ct = threadIdx.x & 1, t = (threadIdx.x & 127) >> 1;
    const bool live = 2 * set + ct < left;
    const int c = blockIdx.x * 2 * SETS + 2 * set + (live ? ct : 0);
    const int n = kp.n;
    PolledRingKeys<float, 2, S> keys{{reinterpret_cast<cpx<float>*>(smem + Plan::ring_off), full, empty, 0, a.err, abort,
                                      threadIdx.x == 0 && !a.stall_keys, reinterpret_cast<const char*>(a.gsw),
                                      (uint32_t)n * kpl, 0}};
    char* sbase = smem + Plan::set_off + (size_t)set * Plan::set;
    const DuoCtx St{TwTable<float>(hot_twiddles<float>(tables), t), make_duo_idx(t, ct),
                    reinterpret_cast<cpx<float>*>(sbase + Plan::acc), reinterpret_cast<int32_t*>(sbase), t, ct, 1 + set,
                    kp.Bgbit, kp.split, kp.offset};

    if (a.acc_in) {
        const int32_t* src = a.acc_in + (size_t)c * 2 * kN;
        for (int i = t; i < 2 * kN; i += 64) St.acc[duo_word(i >> 10, i & (kN - 1), ct)] = src[i];
    } else {
        const int barb = mod_switch_2n(a.x[(size_t)c * (n + 1) + n]);
        for (int i = t; i < kN; i += 64) {
            St.acc[duo_word(0, i, ct)] = 0;
            St.acc[duo_word(1, i, ct)] = test_vector_coef(a, c, barb, i);
        }
    }
    duo_sync(St.bar_id);
    const int32_t* bara = a.bara ? a.bara + (size_t)c * n : nullptr;
    const int32_t* xs = a.x ? a.x + (size_t)c * (n + 1) : nullptr;
    int a_next = bara ? bara[0] : mod_switch_2n(xs[0]);
#pragma unroll 1
    for (int i = 0; i < n; ++i) {
        const int ai = a_next;
        if (i + 1 < n) a_next = bara ? bara[i + 1] : mod_switch_2n(xs[i + 1]);
        keys.row0 = (uint32_t)i * kpl;
        if (__any_sync(0xffffffffu, ai != 0)) {
            duo_step<L, FB>(St, keys, ai);
        } else {  // tfhe_blindRotate_FFT.cpp:114, the same for the set
#pragma unroll
            for (int p = 0; p < kpl; ++p) {
                keys.acquire_polled(p, false);
                keys.release(p);
            }
        }
    }
    if (keys.producer) keys.drain();
    if (!live) return;
    if (a.acc_out) {
        int32_t* dst = a.acc_out + (size_t)c * 2 * kN;
        for (int i = t; i < 2 * kN; i += 64) dst[i] = St.acc[duo_word(i >> 10, i & (kN - 1), ct)];
    }
    if (a.lwe_out) {
        // tLweExtractLweSample: a'_0 = a_0, a'_j = -a_{N-j}, b' = b_0
        int32_t* dst = a.lwe_out + (size_t)c * (kN + 1);
        for (int i = t; i < kN; i += 64)
            dst[i] = i == 0 ? St.acc[duo_word(0, 0, ct)] : (int32_t)(0u - (uint32_t)St.acc[duo_word(0, kN - i, ct)]);
        if (t == 0) dst[kN] = St.acc[duo_word(1, 0, ct)];
    }
}

// ----------------------------------------------------------------------
// Blind rotation with one ciphertext per CTA (low latency, up to one per SM).
// Split-FP32 only.
//
// l sets of 128 threads run transforms in lane pairs (fft512_forward_duo):
// the two lanes of a pair hold the same point of two transforms and share
// addresses of the accumulator and the digits.  Set j < 2 decomposes
// polynomial j and transforms its levels 0 and 1, set 2 (l = 3) level 2 of
// both polynomials; each writes its transformed digits D to shared memory.
// After a barrier, sets 0 and 1 own the output polynomials: lane pair t
// multiplies all 2l rows in row order, the high key part in the even lane and
// the low part in the odd one, which read the same D, transforms both back
// and rounds.  The lanes then exchange halves, so that the even one has the
// whole sum of coefficients t + 64q and the odd one that of the 512 above,
// kept in registers and written out for the next step's rotation.  A producer
// warp copies each step's key rows into shared memory (one 4 KB part of a row
// a lane) as soon as the owners have used the last step's.  The products are
// summed in the same order as in every other shape, so the ciphertexts are
// the same bit for bit; with PAIR, in the pair kernel's order: the rows of
// each input polynomial on their own, then the two sums (for the batch sizes
// that shape 0 has always run in that order).
//
// What bounds it: the shared-memory pipe (about 3,600 wavefronts of a step's
// 5,150 clocks: the key values written and read 1,536, the transforms'
// exchanges 1,280, the digits 580, the accumulator) and the chain of a step's phases.
// Measured against the form with one transform per 64 threads, the high and
// the low part in different groups, keys loaded into registers (the loads
// held the load/store unit for 600 clocks a step) and accumulated by
// shared-memory atomics: 1.755 -> 1.570 ms for 152 ciphertexts; the twiddles
// in registers instead of shared memory are 0.054 ms of that.
// ----------------------------------------------------------------------
template <int L>
struct SpreadPlan {
    static_assert(L == 2 || L == 3, "levels 0, 1 in lane pairs, level 2 apart");
    static constexpr int kSets = L;
    static constexpr int kThreads = kDuoThreads * kSets + 32;  // and the producer warp
    // a step's key values, [row][polynomial][part], each part 64 bytes round
    // so that the two lanes of a pair fall on different banks
    static constexpr int kKeyPart = kHalf * sizeof(cpx<float>) + 64;
    static constexpr int kKeyParts = 2 * L * 2 * 2;
    static constexpr int kDA = 2 * kHalf;               // digits of levels 0, 1 of a polynomial: [q][t][level]
    static constexpr int kDB = L == 3 ? kHalf + 8 : 0;  // of level 2: [q][t], the next polynomial's 64 bytes round
    static constexpr int kD = kDA + kDB;
    static constexpr size_t acc_off = kHotSize * sizeof(cpx<float>);
    // the accumulator's words, see spread_put: from one pair to the next, from
    // one polynomial to the other
    static constexpr int kAccPair = L == 2 ? 2 : 4;
    static constexpr int kAccPoly = L == 2 ? 2 * kN : 2;
    static constexpr size_t d_off = acc_off + 2 * 2 * kN * sizeof(int32_t);
    static constexpr size_t x_off = d_off + 2 * kD * sizeof(cpx<float>);
    static constexpr size_t key_off = x_off + kSets * kDuoSlots * sizeof(cpx<float>);
    static constexpr size_t bar_off = key_off + (size_t)kKeyParts * kKeyPart;  // 2 mbarriers, abort flag
    static constexpr size_t total = bar_off + 2 * sizeof(uint64_t) + 16;
    static_assert(d_off % 16 == 0 && kD * sizeof(cpx<float>) % 16 == 0, "16-byte digit loads");
    static_assert(key_off % 16 == 0 && kKeyParts <= 32, "bulk copies, one a lane");
};

// The accumulator in shared memory: for every s in [0, N) the pair (c(s),
// c(s + N/2)) of both polynomials, c the coefficients continued by X^N = -1,
// so that a rotation reads a folded point with one 64-bit load and needs only
// a sign.  With A and B the coefficients u and u + 512 (u < 512), s = u holds
// (A, B) and s = u + 512 holds (B, -A).
//
// For l = 2 every set reads one polynomial, whose pairs lie one after the
// other: the 16 points that a warp's lane pairs read, or write as 32 words, are
// one wavefront.  With the pairs of both polynomials side by side they are
// two (256 wavefronts of a step more): 1.079 -> 1.000 ms for 152 ciphertexts,
// 2.078 -> 2.033 ms for 304.  For l = 3, whose third set reads both polynomials
// at once, the side by side form is the faster one although it has those
// wavefronts: 1.574 against 1.598 ms for 152 ciphertexts, 3.05 against 3.20 ms
// for 304.  (The addresses are written out per form: one expression for both
// cost l = 2 0.028 ms, and l = 3 0.02 ms the other way round.)
template <int L>
__device__ __forceinline__ int spread_word(int j, int x) {  // of coefficient x < N
    return L == 2 ? j * SpreadPlan<L>::kAccPoly + (x & (kHalf - 1)) * SpreadPlan<L>::kAccPair + (x >> 9)
                  : ((x & (kHalf - 1)) * 2 + j) * 2 + (x >> 9);
}
template <int L>
__device__ __forceinline__ void spread_put(int32_t* acc, int j, int x, uint32_t v) {
    const int half = x >> 9;
    int32_t* w = L == 2 ? acc + j * SpreadPlan<L>::kAccPoly + (x & (kHalf - 1)) * SpreadPlan<L>::kAccPair
                        : acc + ((x & (kHalf - 1)) * 2 + j) * 2;
    w[half] = (int32_t)v;
    w[kHalf * SpreadPlan<L>::kAccPair + 1 - half] = (int32_t)(half ? v : 0u - v);
}
// X^a - 1 applied to the folded point t + 64r of polynomial j, plus the
// gadget offset: r0 for coefficient t + 64r, r1 for that + 512.
template <int L>
__device__ __forceinline__ void rotated_pair(const int32_t* acc, int j, int t, int r, int a, uint32_t offset,
                                             uint32_t& r0, uint32_t& r1) {
    constexpr int kStep = SpreadPlan<L>::kAccPair / 2;
    const int2* src = L == 2 ? reinterpret_cast<const int2*>(acc + j * SpreadPlan<L>::kAccPoly)
                             : reinterpret_cast<const int2*>(acc) + j;
    const int s = t + 64 * r - a;
    const int2 w = src[(s & (kN - 1)) * kStep];
    const int2 p = src[(t + 64 * r) * kStep];
    const uint32_t m = (uint32_t)((s << 21) >> 31);  // all ones when s mod 2N >= N
    r0 = ((uint32_t)w.x ^ m) - (uint32_t)p.x + (offset - m);
    r1 = ((uint32_t)w.y ^ m) - (uint32_t)p.y + (offset - m);
}

// The producer warp of k_blind_rotate_spread: the key values of every step that
// the ciphertext takes, into the one buffer, as soon as the owners have used
// the last step's.  Owners that have given up on a step free its values too, so
// the producer waits for the last copy itself before it fills the buffer again.
// EARLY arms the barrier and prefetches before the owners are done: 263
// ciphertexts in the pair kernel's order with l = 3 3.06 -> 3.04 ms; in the other
// forms it is slower (152 ciphertexts 1.560 -> 1.583 ms).
template <int L, bool EARLY>
__device__ __forceinline__ void spread_stream(const EpArgs& a, char* smem, uint64_t* kfull, uint64_t* kfree,
                                              volatile int* abort, int n, int c) {
    using Plan = SpreadPlan<L>;
    constexpr int kRows = 2 * L;
    constexpr size_t kStep = (size_t)Plan::kKeyParts * kHalf, kRow = kStep / kRows;  // complex values
    constexpr uint32_t kStepBytes = kStep * sizeof(cpx<float>), kRowBytes = kStepBytes / kRows;
    const int u = threadIdx.x & 31;
    const cpx<float>* gsw = reinterpret_cast<const cpx<float>*>(a.gsw);
    const cpx<float>* src = gsw + (size_t)u * kHalf;  // parts lie in order, row by row
    const auto prefetch = [&](int i) {  // rows into L2 two steps ahead of their copies
        if (i + 2 < n && u < kRows) bulk_prefetch_l2(gsw + (size_t)(i + 2) * kStep + (size_t)u * kRow, kRowBytes);
    };
    // 32 steps' rotations, one a lane, loaded 32 steps ahead: a step with
    // a_i = 0 is not taken and has no copy (152 noiseless constants 575 -> 55 us)
    const auto moves = [&](int i) {
        return i < n && (a.bara ? a.bara[(size_t)c * n + i] : mod_switch_2n(a.x[(size_t)c * (n + 1) + i])) != 0;
    };
    uint32_t k = 0;  // steps copied
    bool go = true, next = moves(u);
#pragma unroll 1
    for (int i0 = 0; i0 < n && go; i0 += 32) {
        uint32_t todo = __ballot_sync(0xffffffffu, next);
        next = moves(i0 + 32 + u);
#pragma unroll 1
        for (; todo; todo &= todo - 1) {
            const int i = i0 + __ffs((int)todo) - 1;
            if (EARLY) prefetch(i);
            go = k == 0 || mbar_wait_bounded(kfull, (k - 1) & 1, abort);
            if (EARLY) {
                go = __all_sync(0xffffffffu, go);
                if (u == 0 && go) mbar_arrive_expect_tx(kfull, kStepBytes);
            }
            go = go && (k == 0 || mbar_wait_bounded(kfree, (k - 1) & 1, abort));
            go = __all_sync(0xffffffffu, go);
            if (!go) {
                *abort = 1;
                atomicExch(a.err, 3);
                break;
            }
            if (!EARLY) {
                if (u == 0) mbar_arrive_expect_tx(kfull, kStepBytes);
                __syncwarp();
            }
            if (u < Plan::kKeyParts && !a.stall_keys)
                bulk_copy_g2s(smem + Plan::key_off + (size_t)u * Plan::kKeyPart, src + (size_t)i * kStep,
                              (uint32_t)(kHalf * sizeof(cpx<float>)), kfull);
            if (!EARLY) prefetch(i);
            ++k;
        }
    }
    // no copy in flight at the end of the kernel
    if (k > 0 && !mbar_wait_bounded(kfull, (k - 1) & 1)) atomicExch(a.err, 3);
    __syncwarp();
}

template <int L, bool PAIR>
__global__ void __launch_bounds__(SpreadPlan<L>::kThreads, 1) k_blind_rotate_spread(KParams kp, Tables T, EpArgs a) {
    using Plan = SpreadPlan<L>;
    extern __shared__ __align__(128) char smem[];
    cpx<float>* tables = reinterpret_cast<cpx<float>*>(smem);
    int32_t* acc = reinterpret_cast<int32_t*>(smem + Plan::acc_off);
    cpx<float>* dsh = reinterpret_cast<cpx<float>*>(smem + Plan::d_off);
    uint64_t* kfull = reinterpret_cast<uint64_t*>(smem + Plan::bar_off);  // the step's key values landed
    uint64_t* kfree = kfull + 1;                                          // every owner warp has used them
    volatile int* abort = reinterpret_cast<volatile int*>(kfull + 2);
    const int c = blockIdx.x;
    const int set = threadIdx.x >> 7, e = threadIdx.x & 1, t = (threadIdx.x & 127) >> 1;
    const bool owner = set < 2;          // also the sets with levels 0 and 1 of one polynomial
    const int jp = owner ? set : e;      // polynomial this lane decomposes
    const int lev = owner ? e : 2;       // at this level; owners: output polynomial `set`, key part e
    const int n = kp.n;
    load_hot_tables<float>(tables, T);
    if (a.acc_in) {
        const int32_t* src = a.acc_in + (size_t)c * 2 * kN;
        for (int i = threadIdx.x; i < 2 * kN; i += blockDim.x)
            spread_put<L>(acc, i >> 10, i & (kN - 1), (uint32_t)src[i]);
    } else {
        const int32_t* xs = a.x + (size_t)c * (n + 1);
        const int barb = mod_switch_2n(xs[n]);
        for (int i = threadIdx.x; i < kN; i += blockDim.x) {
            spread_put<L>(acc, 0, i, 0u);
            spread_put<L>(acc, 1, i, (uint32_t)test_vector_coef(a, c, barb, i));
        }
    }
    if (threadIdx.x == 0) {
        mbar_init(kfull, 1);
        mbar_init(kfree, 8);  // owner warps
        *abort = 0;
        fence_mbar_init();
    }
    __syncthreads();

    const auto gave_up = [&]() {
        *abort = 1;
        atomicExch(a.err, 3);
    };
    if (set != Plan::kSets) {
        // barrier of all sets (the producer warp takes no part)
        const auto step_sync = []() {
            asm volatile("barrier.sync 15, %0;" ::"n"(kDuoThreads * Plan::kSets) : "memory");
        };
        const TwRegs<float> tw(hot_twiddles<float>(tables), t);
        const DuoIdx ix = make_duo_idx(t, e);
        cpx<float>* const xbuf[1] = {reinterpret_cast<cpx<float>*>(smem + Plan::x_off) + set * kDuoSlots};
        const int bar_id = 1 + set;
        const int halfBg = 1 << (kp.Bgbit - 1);
        const uint32_t mask = (1u << kp.Bgbit) - 1;
        const int decal = 32 - (lev + 1) * kp.Bgbit;
        const int out_shift = e == 0 ? kp.split : 0;  // the high part counts 2^split
        const float4* keys =
            reinterpret_cast<const float4*>(smem + Plan::key_off + (size_t)(2 * set + e) * Plan::kKeyPart) + t;
        uint32_t own[8] = {};  // owners: coefficients t + 64q (even lane) or 512 above (odd) of the output polynomial
        if (owner) {
#pragma unroll
            for (int q = 0; q < 8; ++q) own[q] = (uint32_t)acc[spread_word<L>(set, t + 64 * q + e * kHalf)];
        }
        const int32_t* bara = a.bara ? a.bara + (size_t)c * n : nullptr;
        const int32_t* xs = a.x ? a.x + (size_t)c * (n + 1) : nullptr;
        const int32_t* rot = bara ? bara : xs;
        int32_t rot_next = rot[0];
        uint32_t k = 0;  // parity of the steps taken, as the producer counts them
#pragma unroll 1
        for (int i = 0; i < n; ++i) {
            const int ai = bara ? rot_next : mod_switch_2n(rot_next);
            if (i + 1 < n) rot_next = rot[i + 1];
            if (ai == 0) continue;  // tfhe_blindRotate_FFT.cpp:114 (uniform over the CTA)
            cpx<float> v[1][8];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                uint32_t u0, u1;
                rotated_pair<L>(acc, jp, t, q, ai, kp.offset, u0, u1);
                v[0][q] = digit_pair<float>(u0, u1, decal, mask, halfBg);
            }
            fft512_forward_duo<1>(v, xbuf, tw, ix, bar_id);
            {
                const int d0 = owner ? jp * Plan::kD + 2 * t + e : jp * Plan::kD + Plan::kDA + t;
                const int dq = owner ? 128 : 64;
#pragma unroll
                for (int q = 0; q < 8; ++q) dsh[d0 + dq * q] = v[0][q];
            }
            step_sync();  // every D in place; every read of acc done
            if (owner) {
                if (!mbar_wait_bounded(kfull, k, abort)) gave_up();
                __syncwarp();
                cpx<float> o[1][8];
#pragma unroll
                for (int q = 0; q < 8; ++q) o[0][q] = {0.f, 0.f};
                cpx<float> other[8];  // PAIR: the rows of the other input polynomial apart
#pragma unroll
                for (int q = 0; q < 8; ++q) other[q] = {0.f, 0.f};
#pragma unroll
                for (int qq = 0; qq < 4; ++qq) {
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        float4 w[L];
#pragma unroll
                        for (int lv = 0; lv < L; ++lv)
                            w[lv] = keys[(j * L + lv) * 4 * (Plan::kKeyPart / 16) + qq * 64];
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const int q = 2 * qq + h;
                            const cpx<float>* D = dsh + j * Plan::kD;
                            const float4 da = reinterpret_cast<const float4*>(D)[q * 64 + t];
                            cpx<float>& z = PAIR && j == 1 ? other[q] : o[0][q];
                            z = cmac(z, cpx<float>{da.x, da.y},
                                     h ? cpx<float>{w[0].z, w[0].w} : cpx<float>{w[0].x, w[0].y});
                            z = cmac(z, cpx<float>{da.z, da.w},
                                     h ? cpx<float>{w[1].z, w[1].w} : cpx<float>{w[1].x, w[1].y});
                            if constexpr (L == 3)
                                z = cmac(z, D[Plan::kDA + q * 64 + t],
                                         h ? cpx<float>{w[2].z, w[2].w} : cpx<float>{w[2].x, w[2].y});
                        }
                    }
                    if constexpr (PAIR) {
                        o[0][2 * qq] = cadd(o[0][2 * qq], other[2 * qq]);
                        o[0][2 * qq + 1] = cadd(o[0][2 * qq + 1], other[2 * qq + 1]);
                    }
                }
                __syncwarp();
                if ((threadIdx.x & 31) == 0) mbar_arrive(kfree);
                fft512_inverse_duo<1>(o, xbuf, tw, ix, bar_id);
                // both parts through the wide rounding: for the high part (below
                // 2^22) it gives round_small_pair's integer, and the lanes stay together
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    uint32_t c0, c1;
                    round_wrap_pair(o[0][q], c0, c1);
                    c0 <<= out_shift;
                    c1 <<= out_shift;
                    const uint32_t other = __shfl_xor_sync(0xffffffffu, e ? c0 : c1, 1);
                    own[q] += (e ? c1 : c0) + other;
                    spread_put<L>(acc, set, t + 64 * q + e * kHalf, own[q]);
                }
            }
            k ^= 1;
            step_sync();  // the accumulator is updated before the next step reads it
        }
    } else {
        spread_stream<L, (L == 3 && PAIR)>(a, smem, kfull, kfree, abort, n, c);
    }
    __syncthreads();
    if (a.acc_out) {
        int32_t* dst = a.acc_out + (size_t)c * 2 * kN;
        for (int i = threadIdx.x; i < 2 * kN; i += blockDim.x) dst[i] = acc[spread_word<L>(i >> 10, i & (kN - 1))];
    }
    if (a.lwe_out) {
        // tLweExtractLweSample: a'_0 = a_0, a'_j = -a_{N-j}, b' = b_0
        int32_t* dst = a.lwe_out + (size_t)c * (kN + 1);
        for (int i = threadIdx.x; i < kN; i += blockDim.x)
            dst[i] = i == 0 ? acc[spread_word<L>(0, 0)] : (int32_t)(0u - (uint32_t)acc[spread_word<L>(0, kN - i)]);
        if (threadIdx.x == 0) dst[kN] = acc[spread_word<L>(1, 0)];
    }
}

// ----------------------------------------------------------------------
// Blind rotation with one ciphertext over a cluster of two CTAs (two SMs).
//
// The work of a step split across two SMs: CTA r of the cluster holds
// accumulator polynomial r, runs the l forward transforms of polynomial r
// (one per group) and owns output polynomial r (groups 0 and 1: the high and
// the low key part).  Each group writes its transformed digits D_(r,lev) to
// its own shared memory and pushes them into the peer CTA's (distributed
// shared memory); once the peer's digits have landed the owners multiply all 2l rows
// -- l local, l from the peer -- in row order with their part of each key
// row, transform back, round and add into the local accumulator with
// integer atomics.  The accumulator never crosses SMs, only 4 KB of digits
// per group and step do.
//
// The pushes are asynchronous stores (st.async) that count their bytes on
// the receiving CTA's mbarrier for that step: the owners wait (bounded) for
// the peer's l x 4 KB to land, with no cluster-wide barrier and no release
// fence on the sender.  Pushes alternate between two buffers, each with its
// own mbarrier.  A push into buffer b at step k cannot overtake the peer's
// reads of b at step k - 2: the pushing CTA has by then received the peer's
// step k - 1 digits, which the peer sends only after its step k - 2
// products.  The products are summed in the same order as every other
// shape, so the ciphertexts are bit-identical to the spread kernel's (and with
// PAIR in the pair kernel's order, as there).
// Split-FP32 only, 1 CTA per SM (the shared-memory request is padded so
// that the two CTAs take two SMs).
// ----------------------------------------------------------------------
template <int L>
struct Spread2Plan {
    static constexpr size_t tables = kHotSize * sizeof(cpx<float>);
    static constexpr size_t acc_off = tables;                                     // own polynomial
    static constexpr size_t dloc_off = acc_off + kN * sizeof(int32_t);           // [lev][q][t]
    static constexpr size_t drem_off = dloc_off + L * kHalf * sizeof(cpx<float>);  // [buf][lev][q][t]
    static constexpr size_t scratch_off = drem_off + 2 * L * kHalf * sizeof(cpx<float>);
    static constexpr size_t scratch = 2 * kScratchStride * sizeof(cpx<float>);
    static constexpr size_t bar_off = scratch_off + L * scratch;  // 2 mbarriers, abort flag
    static constexpr size_t total = bar_off + 2 * sizeof(uint64_t) + 16;
    static constexpr size_t request = total > 120 * 1024 ? total : 120 * 1024;  // one CTA per SM
};

template <int L, bool PAIR>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(64 * L, 1)
    k_blind_rotate_spread2(KParams kp, Tables T, EpArgs a) {
    static_assert(L >= 2, "two owner groups per CTA");
    namespace cg = cooperative_groups;
    using Plan = Spread2Plan<L>;
    constexpr int kRows = 2 * L;
    constexpr int kRowElems = 2 * 2 * kHalf;  // complex values per key row
    extern __shared__ __align__(128) char smem[];
    cg::cluster_group cluster = cg::this_cluster();
    const int r = (int)cluster.block_rank();  // this CTA's polynomial
    cpx<float>* tables = reinterpret_cast<cpx<float>*>(smem);
    int32_t* acc = reinterpret_cast<int32_t*>(smem + Plan::acc_off);
    cpx<float>* dloc = reinterpret_cast<cpx<float>*>(smem + Plan::dloc_off);
    cpx<float>* drem = reinterpret_cast<cpx<float>*>(smem + Plan::drem_off);
    uint64_t* dbar = reinterpret_cast<uint64_t*>(smem + Plan::bar_off);  // per buffer
    volatile int* abort = reinterpret_cast<volatile int*>(smem + Plan::bar_off + 2 * sizeof(uint64_t));
    // the peer's digit buffers and their mbarriers, as shared::cluster addresses
    const uint32_t drem_peer = cluster_map(smem_u32(drem), (uint32_t)(r ^ 1));
    const uint32_t dbar_peer = cluster_map(smem_u32(dbar), (uint32_t)(r ^ 1));
    const int c = blockIdx.x >> 1;
    const int g = threadIdx.x >> 6, t = threadIdx.x & 63;
    const int lev = g;
    const bool owner = g < 2;
    const int opt = g & 1;
    const int n = kp.n;
    load_hot_tables<float>(tables, T);
    if (a.acc_in) {
        const int32_t* src = a.acc_in + (size_t)c * 2 * kN + (size_t)r * kN;
        for (int i = threadIdx.x; i < kN; i += blockDim.x) acc[i] = src[i];
    } else {
        const int32_t* xs = a.x + (size_t)c * (n + 1);
        const int barb = mod_switch_2n(xs[n]);
        for (int i = threadIdx.x; i < kN; i += blockDim.x) acc[i] = r == 0 ? 0 : test_vector_coef(a, c, barb, i);
    }
    if (threadIdx.x == 0) {
        mbar_init(&dbar[0], 1);
        mbar_init(&dbar[1], 1);
        *abort = 0;
        fence_mbar_init();
    }
    cluster.sync();  // both CTAs' barriers initialised before any push

    const FftTwiddles<float> tw = hot_twiddles<float>(tables);
    const FftIdx ix = make_fft_idx(t);
    const FftScratch<float> sc = scratch_at<float>(smem + Plan::scratch_off + (size_t)g * Plan::scratch);
    const int bar_id = 1 + g;
    const int halfBg = 1 << (kp.Bgbit - 1);
    const uint32_t mask = (1u << kp.Bgbit) - 1;
    const int decal = 32 - (lev + 1) * kp.Bgbit;
    const cpx<float>* gsw = reinterpret_cast<const cpx<float>*>(a.gsw);
    const size_t step_elems = (size_t)kRows * kRowElems;
    const int32_t* bara = a.bara ? a.bara + (size_t)c * n : nullptr;
    const int32_t* xs = a.x ? a.x + (size_t)c * (n + 1) : nullptr;
    const int32_t* rot = bara ? bara : xs;
    int32_t rot_next = rot[0];
    // side jobs of the last warp, done once its group's digits are out: with
    // l = 3 that group owns no output (they cost a warp 230 clocks a step)
    const int side = (int)threadIdx.x - (64 * L - 32);
    // Key rows go into L2 eight steps (14 us) ahead.  A gate's key switch
    // streams its table between two blind rotations, so the bootstrapping key
    // comes from HBM again: after a key switch 1,179 -> 1,170 us for one
    // ciphertext and 1,160 -> 1,153 us for 64 against two steps ahead (four:
    // no gain; sixteen: slower).
    constexpr int kAhead = 8;
    const auto prefetch_rows = [&](int step) {
        if (step < n && side >= 0 && side < kRows && (side & 1) == r)
            bulk_prefetch_l2(gsw + (size_t)step * step_elems + (size_t)side * kRowElems,
                             kRowElems * sizeof(cpx<float>));
    };
    // a step's incoming digits: one arrival and l x 4 KB of stores
    const auto expect_digits = [&](int b) {
        if (side == 0) mbar_arrive_expect_tx(&dbar[b], (uint32_t)(L * kHalf * sizeof(cpx<float>)));
    };
    for (int s = 0; s < kAhead; ++s) prefetch_rows(s);
    expect_digits(0);
    uint32_t k = 0;  // steps taken (the same in both CTAs)
#pragma unroll 1
    for (int i = 0; i < n; ++i) {
        const int ai = bara ? rot_next : mod_switch_2n(rot_next);
        if (i + 1 < n) rot_next = rot[i + 1];
        if (ai == 0) continue;  // tfhe_blindRotate_FFT.cpp:114 (uniform over the cluster)
        const int buf = (int)(k & 1);
        const cpx<float>* step_keys = gsw + (size_t)i * step_elems;
        cpx<float> v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int x0 = t + 64 * q;
            const uint32_t u0 = (uint32_t)rot_coef(acc, x0, ai) - (uint32_t)acc[x0] + kp.offset;
            const uint32_t u1 = (uint32_t)rot_coef(acc, x0 + kHalf, ai) - (uint32_t)acc[x0 + kHalf] + kp.offset;
            v[q] = digit_pair<float>(u0, u1, decal, mask, halfBg);
        }
        fft512_forward_ip1(v, sc.b0, tw, ix, t, bar_id);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int e = (lev * 8 + q) * 64 + t;
            dloc[e] = v[q];
            st_async_f2(drem_peer + (uint32_t)((buf * L * kHalf + e) * sizeof(cpx<float>)), v[q].x, v[q].y,
                        dbar_peer + (uint32_t)(buf * sizeof(uint64_t)));
        }
        // the owners' key values, part (r, opt) of every row, loaded while the
        // peer's digits travel: 96 16-byte loads a step and SM hold the
        // load/store unit some 500 clocks, which the rotation and the
        // transform would wait for (1.184 -> 1.119 ms against loads at the
        // start of the step)
        float4 kk[kRows][4];
        if (owner) {
#pragma unroll
            for (int p = 0; p < kRows; ++p) {
                const float4* g4 =
                    reinterpret_cast<const float4*>(step_keys + (size_t)p * kRowElems + (r * 2 + opt) * kHalf);
#pragma unroll
                for (int qq = 0; qq < 4; ++qq) kk[p][qq] = __ldg(g4 + qq * 64 + t);
            }
        }
        __syncthreads();  // every local D in place; every read of acc done
        prefetch_rows(i + kAhead);
        expect_digits(buf ^ 1);  // the other buffer's last digits were used a step ago
        if (owner) {
            if (!mbar_wait_cluster_bounded(&dbar[buf], (k >> 1) & 1, abort)) {  // the peer's D landed
                *abort = 1;
                atomicExch(a.err, 3);
            }
            cpx<float> o[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) o[q] = {0.f, 0.f};
            cpx<float> first[8];  // PAIR: polynomial 0's rows on their own
#pragma unroll
            for (int p = 0; p < kRows; ++p) {
                const int jp = p / L, lv = p - jp * L;
                if (PAIR && p == L) {
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        first[q] = o[q];
                        o[q] = {0.f, 0.f};
                    }
                }
                const cpx<float>* D = jp == r ? dloc + lv * kHalf : drem + (buf * L + lv) * kHalf;
#pragma unroll
                for (int qq = 0; qq < 4; ++qq) {
                    const cpx<float> d0 = D[(2 * qq) * 64 + t];
                    const cpx<float> d1 = D[(2 * qq + 1) * 64 + t];
                    o[2 * qq] = cmac(o[2 * qq], d0, cpx<float>{kk[p][qq].x, kk[p][qq].y});
                    o[2 * qq + 1] = cmac(o[2 * qq + 1], d1, cpx<float>{kk[p][qq].z, kk[p][qq].w});
                }
            }
            if constexpr (PAIR) {
#pragma unroll
                for (int q = 0; q < 8; ++q) o[q] = cadd(first[q], o[q]);
            }
            fft512_inverse_ip1(o, sc.b0, tw, ix, t, bar_id);
            uint32_t c0[8] = {}, c1[8] = {};  // the low part adds into them
            round_part<float, 2>(o, opt, kp.split, c0, c1);
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int x0 = t + 64 * q;
                atomicAdd(reinterpret_cast<unsigned*>(acc + x0), c0[q]);
                atomicAdd(reinterpret_cast<unsigned*>(acc + x0 + kHalf), c1[q]);
            }
        }
        ++k;
        __syncthreads();  // the accumulator is updated before the next step reads it
    }
    if (a.acc_out) {
        int32_t* dst = a.acc_out + (size_t)c * 2 * kN + (size_t)r * kN;
        for (int i = threadIdx.x; i < kN; i += blockDim.x) dst[i] = acc[i];
    }
    if (a.lwe_out) {
        // tLweExtractLweSample: a'_0 = a_0, a'_j = -a_{N-j} (polynomial 0),
        // b' = b_0 (polynomial 1)
        int32_t* dst = a.lwe_out + (size_t)c * (kN + 1);
        if (r == 0) {
            for (int i = threadIdx.x; i < kN; i += blockDim.x)
                dst[i] = i == 0 ? acc[0] : (int32_t)(0u - (uint32_t)acc[kN - i]);
        } else if (threadIdx.x == 0) {
            dst[kN] = acc[0];
        }
    }
    cluster.sync();  // no CTA leaves while its peer could still address its shared memory
}

// ----------------------------------------------------------------------
// The FP64 form's blind rotation over a cluster of two CTAs (lowest FP64
// latency).  The same split as k_blind_rotate_spread2: CTA r holds
// accumulator polynomial r and runs its l forward transforms (one per group),
// pushes the transformed digits into the peer's shared memory (asynchronous
// stores counted on the peer's mbarrier, two alternating buffers), and owns
// output polynomial r.  The FP64 key has one part, so one owner group per
// CTA (group 0) multiplies all 2l rows in row order with output r's part of
// each key row, transforms back and truncates like the reference
// (TorusPolynomial_fft.cpp:40).  The transforms, the products and their
// order are those of the other FP64 shapes.  A single FP64 gate then runs on
// two SMs' FP64 pipes instead of one 64-thread group.
// ----------------------------------------------------------------------
template <int L>
struct Spread2F64Plan {
    static constexpr size_t tables = kHotSize * sizeof(cpx<double>);
    static constexpr size_t acc_off = tables;                                       // own polynomial
    static constexpr size_t dloc_off = acc_off + kN * sizeof(int32_t);             // [lev][q][t]
    static constexpr size_t drem_off = dloc_off + L * kHalf * sizeof(cpx<double>);  // [buf][lev][q][t]
    static constexpr size_t scratch_off = drem_off + 2 * L * kHalf * sizeof(cpx<double>);
    static constexpr size_t scratch = 2 * kScratchStride * sizeof(cpx<double>);
    static constexpr size_t bar_off = scratch_off + L * scratch;  // 2 mbarriers, abort flag
    static constexpr size_t total = bar_off + 2 * sizeof(uint64_t) + 16;
    static constexpr size_t request = total > 120 * 1024 ? total : 120 * 1024;  // one CTA per SM
    static_assert(dloc_off % 16 == 0 && drem_off % 16 == 0 && bar_off % 8 == 0, "alignment");
};

template <int L>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(64 * L, 1)
    k_blind_rotate_spread2_f64(KParams kp, Tables T, EpArgs a) {
    namespace cg = cooperative_groups;
    using Plan = Spread2F64Plan<L>;
    constexpr int kRows = 2 * L;
    constexpr int kRowElems = 2 * kHalf;  // complex values per key row (two outputs, one part)
    constexpr int kEarly = L;             // rows whose key values the owner loads before the transform
    extern __shared__ __align__(128) char smem[];
    cg::cluster_group cluster = cg::this_cluster();
    const int r = (int)cluster.block_rank();  // this CTA's polynomial
    cpx<double>* tables = reinterpret_cast<cpx<double>*>(smem);
    int32_t* acc = reinterpret_cast<int32_t*>(smem + Plan::acc_off);
    cpx<double>* dloc = reinterpret_cast<cpx<double>*>(smem + Plan::dloc_off);
    cpx<double>* drem = reinterpret_cast<cpx<double>*>(smem + Plan::drem_off);
    uint64_t* dbar = reinterpret_cast<uint64_t*>(smem + Plan::bar_off);  // per buffer
    volatile int* abort = reinterpret_cast<volatile int*>(smem + Plan::bar_off + 2 * sizeof(uint64_t));
    const uint32_t drem_peer = cluster_map(smem_u32(drem), (uint32_t)(r ^ 1));
    const uint32_t dbar_peer = cluster_map(smem_u32(dbar), (uint32_t)(r ^ 1));
    const int c = blockIdx.x >> 1;
    const int g = threadIdx.x >> 6, t = threadIdx.x & 63;
    const int lev = g;
    const bool owner = g == 0;
    const int n = kp.n;
    load_hot_tables<double>(tables, T);
    if (a.acc_in) {
        const int32_t* src = a.acc_in + (size_t)c * 2 * kN + (size_t)r * kN;
        for (int i = threadIdx.x; i < kN; i += blockDim.x) acc[i] = src[i];
    } else {
        const int32_t* xs = a.x + (size_t)c * (n + 1);
        const int barb = mod_switch_2n(xs[n]);
        for (int i = threadIdx.x; i < kN; i += blockDim.x) acc[i] = r == 0 ? 0 : test_vector_coef(a, c, barb, i);
    }
    if (threadIdx.x == 0) {
        mbar_init(&dbar[0], 1);
        mbar_init(&dbar[1], 1);
        *abort = a.stall_peers && r == 1;  // self-test: this CTA sends nothing
        fence_mbar_init();
    }
    cluster.sync();  // both CTAs' barriers initialised before any push

    const FftTwiddles<double> tw = hot_twiddles<double>(tables);
    const FftIdx ix = make_fft_idx(t);
    const FftScratch<double> sc = scratch_at<double>(smem + Plan::scratch_off + (size_t)g * Plan::scratch);
    const int bar_id = 1 + g;
    const int halfBg = 1 << (kp.Bgbit - 1);
    const uint32_t mask = (1u << kp.Bgbit) - 1;
    const int decal = 32 - (lev + 1) * kp.Bgbit;
    const cpx<double>* gsw = reinterpret_cast<const cpx<double>*>(a.gsw);
    const size_t step_elems = (size_t)kRows * kRowElems;
    const int32_t* bara = a.bara ? a.bara + (size_t)c * n : nullptr;
    const int32_t* xs = a.x ? a.x + (size_t)c * (n + 1) : nullptr;
    const int32_t* rot = bara ? bara : xs;
    int32_t rot_next = rot[0];
    if (threadIdx.x < kRows)  // output r's part of the first step's rows into L2
        bulk_prefetch_l2(gsw + (size_t)threadIdx.x * kRowElems + r * kHalf, kHalf * sizeof(cpx<double>));
    uint32_t k = 0;  // steps taken (the same in both CTAs)
#pragma unroll 1
    for (int i = 0; i < n; ++i) {
        const int ai = bara ? rot_next : mod_switch_2n(rot_next);
        if (i + 1 < n) rot_next = rot[i + 1];
        if (ai == 0) continue;  // tfhe_blindRotate_FFT.cpp:114 (uniform over the cluster)
        const int stop = *abort;  // the same for the whole CTA: set only between a step's two barriers
        const int buf = (int)(k & 1);
        // this step's incoming digits: one arrival and l x 8 KB of stores
        if (threadIdx.x == 0 && !stop)
            mbar_arrive_expect_tx(&dbar[buf], (uint32_t)(L * kHalf * sizeof(cpx<double>)));
        const cpx<double>* step_keys = gsw + (size_t)i * step_elems;
        if (i + 1 < n && threadIdx.x < kRows)  // the next step's rows into L2
            bulk_prefetch_l2(step_keys + step_elems + (size_t)threadIdx.x * kRowElems + r * kHalf,
                             kHalf * sizeof(cpx<double>));
        // the owner's first rows go out before the transform, so their L2
        // latency overlaps it
        double2 kk[kEarly][8];
        if (owner) {
#pragma unroll
            for (int p = 0; p < kEarly; ++p) {
                const double2* g2 = reinterpret_cast<const double2*>(step_keys + (size_t)p * kRowElems + r * kHalf);
#pragma unroll
                for (int q = 0; q < 8; ++q) kk[p][q] = __ldg(g2 + key_index<double>(t, q));
            }
        }
        cpx<double> v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int x0 = t + 64 * q;
            const uint32_t u0 = (uint32_t)rot_coef(acc, x0, ai) - (uint32_t)acc[x0] + kp.offset;
            const uint32_t u1 = (uint32_t)rot_coef(acc, x0 + kHalf, ai) - (uint32_t)acc[x0 + kHalf] + kp.offset;
            v[q] = digit_pair<double>(u0, u1, decal, mask, halfBg);
        }
        fft512_forward_ip1(v, sc.b0, tw, ix, t, bar_id);
        if (stop) break;  // nothing is armed or sent after a wait has given up
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int e = (lev * 8 + q) * 64 + t;
            dloc[e] = v[q];
            st_async_d2(drem_peer + (uint32_t)((buf * L * kHalf + e) * sizeof(cpx<double>)), v[q].x, v[q].y,
                        dbar_peer + (uint32_t)(buf * sizeof(uint64_t)));
        }
        __syncthreads();  // every local D in place; every read of acc done
        if (owner) {
            if (!mbar_wait_cluster_bounded(&dbar[buf], (k >> 1) & 1, abort)) {  // the peer's D landed
                *abort = 1;
                atomicExch(a.err, 3);
            }
            cpx<double> o[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) o[q] = {0.0, 0.0};
#pragma unroll
            for (int p = 0; p < kRows; ++p) {
                const int jp = p / L, lv = p - jp * L;
                const cpx<double>* D = jp == r ? dloc + lv * kHalf : drem + (buf * L + lv) * kHalf;
                const double2* g2 = reinterpret_cast<const double2*>(step_keys + (size_t)p * kRowElems + r * kHalf);
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const double2 w = p < kEarly ? kk[p < kEarly ? p : 0][q] : __ldg(g2 + key_index<double>(t, q));
                    o[q] = cmac(o[q], D[q * 64 + t], cpx<double>{w.x, w.y});
                }
            }
            fft512_inverse_ip1(o, sc.b0, tw, ix, t, bar_id);
            uint32_t c0[8], c1[8];
            round_part<double, 1>(o, 0, kp.split, c0, c1);
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int x0 = t + 64 * q;
                acc[x0] = (int32_t)((uint32_t)acc[x0] + c0[q]);
                acc[x0 + kHalf] = (int32_t)((uint32_t)acc[x0 + kHalf] + c1[q]);
            }
        }
        ++k;
        __syncthreads();  // the accumulator is updated before the next step reads it
    }
    if (a.acc_out) {
        int32_t* dst = a.acc_out + (size_t)c * 2 * kN + (size_t)r * kN;
        for (int i = threadIdx.x; i < kN; i += blockDim.x) dst[i] = acc[i];
    }
    if (a.lwe_out) {
        // tLweExtractLweSample: a'_0 = a_0, a'_j = -a_{N-j} (polynomial 0),
        // b' = b_0 (polynomial 1)
        int32_t* dst = a.lwe_out + (size_t)c * (kN + 1);
        if (r == 0) {
            for (int i = threadIdx.x; i < kN; i += blockDim.x)
                dst[i] = i == 0 ? acc[0] : (int32_t)(0u - (uint32_t)acc[kN - i]);
        } else if (threadIdx.x == 0) {
            dst[kN] = acc[0];
        }
    }
    if (*abort) let_stores_land();
    cluster.sync();  // no CTA leaves while its peer could still address its shared memory
}

// ----------------------------------------------------------------------
// The FP64 form's blind rotation over a cluster of eight CTAs (lowest FP64
// latency).  One SM's FP64 unit takes 19 clocks per warp instruction (64 for
// a warp alone), so a step's latency is the FP64 work per SM; here a step's
// 5,000 warp instructions are spread over eight SMs in warps of four per SM.
//
//   CTA p < 2l transforms row p's digits (polynomial p / l, level p % l): 128
//   threads, each computing four of a butterfly's eight outputs (its parity,
//   the same for a whole warp: dft8_parity), the inputs exchanged through
//   shared memory, so no operation is done twice.  Positions 64b .. 64b + 63
//   of the result go to CTA b.
//   CTA b multiplies all 2l rows, in row order, at its 64 positions for both
//   output polynomials, one (position, output) a thread, and runs the inverse
//   passes C' and B', which stay within those positions, one output of a
//   butterfly a thread (dft8_one, the output pair the same for a warp).
//   Point t of the block's results goes to CTA t / 8.
//   CTA m runs pass A' for points t = 8m .. 8m + 7, truncates, adds into the
//   coefficients it keeps in registers (t + 64q and + 512), and sends them to
//   the l CTAs that decompose that polynomial.
//
// The three exchanges of a step are asynchronous stores (st.async) counted
// in bytes on the receiver's mbarrier, each into a single buffer: data of
// step k + 1 can only come after every CTA has received all of step k's
// coefficients, and each of those was sent after its sender had read its
// step-k digits and points.  All waits are bounded.
// Every product, sum and rounding is the other FP64 shapes', on the same
// operands, so the ciphertexts agree bit for bit.
// Measured: one ciphertext 20.3 -> 6.2 ms against the two-SM cluster kernel.
// ----------------------------------------------------------------------
template <int L>
struct Cluster8F64Plan {
    static constexpr int kThreads = 128;
    static constexpr size_t acc_off = kHotSize * sizeof(cpx<double>);      // polynomial p / l: (x, x + 512) pairs
    static constexpr size_t x_off = acc_off + kN * sizeof(int32_t);        // transform buffers, ping and pong
    static constexpr size_t d_off = x_off + 2 * kScratchStride * sizeof(cpx<double>);  // [row][q][8] digits received
    static constexpr size_t o_off = d_off + 2 * L * 64 * sizeof(cpx<double>);  // [output][64] block buffers, two
    static constexpr size_t p_off = o_off + 2 * 2 * 72 * sizeof(cpx<double>);  // [output][block][8] points received
    static constexpr size_t bar_off = p_off + 2 * 64 * sizeof(cpx<double>);    // 3 mbarriers, abort flag
    static constexpr size_t total = bar_off + 3 * sizeof(uint64_t) + 16;
    static_assert(acc_off % 16 == 0 && d_off % 16 == 0 && p_off % 16 == 0, "16-byte stores");
};

// one output of the 8-point butterfly v for a thread of class C = its warp
template <int S>
__device__ __forceinline__ cpx<double> dft8_by_warp(const cpx<double> (&v)[8], int cls, bool minus) {
    switch (cls) {
    case 0: return dft8_one<S, 0>(v, minus);
    case 1: return dft8_one<S, 1>(v, minus);
    case 2: return dft8_one<S, 2>(v, minus);
    default: return dft8_one<S, 3>(v, minus);
    }
}

// Barrier of the 128 threads; the two parities reach it from different code.
__device__ __forceinline__ void parity_sync() { asm volatile("barrier.sync 1, 128;" ::: "memory"); }

// Forward transform of one polynomial's digits by 128 threads: (t, H) with
// H the parity of the outputs the thread computes.  In: w[k] = digit of point
// t + 64 (4H + k).  Out: y[k] = position 8t + 2k + H.
template <int H>
__device__ __forceinline__ void forward_parity(cpx<double> (&w)[4], cpx<double> (&y)[4], cpx<double>* x0,
                                               cpx<double>* x1, const FftTwiddles<double>& tw, int t) {
    cpx<double> v[8];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (4 * H + k) w[k] = cmul_alt(w[k], twist_c<double>(4 * H + k));
        x0[spad(t + 64 * (4 * H + k))] = w[k];
    }
    parity_sync();
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = x0[spad(t + 64 * q)];
    dft8_parity<1, H>(v, y);
#pragma unroll
    for (int k = 0; k < 4; ++k) x1[spad(t + 64 * (2 * k + H))] = cmul(y[k], tw.a[(2 * k + H) * 64 + t]);
    parity_sync();
    const int b = t >> 3, j = t & 7;
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = x1[spad(64 * b + j + 8 * q)];
    dft8_parity<1, H>(v, y);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (2 * k + H) y[k] = cmul(y[k], tw.b[(2 * k + H) * 8 + j]);
        x0[spad(64 * b + j + 8 * (2 * k + H))] = y[k];
    }
    parity_sync();
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = x0[spad(8 * t + q)];
    dft8_parity<1, H>(v, y);
}

template <int L>
__global__ void __cluster_dims__(8, 1, 1) __launch_bounds__(Cluster8F64Plan<L>::kThreads, 1)
    k_blind_rotate_cluster8_f64(KParams kp, Tables T, EpArgs a) {
    namespace cg = cooperative_groups;
    using Plan = Cluster8F64Plan<L>;
    constexpr int kRows = 2 * L;
    extern __shared__ __align__(128) char smem[];
    cg::cluster_group cluster = cg::this_cluster();
    const int m = (int)cluster.block_rank();
    cpx<double>* tables = reinterpret_cast<cpx<double>*>(smem);
    int2* acc = reinterpret_cast<int2*>(smem + Plan::acc_off);
    cpx<double>* x0 = reinterpret_cast<cpx<double>*>(smem + Plan::x_off);
    cpx<double>* x1 = x0 + kScratchStride;
    cpx<double>* din = reinterpret_cast<cpx<double>*>(smem + Plan::d_off);
    cpx<double>* o0 = reinterpret_cast<cpx<double>*>(smem + Plan::o_off);
    cpx<double>* o1 = o0 + 2 * 72;
    cpx<double>* pin = reinterpret_cast<cpx<double>*>(smem + Plan::p_off);
    uint64_t* bar_acc = reinterpret_cast<uint64_t*>(smem + Plan::bar_off);  // coefficients received
    uint64_t* bar_d = bar_acc + 1;                                          // digits received
    uint64_t* bar_p = bar_acc + 2;                                          // points received
    volatile int* abort = reinterpret_cast<volatile int*>(bar_acc + 3);
    const int c = blockIdx.x >> 3;
    const int u = threadIdx.x, warp = u >> 5, lane = u & 31;
    const int n = kp.n;
    const bool forward = m < kRows;
    const int jp = m / L, lev = m - jp * L;  // forward: polynomial and level
    load_hot_tables<double>(tables, T);

    // coefficient pairs kept by this thread: output wj, point 8m + wt, q = wq
    // (x = 8m + wt + 64 wq and x + 512); the same thread numbering serves the
    // inverse passes: output wj, butterfly wt, butterfly output wq
    const int wj = (lane >> 3) & 1, wt = lane & 7;
    const bool minus = lane >= 16;
    const int wq = 2 * (warp & 1) + (warp >> 1) + (minus ? 4 : 0);
    uint32_t own0, own1;
    {
        const int x = 8 * m + wt + 64 * wq;
        const int32_t* src = a.acc_in ? a.acc_in + (size_t)c * 2 * kN : nullptr;
        const int barb = src ? 0 : mod_switch_2n(a.x[(size_t)c * (n + 1) + n]);
        const auto start = [&](int j, int i) -> int32_t {
            return src ? src[j * kN + i] : j == 0 ? 0 : test_vector_coef(a, c, barb, i);
        };
        own0 = (uint32_t)start(wj, x);
        own1 = (uint32_t)start(wj, x + kHalf);
        if (forward)
            for (int i = u; i < kHalf; i += Plan::kThreads) acc[i] = make_int2(start(jp, i), start(jp, i + kHalf));
    }
    if (u == 0) {
        mbar_init(bar_acc, 1);
        mbar_init(bar_d, 1);
        mbar_init(bar_p, 1);
        *abort = a.stall_peers && m == 0;  // self-test: this CTA sends no points
        fence_mbar_init();
    }
    cluster.sync();  // every CTA's barriers initialised before any store

    const FftTwiddles<double> tw = hot_twiddles<double>(tables);
    const int halfBg = 1 << (kp.Bgbit - 1);
    const uint32_t mask = (1u << kp.Bgbit) - 1;
    const int decal = 32 - (lev + 1) * kp.Bgbit;
    const cpx<double>* gsw = reinterpret_cast<const cpx<double>*>(a.gsw);
    const size_t step_elems = (size_t)kRows * 2 * kHalf;
    const int32_t* bara = a.bara ? a.bara + (size_t)c * n : nullptr;
    const int32_t* xs = a.x ? a.x + (size_t)c * (n + 1) : nullptr;
    const int32_t* rot = bara ? bara : xs;
    // after a wait that gave up a thread arms nothing more, and its CTA leaves
    // the loop at the next barrier
    bool ok = true;
    const auto wait_for = [&](uint64_t* bar, uint32_t parity) {
        if (!mbar_wait_cluster_bounded(bar, parity, abort)) {
            ok = false;
            *abort = 1;
            atomicExch(a.err, 3);
        }
        __syncwarp();
    };
    int32_t rot_next = rot[0];
    uint32_t k = 0;  // steps taken (the same in all CTAs)
#pragma unroll 1
    for (int i = 0; i < n; ++i) {
        const int ai = bara ? rot_next : mod_switch_2n(rot_next);
        if (i + 1 < n) rot_next = rot[i + 1];
        if (ai == 0) continue;  // tfhe_blindRotate_FFT.cpp:114 (uniform over the cluster)
        if (u == 0 && ok) {
            mbar_arrive_expect_tx(bar_d, kRows * 64 * sizeof(cpx<double>));
            mbar_arrive_expect_tx(bar_p, 2 * 64 * sizeof(cpx<double>));
        }
        // this step's key values at (output mj, position 64m + 8 mt + mq)
        const int mj = u >> 6, mq = (u >> 3) & 7, mt = u & 7;
        double2 kk[kRows];
        {
            const double2* g2 = reinterpret_cast<const double2*>(gsw + (size_t)i * step_elems + mj * kHalf) +
                                key_index<double>(8 * m + mt, mq);
#pragma unroll
            for (int p = 0; p < kRows; ++p) kk[p] = __ldg(g2 + (size_t)p * 2 * kHalf);
        }
        if (forward) {
            if (k > 0) wait_for(bar_acc, (k - 1) & 1);
            if (u == 0 && ok) mbar_arrive_expect_tx(bar_acc, kN * sizeof(int32_t));
            __syncwarp();
            const int t = u & 63, hp = u >> 6;
            cpx<double> w[4], y[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int s = t + 64 * (4 * hp + q);
                const int2 p = acc[s];
                const int rs = s - ai;
                const int2 v = acc[rs & (kHalf - 1)];
                const uint32_t v0 = (uint32_t)(rs & kHalf ? v.y : v.x), v1 = (uint32_t)(rs & kHalf ? v.x : v.y);
                const uint32_t u0 = (rs & kN ? 0u - v0 : v0) - (uint32_t)p.x + kp.offset;
                const uint32_t u1 = ((rs + kHalf) & kN ? 0u - v1 : v1) - (uint32_t)p.y + kp.offset;
                w[q] = digit_pair<double>(u0, u1, decal, mask, halfBg);
            }
            if (hp == 0) forward_parity<0>(w, y, x0, x1, tw, t);
            else forward_parity<1>(w, y, x0, x1, tw, t);
            const uint32_t dst = cluster_map(smem_u32(din), (uint32_t)(t >> 3));
            const uint32_t dbar = cluster_map(smem_u32(bar_d), (uint32_t)(t >> 3));
#pragma unroll
            for (int q = 0; q < 4; ++q)
                st_async_d2(dst + (uint32_t)((m * 64 + (2 * q + hp) * 8 + (t & 7)) * sizeof(cpx<double>)), y[q].x,
                            y[q].y, dbar);
        }
        wait_for(bar_d, k & 1);
        {
            cpx<double> o = {0.0, 0.0};
#pragma unroll
            for (int p = 0; p < kRows; ++p) {
                o = cmac(o, din[p * 64 + mq * 8 + mt], cpx<double>{kk[p].x, kk[p].y});
            }
            o0[mj * 72 + 9 * mt + mq] = o;
        }
        __syncthreads();
        const int stop = *abort;  // the same for the whole CTA: not set between these two barriers
        cpx<double> v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = o0[wj * 72 + 9 * wt + q];
        // pass C' of butterfly wt, output wq, times pass B''s twiddle
        o1[wj * 72 + 9 * wt + wq] = cmulc(dft8_by_warp<-1>(v, warp, minus), tw.b[wt * 8 + wq]);
        __syncthreads();
        if (stop) break;
        // pass B' of butterfly j = wt (positions j + 8r), output wq, times pass A''s twiddle
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = o1[wj * 72 + 9 * q + wt];
        {
            const cpx<double> z = cmulc(dft8_by_warp<-1>(v, warp, minus), tw.a[m * 64 + wt + 8 * wq]);
            st_async_d2(cluster_map(smem_u32(pin), (uint32_t)wq) +
                            (uint32_t)(((wj * 8 + m) * 8 + wt) * sizeof(cpx<double>)),
                        z.x, z.y, cluster_map(smem_u32(bar_p), (uint32_t)wq));
        }
        // pass A' of point 8m + wt, output wq
        wait_for(bar_p, k & 1);
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = pin[(wj * 8 + q) * 8 + wt];
        {
            cpx<double> z = dft8_by_warp<-1>(v, warp, minus);
            cpx<double> un = {1.0, 0.0};
#pragma unroll
            for (int q = 1; q < 8; ++q)
                if (wq == q) un = twist_c<double>(q);
            z = cmulc(z, un);
            own0 += trunc_div512(z.x);
            own1 += trunc_div512(z.y);
            const int x = 8 * m + wt + 64 * wq;
#pragma unroll
            for (int lv = 0; lv < L; ++lv) {
                const uint32_t rank = (uint32_t)(wj * L + lv);
                st_async_i2(cluster_map(smem_u32(acc), rank) + (uint32_t)(x * sizeof(int2)), (int32_t)own0,
                            (int32_t)own1, cluster_map(smem_u32(bar_acc), rank));
            }
        }
        ++k;
    }
    const int x = 8 * m + wt + 64 * wq;
    if (a.acc_out) {
        int32_t* dst = a.acc_out + (size_t)c * 2 * kN + wj * kN;
        dst[x] = (int32_t)own0;
        dst[x + kHalf] = (int32_t)own1;
    }
    if (a.lwe_out) {
        // tLweExtractLweSample: a'_0 = a_0, a'_j = -a_{N-j}, b' = b_0
        int32_t* dst = a.lwe_out + (size_t)c * (kN + 1);
        if (wj == 0) {
            if (x == 0) dst[0] = (int32_t)own0;
            else dst[kN - x] = (int32_t)(0u - own0);
            dst[kHalf - x] = (int32_t)(0u - own1);
        } else if (x == 0) {
            dst[kN] = (int32_t)own0;
        }
    }
    if (forward && k > 0) wait_for(bar_acc, (k - 1) & 1);  // the last coefficients landed
    if (*abort) let_stores_land();
    cluster.sync();  // no CTA leaves while another could still address its shared memory
}

// ----------------------------------------------------------------------
// The FP64 form's blind rotation, one ciphertext per CTA: 2l groups of 64
// threads run a step's 2l forward transforms at once, then groups 0 and 1
// multiply all 2l rows in row order with their output polynomial's part of
// each key row, transform back and truncate.  The FP64 unit bounds it: 19
// clocks per warp instruction and SM when all four SM sub-partitions have a
// warp in FP64 code, 64 when only one has, so the work of a step is laid out
// to keep all four busy in both halves of it (12 warps, then 4).  A step is
// about 5,000 FP64 warp instructions, 95,000 clocks (29 ms for n = 630).
// Measured: 29.8 ms a wave of 152, 59.5 ms for 300, against 43.2 ms (two
// waves of the cluster kernel) and 92.6 ms (a wave of the 3-per-CTA kernel)
// before it.
// The transforms, the products and their order are those of the other FP64
// shapes.
// ----------------------------------------------------------------------
template <int L>
struct SpreadF64Plan {
    static constexpr int kGroups = 2 * L;
    static constexpr size_t acc_off = kHotSize * sizeof(cpx<double>);
    static constexpr size_t d_off = acc_off + 2 * kN * sizeof(int32_t);            // [row][q][t]
    static constexpr size_t x_off = d_off + kGroups * kHalf * sizeof(cpx<double>);  // one exchange buffer a group
    static constexpr size_t total = x_off + kGroups * kScratchStride * sizeof(cpx<double>);
};

template <int L>
__global__ void __launch_bounds__(128 * L, 1) k_blind_rotate_spread_f64(KParams kp, Tables T, EpArgs a) {
    using Plan = SpreadF64Plan<L>;
    constexpr int kRows = 2 * L;
    constexpr int kRowElems = 2 * kHalf;  // complex values per key row (two outputs, one part)
    extern __shared__ __align__(128) char smem[];
    cpx<double>* tables = reinterpret_cast<cpx<double>*>(smem);
    int32_t* acc = reinterpret_cast<int32_t*>(smem + Plan::acc_off);
    cpx<double>* dsh = reinterpret_cast<cpx<double>*>(smem + Plan::d_off);
    const int c = blockIdx.x;
    const int g = threadIdx.x >> 6, t = threadIdx.x & 63;
    const int jp = g / L, lev = g - jp * L;
    const int n = kp.n;
    load_hot_tables<double>(tables, T);
    if (a.acc_in) {
        const int32_t* src = a.acc_in + (size_t)c * 2 * kN;
        for (int i = threadIdx.x; i < 2 * kN; i += blockDim.x) acc[i] = src[i];
    } else {
        const int barb = mod_switch_2n(a.x[(size_t)c * (n + 1) + n]);
        for (int i = threadIdx.x; i < kN; i += blockDim.x) {
            acc[i] = 0;
            acc[kN + i] = test_vector_coef(a, c, barb, i);
        }
    }
    __syncthreads();

    const FftTwiddles<double> tw = hot_twiddles<double>(tables);
    const FftIdx ix = make_fft_idx(t);
    cpx<double>* xbuf = reinterpret_cast<cpx<double>*>(smem + Plan::x_off) + g * kScratchStride;
    const int bar_id = 1 + g;
    const int halfBg = 1 << (kp.Bgbit - 1);
    const uint32_t mask = (1u << kp.Bgbit) - 1;
    const int decal = 32 - (lev + 1) * kp.Bgbit;
    const cpx<double>* gsw = reinterpret_cast<const cpx<double>*>(a.gsw);
    const size_t step_elems = (size_t)kRows * kRowElems;
    const int32_t* bara = a.bara ? a.bara + (size_t)c * n : nullptr;
    const int32_t* xs = a.x ? a.x + (size_t)c * (n + 1) : nullptr;
    const int32_t* rot = bara ? bara : xs;
    int32_t rot_next = rot[0];
#pragma unroll 1
    for (int i = 0; i < n; ++i) {
        const int ai = bara ? rot_next : mod_switch_2n(rot_next);
        if (i + 1 < n) rot_next = rot[i + 1];
        if (ai == 0) continue;  // tfhe_blindRotate_FFT.cpp:114 (uniform over the CTA)
        const cpx<double>* step_keys = gsw + (size_t)i * step_elems;
        if (threadIdx.x < kRows)  // this step's rows into L2 during its transforms
            bulk_prefetch_l2(step_keys + (size_t)threadIdx.x * kRowElems, kRowElems * sizeof(cpx<double>));
        cpx<double> v[8];
        {
            const int32_t* src = acc + jp * kN;
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int x0 = t + 64 * q;
                const uint32_t u0 = (uint32_t)rot_coef(src, x0, ai) - (uint32_t)src[x0] + kp.offset;
                const uint32_t u1 = (uint32_t)rot_coef(src, x0 + kHalf, ai) - (uint32_t)src[x0 + kHalf] + kp.offset;
                v[q] = digit_pair<double>(u0, u1, decal, mask, halfBg);
            }
        }
        fft512_forward_ip1(v, xbuf, tw, ix, t, bar_id);
#pragma unroll
        for (int q = 0; q < 8; ++q) dsh[(g * 8 + q) * 64 + t] = v[q];
        __syncthreads();  // every D in place; every read of acc done
        if (g < 2) {
            cpx<double> o[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) o[q] = {0.0, 0.0};
#pragma unroll
            for (int p = 0; p < kRows; ++p) {
                const double2* g2 = reinterpret_cast<const double2*>(step_keys + (size_t)p * kRowElems + g * kHalf);
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const double2 w = __ldg(g2 + key_index<double>(t, q));
                    o[q] = cmac(o[q], dsh[(p * 8 + q) * 64 + t], cpx<double>{w.x, w.y});
                }
            }
            fft512_inverse_ip1(o, xbuf, tw, ix, t, bar_id);
            uint32_t c0[8], c1[8];
            round_part<double, 1>(o, 0, kp.split, c0, c1);
            int32_t* dst = acc + g * kN;
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int x0 = t + 64 * q;
                dst[x0] = (int32_t)((uint32_t)dst[x0] + c0[q]);
                dst[x0 + kHalf] = (int32_t)((uint32_t)dst[x0 + kHalf] + c1[q]);
            }
        }
        __syncthreads();  // the accumulator is updated before the next step reads it
    }
    if (a.acc_out) {
        int32_t* dst = a.acc_out + (size_t)c * 2 * kN;
        for (int i = threadIdx.x; i < 2 * kN; i += blockDim.x) dst[i] = acc[i];
    }
    if (a.lwe_out) {
        // tLweExtractLweSample: a'_0 = a_0, a'_j = -a_{N-j}, b' = b_0
        int32_t* dst = a.lwe_out + (size_t)c * (kN + 1);
        for (int i = threadIdx.x; i < kN; i += blockDim.x)
            dst[i] = i == 0 ? acc[0] : (int32_t)(0u - (uint32_t)acc[kN - i]);
        if (threadIdx.x == 0) dst[kN] = acc[kN];
    }
}

// ----------------------------------------------------------------------
// Blind rotation with two 64-thread halves per ciphertext (low latency).
//
// Half h of a ciphertext decomposes and transforms input polynomial h (rows
// h l .. h l + l - 1 of every key step), multiply-accumulates them into the
// partial products of both output polynomials, hands the partial of output
// 1 - h to the other half through shared memory, and transforms back only
// output h.  Each half reads and writes only accumulator polynomial h, so the
// halves meet once per step (the partial exchange).  Per step and half: l
// forward and PARTS inverse transforms instead of 2l and 2 PARTS, so a
// ciphertext takes about half the time; used when a batch has at most three
// ciphertexts per SM to spread (the last partial wave of a large batch,
// small batches, single gates).  Key rows come through the same shared ring
// as k_blind_rotate_ring; each row is read by one half of every ciphertext.
// ----------------------------------------------------------------------
__device__ __forceinline__ void pair_sync(int bar_id) { converged_sync(bar_id, 2 * kFftThreads); }

// h is the half; out[h] and out[1 - h] are picked by uniform branches so
// that the accumulators stay in registers with one copy of the code.
template <typename R, int PARTS, int L, typename Keys>
__device__ __forceinline__ void ep_step_half(const StepCtx<R, PARTS, 1, ConvergedBarrier>& S, Keys& keys, int a, int h,
                                             cpx<R>* peer_inbox, int pair_bar) {
    const int t = S.t;
    const int halfBg = 1 << (S.Bgbit - 1);
    const uint32_t mask = (1u << S.Bgbit) - 1;

    cpx<R> out[2][PARTS][8];
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int pt = 0; pt < PARTS; ++pt)
#pragma unroll
            for (int q = 0; q < 8; ++q) out[j][pt][q] = {(R)0, (R)0};

    {
        const int32_t* src = S.acc + h * kN;
        uint32_t r0[8], r1[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const int x0 = t + 64 * r;
            r0[r] = (uint32_t)rot_coef(src, x0, a) - (uint32_t)src[x0] + S.offset;
            r1[r] = (uint32_t)rot_coef(src, x0 + kHalf, a) - (uint32_t)src[x0 + kHalf] + S.offset;
        }
#pragma unroll 1
        for (int lev = 0; lev < L; ++lev) {
            cpx<R> v[8];
            const int decal = 32 - (lev + 1) * S.Bgbit;
#pragma unroll
            for (int r = 0; r < 8; ++r)
                v[r] = digit_pair<R>(r0[r], r1[r], decal, mask, halfBg);
            fft512_forward_tw(v, S.s[0], S.tw, S.ix, t, S.bar_id);
            const int p = h * L + lev;
            mac_row<R, PARTS, Keys::kShared>(out, v, keys.acquire(p), t);
            keys.release(p);
        }
    }
    // every row of this step is issued before the producer waits on its pair
    if (keys.producer) keys.issue_through(keys.row0 + 2 * L - 1);

    // exchange: both halves' forward transforms are done, so their scratch
    // buffers are free; write the partial of output 1 - h into the other
    // half's scratch, then read this half's own
    pair_sync(pair_bar);
#pragma unroll
    for (int pt = 0; pt < PARTS; ++pt) {
        cpx<R> w[8];
        pick_part<R, PARTS>(w, out, 1 - h, pt);
#pragma unroll
        for (int q = 0; q < 8; ++q) peer_inbox[pt * kScratchStride + q * 64 + t] = w[q];
    }
    pair_sync(pair_bar);
    // the next step's first rows land during this step's inverse transforms
    if (keys.producer) {
        keys.stop_if(*keys.abort);  // the other half has given up on a row
        keys.issue_upto(keys.row0 + 2 * L - 1);
    }
    {
        const cpx<R>* inbox = S.s[0].b0;
#pragma unroll
        for (int pt = 0; pt < PARTS; ++pt) {
            cpx<R> w[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) w[q] = inbox[pt * kScratchStride + q * 64 + t];
            add_part<R, PARTS>(out, w, h, pt);
        }
    }
    group_sync(S.bar_id);  // the inbox is the transform's scratch

    uint32_t c0[8], c1[8];
#pragma unroll 1
    for (int pt = 0; pt < PARTS; ++pt) {
        cpx<R> v[8];
        pick_part<R, PARTS>(v, out, h, pt);
        fft512_inverse_tw(v, S.s[0], S.tw, S.ix, t, S.bar_id);
        round_part<R, PARTS>(v, pt, S.split, c0, c1);
    }
    int32_t* dst = S.acc + h * kN;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int x0 = t + 64 * q;
        dst[x0] = (int32_t)((uint32_t)dst[x0] + c0[q]);
        dst[x0 + kHalf] = (int32_t)((uint32_t)dst[x0 + kHalf] + c1[q]);
    }
    group_sync(S.bar_id);
}

template <typename R, int PARTS, int PAIRS, int L, int S>
struct PairPlan {
    static constexpr size_t kRowBytes = (size_t)2 * PARTS * kHalf * sizeof(cpx<R>);
    static constexpr size_t tables = kHotSize * sizeof(cpx<R>);
    static constexpr size_t ring_off = (tables + 127) & ~(size_t)127;
    static constexpr size_t bar_off = ring_off + S * kRowBytes;
    static constexpr size_t flag_off = bar_off + 2 * S * sizeof(uint64_t);
    static constexpr size_t pair_off = (flag_off + sizeof(int) + 127) & ~(size_t)127;
    static constexpr size_t acc = 2 * kN * sizeof(int32_t);
    static constexpr size_t half_scratch = 2 * kScratchStride * sizeof(cpx<R>);
    static constexpr size_t pair = acc + 2 * half_scratch;
    static constexpr size_t total = pair_off + PAIRS * pair;
};

template <typename R, int PARTS, int PAIRS, int L, int S>
__global__ void __launch_bounds__(128 * PAIRS, 1) k_blind_rotate_pair(KParams kp, Tables T, EpArgs a) {
    using Plan = PairPlan<R, PARTS, PAIRS, L, S>;
    static_assert(1 + 2 * PAIRS + PAIRS <= 16, "named barriers");
    static_assert(PARTS * kScratchStride >= PARTS * kHalf, "inbox fits the scratch");
    constexpr int kpl = 2 * L;
    extern __shared__ __align__(128) char smem[];
    cpx<R>* tables = reinterpret_cast<cpx<R>*>(smem);
    cpx<R>* ring = reinterpret_cast<cpx<R>*>(smem + Plan::ring_off);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + Plan::bar_off);
    uint64_t* empty = full + S;
    volatile int* abort = reinterpret_cast<volatile int*>(smem + Plan::flag_off);
    const int active = min(PAIRS, a.count - (int)blockIdx.x * PAIRS);
    if (threadIdx.x == 0) {
        for (int i = 0; i < S; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 64 * active);  // one half of every ciphertext reads a row
        }
        *abort = 0;
        fence_mbar_init();
    }
    load_hot_tables<R>(tables, T);
    __syncthreads();

    const int pr = threadIdx.x >> 7;
    const int h = (threadIdx.x >> 6) & 1;
    const int t = threadIdx.x & 63;
    const int c = blockIdx.x * PAIRS + pr;
    if (pr >= active) return;
    const int n = kp.n;
    RingKeys<R, PARTS, S> keys{ring, full, empty, 0, a.err, abort, threadIdx.x == 0 && !a.stall_keys,
                               reinterpret_cast<const char*>(a.gsw), (uint32_t)n * kpl, 0};

    char* pbase = smem + Plan::pair_off + (size_t)pr * Plan::pair;
    StepCtx<R, PARTS, 1, ConvergedBarrier> St;
    St.tw = hot_twiddles<R>(tables);
    St.ix = make_fft_idx(t);
    St.acc = reinterpret_cast<int32_t*>(pbase);
    St.s[0] = scratch_at<R>(pbase + Plan::acc + h * Plan::half_scratch);
    cpx<R>* peer_inbox = reinterpret_cast<cpx<R>*>(pbase + Plan::acc + (1 - h) * Plan::half_scratch);
    St.t = t;
    St.bar_id = {1 + 2 * pr + h};
    const int pair_bar = 1 + 2 * PAIRS + pr;
    St.Bgbit = kp.Bgbit;
    St.split = kp.split;
    St.offset = kp.offset;

    // half h owns accumulator polynomial h
    int32_t* mine = St.acc + h * kN;
    if (a.acc_in) {
        const int32_t* src = a.acc_in + (size_t)c * 2 * kN + h * kN;
        for (int i = t; i < kN; i += 64) mine[i] = src[i];
    } else {
        const int32_t* xs = a.x + (size_t)c * (n + 1);
        const int barb = mod_switch_2n(xs[n]);
        for (int i = t; i < kN; i += 64)
            mine[i] = h == 0 ? 0 : test_vector_coef(a, c, barb, i);
    }
    group_sync(St.bar_id);
    const int32_t* bara = a.bara ? a.bara + (size_t)c * n : nullptr;
    const int32_t* xs = a.x ? a.x + (size_t)c * (n + 1) : nullptr;
    int a_next = bara ? bara[0] : mod_switch_2n(xs[0]);
#pragma unroll 1
    for (int i = 0; i < n; ++i) {
        const int ai = a_next;
        if (i + 1 < n) a_next = bara ? bara[i + 1] : mod_switch_2n(xs[i + 1]);
        keys.row0 = (uint32_t)i * kpl;
        if (ai == 0) {  // tfhe_blindRotate_FFT.cpp:114 -- this half's rows still pass through
            for (int p = h * L; p < h * L + L; ++p) {
                keys.acquire(p);
                keys.release(p);
            }
            continue;
        }
        ep_step_half<R, PARTS, L>(St, keys, ai, h, peer_inbox, pair_bar);
    }
    if (keys.producer) {
        keys.issue_through(keys.total - 1);  // rows of a skipped last step
        keys.drain();
    }
    pair_sync(pair_bar);  // both polynomials final
    if (a.acc_out) {
        int32_t* dst = a.acc_out + (size_t)c * 2 * kN + h * kN;
        for (int i = t; i < kN; i += 64) dst[i] = mine[i];
    }
    if (a.lwe_out) {
        // tLweExtractLweSample: a'_0 = a_0, a'_j = -a_{N-j}, b' = b_0
        int32_t* dst = a.lwe_out + (size_t)c * (kN + 1);
        const int tt = h * 64 + t;
        for (int i = tt; i < kN; i += 128)
            dst[i] = i == 0 ? St.acc[0] : (int32_t)(0u - (uint32_t)St.acc[kN - i]);
        if (tt == 0) dst[kN] = St.acc[kN];
    }
}

// ----------------------------------------------------------------------
// key conversion: one 64-thread group per polynomial
// ----------------------------------------------------------------------
__device__ __forceinline__ void twisted_forward64(const double* coef, cpx<double> (&v)[8],
                                                  const FftScratch<double>& s,
                                                  const FftTwiddles<double>& tw,
                                                  const cpx<double>* psi, int t, int bar) {
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const int x0 = t + 64 * r;
        v[r] = cmul_alt(cpx<double>{coef[x0], coef[x0 + kHalf]}, psi[x0]);
    }
    fft512_forward(v, s, tw, t, bar);
}

// Per polynomial smem: 1024 doubles of coefficients + scratch.
constexpr size_t kConvGroupBytes = kN * sizeof(double) + 2 * kScratchStride * sizeof(cpx<double>);
constexpr size_t kConvTableBytes = kTabSize * sizeof(cpx<double>);

template <int FORM>
__global__ void __launch_bounds__(256) k_tgsw_to_fft(Tables T, const int32_t* __restrict__ in,
                                                     void* out, int npoly, int split) {
    extern __shared__ __align__(128) char smem[];
    cpx<double>* tables = reinterpret_cast<cpx<double>*>(smem);
    load_tables<double>(tables, T);
    __syncthreads();
    const int g = threadIdx.x >> 6, t = threadIdx.x & 63;
    const int poly = blockIdx.x * (blockDim.x >> 6) + g;
    if (poly >= npoly) return;
    char* gbase = smem + kConvTableBytes + (size_t)g * kConvGroupBytes;
    double* coef = reinterpret_cast<double*>(gbase);
    FftScratch<double> s = scratch_at<double>(gbase + kN * sizeof(double));
    const int32_t* src = in + (size_t)poly * kN;
    const int bar = 1 + g;

    if (FORM == kFormFp64) {
        for (int i = t; i < kN; i += 64) coef[i] = (double)src[i];
        group_sync(bar);
        cpx<double> v[8];
        twisted_forward64(coef, v, s, twiddles_at<double>(tables), tables + kTabPsi, t, bar);
        cpx<double>* dst = reinterpret_cast<cpx<double>*>(out) + (size_t)poly * kHalf;
#pragma unroll
        for (int q = 0; q < 8; ++q) dst[key_index<double>(t, q)] = v[q];
    } else {
        // split K = Khi * 2^s + Klo, Klo in [-2^(s-1), 2^(s-1))
        cpx<float>* dst = reinterpret_cast<cpx<float>*>(out) + (size_t)poly * 2 * kHalf;
        for (int part = 0; part < 2; ++part) {
            for (int i = t; i < kN; i += 64) {
                const int64_t K = src[i];
                const int64_t half = (int64_t)1 << (split - 1);
                const int64_t lo = ((K + half) & (((int64_t)1 << split) - 1)) - half;
                const int64_t hi = (K - lo) >> split;
                coef[i] = (double)(part == 0 ? hi : lo);
            }
            group_sync(bar);
            cpx<double> v[8];
            twisted_forward64(coef, v, s, twiddles_at<double>(tables), tables + kTabPsi, t, bar);
#pragma unroll
            for (int q = 0; q < 8; ++q)
                dst[part * kHalf + key_index<float>(t, q)] = {(float)v[q].x, (float)v[q].y};
            group_sync(bar);
        }
    }
}

// engine FP64 layout -> integer coefficients (rounded to nearest)
__global__ void __launch_bounds__(256) k_fft64_to_tgsw(Tables T, const void* in,
                                                       int32_t* __restrict__ out, int npoly) {
    extern __shared__ __align__(128) char smem[];
    cpx<double>* tables = reinterpret_cast<cpx<double>*>(smem);
    load_tables<double>(tables, T);
    __syncthreads();
    const int g = threadIdx.x >> 6, t = threadIdx.x & 63;
    const int poly = blockIdx.x * (blockDim.x >> 6) + g;
    if (poly >= npoly) return;
    char* gbase = smem + kConvTableBytes + (size_t)g * kConvGroupBytes;
    FftScratch<double> s = scratch_at<double>(gbase + kN * sizeof(double));
    const cpx<double>* src = reinterpret_cast<const cpx<double>*>(in) + (size_t)poly * kHalf;
    cpx<double> v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = src[key_index<double>(t, q)];
    fft512_inverse(v, s, twiddles_at<double>(tables), t, 1 + g);
    int32_t* dst = out + (size_t)poly * kN;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const cpx<double> z = cmulc(v[q], tables[kTabPsi + t + 64 * q]);
        dst[t + 64 * q] = (int32_t)(uint32_t)(uint64_t)llrint(z.x / 512.0);
        dst[t + 64 * q + kHalf] = (int32_t)(uint32_t)(uint64_t)llrint(z.y / 512.0);
    }
}

// ----------------------------------------------------------------------
// Lagrange half-complex form in the reference layout: value m' is
// P(w^(2m'+1)), w = e^{i pi/N}.  Engine frequency m is P(psi^(4m+1)).
// ----------------------------------------------------------------------
__device__ __forceinline__ void engine_to_ref_index(int m, int* ref, bool* conj) {
    const int e = (4 * m + 1) & 2047;
    if (e < kN) {
        *ref = (e - 1) >> 1;
        *conj = false;
    } else {
        *ref = (2048 - e - 1) >> 1;
        *conj = true;
    }
}

// in: count polynomials (int32 coefficients), out: count x 512 complex
// doubles in the reference layout, multiplied by `scale`.
__global__ void __launch_bounds__(256) k_poly_to_lagrange(Tables T, const int32_t* __restrict__ in,
                                                          double* __restrict__ out, int npoly,
                                                          double scale) {
    extern __shared__ __align__(128) char smem[];
    cpx<double>* tables = reinterpret_cast<cpx<double>*>(smem);
    load_tables<double>(tables, T);
    __syncthreads();
    const int g = threadIdx.x >> 6, t = threadIdx.x & 63;
    const int poly = blockIdx.x * (blockDim.x >> 6) + g;
    if (poly >= npoly) return;
    char* gbase = smem + kConvTableBytes + (size_t)g * kConvGroupBytes;
    double* coef = reinterpret_cast<double*>(gbase);
    FftScratch<double> s = scratch_at<double>(gbase + kN * sizeof(double));
    const int32_t* src = in + (size_t)poly * kN;
    for (int i = t; i < kN; i += 64) coef[i] = (double)src[i];
    group_sync(1 + g);
    cpx<double> v[8];
    twisted_forward64(coef, v, s, twiddles_at<double>(tables), tables + kTabPsi, t, 1 + g);
    double* dst = out + (size_t)poly * kN;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        int ref;
        bool cj;
        engine_to_ref_index(freq_of(t, q), &ref, &cj);
        dst[2 * ref] = v[q].x * scale;
        dst[2 * ref + 1] = (cj ? -v[q].y : v[q].y) * scale;
    }
}

// TorusPolynomial_fft: reference-layout values (torus / 2^32 scale) ->
// Torus32 coefficients, truncating like TorusPolynomial_fft.cpp:39-41.
__global__ void __launch_bounds__(256) k_lagrange_to_torus(Tables T, const double* __restrict__ in,
                                                           int32_t* __restrict__ out, int npoly) {
    extern __shared__ __align__(128) char smem[];
    cpx<double>* tables = reinterpret_cast<cpx<double>*>(smem);
    load_tables<double>(tables, T);
    __syncthreads();
    const int g = threadIdx.x >> 6, t = threadIdx.x & 63;
    const int poly = blockIdx.x * (blockDim.x >> 6) + g;
    if (poly >= npoly) return;
    char* gbase = smem + kConvTableBytes + (size_t)g * kConvGroupBytes;
    FftScratch<double> s = scratch_at<double>(gbase + kN * sizeof(double));
    const double* src = in + (size_t)poly * kN;
    cpx<double> v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        int ref;
        bool cj;
        engine_to_ref_index(freq_of(t, q), &ref, &cj);
        const double re = src[2 * ref], im = src[2 * ref + 1];
        v[q] = {re, cj ? -im : im};
    }
    fft512_inverse(v, s, twiddles_at<double>(tables), t, 1 + g);
    const double sc = 4294967296.0 / 512.0;
    int32_t* dst = out + (size_t)poly * kN;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const cpx<double> z = cmulc(v[q], tables[kTabPsi + t + 64 * q]);
        dst[t + 64 * q] = (int32_t)(uint32_t)(uint64_t)__double2ll_rz(z.x * sc);
        dst[t + 64 * q + kHalf] = (int32_t)(uint32_t)(uint64_t)__double2ll_rz(z.y * sc);
    }
}

// reference layout <-> engine FP64 layout, values multiplied by `scale`
__global__ void k_ref_to_engine64(const double* __restrict__ ref, cpx<double>* __restrict__ eng,
                                  int npoly, double scale) {
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= npoly * kHalf) return;
    const int poly = idx / kHalf, e = idx % kHalf;
    const int t = e & 63, q = e >> 6;
    int r;
    bool cj;
    engine_to_ref_index(freq_of(t, q), &r, &cj);
    const double re = ref[(size_t)poly * kN + 2 * r], im = ref[(size_t)poly * kN + 2 * r + 1];
    eng[(size_t)poly * kHalf + key_index<double>(t, q)] = {re * scale, (cj ? -im : im) * scale};
}

__global__ void k_engine64_to_ref(const cpx<double>* __restrict__ eng, double* __restrict__ ref,
                                  int npoly, double scale) {
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= npoly * kHalf) return;
    const int poly = idx / kHalf, e = idx % kHalf;
    const int t = e & 63, q = e >> 6;
    int r;
    bool cj;
    engine_to_ref_index(freq_of(t, q), &r, &cj);
    const cpx<double> v = eng[(size_t)poly * kHalf + key_index<double>(t, q)];
    ref[(size_t)poly * kN + 2 * r] = v.x * scale;
    ref[(size_t)poly * kN + 2 * r + 1] = (cj ? -v.y : v.y) * scale;
}

// LagrangeHalfCPolynomialAddMul (tGswFFTExternMulToTLwe.cpp:172-180)
__global__ void k_lagrange_addmul(const double* __restrict__ a, const double* __restrict__ b,
                                  double* __restrict__ acc, size_t total) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const double ar = a[2 * i], ai = a[2 * i + 1], br = b[2 * i], bi = b[2 * i + 1];
    acc[2 * i] += ar * br - ai * bi;
    acc[2 * i + 1] += ar * bi + ai * br;
}

// ----------------------------------------------------------------------
// small kernels
// ----------------------------------------------------------------------
__device__ __forceinline__ void gate_coeffs(int gate, int32_t e8, int32_t e4, int32_t* c,
                                            int32_t* sa, int32_t* sb) {
    switch (gate) {
    case 0: *c = e8; *sa = -1; *sb = -1; break;   // NAND
    case 1: *c = -e8; *sa = 1; *sb = 1; break;    // AND
    case 2: *c = e8; *sa = 1; *sb = 1; break;     // OR
    case 3: *c = e4; *sa = 2; *sb = 2; break;     // XOR
    case 4: *c = -e4; *sa = -2; *sb = -2; break;  // XNOR
    case 5: *c = -e8; *sa = -1; *sb = -1; break;  // NOR
    case 6: *c = -e8; *sa = -1; *sb = 1; break;   // ANDNY
    case 7: *c = -e8; *sa = 1; *sb = -1; break;   // ANDYN
    case 8: *c = e8; *sa = -1; *sb = 1; break;    // ORNY
    case 9: *c = e8; *sa = 1; *sb = -1; break;    // ORYN
    default: *c = 0; *sa = 0; *sb = 0; break;
    }
}

__global__ void k_gate_combine(int n, const int32_t* __restrict__ gates, int uniform_gate,
                               const int32_t* __restrict__ ca, const int32_t* __restrict__ cb,
                               int32_t* __restrict__ out, int count) {
    const size_t width = (size_t)n + 1;
    const size_t total = (size_t)count * width;
    for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (size_t)gridDim.x * blockDim.x) {
        const size_t c = idx / width;
        const int i = (int)(idx - c * width);
        const int gate = gates ? gates[c] : uniform_gate;
        int32_t k0, sa, sb;
        gate_coeffs(gate, 1 << 29, 1 << 30, &k0, &sa, &sb);
        uint32_t v = (i == n) ? (uint32_t)k0 : 0u;
        v += (uint32_t)sa * (uint32_t)ca[idx];
        v += (uint32_t)sb * (uint32_t)cb[idx];
        out[idx] = (int32_t)v;
    }
}

__global__ void k_lwe_add2_const(const int32_t* __restrict__ u1, const int32_t* __restrict__ u2,
                                 int32_t* __restrict__ out, int width, int32_t mu, int count) {
    const size_t total = (size_t)count * width;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (size_t)gridDim.x * blockDim.x) {
        uint32_t v = (uint32_t)u1[i] + (uint32_t)u2[i];
        if ((int)(i % width) == width - 1) v += (uint32_t)mu;
        out[i] = (int32_t)v;
    }
}

__global__ void k_mul_by_xai_minus_one(const int32_t* __restrict__ in,
                                       const int32_t* __restrict__ ai, int32_t* __restrict__ out,
                                       int polys_per_item, int count) {
    const size_t total = (size_t)count * polys_per_item * kN;
    for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (size_t)gridDim.x * blockDim.x) {
        const size_t poly = idx / kN;
        const int x = (int)(idx - poly * kN);
        const int a = ai[poly / polys_per_item];
        const int32_t* p = in + poly * kN;
        out[idx] = (int32_t)((uint32_t)rot_coef(p, x, a) - (uint32_t)p[x]);
    }
}

__global__ void k_extract(const int32_t* __restrict__ acc, int32_t* __restrict__ out, int count) {
    const int c = blockIdx.x;
    if (c >= count) return;
    const int32_t* a = acc + (size_t)c * 2 * kN;
    int32_t* o = out + (size_t)c * (kN + 1);
    for (int i = threadIdx.x; i < kN; i += blockDim.x)
        o[i] = i == 0 ? a[0] : (int32_t)(0u - (uint32_t)a[kN - i]);
    if (threadIdx.x == 0) o[kN] = a[kN];
}

template <typename Kern>
cudaError_t set_smem(Kern k, size_t bytes) {
    return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

uint32_t decomp_offset(int l, int Bgbit) {
    // constants.h:24 (2164391936 for l = 3, Bgbit = 7)
    uint32_t o = 0;
    for (int i = 0; i < l; ++i) o += 1u << (32 - (i + 1) * Bgbit);
    return o * (uint32_t)(1 << (Bgbit - 1));
}

KParams make_kparams(const DevParams& P) {
    KParams kp;
    kp.n = P.n;
    kp.Bgbit = P.Bgbit;
    kp.split = P.split_bits;
    kp.offset = decomp_offset(P.l, P.Bgbit);
    return kp;
}

// The blind-rotation arguments of items [off, off + cnt) of a batch.
EpArgs slice_blind_rotate(const DevParams& P, const EpArgs& a, int off, int cnt) {
    EpArgs b = a;
    const size_t o = (size_t)off;
    if (a.acc_in) b.acc_in = a.acc_in + o * 2 * kN;
    if (a.acc_out) b.acc_out = a.acc_out + o * 2 * kN;
    if (a.bara) b.bara = a.bara + o * P.n;
    if (a.x) b.x = a.x + o * (P.n + 1);
    if (a.lwe_out) b.lwe_out = a.lwe_out + o * (kN + 1);
    if (a.tv) b.tv = a.tv + o * a.tv_stride;
    b.count = cnt;
    return b;
}

template <typename R, int PARTS, int MODE, int GROUPS, int L>
cudaError_t launch_ep_t(const DevParams& P, const Tables& T, const EpArgs& a, cudaStream_t st) {
    if (a.count <= 0) return cudaSuccess;
    const KParams kp = make_kparams(P);
    const size_t smem = SmemPlan<R, (L > PARTS ? L : PARTS)>::total(GROUPS);
    auto kern = k_external_product<R, PARTS, MODE, GROUPS, L>;
    cudaError_t e = set_smem(kern, smem);
    if (e != cudaSuccess) return e;
    const int grid = MODE == kEpBlindRotate ? (a.count + GROUPS - 1) / GROUPS : std::min(a.count, kSmCount);
    kern<<<grid, 64 * GROUPS, smem, st>>>(kp, T, a);
    return cudaGetLastError();
}

template <int MODE, int L>
cudaError_t launch_products(const DevParams& P, const Tables& T, const EpArgs& a, cudaStream_t st) {
    if (a.count <= 0) return cudaSuccess;
    const KParams kp = make_kparams(P);
    using Plan = ProductPlan<L>;
    auto kern = k_products_stream<MODE, L>;
    cudaError_t e = set_smem(kern, Plan::total);
    if (e != cudaSuccess) return e;
    kern<<<std::min(a.count, kSmCount), 64 * Plan::kGroups, Plan::total, st>>>(kp, T, a);
    return cudaGetLastError();
}

template <typename R, int PARTS, int GROUPS, int L, bool INLINE, int S = 4, int NB = 1>
cudaError_t launch_ring_t(const DevParams& P, const Tables& T, const EpArgs& a, cudaStream_t st) {
    if (a.count <= 0) return cudaSuccess;
    const KParams kp = make_kparams(P);
    using Plan = RingPlan<R, PARTS, GROUPS, L, S, NB>;
    auto kern = k_blind_rotate_ring<R, PARTS, GROUPS, L, S, INLINE, NB>;
    cudaError_t e = set_smem(kern, Plan::total);
    if (e != cudaSuccess) return e;
    const int grid = (a.count + GROUPS - 1) / GROUPS;
    kern<<<grid, 64 * GROUPS + (INLINE ? 0 : 32), Plan::total, st>>>(kp, T, a);
    return cudaGetLastError();
}

template <typename R, int PARTS, int PAIRS, int L, int S>
cudaError_t launch_pair_t(const DevParams& P, const Tables& T, const EpArgs& a, cudaStream_t st) {
    if (a.count <= 0) return cudaSuccess;
    const KParams kp = make_kparams(P);
    using Plan = PairPlan<R, PARTS, PAIRS, L, S>;
    auto kern = k_blind_rotate_pair<R, PARTS, PAIRS, L, S>;
    cudaError_t e = set_smem(kern, Plan::total);
    if (e != cudaSuccess) return e;
    const int grid = (a.count + PAIRS - 1) / PAIRS;
    kern<<<grid, 128 * PAIRS, Plan::total, st>>>(kp, T, a);
    return cudaGetLastError();
}

template <int L, bool PAIR = false>
cudaError_t launch_spread(const DevParams& P, const Tables& T, const EpArgs& a, cudaStream_t st) {
    if (a.count <= 0) return cudaSuccess;
    const KParams kp = make_kparams(P);
    using Plan = SpreadPlan<L>;
    auto kern = k_blind_rotate_spread<L, PAIR>;
    cudaError_t e = set_smem(kern, Plan::total);
    if (e != cudaSuccess) return e;
    kern<<<a.count, Plan::kThreads, Plan::total, st>>>(kp, T, a);
    return cudaGetLastError();
}

template <int L, bool PAIR = false>
cudaError_t launch_spread2(const DevParams& P, const Tables& T, const EpArgs& a, cudaStream_t st) {
    if (a.count <= 0) return cudaSuccess;
    const KParams kp = make_kparams(P);
    using Plan = Spread2Plan<L>;
    auto kern = k_blind_rotate_spread2<L, PAIR>;
    cudaError_t e = set_smem(kern, Plan::request);
    if (e != cudaSuccess) return e;
    kern<<<2 * a.count, 64 * L, Plan::request, st>>>(kp, T, a);
    return cudaGetLastError();
}

// FP64: one ciphertext per cluster of two CTAs
template <int L>
cudaError_t launch_spread2_f64(const DevParams& P, const Tables& T, const EpArgs& a, cudaStream_t st) {
    if (a.count <= 0) return cudaSuccess;
    const KParams kp = make_kparams(P);
    using Plan = Spread2F64Plan<L>;
    auto kern = k_blind_rotate_spread2_f64<L>;
    cudaError_t e = set_smem(kern, Plan::request);
    if (e != cudaSuccess) return e;
    kern<<<2 * a.count, 64 * L, Plan::request, st>>>(kp, T, a);
    return cudaGetLastError();
}

// FP64: one ciphertext per cluster of eight CTAs
template <int L>
cudaError_t launch_cluster8_f64(const DevParams& P, const Tables& T, const EpArgs& a, cudaStream_t st) {
    if (a.count <= 0) return cudaSuccess;
    const KParams kp = make_kparams(P);
    using Plan = Cluster8F64Plan<L>;
    auto kern = k_blind_rotate_cluster8_f64<L>;
    cudaError_t e = set_smem(kern, Plan::total);
    if (e != cudaSuccess) return e;
    kern<<<8 * a.count, Plan::kThreads, Plan::total, st>>>(kp, T, a);
    return cudaGetLastError();
}

// FP64: one ciphertext per CTA
template <int L>
cudaError_t launch_spread_f64(const DevParams& P, const Tables& T, const EpArgs& a, cudaStream_t st) {
    if (a.count <= 0) return cudaSuccess;
    const KParams kp = make_kparams(P);
    using Plan = SpreadF64Plan<L>;
    auto kern = k_blind_rotate_spread_f64<L>;
    cudaError_t e = set_smem(kern, Plan::total);
    if (e != cudaSuccess) return e;
    kern<<<a.count, 128 * L, Plan::total, st>>>(kp, T, a);
    return cudaGetLastError();
}

// split-FP32 pair kernel with `per_cta` (1..3) ciphertexts per CTA
template <int L>
cudaError_t launch_pair_fp32(const DevParams& P, const Tables& T, const EpArgs& a, int per_cta,
                             cudaStream_t st) {
    // a 4-row ring: deeper rings (6, 8 rows) measured slower, the shared
    // memory they take comes out of the L1 cache
    if (per_cta <= 1) return launch_pair_t<float, 2, 1, L, 4>(P, T, a, st);
    if (per_cta == 2) return launch_pair_t<float, 2, 2, L, 4>(P, T, a, st);
    return launch_pair_t<float, 2, 3, L, 4>(P, T, a, st);
}

template <int SETS, int L>
cudaError_t launch_duo(const DevParams& P, const Tables& T, const EpArgs& a, cudaStream_t st) {
    if (a.count <= 0) return cudaSuccess;
    const KParams kp = make_kparams(P);
    using Plan = DuoPlan<SETS, L, 4, 2>;
    auto kern = k_blind_rotate_duo<SETS, L, 4, 2>;
    cudaError_t e = set_smem(kern, Plan::total);
    if (e != cudaSuccess) return e;
    kern<<<(a.count + 2 * SETS - 1) / (2 * SETS), kDuoThreads * SETS, Plan::total, st>>>(kp, T, a);
    return cudaGetLastError();
}

// Batched ring kernels: 4 per CTA (8 warps per SM) -- for l = 3 with a step's
// three forward transforms run together in one ciphertext's 64 threads (4.56
// ms for 608; in lane pairs two at a time 4.71 ms), for l = 2 in lane pairs
// (2.79 ms against 2.90) -- or 6 per CTA in lane pairs, transforms two at a
// time (168 registers, 12 warps per SM).  What 3 per SM can hold runs as 3
// per CTA with a step's transforms together, on more SMs with fewer warps
// each: 448 ciphertexts 4.54 -> 4.29 ms, 305 4.49 -> 4.17 ms, l = 2 448 2.78
// -> 2.68 ms.
template <int L>
cudaError_t launch_ring_batched(const DevParams& P, const Tables& T, const EpArgs& a, cudaStream_t st) {
    if (a.count <= 3 * kSmCount) return launch_ring_t<float, 2, 3, L, true, 4, L>(P, T, a, st);
    if constexpr (L == 2) return launch_duo<2, L>(P, T, a, st);
    else return launch_ring_t<float, 2, 4, L, true, 4, L>(P, T, a, st);
}
template <int L>
cudaError_t launch_ring_pairs(const DevParams& P, const Tables& T, const EpArgs& a, cudaStream_t st) {
    return launch_duo<3, L>(P, T, a, st);
}

// Up to two ciphertexts per SM: one per cluster of two SMs up to half as many
// as SMs, one per CTA up to as many, and two launches (a wave of one per CTA,
// then the rest) above.  In the pair kernel's order with l = 2 the pair kernel
// itself is the faster one from 1.5 per SM on (1.93 ms for 229 to 304, where
// two waves of one per CTA take 2.01 to 2.03 ms; l = 3: 3.22 against 3.05 ms;
// 220 with l = 2 1.80 ms in two launches).
template <int L, bool PAIR>
cudaError_t launch_low_latency(const DevParams& P, const Tables& T, const EpArgs& a, cudaStream_t st) {
    if (a.count <= kSmCount / 2) return launch_spread2<L, PAIR>(P, T, a, st);
    const int rest = a.count - kSmCount;
    if (PAIR && L == 2 && rest > kSmCount / 2) return launch_pair_fp32<L>(P, T, a, 2, st);
    if (rest <= 0 || rest > kSmCount / 2) return launch_spread<L, PAIR>(P, T, a, st);
    const cudaError_t e = launch_spread<L, PAIR>(P, T, slice_blind_rotate(P, a, 0, kSmCount), st);
    if (e != cudaSuccess) return e;
    return launch_spread2<L, PAIR>(P, T, slice_blind_rotate(P, a, kSmCount, rest), st);
}

// Automatic shape of a split-FP32 blind rotation over `count` ciphertexts.
// Measured per launch (default set): a wave of 6 per SM on
// launch_ring_pairs 6.1 ms, of 4 per SM on launch_ring_batched 4.6 ms (4.2 ms
// up to 3 per SM), whatever the fill of the wave; the cluster kernel 1.12 ms
// for up to one per two SMs; the spread kernel 1.57 ms at 1 per SM, 3.0 to 3.1
// ms for two waves.  So: whole waves of 6 per SM; a remainder of up to 2 per SM on those
// two (2.7 ms up to 1.5 per SM, where the pair kernel took 3.24 ms for any
// count of 2 per SM), of up to 4 per SM as one launch_ring_batched wave, of
// up to 5 as that wave and the rest on the low-latency kernels (5.7 or 6.1
// ms), else one more 6-per-SM wave.
//
// A remainder of more than 1 and up to 2 per SM is summed in the pair
// kernel's order, as it always was under shape 0.  fixed_order (shape 15):
// every launch sums the 2l key rows in the same order, and a ciphertext's
// result does not depend on the batch it runs in -- what a server that mixes
// requests needs.
template <int L>
cudaError_t launch_auto_fp32(const DevParams& P, const Tables& T, const EpArgs& a, cudaStream_t st,
                             bool fixed_order = false) {
    const int wave = 6 * kSmCount;
    const int full = (a.count / wave) * wave;
    const int rest = a.count - full;
    if (rest == 0 || rest > 5 * kSmCount) return launch_ring_pairs<L>(P, T, a, st);
    if (full) {
        cudaError_t e = launch_ring_pairs<L>(P, T, slice_blind_rotate(P, a, 0, full), st);
        if (e != cudaSuccess) return e;
    }
    const EpArgs tail = slice_blind_rotate(P, a, full, rest);
    if (rest > 2 * kSmCount) {
        const int most = std::min(rest, 4 * kSmCount);
        cudaError_t e = launch_ring_batched<L>(P, T, slice_blind_rotate(P, tail, 0, most), st);
        if (e != cudaSuccess || most == rest) return e;
        return launch_low_latency<L, false>(P, T, slice_blind_rotate(P, tail, most, rest - most), st);
    }
    if (rest > kSmCount && !fixed_order) return launch_low_latency<L, true>(P, T, tail, st);
    return launch_low_latency<L, false>(P, T, tail, st);
}

// Automatic shape of an FP64 blind rotation.  Every shape gives the same
// ciphertexts, so only time decides.  Measured per launch (default set): the
// eight-SM cluster kernel 6.2 ms for up to 15 ciphertexts, 10.6 ms to 32, 15.6
// ms to 48, 20.9 ms at 57; the two-SM cluster kernel 20.3 ms for up to one
// ciphertext per two SMs; the one-per-CTA kernel 29.8 ms a wave of one per SM; the 3-per-CTA kernel with
// L2-direct key reads 87.0 ms a wave of three per SM (3 waves of the former
// take 89.3 ms).  The rule takes one kernel per remainder (by these times 77 to
// 91, 153 to 228 and 305 to 380 would end sooner split between two): whole
// waves of three per SM, and a remainder of up to
// two per SM on the one-per-CTA kernel, of up to one per two SMs on the
// two-SM cluster kernel, of up to 48 on the eight-SM one.
template <int L>
cudaError_t launch_auto_fp64(const DevParams& P, const Tables& T, const EpArgs& a, cudaStream_t st) {
    const int wave = 3 * kSmCount;
    int full = (a.count / wave) * wave;
    if (a.count - full > 2 * kSmCount) full = a.count;
    if (full) {
        const cudaError_t e =
            launch_ep_t<double, 1, kEpBlindRotate, 3, L>(P, T, slice_blind_rotate(P, a, 0, full), st);
        if (e != cudaSuccess || full == a.count) return e;
    }
    const EpArgs tail = slice_blind_rotate(P, a, full, a.count - full);
    if (tail.count > kSmCount / 2) return launch_spread_f64<L>(P, T, tail, st);
    if (tail.count <= 48) return launch_cluster8_f64<L>(P, T, tail, st);
    return launch_spread2_f64<L>(P, T, tail, st);
}

// FP64: ~250 registers per thread and 2 x L exchange buffers of 9 KB per
// group, so 3 groups (192 threads) per CTA.  split-FP32: GROUPS groups.
template <int L>
cudaError_t launch_ep_l(const DevParams& P, Form f, EpMode mode, const Tables& T, const EpArgs& a,
                        int groups, cudaStream_t st) {
    if (f == kFormFp64) {
        switch (mode) {
        case kEpPlain: return launch_ep_t<double, 1, kEpPlain, 3, L>(P, T, a, st);
        case kEpMuxRotate: return launch_ep_t<double, 1, kEpMuxRotate, 3, L>(P, T, a, st);
        default:
            // 0: automatic (launch_auto_fp64); 3: L2-direct, 3 per CTA; 4:
            // shared key ring; 16: cluster kernel
            if (groups == 0) return launch_auto_fp64<L>(P, T, a, st);
            if (groups == 16) return launch_spread2_f64<L>(P, T, a, st);
            if (groups == 3) return launch_ep_t<double, 1, kEpBlindRotate, 3, L>(P, T, a, st);
            return launch_ring_t<double, 1, 4, L, true>(P, T, a, st);
        }
    }
    switch (mode) {
    case kEpPlain: return launch_products<kEpPlain, L>(P, T, a, st);
    case kEpMuxRotate: return launch_products<kEpMuxRotate, L>(P, T, a, st);
    default:
        if (groups == 0) return launch_auto_fp32<L>(P, T, a, st);
        if (groups == 15) return launch_auto_fp32<L>(P, T, a, st, true);
        if (groups == 16) return launch_spread2<L>(P, T, a, st);
        // 1, 2, 4: L2-direct key reads; 5: shared ring fed by a producer
        // warp; 6, 7, 8: shared ring fed in line by one consumer thread;
        // 9: shared ring, 4 per CTA, a step's l forward transforms run
        // together; 10: shared ring, 6 per CTA, transforms two at a time;
        // 11, 12, 13: pair kernel with 1, 2, 3 ciphertexts per CTA;
        // 15: the automatic shape in fixed summation order (no pair kernel);
        // 16: spread over a cluster of two CTAs
        if (groups >= 11 && groups <= 13) return launch_pair_fp32<L>(P, T, a, groups - 10, st);
        if (groups == 9) return launch_ring_batched<L>(P, T, a, st);
        if (groups == 10) return launch_ring_pairs<L>(P, T, a, st);
        if (groups == 14) return launch_spread<L>(P, T, a, st);
        if (groups == 1) return launch_ep_t<float, 2, kEpBlindRotate, 1, L>(P, T, a, st);
        if (groups == 2) return launch_ep_t<float, 2, kEpBlindRotate, 2, L>(P, T, a, st);
        if (groups == 4) return launch_ep_t<float, 2, kEpBlindRotate, 4, L>(P, T, a, st);
        if (groups == 5) return launch_ring_t<float, 2, 5, L, false>(P, T, a, st);
        if (groups == 7) return launch_ring_t<float, 2, 7, L, true>(P, T, a, st);
        if (groups == 8) return launch_ring_t<float, 2, 8, L, true>(P, T, a, st);
        return launch_ring_t<float, 2, 6, L, true>(P, T, a, st);
    }
}

}  // namespace

// ----------------------------------------------------------------------
// host-side tables and launchers
// ----------------------------------------------------------------------
static void sincos_2pi_frac(long k, long M, double* c, double* s) {
    k %= M;
    const long q = (4 * k) / M;
    const long r = k - q * (M / 4);
    double cr, sr;
    if (8 * r <= M) {
        const double a = 2.0 * M_PI * (double)r / (double)M;
        cr = cos(a);
        sr = sin(a);
    } else {
        const double a = 2.0 * M_PI * (double)(M / 4 - r) / (double)M;
        cr = sin(a);
        sr = cos(a);
    }
    switch (q) {
    case 0: *c = cr; *s = sr; break;
    case 1: *c = -sr; *s = cr; break;
    case 2: *c = -cr; *s = -sr; break;
    default: *c = sr; *s = -cr; break;
    }
}

void make_twiddles_host(double* h) {
    // layout of Tables: [q][t] W^(tq) | [q][j] W^(8jq) | [q][t] psi^t W^(tq) | psi^x,
    // W = e^{2 pi i/512}, psi = e^{pi i/1024}
    for (int q = 0; q < 8; ++q)
        for (int t = 0; t < 64; ++t)
            sincos_2pi_frac(t * q, 512, &h[2 * (kTabA + q * 64 + t)], &h[2 * (kTabA + q * 64 + t) + 1]);
    for (int q = 0; q < 8; ++q)
        for (int j = 0; j < 8; ++j)
            sincos_2pi_frac(8 * j * q, 512, &h[2 * (kTabB + q * 8 + j)], &h[2 * (kTabB + q * 8 + j) + 1]);
    // psi^t W^(tq) = e^{2 pi i (t + 4 t q) / 2048}
    for (int q = 0; q < 8; ++q)
        for (int t = 0; t < 64; ++t)
            sincos_2pi_frac(t + 4 * t * q, 2048, &h[2 * (kTabT + q * 64 + t)], &h[2 * (kTabT + q * 64 + t) + 1]);
    for (int x = 0; x < 512; ++x)
        sincos_2pi_frac(x, 2048, &h[2 * (kTabPsi + x)], &h[2 * (kTabPsi + x) + 1]);
}

int twiddle_table_entries() { return kTabSize; }

size_t tgsw_fft_bytes(const DevParams& P, Form f) {
    const size_t rows = (size_t)(P.k + 1) * P.l;
    if (f == kFormFp64) return rows * 2 * kHalf * sizeof(cpx<double>);
    return rows * 2 * 2 * kHalf * sizeof(cpx<float>);
}

cudaError_t launch_tgsw_to_fft(const DevParams& P, Form f, const Tables& T, const int32_t* tgsw,
                               void* out, int count, cudaStream_t st) {
    const int npoly = count * (P.k + 1) * P.l * (P.k + 1);
    if (npoly <= 0) return cudaSuccess;
    const int groups = 4;
    const size_t smem = kConvTableBytes + groups * kConvGroupBytes;
    const int grid = (npoly + groups - 1) / groups;
    cudaError_t e;
    if (f == kFormFp64) {
        e = set_smem(k_tgsw_to_fft<kFormFp64>, smem);
        if (e != cudaSuccess) return e;
        k_tgsw_to_fft<kFormFp64><<<grid, 64 * groups, smem, st>>>(T, tgsw, out, npoly, 0);
    } else {
        e = set_smem(k_tgsw_to_fft<kFormSplitFp32>, smem);
        if (e != cudaSuccess) return e;
        k_tgsw_to_fft<kFormSplitFp32><<<grid, 64 * groups, smem, st>>>(T, tgsw, out, npoly,
                                                                       P.split_bits);
    }
    return cudaGetLastError();
}

cudaError_t launch_tgsw_from_fft64(const DevParams& P, const Tables& T, const void* in,
                                   int32_t* tgsw, int count, cudaStream_t st) {
    const int npoly = count * (P.k + 1) * P.l * (P.k + 1);
    if (npoly <= 0) return cudaSuccess;
    const int groups = 4;
    const size_t smem = kConvTableBytes + groups * kConvGroupBytes;
    cudaError_t e = set_smem(k_fft64_to_tgsw, smem);
    if (e != cudaSuccess) return e;
    k_fft64_to_tgsw<<<(npoly + groups - 1) / groups, 64 * groups, smem, st>>>(T, in, tgsw, npoly);
    return cudaGetLastError();
}

cudaError_t launch_lagrange_ref_to_engine64(const double* ref, void* eng, int npoly, double scale,
                                            cudaStream_t st) {
    const int total = npoly * kHalf;
    if (total <= 0) return cudaSuccess;
    k_ref_to_engine64<<<(total + 255) / 256, 256, 0, st>>>(ref, reinterpret_cast<cpx<double>*>(eng),
                                                          npoly, scale);
    return cudaGetLastError();
}

cudaError_t launch_engine64_to_lagrange_ref(const void* eng, double* ref, int npoly, double scale,
                                            cudaStream_t st) {
    const int total = npoly * kHalf;
    if (total <= 0) return cudaSuccess;
    k_engine64_to_ref<<<(total + 255) / 256, 256, 0, st>>>(
        reinterpret_cast<const cpx<double>*>(eng), ref, npoly, scale);
    return cudaGetLastError();
}

int blind_rotate_tail_start(Form f, int groups, int count) {
    // launch_auto_fp32's whole 6-per-SM waves, when a remainder of at most 4 per
    // SM follows as its own launches.  The key switch of the full waves beside
    // it saves what SMs without a CTA of the remainder can take of it (a
    // key-switch CTA needs an SM's shared memory to itself): 950 gates 7.38 ->
    // 7.31 ms, 1,300 10.43 -> 10.38, 1,520 10.77 -> 10.75; nothing at 448 over
    // whole waves (150 of 152 SMs taken: 4,096 gates 28.97 ms either way).  A
    // remainder of 4 to 5 per SM is not split off: it leaves SMs free only in its
    // last launch (912 + 760 gates 12.38 ms, with the fork 12.32).
    if (f != kFormSplitFp32 || (groups != 0 && groups != 15)) return 0;
    const int wave = 6 * kSmCount;
    const int full = (count / wave) * wave;
    const int rest = count - full;
    return full > 0 && rest > 0 && rest <= 4 * kSmCount ? full : 0;
}

cudaError_t launch_external_product(const DevParams& P, Form f, EpMode mode, const Tables& T,
                                    const EpArgs& a, int groups, cudaStream_t st) {
    switch (P.l) {
    case 2: return launch_ep_l<2>(P, f, mode, T, a, groups, st);
    case 3: return launch_ep_l<3>(P, f, mode, T, a, groups, st);
    default: return cudaErrorInvalidValue;  // decomposition lengths 2 and 3 are built
    }
}

cudaError_t launch_gate_combine(const DevParams& P, const int32_t* gates, int32_t uniform_gate,
                                const int32_t* ca, const int32_t* cb, int32_t* out, int count,
                                cudaStream_t st) {
    if (count <= 0) return cudaSuccess;
    const size_t total = (size_t)count * (P.n + 1);
    const int blocks = (int)((total + 255) / 256 < 8192 ? (total + 255) / 256 : 8192);
    k_gate_combine<<<blocks, 256, 0, st>>>(P.n, gates, uniform_gate, ca, cb, out, count);
    return cudaGetLastError();
}

cudaError_t launch_lwe_add2_const(const int32_t* u1, const int32_t* u2, int32_t* out,
                                  int32_t width, int32_t mu, int count, cudaStream_t st) {
    if (count <= 0) return cudaSuccess;
    const size_t total = (size_t)count * width;
    int blocks = (int)((total + 255) / 256);
    if (blocks > 4096) blocks = 4096;
    k_lwe_add2_const<<<blocks, 256, 0, st>>>(u1, u2, out, width, mu, count);
    return cudaGetLastError();
}

cudaError_t launch_mul_by_xai_minus_one(const DevParams& P, const int32_t* in, const int32_t* ai,
                                        int32_t* out, int count, cudaStream_t st) {
    if (count <= 0) return cudaSuccess;
    const size_t total = (size_t)count * (P.k + 1) * kN;
    const int blocks = (int)((total + 255) / 256 < 8192 ? (total + 255) / 256 : 8192);
    k_mul_by_xai_minus_one<<<blocks, 256, 0, st>>>(in, ai, out, P.k + 1, count);
    return cudaGetLastError();
}

cudaError_t launch_extract(const DevParams& P, const int32_t* acc, int32_t* out, int count,
                           cudaStream_t st) {
    (void)P;
    if (count <= 0) return cudaSuccess;
    k_extract<<<count, 256, 0, st>>>(acc, out, count);
    return cudaGetLastError();
}

cudaError_t launch_poly_to_lagrange(const DevParams& P, const Tables& T, const int32_t* in,
                                    double* out, int count, double scale, cudaStream_t st) {
    (void)P;
    if (count <= 0) return cudaSuccess;
    const int groups = 4;
    const size_t smem = kConvTableBytes + groups * kConvGroupBytes;
    cudaError_t e = set_smem(k_poly_to_lagrange, smem);
    if (e != cudaSuccess) return e;
    k_poly_to_lagrange<<<(count + groups - 1) / groups, 64 * groups, smem, st>>>(T, in, out, count,
                                                                                 scale);
    return cudaGetLastError();
}

cudaError_t launch_lagrange_to_torus(const DevParams& P, const Tables& T, const double* in,
                                     int32_t* out, int count, cudaStream_t st) {
    (void)P;
    if (count <= 0) return cudaSuccess;
    const int groups = 4;
    const size_t smem = kConvTableBytes + groups * kConvGroupBytes;
    cudaError_t e = set_smem(k_lagrange_to_torus, smem);
    if (e != cudaSuccess) return e;
    k_lagrange_to_torus<<<(count + groups - 1) / groups, 64 * groups, smem, st>>>(T, in, out,
                                                                                  count);
    return cudaGetLastError();
}

cudaError_t launch_lagrange_addmul(const double* a, const double* b, double* acc, int npoly,
                                   int half, cudaStream_t st) {
    const size_t total = (size_t)npoly * half;
    if (total == 0) return cudaSuccess;
    k_lagrange_addmul<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(a, b, acc, total);
    return cudaGetLastError();
}

}  // namespace tfhe_gb300
