// tkd_pack.cu: the weight packer of the dense_reader path.
//
// Replaces the host conversion the reference reaches through ttnn.from_torch(dtype=bfloat8_b | bfloat4_b | bfloat16)
// in native_weight (dense_reader/linear.py:144-156) and block_float (:159-163): float32 -> block-float numbers
// (one shared 8-bit exponent per 16 consecutive output columns at one k, sign + 7 or 3 magnitude bits), by the rule of
// moe/moe8.py:134-150 (truncating alignment shift, then round to nearest even, clamp without an exponent bump, sign
// dropped for zero), and then the re-layout into the HBM stream of tkd_layout.h. Three passes, each a plain
// HBM-bound kernel:
//   1. tkd_quantise_kernel: float32 -> canonical exps [K, G] and codes [K, Npad] (the same numbers the reference's
//      tiles hold, before any re-layout; what the parity tests compare bit for bit);
//   2. tkd_emax_kernel: per group of 16 columns the largest exponent of a row with a non-zero code (a block a group);
//   3. tkd_permute_kernel: canonical -> stream, one thread per 32-bit word of the stream.
// tkd_pack_weight_kernel does all three at once and is what a weight's loading runs; the passes serve callers that hold the
// canonical numbers (int4 and ternary codes, K-block experts), and a K too long for its shared memory.
// tkd_unpack_kernel is the inverse (stream -> float32 [K, Npad]), used for the weight's read-back.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "tkd_internal.h"
#include "tkd_layout.h"

namespace {

__device__ __forceinline__ float src_at(const float* src, int orient, int64_t K, int64_t N, int64_t k, int64_t n,
                                        const float* col_div) {
    // orient 0: src is [N, K] (a torch [out, in] matrix); 1: src is [K, N]
    float v = orient == 0 ? src[n * K + k] : src[k * N + n];
    if (col_div) v = __fdiv_rn(v, col_div[n]);
    return v;
}

// One thread per (group g, k): 16 values -> one exponent byte and 16 code bytes.
__global__ void tkd_quantise_kernel(const float* __restrict__ src, int orient, int64_t K, int64_t N, int64_t npad,
                                    const float* __restrict__ col_div, int mb, uint8_t* __restrict__ exps,
                                    uint8_t* __restrict__ codes) {
    const int64_t G = npad / 16;
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t g = blockIdx.y;
    if (k >= K) return;
    uint32_t bits[16];
    uint32_t shared = 0;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const int64_t n = g * 16 + i;
        bits[i] = n < N ? __float_as_uint(src_at(src, orient, K, N, k, n, col_div)) : 0u;
        shared = max(shared, (bits[i] >> 23) & 0xFFu);
    }
    const int shift = 24 - mb;
    const uint32_t maxm = (1u << mb) - 1;
    uint32_t out[4] = {0, 0, 0, 0};
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const uint32_t e = (bits[i] >> 23) & 0xFFu;
        const uint32_t man = (bits[i] & 0x7FFFFFu) | (1u << 23);
        const uint32_t diff = shared - e;
        uint32_t m = diff > 31 ? 0u : (man >> diff);       // truncating alignment
        const uint32_t rnd = m & ((1u << shift) - 1);
        m >>= shift;
        const uint32_t tie = 1u << (shift - 1);
        m += (rnd > tie) || (rnd == tie && (m & 1u));      // nearest, ties to even
        m = min(m, maxm);                                  // no exponent bump
        if (e == 0) m = 0;                                 // zero or denormal
        const uint32_t s = m ? (bits[i] >> 31) : 0u;
        out[i >> 2] |= ((s << mb) | m) << (8 * (i & 3));
    }
    exps[k * G + g] = (uint8_t)shared;
    *reinterpret_cast<uint4*>(codes + k * npad + g * 16) = make_uint4(out[0], out[1], out[2], out[3]);
}

// bfloat16 weights: float32 -> bf16 bits (round to nearest even), canonical [K, Npad] uint16.
__global__ void tkd_tobf16_kernel(const float* __restrict__ src, int orient, int64_t K, int64_t N, int64_t npad,
                                  const float* __restrict__ col_div, uint16_t* __restrict__ codes) {
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t g = blockIdx.y;
    if (k >= K) return;
    for (int i = 0; i < 16; ++i) {
        const int64_t n = g * 16 + i;
        const float v = n < N ? src_at(src, orient, K, N, k, n, col_div) : 0.f;
        codes[k * npad + n] = __bfloat16_as_ushort(__float2bfloat16_rn(v));
    }
}

__device__ __forceinline__ bool row_nonzero(const uint8_t* codes, int64_t npad, int64_t k, int64_t g) {
    const uint4 c = *reinterpret_cast<const uint4*>(codes + k * npad + g * 16);
    return (c.x | c.y | c.z | c.w) != 0;
}

// One block per group: emax[g] = the largest exponent among its rows that hold a non-zero code (0: none). info[0] is
// OR-ed with 1 when a non-zero row's exponent lies more than TKD_ESPREAD below it (a "wide" weight). The
// block's threads share the rows of K out and reduce (maxima and minima: the order does not matter).
constexpr int kEmaxThreads = 256;
__global__ void __launch_bounds__(kEmaxThreads) tkd_emax_kernel(const uint8_t* __restrict__ exps,
                                                               const uint8_t* __restrict__ codes, int64_t K, int64_t npad,
                                                               uint8_t* __restrict__ emax, int* __restrict__ info) {
    __shared__ int shi[kEmaxThreads / 32], slo[kEmaxThreads / 32];
    const int64_t G = npad / 16, g = blockIdx.x;
    int hi = 0, lo = 255;
    for (int64_t k = threadIdx.x; k < K; k += kEmaxThreads) {
        if (!row_nonzero(codes, npad, k, g)) continue;
        const int e = exps[k * G + g];
        hi = max(hi, e);
        lo = min(lo, e);
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        hi = max(hi, __shfl_xor_sync(0xFFFFFFFFu, hi, o));
        lo = min(lo, __shfl_xor_sync(0xFFFFFFFFu, lo, o));
    }
    if ((threadIdx.x & 31) == 0) shi[threadIdx.x >> 5] = hi, slo[threadIdx.x >> 5] = lo;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < kEmaxThreads / 32; ++w) hi = max(hi, shi[w]), lo = min(lo, slo[w]);
        emax[g] = (uint8_t)hi;
        if (lo <= hi && hi - lo > TKD_ESPREAD) atomicOr(info, 1);
    }
}

// One thread per 32-bit word of the stream.
__global__ void tkd_permute_kernel(int fmt, int64_t K, int64_t npad, const uint8_t* __restrict__ exps,
                                   const void* __restrict__ codes_v, const uint8_t* __restrict__ emax,
                                   uint32_t* __restrict__ stream) {
    const int64_t words = tkd_stream_bytes(fmt, K, npad) / 4;
    const int64_t wi = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (wi >= words) return;
    const int64_t G = npad / 16;
    const int ksa = tkd_ksa(fmt), eb = tkd_exp_bytes(fmt);
    int64_t g, sa;
    int off;  // byte offset of this word inside its super-atom
    tkd_sa_owner(fmt, K, wi * 4, &g, &sa, &off);
    uint32_t word = 0;
    if (fmt == TKD_BF16) {
        const uint16_t* codes = static_cast<const uint16_t*>(codes_v);
        const int jj = off / 512, lane = (off % 512) / 16, ai = (off % 16) / 4;
        const int t = lane & 3, i = (lane >> 2) + 8 * (ai & 1);
        for (int half = 0; half < 2; ++half) {
            const int64_t k = sa * ksa + 8 * t + 4 * jj + 2 * (ai >> 1) + half;
            const uint32_t v = k < K ? codes[k * npad + g * 16 + i] : 0u;
            word |= v << (16 * half);
        }
    } else if (fmt == TKD_INT4 && off < eb) {
        // the scales of the super-atom's k32 block qq for columns g8 and g8 + 8 (exps: bf16 bits [ceil(K / 32), npad]),
        // each times 2^TKD_INT4_SCALE_EXP (exact: a bf16 keeps its significand; the product is a normal number)
        const uint16_t* sc = reinterpret_cast<const uint16_t*>(exps);
        const int g8 = (off / 4) >> 1, qq = (off / 4) & 1;
        const int64_t kg = sa * 2 + qq;
        for (int half = 0; half < 2; ++half) {
            uint32_t b = 0;
            if (kg * 32 < K) {
                const float v = __uint_as_float((uint32_t)sc[kg * npad + g * 16 + g8 + 8 * half] << 16);
                b = __float_as_uint(v * 0x1p65f) >> 16;
            }
            word |= b << (16 * half);
        }
    } else if (off < eb) {
        const uint8_t* codes = static_cast<const uint8_t*>(codes_v);
        const int per_t = fmt == TKD_BFP4 ? 4 : 2;
        const int t = (off / 4) / per_t, j = (off / 4) % per_t;
        const int qq = fmt == TKD_BFP4 ? j >> 1 : 0, jj = fmt == TKD_BFP4 ? j & 1 : j;
        for (int r = 0; r < 4; ++r) {
            const int64_t k = sa * ksa + qq * 32 + 8 * t + 4 * jj + r;
            int e = tkd_ezero(fmt);
            if (k < K && row_nonzero(codes, npad, k, g))
                e = max(tkd_ezero(fmt), (int)exps[k * G + g] - (int)emax[g] + tkd_ebias(fmt));
            word |= tkd_exp_bits(fmt, (uint32_t)e, r);
        }
    } else {
        const uint8_t* codes = static_cast<const uint8_t*>(codes_v);
        const int co = off - eb;
        const int lane = co / 16, wj = (co % 16) / 4;
        const int t = lane & 3, g8 = lane >> 2;
        if (fmt == TKD_BFP8) {
            const int jj = wj >> 1, apair = wj & 1;  // the word holds a(2 apair) and a(2 apair) + 1
            for (int odd = 0; odd < 2; ++odd)
                for (int half = 0; half < 2; ++half) {
                    const int64_t k = sa * ksa + 8 * t + 4 * jj + 2 * apair + half;
                    const uint32_t c = k < K ? codes[k * npad + g * 16 + g8 + 8 * odd] : 0u;
                    word |= tkd_code_bits(fmt, c, 8 * odd, half);
                }
        } else {
            const int qq = wj >> 1, jj = wj & 1;
            for (int ai = 0; ai < 4; ++ai)
                for (int half = 0; half < 2; ++half) {
                    const int64_t k = sa * ksa + qq * 32 + 8 * t + 4 * jj + 2 * (ai >> 1) + half;
                    const uint32_t c = k < K ? codes[k * npad + g * 16 + g8 + 8 * (ai & 1)] : 0u;
                    word |= tkd_code_bits(fmt, c, ai, half);
                }
        }
    }
    stream[wi] = word;
}

// One thread per element: canonical block-float numbers -> bf16 bits [K, npad]. Every block-float value
// +-m * 2^(e - unit) (m below 2^7, e from 1) is a bf16 value exactly, the subnormal ones included (multiples of 2^-132),
// so the float's low 16 bits are zero and its high 16 are the bf16.
__global__ void tkd_dequantise_bf16_kernel(int fmt, int64_t K, int64_t npad, const uint8_t* __restrict__ exps,
                                           const uint8_t* __restrict__ codes, uint16_t* __restrict__ out) {
    const int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (idx >= K * npad) return;
    const int64_t k = idx / npad, n = idx % npad;
    const int mb = tkd_mant_bits(fmt);
    const uint32_t c = codes[idx], m = c & ((1u << mb) - 1);
    const float v = m ? ldexpf((float)m, (int)exps[k * (npad / 16) + (n >> 4)] - tkd_unit_exp(fmt)) : 0.f;
    out[idx] = (uint16_t)((__float_as_uint(v) >> 16) | (((c >> mb) & 1u) << 15));
}

// One thread per element: stream -> float32 [K, npad].
__global__ void tkd_unpack_kernel(int fmt, int64_t K, int64_t npad, const uint8_t* __restrict__ stream,
                                  const uint8_t* __restrict__ emax, float* __restrict__ out) {
    const int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (idx >= K * npad) return;
    const int64_t k = idx / npad, n = idx % npad;
    const TkdLoc L = tkd_locate(fmt, K, k, n);
    float v;
    if (fmt == TKD_BF16) {
        const uint16_t b = *reinterpret_cast<const uint16_t*>(stream + L.code_word);
        v = __uint_as_float((uint32_t)b << 16);
    } else {
        const int mb = tkd_mant_bits(fmt);
        const uint32_t w = *reinterpret_cast<const uint32_t*>(stream + L.code_word);
        const uint32_t c = tkd_code_from_word(fmt, w, L.rot, L.half);
        const uint32_t m = c & ((1u << mb) - 1);
        const uint32_t ew = *reinterpret_cast<const uint32_t*>(stream + L.exp_word);
        if (fmt == TKD_INT4) {
            // q * s: the stored scale is s * 2^65
            const float s65 = __uint_as_float(((ew >> (16 * L.exp_r)) & 0xFFFFu) << 16);
            v = (float)m * (s65 * 0x1p-65f);
        } else {
            const int e = (int)tkd_exp_from_word(fmt, ew, L.exp_r) + (int)emax[n >> 4] - tkd_ebias(fmt);
            v = m ? ldexpf((float)m, e - tkd_unit_exp(fmt)) : 0.f;
        }
        if ((c >> mb) & 1u) v = -v;
    }
    out[idx] = v;
}

// The three passes above in one, for float32 -> stream at load time: a CTA owns a group of 16 columns and all of K, and a
// warp takes a super-atom at a time. A lane loads exactly the numbers whose codes it will write (8 consecutive k of columns
// g and g + 8 per block of 32 k: the fragment layout of tkd_layout.h), the shared exponents of its 8 k come from three
// shuffles over the lanes of the same k, and its 16 bytes of codes go straight to the stream. Only the exponents wait for
// the group's largest: two bytes a k in shared memory, written as the stream's words at the end. A row of the group holds a
// non-zero code exactly when its shared exponent is not zero (the largest value's implicit bit survives the rounding).
// SCALE 1: the columns are divided by col_div first; 2: by their largest magnitude rounded up to bf16 (native_weight's
// col_scale), found by a first walk over the CTA's 16 columns, whose second reading then comes from L2, and written out.
// Bound: HBM. [14336, 4096] float32 to bfloat4_b (235 MB in, 33 MB out): tkd_quantise, the emax and the permute pass 410 us
// together (1 byte a weight of codes written and read back, uncoalesced loads of the [N, K] matrix); here 54 us without
// column scales (5.0 TB/s), 84 with its own.
// threads of a CTA: with the columns' own scales two large CTAs an SM (77 MB of the matrix between the two readings: it stays
// in the 126 MB L2), else as many as fit
__host__ __device__ constexpr int pack_threads(int scale) { return scale == 2 ? 512 : 256; }

// The largest of three magnitudes, a NaN if there is one: one operation for two values, where an AND and a maximum each were four
// on the half-rate integer pipe, which the kernel keeps busy (a [14336, 4096] call with its own scales: bfloat8_b 126 to 113 us,
// bfloat4_b 107 to 105).
__device__ __forceinline__ float max3_abs(float a, float b, float c) {
    float d;
    asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// |v|'s bits rounded up to bf16, as a float (linear.bf16_ceil), of at least 1e-8
__device__ __forceinline__ float pack_col_scale(uint32_t bits) {
    const float a = __uint_as_float(bits), s = a < 1e-8f ? 1e-8f : a;  // (a NaN stays)
    const float down = __bfloat162float(__float2bfloat16_rn(s));
    return down >= s ? down : __uint_as_float(__float_as_uint(down) + 0x10000u);
}

// One value's code in place: sign at bit 15, the magnitude from bit `p` (0 for 7 bits, 4 for 3), by the rule of
// tkd_quantise_kernel. Rounding to nearest even is one addition: half less one, plus the kept part's last bit.
template <int FMT>
__device__ __forceinline__ uint32_t pack_code(uint32_t bits, uint32_t shared) {
    constexpr int mb = FMT == TKD_BFP8 ? 7 : 3, shift = 24 - mb, p = FMT == TKD_BFP8 ? 0 : 4;
    const uint32_t e = (bits >> 23) & 0xFFu;
    uint32_t m = ((bits & 0x7FFFFFu) | 0x800000u) >> min(shared - e, 31u);
    m = (m + ((1u << (shift - 1)) - 1u) + ((m >> shift) & 1u)) >> shift;
    m = e ? min(m, (1u << mb) - 1u) : 0u;
    return m ? ((bits >> 16) & 0x8000u) | (m << p) : 0u;
}

// The codes of two values (k even in the low half) in floating point, six instructions a value instead of sixteen on the
// half-rate integer pipe: y = |v| / the code's unit (s, a power of two, so exact); the alignment's truncation is y - 2^mb
// rounded down (its last place is the one the rule keeps, and a y of 2^(mb - 1) or more, not shifted, is exact); adding
// 1.5 * 2^23 + 2^mb rounds that to the nearest integer, ties to even, in the sum's low bits. Denormals are flushed to the
// rule's zero. For shared exponents of 8 to 254, or 0.
template <int FMT>
__device__ __forceinline__ uint32_t pack_pair(float v0, float v1, float s0, float s1) {
    constexpr float top = FMT == TKD_BFP8 ? 128.f : 8.f;
    float z[2];
    const float v[2] = {v0, v1}, s[2] = {s0, s1};
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        float y;
        asm("{\n\t.reg .f32 a;\n\tabs.ftz.f32 a, %1;\n\tmul.ftz.f32 %0, a, %2;\n\t}" : "=f"(y) : "f"(v[i]), "f"(s[i]));
        z[i] = __fadd_rn(__fadd_rd(fminf(y, top - 1.f), -top), 12582912.f + top);
    }
    const uint32_t m = __byte_perm(__float_as_uint(z[0]), __float_as_uint(z[1]), 0x5410);
    const uint32_t sign = __byte_perm(__float_as_uint(v0), __float_as_uint(v1), 0x7632) & (m + 0x7FFF7FFFu) & 0x80008000u;
    return FMT == TKD_BFP8 ? m | sign : m * 16u + sign;
}

template <int FMT, int ORIENT, int SCALE>
__global__ void __launch_bounds__(pack_threads(SCALE)) tkd_pack_weight_kernel(const float* __restrict__ src, int64_t ld, int K, int64_t N,
                                                                       const float* __restrict__ col_div,
                                                                       uint16_t* __restrict__ scale_out, uint8_t* __restrict__ stream,
                                                                       uint8_t* __restrict__ emax, int* info) {
    constexpr int KSA = FMT == TKD_BFP4 ? 64 : 32, XB = KSA / 32, EB = FMT == TKD_BFP8 ? 32 : FMT == TKD_BFP4 ? 64 : 0;
    constexpr int kPackThreads = pack_threads(SCALE), kPackWarps = kPackThreads / 32;
    extern __shared__ __align__(16) uint8_t exps[];  // the shared exponent of every k, 16 bits each, from bit 7 (not for bf16)
    __shared__ uint32_t cmax[kPackWarps][16];
    __shared__ float cdiv[16];
    __shared__ int shi[kPackWarps], slo[kPackWarps];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int64_t grp = blockIdx.x, n0 = grp * 16 + g, n1 = n0 + 8;
    const bool in0 = n0 < N, in1 = n1 < N;
    const int nsa = (K + KSA - 1) / KSA;
    // 8 consecutive k of one column
    auto load8 = [&](float (&v)[8], int64_t n, bool in, int k) {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = 0.f;
        if (!in || k >= K) return;
        if constexpr (ORIENT == 0) {
            const float4* s = reinterpret_cast<const float4*>(src + n * ld + k);
            const float4 a = __ldg(s), b = __ldg(s + 1);
            v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
        } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = __ldg(src + (int64_t)(k + i) * ld + n);
        }
    };
    float d0 = 1.f, d1 = 1.f, r0 = 1.f, r1 = 1.f;
    bool slow = SCALE == 1;  // divide by the division
    // (scales of one, for a caller that wants some beside undivided columns)
    if (SCALE == 0 && scale_out && tid < 16 && grp * 16 + tid < N) scale_out[grp * 16 + tid] = 0x3F80;
    if constexpr (SCALE == 1) {
        if (in0) d0 = col_div[n0];
        if (in1) d1 = col_div[n1];
    } else if constexpr (SCALE == 2) {
        float f0 = 0.f, f1 = 0.f;
#pragma unroll 2  // (four need 75 registers: one CTA an SM)
        for (int b = warp; b < K / 32; b += kPackWarps) {
            float v0[8], v1[8];
            load8(v0, n0, in0, 32 * b + 8 * t);
            load8(v1, n1, in1, 32 * b + 8 * t);
#pragma unroll
            for (int i = 0; i < 8; i += 2) f0 = max3_abs(f0, v0[i], v0[i + 1]), f1 = max3_abs(f1, v1[i], v1[i + 1]);
        }
        uint32_t m0 = __float_as_uint(f0), m1 = __float_as_uint(f1);  // (magnitudes order as their bits do, a NaN above all)
#pragma unroll
        for (int o = 1; o < 4; o <<= 1) {
            m0 = max(m0, __shfl_xor_sync(0xFFFFFFFFu, m0, o));
            m1 = max(m1, __shfl_xor_sync(0xFFFFFFFFu, m1, o));
        }
        if (t == 0) cmax[warp][g] = m0, cmax[warp][g + 8] = m1;
        __syncthreads();
        if (tid < 16) {
            uint32_t m = 0;
#pragma unroll
            for (int w = 0; w < kPackWarps; ++w) m = max(m, cmax[w][tid]);
            const float c = pack_col_scale(m);
            cdiv[tid] = c;
            if (grp * 16 + tid < N) scale_out[grp * 16 + tid] = __bfloat16_as_ushort(__float2bfloat16_rn(c));
        }
        __syncthreads();
        d0 = cdiv[g], d1 = cdiv[g + 8];
        r0 = __frcp_rn(d0), r1 = __frcp_rn(d1);
        slow = __any_sync(0xFFFFFFFFu, !(d0 < 0x1p60f) || !(d1 < 0x1p60f));
    }
    for (int sa = warp; sa < nsa; sa += kPackWarps) {
        uint8_t* dst = stream + tkd_sa_offset(FMT, K, grp, sa) + EB + lane * 16;
        float v[2][XB][8];
#pragma unroll
        for (int q = 0; q < XB; ++q) {
            load8(v[0][q], n0, in0, sa * KSA + 32 * q + 8 * t);
            load8(v[1][q], n1, in1, sa * KSA + 32 * q + 8 * t);
        }
        if constexpr (SCALE != 0) {
            // (own scales) v / d correctly rounded: q = v r, r the rounded reciprocal, then q + (v - q d) r (P. Markstein, IBM J. Res.
            // Dev. 34, 1990). q is within 1.5 units of its last place, d has 8 significant bits: v - q d is exact, the last sum
            // is v / d within 2^-23 units, and a quotient by such a d lies at least 2^-9 units from where rounding changes.
            // It needs v - q d in the normal numbers: a block whose largest quotients lie near the denormals is divided below.
            if (SCALE == 2 && FMT != TKD_BF16 && !slow) {
#pragma unroll
                for (int q = 0; q < XB; ++q)
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float x = v[0][q][i] * r0, y = v[1][q][i] * r1;
                        v[0][q][i] = fmaf(fmaf(-x, d0, v[0][q][i]), r0, x), v[1][q][i] = fmaf(fmaf(-y, d1, v[1][q][i]), r1, y);
                    }
            } else {
#pragma unroll
                for (int q = 0; q < XB; ++q)
#pragma unroll
                    for (int i = 0; i < 8; ++i) v[0][q][i] = __fdiv_rn(v[0][q][i], d0), v[1][q][i] = __fdiv_rn(v[1][q][i], d1);
            }
        }
        uint32_t words[4];
#pragma unroll
        for (int q = 0; q < XB; ++q) {
            if constexpr (FMT == TKD_BF16) {
                uint32_t b[2][4];  // the column's pairs of k
#pragma unroll
                for (int c = 0; c < 2; ++c)
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        b[c][i] = (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(v[c][q][2 * i])) |
                                  ((uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(v[c][q][2 * i + 1])) << 16);
#pragma unroll
                for (int jj = 0; jj < 2; ++jj)
                    *reinterpret_cast<uint4*>(dst + 512 * jj) = make_uint4(b[0][2 * jj], b[1][2 * jj], b[0][2 * jj + 1], b[1][2 * jj + 1]);
            } else {
                // the largest upper halves (exponent and seven bits) of the 16 columns at each k, two k to a word
                uint32_t both[4];
                auto maxima = [&]() {
                    uint32_t odd = 0;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        uint32_t w[2];
#pragma unroll
                        for (int c = 0; c < 2; ++c)
                            w[c] = __byte_perm(__float_as_uint(v[c][q][2 * i]), __float_as_uint(v[c][q][2 * i + 1]), 0x7632) & 0x7FFF7FFFu;
                        both[i] = __vmaxu2(w[0], w[1]);
#pragma unroll
                        for (int o = 4; o < 32; o <<= 1) both[i] = __vmaxu2(both[i], __shfl_xor_sync(0xFFFFFFFFu, both[i], o));
                        // an exponent of 1 to 7, or of 255, leaves pack_pair's scale outside the normal numbers; (own scales)
                        // one below 100 may come of a quotient that was not exact, unless the largest upper half is zero: then all
                        // are zeros by the rule, exact or not. (As they counted among the others, the columns that pad N to a
                        // panel's 128 took the division for every number: [2912, 1376] to bfloat8_b 20.5 us for 8.9 without scales.)
                        if constexpr (SCALE == 2) {
                            const uint32_t z0 = both[i] & 0xFFFFu, z1 = both[i] >> 16, low = 100u << 7;
                            odd |= (z0 - 1u < low - 1u) | (z1 - 1u < low - 1u);
                        }
                        both[i] &= 0x7F807F80u;
                        const uint32_t e0 = both[i] & 0xFFFFu, e1 = both[i] >> 16, low = 8u << 7;
                        if constexpr (SCALE != 2) odd |= (e0 - 1u < low - 1u) | (e1 - 1u < low - 1u);
                        odd |= (e0 == 0x7F80u) | (e1 == 0x7F80u);
                    }
                    return __any_sync(0xFFFFFFFFu, odd) != 0;
                };
                bool odd = maxima();
                if (SCALE == 2 && odd && !slow) {
                    load8(v[0][q], n0, in0, sa * KSA + 32 * q + 8 * t);
                    load8(v[1][q], n1, in1, sa * KSA + 32 * q + 8 * t);
#pragma unroll
                    for (int i = 0; i < 8; ++i) v[0][q][i] = __fdiv_rn(v[0][q][i], d0), v[1][q][i] = __fdiv_rn(v[1][q][i], d1);
                    (void)maxima();
                }
                if (g == 0) *reinterpret_cast<uint4*>(exps + (sa * KSA + 32 * q + 8 * t) * 2) = make_uint4(both[0], both[1], both[2], both[3]);
                uint32_t r[2][4];  // (column g or g + 8, pair of k): a fragment register
                if (!odd) {
                    constexpr uint32_t unit = (uint32_t)(253 + (FMT == TKD_BFP8 ? 7 : 3)) << 23;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float s0 = __uint_as_float(unit - (both[i] << 16)), s1 = __uint_as_float(unit - (both[i] & 0xFFFF0000u));
#pragma unroll
                        for (int c = 0; c < 2; ++c) r[c][i] = pack_pair<FMT>(v[c][q][2 * i], v[c][q][2 * i + 1], s0, s1);
                    }
                } else {
#pragma unroll
                    for (int c = 0; c < 2; ++c)
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            r[c][i] = pack_code<FMT>(__float_as_uint(v[c][q][2 * i]), (both[i] >> 7) & 0xFFu) |
                                      (pack_code<FMT>(__float_as_uint(v[c][q][2 * i + 1]), both[i] >> 23) << 16);
                }
                if constexpr (FMT == TKD_BFP8) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) words[i] = r[0][i] | tkd_rotl(r[1][i], 8);
                } else {
#pragma unroll
                    for (int jj = 0; jj < 2; ++jj)
                        words[2 * q + jj] = r[0][2 * jj] | (r[1][2 * jj] >> 4) | tkd_rotl(r[0][2 * jj + 1] | (r[1][2 * jj + 1] >> 4), 8);
                }
            }
        }
        if constexpr (FMT != TKD_BF16) *reinterpret_cast<uint4*>(dst) = make_uint4(words[0], words[1], words[2], words[3]);
    }
    if constexpr (FMT != TKD_BF16) {
        __syncthreads();
        uint32_t hi = 0, lo = 255;
        for (int i = tid; i < nsa * KSA; i += kPackThreads) {
            const uint32_t sh = *reinterpret_cast<const uint16_t*>(exps + 2 * i) >> 7;
            hi = max(hi, sh), lo = min(lo, sh ? sh : 255u);
        }
        hi = __reduce_max_sync(0xFFFFFFFFu, hi), lo = __reduce_min_sync(0xFFFFFFFFu, lo);
        if (lane == 0) shi[warp] = (int)hi, slo[warp] = (int)lo;
        __syncthreads();
        int top = 0, low = 255;
#pragma unroll
        for (int w = 0; w < kPackWarps; ++w) top = max(top, shi[w]), low = min(low, slo[w]);
        if (tid == 0) {
            emax[grp] = (uint8_t)top;
            if (low <= top && top - low > TKD_ESPREAD) *static_cast<volatile int*>(info) = 1;
        }
        // the exponent words: word (t, j) of a super-atom covers k = 32 (j / 2) + 8 t + 4 (j % 2) .. + 3
        constexpr int PT = 2 * XB, PW = 4 * PT;
        for (int i = tid; i < nsa * PW; i += kPackThreads) {
            const int sa = i / PW, wi = i % PW, wt = wi / PT, j = wi % PT;
            const uint2 e4 = *reinterpret_cast<const uint2*>(exps + 2 * (sa * KSA + 32 * (j >> 1) + 8 * wt + 4 * (j & 1)));
            uint32_t word = 0;
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int sh = (int)(((r & 2 ? e4.y : e4.x) >> (16 * (r & 1) + 7)) & 0xFFu);
                const int e = sh ? max(tkd_ezero(FMT), sh - top + tkd_ebias(FMT)) : tkd_ezero(FMT);
                word |= tkd_exp_bits(FMT, (uint32_t)e, r);
            }
            *reinterpret_cast<uint32_t*>(stream + tkd_sa_offset(FMT, K, grp, sa) + wi * 4) = word;
        }
    }
}

template <int FMT, int ORIENT>
int launch_pack_weight(const float* src, int64_t ld, int64_t K, int64_t N, int64_t npad, const float* col_div, uint16_t* scale_out,
                       bool unit, void* packed, uint8_t* emax, int* info, cudaStream_t st) {
    const size_t smem = FMT == TKD_BF16 ? 0 : (size_t)(K + 63) / 64 * 128;
    auto kern = scale_out && !unit ? tkd_pack_weight_kernel<FMT, ORIENT, 2>
                          : col_div ? tkd_pack_weight_kernel<FMT, ORIENT, 1> : tkd_pack_weight_kernel<FMT, ORIENT, 0>;
    if (smem > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
    }
    kern<<<(unsigned)(npad / 16), pack_threads(scale_out && !unit ? 2 : 0), smem, st>>>(src, ld, (int)K, N, col_div, scale_out, static_cast<uint8_t*>(packed), emax, info);
    return (int)cudaGetLastError();
}

}  // namespace

int tkd_launch_pack_weight(int fmt, const float* src, int orient, int64_t ld, int64_t K, int64_t N, int64_t npad, const float* col_div,
                           uint16_t* scale_out, bool unit, void* packed, uint8_t* emax, int* info, cudaStream_t st) {
    auto go = [&](auto f) {
        constexpr int F = decltype(f)::value;
        return orient == 0 ? launch_pack_weight<F, 0>(src, ld, K, N, npad, col_div, scale_out, unit, packed, emax, info, st)
                           : launch_pack_weight<F, 1>(src, ld, K, N, npad, col_div, scale_out, unit, packed, emax, info, st);
    };
    return fmt == TKD_BFP8 ? go(std::integral_constant<int, TKD_BFP8>{}) : fmt == TKD_BFP4 ? go(std::integral_constant<int, TKD_BFP4>{})
                                                                                           : go(std::integral_constant<int, TKD_BF16>{});
}

int tkd_launch_quantise(int fmt, const float* src, int orient, int64_t K, int64_t N, int64_t npad,
                        const float* col_div, uint8_t* exps, void* codes, cudaStream_t st) {
    dim3 grid((unsigned)((K + 127) / 128), (unsigned)(npad / 16));
    if (fmt == TKD_BF16)
        tkd_tobf16_kernel<<<grid, 128, 0, st>>>(src, orient, K, N, npad, col_div, static_cast<uint16_t*>(codes));
    else
        tkd_quantise_kernel<<<grid, 128, 0, st>>>(src, orient, K, N, npad, col_div, tkd_mant_bits(fmt), exps,
                                                  static_cast<uint8_t*>(codes));
    return (int)cudaGetLastError();
}

int tkd_launch_permute(int fmt, int64_t K, int64_t npad, const uint8_t* exps, const void* codes, uint8_t* emax,
                       int* info, void* stream, cudaStream_t st) {
    const int64_t G = npad / 16;
    if (fmt != TKD_BF16 && fmt != TKD_INT4) {
        tkd_emax_kernel<<<(unsigned)G, kEmaxThreads, 0, st>>>(exps, static_cast<const uint8_t*>(codes), K, npad, emax, info);
    }
    const int64_t words = tkd_stream_bytes(fmt, K, npad) / 4;
    tkd_permute_kernel<<<(unsigned)((words + 255) / 256), 256, 0, st>>>(fmt, K, npad, exps, codes, emax,
                                                                       static_cast<uint32_t*>(stream));
    return (int)cudaGetLastError();
}

int tkd_launch_dequantise_bf16(int fmt, int64_t K, int64_t npad, const uint8_t* exps, const void* codes, void* out,
                               cudaStream_t st) {
    const int64_t n = K * npad;
    tkd_dequantise_bf16_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(fmt, K, npad, exps, static_cast<const uint8_t*>(codes),
                                                                            static_cast<uint16_t*>(out));
    return (int)cudaGetLastError();
}

int tkd_launch_unpack(int fmt, int64_t K, int64_t npad, const void* stream, const uint8_t* emax, float* out,
                      cudaStream_t st) {
    const int64_t n = K * npad;
    tkd_unpack_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(fmt, K, npad, static_cast<const uint8_t*>(stream),
                                                                  emax, out);
    return (int)cudaGetLastError();
}
