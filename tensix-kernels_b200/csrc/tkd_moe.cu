// tkd_moe.cu: the mixture-of-experts layer's two matmuls over the chosen experts only, for sm_100a. They take the
// place of the reference's gate_up / down and gate_up_rows / down_rows (moe/moe8.py:710-911, 928-1136; kernels
// moe_gu_reader.cpp, moe_gu_compute.cpp, moe_gu_writer.cpp, moe_dn_reader.cpp, moe_dn_compute.cpp, moe_dn_writer.cpp
// and kernels/moe8_rows.h for the union of the rows' experts).
//
// Every expert's weight is a bfloat4_b stream of tkd_layout.h (tkd_pack), all experts back to back, so the kernel
// finds a chosen expert by its id alone: the ids are read on the device and nothing goes to the host. What a call reads
// is small (k experts of a few MB) and scattered, so instead of the persistent ring of tkd_stream_kernel.cuh this is a plain grid of
// warps that each take a run of super-atoms of one group of 16 columns: the run's weights and its inputs come into the warp's own
// shared memory by bulk copies, all asked for as soon as the expert's id is known, and the decode is the stream kernel's (block_mma).
// The layer is a chain of latencies (the ids, the weights from DRAM, the sums, the launch): as loads into registers, four super-atoms
// at a time behind a block's copy of the inputs, gate_up took 7.9 us of a layer of 8 experts of 2048 x 1536, and down, whose slots met
// through L2 by an atomic, 6.8.
//   gate_up: a CTA is 16 columns of a gate tile and the same 16 of its up tile of one slot's expert, two runs each: it finishes 16
//            outputs, h = routing weight * act(x G + b) * (x U + b), rounded to bf16 once.
//   down:    a CTA is 16 columns of y, two runs of every slot's expert: the slots' sums are added in slot order in shared memory.
// Several rows (by_union): tkd_moe_rows.cuh.
#include "tkd_moe_rows.cuh"

namespace {

constexpr int kMoeSplit = 2;  // runs of K a group
constexpr int kMoeHalf = 8;   // super-atoms of a half of a warp's buffer
constexpr int kMoeCols = 32;  // columns a counter of the workspace stands for

struct MoeParams {
    const uint8_t* w;
    const uint8_t* emax;
    int64_t wbytes;
    int E, K, N, npad;
    const uint16_t* x;
    const void* ids;
    int ids32;
    const uint16_t* rw;
    int slots, act;
    const uint16_t* bias;
    uint16_t* out;
    int* status;
    uint32_t mul16, mul128;
};

__device__ __forceinline__ uint32_t moe_id(const MoeParams& p, int64_t i) {
    return p.ids32 ? static_cast<const uint32_t*>(p.ids)[i] : static_cast<const uint16_t*>(p.ids)[i];
}
// a column sum in the stream's units -> its value (tkd_layout.h: 2^tkd_out_exp, in two factors that are normal floats)
__device__ __forceinline__ float moe_scale(float v, int ebyte) {
    const int e = tkd_out_exp(TKD_BFP4, ebyte), e1 = e / 2, e2 = e - e1;
    return v * __uint_as_float((uint32_t)(e1 + 127) << 23) * __uint_as_float((uint32_t)(e2 + 127) << 23);
}
// Bytes of a warp's buffer: two halves of weights and of the inputs for them.
template <int FMT>
constexpr int kMoeHalfBytes = kMoeHalf * (Fmt<FMT>::SAB + Fmt<FMT>::KSA * 2);

// A warp's run of super-atoms of a group, through its buffer `buf` and its two barriers: the sums in acc. st: halves before this run.
// xs: the inputs at k = 0. false: a wait gave up.
template <int FMT>
__device__ __forceinline__ bool moe_run(const MoeParams& p, float (&acc)[2][1][4], const uint8_t* wb, int group, int sa0, int sa1,
                                        const uint16_t* xs, uint32_t buf, uint32_t bars, uint32_t& st, const uint2 sh) {
    using F = Fmt<FMT>;
    constexpr int XB = F::KSA * 2;  // bytes of x a super-atom
    const int lane = threadIdx.x & 31, t = lane & 3;
    const int halves = (sa1 - sa0 + kMoeHalf - 1) / kMoeHalf;
    auto issue = [&](int h) {
        const uint32_t q = (st + h) & 1, to = buf + q * kMoeHalfBytes<FMT>, bar = bars + 8 * q;
        const int a = sa0 + h * kMoeHalf, b = min(sa1, a + kMoeHalf);
        const uint32_t xbytes = (uint32_t)(min(b * F::KSA, p.K) - a * F::KSA) * 2;
        mbar_expect_tx(bar, (b - a) * F::SAB + xbytes);
        for (int sa = a; sa < b;) {  // (a group's super-atoms lie back to back inside a chunk)
            const int end = min(b, (sa | (F::SUBSA - 1)) + 1);
            bulk_g2s(to + (sa - a) * F::SAB, wb + tkd_sa_offset(FMT, p.K, group, sa), (end - sa) * F::SAB, bar);
            sa = end;
        }
        bulk_g2s(to + kMoeHalf * F::SAB, xs + a * F::KSA, xbytes, bar);
    };
    if (lane == 0) {
        issue(0);
        if (halves > 1) issue(1);
    }
    __syncwarp();
    for (int h = 0; h < halves; ++h) {
        const uint32_t q = (st + h) & 1, from = buf + q * kMoeHalfBytes<FMT>, x0 = from + kMoeHalf * F::SAB + 16 * t;
        if (!mbar_wait(bars + 8 * q, ((st + h) >> 1) & 1, p.status)) {
            for (uint32_t i = 0; h + 1 < halves && i < 64; ++i)  // (the copies in flight land before the warp goes)
                if (mbar_try_wait(bars + 8 * (q ^ 1), ((st + h + 1) >> 1) & 1)) break;
            return false;
        }
        const int a = sa0 + h * kMoeHalf, n = min(sa1 - a, kMoeHalf);
        if (FMT == TKD_BFP4 && (a + n) * F::KSA > p.K) {  // (a K that ends inside a super-atom: zeros after it)
            if (lane < 4) asm volatile("st.shared.v4.u32 [%0], {%1,%1,%1,%1};" ::"r"(x0 + n * XB - 64), "r"(0u) : "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // (before the next run's copies)
            __syncwarp();
        }
        auto one = [&](int b) {
            const uint32_t s = from + b * F::SAB, x = x0 + b * XB;
            if constexpr (FMT == TKD_BFP4) {
                const uint4 ev = lds128(s + t * 16), cv = lds128(s + 64 + lane * 16);
#pragma unroll
                for (int qq = 0; qq < 2; ++qq) {
                    const uint32_t cw[4] = {qq ? cv.z : cv.x, qq ? cv.w : cv.y, 0u, 0u}, ew[2] = {qq ? ev.z : ev.x, qq ? ev.w : ev.y};
                    const uint4 xv[1] = {lds128(x + 64 * qq)};
                    block_mma<TKD_BFP4, 1, 2>(acc, cw, ew, xv, sh);
                }
            } else {  // (bf16: the A fragments of the super-atom's two mmas as they are)
                const uint4 wa = lds128(s + lane * 16), wc = lds128(s + 512 + lane * 16), xv = lds128(x);
                mma_bf16(acc[0][0], wa.x, wa.y, wa.z, wa.w, xv.x, xv.y);
                mma_bf16(acc[1][0], wc.x, wc.y, wc.z, wc.w, xv.z, xv.w);
            }
        };
        if (n == kMoeHalf) {
#pragma unroll
            for (int b = 0; b < kMoeHalf; ++b) one(b);
        } else {
#pragma unroll 2
            for (int b = 0; b < n; ++b) one(b);
        }
        __syncwarp();
        if (lane == 0 && h + 2 < halves) issue(h + 2);
    }
    st += halves;
    return true;
}

// One row. FMT: the experts' stream format (bfloat4_b, or bf16 for a pack held exactly). DOWN: the down matmul.
template <int FMT, bool DOWN>
__global__ void __launch_bounds__(DOWN ? 512 : 128, DOWN ? 1 : 4) tkd_moe_kernel(const MoeParams p) {
    using F = Fmt<FMT>;  // (k and bytes of a super-atom, super-atoms of a group in a chunk)
    extern __shared__ __align__(128) uint8_t moe_dsm[];
    __shared__ uint64_t s_bars[2 * 16];
    __shared__ int s_e[DOWN ? 17 : 1];  // down: a slot's exponent byte, -1 without an expert
    __shared__ float red[DOWN ? 17 : 1][kMoeSplit][DOWN ? 16 : 32];  // [slot][run][column]
    // (the warp's number by a shuffle, as in tkd_narrow_kernel: gate_up of 8 of 128 experts, 2048 -> 2 x 768, 6.3 us without, 6.0 so, down 3.76
    // and 3.72)
    const int tid = threadIdx.x, warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0), lane = tid & 31, g = lane >> 2, t = lane & 3;
    const uint32_t buf = smem_u32(moe_dsm) + warp * 2 * kMoeHalfBytes<FMT>, bars = smem_u32(s_bars) + warp * 16;
    if (lane == 0) {
        mbar_init(bars, 1), mbar_init(bars + 8, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    // (launched as a programmatic dependent: nothing the kernels before wrote is read above the wait, and the kernel after may bring
    // its CTAs in while this one runs: it waits at the same place)
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");

    const int u = blockIdx.x, nsa = (p.K + F::KSA - 1) / F::KSA, per = (nsa + kMoeSplit - 1) / kMoeSplit;
    const uint2 sh = make_uint2(p.mul16, p.mul128);
    uint32_t st = 0;
    // the sums of group `group` of expert e over run ksp, its inputs from xs on, to d: columns g and g + 8
    auto run = [&](int e, int group, int ksp, const uint16_t* xs, float* d) {
        float acc[2][1][4] = {};
        const int sa0 = min(ksp * per, nsa), sa1 = min(nsa, sa0 + per);
        if (e >= 0 && sa0 < sa1) moe_run<FMT>(p, acc, p.w + (int64_t)e * p.wbytes, group, sa0, sa1, xs, buf, bars, st, sh);
        // (every column of D is the one row's; its first is kept: lanes with t = 0 hold columns g and g + 8 of the weight)
        if (t == 0) d[g] = acc[0][0][0] + acc[1][0][0], d[g + 8] = acc[0][0][2] + acc[1][0][2];
    };
    auto expert = [&](int q) {
        const uint32_t id = moe_id(p, q);
        return id < (uint32_t)p.E ? (int)id : -1;
    };
    if constexpr (!DOWN) {
        // unit u is half hf = u & 1 of the tile pair j = u >> 1: columns hf * 16 .. + 15 of gate tile j (warps gi 0) and of up tile j
        // (gi 1), 16 outputs
        const int q = blockIdx.y, e = expert(q), gi = warp & 1, j = u >> 1, hf = u & 1;
        int eg = 0, eu = 0;
        float w1 = 0.f, bg = 0.f, bu = 0.f;
        if (tid < 16 && e >= 0) {  // (asked for ahead of the weights' wait)
            w1 = bf16_bits_to_f32(p.rw[q]);  // the slot's routing weight
            if constexpr (FMT == TKD_BFP4) {
                const uint8_t* emx = p.emax + (int64_t)e * (p.npad / 16) + j * 4 + hf;
                eg = emx[0], eu = emx[2];
            }
            if (p.bias) {
                const uint16_t* b = p.bias + (int64_t)e * p.npad + j * 64 + hf * 16 + tid;
                bg = bf16_bits_to_f32(b[0]), bu = bf16_bits_to_f32(b[32]);
            }
        }
        run(e, j * 4 + 2 * gi + hf, warp >> 1, p.x, &red[0][warp >> 1][gi * 16]);
        __syncthreads();
        if (tid < 16) {
            float val = 0.f;
            if (e >= 0) {
                float gt = red[0][0][tid] + red[0][1][tid], up = red[0][0][16 + tid] + red[0][1][16 + tid];
                if constexpr (FMT == TKD_BFP4) gt = moe_scale(gt, eg), up = moe_scale(up, eu);
                val = moe_glu(gt + bg, up + bu, p.act) * w1;
            }
            p.out[(int64_t)q * (p.N / 2) + j * 32 + hf * 16 + tid] = f32_to_bf16_bits(val);
        }
    } else {
        for (int i = warp; i < p.slots * kMoeSplit; i += blockDim.x >> 5) {
            const int q = i / kMoeSplit, ksp = i - q * kMoeSplit, e = expert(q);
            int eb = e >= 0 ? 0 : -1;
            if (FMT == TKD_BFP4 && e >= 0) eb = p.emax[(int64_t)e * (p.npad / 16) + u];
            run(e, u, ksp, p.x + (int64_t)q * p.K, red[q][ksp]);
            if (lane == 0 && ksp == 0) s_e[q] = eb;
        }
        __syncthreads();
        if (tid < 16) {
            float v = 0.f;
            for (int q = 0; q < p.slots; ++q) {  // (in slot order)
                float s = red[q][0][tid] + red[q][1][tid];
                if constexpr (FMT == TKD_BFP4) s = moe_scale(s, max(s_e[q], 0));
                v += s_e[q] >= 0 ? s : 0.f;
            }
            p.out[u * 16 + tid] = f32_to_bf16_bits(v);
        }
    }
}

// ---- the router's top k and their weights (moe/moe8.py:1139-1253 route, kernels/moe_route.cpp of the reference). One warp a
// row. The keys are float64's (the reference's core works in fixed point to the same end: picks that equal a float64 host
// computation's) as unsigned words that order as they do, a lane's experts in its registers. A round is two or three warp-wide
// maxima in hardware: the key's words, then among equals the lower id. A pick by logit needs no sigmoid and one word, and the
// sigmoids and exponentials of the weights are the picks' alone. Bound by latency: 8 of 128 experts took 8.3 us as rounds of
// float64 shuffles after 128 sigmoids.
constexpr int kRouteMaxE = 1024;

struct RouteParams {
    const float* logits;
    int64_t ld;
    int E, k, kind, norm, ng, tg, has_slot, ids32;
    const float* bias;
    double scale;
    uint32_t slot;
    void* ids;
    int64_t ld_ids;
    uint16_t* w;
    int64_t ld_w;
    uint16_t* shared;
    int64_t ld_sh;
};

__device__ __forceinline__ uint16_t route_bf16(double v) { return f32_to_bf16_bits((float)v); }
__device__ __forceinline__ double route_sigmoid(double x) { return 1.0 / (1.0 + exp(-x)); }
// words that order as the numbers do, above 0; -0 as +0
__device__ __forceinline__ uint32_t route_key(float x) {
    const uint32_t b = __float_as_uint(x + 0.f);
    return b & 0x80000000u ? ~b : b | 0x80000000u;
}
__device__ __forceinline__ unsigned long long route_key(double x) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x + 0.0);
    return b >> 63 ? ~b : b | (1ull << 63);
}

// BIASED: kind 1 (keys of 64 bits, groups). PER: experts a lane holds, at most.
template <bool BIASED, int PER>
__global__ void __launch_bounds__(32) tkd_moe_route_kernel(const RouteParams p) {
    using Key = std::conditional_t<BIASED, unsigned long long, uint32_t>;
    __shared__ double skey[BIASED ? 32 * PER : 1];
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int row = blockIdx.x, lane = threadIdx.x;
    const float* lg = p.logits + (int64_t)row * p.ld;
    Key own[PER];  // expert 32 j + lane's key; 0: out
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const int e = 32 * j + lane;
        own[j] = 0;
        if (32 * j >= p.E) continue;  // (E is a multiple of 32)
        if constexpr (BIASED) {
            const double v = route_sigmoid((double)lg[e]) + (double)p.bias[e];
            skey[e] = v;
            own[j] = route_key(v);
        } else {
            own[j] = route_key(lg[e]);
        }
    }
    if constexpr (BIASED) {
        __syncwarp();
        if (p.ng > 1) {
            // group-limited routing: a group's score is the sum of its two largest keys; the tg best groups stay (the lower
            // group among equal scores), the others' experts are out
            const int ge = p.E / p.ng;
            unsigned long long score = 0;
            if (lane < p.ng) {
                double a = skey[lane * ge], b = -__longlong_as_double(0x7FF0000000000000LL);
                for (int i = 1; i < ge; ++i) {
                    const double v = skey[lane * ge + i];
                    if (v > a) b = a, a = v;
                    else if (v > b) b = v;
                }
                score = route_key(a + b);
            }
            uint32_t kept = 0;
            for (int j = 0; j < p.tg; ++j) {
                const uint32_t hi = __reduce_max_sync(0xFFFFFFFFu, (uint32_t)(score >> 32));
                const uint32_t lo = __reduce_max_sync(0xFFFFFFFFu, (uint32_t)(score >> 32) == hi ? (uint32_t)score : 0u);
                const uint32_t who = __ballot_sync(0xFFFFFFFFu, score == (((unsigned long long)hi << 32) | lo));
                kept |= who & -who;
                if (lane == __ffs(who) - 1) score = 0;
            }
#pragma unroll
            for (int j = 0; j < PER; ++j)
                if (32 * j < p.E && !((kept >> ((32 * j + lane) / ge)) & 1u)) own[j] = 0;
        }
    }
    int id = -1;  // lane j: pick j
    for (int j = 0; j < p.k; ++j) {
        Key best = 0;
        int at = 0;
#pragma unroll
        for (int q = 0; q < PER; ++q)
            if (own[q] > best) best = own[q], at = q;  // (the lowest of a lane's equal keys)
        bool mine;
        if constexpr (BIASED) {
            const uint32_t hi = __reduce_max_sync(0xFFFFFFFFu, (uint32_t)(best >> 32));
            const uint32_t lo = __reduce_max_sync(0xFFFFFFFFu, (uint32_t)(best >> 32) == hi ? (uint32_t)best : 0u);
            mine = best != 0 && best == (((unsigned long long)hi << 32) | lo);
        } else {
            const uint32_t most = __reduce_max_sync(0xFFFFFFFFu, best);  // (by all lanes, those with nothing left too)
            mine = best != 0 && best == most;
        }
        const uint32_t e = __reduce_min_sync(0xFFFFFFFFu, mine ? (uint32_t)(32 * at + lane) : 0xFFFFFFFFu);
        if (lane == j) id = (int)e;  // (none left: -1)
#pragma unroll
        for (int q = 0; q < PER; ++q)
            if (e == (uint32_t)(32 * q + lane)) own[q] = 0;
    }
    // the weights: softmax over the picks' logits, or the picks' sigmoids (over their sum unless norm is off), times scale
    const double x = id >= 0 ? (double)lg[id] : 0.0;
    const double top = __shfl_sync(0xFFFFFFFFu, x, 0);
    const double v = id < 0 ? 0.0 : p.kind == 0 ? exp(x - top) : route_sigmoid(x);
    double sum = v;
#pragma unroll
    for (int d = 8; d > 0; d >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, d);  // (at most 16 picks)
    const double wv = (p.kind == 0 || p.norm ? v / sum : v) * p.scale;
    const int slots = p.k + p.has_slot;
    if (lane < slots) {
        const bool extra = lane == p.k;  // the fixed slot: that id at weight 1
        const uint32_t out_id = extra ? p.slot : (uint32_t)max(id, 0);
        if (p.ids32) static_cast<uint32_t*>(p.ids)[(int64_t)row * p.ld_ids + lane] = out_id;
        else static_cast<uint16_t*>(p.ids)[(int64_t)row * p.ld_ids + lane] = (uint16_t)out_id;
        p.w[(int64_t)row * p.ld_w + lane] = route_bf16(extra ? 1.0 : (id >= 0 ? wv : 0.0));
    }
    if (p.shared && lane == 0) p.shared[(int64_t)row * p.ld_sh] = route_bf16(route_sigmoid((double)lg[p.E]));
}

template <int FMT, bool DOWN>
int moe_launch(const MoeParams& p, cudaStream_t st) {
    auto kern = tkd_moe_kernel<FMT, DOWN>;
    const int room = 200 * 1024 / (2 * kMoeHalfBytes<FMT>), most = room < 16 ? room : 16;  // warps of down: a run each, if they fit
    const int warps = DOWN ? (p.slots * kMoeSplit < most ? p.slots * kMoeSplit : most) : 2 * kMoeSplit;
    const size_t smem = (size_t)warps * 2 * kMoeHalfBytes<FMT>;
    if (smem > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = DOWN ? dim3((unsigned)(p.N / 16)) : dim3((unsigned)(p.N / 32), (unsigned)p.slots);
    cfg.blockDim = dim3(warps * 32), cfg.dynamicSmemBytes = smem, cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr, cfg.numAttrs = 1;
    return (int)cudaLaunchKernelEx(&cfg, kern, p);
}

bool moe_args_ok(const TkdMoe* a, bool down) {
    if (!a || !a->w || !a->x || !a->ids || !a->out) return false;
    if (a->fmt != TKD_FMT_BFP4 && a->fmt != TKD_FMT_BF16) return false;
    if (a->fmt == TKD_FMT_BFP4 && !a->emax) return false;
    if (a->experts < 1 || a->k_in < 32 || a->k_in % 32 || a->n < 32 || a->n % 32 || a->k < 1 || a->k > 16) return false;
    if (a->rows < 1 || a->rows > 32 || (!a->by_union && a->rows != 1)) return false;
    if (a->by_union && (a->experts > 1024 || a->slots < 1 || a->ld_ids < a->k)) return false;
    if (!a->by_union && a->slots != a->k) return false;
    if (a->expert_bytes < tkd_packed_bytes(a->fmt, a->k_in, a->n) || a->expert_bytes % 16) return false;
    if (a->ldx % 8 || (reinterpret_cast<uintptr_t>(a->x) | reinterpret_cast<uintptr_t>(a->w)) & 15) return false;
    if (down) {
        if (a->ldx < (int64_t)a->slots * a->k_in || a->ldo < a->n) return false;
    } else {
        if (a->n % 64 || !a->route_w || a->ldx < a->k_in || a->ldo < (int64_t)a->slots * (a->n / 2)) return false;
        if (a->act < 0 || a->act > 2 || (a->by_union && a->ld_w < a->k)) return false;
    }
    return true;
}

MoeParams moe_params(const TkdMoe* a) {
    MoeParams p = {};
    p.w = static_cast<const uint8_t*>(a->w), p.emax = a->emax, p.wbytes = a->expert_bytes;
    p.E = a->experts, p.K = a->k_in, p.N = a->n, p.npad = (int)tkd_padded_cols(a->n);
    p.x = static_cast<const uint16_t*>(a->x), p.ids = a->ids, p.ids32 = a->ids32;
    p.rw = static_cast<const uint16_t*>(a->route_w);
    p.slots = a->slots, p.act = a->act, p.bias = static_cast<const uint16_t*>(a->bias);
    p.out = static_cast<uint16_t*>(a->out);
    p.status = a->status;
    p.mul16 = 16, p.mul128 = 128;
    return p;
}

int moe_sms() {
    static int cached[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    if (!cached[dev]) {
        int v = 0;
        if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 148;
        cached[dev] = v;
    }
    return cached[dev];
}

// the counters of a workspace, before the partial sums: a cut tile each of the rows form's gate_up (down has fewer)
int64_t moe_rows_counters(const TkdMoe* a, bool down) {
    const int64_t npad = tkd_padded_cols(a->n);
    return ((down ? npad / kMoeCols : a->experts * (npad / 128)) * 4 + 255) & ~(int64_t)255;
}

template <bool DOWN>
int moe_rows(const TkdMoe* a, cudaStream_t st) {
    MoeRowsParams p = {};
    p.w = static_cast<const uint8_t*>(a->w), p.emax = a->emax, p.wbytes = a->expert_bytes;
    p.panel_bytes = tkd_panel_bytes(a->fmt, a->k_in);
    p.E = a->experts, p.K = a->k_in, p.N = a->n, p.npad = (int)tkd_padded_cols(a->n), p.R = a->rows, p.k = a->k, p.slots = a->slots;
    p.x = static_cast<const uint16_t*>(a->x), p.ldx = a->ldx, p.ids = a->ids, p.ids32 = a->ids32, p.ld_ids = a->ld_ids;
    p.rw = static_cast<const uint16_t*>(a->route_w), p.ld_w = a->ld_w, p.act = a->act, p.bias = static_cast<const uint16_t*>(a->bias);
    p.out = static_cast<uint16_t*>(a->out), p.ldo = a->ldo, p.out_rows = a->out_rows;
    p.status = a->status;
    p.mul16 = 16, p.mul128 = 128;
    const int mt = (a->rows + 7) / 8;
    size_t smem = 0;
    if (!(a->fmt == TKD_FMT_BFP4 ? moe_rows_smem<TKD_BFP4>(p, mt, &smem) : moe_rows_smem<TKD_BF16>(p, mt, &smem))) return TKD_ERR_UNSUPPORTED;
    // one CTA an SM, or as many as the workspace has room for (two partial sums each)
    int grid = moe_sms();
    const int64_t head = moe_rows_counters(a, DOWN), part = 2 * 128 * 8 * mt * (int64_t)sizeof(float);
    const int64_t room = a->workspace ? ((int64_t)a->workspace_bytes - head) / part : 0;
    if (DOWN || room >= grid) {
        if (room < grid) grid = room < 1 ? 1 : (int)room;  // (one CTA cuts nothing)
        p.counters = static_cast<int*>(a->workspace);
        p.scratch = reinterpret_cast<float*>(static_cast<uint8_t*>(a->workspace) + head);
    }
    auto go = [&](auto f) -> int {
        constexpr int F = decltype(f)::value;
        switch (mt) {
            case 1: return moe_rows_launch<F, 1, DOWN>(p, grid, smem, st);
            case 2: return moe_rows_launch<F, 2, DOWN>(p, grid, smem, st);
            case 3: return moe_rows_launch<F, 3, DOWN>(p, grid, smem, st);
            default: return moe_rows_launch<F, 4, DOWN>(p, grid, smem, st);
        }
    };
    const int e = a->fmt == TKD_FMT_BF16 ? go(std::integral_constant<int, TKD_BF16>{}) : go(std::integral_constant<int, TKD_BFP4>{});
    return e == 0 ? TKD_OK : TKD_ERR_CUDA + e;
}

template <bool DOWN>
int moe_one(const TkdMoe* a, cudaStream_t st) {
    const MoeParams p = moe_params(a);
    if (p.K > 112 * 1024) return TKD_ERR_UNSUPPORTED;  // (no limit of this kernel: what tkd_moe_gate_up and _down always refused)
    const int e = a->fmt == TKD_FMT_BF16 ? moe_launch<TKD_BF16, DOWN>(p, st) : moe_launch<TKD_BFP4, DOWN>(p, st);
    return e == 0 ? TKD_OK : TKD_ERR_CUDA + e;
}

}  // namespace

extern "C" {

int tkd_moe_workspace(const TkdMoe* a, uint64_t* bytes) {
    if (!a || !bytes || a->slots < 1 || a->rows < 1 || a->n < 1) return TKD_ERR_BAD_ARG;
    const int64_t npad = tkd_padded_cols(a->n);
    // the column blocks' counters, then the slots' partial sums (more than the rows form needs of several slots and rows)
    *bytes = (uint64_t)(((npad / kMoeCols) * 4 + 255) & ~(int64_t)255) + (uint64_t)a->slots * a->rows * npad * sizeof(float);
    return TKD_OK;
}

int tkd_moe_rows_workspace(const TkdMoe* a, int down, uint64_t* bytes) {
    if (!a || !bytes || a->rows < 1 || a->rows > 32 || a->n < 1 || a->experts < 1) return TKD_ERR_BAD_ARG;
    *bytes = (uint64_t)(moe_rows_counters(a, down != 0) + (int64_t)moe_sms() * 2 * 128 * ((a->rows + 7) / 8 * 8) * (int64_t)sizeof(float));
    return TKD_OK;
}

int tkd_moe_gate_up(const TkdMoe* a, void* stream) {
    if (!moe_args_ok(a, false)) return TKD_ERR_BAD_ARG;
    if (a->workspace && (reinterpret_cast<uintptr_t>(a->workspace) & 15)) return TKD_ERR_WORKSPACE;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    return a->by_union ? moe_rows<false>(a, st) : moe_one<false>(a, st);
}

int tkd_moe_down(const TkdMoe* a, void* stream) {
    if (!moe_args_ok(a, true)) return TKD_ERR_BAD_ARG;
    uint64_t need = 0, rows = 0;
    tkd_moe_workspace(a, &need);
    if (a->by_union && tkd_moe_rows_workspace(a, 1, &rows) == TKD_OK && rows < need) need = rows;
    if (!a->workspace || a->workspace_bytes < need || (reinterpret_cast<uintptr_t>(a->workspace) & 15)) return TKD_ERR_WORKSPACE;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    return a->by_union ? moe_rows<true>(a, st) : moe_one<true>(a, st);
}

int tkd_moe_route(const float* logits, int64_t ld, int rows, int experts, int k, int kind, const float* bias, double scale,
                  int norm, int n_group, int topk_group, int has_slot, uint32_t slot, void* ids, int ids32, int64_t ld_ids,
                  void* w, int64_t ld_w, void* shared, int64_t ld_shared, void* stream) {
    if (!logits || !ids || !w || rows < 1 || rows > 32 || experts < 32 || experts % 32 || experts > kRouteMaxE) return TKD_ERR_BAD_ARG;
    if (k < 1 || k > 16 || k > experts || (has_slot && k + 1 > 16) || kind < 0 || kind > 2 || (kind == 1 && !bias)) return TKD_ERR_BAD_ARG;
    if (!(scale > 0.0 && scale < 4.0) || (!norm && kind == 0)) return TKD_ERR_BAD_ARG;
    if (ld < experts + (shared ? 1 : 0) || ld_ids < k + (has_slot ? 1 : 0) || ld_w < k + (has_slot ? 1 : 0)) return TKD_ERR_BAD_ARG;
    if (n_group > 1) {
        if (kind != 1 || n_group > 32 || experts % n_group || experts / n_group < 2 || topk_group < 1 || topk_group > n_group ||
            topk_group * (experts / n_group) < k)
            return TKD_ERR_BAD_ARG;
    }
    RouteParams p = {};
    p.logits = logits, p.ld = ld, p.E = experts, p.k = k, p.kind = kind, p.norm = norm, p.ng = n_group > 1 ? n_group : 1;
    p.tg = topk_group, p.has_slot = has_slot ? 1 : 0, p.ids32 = ids32, p.bias = bias, p.scale = scale, p.slot = slot;
    p.ids = ids, p.ld_ids = ld_ids, p.w = static_cast<uint16_t*>(w), p.ld_w = ld_w;
    p.shared = static_cast<uint16_t*>(shared), p.ld_sh = ld_shared;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)rows), cfg.blockDim = dim3(32), cfg.stream = static_cast<cudaStream_t>(stream);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr, cfg.numAttrs = 1;
    // (few experts in few registers: 128 are the usual number, and every round goes through all of a lane's)
    auto kern = experts <= 128 ? (kind == 1 ? tkd_moe_route_kernel<true, 4> : tkd_moe_route_kernel<false, 4>)
                : experts <= 512 ? (kind == 1 ? tkd_moe_route_kernel<true, 16> : tkd_moe_route_kernel<false, 16>)
                                 : (kind == 1 ? tkd_moe_route_kernel<true, 32> : tkd_moe_route_kernel<false, 32>);
    const int e = (int)cudaLaunchKernelEx(&cfg, kern, p);
    return e == 0 ? TKD_OK : TKD_ERR_CUDA + e;
}
}
