// tkd_moe.cu: the mixture-of-experts layer's two matmuls over the chosen experts only, for sm_100a. They take the
// place of the reference's gate_up / down and gate_up_rows / down_rows (moe/moe8.py:710-911, 928-1136; kernels
// moe_gu_reader.cpp, moe_gu_compute.cpp, moe_gu_writer.cpp, moe_dn_reader.cpp, moe_dn_compute.cpp, moe_dn_writer.cpp
// and kernels/moe8_rows.h for the union of the rows' experts).
//
// Every expert's weight is a bfloat4_b stream of tkd_layout.h (tkd_pack), all experts back to back, so the kernel
// finds a chosen expert by its id alone: the ids are read on the device and nothing goes to the host. What a call reads
// is small (k experts of a few MB) and scattered, so instead of the persistent ring of tkd_stream_kernel.cuh this is
// a plain grid: a CTA owns (32 columns of one slot's expert, all of its K), its 4 warps are 2 groups of 16 columns x 2
// runs of super-atoms, and a lane loads its own 16 bytes of codes and 16 bytes of exponents of a super-atom straight
// from global memory into the mma.sync A fragment's registers (the stream is laid out lane by lane, so a warp's load
// is one contiguous 512 bytes), four super-atoms at a time. The decode is the stream kernel's (block_mma), and like it
// the kernel is bound by instruction issue, not by HBM: units this small (384 and 512 CTAs of 128 threads for a layer
// of 8 experts of 2048 x 1536) are what spreads that work evenly over the SMs.
//   gate_up: a unit is 16 columns of a gate tile and the same 16 of its up tile: the CTA finishes 16 outputs,
//            h = routing weight * act(x G + b) * (x U + b), rounded to bf16 once.
//   down:    a CTA writes its slot's partial sums of 32 columns of y to the workspace; the CTA that arrives last at
//            the unit's counter adds the slots up in slot order and writes y (no CTA waits for another).
// Several rows (by_union): tkd_moe_rows.cuh.
#include "tkd_moe_rows.cuh"

namespace {

constexpr int kMoeGroups = 2;  // groups of 16 columns a CTA covers at a time (gate_up: 16 gate columns and their 16 up columns)
// warps along K per group: 4 warps a CTA, four CTAs an SM (with 4 a warp had too few super-atoms to spread its set-up over: the
// layer of the benchmark 16.9 us, 16.35 with down at 2, 16.8 with gate_up at 2; down at 1: 17.6)
constexpr int kMoeSplit = 2, kMoeThreads = kMoeGroups * kMoeSplit * 32;
constexpr int kMoeBatch = 4;  // super-atoms whose loads are issued before the first is used (8: spills, slower)
constexpr int kMoeCols = kMoeGroups * 16;

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
    float* part;    // down: [slot][npad] partial sums
    int* counters;  // down: one per block of 64 columns; back to zero when the call ends
    uint32_t mul16, mul128;
};

__device__ __forceinline__ uint4 ldg_stream(const uint8_t* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
    return v;
}
__device__ __forceinline__ uint32_t moe_id(const MoeParams& p, int64_t i) {
    return p.ids32 ? static_cast<const uint32_t*>(p.ids)[i] : static_cast<const uint16_t*>(p.ids)[i];
}
// a column sum in the stream's units -> its value (tkd_layout.h: 2^tkd_out_exp, in two factors that are normal floats)
__device__ __forceinline__ float moe_scale(float v, int ebyte) {
    const int e = tkd_out_exp(TKD_BFP4, ebyte), e1 = e / 2, e2 = e - e1;
    return v * __uint_as_float((uint32_t)(e1 + 127) << 23) * __uint_as_float((uint32_t)(e2 + 127) << 23);
}
// One row. FMT: the experts' stream format (bfloat4_b, or bf16 for a pack held exactly). DOWN: the down matmul.
template <int FMT, bool DOWN>
__global__ void __launch_bounds__(kMoeThreads, 4) tkd_moe_kernel(const MoeParams p) {
    using F = Fmt<FMT>;  // (k and bytes of a super-atom, super-atoms of a group in a chunk)
    extern __shared__ __align__(16) uint8_t moe_dsm[];
    __shared__ int s_last;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int gi = warp & (kMoeGroups - 1), ksp = warp / kMoeGroups;
    const int q = blockIdx.y;
    const int Kpad = (p.K + 63) & ~63;
    uint8_t* xs = moe_dsm;
    float* red = reinterpret_cast<float*>(moe_dsm + Kpad * 2);  // [ksp][column]

    // (launched as a programmatic dependent: nothing the kernels before wrote is read above this line, and the kernel
    // after may bring its CTAs in while this one runs: it waits at the same place)
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    const uint32_t id = moe_id(p, q);
    const int e = id < (uint32_t)p.E ? (int)id : -1;
    float w1 = 0.f;  // the slot's routing weight
    if constexpr (!DOWN)
        if (e >= 0) w1 = bf16_bits_to_f32(p.rw[q]);
    // a unit of 32 weight columns. gate_up: unit u is half hf = u & 1 of the tile pair j = u >> 1: columns hf * 16 .. + 15 of
    // gate tile j (warps gi 0) and of up tile j (gi 1), 16 outputs.
    const int u = blockIdx.x, group = DOWN ? u * kMoeGroups + gi : (u >> 1) * 4 + 2 * gi + (u & 1);
    const uint8_t* wb = p.w + (int64_t)max(e, 0) * p.wbytes;
    const uint8_t* emx = FMT == TKD_BFP4 ? p.emax + (int64_t)max(e, 0) * (p.npad / 16) : nullptr;
    const int nsa = (p.K + F::KSA - 1) / F::KSA, per = (nsa + kMoeSplit - 1) / kMoeSplit;
    const int sa0 = ksp * per, sa1 = min(nsa, sa0 + per);
    const uint2 sh = make_uint2(p.mul16, p.mul128);
    if (e >= 0) {
        // This warp's super-atoms are asked into L2 at once (one instruction per run inside a chunk), so that the loads behind
        // the first batch, which wait for registers, find them there: one trip to HBM, not two.
        if (lane == 0)
            for (int sa = sa0; sa < sa1;) {
                const int end = min(sa1, (sa | (F::SUBSA - 1)) + 1);
                const uint8_t* s = wb + tkd_sa_offset(FMT, p.K, group, sa);
                asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(s), "r"((end - sa) * F::SAB) : "memory");
                sa = end;
            }
        // the activations: gate_up: x; down: the inputs of slot q. Zeros past K up to a super-atom.
        const uint16_t* xsrc = p.x + (DOWN ? (int64_t)q * p.K : 0);
        for (int c = tid; c < Kpad / 8; c += kMoeThreads)
            reinterpret_cast<uint4*>(xs)[c] = c * 8 < p.K ? __ldg(reinterpret_cast<const uint4*>(xsrc) + c) : make_uint4(0u, 0u, 0u, 0u);
    }
    __syncthreads();
    const uint32_t xa = smem_u32(xs) + 16 * t;
    if (e >= 0) {
        // ---- the group's sums over this warp's run of super-atoms
        float acc[2][1][4] = {};
        // (the super-atoms of a group lie back to back inside a chunk of 8: the layout is asked at its starts only)
        const uint8_t* s = wb;
        for (int sa = sa0; sa < sa1; sa += kMoeBatch) {
            uint4 cv[kMoeBatch], ev[kMoeBatch];
#pragma unroll
            for (int b = 0; b < kMoeBatch; ++b)
                if (sa + b < sa1) {
                    s = (b == 0 && sa == sa0) || ((sa + b) & (F::SUBSA - 1)) == 0 ? wb + tkd_sa_offset(FMT, p.K, group, sa + b) : s + F::SAB;
                    if constexpr (FMT == TKD_BFP4) {
                        ev[b] = ldg_stream(s + t * 16);
                        cv[b] = ldg_stream(s + 64 + lane * 16);
                    } else {  // (bf16: the A fragments of the super-atom's two mmas as they are)
                        cv[b] = ldg_stream(s + lane * 16);
                        ev[b] = ldg_stream(s + 512 + lane * 16);
                    }
                }
#pragma unroll
            for (int b = 0; b < kMoeBatch; ++b)
                if (sa + b < sa1) {
                    if constexpr (FMT == TKD_BFP4) {
#pragma unroll
                        for (int qq = 0; qq < 2; ++qq) {
                            const uint32_t cw[4] = {qq ? cv[b].z : cv[b].x, qq ? cv[b].w : cv[b].y, 0u, 0u};
                            const uint32_t ew[2] = {qq ? ev[b].z : ev[b].x, qq ? ev[b].w : ev[b].y};
                            const uint4 xv[1] = {lds128(xa + (uint32_t)(sa + b) * 128 + 64 * qq)};
                            block_mma<TKD_BFP4, 1, 2>(acc, cw, ew, xv, sh);
                        }
                    } else {
                        const uint4 xv = lds128(xa + (uint32_t)(sa + b) * 64);
                        mma_bf16(acc[0][0], cv[b].x, cv[b].y, cv[b].z, cv[b].w, xv.x, xv.y);
                        mma_bf16(acc[1][0], ev[b].x, ev[b].y, ev[b].z, ev[b].w, xv.z, xv.w);
                    }
                }
        }
        // (every column of D is the one row's; its first is kept: lanes with t = 0 hold columns g and g + 8 of the weight)
        if (t == 0) {
            float* d = red + ksp * kMoeCols + gi * 16 + g;
            d[0] = acc[0][0][0] + acc[1][0][0], d[8] = acc[0][0][2] + acc[1][0][2];
        }
    }
    __syncthreads();

    // column c of the unit (gate_up: 0-15 the gate's, 16-31 the up's): the K sum, in the weight's units
    auto column_sum = [&](int c, int grp) {
        float v = 0.f;
#pragma unroll
        for (int sp = 0; sp < kMoeSplit; ++sp) v += red[sp * kMoeCols + c];
        if constexpr (FMT == TKD_BFP4) v = moe_scale(v, emx[grp]);
        return v;
    };
    if constexpr (!DOWN) {
        const int j = u >> 1, hf = u & 1;
        if (tid < 16) {
            float val = 0.f;
            if (e >= 0) {
                float gt = column_sum(tid, j * 4 + hf), up = column_sum(16 + tid, j * 4 + 2 + hf);
                if (p.bias) {
                    const uint16_t* b = p.bias + (int64_t)e * p.npad + j * 64 + hf * 16 + tid;
                    gt += bf16_bits_to_f32(b[0]), up += bf16_bits_to_f32(b[32]);
                }
                val = moe_glu(gt, up, p.act) * w1;
            }
            p.out[(int64_t)q * (p.N / 2) + j * 32 + hf * 16 + tid] = f32_to_bf16_bits(val);
        }
    } else {
        // this slot's sums of the unit's columns are written: the CTA that arrives last adds the slots up
        if (tid < kMoeCols) {
            if (e >= 0) p.part[(int64_t)q * p.npad + u * kMoeCols + tid] = column_sum(tid, u * kMoeGroups + (tid >> 4));
            __threadfence();
        }
        __syncthreads();
        if (tid == 0) s_last = atomicAdd(&p.counters[u], 1) == p.slots - 1;
        __syncthreads();
        if (s_last && tid < kMoeCols) {
            __threadfence();
            const int col = u * kMoeCols + tid;
            if (col < p.N) {
                float v = 0.f;
                for (int sl = 0; sl < p.slots; sl += 8) {  // (eight loads in flight; added in slot order)
                    float part[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        part[j] = sl + j < p.slots && moe_id(p, sl + j) < (uint32_t)p.E ? __ldcg(p.part + (int64_t)(sl + j) * p.npad + col) : 0.f;
#pragma unroll
                    for (int j = 0; j < 8; ++j) v += part[j];
                }
                p.out[col] = f32_to_bf16_bits(v);
            }
            if (tid == 0) p.counters[u] = 0;
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
int moe_launch(const MoeParams& p, dim3 grid, cudaStream_t st) {
    auto kern = tkd_moe_kernel<FMT, DOWN>;
    const size_t smem = (size_t)((p.K + 63) & ~63) * 2 + kMoeSplit * kMoeCols * sizeof(float);
    if (smem > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid, cfg.blockDim = dim3(kMoeThreads), cfg.dynamicSmemBytes = smem, cfg.stream = st;
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
    MoeParams p = moe_params(a);
    if ((int64_t)((p.K + 63) & ~63) * 2 > 224 * 1024) return TKD_ERR_UNSUPPORTED;  // (the row in shared memory)
    if (DOWN) {
        p.counters = static_cast<int*>(a->workspace);
        p.part = reinterpret_cast<float*>(static_cast<uint8_t*>(a->workspace) + moe_rows_counters(a, true));
    }
    const dim3 grid((unsigned)((DOWN ? p.npad : p.N) / kMoeCols), (unsigned)a->slots);
    const int e = a->fmt == TKD_FMT_BF16 ? moe_launch<TKD_BF16, DOWN>(p, grid, st) : moe_launch<TKD_BFP4, DOWN>(p, grid, st);
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
