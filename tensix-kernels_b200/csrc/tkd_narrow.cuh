// tkd_narrow.cuh: the streaming matmul of one to eight rows as items of 32 columns and all of K.
//
// tkd_stream_kernel.cuh's items are 128 columns and a slice of K: a panel's four slices fall to several CTAs, and its end is a
// chain of trips through L2 (the sums stored, counted in by an atomic, the last to arrive reading all of them back), 1.4 us of
// a launch of one row and 2.5 of one of eight, where one token through [4096, 2048] takes 5.5 us. Here a CTA takes two groups
// of 16 columns over all of K, the same bytes, and its sixteen streaming warps are (slice, half of a chunk's super-atoms,
// group): the sums are the same sums in the same order (T_h ascending over the slices, then T0 + T1: see there, the two kernels
// give the same bits), but they meet in shared memory, and no CTA waits for another. Plain calls of one to four
// slices whose rows of x fit in shared memory run this kernel, but for large weights of one to three (make_layout has the limits); FOUR: of four, an instance of its own, because what
// fewer need (a count instead of a constant here and there) cost the calls of four 0.15 us. Measured, a launch of a sequence in a graph:
// one row, [4096, 4096] of bfloat8_b 8.3 us before, 6.2 now (2.8 at the memory's rate), [2048, 3072] 5.3 and 3.5; eight rows of
// bf16, [2048, 2048] 7.2 and 4.2 (1.3). Where an SM has several items the decode of the weights bounds both kernels.
//
//   warp 0       producer: a stage of the ring is the next chunk of all four slices, 2 groups each: a copy for each slice, by a
//                lane each (GLU: the gate's group and the up's apart)
//   warps 1-16   streaming
//   warps 17-18  output: a warp takes every other item, a lane a column (GLU: 16 gate columns and their 16 up columns)
#pragma once
#include "tkd_stream_kernel.cuh"

namespace {

constexpr int kNarrowWarps = 19;

__device__ __forceinline__ void sts32(uint32_t a, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory"); }
__device__ __forceinline__ void sts64(uint32_t a, float v, float w) {
    asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(v), "f"(w) : "memory");
}

// Where item `pl` of a segment lies: the panel and the two groups in it.
struct NarrowItem {
    int panel, ga, gb;
};
__device__ __forceinline__ NarrowItem narrow_item(const TkdParams& p, int pl) {
    if (p.epi == TKD_EPI_GLU2) return {pl >> 3, pl & 7, pl & 7};  // (group pl of the gate's and of the up's weight)
    if (p.epi == TKD_EPI_GLU_IL) {
        const int g = (pl >> 1) * 4 + (pl & 1);  // (interleaved: two groups of gate columns, their two of up columns)
        return {g >> 3, g & 7, (g & 7) + 2};
    }
    return {pl >> 2, 2 * (pl & 3), 2 * (pl & 3) + 1};
}

template <int FMT, bool ONE, bool KWHOLE, bool FOUR>
__global__ void __launch_bounds__(kNarrowWarps * 32, 1) tkd_narrow_kernel(const __grid_constant__ TkdParams p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    using F = Fmt<FMT>;
    constexpr int SW = kStreamWarps, MR = ONE ? 1 : 8, CK = F::SUBSA * F::KSA, GB = F::SUBSA * F::SAB;
    constexpr int EXPB = FMT == TKD_BFP4 || FMT == TKD_INT4 ? 64 : (FMT == TKD_BFP8 ? 32 : 0);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem);
    const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + TKD_MAX_STAGES);
    const uint32_t pfull0 = smem_u32(bars + 2 * TKD_MAX_STAGES), pempty0 = pfull0 + 16, xbar = pfull0 + 32;
    float* pbuf = reinterpret_cast<float*>(smem + p.off_pbuf);  // [2 items][4 slices][2 halves][32 columns][MR]
    const uint32_t ring_a = smem_u32(smem + p.off_ring), xt0 = smem_u32(smem + p.off_xt);
    // (the warp's number by a shuffle: what follows from it is then known to be the same in all lanes, and the loop's addresses and counts
    // are reckoned once a warp, beside the lanes' arithmetic that bounds it. Launches in a graph: a layer (4096, 1024, 14336), one row,
    // 45.1 us with the thread's number divided, 43.2 so; (2048, 512, 5632) of bf16, 8 rows, 26.9 and 26.0)
    const int tid = threadIdx.x, warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0), lane = tid & 31;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (tid == 0) {
        for (int s = 0; s < p.nstages; ++s) mbar_init(full0 + 8 * s, 1), mbar_init(empty0 + 8 * s, SW);
        for (int s = 0; s < 2; ++s) mbar_init(pfull0 + 8 * s, SW), mbar_init(pempty0 + 8 * s, 1);
        mbar_init(xbar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    const uint32_t T = 4u * (uint32_t)p.total_panels;  // items
    const int i0 = (int)((uint64_t)T * blockIdx.x / gridDim.x), i1 = (int)((uint64_t)T * (blockIdx.x + 1) / gridDim.x);
    const int nst = p.nstages, M = ONE ? 1 : p.M, K = p.K, cps = p.ks / CK, nch = (K + CK - 1) / CK;
    const int nsa_total = (K + F::KSA - 1) / F::KSA;
    const bool glu = p.epi == TKD_EPI_GLU2 || p.epi == TKD_EPI_GLU_IL, silu = p.epi == TKD_EPI_SILU;
    auto seg_of = [&](int it) {
        int s = 0;
#pragma unroll
        for (int q = 1; q < 4; ++q)
            if (q < p.nseg && it >= 4 * p.seg[q].panel0) s = q;
        return s;
    };

    if (warp == 0) {
        // ---------------------------------------------------------------- producer: lane 2 s + g brings slice s's share of group g
        // (not GLU: lane 2 s both groups', which lie together)
        uint32_t st = 0;
        bool ok = true;
        const int s = lane >> 1, g = lane & 1;
        for (int it = i0; ok && it < i1; ++it) {
            const TkdSegDev& sg = p.seg[seg_of(it)];
            const NarrowItem n = narrow_item(p, it - 4 * sg.panel0);
            const uint8_t* src = (g && p.epi == TKD_EPI_GLU2 ? sg.w2 : sg.w) + (int64_t)n.panel * p.panel_bytes;
            for (int i = 0; i < cps; ++i, ++st) {
                const uint32_t q = st % nst;
                ok = __all_sync(0xFFFFFFFFu, mbar_wait_parked(empty0 + 8 * q, ((st / nst) & 1) ^ 1, p.status));
                if (!ok) break;
                const int c = s * cps + i;  // this lane's chunk, if there is one
                const bool mine = s < (FOUR ? 4 : p.nslices) && c < nch && (glu || !g);
                const uint32_t gb = mine ? (uint32_t)min(F::SUBSA, nsa_total - c * F::SUBSA) * F::SAB : 0u, bytes = glu ? gb : 2 * gb;
                const uint32_t all = __reduce_add_sync(0xFFFFFFFFu, bytes);
                if (lane == 0) mbar_expect_tx(full0 + 8 * q, all);
                __syncwarp();
                if (mine)
                    bulk_g2s(ring_a + q * p.stage_bytes + s * 2 * GB + g * gb, src + (int64_t)c * (GB * 8) + (int64_t)(g ? n.gb : n.ga) * gb, bytes,
                             full0 + 8 * q);
            }
        }
        if (!ok)  // (the copies in flight land before the CTA goes)
            for (uint32_t back = 1; back <= (uint32_t)nst && back <= st; ++back)
                for (uint32_t i = 0; i < 64; ++i)
                    if (mbar_try_wait(full0 + 8 * ((st - back) % nst), ((st - back) / nst) & 1)) break;
    } else if (warp <= SW) {
        // ---------------------------------------------------------------- streaming warps
        const int cw = warp - 1, gsel = cw & 1, h = (cw >> 1) & 1, sl = cw >> 2;
        if constexpr (!KWHOLE) {
            // the rows of x in shared memory end in zeros up to a whole chunk
            const int pieces = nch * (CK / 8);
            for (int r = 0; r < M; ++r)
                for (int e = K / 8 + cw * 32 + lane; e < pieces; e += SW * 32)
                    asm volatile("st.shared.v4.u32 [%0], {%1,%1,%1,%1};" ::"r"(xt0 + r * p.x_stride + e * 16), "r"(0u) : "memory");
            asm volatile("bar.sync 2, %0;" ::"n"(SW * 32) : "memory");
        }
        // (x and the outputs may belong to the kernel before this one: wait for it to complete)
        asm volatile("griddepcontrol.wait;" ::: "memory");
        if (cw == 0 && lane == 0) {
            mbar_expect_tx(xbar, (uint32_t)(M * K * 2));
            for (int r = 0; r < M; ++r) bulk_g2s(xt0 + (ONE ? 0 : r * p.x_stride), p.x + (int64_t)r * p.ldx, (uint32_t)(K * 2), xbar);
        }
        const int g = lane >> 2, t = lane & 3;
        const uint32_t exp_lane = FMT == TKD_INT4 ? g * 8 : t * (EXPB / 4);
        const uint32_t lane_off = sl * 2 * GB + gsel * GB + h * F::SAB;
        // (a lane whose row lies beyond M reads row M - 1: a column of B only feeds its own column of D)
        const uint32_t xs_lane = xt0 + (ONE ? 0 : min(g, M - 1) * p.x_stride) + (8 * t + h * F::KSA) * 2;
        const uint2 sh = make_uint2(p.mul16, p.mul128);
        const uint16_t* const no_x[1] = {nullptr};
        const uint4 no_pre[F::SUBSA / 2 * F::XB][1] = {};
        float acc[2][1][4];
        bool ok = mbar_wait(xbar, 0, p.status);
        if constexpr (FMT == TKD_INT4)
            rows_for_int4<ONE>(p, xt0, cw, lane, M);
        const int c0 = sl * cps, mine = min(cps, nch - c0);  // (the last slice may have fewer chunks)
        // (the sums of a slice that K does not have: -0, which changes no float32 that it is added to)
        const float zero = FOUR || sl < p.nslices ? 0.f : -0.f;
        const uint32_t xs0 = xs_lane + c0 * CK * 2;
        const uint32_t ring_end = ring_a + nst * p.stage_bytes;
        uint32_t at = ring_a, bar = full0, phase = 0;  // the stage, its barrier, its parity
        // (where this lane's sums go, of two buffers)
        uint32_t pc = smem_u32(pbuf) + (((sl * 2 + h) * 32 + gsel * 16 + g) * MR + (ONE ? 0 : 2 * t)) * 4, pbar = pfull0, pphase = 1;
        int other = 8 * 32 * MR * 4;
        for (int j = 0; ok && j < i1 - i0; ++j) {
#pragma unroll
            for (int a = 0; a < 2; ++a) acc[a][0][0] = acc[a][0][1] = acc[a][0][2] = acc[a][0][3] = zero;
            uint32_t xs = xs0;
#pragma unroll 1
            for (int i = 0; i < cps; ++i, xs += CK * 2) {
                ok = mbar_wait(bar, phase, p.status);
                if (!ok) break;
                const uint32_t a = at + lane_off;
                if (i < mine) {
                    if (KWHOLE || (c0 + i + 1) * CK <= K) {
                        chunk_mma<FMT, 1, 2, true, false, true>(acc, a + EXPB + lane * 16, a + exp_lane, no_pre, no_x, 0, K, h, F::SUBSA, sh, xs);
                    } else {
                        const int nsa = nsa_total - (c0 + i) * F::SUBSA;  // (the groups lie closer together)
                        const uint32_t b = a - gsel * (GB - nsa * F::SAB);
                        chunk_mma<FMT, 1, 2, false, false, true>(acc, b + EXPB + lane * 16, b + exp_lane, no_pre, no_x, (c0 + i) * CK, K, h, nsa, sh, xs);
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(bar + 8 * TKD_MAX_STAGES);
                at += p.stage_bytes, bar += 8;
                if (at == ring_end) at = ring_a, bar = full0, phase ^= 1;
            }
            if (!ok) break;
            // ---- the item's sums of this slice, half and group
            if (!mbar_wait(pbar + 16, pphase, p.status)) break;
            if constexpr (ONE) {
                if (t == 0) sts32(pc, acc[0][0][0] + acc[1][0][0]), sts32(pc + 32, acc[0][0][2] + acc[1][0][2]);
            } else {
                sts64(pc, acc[0][0][0] + acc[1][0][0], acc[0][0][1] + acc[1][0][1]);
                sts64(pc + 8 * MR * 4, acc[0][0][2] + acc[1][0][2], acc[0][0][3] + acc[1][0][3]);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(pbar);
            pc += other, other = -other, pbar ^= 8;
            if (pbar == pfull0) pphase ^= 1;
        }
    } else {
        // ---------------------------------------------------------------- output warps
        asm volatile("griddepcontrol.wait;" ::: "memory");
        const int b = warp - 1 - SW;
        const bool up = glu && lane >= 16;
        for (int it = i0 + b; it < i1; it += 2) {
            const TkdSegDev& sg = p.seg[seg_of(it)];
            const int pl = it - 4 * sg.panel0;
            // this lane's column of its weight, and what it stores
            int n, oc;
            if (p.epi == TKD_EPI_GLU2) {
                n = pl * 16 + (lane & 15);
                oc = !up && n < sg.n_valid ? sg.out_col0 + n : -1;
            } else if (glu) {
                n = (pl >> 1) * 64 + (pl & 1) * 16 + (up ? 32 : 0) + (lane & 15);
                oc = !up && n < sg.n_valid ? sg.out_col0 + pl * 16 + lane : -1;
            } else {
                n = pl * 32 + lane;
                oc = n < sg.n_valid ? sg.out_col0 + n : -1;
            }
            const bool other = up && p.epi == TKD_EPI_GLU2;
            float f1 = 1.f, f2 = 1.f, sc = 1.f;  // 2^e of the group in two normal floats, the column's scale
            if constexpr (FMT == TKD_BFP8 || FMT == TKD_BFP4) {
                const int e = tkd_out_exp(FMT, (other ? sg.emax2 : sg.emax)[n >> 4]), e1 = e / 2;
                f1 = __uint_as_float((uint32_t)(e1 + 127) << 23), f2 = __uint_as_float((uint32_t)(e - e1 + 127) << 23);
            }
            if (p.scale_dt != TKD_DT_NONE && n < sg.n_valid) {
                const void* sp = other ? p.scale2 : p.scale;
                sc = p.scale_dt == TKD_DT_BF16 ? bf16_bits_to_f32(static_cast<const uint16_t*>(sp)[n]) : static_cast<const float*>(sp)[n];
            }
            // (the residual is asked for now, so that its latency passes while the streaming warps are at work; a row past M reads
            // the last again)
            uint32_t q[MR];
            if (p.res_dt != TKD_DT_NONE && oc >= 0) {
                const int rsz = p.res_dt == TKD_DT_F32 ? 4 : 2;
                const char* rp = static_cast<const char*>(p.res) + (int64_t)oc * rsz;
#pragma unroll
                for (int m = 0; m < MR; ++m) {
                    q[m] = rsz == 4 ? *reinterpret_cast<const uint32_t*>(rp) : (uint32_t)*reinterpret_cast<const uint16_t*>(rp) << 16;
                    if (m + 1 < M) rp += p.ldr * rsz;
                }
            } else {
#pragma unroll
                for (int m = 0; m < MR; ++m) q[m] = 0u;
            }
            if (!mbar_wait(pfull0 + 8 * b, ((it - i0) >> 1) & 1, p.status)) break;
            // T_h = the slices' sums in order, then T0 + T1
            float v[MR];
            const float* pc = pbuf + ((size_t)b * 8 * 32 + lane) * MR;
            auto get = [&](int s, int hh, float (&o)[MR]) {
                const float* a = pc + (size_t)(s * 2 + hh) * 32 * MR;
                if constexpr (ONE) {
                    o[0] = a[0];
                } else {
                    const float4 lo = *reinterpret_cast<const float4*>(a), hi = *reinterpret_cast<const float4*>(a + 4);
                    o[0] = lo.x, o[1] = lo.y, o[2] = lo.z, o[3] = lo.w, o[4] = hi.x, o[5] = hi.y, o[6] = hi.z, o[7] = hi.w;
                }
            };
            float t1[MR];
            get(0, 0, v), get(0, 1, t1);
#pragma unroll
            for (int s = 1; s < 4; ++s) {
                float a[MR], c[MR];
                get(s, 0, a), get(s, 1, c);
#pragma unroll
                for (int m = 0; m < MR; ++m) v[m] += a[m], t1[m] += c[m];
            }
#pragma unroll
            for (int m = 0; m < MR; ++m) v[m] += t1[m];
            __syncwarp();
            if (lane == 0) mbar_arrive(pempty0 + 8 * b);
            if constexpr (FMT == TKD_BFP8 || FMT == TKD_BFP4) {
#pragma unroll
                for (int m = 0; m < MR; ++m) v[m] = v[m] * f1 * f2;
            }
            if (p.scale_dt != TKD_DT_NONE) {
#pragma unroll
                for (int m = 0; m < MR; ++m) v[m] *= sc;
            }
            if (glu || silu) {  // (one copy of the activation's code for both: a GLU's other factor, or 1)
#pragma unroll
                for (int m = 0; m < MR; ++m) {
                    const float u = __shfl_xor_sync(0xFFFFFFFFu, v[m], 16);
                    v[m] = act_gate(v[m], p.act) * (glu ? u : 1.f);
                }
            }
            if (p.res_dt != TKD_DT_NONE) {
#pragma unroll
                for (int m = 0; m < MR; ++m) v[m] += __uint_as_float(q[m]);
            }
            const bool f32out = p.epi == TKD_EPI_OUT32;
            char* yp = static_cast<char*>(p.out) + (int64_t)oc * (f32out ? 4 : 2);
            const int rows = oc >= 0 ? M : 0;
#pragma unroll
            for (int m = 0; m < MR; ++m, yp += p.ldo * (f32out ? 4 : 2)) {
                if (f32out)
                    st_if(m < rows, yp, __float_as_uint(v[m]));
                else
                    st16_if(m < rows, yp, f32_to_bf16_bits(v[m]));
            }
        }
    }
}

template <int FMT, bool ONE, bool KWHOLE, bool FOUR>
int launch_narrow_one(const TkdParams& p, int grid, size_t smem, cudaStream_t st) {
    auto kern = tkd_narrow_kernel<FMT, ONE, KWHOLE, FOUR>;
    static bool allowed[64] = {false};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    if (dev < 0 || dev >= 64 || !allowed[dev]) {
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        if (e != cudaSuccess) return (int)e;
        if (dev >= 0 && dev < 64) allowed[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid), cfg.blockDim = dim3(kNarrowWarps * 32), cfg.stream = st;
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr, cfg.numAttrs = p.no_pdl ? 0 : 1;
    return (int)cudaLaunchKernelEx(&cfg, kern, p);
}
template <int FMT, bool ONE, bool KWHOLE>
int launch_narrow_k(const TkdParams& p, int grid, size_t smem, cudaStream_t st) {
    return p.nslices == 4 ? launch_narrow_one<FMT, ONE, KWHOLE, true>(p, grid, smem, st) : launch_narrow_one<FMT, ONE, KWHOLE, false>(p, grid, smem, st);
}
template <int FMT>
int launch_narrow(const TkdParams& p, int grid, size_t smem, cudaStream_t st) {
    const bool whole = p.K % (Fmt<FMT>::SUBSA * Fmt<FMT>::KSA) == 0;
    if (p.M == 1) return whole ? launch_narrow_k<FMT, true, true>(p, grid, smem, st) : launch_narrow_k<FMT, true, false>(p, grid, smem, st);
    return whole ? launch_narrow_k<FMT, false, true>(p, grid, smem, st) : launch_narrow_k<FMT, false, false>(p, grid, smem, st);
}

}  // namespace
