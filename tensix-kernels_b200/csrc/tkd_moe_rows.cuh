// tkd_moe_rows.cuh: the mixture-of-experts layer's two matmuls for several rows (gate_up_rows / down_rows, moe/moe8.py:928-1136
// of the reference): every expert that some row chose, streamed once for all rows.
//
// As a CTA per slot and run of columns (the one-row kernel's plan, tkd_moe.cu) 16 rows of 8 of 128 experts left the slots past
// the union without work, waited for global loads unit by unit and added 80 partial sums a column at the end: 359 us a layer
// of 108 MB. Here one persistent CTA an SM takes an equal share of the union's work through a ring of bulk copies, as
// tkd_stream_kernel does:
//   warp 0       producer: a stage is one chunk (128 columns x 512 k of bfloat4_b, 128 k of bf16) of one expert's panel by one
//                bulk copy, and the rows' activations for those k by the warp's own 16-byte asynchronous copies, both counted
//                on the stage's barrier
//   warps 1-16   streaming: warp (g, h) multiplies the 16 columns of group g by every other super-atom with mma.sync, 8 rows an
//                MMA; from nine rows on the scales go into the weights instead (exact: a code times a power of two), once for
//                all rows, and where an expert's few rows take one MMA too: an activation times the largest scale, 2^64, may be
//                past bf16's range. An expert's sums, times its group's factor, are added to the tile's in registers
//   warps 17-20  output (thread = column)
//
// A tile is 128 columns of the result: gate_up: of one expert (64 outputs act(x G + b) * (x U + b) * routing weight); down: of
// y, its K running on over all the union's experts. A tile's work is its blocks, one per (expert, chunk). The blocks of all
// tiles are dealt out in equal contiguous runs, one per CTA; a tile that falls to several goes through scratch, a partial sum
// per CTA, added up in order by the one that delivers last. Whole tiles are dealt out where that is as even.
#pragma once
#include "tkd_stream_kernel.cuh"

namespace {

// moe8.py:83-85, 607-616: silu, gelu_tanh, or gpt-oss's clamped SwiGLU min(g, 7) * sigmoid(1.702 min(g, 7)) * (clamp(u, -7, 7) + 1)
__device__ __forceinline__ float moe_glu(float gt, float u, int act) {
    if (act == 2) {
        const float gc = fminf(gt, 7.f);
        return over_one_plus_exp(gc, -1.702f * gc) * (fminf(fmaxf(u, -7.f), 7.f) + 1.f);
    }
    return act_gate(gt, act) * u;
}

constexpr int kMrWarps = 21, kMrStream = 16;
// shared memory: barriers, the experts chosen (a bit each), flags, the current expert's routing weights, the union, the ids, the weights
constexpr int kMrBits = 512, kMrFlags = 640, kMrRow = 768, kMrUnion = 1024, kMrIds = 3072, kMrW = 4096, kMrHead = 5120;

struct MoeRowsParams {
    const uint8_t* w;
    const uint8_t* emax;
    int64_t wbytes, panel_bytes;
    int E, K, N, npad, R, k, slots;
    const uint16_t* x;
    int64_t ldx;
    const void* ids;
    int ids32;
    int64_t ld_ids;
    const uint16_t* rw;
    int64_t ld_w;
    int act;
    const uint16_t* bias;
    uint16_t* out;
    int64_t ldo;
    int out_rows;    // rows of out: those past R are zeroed
    float* scratch;  // [cta][2][8 MT rows / 4][128 columns][4]
    int* counters;   // per tile: blocks delivered. null: tiles are not cut
    int* status;
    int nstages, stage_bytes, w_bytes, x_stride, off_pbuf, off_ring;
    uint32_t mul16, mul128;
};

template <int FMT, int MT, bool DOWN>
__global__ void __launch_bounds__(kMrWarps * 32, 1) tkd_moe_rows_kernel(const __grid_constant__ MoeRowsParams p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    using F = Fmt<FMT>;
    constexpr int CK = F::SUBSA * F::KSA, RW = 8 * MT, MP = RW + 4, EXPB = FMT == TKD_BFP4 ? 64 : 0;
    const uint32_t full0 = smem_u32(smem), empty0 = full0 + 8 * TKD_MAX_STAGES;
    const uint32_t pfull = empty0 + 8 * TKD_MAX_STAGES, pempty = pfull + 8;
    uint32_t* bm = reinterpret_cast<uint32_t*>(smem + kMrBits);
    volatile int* sflag = reinterpret_cast<volatile int*>(smem + kMrFlags);  // [0] a flag, [1] the union's size
    float* wrow = reinterpret_cast<float*>(smem + kMrRow);
    uint16_t* ulist = reinterpret_cast<uint16_t*>(smem + kMrUnion);
    uint16_t* sids = reinterpret_cast<uint16_t*>(smem + kMrIds);
    uint16_t* srw = reinterpret_cast<uint16_t*>(smem + kMrW);
    float* pbuf = reinterpret_cast<float*>(smem + p.off_pbuf);  // [2 halves][128 columns][MP]
    const uint32_t ring0 = smem_u32(smem + p.off_ring);
    // (the warp's number by a shuffle, as in tkd_narrow_kernel: a layer of 16 rows, 8 of 128 experts, 85.2 us without, 83.6 so)
    const int tid = threadIdx.x, warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0), lane = tid & 31;
    if (tid == 0) {
        for (int s = 0; s < p.nstages; ++s) mbar_init(full0 + 8 * s, 33), mbar_init(empty0 + 8 * s, kMrStream);
        mbar_init(pfull, kMrStream), mbar_init(pempty, 4);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (tid < 32) bm[tid] = 0;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    __syncthreads();
    // ---- the union of the rows' experts, in increasing order
    for (int i = tid; i < p.R * p.k; i += kMrWarps * 32) {
        const int r = i / p.k, s = i - r * p.k;
        const int64_t at = r * p.ld_ids + s;
        const uint32_t id = p.ids32 ? static_cast<const uint32_t*>(p.ids)[at] : static_cast<const uint16_t*>(p.ids)[at];
        if (!DOWN) srw[i] = p.rw[r * p.ld_w + s];
        sids[i] = id < (uint32_t)p.E ? (uint16_t)id : (uint16_t)0xFFFF;
        if (id < (uint32_t)p.E) atomicOr(&bm[id >> 5], 1u << (id & 31));
    }
    __syncthreads();
    if (warp == 0) {
        uint32_t word = bm[lane];
        const int c = __popc(word);
        int upto = c;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int v = __shfl_up_sync(0xFFFFFFFFu, upto, d);
            if (lane >= d) upto += v;
        }
        if (lane == 31) sflag[1] = min(upto, p.slots);
        for (int at = upto - c; word; word &= word - 1) ulist[at++] = (uint16_t)(lane * 32 + __ffs(word) - 1);
    }
    __syncthreads();
    const int U = sflag[1], NP = p.npad / 128, R = p.R, K = p.K, nst = p.nstages, nch = (K + CK - 1) / CK;
    const int nsa_total = (K + F::KSA - 1) / F::KSA;
    const int tiles = DOWN ? (U ? NP : 0) : U * NP, nb = DOWN ? U * nch : nch;
    // runs of units: whole tiles, or blocks where that saves the longest run two blocks (what cutting costs); no CTA's run is
    // empty (those past the last unit have none at all)
    const int whole = (tiles + (int)gridDim.x - 1) / (int)gridDim.x * nb, fine = (tiles * nb + (int)gridDim.x - 1) / (int)gridDim.x;
    const int step = !p.counters || whole <= fine + 2 ? nb : 1;
    const int64_t units = step == 1 ? (int64_t)tiles * nb : tiles;
    const int grid = (int)min((int64_t)gridDim.x, max(units, (int64_t)1)), cta = min((int)blockIdx.x, grid);
    const int i0 = (int)(units * cta / grid) * step, i1 = (int)(units * min(cta + 1, grid) / grid) * step;
    // where block `it` lies
    struct At {
        int tile, j, q, c;  // tile, block of the tile, slot of the union, chunk
    };
    auto at_of = [&](int it) {
        At a;
        a.tile = it / nb, a.j = it - a.tile * nb;
        a.q = DOWN ? a.j / nch : a.tile / NP, a.c = DOWN ? a.j - a.q * nch : a.j;
        return a;
    };
    auto advance = [&](At& a) {
        ++a.j;
        if (++a.c == nch) {
            a.c = 0;
            if (DOWN) ++a.q;
        }
        if (a.j == nb) {
            a.j = a.c = 0, ++a.tile;
            if (DOWN)
                a.q = 0;
            else if (a.tile % NP == 0)
                ++a.q;
        }
    };

    // gate_up: the rows that chose the expert of slot q, a bit each (by a whole warp). Up to eight of them (of 16 rows and 8 of 128 experts
    // one or two as a rule) are brought and multiplied alone, as rows 0, 1, ..: one MMA a fragment. Us of gate_up with all rows multiplied /
    // so: 8 of 128 experts of 2048 x 1536, 16 rows 54.1 / 47.6, 24 rows 80.9 / 72.7, 32 rows 106.3 / 78.1; 2 of 8 of 4096 x 4096, 16
    // rows 30.5 / 29.3, 24 rows 38.7 / 40.2, 32 rows 46.5 / 47.9. (A producer that walks the bits, a row after the other, took the
    // latter's 16 rows to 33.5; one that brings all rows the former's 15 rows from 44.2 to 48.5. With the scales in the activations
    // instead of the weights 16 rows of the former take 0.7 us less, but then an input's range depends on how many rows chose the expert.)
    constexpr bool PICK = !DOWN && MT > 1 && FMT == TKD_BFP4;
    auto rows_of = [&](int q) {
        const int e = ulist[q];
        bool mine = false;
        if (lane < R)
            for (int s = 0; s < p.k; ++s) mine |= sids[lane * p.k + s] == e;
        return __ballot_sync(0xFFFFFFFFu, mine);
    };

    if (warp == 0) {
        // ---------------------------------------------------------------- producer
        int qm = -1, row = 0, nfew = 0;
        uint32_t st = 0;
        bool ok = true;
        if (i0 < i1) {
            At a = at_of(i0);
            for (int it = i0; it < i1; ++it, ++st, advance(a)) {
                const int panel = DOWN ? a.tile : a.tile - a.q * NP;
                const uint32_t s = st % nst, dst = ring0 + s * p.stage_bytes;
                ok = mbar_wait_parked(empty0 + 8 * s, ((st / nst) & 1) ^ 1, p.status);
                if (!ok) break;
                if (lane == 0) {
                    const uint32_t bytes = (uint32_t)min(F::SUBSA, nsa_total - a.c * F::SUBSA) * F::SAB * 8;
                    mbar_expect_tx(full0 + 8 * s, bytes);
                    bulk_g2s(dst, p.w + (int64_t)ulist[a.q] * p.wbytes + (int64_t)panel * p.panel_bytes + (int64_t)a.c * (F::SUBSA * F::SAB * 8),
                             bytes, full0 + 8 * s);
                }
                // the rows' inputs, 8 k a piece
                const uint16_t* xq = p.x + (DOWN ? (int64_t)a.q * K : 0) + a.c * CK;
                const int pieces = min(CK, K - a.c * CK) / 8;
                if (PICK && a.q != qm) {  // (lane i < 8: the i-th of the rows that chose the expert)
                    qm = a.q;
                    const uint32_t mask = rows_of(qm);
                    nfew = __popc(mask);
                    row = nfew <= 8 && lane < nfew ? (int)__fns(mask, 0, lane + 1) : 0;
                }
                const bool few = PICK && nfew <= 8;
                if (few) {
                    const uint16_t* xl = xq + lane * 8;
                    const uint32_t xd = dst + p.w_bytes + lane * 16;
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int64_t off = (int64_t)__shfl_sync(0xFFFFFFFFu, row, i) * p.ldx;
                        if (i < nfew) {
#pragma unroll
                            for (int e = 0; e < CK / 8; e += 32)
                                if (lane + e < pieces)
                                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(xd + i * p.x_stride + e * 16), "l"(xl + off + e * 8) : "memory");
                        }
                    }
                }
                for (int e = lane; !few && e < pieces; e += 32) {
                    const uint16_t* xr = xq + e * 8;
                    uint32_t xd = dst + p.w_bytes + e * 16;
#pragma unroll 8
                    for (int r = 0; r < R; ++r, xr += p.ldx, xd += p.x_stride)
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(xd), "l"(xr) : "memory");
                }
                asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(full0 + 8 * s) : "memory");
                __syncwarp();
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        if (!ok)  // (the bulk copies in flight land before the CTA goes)
            for (uint32_t back = 1; back <= (uint32_t)nst && back <= st; ++back)
                for (uint32_t i = 0; i < 64; ++i)
                    if (mbar_try_wait(full0 + 8 * ((st - back) % nst), ((st - back) / nst) & 1)) break;
    } else if (warp <= kMrStream) {
        // ---------------------------------------------------------------- streaming warps
        const int cw = warp - 1, g8 = cw & 7, h = cw >> 3, g = lane >> 2, t = lane & 3;
        const uint2 sh = make_uint2(p.mul16, p.mul128);
        uint32_t xrow[MT];  // this lane's rows (one past R reads the last: a column of B only feeds its own column of D)
#pragma unroll
        for (int m = 0; m < MT; ++m) xrow[m] = p.w_bytes + min(8 * m + g, R - 1) * p.x_stride + 16 * t;
        float acc[2][MT][4], tot[MT][4];
        auto clear = [&]() {
#pragma unroll
            for (int a = 0; a < 2; ++a)
#pragma unroll
                for (int m = 0; m < MT; ++m) acc[a][m][0] = acc[a][m][1] = acc[a][m][2] = acc[a][m][3] = 0.f;
        };
        auto clear_tot = [&]() {
#pragma unroll
            for (int m = 0; m < MT; ++m) tot[m][0] = tot[m][1] = tot[m][2] = tot[m][3] = 0.f;
        };
        uint32_t slot = 0, phase = 0, np = 0;
        int qm = -1;
        bool few = false;
        clear(), clear_tot();
        At a = {0, 0, 0, 0};
        if (i0 < i1) a = at_of(i0);
        for (int it = i0; it < i1; ++it) {
            const int c = a.c;
            if (PICK && a.q != qm) {
                qm = a.q;
                const int n = __popc(rows_of(qm));
                few = n <= 8;  // (then this lane's one row is in xrow[0]: another register for it spilled at 17 to 24 rows)
                xrow[0] = p.w_bytes + (uint32_t)max(min(g, (few ? n : R) - 1), 0) * p.x_stride + 16 * t;
            }
            // (the expert's last block here: its group's largest exponent is asked for before the stage is waited for)
            const bool fold = c == nch - 1 || it == i1 - 1, deliver = a.j == nb - 1 || it == i1 - 1;
            int ebyte = 0;
            if constexpr (FMT == TKD_BFP4)
                if (fold) ebyte = p.emax[(int64_t)ulist[a.q] * (p.npad / 16) + (DOWN ? a.tile : a.tile - a.q * NP) * 8 + g8];
            if (!mbar_wait(full0 + 8 * slot, phase, p.status)) break;
            const int nsa = min(F::SUBSA, nsa_total - c * F::SUBSA);
            const uint32_t sb = ring0 + slot * p.stage_bytes, gb = sb + g8 * nsa * F::SAB;
            // (a whole chunk without the checks, so that its loads run ahead of its arithmetic)
            auto chunk = [&](auto full, auto picked) {
                constexpr bool FULL = decltype(full)::value, FEW = decltype(picked)::value;
#pragma unroll
                for (int i = 0; i < F::SUBSA / 2; ++i) {
                    const int sa = h + 2 * i;
                    if (!FULL && sa >= nsa) break;
                    const uint32_t ab = gb + sa * F::SAB;
                    if constexpr (FMT == TKD_BFP4) {
                        const uint4 ev = lds128(ab + t * 16), cv = lds128(ab + EXPB + lane * 16);
#pragma unroll
                        for (int q = 0; q < 2; ++q) {
                            if (!FULL && c * CK + sa * F::KSA + 32 * q >= K) break;  // (a K that ends inside the super-atom)
                            uint4 xv[MT];
#pragma unroll
                            for (int m = 0; m < (FEW ? 1 : MT); ++m) xv[m] = lds128(sb + xrow[m] + (sa * F::KSA + 32 * q) * 2);
                            const uint32_t cwd[4] = {q ? cv.z : cv.x, q ? cv.w : cv.y, 0u, 0u}, ewd[2] = {q ? ev.z : ev.x, q ? ev.w : ev.y};
                            if constexpr (MT == 1) {
                                block_mma<TKD_BFP4, MT, 2>(acc, cwd, ewd, xv, sh);
                            } else {
#pragma unroll
                                for (int jj = 0; jj < 2; ++jj) {
                                    const uint32_t w = cwd[jj], w8 = __funnelshift_r(w, w, 8);
                                    const uint32_t s0 = and_or(ewd[jj], TKD_EMASK_BFP4, ebase(sh));
                                    const uint32_t s1 = and_or(shl_fma<7>(ewd[jj], sh.y), TKD_EMASK_BFP4, ebase(sh));
                                    const uint32_t a0 = mul_bf16x2(w & TKD_MASK_BFP4, s0), a1 = mul_bf16x2(shl_fma<4>(w, sh.x) & TKD_MASK_BFP4, s0);
                                    const uint32_t a2 = mul_bf16x2(w8 & TKD_MASK_BFP4, s1), a3 = mul_bf16x2(shl_fma<4>(w8, sh.x) & TKD_MASK_BFP4, s1);
#pragma unroll
                                    for (int m = 0; m < (FEW ? 1 : MT); ++m)
                                        mma_bf16(acc[jj][m], a0, a1, a2, a3, jj ? xv[m].z : xv[m].x, jj ? xv[m].w : xv[m].y);
                                }
                            }
                        }
                    } else {
                        const uint4 wa = lds128(ab + lane * 16), wb = lds128(ab + 512 + lane * 16);
#pragma unroll
                        for (int m = 0; m < MT; ++m) {
                            const uint4 xv = lds128(sb + xrow[m] + sa * F::KSA * 2);
                            mma_bf16(acc[0][m], wa.x, wa.y, wa.z, wa.w, xv.x, xv.y);
                            mma_bf16(acc[1][m], wb.x, wb.y, wb.z, wb.w, xv.z, xv.w);
                        }
                    }
                }
            };
            if (PICK && few) {
                if constexpr (PICK) {
                    if (c * CK + CK <= K)
                        chunk(std::true_type{}, std::true_type{});
                    else
                        chunk(std::false_type{}, std::true_type{});
                }
            } else if (c * CK + CK <= K) {
                chunk(std::true_type{}, std::false_type{});
            } else {
                chunk(std::false_type{}, std::false_type{});
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(empty0 + 8 * slot);
            if (++slot == (uint32_t)nst) slot = 0, phase ^= 1;
            if (fold) {
                float f1 = 1.f, f2 = 1.f;  // 2^e in two normal floats
                if constexpr (FMT == TKD_BFP4) {
                    const int e = tkd_out_exp(FMT, ebyte), e1 = e / 2;
                    f1 = __uint_as_float((uint32_t)(e1 + 127) << 23), f2 = __uint_as_float((uint32_t)(e - e1 + 127) << 23);
                }
#pragma unroll
                for (int m = 0; m < MT; ++m)
#pragma unroll
                    for (int e = 0; e < 4; ++e) tot[m][e] += (acc[0][m][e] + acc[1][m][e]) * f1 * f2;
                clear();
            }
            if (deliver) {
                if (!mbar_wait(pempty, (np & 1) ^ 1, p.status)) break;
                float* d = pbuf + ((size_t)h * 128 + g8 * 16 + g) * MP + 2 * t;
#pragma unroll
                for (int m = 0; m < MT; ++m) {
                    *reinterpret_cast<float2*>(d + 8 * m) = make_float2(tot[m][0], tot[m][1]);
                    *reinterpret_cast<float2*>(d + 8 * MP + 8 * m) = make_float2(tot[m][2], tot[m][3]);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(pfull);
                ++np;
                clear_tot();
            }
            advance(a);
        }
    } else {
        // ---------------------------------------------------------------- output warps
        const int et = tid - (1 + kMrStream) * 32;
        // zeros: rows past R, and what no expert fills (gate_up: the slots past the union; down: all of y without any expert)
        {
            const int wide = DOWN ? p.N : p.slots * (p.N / 2), used = DOWN ? (U ? p.N : 0) : U * (p.N / 2);  // (multiples of 8)
            const int tail = (wide - used) / 8, per = wide / 8, n1 = R * tail, n2 = max(0, p.out_rows - R) * per;
            for (int i = (int)blockIdx.x * 128 + et; i < n1 + n2; i += (int)gridDim.x * 128) {
                const int r = i < n1 ? i / tail : R + (i - n1) / per, c = i < n1 ? used / 8 + i % tail : (i - n1) % per;
                uint16_t* o = p.out + (int64_t)r * p.ldo + c * 8;
                if (!((reinterpret_cast<uintptr_t>(p.out) & 15) | (p.ldo & 7))) {
                    *reinterpret_cast<uint4*>(o) = make_uint4(0u, 0u, 0u, 0u);
                } else {
                    for (int b = 0; b < 8; ++b) o[b] = 0;
                }
            }
        }
        uint32_t np = 0;
        bool met = true;
        int qw = -1;  // the slot whose routing weights are in wrow
        uint32_t mask = 0;
        float* const col = pbuf + (size_t)et * MP;
        for (int it = i0; it < i1; ++np) {
            const int tile = it / nb, j0 = it - tile * nb, j1 = min(nb, j0 + i1 - it);
            it += j1 - j0;
            const int q = DOWN ? 0 : tile / NP, panel = DOWN ? tile : tile - q * NP;
            const int o = et & 63, r0 = (et >> 6) * (4 * MT), gc = 64 * (o >> 5) + (o & 31);  // (gate_up: output o, half of the rows)
            float bg = 0.f, bu = 0.f;
            if constexpr (!DOWN) {
                const int e = ulist[q];
                if (q != qw && et < 32) {
                    float wv = 0.f;
                    if (et < R)
                        for (int s = 0; s < p.k; ++s)
                            if (sids[et * p.k + s] == e) wv = bf16_bits_to_f32(srw[et * p.k + s]);
                    wrow[et] = wv;  // (the tile before ended with a barrier)
                }
                if (PICK && q != qw) mask = rows_of(q);
                qw = q;
                if (p.bias) {
                    const uint16_t* b = p.bias + (int64_t)e * p.npad + panel * 128 + gc;
                    bg = bf16_bits_to_f32(b[0]), bu = bf16_bits_to_f32(b[32]);
                }
            }
            if (!mbar_wait_parked(pfull, np & 1, p.status, met)) met = false;  // (and on: see mbar_wait)
            float v[RW];  // the column's sums
#pragma unroll
            for (int m = 0; m < RW; m += 4) {
                const float4 x0 = *reinterpret_cast<const float4*>(col + m), x1 = *reinterpret_cast<const float4*>(col + 128 * MP + m);
                v[m] = x0.x + x1.x, v[m + 1] = x0.y + x1.y, v[m + 2] = x0.z + x1.z, v[m + 3] = x0.w + x1.w;
            }
            bool finish = j1 - j0 == nb;
            if (!finish) {
                constexpr int part = 128 * RW;
                float* dst = p.scratch + ((int64_t)blockIdx.x * 2 + (i0 < tile * nb ? 1 : 0)) * part + et * 4;
#pragma unroll
                for (int m = 0; m < RW; m += 4) __stcg(reinterpret_cast<float4*>(dst + m * 128), make_float4(v[m], v[m + 1], v[m + 2], v[m + 3]));
                bar_output_warps();  // (orders the 128 threads' stores before thread 0's release)
                if (et == 0) {
                    const int last = atom_add_acq_rel(p.counters + tile, j1 - j0) + j1 - j0 == nb;
                    if (last) p.counters[tile] = 0;
                    sflag[0] = last;
                }
                bar_output_warps();
                finish = sflag[0] != 0;
                if (finish) {
                    // the parts in order: the CTAs whose runs meet the tile's blocks
                    const int b0 = (int)((((int64_t)tile * nb + 1) * grid - 1) / units), b1 = (int)((((int64_t)tile * nb + nb) * grid - 1) / units);
                    auto part_of = [&](int b) {
                        return p.scratch + ((int64_t)b * 2 + ((int)(units * b / grid) < tile * nb ? 1 : 0)) * part + et * 4;
                    };
                    // the CTA's last tile: the ring is idle, and the parts come into it together (one trip to L2 instead of one
                    // for every two parts)
                    const bool staged = it >= i1 && (b1 - b0 + 1) * part * 4 <= nst * p.stage_bytes;
                    if (staged) {
                        for (int b = b0; b <= b1; ++b) {
                            const float* src = part_of(b);
#pragma unroll
                            for (int m = 0; m < RW; m += 4)
                                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(ring0 + ((b - b0) * part + m * 128 + et * 4) * 4),
                                             "l"(src + m * 128)
                                             : "memory");
                        }
                        asm volatile("cp.async.wait_all;" ::: "memory");
                    }
#pragma unroll
                    for (int m = 0; m < RW; ++m) v[m] = 0.f;
#pragma unroll 2
                    for (int b = b0; b <= b1; ++b) {
                        const float* src = part_of(b);
#pragma unroll
                        for (int m = 0; m < RW; m += 4) {
                            float4 f;
                            if (staged) {
                                const uint4 w = lds128(ring0 + ((b - b0) * part + m * 128 + et * 4) * 4);
                                f = make_float4(__uint_as_float(w.x), __uint_as_float(w.y), __uint_as_float(w.z), __uint_as_float(w.w));
                            } else {
                                f = __ldcg(reinterpret_cast<const float4*>(src + m * 128));
                            }
                            v[m] += f.x, v[m + 1] += f.y, v[m + 2] += f.z, v[m + 3] += f.w;
                        }
                    }
                }
            }
            if constexpr (DOWN) {
                const int n = panel * 128 + et, left = finish && n < p.N ? R : 0;
                uint16_t* op = p.out + n;
#pragma unroll
                for (int m = 0; m < RW; ++m, op += p.ldo) st16_if(m < left, op, f32_to_bf16_bits(v[m]));
            } else if (finish) {
#pragma unroll
                for (int m = 0; m < RW; m += 4) *reinterpret_cast<float4*>(col + m) = make_float4(v[m], v[m + 1], v[m + 2], v[m + 3]);
                bar_output_warps();
                const float *gp = pbuf + gc * MP + r0, *up = gp + 32 * MP;
                uint16_t* op = p.out + (int64_t)r0 * p.ldo + (int64_t)q * (p.N / 2) + panel * 64 + o;
                const int left = panel * 64 + o < p.N / 2 ? R - r0 : 0;
                auto value = [&](int at, int m) { return f32_to_bf16_bits(moe_glu(gp[at] + bg, up[at] + bu, p.act) * wrow[r0 + m]); };
                if (PICK && __popc(mask) <= 8) {
                    // (the rows multiplied lie together, in order; the others' outputs are zeros)
                    const uint32_t mine = mask >> r0 & ((1u << 4 * MT) - 1u);
                    int at = __popc(mask & ((1u << r0) - 1u)) - r0;
#pragma unroll
                    for (int m = 0; m < 4 * MT; ++m) st16_if(m < left && !(mine >> m & 1u), op + m * p.ldo, (uint16_t)0);
#pragma unroll 1
                    for (uint32_t b = left > 0 ? mine : 0u; b; b &= b - 1, ++at) {
                        const int m = __ffs(b) - 1;
                        op[m * p.ldo] = value(at, m);
                    }
                } else {
#pragma unroll
                    for (int m = 0; m < 4 * MT; ++m, op += p.ldo) st16_if(m < left, op, value(m, m));
                }
            }
            bar_output_warps();  // (the sums, wrow and sflag are read)
            if (lane == 0) mbar_arrive(pempty);
        }
    }
}

// The stages of the ring that fit, and the shared memory; false: fewer than two.
template <int FMT>
bool moe_rows_smem(MoeRowsParams& p, int mt, size_t* smem) {
    using F = Fmt<FMT>;
    p.w_bytes = 8 * F::SUBSA * F::SAB;
    p.x_stride = F::SUBSA * F::KSA * 2 + 64;  // (16 banks on from row to row: the 8 rows a quarter-warp reads lie in different ones)
    p.stage_bytes = (p.w_bytes + p.R * p.x_stride + 127) & ~127;
    p.off_pbuf = kMrHead;
    p.off_ring = (p.off_pbuf + 2 * 128 * (8 * mt + 4) * 4 + 127) & ~127;
    p.nstages = (227 * 1024 - p.off_ring) / p.stage_bytes;
    if (p.nstages > TKD_MAX_STAGES) p.nstages = TKD_MAX_STAGES;
    *smem = (size_t)p.off_ring + (size_t)p.nstages * p.stage_bytes;
    return p.nstages >= 2;
}

template <int FMT, int MT, bool DOWN>
int moe_rows_launch(const MoeRowsParams& p, int grid, size_t smem, cudaStream_t st) {
    auto kern = tkd_moe_rows_kernel<FMT, MT, DOWN>;
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
    cfg.gridDim = dim3((unsigned)grid), cfg.blockDim = dim3(kMrWarps * 32), cfg.dynamicSmemBytes = smem, cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr, cfg.numAttrs = 1;
    return (int)cudaLaunchKernelEx(&cfg, kern, p);
}

}  // namespace
