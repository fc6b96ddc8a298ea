// tkd_rows.cuh: the streaming matmul of 9 to 32 rows as items of 32 columns over all of K, the rows of x whole in shared memory.
//
// The tensor-memory kernel (tkd_stream_tc.cuh) pays for a launch: 1.1 us of tensor-memory allocation, a unit's way from decode warps
// over an MMA warp to output warps, and unless K makes four slices a panel's sums through L2; and it brings every tile of x for every
// panel anew. Where x fits in shared memory, mma.sync on weights in registers does without all of that: 16 rows of bfloat8_b,
// [2048, 4096] 7.8 us before, 5.5 now (1.4 at the memory's rate), bfloat4_b [1280, 4096] 7.6 and 5.0. What bounds it on large weights is
// instruction issue: 39 warp instructions for 256 weights and 16 rows, issue active in 0.56 of the cycles (bfloat8_b [2048, 28672]). rows_layout (tkd_api.cu) says where which kernel runs.
//
//   warps 0-3      output: a quarter of the rows each, a lane a column (GLU: 16 gate columns and their 16 up columns). The first
//                  warps: the schedulers favour older ones, and beside four streaming warps that are always ready these took 1.4 us an
//                  item
//   warp 4         producer: a stage of the ring is SC chunks of K, 2 groups of 16 columns each (a copy each; GLU: the gate's group
//                  and the up's apart)
//   warps 5-20     streaming: a warp takes every sixteenth super-atom of a stage, both groups of it: the weights become bf16 once (a
//                  code times 2^e', which is exact) and are multiplied with mma.sync, 8 rows an MMA, by rows of x that both groups
//                  share. They bring x as well, 16 bytes a lane, a stage's part of K after the other
//
// A column's sum: streaming warp w's sums T_w over all its super-atoms, U_i = T_i + T_{i + 8}, then U_0 + U_1 + .. + U_7 in order. It
// depends on K and the format only; where this kernel runs goes by the number of rows as well (rows_layout).
#pragma once
#include "tkd_narrow.cuh"

namespace {

constexpr int kRowsStream = 16, kRowsPitch = TKD_ROWS_PITCH, kRowsSegs = 8, kRowsOut = 4, kRowsWarps = kRowsOut + 1 + kRowsStream;

__device__ __forceinline__ float lds32f(uint32_t a) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
    return v;
}

// The two k16 blocks of a k32 block of 16 columns as bf16 A fragments. cw, ew: the lane's code and exponent words.
template <int FMT>
__device__ __forceinline__ void rows_decode(uint32_t (&a)[2][4], const uint32_t (&cw)[4], const uint32_t (&ew)[2], const uint2 sh) {
#pragma unroll
    for (int jj = 0; jj < 2; ++jj) {
        uint32_t a0, a1, a2, a3, s0, s1;
        if constexpr (FMT == TKD_BFP4) {
            const uint32_t w = cw[jj], t = __funnelshift_r(w, w, 8);
            a0 = w & TKD_MASK_BFP4, a1 = shl_fma<4>(w, sh.x) & TKD_MASK_BFP4;
            a2 = t & TKD_MASK_BFP4, a3 = shl_fma<4>(t, sh.x) & TKD_MASK_BFP4;
            s0 = and_or(ew[jj], TKD_EMASK_BFP4, ebase(sh));
            s1 = and_or(shl_fma<7>(ew[jj], sh.y), TKD_EMASK_BFP4, ebase(sh));
        } else {
            const uint32_t w0 = cw[2 * jj], w1 = cw[2 * jj + 1];
            a0 = w0 & TKD_MASK_BFP8, a1 = rot_and<8>(w0, TKD_MASK_BFP8);
            a2 = w1 & TKD_MASK_BFP8, a3 = rot_and<8>(w1, TKD_MASK_BFP8);
            s0 = ew[jj] & 0x7F807F80u, s1 = rot_and<8>(ew[jj], 0x7F807F80u);
        }
        a[jj][0] = mul_bf16x2(a0, s0), a[jj][1] = mul_bf16x2(a1, s0);
        a[jj][2] = mul_bf16x2(a2, s1), a[jj][3] = mul_bf16x2(a3, s1);
    }
}

// One super-atom of two groups of columns: ca, ea: the lane's code and exponent words of the first group's, GS bytes on (0: gs) the
// second's; xa: its 16 bytes of x of each eight rows. OW, OX: distances from there, known at compile time.
template <int FMT, int MT, int OW, int OX, int GS>
__device__ __forceinline__ void rows_block(float (&acc)[2][MT][4], uint32_t ca, uint32_t ea, uint32_t gs, const uint32_t (&xa)[MT], const uint2 sh) {
    using F = Fmt<FMT>;
    const uint32_t cb = GS ? ca : ca + gs, eb = GS ? ea : ea + gs;
    if constexpr (FMT == TKD_BF16) {
        const uint4 wv[2][2] = {{lds128_at<OW>(ca), lds128_at<OW + 512>(ca)}, {lds128_at<OW + GS>(cb), lds128_at<OW + GS + 512>(cb)}};
        uint4 xv[MT];
#pragma unroll
        for (int m = 0; m < MT; ++m) xv[m] = lds128_at<OX>(xa[m]);
#pragma unroll
        for (int gr = 0; gr < 2; ++gr)
#pragma unroll
            for (int jj = 0; jj < 2; ++jj)
#pragma unroll
                for (int m = 0; m < MT; ++m)
                    mma_bf16(acc[gr][m], wv[gr][jj].x, wv[gr][jj].y, wv[gr][jj].z, wv[gr][jj].w, jj ? xv[m].z : xv[m].x, jj ? xv[m].w : xv[m].y);
    } else {
        const uint4 cv[2] = {lds128_at<OW>(ca), lds128_at<OW + GS>(cb)};
        uint4 ev[2];
        if constexpr (FMT == TKD_BFP4) {
            ev[0] = lds128_at<OW>(ea), ev[1] = lds128_at<OW + GS>(eb);
        } else {
            const uint2 e0 = lds64_at<OW>(ea), e1 = lds64_at<OW + GS>(eb);
            ev[0] = make_uint4(e0.x, e0.y, 0u, 0u), ev[1] = make_uint4(e1.x, e1.y, 0u, 0u);
        }
        unrolled(std::make_integer_sequence<int, F::XB>{}, [&](auto qc) {
            constexpr int q = decltype(qc)::value;
            uint4 xv[MT];
#pragma unroll
            for (int m = 0; m < MT; ++m) xv[m] = lds128_at<OX + q * 64>(xa[m]);
#pragma unroll
            for (int gr = 0; gr < 2; ++gr) {
                uint32_t w[2][4];
                const uint4 v = cv[gr];
                const uint32_t cws[4] = {FMT == TKD_BFP4 && q ? v.z : v.x, FMT == TKD_BFP4 && q ? v.w : v.y, v.z, v.w};
                const uint32_t ews[2] = {q ? ev[gr].z : ev[gr].x, q ? ev[gr].w : ev[gr].y};
                rows_decode<FMT>(w, cws, ews, sh);
#pragma unroll
                for (int jj = 0; jj < 2; ++jj)
#pragma unroll
                    for (int m = 0; m < MT; ++m)
                        mma_bf16(acc[gr][m], w[jj][0], w[jj][1], w[jj][2], w[jj][3], jj ? xv[m].z : xv[m].x, jj ? xv[m].w : xv[m].y);
            }
        });
    }
}

// SC: chunks of a stage (TkdParams.rows_chunks). PLAIN: no top-k records and no exchange with other GPUs. TURNS: fewer CTAs than
// tiles of rows (two tiles, and max_ctas leaves one CTA), which take their tiles in turn, the ring and the hand-over of sums running on;
// an instance of its own, so that the others keep their code.
template <int FMT, int MT, int SC, bool PLAIN, bool TURNS>
__global__ void __launch_bounds__(kRowsWarps * 32, 1) tkd_rows_kernel(const __grid_constant__ TkdParams p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    using F = Fmt<FMT>;
    constexpr int SW = kRowsStream, CK = F::SUBSA * F::KSA, GB = F::SUBSA * F::SAB, PP = kRowsPitch;
    constexpr int EXPB = FMT == TKD_BFP4 ? 64 : (FMT == TKD_BFP8 ? 32 : 0);
    constexpr int SLOT = 8 * MT * PP * 4;  // bytes of a warp's sums: [row][column]
    constexpr int RW = 2 * MT;             // rows of an output warp
    static_assert(SC * F::SUBSA % SW == 0, "a stage is as many super-atoms for every streaming warp");
    const uint32_t full0 = smem_u32(smem), empty0 = full0 + 8 * TKD_MAX_STAGES, xbar0 = empty0 + 8 * TKD_MAX_STAGES;
    const uint32_t half0 = xbar0 + 8 * kRowsSegs, pfull = half0 + 64, pempty = pfull + 8;
    const uint32_t pbuf = smem_u32(smem + p.off_pbuf), ring0 = smem_u32(smem + p.off_ring), xt0 = smem_u32(smem + p.off_xt);
    volatile int* sflag = reinterpret_cast<volatile int*>(smem + TKD_SMEM_HEAD - 16);
    // (the warp's number by a shuffle, as in tkd_narrow_kernel: 9 rows of bfloat4_b [4096, 57344] 41.2 us without, 37.3 so; bfloat8_b 48.7
    // and 47.6; 17 rows of bfloat4_b [1152, 4288], two tiles, 6.5 and 5.1)
    const int tid = threadIdx.x, warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0), lane = tid & 31;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (tid == 0) {
        for (int s = 0; s < p.nstages; ++s) mbar_init(full0 + 8 * s, 1), mbar_init(empty0 + 8 * s, SW);
        for (int s = 0; s < kRowsSegs; ++s) mbar_init(xbar0 + 8 * s, SW * 32);
        for (int s = 0; s < 8; ++s) mbar_init(half0 + 8 * s, 1);
        mbar_init(pfull, 8), mbar_init(pempty, kRowsOut);
        sflag[0] = sflag[1] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    const uint32_t T = 4u * (uint32_t)p.total_panels;  // items
    // (tiles of rows: a team of CTAs each)
    const uint32_t team = p.rows_team ? p.rows_team : gridDim.x, tile = blockIdx.x / team, cta = blockIdx.x - tile * team;
    const int i0 = (int)((uint64_t)T * cta / team), i1 = (int)((uint64_t)T * (cta + 1) / team);
    int row0 = (int)tile * p.rows_tile, M = p.rows_tile ? min(p.rows_tile, p.M - row0) : p.M;
    // (TURNS: the first row and the number of rows of the tile after this one, `step` tiles on; false: there is none)
    const int step = TURNS ? gridDim.x / team * p.rows_tile : 0;
    auto next_tile = [&]() {
        row0 += step, M = min(p.rows_tile, p.M - row0);
        return TURNS && row0 < p.M;
    };
    const int nst = p.nstages, K = p.K, nch = (K + CK - 1) / CK, nsa_total = (K + F::KSA - 1) / F::KSA;
    const int spi = (nch + SC - 1) / SC;  // stages of an item
    const int epi = p.epi;
    const bool glu = epi == TKD_EPI_GLU2 || epi == TKD_EPI_GLU_IL;
    auto seg_of = [&](int it) {
        int s = 0;
#pragma unroll
        for (int q = 1; q < 4; ++q)
            if (q < p.nseg && it >= 4 * p.seg[q].panel0) s = q;
        return s;
    };

    if (warp == kRowsOut) {
        // ---------------------------------------------------------------- producer: lane 2 s + g brings chunk s's share of group g
        // (not GLU: lane 2 s both groups', which lie together)
        uint32_t st = 0;
        bool ok = true;
        const int s = lane >> 1, g = lane & 1;
        do {
            for (int it = i0; ok && it < i1; ++it) {
                const TkdSegDev& sg = p.seg[seg_of(it)];
                const NarrowItem n = narrow_item(p, it - 4 * sg.panel0);
                const uint8_t* src = (g && epi == TKD_EPI_GLU2 ? sg.w2 : sg.w) + (int64_t)n.panel * p.panel_bytes;
                for (int i = 0; i < spi; ++i, ++st) {
                    const uint32_t q = st % nst;
                    ok = __all_sync(0xFFFFFFFFu, mbar_wait_parked(empty0 + 8 * q, ((st / nst) & 1) ^ 1, p.status));
                    if (!ok) break;
                    const int c = i * SC + s;  // this lane's chunk, if there is one
                    const bool mine = s < SC && c < nch && (glu || !g);
                    const uint32_t gb = mine ? (uint32_t)min(F::SUBSA, nsa_total - c * F::SUBSA) * F::SAB : 0u, bytes = glu ? gb : 2 * gb;
                    const uint32_t all = __reduce_add_sync(0xFFFFFFFFu, bytes);
                    if (lane == 0) mbar_expect_tx(full0 + 8 * q, all);
                    __syncwarp();
                    if (mine)
                        bulk_g2s(ring0 + q * p.stage_bytes + s * 2 * GB + g * gb, src + (int64_t)c * (GB * 8) + (int64_t)(g ? n.gb : n.ga) * gb, bytes,
                                 full0 + 8 * q);
                }
            }
        } while (TURNS && next_tile());
        if (!ok)  // (the copies in flight land before the CTA goes)
            for (uint32_t back = 1; back <= (uint32_t)nst && back <= st; ++back)
                for (uint32_t i = 0; i < 64; ++i)
                    if (mbar_try_wait(full0 + 8 * ((st - back) % nst), ((st - back) / nst) & 1)) break;
    } else if (warp > kRowsOut) {
        // ---------------------------------------------------------------- streaming warps
        const int cw = warp - kRowsOut - 1, g = lane >> 2, t = lane & 3;
        if (nch * CK > K) {
            // the rows of x end in zeros up to a whole chunk
            for (int r = cw; r < M; r += SW)  // (no later tile has more)
                for (int e = K / 8 + lane; e < nch * (CK / 8); e += 32)
                    asm volatile("st.shared.v4.u32 [%0], {%1,%1,%1,%1};" ::"r"(xt0 + r * p.x_stride + e * 16), "r"(0u) : "memory");
            asm volatile("bar.sync 2, %0;" ::"n"(SW * 32) : "memory");
        }
        // (x and the outputs may belong to the kernel before this one: wait for it to complete)
        asm volatile("griddepcontrol.wait;" ::: "memory");
        uint32_t at = ring0, bar = full0, phase = 0;
        bool ok = true;
        int n = 0;              // items of the tiles before this one
        uint32_t xphase = 0;
        do {
            for (int s = 0; s < kRowsSegs; ++s) {  // (the last part: all that is left)
                const int e0 = min(s * SC * CK, K) / 8, e1 = s == kRowsSegs - 1 ? K / 8 : min((s + 1) * SC * CK, K) / 8;
                for (int r = cw; r < M; r += SW) {
                    const uint16_t* src = p.x + (int64_t)(row0 + r) * p.ldx;
                    const uint32_t dst = xt0 + r * p.x_stride;
#pragma unroll 4
                    for (int e = e0 + lane; e < e1; e += 32)
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + e * 16), "l"(src + e * 8) : "memory");
                }
                asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(xbar0 + 8 * s) : "memory");
            }
            const uint2 sh = make_uint2(p.mul16, p.mul128);
            // (a lane whose row lies beyond M reads row M - 1: a column of B only feeds its own column of D)
            uint32_t xrow[MT];
#pragma unroll
            for (int m = 0; m < MT; ++m) xrow[m] = xt0 + min(8 * m + g, M - 1) * p.x_stride + t * 16;
            const int cc = cw / F::SUBSA, si = cw % F::SUBSA;  // this warp's (first) super-atom of a stage
            constexpr int NU = SC * F::SUBSA / SW, CSTEP = SW / F::SUBSA;
            const uint32_t gbl = (nsa_total - (nch - 1) * F::SUBSA) * F::SAB;  // a group's share of K's last chunk
            const int cwhole = nsa_total / F::SUBSA;                           // whole chunks
            const uint32_t exp_lane = cc * 2 * GB + si * F::SAB + t * (EXPB / 4), code_lane = cc * 2 * GB + si * F::SAB + EXPB + lane * 16;
            const uint32_t xk0 = (cc * CK + si * F::KSA) * 2;
            const uint32_t ring_end = ring0 + nst * p.stage_bytes;
            const uint32_t slot = pbuf + (cw & 7) * SLOT + ((2 * t) * PP + g) * 4;  // (where this lane's sums go)
            float acc[2][MT][4];
            for (int j0 = 0; ok && j0 < i1 - i0; ++j0) {
                const int j = n + j0;
#pragma unroll
                for (int a = 0; a < 2; ++a)
#pragma unroll
                    for (int m = 0; m < MT; ++m) acc[a][m][0] = acc[a][m][1] = acc[a][m][2] = acc[a][m][3] = 0.f;
                uint32_t xk = xk0;
                int c = 0;
#pragma unroll 1
                for (int i = 0; i < spi; ++i, xk += SC * CK * 2, c += SC) {
                    if (j0 == 0) ok = mbar_wait(xbar0 + 8 * min(i, kRowsSegs - 1), xphase, p.status);
                    ok = ok && mbar_wait(bar, phase, p.status);
                    if (!ok) break;
                    const uint32_t ca = at + code_lane, ea = at + exp_lane;
                    uint32_t xa[MT];
#pragma unroll
                    for (int m = 0; m < MT; ++m) xa[m] = xrow[m] + xk;
                    if (c + SC <= cwhole && MT == 2) {
                        unrolled(std::make_integer_sequence<int, NU>{}, [&](auto uc) {
                            constexpr int u = decltype(uc)::value;
                            rows_block<FMT, MT, u * CSTEP * 2 * GB, u * CSTEP * CK * 2, GB>(acc, ca, ea, 0u, xa, sh);
                        });
                    } else if (c + SC <= cwhole) {
                        // (one after the other: side by side they spill)
#pragma unroll 1
                        for (int u = 0; u < NU; ++u) {
                            const uint32_t by = u * CSTEP * 2 * GB;
                            uint32_t xu[MT];
#pragma unroll
                            for (int m = 0; m < MT; ++m) xu[m] = xa[m] + u * CSTEP * CK * 2;
                            rows_block<FMT, MT, 0, 0, GB>(acc, ca + by, ea + by, 0u, xu, sh);
                        }
                    } else {
                        // (K's last chunk may have fewer super-atoms: its groups lie closer together)
#pragma unroll 1
                        for (int u = 0; u < NU; ++u) {
                            const int ch = c + cc + u * CSTEP;
                            if (ch >= nch || ch * F::SUBSA + si >= nsa_total) break;
                            const uint32_t by = u * CSTEP * 2 * GB;
                            uint32_t xu[MT];
#pragma unroll
                            for (int m = 0; m < MT; ++m) xu[m] = xa[m] + u * CSTEP * CK * 2;
                            rows_block<FMT, MT, 0, 0, 0>(acc, ca + by, ea + by, ch == nch - 1 ? gbl : (uint32_t)GB, xu, sh);
                        }
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar + 8 * TKD_MAX_STAGES);
                    at += p.stage_bytes, bar += 8;
                    if (at == ring_end) at = ring0, bar = full0, phase ^= 1;
                }
                if (!ok) break;
                // ---- the item's sums: the upper eight warps' through shared memory to the lower eight, theirs to the output warps
                if (cw >= 8) {
                    ok = mbar_wait(pempty, (j & 1) ^ 1, p.status);
                    if (!ok) break;
                } else {
                    ok = mbar_wait(half0 + 8 * cw, j & 1, p.status);
                    if (!ok) break;
#pragma unroll
                    for (int a = 0; a < 2; ++a)
#pragma unroll
                        for (int m = 0; m < MT; ++m)
#pragma unroll
                            for (int e = 0; e < 4; ++e) acc[a][m][e] += lds32f(slot + ((8 * m + (e & 1)) * PP + a * 16 + (e >> 1) * 8) * 4);
                }
#pragma unroll
                for (int a = 0; a < 2; ++a)
#pragma unroll
                    for (int m = 0; m < MT; ++m)
#pragma unroll
                        for (int e = 0; e < 4; ++e) sts32(slot + ((8 * m + (e & 1)) * PP + a * 16 + (e >> 1) * 8) * 4, acc[a][m][e]);
                __syncwarp();
                if (lane == 0) mbar_arrive(cw >= 8 ? half0 + 8 * (cw - 8) : pfull);
            }
            if (!TURNS || !next_tile()) break;
            // (every warp has read this tile's rows: one whose wait gave up comes here too)
            asm volatile("bar.sync 2, %0;" ::"n"(SW * 32) : "memory");
            n += i1 - i0, xphase ^= 1;
        } while (true);
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else {
        // ---------------------------------------------------------------- output warps
        asm volatile("griddepcontrol.wait;" ::: "memory");
        const int ow = warp, npeers = PLAIN ? 0 : p.npeers;
        int left = M - RW * ow;  // rows from this warp's first on
        int topk_k = PLAIN || tile ? 0 : p.topk_k;
        const bool up = glu && lane >= 16, f32out = epi == TKD_EPI_OUT32;
        bool met = true;
        int counted = 0;  // items of the current unit of top-k records whose outputs are written and not counted
        for (int j = 0, it = i0;; ++j, ++it) {
            if (it == i1) {
                if (!TURNS || !next_tile()) break;
                it = i0, left = M - RW * ow, topk_k = 0;
            }
            const int seg = seg_of(it);
            const TkdSegDev& sg = p.seg[seg];
            const int pl = it - 4 * sg.panel0;
            const int plw = !PLAIN && p.rep_panels ? pl % (4 * p.rep_panels) : pl;  // (the item's number in its weight)
            // this lane's column of its weight, and what it stores
            int n, oc;
            if (epi == TKD_EPI_GLU2) {
                n = pl * 16 + (lane & 15);
                oc = !up && n < sg.n_valid ? sg.out_col0 + n : -1;
            } else if (glu) {
                n = (pl >> 1) * 64 + (pl & 1) * 16 + (up ? 32 : 0) + (lane & 15);
                oc = !up && n < sg.n_valid ? sg.out_col0 + pl * 16 + lane : -1;
            } else {
                n = plw * 32 + lane;
                oc = n < sg.n_valid ? sg.out_col0 + n : -1;
            }
            const bool other = up && epi == TKD_EPI_GLU2;
            float f1 = 1.f, f2 = 1.f, sc = 1.f;  // 2^e of the group in two normal floats, the column's scale
            if constexpr (FMT != TKD_BF16) {
                const int e = tkd_out_exp(FMT, (other ? sg.emax2 : sg.emax)[(PLAIN || glu ? n : pl * 32 + lane) >> 4]), e1 = e / 2;
                f1 = __uint_as_float((uint32_t)(e1 + 127) << 23), f2 = __uint_as_float((uint32_t)(e - e1 + 127) << 23);
            }
            if (p.scale_dt != TKD_DT_NONE && n < sg.n_valid) {
                const void* sp = other ? p.scale2 : p.scale;
                sc = p.scale_dt == TKD_DT_BF16 ? bf16_bits_to_f32(static_cast<const uint16_t*>(sp)[n]) : static_cast<const float*>(sp)[n];
            }
            // (the residual is asked for now, so that its latency passes while the streaming warps are at work; a row past M reads
            // the last again)
            uint32_t q[RW] = {};
            if (p.res_dt != TKD_DT_NONE && oc >= 0 && left > 0) {
                const int rsz = p.res_dt == TKD_DT_F32 ? 4 : 2;
                const char* rp = static_cast<const char*>(p.res) + ((int64_t)(row0 + RW * ow) * p.ldr + oc) * rsz;
#pragma unroll
                for (int m = 0; m < RW; ++m) {
                    q[m] = rsz == 4 ? *reinterpret_cast<const uint32_t*>(rp) : (uint32_t)*reinterpret_cast<const uint16_t*>(rp) << 16;
                    if (m + 1 < left) rp += p.ldr * rsz;
                }
            }
            // (on after a wait that gave up, where the warps meet at barriers: see mbar_wait)
            if (!mbar_wait(pfull, j & 1, p.status, met)) {
                met = false;
                if (PLAIN) break;
            }
            float v[RW];
            const uint32_t a = pbuf + ((RW * ow) * PP + lane) * 4;
#pragma unroll
            for (int m = 0; m < RW; ++m) v[m] = lds32f(a + m * PP * 4);
#pragma unroll
            for (int s = 1; s < 8; ++s)
#pragma unroll
                for (int m = 0; m < RW; ++m) v[m] += lds32f(a + s * SLOT + m * PP * 4);
            __syncwarp();
            if (lane == 0) mbar_arrive(pempty);
#pragma unroll
            for (int m = 0; m < RW; ++m) v[m] = v[m] * f1 * f2 * sc;
            if (glu || epi == TKD_EPI_SILU) {
#pragma unroll
                for (int m = 0; m < RW; ++m) {
                    const float u = __shfl_xor_sync(0xFFFFFFFFu, v[m], 16);
                    v[m] = act_gate(v[m], p.act) * (glu ? u : 1.f);
                }
            }
            if (p.res_dt != TKD_DT_NONE) {
#pragma unroll
                for (int m = 0; m < RW; ++m) v[m] += __uint_as_float(q[m]);
            }
            char* yp = static_cast<char*>(p.out) + ((int64_t)(row0 + RW * ow) * p.ldo + oc) * (f32out ? 4 : 2);
            const int rows = oc >= 0 && (PLAIN || p.topk_k == 0 || p.write_y) ? left : 0;
#pragma unroll
            for (int m = 0; m < RW; ++m, yp += p.ldo * (f32out ? 4 : 2)) {
                if (f32out)
                    st_if(m < rows, yp, __float_as_uint(v[m]));
                else
                    st16_if(m < rows, yp, f32_to_bf16_bits(v[m]));
            }
            if constexpr (!PLAIN) {
#pragma unroll
                for (int m = 0; m < RW; ++m) {
                    const int r = RW * ow + m;
                    const size_t to = (size_t)(row0 + r) * p.ldo + oc;
                    const uint16_t b = f32_to_bf16_bits(v[m]);
#pragma unroll 1
                    for (int pq = 0; m < rows && pq < npeers; ++pq) {
                        if (!p.peer_out[pq]) continue;
                        if (f32out)
                            static_cast<float*>(p.peer_out[pq])[to] = v[m];
                        else
                            static_cast<uint16_t*>(p.peer_out[pq])[to] = b;
                    }
                    if (topk_k && !p.write_y && oc >= 0 && r < p.topk_rows) p.ytmp[(size_t)r * p.ld_ytmp + it * 32 + lane] = b;
                }
                // (the items of a unit that this CTA has in a row are counted once, after the last: a count is a fence, an atomic and
                // barriers. Counted item by item 16 rows of bfloat8_b [1536, 75968] with records of 4 took 86.8 us, 60.3 now)
                const int wide = 4 * (p.rep_panels ? p.rep_panels : p.total_panels / p.nseg);
                if (topk_k) ++counted;
                if (topk_k && (it + 1 == i1 || plw + 1 == wide || (plw + 1) % (p.topk_unit / 32) == 0)) {
                    const Cursor c = {it >> 2, 0, seg, pl >> 2};
                    const int add = counted;
                    counted = 0;
                    topk_records(p, c, sg, 4, add, tid, ow, lane, reinterpret_cast<float*>(smem + p.off_tbuf), sflag, static_cast<uint16_t*>(p.out), topk_k, npeers);
                }
            }
        }
        if (npeers) exchange_done(p, lane, npeers, sflag);
    }
}

template <int FMT, int MT, int SC, bool PLAIN, bool TURNS = false>
int launch_rows_one(const TkdParams& p, int grid, size_t smem, cudaStream_t st) {
    auto kern = tkd_rows_kernel<FMT, MT, SC, PLAIN, TURNS>;
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
    cfg.gridDim = dim3((unsigned)grid), cfg.blockDim = dim3(kRowsWarps * 32), cfg.stream = st;
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr, cfg.numAttrs = p.no_pdl ? 0 : 1;
    return (int)cudaLaunchKernelEx(&cfg, kern, p);
}
template <int FMT>
int launch_rows_kernel(const TkdParams& p, int grid, size_t smem, cudaStream_t st) {
    auto go = [&](auto mt, auto sc) {
        constexpr int MT = decltype(mt)::value, SC = decltype(sc)::value;
        if constexpr (FMT != TKD_BF16 && MT == 2)  // (two tiles of 17 to 32 rows are a block-float weight's: rows_layout)
            if (p.rows_turns)
                return p.topk_k || p.npeers ? launch_rows_one<FMT, MT, SC, false, true>(p, grid, smem, st)
                                            : launch_rows_one<FMT, MT, SC, true, true>(p, grid, smem, st);
        return p.topk_k || p.npeers ? launch_rows_one<FMT, MT, SC, false>(p, grid, smem, st) : launch_rows_one<FMT, MT, SC, true>(p, grid, smem, st);
    };
    const int rows = p.rows_tile ? p.rows_tile : p.M;
    auto chunks = [&](auto mt) {
        if constexpr (FMT != TKD_BF16)
            if (p.rows_chunks == 2) return go(mt, std::integral_constant<int, 2>{});
        return go(mt, std::integral_constant<int, 4>{});
    };
    if constexpr (FMT == TKD_BF16)
        if (rows > 24) return chunks(std::integral_constant<int, 4>{});
    return rows <= 16 ? chunks(std::integral_constant<int, 2>{}) : chunks(std::integral_constant<int, 3>{});
}

}  // namespace
