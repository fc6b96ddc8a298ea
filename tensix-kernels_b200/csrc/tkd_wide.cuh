// tkd_wide.cuh: the matmul of more than 32 activation rows (a prompt's prefill, a large batch) against a packed weight, on
// the fifth-generation tensor cores.
//
// The reference takes such calls as slices of rows, each reading all the weights again (dense_reader/linear.py:179-184). So
// did this library: 512 rows through a [14336, 4096] bfloat8_b weight were 16 launches of the kernel for 32 rows, 387 us,
// each bound by taking the weights apart, which is the same work for 32 rows as for 256. Here a weight is taken apart once
// for up to 256 rows: a tile is 128 weight columns (the MMA's M: a panel of the stream) by NT rows (its N), all of K
// accumulated in tensor memory.
//
//   tkd_wide_x_kernel  lays the activations out as the MMA's B operand first: tiles of NT rows x 64 k, K-major with the
//                      128-byte swizzle, k in the order of the weight fragments, rows past M and k past K zero; each tile
//                      contiguous, so that it comes into shared memory by one bulk copy.
//   tkd_wide_kernel    warp 0 (and 2)  one lane issues the MMAs, A from tensor memory, B from shared memory. Up to 128 rows
//                                      two warps share the units (of 128 k): an MMA of few rows is shorter than its issue.
//                      warp 1          producer of the ring of weight chunks; warp 3: of the x tiles
//                      warps 4-7       output: a thread is a column (a tensor-memory lane); the decode warps help where they cannot go on. Before the decode warps: the
//                                      schedulers favour older warps, and the next tile waits for these to free its accumulators
//                      warps 8-23      decode: tkd_stream_tc_kernel's, without the activations
//
// Work split: tiles are numbered panel-major (the tiles of a panel run at the same time on different SMs and share its
// chunks in L2), each cut into `blocks` blocks of q chunks of K; all blocks are dealt out in equal contiguous runs, one per
// CTA. A tile whose blocks fall to several CTAs goes through scratch, a partial sum per CTA, and the one that delivers last
// adds them up in order of k. How many rows a tile has and how fine it is cut is the host's choice (make_wide).
#pragma once
#include "tkd_stream_tc.cuh"

namespace {

constexpr int kWideWarps = 24, kWideRing = 1, kWideX = 3, kWideDecode0 = 8;
constexpr int kWideWorkers = 5;  // of a tile's output: the output warps and four times four decode warps
constexpr int kWideASlots = 4;                    // units of A in tensor memory, 64 columns each
constexpr int kWideA0 = 256;                      // their first column: the accumulators have 0-255
static_assert(kWideA0 + kWideASlots * 64 <= 512, "tensor memory");

// One CTA lays out 64 rows of one tile: thread (row, piece of 8 k).
__global__ void __launch_bounds__(512) tkd_wide_x_kernel(const uint16_t* __restrict__ x, int64_t ldx, int M, int K, int nt, int nkb,
                                                         uint8_t* __restrict__ xt) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int kb = blockIdx.x, rt = blockIdx.z, r = blockIdx.y * 64 + (threadIdx.x >> 3), c = threadIdx.x & 7;
    if (r >= nt) return;
    const int row = rt * nt + r, k = kb * 64 + 8 * c;
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (row < M && k < K) v = __ldg(reinterpret_cast<const uint4*>(x + (int64_t)row * ldx + k));
    uint8_t* t = xt + ((int64_t)rt * nkb + kb) * nt * 128 + r * 128;
    const int o0 = 64 * (c >> 2) + 8 * (c & 3), o1 = o0 + 32;  // (k 0-3 and k 4-7: see tkd_stream_tc.cuh)
    *reinterpret_cast<uint2*>(t + ((((o0 >> 4) ^ (r & 7)) << 4) | (o0 & 15))) = make_uint2(v.x, v.y);
    *reinterpret_cast<uint2*>(t + ((((o1 >> 4) ^ (r & 7)) << 4) | (o1 & 15))) = make_uint2(v.z, v.w);
}

// D (tensor memory) (+)= A (tensor memory) x B (shared memory), M 128, N from the instruction descriptor
__device__ __forceinline__ void wide_mma(uint32_t d, uint32_t a, uint32_t blo, uint32_t bhi, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "mov.b64 db, {%2, %3};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t}"
        ::"r"(d), "r"(a), "r"(blo), "r"(bhi), "r"(idesc), "r"(accumulate)
        : "memory");
}

// A part of a CTA's run that lies in one tile.
struct WideSeg {
    int tile, c0, c1;  // chunks c0 .. c1 - 1 of the tile
};
__device__ __forceinline__ bool wide_next(const TkdWide& p, int& it, int i1, WideSeg& s) {
    if (it >= i1) return false;
    s.tile = it / p.blocks;
    const int b0 = it - s.tile * p.blocks, b1 = min(p.blocks, b0 + i1 - it);
    s.c0 = b0 * p.q, s.c1 = min(p.chunks, b1 * p.q);
    it += b1 - b0;
    return true;
}
__device__ __forceinline__ int wide_begin(const TkdWide& p, int cta) { return (int)((int64_t)p.total * cta / p.grid); }
// the CTA whose run holds item i
__device__ __forceinline__ int wide_owner(const TkdWide& p, int i) { return (int)((((int64_t)i + 1) * p.grid - 1) / p.total); }

__device__ __forceinline__ void tmem_ld16(uint32_t at, uint32_t (&q)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(q[0]), "=r"(q[1]), "=r"(q[2]), "=r"(q[3]), "=r"(q[4]), "=r"(q[5]), "=r"(q[6]), "=r"(q[7]), "=r"(q[8]), "=r"(q[9]),
                   "=r"(q[10]), "=r"(q[11]), "=r"(q[12]), "=r"(q[13]), "=r"(q[14]), "=r"(q[15])
                 : "r"(at)
                 : "memory");
}
// (the registers named, so that nothing reads them before the wait)
__device__ __forceinline__ void tmem_wait16(uint32_t (&q)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(q[0]), "+r"(q[1]), "+r"(q[2]), "+r"(q[3]), "+r"(q[4]), "+r"(q[5]), "+r"(q[6]), "+r"(q[7]), "+r"(q[8]), "+r"(q[9]),
                   "+r"(q[10]), "+r"(q[11]), "+r"(q[12]), "+r"(q[13]), "+r"(q[14]), "+r"(q[15])
                 :
                 : "memory");
}

// The output of segment j of the CTA's run: a thread is the column et of its tile's panel, rows go in batches of 16. Four warps
// (one to a quarter of the tensor memory's lanes) are a worker, and worker wk of nwk takes every nwk-th batch: the output
// warps alone where a second set of accumulators lets the next tile's MMAs run beside them; with the decode warps as workers
// 1-4 where there is one set, since nothing can run before it is free (256 rows: 9 us with four warps, of 77 for 512 rows of
// [4096, 14336] in which a CTA has two tiles). met: whether the warp's waits so far were (it goes on either way: see mbar_wait).
template <int FMT, int EK, int nwk>
__device__ __forceinline__ void wide_segment(const TkdWide& p, const WideSeg& sg, uint32_t j, bool more, int wk, uint32_t tmem0,
                                             uint8_t* smem, uint32_t accfull0, uint32_t accempty0, volatile int* sflag, uint32_t xs0,
                                             bool& met) {
    constexpr int CK = Fmt<FMT>::SUBSA * Fmt<FMT>::KSA;
    const int lane = threadIdx.x & 31, ow = (threadIdx.x >> 5) & 3, et = ow * 32 + lane;
    const bool leader = wk == 0 && et == 0;
    const int NT = p.nt, nm = p.nmma, r0 = 16 * wk, rstep = 16 * nwk;
    constexpr bool glu = EK == TKD_EPI_GLU2, f32out = EK == TKD_EPI_OUT32, res16 = EK == TKD_EPI_RESIDUAL;
    const bool glu2 = glu && p.epi == TKD_EPI_GLU2, res32 = f32out && p.res;
    float* stage = reinterpret_cast<float*>(smem + p.off_stage) + wk * 1024;  // GLU: [16 rows][64 columns] of the up half
    // GLU: the warps of a panel's gate columns (interleaved: 32 gate, their 32 up, ...; two weights: 64 and 64)
    const bool gate = glu2 ? ow < 2 : (ow & 1) == 0;
    const int gcol = glu2 ? (ow & 1) * 32 + lane : (ow >> 1) * 32 + lane;  // the column within the tile's 64 outputs
    auto bar_workers = [&]() {
        if (nwk > 1)
            asm volatile("bar.sync 3, %0;" ::"n"(kWideWorkers * 128) : "memory");
        else
            bar_output_warps();
    };
    auto bar_worker = [&]() { asm volatile("bar.sync %0, 128;" ::"r"(4 + wk) : "memory"); };
    {
        const int panel = sg.tile / p.nrt, rt = sg.tile - panel * p.nrt;
        const int n = glu2 ? (panel >> 1) * 128 + (panel & 1) * 64 + (et & 63) : panel * 128 + et;  // the column of its weight
        const bool in_w = n < p.n_valid;
        float colf = 1.f, colg = 1.f;  // the column's factor: 2^e of its group in two normal floats, times its scale
        if constexpr (FMT != TKD_BF16) {
            const int e = tkd_out_exp(FMT, (glu2 && et >= 64 ? p.emax2 : p.emax)[n >> 4]), e1 = e / 2, e2 = e - e1;
            colf = __uint_as_float((uint32_t)(e1 + 127) << 23), colg = __uint_as_float((uint32_t)(e2 + 127) << 23);
        }
        if (p.scale_dt != TKD_DT_NONE && in_w) {
            const void* sp = glu2 && et >= 64 ? p.scale2 : p.scale;
            colg *= p.scale_dt == TKD_DT_BF16 ? bf16_bits_to_f32(static_cast<const uint16_t*>(sp)[n]) : static_cast<const float*>(sp)[n];
        }
        // the output column this thread stores, or -1
        int oc = -1;
        if (!glu) {
            if (in_w) oc = p.out_col0 + n;
        } else if (gate) {
            const int o = panel * 64 + gcol;
            if (o < (glu2 ? p.n_valid : p.n_valid / 2)) oc = p.out_col0 + o;
        }
        const int row0 = rt * NT, rows = min(NT, p.M - row0);
        const bool whole = sg.c0 == 0 && sg.c1 == p.chunks;
        const int kv = min(p.K, sg.c1 * CK) - sg.c0 * CK;
        const bool two = nm == 2 && kv > 128;
        const uint32_t set = j % p.nset;
        if (!mbar_wait_parked(accfull0 + 8 * set, (j / p.nset) & 1, p.status, met)) met = false;
        tc_fence_after();
        const uint32_t ta = tmem0 + ((uint32_t)(ow * 32) << 16) + set * nm * NT;
        // sixteen rows of the segment's sums
        auto sums = [&](int r, float (&v)[16]) {
            uint32_t a[16], b[16];
            tmem_ld16(ta + r, a);
            if (two) tmem_ld16(ta + NT + r, b);
            tmem_wait16(a);
            if (two) {
                tmem_wait16(b);
#pragma unroll
                for (int m = 0; m < 16; ++m) v[m] = __uint_as_float(a[m]) + __uint_as_float(b[m]);
            } else {
#pragma unroll
                for (int m = 0; m < 16; ++m) v[m] = __uint_as_float(a[m]);
            }
        };
        auto release = [&]() {
            tc_fence_before();
            if (nwk > 1)
                bar_workers();
            else
                __syncwarp();
            if (wk == 0 && lane == 0) mbar_arrive(accempty0 + 8 * set);
        };
        // ---- a cut tile: partial sums in scratch, [segment][row / 4][column][4]. The later of two CTAs adds the other's to its
        // own, still in tensor memory, without storing that; of more than two each stores its own, and the last adds them all.
        const int64_t part = (int64_t)NT * 128;
        const int b0 = whole ? 0 : wide_owner(p, sg.tile * p.blocks);
        const int nseg = whole ? 1 : wide_owner(p, sg.tile * p.blocks + p.blocks - 1) - b0 + 1, own = (int)blockIdx.x - b0;
        // where segment s of the tile leaves its sums
        auto part_of = [&](int s) {
            return p.scratch + ((int64_t)(b0 + s) * 2 + (wide_begin(p, b0 + s) < sg.tile * p.blocks ? 1 : 0)) * part + et * 4;
        };
        bool staged = false;  // the other parts are copied into the (then idle) x tiles first, `per` rows at a time
        int per = 0;
        if (!whole) {
            bool last = false;
            if (nseg == 2) {
                if (leader) sflag[0] = atom_add_acq_rel(p.counters + sg.tile, 0) == 1;
                bar_workers();
                last = sflag[0] != 0;
                bar_workers();  // (sflag may be written again only after everyone has read it)
            }
            if (!last) {
                float* dst = part_of(own);
#pragma unroll 1
                for (int r = r0; r < rows; r += rstep) {
                    float v[16];
                    sums(r, v);
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        __stcg(reinterpret_cast<float4*>(dst + r * 128 + q * 512), make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]));
                }
                bar_workers();  // (orders all threads' stores before thread 0's release)
                if (leader) sflag[0] = atom_add_acq_rel(p.counters + sg.tile, 1) == nseg - 1;
                bar_workers();
                last = sflag[0] != 0;
                bar_workers();
            }
            if (!last) {
                release();
                return;
            }
            if (leader) p.counters[sg.tile] = 0;
            per = p.nx * NT * 128 / ((nseg == 2 ? 1 : nseg) * 512) & ~15;
            staged = !more && (nwk > 1 ? nseg == 2 && per >= NT : per >= 16);  // (this CTA's last tile: every x tile has been multiplied)
        }
        // ---- the output stage, sixteen rows at a time (a warp has its scheduler nearly to itself here: the loop is bound by the
        // latency of its chains, so the rows go side by side; eight at a time a tile of 256 rows took twice as long)
        const bool odd = lane & 1;
        const bool pairs = !f32out && !((reinterpret_cast<uintptr_t>(p.out) & 3) | (p.ldo & 1) | (p.out_col0 & 1)) &&
                           !(res16 && ((reinterpret_cast<uintptr_t>(p.res) & 3) | (p.ldr & 1)));
        const bool fast = __all_sync(0xFFFFFFFFu, pairs && oc >= 0);  // (two columns a store)
        const uint32_t pick = odd ? 0x3276u : 0x5410u;  // (own word first: an even lane both lower halves, an odd one both upper)
        // fast, with a residual: the pairs of columns of every other row of a batch, asked for a batch ahead
        uint32_t rq[8];
        auto load_res = [&](int r) {
            const uint16_t* rp = static_cast<const uint16_t*>(p.res) + (int64_t)(row0 + r + odd) * p.ldr + oc - odd;
#pragma unroll
            for (int m = 0; m < 8; ++m) {
                // (a row past the last reads the last of its kind again)
                rq[m] = *reinterpret_cast<const uint32_t*>(rp);
                if (r + 2 * m + 2 + odd < rows) rp += 2 * p.ldr;
            }
        };
        if (fast && res16 && r0 + odd < rows) load_res(r0);
        uint16_t* y16 = static_cast<uint16_t*>(p.out) + (int64_t)row0 * p.ldo + oc;
        int staged_from = 0, staged_to = 0;  // the rows whose other parts lie in the x tiles
        if (staged && nwk > 1) {
            // (one other part, and room for all of it: each thread copies its own batches')
            const float* src = part_of(1 - own);
            for (int r = r0; r < rows; r += rstep)
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(xs0 + ((r / 4 + q) * 128 + et) * 16), "l"(src + r * 128 + q * 512)
                                 : "memory");
            asm volatile("cp.async.wait_all;" ::: "memory");
            staged_to = NT;
        }
#pragma unroll 1
        for (int r = r0; r < rows; r += rstep) {
            float v[16];
            if (staged && r >= staged_to) {
                staged_from = r, staged_to = r + per;
                const int n4 = min(per, NT - r) / 4;
                for (int s = nseg == 2 ? 1 - own : 0, i = 0; s < nseg && (nseg > 2 || i == 0); ++s, ++i) {
                    const float* src = part_of(s) + r * 128;
                    const uint32_t dst = xs0 + (i * (per / 4) * 128 + et) * 16;
#pragma unroll 8
                    for (int q = 0; q < n4; ++q)
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + q * 2048), "l"(src + q * 512) : "memory");
                }
                asm volatile("cp.async.wait_all;" ::: "memory");
            }
            // + sixteen rows of the i-th part that is added here, segment s's
            auto add = [&](int s, int i) {
                float4 f[4];
                if (staged) {
                    const uint32_t at = xs0 + ((i * (per / 4) + (r - staged_from) / 4) * 128 + et) * 16;
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const uint4 w = lds128(at + 2048 * q);
                        f[q] = make_float4(__uint_as_float(w.x), __uint_as_float(w.y), __uint_as_float(w.z), __uint_as_float(w.w));
                    }
                } else {
                    const float4* src = reinterpret_cast<const float4*>(part_of(s) + r * 128);
#pragma unroll
                    for (int q = 0; q < 4; ++q) f[q] = __ldcg(src + 128 * q);
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) v[4 * q] += f[q].x, v[4 * q + 1] += f[q].y, v[4 * q + 2] += f[q].z, v[4 * q + 3] += f[q].w;
            };
            if (nseg <= 2) {
                sums(r, v);
                if (nseg == 2) add(1 - own, 0);  // (which of two terms comes first does not matter)
            } else {
#pragma unroll
                for (int m = 0; m < 16; ++m) v[m] = 0.f;
#pragma unroll 1
                for (int s = 0; s < nseg; ++s) add(s, s);  // in order of k
            }
#pragma unroll
            for (int m = 0; m < 16; ++m) v[m] = v[m] * colf * colg;
            if (EK == TKD_EPI_SILU) {
#pragma unroll
                for (int m = 0; m < 16; ++m) v[m] = act_gate(v[m], 0);
            }
            if (glu) {
                bar_worker();  // (the batch before has been read)
                if (!gate)
#pragma unroll
                    for (int m = 0; m < 16; ++m) stage[m * 64 + gcol] = v[m];
                bar_worker();
                if (!gate) continue;
#pragma unroll
                for (int m = 0; m < 16; ++m) v[m] = act_gate(v[m], p.act) * stage[m * 64 + gcol];
            }
            if (fast) {
                // an even lane stores both columns of the even rows, its neighbour those of the odd ones
                uint16_t* yp = y16 + (int64_t)(r + odd) * p.ldo - odd;
                const int left = rows - r - odd;  // (rows from this lane's first on)
                uint32_t w[8];
                if (!res16) {
#pragma unroll
                    for (int m = 0; m < 8; ++m) {
                        const uint32_t mine = f32x2_to_bf16x2(v[2 * m], v[2 * m + 1]);
                        w[m] = __byte_perm(mine, __shfl_xor_sync(0xFFFFFFFFu, mine, 1), pick);
                    }
                } else {
#pragma unroll
                    for (int m = 0; m < 8; ++m) {
                        const float got = __shfl_xor_sync(0xFFFFFFFFu, odd ? v[2 * m] : v[2 * m + 1], 1);
                        const float lo = odd ? got : v[2 * m], hi = odd ? v[2 * m + 1] : got;
                        w[m] = f32x2_to_bf16x2(lo + __uint_as_float(rq[m] << 16), hi + __uint_as_float(rq[m] & 0xFFFF0000u));
                    }
                    if (r + rstep + odd < rows) load_res(r + rstep);
                }
#pragma unroll
                for (int m = 0; m < 8; ++m, yp += 2 * p.ldo) st_if(2 * m < left, yp, w[m]);
            } else if (f32out && !res32) {
                float* yp = static_cast<float*>(p.out) + (int64_t)(row0 + r) * p.ldo + oc;
                const int left = oc >= 0 ? rows - r : 0;
#pragma unroll
                for (int m = 0; m < 16; ++m, yp += p.ldo) st_if(m < left, yp, __float_as_uint(v[m]));
            } else if (oc >= 0) {
                int64_t at = (int64_t)(row0 + r) * p.ldo + oc, ra = (int64_t)(row0 + r) * p.ldr + oc;
                const int esz = f32out ? 4 : 2, rsz = res32 ? 4 : 2;
                char *yp = static_cast<char*>(p.out) + at * esz;
                const char* rp = static_cast<const char*>(p.res) + ra * rsz;
                uint32_t q[16];
                if (res32 || res16) {
#pragma unroll
                    for (int m = 0; m < 16; ++m) {
                        q[m] = res32 ? *reinterpret_cast<const uint32_t*>(rp) : (uint32_t)*reinterpret_cast<const uint16_t*>(rp) << 16;
                        if (r + m + 1 < rows) rp += p.ldr * rsz;
                    }
#pragma unroll
                    for (int m = 0; m < 16; ++m) v[m] += __uint_as_float(q[m]);
                }
#pragma unroll
                for (int m = 0; m < 16; ++m, yp += p.ldo * esz) {
                    if (f32out)
                        st_if(r + m < rows, yp, __float_as_uint(v[m]));
                    else
                        st16_if(r + m < rows, yp, f32_to_bf16_bits(v[m]));
                }
            }
        }
        release();
    }
}

// EK: the kind of output (TKD_EPI_GLU2 for both GLU forms). One kernel for all of them was 3 us slower at any size: every launch
// fetches its code anew, and most of it was outputs that the call does not have. SHARED: the decode warps share the output.
template <int FMT, bool KWHOLE, int EK, bool SHARED>
__global__ void __launch_bounds__(kWideWarps * 32, 1) tkd_wide_kernel(const __grid_constant__ TkdWide p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    using F = Fmt<FMT>;
    constexpr int CK = F::SUBSA * F::KSA, SW = 16, G = kTcGroups;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem);
    const uint32_t full0 = smem_u32(bars), empty0 = full0 + 8 * TKD_MAX_STAGES;
    const uint32_t xfull0 = empty0 + 8 * TKD_MAX_STAGES, xempty0 = xfull0 + 8 * TKD_WIDE_XT;
    const uint32_t afull0 = xempty0 + 8 * TKD_WIDE_XT, aempty0 = afull0 + 8 * kWideASlots;
    const uint32_t accfull0 = aempty0 + 8 * kWideASlots, accempty0 = accfull0 + 16;
    static_assert(8 * (2 * TKD_MAX_STAGES + 2 * TKD_WIDE_XT + 2 * kWideASlots + 4) <= TKD_SMEM_HEAD - 32, "barriers");
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + TKD_SMEM_HEAD - 32);
    volatile int* sflag = reinterpret_cast<volatile int*>(smem + TKD_SMEM_HEAD - 16);
    const uint32_t xs0 = (smem_u32(smem + p.off_x) + 1023u) & ~1023u;  // (the swizzle is a function of the address)
    const uint32_t ring0 = smem_u32(smem + p.off_ring);

    // (the warp's number by a shuffle: what follows from it is then known to be the same in all lanes, as the operands of an MMA have
    // to be; else each is taken from a lane before it is issued. 512 rows of [14336, 4096] bfloat8_b, launches in a graph: 67.2 to 58.7 us)
    const int tid = threadIdx.x, warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0), lane = tid & 31;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (tid == 0) {
        for (int s = 0; s < p.nstages; ++s) mbar_init(full0 + 8 * s, 1), mbar_init(empty0 + 8 * s, SW);
        for (int s = 0; s < p.nx; ++s) mbar_init(xfull0 + 8 * s, 1), mbar_init(xempty0 + 8 * s, 1);
        for (int s = 0; s < kWideASlots; ++s) mbar_init(afull0 + 8 * s, SW / G), mbar_init(aempty0 + 8 * s, 1);
        for (int s = 0; s < 2; ++s) mbar_init(accfull0 + 8 * s, p.nmma), mbar_init(accempty0 + 8 * s, 4);
        sflag[0] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem0 = *tmem_slot;
    const int i0 = wide_begin(p, blockIdx.x), i1 = wide_begin(p, blockIdx.x + 1);
    const int K = p.K, nst = p.nstages, NT = p.nt, nx = p.nx;
    const bool glu2 = p.epi == TKD_EPI_GLU2;
    const int nsa_total = (K + F::KSA - 1) / F::KSA;
    WideSeg sg;

    if (warp == kWideRing) {
        // ---------------------------------------------------------------- producer of the weight chunks
        uint32_t st = 0;
        bool ok = true;
        for (int it = i0; ok && wide_next(p, it, i1, sg);) {
            const int panel = sg.tile / p.nrt;
            const uint8_t* src = p.w + (int64_t)(glu2 ? panel >> 1 : panel) * p.panel_bytes;
            const uint8_t* src2 = glu2 ? p.w2 + (int64_t)(panel >> 1) * p.panel_bytes : nullptr;
            for (int c = sg.c0; c < sg.c1; ++c, ++st) {
                const uint32_t s = st % nst;
                ok = mbar_wait_parked(empty0 + 8 * s, ((st / nst) & 1) ^ 1, p.status);
                if (!ok) break;
                const uint32_t gbytes = (uint32_t)min(F::SUBSA, nsa_total - c * F::SUBSA) * F::SAB;  // one group's share
                const int64_t coff = (int64_t)c * (F::SUBSA * F::SAB * 8);
                const uint32_t dst = ring0 + s * p.stage_bytes;
                if (lane == 0) {
                    mbar_expect_tx(full0 + 8 * s, 8 * gbytes);
                    if (glu2) {
                        const int64_t hoff = coff + (int64_t)(panel & 1) * 4 * gbytes;
                        bulk_g2s(dst, src + hoff, 4 * gbytes, full0 + 8 * s);
                        bulk_g2s(dst + 4 * gbytes, src2 + hoff, 4 * gbytes, full0 + 8 * s);
                    } else {
                        bulk_g2s(dst, src + coff, 8 * gbytes, full0 + 8 * s);
                    }
                }
                __syncwarp();
            }
        }
        if (!ok)  // (the copies in flight land before the CTA goes)
            for (uint32_t back = 1; back <= (uint32_t)nst && back <= st; ++back)
                for (uint32_t i = 0; i < 64; ++i)
                    if (mbar_try_wait(full0 + 8 * ((st - back) % nst), ((st - back) / nst) & 1)) break;
    } else if (warp == kWideX) {
        // ---------------------------------------------------------------- producer of the x tiles, two a unit
        asm volatile("griddepcontrol.wait;" ::: "memory");
        const uint32_t bytes = (uint32_t)NT * 128;
        uint32_t st = 0, s = 0, phase = 1;
        bool ok = true;
        for (int it = i0; ok && wide_next(p, it, i1, sg);) {
            const uint8_t* src = p.xt + (int64_t)(sg.tile % p.nrt) * p.nkb * bytes;
            const int kb1 = 2 * ((min(K, sg.c1 * CK) + 127) / 128);
            for (int kb = sg.c0 * (CK / 64); kb < kb1; ++kb, ++st) {
                ok = mbar_wait(xempty0 + 8 * s, phase, p.status);
                if (!ok) break;
                if (lane == 0) {
                    mbar_expect_tx(xfull0 + 8 * s, bytes);
                    bulk_g2s(xs0 + s * bytes, src + (int64_t)kb * bytes, bytes, xfull0 + 8 * s);
                }
                __syncwarp();
                if (++s == (uint32_t)nx) s = 0, phase ^= 1;
            }
        }
        if (!ok)
            for (uint32_t back = 1; back <= (uint32_t)nx && back <= st; ++back)
                for (uint32_t i = 0; i < 64; ++i)
                    if (mbar_try_wait(xfull0 + 8 * ((st - back) % nx), ((st - back) / nx) & 1)) break;
    } else if (warp == 0 || warp == 2) {
        // ---------------------------------------------------------------- MMA issue. A unit belongs to the warp of its number's
        // parity in the CTA's sequence (so a slot's barriers are one warp's and it sees every phase of them), an accumulator
        // to the parity within the segment. The loop is on every unit's way from decoded to multiplied, a warp alone: slots and their
        // parities are counted, not divided out of the unit's number (the x tiles' number is no constant), and a whole unit's MMAs
        // stand without a test between them. With divisions a unit took the warp 1540 cycles at 256 rows, where its eight MMAs run
        // 1050: 384 rows of [14336, 4096] bfloat8_b 63.4 us, 45.4 so (with the shuffle above).
        const int mw = warp >> 1, nm = p.nmma;
        if (mw < nm) {
            const uint64_t bd0 = tc_desc(xs0);
            const uint32_t dhi = (uint32_t)(bd0 >> 32), blo0 = (uint32_t)bd0, xstep = (uint32_t)NT * 128 >> 4;
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (((uint32_t)NT >> 3) << 17) | ((128u >> 4) << 24);
            uint32_t us = 0, j = 0;
            uint32_t ps = mw, aphase = 0, xs = 2 * mw, xphase = 0;  // this warp's next slots and their parities
            bool ok = true;
            for (int it = i0; ok && wide_next(p, it, i1, sg); ++j) {
                const int kv = min(K, sg.c1 * CK) - sg.c0 * CK, nu = (kv + 127) >> 7;
                const uint32_t set = p.nset == 2 ? j & 1 : 0;
                ok = mbar_wait(accempty0 + 8 * set, ((p.nset == 2 ? j >> 1 : j) & 1) ^ 1, p.status);
                if (!ok) break;
                tc_fence_after();
                for (int ui = nm == 2 ? (int)((mw - us) & 1u) : 0; ui < nu; ui += nm) {
                    ok = mbar_wait(afull0 + 8 * ps, aphase, p.status);
                    if (!ok) break;
                    const int kleft = kv - 128 * ui;
                    const uint32_t d = tmem0 + (set * nm + (ui & (nm - 1))) * NT, acc = ui >= nm;
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        ok = ok && mbar_wait(xfull0 + 8 * (xs + h), xphase, p.status);
                        if (!ok) break;
                        tc_fence_after();
                        if (tc_elect()) {
                            const uint32_t al = tmem0 + kWideA0 + ps * 64 + h * 32, bl = blo0 + (xs + h) * xstep;
                            auto issue = [&](int nb) {
#pragma unroll
                                for (int b = 0; b < 4; ++b)
                                    if (b < nb) wide_mma(d, al + 8 * b, bl + 2 * b, dhi, idesc, h || b ? 1u : acc);
                            };
                            if (kleft >= 128)
                                issue(4);
                            else
                                issue((kleft >> 4) - 4 * h);
                            tc_commit(xempty0 + 8 * (xs + h));
                            if (h == 1) tc_commit(aempty0 + 8 * ps);
                        }
                        __syncwarp();
                    }
                    if (!ok) break;
                    if ((ps += nm) >= kWideASlots) ps -= kWideASlots, aphase ^= 1;
                    if ((xs += 2 * nm) >= (uint32_t)nx) xs -= nx, xphase ^= 1;
                }
                us += nu;
                if (ok && tc_elect()) tc_commit(accfull0 + 8 * set);
                __syncwarp();
            }
        }
    } else {
        // ---------------------------------------------------------------- output warps (4-7), and decode warps, as tkd_stream_tc_kernel's: two groups of
        // eight, a unit of two tiles of 64 k is one group's; a warp stores its 16 columns' share into tensor memory
        const bool decode = warp >= kWideDecode0;
        const int cw = warp - kWideDecode0, qtr = warp & 3, sub4 = cw >> 2, grp = sub4 >> 1, rg = 2 * qtr + (sub4 & 1), t = lane & 3;
        constexpr int EXPB = FMT == TKD_BFP4 ? 64 : (FMT == TKD_BFP8 ? 32 : 0), UPC = CK / 128, MU = (UPC + G - 1) / G;
        const uint2 sh = make_uint2(p.mul16, p.mul128);
        const uint32_t alane = tmem0 + ((uint32_t)(16 * rg) << 16) + kWideA0;
        uint32_t slot = 0, phase = 0, useq = 0;
        auto st_a = [&](uint32_t taddr, const uint32_t* r) {
            asm volatile("tcgen05.st.sync.aligned.16x256b.x2.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]),
                         "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                         : "memory");
        };
        // 32 k (bfloat4_b: 64 k) of the warp's columns from shared memory at `sab` to tensor-memory columns tb on
        auto decode_sa = [&](uint32_t sab, uint32_t tb) {
            if constexpr (FMT == TKD_BF16) {
                const uint4 a = lds128(sab + lane * 16), b = lds128(sab + 512 + lane * 16);
                const uint32_t r[8] = {a.x, a.z, a.y, a.w, b.x, b.z, b.y, b.w};
                st_a(tb, r);
            } else {
                uint32_t cw_[4], ew_[4];
                const uint4 cv = lds128(sab + EXPB + lane * 16);
                cw_[0] = cv.x, cw_[1] = cv.y, cw_[2] = cv.z, cw_[3] = cv.w;
                if constexpr (FMT == TKD_BFP8) {
                    const uint2 ev = lds64(sab + t * 8);
                    ew_[0] = ev.x, ew_[1] = ev.y, ew_[2] = ew_[3] = 0;
                } else {
                    const uint4 ev = lds128(sab + t * 16);
                    ew_[0] = ev.x, ew_[1] = ev.y, ew_[2] = ev.z, ew_[3] = ev.w;
                }
#pragma unroll
                for (int q = 0; q < F::XB; ++q) {
                    uint32_t r[8];
#pragma unroll
                    for (int jj = 0; jj < 2; ++jj) {
                        uint32_t a0, a1, a2, a3, s0, s1;
                        if constexpr (FMT == TKD_BFP4) {
                            const uint32_t w = cw_[2 * q + jj], tt = __funnelshift_r(w, w, 8), ew = ew_[2 * q + jj];
                            a0 = w & TKD_MASK_BFP4, a1 = shl_fma<4>(w, sh.x) & TKD_MASK_BFP4;
                            a2 = tt & TKD_MASK_BFP4, a3 = shl_fma<4>(tt, sh.x) & TKD_MASK_BFP4;
                            s0 = and_or(ew, TKD_EMASK_BFP4, ebase(sh)), s1 = and_or(shl_fma<7>(ew, sh.y), TKD_EMASK_BFP4, ebase(sh));
                        } else {
                            const uint32_t w0 = cw_[2 * jj], w1 = cw_[2 * jj + 1], ew = ew_[jj];
                            a0 = w0 & TKD_MASK_BFP8, a1 = rot_and<8>(w0, TKD_MASK_BFP8);
                            a2 = w1 & TKD_MASK_BFP8, a3 = rot_and<8>(w1, TKD_MASK_BFP8);
                            s0 = ew & 0x7F807F80u, s1 = rot_and<8>(ew, 0x7F807F80u);
                        }
                        r[4 * jj] = mul_bf16x2(a0, s0), r[4 * jj + 1] = mul_bf16x2(a2, s1);
                        r[4 * jj + 2] = mul_bf16x2(a1, s0), r[4 * jj + 3] = mul_bf16x2(a3, s1);
                    }
                    st_a(tb + 16 * q, r);
                }
            }
        };
        bool met = true;
        uint32_t j = 0;
        for (int it = i0; wide_next(p, it, i1, sg);) {
            bool ok = true;
            for (int c = decode && met ? sg.c0 : sg.c1; ok && c < sg.c1; ++c) {
                ok = mbar_wait(full0 + 8 * slot, phase, p.status);
                if (!ok) break;
                const int nsa = KWHOLE ? F::SUBSA : min(F::SUBSA, nsa_total - c * F::SUBSA);
                const int ntiles = (nsa * F::KSA + 63) / 64, nunits = (ntiles + 1) >> 1;
                const int u0 = (int)((uint32_t)grp - useq) & (G - 1);
                const uint32_t gb = ring0 + slot * p.stage_bytes + rg * nsa * F::SAB;
#pragma unroll
                for (int i = 0; i < MU; ++i) {
                    const int u = u0 + G * i;
                    if (u >= nunits) break;
                    const uint32_t us = useq + u, ps = us % kWideASlots;
                    ok = mbar_wait(aempty0 + 8 * ps, ((us / kWideASlots) & 1) ^ 1, p.status);
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t ta = alane + ps * 64;
#pragma unroll
                    for (int sub = 0; sub < 2; ++sub) {
                        const int ti = 2 * u + sub;
                        if (ti >= ntiles) break;
                        if constexpr (FMT == TKD_BFP4) {
                            decode_sa(gb + ti * F::SAB, ta + sub * 32);
                        } else {
                            decode_sa(gb + 2 * ti * F::SAB, ta + sub * 32);
                            if (2 * ti + 1 < nsa) decode_sa(gb + (2 * ti + 1) * F::SAB, ta + sub * 32 + 16);
                        }
                    }
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(afull0 + 8 * ps);
                }
                useq += nunits;
                __syncwarp();
                if (ok && lane == 0) mbar_arrive(empty0 + 8 * slot);
                if (++slot == (uint32_t)nst) slot = 0, phase ^= 1;
            }
            met = met && ok;
            // (the output and the residual may be the kernel before's: waited for once)
            if (j == 0 && (SHARED || !decode)) asm volatile("griddepcontrol.wait;" ::: "memory");
            if (SHARED || !decode)
                wide_segment<FMT, EK, SHARED ? kWideWorkers : 1>(p, sg, j, it < i1, SHARED ? 1 + sub4 : 0, tmem0, smem, accfull0, accempty0, sflag,
                                                                 xs0, met);
            ++j;
        }
    }
    // ---- the end: everyone comes here, also after a wait that gave up
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem0), "r"(512u) : "memory");
    }
}

template <int FMT, bool KWHOLE, int EK, bool SHARED>
int launch_wide(const TkdWide& p, size_t smem, cudaStream_t st) {
    auto kern = tkd_wide_kernel<FMT, KWHOLE, EK, SHARED>;
    static bool allowed[64] = {false};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    if (dev < 0 || dev >= 64 || !allowed[dev]) {
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        if (e != cudaSuccess) return (int)e;
        if (dev >= 0 && dev < 64) allowed[dev] = true;
    }
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.stream = st, cfg.attrs = attr, cfg.numAttrs = p.no_pdl ? 0 : 1;
    cfg.gridDim = dim3((unsigned)p.nkb, (unsigned)((p.nt + 63) / 64), (unsigned)p.nrt), cfg.blockDim = dim3(512);
    e = cudaLaunchKernelEx(&cfg, tkd_wide_x_kernel, p.x, p.ldx, p.M, p.K, p.nt, p.nkb, p.xt);
    if (e != cudaSuccess) return (int)e;
    cfg.gridDim = dim3((unsigned)p.grid), cfg.blockDim = dim3(kWideWarps * 32), cfg.dynamicSmemBytes = smem;
    return (int)cudaLaunchKernelEx(&cfg, kern, p);
}
template <int FMT, int EK>
int launch_wide_k(const TkdWide& p, size_t smem, cudaStream_t st) {
    const bool whole = p.K % (Fmt<FMT>::SUBSA * Fmt<FMT>::KSA) == 0;
    if (p.nset == 1) return whole ? launch_wide<FMT, true, EK, true>(p, smem, st) : launch_wide<FMT, false, EK, true>(p, smem, st);
    return whole ? launch_wide<FMT, true, EK, false>(p, smem, st) : launch_wide<FMT, false, EK, false>(p, smem, st);
}
template <int FMT>
int launch_wide_fmt(const TkdWide& p, size_t smem, cudaStream_t st) {
    return for_epilogue(p.epi, [&](auto ek) { return launch_wide_k<FMT, decltype(ek)::value>(p, smem, st); });
}

}  // namespace
