// tkd_topk.cu: the best `top` candidates of every row out of a set of top-k records (include/tkd.h: tkd_topk_merge).
//
// One CTA per row. A candidate is (key, index); the order is key descending, index ascending among equal keys, which
// is total (indices are distinct), so every GPU merging the same records gets the same answer. Packed as
// key << 32 | ~index the order is that of 64-bit integers. The candidates (records * k of them, 600 for the
// 151936-column LM head) are held by the threads in a strided fashion; `top` rounds each pick the largest candidate
// below the one picked before: a maximum over the thread's own, a warp shuffle reduction, one exchange through shared
// memory.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "tkd_internal.h"

namespace {

constexpr int kThreads = 256;
constexpr int kOwn = 4;  // candidates a thread keeps in registers; more are re-read from memory every round

__global__ void __launch_bounds__(kThreads) tkd_topk_merge_kernel(const uint32_t* __restrict__ records, int nrec, int rows,
                                                                  int k, int top, uint32_t* __restrict__ out) {
    __shared__ unsigned long long red[kThreads / 32];
    // (launched as a programmatic dependent of the kernel before it, normally the stream kernel that writes the
    // records: let the kernel after this one start its CTAs, then wait for the records to be complete)
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int r = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n = nrec * k;
    auto cand = [&](int c) -> unsigned long long {
        const int rec = c / k, q = c - rec * k;
        const uint32_t* page = records + (size_t)rec * 2 * rows * k;
        const uint32_t key = __ldg(page + r * k + q), idx = __ldg(page + (rows + r) * k + q);
        return key ? ((unsigned long long)key << 32) | (uint32_t)~idx : 0ull;  // (0: an empty slot)
    };
    unsigned long long own[kOwn];
#pragma unroll
    for (int j = 0; j < kOwn; ++j) own[j] = tid + j * kThreads < n ? cand(tid + j * kThreads) : 0ull;
    unsigned long long bound = ~0ull;
    for (int t = 0; t < top; ++t) {
        unsigned long long best = 0;
#pragma unroll
        for (int j = 0; j < kOwn; ++j)
            if (own[j] < bound && own[j] > best) best = own[j];
        for (int c = tid + kOwn * kThreads; c < n; c += kThreads) {
            const unsigned long long v = cand(c);
            if (v < bound && v > best) best = v;
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            const unsigned long long other = __shfl_xor_sync(0xFFFFFFFFu, best, o);
            best = other > best ? other : best;
        }
        if (lane == 0) red[warp] = best;
        __syncthreads();
        best = red[0];
#pragma unroll
        for (int w = 1; w < kThreads / 32; ++w) best = red[w] > best ? red[w] : best;
        __syncthreads();
        if (tid == 0) {
            out[r * top + t] = (uint32_t)(best >> 32);
            out[(rows + r) * top + t] = best ? ~(uint32_t)best : 0xFFFFFFFFu;
        }
        bound = best;  // (0: nothing left; the remaining slots come out empty)
    }
}

// The same for up to kWarpMax candidates a row (the LM head's 600): one warp, the candidates in registers (32 a lane,
// fetched with all their loads in flight), and per round two warp-wide reductions in hardware (redux.sync) instead of
// ten shuffles: the largest key, then among the lanes holding it the largest ~index.
constexpr int kWarpMax = 1024;
__global__ void __launch_bounds__(32) tkd_topk_merge_warp_kernel(const uint32_t* __restrict__ records, int nrec, int rows,
                                                                 int k, int top, uint32_t* __restrict__ out) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int r = blockIdx.x, lane = threadIdx.x;
    const int n = nrec * k;
    unsigned long long own[kWarpMax / 32];
#pragma unroll
    for (int j = 0; j < kWarpMax / 32; ++j) {
        const int c = lane + 32 * j;
        own[j] = 0ull;
        if (c < n) {
            const int rec = c / k, q = c - rec * k;
            const uint32_t* page = records + (size_t)rec * 2 * rows * k;
            const uint32_t key = __ldg(page + r * k + q), idx = __ldg(page + (rows + r) * k + q);
            own[j] = key ? ((unsigned long long)key << 32) | (uint32_t)~idx : 0ull;
        }
    }
    unsigned long long bound = ~0ull;
    for (int t = 0; t < top; ++t) {
        unsigned long long mine = 0;
#pragma unroll
        for (int j = 0; j < kWarpMax / 32; ++j)
            if (own[j] < bound && own[j] > mine) mine = own[j];
        const uint32_t key = __reduce_max_sync(0xFFFFFFFFu, (uint32_t)(mine >> 32));
        const uint32_t low = __reduce_max_sync(0xFFFFFFFFu, key && (uint32_t)(mine >> 32) == key ? (uint32_t)mine : 0u);
        const unsigned long long best = key ? ((unsigned long long)key << 32) | low : 0ull;
        if (lane == 0) {
            out[r * top + t] = key;
            out[(rows + r) * top + t] = best ? ~low : 0xFFFFFFFFu;
        }
        bound = best;  // (0: nothing left; the remaining slots come out empty)
    }
}

}  // namespace

int tkd_launch_topk_merge(const uint32_t* records, int nrec, int rows, int k, int top, uint32_t* out, cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)rows);
    cfg.blockDim = dim3(kThreads);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (nrec * k <= kWarpMax) {
        cfg.blockDim = dim3(32);
        return (int)cudaLaunchKernelEx(&cfg, tkd_topk_merge_warp_kernel, records, nrec, rows, k, top, out);
    }
    return (int)cudaLaunchKernelEx(&cfg, tkd_topk_merge_kernel, records, nrec, rows, k, top, out);
}

// ---- the LM head's rescore and pick (include/tkd.h: tkd_head_pick, tkd_head_pick_records) --------------------------
namespace {

// a float's bits as an unsigned key in the float order: NaN above everything, -0 equal to +0 (torch's compare)
__device__ __forceinline__ uint32_t order32(uint32_t b) {
    if ((b & 0x7FFFFFFFu) == 0) b = 0;
    if ((b & 0x7F800000u) == 0x7F800000u && (b & 0x007FFFFFu)) return 0xFFFFFFFFu;
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
// a record key's rank for the records-only pick: a NaN of either sign above every key, -0 equal to +0 (key != 0)
__device__ __forceinline__ uint32_t rank16(uint32_t kk) {
    const uint32_t mag = (kk >= 0x8000u ? kk : ~kk) & 0x7FFFu;
    if ((mag & 0x7F80u) == 0x7F80u && (mag & 0x007Fu)) return 0x10000u;
    return kk == 0x7FFFu ? 0x8000u : kk;
}

constexpr int kPickWarps = 16, kPickOwn = 8, kPickCluster = 4;

// The best `top` (at most 32) of a warp's candidates, lane t the t-th: (rank, id), rank 0 where there are none. A candidate's
// word is rank << 12 | 4095 - its place, so that an equal rank keeps the earlier place; a round is one warp-wide maximum in
// hardware, and the lane that gave it moves on to its next.
template <int N>
__device__ __forceinline__ void pick_rounds(const uint32_t (&word)[N], const uint32_t (&id)[N], int top, int lane, uint32_t& rank_out,
                                            uint32_t& id_out) {
    uint32_t best = 0, bid = 0;
    auto next = [&](uint32_t bound) {
        best = 0;
#pragma unroll
        for (int j = 0; j < N; ++j)
            if (word[j] < bound && word[j] > best) best = word[j], bid = id[j];
    };
    next(0xFFFFFFFFu);
    rank_out = 0, id_out = 0;
    for (int t = 0; t < top; ++t) {
        const uint32_t m = __reduce_max_sync(0xFFFFFFFFu, best);
        if (m >> 12 == 0) break;
        const uint32_t src = __ballot_sync(0xFFFFFFFFu, best == m);
        const uint32_t won = __shfl_sync(0xFFFFFFFFu, bid, __ffs(src) - 1);
        if (lane == t) rank_out = m >> 12, id_out = won;
        if (best == m) next(m);
    }
}

// The same by counting, for up to kPickSlots slots of up to kPickRecs records: a slot's place among the best is the number of
// slots before it, and only the `top` records whose best slots are the best of all can hold one of the best. Four threads a record,
// then a slot, no chain of rounds: as `top` rounds of maxima in every warp and again over the warps' lists the pick of 16
// from 19 records of 8 took 11.7 us of a launch (2 rows, 37888 columns), 8.2 now; the rest is the rescore, rows of the head at
// random places in its memory. (Where: launch_pick.) word: rank << 32 | ~place (0: empty), id: the slots' in shared memory.
constexpr int kPickSlots = 2048, kPickRecs = 512;
struct PickCount {
    unsigned long long word[kPickSlots], most[kPickRecs];
    uint32_t id[kPickSlots];
    int kept[32], nkept;
};
__device__ __forceinline__ void pick_count(PickCount& s, int nrec, int k, int top, int tid, uint32_t* cid, int* held) {
    constexpr int T = kPickWarps * 32, G = T / 4;
    const int sub = tid & 3;
    auto before = [&](const unsigned long long* w, int n, unsigned long long mine) {  // (by four threads together)
        int c = 0;
#pragma unroll 4
        for (int i = sub; i < n; i += 4) c += w[i] > mine;
        c += __shfl_xor_sync(0xFFFFFFFFu, c, 1);
        return c + __shfl_xor_sync(0xFFFFFFFFu, c, 2);
    };
    for (int b = 0; b < nrec; b += G) {
        const int rec = b + (tid >> 2);
        unsigned long long m = 0;
        for (int q = sub; rec < nrec && q < k; q += 4) m = max(m, s.word[rec * k + q]);
        m = max(m, __shfl_xor_sync(0xFFFFFFFFu, m, 1));
        m = max(m, __shfl_xor_sync(0xFFFFFFFFu, m, 2));
        if (sub == 0 && rec < nrec) s.most[rec] = m;
    }
    if (tid == 0) s.nkept = *held = 0;
    __syncthreads();
    for (int b = 0; b < nrec; b += G) {
        const int rec = b + (tid >> 2);
        const unsigned long long m = rec < nrec ? s.most[rec] : 0ull;
        const int c = before(s.most, nrec, m);
        if (sub == 0 && m && c < top) s.kept[c] = rec, atomicAdd(&s.nkept, 1);
    }
    __syncthreads();
    // (the kept records' slots, in place of the records' maxima)
    const int n = s.nkept * k;
    for (int b = 0; b < n; b += G) {
        const int i = b + (tid >> 2), at = i < n ? s.kept[i / k] * k + i % k : 0;
        const unsigned long long m = i < n ? s.word[at] : 0ull;
        int c = 0;
        for (int j = 0; j < s.nkept; ++j) {
            const unsigned long long* w = s.word + s.kept[j] * k;
#pragma unroll 2
            for (int q = sub; q < k; q += 4) c += w[q] > m;
        }
        c += __shfl_xor_sync(0xFFFFFFFFu, c, 1);
        c += __shfl_xor_sync(0xFFFFFFFFu, c, 2);
        if (sub == 0 && m && c < top) cid[c] = s.id[at], atomicAdd(held, 1);
    }
}

// One CTA, or one cluster of CL CTAs, per row r of the step.
//   1. The best `top` slots of row r over the records in order (record by record, slot by slot), by key (RECORDS: by
//      rank16, and top is 1); an equal key keeps the earlier slot; a slot with key 0 or an id at or past `vocab` is empty: by
//      counting (COUNT: pick_count), or a warp takes a run of slots, 256 at a time beside its best so far; one warp merges the warps' lists.
//   2. (not RECORDS) Their exact logits: bf16 x row times the candidates' bf16 head rows, float32 sums (a warp per
//      candidate: every lane sums its 8-element pieces in order, then a shuffle tree), rounded to bf16 with `round`.
//   3. The pick: the largest logit (order32), the lowest id among equals. Row r of out (32 words):
//      [token, the first candidate by the device's own logit, count, 0 ...]; count is the candidates held (RECORDS: all
//      valid slots). No valid slot: [0, 0xFFFFFFFF, 0].
// Bound by latency: as `top` rounds over all slots read anew, with two barriers each, and one candidate after the other, it
// took a fifth of a vocabulary's call. CL, of three and more rows: a row is a cluster of CL CTAs; each finds the same
// candidates and takes its share of their rows, whose exact logits meet in the first one's shared memory. The candidates lie anywhere in
// the head, each in a page of its own as a rule, and sixteen such rows at a time were more than an SM has under way beside other CTAs
// that ask for theirs: records and pick of 8 rows of a head of 118656 columns of 3328 89.4 us with a CTA a row, 88.3 so, 4 rows 78.3 and
// 77.3; 4 rows of 34304 columns of 3712 45.2 and 41.6. One and two rows keep a CTA each: 65.9 and 66.4, 72.5 and 72.4 (31.7 and 31.6, 38.8
// and 38.5).
template <bool RECORDS, bool COUNT, int CL>
__global__ void __launch_bounds__(kPickWarps * 32) tkd_head_pick_kernel(const uint32_t* __restrict__ records, int nrec, int rows,
                                                                        int k, int top, uint32_t vocab,
                                                                        const uint16_t* __restrict__ x, int64_t ldx, int dim,
                                                                        const uint16_t* __restrict__ head, int64_t ld_head,
                                                                        int round, const uint32_t* __restrict__ tmap,
                                                                        uint32_t* __restrict__ out, uint32_t* __restrict__ ids_out) {
    __shared__ uint32_t srank[COUNT ? 1 : kPickWarps][32], sid[COUNT ? 1 : kPickWarps][32], cid[32], clogit[32];
    extern __shared__ __align__(16) uint8_t pick_smem[];
    __shared__ int held, nvalid[kPickWarps];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if constexpr (CL > 1) asm volatile("barrier.cluster.arrive.release;" ::: "memory");  // (waited for before the first store to another CTA)
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int r = blockIdx.x / CL, part = blockIdx.x % CL, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n = nrec * k;
    int mine = 0;
    if constexpr (COUNT) {
        PickCount& pc = *reinterpret_cast<PickCount*>(pick_smem);
#pragma unroll 4
        for (int c = tid; c < n; c += kPickWarps * 32) {
            const int rec = c / k, q = c - rec * k;
            const uint32_t* page = records + (size_t)rec * 2 * rows * k;
            const uint32_t key = __ldg(page + r * k + q) & 0xFFFFu, id = __ldg(page + (rows + r) * k + q);
            const bool ok = key && id < vocab;
            mine += ok;
            pc.id[c] = id;
            pc.word[c] = ok ? (unsigned long long)key << 32 | (0xFFFFFFFFu - (uint32_t)c) : 0ull;
        }
        mine = __reduce_add_sync(0xFFFFFFFFu, mine);
        if (lane == 0) nvalid[warp] = mine;
        __syncthreads();
        pick_count(pc, nrec, k, top, tid, cid, &held);
    } else {
        const int per = (n + kPickWarps - 1) / kPickWarps, c1 = min(n, (warp + 1) * per);
        uint32_t rank = 0, id = 0;  // lane t: the t-th so far
        for (int c0 = warp * per; c0 < c1; c0 += 32 * kPickOwn) {
            uint32_t word[kPickOwn + 1], ids[kPickOwn + 1];
#pragma unroll
            for (int j = 0; j < kPickOwn; ++j) {
                const int c = c0 + 32 * j + lane;
                word[j] = ids[j] = 0;
                if (c < c1) {
                    const int rec = c / k, q = c - rec * k;
                    const uint32_t* page = records + (size_t)rec * 2 * rows * k;
                    const uint32_t key = __ldg(page + r * k + q) & 0xFFFFu;
                    ids[j] = __ldg(page + (rows + r) * k + q);
                    if (key && ids[j] < vocab) {
                        word[j] = (RECORDS ? rank16(key) : key) << 12 | (uint32_t)(4095 - 32 - 32 * j - lane);
                        ++mine;
                    }
                }
            }
            word[kPickOwn] = rank ? rank << 12 | (uint32_t)(4095 - lane) : 0u, ids[kPickOwn] = id;
            pick_rounds(word, ids, top, lane, rank, id);
        }
        srank[warp][lane] = rank, sid[warp][lane] = id;
        mine = __reduce_add_sync(0xFFFFFFFFu, mine);
        if (lane == 0) nvalid[warp] = mine;
        __syncthreads();
        if (warp == 0) {
            uint32_t word[kPickWarps], ids[kPickWarps];
#pragma unroll
            for (int w = 0; w < kPickWarps; ++w) {
                const uint32_t rk = srank[w][lane];
                word[w] = rk ? rk << 12 | (uint32_t)(4095 - 32 * w - lane) : 0u, ids[w] = sid[w][lane];
            }
            pick_rounds(word, ids, top, lane, rank, id);
            cid[lane] = id;
            const uint32_t any = __ballot_sync(0xFFFFFFFFu, rank != 0);
            if (lane == 0) held = __popc(any);
        }
    }
    __syncthreads();
    const int nc = held;
    if constexpr (!RECORDS) {
        const uint16_t* xr = x + (size_t)r * ldx;
        if constexpr (CL > 1) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
        for (int c = warp * CL + part; c < nc; c += kPickWarps * CL) {
            const uint16_t* wr = head + (size_t)cid[c] * ld_head;
            float acc = 0.f;
#pragma unroll 16
            for (int d = lane * 8; d < dim; d += 256) {
                const uint4 wv = __ldg(reinterpret_cast<const uint4*>(wr + d));
                const uint4 xv = __ldg(reinterpret_cast<const uint4*>(xr + d));
                const uint32_t ww[4] = {wv.x, wv.y, wv.z, wv.w}, xx[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    acc = fmaf(__uint_as_float(ww[e] << 16), __uint_as_float(xx[e] << 16), acc);
                    acc = fmaf(__uint_as_float(ww[e] & 0xFFFF0000u), __uint_as_float(xx[e] & 0xFFFF0000u), acc);
                }
            }
#pragma unroll
            for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xFFFFFFFFu, acc, o);
            if (lane == 0) {
                uint32_t bits = __float_as_uint(acc);
                if (round) bits = (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(acc)) << 16;
                if constexpr (CL > 1) {
                    uint32_t to;  // (clogit[c] of the cluster's first CTA)
                    asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(to) : "r"((uint32_t)__cvta_generic_to_shared(&clogit[c])));
                    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(to), "r"(order32(bits)) : "memory");
                } else {
                    clogit[c] = order32(bits);
                }
            }
        }
        if constexpr (CL > 1) {
            asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
            if (part) return;
        } else {
            __syncthreads();
        }
    }
    if (warp == 0) {
        const bool have = lane < nc;
        uint32_t best = 0xFFFFFFFFu, count = (uint32_t)nc;
        if constexpr (RECORDS) {
            count = (uint32_t)__reduce_add_sync(0xFFFFFFFFu, lane < kPickWarps ? nvalid[lane] : 0);
            if (nc) best = cid[0];
        } else if (nc) {
            const uint32_t logit = have ? clogit[lane] : 0u, most = __reduce_max_sync(0xFFFFFFFFu, logit);
            best = __reduce_min_sync(0xFFFFFFFFu, have && logit == most ? cid[lane] : 0xFFFFFFFFu);
        }
        uint32_t tok = nc ? best : 0u;
        if (RECORDS && nc && tmap) tok = __ldg(tmap + best);
        out[(size_t)r * 32 + lane] = lane == 0 ? tok : lane == 1 ? (nc ? cid[0] : 0xFFFFFFFFu) : lane == 2 ? count : 0u;
        if (ids_out && r == 0 && lane == 0) ids_out[0] = tok;
    }
}

template <bool RECORDS, bool COUNT, int CL>
int launch_pick_by(const uint32_t* records, int nrec, int rows, int k, int top, uint32_t vocab, const uint16_t* x, int64_t ldx,
                int dim, const uint16_t* head, int64_t ld_head, int round, const uint32_t* tmap, uint32_t* out,
                uint32_t* ids_out, cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(rows * CL));
    cfg.blockDim = dim3(kPickWarps * 32);
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (CL > 1) attr[1].id = cudaLaunchAttributeClusterDimension, attr[1].val.clusterDim = {CL, 1, 1}, cfg.numAttrs = 2;
    cfg.dynamicSmemBytes = COUNT ? sizeof(PickCount) : 0;
    return (int)cudaLaunchKernelEx(&cfg, tkd_head_pick_kernel<RECORDS, COUNT, CL>, records, nrec, rows, k, top, vocab, x, ldx, dim, head,
                                   ld_head, round, tmap, out, ids_out);
}
// Counting compares every record with every other, rounds take `top` turns: counting up to twenty records for each of the top. Measured,
// us in rounds / by counting: top 4, records of 2, 75 of them 4.8 / 4.1, 150 4.8 / 5.5; top 16, records of 4, 75 9.9 / 5.4, 256 10.2 / 7.9,
// 400 10.8 / 13.2; top 32, 512 18.5 / 17.7. One turn, as of the records' own pick, is shorter nearly always (75 of 8 2.7 / 3.1, 512 of
// 4 3.4 / 12.3).
template <bool RECORDS, class... A>
int launch_pick(const uint32_t* records, int nrec, int rows, int k, int top, A... more) {
    if constexpr (!RECORDS)
        if (nrec <= 20 * top && nrec <= kPickRecs && (int64_t)nrec * k <= kPickSlots)
            return rows > 2 ? launch_pick_by<RECORDS, true, kPickCluster>(records, nrec, rows, k, top, more...)
                            : launch_pick_by<RECORDS, true, 1>(records, nrec, rows, k, top, more...);
    if constexpr (!RECORDS)
        if (rows > 2) return launch_pick_by<RECORDS, false, kPickCluster>(records, nrec, rows, k, top, more...);
    return launch_pick_by<RECORDS, false, 1>(records, nrec, rows, k, top, more...);
}

}  // namespace

int tkd_launch_head_pick(const uint32_t* records, int nrec, int rows, int k, int top, uint32_t vocab, const uint16_t* x,
                         int64_t ldx, int dim, const uint16_t* head, int64_t ld_head, int round, uint32_t* out,
                         uint32_t* ids_out, cudaStream_t st) {
    return launch_pick<false>(records, nrec, rows, k, top, vocab, x, ldx, dim, head, ld_head, round, nullptr, out, ids_out, st);
}

int tkd_launch_head_pick_records(const uint32_t* records, int nrec, int rows, int k, uint32_t vocab, const uint32_t* tmap,
                                 uint32_t* out, uint32_t* ids_out, cudaStream_t st) {
    return launch_pick<true>(records, nrec, rows, k, 1, vocab, nullptr, 0, 0, nullptr, 0, 0, tmap, out, ids_out, st);
}
