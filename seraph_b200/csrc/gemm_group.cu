// gemm_group.cu - several independent products in one persistent launch, on FP16 operand parts.
//
//   C_p[M,N] (+)= sum over segments s of p of  A_s[M,K_s] B_s[N,K_s]^T        p = 0 .. nprob-1
//
// The plain products of a training step come in groups that share operands or a destination: q, k and v; gate and up; a
// projection's weight gradient with its input gradient; the input gradients that are summed (three for q, k, v).  As launches of their
// own each pays for a ramp, a tail and (when its tiles do not fill the SMs) a split-K pass; a small model's step was mostly that.  Here a
// group is one launch: the tiles of all its products are dealt together, and products that are added into one destination are
// segments of one k loop, so their sum never leaves the accumulators.
//
// As in gemm_tc_kernel's prepared-FP16 form (gemm_tc.cuh), CTA pairs (cta_group::2) compute 256 x BN tiles, and accumulation in tensor memory
// is cut every 64 k (twelve instructions) and added into registers with round-to-nearest adds.  What differs:
//   * a stage is 64 k (one such chunk) of the hi or of the lo parts: rows of 128 bytes, whole lines, where 32 k of both asked L2 twice for each;
//   * an operand's hi and lo parts are the third dimension of one tensor map; either operand may be K-major or MN-major, per segment, at
//     run time;
//   * the power-of-two scales of the two operands are applied as a chunk is added (an fma), since segments have their own;
//   * work items are handed out at run time: one warp of the pair's leader takes the next item from a counter and passes it to the
//     roles of both CTAs through a ring in shared memory.  Items are ordered longest first, so the schedule is a greedy one whatever the mix
//     of products; the order of the additions inside a tile does not depend on it;
//   * what a role does between two chunks is kept short, for a chunk is 768 (BN = 128) or 1536 cycles of the tensor core and the roles took longer: the
//     epilogue's loop has its width as a constant, waits that are over read no clock, an item arrives decoded.  In all, with the schedule below and
//     roles that wait for the preceding kernel only where they need it: 2048 x 8192 x 512 from 58.5 to 44.3 us, 64 x 128 x 512 (one tile) from
//     8.4 to 6.2 us, 256 x 256 tiles at one pass from 0.88 to 0.45 us a chunk;
//   * each epilogue warp sends its 32 rows out itself, 32 columns at a time, through two 4 KB buffers and tensor stores (or reductions).
//     An SM writes about 32 bytes a cycle to L2, 4096 cycles for its half of a 256 x 256 tile; with buffers that are refilled as they drain the
//     warps are back at the next tile's chunks after about 2900 cycles, which is what the two accumulators hide of it.  (Whole rows through
//     one buffer of 64 rows and store warps: 4900 cycles, a stall of 1.3 us a tile.)
// NT = 3: FP32-accurate (hi hi + lo hi + hi lo).  NT = 1: hi parts only, the 11 leading significant bits (what a TF32 instruction reads of an
// FP32 word, at twice its rate): the reduced-precision mode, for all but its smallest products (gg_single).
#include <stdio.h>
#include <type_traits>
#include "gemm_tc.cuh"
#include "attention_fused.cuh"
#include "gemm_plan.h"

#define GG_MAXS 10               // segments per launch
#define GG_RING 4                // items the slowest role may lag behind the scheduling warp
#define GG_AHEAD 8               // k blocks left to load of an item when the next one is asked for: enough to hide the hand-over, not more, so
                                 // that items go to the pairs that really are free first
#define GG_THREADS 384          // warps 0-3: loads, instructions, items; 4-11: epilogue
// Registers of a thread of the one and of the other: 128 accumulators, 32 words on their way and the addresses need more than the 184 that sixteen warps
// leave an epilogue thread; with twelve it has 216, and a chunk of 256 columns is drained in 800 cycles instead of 1300 (spills).  Their sum is what
// the CTA is launched with (384 x 168).
#define GG_REGS_LIGHT 72
#define GG_REGS_EPI 216
#define GG_EMPTY_ARRIVALS 21     // roles that take an item: 2 producers and 8 epilogue warps in both CTAs, the MMA warp in the leader

struct __align__(64) GgSeg {
    CUtensorMap a, b;            // parts: K-major {K, rows, part}, MN-major {rows, K, part}
    const float *amax_a, *amax_b;
    int K, kb;                   // kb: k blocks of 64
    float alpha;                 // factor of this segment
    int mn;                      // bit 0: A is MN-major, bit 1: B is
};
struct __align__(64) GgProb {
    CUtensorMap c;               // FP32 {N, M}, boxes of 32 columns x 32 rows, 128-byte swizzle
    unsigned* out_amax;          // largest |C| is left here (whole tiles; the fix-up leaves it for split ones), or NULL
    int M, N, bn, tiles_m, tiles_n, seg0, nseg, kb, acc;      // bn: width of its tiles
};
struct GgRun { int item0, prob, tile0, split, slot0; };      // items item0 .. : tiles tile0 .. of the product, `split` pieces each
struct GgParams {
    int nruns, items, nsegs, nprob;
    int heads, group;            // BATCH: query heads, and those of one K/V head
    unsigned* counter; int* status;
    CUtensorMap partial;         // workspace of the split tiles: {BN, 256 rows per piece}, the same boxes
    GgRun run[GG_MAXE];
    GgProb prob[GG_MAXP];
    GgSeg seg[GG_MAXS];
};

__device__ __forceinline__ bool gg_try_cluster(uint32_t addr, uint32_t parity) {
    uint32_t done;
    asm volatile("{\n\t.reg .pred P;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 P, [%1], %2;\n\tselp.u32 %0, 1, 0, P;\n\t}"
                 : "=r"(done) : "r"(addr), "r"(parity) : "memory");
    return done != 0;
}
__device__ __forceinline__ bool gg_wait_cluster(uint64_t* bar, uint32_t parity) {      // as mbar_wait, for data written by the other CTA of the pair
    const uint32_t addr = smem_u32(bar);
    if (gg_try_cluster(addr, parity)) return true;
    const long long t0 = clock64();
    for (;;) {
        if (gg_try_cluster(addr, parity)) return true;
        if (clock64() - t0 > TC_SPIN_CYCLES) return false;
    }
}
// An item's hand-over: decoded once by the warp that takes it from the counter (1000 cycles of table look-ups and divisions), not by every role.  The words
// travel with their own completion on the receiver's barrier (st.async), and a role gives a slot back without a release: it has only read the slot.
// Arrivals with release semantics waited 3000 cycles each for whatever their thread had in flight, half of a short item.
struct __align__(16) GgItem { int prob, mt, nt, kb0, kb1, slot, split, pad; };      // prob: -1 after the last item; slot: of the workspace, where split
__device__ __forceinline__ void gg_send_item(uint32_t slot_cluster, uint32_t bar_cluster, const GgItem& v) {
    asm volatile("mbarrier.arrive.expect_tx.relaxed.cluster.shared::cluster.b64 _, [%0], 32;" ::"r"(bar_cluster) : "memory");
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(slot_cluster), "r"(v.prob), "r"(v.mt), "r"(v.nt), "r"(v.kb0), "r"(bar_cluster) : "memory");
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(slot_cluster + 16), "r"(v.kb1), "r"(v.slot), "r"(v.split), "r"(0), "r"(bar_cluster) : "memory");
}
__device__ __forceinline__ void gg_arrive_relaxed(uint32_t bar_cluster) {
    asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar_cluster) : "memory");
}

__device__ __forceinline__ void gg_load_4d_pair(void* dst, const CUtensorMap* map, uint32_t bar_cluster, int c0, int c1, int c2, int c3) {
    asm volatile("cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
                 ::"r"(smem_u32(dst)), "l"(map), "r"(bar_cluster), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
}
__device__ __forceinline__ void af_arrive_local(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
struct GgWork { int prob, m0, n0, nb0, kb0, kb1, slot, head; bool split; };
template <bool BATCH>
__device__ __forceinline__ void gg_decode(const GgParams& p, int item, GgItem& w) {
    int r = 0;
    while (r + 1 < p.nruns && p.run[r + 1].item0 <= item) r++;
    const GgRun& run = p.run[r];
    const GgProb& pr = p.prob[run.prob];
    const int local = item - run.item0;
    if constexpr (BATCH) {                                         // the lowest rows first: they have the most k
        w.prob = run.prob; w.mt = pr.tiles_m - 1 - local / p.heads; w.nt = local % p.heads;
        w.split = w.slot = w.kb0 = 0; w.kb1 = min(pr.kb, (w.mt + 1) * 4);
        return;
    }
    const int t = run.split > 1 ? local / run.split : local, piece = run.split > 1 ? local % run.split : 0;
    tc_raster(run.tile0 + t, pr.tiles_m, pr.tiles_n, TC_GROUP_M / 2, &w.mt, &w.nt);
    w.prob = run.prob;
    w.split = run.split > 1;
    w.slot = run.slot0 + local;
    w.kb0 = 0; w.kb1 = pr.kb;
    if (w.split) {
        const int per = (pr.kb + run.split - 1) / run.split;
        w.kb0 = min(pr.kb, piece * per); w.kb1 = min(pr.kb, w.kb0 + per);
    }
}

template <int BN, int NT>
struct GgShape {
    static constexpr int NP = NT == 3 ? 2 : 1;                     // parts per operand
    static constexpr int A_PART = 128 * 128, B_PART = (BN / 2) * 128;
    static constexpr int STAGE = A_PART + B_PART;                  // one part of both operands
    // A load takes about a microsecond under load: 1.5 (BN = 256) to 3 (BN = 128) chunks of MMA time ahead of the one being multiplied.  With the
    // narrow tile six stages and two buffers per warp take 0.97 to 1.03 of the time of eight and one.
    static constexpr int STAGES = BN == 256 ? 5 : 8;
    static constexpr int NBUF = BN == 256 ? 2 : 1;                 // output staging: blocks of 32 rows x 32 columns per epilogue warp
    static constexpr int STG = 8 * NBUF * 4096;
    // accumulators in tensor memory.  Between a chunk's last instruction and the return of its accumulator lie a commit, the drain and two arrivals,
    // as long as a chunk of the narrow tile takes: with two of them its instructions waited (2048 x 8192 x 512: 58.7 us, with four 54.3).
    static constexpr int NACC = 512 / BN;
    static constexpr int SMEM = STAGES * STAGE + STG + 1024 + 512;
};

template <int BN, int NT, bool BATCH>
__global__ void __launch_bounds__(GG_THREADS, 1)
gg_kernel(const __grid_constant__ GgParams p) {
    using Sh = GgShape<BN, NT>;
    constexpr int NP = Sh::NP, A_PART = Sh::A_PART, STAGE = Sh::STAGE, STAGES = Sh::STAGES;
    constexpr int NACC = Sh::NACC;
    constexpr uint32_t TMEM_COLS = NACC * BN;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* stg = smem + STAGES * STAGE;
    uint64_t* full = (uint64_t*)(stg + Sh::STG);
    uint64_t* empty = full + STAGES;
    uint64_t* acc_full = empty + STAGES;          // [NACC]
    uint64_t* acc_empty = acc_full + NACC;        // [NACC]
    uint64_t* item_full = acc_empty + NACC;       // [GG_RING]
    uint64_t* item_empty = item_full + GG_RING;   // [GG_RING] (the leader's are used)
    uint64_t* item_req = item_empty + GG_RING;    // 1: the leader's producer asks for the next item
    GgItem* item_slot = (GgItem*)(((uintptr_t)(item_req + 1) + 15) & ~(uintptr_t)15);
    uint32_t* tmem_slot = (uint32_t*)(item_slot + GG_RING);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    const bool leader = rank == 0;
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; s++) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int b = 0; b < NACC; b++) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 16); }
        mbar_init(item_req, 1);
        for (int b = 0; b < GG_RING; b++) { mbar_init(&item_full[b], 1); mbar_init(&item_empty[b], GG_EMPTY_ARRIVALS); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 3 && lane < p.nsegs) {            // the tensor maps on their way to the cache
        asm volatile("prefetch.tensormap [%0];" ::"l"(&p.seg[lane].a) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&p.seg[lane].b) : "memory");
        if (lane < p.nprob) asm volatile("prefetch.tensormap [%0];" ::"l"(&p.prob[lane].c) : "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();                           // the peer's barriers exist before anything signals them
    // Every role waits for the kernel before this one where it first touches what that may still write: the operands, the scale words, the counter.
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    bool ok = true;
    // the n-th item of this CTA's roles: the first is the pair's number, the others are waited for, read, and their slot handed back; false after the last.
    // The arrival that hands a slot back is relaxed; it follows the reads because it depends on the words they brought.  A role that is a warp
    // (`whole`) votes on them, so that its one arrival depends on every lane's.
    auto next_item = [&](int n, bool whole, int rk, GgWork& w) -> bool {
        GgItem it;
        if (n == 0) gg_decode<BATCH>(p, (int)(blockIdx.x >> 1), it);
        else {
            const int s = (n - 1) % GG_RING;
            it.prob = -2; it.pad = 0;             // the wait ran out
            if (gg_wait_cluster(&item_full[s], ((n - 1) / GG_RING) & 1)) {
                const uint32_t a = smem_u32(&item_slot[s]);
                asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(it.prob), "=r"(it.mt), "=r"(it.nt), "=r"(it.kb0) : "r"(a) : "memory");
                asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(it.kb1), "=r"(it.slot), "=r"(it.split), "=r"(it.pad) : "r"(a + 16) : "memory");
            }
            bool read = it.prob >= -1 && it.pad == 0;      // so whenever the words have come
            if (whole) read = __all_sync(0xffffffffu, read);
            if (!read) { ok = false; return false; }
            if (!whole || lane == 0) gg_arrive_relaxed(mapa_u32(smem_u32(&item_empty[s]), 0));
            if (it.prob < 0) return false;
        }
        const int bn = p.prob[it.prob].bn;
        w.prob = it.prob; w.kb0 = it.kb0; w.kb1 = it.kb1; w.slot = it.slot; w.split = it.split != 0;
        w.m0 = it.mt * 256 + rk * 128; w.n0 = it.nt * bn; w.nb0 = (BATCH ? it.nt / p.group * bn : w.n0) + rk * (bn / 2); w.head = it.nt;
        return true;
    };

    const bool is_epi = warp >= 4 && warp < 12;
    if (!is_epi) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(GG_REGS_LIGHT));
        if (warp == 0 || warp == 3) {
            // ---------------- TMA producers: warp 0 fetches A, asks for items and announces the bytes, warp 3 fetches B ----------------
            // (one thread for both took 430 cycles a stage, as long as the tensor core has for half a chunk of the narrow tile)
            if (elect_one()) {
                const bool is_a = warp == 0;
                const uint32_t full0 = mapa_u32(smem_u32(full), 0);      // both CTAs' bytes land on the leader's barriers
                int s = 0;
                uint32_t par = 1;
                for (int n = 0; ok; n++) {
                    GgWork w;
                    if (!next_item(n, false, (int)rank, w)) break;
                    if (n == 0) sb_pdl_enter();
                    const GgProb& pr = p.prob[w.prob];
                    int off = 0, left = w.kb1 - w.kb0;
                    const int ask = is_a && leader ? min(left, GG_AHEAD) : -1;
                    if (left == 0 && ask == 0) af_arrive_local(item_req);
                    for (int sg = pr.seg0; sg < pr.seg0 + pr.nseg && ok; sg++) {
                        const GgSeg& g = p.seg[sg];
                        const int lo = max(w.kb0, off) - off, hi = min(w.kb1, off + g.kb) - off;
                        off += g.kb;
                        const bool mn = (g.mn & (is_a ? 1 : 2)) != 0;
                        const int boxes = is_a ? 2 : (pr.bn + 127) / 128;             // of 64 rows: an MN-major operand is fetched in whole lines
                        const uint32_t bytes = (uint32_t)(A_PART + ((g.mn & 2) ? (pr.bn + 127) / 128 * 8192 : pr.bn * 64)) * 2;
                        const CUtensorMap* map = is_a ? &g.a : &g.b;
                        const int row = is_a ? w.m0 : w.nb0;
                        uint8_t* base = is_a ? smem : smem + A_PART;
                        for (int kb = lo; kb < hi && ok; kb++) {
                            if (left-- == ask) af_arrive_local(item_req);
                            for (int part = 0; part < NP; part++) {
                                ok = mbar_wait(&empty[s], par);
                                if (!ok) break;
                                if (is_a && leader) mbar_expect_tx(&full[s], bytes);
                                uint8_t* st = base + s * STAGE;
                                const uint32_t fb = full0 + (uint32_t)(s * 8);
                                if (!mn) tma_load_3d_pair(st, map, fb, kb * 64, row, part);
                                else {
#pragma unroll
                                    for (int j = 0; j < 2; j++) {
                                        if (j >= boxes) continue;
                                        if (BATCH && is_a) gg_load_4d_pair(st + j * 8192, map, fb, row + 64 * j, kb * 64, w.head, part);
                                        else tma_load_3d_pair(st + j * 8192, map, fb, row + 64 * j, kb * 64, part);
                                    }
                                }
                                if (++s == STAGES) { s = 0; par ^= 1; }
                            }
                        }
                    }
                }
                if (!ok) atomicExch(p.status, SB_ERR_TIMEOUT);
            }
        } else if (warp == 1) {
            // ---------------- MMA issuer ----------------
            if (leader && elect_one()) {
                uint32_t git = 0, gch = 0;
                for (int n = 0; ok; n++) {
                    GgWork w;
                    if (!next_item(n, false, 0, w)) break;
                    const GgProb& pr = p.prob[w.prob];
                    int off = 0;
                    for (int sg = pr.seg0; sg < pr.seg0 + pr.nseg && ok; sg++) {
                        const GgSeg& g = p.seg[sg];
                        const int lo = max(w.kb0, off) - off, hi = min(w.kb1, off + g.kb) - off;
                        off += g.kb;
                        const bool amn = (g.mn & 1) != 0, bmn = (g.mn & 2) != 0;
                        const uint32_t idesc = (1u << 4) | ((amn ? 1u : 0u) << 15) | ((bmn ? 1u : 0u) << 16) | ((uint32_t)(pr.bn >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
                        const uint64_t adva = amn ? 128 : 2, advb = bmn ? 128 : 2;      // 16 k in 16-byte units
                        const int K = g.K;
                        auto step = [&](uint32_t tmem_d, uint64_t a1, uint64_t b1, uint64_t a2, uint64_t b2, uint32_t acc) {
                            // consecutive instructions share an operand (hi hi, lo hi, hi lo): with the narrow tile, whose operand reads take as long
                            // as its arithmetic, all of hi hi first was 40 % slower
                            tc_mma_f16_pair(tmem_d, a1, b1, idesc, acc);
                            if (NT == 3) {
                                tc_mma_f16_pair(tmem_d, a2, b1, idesc, 1);
                                tc_mma_f16_pair(tmem_d, a1, b2, idesc, 1);
                            }
                        };
                        for (int kb = lo; kb < hi && ok; kb++, git += NP, gch++) {
                            const int buf = gch % NACC, s = git % STAGES, s2 = (git + 1) % STAGES;
                            ok = mbar_wait(&acc_empty[buf], ((gch / NACC) & 1) ^ 1) && mbar_wait(&full[s], (git / STAGES) & 1);
                            if (!ok) break;
                            tc_fence_after();
                            const uint32_t tmem_d = tmem_base + (uint32_t)(buf * BN);
                            const uint32_t sa = smem_u32(smem + s * STAGE), sb = sa + A_PART;
                            const uint64_t a1 = amn ? make_mn16_desc<64>(sa) : make_kmajor_desc<128>(sa);
                            const uint64_t b1 = bmn ? make_mn16_desc<64>(sb) : make_kmajor_desc<128>(sb);
                            if (NT == 3) {
                                ok = mbar_wait(&full[s2], ((git + 1) / STAGES) & 1);
                                if (!ok) break;
                                tc_fence_after();
                            }
                            const uint64_t lo_off = NT == 3 ? (uint64_t)((s2 - s) * (STAGE >> 4)) : 0, a2 = a1 + lo_off, b2 = b1 + lo_off;
                            const int left = K - kb * 64;
                            if (left >= 64) {
#pragma unroll
                                for (int kk = 0; kk < 4; kk++) step(tmem_d, a1 + kk * adva, b1 + kk * advb, a2 + kk * adva, b2 + kk * advb, kk ? 1u : 0u);
                            } else {
                                for (int kk = 0; kk < (left + 15) >> 4; kk++)      // the rest of a short last block is zeros
                                    step(tmem_d, a1 + kk * adva, b1 + kk * advb, a2 + kk * adva, b2 + kk * advb, kk ? 1u : 0u);
                            }
                            tc_commit_pair(&empty[s]);
                            if (NT == 3) tc_commit_pair(&empty[s2]);
                            tc_commit_pair(&acc_full[buf]);
                        }
                    }
                }
                if (!ok) atomicExch(p.status, SB_ERR_TIMEOUT);
            }
        } else if (warp == 2) {
            // ---------------- scheduler: hands the next item to the roles of both CTAs ----------------
            if (leader && elect_one()) {
                const int G = gridDim.x / 2;
                sb_pdl_wait();
                const uint32_t slot0 = mapa_u32(smem_u32(item_slot), 0), slot1 = mapa_u32(smem_u32(item_slot), 1), full1 = mapa_u32(smem_u32(item_full), 1), full0 = mapa_u32(smem_u32(item_full), 0);
                for (int n = 0; ok; n++) {
                    const int s = n % GG_RING;
                    ok = mbar_wait(item_req, n & 1) && gg_wait_cluster(&item_empty[s], ((n / GG_RING) & 1) ^ 1);
                    if (!ok) break;
                    const int item = G + (int)atomicAdd(p.counter, 1u);
                    GgItem v;
                    v.prob = -1; v.mt = v.nt = v.kb0 = v.kb1 = v.slot = v.split = 0;
                    if (item < p.items) gg_decode<BATCH>(p, item, v);
                    gg_send_item(slot0 + (uint32_t)(s * sizeof(GgItem)), full0 + (uint32_t)(s * 8), v);
                    gg_send_item(slot1 + (uint32_t)(s * sizeof(GgItem)), full1 + (uint32_t)(s * 8), v);
                    if (v.prob < 0) break;
                }
                if (!ok) atomicExch(p.status, SB_ERR_TIMEOUT);
            }
        }
    } else {
        // ---------------- epilogue: chunks from tensor memory, scaled, into register accumulators; tiles to the staging buffer ----------------
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(GG_REGS_EPI));
        const int q = warp & 3, half = (warp - 4) >> 2;
        const uint32_t sbuf = smem_u32(stg + (warp - 4) * Sh::NBUF * 4096);
        uint32_t gch = 0, pieces = 0;
        sb_pdl_wait();
        // The factor of each segment, in the lane of its number (read once: at every item the two words took 1400 cycles).  It undoes the operands'
        // power-of-two scales; where their product leaves the float range it takes two multiplications.
        float my_s1 = 0.f, my_s2 = 0.f;
        if (lane < p.nsegs) {
            const GgSeg& g = p.seg[lane];
            const int e = -tc_f16_shift(sb_word(g.amax_a)) - tc_f16_shift(sb_word(g.amax_b));
            const bool far = e < -120 || e > 120;
            my_s1 = (far ? tc_pow2(e / 2) : tc_pow2(e)) * g.alpha; my_s2 = far ? tc_pow2(e - e / 2) : 0.f;
        }
        __syncwarp();
        for (int n = 0; ok; n++) {
            GgWork w;
            if (!next_item(n, true, (int)rank, w)) break;
            const GgProb& pr = p.prob[w.prob];
            const int groups = pr.bn / 64, col0 = half * groups * 32;      // 32 columns at a time, half of the tile's per warp
            float accr[BN / 2];
#pragma unroll
            for (int j = 0; j < BN / 2; j++) accr[j] = 0.f;
            int off = 0;
            for (int sg = pr.seg0; sg < pr.seg0 + pr.nseg && ok; sg++) {
                const GgSeg& g = p.seg[sg];
                const int lo = max(w.kb0, off) - off, hi = min(w.kb1, off + g.kb) - off;
                off += g.kb;
                if (lo >= hi) continue;
                const float s1 = __shfl_sync(0xffffffffu, my_s1, sg), s2 = __shfl_sync(0xffffffffu, my_s2, sg);
                const bool far = s2 != 0.f;
                // W: groups of 32 columns of this warp, a constant of the loop; 0: `groups` of them with scales that take two factors
                auto drain = [&](auto w_t) {
                constexpr int W = decltype(w_t)::value;
                constexpr bool FAR = W == 0;
                for (int kb = lo; kb < hi && ok; kb++, gch++) {
                    const int buf = gch % NACC;
                    ok = mbar_wait(&acc_full[buf], (gch / NACC) & 1);
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * BN + col0);
#pragma unroll
                    for (int gi = 0; gi < (FAR ? BN / 64 : W); gi++) {
                        if (FAR && gi >= groups) continue;
                        uint32_t r[32];
                        tc_ld32(taddr + (uint32_t)(gi * 32), r);
                        if (gi == (FAR ? groups : W) - 1) {
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) mbar_arrive_cluster(mapa_u32(smem_u32(&acc_empty[buf]), 0));
                        }
#pragma unroll
                        for (int j = 0; j < 32; j++) accr[gi * 32 + j] = FAR ? accr[gi * 32 + j] + __uint_as_float(r[j]) * s1 * s2 : fmaf(__uint_as_float(r[j]), s1, accr[gi * 32 + j]);
                    }
                }
                };
                // A loop for each width, and one for far scales, chosen outside: with the choices inside, a chunk of 256 columns cost the warps 1250 cycles
                // instead of 640 (moves between copies of the accumulators), more than the tensor core takes for the single-pass form of it.
                if (far) drain(std::integral_constant<int, 0>());
                else if (BN == 256 && groups == 4) drain(std::integral_constant<int, BN / 64>());
                else if (BN == 256 && groups == 3) drain(std::integral_constant<int, BN == 256 ? 3 : 1>());
                else if (groups == 2) drain(std::integral_constant<int, 2>());
                else drain(std::integral_constant<int, 1>());
            }
            if (pr.out_amax && !w.split) {
                float m = 0.f;
#pragma unroll
                for (int j = 0; j < BN / 2; j++) m = fmaxf(m, fabsf(accr[j]));
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
                if (lane == 0 && m > 0.f) atomicMax(pr.out_amax, __float_as_uint(m));
            }
            if (!ok) break;
            const CUtensorMap* map = w.split ? &p.partial : &pr.c;
            const int x0 = (w.split ? 0 : w.n0) + col0, y0 = (w.split ? (w.slot * 2 + (int)rank) * 128 : w.m0) + q * 32;
            const bool inside = w.split || y0 < pr.M, accf = !w.split && pr.acc;
#pragma unroll
            for (int g = 0; g < BN / 64; g++) {
                if (g >= groups || !inside || !(w.split || x0 + g * 32 < pr.N)) continue;
                const uint32_t buf = sbuf + (pieces++ % Sh::NBUF) * 4096;      // the buffers in turn, whatever was skipped: the wait leaves the other one's store pending
                if (lane == 0) asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(Sh::NBUF - 1) : "memory");      // what was staged here before has been read
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 8; i++)
                    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(buf + (uint32_t)(lane * 128 + ((i ^ (lane & 7)) << 4))),
                                 "f"(accr[g * 32 + 4 * i]), "f"(accr[g * 32 + 4 * i + 1]), "f"(accr[g * 32 + 4 * i + 2]), "f"(accr[g * 32 + 4 * i + 3]) : "memory");
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) {
                    if (accf) asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.tile.bulk_group [%0, {%1, %2}], [%3];" ::"l"(map), "r"(x0 + g * 32), "r"(y0), "r"(buf) : "memory");
                    else      asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(map), "r"(x0 + g * 32), "r"(y0), "r"(buf) : "memory");
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                }
            }
        }
        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");      // the buffers are read out before the CTA gives its shared memory back
        if (!ok && lane == 0) atomicExch(p.status, SB_ERR_TIMEOUT);
        tc_fence_before();
    }
    __syncthreads();
    asm volatile("barrier.cluster.arrive.relaxed.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");      // neither CTA leaves while the other may still signal it or read its operands
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS));
    }
}

// Adds the pieces of the split tiles into C in piece order: one thread per four columns of one row, all products of the launch.
struct GgFixRun { float* C; long ldc; unsigned* out_amax; int M, N, bn, tiles_m, tiles_n, acc, tile0, split, slot0, block0; };
struct GgFixParams { int n, blocks, bn; const float* partial; GgFixRun f[GG_MAXP]; };
static __global__ void __launch_bounds__(256) gg_fixup_kernel(const __grid_constant__ GgFixParams p) {
    sb_pdl_enter();
    const int bn4 = p.bn >> 2;
    const long item = (long)blockIdx.x * blockDim.x + threadIdx.x;
    const int blk = (int)(item / (128 * bn4)), i = (int)(item % (128 * bn4));
    if (blk >= p.blocks) return;
    int k = 0;
    while (k + 1 < p.n && p.f[k + 1].block0 <= blk) k++;
    const GgFixRun& f = p.f[k];
    const int t = (blk - f.block0) >> 1, rank = (blk - f.block0) & 1;
    int mt, nt;
    tc_raster(f.tile0 + t, f.tiles_m, f.tiles_n, TC_GROUP_M / 2, &mt, &nt);
    const int r = i / bn4, col = (i % bn4) * 4;
    const int row = mt * 256 + rank * 128 + r, c0 = nt * f.bn + col;
    if (row >= f.M || c0 >= f.N || col >= f.bn) return;         // N is a multiple of 4: a group of columns is inside or outside
    const size_t block = (size_t)128 * p.bn;
    const float* p0 = p.partial + ((size_t)(f.slot0 + t * f.split) * 2 + rank) * block + (size_t)r * p.bn + col;
    float4* cp = (float4*)(f.C + (size_t)row * f.ldc + c0);
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (f.acc) v = *cp;
    float4 o[8];
#pragma unroll
    for (int s = 0; s < 8; s++) if (s < f.split) o[s] = __ldcg((const float4*)(p0 + (size_t)s * 2 * block));
#pragma unroll
    for (int s = 0; s < 8; s++) if (s < f.split) { v.x += o[s].x; v.y += o[s].y; v.z += o[s].z; v.w += o[s].w; }
    *cp = v;
    if (f.out_amax) {
        const float m = sb_amax4(0.f, v);
        const unsigned live = __activemask();
        const unsigned wm = __reduce_max_sync(live, __float_as_uint(m));
        if ((int)(threadIdx.x & 31) == __ffs(live) - 1 && wm != 0u) atomicMax(f.out_amax, wm);
    }
}

// the schedule of a group (gemm_plan.h)
static const GgPlan* gg_plan(sb_ctx_t* c, const GgPlanKey* key) {
    if (!c->gg_plans) c->gg_plans = calloc(1, sizeof(GgPlanTable));
    return c->gg_plans ? gg_plan_find((GgPlanTable*)c->gg_plans, key) : nullptr;
}

template <int BN, int NT, bool BATCH = false>
static bool gg_launch_t(sb_ctx_t* c, const GgParams& p, int G) {
    auto kern = gg_kernel<BN, NT, BATCH>;
    constexpr int smem = GgShape<BN, NT>::SMEM;
    static_assert(smem <= 232448, "shared memory of one CTA");
    static bool attr_set = false;
    if (!attr_set) {
        cudaFuncAttributes fa;
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess || cudaFuncGetAttributes(&fa, kern) != cudaSuccess) return false;
        // setmaxnreg.inc takes from the registers the CTA was launched with and would wait for good on a build that has fewer
        if (fa.numRegs * GG_THREADS < GG_REGS_LIGHT * 128 + GG_REGS_EPI * 256) return false;
        attr_set = true;
    }
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof cfg);
    cfg.gridDim = dim3((unsigned)(2 * G)); cfg.blockDim = dim3(GG_THREADS); cfg.dynamicSmemBytes = smem; cfg.stream = (cudaStream_t)c->pub.stream;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at; cfg.numAttrs = 2;
    c->launches++;
    return cudaLaunchKernelEx(&cfg, kern, p) == cudaSuccess;
}

// --------------------------------------------------------------------------- host side
bool gg_shape_ok(int M, int N, int K, int tA, int tB) {
    if (M < 8 || N < 8 || K < 8 || (N & 3) || (double)M * N * K < (double)(1 << 19)) return false;      // smaller: the CUDA-core kernel
    if (tA && tB) tA = tB = 0;
    return (tA ? (M & 7) == 0 : (K & 7) == 0) && (tB ? (K & 7) == 0 : (N & 7) == 0);
}
// In the single-pass mode a product of fewer than 32 rows or columns, or under 2^21 multiply-adds, stays FP32-accurate: that mode's TF32 kernel left
// those to the FP32 cores, and so few operations gain nothing from two passes less.  The rank of an adapter counts as the multiple of 128 that it
// was padded to there.  One such product and the launch takes three passes.
static bool gg_single(const sb_gemm_job_t* b) {
    int d[3] = {b->M, b->N, b->K};
    if (b->rank) d[b->rank - 1] = (d[b->rank - 1] + 127) / 128 * 128;
    return d[0] >= 32 && d[1] >= 32 && (double)d[0] * d[1] * d[2] >= (double)(1 << 21);
}
static bool gg_mode(const sb_ctx_t* c, int* nt) {
    const int mode = c->pub.use_bf16 ? SB_GEMM_BF16 : c->gemm_mode;
    *nt = mode == SB_GEMM_BF16 ? 1 : 3;
    return c->gemm_pair && (mode == SB_GEMM_FP16X3 || mode == SB_GEMM_BF16) && tc_load_encode();
}
extern "C" int sb_gemm_group_takes(sb_ctx_t* c, int M, int N, int K, int tA, int tB) {
    int nt;
    return gg_mode(c, &nt) && gg_shape_ok(M, N, K, tA, tB) ? 1 : 0;
}

struct GgOperand { const float* x; size_t n; __half* h; float* amax; float* guess; bool fresh, kept; int slot; };      // kept: the parts outlive the step
// the parts of an operand: those a producer or an earlier product of the step left, or a slot to make them in
static int gg_operand(sb_ctx_t* c, GgOperand* ops, int* nops, const float* x, size_t n) {
    for (int i = 0; i < *nops; i++) if (ops[i].x == x && ops[i].n == n) return i;
    GgOperand* o = &ops[*nops];
    o->x = x; o->n = n; o->slot = -1; o->kept = false;
    void* h; int fresh;
    if (sb_parts_find(c, x, n, &h, &o->amax, &fresh)) { o->h = (__half*)h; o->fresh = fresh != 0; o->kept = fresh == SB_PARTS_MAKE_KEPT; o->guess = sb_parts_guess(c, x); }
    else {
        bool fr;
        const int s = sb_f16_slot(c, x, n, -1, &fr);
        if (s < 0) return -1;
        o->h = (__half*)c->f16_slot[s].h; o->fresh = fr; o->slot = s;
        if (fr) c->f16_slot[s].amax = c->d_amax + s;
        o->amax = c->f16_slot[s].amax; o->guess = c->d_amax + SB_F16_SLOTS + 2 * s;
    }
    return (*nops)++;
}
// Parts of the operands that have none yet: one launch, or three where some larger ones have no known maximum
static void gg_prepare(sb_ctx_t* c, GgOperand* ops, int n) {
    TcMulti sp;
    tc_multi_begin(&sp);
    double bytes = 0;
    int tk = -1;
    bool any = false;
    for (int i = 0; i < n; i++) {
        GgOperand* o = &ops[i];
        if (o->fresh) {
            if (!any) { tk = sb_tick_begin(c, SB_CLS_GEMM_PREP); any = true; }
            float* left = o->kept ? NULL : sb_amax_lookup(c, o->x, o->n);
            if (left) { o->amax = left; if (o->slot >= 0) c->f16_slot[o->slot].amax = left; else sb_parts_set_amax(c, o->x, left); }
            tc_multi_add(&sp, o->x, o->n, o->h, o->amax, left ? nullptr : o->guess);
            bytes += 8.0 * o->n;
        }
        if (sp.n == TC_MULTI || i + 1 == n) { tc_multi_split(c, sp); tc_multi_begin(&sp); }
    }
    if (any) sb_tick_end(c, tk, 0.0, bytes);
}
// Parts of registered tensors (weights) ahead of the products that read them: one to three launches instead of as many per tensor
extern "C" void sb_parts_prepare(sb_ctx_t* c, const float* const* x, const size_t* n, int count) {
    GgOperand ops[TC_MULTI];
    for (int i0 = 0; i0 < count; ) {
        int k = 0;
        for (; i0 < count && k < TC_MULTI; i0++) {
            void* h; int fresh;
            if (!sb_parts_find(c, x[i0], n[i0], &h, &ops[k].amax, &fresh)) continue;      // no parts for it: its products prepare it
            ops[k].x = x[i0]; ops[k].n = n[i0]; ops[k].h = (__half*)h; ops[k].fresh = fresh != 0; ops[k].kept = fresh == SB_PARTS_MAKE_KEPT; ops[k].slot = -1; ops[k].guess = sb_parts_guess(c, x[i0]);
            k++;
        }
        gg_prepare(c, ops, k);
    }
}

static bool gg_map(sb_ctx_t* c, CUtensorMap* m, const __half* h, size_t n, int rows, int K, bool mn, int box_rows) {
    // parts are n halfs apart; K-major [rows, K]: {K, rows, part}; MN-major [K, rows]: {rows, K, part}
    const cuuint64_t dims[3] = {(cuuint64_t)(mn ? rows : K), (cuuint64_t)(mn ? K : rows), 2};
    const cuuint64_t strides[2] = {(cuuint64_t)(mn ? rows : K) * 2, (cuuint64_t)n * 2};
    const cuuint32_t box[3] = {64u, mn ? 64u : (cuuint32_t)box_rows, 1u};
    return tc_encode(c, m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, h, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
}

static bool gg_map_out(sb_ctx_t* c, CUtensorMap* m, const float* C, int M, int N) {
    const cuuint64_t dims[2] = {(cuuint64_t)N, (cuuint64_t)M}, strides[1] = {(cuuint64_t)N * 4};
    const cuuint32_t box[2] = {32u, 32u};
    return tc_encode(c, m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, C, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE);
}

// one launch (and the fix-up pass of its split tiles); jobs with the same destination as the one before are its further segments
static bool gg_run(sb_ctx_t* c, const sb_gemm_job_t* jobs, int njobs, int nt) {
    GgOperand ops[2 * GG_MAXS];
    int nops = 0, ia[GG_MAXS], ib[GG_MAXS];
    for (int j = 0; j < njobs; j++) {
        ia[j] = gg_operand(c, ops, &nops, jobs[j].A, (size_t)jobs[j].M * jobs[j].K);
        ib[j] = gg_operand(c, ops, &nops, jobs[j].B, (size_t)jobs[j].N * jobs[j].K);
        if (ia[j] < 0 || ib[j] < 0) return false;
    }
    gg_prepare(c, ops, nops);
    GgParams p;
    memset(&p, 0, sizeof p);
    GgPlanKey key;
    memset(&key, 0, sizeof key);
    int np = 0, of[GG_MAXS];      // of: product of each job
    double flops = 0, bytes = 0;
    for (int j = 0; j < njobs; j++) {
        const sb_gemm_job_t* b = &jobs[j];
        const bool more = j > 0 && b->C == jobs[j - 1].C && b->acc;
        flops += 2.0 * b->M * b->N * b->K;
        bytes += 4.0 * ((double)b->M * b->K + (double)b->N * b->K + (more ? 0.0 : (double)b->M * b->N * (b->acc ? 2 : 1)));
        if (!more) {
            GgProb* q = &p.prob[np++];
            q->M = b->M; q->N = b->N; q->seg0 = j; q->nseg = 0; q->kb = 0; q->acc = b->acc;
        }
        GgProb* q = &p.prob[np - 1];
        p.seg[j].K = b->K; p.seg[j].alpha = b->alpha == 0.f ? 1.f : b->alpha; p.seg[j].kb = (b->K + 63) / 64;
        q->nseg++; q->kb += p.seg[j].kb;
        of[j] = np - 1;
    }
    const int sms = c->pub.gpu_sm_count > 0 ? c->pub.gpu_sm_count : 148;
    key.nt = nt; key.G = max(1, (sms - (c->gemm_reserve_sms < sms ? c->gemm_reserve_sms : 0)) / 2);
    for (int i = 0; i < np; i++) gg_key_add(&key, p.prob[i].M, p.prob[i].N, p.prob[i].kb);
    const GgPlan* plan = gg_plan(c, &key);
    if (!plan) return false;
    const int bn = plan->bn;
    for (int j = 0; j < njobs; j++) {
        const sb_gemm_job_t* b = &jobs[j];
        int tA = b->tA, tB = b->tB;
        if (tA && tB) tA = tB = 0;
        const GgOperand *oa = &ops[ia[j]], *ob = &ops[ib[j]];
        p.seg[j].mn = (tA ? 1 : 0) | (tB ? 0 : 2);
        p.seg[j].amax_a = oa->amax; p.seg[j].amax_b = ob->amax;
        if (!gg_map(c, &p.seg[j].a, oa->h, oa->n, b->M, b->K, tA != 0, 128) ||
            !gg_map(c, &p.seg[j].b, ob->h, ob->n, b->N, b->K, !tB, plan->w[of[j]] / 2)) return false;
    }
    GgFixParams fx;
    fx.n = fx.blocks = 0; fx.bn = bn;
    int slots = 0;
    for (int i = 0; i < np; i++) {
        GgProb* q = &p.prob[i];
        q->bn = plan->w[i];
        q->tiles_m = (q->M + 255) / 256; q->tiles_n = (q->N + q->bn - 1) / q->bn;
        float* C = jobs[q->seg0].C;
        if (!q->acc) q->out_amax = sb_amax_take(c, C, (size_t)q->M * q->N);      // an announced output: the epilogue leaves max |C|
        if (!gg_map_out(c, &q->c, C, q->M, q->N)) return false;
    }
    for (int r = 0; r < plan->nruns; r++) {
        const GgPlanRun* pr = &plan->run[r];
        GgProb* q = &p.prob[pr->prob];
        p.run[r].item0 = p.items; p.run[r].prob = pr->prob; p.run[r].tile0 = pr->tile0; p.run[r].split = pr->split; p.run[r].slot0 = slots;
        p.items += pr->tiles * pr->split;
        if (pr->split > 1) {
            GgFixRun* f = &fx.f[fx.n++];
            f->C = jobs[q->seg0].C; f->ldc = q->N; f->out_amax = q->out_amax; f->M = q->M; f->N = q->N; f->bn = q->bn; f->tiles_m = q->tiles_m; f->tiles_n = q->tiles_n;
            f->acc = q->acc; f->tile0 = pr->tile0; f->split = pr->split; f->slot0 = slots; f->block0 = fx.blocks;
            fx.blocks += pr->tiles * 2;
            slots += pr->tiles * pr->split;
        }
    }
    p.nruns = plan->nruns; p.nsegs = njobs; p.nprob = np;
    float* partial = nullptr;
    if (slots) {
        partial = (float*)sb_gemm_stage(c, 4, (size_t)slots * 2 * 128 * bn * sizeof(float));
        if (!partial || !gg_map_out(c, &p.partial, partial, slots * 256, bn)) return false;
    }
    p.counter = sb_item_counter(c);
    if (!p.counter) return false;
    p.status = c->d_status;
    int tg = sb_tick_begin(c, SB_CLS_GEMM);
    const int G = p.items < key.G ? p.items : key.G;
    bool ok = bn == 256 ? (nt == 3 ? gg_launch_t<256, 3>(c, p, G) : gg_launch_t<256, 1>(c, p, G))
                        : (nt == 3 ? gg_launch_t<128, 3>(c, p, G) : gg_launch_t<128, 1>(c, p, G));
    if (ok && fx.blocks) {
        fx.partial = partial;
        const long items = (long)fx.blocks * 128 * (bn / 4);
        sb_launch(gg_fixup_kernel, dim3((unsigned)((items + 255) / 256)), dim3(256), 0, (cudaStream_t)c->pub.stream, fx);
        c->launches++;
    }
    sb_tick_end(c, tg, flops, bytes);
    return ok && cudaGetLastError() == cudaSuccess;
}

// Returns 0 when the products were launched, 1 when some are not for this kernel (nothing has been launched then).
extern "C" int sb_gemm_group_try(sb_ctx_t* c, const sb_gemm_job_t* jobs, int njobs) {
    int nt;
    if (njobs <= 0 || !gg_mode(c, &nt)) return 1;
    for (int j = 0; j < njobs; j++)
        if (!gg_shape_ok(jobs[j].M, jobs[j].N, jobs[j].K, jobs[j].tA, jobs[j].tB) || !tc_aligned16(jobs[j].A) || !tc_aligned16(jobs[j].B) || !tc_aligned16(jobs[j].C)) return 1;
    const int keep = c->f16_keep;
    if (!keep) c->f16_keep = 1;                                   // operands of one group never share a slot
    bool ok = true;
    for (int j = 0; j < njobs && ok; ) {
        int k = j + 1;
        while (k < njobs && k - j < GG_MAXS) k++;
        if (k < njobs) while (k > j + 1 && jobs[k].C == jobs[k - 1].C && jobs[k].acc) k--;      // a sum stays in one launch
        int passes = nt;
        for (int i = j; i < k; i++) if (!gg_single(&jobs[i])) passes = 3;
        ok = gg_run(c, jobs + j, k - j, passes);
        j = k;
    }
    if (!keep) sb_gemm_keep_end(c);
    if (!ok) sb_set_status(c, SB_ERR_CUDA);
    return 0;
}

// dQ = dS K of an attention backward: for every sequence and query head [S, 128] from the parts of dS^T ([slot of (sequence, head): af_slot_row][key][query], rows of Sp) and
// of K.  The query rows of a tile of 256 need the keys up to its last row.  A product is a sequence; its tiles of all heads are items of one launch, which
// takes GG_MAXP sequences.  (A launch per sequence of gemm_tc_kernel, two of them side by side: 8 x 2048 tokens, 16 heads, 296 us; this 250,
// of which the parts of dS alone, 1.07 GB, take 164.)  starts: boundaries on the host.  0: launched.
extern "C" int sb_gemm_dq(sb_ctx_t* c, const void* ds, size_t ds_part, const float* ds_bound, const void* k, size_t k_part, const float* amax_k, float* dQ,
                          const int* starts, int nseq, int Sp, int Hq, int g) {
    if (!tc_load_encode()) return 1;
    const int qd = Hq * 128, kvd = qd / g;
    const int sms = c->pub.gpu_sm_count > 0 ? c->pub.gpu_sm_count : 148, pairs = max(1, (sms - (c->gemm_reserve_sms < sms ? c->gemm_reserve_sms : 0)) / 2);
    for (int b0 = 0; b0 < nseq; ) {
        GgParams p;
        memset(&p, 0, sizeof p);
        int seq[GG_MAXP], n = 0;
        for (; b0 < nseq && n < GG_MAXP; b0++) {                  // the longest first
            const int S = starts[b0 + 1] - starts[b0];
            if (S <= 0) continue;
            int j = n++;
            for (; j > 0 && starts[seq[j - 1] + 1] - starts[seq[j - 1]] < S; j--) seq[j] = seq[j - 1];
            seq[j] = b0;
        }
        if (!n) break;
        for (int i = 0; i < n; i++) {
            const int t0 = starts[seq[i]], S = starts[seq[i] + 1] - t0;
            GgSeg* sg = &p.seg[i];
            GgProb* q = &p.prob[i];
            sg->K = S; sg->kb = (S + 63) / 64; sg->alpha = 1.f; sg->mn = 3; sg->amax_a = ds_bound; sg->amax_b = amax_k;
            q->M = S; q->N = qd; q->bn = 128; q->tiles_m = (S + 255) / 256; q->tiles_n = Hq; q->seg0 = i; q->nseg = 1; q->kb = sg->kb;
            p.run[i].item0 = p.items; p.run[i].prob = i; p.run[i].split = 1;
            p.items += q->tiles_m * Hq;
            const cuuint64_t ad[4] = {(cuuint64_t)S, (cuuint64_t)S, (cuuint64_t)Hq, 2}, as[3] = {(cuuint64_t)Sp * 2, (cuuint64_t)((S + 127) & ~127) * Sp * 2, (cuuint64_t)ds_part * 2};
            const cuuint32_t abox[4] = {64u, 64u, 1u, 1u}, one[4] = {1u, 1u, 1u, 1u};
            if (g_tc_encode(&sg->a, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, (void*)((const __half*)ds + (size_t)af_slot_row(Hq, seq[i], 0, t0, S) * Sp), ad, as, abox, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
                            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) return 1;
            const cuuint64_t bd[3] = {(cuuint64_t)kvd, (cuuint64_t)S, 2}, bs[2] = {(cuuint64_t)kvd * 2, (cuuint64_t)k_part * 2};
            const cuuint32_t bbox[3] = {64u, 64u, 1u};
            if (!tc_encode(c, &sg->b, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, (const __half*)k + (size_t)t0 * kvd, bd, bs, bbox, CU_TENSOR_MAP_SWIZZLE_128B) ||
                !gg_map_out(c, &q->c, dQ + (size_t)t0 * qd, S, qd)) return 1;
        }
        p.nruns = p.nsegs = p.nprob = n;
        p.heads = Hq; p.group = g;
        p.counter = sb_item_counter(c);
        if (!p.counter) return 1;
        p.status = c->d_status;
        if (!gg_launch_t<128, 3, true>(c, p, p.items < pairs ? p.items : pairs)) return 1;
    }
    return cudaGetLastError() == cudaSuccess ? 0 : 1;
}
