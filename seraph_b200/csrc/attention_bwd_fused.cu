// attention_bwd_fused.cu - causal attention backward with dK and dV kept on chip (head sizes 64 and 128, FP16 hi/lo parts,
// FP32-level accuracy).  Replaces batch_attention_backward_packed_kernel / flash_attention_bwd_packed_kernel of the
// reference (src/cuda_train_context.cu:1013, :2012), which add into dK and dV with float atomics from every query tile.
//
// One CTA owns 128 consecutive keys of one (sequence, K/V head) for its whole life: the FP16 parts of those rows of V
// stay in shared memory (64 KB), those of K in tensor memory (128 columns), where they are the A operand of the S^T
// product: an MMA of 32 queries then reads 1 KB instead of 5 KB from shared memory, which is what its time went by.
// The CTA walks over the query heads of the K/V head's group and, for each, over the sequence's queries from the
// diagonal to the end in blocks of 32 (Q and dO parts, 32 KB per block, three stages):
//
//   S^T  = K Q_j^T,  dP^T = V dO_j^T     tcgen05.mma kind::f16, M 128 (keys) x N 32 (queries) x K 128, three passes each
//                                        (k1 q1 + k2 q1 + k1 q2), accumulators in tensor memory, two buffers
//   P^T  = exp(S^T/sqrt(hd) - lse),  dS^T = P^T o (dP^T - D)/sqrt(hd)      by the elementwise warps, one key row per
//                                        thread; both go BACK INTO TENSOR MEMORY as FP16 hi/lo parts, over the very
//                                        columns S^T and dP^T came from (tcgen05.st), to be the A operand of
//   dV  += P^T dO_j,  dK += dS^T Q_j     M 128 (keys) x N 128 (head dim) x K 32 (queries), A from tensor memory, B = the
//                                        same Q / dO tiles read in place MN-major; accumulators of 128 columns each in
//                                        tensor memory, summed over the query blocks and heads
//
// (128-wide heads; for 64-wide ones see AB_DRAIN.)  The tensor core adds into its accumulator with truncation, so a chain of accumulation is cut after AB_DRAIN query
// blocks: four drain warps read dK and dV out of tensor memory and add them into the output (round to nearest,
// performed in L2).  A dK/dV element is only ever touched by the one CTA that owns its key, one chain's additions have
// been performed before the next chain's are issued, and the output is zeroed (or holds the caller's values) before the
// launch: the result does not depend on scheduling and is the same bits on every run.
// dS^T also leaves the chip, as FP16 parts laid out [head slot = (sequence, K/V head, group member)][key][query]: dQ = dS K is one more launch, of the
// grouped kernel (long 128-wide sequences) or of at_dq_bwd_kernel below (keys up to the diagonal, A read MN-major).  P never reaches memory, dS is written once
// and read once: 8 bytes per score element instead of the 20 of the score-materialising path.
//
// Everything that leaves the CTA goes through shared memory and the TMA unit.  With one key row per thread (the layout
// tensor memory gives), a warp's direct stores and reductions touch 32 different rows per instruction, 32 memory
// transactions each; cycle counters in the warps showed the load/store unit busy two thirds of a step with them and the
// elementwise warps, which bound the step, waiting on it.  So the elementwise warps stage a step's dS^T parts in shared memory
// and one thread stores them as two tiles of 128 keys x 32 queries (a store per warp cost the issuing lane 500 cycles a step: the
// TMA unit takes few, large requests), each drain warp stages 32 rows x 32 columns of a chain at a time
// (128-byte swizzle, conflict-free for row-per-lane writes) and adds it with a TMA reduction, and the log-sum-exp and the row
// dot products D come from copies transposed to [sequence][head][query] (at_bwd_prep2_kernel): a bulk copy brings a step's 32 of each
// beside its tiles, and a warp reads its 16 as four 16-byte loads from one address.  A key block that reaches past its sequence's end keeps the
// per-thread reductions, so that no CTA ever adds (even a zero) into a row of the next sequence.
//
// Warps (16): 0 TMA producer, 1 MMA issuer (owns the tensor-memory allocation), 4-11 elementwise (a lane quarter and half of
// a step's queries each), 12-15 drain.  Every mbarrier wait is bounded; a wait that runs out sets the status word and the CTA drains
// and frees its tensor memory.
#include <type_traits>
#include "attention_fused.cuh"

#define AB_BK 128                 // keys per CTA
#define AB_BQ 32                  // queries per step
#define AB_STAGES 3
#define AB_THREADS 512
// Steps per accumulation chain in tensor memory.  128-wide heads: 8 (48 instructions, 3e-6 of one-sided truncation), a chain is added into
// the output in L2.  64-wide heads: 2 (12 instructions, as in the GEMM kernel); their rows of dK and dV fit the drain warps' registers, where
// the chains are added up, and a second set of accumulators in tensor memory takes the next chain meanwhile: the output is written once.
// (Chains of 8 here made the 33M model's gradients 1.5 times less accurate.)
#define AB_DRAIN(NH) ((NH) == 1 ? 2 : 8)
// shared memory, for NH = head size / 64 halves of 128-byte rows:
#define AB_KV_BYTES(NH) ((NH) * 32768)        // the parts of 128 rows of V: 2 parts x NH halves of the head dimension x 128 x 128 B
#define AB_STAGE_BYTES(NH) ((NH) * 16384)     // one step's Q parts and dO parts, 32 rows each
#define AB_OFF_EWS(NH) (AB_KV_BYTES(NH) + AB_STAGES * AB_STAGE_BYTES(NH))      // dS^T staging: 2 buffers x (hi tile 8 KB, lo tile 8 KB); a tile is 128 keys x 32 queries (64-byte rows)
#define AB_OFF_DRS(NH) (AB_OFF_EWS(NH) + 2 * 16384)                      // per drain warp 2 buffers x 4 KB: 32 rows x 32 floats, 128-byte swizzle
                                                                 // (before the first step these 64 KB receive the parts of K on their way to tensor memory)
#define AB_OFF_BAR(NH) (AB_OFF_DRS(NH) + 4 * 8192)
#define AB_SMEM(NH) (AB_OFF_BAR(NH) + 1024 + 1024)
#define AB_REGS_LIGHT 72          // producer / MMA issuer warpgroup
#define AB_REGS_EW 120             // the two elementwise warpgroups
#define AB_REGS_DRAIN 200          // the drain warpgroup holds 128 accumulator values at a time   (128*72 + 256*120 + 128*200 = 65536)
// tensor-memory columns: dK 0..127, dV 128..255, the parts of K 256..383 (for each k-step of 16 head-dimension elements, 8 columns
// of hi parts then 8 of lo parts, two halfs per column), then per buffer e: S^T at 384 + 64 e (32 columns, one per query), dP^T 32
// further.  The FP16 parts of P^T and dS^T replace them in place: for each k-step of 16 queries, 8 columns of hi parts then 8 of lo parts.
// 64-wide heads: dK 0..63, dV 64..127, K 128..191, the score buffers 192..319, and there is room for the parts of V, 320..383, and for a second
// set of accumulators, 384..511.

__device__ __forceinline__ void ab_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr));
}
#define AB_REGS16(r) "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), \
                     "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
__device__ __forceinline__ void ab_ld_wait2(uint32_t (&a)[16], uint32_t (&b)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" : AB_REGS16(a), AB_REGS16(b) :: "memory");
}
__device__ __forceinline__ void ab_red4(float* p, float a, float b, float c, float d) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}
__device__ __forceinline__ void ab_sts4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
// tile in shared memory -> global memory through a tensor map, as a store or as an FP32 addition; completion by bulk group
__device__ __forceinline__ void ab_tma_store(const CUtensorMap* map, uint32_t src, int c0, int c1) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(map), "r"(c0), "r"(c1), "r"(src) : "memory");
}
__device__ __forceinline__ void ab_tma_add(const CUtensorMap* map, uint32_t src, int c0, int c1) {
    asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.tile.bulk_group [%0, {%1, %2}], [%3];" ::"l"(map), "r"(c0), "r"(c1), "r"(src) : "memory");
}
__device__ __forceinline__ void ab_bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
#define AB_BULK_COMMIT() asm volatile("cp.async.bulk.commit_group;" ::: "memory")
#define AB_BULK_WAIT_READ(n) asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(n) : "memory")
#define AB_BULK_WAIT(n) asm volatile("cp.async.bulk.wait_group %0;" ::"n"(n) : "memory")
#define AB_FENCE_ASYNC() asm volatile("fence.proxy.async.shared::cta;" ::: "memory")

template <int HD>
__global__ void __launch_bounds__(AB_THREADS, 1)
at_dkv_bwd_kernel(const __grid_constant__ CUtensorMap mQ1, const __grid_constant__ CUtensorMap mQ2,
                  const __grid_constant__ CUtensorMap mD1, const __grid_constant__ CUtensorMap mD2,
                  const __grid_constant__ CUtensorMap mK1, const __grid_constant__ CUtensorMap mK2,
                  const __grid_constant__ CUtensorMap mV1, const __grid_constant__ CUtensorMap mV2,
                  const __grid_constant__ CUtensorMap mS1, const __grid_constant__ CUtensorMap mS2,
                  const __grid_constant__ CUtensorMap mdK, const __grid_constant__ CUtensorMap mdV,
                  const float* __restrict__ LT, const float* __restrict__ DT,
                  __half* __restrict__ dS1, __half* __restrict__ dS2, float* __restrict__ dK, float* __restrict__ dV,
                  const float* __restrict__ amax_q, const float* __restrict__ amax_k, const float* __restrict__ amax_v,
                  const float* __restrict__ amax_do, const float* __restrict__ ds_bound,
                  const AfSeqTab seqs, int Sp, int Hq, int g, int nkb, int chunk, int accumulate, int upper, float scale, int* status,
                  unsigned* amax_dk, unsigned* amax_dv) {
    constexpr int NH = HD / 64;
    constexpr int KV_PART = NH * 16384, ST_PART = NH * 4096;
    constexpr int COL_DK = 0, COL_DV = HD, COL_K = 2 * HD, COL_S0 = 3 * HD, COL_V = COL_S0 + 128;
    constexpr bool V_TMEM = HD == 64;                  // the parts of V sit in tensor memory too
    constexpr int DRAIN = AB_DRAIN(NH);
    constexpr bool REG_ACC = HD == 64;                 // chains are added up in the drain warps' registers, two sets of accumulators
    constexpr int COL_ACC2 = 384;                      // the second set, relative to COL_DK / COL_DV
    // which (key block, sequence, K/V head).  Key blocks from the start of the sequences have the most queries, so the launch runs
    // in up to four phases over ranges of key blocks, the longest first, and ends on CTAs of a few steps that fill the last wave.
    // Inside a phase the (sequence, head) pairs are taken `chunk` at a time, so that the Q and dO parts the CTAs in flight read
    // again and again (once per key block) stay in L2.
    const int Hkv = Hq / g;
    const int pairs = seqs.n * Hkv;
    const int nph = min(4, nkb);
    int bid = (int)blockIdx.x, ph = 0;
    while (ph + 1 < nph && bid >= pairs * ((ph + 1) * nkb / nph - ph * nkb / nph)) { bid -= pairs * ((ph + 1) * nkb / nph - ph * nkb / nph); ph++; }
    const int kb_lo = ph * nkb / nph, nk = (ph + 1) * nkb / nph - kb_lo;
    const int ci = bid / (chunk * nk);
    const int in_chunk = min(chunk, pairs - ci * chunk);
    const int cr = bid - ci * chunk * nk;
    const int kb = kb_lo + cr / in_chunk;
    const int rem = ci * chunk + cr % in_chunk;
    const int b = rem / Hkv, kvh = rem % Hkv;
    const int k0 = kb * AB_BK;
    int t0, S;
    auto take = [&]() -> bool {                        // false: no keys for this CTA
        sb_pdl_enter();
        t0 = (int)seqs.start[b]; S = (int)seqs.start[b + 1] - t0;
        const bool gave_up = __syncthreads_or(*(volatile int*)status != 0);      // an earlier CTA did (it may do so while this one reads: all threads decide alike)
        return kb < nkb && k0 < S && !gave_up;
    };
    const bool first = gridDim.x > AF_ONE_WAVE;
    if (first && !take()) return;
    const int kvd = Hkv * HD;

    extern __shared__ uint8_t af_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)af_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = (uint64_t*)(smem + AB_OFF_BAR(NH));
    uint64_t* kv_full = bars;                          // 1: V in shared memory
    uint64_t* full = bars + 1;                         // AB_STAGES
    uint64_t* empty = full + AB_STAGES;                // AB_STAGES
    uint64_t* sdp_full = empty + AB_STAGES;            // 2
    uint64_t* p_full = sdp_full + 2;                   // 2
    uint64_t* acc_ready = p_full + 2;                  // 2 (128-wide heads use one)
    uint64_t* acc_free = acc_ready + 2;                // 2
    uint64_t* k_ready = acc_free + 2;                  // 1: K in tensor memory
    uint64_t* k_full = k_ready + 1;                    // 1: K in shared memory, on its way there
    uint64_t* ew_sync = k_full + 1;                    // 1: the elementwise warps have staged their rows of a step's dS^T tiles
    uint32_t* tmem_slot = (uint32_t*)(ew_sync + 1);
    float* rows_s = (float*)(smem + AB_OFF_BAR(NH) + 256);      // per stage the log-sum-exp and D of its 32 queries

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        mbar_init(kv_full, 1); mbar_init(k_ready, 8); mbar_init(k_full, 1); mbar_init(ew_sync, 8);
        for (int i = 0; i < AB_STAGES; i++) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
        for (int i = 0; i < 2; i++) { mbar_init(&sdp_full[i], 1); mbar_init(&p_full[i], 8); mbar_init(&acc_ready[i], 1); mbar_init(&acc_free[i], 4); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    if (!first && !take()) {
        if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512));
        return;
    }
    bool ok = true;
    const int nq = (S + AB_BQ - 1) / AB_BQ, j0 = k0 / AB_BQ, per_head = nq - j0;
    const int nsteps = g * per_head;
    const int nchains = (nsteps + DRAIN - 1) / DRAIN;

    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(AB_REGS_LIGHT));
        if (warp == 0) {
            // ---------------- TMA producer ----------------
            if (elect_one()) {
                mbar_expect_tx(k_full, AB_KV_BYTES(NH));
                for (int p = 0; p < NH; p++) {
                    af_tma_2d(smem + AB_OFF_EWS(NH) + p * 16384, &mK1, k_full, kvh * HD + p * 64, t0 + k0);
                    af_tma_2d(smem + AB_OFF_EWS(NH) + KV_PART + p * 16384, &mK2, k_full, kvh * HD + p * 64, t0 + k0);
                }
                mbar_expect_tx(kv_full, AB_KV_BYTES(NH));
                for (int p = 0; p < NH; p++) {
                    af_tma_2d(smem + p * 16384, &mV1, kv_full, kvh * HD + p * 64, t0 + k0);
                    af_tma_2d(smem + KV_PART + p * 16384, &mV2, kv_full, kvh * HD + p * 64, t0 + k0);
                }
                const int slot0 = af_slot_row(Hq, b, kvh * g, t0, S), slot_rows = (S + 127) & ~127;
                for (int t = 0; t < nsteps && ok; t++) {
                    const int s = t % AB_STAGES, u = t / AB_STAGES;
                    const int h = kvh * g + t / per_head, j = j0 + t % per_head;
                    ok = mbar_wait(&empty[s], (u & 1) ^ 1);
                    if (!ok) break;
                    uint8_t* st = smem + AB_KV_BYTES(NH) + s * AB_STAGE_BYTES(NH);
                    mbar_expect_tx(&full[s], AB_STAGE_BYTES(NH) + 256);
                    const size_t row = (size_t)(slot0 + t / per_head * slot_rows) + j * AB_BQ;
                    ab_bulk_load(rows_s + s * 64, LT + row, 128, &full[s]);
                    ab_bulk_load(rows_s + s * 64 + 32, DT + row, 128, &full[s]);
                    for (int p = 0; p < NH; p++) {
                        af_tma_2d(st + p * 4096, &mQ1, &full[s], h * HD + p * 64, t0 + j * AB_BQ);
                        af_tma_2d(st + ST_PART + p * 4096, &mQ2, &full[s], h * HD + p * 64, t0 + j * AB_BQ);
                        af_tma_2d(st + 2 * ST_PART + p * 4096, &mD1, &full[s], h * HD + p * 64, t0 + j * AB_BQ);
                        af_tma_2d(st + 3 * ST_PART + p * 4096, &mD2, &full[s], h * HD + p * 64, t0 + j * AB_BQ);
                    }
                }
                if (!ok) atomicExch(status, SB_ERR_TIMEOUT);
            }
        } else if (warp == 1) {
            // ---------------- MMA issuer ----------------
            if (elect_one()) {
                const uint32_t idesc_s = (1u << 4) | ((uint32_t)(AB_BQ >> 3) << 17) | ((uint32_t)(AB_BK >> 4) << 24);
                const uint32_t idesc_o = (1u << 4) | (1u << 16) | ((uint32_t)(HD >> 3) << 17) | ((uint32_t)(AB_BK >> 4) << 24);
                const uint32_t sv = smem_u32(smem), tk = tmem_base + COL_K;
                ok = mbar_wait(k_ready, 0) && (V_TMEM || mbar_wait(kv_full, 0));
                for (int t = 0; t <= nsteps && ok; t++) {
                    if (t < nsteps) {
                        // S^T and dP^T of step t into buffer t & 1 (its parts of step t - 2 were consumed by instructions issued before these)
                        const int s = t % AB_STAGES, e = t & 1;
                        ok = mbar_wait(&full[s], (t / AB_STAGES) & 1);
                        if (!ok) break;
                        tc_fence_after();
                        const uint32_t st = smem_u32(smem + AB_KV_BYTES(NH) + s * AB_STAGE_BYTES(NH));
                        {                                          // S^T: K parts from tensor memory
                            const uint32_t d = tmem_base + (uint32_t)COL_S0 + 64 * e;
#pragma unroll
                            for (int p = 0; p < NH; p++) {
                                const uint64_t b1 = make_kmajor_desc<128>(st + p * 4096), b2 = make_kmajor_desc<128>(st + ST_PART + p * 4096);
#pragma unroll
                                for (int kk = 0; kk < 4; kk++) {
                                    const uint64_t adv = (uint64_t)(kk * 2);
                                    const uint32_t ta = tk + (uint32_t)((p * 4 + kk) * 16);
                                    af_mma_ts(d, ta, b1 + adv, idesc_s, (p | kk) ? 1u : 0u);
                                    af_mma_ts(d, ta + 8, b1 + adv, idesc_s, 1);
                                    af_mma_ts(d, ta, b2 + adv, idesc_s, 1);
                                }
                            }
                        }
                        {                                          // dP^T: V parts from shared memory (64-wide heads: tensor memory)
                            const uint32_t sb = st + 2 * ST_PART;
                            const uint32_t d = tmem_base + (uint32_t)COL_S0 + 64 * e + 32;
#pragma unroll
                            for (int p = 0; p < NH; p++) {
                                const uint64_t a1 = make_kmajor_desc<128>(sv + p * 16384), a2 = make_kmajor_desc<128>(sv + KV_PART + p * 16384);
                                const uint64_t b1 = make_kmajor_desc<128>(sb + p * 4096), b2 = make_kmajor_desc<128>(sb + ST_PART + p * 4096);
#pragma unroll
                                for (int kk = 0; kk < 4; kk++) {
                                    const uint64_t adv = (uint64_t)(kk * 2);
                                    if constexpr (V_TMEM) {
                                        const uint32_t ta = tmem_base + (uint32_t)(COL_V + kk * 16);
                                        af_mma_ts(d, ta, b1 + adv, idesc_s, kk ? 1u : 0u);
                                        af_mma_ts(d, ta + 8, b1 + adv, idesc_s, 1);
                                        af_mma_ts(d, ta, b2 + adv, idesc_s, 1);
                                    } else {
                                        af_mma_f16_two(d, a1 + adv, b1 + adv, b2 + adv, idesc_s, (p | kk) ? 1u : 0u);
                                        af_mma_f16(d, a2 + adv, b1 + adv, idesc_s, 1);
                                    }
                                }
                            }
                        }
                        tc_commit(&sdp_full[e]);
                    }
                    if (t >= 1) {
                        // dV += P^T dO and dK += dS^T Q of step t - 1
                        const int u = t - 1, e = u & 1, s = u % AB_STAGES;
                        ok = mbar_wait(&p_full[e], (u >> 1) & 1);
                        if (!ok) break;
                        const bool first = (u % DRAIN) == 0;
                        const int ch = u / DRAIN, as = REG_ACC ? ch & 1 : 0, au = REG_ACC ? ch >> 1 : ch;      // chain, its accumulators, how often they were used before
                        if (first && au > 0) {                       // the drain warps have read the chain before out of them
                            ok = mbar_wait(&acc_free[as], (au - 1) & 1);
                            if (!ok) break;
                        }
                        tc_fence_after();
                        const uint32_t st = smem_u32(smem + AB_KV_BYTES(NH) + s * AB_STAGE_BYTES(NH));
#pragma unroll
                        for (int prod = 0; prod < 2; prod++) {
                            const uint32_t ta = tmem_base + (uint32_t)(prod ? COL_S0 + 64 * e + 32 : COL_S0 + 64 * e);      // per k-step of 16 queries: hi part 8 columns, lo part the next 8
                            const uint32_t sb = st + (prod ? 0 : 2 * ST_PART);                                       // dK takes Q, dV takes dO
                            const uint64_t b1 = make_mn16_desc<AB_BQ>(sb), b2 = make_mn16_desc<AB_BQ>(sb + ST_PART);
                            const uint32_t d = tmem_base + (uint32_t)((prod ? COL_DK : COL_DV) + (REG_ACC ? as * COL_ACC2 : 0));
#pragma unroll
                            for (int kk = 0; kk < 2; kk++) {
                                const uint64_t advb = (uint64_t)(kk * 128);
                                af_mma_ts(d, ta + kk * 16, b1 + advb, idesc_o, (first && kk == 0) ? 0u : 1u);
                                af_mma_ts(d, ta + kk * 16 + 8, b1 + advb, idesc_o, 1);
                                af_mma_ts(d, ta + kk * 16, b2 + advb, idesc_o, 1);
                            }
                        }
                        tc_commit(&empty[s]);
                        if (((u + 1) % DRAIN) == 0 || u == nsteps - 1) tc_commit(&acc_ready[as]);
                    }
                }
                if (!ok) atomicExch(status, SB_ERR_TIMEOUT);
            }
        }
    } else if (warp >= 12) {
        // ---------------- drain: dK and dV chains out of tensor memory, added into the output ----------------
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(AB_REGS_DRAIN));
        {
            const int q = warp & 3, r = q * 32 + lane, kg = k0 + r;
            const bool live = kg < S;
            // dV accumulates (P 2^14) (dO 2^s_do), dK accumulates (dS 2^s_ds) (Q 2^s_q)
            const float fv = tc_pow2(-14) * tc_pow2(-tc_f16_shift(sb_word(amax_do)));
            const float fk = tc_pow2(-tc_f16_shift(sb_word(ds_bound))) * tc_pow2(-tc_f16_shift(sb_word(amax_q)));
            float* rowk = dK + (size_t)(t0 + (live ? kg : 0)) * kvd + (size_t)kvh * HD;
            float* rowv = dV + (size_t)(t0 + (live ? kg : 0)) * kvd + (size_t)kvh * HD;
            const uint32_t ta = tmem_base + ((uint32_t)(q * 32) << 16);
            const bool whole = k0 + AB_BK <= S;                // all 128 keys belong to this sequence: tiles through the TMA unit
            ok = mbar_wait(k_ready, 0);                         // the staging area held the parts of K until now
            const uint32_t stg = smem_u32(smem + AB_OFF_DRS(NH) + q * 8192);
            const int row0 = t0 + k0 + q * 32, col0 = kvh * HD;
            int pieces = 0;                                     // tiles this warp has handed to the TMA unit
            // one row of dK (which = 0) or dV, scaled, to memory: stored (`first`: nothing has to zero the output before) or added
            auto emit = [&](int which, bool first, uint32_t (&v0)[32], uint32_t (&v1)[32], uint32_t (&v2)[32], uint32_t (&v3)[32]) {
                const float f = which ? fv : fk;
                if (whole) {
                    auto piece = [&](uint32_t (&v)[32], int pc) {
                        const uint32_t buf = stg + (uint32_t)((pieces & 1) * 4096);
                        if (pieces >= 2) { if (lane == 0) AB_BULK_WAIT_READ(1); __syncwarp(); }     // the tile staged here two pieces ago has been read
#pragma unroll
                        for (int i = 0; i < 8; i++)
                            ab_sts4(buf + (uint32_t)(lane * 128 + ((i ^ (lane & 7)) << 4)),
                                    __float_as_uint(__uint_as_float(v[4 * i]) * f), __float_as_uint(__uint_as_float(v[4 * i + 1]) * f),
                                    __float_as_uint(__uint_as_float(v[4 * i + 2]) * f), __float_as_uint(__uint_as_float(v[4 * i + 3]) * f));
                        AB_FENCE_ASYNC();
                        __syncwarp();
                        if (lane == 0) {
                            if (first) ab_tma_store(which ? &mdV : &mdK, buf, col0 + pc * 32, row0);
                            else ab_tma_add(which ? &mdV : &mdK, buf, col0 + pc * 32, row0);
                            AB_BULK_COMMIT();
                        }
                        pieces++;
                    };
                    piece(v0, 0); piece(v1, 1);
                    if constexpr (NH == 2) { piece(v2, 2); piece(v3, 3); }
                } else if (live) {
                    float* dst = which ? rowv : rowk;
                    auto piece = [&](uint32_t (&v)[32], int pc) {
#pragma unroll
                        for (int i = 0; i < 8; i++) {
                            const float x0 = __uint_as_float(v[4 * i]) * f, x1 = __uint_as_float(v[4 * i + 1]) * f,
                                        x2 = __uint_as_float(v[4 * i + 2]) * f, x3 = __uint_as_float(v[4 * i + 3]) * f;
                            if (first) *(float4*)(dst + pc * 32 + 4 * i) = make_float4(x0, x1, x2, x3);
                            else ab_red4(dst + pc * 32 + 4 * i, x0, x1, x2, x3);
                        }
                    };
                    piece(v0, 0); piece(v1, 1);
                    if constexpr (NH == 2) { piece(v2, 2); piece(v3, 3); }
                }
            };
            if constexpr (REG_ACC) {
                uint32_t a0[32], a1[32], a2[32], a3[32];           // running sums (floats): dK columns 0..31, 32..63, dV columns 0..31, 32..63
#pragma unroll
                for (int i = 0; i < 32; i++) a0[i] = a1[i] = a2[i] = a3[i] = 0u;
                auto add = [&](uint32_t (&s)[32], uint32_t (&v)[32]) {
#pragma unroll
                    for (int i = 0; i < 32; i++) s[i] = __float_as_uint(__uint_as_float(s[i]) + __uint_as_float(v[i]));
                };
                for (int c = 0; c < nchains && ok; c++) {
                    const int as = c & 1;
                    ok = mbar_wait(&acc_ready[as], (c >> 1) & 1);
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t tb = ta + (uint32_t)(as * COL_ACC2);
                    uint32_t v[32];
                    af_ld32_issue(tb + COL_DK, v); af_ld_wait(v); add(a0, v);
                    af_ld32_issue(tb + COL_DK + 32, v); af_ld_wait(v); add(a1, v);
                    af_ld32_issue(tb + COL_DV, v); af_ld_wait(v); add(a2, v);
                    af_ld32_issue(tb + COL_DV + 32, v); af_ld_wait(v);
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) af_arrive(&acc_free[as]);
                    add(a3, v);
                }
                if (ok) { emit(0, !accumulate, a0, a1, a0, a1); emit(1, !accumulate, a2, a3, a2, a3); }
                if (amax_dk && amax_dv) {
                    float mk = 0.f, mv = 0.f;
#pragma unroll
                    for (int i = 0; i < 32; i++) {
                        mk = fmaxf(mk, fmaxf(fabsf(__uint_as_float(a0[i])), fabsf(__uint_as_float(a1[i]))));
                        mv = fmaxf(mv, fmaxf(fabsf(__uint_as_float(a2[i])), fabsf(__uint_as_float(a3[i]))));
                    }
                    mk = live ? mk * fk : 0.f; mv = live ? mv * fv : 0.f;
                    for (int d = 16; d > 0; d >>= 1) { mk = fmaxf(mk, __shfl_xor_sync(0xffffffffu, mk, d)); mv = fmaxf(mv, __shfl_xor_sync(0xffffffffu, mv, d)); }
                    if (lane == 0 && mk > 0.f) atomicMax(amax_dk, __float_as_uint(mk));
                    if (lane == 0 && mv > 0.f) atomicMax(amax_dv, __float_as_uint(mv));
                }
            } else {
                for (int c = 0; c < nchains && ok; c++) {
                    ok = mbar_wait(acc_ready, c & 1);
                    if (!ok) break;
                    tc_fence_after();
                    if (whole && c > 0) {                       // the previous chain's additions have been performed: one order per element
                        if (lane == 0) AB_BULK_WAIT(0);
                        __syncwarp();
                    }
#pragma unroll
                    for (int which = 0; which < 2; which++) {   // dK, then dV: all loads of one in flight, one wait
                        uint32_t v0[32], v1[32], v2[32], v3[32];
                        af_ld32_issue(ta + (uint32_t)(which * HD), v0);
                        af_ld32_issue(ta + (uint32_t)(which * HD + 32), v1);
                        af_ld32_issue(ta + (uint32_t)(which * HD + 64), v2);
                        af_ld32_issue(ta + (uint32_t)(which * HD + 96), v3);
                        af_ld_wait(v0); af_ld_dep(v1); af_ld_dep(v2); af_ld_dep(v3);
                        if (which == 1) {                       // everything is in registers: the next chain may overwrite the accumulators
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) af_arrive(acc_free);
                        }
                        emit(which, c == 0 && !accumulate, v0, v1, v2, v3);
                    }
                }
            }
            if (lane == 0) AB_BULK_WAIT_READ(0);               // the staging buffers are read out before the CTA gives its shared memory back
            if (!ok && lane == 0) atomicExch(status, SB_ERR_TIMEOUT);
        }
    } else {
        // ---------------- elementwise: one key row and 16 of the step's 32 queries per thread (warps 4-7: queries 0..15, 8-11: 16..31) ----------------
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(AB_REGS_EW));
        const int ch = (warp - 4) >> 2, q = warp & 3, r = q * 32 + lane, kg = k0 + r;
        const float cs = tc_pow2(-tc_f16_shift(sb_word(amax_q))) * tc_pow2(-tc_f16_shift(sb_word(amax_k))) * (HD == 64 ? scale : scale * 1.4426950408889634f);
        const float cp = tc_pow2(-tc_f16_shift(sb_word(amax_do))) * tc_pow2(-tc_f16_shift(sb_word(amax_v)));
        const float cpd = cp * (tc_pow2(tc_f16_shift(sb_word(ds_bound))) * scale * (1.0f / 16384.f));      // p holds P * 2^14
        const uint32_t lane_addr = (uint32_t)(q * 32) << 16;
        // This key row's parts of K from shared memory (128-byte-swizzled tiles: hi and lo part of each half of the head
        // dimension) into tensor memory: head-dimension k-steps ch*4 .. ch*4+3 are half `ch`, two consecutive halfs per column.
        // 64-wide heads have one half: warps with ch = 1 bring the parts of V in the same way.
        ok = mbar_wait(V_TMEM && ch == 1 ? kv_full : k_full, 0);
        {
            const uint32_t kt = smem_u32(smem + (V_TMEM && ch == 1 ? 0 : AB_OFF_EWS(NH) + (V_TMEM ? 0 : ch * 16384))) + (uint32_t)(r * 128);
            const uint32_t kcol = tmem_base + lane_addr + (uint32_t)(V_TMEM ? (ch ? COL_V : COL_K) : COL_K + ch * 64);
#pragma unroll
            for (int kk = 0; kk < 4; kk++) {
                uint32_t h8[8], l8[8];
                const uint32_t c0 = (uint32_t)(((2 * kk) ^ (r & 7)) << 4), c1 = (uint32_t)(((2 * kk + 1) ^ (r & 7)) << 4);
                asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(h8[0]), "=r"(h8[1]), "=r"(h8[2]), "=r"(h8[3]) : "r"(kt + c0) : "memory");
                asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(h8[4]), "=r"(h8[5]), "=r"(h8[6]), "=r"(h8[7]) : "r"(kt + c1) : "memory");
                asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(l8[0]), "=r"(l8[1]), "=r"(l8[2]), "=r"(l8[3]) : "r"(kt + KV_PART + c0) : "memory");
                asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(l8[4]), "=r"(l8[5]), "=r"(l8[6]), "=r"(l8[7]) : "r"(kt + KV_PART + c1) : "memory");
                af_st8(kcol + (uint32_t)(kk * 16), h8);
                af_st8(kcol + (uint32_t)(kk * 16 + 8), l8);
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane == 0) af_arrive(k_ready);
        }
        ok = ok && mbar_wait(k_ready, 0);                       // every warp has its rows of K out of the staging area
        const int slot0 = af_slot_row(Hq, b, kvh * g, t0, S), slot_rows = (S + 127) & ~127;      // this K/V head's slots
        const uint32_t ews = smem_u32(smem + AB_OFF_EWS(NH));
        const bool issuer = warp == 4 && lane == 0;            // hands the staged tiles to the TMA unit
        // Columns before this key block that the dQ product reads together with it (its query tiles are 256 wide): zeros, stored
        // from a tile of zeros that sits where the second step will stage its hi parts
        // ew_sync counts one phase per hand-over: a warp arrives when its rows are staged; the issuing thread waits for all eight, and
        // before it arrives it makes sure that everything it handed over earlier has been read.  So a completed phase n tells every
        // warp that the tiles handed over in phases < n are read out: a buffer is written again one phase after the next.
        int sync_n = 0;
        if (upper && (k0 & 255) != 0 && ok) {
            ab_sts4(ews + 16384 + (uint32_t)((warp - 4) * 1024 + lane * 32), 0, 0, 0, 0);
            ab_sts4(ews + 16384 + (uint32_t)((warp - 4) * 1024 + lane * 32 + 16), 0, 0, 0, 0);
            AB_FENCE_ASYNC();
            __syncwarp();
            if (lane == 0) af_arrive(ew_sync);
            if (warp == 4) {
                ok = mbar_wait(ew_sync, 0);
                if (issuer && ok) {
                    for (int hi = 0; hi < g; hi++) {
                        const int y = slot0 + hi * slot_rows + k0;
                        for (int i = 0; i < 4; i++) { ab_tma_store(&mS1, ews + 16384, k0 - 128 + i * 32, y); ab_tma_store(&mS2, ews + 16384, k0 - 128 + i * 32, y); }
                    }
                    AB_BULK_COMMIT();
                }
            }
            sync_n = 1;
        }
        int hi = 0, j = j0;                                     // query head within the group, query block
        for (int t = 0; t < nsteps && ok; t++) {
            const int e = t & 1;
            const int q0 = j * AB_BQ;
            ok = mbar_wait(&sdp_full[e], (t >> 1) & 1) && mbar_wait(&full[t % AB_STAGES], (t / AB_STAGES) & 1);
            if (!ok) break;
            tc_fence_after();
            const int hb = slot0 + hi * slot_rows;
            uint32_t sr[16], dr[16];
            ab_ld16(tmem_base + lane_addr + (uint32_t)(COL_S0 + 64 * e + ch * 16), sr);
            ab_ld16(tmem_base + lane_addr + (uint32_t)(COL_S0 + 64 * e + 32 + ch * 16), dr);
            // log-sum-exp (times log2 e) and D of this warp's 16 queries, which came with the step's tiles: the same addresses for every lane (from global memory
            // they were late by most of a step's 1400 cycles of arithmetic)
            float4 L4[4], D4[4];
            {
                const float4* lp = (const float4*)(rows_s + t % AB_STAGES * 64 + ch * 16);
#pragma unroll
                for (int i = 0; i < 4; i++) { L4[i] = lp[i]; D4[i] = lp[8 + i]; }
            }
            ab_ld_wait2(sr, dr);
            uint32_t p1[8], p2[8], d1[8], d2[8];
            // away from the diagonal and from the sequence's end no element of the step is masked
            const bool nomask = q0 >= k0 + AB_BK && q0 + AB_BQ <= S && k0 + AB_BK <= S;
            auto columns = [&](auto masked) {
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    float pv[2], dv[2];
#pragma unroll
                    for (int w = 0; w < 2; w++) {
                        const int c = 2 * i + w;
                        const float4 l4 = L4[c >> 2], dq4 = D4[c >> 2];
                        const float Lq = (c & 3) == 0 ? l4.x : (c & 3) == 1 ? l4.y : (c & 3) == 2 ? l4.z : l4.w;      // 14 - lse log2 e (64-wide heads: - lse)
                        const float Dq = (c & 3) == 0 ? dq4.x : (c & 3) == 1 ? dq4.y : (c & 3) == 2 ? dq4.z : dq4.w;  // D dsc
                        const int qi = q0 + ch * 16 + c;
                        const bool valid = !decltype(masked)::value || (kg <= qi && qi < S && kg < S);
                        const float y = fmaf(__uint_as_float(sr[c]), cs, Lq);
                        pv[w] = valid ? (HD == 64 ? af_ex2(y * 1.4426950408889634f) * 16384.f : af_ex2(y)) : 0.f;      // P * 2^14
                        dv[w] = pv[w] * fmaf(__uint_as_float(dr[c]), cpd, -Dq);
                    }
                    af_split2(pv[0], pv[1], p1[i], p2[i]);
                    af_split2(dv[0], dv[1], d1[i], d2[i]);
                }
            };
            if (nomask) columns(std::false_type{}); else columns(std::true_type{});
            // The parts of these 16 queries go back over the 16 columns their scores came from (all of them are in registers by now):
            // hi part in the first 8 columns, lo part in the next 8, which is where the MMA issuer looks for k-step `ch`.
            af_st8(tmem_base + lane_addr + (uint32_t)(COL_S0 + 64 * e + ch * 16), p1);
            af_st8(tmem_base + lane_addr + (uint32_t)(COL_S0 + 64 * e + ch * 16 + 8), p2);
            af_st8(tmem_base + lane_addr + (uint32_t)(COL_S0 + 64 * e + 32 + ch * 16), d1);
            af_st8(tmem_base + lane_addr + (uint32_t)(COL_S0 + 64 * e + 32 + ch * 16 + 8), d2);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane == 0) af_arrive(&p_full[e]);
            // dS^T parts of this key row, 16 queries = 32 bytes per part, into the step's two tiles (64-byte rows).  The issuing thread
            // first makes sure that everything it handed over earlier has been read (the other buffer is written in the next step),
            // then all eight warps meet and it hands this step's tiles to the TMA unit.
            {
                const uint32_t buf = ews + (uint32_t)(e * 16384);
                const uint32_t row = buf + (uint32_t)(r * 64), x0 = (uint32_t)((2 * ch) ^ ((r >> 1) & 3)) << 4, x1 = x0 ^ 16;      // 64-byte swizzle: without it four lanes of eight met in a bank
                if (warp != 4 && sync_n > 0) {                  // (the issuer's warp waited for this phase when it handed the tiles over)
                    ok = mbar_wait(ew_sync, (sync_n - 1) & 1);
                    if (!ok) break;
                }
                ab_sts4(row + x0, d1[0], d1[1], d1[2], d1[3]); ab_sts4(row + x1, d1[4], d1[5], d1[6], d1[7]);
                ab_sts4(row + 8192 + x0, d2[0], d2[1], d2[2], d2[3]); ab_sts4(row + 8192 + x1, d2[4], d2[5], d2[6], d2[7]);
                AB_FENCE_ASYNC();
                __syncwarp();
                if (issuer) AB_BULK_WAIT_READ(0);
                if (lane == 0) af_arrive(ew_sync);
                if (warp == 4) {
                    ok = mbar_wait(ew_sync, sync_n & 1);
                    if (!ok) break;
                    if (issuer) {
                        const int y = hb + k0;
                        ab_tma_store(&mS1, buf, q0, y); ab_tma_store(&mS2, buf + 8192, q0, y);
                        AB_BULK_COMMIT();
                    }
                }
                sync_n++;
            }
            if (++j == nq) { j = j0; hi++; }
        }
        if (issuer) AB_BULK_WAIT_READ(0);                      // the staging tiles are read out before the CTA gives its shared memory back
        if (!ok && lane == 0) atomicExch(status, SB_ERR_TIMEOUT);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512));
    }
}

// ---------------------------------------------------------------------------------------------------------------
// dQ = dS K.  One CTA owns 128 queries of one (sequence, query head) and walks over the keys up to the diagonal in blocks of 64:
// dS^T parts ([key][query], read MN-major as the 128-row A operand) and K parts (MN-major B operand) through a ring of stages, twelve
// MMAs per block into one of two tensor-memory accumulators, which eight warps add into registers (round-to-nearest FP32).  All
// sequences and heads in one launch, longest query blocks first.  32 rows of a sequence leave through tensor stores, staged where the ring was
// (a thread's own stores touch 32 lines an instruction).  Bound by the bytes of dS and K that an SM takes in.
#define AQ_THREADS 320
// 64-wide heads, more CTAs than SMs: two stages, so that two CTAs share an SM and one loads and starts while the other ends (24 sequences of 383
// tokens, 8 heads: backward call 155 -> 146 us, 8 x 2048: 517 -> 500).  A grid of one wave keeps three: launched early, beside what still runs,
// small CTAs would share an SM while others idle (8 x 256: 47 -> 49 us).
#define AQ_STAGES(NH, GRID) ((NH) == 1 && (GRID) > AF_ONE_WAVE ? 2 : 3)
#define AQ_A_BYTES 32768                                // dS^T: 2 parts x 64 keys x 128 queries
#define AQ_STAGE_BYTES(NH) (AQ_A_BYTES + (NH) * 16384)  // and K: 2 parts x 64 keys x head size
#define AQ_SMEM(NH, STAGES) ((STAGES) * AQ_STAGE_BYTES(NH) + 1024 + 256)

template <int HD>
__global__ void __launch_bounds__(AQ_THREADS, HD == 64 ? 2 : 1)
at_dq_bwd_kernel(const __grid_constant__ CUtensorMap mS1, const __grid_constant__ CUtensorMap mS2,
                 const __grid_constant__ CUtensorMap mK1, const __grid_constant__ CUtensorMap mK2, const __grid_constant__ CUtensorMap mdQ,
                 const AfSeqTab seqs, float* __restrict__ dQ, const float* __restrict__ ds_bound, const float* __restrict__ amax_k,
                 int Sp, int Hq, int g, int nqb_max, int* status, unsigned* amax_dq) {
    constexpr int NH = HD / 64, OC = HD / 2;
    const int stages = AQ_STAGES(NH, gridDim.x);
    const int per_i = seqs.n * Hq;
    const int qb = nqb_max - 1 - (int)blockIdx.x / per_i;
    const int rem = (int)blockIdx.x % per_i;
    const int b = rem / Hq, h = rem % Hq;
    int t0, S, nkv;
    auto take = [&]() -> bool {                         // false: no rows for this CTA
        sb_pdl_enter();
        t0 = (int)seqs.start[b]; S = (int)seqs.start[b + 1] - t0;
        nkv = min((S + 63) / 64, 2 * qb + 2);
        const bool gave_up = __syncthreads_or(*(volatile int*)status != 0);      // as above
        return qb * 128 < S && !gave_up;
    };
    const bool first = gridDim.x > AF_ONE_WAVE;
    if (first && !take()) return;

    extern __shared__ uint8_t af_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)af_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* full = (uint64_t*)(smem + stages * AQ_STAGE_BYTES(NH));
    uint64_t* empty = full + stages;
    uint64_t* acc_full = empty + stages;             // 2
    uint64_t* acc_empty = acc_full + 2;                 // 2
    uint32_t* tmem_slot = (uint32_t*)(acc_empty + 2);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int i = 0; i < stages; i++) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
        for (int i = 0; i < 2; i++) { mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], 8); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(2 * HD));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    if (!first && !take()) {
        if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(2 * HD));
        return;
    }
    bool ok = true;
    if (warp == 0) {
        // ---------------- TMA producer ----------------
        if (elect_one()) {
            const int y0 = af_slot_row(Hq, b, h, t0, S);
            for (int j = 0, s = 0, turn = 0; j < nkv && ok; j++, s = s + 1 < stages ? s + 1 : 0, turn += s == 0) {
                ok = mbar_wait(&empty[s], (turn & 1) ^ 1);
                if (!ok) break;
                uint8_t* st = smem + s * AQ_STAGE_BYTES(NH);
                mbar_expect_tx(&full[s], AQ_STAGE_BYTES(NH));
                for (int p = 0; p < 2; p++) {
                    af_tma_2d(st + p * 8192, &mS1, &full[s], qb * 128 + p * 64, y0 + j * 64);
                    af_tma_2d(st + 16384 + p * 8192, &mS2, &full[s], qb * 128 + p * 64, y0 + j * 64);
                }
                for (int p = 0; p < NH; p++) {
                    af_tma_2d(st + AQ_A_BYTES + p * 8192, &mK1, &full[s], (h / g) * HD + p * 64, t0 + j * 64);
                    af_tma_2d(st + AQ_A_BYTES + NH * 8192 + p * 8192, &mK2, &full[s], (h / g) * HD + p * 64, t0 + j * 64);
                }
            }
            if (!ok) atomicExch(status, SB_ERR_TIMEOUT);
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        if (elect_one()) {
            const uint32_t idesc = (1u << 4) | (1u << 15) | (1u << 16) | ((uint32_t)(HD >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
            for (int j = 0, s = 0, turn = 0; j < nkv && ok; j++, s = s + 1 < stages ? s + 1 : 0, turn += s == 0) {
                const int e = j & 1;
                ok = mbar_wait(&full[s], turn & 1) && mbar_wait(&acc_empty[e], ((j >> 1) & 1) ^ 1);
                if (!ok) break;
                tc_fence_after();
                const uint32_t st = smem_u32(smem + s * AQ_STAGE_BYTES(NH));
                const uint64_t a1 = make_mn16_desc<64>(st), a2 = make_mn16_desc<64>(st + 16384);
                const uint64_t b1 = make_mn16_desc<64>(st + AQ_A_BYTES), b2 = make_mn16_desc<64>(st + AQ_A_BYTES + NH * 8192);
                const uint32_t d = tmem_base + (uint32_t)(e * HD);
#pragma unroll
                for (int kk = 0; kk < 4; kk++) {
                    const uint64_t adv = (uint64_t)(kk * 128);
                    af_mma_f16(d, a1 + adv, b1 + adv, idesc, kk ? 1u : 0u);
                    af_mma_f16(d, a2 + adv, b1 + adv, idesc, 1);
                    af_mma_f16(d, a1 + adv, b2 + adv, idesc, 1);
                }
                tc_commit(&empty[s]);
                tc_commit(&acc_full[e]);
            }
            if (!ok) atomicExch(status, SB_ERR_TIMEOUT);
        }
    } else {
        // ---------------- accumulation: one query row and half of the columns per thread ----------------
        const int q = warp & 3, r = q * 32 + lane, ch = (warp - 2) >> 2;
        const int qi = qb * 128 + r;
        float o[OC];
#pragma unroll
        for (int i = 0; i < OC; i++) o[i] = 0.f;
        for (int j = 0; j < nkv && ok; j++) {
            const int e = j & 1;
            ok = mbar_wait(&acc_full[e], (j >> 1) & 1);
            if (!ok) break;
            tc_fence_after();
            const uint32_t ta = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(e * HD + ch * OC);
            uint32_t t[32], t2[32];
            af_ld32_issue(ta, t);
            if constexpr (OC == 64) af_ld32_issue(ta + 32, t2);
            af_ld_wait(t);
            if constexpr (OC == 64) af_ld_dep(t2);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) af_arrive(&acc_empty[e]);
#pragma unroll
            for (int i = 0; i < 32; i++) {
                o[i] += __uint_as_float(t[i]);
                if constexpr (OC == 64) o[32 + i] += __uint_as_float(t2[i]);
            }
        }
        ok = __all_sync(0xffffffffu, ok);
        float am = 0.f;
        if (ok) {
            const float f1 = tc_pow2(-tc_f16_shift(sb_word(ds_bound))), f2 = tc_pow2(-tc_f16_shift(sb_word(amax_k)));
#pragma unroll
            for (int i = 0; i < OC; i++) o[i] = o[i] * f1 * f2;
        }
        if (ok && qb * 128 + q * 32 + 32 <= S) {
            // 32 rows of the sequence: as tiles, through the ring (every load has been consumed)
#pragma unroll
            for (int c = 0; c < NH; c++) {
                const uint32_t buf = smem_u32(smem) + (uint32_t)(((warp - 2) * NH + c) * 4096);
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const float4 v = make_float4(o[c * 32 + 4 * i], o[c * 32 + 4 * i + 1], o[c * 32 + 4 * i + 2], o[c * 32 + 4 * i + 3]);
                    ab_sts4(buf + (uint32_t)(lane * 128 + ((i ^ (lane & 7)) << 4)), __float_as_uint(v.x), __float_as_uint(v.y), __float_as_uint(v.z), __float_as_uint(v.w));
                    am = sb_amax4(am, v);
                }
                AB_FENCE_ASYNC();
                __syncwarp();
                if (lane == 0) ab_tma_store(&mdQ, buf, h * HD + ch * OC + c * 32, t0 + qb * 128 + q * 32);
            }
            if (lane == 0) { AB_BULK_COMMIT(); AB_BULK_WAIT_READ(0); }
        } else if (ok && qi < S) {
            float4* dst = (float4*)(dQ + (size_t)(t0 + qi) * Hq * HD + (size_t)h * HD + ch * OC);
#pragma unroll
            for (int i = 0; i < OC / 4; i++) {
                const float4 v = make_float4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
                dst[i] = v;
                am = sb_amax4(am, v);
            }
        }
        if (amax_dq) {
            for (int d = 16; d > 0; d >>= 1) am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, d));
            if (lane == 0 && am > 0.f) atomicMax(amax_dq, __float_as_uint(am));
        }
        if (!ok && lane == 0) atomicExch(status, SB_ERR_TIMEOUT);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(2 * HD));
    }
}

template <int HD>
static int ab_launch(sb_ctx_t* c, const AbCall& p) {
    auto kern = at_dkv_bwd_kernel<HD>;
    constexpr int NH = HD / 64;
    static bool attr_done = false;
    if (!attr_done) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, AB_SMEM(NH)) != cudaSuccess ||
            cudaFuncSetAttribute(at_dq_bwd_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, AQ_SMEM(NH, 3)) != cudaSuccess) { cudaGetLastError(); return 1; }
        attr_done = true;
    }
    const AfSeqTab seqs = {c->h_seq_n, c->attn_seq_starts};
    int Smax = 0;
    for (int b = 0; b < c->h_seq_n; b++) Smax = max(Smax, c->h_seq[b + 1] - c->h_seq[b]);
    if (Smax <= 0 || Smax > p.Sp) return 1;
    const int qd = p.Hq * HD, kvd = p.Hkv * HD, nkb = (Smax + AB_BK - 1) / AB_BK, g = p.Hq / p.Hkv;
    const int upper = !p.dQ;                             // the product over tiles of 256 queries reads 128 columns left of odd key blocks: zeros
    CUtensorMap mQ1, mQ2, mD1, mD2, mK1, mK2, mV1, mV2, mS1, mS2, mdK, mdV, mdQ, mA1, mA2, mB1, mB2;
    if (!af_make_map(c, &mQ1, p.q1, p.T, qd, AB_BQ) || !af_make_map(c, &mQ2, p.q2, p.T, qd, AB_BQ) ||
        !af_make_map(c, &mD1, p.do1, p.T, qd, AB_BQ) || !af_make_map(c, &mD2, p.do2, p.T, qd, AB_BQ) ||
        !af_make_map(c, &mK1, p.k1, p.T, kvd, AB_BK) || !af_make_map(c, &mK2, p.k2, p.T, kvd, AB_BK) ||
        !af_make_map(c, &mV1, p.v1, p.T, kvd, AB_BK) || !af_make_map(c, &mV2, p.v2, p.T, kvd, AB_BK)) return 1;
    {
        // dS^T parts: [rows of the head slots: keys][Sp queries] halfs, tiles of 32 queries x 128 keys, rows of 64 bytes with the 64-byte swizzle in shared memory;
        // dK, dV: [T][kvd] floats, tiles of 32 columns x 32 keys, 128-byte swizzle
        const cuuint64_t rows = af_slot_rows(p.Hq, seqs.n, p.T);
        const cuuint64_t sd[2] = {(cuuint64_t)p.Sp, rows}, ss[1] = {(cuuint64_t)p.Sp * 2};
        const cuuint32_t sbx[2] = {32u, 128u}, abx[2] = {64u, 64u};
        const cuuint64_t gd[2] = {(cuuint64_t)kvd, (cuuint64_t)p.T}, gs[1] = {(cuuint64_t)kvd * 4};
        const cuuint32_t gbx[2] = {32u, 32u};
        const CUtensorMapL2promotion np = CU_TENSOR_MAP_L2_PROMOTION_NONE;
        if (rows > 0x7fffffffull || !tc_aligned16(p.dS1) || !tc_aligned16(p.dS2) ||
            !tc_encode(c, &mS1, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, p.dS1, sd, ss, sbx, CU_TENSOR_MAP_SWIZZLE_64B, np) ||
            !tc_encode(c, &mS2, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, p.dS2, sd, ss, sbx, CU_TENSOR_MAP_SWIZZLE_64B, np) ||
            !tc_encode(c, &mdK, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, p.dK, gd, gs, gbx, CU_TENSOR_MAP_SWIZZLE_128B, np) ||
            !tc_encode(c, &mdV, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, p.dV, gd, gs, gbx, CU_TENSOR_MAP_SWIZZLE_128B, np)) return 1;
        const cuuint64_t qdim[2] = {(cuuint64_t)qd, (cuuint64_t)p.T}, qst[1] = {(cuuint64_t)qd * 4};
        if (p.dQ && (!tc_encode(c, &mdQ, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, p.dQ, qdim, qst, gbx, CU_TENSOR_MAP_SWIZZLE_128B, np) ||
                     !tc_encode(c, &mA1, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, p.dS1, sd, ss, abx, CU_TENSOR_MAP_SWIZZLE_128B) ||
                     !tc_encode(c, &mA2, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, p.dS2, sd, ss, abx, CU_TENSOR_MAP_SWIZZLE_128B) ||
                     !af_make_map(c, &mB1, p.k1, p.T, kvd, 64) || !af_make_map(c, &mB2, p.k2, p.T, kvd, 64))) return 1;
    }
    const long blocks = (long)nkb * seqs.n * p.Hkv, qblocks = (long)nkb * seqs.n * p.Hq;
    // pairs per chunk: their Q and dO parts (8 bytes per element) within about a third of the L2
    const size_t pair_bytes = (size_t)g * Smax * HD * 8;
    int chunk = (int)((size_t)(40u << 20) / pair_bytes);
    chunk = max(1, min(chunk, seqs.n * p.Hkv));
    if (qblocks > 0x7fffffffL) return 1;
    cudaStream_t st = (cudaStream_t)c->pub.stream;
    sb_launch(kern, dim3((unsigned)blocks), dim3(AB_THREADS), AB_SMEM(NH), st, mQ1, mQ2, mD1, mD2, mK1, mK2, mV1, mV2, mS1, mS2, mdK, mdV, p.LT, p.DT, (__half*)p.dS1, (__half*)p.dS2, p.dK, p.dV,
        p.amax_q, p.amax_k, p.amax_v, p.amax_do, p.ds_bound, seqs, p.Sp, p.Hq, g, nkb, chunk, p.accumulate, upper, 1.0f / sqrtf((float)HD), c->d_status, p.amax_dk, p.amax_dv);
    c->launches++;
    if (p.dQ) {
        sb_launch(at_dq_bwd_kernel<HD>, dim3((unsigned)qblocks), dim3(AQ_THREADS), AQ_SMEM(NH, AQ_STAGES(NH, qblocks)), st, mA1, mA2, mB1, mB2, mdQ, seqs, p.dQ, p.ds_bound, p.amax_k, p.Sp, p.Hq, g, nkb, c->d_status, p.amax_dq);
        c->launches++;
    }
    return cudaGetLastError() == cudaSuccess ? 0 : 1;
}

// See AbCall for the operands.  Returns 0 when launched, 1 when this path does not take the call.
int sb_attention_fused_dkv(sb_ctx_t* c, const AbCall& p, int hd) {
    if (p.Sp % 128 || p.Hkv <= 0 || p.Hq % p.Hkv || !tc_load_encode()) return 1;
    if (c->h_seq_n <= 0 || !c->attn_seq_starts) return 1;
    if (!tc_aligned16(p.dK) || !tc_aligned16(p.dV) || !tc_aligned16(p.dQ)) return 1;
    if (hd == 128) return ab_launch<128>(c, p);
    if (hd == 64) return ab_launch<64>(c, p);
    return 1;
}
