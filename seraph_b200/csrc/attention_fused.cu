// attention_fused.cu - causal attention forward in one kernel (head sizes 64 and 128, FP16 hi/lo parts, FP32-level accuracy).
//
// A tile is 128 consecutive queries of one (sequence, query head); a CTA per SM takes tiles in turn, those with the most keys first, from a counter, and
// walks over each one's keys in blocks of 64, up to the diagonal.  Nothing of size S x S ever reaches memory:
//
//   S_j  = Q K_j^T          tcgen05.mma kind::f16, M 128 x N 64 x K 128, three passes (q1 k1 + q2 k1 + q1 k2) on the
//                           prepared parts of Q and K (x * 2^s = h1 + h2), Q from tensor memory, accumulator in tensor memory: the two halves
//                           of the head dimension go to two accumulators of twelve instructions each, added in FP32
//   P_j  = exp(S_j/sqrt(hd) - m)   by the softmax warps, half a query row per thread, running maximum m and sum l;
//                           written back over the scores in tensor memory as two FP16 parts of P * 2^14
//   O    = O * alpha + P_j V_j     M 128 x N 128 x K 64, three passes on the parts of P (tensor memory) and V (read in place,
//                           MN-major), twelve instructions into a fresh accumulator that the O warps add into
//                           registers (round-to-nearest FP32) after scaling by alpha = exp(m_old - m_new)
//   out  = O / l,  lse = m + log l
//
// Warps: 0 tiles and TMA loads, 1 MMA issuer (owns the tensor-memory allocation), 4-11 softmax (two warps per lane quarter, 32 of a block's keys
// each, the maxima exchanged through shared memory), 12-15 O accumulation (a whole row per thread).  Shared memory: Q parts 64 KB on their way to tensor
// memory, K and V parts 2 x 32 KB each (double buffered), 32 KB of output staging.  64-wide heads run the same kernel with half of everything but the
// score block (one accumulator of twelve instructions per S).
//
// What bounds it: a block of 128-wide heads is 1536 cycles of the tensor core and 1900 of the softmax warps, at the clock that the power leaves
// (1.4 GHz under continuous load).  Before, one softmax warp per lane quarter, Q and P in shared memory (56 cycles an instruction of S instead of 32) and a
// CTA per tile, of whose 48000 cycles 8000 went before its first block and 8000, most of them a thread's 16-byte stores, after its last:
// 8 x 2048 tokens, 16 heads of 128: 490 -> 410 us; 8 heads of 64: 180 -> 115; 24 sequences of 383, 8 heads of 64: 60 -> 36.
// Every mbarrier wait is bounded; a wait that runs out sets the status word and the CTA drains and frees its
// tensor memory.
#include "attention_fused.cuh"

// Registers of a thread by warpgroup: 128 x (72 + 2 x 120 + 200) = 512 x 128, what the CTA is launched with
#define AF_REGS_LIGHT 72
#define AF_REGS_SOFTMAX 120
#define AF_REGS_O 200
#define AF_BAR_BYTES 320           // 28 barriers, the tensor-memory address, two tiles, eight flags
struct __align__(16) AfTile { int qb, h, t0, S; };      // qb: query block, -1 after the last tile; h: query head; the sequence's first row and length
template <int HD>
__global__ void __launch_bounds__(AF_THREADS, 1)
at_fused_fwd_kernel(const __grid_constant__ CUtensorMap mQ1, const __grid_constant__ CUtensorMap mQ2,
                    const __grid_constant__ CUtensorMap mK1, const __grid_constant__ CUtensorMap mK2,
                    const __grid_constant__ CUtensorMap mV1, const __grid_constant__ CUtensorMap mV2,
                    const __grid_constant__ CUtensorMap mO, const __grid_constant__ CUtensorMap mH1, const __grid_constant__ CUtensorMap mH2,
                    const AfSeqTab seqs, float* __restrict__ O, float* __restrict__ lse,
                    const float* __restrict__ amax_q, const float* __restrict__ amax_k, const float* __restrict__ amax_v,
                    int Hq, int g, int nqb_max, int tiles, unsigned* counter, float scale, int* status, float* bound_o, uint4* __restrict__ Oh, size_t n_o, unsigned keep) {
    constexpr int NH = HD / 64;                              // 64-column halves of the head dimension (one 128-byte row of halfs each)
    constexpr int Q_BYTES = NH * 32768, KV_STAGE = NH * 16384, Q_PART = NH * 16384, KV_PART = NH * 8192;
    constexpr int OFF_K = Q_BYTES, OFF_V = OFF_K + 2 * KV_STAGE, OFF_STG = OFF_V + 2 * KV_STAGE, OFF_BAR = OFF_STG + 32768;
    // tensor memory: two S buffers of NH x 64 columns (their first 64 become the parts of P), P V accumulators of HD, the parts of Q; in the parts 16
    // elements of k are 8 columns of hi and 8 of lo parts
    constexpr int NPV = HD == 64 ? 2 : 1;
    constexpr int COL_PV = 2 * NH * AF_BKV, COL_Q = COL_PV + NPV * HD, TMEM_COLS = 512;
    static_assert(COL_Q + HD <= TMEM_COLS, "tensor memory");
    const int qd = Hq * HD;

    extern __shared__ uint8_t af_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)af_raw + 1023) & ~(uintptr_t)1023);
    // what is left beside the tiles (3072 bytes) lies before and behind them as the alignment has it; 1008 bytes is the most that can lie before
    const bool front = (uint8_t*)smem - af_raw >= 512;
    uint64_t* bars = (uint64_t*)(front ? af_raw : smem + OFF_BAR);
    uint64_t* q_full = bars;            // 1: Q in shared memory
    uint64_t* q_empty = bars + 1;       // 1: and out of it again
    uint64_t* q_ready = bars + 2;       // 1: Q in tensor memory
    uint64_t* k_full = bars + 3;        // 2
    uint64_t* k_empty = bars + 5;       // 2
    uint64_t* v_full = bars + 7;        // 2
    uint64_t* v_empty = bars + 9;       // 2
    uint64_t* s_full = bars + 11;       // 2
    uint64_t* p_full = bars + 13;       // 2
    uint64_t* pv_full = bars + 15;      // 2
    uint64_t* pv_empty = bars + 17;     // 2
    uint64_t* h_full = bars + 19;       // 2
    uint64_t* h_empty = bars + 21;      // 2
    uint64_t* tile_full = bars + 23;    // 2
    uint64_t* tile_empty = bars + 25;   // 2
    uint32_t* tmem_slot = (uint32_t*)(bars + 28);
    AfTile* tile_s = (AfTile*)(bars + 30);                    // [2]
    volatile int* bad = (volatile int*)(tile_s + 2);          // [8]: a softmax warp that gave up
    // [2][2][128]: the maximum of each row's two halves of a block.  The softmax warps and the O warps form the running maximum and its factors from
    // them, each for themselves.  After a tile's last block the next slot passes the sums.
    float* half_s = (float*)(smem + OFF_BAR + (front ? 0 : AF_BAR_BYTES));

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        mbar_init(q_full, 1); mbar_init(q_empty, 8); mbar_init(q_ready, 8);
        for (int i = 0; i < 2; i++) {
            mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1); mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1);
            mbar_init(&s_full[i], 1); mbar_init(&p_full[i], 8); mbar_init(&pv_full[i], 1); mbar_init(&pv_empty[i], 4);
            mbar_init(&h_full[i], 8); mbar_init(&h_empty[i], 4); mbar_init(&tile_full[i], 1); mbar_init(&tile_empty[i], 13);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (threadIdx.x < 8) bad[threadIdx.x] = 0;
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    sb_pdl_enter();
    if (bound_o && blockIdx.x == 0 && threadIdx.x == 0) *bound_o = sb_word(amax_v);
    bool ok = true;
    // the n-th tile of this CTA, for one role; `arrive`: the lane that gives the slot back.  False: no more, or the wait ran out (then ok is false)
    auto next_tile = [&](int n, bool arrive, AfTile& t, int& nkv) -> bool {
        ok = ok && mbar_wait(&tile_full[n & 1], (n >> 1) & 1);
        if (!ok) return false;
        const uint32_t a = smem_u32(&tile_s[n & 1]);
        asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(t.qb), "=r"(t.h), "=r"(t.t0), "=r"(t.S) : "r"(a) : "memory");
        __syncwarp(__activemask());
        if (arrive) af_arrive(&tile_empty[n & 1]);
        nkv = min((t.S + AF_BKV - 1) / AF_BKV, 2 * t.qb + 2);
        return t.qb >= 0;
    };

    if (warp < 4) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(AF_REGS_LIGHT));
    if (warp == 0) {
        // ---------------- tiles and TMA loads ----------------
        if (elect_one()) {
            const int per_i = seqs.n * Hq;
            const int gave_up = *(volatile int*)status;        // an earlier CTA did: do not queue behind its cause (on its way together with the boundaries)
            int tile = (int)blockIdx.x;
            uint32_t gk = 0;                                   // blocks so far
            for (int n = 0; ok; n++) {
                // tiles with the most keys first, the query heads of one K/V head side by side; some have no rows
                AfTile t;
                for (;; tile = (int)gridDim.x + (int)atomicAdd(counter, 1u)) {
                    t.qb = -1; t.h = t.t0 = t.S = 0;
                    if (tile >= tiles) break;
                    const int rem = tile % per_i, b = rem / Hq;
                    t.qb = nqb_max - 1 - tile / per_i; t.h = rem % Hq;
                    t.t0 = (int)seqs.start[b]; t.S = (int)seqs.start[b + 1] - t.t0;
                    if (t.qb * AF_BQ < t.S || gave_up) break;
                }
                if (gave_up) t.qb = -1;
                ok = mbar_wait(&tile_empty[n & 1], ((n >> 1) & 1) ^ 1);
                if (!ok) break;
                tile_s[n & 1] = t;
                af_arrive(&tile_full[n & 1]);
                if (t.qb < 0) break;
                tile = (int)gridDim.x + (int)atomicAdd(counter, 1u);
                const int nkv = min((t.S + AF_BKV - 1) / AF_BKV, 2 * t.qb + 2), kvh = t.h / g;
                ok = mbar_wait(q_empty, (n & 1) ^ 1);
                if (!ok) break;
                mbar_expect_tx(q_full, Q_BYTES);
                for (int p = 0; p < NH; p++) {
                    af_tma_2d(smem + p * 16384, &mQ1, q_full, t.h * HD + p * 64, t.t0 + t.qb * AF_BQ);
                    af_tma_2d(smem + Q_PART + p * 16384, &mQ2, q_full, t.h * HD + p * 64, t.t0 + t.qb * AF_BQ);
                }
                // order of need: K_0, K_1, V_0, K_2, V_1, ...
                for (int jj = -1; jj < nkv && ok; jj++) {
                    if (jj + 1 < nkv) {
                        const uint32_t i = gk + (uint32_t)(jj + 1), s = i & 1;
                        ok = mbar_wait(&k_empty[s], ((i >> 1) & 1) ^ 1);
                        if (!ok) break;
                        uint8_t* dst = smem + OFF_K + s * KV_STAGE;
                        mbar_expect_tx(&k_full[s], KV_STAGE);
                        for (int p = 0; p < NH; p++) {
                            af_tma_2d(dst + p * 8192, &mK1, &k_full[s], kvh * HD + p * 64, t.t0 + (jj + 1) * AF_BKV);
                            af_tma_2d(dst + KV_PART + p * 8192, &mK2, &k_full[s], kvh * HD + p * 64, t.t0 + (jj + 1) * AF_BKV);
                        }
                    }
                    if (jj >= 0) {
                        const uint32_t i = gk + (uint32_t)jj, s = i & 1;
                        ok = mbar_wait(&v_empty[s], ((i >> 1) & 1) ^ 1);
                        if (!ok) break;
                        uint8_t* dst = smem + OFF_V + s * KV_STAGE;
                        mbar_expect_tx(&v_full[s], KV_STAGE);
                        for (int p = 0; p < NH; p++) {
                            af_tma_2d(dst + p * 8192, &mV1, &v_full[s], kvh * HD + p * 64, t.t0 + jj * AF_BKV);
                            af_tma_2d(dst + KV_PART + p * 8192, &mV2, &v_full[s], kvh * HD + p * 64, t.t0 + jj * AF_BKV);
                        }
                    }
                }
                gk += (uint32_t)nkv;
            }
            if (!ok) atomicExch(status, SB_ERR_TIMEOUT);
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        if (elect_one()) {
            const uint32_t idesc_s = (1u << 4) | ((uint32_t)(AF_BKV >> 3) << 17) | ((uint32_t)(AF_BQ >> 4) << 24);
            const uint32_t idesc_o = (1u << 4) | (1u << 16) | ((uint32_t)(HD >> 3) << 17) | ((uint32_t)(AF_BQ >> 4) << 24);
            uint32_t gk = 0;
            AfTile t;
            int nkv;
            for (int n = 0; next_tile(n, true, t, nkv); n++) {
                ok = mbar_wait(q_ready, n & 1);
                for (int jj = -1; jj < nkv && ok; jj++) {
                    if (jj + 1 < nkv) {
                        // S = Q K^T of the next block: head-dimension half p into accumulator p of its S buffer (the parts of P two blocks before, which lie
                        // there, were consumed by instructions issued before these)
                        const uint32_t i = gk + (uint32_t)(jj + 1), s = i & 1;
                        ok = mbar_wait(&k_full[s], (i >> 1) & 1);
                        if (!ok) break;
                        tc_fence_after();
                        const uint32_t sk = smem_u32(smem + OFF_K + s * KV_STAGE);
#pragma unroll
                        for (int p = 0; p < NH; p++) {
                            const uint64_t b1 = make_kmajor_desc<128>(sk + p * 8192), b2 = make_kmajor_desc<128>(sk + KV_PART + p * 8192);
                            const uint32_t d = tmem_base + s * (NH * AF_BKV) + (uint32_t)(p * AF_BKV);
#pragma unroll
                            for (int kk = 0; kk < 4; kk++) {
                                const uint64_t adv = (uint64_t)(kk * 2);
                                const uint32_t ta = tmem_base + (uint32_t)(COL_Q + (p * 4 + kk) * 16);
                                af_mma_ts(d, ta, b1 + adv, idesc_s, kk ? 1u : 0u);
                                af_mma_ts(d, ta + 8, b1 + adv, idesc_s, 1);
                                af_mma_ts(d, ta, b2 + adv, idesc_s, 1);
                            }
                        }
                        tc_commit(&s_full[s]);
                        tc_commit(&k_empty[s]);
                    }
                    if (jj >= 0) {
                        // O contribution of block jj: P V
                        const uint32_t i = gk + (uint32_t)jj, s = i & 1, v = i % NPV;
                        ok = mbar_wait(&v_full[s], (i >> 1) & 1) && mbar_wait(&pv_empty[v], ((i / NPV) & 1) ^ 1) && mbar_wait(&p_full[s], (i >> 1) & 1);
                        if (!ok) break;
                        tc_fence_after();
                        const uint32_t sv = smem_u32(smem + OFF_V + s * KV_STAGE);
                        const uint64_t b1 = make_mn16_desc<AF_BKV>(sv), b2 = make_mn16_desc<AF_BKV>(sv + KV_PART);
                        const uint32_t d = tmem_base + (uint32_t)COL_PV + v * HD;
#pragma unroll
                        for (int kk = 0; kk < 4; kk++) {
                            const uint64_t advb = (uint64_t)(kk * 128);
                            const uint32_t ta = tmem_base + s * (NH * AF_BKV) + (uint32_t)(kk * 16);
                            af_mma_ts(d, ta, b1 + advb, idesc_o, kk ? 1u : 0u);
                            af_mma_ts(d, ta + 8, b1 + advb, idesc_o, 1);
                            af_mma_ts(d, ta, b2 + advb, idesc_o, 1);
                        }
                        tc_commit(&pv_full[v]);
                        tc_commit(&v_empty[s]);
                    }
                }
                gk += (uint32_t)nkv;
            }
            if (!ok) atomicExch(status, SB_ERR_TIMEOUT);
        }
    } else if (warp >= 4 && warp < 12) {
        // ---------------- softmax: half a query row (32 of the block's keys) per thread ----------------
        // The two warps of a lane quarter meet at a named barrier in every block, once before they leave, and learn there whether the other one's waits
        // ran out: both meet the same number of times, whichever of them gives up.  A warp that gives up leaves the number of the meeting it does so at: the other
        // one may look only after that warp has gone on to the next meeting, and must not leave before it.
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(AF_REGS_SOFTMAX));
        const int q = warp & 3, half = (warp - 4) >> 2, r = q * 32 + lane;
        const uint32_t lanes = tmem_base + ((uint32_t)(q * 32) << 16);
        const float cs = tc_pow2(-tc_f16_shift(sb_word(amax_q))) * tc_pow2(-tc_f16_shift(sb_word(amax_k))) * (scale * 1.4426950408889634f);
        auto meet = [&](uint32_t id) {                         // id: as many meetings before this one, the same in both warps
            if (!ok && lane == 0) bad[q * 2 + half] = (int)id + 1;
            __syncwarp();
            asm volatile("bar.sync %0, 64;" ::"r"(1 + q) : "memory");
            const int other = bad[q * 2 + (half ^ 1)];
            if (other != 0 && other <= (int)id + 1) ok = false;
        };
        uint32_t gk = 0, gh = 0;                               // blocks so far, slots of half_s used so far
        for (int n = 0;; n++) {
            AfTile t;
            int nkv;
            if (!next_tile(n, lane == 0, t, nkv)) { meet(gh); break; }
            const int qi = t.qb * AF_BQ + r;                   // position of this row inside the sequence
            float m = -INFINITY, l = 0.f;
            // This row's parts of Q from shared memory (128-byte-swizzled tiles) into tensor memory, where an instruction of 64 columns reads them without
            // waiting for 4 KB of shared memory (56 cycles instead of 32); half of the k-steps each.  The last S of the tile before was complete when
            // this warp read it.
            ok = ok && mbar_wait(q_full, n & 1);
            {
                const uint32_t qt = smem_u32(smem) + (uint32_t)(r * 128);
#pragma unroll
                for (int k = 0; k < NH * 2; k++) {
                    const int kk = half * (NH * 2) + k;
                    uint32_t h8[8], l8[8];
                    const uint32_t at = qt + (uint32_t)((kk >> 2) * 16384), c0 = (uint32_t)(((2 * (kk & 3)) ^ (r & 7)) << 4), c1 = (uint32_t)(((2 * (kk & 3) + 1) ^ (r & 7)) << 4);
                    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(h8[0]), "=r"(h8[1]), "=r"(h8[2]), "=r"(h8[3]) : "r"(at + c0) : "memory");
                    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(h8[4]), "=r"(h8[5]), "=r"(h8[6]), "=r"(h8[7]) : "r"(at + c1) : "memory");
                    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(l8[0]), "=r"(l8[1]), "=r"(l8[2]), "=r"(l8[3]) : "r"(at + Q_PART + c0) : "memory");
                    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(l8[4]), "=r"(l8[5]), "=r"(l8[6]), "=r"(l8[7]) : "r"(at + Q_PART + c1) : "memory");
                    af_st8(lanes + (uint32_t)(COL_Q + kk * 16), h8);
                    af_st8(lanes + (uint32_t)(COL_Q + kk * 16 + 8), l8);
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                tc_fence_before();
                __syncwarp();
                if (lane == 0) { af_arrive(q_ready); af_arrive(q_empty); }
            }
            for (int j = 0; j < nkv; j++) {
                const uint32_t i = gk + (uint32_t)j, s = i & 1, hi = gh + (uint32_t)j, hs = (hi & 1) * 256;
                ok = ok && mbar_wait(&s_full[s], (i >> 1) & 1);
                tc_fence_after();
                float y[32];                                    // raw scores (the two accumulators added)
                {
                    const uint32_t ta = lanes + s * (NH * AF_BKV) + (uint32_t)(half * 32);
                    uint32_t a[32], c[32];
                    af_ld32_issue(ta, a);
                    if constexpr (NH == 2) af_ld32_issue(ta + 64, c);
                    af_ld_wait(a);
                    if constexpr (NH == 2) af_ld_dep(c);
#pragma unroll
                    for (int e = 0; e < 32; e++) y[e] = NH == 2 ? __uint_as_float(a[e]) + __uint_as_float(c[e]) : __uint_as_float(a[e]);
                }
                if (j >= 2 * t.qb) {                           // blocks that reach the diagonal: keys after the query do not count
                    const int k0 = j * AF_BKV + half * 32;
#pragma unroll
                    for (int e = 0; e < 32; e++) if (k0 + e > qi) y[e] = -INFINITY;
                }
                float mx4[4] = {y[0], y[1], y[2], y[3]};
#pragma unroll
                for (int e = 4; e < 32; e++) mx4[e & 3] = fmaxf(mx4[e & 3], y[e]);
                const float mine = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * cs;      // cs > 0
                ok = ok && mbar_wait(&h_empty[hi & 1], ((hi >> 1) & 1) ^ 1);
                half_s[hs + half * 128 + r] = mine;
                meet(hi);
                if (!ok) break;
                if (lane == 0) af_arrive(&h_full[hi & 1]);
                const float m_new = fmaxf(m, fmaxf(mine, half_s[hs + (half ^ 1) * 128 + r]));      // finite from block 0 on: key 0 counts for every row
                const float alpha = af_ex2(m - m_new);
                // P leaves as P * 2^14.  128-wide heads: the 14 rides on the exponent, which costs nothing and rounds an exponent of up to 14;
                // 64-wide heads have the issue slots for an exact multiplication instead
                constexpr bool EXACT = HD == 64;
                const float off = EXACT ? -m_new : 14.f - m_new;
                float sm4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int e = 0; e < 32; e++) { y[e] = af_ex2(fmaf(y[e], cs, off)); if (EXACT) y[e] *= 16384.f; sm4[e & 3] += y[e]; }
                l = l * alpha + ((sm4[0] + sm4[1]) + (sm4[2] + sm4[3]));          // in units of 2^-14
                m = m_new;
                // P * 2^14 as two FP16 parts, over the columns that its scores came from (all of them are in registers by now)
                const uint32_t tp = lanes + s * (NH * AF_BKV) + (uint32_t)(half * 32);
#pragma unroll
                for (int kk = 0; kk < 2; kk++) {
                    uint32_t w1[8], w2[8];
#pragma unroll
                    for (int e = 0; e < 8; e++) af_split2(y[kk * 16 + 2 * e], y[kk * 16 + 2 * e + 1], w1[e], w2[e]);
                    af_st8(tp + kk * 16, w1);
                    af_st8(tp + kk * 16 + 8, w2);
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                tc_fence_before();
                __syncwarp();
                if (lane == 0) af_arrive(&p_full[s]);
            }
            if (!ok) break;                                    // agreed on at the last meeting
            // the row's sum, of both halves, through the next slot
            const uint32_t hi = gh + (uint32_t)nkv, hs = (hi & 1) * 256;
            ok = ok && mbar_wait(&h_empty[hi & 1], ((hi >> 1) & 1) ^ 1);
            if (half) half_s[hs + 128 + r] = l;
            meet(hi);
            if (!ok) break;
            if (!half) {
                l += half_s[hs + 128 + r];
                half_s[hs + r] = l > 0.f ? 1.0f / l : 0.f;
                if (lse && qi < t.S) lse[(size_t)(t.t0 + qi) * Hq + t.h] = fmaf(m, 0.6931471805599453f, logf(l * (1.0f / 16384.f)));
            }
            __syncwarp();
            if (lane == 0) af_arrive(&h_full[hi & 1]);
            gk += (uint32_t)nkv; gh += (uint32_t)nkv + 1;
        }
        if (!ok && lane == 0) atomicExch(status, SB_ERR_TIMEOUT);
    } else if (warp >= 12) {
        // ---------------- O accumulation: one row per thread ----------------
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(AF_REGS_O));
        const int q = warp & 3, r = q * 32 + lane;
        const uint32_t stg = smem_u32(smem + OFF_STG + q * 8192);      // two blocks of 32 rows x 128 bytes on their way out
        const float fv = tc_pow2(-tc_f16_shift(sb_word(amax_v))), sc = tc_pow2(tc_f16_shift(sb_word(amax_v)));
        uint32_t gk = 0, gh = 0;
        AfTile t;
        int nkv;
        for (int n = 0; next_tile(n, lane == 0, t, nkv); n++) {
            const int qi = t.qb * AF_BQ + r;
            float o[HD], m = -INFINITY;
#pragma unroll
            for (int i = 0; i < HD; i++) o[i] = 0.f;
            for (int j = 0; j < nkv; j++) {
                const uint32_t i = gk + (uint32_t)j, v = i % NPV, hi = gh + (uint32_t)j, hs = (hi & 1) * 256;
                ok = mbar_wait(&h_full[hi & 1], (hi >> 1) & 1);
                if (!ok) break;
                const float m_new = fmaxf(m, fmaxf(half_s[hs + r], half_s[hs + 128 + r])), alpha = af_ex2(m - m_new);      // as the softmax warps
                m = m_new;
                __syncwarp();
                if (lane == 0) af_arrive(&h_empty[hi & 1]);
                ok = mbar_wait(&pv_full[v], (i / NPV) & 1);
                if (!ok) break;
                tc_fence_after();
                const uint32_t ta = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)COL_PV + v * HD;
#pragma unroll
                for (int c = 0; c < HD / 32; c++) {
                    uint32_t w[32];
                    af_ld32_issue(ta + c * 32, w);
                    af_ld_wait(w);
                    if (c == HD / 32 - 1) {
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) af_arrive(&pv_empty[v]);
                    }
#pragma unroll
                    for (int e = 0; e < 32; e++) o[c * 32 + e] = fmaf(o[c * 32 + e], alpha, __uint_as_float(w[e]));
                }
            }
            const uint32_t hi = gh + (uint32_t)nkv;
            ok = ok && mbar_wait(&h_full[hi & 1], (hi >> 1) & 1);
            if (!ok) break;
            const float f = half_s[(hi & 1) * 256 + r] * fv;      // 1 / l with l in units of 2^-14, O holds (P * 2^14) V' products
            __syncwarp();
            if (lane == 0) af_arrive(&h_empty[hi & 1]);
            gk += (uint32_t)nkv; gh += (uint32_t)nkv + 1;
#pragma unroll
            for (int i = 0; i < HD; i++) o[i] *= f;
            // O is a weighted mean of rows of V, so max |V| bounds it: its word for the output projection's operand, and the scale of the parts that
            // are written here beside O (a split pass over O less).  32 rows that all belong to the sequence go out as tiles (a thread's own row, 16 bytes at
            // a time, took 5500 cycles a tile); the last rows of a sequence as they are.
            const int y0 = t.t0 + t.qb * AF_BQ + q * 32;
            if (t.qb * AF_BQ + q * 32 + 32 <= t.S) {
                auto room = [&]() { if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory"); __syncwarp(); };
                auto send = [&](const CUtensorMap* map, uint32_t buf, int x) {
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) {
                        asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(map), "r"(x), "r"(y0), "r"(buf) : "memory");
                        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                    }
                };
#pragma unroll
                for (int c = 0; c < HD / 32; c++) {
                    const uint32_t buf = stg + (uint32_t)((c & 1) * 4096);
                    room();
#pragma unroll
                    for (int i = 0; i < 8; i++)
                        asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(buf + (uint32_t)(lane * 128 + ((i ^ (lane & 7)) << 4))),
                                     "f"(o[c * 32 + 4 * i]), "f"(o[c * 32 + 4 * i + 1]), "f"(o[c * 32 + 4 * i + 2]), "f"(o[c * 32 + 4 * i + 3]) : "memory");
                    send(&mO, buf, t.h * HD + c * 32);
                }
                if (Oh) {
#pragma unroll
                    for (int c = 0; c < NH; c++)
#pragma unroll
                        for (int part = 0; part < 2; part++) {
                            const uint32_t buf = stg + (uint32_t)(part * 4096);
                            room();
#pragma unroll
                            for (int i = 0; i < 8; i++) {
                                uint32_t a[4], b[4];
#pragma unroll
                                for (int e = 0; e < 4; e++) sb_split2(o[c * 64 + 8 * i + 2 * e] * sc, o[c * 64 + 8 * i + 2 * e + 1] * sc, a[e], b[e], keep);
                                const uint32_t at = buf + (uint32_t)(lane * 128 + ((i ^ (lane & 7)) << 4));
                                if (part == 0) asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]) : "memory");
                                else           asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]) : "memory");
                            }
                            send(part == 0 ? &mH1 : &mH2, buf, t.h * HD + c * 64);
                        }
                }
            } else if (qi < t.S) {
                const size_t at = (size_t)(t.t0 + qi) * qd + (size_t)t.h * HD;
                float4* dst = (float4*)(O + at);
#pragma unroll
                for (int i = 0; i < HD / 4; i++) dst[i] = make_float4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
                if (Oh) {
#pragma unroll
                    for (int i = 0; i < HD / 8; i++) {
                        uint4 a, b;
                        sb_split2(o[8 * i] * sc, o[8 * i + 1] * sc, a.x, b.x, keep); sb_split2(o[8 * i + 2] * sc, o[8 * i + 3] * sc, a.y, b.y, keep);
                        sb_split2(o[8 * i + 4] * sc, o[8 * i + 5] * sc, a.z, b.z, keep); sb_split2(o[8 * i + 6] * sc, o[8 * i + 7] * sc, a.w, b.w, keep);
                        Oh[at / 8 + i] = a; Oh[(n_o + at) / 8 + i] = b;
                    }
                }
            }
        }
        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");      // the buffers are read out before the CTA gives its shared memory back
        if (!ok && lane == 0) atomicExch(status, SB_ERR_TIMEOUT);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS));
    }
}

// ---------------------------------------------------------------------------------------------------------------
// Backward scores in one kernel: for 128 queries of one (sequence, head) and every block of 64 keys up to the diagonal
//   S = Q K^T, dP = dO V^T   (three FP16 passes each, two twelve-instruction accumulators per product, in tensor memory)
//   P = exp(S/sqrt(hd) - lse),  dS = P o (dP - D) / sqrt(hd)
// and P, dS leave as the FP16 parts the three long products of the backward pass read (P * 2^14; dS times the power
// of two that brings its bound to [2^14, 2^15)), laid out [head][Sp][Sp] like the score scratch.  Columns past the
// diagonal are written as zeros up to the end of the row's 256-column tile, which is as far as those products read.
// Warps: 0 TMA producer, 1 MMA issuer, 4-11 elementwise (two per lane quarter, 32 of the 64 columns each).
// Shared memory: Q and dO parts 2 x 64 KB, K parts 2 x 32 KB (double buffered), V parts 32 KB.
#define AS_OFF_DO 65536
#define AS_OFF_K 131072
#define AS_OFF_V (AS_OFF_K + 2 * AF_KV_STAGE)
#define AS_OFF_BAR (AS_OFF_V + AF_KV_STAGE)
#define AS_SMEM (AS_OFF_BAR + 1024 + 1024)
#define AS_THREADS 384

__global__ void __launch_bounds__(AS_THREADS, 1)
at_score_bwd_kernel(const __grid_constant__ CUtensorMap mQ1, const __grid_constant__ CUtensorMap mQ2,
                    const __grid_constant__ CUtensorMap mD1, const __grid_constant__ CUtensorMap mD2,
                    const __grid_constant__ CUtensorMap mK1, const __grid_constant__ CUtensorMap mK2,
                    const __grid_constant__ CUtensorMap mV1, const __grid_constant__ CUtensorMap mV2,
                    const float* __restrict__ lse, const float* __restrict__ D,
                    __half* __restrict__ P1, __half* __restrict__ P2, __half* __restrict__ dS1, __half* __restrict__ dS2,
                    const float* __restrict__ amax_q, const float* __restrict__ amax_k, const float* __restrict__ amax_v,
                    const float* __restrict__ amax_do, const float* __restrict__ ds_bound,
                    const __grid_constant__ AfSeqs seqs, int Sp, int Hq, int g, int head0, int head_step, int nb, int nqb, float scale, int* status) {
    sb_pdl_enter();
    // nb > 0: one sequence, heads head0 + i * head_step, output slot i.  nb == 0: every sequence and head of the call,
    // output slot ((sequence * g + head % g) * Hkv + head / g), i.e. the Hkv heads of one (sequence, group member) side by side
    const int nheads = nb > 0 ? nb : Hq;
    const int per_i = seqs.n * nheads;
    const int qb = nqb - 1 - (int)blockIdx.x / per_i;
    const int rem = (int)blockIdx.x % per_i;
    const int b = rem / nheads, hi = rem % nheads;
    const int h = nb > 0 ? head0 + hi * head_step : hi;
    const int hb = nb > 0 ? hi : (b * g + h % g) * (Hq / g) + h / g;
    const int t0 = seqs.start[b], S = seqs.start[b + 1] - t0;
    if (qb * AF_BQ >= S) return;
    if (__syncthreads_or(*(volatile int*)status != 0)) return;            // all threads or none, also while another CTA sets it
    const int nkv = min((S + AF_BKV - 1) / AF_BKV, 2 * qb + 2);           // key blocks that hold scores
    const int nz = min(Sp / AF_BKV, 4 * (qb / 2 + 1));                    // key blocks that are written
    const int kvh = h / g;

    extern __shared__ uint8_t af_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)af_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = (uint64_t*)(smem + AS_OFF_BAR);
    uint64_t* q_full = bars;            // 1
    uint64_t* k_full = bars + 1;        // 2
    uint64_t* k_empty = bars + 3;       // 2
    uint64_t* v_full = bars + 5;        // 1
    uint64_t* v_empty = bars + 6;       // 1
    uint64_t* acc_full = bars + 7;      // 2
    uint64_t* acc_empty = bars + 9;     // 2
    uint32_t* tmem_slot = (uint32_t*)(bars + 12);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        mbar_init(q_full, 1); mbar_init(v_full, 1); mbar_init(v_empty, 1);
        for (int i = 0; i < 2; i++) { mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1); mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], 8); }
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
    bool ok = true;

    if (warp == 0) {
        if (elect_one()) {
            mbar_expect_tx(q_full, 2 * AF_Q_BYTES);
            for (int p = 0; p < 2; p++) {
                af_tma_2d(smem + p * 16384, &mQ1, q_full, h * AF_HD + p * 64, t0 + qb * AF_BQ);
                af_tma_2d(smem + 32768 + p * 16384, &mQ2, q_full, h * AF_HD + p * 64, t0 + qb * AF_BQ);
                af_tma_2d(smem + AS_OFF_DO + p * 16384, &mD1, q_full, h * AF_HD + p * 64, t0 + qb * AF_BQ);
                af_tma_2d(smem + AS_OFF_DO + 32768 + p * 16384, &mD2, q_full, h * AF_HD + p * 64, t0 + qb * AF_BQ);
            }
            for (int j = 0; j < nkv && ok; j++) {
                const int s = j & 1, u = j >> 1;
                ok = mbar_wait(&k_empty[s], (u & 1) ^ 1);
                if (!ok) break;
                uint8_t* dk = smem + AS_OFF_K + s * AF_KV_STAGE;
                mbar_expect_tx(&k_full[s], AF_KV_STAGE);
                for (int p = 0; p < 2; p++) {
                    af_tma_2d(dk + p * 8192, &mK1, &k_full[s], kvh * AF_HD + p * 64, t0 + j * AF_BKV);
                    af_tma_2d(dk + 16384 + p * 8192, &mK2, &k_full[s], kvh * AF_HD + p * 64, t0 + j * AF_BKV);
                }
                ok = mbar_wait(v_empty, (j & 1) ^ 1);
                if (!ok) break;
                uint8_t* dv = smem + AS_OFF_V;
                mbar_expect_tx(v_full, AF_KV_STAGE);
                for (int p = 0; p < 2; p++) {
                    af_tma_2d(dv + p * 8192, &mV1, v_full, kvh * AF_HD + p * 64, t0 + j * AF_BKV);
                    af_tma_2d(dv + 16384 + p * 8192, &mV2, v_full, kvh * AF_HD + p * 64, t0 + j * AF_BKV);
                }
            }
            if (!ok) atomicExch(status, SB_ERR_TIMEOUT);
        }
    } else if (warp == 1) {
        if (elect_one()) {
            const uint32_t idesc = (1u << 4) | ((uint32_t)(AF_BKV >> 3) << 17) | ((uint32_t)(AF_BQ >> 4) << 24);
            const uint32_t sq = smem_u32(smem), sdo = smem_u32(smem + AS_OFF_DO), sv = smem_u32(smem + AS_OFF_V);
            ok = mbar_wait(q_full, 0);
            for (int j = 0; j < nkv && ok; j++) {
                const int s = j & 1, u = j >> 1;
                ok = mbar_wait(&acc_empty[s], (u & 1) ^ 1) && mbar_wait(&k_full[s], u & 1);
                if (!ok) break;
                tc_fence_after();
                const uint32_t sk = smem_u32(smem + AS_OFF_K + s * AF_KV_STAGE);
#pragma unroll
                for (int p = 0; p < 2; p++) {
                    const uint64_t a1 = make_kmajor_desc<128>(sq + p * 16384), a2 = make_kmajor_desc<128>(sq + 32768 + p * 16384);
                    const uint64_t b1 = make_kmajor_desc<128>(sk + p * 8192), b2 = make_kmajor_desc<128>(sk + 16384 + p * 8192);
                    const uint32_t d = tmem_base + (uint32_t)(s * 256 + p * 64);
#pragma unroll
                    for (int kk = 0; kk < 4; kk++) {
                        const uint64_t adv = (uint64_t)(kk * 2);
                        af_mma_f16(d, a1 + adv, b1 + adv, idesc, kk ? 1u : 0u);
                        af_mma_f16(d, a2 + adv, b1 + adv, idesc, 1);
                        af_mma_f16(d, a1 + adv, b2 + adv, idesc, 1);
                    }
                }
                tc_commit(&k_empty[s]);
                ok = mbar_wait(v_full, j & 1);
                if (!ok) break;
                tc_fence_after();
#pragma unroll
                for (int p = 0; p < 2; p++) {
                    const uint64_t a1 = make_kmajor_desc<128>(sdo + p * 16384), a2 = make_kmajor_desc<128>(sdo + 32768 + p * 16384);
                    const uint64_t b1 = make_kmajor_desc<128>(sv + p * 8192), b2 = make_kmajor_desc<128>(sv + 16384 + p * 8192);
                    const uint32_t d = tmem_base + (uint32_t)(s * 256 + 128 + p * 64);
#pragma unroll
                    for (int kk = 0; kk < 4; kk++) {
                        const uint64_t adv = (uint64_t)(kk * 2);
                        af_mma_f16(d, a1 + adv, b1 + adv, idesc, kk ? 1u : 0u);
                        af_mma_f16(d, a2 + adv, b1 + adv, idesc, 1);
                        af_mma_f16(d, a1 + adv, b2 + adv, idesc, 1);
                    }
                }
                tc_commit(v_empty);
                tc_commit(&acc_full[s]);
            }
            if (!ok) atomicExch(status, SB_ERR_TIMEOUT);
        }
    } else if (warp >= 4) {
        // ---------------- elementwise: one query row and 32 of the block's 64 keys per thread ----------------
        const int q = warp & 3, r = q * 32 + lane, half = (warp - 4) >> 2;
        const int qi = qb * AF_BQ + r;
        const bool live = qi < S;
        const float cs = tc_pow2(-tc_f16_shift(sb_word(amax_q))) * tc_pow2(-tc_f16_shift(sb_word(amax_k))) * (scale * 1.4426950408889634f);
        const float cp = tc_pow2(-tc_f16_shift(sb_word(amax_do))) * tc_pow2(-tc_f16_shift(sb_word(amax_v)));
        const float dsc = tc_pow2(tc_f16_shift(sb_word(ds_bound))) * scale * (1.0f / 16384.f);      // pr holds P * 2^14
        const float L2 = live ? lse[(size_t)(t0 + qi) * Hq + h] * 1.4426950408889634f : 0.f;
        const float Dq = live ? D[(size_t)(t0 + qi) * Hq + h] : 0.f;
        // after the transpose: lane (a, c) = (lane / 4, lane % 4) writes chunk c of the warp's rows 4a + t, t = 0..3
        const size_t qrowbase = ((size_t)hb * Sp + (size_t)(qb * AF_BQ + q * 32 + 4 * (lane >> 2))) * Sp + half * 32 + (lane & 3) * 8;
        for (int j = 0; j < nz && ok; j++) {
            uint4 w[4][4];                                      // P1, P2, dS1, dS2: 32 halfs each
            if (j < nkv) {
                const int s = j & 1, u = j >> 1;
                ok = mbar_wait(&acc_full[s], u & 1);
                if (!ok) break;
                tc_fence_after();
                const uint32_t ta = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(s * 256 + half * 32);
                float pr[32];
                {
                    uint32_t a[32], c[32];
                    uint32_t a2[32], c2[32];
                    af_ld32_issue(ta, a);
                    af_ld32_issue(ta + 64, c);
                    af_ld32_issue(ta + 128, a2);
                    af_ld32_issue(ta + 192, c2);
                    af_ld_wait(a); af_ld_dep(c); af_ld_dep(a2); af_ld_dep(c2);
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) af_arrive(&acc_empty[s]);
                    const int k0 = j * AF_BKV + half * 32;
#pragma unroll
                    for (int i = 0; i < 32; i++) {
                        const float y = fmaf(__uint_as_float(a[i]) + __uint_as_float(c[i]), cs, 14.f - L2);
                        pr[i] = (live && k0 + i <= qi) ? af_ex2(y) : 0.f;                   // P * 2^14
                    }
                    uint32_t* w0 = (uint32_t*)&w[0][0]; uint32_t* w1 = (uint32_t*)&w[1][0];
                    uint32_t* w2 = (uint32_t*)&w[2][0]; uint32_t* w3 = (uint32_t*)&w[3][0];
#pragma unroll
                    for (int e = 0; e < 16; e++) {
                        const float p0 = pr[2 * e], p1 = pr[2 * e + 1];
                        const float d0 = p0 * ((__uint_as_float(a2[2 * e]) + __uint_as_float(c2[2 * e])) * cp - Dq) * dsc;
                        const float d1 = p1 * ((__uint_as_float(a2[2 * e + 1]) + __uint_as_float(c2[2 * e + 1])) * cp - Dq) * dsc;
                        af_split2(p0, p1, w0[e], w1[e]);
                        af_split2(d0, d1, w2[e], w3[e]);
                    }
                }
            } else {
#pragma unroll
                for (int a = 0; a < 4; a++)
#pragma unroll
                    for (int i = 0; i < 4; i++) w[a][i] = make_uint4(0, 0, 0, 0);
            }
            // A lane holds 64 bytes of its own row per array; lanes 4a..4a+3 transpose their 4 x 4 chunks of 16 bytes so that one
            // store instruction writes whole 64-byte row pieces (8 rows) instead of one chunk in each of 32 rows.
            if (j < nkv) {
#pragma unroll
                for (int a = 0; a < 4; a++) af_quad_transpose(w[a], lane);
            }
            const size_t o = qrowbase + (size_t)j * AF_BKV;
#pragma unroll
            for (int t = 0; t < 4; t++) {
                const size_t ot = o + (size_t)t * Sp;
                *(uint4*)(P1 + ot) = w[0][t]; *(uint4*)(P2 + ot) = w[1][t]; *(uint4*)(dS1 + ot) = w[2][t]; *(uint4*)(dS2 + ot) = w[3][t];
            }
        }
        if (!ok && lane == 0) atomicExch(status, SB_ERR_TIMEOUT);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512));
    }
}

template <int HD>
static int af_launch_fwd(sb_ctx_t* c, const void* q1, const void* q2, const void* k1, const void* k2, const void* v1, const void* v2,
                         const float* amax_q, const float* amax_k, const float* amax_v, float* O, float* lse, int T, int Hq, int Hkv) {
    constexpr int smem = HD / 64 * (32768 + 4 * 16384) + 32768 + 3072;      // tiles, output staging, alignment, barriers, the rows' maxima
    auto kern = at_fused_fwd_kernel<HD>;
    static bool attr_done = false;
    if (!attr_done) {
        cudaFuncAttributes fa;
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess || cudaFuncGetAttributes(&fa, kern) != cudaSuccess ||
            fa.numRegs * AF_THREADS < 128 * (AF_REGS_LIGHT + 2 * AF_REGS_SOFTMAX + AF_REGS_O)) { cudaGetLastError(); return 1; }      // (setmaxnreg.inc would wait for good)
        attr_done = true;
    }
    const int qd = Hq * HD, kvd = Hkv * HD;
    CUtensorMap mQ1, mQ2, mK1, mK2, mV1, mV2;
    if (!af_make_map(c, &mQ1, q1, T, qd, AF_BQ) || !af_make_map(c, &mQ2, q2, T, qd, AF_BQ) ||
        !af_make_map(c, &mK1, k1, T, kvd, AF_BKV) || !af_make_map(c, &mK2, k2, T, kvd, AF_BKV) ||
        !af_make_map(c, &mV1, v1, T, kvd, AF_BKV) || !af_make_map(c, &mV2, v2, T, kvd, AF_BKV)) return 1;
    const size_t n_o = (size_t)T * qd;
    CUtensorMap mO, mH1, mH2;
    {
        const cuuint64_t dims[2] = {(cuuint64_t)qd, (cuuint64_t)T}, pitch[1] = {(cuuint64_t)qd * 4};
        const cuuint32_t box[2] = {32u, 32u};
        if (!tc_encode(c, &mO, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, O, dims, pitch, box, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE)) return 1;
    }
    unsigned* counter = sb_item_counter(c);
    if (!counter) return 1;
    sb_resolve_host_seq(c);                                  // only now: a single call's boundaries are on their way to the host while the maps are made
    if (c->h_seq_n <= 0 || !c->h_seq || c->h_seq[c->h_seq_n] != T) return 1;
    int Smax = 0;
    for (int b = 0; b < c->h_seq_n; b++) Smax = max(Smax, c->h_seq[b + 1] - c->h_seq[b]);
    if (Smax <= 0) return 1;
    const AfSeqTab seqs = {c->h_seq_n, c->attn_seq_starts};
    const int nqb = (Smax + AF_BQ - 1) / AF_BQ;
    const long blocks = (long)nqb * seqs.n * Hq;
    if (blocks > 0x7fffffffL) return 1;
    // From here on the step's tables say that the kernel leaves the maximum and the parts of O (an operand of a training step).  Where it is not
    // launched after all, they must not: the kernels that then form O write neither.
    void* oh; float* own; int fresh;
    float* bound_o = (float*)sb_amax_take(c, O, n_o);
    if (sb_parts_find(c, O, n_o, &oh, &own, &fresh)) sb_parts_set_amax(c, O, (float*)amax_v); else oh = nullptr;
    mH1 = mH2 = mO;
    bool ok = !oh || (af_make_map(c, &mH1, oh, T, qd, 32) && af_make_map(c, &mH2, (__half*)oh + n_o, T, qd, 32));
    if (ok) {
        const int sms = c->pub.gpu_sm_count > 0 ? c->pub.gpu_sm_count : 148;
        sb_launch(kern, dim3((unsigned)(blocks < sms ? blocks : sms)), dim3(AF_THREADS), smem, (cudaStream_t)c->pub.stream, mQ1, mQ2, mK1, mK2, mV1, mV2, mO, mH1, mH2, seqs, O, lse, amax_q, amax_k, amax_v, Hq, Hq / Hkv, nqb, (int)blocks,
            counter, 1.0f / sqrtf((float)HD), c->d_status, bound_o, (uint4*)oh, n_o, sb_parts_keep(c));
        c->launches++;
        ok = cudaGetLastError() == cudaSuccess;
    }
    if (!ok) { sb_amax_forget(c, O); sb_parts_invalidate(c, O); }
    return ok ? 0 : 1;
}
// q1/q2, k1/k2, v1/v2: the FP16 parts of Q [T, Hq*hd], K and V [T, Hkv*hd]; amax_*: the device words their scales derive from.
// Returns 0 when the kernel was launched, 1 when this path does not take the call.
extern "C" int sb_attention_fused_forward(sb_ctx_t* c, const void* q1, const void* q2, const void* k1, const void* k2,
                                          const void* v1, const void* v2, const float* amax_q, const float* amax_k, const float* amax_v,
                                          float* O, float* lse, int T, int Hq, int Hkv, int hd) {
    if (!c->attn_seq_starts || Hq % Hkv || !tc_aligned16(O) || !tc_load_encode()) return 1;
    if (hd == 128) return af_launch_fwd<128>(c, q1, q2, k1, k2, v1, v2, amax_q, amax_k, amax_v, O, lse, T, Hq, Hkv);
    if (hd == 64) return af_launch_fwd<64>(c, q1, q2, k1, k2, v1, v2, amax_q, amax_k, amax_v, O, lse, T, Hq, Hkv);
    return 1;
}

// The backward score kernel.  nb > 0: one sequence [t0, t0 + S) and the heads head0, head0 + head_step, ... (nb of them), the
// parts P1..dS2 laid out [nb][Sp][Sp].  nb == 0: every sequence and head of the batch in one launch, parts laid out
// [sequence][group member][K-V head][Sp][Sp] (t0, S, head0, head_step unused).  Returns 0 when launched.
extern "C" int sb_attention_fused_scores(sb_ctx_t* c, const void* q1, const void* q2, const void* do1, const void* do2,
                                         const void* k1, const void* k2, const void* v1, const void* v2,
                                         const float* amax_q, const float* amax_k, const float* amax_v, const float* amax_do, const float* ds_bound,
                                         const float* lse, const float* D, void* P1, void* P2, void* dS1, void* dS2,
                                         int t0, int S, int Sp, int T, int Hq, int Hkv, int hd, int head0, int head_step, int nb) {
    if (hd != AF_HD || (Sp % 256) || nb < 0 || !tc_load_encode()) return 1;
    if (nb > 0 && S <= 0) return 1;
    if (nb == 0 && (c->h_seq_n <= 0 || c->h_seq_n > AF_MAXSEQ)) return 1;
    static bool attr_done = false;
    if (!attr_done) {
        if (cudaFuncSetAttribute(at_score_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, AS_SMEM) != cudaSuccess) { cudaGetLastError(); return 1; }
        attr_done = true;
    }
    AfSeqs seqs;
    int Smax = S;
    if (nb > 0) { seqs.n = 1; seqs.start[0] = t0; seqs.start[1] = t0 + S; }
    else {
        seqs.n = c->h_seq_n; Smax = 0;
        for (int b = 0; b <= c->h_seq_n; b++) seqs.start[b] = c->h_seq[b];
        for (int b = 0; b < c->h_seq_n; b++) Smax = max(Smax, c->h_seq[b + 1] - c->h_seq[b]);
        if (Smax <= 0) return 1;
    }
    const int qd = Hq * hd, kvd = Hkv * hd, nqb = (Smax + AF_BQ - 1) / AF_BQ;
    CUtensorMap mQ1, mQ2, mD1, mD2, mK1, mK2, mV1, mV2;
    if (!af_make_map(c, &mQ1, q1, T, qd, AF_BQ) || !af_make_map(c, &mQ2, q2, T, qd, AF_BQ) ||
        !af_make_map(c, &mD1, do1, T, qd, AF_BQ) || !af_make_map(c, &mD2, do2, T, qd, AF_BQ) ||
        !af_make_map(c, &mK1, k1, T, kvd, AF_BKV) || !af_make_map(c, &mK2, k2, T, kvd, AF_BKV) ||
        !af_make_map(c, &mV1, v1, T, kvd, AF_BKV) || !af_make_map(c, &mV2, v2, T, kvd, AF_BKV)) return 1;
    const long blocks = (long)nqb * seqs.n * (nb > 0 ? nb : Hq);
    if (blocks > 0x7fffffffL) return 1;
    sb_launch(at_score_bwd_kernel, dim3((unsigned)blocks), dim3(AS_THREADS), AS_SMEM, (cudaStream_t)c->pub.stream, mQ1, mQ2, mD1, mD2, mK1, mK2, mV1, mV2, lse, D, (__half*)P1, (__half*)P2, (__half*)dS1, (__half*)dS2,
        amax_q, amax_k, amax_v, amax_do, ds_bound, seqs, Sp, Hq, Hq / Hkv, head0, head_step, nb, nqb, 1.0f / sqrtf((float)hd), c->d_status);
    c->launches++;
    return cudaGetLastError() == cudaSuccess ? 0 : 1;
}
