// kernels_reduce.cu - row-reduction and optimizer kernels (sm_100a), all deterministic:
// no floating-point atomics anywhere, so two runs give the same bits.
//
// Reference kernels replaced (src/cuda_train_context.cu): rmsnorm :148,
// rmsnorm_backward :1767 (atomicAdd on grad_scale), softmax :1486,
// cross_entropy_grad[_packed] :1566/:1657, reduce_sum :2209 (atomicAdd),
// embedding_backward :2175 (atomicAdd, blockDim = hidden_size), adamw :2187.
#include <cuda_runtime.h>
#include <cuda_fp16.h>
#include <math.h>
#include <stdio.h>
#include <string.h>
#include <stdint.h>
#include "sb_internal.h"

#define RB_THREADS 256

static inline int aligned16(const void* p) { return (((uintptr_t)p) & 15) == 0; }
static inline int sm_count(sb_ctx_t* c) { return c->pub.gpu_sm_count > 0 ? c->pub.gpu_sm_count : 148; }

__device__ __forceinline__ float warp_sum(float v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
// block-wide sum of up to two values; every thread gets the result.  red: >= 2*32 floats of smem
__device__ __forceinline__ void block_sum2(float& a, float& b, float* red) {
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    a = warp_sum(a); b = warp_sum(b);
    __syncthreads();
    if (lane == 0) { red[w] = a; red[32 + w] = b; }
    __syncthreads();
    float x = 0.f, y = 0.f;
    for (int i = 0; i < nw; i++) { x += red[i]; y += red[32 + i]; }   // fixed order
    a = x; b = y;
}

// ---------------------------------------------------------------------------
// RMSNorm forward: y = x * (1/sqrt(mean(x^2)+eps)) * w.   8 bytes per element + w.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(RB_THREADS) rmsnorm_kernel(const float* __restrict__ x, const float* __restrict__ w,
                                                             float* __restrict__ y, int rows, int cols, float eps, int vec) {
    sb_pdl_enter();
    __shared__ float red[64];
    for (int r = blockIdx.x; r < rows; r += gridDim.x) {
        const float* xr = x + (size_t)r * cols; float* yr = y + (size_t)r * cols;
        float ss = 0.f, dummy = 0.f;
        if (vec) for (int i = threadIdx.x; i < cols / 4; i += blockDim.x) { float4 v = ((const float4*)xr)[i]; ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w; }
        else     for (int i = threadIdx.x; i < cols; i += blockDim.x) { float v = xr[i]; ss += v * v; }
        block_sum2(ss, dummy, red);
        float inv = 1.0f / sqrtf(ss / cols + eps);
        if (vec) for (int i = threadIdx.x; i < cols / 4; i += blockDim.x) {
            float4 v = ((const float4*)xr)[i], s = ((const float4*)w)[i];
            ((float4*)yr)[i] = make_float4(v.x * inv * s.x, v.y * inv * s.y, v.z * inv * s.z, v.w * inv * s.w);
        } else for (int i = threadIdx.x; i < cols; i += blockDim.x) yr[i] = xr[i] * inv * w[i];
    }
}

// ---------------------------------------------------------------------------
// RMSNorm backward.  Each CTA owns rows r = blockIdx.x, +gridDim.x, ...; it
// writes dx for them (optionally fused with the residual-gradient add) and
// keeps a per-column partial of dscale in registers, stored once to
// partial[blockIdx.x][cols].  A second kernel adds the partials in block
// order into dscale.  Algorithmic traffic: 12 bytes per element (+4 when the
// residual is fused) + cols*4.
// ---------------------------------------------------------------------------
#define RN_MAX_SWEEP 16     // cols <= RB_THREADS*4*RN_MAX_SWEEP = 16384
__global__ void __launch_bounds__(RB_THREADS) rmsnorm_bwd_kernel(const float* __restrict__ x, const float* __restrict__ w,
                                                                 const float* __restrict__ dy, const float* __restrict__ resid,
                                                                 float* __restrict__ dx, float* __restrict__ partial,
                                                                 int rows, int cols, float eps, int vec) {
    sb_pdl_enter();
    __shared__ float red[64];
    float acc[RN_MAX_SWEEP * 4];
#pragma unroll
    for (int i = 0; i < RN_MAX_SWEEP * 4; i++) acc[i] = 0.f;
    const int c4 = cols / 4;
    for (int r = blockIdx.x; r < rows; r += gridDim.x) {
        const float* xr = x + (size_t)r * cols; const float* gr = dy + (size_t)r * cols;
        float ss = 0.f, cp = 0.f;
        if (vec) for (int i = threadIdx.x; i < c4; i += blockDim.x) {
            float4 v = ((const float4*)xr)[i], g = ((const float4*)gr)[i], s = ((const float4*)w)[i];
            ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
            cp += g.x * s.x * v.x + g.y * s.y * v.y + g.z * s.z * v.z + g.w * s.w * v.w;
        } else for (int i = threadIdx.x; i < cols; i += blockDim.x) { float v = xr[i]; ss += v * v; cp += gr[i] * w[i] * v; }
        block_sum2(ss, cp, red);
        float inv = 1.0f / sqrtf(ss / cols + eps);
        float k = inv * inv * inv / cols * cp;
        float* dr = dx + (size_t)r * cols; const float* rr = resid ? resid + (size_t)r * cols : nullptr;
        if (vec) {
#pragma unroll
            for (int sw = 0; sw < RN_MAX_SWEEP; sw++) {
                int i = threadIdx.x + sw * RB_THREADS;
                if (i < c4) {
                    float4 v = ((const float4*)xr)[i], g = ((const float4*)gr)[i], s = ((const float4*)w)[i], o;
                    acc[sw * 4 + 0] += g.x * v.x * inv; acc[sw * 4 + 1] += g.y * v.y * inv;
                    acc[sw * 4 + 2] += g.z * v.z * inv; acc[sw * 4 + 3] += g.w * v.w * inv;
                    o.x = g.x * s.x * inv - v.x * k; o.y = g.y * s.y * inv - v.y * k;
                    o.z = g.z * s.z * inv - v.z * k; o.w = g.w * s.w * inv - v.w * k;
                    if (rr) { float4 q = ((const float4*)rr)[i]; o.x += q.x; o.y += q.y; o.z += q.z; o.w += q.w; }
                    ((float4*)dr)[i] = o;
                }
            }
        } else {
#pragma unroll
            for (int sw = 0; sw < RN_MAX_SWEEP * 4; sw++) {
                int i = threadIdx.x + sw * RB_THREADS;
                if (i < cols) {
                    float v = xr[i], g = gr[i];
                    acc[sw] += g * v * inv;
                    float o = g * w[i] * inv - v * k;
                    if (rr) o += rr[i];
                    dr[i] = o;
                }
            }
        }
    }
    float* pr = partial + (size_t)blockIdx.x * cols;
    if (vec) {
#pragma unroll
        for (int sw = 0; sw < RN_MAX_SWEEP; sw++) {
            int i = threadIdx.x + sw * RB_THREADS;
            if (i < c4) ((float4*)pr)[i] = make_float4(acc[sw * 4], acc[sw * 4 + 1], acc[sw * 4 + 2], acc[sw * 4 + 3]);
        }
    } else {
#pragma unroll
        for (int sw = 0; sw < RN_MAX_SWEEP * 4; sw++) { int i = threadIdx.x + sw * RB_THREADS; if (i < cols) pr[i] = acc[sw]; }
    }
}

// ---------------------------------------------------------------------------
// Warp-per-row variants for rows of up to 128*NV floats (cols % 4 == 0): the whole row lives in
// registers, every lane has NV independent 16-byte loads in flight, reductions are warp shuffles
// only, and the row is read from memory exactly once.
// ---------------------------------------------------------------------------
template <int NV>
__global__ void __launch_bounds__(RB_THREADS) rmsnorm_warp_kernel(const float* __restrict__ x, const float* __restrict__ w,
                                                                  float* __restrict__ y, float* __restrict__ copy, int rows, int cols, float eps, unsigned* amax_out, unsigned* inv_max) {
    sb_pdl_enter();
    const int lane = threadIdx.x & 31, warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
    const int c4 = cols >> 2;
    float am = 0.f, im = 0.f;
    for (int r = warp; r < rows; r += nwarps) {
        const float4* xr = (const float4*)(x + (size_t)r * cols);
        float4 v[NV];
        float ss = 0.f;
#pragma unroll
        for (int i = 0; i < NV; i++) {
            int j = lane + 32 * i;
            v[i] = j < c4 ? xr[j] : make_float4(0.f, 0.f, 0.f, 0.f);
            if (copy && j < c4) ((float4*)(copy + (size_t)r * cols))[j] = v[i];
            ss += v[i].x * v[i].x + v[i].y * v[i].y + v[i].z * v[i].z + v[i].w * v[i].w;
        }
        ss = warp_sum(ss);
        const float inv = 1.0f / sqrtf(ss / cols + eps);
        im = fmaxf(im, inv);
        float4* yr = (float4*)(y + (size_t)r * cols);
#pragma unroll
        for (int i = 0; i < NV; i++) {
            int j = lane + 32 * i;
            if (j < c4) {
                float4 s = ((const float4*)w)[j];
                const float4 o = make_float4(v[i].x * inv * s.x, v[i].y * inv * s.y, v[i].z * inv * s.z, v[i].w * inv * s.w);
                yr[j] = o;
                am = sb_amax4(am, o);
            }
        }
    }
    sb_block_amax(am, amax_out);
    if (inv_max && lane == 0 && im > 0.f) atomicMax(inv_max, __float_as_uint(im));
}

// Rows of exactly 128 columns (the learned per-head norm: rows = tokens x heads): one float4 per lane, four rows of a warp in
// flight together, so that a warp has 2 KB of loads outstanding instead of 512 bytes.
__global__ void __launch_bounds__(RB_THREADS) rmsnorm_w128_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ y,
                                                                  int rows, float eps, unsigned* amax_out) {
    sb_pdl_enter();
    const int lane = threadIdx.x & 31, warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
    const float4 s = ((const float4*)w)[lane];
    float am = 0.f;
    for (int r0 = warp * 4; r0 < rows; r0 += nwarps * 4) {
        float4 v[4];
#pragma unroll
        for (int i = 0; i < 4; i++) v[i] = r0 + i < rows ? ((const float4*)x)[(size_t)(r0 + i) * 32 + lane] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            if (r0 + i >= rows) break;
            const float ss = warp_sum(v[i].x * v[i].x + v[i].y * v[i].y + v[i].z * v[i].z + v[i].w * v[i].w);
            const float inv = 1.0f / sqrtf(ss / 128.f + eps);
            const float4 o = make_float4(v[i].x * inv * s.x, v[i].y * inv * s.y, v[i].z * inv * s.z, v[i].w * inv * s.w);
            ((float4*)y)[(size_t)(r0 + i) * 32 + lane] = o;
            am = sb_amax4(am, o);
        }
    }
    sb_block_amax(am, amax_out);
}

// RMSNorm backward for a 256-thread CTA that visits groups of ROWS rows.  Thread t owns the float4 column
// chunks t, t+256, ... (NC of them) of every row the CTA visits, so its dscale partial stays in NC float4
// registers.  The loads of the next group (x, dy, residual) are issued before the current group is reduced,
// so memory requests are in flight during the two CTA-wide reductions (sum x^2 and sum dy*w*x of each row);
// two CTAs share an SM.  One dscale partial row per CTA, summed in CTA order by colsum_partials_kernel.
// With RnbOut the result leaves as FP16 operand parts beside FP32, for the products that read the gradient next.  Its bound: with g = dy o w and
// xh = x / rms, dx = (g - xh mean(g o xh)) / rms + residual, |xh_i| <= sqrt(cols) and |mean(g o xh)| <= rms(g) <= max|g|, so
//   |dx| <= max|residual| + (1 + sqrt(cols)) max(1/rms) max|w| max|dy|.
// It is some 2^5 above the true maximum, which costs only values below 2^-13 of that maximum a part of their low halves (see sb_f16_shift).
struct RnbOut {
    uint2 *h1, *h2;                                   // NULL: only the bound is formed
    const float *amax_dy, *amax_resid, *inv_max;      // amax_resid NULL: no residual
    float* bound;                                     // NULL: neither parts nor bound
    unsigned keep;
};
template <int NC, int ROWS>
struct RnbSet { float4 v[ROWS][NC], g[ROWS][NC], q[ROWS][NC]; };

template <int NC, int ROWS>
__device__ __forceinline__ void rnb_load(RnbSet<NC, ROWS>& s, const float* __restrict__ x, const float* __restrict__ dy, const float* resid,
                                         int r0, int rows, int c4) {
#pragma unroll
    for (int rr = 0; rr < ROWS; rr++)
#pragma unroll
        for (int i = 0; i < NC; i++) {
            const int j = threadIdx.x + RB_THREADS * i;
            const bool in = r0 + rr < rows && j < c4;
            const size_t o = (size_t)(r0 + rr) * c4 + j;
            s.v[rr][i] = in ? ((const float4*)x)[o] : make_float4(0.f, 0.f, 0.f, 0.f);
            s.g[rr][i] = in ? ((const float4*)dy)[o] : make_float4(0.f, 0.f, 0.f, 0.f);
            s.q[rr][i] = (in && resid) ? ((const float4*)resid)[o] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
}

// the row's scales: in registers, or with four chunks a thread read from cache again where they are used (registers are what limits it)
template <int NC>
__device__ __forceinline__ float4 rnb_scale(const float4 (&scr)[NC], const float* __restrict__ w, int i, int c4) {
    if constexpr (NC < 4) return scr[i];
    const int j = threadIdx.x + RB_THREADS * i;
    return j < c4 ? __ldg((const float4*)w + j) : make_float4(0.f, 0.f, 0.f, 0.f);
}

template <int NC, int ROWS>
__device__ __forceinline__ void rnb_compute(const RnbSet<NC, ROWS>& s, const float4 (&scr)[NC], const float* __restrict__ w, float4 (&acc)[NC], float* dx, int r0, int rows,
                                            int cols, int c4, float eps, float (*s_red)[2 * ROWS], float* s_tot, float& am, const RnbOut& out, float osc) {
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    float part[2 * ROWS];
#pragma unroll
    for (int rr = 0; rr < ROWS; rr++) {
        float ss = 0.f, cp = 0.f;
#pragma unroll
        for (int i = 0; i < NC; i++) {
            const float4 v = s.v[rr][i], g = s.g[rr][i], sc = rnb_scale<NC>(scr, w, i, c4);
            ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
            cp += g.x * sc.x * v.x + g.y * sc.y * v.y + g.z * sc.z * v.z + g.w * sc.w * v.w;
        }
        part[2 * rr] = warp_sum(ss); part[2 * rr + 1] = warp_sum(cp);
    }
    if (lane == 0) {
#pragma unroll
        for (int k = 0; k < 2 * ROWS; k++) s_red[wib][k] = part[k];
    }
    __syncthreads();
    if (threadIdx.x < 2 * ROWS) {
        float t = 0.f;
#pragma unroll
        for (int wv = 0; wv < RB_THREADS / 32; wv++) t += s_red[wv][threadIdx.x];
        s_tot[threadIdx.x] = t;
    }
    __syncthreads();
#pragma unroll
    for (int rr = 0; rr < ROWS; rr++) {
        if (r0 + rr >= rows) break;
        const float inv = 1.0f / sqrtf(s_tot[2 * rr] / cols + eps);
        const float k = inv * inv * inv / cols * s_tot[2 * rr + 1];
#pragma unroll
        for (int i = 0; i < NC; i++) {
            const int j = threadIdx.x + RB_THREADS * i;
            if (j < c4) {
                const float4 v = s.v[rr][i], g = s.g[rr][i], q = s.q[rr][i], sc = rnb_scale<NC>(scr, w, i, c4);
                float4 o;
                acc[i].x += g.x * v.x * inv; acc[i].y += g.y * v.y * inv; acc[i].z += g.z * v.z * inv; acc[i].w += g.w * v.w * inv;
                o.x = g.x * sc.x * inv - v.x * k + q.x; o.y = g.y * sc.y * inv - v.y * k + q.y;
                o.z = g.z * sc.z * inv - v.z * k + q.z; o.w = g.w * sc.w * inv - v.w * k + q.w;
                ((float4*)dx)[(size_t)(r0 + rr) * c4 + j] = o;
                if (out.h1) {
                    uint2 hh, hl;
                    sb_split2(o.x * osc, o.y * osc, hh.x, hl.x, out.keep); sb_split2(o.z * osc, o.w * osc, hh.y, hl.y, out.keep);
                    out.h1[(size_t)(r0 + rr) * c4 + j] = hh; out.h2[(size_t)(r0 + rr) * c4 + j] = hl;
                }
                am = sb_amax4(am, o);
            }
        }
    }
}

template <int NC, int ROWS>
__global__ void __launch_bounds__(RB_THREADS, 2) rmsnorm_bwd_rows_kernel(const float* __restrict__ x, const float* __restrict__ w,
                                                                         const float* __restrict__ dy, const float* resid, float* dx,
                                                                         float* __restrict__ partial, int rows, int cols, float eps, unsigned* amax_dx, const RnbOut out) {
    sb_pdl_enter();
    float am = 0.f;
    __shared__ float s_red[2][RB_THREADS / 32][2 * ROWS];
    __shared__ float s_tot[2][2 * ROWS];
    __shared__ float s_w[RB_THREADS / 32];
    const int c4 = cols >> 2;
    float4 acc[NC], sc[NC];
#pragma unroll
    for (int i = 0; i < NC; i++) {
        acc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        const int j = threadIdx.x + RB_THREADS * i;
        sc[i] = j < c4 ? ((const float4*)w)[j] : acc[i];
    }
    const int ngroups = (rows + ROWS - 1) / ROWS, stride = gridDim.x;
    RnbSet<NC, ROWS> a, b;
    int gidx = blockIdx.x;
    if (gidx < ngroups) rnb_load<NC, ROWS>(a, x, dy, resid, gidx * ROWS, rows, c4);
    float osc = 1.f;
    if (out.bound) {
        float wm = 0.f;
#pragma unroll
        for (int i = 0; i < NC; i++) wm = sb_amax4(wm, sc[i]);
        wm = warp_max(wm);
        if ((threadIdx.x & 31) == 0) s_w[threadIdx.x >> 5] = wm;
        __syncthreads();
        wm = warp_max(s_w[threadIdx.x & (RB_THREADS / 32 - 1)]);
        const float bound = fminf((out.amax_resid ? sb_word(out.amax_resid) : 0.f) + 1.0001f * (1.f + sqrtf((float)cols)) * sb_word(out.inv_max) * wm * sb_word(out.amax_dy), 3.0e38f);
        osc = sb_pow2(sb_f16_shift(bound));
        if (blockIdx.x == 0 && threadIdx.x == 0) *out.bound = bound;
    }
    while (gidx < ngroups) {
        if (gidx + stride < ngroups) rnb_load<NC, ROWS>(b, x, dy, resid, (gidx + stride) * ROWS, rows, c4);
        rnb_compute<NC, ROWS>(a, sc, w, acc, dx, gidx * ROWS, rows, cols, c4, eps, s_red[0], s_tot[0], am, out, osc);
        gidx += stride;
        if (gidx >= ngroups) break;
        if (gidx + stride < ngroups) rnb_load<NC, ROWS>(a, x, dy, resid, (gidx + stride) * ROWS, rows, c4);
        rnb_compute<NC, ROWS>(b, sc, w, acc, dx, gidx * ROWS, rows, cols, c4, eps, s_red[1], s_tot[1], am, out, osc);
        gidx += stride;
    }
#pragma unroll
    for (int i = 0; i < NC; i++) {
        const int j = threadIdx.x + RB_THREADS * i;
        if (j < c4) ((float4*)(partial + (size_t)blockIdx.x * cols))[j] = acc[i];
    }
    sb_block_amax(am, amax_dx);
}

// Rows of up to 512 columns: a warp per row (4 vectors of x, dy, residual and scale per lane), so that all threads have work (in the kernel above a
// row of 512 columns occupies half of a CTA) and a row needs no CTA-wide sums; a warp's dscale partial stays in registers, the CTA adds its
// warps' in warp order.  From 512 rows up: fewer leave most SMs without a CTA (61 rows: 8 CTAs, 2 us a launch slower than two rows per CTA).
// 2048 x 512: 13 -> 11 us a launch, 5800 x 512: 19 -> 15.
template <int NV>
__global__ void __launch_bounds__(RB_THREADS, 2) rmsnorm_bwd_warp_kernel(const float* __restrict__ x, const float* __restrict__ w,
                                                                         const float* __restrict__ dy, const float* resid, float* dx,
                                                                         float* __restrict__ partial, int rows, int cols, float eps, unsigned* amax_dx, const RnbOut out) {
    sb_pdl_enter();
    __shared__ float4 s_acc[RB_THREADS / 32][32 * NV];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, c4 = cols >> 2, stride = gridDim.x * (RB_THREADS / 32);
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 acc[NV], v[NV], g[NV], q[NV];
    auto load = [&](int r) {
        const size_t o0 = (size_t)r * c4;
#pragma unroll
        for (int i = 0; i < NV; i++) {
            const int j = lane + 32 * i;
            const bool in = j < c4;
            v[i] = in ? ((const float4*)x)[o0 + j] : zero;
            g[i] = in ? ((const float4*)dy)[o0 + j] : zero;
            q[i] = in && resid ? ((const float4*)resid)[o0 + j] : zero;
        }
    };
    const int r0 = blockIdx.x * (RB_THREADS / 32) + wib;
    if (r0 < rows) load(r0);              // on its way while the scales and the words are looked at
    float wm = 0.f, am = 0.f;
#pragma unroll
    for (int i = 0; i < NV; i++) {
        const int j = lane + 32 * i;
        acc[i] = zero;
        wm = sb_amax4(wm, j < c4 ? ((const float4*)w)[j] : zero);      // (read again from cache below)
    }
    float osc = 1.f;
    if (out.bound) {
        wm = warp_max(wm);
        const float bound = fminf((out.amax_resid ? sb_word(out.amax_resid) : 0.f) + 1.0001f * (1.f + sqrtf((float)cols)) * sb_word(out.inv_max) * wm * sb_word(out.amax_dy), 3.0e38f);
        osc = sb_pow2(sb_f16_shift(bound));
        if (blockIdx.x == 0 && threadIdx.x == 0) *out.bound = bound;
    }
    for (int r = r0; r < rows; r += stride) {
        const size_t o0 = (size_t)r * c4;
        if (r != r0) load(r);
        float ss = 0.f, cp = 0.f;
        float4 sc[NV];
#pragma unroll
        for (int i = 0; i < NV; i++) {
            sc[i] = lane + 32 * i < c4 ? __ldg((const float4*)w + lane + 32 * i) : zero;
            ss += v[i].x * v[i].x + v[i].y * v[i].y + v[i].z * v[i].z + v[i].w * v[i].w;
            cp += g[i].x * sc[i].x * v[i].x + g[i].y * sc[i].y * v[i].y + g[i].z * sc[i].z * v[i].z + g[i].w * sc[i].w * v[i].w;
        }
        ss = warp_sum(ss); cp = warp_sum(cp);
        const float inv = 1.0f / sqrtf(ss / cols + eps), k = inv * inv * inv / cols * cp;
#pragma unroll
        for (int i = 0; i < NV; i++) {
            const int j = lane + 32 * i;
            if (j >= c4) continue;
            acc[i].x += g[i].x * v[i].x * inv; acc[i].y += g[i].y * v[i].y * inv; acc[i].z += g[i].z * v[i].z * inv; acc[i].w += g[i].w * v[i].w * inv;
            float4 o;
            o.x = g[i].x * sc[i].x * inv - v[i].x * k + q[i].x; o.y = g[i].y * sc[i].y * inv - v[i].y * k + q[i].y;
            o.z = g[i].z * sc[i].z * inv - v[i].z * k + q[i].z; o.w = g[i].w * sc[i].w * inv - v[i].w * k + q[i].w;
            ((float4*)dx)[o0 + j] = o;
            am = sb_amax4(am, o);
            if (out.h1) {
                uint2 hh, hl;
                sb_split2(o.x * osc, o.y * osc, hh.x, hl.x, out.keep); sb_split2(o.z * osc, o.w * osc, hh.y, hl.y, out.keep);
                out.h1[o0 + j] = hh; out.h2[o0 + j] = hl;
            }
        }
    }
#pragma unroll
    for (int i = 0; i < NV; i++) s_acc[wib][lane + 32 * i] = acc[i];
    __syncthreads();
    for (int j = threadIdx.x; j < c4; j += RB_THREADS) {
        float4 t = s_acc[0][j];
#pragma unroll
        for (int k = 1; k < RB_THREADS / 32; k++) { const float4 u = s_acc[k][j]; t.x += u.x; t.y += u.y; t.z += u.z; t.w += u.w; }
        ((float4*)(partial + (size_t)blockIdx.x * cols))[j] = t;
    }
    sb_block_amax(am, amax_dx);
}

// RMSNorm backward for rows of exactly 128 columns (the learned per-head norm of q and k: rows = tokens x heads): one warp per
// row, a float4 per lane, four rows in flight per warp; no CTA-wide reduction per row.  A lane's dscale partial stays in a
// float4 over all rows its warp visits; the warps of a CTA add theirs in warp order into one partial row per CTA.
__global__ void __launch_bounds__(RB_THREADS, 4) rmsnorm_bwd_w128_kernel(const float* __restrict__ x, const float* __restrict__ w,
                                                                         const float* __restrict__ dy, const float* resid, float* dx,
                                                                         float* __restrict__ partial, int rows, float eps, unsigned* amax_dx) {
    sb_pdl_enter();
    __shared__ float4 s_acc[RB_THREADS / 32][32];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, nw = (gridDim.x * RB_THREADS) >> 5;
    const float4 sc = ((const float4*)w)[lane];
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    float am = 0.f;
    for (int r0 = (blockIdx.x * (RB_THREADS / 32) + wib) * 4; r0 < rows; r0 += nw * 4) {
        float4 v[4], g[4], q[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const bool in = r0 + i < rows;
            const size_t o = (size_t)(r0 + i) * 32 + lane;
            v[i] = in ? ((const float4*)x)[o] : make_float4(0.f, 0.f, 0.f, 0.f);
            g[i] = in ? ((const float4*)dy)[o] : make_float4(0.f, 0.f, 0.f, 0.f);
            q[i] = (in && resid) ? ((const float4*)resid)[o] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            if (r0 + i >= rows) break;
            float ss = v[i].x * v[i].x + v[i].y * v[i].y + v[i].z * v[i].z + v[i].w * v[i].w;
            float cp = g[i].x * sc.x * v[i].x + g[i].y * sc.y * v[i].y + g[i].z * sc.z * v[i].z + g[i].w * sc.w * v[i].w;
            ss = warp_sum(ss); cp = warp_sum(cp);
            const float inv = 1.0f / sqrtf(ss / 128.f + eps);
            const float k = inv * inv * inv / 128.f * cp;
            acc.x += g[i].x * v[i].x * inv; acc.y += g[i].y * v[i].y * inv; acc.z += g[i].z * v[i].z * inv; acc.w += g[i].w * v[i].w * inv;
            float4 o;
            o.x = g[i].x * sc.x * inv - v[i].x * k + q[i].x; o.y = g[i].y * sc.y * inv - v[i].y * k + q[i].y;
            o.z = g[i].z * sc.z * inv - v[i].z * k + q[i].z; o.w = g[i].w * sc.w * inv - v[i].w * k + q[i].w;
            ((float4*)dx)[(size_t)(r0 + i) * 32 + lane] = o;
            am = sb_amax4(am, o);
        }
    }
    s_acc[wib][lane] = acc;
    __syncthreads();
    if (wib == 0) {
        float4 t = s_acc[0][lane];
#pragma unroll
        for (int k = 1; k < RB_THREADS / 32; k++) { const float4 u = s_acc[k][lane]; t.x += u.x; t.y += u.y; t.z += u.z; t.w += u.w; }
        ((float4*)(partial + (size_t)blockIdx.x * 128))[lane] = t;
    }
    sb_block_amax(am, amax_dx);
}

// dscale[c] += sum over partial rows of partial[b][c], in a fixed order: 32 columns per CTA, the rows dealt to
// 32 row groups (group g takes rows g, g+32, ...; ten independent loads are in flight per thread), the 32 group
// sums then added in group order.
#define CS_GROUPS 32
#define CS_BATCH 10
#define CS_TAB 64
struct CsEntry { const float* partial; float* dscale; int nblocks, cols; };
struct CsTab { int store; CsEntry e[CS_TAB]; };      // blockIdx.y = entry; store: dscale is written, not added to
__global__ void __launch_bounds__(32 * CS_GROUPS) colsum_partials_kernel(const __grid_constant__ CsTab tab) {
    sb_pdl_enter();
    const float* __restrict__ partial = tab.e[blockIdx.y].partial; float* __restrict__ dscale = tab.e[blockIdx.y].dscale;
    const int nblocks = tab.e[blockIdx.y].nblocks, cols = tab.e[blockIdx.y].cols;
    if ((int)blockIdx.x * 32 >= cols) return;
    __shared__ float s_part[CS_GROUPS][33];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int cidx = blockIdx.x * 32 + tx;
    float s = 0.f;
    if (cidx < cols) {
        for (int b0 = ty; b0 < nblocks; b0 += CS_GROUPS * CS_BATCH) {
            float v[CS_BATCH];
#pragma unroll
            for (int i = 0; i < CS_BATCH; i++) {
                const int b = b0 + i * CS_GROUPS;
                v[i] = b < nblocks ? partial[(size_t)b * cols + cidx] : 0.f;
            }
#pragma unroll
            for (int i = 0; i < CS_BATCH; i++) s += v[i];
        }
    }
    s_part[ty][tx] = s;
    __syncthreads();
    if (ty == 0 && cidx < cols) {
        float t = s_part[0][tx];
#pragma unroll
        for (int g = 1; g < CS_GROUPS; g++) t += s_part[g][tx];
        dscale[cidx] = tab.store ? t : dscale[cidx] + t;
    }
}

// ---------------------------------------------------------------------------
// Row softmax (kept for API completeness; no training step uses it)
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(RB_THREADS) softmax_kernel(const float* __restrict__ x, float* __restrict__ y, int rows, int cols) {
    sb_pdl_enter();
    __shared__ float red[64];
    for (int r = blockIdx.x; r < rows; r += gridDim.x) {
        const float* xr = x + (size_t)r * cols; float* yr = y + (size_t)r * cols;
        float m = -INFINITY;
        for (int i = threadIdx.x; i < cols; i += blockDim.x) m = fmaxf(m, xr[i]);
        m = warp_max(m);
        __syncthreads();
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
        __syncthreads();
        m = -INFINITY;
        for (int i = 0; i < (blockDim.x + 31) / 32; i++) m = fmaxf(m, red[i]);
        float s = 0.f, d0 = 0.f;
        for (int i = threadIdx.x; i < cols; i += blockDim.x) s += expf(xr[i] - m);
        block_sum2(s, d0, red);
        float inv = 1.0f / s;
        for (int i = threadIdx.x; i < cols; i += blockDim.x) yr[i] = expf(xr[i] - m) * inv;
    }
}

// ---------------------------------------------------------------------------
// Q/K normalisation over the whole token row (all heads): y = x / max(sqrt(mean(x^2)), eps), in place
// (shaders/qk_norm.comp:30-76; the CUDA backend of the reference does not have it), and its backward, which the
// reference lacks: r > eps: dx = (dy - y * mean(dy o y)) / r;  clamp active: dx = dy / eps.  The forward keeps r per
// row because it overwrites x.  One warp per row, the row in registers (cols % 4 == 0, cols <= 128 * NV): 8 bytes
// per element forward, 12 backward.  Other shapes: one CTA per row.
// ---------------------------------------------------------------------------
// RMSNorm of rows of 1028 to 4096 columns: a CTA per row, NC vectors of it per thread, the next row's loads in flight during this row's sum.  (A warp
// per row needs 64 to 128 registers for the row alone, one or two CTAs per SM: 2.0 to 3.3 TB/s at 2048 and 4096 columns.)  The row leaves as FP32
// (y) or as FP16 operand parts under the bound that rmsnorm_warp_parts_kernel explains; copy, inv_max and amax_out as there.
template <int NC>
__global__ void __launch_bounds__(RB_THREADS, 4) rmsnorm_rows_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ y,
                                                                     uint2* __restrict__ h1, uint2* __restrict__ h2, float* __restrict__ copy, int rows, int cols, float eps,
                                                                     float* bound_out, unsigned keep, unsigned* inv_max, unsigned* amax_out) {
    sb_pdl_enter();
    __shared__ float red[2][RB_THREADS / 32], s_w[RB_THREADS / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c4 = cols >> 2;
    float4 s[NC], v[NC], nx[NC];
    int r = blockIdx.x;
#pragma unroll
    for (int i = 0; i < NC; i++) {
        const int j = threadIdx.x + RB_THREADS * i;
        s[i] = j < c4 ? ((const float4*)w)[j] : make_float4(0.f, 0.f, 0.f, 0.f);
        v[i] = j < c4 && r < rows ? ((const float4*)x)[(size_t)r * c4 + j] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    float sc = 1.f, im = 0.f, am = 0.f;
    if (bound_out) {
        float wm = 0.f;
#pragma unroll
        for (int i = 0; i < NC; i++) wm = sb_amax4(wm, s[i]);
        wm = warp_max(wm);
        if (lane == 0) s_w[warp] = wm;
        __syncthreads();
        wm = warp_max(s_w[threadIdx.x & (RB_THREADS / 32 - 1)]);
        const float bound = fminf(sqrtf((float)cols) * wm * 1.0001f, 3.0e38f);
        sc = sb_pow2(sb_f16_shift(bound));
        if (blockIdx.x == 0 && threadIdx.x == 0) *bound_out = bound;
    }
    for (int it = 0; r < rows; r += gridDim.x, it++) {
        const int rn = r + gridDim.x;
        float ss = 0.f;
#pragma unroll
        for (int i = 0; i < NC; i++) {
            const int j = threadIdx.x + RB_THREADS * i;
            if (j < c4 && rn < rows) nx[i] = ((const float4*)x)[(size_t)rn * c4 + j];
            ss += v[i].x * v[i].x + v[i].y * v[i].y + v[i].z * v[i].z + v[i].w * v[i].w;
        }
        ss = warp_sum(ss);
        if (lane == 0) red[it & 1][warp] = ss;
        __syncthreads();                        // the other half of red is written next: one barrier a row is enough
        ss = red[it & 1][0];
#pragma unroll
        for (int k = 1; k < RB_THREADS / 32; k++) ss += red[it & 1][k];
        const float inv = 1.0f / sqrtf(ss / cols + eps);
        im = fmaxf(im, inv);
#pragma unroll
        for (int i = 0; i < NC; i++) {
            const int j = threadIdx.x + RB_THREADS * i;
            if (j < c4) {
                const size_t o = (size_t)r * c4 + j;
                if (copy) ((float4*)copy)[o] = v[i];
                const float4 q = make_float4(v[i].x * inv * s[i].x, v[i].y * inv * s[i].y, v[i].z * inv * s[i].z, v[i].w * inv * s[i].w);
                if (h1) {
                    uint2 a, b;
                    sb_split2(q.x * sc, q.y * sc, a.x, b.x, keep); sb_split2(q.z * sc, q.w * sc, a.y, b.y, keep);
                    h1[o] = a; h2[o] = b;
                } else {
                    ((float4*)y)[o] = q;
                    am = sb_amax4(am, q);
                }
                v[i] = nx[i];
            }
        }
    }
    if (inv_max && threadIdx.x == 0 && im > 0.f) atomicMax(inv_max, __float_as_uint(im));
    sb_block_amax(am, amax_out);
}

// The same rows with y written only as FP16 operand parts: every |y_i| = |x_i| rstd |w_i| is at most sqrt(cols) max|w| (x_i^2 cannot
// exceed the row's sum of squares), so that bound sets the scale and no pass over y looks for its maximum or splits it again.
template <int NV>
__global__ void __launch_bounds__(RB_THREADS) rmsnorm_warp_parts_kernel(const float* __restrict__ x, const float* __restrict__ w,
                                                                        float* __restrict__ y, uint2* __restrict__ h1, uint2* __restrict__ h2, int rows, int cols, float eps,
                                                                        float* __restrict__ bound_out, unsigned keep, float* __restrict__ copy, unsigned* inv_max) {
    sb_pdl_enter();
    constexpr bool KEEP = NV <= 4;        // the scales stay in registers; wider rows read them again from cache
    const int lane = threadIdx.x & 31, warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
    const int c4 = cols >> 2;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 v[NV], s[KEEP ? NV : 1];
    auto load = [&](int r) {
        const float4* xr = (const float4*)(x + (size_t)r * cols);
#pragma unroll
        for (int i = 0; i < NV; i++) v[i] = lane + 32 * i < c4 ? xr[lane + 32 * i] : zero;
    };
    if (warp < rows) load(warp);          // on its way while the scales are looked at
    float wm = 0.f;
#pragma unroll
    for (int i = 0; i < NV; i++) {
        const int j = lane + 32 * i;
        const float4 q = j < c4 ? ((const float4*)w)[j] : zero;
        if constexpr (KEEP) s[i] = q;
        wm = sb_amax4(wm, q);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) wm = fmaxf(wm, __shfl_xor_sync(0xffffffffu, wm, o));
    const float bound = fminf(sqrtf((float)cols) * wm * 1.0001f, 3.0e38f);
    const float sc = sb_pow2(sb_f16_shift(bound));
    if (warp == 0 && lane == 0) *bound_out = bound;
    float im = 0.f;
    for (int r = warp; r < rows; r += nwarps) {
        if (r != warp) load(r);
        float ss = 0.f;
#pragma unroll
        for (int i = 0; i < NV; i++) {
            const int j = lane + 32 * i;
            if (copy && j < c4) ((float4*)(copy + (size_t)r * cols))[j] = v[i];
            ss += v[i].x * v[i].x + v[i].y * v[i].y + v[i].z * v[i].z + v[i].w * v[i].w;
        }
        ss = warp_sum(ss);
        const float inv = 1.0f / sqrtf(ss / cols + eps);
        im = fmaxf(im, inv);
        uint2* o1 = h1 + (size_t)r * c4; uint2* o2 = h2 + (size_t)r * c4;
#pragma unroll
        for (int i = 0; i < NV; i++) {
            int j = lane + 32 * i;
            if (j < c4) {
                // the FP32 value first, exactly as the plain kernel forms it, then the scale (a power of two: exact)
                const float4 q = KEEP ? s[KEEP ? i : 0] : ((const float4*)w)[j];
                const float y0 = v[i].x * inv * q.x, y1 = v[i].y * inv * q.y, y2 = v[i].z * inv * q.z, y3 = v[i].w * inv * q.w;
                if (y) { ((float4*)(y + (size_t)r * cols))[j] = make_float4(y0, y1, y2, y3); continue; }      // no arena for the parts
                uint2 a, b;
                sb_split2(y0 * sc, y1 * sc, a.x, b.x, keep); sb_split2(y2 * sc, y3 * sc, a.y, b.y, keep);
                o1[j] = a; o2[j] = b;
            }
        }
    }
    sb_block_amax(im, inv_max);           // (a word that all warps raise one by one: 5800 of them took longer than the rows)
}
template <int NV>
__global__ void __launch_bounds__(RB_THREADS) qk_norm_warp_kernel(float* __restrict__ x, float* __restrict__ rms_out, int rows, int cols, float eps) {
    sb_pdl_enter();
    const int lane = threadIdx.x & 31, warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
    const int c4 = cols >> 2;
    for (int r = warp; r < rows; r += nwarps) {
        float4* xr = (float4*)(x + (size_t)r * cols);
        float4 v[NV];
        float ss = 0.f;
#pragma unroll
        for (int i = 0; i < NV; i++) {
            const int j = lane + 32 * i;
            v[i] = j < c4 ? xr[j] : make_float4(0.f, 0.f, 0.f, 0.f);
            ss += v[i].x * v[i].x + v[i].y * v[i].y + v[i].z * v[i].z + v[i].w * v[i].w;
        }
        ss = warp_sum(ss);
        const float rms = sqrtf(ss / cols);
        if (lane == 0 && rms_out) rms_out[r] = rms;
        const float inv = 1.0f / fmaxf(rms, eps);
#pragma unroll
        for (int i = 0; i < NV; i++) {
            const int j = lane + 32 * i;
            if (j < c4) xr[j] = make_float4(v[i].x * inv, v[i].y * inv, v[i].z * inv, v[i].w * inv);
        }
    }
}
template <int NV>
__global__ void __launch_bounds__(RB_THREADS) qk_norm_bwd_warp_kernel(const float* __restrict__ y, const float* __restrict__ rms,
                                                                      const float* dy, float* dx, int rows, int cols, float eps) {
    sb_pdl_enter();
    const int lane = threadIdx.x & 31, warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
    const int c4 = cols >> 2;
    for (int r = warp; r < rows; r += nwarps) {
        const float4* yr = (const float4*)(y + (size_t)r * cols);
        const float4* gr = (const float4*)(dy + (size_t)r * cols);
        float4 v[NV], g[NV];
        float dot = 0.f;
#pragma unroll
        for (int i = 0; i < NV; i++) {
            const int j = lane + 32 * i;
            v[i] = j < c4 ? yr[j] : make_float4(0.f, 0.f, 0.f, 0.f);
            g[i] = j < c4 ? gr[j] : make_float4(0.f, 0.f, 0.f, 0.f);
            dot += v[i].x * g[i].x + v[i].y * g[i].y + v[i].z * g[i].z + v[i].w * g[i].w;
        }
        dot = warp_sum(dot);
        const float rr = rms[r];
        const bool live = rr > eps;
        const float m = live ? dot / cols : 0.f, inv = 1.0f / (live ? rr : eps);
        float4* o = (float4*)(dx + (size_t)r * cols);
#pragma unroll
        for (int i = 0; i < NV; i++) {
            const int j = lane + 32 * i;
            if (j < c4) o[j] = make_float4((g[i].x - v[i].x * m) * inv, (g[i].y - v[i].y * m) * inv, (g[i].z - v[i].z * m) * inv, (g[i].w - v[i].w * m) * inv);
        }
    }
}
// any shape: one CTA per row, two passes over the row
__global__ void __launch_bounds__(RB_THREADS) qk_norm_row_kernel(float* __restrict__ x, float* __restrict__ rms_out, const float* __restrict__ rms_in,
                                                                 const float* dy, float* dx, int rows, int cols, float eps) {
    sb_pdl_enter();
    __shared__ float red[RB_THREADS / 32];
    __shared__ float tot;
    for (int r = blockIdx.x; r < rows; r += gridDim.x) {
        // forward (dy == NULL): sum of x^2; backward: sum of dy*y (x then holds y)
        const float* a = x + (size_t)r * cols; const float* b = dy ? dy + (size_t)r * cols : a;
        float s = 0.f;
        for (int i = threadIdx.x; i < cols; i += blockDim.x) s += a[i] * b[i];
        s = warp_sum(s);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
        __syncthreads();
        if (threadIdx.x == 0) { float t = 0.f; for (int w = 0; w < RB_THREADS / 32; w++) t += red[w]; tot = t; }
        __syncthreads();
        if (!dy) {
            const float rms = sqrtf(tot / cols), inv = 1.0f / fmaxf(rms, eps);
            if (threadIdx.x == 0 && rms_out) rms_out[r] = rms;
            for (int i = threadIdx.x; i < cols; i += blockDim.x) x[(size_t)r * cols + i] = a[i] * inv;
        } else {
            const float rr = rms_in[r];
            const bool live = rr > eps;
            const float m = live ? tot / cols : 0.f, inv = 1.0f / (live ? rr : eps);
            for (int i = threadIdx.x; i < cols; i += blockDim.x) dx[(size_t)r * cols + i] = (b[i] - a[i] * m) * inv;
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// Cross-entropy loss and gradient, packed.
//   last token of a sequence -> zero row and zero loss
//   loss = -(logit[target] - max - log(sum));  grad = (softmax - onehot)/num_valid
// A cluster of CL CTAs holds one row of logits in shared memory, a slice of V / CL each: every logit is read once and exponentiated once, and
// the maximum and the sum of the row are exchanged through distributed shared memory.  8 bytes per logit (4 when no gradient is asked for).
// (An online maximum and sum, then a second read for the gradient: 12 bytes and two or more exponentials per logit.)
// The gradient leaves as FP32 (`grad`), or as the two FP16 parts the LM-head backward products read (g1: h1 = fp16(g * part_scale),
// h2 = fp16(g * part_scale - h1), laid out like grad): |g| <= inv_valid everywhere (softmax minus one-hot, over the number of predictions),
// so the parts' scale is known before a single logit is read, *part_amax = inv_valid; or, both NULL, not at all.
// ---------------------------------------------------------------------------
#define CE_THREADS 512
struct CeArgs {
    const float* logits; const uint32_t* targets; float *grad, *loss_rows;
    const uint32_t *pos_ids, *seq_ids, *seq_starts;
    int T, V; float inv_valid; int* status; unsigned* amax_grad;
    __half *g1, *g2; float part_scale; float* part_amax; unsigned keep;
};
// the CTAs of a cluster combine one value each: v of rank i lands in slot[i] of every CTA
template <int CL>
__device__ __forceinline__ void ce_exchange(float* slot, float v) {
    if (CL == 1) { if (threadIdx.x == 0) slot[0] = v; __syncthreads(); return; }
    if (threadIdx.x < CL) {
        uint32_t rank, a;
        asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(slot + rank)), "r"((uint32_t)threadIdx.x));
        asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
    }
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
template <int CL>
__global__ void __launch_bounds__(CE_THREADS) cross_entropy_kernel(const __grid_constant__ CeArgs p) {
    sb_pdl_enter();
    extern __shared__ float4 row[];
    __shared__ float red[CE_THREADS / 32], smax[CL], ssum[CL];
    const int r = blockIdx.x / CL, rank = blockIdx.x % CL, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n4 = p.V / 4, per = (n4 + CL - 1) / CL, lo = min(n4, rank * per), n = min(n4, lo + per) - lo;
    const float4* lr = (const float4*)(p.logits + (size_t)r * p.V) + lo;
    const size_t out = (size_t)r * n4 + lo;
    float4* gr = p.grad ? (float4*)p.grad + out : nullptr;
    uint2* p1 = p.g1 ? (uint2*)p.g1 + out : nullptr; uint2* p2 = p.g1 ? (uint2*)p.g2 + out : nullptr;
    if (p.part_amax && blockIdx.x == 0 && threadIdx.x == 0) *p.part_amax = p.inv_valid;
    const uint32_t s = p.seq_ids[r];
    if ((int)p.pos_ids[r] >= (int)(p.seq_starts[s + 1] - p.seq_starts[s]) - 1) {
        for (int i = threadIdx.x; i < n; i += CE_THREADS) {
            if (p1) { p1[i] = make_uint2(0u, 0u); p2[i] = make_uint2(0u, 0u); }
            else if (gr) gr[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        if (rank == 0 && threadIdx.x == 0) p.loss_rows[r] = 0.f;
        return;
    }
    uint32_t tg = p.targets[r];
    if (tg >= (uint32_t)p.V) { if (threadIdx.x == 0) atomicExch(p.status, SB_ERR_TOKEN_RANGE); tg = 0; }
    const float lt = p.logits[(size_t)r * p.V + tg];        // (grad may be the same array as logits)
    if (CL > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    float m = -INFINITY;
    for (int i0 = threadIdx.x; i0 < n; i0 += 4 * CE_THREADS) {
        float4 v[4];
#pragma unroll
        for (int u = 0; u < 4; u++) if (i0 + u * CE_THREADS < n) v[u] = __ldcs(lr + i0 + u * CE_THREADS);
#pragma unroll
        for (int u = 0; u < 4; u++) if (i0 + u * CE_THREADS < n) {
            row[i0 + u * CE_THREADS] = v[u];
            m = fmaxf(m, fmaxf(fmaxf(v[u].x, v[u].y), fmaxf(v[u].z, v[u].w)));
        }
    }
    m = warp_max(m);
    if (lane == 0) red[warp] = m;
    __syncthreads();
    m = warp_max(red[lane & (CE_THREADS / 32 - 1)]);
    if (CL > 1) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");      // every CTA of the cluster is running: its shared memory may be written
    ce_exchange<CL>(smax, m);
    m = smax[0];
#pragma unroll
    for (int i = 1; i < CL; i++) m = fmaxf(m, smax[i]);
    float sum = 0.f;
    for (int i = threadIdx.x; i < n; i += CE_THREADS) {     // a thread reads back what it stored itself
        float4 v = row[i];
        v.x = expf(v.x - m); v.y = expf(v.y - m); v.z = expf(v.z - m); v.w = expf(v.w - m);
        row[i] = v;
        sum += (v.x + v.y) + (v.z + v.w);
    }
    sum = warp_sum(sum);
    __syncthreads();                                        // red has been read
    if (lane == 0) red[warp] = sum;
    __syncthreads();
    sum = red[0];
#pragma unroll
    for (int i = 1; i < CE_THREADS / 32; i++) sum += red[i];
    ce_exchange<CL>(ssum, sum);
    sum = ssum[0];
#pragma unroll
    for (int i = 1; i < CL; i++) sum += ssum[i];
    if (rank == 0 && threadIdx.x == 0) p.loss_rows[r] = -((lt - m) - logf(sum));
    if (!p1 && !gr) return;
    const float inv = 1.0f / sum;
    float am = 0.f;
    for (int i = threadIdx.x; i < n; i += CE_THREADS) {
        float4 g = row[i];
        g.x *= inv; g.y *= inv; g.z *= inv; g.w *= inv;
        const uint32_t b = (uint32_t)(lo + i) * 4;
        if (tg - b < 4u) { if (tg == b) g.x -= 1.f; else if (tg == b + 1) g.y -= 1.f; else if (tg == b + 2) g.z -= 1.f; else g.w -= 1.f; }
        g.x *= p.inv_valid; g.y *= p.inv_valid; g.z *= p.inv_valid; g.w *= p.inv_valid;
        if (p1) {
            uint2 h, l;
            sb_split2(g.x * p.part_scale, g.y * p.part_scale, h.x, l.x, p.keep); sb_split2(g.z * p.part_scale, g.w * p.part_scale, h.y, l.y, p.keep);
            p1[i] = h; p2[i] = l;
        } else {
            gr[i] = g;
            am = sb_amax4(am, g);
        }
    }
    sb_block_amax(am, p.amax_grad);
}

// Rows too long for that (a vocabulary of 152k is 608 KB a row): one CTA of 1024 threads per row and SM, an online (max, sum) pass in batches of 16
// logits (one comparison and at most one rescaling each), then the gradient pass from the end of the row backwards, which finds what the rows in
// flight (148 x 608 KB) still have in L2.  (Clusters of 8 and 16 CTAs with slices in shared memory read each logit once, but their phases and
// the cluster's launch leave memory idle: 3.3 and 4.1 ms at 8192 x 151936, against 2.85 here and 2.96 for an
// online pass of 512 threads that compared every logit.)
#define CE_LONG 1024
__global__ void __launch_bounds__(CE_LONG, 1) cross_entropy_long_kernel(const __grid_constant__ CeArgs p) {
    sb_pdl_enter();
    __shared__ float redm[32], reds[32];
    const int r = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n = p.V / 4;
    const float4* lr = (const float4*)(p.logits + (size_t)r * p.V);
    const size_t out = (size_t)r * n;
    float4* gr = p.grad ? (float4*)p.grad + out : nullptr;
    uint2* p1 = p.g1 ? (uint2*)p.g1 + out : nullptr; uint2* p2 = p.g1 ? (uint2*)p.g2 + out : nullptr;
    if (p.part_amax && r == 0 && threadIdx.x == 0) *p.part_amax = p.inv_valid;
    const uint32_t s = p.seq_ids[r];
    if ((int)p.pos_ids[r] >= (int)(p.seq_starts[s + 1] - p.seq_starts[s]) - 1) {
        for (int i = threadIdx.x; i < n; i += CE_LONG) {
            if (p1) { p1[i] = make_uint2(0u, 0u); p2[i] = make_uint2(0u, 0u); }
            else if (gr) gr[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        if (threadIdx.x == 0) p.loss_rows[r] = 0.f;
        return;
    }
    uint32_t tg = p.targets[r];
    if (tg >= (uint32_t)p.V) { if (threadIdx.x == 0) atomicExch(p.status, SB_ERR_TOKEN_RANGE); tg = 0; }
    const float lt = p.logits[(size_t)r * p.V + tg];
    float m = -INFINITY, sum = 0.f;
    for (int i0 = threadIdx.x; i0 < n; i0 += 4 * CE_LONG) {
        float4 v[4];
#pragma unroll
        for (int u = 0; u < 4; u++) v[u] = i0 + u * CE_LONG < n ? lr[i0 + u * CE_LONG] : make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
        float bm = -INFINITY;
#pragma unroll
        for (int u = 0; u < 4; u++) bm = fmaxf(bm, fmaxf(fmaxf(v[u].x, v[u].y), fmaxf(v[u].z, v[u].w)));
        if (bm > m) { sum = m == -INFINITY ? sum : sum * expf(m - bm); m = bm; }
#pragma unroll
        for (int u = 0; u < 4; u++) if (i0 + u * CE_LONG < n) sum += (expf(v[u].x - m) + expf(v[u].y - m)) + (expf(v[u].z - m) + expf(v[u].w - m));
    }
    float wm = warp_max(m);
    sum = warp_sum(m == -INFINITY ? sum : sum * expf(m - wm));
    if (lane == 0) { redm[warp] = wm; reds[warp] = sum; }
    __syncthreads();
    m = warp_max(redm[lane]);
    sum = warp_sum(redm[lane] == -INFINITY ? reds[lane] : reds[lane] * expf(redm[lane] - m));
    if (threadIdx.x == 0) p.loss_rows[r] = -((lt - m) - logf(sum));
    if (!p1 && !gr) return;
    const float inv = 1.0f / sum;
    float am = 0.f;
    auto grad_of = [&](int i, float4 g) {
        g.x = expf(g.x - m) * inv; g.y = expf(g.y - m) * inv; g.z = expf(g.z - m) * inv; g.w = expf(g.w - m) * inv;
        const uint32_t b = (uint32_t)i * 4;
        if (tg - b < 4u) { if (tg == b) g.x -= 1.f; else if (tg == b + 1) g.y -= 1.f; else if (tg == b + 2) g.z -= 1.f; else g.w -= 1.f; }
        g.x *= p.inv_valid; g.y *= p.inv_valid; g.z *= p.inv_valid; g.w *= p.inv_valid;
        if (p1) {
            uint2 h, l;
            sb_split2(g.x * p.part_scale, g.y * p.part_scale, h.x, l.x, p.keep); sb_split2(g.z * p.part_scale, g.w * p.part_scale, h.y, l.y, p.keep);
            __stcs(p1 + i, h); __stcs(p2 + i, l);
        } else {
            gr[i] = g;
            am = sb_amax4(am, g);
        }
    };
    for (int j0 = threadIdx.x; j0 < n; j0 += 4 * CE_LONG) {
        float4 v[4];
#pragma unroll
        for (int u = 0; u < 4; u++) if (j0 + u * CE_LONG < n) v[u] = __ldcs(lr + (n - 1 - j0 - u * CE_LONG));
#pragma unroll
        for (int u = 0; u < 4; u++) if (j0 + u * CE_LONG < n) grad_of(n - 1 - j0 - u * CE_LONG, v[u]);
    }
    sb_block_amax(am, p.amax_grad);
}

// rows that are not a multiple of four logits or not aligned: one CTA per row, an online (max, sum) pass over the
// logits, then one pass that writes the gradient
__global__ void __launch_bounds__(CE_THREADS) cross_entropy_any_kernel(const float* __restrict__ logits, const uint32_t* __restrict__ targets,
                                                                   float* __restrict__ grad, float* __restrict__ loss_rows,
                                                                   const uint32_t* __restrict__ pos_ids, const uint32_t* __restrict__ seq_ids,
                                                                   const uint32_t* __restrict__ seq_starts,
                                                                   int T, int V, float inv_valid, int* status, unsigned* amax_grad) {
    sb_pdl_enter();
    __shared__ float redm[32], reds[32];
    float am = 0.f;
    int r = blockIdx.x;
    if (r >= T) return;
    const float* lr = logits + (size_t)r * V; float* gr = grad + (size_t)r * V;
    uint32_t s = seq_ids[r];
    int seq_len = (int)(seq_starts[s + 1] - seq_starts[s]);
    if ((int)pos_ids[r] >= seq_len - 1) {
        if (grad) for (int i = threadIdx.x; i < V; i += blockDim.x) gr[i] = 0.f;
        if (threadIdx.x == 0) loss_rows[r] = 0.f;
        return;
    }
    uint32_t tg = targets[r];
    if (tg >= (uint32_t)V) { if (threadIdx.x == 0) atomicExch(status, SB_ERR_TOKEN_RANGE); tg = 0; }
    float m = -INFINITY, sum = 0.f;
#define CE_ONLINE(v) { float nv = (v); if (nv > m) { sum = sum * expf(m - nv) + 1.0f; m = nv; } else sum += expf(nv - m); }
    for (int i = threadIdx.x; i < V; i += blockDim.x) CE_ONLINE(lr[i])
    // combine (m,sum) pairs: warp, then block
    for (int o = 16; o > 0; o >>= 1) {
        float om = __shfl_xor_sync(0xffffffffu, m, o), os = __shfl_xor_sync(0xffffffffu, sum, o);
        float nm = fmaxf(m, om);
        sum = (m == -INFINITY ? 0.f : sum * expf(m - nm)) + (om == -INFINITY ? 0.f : os * expf(om - nm));
        m = nm;
    }
    if ((threadIdx.x & 31) == 0) { redm[threadIdx.x >> 5] = m; reds[threadIdx.x >> 5] = sum; }
    __syncthreads();
    m = -INFINITY; sum = 0.f;
    for (int i = 0; i < CE_THREADS / 32; i++) {
        float om = redm[i], os = reds[i], nm = fmaxf(m, om);
        sum = (m == -INFINITY ? 0.f : sum * expf(m - nm)) + (om == -INFINITY ? 0.f : os * expf(om - nm));
        m = nm;
    }
    float inv = 1.0f / sum;
    if (threadIdx.x == 0) loss_rows[r] = -((lr[tg] - m) - logf(sum));
    if (grad) for (int i = threadIdx.x; i < V; i += blockDim.x) {
        float g = expf(lr[i] - m) * inv;
        if ((uint32_t)i == tg) g -= 1.f;
        gr[i] = g * inv_valid;
        am = fmaxf(am, fabsf(g * inv_valid));
    }
    sb_block_amax(am, amax_grad);
}

// ---------------------------------------------------------------------------
// Deterministic sums: fixed grid, fixed per-thread assignment, fixed-order combine.
// ---------------------------------------------------------------------------
template <bool SQUARE>
__global__ void __launch_bounds__(RB_THREADS) partial_sum_kernel(const float* __restrict__ x, size_t n, float* __restrict__ partial, int vec) {
    sb_pdl_enter();
    __shared__ float red[64];
    size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x, nth = (size_t)gridDim.x * blockDim.x;
    float s = 0.f, d0 = 0.f;
    if (vec) {
        size_t n4 = n >> 2;
        for (size_t i = tid; i < n4; i += nth) {
            float4 v = ((const float4*)x)[i];
            s += SQUARE ? (v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w) : (v.x + v.y + v.z + v.w);
        }
        for (size_t i = (n4 << 2) + tid; i < n; i += nth) s += SQUARE ? x[i] * x[i] : x[i];
    } else for (size_t i = tid; i < n; i += nth) s += SQUARE ? x[i] * x[i] : x[i];
    block_sum2(s, d0, red);
    if (threadIdx.x == 0) partial[blockIdx.x] = s;
}
__global__ void final_sum_kernel(const float* __restrict__ partial, int n, float* out) {
    sb_pdl_enter();
    __shared__ float red[64];
    float s = 0.f, d0 = 0.f;
    for (int i = threadIdx.x; i < n; i += blockDim.x) s += partial[i];
    block_sum2(s, d0, red);
    if (threadIdx.x == 0) out[0] = s;
}

// ---------------------------------------------------------------------------
// Embedding backward as a sorted-segment reduction.
//   1. count_kernel     per-chunk token histograms (integer atomics: exact)
//   2. scan_kernel      bucket starts over the vocabulary, list of rows that occur
//   3. place_kernel     stable position of every token inside its bucket
//   4. segsum_kernel    one CTA per occurring row adds its gradient rows in
//                       ascending token position and does ONE += into dE
// Integer work is exact, the float sums have a fixed order: bit-reproducible.
// Algorithmic bytes: 4*T*d read + 8*U*d (read+write of U touched rows) + 4*T.
// ---------------------------------------------------------------------------
#define EB_CHUNK 1024
__global__ void __launch_bounds__(EB_CHUNK) eb_count_kernel(const uint32_t* __restrict__ tok, int T, int V,
                                                            int* __restrict__ chunk_cnt, int* __restrict__ cnt, int* status) {
    sb_pdl_enter();
    int t = blockIdx.x * EB_CHUNK + threadIdx.x;
    if (t >= T) return;
    uint32_t id = tok[t];
    if (id >= (uint32_t)V) { atomicExch(status, SB_ERR_TOKEN_RANGE); return; }
    atomicAdd(&chunk_cnt[(size_t)blockIdx.x * V + id], 1);
    atomicAdd(&cnt[id], 1);
}

// single CTA: exclusive scan of cnt[V] -> start[V]; compaction of rows with cnt>0 -> rows[], meta[0] = U
__global__ void __launch_bounds__(1024) eb_scan_kernel(const int* __restrict__ cnt, int V, int* __restrict__ start,
                                                       int* __restrict__ rows, int* __restrict__ meta) {
    sb_pdl_enter();
    __shared__ int s_cnt[1024], s_u[1024];
    int per = (V + 1023) / 1024, b = threadIdx.x * per, e = min(b + per, V);
    int c = 0, u = 0;
    for (int i = b; i < e; i++) { int k = cnt[i]; c += k; u += (k > 0); }
    s_cnt[threadIdx.x] = c; s_u[threadIdx.x] = u;
    __syncthreads();
    for (int off = 1; off < 1024; off <<= 1) {            // Hillis-Steele inclusive scan
        int vc = 0, vu = 0;
        if ((int)threadIdx.x >= off) { vc = s_cnt[threadIdx.x - off]; vu = s_u[threadIdx.x - off]; }
        __syncthreads();
        s_cnt[threadIdx.x] += vc; s_u[threadIdx.x] += vu;
        __syncthreads();
    }
    int base_c = s_cnt[threadIdx.x] - c, base_u = s_u[threadIdx.x] - u;
    for (int i = b; i < e; i++) {
        int k = cnt[i];
        start[i] = base_c; base_c += k;
        if (k > 0) rows[base_u++] = i;
    }
    if (threadIdx.x == 1023) { meta[0] = s_u[1023]; meta[1] = s_cnt[1023]; }
}

__global__ void __launch_bounds__(EB_CHUNK) eb_place_kernel(const uint32_t* __restrict__ tok, int T, int V,
                                                            const int* __restrict__ chunk_cnt, const int* __restrict__ start,
                                                            int* __restrict__ sorted_pos) {
    sb_pdl_enter();
    __shared__ __align__(16) uint32_t s_tok[EB_CHUNK];
    int t = blockIdx.x * EB_CHUNK + threadIdx.x;
    uint32_t id = t < T ? tok[t] : 0xffffffffu;
    s_tok[threadIdx.x] = id;
    __syncthreads();
    if (t >= T || id >= (uint32_t)V) return;
    int rank = 0;
    for (int cb = 0; cb < (int)blockIdx.x; cb++) rank += chunk_cnt[(size_t)cb * V + id];   // earlier chunks
    // earlier in this chunk: four tokens per read (one per read was most of the kernel's 16 us at 2048 tokens)
    const int j4 = (int)threadIdx.x >> 2;
    for (int j = 0; j < j4; j++) { const uint4 k = ((const uint4*)s_tok)[j]; rank += (k.x == id) + (k.y == id) + (k.z == id) + (k.w == id); }
    for (int j = j4 * 4; j < (int)threadIdx.x; j++) rank += (s_tok[j] == id);
    sorted_pos[start[id] + rank] = t;
}

__global__ void __launch_bounds__(RB_THREADS) eb_segsum_kernel(const float* __restrict__ g, float* __restrict__ dE,
                                                               const int* __restrict__ rows, const int* __restrict__ start,
                                                               const int* __restrict__ cnt, const int* __restrict__ sorted_pos,
                                                               const int* __restrict__ meta, int d, int vec) {
    sb_pdl_enter();
    int U = meta[0];
    for (int u = blockIdx.x; u < U; u += gridDim.x) {
        int row = rows[u], s0 = start[row], n = cnt[row];
        float* er = dE + (size_t)row * d;
        if (vec) for (int i = threadIdx.x; i < d / 4; i += blockDim.x) {
            float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int j = 0; j < n; j++) { float4 v = ((const float4*)(g + (size_t)sorted_pos[s0 + j] * d))[i]; a.x += v.x; a.y += v.y; a.z += v.z; a.w += v.w; }
            float4 e = ((float4*)er)[i]; e.x += a.x; e.y += a.y; e.z += a.z; e.w += a.w; ((float4*)er)[i] = e;
        } else for (int i = threadIdx.x; i < d; i += blockDim.x) {
            float a = 0.f;
            for (int j = 0; j < n; j++) a += g[(size_t)sorted_pos[s0 + j] * d + i];
            er[i] += a;
        }
    }
}

// The same sums in one launch for a training step of up to EB_DIRECT tokens, which does not ask for the tables: a CTA per token looks for its id
// among the earlier tokens (then the row belongs to another CTA), lists the later ones that share it in ascending order, and adds their gradient
// rows.  T^2 ids are compared, 4 T^2 bytes from L2 (34 us at 8192 tokens); the sort's two clears and four dependent kernels, one of them a
// single CTA over the vocabulary, took 25 us at 61 tokens, 45 at 2048 and 320 at 8192 tokens of 152k words.
#define EB_DIRECT 8192
__global__ void __launch_bounds__(128) eb_direct_kernel(const uint32_t* __restrict__ tok, const float* __restrict__ g, float* __restrict__ dE,
                                                        int T, int d, int V, int vec, int* status) {
    sb_pdl_enter();
    extern __shared__ uint16_t list[];
    __shared__ int s_cnt[4];
    const int t = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t id = tok[t];
    if (id >= (uint32_t)V) { if (threadIdx.x == 0) atomicExch(status, SB_ERR_TOKEN_RANGE); return; }
    bool seen = false;
    for (int i = threadIdx.x; i < t / 4; i += 128) { const uint4 k = ((const uint4*)tok)[i]; seen |= k.x == id || k.y == id || k.z == id || k.w == id; }
    for (int i = (t & ~3) + threadIdx.x; i < t; i += 128) seen |= tok[i] == id;
    if (__syncthreads_or(seen)) return;
    int n = 0;
    for (int b0 = t & ~3; b0 < T; b0 += 512) {
        const int j = b0 + threadIdx.x * 4;
        unsigned m = 0;
        if (j + 3 < T) { const uint4 k = ((const uint4*)tok)[j >> 2]; m = (k.x == id) | (k.y == id) << 1 | (k.z == id) << 2 | (k.w == id) << 3; }
        else for (int u = 0; j + u < T && u < 4; u++) m |= (unsigned)(tok[j + u] == id) << u;
        if (!__syncthreads_or((int)m)) continue;                 // (tokens before t do not match)
        const int c = __popc(m);
        int pre = c;
        for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xffffffffu, pre, o); if (lane >= o) pre += v; }
        if (lane == 31) s_cnt[warp] = pre;
        __syncthreads();
        int at = n + pre - c;
        for (int w = 0; w < 4; w++) { if (w < warp) at += s_cnt[w]; n += s_cnt[w]; }
        for (int u = 0; u < 4; u++) if (m >> u & 1) list[at++] = (uint16_t)(j + u);
        __syncthreads();
    }
    float* er = dE + (size_t)id * d;
    if (vec) for (int i = threadIdx.x; i < d / 4; i += 128) {
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int j = 0; j < n; j++) { const float4 v = ((const float4*)(g + (size_t)list[j] * d))[i]; a.x += v.x; a.y += v.y; a.z += v.z; a.w += v.w; }
        float4 e = ((float4*)er)[i]; e.x += a.x; e.y += a.y; e.z += a.z; e.w += a.w; ((float4*)er)[i] = e;
    } else for (int i = threadIdx.x; i < d; i += 128) {
        float a = 0.f;
        for (int j = 0; j < n; j++) a += g[(size_t)list[j] * d + i];
        er[i] += a;
    }
}

// ---------------------------------------------------------------------------
// AdamW over a flat range: decoupled decay, bias correction (host-computed
// 1-beta^t), optional global-norm clip and data-parallel 1/world folded into
// the gradient read.  28 bytes per parameter.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(RB_THREADS) adamw_kernel(float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m,
                                                           float* __restrict__ v, size_t n, float lr, float b1, float b2, float wd,
                                                           float eps, float c1, float c2, float grad_scale,
                                                           const float* __restrict__ sumsq, float clip, int vec) {
    sb_pdl_enter();
    float gs = grad_scale;
    if (clip > 0.f && sumsq) {
        float norm = sqrtf(sumsq[0]) * grad_scale;
        if (norm > clip) gs *= clip / (norm + 1e-6f);
    }
    const float decay = 1.0f - lr * wd, ob1 = 1.0f - b1, ob2 = 1.0f - b2;
    size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x, nth = (size_t)gridDim.x * blockDim.x;
#define ADAMW_ONE(W, G, M, V) { float gi = (G) * gs; float mi = b1 * (M) + ob1 * gi; float vi = b2 * (V) + ob2 * gi * gi; \
        (M) = mi; (V) = vi; float mh = mi / c1, vh = vi / c2; (W) = (W) * decay - lr * mh / (sqrtf(vh) + eps); }
    if (vec) {
        size_t n4 = n >> 2;
        for (size_t i = tid; i < n4; i += nth) {
            float4 W = ((float4*)w)[i], G = ((const float4*)g)[i], M = ((float4*)m)[i], Vv = ((float4*)v)[i];
            ADAMW_ONE(W.x, G.x, M.x, Vv.x) ADAMW_ONE(W.y, G.y, M.y, Vv.y) ADAMW_ONE(W.z, G.z, M.z, Vv.z) ADAMW_ONE(W.w, G.w, M.w, Vv.w)
            ((float4*)w)[i] = W; ((float4*)m)[i] = M; ((float4*)v)[i] = Vv;
        }
        for (size_t i = (n4 << 2) + tid; i < n; i += nth) ADAMW_ONE(w[i], g[i], m[i], v[i])
    } else for (size_t i = tid; i < n; i += nth) ADAMW_ONE(w[i], g[i], m[i], v[i])
}

extern "C" {

// `copy` (may be NULL) receives the rows x as well: the residual stream that the layer's next product adds into, written while x is in registers
// inv_word (may be NULL): a word raised to the largest 1 / rms of the rows, for the bound of the backward pass; *inv_word = NULL on return when it was not formed
void sb_rmsnorm_copy(sb_ctx_t* c, const float* x, const float* w, float* y, float* copy, int rows, int cols, float eps, float** inv_word) {
    float* inv_max = inv_word ? *inv_word : NULL;
    if (rows <= 0 || cols <= 0) return;
    sb_parts_invalidate(c, y);
    int grid = rows < sm_count(c) * 8 ? rows : sm_count(c) * 8;
    int vec = (cols % 4 == 0) && aligned16(x) && aligned16(w) && aligned16(y);
    if (copy && !(vec && aligned16(copy) && cols <= 4096 && !(cols == 128 && rows >= 1024))) { sb_copy(c, copy, x, (size_t)rows * cols * sizeof(float)); copy = NULL; }
    int tk = sb_tick_begin(c, SB_CLS_NORM_FWD);
    if (vec && cols <= 4096) {
        // warp per row, 8 warps per CTA, two CTAs resident per SM: every warp gets the same number of rows (no tail)
        int wgrid = (rows + 7) / 8;
        { int cap = sm_count(c) * 2, k = (wgrid + cap - 1) / cap; wgrid = (wgrid + k - 1) / k; }
        cudaStream_t st = (cudaStream_t)c->pub.stream;
        unsigned* am = sb_amax_take(c, y, (size_t)rows * cols);
        if (cols == 128 && rows >= 1024) {
            if (inv_word) *inv_word = NULL;
            int g4 = (rows + 31) / 32; if (g4 > sm_count(c) * 4) g4 = sm_count(c) * 4;      // 8 warps x 4 rows per CTA and pass
            sb_launch(rmsnorm_w128_kernel, dim3(g4), dim3(RB_THREADS), 0, st, x, w, y, rows, eps, am);
        } else
        if (cols <= 512)       sb_launch(rmsnorm_warp_kernel<4>, dim3(wgrid), dim3(RB_THREADS), 0, st, x, w, y, copy, rows, cols, eps, am, (unsigned*)inv_max);
        else if (cols <= 1024) sb_launch(rmsnorm_warp_kernel<8>, dim3(wgrid), dim3(RB_THREADS), 0, st, x, w, y, copy, rows, cols, eps, am, (unsigned*)inv_max);
        else {
            const int g = rows < 4 * sm_count(c) ? rows : 4 * sm_count(c);
            if (cols <= 2048) sb_launch(rmsnorm_rows_kernel<2>, dim3(g), dim3(RB_THREADS), 0, st, x, w, y, nullptr, nullptr, copy, rows, cols, eps, nullptr, 0u, (unsigned*)inv_max, am);
            else              sb_launch(rmsnorm_rows_kernel<4>, dim3(g), dim3(RB_THREADS), 0, st, x, w, y, nullptr, nullptr, copy, rows, cols, eps, nullptr, 0u, (unsigned*)inv_max, am);
        }
    } else {
    if (inv_word) *inv_word = NULL;
    sb_launch(rmsnorm_kernel, dim3(grid), dim3(RB_THREADS), 0, (cudaStream_t)c->pub.stream, x, w, y, rows, cols, eps, vec);
    }
    sb_tick_end(c, tk, 0.0, (copy ? 12.0 : 8.0) * rows * cols);
    c->launches++;
}
void sb_rmsnorm(sb_ctx_t* c, const float* x, const float* w, float* y, int rows, int cols, float eps) { sb_rmsnorm_copy(c, x, w, y, NULL, rows, cols, eps, NULL); }

// y only as the FP16 parts of the registered tensor `y`; 1 = done, 0 = not possible here (call sb_rmsnorm)
int sb_rmsnorm_parts(sb_ctx_t* c, const float* x, const float* w, float* y, float* copy, int rows, int cols, float eps, float** inv_word) {
    float* inv_max = inv_word ? *inv_word : NULL;
    if (rows < 1 || cols <= 0 || (cols & 7) || cols > 4096 || !aligned16(x) || !aligned16(w) || (copy && !aligned16(copy))) return 0;
    void* h; float* bound;
    const size_t n = (size_t)rows * cols;
    if (!aligned16(y) || !sb_bound_out(c, y, n, &h, &bound)) return 0;
    float* y32 = h ? NULL : y;
    // a row per warp: what a row costs is the way to memory and back.  5800 x 512 in a step: 8.4 us, 15 with three rows one after the other in two CTAs an
    // SM and an atomic a warp; 2048 x 512: 5.0 (6.5)
    int wgrid = (rows + 7) / 8;
    if (wgrid > sm_count(c) * 16) wgrid = sm_count(c) * 16;
    cudaStream_t st = (cudaStream_t)c->pub.stream;
    uint2* h1 = (uint2*)h; uint2* h2 = (uint2*)((uint16_t*)h + n);
    int tk = sb_tick_begin(c, SB_CLS_NORM_FWD);
    if (cols <= 512)       sb_launch(rmsnorm_warp_parts_kernel<4>, dim3(wgrid), dim3(RB_THREADS), 0, st, x, w, y32, h1, h2, rows, cols, eps, bound, sb_parts_keep(c), copy, (unsigned*)inv_max);
    else if (cols <= 1024) sb_launch(rmsnorm_warp_parts_kernel<8>, dim3(wgrid), dim3(RB_THREADS), 0, st, x, w, y32, h1, h2, rows, cols, eps, bound, sb_parts_keep(c), copy, (unsigned*)inv_max);
    else {
        const int g = rows < 4 * sm_count(c) ? rows : 4 * sm_count(c);
        if (cols <= 2048) sb_launch(rmsnorm_rows_kernel<2>, dim3(g), dim3(RB_THREADS), 0, st, x, w, y32, h ? h1 : nullptr, h2, copy, rows, cols, eps, bound, sb_parts_keep(c), (unsigned*)inv_max, nullptr);
        else              sb_launch(rmsnorm_rows_kernel<4>, dim3(g), dim3(RB_THREADS), 0, st, x, w, y32, h ? h1 : nullptr, h2, copy, rows, cols, eps, bound, sb_parts_keep(c), (unsigned*)inv_max, nullptr);
    }
    sb_tick_end(c, tk, 0.0, (copy ? 12.0 : 8.0) * rows * cols);
    c->launches++;
    return 1;
}

// number of CTAs the rmsnorm backward uses for `rows` rows (also the row count of its partial buffer)
// The sums of dscale partials: at once, or (between sb_colsum_defer and sb_colsum_flush) noted and formed together, up to CS_TAB norms in one
// launch.  A sum is 3 us of work in a launch of its own; a training step of an eight-layer model has 17 of them.
struct CsPending { CsTab tab; int n, maxcols; float* arena; size_t cap, used; };
#define CS_ARENA ((size_t)8 << 20)      // floats (32 MB): 13 norms of 2048 columns; filling up only means a launch
static void cs_launch(sb_ctx_t* c, const CsTab& t, int n, int maxcols) {
    sb_launch(colsum_partials_kernel, dim3((maxcols + 31) / 32, n), dim3(32 * CS_GROUPS), 0, (cudaStream_t)c->pub.stream, t);
    c->launches++;
}
extern "C" void sb_colsum_flush(sb_ctx_t* c) {
    CsPending* p = (CsPending*)c->cs_pending;
    if (!p) return;
    if (p->n) {
        int tk = sb_tick_begin(c, SB_CLS_NORM_BWD);
        cs_launch(c, p->tab, p->n, p->maxcols);
        sb_tick_end(c, tk, 0.0, 0.0);
    }
    p->n = 0; p->maxcols = 0; p->used = 0;
}
extern "C" void sb_colsum_defer(sb_ctx_t* c, int on, int store, size_t floats) {
    sb_colsum_flush(c);
    c->cs_defer = 0; c->cs_store = store;
    if (!on) return;
    CsPending* p = (CsPending*)c->cs_pending;
    if (!p) { p = (CsPending*)calloc(1, sizeof *p); c->cs_pending = p; }
    if (!p) return;
    if (floats > CS_ARENA) floats = CS_ARENA;
    if (p->cap < floats) {
        cudaStreamSynchronize((cudaStream_t)c->pub.stream);
        if (p->arena) cudaFree(p->arena);
        p->arena = NULL; p->cap = 0;
        if (cudaMalloc((void**)&p->arena, floats * sizeof(float)) != cudaSuccess) { cudaGetLastError(); return; }      // no room: one launch per sum
        p->cap = floats;
    }
    c->cs_defer = 1;
}
extern "C" void sb_colsum_free(sb_ctx_t* c) {
    CsPending* p = (CsPending*)c->cs_pending;
    if (p) { if (p->arena) cudaFree(p->arena); free(p); }
    c->cs_pending = NULL; c->cs_defer = 0;
}
// room for the partials of one norm
static float* rn_partials(sb_ctx_t* c, size_t floats) {
    CsPending* p = (CsPending*)c->cs_pending;
    if (c->cs_defer && floats <= p->cap) {
        if (p->n == CS_TAB || p->used + floats > p->cap) sb_colsum_flush(c);
        float* r = p->arena + p->used;
        p->used += (floats + 31) & ~(size_t)31;
        return r;
    }
    return (float*)sb_scratch(c, floats * sizeof(float));
}
static void rn_dscale(sb_ctx_t* c, const float* partial, float* dscale, int nblocks, int cols) {
    CsPending* p = (CsPending*)c->cs_pending;
    const CsEntry e = {partial, dscale, nblocks, cols};
    if (c->cs_defer && partial >= p->arena && partial < p->arena + p->cap) {
        p->tab.store = c->cs_store; p->tab.e[p->n++] = e;
        if (cols > p->maxcols) p->maxcols = cols;
        return;
    }
    CsTab t; t.store = c->cs_store; t.e[0] = e;
    cs_launch(c, t, 1, cols);
}

static int rn_bwd_grid(sb_ctx_t* c, int rows) { int cap = sm_count(c) * 2; return rows < cap ? rows : cap; }

void sb_rmsnorm_backward_with_partials(sb_ctx_t* c, const float* x, const float* w, const float* dy, const float* resid,
                                       float* dx_out, float* dscale, int rows, int cols, float eps, float* partial, int grid) {
    int vec = (cols % 4 == 0) && aligned16(x) && aligned16(w) && aligned16(dy) && aligned16(dx_out) && (!resid || aligned16(resid));
    cudaStream_t s = (cudaStream_t)c->pub.stream;
    int tk = sb_tick_begin(c, SB_CLS_NORM_BWD);
    sb_launch(rmsnorm_bwd_kernel, dim3(grid), dim3(RB_THREADS), 0, s, x, w, dy, resid, dx_out, partial, rows, cols, eps, vec);
    c->launches++;
    if (dscale) rn_dscale(c, partial, dscale, grid, cols);
    sb_tick_end(c, tk, 0.0, (resid ? 16.0 : 12.0) * rows * cols);
}

static bool rn_rows_ok(int vec, int cols) { return vec && cols <= 4096; }
static void rn_backward(sb_ctx_t* c, const float* x, const float* w, const float* dy, const float* resid,
                        float* dx_out, float* dscale, int rows, int cols, float eps, const RnbOut& out, unsigned* exact) {
    if (rows <= 0 || cols <= 0) return;
    if (cols > RB_THREADS * 4 * RN_MAX_SWEEP || (cols % 4 != 0 && cols > RB_THREADS * RN_MAX_SWEEP * 4)) { sb_set_status(c, SB_ERR_SIZE); return; }
    int vec = (cols % 4 == 0) && aligned16(x) && aligned16(w) && aligned16(dy) && aligned16(dx_out) && (!resid || aligned16(resid));
    if (vec && cols == 128 && rows >= 1024 && !out.bound) {
        // many short rows (the per-head norm): a warp per row
        int wgrid = (rows + 31) / 32; if (wgrid > 4 * sm_count(c)) wgrid = 4 * sm_count(c);
        float* partial = rn_partials(c, (size_t)wgrid * cols);
        if (!partial) return;
        cudaStream_t st = (cudaStream_t)c->pub.stream;
        int tk = sb_tick_begin(c, SB_CLS_NORM_BWD);
        unsigned* am = sb_amax_take(c, dx_out, (size_t)rows * cols);
        sb_launch(rmsnorm_bwd_w128_kernel, dim3(wgrid), dim3(RB_THREADS), 0, st, x, w, dy, resid, dx_out, partial, rows, eps, am);
        c->launches++;
        if (dscale) rn_dscale(c, partial, dscale, wgrid, cols);
        sb_tick_end(c, tk, 0.0, (resid ? 16.0 : 12.0) * rows * cols);
        return;
    }
    if (rn_rows_ok(vec, cols)) {
        // row groups with the next group's loads in flight, two CTAs per SM; one dscale partial per CTA, summed in CTA order.  Groups of two
        // rows, of one above 2048 columns (a thread then holds four chunks of a row, and two rows would not fit its registers).
        const bool narrow = cols <= 512 && rows >= 512;
        const int per = narrow ? RB_THREADS / 32 : cols <= 2048 ? 2 : 1;
        int wgrid = (rows + per - 1) / per; if (wgrid > 2 * sm_count(c)) wgrid = 2 * sm_count(c);
        float* partial = rn_partials(c, (size_t)wgrid * cols);
        if (!partial) return;
        cudaStream_t st = (cudaStream_t)c->pub.stream;
        int tk = sb_tick_begin(c, SB_CLS_NORM_BWD);
        unsigned* am = exact ? exact : sb_amax_take(c, dx_out, (size_t)rows * cols);
        if (narrow)            sb_launch(rmsnorm_bwd_warp_kernel<4>, dim3(wgrid), dim3(RB_THREADS), 0, st, x, w, dy, resid, dx_out, partial, rows, cols, eps, am, out);
        else if (cols <= 1024) sb_launch(rmsnorm_bwd_rows_kernel<1, 2>, dim3(wgrid), dim3(RB_THREADS), 0, st, x, w, dy, resid, dx_out, partial, rows, cols, eps, am, out);
        else if (cols > 2048)  sb_launch(rmsnorm_bwd_rows_kernel<4, 1>, dim3(wgrid), dim3(RB_THREADS), 0, st, x, w, dy, resid, dx_out, partial, rows, cols, eps, am, out);
        else                   sb_launch(rmsnorm_bwd_rows_kernel<2, 2>, dim3(wgrid), dim3(RB_THREADS), 0, st, x, w, dy, resid, dx_out, partial, rows, cols, eps, am, out);
        c->launches++;
        if (dscale) rn_dscale(c, partial, dscale, wgrid, cols);
        sb_tick_end(c, tk, 0.0, (resid ? 16.0 : 12.0) * rows * cols);
        return;
    }
    int grid = rn_bwd_grid(c, rows);
    float* partial = rn_partials(c, (size_t)grid * cols);
    if (!partial) return;
    sb_rmsnorm_backward_with_partials(c, x, w, dy, resid, dx_out, dscale, rows, cols, eps, partial, grid);
}
void sb_rmsnorm_backward(sb_ctx_t* c, const float* x, const float* w, const float* dy, const float* resid,
                         float* dx_out, float* dscale, int rows, int cols, float eps) {
    const RnbOut none = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, 0u};
    sb_parts_invalidate(c, dx_out);
    rn_backward(c, x, w, dy, resid, dx_out, dscale, rows, cols, eps, none, nullptr);
}
// The same, with dx handed on as operand parts under a bound where max|dy|, max|residual| and max(1/rms) are known (a pass over dx less);
// *amax: in, the word with max|residual|; out, the word with max|dx| (NULL: not known).
void sb_rmsnorm_backward_parts(sb_ctx_t* c, const float* x, const float* w, const float* dy, const float* resid,
                               float* dx_out, float* dscale, int rows, int cols, float eps, const float* inv_max, float** amax) {
    const size_t n = (size_t)rows * cols;
    const int vec = (cols % 8 == 0) && aligned16(x) && aligned16(w) && aligned16(dy) && aligned16(dx_out) && (!resid || aligned16(resid));
    RnbOut out = {nullptr, nullptr, sb_amax_lookup(c, dy, n), resid ? *amax : nullptr, inv_max, nullptr, sb_parts_keep(c)};
    float* exact = rn_rows_ok(vec, cols) && inv_max && out.amax_dy && (!resid || *amax) ? sb_zero_word(c) : nullptr;
    if (exact) { sb_amax_announce(c, dx_out, n); out.bound = (float*)sb_amax_take(c, dx_out, n); }
    if (!out.bound) {
        sb_amax_announce(c, dx_out, n);
        sb_rmsnorm_backward(c, x, w, dy, resid, dx_out, dscale, rows, cols, eps);
        *amax = sb_amax_lookup(c, dx_out, n);
        return;
    }
    void* h; float* own; int fresh;
    if (sb_parts_find(c, dx_out, n, &h, &own, &fresh)) { sb_parts_set_amax(c, dx_out, out.bound); out.h1 = (uint2*)h; out.h2 = (uint2*)((uint16_t*)h + n); }
    rn_backward(c, x, w, dy, resid, dx_out, dscale, rows, cols, eps, out, (unsigned*)exact);
    *amax = exact;
}

void sb_softmax(sb_ctx_t* c, const float* x, float* y, int rows, int cols) {
    if (rows <= 0 || cols <= 0) return;
    int grid = rows < sm_count(c) * 8 ? rows : sm_count(c) * 8;
    sb_launch(softmax_kernel, dim3(grid), dim3(RB_THREADS), 0, (cudaStream_t)c->pub.stream, x, y, rows, cols);
    c->launches++;
}

static int qk_wgrid(sb_ctx_t* c, int rows) {
    int wgrid = (rows + 7) / 8, cap = sm_count(c) * 2;
    int k = (wgrid + cap - 1) / cap; if (k < 1) k = 1;
    return (wgrid + k - 1) / k;
}
void sb_qk_norm(sb_ctx_t* c, float* x, float* rms_out, int rows, int cols, float eps) {
    if (rows <= 0 || cols <= 0) return;
    cudaStream_t st = (cudaStream_t)c->pub.stream;
    int tk = sb_tick_begin(c, SB_CLS_NORM_FWD);
    if ((cols % 4) == 0 && cols <= 4096 && aligned16(x) && rows >= 64) {
        const int g = qk_wgrid(c, rows);
        if (cols <= 512)       sb_launch(qk_norm_warp_kernel<4>, dim3(g), dim3(RB_THREADS), 0, st, x, rms_out, rows, cols, eps);
        else if (cols <= 1024) sb_launch(qk_norm_warp_kernel<8>, dim3(g), dim3(RB_THREADS), 0, st, x, rms_out, rows, cols, eps);
        else if (cols <= 2048) sb_launch(qk_norm_warp_kernel<16>, dim3(g), dim3(RB_THREADS), 0, st, x, rms_out, rows, cols, eps);
        else                   sb_launch(qk_norm_warp_kernel<32>, dim3(g), dim3(RB_THREADS), 0, st, x, rms_out, rows, cols, eps);
    } else {
        int grid = rows < sm_count(c) * 8 ? rows : sm_count(c) * 8;
        sb_launch(qk_norm_row_kernel, dim3(grid), dim3(RB_THREADS), 0, st, x, rms_out, nullptr, nullptr, nullptr, rows, cols, eps);
    }
    sb_tick_end(c, tk, 0.0, 8.0 * rows * cols);
    c->launches++;
}
void sb_qk_norm_backward(sb_ctx_t* c, const float* y, const float* rms, const float* dy, float* dx, int rows, int cols, float eps) {
    if (rows <= 0 || cols <= 0) return;
    cudaStream_t st = (cudaStream_t)c->pub.stream;
    int tk = sb_tick_begin(c, SB_CLS_NORM_BWD);
    if ((cols % 4) == 0 && cols <= 4096 && aligned16(y) && aligned16(dy) && aligned16(dx) && rows >= 64) {
        const int g = qk_wgrid(c, rows);
        if (cols <= 512)       sb_launch(qk_norm_bwd_warp_kernel<4>, dim3(g), dim3(RB_THREADS), 0, st, y, rms, dy, dx, rows, cols, eps);
        else if (cols <= 1024) sb_launch(qk_norm_bwd_warp_kernel<8>, dim3(g), dim3(RB_THREADS), 0, st, y, rms, dy, dx, rows, cols, eps);
        else if (cols <= 2048) sb_launch(qk_norm_bwd_warp_kernel<16>, dim3(g), dim3(RB_THREADS), 0, st, y, rms, dy, dx, rows, cols, eps);
        else                   sb_launch(qk_norm_bwd_warp_kernel<32>, dim3(g), dim3(RB_THREADS), 0, st, y, rms, dy, dx, rows, cols, eps);
    } else {
        int grid = rows < sm_count(c) * 8 ? rows : sm_count(c) * 8;
        sb_launch(qk_norm_row_kernel, dim3(grid), dim3(RB_THREADS), 0, st, (float*)y, nullptr, rms, dy, dx, rows, cols, eps);
    }
    sb_tick_end(c, tk, 0.0, 12.0 * rows * cols);
    c->launches++;
}

#define CE_MAX_SLICE (64 * 1024)      // bytes of a row in one CTA's shared memory
// CTAs per row: slices of at most 64 KB, so that three or more CTAs share an SM, in clusters of one or two (four at 32 KB each: 0.63 instead of
// 0.50 ms at 8192 x 32768); up to eight only when there are too few rows to fill the device.  0: the row is too long.
static int ce_cluster(sb_ctx_t* c, int T, int V) {
    int cl = 1;
    if ((size_t)V * 4 > 64 * 1024) cl = 2;
    while (cl < 8 && (long)T * cl <= (long)sm_count(c)) cl *= 2;
    return (size_t)((V / 4 + cl - 1) / cl) * 16 <= CE_MAX_SLICE ? cl : 0;
}
extern "C++" {
template <int CL>
static bool ce_launch(sb_ctx_t* c, const CeArgs& a) {
    const size_t smem = (size_t)((a.V / 4 + CL - 1) / CL) * 16;
    static bool attr = false;
    if (!attr) {
        if (cudaFuncSetAttribute(cross_entropy_kernel<CL>, cudaFuncAttributeMaxDynamicSharedMemorySize, CE_MAX_SLICE) != cudaSuccess) { cudaGetLastError(); return false; }
        attr = true;
    }
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof cfg);
    cfg.gridDim = dim3((unsigned)a.T * CL); cfg.blockDim = dim3(CE_THREADS); cfg.dynamicSmemBytes = smem; cfg.stream = (cudaStream_t)c->pub.stream;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = CL; at[1].val.clusterDim.y = 1; at[1].val.clusterDim.z = 1;
    cfg.attrs = at; cfg.numAttrs = CL > 1 ? 2 : 1;
    c->launches++;
    return cudaLaunchKernelEx(&cfg, cross_entropy_kernel<CL>, a) == cudaSuccess;
}
static bool ce_launch_any(sb_ctx_t* c, const CeArgs& a) {
    switch (ce_cluster(c, a.T, a.V)) {
        case 1: return ce_launch<1>(c, a);
        case 2: return ce_launch<2>(c, a);
        case 4: return ce_launch<4>(c, a);
        case 8: return ce_launch<8>(c, a);
        default:
            c->launches++;
            return sb_launch(cross_entropy_long_kernel, dim3(a.T), dim3(CE_LONG), 0, (cudaStream_t)c->pub.stream, a) == cudaSuccess;
    }
}
}
// grad NULL: the loss alone
void sb_cross_entropy(sb_ctx_t* c, const float* logits, const uint32_t* targets, float* grad, float* loss_rows,
                      const uint32_t* pos_ids, const uint32_t* seq_ids, const uint32_t* seq_starts, int T, int V, int num_valid) {
    if (T <= 0 || V <= 0) return;
    int tk = sb_tick_begin(c, SB_CLS_CE);
    const CeArgs a = {logits, targets, grad, loss_rows, pos_ids, seq_ids, seq_starts, T, V, 1.0f / (float)num_valid, c->d_status,
                      grad ? sb_amax_take(c, grad, (size_t)T * V) : nullptr, nullptr, nullptr, 0.f, nullptr, 0u};
    if (!((V % 4) == 0 && aligned16(logits) && (!grad || aligned16(grad)) && ce_launch_any(c, a))) {
        sb_launch(cross_entropy_any_kernel, dim3(T), dim3(CE_THREADS), 0, (cudaStream_t)c->pub.stream, logits, targets, grad, loss_rows, pos_ids, seq_ids,
                  seq_starts, T, V, a.inv_valid, c->d_status, a.amax_grad);
        c->launches++;
    }
    sb_tick_end(c, tk, 0.0, (grad ? 8.0 : 4.0) * T * V);
}

// The same, with the gradient written only as the FP16 parts of the registered tensor `grad` (its FP32 array is not touched): the
// two LM-head backward products then find their operand prepared and no pass splits 4 T V bytes of gradient again.
// Returns 1 when done, 0 when the parts of `grad` are not available (not registered, cache off, no memory): use sb_cross_entropy.
static __device__ __host__ inline int ce_shift(float amax) {
    int e; frexpf(amax, &e);                       // amax = f * 2^e, f in [0.5, 1): exponent of the leading bit is e - 1
    return 14 - (e - 1);
}
int sb_cross_entropy_parts(sb_ctx_t* c, const float* logits, const uint32_t* targets, float* grad, float* loss_rows,
                           const uint32_t* pos_ids, const uint32_t* seq_ids, const uint32_t* seq_starts, int T, int V, int num_valid) {
    if (T <= 0 || V <= 0 || (V % 4) || !aligned16(logits) || num_valid <= 0) return 0;
    void* h; float* amax;
    if (!aligned16(grad) || !sb_bound_out(c, grad, (size_t)T * V, &h, &amax)) return 0;
    const float inv_valid = 1.0f / (float)num_valid;
    int sh = ce_shift(inv_valid); sh = sh < -100 ? -100 : (sh > 100 ? 100 : sh);      // the rule the products apply to *amax
    const float sc = ldexpf(1.0f, sh);
    int tk = sb_tick_begin(c, SB_CLS_CE);
    const CeArgs a = {logits, targets, h ? nullptr : grad, loss_rows, pos_ids, seq_ids, seq_starts, T, V, inv_valid, c->d_status, nullptr,
                      (__half*)h, h ? (__half*)h + (size_t)T * V : nullptr, sc, amax, sb_parts_keep(c)};
    const bool ok = ce_launch_any(c, a);
    sb_tick_end(c, tk, 0.0, 8.0 * T * V);
    if (!ok) sb_set_status(c, SB_ERR_CUDA);
    return 1;
}

static void sum_impl(sb_ctx_t* c, const float* in, float* out, size_t n, bool square) {
    cudaStream_t s = (cudaStream_t)c->pub.stream;
    if (n == 0) { cudaMemsetAsync(out, 0, sizeof(float), s); return; }
    int grid = sm_count(c) * 4;
    size_t need = (n + RB_THREADS * 4 - 1) / (RB_THREADS * 4);
    if ((size_t)grid > need) grid = (int)need;
    float* partial = (float*)sb_scratch(c, (size_t)grid * sizeof(float));
    if (!partial) return;
    int vec = aligned16(in);
    int tk = sb_tick_begin(c, SB_CLS_OTHER);
    if (square) sb_launch(partial_sum_kernel<true>, dim3(grid), dim3(RB_THREADS), 0, s, in, n, partial, vec);
    else        sb_launch(partial_sum_kernel<false>, dim3(grid), dim3(RB_THREADS), 0, s, in, n, partial, vec);
    sb_launch(final_sum_kernel, dim3(1), dim3(RB_THREADS), 0, s, partial, grid, out);
    sb_tick_end(c, tk, 0.0, 4.0 * (double)n);
    c->launches += 2;
}
void sb_reduce_sum(sb_ctx_t* c, const float* in, float* out, size_t n) { sum_impl(c, in, out, n, false); }
void sb_sumsq(sb_ctx_t* c, const float* g, size_t n, float* d_out) { sum_impl(c, g, d_out, n, true); }

// Scratch layout of the embedding backward (ints): cnt[V] start[V] rows[V] meta[4] sorted_pos[T] chunk_cnt[nchunk*V]
size_t sb_embedding_scratch_ints(int T, int V) {
    size_t nchunk = ((size_t)T + EB_CHUNK - 1) / EB_CHUNK;
    return 3 * (size_t)V + 4 + (size_t)T + nchunk * (size_t)V;
}

void sb_embedding_backward(sb_ctx_t* c, const uint32_t* tok, const float* g, float* dE, int T, int d, int V) {
    if (T <= 0 || d <= 0 || V <= 0) return;
    cudaStream_t s = (cudaStream_t)c->pub.stream;
    int nchunk = (T + EB_CHUNK - 1) / EB_CHUNK;
    size_t ints = sb_embedding_scratch_ints(T, V);
    int* base = (int*)sb_scratch(c, ints * sizeof(int));
    if (!base) return;
    int *cnt = base, *start = cnt + V, *rows = start + V, *meta = rows + V, *sorted_pos = meta + 4, *chunk_cnt = sorted_pos + T;      // sb_embedding_segments reads the same layout
    int tk = sb_tick_begin(c, SB_CLS_EMBED);
    cudaMemsetAsync(cnt, 0, (size_t)V * sizeof(int), s);
    cudaMemsetAsync(chunk_cnt, 0, (size_t)nchunk * V * sizeof(int), s);
    sb_launch(eb_count_kernel, dim3(nchunk), dim3(EB_CHUNK), 0, s, tok, T, V, chunk_cnt, cnt, c->d_status);
    sb_launch(eb_scan_kernel, dim3(1), dim3(1024), 0, s, cnt, V, start, rows, meta);
    sb_launch(eb_place_kernel, dim3(nchunk), dim3(EB_CHUNK), 0, s, tok, T, V, chunk_cnt, start, sorted_pos);
    int grid = T < V ? T : V;
    if (grid > sm_count(c) * 8) grid = sm_count(c) * 8;
    int vec = (d % 4 == 0) && aligned16(g) && aligned16(dE);
    sb_launch(eb_segsum_kernel, dim3(grid), dim3(RB_THREADS), 0, s, g, dE, rows, start, cnt, sorted_pos, meta, d, vec);
    sb_tick_end(c, tk, 0.0, 12.0 * T * d);      // upper bound: every token a distinct row
    c->launches += 4;
}
// without the tables that sb_embedding_segments reads
void sb_embedding_backward_step(sb_ctx_t* c, const uint32_t* tok, const float* g, float* dE, int T, int d, int V) {
    if (T <= 0 || T > EB_DIRECT || d <= 0 || V <= 0 || !aligned16(tok)) { sb_embedding_backward(c, tok, g, dE, T, d, V); return; }
    int tk = sb_tick_begin(c, SB_CLS_EMBED);
    sb_launch(eb_direct_kernel, dim3(T), dim3(128), (size_t)T * sizeof(uint16_t), (cudaStream_t)c->pub.stream, tok, g, dE, T, d, V,
              (int)((d % 4 == 0) && aligned16(g) && aligned16(dE)), c->d_status);
    sb_tick_end(c, tk, 0.0, 12.0 * T * d);
    c->launches++;
}

// copies the segment tables of the last sb_embedding_backward(T, V) to the host:
// rows[U] (ascending), counts[U], sorted_pos[T]; returns U, or -1 on error
int sb_embedding_segments(sb_ctx_t* c, int T, int V, int* rows_out, int* counts_out, int* sorted_pos_out) {
    size_t ints = sb_embedding_scratch_ints(T, V);
    if (!c->scratch || c->scratch_bytes < ints * sizeof(int)) return -1;
    cudaStream_t s = (cudaStream_t)c->pub.stream;
    cudaStreamSynchronize(s);
    int* base = (int*)c->scratch;
    int *cnt = base, *start = cnt + V, *rows = start + V, *meta = rows + V, *sorted_pos = meta + 4;
    int h_meta[4];
    if (cudaMemcpy(h_meta, meta, sizeof h_meta, cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
    int U = h_meta[0];
    if (U < 0 || U > V) return -1;
    int* h_cnt = (int*)malloc((size_t)V * sizeof(int));
    if (!h_cnt) return -1;
    cudaMemcpy(h_cnt, cnt, (size_t)V * sizeof(int), cudaMemcpyDeviceToHost);
    cudaMemcpy(rows_out, rows, (size_t)U * sizeof(int), cudaMemcpyDeviceToHost);
    cudaMemcpy(sorted_pos_out, sorted_pos, (size_t)T * sizeof(int), cudaMemcpyDeviceToHost);
    for (int i = 0; i < U; i++) counts_out[i] = h_cnt[rows_out[i]];
    free(h_cnt);
    (void)start;
    return U;
}

void sb_adamw(sb_ctx_t* c, float* w, const float* g, float* m, float* v, size_t n, float lr, float b1, float b2,
              float wd, float eps, int step, float grad_scale, const float* d_sumsq, float clip) {
    if (!n) return;
    float c1 = 1.0f - powf(b1, (float)step), c2 = 1.0f - powf(b2, (float)step);
    int vec = aligned16(w) && aligned16(g) && aligned16(m) && aligned16(v);
    size_t need = (n + RB_THREADS * 4 - 1) / (RB_THREADS * 4);
    size_t grid = (size_t)sm_count(c) * 8;
    if (grid > need) grid = need;
    int tk = sb_tick_begin(c, SB_CLS_ADAMW);
    sb_launch(adamw_kernel, dim3((int)grid), dim3(RB_THREADS), 0, (cudaStream_t)c->pub.stream, w, g, m, v, n, lr, b1, b2, wd, eps, c1, c2,
                                                                         grad_scale, d_sumsq, clip, vec);
    sb_tick_end(c, tk, 0.0, 28.0 * (double)n);
    c->launches++;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// RMSNorm backward for callers that must not allocate.
//
// Some hosts of this library may not touch the CUDA allocator at the moment
// they need a backward op: code running while a stream capture is open on
// another thread, real-time loops and allocator-owning frameworks that forbid
// cudaMalloc after start-up, and embedders that hand out every byte of device
// memory themselves.  For them the two-stage reduction of dscale keeps its
// per-CTA partial sums in a fixed array that lives in the library image
// instead of in grow-on-demand scratch.
//
// The array belongs to the device that loaded the library and stays resident
// until the process exits: SB_NOALLOC_MAX_CTAS * SB_NOALLOC_MAX_COLS floats
// (296 * 8192 * 4 bytes = 9.7 MB) on every GPU that uses the library.
// ---------------------------------------------------------------------------
#define SB_NOALLOC_MAX_COLS 8192
#define SB_NOALLOC_MAX_CTAS 296          // two CTAs per SM on a 148-SM part
#define SB_NOALLOC_MAX_DEVICES 64

static __device__ __align__(256) float g_rn_static_partials[(size_t)SB_NOALLOC_MAX_CTAS * SB_NOALLOC_MAX_COLS];

// Device address of the array, looked up once per device.  In host code the
// symbol's name is only a handle; the kernels need what cudaGetSymbolAddress
// returns for the device that is current.
static float* g_rn_static_ptr[SB_NOALLOC_MAX_DEVICES];
static int g_rn_static_sms[SB_NOALLOC_MAX_DEVICES];

extern "C" int seraph_b200_rmsnorm_backward_static(const float* input, const float* scale, const float* grad_output,
                                                   float* grad_input, float* grad_scale, int rows, int cols, float eps,
                                                   void* stream) {
    if (!input || !scale || !grad_output || !grad_input || !grad_scale || rows < 0 || cols <= 0) {
        fprintf(stderr, "seraph_b200_rmsnorm_backward_static: NULL pointer or bad shape (rows %d, cols %d)\n", rows, cols);
        return SB_ERR_ARG;
    }
    if (cols > SB_NOALLOC_MAX_COLS) {
        fprintf(stderr, "seraph_b200_rmsnorm_backward_static: cols %d exceeds the fixed scratch (at most %d columns); "
                        "use cuda_train_rmsnorm_backward_batch, which may allocate\n", cols, SB_NOALLOC_MAX_COLS);
        return SB_ERR_SIZE;
    }
    if (rows == 0) return SB_OK;
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= SB_NOALLOC_MAX_DEVICES) {
        fprintf(stderr, "seraph_b200_rmsnorm_backward_static: no usable current device\n");
        return SB_ERR_CUDA;
    }
    if (!g_rn_static_ptr[dev]) {
        // first call on this device: resolve the array's device address and the SM count
        float* p = NULL;
        cudaError_t e = cudaGetSymbolAddress((void**)&p, g_rn_static_partials);
        if (e != cudaSuccess || !p) {
            fprintf(stderr, "seraph_b200_rmsnorm_backward_static: cudaGetSymbolAddress failed: %s\n", cudaGetErrorString(e));
            return SB_ERR_CUDA;
        }
        int sms = 0;
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 148;
        g_rn_static_sms[dev] = sms;
        g_rn_static_ptr[dev] = p;
    }
    int grid = 2 * g_rn_static_sms[dev];
    if (grid > SB_NOALLOC_MAX_CTAS) grid = SB_NOALLOC_MAX_CTAS;
    if (grid > rows) grid = rows;
    float* partial = g_rn_static_ptr[dev];
    int vec = (cols % 4 == 0) && aligned16(input) && aligned16(scale) && aligned16(grad_output) && aligned16(grad_input);
    cudaStream_t s = (cudaStream_t)stream;
    // every CTA overwrites its whole row of partials before the column sum reads it,
    // so nothing left over from an earlier call is ever read and no clearing is needed
    // plain launches on the caller's stream, which may be under capture
    rmsnorm_bwd_kernel<<<grid, RB_THREADS, 0, s>>>(input, scale, grad_output, nullptr, grad_input, partial, rows, cols, eps, vec);
    CsTab tab;
    tab.store = 0; tab.e[0] = {partial, grad_scale, grid, cols};
    colsum_partials_kernel<<<(cols + 31) / 32, 32 * CS_GROUPS, 0, s>>>(tab);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        fprintf(stderr, "seraph_b200_rmsnorm_backward_static: launch failed: %s\n", cudaGetErrorString(e));
        return SB_ERR_CUDA;
    }
    return SB_OK;
}
