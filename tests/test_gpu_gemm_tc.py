"""Tensor-core GEMM (tcgen05, TMA, TMEM) against the FP64-accumulate oracle, through the C ABI.
Stated bounds (relative L2 of the whole result, standard-normal operands):
  mode 0, FP32-accurate (three TF32 passes on a hi/lo split):  <= 2e-6   (the FP32 path; whole-model gradients must meet 1e-5)
  mode 1, single-pass TF32:                                    <= 2e-3
  mode 4, FP32-accurate with scaled FP16 hi/lo parts where the layout allows (three FP16 passes): <= 2e-6
Shapes include ragged M/N/K edges (TMA zero fill), all three layouts, accumulate, long K."""
import numpy as np
import pytest

import oracle_lib as O
from oracle_lib import rel_l2

pytestmark = pytest.mark.gpu
BOUND = {0: 2e-6, 1: 2e-3, 4: 2e-6}

SHAPES = [(128, 256, 64), (256, 128, 32), (130, 257, 96), (384, 512, 1024), (100, 200, 4096), (1000, 1000, 40),
          (129, 33, 512), (2048, 64, 256), (300, 300, 64), (257, 512, 160), (512, 384, 2048)]


@pytest.fixture(scope="module")
def ctx():
    from seraph_b200 import api
    c = api.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("pair", [1, 0])
@pytest.mark.parametrize("mode", [0, 1, 4])
@pytest.mark.parametrize("tA,tB,acc", [(0, 1, 0), (0, 0, 0), (1, 0, 1), (0, 1, 1)])
@pytest.mark.parametrize("M,N,K", SHAPES)
def test_tc_gemm_matches_oracle(ctx, M, N, K, tA, tB, acc, mode, pair):
    """pair = 1: tiles of 256 rows on CTA pairs (cta_group::2) where the shape allows; 0: one CTA per tile."""
    if pair and (M <= 128 or N <= 128):
        pytest.skip("shape runs on single CTAs either way")
    r = np.random.default_rng(M + 3 * N + 7 * K + tA + 2 * tB)
    A = r.standard_normal((K, M) if tA else (M, K)).astype(np.float32)
    B = r.standard_normal((N, K) if tB else (K, N)).astype(np.float32)
    C0 = r.standard_normal((M, N)).astype(np.float32)
    ref = C0.copy()
    O.lib().ref_matmul(A, B, ref, M, N, K, tA, tB, acc)
    a, b, c = ctx.upload(A), ctx.upload(B), ctx.upload(C0)
    ctx.set_gemm_mode(mode)
    ctx.set_gemm_pair(pair)
    n0 = ctx.launches()
    ctx.lib.cuda_train_matmul_transpose(ctx.h, a.b, b.b, c.b, M, N, K, tA, tB, acc)
    out = c.numpy(shape=(M, N))
    ctx.set_gemm_mode(4)
    ctx.set_gemm_pair(1)
    ctx.check()
    assert ctx.launches() > n0
    assert rel_l2(out, ref) < BOUND[mode], rel_l2(out, ref)
    ctx.release(a, b, c)


@pytest.mark.parametrize("tA,tB,acc", [(0, 1, 0), (0, 0, 1), (1, 0, 0), (1, 0, 1)])
@pytest.mark.parametrize("M,N,K", [(8, 512, 1024), (61, 1408, 512), (264, 136, 72), (256, 128, 64), (512, 264, 1000), (2056, 8, 4096), (24, 16, 8192)])
def test_grouped_kernel_at_tile_edges(ctx, M, N, K, tA, tB, acc):
    """The persistent kernel of grouped products from eight rows or columns up: single and partial tiles of 256, a short last block of k, tiles cut
    along k."""
    r = np.random.default_rng(M + N + K)
    A = r.standard_normal((K, M) if tA else (M, K)).astype(np.float32)
    B = r.standard_normal((N, K) if tB else (K, N)).astype(np.float32)
    C0 = r.standard_normal((M, N)).astype(np.float32)
    ref = C0.copy()
    O.lib().ref_matmul(A, B, ref, M, N, K, tA, tB, acc)
    a, b, c = ctx.upload(A), ctx.upload(B), ctx.upload(C0)
    ctx.lib.cuda_train_matmul_transpose(ctx.h, a.b, b.b, c.b, M, N, K, tA, tB, acc)
    out = c.numpy(shape=(M, N))
    ctx.check()
    assert rel_l2(out, ref) < BOUND[4], rel_l2(out, ref)
    ctx.release(a, b, c)


@pytest.mark.parametrize("mode", [4, 2])
@pytest.mark.parametrize("tA,tB,acc", [(0, 1, 0), (0, 0, 1), (1, 0, 1)])
@pytest.mark.parametrize("M,N,K", [(64, 512, 512), (64, 520, 1408), (512, 520, 1408), (2048, 2816, 256), (5800, 520, 512), (5800, 1000, 512), (10240, 344, 64),
                                   (18944, 88, 64), (4096, 2048, 136)])
def test_grouped_kernel_widths_of_tiles(ctx, M, N, K, tA, tB, acc, mode):
    """Tiles of 64, 128, 192 and 256 columns, whole and in pieces, with ragged last tiles; several items per CTA pair where a warp sends an odd number of
    blocks of a tile out (88 columns are three of a half tile's four), so that its staging buffers change turns.  The bounds are those of every product."""
    r = np.random.default_rng(M + 2 * N + 3 * K + tA)
    A = r.standard_normal((K, M) if tA else (M, K)).astype(np.float32)
    B = r.standard_normal((N, K) if tB else (K, N)).astype(np.float32)
    C0 = r.standard_normal((M, N)).astype(np.float32)
    ref = (A.T if tA else A).astype(np.float64) @ (B.T if tB else B).astype(np.float64) + (C0 if acc else 0)
    a, b, c = ctx.upload(A), ctx.upload(B), ctx.upload(C0)
    ctx.set_gemm_mode(mode)
    ctx.lib.cuda_train_matmul_transpose(ctx.h, a.b, b.b, c.b, M, N, K, tA, tB, acc)
    out = c.numpy(shape=(M, N))
    ctx.set_gemm_mode(4)
    ctx.check()
    bound = BOUND[4] if mode == 4 else BOUND[1]
    assert rel_l2(out, ref) < bound, rel_l2(out, ref)
    for y in range(0, M, 256):                        # a wrong tile does not hide in the norm of the whole
        assert rel_l2(out[y:y + 256], ref[y:y + 256]) < 2 * bound
    ctx.release(a, b, c)


@pytest.mark.parametrize("tA,tB,acc", [(0, 1, 0), (0, 0, 1), (1, 0, 1)])
@pytest.mark.parametrize("M,N,K,single", [(8, 512, 1024, 0), (24, 2048, 512, 0), (512, 16, 4096, 0), (64, 128, 248, 0), (64, 128, 256, 1), (32, 512, 128, 1)])
def test_single_pass_mode_keeps_small_products_accurate(ctx, M, N, K, single, tA, tB, acc):
    """use_bf16 / mode 2: operands of 11 significant bits from 32 rows and columns and 2^21 multiply-adds up, FP32 accuracy below."""
    r = np.random.default_rng(M + N + K)
    A = r.standard_normal((K, M) if tA else (M, K)).astype(np.float32)
    B = r.standard_normal((N, K) if tB else (K, N)).astype(np.float32)
    C0 = r.standard_normal((M, N)).astype(np.float32)
    ref = C0.copy()
    O.lib().ref_matmul(A, B, ref, M, N, K, tA, tB, acc)
    a, b, c = ctx.upload(A), ctx.upload(B), ctx.upload(C0)
    ctx.set_gemm_mode(2)
    ctx.lib.cuda_train_matmul_transpose(ctx.h, a.b, b.b, c.b, M, N, K, tA, tB, acc)
    out = c.numpy(shape=(M, N))
    ctx.set_gemm_mode(4)
    ctx.check()
    e = rel_l2(out, ref)
    assert (1e-4 < e < BOUND[1]) if single else e < BOUND[4], e
    ctx.release(a, b, c)


@pytest.mark.parametrize("kind", ["normal", "outlier", "one element", "zeros", "inf", "nan"])
@pytest.mark.parametrize("M,N,K", [(512, 256, 1024), (64, 128, 256), (1000, 264, 136), (4200, 264, 1024)])
def test_scale_of_the_parts_is_checked_against_every_element(ctx, M, N, K, kind):
    """The scale of an operand's FP16 parts is guessed from 16384 of its elements; one that FP16 cannot hold under it (an element that few samples
    hit, the only one that is not zero) must give the scale of the true maximum, and not the overflow of the guessed one."""
    r = np.random.default_rng(M + K)
    A, B = r.standard_normal((M, K)).astype(np.float32), r.standard_normal((N, K)).astype(np.float32)
    if kind in ("one element", "zeros"):
        A[:] = 0
    for y, x in ([(M - 3, K - 5), (M // 2, 77)] if kind not in ("normal", "zeros") else []):
        A[y, x] = {"outlier": 3.0e5, "one element": -7.25, "inf": np.inf, "nan": np.nan}[kind]
    a, b, c = ctx.upload(A), ctx.upload(B), ctx.zeros(M * N)
    ctx.lib.cuda_train_matmul_transpose(ctx.h, a.b, b.b, c.b, M, N, K, 0, 1, 0)
    out = c.numpy(shape=(M, N))
    ctx.check()
    if kind in ("inf", "nan"):
        assert not np.isfinite(out[[M - 3, M // 2]]).any() and (kind == "inf" or np.isfinite(np.delete(out, [M - 3, M // 2], 0)).all())
    else:
        # parts hold 22 bits of what is within 2^-17 of the largest element (3e5 is 2^18: elements near 1 keep 21) and 2^-39 of it below
        ref = A.astype(np.float64) @ B.T.astype(np.float64)
        for y in range(0, M, 64):
            assert rel_l2(out[y:y + 64], ref[y:y + 64]) < BOUND[4] or not ref[y:y + 64].any() and not out[y:y + 64].any()
    ctx.release(a, b, c)


@pytest.mark.parametrize("M,K,peak,unit", [(8, 256, 1.0, 1.0), (120, 256, 1.99, 1.0), (512, 64, 1.99, 1.0), (520, 64, 1.0, 1.0), (512, 256, 3.9, 1.0), (513, 256, 1.99, 1.0),
                                           (1024, 256, 2.0 ** 80, 1.0), (1024, 256, 1.99, 2.0 ** -60), (1025, 256, 1.0, 1.0), (4096, 256, 3.9, 1.0), (4097, 256, 1.99, 2.0 ** -60),
                                           (4096, 256, 2.0 ** 80, 1.0)] +
                         [(4200, 1024, p, u) for p in (1.0, 1.99, 2.6, 3.9, 7.0) for u in (1.0, 2.0 ** -60)] + [(4200, 1024, 2.0 ** 80, 1.0)])
def test_parts_keep_the_bits_of_the_true_scale(ctx, M, K, peak, unit):
    """An operand times the identity is its two parts, added: under the scale of its true maximum, 2^s with max 2^s in [2^14, 2^15), each element is within
    2^-23 of itself (hi and lo part, 11 bits each, rounded to nearest) or within half of FP16's smallest step, 2^-25, whichever is larger.  No guess of
    that scale may cost more.  The largest element lies where a sample of 16384 need not see it, among others below 1.  Up to 1024 x 256 elements one launch
    of clusters of one to eight CTAs prepares an operand, 8192 float4s a CTA; up to 16 MB the maximum is found first; beyond that it is guessed."""
    r = np.random.default_rng(M)
    A = (r.choice([-1, 1], (M, K)) * 2.0 ** r.uniform(-34, 0, (M, K))).astype(np.float32)
    A[M - 3, K - 5] = peak
    A *= np.float32(unit)
    top = float(np.abs(A).max())
    a, b, c = ctx.upload(A), ctx.upload(np.eye(K, dtype=np.float32)), ctx.zeros(M * K)
    ctx.lib.cuda_train_matmul_transpose(ctx.h, a.b, b.b, c.b, M, K, K, 0, 1, 0)
    out = c.numpy(shape=(M, K)).astype(np.float64)
    ctx.check()
    s = 14 - int(np.floor(np.log2(top)))
    bound = np.maximum(np.abs(A) * 2.0 ** -23, 2.0 ** (-25 - s))
    worst = float((np.abs(out - A) / bound).max())
    assert worst <= 1.0, worst
    ctx.release(a, b, c)


@pytest.mark.parametrize("peak", [1.0, 1.99, 3.9, 7.0])
@pytest.mark.parametrize("M", [120, 520, 1032])
def test_parts_do_not_depend_on_the_way_they_are_made(ctx, M, peak):
    """The same operand beside a small one (one launch, or the maximum first: from 1025 rows on) and beside one of 18 MB (the scale from a sample): the same parts."""
    K, N = 256, 17408
    r = np.random.default_rng(M)
    A = (r.choice([-1, 1], (M, K)) * 2.0 ** r.uniform(-34, 0, (M, K))).astype(np.float32)
    A[M - 3, K - 5] = peak
    E = np.zeros((N, K), np.float32)
    E[:K] = np.eye(K)
    a, e, c, cl = ctx.upload(A), ctx.upload(E), ctx.zeros(M * K), ctx.zeros(M * N)
    ctx.lib.cuda_train_matmul_transpose(ctx.h, a.b, e.b, c.b, M, K, K, 0, 1, 0)
    ctx.lib.cuda_train_matmul_transpose(ctx.h, a.b, e.b, cl.b, M, N, K, 0, 1, 0)
    out, large = c.numpy(shape=(M, K)), cl.numpy(shape=(M, N))
    ctx.check()
    assert np.array_equal(out, large[:, :K]) and not large[:, K:].any()
    ctx.release(a, e, c, cl)


def test_tc_gemm_long_k_and_reproducible(ctx):
    """K = 16384 (longer than the 8192-token reduction of the weight gradients): accumulation error stays in bound."""
    M, N, K = 256, 512, 16384
    r = np.random.default_rng(5)
    A, B = r.standard_normal((M, K)).astype(np.float32), r.standard_normal((N, K)).astype(np.float32)
    ref = np.zeros((M, N), np.float32)
    O.lib().ref_matmul(A, B, ref, M, N, K, 0, 1, 0)
    a, b, c, c2 = ctx.upload(A), ctx.upload(B), ctx.zeros(M * N), ctx.zeros(M * N)
    ctx.lib.cuda_train_matmul_transpose(ctx.h, a.b, b.b, c.b, M, N, K, 0, 1, 0)
    ctx.lib.cuda_train_matmul_transpose(ctx.h, a.b, b.b, c2.b, M, N, K, 0, 1, 0)
    o1, o2 = c.numpy(shape=(M, N)), c2.numpy(shape=(M, N))
    ctx.check()
    e = rel_l2(o1, ref)
    print("FP32-accurate tensor-core GEMM, K=16384: rel-L2 vs FP64 accumulate =", e)
    assert e < 2e-6 and np.array_equal(o1, o2)
    # the same product with whole tiles only (no k pieces in the last wave) meets the same bound
    ctx.set_gemm_tail_split(0)
    ctx.lib.cuda_train_matmul_transpose(ctx.h, a.b, b.b, c2.b, M, N, K, 0, 1, 0)
    o3 = c2.numpy(shape=(M, N))
    ctx.set_gemm_tail_split(1)
    ctx.check()
    assert rel_l2(o3, ref) < 2e-6
    ctx.release(a, b, c, c2)


@pytest.mark.parametrize("mode", [4, 0])
@pytest.mark.parametrize("tA,tB", [(0, 1), (0, 0), (1, 0)])
@pytest.mark.parametrize("M,N,K", [(384, 512, 1024), (130, 257, 96), (1000, 1000, 40), (2048, 2048, 512), (256, 512, 16384),
                                   (4096, 1024, 256), (300, 300, 64), (2049, 6144, 128)])
def test_epilogue_leaves_the_largest_magnitude_of_the_output(ctx, M, N, K, tA, tB, mode):
    """Inside a training step the product's epilogue (and the fix-up pass of tiles whose k range was cut into pieces) leaves
    max |C| behind, and the kernels that write the next operand as FP16 parts scale by bounds formed from it: a value below the
    true maximum would overflow FP16.  The maximum of floats is exact, so it must equal the maximum of the downloaded result,
    with ragged edges, with whole and split tiles, in every layout."""
    import ctypes
    r = np.random.default_rng(11 * M + 5 * N + K + tA + 2 * tB)
    A = r.standard_normal((K, M) if tA else (M, K)).astype(np.float32)
    B = r.standard_normal((N, K) if tB else (K, N)).astype(np.float32)
    A[r.integers(0, A.shape[0]), r.integers(0, A.shape[1])] = 37.0            # one outlier, so that the maximum sits in one tile
    a, b, c = ctx.upload(A), ctx.upload(B), ctx.upload(np.full((M, N), 1e9, np.float32))
    ctx.set_gemm_mode(mode)
    am = ctypes.c_float(-1.0)
    got = ctx.lib.seraph_b200_matmul_amax(ctx.h, a.b, b.b, c.b, M, N, K, tA, tB, ctypes.byref(am))
    out = c.numpy(shape=(M, N))
    ctx.set_gemm_mode(4)
    ctx.check()
    assert got == 1, "shape expected on the tensor-core kernel"
    assert am.value == float(np.abs(out).max()), (am.value, float(np.abs(out).max()))
    ctx.release(a, b, c)
