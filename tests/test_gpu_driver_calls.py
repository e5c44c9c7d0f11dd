"""What a training step asks of the CUDA runtime besides its kernel launches: calls are counted by a small library that is loaded in front of the
runtime, in a process of its own."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
static void* next(const char* name) { return dlsym(dlopen("libcudart.so.12", RTLD_NOW | RTLD_NOLOAD), name); }
int n_malloc, n_memset;
int cudaMalloc(void** p, size_t n) {
    static int (*f)(void**, size_t);
    if (!f) f = (int (*)(void**, size_t))next("cudaMalloc");
    n_malloc++;
    return f(p, n);
}
int cudaMemsetAsync(void* p, int v, size_t n, void* s) {
    static int (*f)(void*, int, size_t, void*);
    if (!f) f = (int (*)(void*, int, size_t, void*))next("cudaMemsetAsync");
    n_memset++;
    return f(p, v, n, s);
}
"""

PRELUDE = """
import ctypes as C, sys
import numpy as np
sys.path.insert(0, %r)
import oracle_lib as O
from seraph_b200 import api
SHIM = C.CDLL(%r)
def count(name): return C.c_int.in_dll(SHIM, name).value
def lora_state(ctx, cfg, rank, mask):
    ctx.lib.seraph_b200_reset_model(ctx.h)
    st = api.TrainState(cfg, cfg.init_params(1))
    n = cfg.lora_tensors(rank, mask)[1]
    st.attach_lora(rank, 2.0 * rank, mask, (0.02 * np.random.default_rng(2).standard_normal(n)).astype(np.float32))
    return st
def step(ctx, cfg, st, T):
    tok = np.random.default_rng(T).integers(0, cfg.V, T).astype(np.int32)
    before = count("n_malloc"), count("n_memset")
    assert api.step_lora_batch(ctx, st, tok, [0, T // 3, T]) > 0
    ctx.check()
    return count("n_malloc") - before[0], count("n_memset") - before[1]
cfg = O.ModelCfg(V=512, d=256, L=2, Hq=4, Hkv=2, hd=64, F=512)
ctx = api.Context(0)
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    d = tmp_path_factory.mktemp("shim")
    (d / "shim.c").write_text(SHIM)
    so = str(d / "shim.so")
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", so, str(d / "shim.c"), "-ldl"], check=True)

    def go(code):
        r = subprocess.run([sys.executable, "-c", PRELUDE % (HERE, so) + code], env=dict(os.environ, LD_PRELOAD=so), capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        return r.stdout
    return go


def test_clearing_in_a_lora_step_does_not_grow_with_its_adapters(run):
    out = run("""
for mask in (0x05, 0x7F):
    st = lora_state(ctx, cfg, 8, mask)
    for _ in range(3): m = step(ctx, cfg, st, 512)[1]
    print(m)
    st.close()
""").split()
    few, many = (int(x) for x in out)
    assert few > 0 and many == few, out


def test_lora_steps_of_lengths_seen_before_allocate_nothing(run):
    out = run("""
st = lora_state(ctx, cfg, 16, 0x7F)
print(*[step(ctx, cfg, st, T)[0] for _ in range(2) for T in (512, 300, 40, 411)])
st.close()
""").split()
    calls = [int(x) for x in out]
    assert calls[0] > 0 and calls[4:] == [0, 0, 0, 0], calls


def test_a_smaller_product_than_the_last_allocates_nothing(run):
    """Operands are prepared in one, two or three launches by their size; whichever way it is, a call that follows a larger one needs no more memory."""
    out = run("""
for M, K in ((8192, 1024), (4096, 512), (512, 256)):
    a, b, c = ctx.zeros(M * K), ctx.zeros(K * K), ctx.zeros(M * K)
    before = count("n_malloc")
    ctx.lib.cuda_train_matmul_transpose(ctx.h, a.b, b.b, c.b, M, K, K, 0, 1, 0)
    ctx.check()
    print(count("n_malloc") - before)
    ctx.release(a, b, c)
""").split()
    assert int(out[0]) > 0 and out[1:] == ["0", "0"], out
