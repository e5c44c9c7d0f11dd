"""The work a user of this library has it do, as measurable cases.

Every case goes through the public C entry points (over the ctypes mirror seraph_b200.api):

  full   cuda_train_step_gpu_full / _full_batch: forward, loss, backward and AdamW of a full-weight model
  lora   cuda_train_step_gpu_lora / _lora_batch: the same for adapters on a frozen base
  eval   cuda_evaluate: mean loss and perplexity over validation samples
  attn   cuda_train_batch_attention_packed and its backward, for hosts that call single operations

The models are the ones of this repository's benchmark and tests: the 33M Llama-style decoder (8 heads of 64), slices of the
Qwen3-1.7B-shaped decoder (16/8 heads of 128, learned per-head q/k norm) and of the Mistral-7B-shaped one (32/8 heads of 128,
separate lm_head).  Token ids are uniform, weights N(0, 0.02) with norm scales near 1, as there.

The outputs are the loss and the resident device arrays the context publishes (parameters, gradients and both Adam moments of
the trained set), read in place through its cuda_buffer_t views."""
import ctypes as C
import random

import numpy as np
import torch

from seraph_b200 import api
from seraph_b200.config import ModelCfg

M33 = dict(V=8192, d=512, L=8, Hq=8, Hkv=8, hd=64, F=1408, theta=10000.0)
QWEN = dict(d=2048, L=2, Hq=16, Hkv=8, hd=128, F=6144, theta=1e6, head_norm=1)
MISTRAL = dict(V=32000, d=4096, L=2, Hq=32, Hkv=8, hd=128, F=14336, theta=1e6, untied=1)


def model(case):
    if case["model"] == "33m":
        return ModelCfg(**M33)
    if case["model"] == "qwen":
        return ModelCfg(V=case["vocab"], **QWEN)
    return ModelCfg(**MISTRAL)


def lengths(case):
    """Token counts of the packed sequences: all `seq`, or (ragged) from a quarter of it up, odd ones among them, the longest `seq`."""
    B, S = case["batch"], case["seq"]
    if not case["ragged"]:
        return [S] * B
    r = random.Random(1000 * B + S)
    return [S] + [r.randint(max(2, S // 4), S) for _ in range(B - 1)]


# ----------------------------------------------------------------------------------------------------------------------
# the cases
# ----------------------------------------------------------------------------------------------------------------------
def full(name, mdl, batch, seq, ragged=False, vocab=0, clip=0.0, bf16=False):
    return dict(name=name, kind="full", model=mdl, vocab=vocab, batch=batch, seq=seq, ragged=ragged, clip=clip, bf16=bf16)


def lora(name, mdl, batch, seq, rank, mask, ragged=False, vocab=0):
    return dict(name=name, kind="lora", model=mdl, vocab=vocab, batch=batch, seq=seq, ragged=ragged, rank=rank, mask=mask)


def evaluation(name, mdl, batch, seq, ragged=True, vocab=0):
    return dict(name=name, kind="eval", model=mdl, vocab=vocab, batch=batch, seq=seq, ragged=ragged)


def attention(name, batch, seq, heads, kv_heads, head_dim, ragged=False):
    return dict(name=name, kind="attn", batch=batch, seq=seq, ragged=ragged, heads=heads, kv_heads=kv_heads, head_dim=head_dim)


def listed():
    return [
        # one short sample, no packing: what the trainer does at batch size 1; launches and latency are nearly all of it
        full("33m full 1x61", "33m", 1, 61),
        # the baseline's first configuration, with the clipping it names
        full("33m full 8x256 clip", "33m", 8, 256, clip=1.0),
        # a packed batch as the trainer fills it from samples of unequal length
        full("33m full 24 ragged <=383", "33m", 24, 383, ragged=True),
        # the same model with the context's use_bf16 switch (reduced-precision products)
        full("33m full 8x256 use_bf16", "33m", 8, 256, bf16=True),
        # two layers of the benchmark model: the shape of its layers at half its batch
        full("qwen full 2x2048", "qwen", 2, 2048, vocab=16384),
        # the benchmark model's micro-batch and vocabulary on two layers: the loss and the LM head weigh most
        full("qwen full 4x2048 vocab 152k", "qwen", 4, 2048, vocab=151936),
        # long and short samples packed together
        full("qwen full 5 ragged <=1500", "qwen", 5, 1500, ragged=True, vocab=16384),
        # rank-8 q and v adapters (the trainer's default set) on the small model
        lora("33m lora r8 qv 4x128", "33m", 4, 128, 8, 0b0000101),
        # the baseline's adapter configuration on two layers: rank 16 on q, k, v, o
        lora("qwen lora r16 qkvo 4x2048", "qwen", 4, 2048, 16, 0b0001111, vocab=32768),
        # rank 64 on all seven projections, long sequences, 4:1 head grouping
        lora("mistral lora r64 all 2x4096", "mistral", 2, 4096, 64, 0x7F),
        # validation between epochs: 64 samples of unequal length
        evaluation("33m evaluate 64 ragged <=256", "33m", 64, 256),
        # the baseline's isolated attention configuration, forward and backward
        attention("attention 8x2048 16x128", 8, 2048, 16, 16, 128),
    ]


def spread(rng, lo, hi):
    """log-uniform whole number"""
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["33m", "33m", "qwen", "qwen", "lora33m", "loraq", "loram", "eval", "attn", "attn"])
    ragged = rng.random() < 0.5
    if kind == "33m":
        seq = spread(rng, 16, 1024)
        c = full("", "33m", spread(rng, 1, max(1, min(64, 8192 // seq))), seq, ragged, 0, rng.choice([0.0, 1.0]), rng.random() < 0.25)
    elif kind == "qwen":
        seq = spread(rng, 128, 2048)
        c = full("", "qwen", spread(rng, 1, max(1, min(32, 8192 // seq))), seq, ragged, rng.choice([16384, 32768, 151936]))
    elif kind == "lora33m":
        seq = spread(rng, 16, 1024)
        c = lora("", "33m", spread(rng, 1, max(1, min(64, 8192 // seq))), seq, rng.choice([4, 8, 16]), rng.choice([0b0000101, 0b0001111, 0x7F]), ragged)
    elif kind == "loraq":
        seq = spread(rng, 128, 2048)
        c = lora("", "qwen", spread(rng, 1, max(1, min(32, 8192 // seq))), seq, rng.choice([8, 16, 32]), rng.choice([0b0000101, 0b0001111, 0x7F]), ragged, 32768)
    elif kind == "loram":
        seq = spread(rng, 256, 4096)
        c = lora("", "mistral", spread(rng, 1, max(1, min(16, 8192 // seq))), seq, rng.choice([16, 64]), rng.choice([0b0001111, 0x7F]), ragged)
    elif kind == "eval":
        mdl = rng.choice(["33m", "qwen"])
        seq = spread(rng, 32, 1024)
        c = evaluation("", mdl, spread(rng, 1, max(1, min(256, 32768 // seq))), seq, ragged, 32768 if mdl == "qwen" else 0)
    else:
        seq = spread(rng, 64, 4096)
        hd = rng.choice([64, 128])
        kv = rng.choice([2, 4, 8])
        c = attention("", spread(rng, 1, max(1, min(32, 16384 // seq))), seq, kv * rng.choice([1, 2, 4]) if kv < 8 else kv * rng.choice([1, 2]), kv, hd, ragged)
    del c["name"]
    return c


# ----------------------------------------------------------------------------------------------------------------------
# what the context publishes on the device
# ----------------------------------------------------------------------------------------------------------------------
_PB = C.POINTER(api.CudaBuffer)
_PPB = C.POINTER(_PB)
_TENSORS = ["q", "k", "v", "o", "gate", "up", "down", "in_norm", "post_norm"]


class _CtxHead(C.Structure):
    """cuda_train_context_t of include/seraph_b200_abi.h"""
    _fields_ = (
        [("device_id", C.c_int), ("stream", C.c_void_p), ("initialized", C.c_int), ("gpu_", C.c_int * 11), ("use_bf16", C.c_int),
         ("use_flash_attn", C.c_int), ("batch_size", C.c_int), ("tiles_", C.c_int * 5),
         ("opt_", C.c_void_p * 4), ("max_buffer_size", C.c_size_t), ("fwd_", C.c_void_p * 3), ("max_fwd_buffer_size", C.c_size_t),
         ("attn_", C.c_void_p * 4), ("max_attn_buffer_size", C.c_size_t), ("act_", C.c_void_p * 8), ("max_fwd_act_bytes", C.c_size_t),
         ("cache_dims_", C.c_int * 5), ("cache_", C.c_void_p * 13), ("train_", C.c_void_p * 18), ("weights_dims_", C.c_int * 6),
         ("embed", _PB * 4), ("final_norm", _PB * 4)]
        + [(t, _PPB * 4) for t in _TENSORS]
        + [("debug_nan_flags", _PB), ("lora_gpu", C.c_void_p)])


class _LoraAdapter(C.Structure):
    _fields_ = [(k, _PPB) for k in ("A", "B", "gA", "gB", "mA", "vA", "mB", "vB")] + [("active", C.c_int)]


class _LoraState(C.Structure):
    _fields_ = [("num_layers", C.c_int), ("rank", C.c_int), ("alpha", C.c_float), ("scale", C.c_float)] + \
               [(t, _LoraAdapter) for t in ("q", "k", "v", "o", "gate", "up", "down")]


class Owner:
    """A context with what was made in it; closed when the last reference (a state, or an output that views its memory) goes."""

    def __init__(self):
        self.ctx, self.st = api.Context(0), None

    def head(self):
        return _CtxHead.from_address(self.ctx.h)

    def __del__(self):
        try:
            if self.st is not None:
                self.st.close()
            self.ctx.close()
        except Exception:
            pass


class _Array:
    def __init__(self, owner, addr, n):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f4", "data": (addr, False), "version": 2}


def on_device(owner, addr, n):
    """float32 tensor over n floats at a device address of `owner`"""
    return torch.as_tensor(_Array(owner, addr, n), device="cuda")


def _address(buffer):
    return C.cast(buffer.contents.data, C.c_void_p).value


def trained_arrays(owner, cfg, n):
    """The parameters, gradients and Adam moments of a full-weight model: each kind is one array in the flat parameter order."""
    h, out = owner.head(), {}
    for k, name in enumerate(("weights", "grads", "m", "v")):
        base = _address(h.embed[k])
        last = _address(h.post_norm[k][cfg.L - 1])
        assert last + 4 * cfg.d == base + 4 * n, "the published views are one flat array"
        out[name] = on_device(owner, base, n)
    return out


def adapter_arrays(owner, cfg, n, mask):
    h = _LoraState.from_address(owner.head().lora_gpu)
    first = getattr(h, cfg.LORA_NAMES[(mask & -mask).bit_length() - 1])
    return {name: on_device(owner, _address(getattr(first, f)[0]), n) for name, f in (("adapters", "A"), ("grads", "gA"), ("m", "mA"), ("v", "vA"))}


# ----------------------------------------------------------------------------------------------------------------------
# states
# ----------------------------------------------------------------------------------------------------------------------
def seeded_weights(cfg, gen):
    """N(0, 0.02) weights, norm scales 1 with a little spread, flat, on the host"""
    p = torch.empty(cfg.n_params(), device="cuda").normal_(0.0, 0.02, generator=gen)
    for name, shp, off in cfg.tensors():
        if name.endswith("norm"):
            p[off:off + shp[0]].mul_(2.0).add_(1.0)
    return p.cpu().numpy()


def seeded_extras(cfg, gen):
    tens, n = cfg.extras_tensors()
    x = torch.empty(n, device="cuda").normal_(0.0, 0.02, generator=gen)
    for name, shp, off in tens:
        if name.endswith("norm"):
            x[off:off + shp[0]].mul_(2.0).add_(1.0)
    return x.cpu().numpy()


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    lens = lengths(case)
    starts = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    T = int(starts[-1])
    own = Owner()
    ctx = own.ctx
    if case["kind"] == "attn":
        return prepare_attention(case, gen, own, starts, T)
    cfg = model(case)
    tokens = torch.randint(0, cfg.V, (T,), device="cuda", generator=gen, dtype=torch.int32).cpu().numpy()
    own.st = api.TrainState(cfg, seeded_weights(cfg, gen), lean=True)
    extras = seeded_extras(cfg, gen)
    if extras.size:
        rc = ctx.lib.seraph_b200_set_model_extras(ctx.h, cfg.head_norm, cfg.untied, extras.ctypes.data, extras.size)
        assert rc == 0, rc
    s = dict(kind=case["kind"], own=own, tokens=tokens, starts=starts, views={})
    if case["kind"] == "lora":
        _, n = cfg.lora_tensors(case["rank"], case["mask"])
        adapters = torch.empty(n, device="cuda").normal_(0.0, 0.02, generator=gen).cpu().numpy()      # past the first steps: B is no longer zero
        own.st.attach_lora(case["rank"], 2.0 * case["rank"], case["mask"], adapters)
    if case.get("bf16"):
        own.head().use_bf16 = 1
    if case.get("clip"):
        assert ctx.lib.seraph_b200_set_grad_clip(ctx.h, case["clip"]) == 0
    # the loss before training, on a few tokens: the model is on the device from here on
    few = np.ascontiguousarray(tokens[:min(16, lens[0])])
    ctx.lib.cuda_eval_forward(own.st.h, few.ctypes.data, len(few), ctx.h)
    ctx.check()
    if case["kind"] == "full":
        s["views"] = trained_arrays(own, cfg, own.st.n)
    elif case["kind"] == "lora":
        s["views"] = adapter_arrays(own, cfg, own.st.n_lora, case["mask"])
    else:
        s["offsets"], s["longest"] = np.ascontiguousarray(starts[:-1]), max(lens)
    return s


def prepare_attention(case, gen, own, starts, T):
    ctx = own.ctx
    q, kv, h = case["heads"] * case["head_dim"], case["kv_heads"] * case["head_dim"], case["heads"]
    s = dict(kind="attn", own=own, dims=(T, len(starts) - 1, h, case["kv_heads"], case["head_dim"], int(np.diff(starts).max())),
             starts=ctx.upload(starts.astype(np.uint32)), buf={}, views={}, kv_bytes=4 * T * kv)
    for name, n, random_input in (("Q", q, 1), ("K", kv, 1), ("V", kv, 1), ("dO", q, 1), ("out", q, 0), ("lse", h, 0), ("dQ", q, 0), ("dK", kv, 0), ("dV", kv, 0)):
        b = s["buf"][name] = ctx.empty(T * n).b
        v = on_device(own, _address(b), T * n)
        if random_input:
            v.normal_(generator=gen)
        else:
            s["views"][name] = v
    torch.cuda.synchronize()
    return s


# ----------------------------------------------------------------------------------------------------------------------
# one pass
# ----------------------------------------------------------------------------------------------------------------------
def run(s):
    own, kind = s["own"], s["kind"]
    ctx, lib = own.ctx, own.ctx.lib
    if kind == "attn":
        b, d = s["buf"], s["dims"]
        lib.cuda_train_batch_attention_packed(ctx.h, b["Q"], b["K"], b["V"], b["out"], b["lse"], s["starts"].b, *d)
        lib.cuda_train_fill_buffer(ctx.h, b["dK"], 0, s["kv_bytes"])      # the backward adds into dK and dV
        lib.cuda_train_fill_buffer(ctx.h, b["dV"], 0, s["kv_bytes"])
        lib.cuda_train_batch_attention_backward_packed(ctx.h, b["Q"], b["K"], b["V"], b["out"], b["lse"], b["dO"], b["dQ"], b["dK"], b["dV"],
                                                       s["starts"].b, *d)
        return s["views"]
    tok, ss = s["tokens"], s["starts"]
    if kind == "eval":
        ppl = C.c_float(0.0)
        loss = lib.cuda_evaluate(own.st.h, tok.ctypes.data, len(tok), s["offsets"].ctypes.data, len(s["offsets"]), s["longest"], 0, ctx.h, C.byref(ppl))
        return {"loss": float(loss), "perplexity": ppl.value}
    one = len(ss) == 2
    if kind == "full":
        loss = (lib.cuda_train_step_gpu_full(own.st.h, tok.ctypes.data, len(tok), ctx.h) if one else
                lib.cuda_train_step_gpu_full_batch(own.st.h, tok.ctypes.data, len(tok), ss.ctypes.data, len(ss) - 1, ctx.h))
    else:
        loss = (lib.cuda_train_step_gpu_lora(own.st.h, tok.ctypes.data, len(tok), ctx.h) if one else
                lib.cuda_train_step_gpu_lora_batch(own.st.h, tok.ctypes.data, len(tok), ss.ctypes.data, len(ss) - 1, ctx.h))
    return {"loss": float(loss), **s["views"]}


# ----------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without, and how far two correct implementations may differ
# ----------------------------------------------------------------------------------------------------------------------
def work(case):
    lens = lengths(case)
    T, sq = float(sum(lens)), float(sum(n * n for n in lens))
    if case["kind"] == "attn":
        H, KV, D = case["heads"], case["kv_heads"], case["head_dim"]
        # Q, K, V, dO in; out, lse, dQ, dK, dV out (the backward's reads of out and lse come after they were written: once more)
        return {"bytes": 4.0 * T * (5 * H * D + 4 * KV * D + 2 * H), "flops": 7.0 * H * D * sq}
    cfg = model(case)
    lin = cfg.L * (2 * cfg.qd * cfg.d + 2 * cfg.kvd * cfg.d + 3 * cfg.F * cfg.d)
    head = cfg.V * cfg.d
    params = cfg.n_params() + cfg.extras_tensors()[1]
    attn = cfg.L * cfg.qd * sq
    if case["kind"] == "eval":
        return {"bytes": 4.0 * params, "flops": 2.0 * (lin + head) * T + 2.0 * attn}
    if case["kind"] == "full":
        # parameters and both moments in; parameters, gradients and both moments out
        return {"bytes": 28.0 * params, "flops": 6.0 * (lin + head) * T + 7.0 * attn}
    n = cfg.lora_tensors(case["rank"], case["mask"])[1]
    return {"bytes": 4.0 * params + 28.0 * n, "flops": 4.0 * (lin + head) * T + 7.0 * attn + 6.0 * n * T}


def tolerance(case):
    if case.get("bf16"):
        return {"rel": 5e-3, "max": 0.2}       # products of operands with 11 significant bits
    # FP32 sums through the whole model; the second moment is a square.  "max": AdamW divides a gradient by its own magnitude, so a
    # weight whose gradient is all rounding may move the other way (twice the step's learning rate, against weights of 0.02)
    return {"rel": 2e-5, "max": 2e-3}
