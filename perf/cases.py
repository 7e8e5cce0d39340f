"""What the framework's performance is measured on: the work that a user's program has it do on one GPU, through
the public entry points.

Families:

* ``ep``    one expert-parallel exchange: ``EpDispatcher.dispatch`` and ``EpDispatcher.combine``;
* ``moe``   one forward pass of ``models.MoEFeedForward`` (dispatch, grouped expert GEMMs, combine), prefill batches
            and low-latency decode batches, e4m3 and bf16 experts;
* ``tp``    one forward pass of ``models.TensorParallelMLP`` / ``TensorParallelMLPFp8``;
* ``gemm``  one ``gemm_bf16`` or ``gemm_fp8_blockscaled`` call on ordinary tensors;
* ``coll``  one stream-ordered collective between several PEs that one process hosts on the GPU.

Every family but ``coll`` runs with one PE in the process, as ``bench.py`` does on one GPU.
"""
from __future__ import annotations

import torch

import rocshmem_b200 as shm
from rocshmem_b200.models import moe_ffn, tp_mlp
from rocshmem_b200.ops import collectives, gemm, moe

BF16 = torch.bfloat16


def listed():
    """The listed cases."""
    return [
        # The workload of bench.py: a prefill or training micro-batch of 4096 tokens, top-8 of 256 experts, e4m3 rows.
        {"name": "ep_fp8_4096", "kind": "ep", "tokens": 4096, "hidden": 7168, "experts": 256, "top_k": 8,
         "quantize": True, "unused": False},
        # A ragged batch of a smaller model that keeps bf16 rows; some tokens select fewer experts than top-k allows.
        {"name": "ep_bf16_ragged", "kind": "ep", "tokens": 611, "hidden": 4096, "experts": 64, "top_k": 6,
         "quantize": False, "unused": True},
        # Prefill through one rank's experts of a wide mixture-of-experts layer, about 1024 rows per expert.
        {"name": "moe_fp8_prefill", "kind": "moe", "tokens": 2048, "hidden": 7168, "inter": 2048, "experts": 16,
         "top_k": 8, "quantize": True, "fp8_experts": True, "low_latency": False},
        # The same layer in a decode step: 128 tokens, bound by the weights it has to read.
        {"name": "moe_fp8_decode", "kind": "moe", "tokens": 128, "hidden": 7168, "inter": 2048, "experts": 16,
         "top_k": 8, "quantize": True, "fp8_experts": True, "low_latency": True},
        # A ragged prefill batch with bf16 rows and bf16 experts.
        {"name": "moe_bf16_ragged", "kind": "moe", "tokens": 1111, "hidden": 4096, "inter": 1536, "experts": 8,
         "top_k": 4, "quantize": False, "fp8_experts": False, "low_latency": False},
        # A long-prompt prefill through one rank's share (1/8) of a dense SwiGLU MLP.
        {"name": "tp_bf16_8192", "kind": "tp", "m": 8192, "d_model": 8192, "d_ff": 3584, "fp8": False},
        # A medium batch through the block-scaled form of the same layer.
        {"name": "tp_fp8_2048", "kind": "tp", "m": 2048, "d_model": 8192, "d_ff": 3584, "fp8": True},
        # A projection in a decode step: few rows, bound by reading the weight.
        {"name": "gemm_bf16_decode", "kind": "gemm", "m": 32, "n": 7168, "k": 8192, "fp8": False},
        # A ragged number of rows, and dimensions that are no multiple of a tile.
        {"name": "gemm_bf16_ragged", "kind": "gemm", "m": 1000, "n": 4104, "k": 4040, "fp8": False},
        # A small block-scaled projection in a decode step: launch latency and the weight's bytes.
        {"name": "gemm_fp8_decode", "kind": "gemm", "m": 64, "n": 2048, "k": 7168, "fp8": True},
        # A gradient bucket summed over four PEs.
        {"name": "allreduce_bf16_bucket", "kind": "coll", "op": "allreduce", "pes": 4, "elems": 16 << 20,
         "dtype": "bfloat16"},
        # A small fp32 vector (statistics, a norm) summed over four PEs: latency.
        {"name": "allreduce_fp32_small", "kind": "coll", "op": "allreduce", "pes": 4, "elems": 2000,
         "dtype": "float32"},
    ]


def _log(rng, lo, hi):
    """A whole number in [lo, hi], spread evenly over its logarithm."""
    return min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    """One more case of the ranges that the listed ones stand for."""
    kind = rng.choice(["ep", "ep", "moe", "moe", "tp", "gemm", "gemm", "coll"])
    if kind == "ep":
        experts = rng.choice([8, 16, 32, 64, 128, 256])
        return {"kind": "ep", "tokens": _log(rng, 1, 8192), "hidden": 512 * rng.randint(2, 16), "experts": experts,
                "top_k": rng.randint(1, 8), "quantize": rng.random() < 0.6, "unused": rng.random() < 0.3}
    if kind == "moe":
        experts, hidden, inter = rng.choice([(8, 2048, 1024), (8, 4096, 1536), (16, 4096, 1536), (16, 2048, 1024),
                                             (8, 7168, 2048)])
        decode = rng.random() < 0.5
        fp8 = rng.random() < 0.6
        return {"kind": "moe", "tokens": _log(rng, 1, 256) if decode else _log(rng, 128, 2048), "hidden": hidden,
                "inter": inter, "experts": experts, "top_k": rng.randint(1, 8),
                "quantize": fp8 or rng.random() < 0.5, "fp8_experts": fp8, "low_latency": decode}
    if kind == "tp":
        return {"kind": "tp", "m": 128 * _log(rng, 1, 48), "d_model": 512 * rng.randint(2, 16),
                "d_ff": 512 * rng.randint(2, 7), "fp8": rng.random() < 0.5}
    if kind == "gemm":
        fp8 = rng.random() < 0.5
        m = _log(rng, 1, 8192)
        if fp8:
            return {"kind": "gemm", "m": m, "n": 128 * rng.randint(4, 64), "k": 512 * rng.randint(1, 16), "fp8": True}
        n = rng.randint(256, 8192)
        return {"kind": "gemm", "m": m, "n": n if rng.random() < 0.2 else n // 8 * 8, "k": 8 * rng.randint(32, 1024),
                "fp8": False}
    op = rng.choice(["allreduce", "allreduce", "alltoall", "fcollect", "broadcast"])
    elems = _log(rng, 128, 8 << 20)
    return {"kind": "coll", "op": op, "pes": 4, "elems": elems, "dtype": rng.choice(["bfloat16", "float32", "int32"])}


# ---- the runtime and the objects that a program keeps ----------------------------------------------------------

_generation = 0     # counts the initialisations of the runtime: objects of an earlier one are not given back to it
_kept = {}          # layers with their weights, by configuration (the last two)


def _runtime(pes):
    """The runtime with `pes` PEs in this process."""
    global _generation
    if shm.is_initialized() and shm.n_local_pes() == pes:
        return
    while _kept:
        _forget(next(iter(_kept)))
    if shm.is_initialized():
        shm.finalize()
    shm.init(n_local=pes, heap_size="8G" if pes == 1 else "1G", device=0)
    _generation += 1


def _forget(key):
    _kept.pop(key).destroy()


def _layer(key, make):
    """The layer of one configuration, with its weights: a program builds it once and calls it on many inputs."""
    if key in _kept:
        _kept[key] = _kept.pop(key)
    else:
        while len(_kept) >= 2:
            _forget(next(iter(_kept)))
        _kept[key] = make()
    return _kept[key]


class _State:
    """What a program has in hand; its symmetric memory goes back to the heap with it."""

    def __init__(self, give_back=None):
        self._give_back, self._generation = give_back, _generation

    def __del__(self):
        if self._give_back is not None and self._generation == _generation and shm.is_initialized():
            self._give_back()


def _routing(tokens, experts, top_k, g, unused):
    """Top-k gating of N(0, 1) logits with softmax weights."""
    top_k = min(top_k, experts)
    val, idx = torch.randn(tokens, experts, generator=g, device="cuda").topk(top_k, dim=-1)
    idx = idx.to(torch.int32)
    if unused:
        idx[torch.rand(tokens, top_k, generator=g, device="cuda") < 0.15] = -1
    return idx.contiguous(), torch.softmax(val, dim=-1).contiguous()


def _randn(shape, g, scale=1.0):
    return (torch.randn(shape, generator=g, device="cuda") * scale).to(BF16)


def prepare(case, seed):
    """Inputs made from the seed, and the layer, dispatcher or symmetric buffers that a program keeps."""
    kind = case["kind"]
    _runtime(case["pes"] if kind == "coll" else 1)
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    if kind == "ep":
        T, H, E, K = case["tokens"], case["hidden"], case["experts"], min(case["top_k"], case["experts"])
        d = moe.EpDispatcher(E, K, H, T, quantize=case["quantize"])
        s = _State(d.destroy)
        s.d, s.tokens = d, T
        s.x = _randn((T, H), g)
        s.idx, s.w = _routing(T, E, K, g, case["unused"])
        s.y = d.result_buffer()       # the experts' result rows, as they stand when combine is called
        s.y.copy_(_randn(tuple(s.y.shape), g))
    elif kind == "moe":
        T, H, I, E, K = case["tokens"], case["hidden"], case["inter"], case["experts"], case["top_k"]
        key = ("moe", T, H, I, E, K, case["quantize"], case["fp8_experts"], case["low_latency"])
        s = _State()
        s.layer = _layer(key, lambda: moe_ffn.MoEFeedForward(
            E, K, H, I, max_tokens=T, seed=1, quantize=case["quantize"], fp8_experts=case["fp8_experts"],
            low_latency=case["low_latency"]))
        s.x = _randn((T, H), g)
        s.idx, s.w = _routing(T, E, K, g, False)
    elif kind == "tp":
        make = tp_mlp.TensorParallelMLPFp8 if case["fp8"] else tp_mlp.TensorParallelMLP
        key = ("tp", case["m"], case["d_model"], case["d_ff"], case["fp8"])
        s = _State()
        s.layer = _layer(key, lambda: make(case["d_model"], case["d_ff"], case["m"], seed=1))
        s.x = _randn((case["m"], case["d_model"]), g)
    elif kind == "gemm":
        s = _State()
        s.a = _randn((case["m"], case["k"]), g)
        s.b = _randn((case["n"], case["k"]), g, case["k"] ** -0.5)
        if case["fp8"]:
            s.a, s.a_s = moe.fp8_quantize_1x128(s.a)
            s.b, s.b_s = gemm.quantize_weight_128x128(s.b)
    else:
        n, elems, dtype = case["pes"], case["elems"], getattr(torch, case["dtype"])
        if case["op"] == "alltoall":
            elems = (elems + n - 1) // n * n
        src = shm.zeros(elems, dtype)
        dst = shm.zeros(elems * n if case["op"] == "fcollect" else elems, dtype)
        s = _State(lambda: (torch.cuda.synchronize(), shm.free(dst), shm.free(src)))
        s.src, s.dst = src, dst
        for pe in range(n):
            v = shm.local_view(src, pe)
            if dtype.is_floating_point:
                v.copy_(torch.randn(elems, generator=g, device="cuda"))
            else:
                v.copy_(torch.randint(-1000, 1000, (elems,), generator=g, device="cuda"))
        s.dsts = [shm.local_view(dst, pe) for pe in range(n)]
    s.case = case
    torch.cuda.synchronize()
    return s


def run(s):
    """One pass."""
    case = s.case
    kind = case["kind"]
    if kind == "ep":
        r = s.d.dispatch(s.x, s.idx, s.w)
        out = s.d.combine(s.y, s.idx, s.w, s.tokens)
        # Without quantisation there are no scales; word positions that the API does not name are left out.
        got = {"rows": r.recv_x, "expert": r.local_expert_idx(), "gate": r.gate_weights(), "token": r.src_token(),
               "per_expert": r.rows_per_expert(), "out": out}
        if case["quantize"]:
            got["scales"] = r.recv_scales
        return got
    if kind in ("moe", "tp"):
        return s.layer(s.x, s.idx, s.w) if kind == "moe" else s.layer(s.x)
    if kind == "gemm":
        if case["fp8"]:
            return gemm.gemm_fp8_blockscaled(s.a, s.a_s, s.b, s.b_s)
        return gemm.gemm_bf16(s.a, s.b)
    if case["op"] == "allreduce":
        collectives.allreduce_async(s.dst, s.src)
    elif case["op"] == "alltoall":
        collectives.alltoall_async(s.dst, s.src)
    elif case["op"] == "fcollect":
        collectives.fcollect_async(s.dst, s.src)
    else:
        collectives.broadcast_async(s.dst, s.src, 0)
    return s.dsts


def work(case):
    """Bytes that a pass has to read and write, each once, and its floating-point operations."""
    kind = case["kind"]
    if kind == "ep":
        T, H, K = case["tokens"], case["hidden"], case["top_k"]
        row = H + H // 128 * 4 if case["quantize"] else 2 * H
        return {"bytes": T * (2 * H + row + 2 * H + 2 * H + 16 * K), "flops": 2.0 * T * H}
    if kind == "moe":
        T, H, I, E, K = case["tokens"], case["hidden"], case["inter"], case["experts"], case["top_k"]
        used = E * (1.0 - (1.0 - K / E) ** T)        # experts that some token selects
        weight = 3 * H * I * (1 if case["fp8_experts"] else 2)
        return {"bytes": used * weight + T * H * 4 + T * K * 8, "flops": 6.0 * T * K * H * I}
    if kind == "tp":
        m, d, ff = case["m"], case["d_model"], case["d_ff"]
        return {"bytes": 3 * d * ff * (1 if case["fp8"] else 2) + 4 * m * d, "flops": 6.0 * m * d * ff}
    if kind == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": (m + n) * k * (1 if case["fp8"] else 2) + 2 * m * n, "flops": 2.0 * m * n * k}
    n, size = case["pes"], case["elems"] * torch.empty((), dtype=getattr(torch, case["dtype"])).element_size()
    reads, writes = {"allreduce": (n, n), "alltoall": (n, n), "fcollect": (n, n * n), "broadcast": (1, n - 1)}[case["op"]]
    return {"bytes": (reads + writes) * size, "flops": float((n - 1) * case["elems"]) if case["op"] == "allreduce" else 0.0}


def tolerance(case):
    """What another correct implementation at the same precision would differ by: about four times what was measured
    against the same computation in 64 bits, or, where that is more, between two passes on the same inputs."""
    kind = case["kind"]
    if kind == "coll" and (case["op"] != "allreduce" or case["dtype"] == "int32"):
        return "exact"
    if kind == "coll" and case["dtype"] == "float32":
        return {"rel": 1e-6, "max": 1e-5}       # sums of four values in another order
    if kind == "moe":
        # A token's experts are added up in bf16, in an order that is not fixed: 0.0045, largest 0.034.
        return {"rel": 1.8e-2, "max": 0.14}
    if kind == "tp" and case["fp8"]:
        # The hidden activation quantised from its bf16 or from its fp32 values: 0.0113, largest 0.074.
        return {"rel": 3e-2, "max": 0.29}
    return {"rel": 7e-3, "max": 2.4e-2}         # one rounding to bf16: 0.0017, largest 0.0059


# ---- the same in 64 bits, in plain torch ------------------------------------------------------------------------

def _wide(q, scale=None):
    """A matrix in 64 bits; `scale` holds one factor for each block of it."""
    v = q.double() if scale is None else q.float().double()
    if scale is not None:
        f = scale.double()
        f = f.repeat_interleave(v.shape[-1] // f.shape[-1], -1)
        v = v * f.repeat_interleave(v.shape[-2] // f.shape[-2], -2)
    return v


def _swiglu_mlp(x, w13, w2):
    gate, up = (x @ w13.t()).chunk(2, dim=-1)
    return (torch.nn.functional.silu(gate) * up) @ w2.t()


def exact(case, seed):
    """What `run` returns for these inputs, in 64 bits; None for what is no computed number. The quantisation of
    activations inside a layer is left out: its error is the layer's own."""
    kind = case["kind"]
    if kind == "coll" and case["op"] != "allreduce":
        return None
    s = prepare(case, seed)
    if kind == "ep":
        # One row for each token that selects an expert, in the order of the tokens.
        used = (s.idx >= 0).any(dim=1)
        row = (used.long().cumsum(0) - 1).clamp(min=0)
        gate = torch.where(s.idx >= 0, s.w, torch.zeros_like(s.w)).double().sum(dim=1, keepdim=True)
        out = torch.where(used[:, None], gate * s.y[row].double(), 0.0)
        got = {"rows": None, "expert": None, "gate": None, "token": None, "per_expert": None, "out": out}
        if case["quantize"]:
            got["scales"] = None
        return got
    if kind == "moe":
        layer, x, out = s.layer, s.x.double(), torch.zeros(s.x.shape, dtype=torch.float64, device=s.x.device)
        for e in range(case["experts"]):
            tok, k = (s.idx == e).nonzero(as_tuple=True)
            if case["fp8_experts"]:
                w13, w2 = _wide(layer.w13_q[e], layer.w13_s[e]), _wide(layer.w2_q[e], layer.w2_s[e])
            else:
                w13, w2 = _wide(layer.w13[e]), _wide(layer.w2[e])
            out.index_add_(0, tok, _swiglu_mlp(x[tok], w13, w2) * s.w[tok, k].double()[:, None])
        return out
    if kind == "tp":
        layer = s.layer
        if case["fp8"]:
            return _swiglu_mlp(s.x.double(), _wide(layer.w1_q, layer.w1_s), _wide(layer.w2_q, layer.w2_s))
        return _swiglu_mlp(s.x.double(), _wide(layer.w_gate_up), _wide(layer.w_down))
    if kind == "gemm":
        if case["fp8"]:
            return _wide(s.a, s.a_s) @ _wide(s.b, s.b_s).t()
        return s.a.double() @ s.b.double().t()
    total = sum(shm.local_view(s.src, pe).to(torch.float64 if s.src.dtype.is_floating_point else torch.int64)
                for pe in range(case["pes"]))
    return [total.to(s.src.dtype) if case["dtype"] == "int32" else total for _ in range(case["pes"])]
