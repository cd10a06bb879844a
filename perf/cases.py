"""The work a user of asca_b200 has it do, as cases that can be timed one by one.

A case is a plain dict; ``prepare`` makes what a program holds before the call (weights, a model, device tensors or host
arrays), ``run`` is one pass through the public entry points, ``work`` and ``tolerance`` say what the pass cannot do
without and how closely two correct implementations agree. Kinds of work:

* ``train``    one optimizer step: ``Model.zero_grads`` + ``forward_backward`` + ``adamw_step``
* ``decode``   ``Model.decode_greedy`` (several tokens a call) or ``Model.decode_step`` with logits (a sampler's loop)
* ``prefill``  ``Model.prefill`` of a batch of prompts
* ``delta``    ``ops.delta_fwd`` + ``ops.delta_bwd`` on device tensors, or (``host``) ``Gpu.delta_scan`` + ``delta_bwd_dev``
* ``moe``      ``ops.moe_dispatch`` + ``moe_fwd`` + ``moe_bwd`` on device tensors
"""
import math

import numpy as np
import torch

import asca_b200
from asca_b200 import ops

#: vocab, d, heads, blocks, experts, expert width
MODELS = {
    "331k": (256, 64, 4, 2, 4, 256),         # the reference's CPU-runnable model
    "12.7m": (256, 192, 6, 6, 8, 640),       # the model of its GPU measurements
    "125m": (256, 768, 12, 12, 16, 3072),    # the decode configuration
    "1.3b-block": (256, 2048, 16, 1, 64, 4096),   # one block of the training configuration
}
LR = 3e-4


def listed():
    return [
        # the smallest training run: an optimizer step on 16 sequences of 128 bytes, a wait for the loss in every step
        {"name": "train_331k_f32", "kind": "train", "model": "331k", "dtype": "f32", "B": 16, "T": 128},
        # the reference's own GPU training run: 8 sequences of 256 bytes, six blocks of head dim 32
        {"name": "train_12.7m_f32", "kind": "train", "model": "12.7m", "dtype": "f32", "B": 8, "T": 256},
        # a block of the 1.3B-class model: 8 sequences of 4096 bytes in bf16, the largest work here
        {"name": "train_1.3b_block_bf16", "kind": "train", "model": "1.3b-block", "dtype": "bf16", "B": 8, "T": 4096},
        # one user generating text with the small model: pure latency
        {"name": "decode_331k_f32", "kind": "decode", "model": "331k", "dtype": "f32", "streams": 1, "steps": 128, "logits": False},
        # a serving batch at the decode configuration
        {"name": "decode_125m_bf16", "kind": "decode", "model": "125m", "dtype": "bf16", "streams": 256, "steps": 64, "logits": False},
        # a handful of streams whose tokens are sampled on the host: the logits come back after each step
        {"name": "decode_125m_sampled_bf16", "kind": "decode", "model": "125m", "dtype": "bf16", "streams": 12, "steps": 1, "logits": True},
        # new requests joining: prompts of a length that is no multiple of anything
        {"name": "prefill_125m_bf16", "kind": "prefill", "model": "125m", "dtype": "bf16", "streams": 48, "T": 301},
        # the isolated recurrence at the benchmark's size, forward and backward, both data types
        {"name": "delta_bf16", "kind": "delta", "dtype": "bf16", "B": 8, "T": 4096, "H": 16, "dh": 128, "host": False},
        {"name": "delta_f32", "kind": "delta", "dtype": "f32", "B": 8, "T": 4096, "H": 16, "dh": 128, "host": False},
        # the drop-in form: host arrays in, host arrays out, as the reference's trainer calls its GPU backend
        {"name": "delta_host_f32", "kind": "delta", "dtype": "f32", "B": 3, "T": 777, "H": 6, "dh": 32, "host": True},
        # the isolated expert layer: a skewed load of 65,536 tokens in bf16, and the small f32 layer at a ragged size
        {"name": "moe_bf16", "kind": "moe", "dtype": "bf16", "N": 65536, "d": 1024, "F": 4096, "E": 64},
        {"name": "moe_f32", "kind": "moe", "dtype": "f32", "N": 1500, "d": 192, "F": 384, "E": 8},
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, spread over its logarithm."""
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def _sequences(rng, lo, hi, t_lo, t_hi, b_hi=64):
    """(B, T) with lo <= about B * T <= hi."""
    n = _log(rng, lo, hi)
    t = _log(rng, t_lo, min(t_hi, n))
    return max(1, min(b_hi, n // t)), t


def draw(rng):
    kind = rng.choice(["train_f32", "train_bf16", "decode_f32", "decode_bf16", "prefill", "delta_bf16", "delta_f32", "delta_host",
                       "moe_bf16", "moe_f32"])
    if kind == "train_f32":
        model = rng.choice(["331k", "12.7m"])
        b, t = _sequences(rng, 256, 8192 if model == "331k" else 4096, 16, 512)
        return {"kind": "train", "model": model, "dtype": "f32", "B": b, "T": t}
    if kind == "train_bf16":
        model = rng.choice(["125m", "1.3b-block"])
        b, t = _sequences(rng, 1024, 8192 if model == "125m" else 32768, 128, 4096, 16)
        return {"kind": "train", "model": model, "dtype": "bf16", "B": b, "T": t}
    if kind == "decode_f32":
        model = rng.choice(["331k", "12.7m"])
        return {"kind": "decode", "model": model, "dtype": "f32", "streams": _log(rng, 1, 64),
                "steps": _log(rng, 16, 128 if model == "331k" else 48), "logits": False}
    if kind == "decode_bf16":
        logits = rng.random() < 0.4
        return {"kind": "decode", "model": "125m", "dtype": "bf16", "streams": _log(rng, 1, 256), "steps": 1 if logits else _log(rng, 8, 64),
                "logits": logits}
    if kind == "prefill":
        b, t = _sequences(rng, 256, 24576, 32, 1024)
        return {"kind": "prefill", "model": "125m", "dtype": "bf16", "streams": b, "T": t}
    if kind in ("delta_bf16", "delta_f32"):
        dh = rng.choice([64, 128] if kind == "delta_bf16" else [32, 64, 128])
        h = rng.randint(4, 16)
        b, t = _sequences(rng, 2048 // h, 65536 // h, 64, 4096)
        return {"kind": "delta", "dtype": kind[6:], "B": b, "T": t, "H": h, "dh": dh, "host": False}
    if kind == "delta_host":
        b, t = _sequences(rng, 256, 8192, 64, 1024, 16)
        return {"kind": "delta", "dtype": "f32", "B": b, "T": t, "H": rng.randint(2, 8), "dh": rng.choice([16, 32, 64]), "host": True}
    if kind == "moe_bf16":
        return {"kind": "moe", "dtype": "bf16", "N": _log(rng, 1024, 65536), "d": rng.choice([512, 768, 1024]),
                "F": rng.choice([2048, 3072, 4096]), "E": rng.choice([8, 16, 32, 64])}
    d = rng.choice([64, 128, 192, 256])
    return {"kind": "moe", "dtype": "f32", "N": _log(rng, 256, 4096), "d": d, "F": d * rng.choice([2, 3, 4]), "E": rng.choice([4, 8, 16])}


# ------------------------------------------------------------------ inputs
_gpu_handle = None


def _gpu():
    """The process's one context, on torch's stream."""
    global _gpu_handle
    if _gpu_handle is None:
        _gpu_handle = asca_b200.Gpu(0)
    _gpu_handle.use_torch_stream()
    return _gpu_handle


class _Flat:
    """A flat f32 buffer of a model as a CUDA array (keeps the model that owns it alive)."""

    def __init__(self, owner, ptr, n):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f4", "data": (ptr, False), "version": 2}


class _Model:
    """A model and torch views of its parameters, gradients and moments; freed with the last of them."""

    def __init__(self, cfg, dtype):
        self.model = asca_b200.Model(_gpu(), *cfg)
        if dtype == "bf16":
            self.model.set_compute(asca_b200.BF16)

    def views(self):
        return [torch.as_tensor(_Flat(self, p, self.model.n), device="cuda") for p in self.model.buffers()]

    def __del__(self):
        self.model.free()


def _dtype(case):
    return torch.bfloat16 if case["dtype"] == "bf16" else torch.float32


def _zipf_ids(rng, n, s=1.1):
    p = 1.0 / np.arange(1, 257) ** s
    return rng.choice(256, size=n, p=p / p.sum()).astype(np.uint32)


def _delta_inputs(case, seed):
    """q and k L2-normalised, the norms beside them; slow decay (alpha near 0.88), beta around a half."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    n, H, dh = case["B"] * case["T"], case["H"], case["dh"]
    norm = lambda *shape: torch.randn(*shape, generator=g, device="cuda")  # noqa: E731
    q, k = norm(n, H, dh), norm(n, H, dh)
    qn, kn = q.norm(dim=-1), k.norm(dim=-1)
    q, k = ((x / xn[..., None]).reshape(n, H * dh).to(_dtype(case)) for x, xn in ((q, qn), (k, kn)))
    v, d_o = (norm(n, H * dh).to(_dtype(case)) for _ in range(2))
    alpha, beta = torch.sigmoid(2 + 0.5 * norm(n, H)), torch.sigmoid(norm(n, H))
    return dict(q=q, k=k, v=v, alpha=alpha, beta=beta, qn=qn, kn=kn, d_o=d_o)


def _generator_params(p, cfg, g):
    """Weights whose next byte is clear, as a trained model's is: the head answers each byte's embedding with one other
    byte, so that rounding does not send a greedy decode down another path."""
    V, d = cfg[:2]
    p.normal_(0, 0.02, generator=g)
    embed = torch.randn(V, d, generator=g, device="cuda")
    p[: V * d] = embed.reshape(-1)
    p[V * d: 2 * V * d] = embed[torch.randperm(V, generator=g, device="cuda")].t().reshape(-1)


def prepare(case, seed):
    gpu = _gpu()
    s = {"case": case, "gpu": gpu}
    rng = np.random.default_rng(seed)
    if case["kind"] in ("train", "decode", "prefill"):
        cfg = MODELS[case["model"]]
        holder = _Model(cfg, case["dtype"])
        params, grads, m, v = holder.views()
        g = torch.Generator(device="cuda").manual_seed(seed)
        if case["kind"] == "train":
            params.normal_(0, 0.02, generator=g)
            n = case["B"] * case["T"]
            text = rng.integers(0, 256, n + 1, dtype=np.uint32)
            s.update(ids=text[:-1].copy(), targets=text[1:].copy(), updated={"params": params, "grads": grads, "m": m, "v": v})
        else:
            _generator_params(params, cfg, g)
            ns = case["streams"]
            s["state"] = holder.model.new_decode_state(ns)
            if case["kind"] == "decode":
                dh = cfg[1] // cfg[2]   # the state a prompt has left behind
                s["state"].normal_(0, dh ** -0.5, generator=g)
                s["ids"] = rng.integers(0, 256, ns, dtype=np.uint32)
            else:
                s["ids"] = rng.integers(0, 256, (ns, case["T"]), dtype=np.uint32)
        holder.model.params_changed()
        s["model"], s["holder"] = holder.model, holder
    elif case["kind"] == "delta":
        t = _delta_inputs(case, seed)
        s.update({key: x.cpu().numpy() for key, x in t.items()} if case["host"] else t)
    else:
        g = torch.Generator(device="cuda").manual_seed(seed)
        n, d, F, E = (case[key] for key in ("N", "d", "F", "E"))
        dt = _dtype(case)

        def norm(*shape, scale=1.0):
            x = torch.empty(*shape, dtype=dt, device="cuda")
            return x.normal_(0, scale, generator=g)

        s.update(ids=torch.from_numpy(_zipf_ids(rng, n).view(np.int32)).cuda(), xn=norm(n, d), w1=norm(d, E * F, scale=0.02),
                 w2=norm(E * F, d, scale=0.02), b1=norm(E * F, scale=0.02).float(), b2=norm(d, scale=0.02).float(), dout=norm(n, d).float())
    return s


# ------------------------------------------------------------------ one pass
def run(s):
    case, gpu = s["case"], s["gpu"]
    if case["kind"] == "train":
        model = s["model"]
        model.zero_grads()
        loss = model.forward_backward(s["ids"], s["targets"], case["B"])
        model.adamw_step(LR)
        return {"loss": loss, **s["updated"]}
    if case["kind"] == "decode":
        model = s["model"]
        if case["logits"]:
            logits, nxt = model.decode_step(s["state"], s["ids"])
            return {"logits": logits, "next": nxt, "state": s["state"]}
        return {"tokens": model.decode_greedy(s["state"], s["ids"], case["steps"]), "state": s["state"]}
    if case["kind"] == "prefill":
        logits, nxt = s["model"].prefill(s["state"], s["ids"])
        return {"logits": logits, "next": nxt, "state": s["state"]}
    if case["kind"] == "delta":
        B, T, H, dh = (case[key] for key in ("B", "T", "H", "dh"))
        q, k, v, al, be, qn, kn, d_o = (s[key] for key in ("q", "k", "v", "alpha", "beta", "qn", "kn", "d_o"))
        if case["host"]:
            o, dev = gpu.delta_scan(q, k, v, al, be, B, T, H, dh)
            d_qkv, d_gate = gpu.delta_bwd_dev(dev, d_o, qn, kn)
            dev.free()
        else:
            o, _, ckpt = ops.delta_fwd(gpu, q, k, v, al, be, B, T, H, dh)
            d_qkv, d_gate = ops.delta_bwd(gpu, q, k, v, al, be, qn, kn, d_o, ckpt, B, T, H, dh)
        return {"o": o, "d_qkv": d_qkv, "d_gate": d_gate}
    F, E = case["F"], case["E"]
    perm, offsets = ops.moe_dispatch(gpu, s["ids"], E)
    out, pre, hid = ops.moe_fwd(gpu, s["xn"], s["w1"], s["b1"], s["w2"], s["b2"], perm, offsets, F, E)
    grads = ops.moe_bwd(gpu, s["xn"], s["w1"], s["w2"], pre, hid, s["dout"], perm, offsets, F, E)
    return {"perm": perm, "offsets": offsets, "out": out, "grads": grads}


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    size = 2 if case["dtype"] == "bf16" else 4
    if case["kind"] in ("train", "decode", "prefill"):
        V, d, H, L, E, F = MODELS[case["model"]]
        dh = d // H
        dense = d * 3 * d + d * 2 * H + d * d
        per_token = L * (dense + 2 * d * F)   # weights a token meets, without the head
        if case["kind"] == "train":
            n = case["B"] * case["T"]
            total = 2 * V * d + L * (dense + 3 * d + 2 * H + d + 2 * d * E * F + E * F + d)
            # master weights and both moments read and written, the gradient written; the ids are nothing beside them
            return {"bytes": 28 * total, "flops": n * (6 * (per_token + d * V) + 22 * dh * dh * H * L)}
        ns = case["streams"]
        state = 2 * 4 * L * ns * H * dh * dh
        tokens = ns * (case["steps"] if case["kind"] == "decode" else case["T"])
        hit = E * (1 - (1 - 1 / E) ** (ns if case["kind"] == "decode" else tokens))   # experts that get a token
        weights = size * (L * (dense + 2 * hit * d * F) + V * d)
        flops = tokens * (2 * per_token + 6 * dh * dh * H * L)
        if case["kind"] == "prefill":
            return {"bytes": weights + state, "flops": flops + ns * 2 * d * V}
        # weights and state that no cache holds are met again in every step
        times = case["steps"] if weights + state > 1e8 else 1
        return {"bytes": times * (weights + state), "flops": flops + tokens * 2 * d * V}
    if case["kind"] == "delta":
        n, H, dh = case["B"] * case["T"], case["H"], case["dh"]
        # q, k, v, d_o in and o out; d_qkv in f32 and the six gate-sized arrays
        return {"bytes": n * H * (dh * (5 * size + 12) + 6 * 4), "flops": 22 * dh * dh * H * n}
    n, d, F, E = (case[key] for key in ("N", "d", "F", "E"))
    weights = 2 * d * E * F
    return {"bytes": n * d * (size + 12) + weights * (size + 4) + 8 * (E * F + d) + 8 * n, "flops": 12 * n * d * F}


def tolerance(case):
    if case["dtype"] == "bf16":
        # products of bf16 operands with rounded intermediates; the largest difference is set against the whole flat
        # buffer's root mean square, which tensors with large entries exceed many times over
        return {"rel": 2e-2 if case["kind"] in ("train", "decode", "prefill") else 1e-2, "max": 0.9}
    # 32-bit sums in another order; where a gradient is all rounding, the first optimizer steps may differ by their length
    return {"rel": 3e-5, "max": 0.05} if case["kind"] == "train" else {"rel": 1e-5, "max": 1e-3}
