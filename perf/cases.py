"""The work this framework is timed on, through its public entry points.

A case is a dict of plain values; ``listed()`` names the fixed ones, ``draw(rng)`` gives more of the same ranges,
``prepare(case, seed)`` makes what a user's program holds before the call, ``run(state)`` is one pass, ``work(case)``
the bytes and operations that no implementation can do without, ``tolerance(case)`` what the data types allow.

Kinds of work:
  scan       ops.scan_fused: the scan path of one block (training-time forward, prefill of one layer)
  scan_long  ops.scan_fused_long: one long sequence cut into chunk-aligned segments
  step       ops.decode_step: one token of one layer, states updated in place
  train      the six operators as a block of the reference's trainer calls them, forward and backward
  forward    CdssmLM.forward: logits of every position of a batch
  prompt     CdssmLM.prefill: a prompt is read into a decode cache, logits of the last position
  decode     CdssmLM.decode: one token per sequence from that cache
"""
import functools
import math

import torch
import torch.nn.functional as F

from cdssm_b200 import ops
from cdssm_b200.model import CdssmConfig, CdssmLM

DTYPES = {"bf16": torch.bfloat16, "f32": torch.float32}
SIZE = {"bf16": 2, "f32": 4}
VOCAB = 32000


def listed():
    return [
        # one layer's token of a single generation stream, the default model's shape: launch latency and host time
        dict(name="step_stream", kind="step", B=1, H=24, D=64, N=16, dtype="bf16"),
        # one layer's token of a full decode batch of the 2048-wide model: bytes of the states
        dict(name="step_batch", kind="step", B=256, H=64, D=64, N=2, dtype="bf16"),
        # a token of the 12-layer LM for a handful of concurrent streams, logits handed to the caller's sampler
        dict(name="decode_lm", kind="decode", B=16, L=128, d_model=768, layers=12, N=2, dtype="bf16"),
        # a single user's prompt read into a cache (time to the first token); the length is nobody's multiple
        dict(name="prompt_lm", kind="prompt", B=1, L=523, d_model=768, layers=12, N=16, dtype="bf16"),
        # whole-batch forward of the 12-layer LM (scoring, evaluation)
        dict(name="forward_lm", kind="forward", B=8, L=2048, d_model=768, layers=12, N=2, dtype="bf16"),
        # the scan in full precision at the size used to check numerics
        dict(name="scan_f32", kind="scan", B=2, L=512, H=4, D=64, N=2, dtype="f32", carry=False, tail=False),
        # a few ragged prompts of one layer whose recurrent state is kept for decoding
        dict(name="scan_prompts", kind="scan", B=3, L=777, H=24, D=64, N=2, dtype="bf16", carry=False, tail=True),
        # one layer of the batch forward above
        dict(name="scan_lm", kind="scan", B=8, L=2048, H=24, D=64, N=2, dtype="bf16", carry=False, tail=False),
        # the same layer with the default state size of the model configuration
        dict(name="scan_lm_n16", kind="scan", B=8, L=2048, H=24, D=64, N=16, dtype="bf16", carry=False, tail=False),
        # the scan-kernel sweep at head_dim 128
        dict(name="scan_sweep", kind="scan", B=16, L=4096, H=32, D=128, N=2, dtype="bf16", carry=False, tail=False),
        # one document-length sequence
        dict(name="scan_long", kind="scan_long", B=1, L=1 << 18, H=32, D=128, N=2, dtype="bf16", segments=16),
        # a training step's share of one block: operators forward and backward
        dict(name="train_block", kind="train", B=4, L=1024, H=24, D=64, N=16, dtype="bf16"),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


# The largest scan pass: token-heads x state rows x head_dim of scan_sweep.
SCAN_MOST = 16 * 4096 * 32 * 2 * 128


def draw(rng):
    kind = rng.choice(["scan", "scan", "scan", "scan", "step", "step", "train", "scan_long", "forward", "prompt",
                       "decode", "decode"])
    dtype = "f32" if rng.random() < 0.15 else "bf16"
    N = rng.choice([2, 2, 4, 8, 16, 16])
    if kind == "scan":
        H, D = rng.choice([4, 6, 12, 24, 32, 40]), rng.choice([64, 64, 128])
        L = _log_int(rng, 40, 16384)
        most = SCAN_MOST // (L * H * N * D) // (4 if dtype == "f32" else 1)
        B = _log_int(rng, 1, max(1, min(32, most)))
        return dict(kind=kind, B=B, L=L, H=H, D=D, N=N, dtype=dtype, carry=rng.random() < 0.3,
                    tail=rng.random() < 0.3)
    if kind == "scan_long":
        D, S = rng.choice([64, 128]), rng.choice([4, 8, 16])
        return dict(kind=kind, B=1, L=S * D * _log_int(rng, 8, (1 << 17) // (S * D)), H=rng.choice([8, 16, 24, 32]),
                    D=D, N=2, dtype="bf16", segments=S)
    if kind == "step":
        return dict(kind=kind, B=_log_int(rng, 1, 256), H=rng.choice([6, 12, 24, 32, 64]), D=64, N=N, dtype=dtype)
    if kind == "train":
        H, L = rng.choice([4, 8, 12, 24]), _log_int(rng, 100, 2048)
        return dict(kind=kind, B=_log_int(rng, 1, max(1, 4 * 1024 * 24 * 16 // (L * H * N))), L=L, H=H, D=64, N=N,
                    dtype="bf16")
    d, layers = rng.choice([256, 512, 768]), rng.choice([4, 8, 12])
    if kind == "forward":
        L = _log_int(rng, 64, 4096)
        return dict(kind=kind, B=_log_int(rng, 1, max(1, min(32, 8 * 2048 // L))), L=L, d_model=d, layers=layers,
                    N=rng.choice([2, 2, 4]), dtype="bf16")
    if kind == "prompt":
        return dict(kind=kind, B=_log_int(rng, 1, 4), L=_log_int(rng, 16, 2000), d_model=d, layers=layers, N=N,
                    dtype="bf16")
    return dict(kind=kind, B=_log_int(rng, 1, 128), L=rng.randint(16, 300), d_model=d, layers=layers, N=N, dtype="bf16")


def _constants(length):
    """The five scalars a model of that context length hands to the dynamics (CdssmConfig.dyn_consts)."""
    eps = 2.0 ** -7
    thr = math.sqrt(eps)
    return (math.log(length), thr, 16.0 * eps, thr / 5.0, 1.0)


class _Inputs:
    """Tensors of one layer's scan: unit-variance projections, gates around the biases a model is initialised with."""

    def __init__(self, case, seed, length):
        self.g = torch.Generator(device="cuda").manual_seed(seed)
        self.dtype = DTYPES[case["dtype"]]
        self.H, self.D, self.N = case["H"], case["D"], case["N"]
        self.log_dt_scale = 0.5 * self.randn(self.H)
        self.rope_freqs = 1.0 / (float(length) ** (torch.arange(self.H, dtype=torch.float32, device="cuda") / self.H))
        self.consts = _constants(length)

    def randn(self, *shape):
        return torch.randn(*shape, generator=self.g, device="cuda", dtype=torch.float32)

    def tensor(self, *shape):
        return self.randn(*shape).to(self.dtype)

    def gates(self, *lead):
        """(..., (N+5) H): alpha_raw ~ N(-1, 0.5) and omega ~ U(-pi, pi) per head and pair, the rest N(0, 1)."""
        H, NH = self.H, self.N // 2
        g = self.randn(*lead, (self.N + 5) * H)
        bias = torch.zeros((self.N + 5) * H, device="cuda")
        bias[:NH * H] = -1.0 + 0.5 * self.randn(NH * H)
        bias[NH * H:2 * NH * H] = (torch.rand(NH * H, generator=self.g, device="cuda") * 2 - 1) * math.pi
        g[..., :2 * NH * H] *= 0.1
        return (g + bias).to(self.dtype)


@functools.lru_cache(maxsize=8)
def _model(d_model, layers, N, dtype):
    """A model as a serving or scoring process keeps it, with the terms that training switches on present."""
    cfg = CdssmConfig(d_model=d_model, n_layers=layers, context_length=4096, vocab_size=VOCAB, state_dim=N)
    lm = CdssmLM(cfg, device="cuda", dtype=DTYPES[dtype], seed=7)
    for i, p in enumerate(lm.blocks):
        p.shortcut_scale = 0.2
        p.D = torch.full_like(p.D, 0.1)
        p.v_residual_gate += 0.2 * i - 1.0
    return lm


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case)
    if kind in ("forward", "prompt", "decode"):
        s["lm"] = _model(case["d_model"], case["layers"], case["N"], case["dtype"])
        g = torch.Generator(device="cuda").manual_seed(seed)
        s["ids"] = torch.randint(0, VOCAB, (case["B"], case["L"]), generator=g, device="cuda")
        if kind == "decode":      # a cache that has read a prompt, and the next token of every sequence
            s["tokens"] = torch.randint(0, VOCAB, (case["B"],), generator=g, device="cuda")
            _, s["cache"] = s["lm"].prefill(s["ids"])
        return s
    B, H, D, N = case["B"], case["H"], case["D"], case["N"]
    if kind == "step":
        inp = _Inputs(case, seed, 4096)
        s.update(inp=inp, state=0.1 * inp.randn(B, H, N, D), q=inp.tensor(B, H, D), k=inp.tensor(B, H, D),
                 v=inp.tensor(B, H, N), gates=inp.gates(B), pos=1000)
        return s
    L = case["L"]
    inp = _Inputs(case, seed, max(L, 2048))
    s.update(inp=inp, q=inp.tensor(B, L, H, D), k=inp.tensor(B, L, H, D), v=inp.tensor(B, L, H, N),
             gates=inp.gates(B, L))
    if kind == "scan":
        s["h0"] = 0.1 * inp.randn(B, H, N, D) if case["carry"] else None
        s["pos0"] = 4 * D if case["carry"] else 0
    if kind == "train":
        s["x"] = inp.tensor(B, L, H * D)                                          # input of the short convolution
        s["conv_w"], s["conv_b"] = (0.5 * inp.randn(H * D, 1, 4)).to(inp.dtype), torch.zeros(H * D, device="cuda",
                                                                                           dtype=inp.dtype)
        s["grad_y"], s["grad_conv"] = inp.tensor(B, L, H, N), inp.tensor(B, L, H * D)
    return s


def run(s):
    kind = s["kind"]
    if kind == "forward":
        return s["lm"].forward(s["ids"])
    if kind == "prompt":
        logits, cache = s["lm"].prefill(s["ids"])
        return [logits] + [c[n] for c in cache["layers"] for n in ("state", "conv")]
    if kind == "decode":
        logits = s["lm"].decode(s["tokens"], s["cache"])
        return [logits] + [c[n] for c in s["cache"]["layers"] for n in ("state", "conv")]
    inp = s["inp"]
    if kind == "step":
        y = ops.decode_step(s["state"], s["q"], s["k"], s["v"], s["gates"], inp.log_dt_scale, inp.rope_freqs,
                            *inp.consts, inp.H, inp.N, s["pos"])
        return y, s["state"]
    if kind == "scan":
        return ops.scan_fused(s["q"], s["k"], s["v"], s["gates"], inp.log_dt_scale, inp.rope_freqs, *inp.consts,
                              inp.H, inp.N, inp.D, s["h0"], pos0=s["pos0"], return_tail_state=s["tail"])
    if kind == "scan_long":
        return ops.scan_fused_long(s["q"], s["k"], s["v"], s["gates"], inp.log_dt_scale, inp.rope_freqs, *inp.consts,
                                   inp.H, inp.N, inp.D, segments=s["segments"])
    return _train(s, inp)


def _train(s, inp):
    """Convolution, dynamics, normalisation and chunked scan the way the reference's block and scan driver call them,
    then the backward pass from the gradients of the read-out and of the convolution."""
    B, L, H, D, N = s["B"], s["L"], inp.H, inp.D, inp.N
    leaves = [s[n].detach().requires_grad_() for n in ("x", "conv_w", "conv_b", "q", "k", "v", "gates")]
    lds = inp.log_dt_scale.detach().requires_grad_()
    x, cw, cb, q, k, v, gates = leaves
    conv = ops.CUDAConv1dSiLUOp.apply(x, cw, cb)
    A, vp, beta, sel_C = ops.DynamicsFusedFn.apply(gates, lds, inp.rope_freqs, *inp.consts, H, N)
    kn, qn = ops.NormalizeKQFn.apply(k, q)
    vg = v * vp.repeat_interleave(2, dim=-1)
    NC = -(-L // D)
    pad = NC * D - L
    if pad:
        A, kp, vg = (F.pad(t, (0, 0, 0, 0, 0, pad)) for t in (A, kn, vg))
        beta = F.pad(beta, (0, 0, 0, pad))
    else:
        kp = kn
    local_h, cum_A = ops.IntraChunkScanFn.apply(A.reshape(B * NC, D, H, N), kp.reshape(B * NC, D, H, D),
                                                vg.reshape(B * NC, D, H, N), beta.reshape(B * NC, D, H), N)
    local_h, cum_A = local_h.view(B, NC, D, H, N, D), cum_A.view(B, NC, D, H, N)
    carry = ops.InterChunkScanFn.apply(cum_A[:, :, -1], local_h[:, :, -1], N)
    corr = ops.ExactCorrectionFn.apply(A.reshape(B, NC, D, H, N), kp.reshape(B, NC, D, H, D),
                                       beta.reshape(B, NC, D, H), carry, N)
    Y = (local_h + corr).reshape(B, NC * D, H, N, D)[:, :L]
    y = torch.einsum("blhsd,blhd->blhs", Y, qn) * sel_C.unsqueeze(-1)
    grads = torch.autograd.grad([y, conv], leaves + [lds], [s["grad_y"], s["grad_conv"]])
    return [y.detach(), conv.detach()] + list(grads)


def _scan_work(c, tokens):
    """q, k, v, the N + 5 gate values in and y out per token-head; per state row the products with k (twice: erase and
    update, local and correction walk) and q, two operations a column each."""
    th = tokens * c["H"]
    return th * (2 * c["D"] + c["N"] + c["N"] + 5 + c["N"]) * SIZE[c["dtype"]], th * c["N"] * c["D"] * 12


def work(case):
    c = dict(case)
    kind, B, N = c["kind"], c["B"], c["N"]
    if kind in ("scan", "scan_long"):
        nbytes, flops = _scan_work(c, B * c["L"])
        states = 1 + (1 if c.get("carry") else 0) + (1 if c.get("tail") else 0)      # final state, h0, tail state
        return {"bytes": nbytes + states * B * c["H"] * N * c["D"] * 4, "flops": flops}
    if kind == "step":
        nbytes, flops = _scan_work(c, B)
        return {"bytes": nbytes + 2 * B * c["H"] * N * c["D"] * 4, "flops": flops}
    if kind == "train":      # every operator's inputs and outputs once, forward and backward; five (.., N, D) tensors
        th = B * c["L"] * c["H"]
        small = 4 * c["D"] * 3 + 2 * c["D"] * 3 + (N + 5) * 3 + 6 * (2 * N + 2)
        big = N * c["D"] * (2 + 3 + 2 + 4)   # forward: two written; add: read, read, write; read-out and its gradient; backward
        return {"bytes": th * (small + big) * SIZE[c["dtype"]], "flops": th * N * c["D"] * 60}
    d, di, layers = c["d_model"], 2 * c["d_model"], c["layers"]
    H = di // 64
    es = SIZE[c["dtype"]]
    per_layer = d * (3 * di + H * N) + di * (di + (N + 5) * H) + H * N * di + di * d
    weights = layers * per_layer + VOCAB * d
    scan = dict(c, H=H, D=64)
    if kind == "decode":
        state = layers * B * (H * N * 64 * 8 + 6 * di * es)                          # read and written
        return {"bytes": weights * es + state + B * VOCAB * es,
                "flops": 2 * B * weights + layers * _scan_work(scan, B)[1]}
    tokens = B * c["L"]
    heads = tokens if kind == "forward" else B                                       # positions whose logits are made
    keep = layers * B * (H * N * 64 * 4 + 3 * di * es) if kind == "prompt" else 0
    flops = 2 * tokens * layers * per_layer + 2 * heads * VOCAB * d + layers * _scan_work(scan, tokens)[1]
    return {"bytes": weights * es + tokens * (8 + d * es) + heads * VOCAB * es + keep, "flops": flops}


def tolerance(case):
    if case["dtype"] == "f32":
        return {"rel": 2e-5, "max": 2e-3}      # 32-bit sums over a chain of up to thousands of steps
    if case["kind"] in ("forward", "prompt", "decode"):
        return {"rel": 2e-2, "max": 0.8}       # bf16 roundings of every layer's activations add up along the residual
    return {"rel": 1e-2, "max": 0.4}           # bf16 storage, 32-bit states
