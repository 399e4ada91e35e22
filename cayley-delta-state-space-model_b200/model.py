"""CD-SSM language model glue around the fused scan path: prefill and cached one-token decode.

This is the caller side of the hot path (the reference's cdssm/models/{model,block}.py), written
from the behaviour of the reference so that benchmark configurations 1 (prefill) and 3 (batched
recurrent decode) can run on random-initialised weights.  The passes themselves are native (csrc/host/lm.cpp):
large projections and the LM head are ordinary library products (plumbing), everything else this library's kernels.

Layer structure restated from cdssm/models/block.py:140-229, constants from
cdssm/config/model.py:38-109, initialisation from cdssm/models/init.py:13-126 and
cdssm/models/block.py:90-138.
"""
import math
from dataclasses import dataclass

import torch

from . import ops


@dataclass
class CdssmConfig:
    """The five user values of the reference config plus everything it derives from them."""
    d_model: int = 768
    n_layers: int = 12
    context_length: int = 8192
    vocab_size: int = 50257
    state_dim: int = 16

    def __post_init__(self):
        assert self.state_dim % 2 == 0
        self.d_inner = 2 * self.d_model
        self.head_dim = 64
        self.n_heads = self.d_inner // self.head_dim
        self.chunk_size = self.head_dim
        self.ssm_norm_groups = 32
        self.conv_kernel_size = 4
        self.rope_base = float(self.context_length)
        self.gating_c = math.log(self.context_length)
        self.band_fraction = 2.0 / (self.n_layers + 1)
        io_eps = 2.0 ** -7                                    # bfloat16 machine epsilon
        self.eps_norm = io_eps ** 2
        self.eps_log = io_eps ** 2
        self.adt_eps = 1.0
        self.omega_thresh = math.sqrt(io_eps)
        self.adt_delta = 16.0 * io_eps
        self.adt_smoothness = self.omega_thresh / 5.0

    @property
    def dyn_consts(self):
        return (self.gating_c, self.omega_thresh, self.adt_delta, self.adt_smoothness, self.adt_eps)


class CdssmBlockParams:
    """Weights of one block, initialised like the reference (T-Fixup scaling, spectral gate biases,
    identity Q projection, shortcut and skip switched off)."""

    def __init__(self, cfg: CdssmConfig, layer_idx: int, gen: torch.Generator, device, dtype):
        N, H, di, dm = cfg.state_dim, cfg.n_heads, cfg.d_inner, cfg.d_model
        G = N + 5
        layer_scale = 1.0 / math.sqrt(2 * cfg.n_layers)
        std_in = math.sqrt(2.0 / (dm + di)) * layer_scale
        std_dyn = math.sqrt(2.0 / (di + di)) * layer_scale / math.sqrt(cfg.n_layers)
        rn = lambda *s: torch.randn(*s, generator=gen, dtype=torch.float32)
        w_in = rn(3 * di + H * N, dm) * std_in
        w_in[3 * di:] = rn(H * N, dm) * (std_in / math.sqrt(cfg.head_dim))      # V rows: small init
        w_gate = torch.cat([rn(N * H, di) * std_dyn, rn(5 * H, di) / math.sqrt(di)])
        b_gate = torch.zeros(G * H)
        ln2 = math.log(2.0)
        b_gate[N * H:(N + 1) * H] = ln2              # sel_B
        b_gate[(N + 1) * H:(N + 2) * H] = ln2        # sel_C
        b_gate[(N + 4) * H:(N + 5) * H] = ln2        # r_gate
        # spectral init: per layer a sliding log-timescale band; alpha = 1/tau, omega log-spaced
        log_range = math.log(float(cfg.context_length))
        frac = layer_idx / max(cfg.n_layers - 1, 1)
        width = cfg.band_fraction * log_range
        start = frac * (log_range - width)
        NH = N // 2
        sub = width / max(NH, 1)
        for j in range(NH):
            j0 = start + j * sub / NH
            j1 = j0 + width
            tau = torch.exp(torch.linspace(j0, j1, H))
            b_gate[j * H:(j + 1) * H] = torch.log(torch.exp(1.0 / tau) - 1 + cfg.eps_log)
            fmin, fmax = 1.0 / math.exp(j1), min(0.5, 1.0 / math.exp(j0))
            b_gate[(NH + j) * H:(NH + j + 1) * H] = torch.exp(
                torch.linspace(math.log(max(fmin, cfg.eps_log)), math.log(fmax), H))
        to = lambda t: t.to(device=device, dtype=dtype).contiguous()
        self.norm_w = to(torch.ones(dm))
        self.w_in, self.b_in = to(w_in), to(torch.zeros(3 * di + H * N))
        self.conv_w = to(rn(di, 1, 4) / 2.0)          # std 1/sqrt(kernel)
        self.conv_b = to(torch.zeros(di))
        self.w_gate, self.b_gate = to(w_gate), to(b_gate)
        self.log_dt_scale = torch.zeros(H, device=device, dtype=torch.float32)
        self.rope_freqs = (1.0 / (cfg.rope_base ** (torch.arange(H, dtype=torch.float32) / H))).to(device)
        self.w_q = to(torch.eye(di))
        self.w_readout = to(rn(di, H * N) / math.sqrt(H * N))
        self.w_out = to(rn(dm, di) * std_in)
        self.gn_w, self.gn_b = to(torch.ones(di)), to(torch.zeros(di))
        self.D = to(torch.zeros(di))
        self.v_residual_gate = torch.zeros(H, device=device, dtype=torch.float32)
        self.shortcut_scale = 0.0
        self.merge_q_and_gate_projections()


    def merge_q_and_gate_projections(self):
        """Q_proj and gate_proj read the same conv output: keep their weights as the two row blocks of ONE matrix, so that
        one product serves both.  The separate weights stay available as views: a write into one is seen, and after an
        assignment to one each has its own product until this is called again."""
        di = self.w_q.shape[0]
        self.w_qg = torch.cat([self.w_q, self.w_gate]).contiguous()
        self.b_qg = torch.cat([torch.zeros(di, device=self.b_gate.device, dtype=self.b_gate.dtype), self.b_gate])
        self.w_q, self.w_gate, self.b_gate = self.w_qg[:di], self.w_qg[di:], self.b_qg[di:]

    def residual_mix(self, dtype):
        """sigmoid(v_residual_gate) in the activation dtype (block.py:167-171)."""
        return torch.sigmoid(self.v_residual_gate).to(dtype)[None, None, :, None]

    # Every assignment to an attribute counts: the model lays its weights out for the native path once per state.
    version = 0

    def __setattr__(self, name, value):
        self.__dict__[name] = value
        self.__dict__["version"] = self.version + 1

    def native(self):
        return (self.norm_w, self.w_in, self.b_in, self.conv_w, self.conv_b, self.w_gate, self.b_gate, self.log_dt_scale,
                self.rope_freqs, self.w_q, self.w_readout, self.w_out, self.gn_w, self.gn_b, self.D, self.v_residual_gate,
                self.w_qg, self.b_qg, float(self.shortcut_scale))

    def load_reference(self, sd, prefix, device, dtype):
        """Take this block's weights from a reference state dict (parameter names of
        cdssm/models/block.py:35-88 under `prefix`, e.g. "blocks.3.")."""
        to = lambda name: sd[prefix + name].to(device=device, dtype=dtype).contiguous()
        f32 = lambda name: sd[prefix + name].to(device=device, dtype=torch.float32).contiguous()
        self.norm_w = to("norm.weight")
        self.w_in, self.b_in = to("in_proj.weight"), to("in_proj.bias")
        self.conv_w, self.conv_b = to("conv.weight"), to("conv.bias")
        self.w_gate, self.b_gate = to("gate_proj.weight"), to("gate_proj.bias")
        self.log_dt_scale = f32("log_dt_scale")
        self.w_q, self.w_readout, self.w_out = to("Q_proj.weight"), to("readout_proj.weight"), to("out_proj.weight")
        self.gn_w, self.gn_b = to("ssm_norm.weight"), to("ssm_norm.bias")
        self.D = to("D")
        self.v_residual_gate = f32("v_residual_gate")
        self.shortcut_scale = float(sd[prefix + "shortcut_scale"].float().item())
        self.merge_q_and_gate_projections()


class CdssmLM:
    """Embedding -> n_layers blocks -> RMSNorm -> tied LM head, inference only."""

    @classmethod
    def from_reference_checkpoint(cls, ckpt, device="cuda", dtype=torch.bfloat16):
        """Build the model from a checkpoint of the reference trainer: a dict (or the path of a torch.save'd
        dict) with "config" (the dataclass fields of cdssm/config/model.py; the derived ones are recomputed)
        and "model_state_dict" (cdssm/training/trainer.py:205-214, read like cdssm/inference/predict.py:10-30,
        including the "_orig_mod." prefix a compiled model leaves on its keys)."""
        if isinstance(ckpt, (str, bytes)) or hasattr(ckpt, "__fspath__"):
            ckpt = torch.load(ckpt, map_location="cpu", weights_only=False)
        c = ckpt["config"]
        cfg = CdssmConfig(**{k: c[k] for k in ("d_model", "n_layers", "context_length", "vocab_size", "state_dim")})
        sd = {k.replace("_orig_mod.", ""): v for k, v in ckpt["model_state_dict"].items()}
        lm = cls(cfg, device=device, dtype=dtype, seed=0)
        lm.load_reference_state_dict(sd)
        return lm

    def load_reference_state_dict(self, sd):
        self.embedding = sd["embedding.weight"].to(device=self.device, dtype=self.dtype).contiguous()
        self.final_norm_w = sd["final_norm.weight"].to(device=self.device, dtype=self.dtype).contiguous()
        for i, p in enumerate(self.blocks):
            p.load_reference(sd, f"blocks.{i}.", self.device, self.dtype)

    def __init__(self, cfg: CdssmConfig, device="cuda", dtype=torch.bfloat16, seed=0):
        self.cfg, self.device, self.dtype = cfg, torch.device(device), dtype
        gen = torch.Generator().manual_seed(seed)
        self.embedding = (torch.randn(cfg.vocab_size, cfg.d_model, generator=gen) *
                          math.sqrt(1.0 / cfg.d_model)).to(device=device, dtype=dtype)
        self.blocks = [CdssmBlockParams(cfg, i, gen, device, dtype) for i in range(cfg.n_layers)]
        self.final_norm_w = torch.ones(cfg.d_model, device=device, dtype=dtype)
        self.per_token_group_norm = False   # False = the reference's sequence-wide GroupNorm statistics

    _plan = None   # of the native path: not part of a copy or a saved model

    def __getstate__(self):
        return {k: v for k, v in self.__dict__.items() if k != "_plan"}

    def _native(self):
        """The model as the native path holds it (csrc/host/lm.cpp: the blocks' layers, one call per pass).  Rebuilt when a
        weight tensor was replaced; writes into the tensors and assignments to their ``data`` are seen anyway."""
        c = self.cfg
        key = (id(self.embedding), id(self.final_norm_w), c.state_dim, c.chunk_size, c.ssm_norm_groups, c.eps_norm, *c.dyn_consts,
               *[(id(p), p.version) for p in self.blocks])
        if self._plan is None or self._plan[0] != key:
            plan = ops._lib.host().lm_plan(c.d_model, c.d_inner, c.n_heads, c.state_dim, c.chunk_size, c.ssm_norm_groups,
                                           c.eps_norm, *c.dyn_consts, self.embedding, self.final_norm_w,
                                           [p.native() for p in self.blocks])
            self._plan = (key, plan, self.embedding, self.final_norm_w, list(self.blocks))   # ids stay taken
        return self._plan[1]

    def _ids(self, ids):
        return ids if isinstance(ids, torch.Tensor) else torch.as_tensor(ids, device=self.device)

    # ------------------------------------------------------------------ public API
    @torch.no_grad()
    def forward(self, input_ids, scan_flags=0):
        """Prefill: (B,L) token ids -> (B,L,vocab) logits (cdssm/models/model.py:37-51)."""
        return ops._lib.host().lm_forward(self._native(), self._ids(input_ids), self.per_token_group_norm, scan_flags)

    @torch.no_grad()
    def prefill(self, input_ids, last_only=True):
        """Prefill that also returns the decode cache: per layer the recurrent state after the last
        token (B,H,N,D) fp32 and the last three conv inputs; plus the position counter."""
        logits, flat = ops._lib.host().lm_prefill(self._native(), self._ids(input_ids), last_only)
        layers = [{"state": flat[i], "conv": flat[i + 1]} for i in range(0, len(flat), 2)]
        return logits, {"layers": layers, "pos": input_ids.shape[1]}

    @torch.no_grad()
    def decode(self, token_ids, cache):
        """One token per sequence: (B,) ids -> (B,vocab) logits; the cache is updated in place.
        The reference instead re-runs the whole window per token (cdssm/inference/predict.py:53-67)."""
        # one position counter: the host integer, or - once a decode graph exists - the device int32 that
        # makes the step graph-replayable (see position())
        name = "pos_dev" if "pos_dev" in cache else "pos"
        flat = [c[n] for c in cache["layers"] for n in ("state", "conv")]
        logits = ops._lib.host().lm_decode(self._native(), self._ids(token_ids), flat, cache[name])
        cache[name] += 1
        return logits

    @staticmethod
    def position(cache):
        """Number of tokens the cache has seen (reads the device counter if a decode graph owns it)."""
        return int(cache["pos_dev"].item()) if "pos_dev" in cache else int(cache["pos"])

    def make_forward_graph(self, batch, length, scan_flags=0):
        """Capture forward() for a fixed (batch, length) as one CUDA graph: a prefill of a few thousand tokens is
        some 200 short launches per pass and otherwise bound by the host that issues them.  Returns
        (graph, ids, logits): write token ids into ``ids`` (batch, length), ``graph.replay()``, read ``logits``
        (batch, length, vocab).  The scan workspace belongs to the capture stream and stays alive with the graph."""
        dev = self.device
        ids = torch.zeros(batch, length, dtype=torch.int64, device=dev)
        side = torch.cuda.Stream(device=dev)
        side.wait_stream(torch.cuda.current_stream(dev))
        with torch.cuda.stream(side):               # warm-up outside capture: workspaces, lazy library handles
            for _ in range(2):
                self.forward(ids, scan_flags)
        torch.cuda.current_stream(dev).wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            logits = self.forward(ids, scan_flags)
        return graph, ids, logits

    def make_decode_graph(self, cache, batch):
        """Capture one greedy decode step as a CUDA graph: static token buffer in, next tokens out,
        position in device memory.  Returns (graph, token_buffer); replay advances the cache."""
        dev = self.device
        cache["pos_dev"] = torch.tensor([cache.pop("pos")], dtype=torch.int32, device=dev)
        tok = torch.zeros(batch, dtype=torch.int64, device=dev)
        side = torch.cuda.Stream(device=dev)
        side.wait_stream(torch.cuda.current_stream(dev))
        snapshot = [{k: v.clone() for k, v in c.items()} for c in cache["layers"]]
        with torch.cuda.stream(side):               # warm-up outside capture, then restore the cache
            for _ in range(2):
                tok.copy_(self.decode(tok, cache).argmax(-1))
        torch.cuda.current_stream(dev).wait_stream(side)
        for c, s0 in zip(cache["layers"], snapshot):
            for k in c:
                c[k].copy_(s0[k])
        cache["pos_dev"] -= 2
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            tok.copy_(self.decode(tok, cache).argmax(-1))
        return graph, tok
