"""Operator API of the CD-SSM scan path on B200.

Level 1 mirrors the reference's cdssm/ops.py: the same six ``torch.autograd.Function``
classes, positional signatures, tensor layouts and dtypes (cdssm/ops.py:13-195), so
cdssm/models/{block,ssd,modules}.py can import this module in its place, for inference and training.

Level 2 is the fused path: :func:`scan_fused` (dynamics + normalisation + vp scale + chunked
scan + read-out in one call) and :func:`decode_step`.

Every function launches hand-written sm_100a kernels of libcdssm_b200.so on the current CUDA stream, from the
native host path (csrc/host) or through the C ABI.  There is no CPU, eager-PyTorch or Triton
fallback: tensors must be CUDA tensors and the library must be built.
"""
import torch
from torch import Tensor
from torch.autograd import Function

from . import _lib
from ._lib import CdssmError, check

__all__ = ["CUDAConv1dSiLUOp", "DynamicsFusedFn", "NormalizeKQFn", "IntraChunkScanFn",
           "InterChunkScanFn", "ExactCorrectionFn", "scan_fused", "decode_step", "decode_step_reference", "reference_decode_state",
           "scan_fused_workspace_bytes", "scan_fused_status", "set_wait_limit_ns", "selftest_bounded_wait", "rms_norm", "groupnorm_gate", "conv1d_silu_step", "scan_summary", "scan_fused_long", "compose_carries",
           "CdssmError"]

_DT = {torch.bfloat16: _lib.BF16, torch.float32: _lib.F32}


def _dtype_code(t: Tensor) -> int:
    if t.dtype not in _DT:
        raise CdssmError(f"unsupported dtype {t.dtype}: use bfloat16 (the reference's type) or float32")
    return _DT[t.dtype]


def _prep(t: Tensor, dtype=None, name="tensor") -> Tensor:
    """The reference launchers call .contiguous() and never check dtypes (e.g.
    intra_chunk_scan.cu:573-603); here a wrong device or dtype is an error, not garbage."""
    if not t.is_cuda:
        raise CdssmError(f"{name} must be a CUDA tensor (no CPU fallback exists)")
    if dtype is not None and t.dtype != dtype:
        raise CdssmError(f"{name} has dtype {t.dtype}, expected {dtype}")
    return t.contiguous()


def _f32(t: Tensor, name) -> Tensor:
    """Per-head fp32 vectors; a bf16 buffer (a model cast with .bfloat16()) is converted."""
    if not t.is_cuda:
        raise CdssmError(f"{name} must be a CUDA tensor")
    return t.detach().to(torch.float32).contiguous()


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _p(t):
    return None if t is None else t.data_ptr()


class CUDAConv1dSiLUOp(Function):
    """Causal depthwise conv (kernel 4) + bias + SiLU; cdssm/ops.py:13-28."""

    @staticmethod
    def forward(ctx, x: Tensor, weight: Tensor, bias: Tensor) -> Tensor:
        out, x, w, b = _lib.host().conv_fwd(x, weight, bias)
        ctx.save_for_backward(x, w, b)
        ctx.param_meta = (weight.shape, weight.dtype, bias.dtype)
        return out

    @staticmethod
    def backward(ctx, grad_out):
        """(grad_x, grad_weight, grad_bias), as cdssm/ops.py:22-28 (conv1d_silu.cu:94-219)."""
        gx, gw, gb = _lib.host().conv_bwd(grad_out, *ctx.saved_tensors)
        wshape, wdt, bdt = ctx.param_meta
        return gx, gw.reshape(wshape).to(wdt), gb.to(bdt)


class DynamicsFusedFn(Function):
    """gate_raw -> A_bar, vp_scale, beta, sel_C_gate; cdssm/ops.py:31-81."""

    @staticmethod
    def forward(ctx, gate_raw: Tensor, log_dt_scale: Tensor, rope_freqs: Tensor, gating_c: float,
                omega_thresh: float, adt_delta: float, adt_smoothness: float, adt_eps: float,
                n_heads: int, state_dim: int):
        ctx.args = (gating_c, omega_thresh, adt_delta, adt_smoothness, adt_eps, n_heads, state_dim)
        A, vp, beta, selc, g, lds, rf = _lib.host().dynamics_fwd(gate_raw, log_dt_scale, rope_freqs, *ctx.args)
        ctx.save_for_backward(g, lds, rf)
        ctx.lds_dtype = log_dt_scale.dtype
        return A, vp, beta, selc

    @staticmethod
    def backward(ctx, grad_A_bar, grad_vp_scale, grad_beta, grad_sel_C):
        """(grad_gate_raw, grad_log_dt_scale, None x 8), as cdssm/ops.py:68-81 (dynamics_fused.cu:145-387)."""
        gg, glds = _lib.host().dynamics_bwd(grad_A_bar, grad_vp_scale, grad_beta, grad_sel_C, *ctx.saved_tensors, *ctx.args)
        return (gg, glds.to(ctx.lds_dtype)) + (None,) * 8


class NormalizeKQFn(Function):
    """L2-normalise K and Q over the last dim; cdssm/ops.py:84-97."""

    @staticmethod
    def forward(ctx, K: Tensor, Q: Tensor):
        Ko, Qo, K, Q = _lib.host().normalize_fwd(K, Q)
        ctx.save_for_backward(K, Q)
        return Ko, Qo

    @staticmethod
    def backward(ctx, grad_K_out, grad_Q_out):
        """(grad_K, grad_Q), as cdssm/ops.py:93-97 (normalize_kq.cu:89-163)."""
        return _lib.host().normalize_bwd(grad_K_out, grad_Q_out, *ctx.saved_tensors)


class IntraChunkScanFn(Function):
    """Chunk-local delta-rule scan from a zero state; cdssm/ops.py:100-135."""

    @staticmethod
    def forward(ctx, A_flat: Tensor, K_flat: Tensor, V_flat: Tensor, beta_flat: Tensor, state_dim: int):
        local_h, cum_A, A, K, V, be = _lib.host().intra_fwd(A_flat, K_flat, V_flat, beta_flat, state_dim)
        ctx.save_for_backward(A, K, V, be, local_h, cum_A)
        ctx.state_dim = int(state_dim)
        return local_h, cum_A

    @staticmethod
    def backward(ctx, grad_local_h, grad_cum_A):
        """(grad_A, grad_K, grad_V, grad_beta, None), as cdssm/ops.py:123-135 (intra_chunk_scan.cu:215-553)."""
        return _lib.host().intra_bwd(grad_local_h, grad_cum_A, *ctx.saved_tensors, ctx.state_dim) + (None,)


class InterChunkScanFn(Function):
    """Carry recurrence across chunks; cdssm/ops.py:138-163."""

    @staticmethod
    def forward(ctx, total_A: Tensor, final_local_h: Tensor, state_dim: int) -> Tensor:
        out, a = _lib.host().inter_fwd(total_A, final_local_h, state_dim)
        ctx.save_for_backward(a, out)
        ctx.state_dim = int(state_dim)
        return out

    @staticmethod
    def backward(ctx, grad_chunk_states):
        """(grad_total_A, grad_final_local_h, None), as cdssm/ops.py:157-163 (inter_chunk_scan.cu:89-196)."""
        return _lib.host().inter_bwd(grad_chunk_states, *ctx.saved_tensors, ctx.state_dim) + (None,)


# The reference's correction backward kernel adds the upstream gradient of corrections[t] BEFORE it walks step t
# back (exact_correction.cu:219-223), although the forward stores corrections[t] before the step (:90-94), and its
# grad_beta is head_dim times too large (:347-359): its gradient is not the derivative of its forward.  The drop-in default reproduces the reference (what its training
# runs with); set this to True for the true derivative.
EXACT_CORRECTION_TRUE_GRADIENT = False


class ExactCorrectionFn(Function):
    """Propagate chunk carries through erase+rotate; cdssm/ops.py:166-195."""

    @staticmethod
    def forward(ctx, A_chunk: Tensor, K_chunk: Tensor, beta_chunk: Tensor, chunk_states: Tensor,
                state_dim: int) -> Tensor:
        out, A, K, be = _lib.host().correction_fwd(A_chunk, K_chunk, beta_chunk, chunk_states, state_dim)
        ctx.save_for_backward(A, K, be, out)
        ctx.state_dim = int(state_dim)
        return out

    @staticmethod
    def backward(ctx, grad_corrections):
        """(grad_A, grad_K, grad_beta, grad_chunk_states, None), as cdssm/ops.py:188-195
        (exact_correction.cu:169-383)."""
        return _lib.host().correction_bwd(grad_corrections, *ctx.saved_tensors, ctx.state_dim,
                                          0 if EXACT_CORRECTION_TRUE_GRADIENT else 1) + (None,)


# ------------------------------------------------------------------------------------------
# Level 2: the fused path
# ------------------------------------------------------------------------------------------
FORCE_SIMT = 1
REUSE_LOCAL = 8
EXACT = 32
TENSOR_CORE_WA = 128
KEEP_SIMT_LOCAL, KEEP_SIMT_OUTPUT = 256, 512   # tests: one tensor-core pass at a time
TEST_WITHHOLD = 2048   # self-test of the bounded waits: see include/cdssm_b200.h
FP32_DECAY = 4096      # keep the transition A_bar in float32 (NOT the reference's arithmetic): the reference's
#                        bfloat16 A_bar lets its carry grow without bound over some 1e5 tokens, see the header

def scan_fused_workspace_bytes(B, L, H, D, N, C) -> int:
    return int(_lib.lib().cdssm_b200_scan_fused_workspace_bytes(B, L, H, D, N, C))


def _workspace(on: Tensor, nbytes):
    """(address, bytes) of the grow-only scratch buffer of the tensor's device and its current stream; the library
    itself allocates nothing."""
    return _lib.host().workspace(on, nbytes)


def scan_fused(q: Tensor, k: Tensor, v: Tensor, gate_raw: Tensor, log_dt_scale: Tensor,
               rope_freqs: Tensor, gating_c: float, omega_thresh: float, adt_delta: float,
               adt_smoothness: float, adt_eps: float, n_heads: int, state_dim: int,
               chunk_size: int, h0: Tensor = None, *, shortcut_scale: float = 0.0, pos0: int = 0,
               return_tail_state: bool = False, flags: int = 0, out: Tensor = None, segs: int = 1,
               semantics: str = "reference", strict: bool = False):
    """The scan path of one CD-SSM block in a single call.

    Equals, in the reference (cdssm/models/block.py:181-211): DynamicsFusedFn -> NormalizeKQFn
    -> V * vp_scale -> SSDChunkwiseScan (cdssm/models/ssd.py:39-111) -> shortcut -> einsum
    read-out -> sel_C gate, with the reference's chunk semantics, but without ever storing a
    (B,L,H,N,D) tensor.

    q, k: (B,L,H,D) un-normalised; v: (B,L,H,N) before the vp scale; gate_raw: (B,L,(N+5)H);
    log_dt_scale, rope_freqs: (H).  h0: optional (B,H,N,D) float32 carry into the first chunk.
    segs > 1: the batch rows are ``segs`` consecutive segments of B/segs longer sequences (row b
    starts at position pos0 + (b % segs) * L); see :func:`scan_fused_long`.
    Returns (y (B,L,H,N), final_state (B,H,N,D) float32[, tail_state]); final_state is the carry
    after the last chunk (feed it as h0 of the next chunk-aligned segment together with pos0);
    tail_state is the recurrent state after the last token (what decode_step continues from).
    semantics="exact" runs the plain sequential recurrence instead of the reference's chunk semantics
    (identical inside the first chunk); h0/final_state are then the recurrent state.
    strict=True synchronises the stream after the call and raises if a bounded device-side wait of the
    tensor-core kernels ran out (the outputs are undefined then); without it the call stays asynchronous
    and :func:`scan_fused_status` reports the same word on demand.
    """
    if semantics != "reference":
        if semantics != "exact":
            raise CdssmError("semantics must be 'reference' (the reference's chunked scan, bug for bug) or "
                             "'exact' (the sequential recurrence)")
        flags = int(flags) | EXACT
    res = _lib.host().scan_fused(q, k, v, gate_raw, log_dt_scale, rope_freqs, gating_c, omega_thresh, adt_delta,
                                 adt_smoothness, adt_eps, n_heads, state_dim, chunk_size, h0, shortcut_scale, pos0,
                                 return_tail_state, flags, out, segs)
    if strict:
        code = scan_fused_status(q.device)
        if code != 0:
            raise CdssmError(f"scan_fused: a device-side wait ran out (status {code}); the outputs are undefined")
    return res


def decode_step(state: Tensor, q: Tensor, k: Tensor, v: Tensor, gate_raw: Tensor,
                log_dt_scale: Tensor, rope_freqs: Tensor, gating_c: float, omega_thresh: float,
                adt_delta: float, adt_smoothness: float, adt_eps: float, n_heads: int,
                state_dim: int, pos: int, *, shortcut_scale: float = 0.0, out: Tensor = None,
                v_first: Tensor = None, mix: Tensor = None) -> Tensor:
    """One recurrent step for every sequence of a batch; ``state`` (B,H,N,D) float32 is updated
    in place.  q, k: (B,H,D); v: (B,H,N); gate_raw: (B,(N+5)H); returns y (B,H,N).
    k and v may be column slices of a wider per-token projection (only their batch stride is free).
    ``v_first`` (B,H,N) with ``mix`` (H): the value residual v <- lerp(v_first, v, mix[head]) of
    cdssm/models/block.py:167-171 is applied inside the kernel.

    The reference has no such step (cdssm/inference/predict.py:53-67 re-runs the full forward
    for every new token); the update is one iteration of intra_chunk_scan.cu:117-167 with the
    gates of dynamics_fused.cu:64-139 at position ``pos``.
    """
    return _lib.host().decode_step(state, q, k, v, gate_raw, log_dt_scale, rope_freqs, gating_c, omega_thresh, adt_delta,
                                   adt_smoothness, adt_eps, n_heads, state_dim, pos, shortcut_scale, out, v_first, mix)


def reference_decode_state(carry: Tensor, dtype=torch.bfloat16):
    """State of :func:`decode_step_reference` at a chunk boundary from the carry (B,H,N,D) float32 that
    scan_fused returned as final_state (or zeros at the start of a sequence): a dict of the local state, the
    correction (the carry rounded to the storage type), the carry and the chunk's cumulative decay."""
    carry = _prep(carry, dtype=torch.float32, name="carry").clone()
    B, H, N, D = carry.shape
    gamma = torch.zeros(B, H, N, dtype=torch.float32, device=carry.device)
    gamma[..., 0::2] = 1.0
    return {"local": torch.zeros_like(carry), "correction": carry.to(dtype).float().clone(), "carry": carry, "decay": gamma}


def decode_step_reference(state: dict, q: Tensor, k: Tensor, v: Tensor, gate_raw: Tensor, log_dt_scale: Tensor,
                          rope_freqs: Tensor, gating_c: float, omega_thresh: float, adt_delta: float,
                          adt_smoothness: float, adt_eps: float, n_heads: int, state_dim: int, chunk_size: int,
                          pos, *, shortcut_scale: float = 0.0, out: Tensor = None) -> Tensor:
    """One token of the reference's CHUNKED scan (see cdssm_b200_decode_step_reference): unlike
    :func:`decode_step`, T of these steps reproduce scan_fused / the reference forward over T tokens for any T.
    ``state`` comes from :func:`reference_decode_state` and is updated in place; ``pos`` is the token's position
    from the start of the sequence (int, or an int32 CUDA tensor for graph replay)."""
    q = _prep(q, name="q")
    k = _prep(k, dtype=q.dtype, name="k")
    v = _prep(v, dtype=q.dtype, name="v")
    g = _prep(gate_raw, dtype=q.dtype, name="gate_raw")
    B, H, D = q.shape
    N = int(state_dim)
    for name in ("local", "correction", "carry"):
        t = state[name]
        if not t.is_cuda or t.dtype != torch.float32 or not t.is_contiguous() or tuple(t.shape) != (B, H, N, D):
            raise CdssmError(f"decode_step_reference: state['{name}'] must be a contiguous float32 (B,H,N,D) CUDA tensor")
    if tuple(state["decay"].shape) != (B, H, N) or state["decay"].dtype != torch.float32:
        raise CdssmError("decode_step_reference: state['decay'] must be float32 (B,H,N)")
    if H != int(n_heads) or tuple(v.shape) != (B, H, N) or tuple(g.shape) != (B, (N + 5) * H):
        raise CdssmError("decode_step_reference: inconsistent shapes")
    lds, rf = _f32(log_dt_scale, "log_dt_scale"), _f32(rope_freqs, "rope_freqs")
    y = out if out is not None else torch.empty(B, H, N, dtype=q.dtype, device=q.device)
    pos_dev, pos_i = (pos, 0) if isinstance(pos, Tensor) else (None, int(pos))
    if pos_dev is not None and (pos_dev.dtype != torch.int32 or not pos_dev.is_cuda):
        raise CdssmError("a tensor position must be an int32 CUDA tensor")
    with torch.cuda.device(q.device):
        check(_lib.lib().cdssm_b200_decode_step_reference(
            _p(state["local"]), _p(state["correction"]), _p(state["carry"]), _p(state["decay"]), _p(q), _p(k), _p(v),
            _p(g), _p(lds), _p(rf), _p(y), gating_c, omega_thresh, adt_delta, adt_smoothness, adt_eps,
            shortcut_scale, B, H, D, N, int(chunk_size), pos_i, _p(pos_dev), _dtype_code(q), _stream()),
            "decode_step_reference")
    return y


def scan_fused_status(device=None) -> int:
    """Status word of the last scan_fused call on this device and stream (synchronises the stream).
    0 means every bounded device-side wait of the tensor-core kernel completed; anything else is
    the code of the wait that ran out, and that call's outputs are undefined."""
    import ctypes
    device = torch.device("cuda" if device is None else device)
    index = torch.cuda.current_device() if device.index is None else device.index
    ptr = _lib.host().workspace_address(index)
    if ptr == 0:
        return 0
    out = ctypes.c_int(0)
    with torch.cuda.device(index):
        rc = _lib.lib().cdssm_b200_scan_fused_status(ptr, ctypes.addressof(out), _stream())
    if rc not in (0, -5):
        check(rc, "scan_fused_status")
    return out.value


def rms_norm(x: Tensor, weight: Tensor, eps: float) -> Tensor:
    """RMSNorm over the last dimension in one kernel (cdssm/models/modules.py:50-53)."""
    return _lib.host().rms_norm(x, weight, eps)


def groupnorm_gate(y: Tensor, gn_weight: Tensor, gn_bias: Tensor, z: Tensor, skip: Tensor, x_conv: Tensor,
                   groups: int, eps: float = 1e-5, per_token: bool = False) -> Tensor:
    """GroupNorm(y) * silu(z) + skip * x_conv for (B,L,di) tensors (cdssm/models/block.py:213-224) in two kernels
    (statistics over channels x all positions, as the reference takes them) or, with per_token=True, in one
    (statistics per token: the causal form used with a decode cache).  z may be a column slice of a wider
    projection (rows strided)."""
    return _lib.host().groupnorm_gate(y, gn_weight, gn_bias, z, skip, x_conv, groups, eps, per_token)


def conv1d_silu_step(x: Tensor, hist: Tensor, weight: Tensor, bias: Tensor) -> Tensor:
    """One position of the causal depthwise conv + SiLU: x (B,Dm) (rows may be strided), hist (B,3,Dm) the last
    three inputs, shifted in place.  Returns (B,Dm)."""
    return _lib.host().conv1d_silu_step(x, hist, weight, bias)


def set_wait_limit_ns(limit_ns: int) -> int:
    """Limit of the bounded device-side waits of the tensor-core kernels (0 = the 400 ms default).
    Returns the previous limit."""
    return int(_lib.lib().cdssm_b200_set_wait_limit_ns(int(limit_ns)))


def selftest_bounded_wait(limit_ns: int = 1_000_000, device=None) -> int:
    """Runs the wait primitive of the tensor-core kernels on a barrier that nothing signals.
    Returns 1 if the wait gave up after ``limit_ns`` as it must, 2 if it claimed to be signalled."""
    device = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
    st = torch.zeros(1, dtype=torch.int32, device=device)
    with torch.cuda.device(device):
        check(_lib.lib().cdssm_b200_selftest_bounded_wait(_p(st), int(limit_ns), _stream()), "selftest_bounded_wait")
    return int(st.item())


def scan_summary(k: Tensor, v: Tensor, gate_raw: Tensor, log_dt_scale: Tensor, rope_freqs: Tensor,
                 gating_c: float, omega_thresh: float, adt_delta: float, adt_smoothness: float,
                 adt_eps: float, n_heads: int, state_dim: int, chunk_size: int, h0: Tensor = None, *,
                 pos0: int = 0, segs: int = 1, flags: int = 0):
    """Summary of chunk-aligned segments: (carry_out (B,H,N,D), total_decay (B,H,N)) float32, the
    carry after the last chunk for carry-in h0 and the product of the chunk decays.  Reads k, v and
    the gates only (about half of the scan's bytes).  Of ``flags`` only FP32_DECAY applies."""
    k = _prep(k, name="k")
    v = _prep(v, dtype=k.dtype, name="v")
    g = _prep(gate_raw, dtype=k.dtype, name="gate_raw")
    B, L, H, D = k.shape
    N, C = int(state_dim), int(chunk_size)
    lds, rf = _f32(log_dt_scale, "log_dt_scale"), _f32(rope_freqs, "rope_freqs")
    if h0 is not None:
        h0 = _prep(h0, dtype=torch.float32, name="h0")
    carry = torch.zeros(B, H, N, D, dtype=torch.float32, device=k.device)
    decay = torch.zeros(B, H, N, dtype=torch.float32, device=k.device)
    decay[..., 0::2] = 1.0
    if B * L == 0:
        return (carry if h0 is None else h0.clone()), decay
    with torch.cuda.device(k.device):
        # (as scan_fused asks for it: a call that reuses the local results must find the buffer as it is)
        need = _lib.lib().cdssm_b200_scan_fused_workspace_bytes_for(B, L, H, D, N, C, _dtype_code(k), 0)
        ws_ptr, ws_bytes = _workspace(k, int(need))
        check(_lib.lib().cdssm_b200_scan_summary_fwd(
            _p(k), _p(v), _p(g), _p(lds), _p(rf), _p(h0), _p(carry), _p(decay), ws_ptr, ws_bytes, gating_c,
            omega_thresh, adt_delta, adt_smoothness, adt_eps, B, L, H, D, N, C, int(pos0), int(segs),
            _dtype_code(k), int(flags) & FP32_DECAY, _stream()), "scan_summary_fwd")
    return carry, decay


def scan_fused_long(q: Tensor, k: Tensor, v: Tensor, gate_raw: Tensor, log_dt_scale: Tensor,
                    rope_freqs: Tensor, gating_c: float, omega_thresh: float, adt_delta: float,
                    adt_smoothness: float, adt_eps: float, n_heads: int, state_dim: int, chunk_size: int,
                    h0: Tensor = None, *, segments: int = 1, sequence_parallel: bool = False, group=None,
                    shortcut_scale: float = 0.0, pos0: int = 0, flags: int = 0, timings: dict = None):
    """The fused scan of long sequences cut into chunk-aligned segments, on one GPU or - only with
    ``sequence_parallel=True`` (or an explicit ``group``) - one contiguous piece per rank of a
    torch.distributed group (rank r holds tokens [r*L, (r+1)*L) of every sequence; ``group=None`` is then
    the default group).  Without either, an initialised process group is ignored: in a data-parallel job
    every rank scans its own sequences.  ``h0`` is the carry into the FIRST token of the whole sequence;
    rank 0's value is broadcast to the group.

    Pass A summarises every segment (k, v, gates only); the ranks exchange their (decay, carry)
    summaries with one small all-gather; the carries into all segments follow from the serial
    composition; pass B scans all segments at once as a batch of B*segments rows.
    Returns (y (B,L,H,N), final_state (B,H,N,D)): final_state is the carry after this rank's last
    token (on the last rank: of the whole sequence)."""
    from . import sharding
    B, L, H, D = q.shape
    N, C, S = int(state_dim), int(chunk_size), int(segments)
    if L % (S * C):
        raise CdssmError(f"length {L} does not split into {S} chunk-aligned segments of chunk {C}")
    Ls = L // S
    seg = lambda t: t.contiguous().view(B * S, Ls, *t.shape[2:])
    consts = (gating_c, omega_thresh, adt_delta, adt_smoothness, adt_eps)
    rank, world = sharding.sequence_ranks(sequence_parallel, group)
    if world == 1 and timings is None and B * L > 0:
        return _lib.host().scan_fused_long(q, k, v, gate_raw, log_dt_scale, rope_freqs, *consts, n_heads, N, C, h0,
                                           shortcut_scale, pos0, flags, S)
    if world > 1 and h0 is not None:
        h0 = _prep(h0, dtype=torch.float32, name="h0").clone()
        torch.distributed.broadcast(h0, torch.distributed.get_global_rank(group, 0) if group is not None else 0,
                                    group=group)
    base = pos0 + rank * L
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(4)] if timings is not None else None
    if ev: ev[0].record()
    carry, decay = scan_summary(seg(k), seg(v), seg(gate_raw), log_dt_scale, rope_freqs, *consts, n_heads, N, C,
                                pos0=base, segs=S, flags=flags)
    if ev: ev[1].record()
    if world > 1:
        # this rank's piece as one summary, exchanged with the other ranks (one small all-gather)
        _, piece_out, piece_dec = compose_carries(decay, carry, None, B, S, layout="rows", want_carry_in=False)
        decs, outs = sharding.exchange_summaries(piece_dec, piece_out, group)
        ins, _, _ = compose_carries(decs, outs, h0, B, world, layout="gathered")
        h_in = ins[rank].contiguous()
    else:
        h_in = h0
    h_rows, final, _ = compose_carries(decay, carry, h_in, B, S, layout="rows")
    if ev: ev[2].record()
    y, _ = scan_fused(seg(q), seg(k), seg(v), seg(gate_raw), log_dt_scale, rope_freqs, *consts, n_heads, N, C,
                      h_rows, shortcut_scale=shortcut_scale, pos0=base, segs=S,
                      flags=flags | REUSE_LOCAL)   # pass A's local results
    if ev:
        ev[3].record()
        torch.cuda.synchronize()
        timings.update(summary_ms=ev[0].elapsed_time(ev[1]), handoff_ms=ev[1].elapsed_time(ev[2]),
                       scan_ms=ev[2].elapsed_time(ev[3]))
    return y.view(B, L, H, N), final


def compose_carries(decay: Tensor, carry_out: Tensor, h0, batch: int, segments: int, layout: str = "rows",
                    want_carry_in: bool = True):
    """Chain segment summaries on the GPU: carry_in[g] = s; s <- decay[g] * s + carry_out[g].

    layout "rows": decay (B*S,H,N), carry_out (B*S,H,N,D) are the rows of a segmented batch;
    layout "gathered": decay (S,B,H,N), carry_out (S,B,H,N,D) (one summary per rank).
    Returns (carry_in like carry_out or None, final (B,H,N,D), total_decay (B,H,N))."""
    decay = _prep(decay, dtype=torch.float32, name="decay")
    carry_out = _prep(carry_out, dtype=torch.float32, name="carry_out")
    H, N, D = carry_out.shape[-3:]
    B, S = int(batch), int(segments)
    bs, ss = (S, 1) if layout == "rows" else (1, B)
    if h0 is not None:
        h0 = _prep(h0, dtype=torch.float32, name="h0")
    dev = carry_out.device
    cin = torch.empty_like(carry_out) if want_carry_in else None
    final = torch.empty(B, H, N, D, dtype=torch.float32, device=dev)
    tot = torch.empty(B, H, N, dtype=torch.float32, device=dev)
    with torch.cuda.device(dev):
        check(_lib.lib().cdssm_b200_compose_carries(_p(decay), _p(carry_out), _p(h0), _p(cin), _p(final), _p(tot),
                                                    B, S, H, D, N, bs, ss, _stream()), "compose_carries")
    return cin, final, tot
