"""The six operator-level kernels against the CPU oracle, through the C ABI."""
import numpy as np
import pytest
import torch

from util import BF16_TOL, FP32_TOL, const_args, rel_err, to_dev, to_np

pytestmark = pytest.mark.gpu
DT = [(torch.float32, 0, FP32_TOL), (torch.bfloat16, 15, 2.0 ** -7)]


@pytest.mark.parametrize("dtype,mask,tol", DT)
@pytest.mark.parametrize("N", [2, 4, 16])
def test_dynamics(ops, orc, dtype, mask, tol, N):
    inp = orc.make_inputs(2, 6, 300, 32, N=N, seed=N, bf16=mask != 0)
    want = orc.dynamics(inp["gate_raw"], inp["log_dt_scale"], inp["rope_freqs"], inp["consts"], 6, N,
                        round_bf16=mask)
    got = ops.DynamicsFusedFn.apply(to_dev(inp["gate_raw"], dtype), to_dev(inp["log_dt_scale"], torch.float32),
                                    to_dev(inp["rope_freqs"], torch.float32), *const_args(inp["consts"]), 6, N)
    for g, w, name in zip(got, want, ("A_bar", "vp", "beta", "sel_C")):
        assert g.dtype == dtype and tuple(g.shape) == w.shape
        assert rel_err(to_np(g), w) <= tol, name


@pytest.mark.parametrize("dtype,mask,tol", DT)
@pytest.mark.parametrize("D", [64, 128, 48])
def test_normalize_kq(ops, orc, dtype, mask, tol, D):
    rng = np.random.default_rng(D)
    K = (rng.standard_normal((2, 33, 3, D)) * 3).astype(np.float32)
    Q = (rng.standard_normal((2, 33, 3, D)) * 0.2).astype(np.float32)
    if mask:
        K, Q = orc.bf16_round(K), orc.bf16_round(Q)
    wk, wq = orc.normalize_kq(K, Q, round_bf16=mask)
    gk, gq = ops.NormalizeKQFn.apply(to_dev(K, dtype), to_dev(Q, dtype))
    assert rel_err(to_np(gk), wk) <= tol and rel_err(to_np(gq), wq) <= tol


def _chunk_inputs(orc, BNC, C, H, D, N, seed, bf16):
    rng = np.random.default_rng(seed)
    mag = rng.uniform(0.3, 1.0, (BNC, C, H, N // 2))
    ang = rng.uniform(-3, 3, (BNC, C, H, N // 2))
    A = np.stack([mag * np.cos(ang), mag * np.sin(ang)], -1).reshape(BNC, C, H, N).astype(np.float32)
    K = rng.standard_normal((BNC, C, H, D)).astype(np.float32)
    K /= np.linalg.norm(K, axis=-1, keepdims=True)
    V = rng.standard_normal((BNC, C, H, N)).astype(np.float32)
    beta = rng.uniform(0, 1, (BNC, C, H)).astype(np.float32)
    if bf16:
        A, K, V, beta = (orc.bf16_round(x) for x in (A, K, V, beta))
    return A, K, V, beta


@pytest.mark.parametrize("dtype,mask,tol", [(torch.float32, 0, FP32_TOL), (torch.bfloat16, 15, BF16_TOL)])
@pytest.mark.parametrize("C,H,D,N", [(64, 3, 64, 2), (128, 2, 128, 2), (16, 2, 64, 16), (7, 1, 40, 4)])
def test_intra_inter_correction(ops, orc, dtype, mask, tol, C, H, D, N):
    B, NC = 2, 3
    A, K, V, beta = _chunk_inputs(orc, B * NC, C, H, D, N, seed=C + N, bf16=mask != 0)
    d = lambda x: to_dev(x, dtype)
    lh, cA = ops.IntraChunkScanFn.apply(d(A), d(K), d(V), d(beta), N)
    wlh, wcA = orc.intra_chunk(A, K, V, beta, N, round_bf16=mask)
    assert rel_err(to_np(lh), wlh) <= tol and rel_err(to_np(cA), wcA) <= tol
    tA = wcA.reshape(B, NC, C, H, N)[:, :, -1]
    fl = wlh.reshape(B, NC, C, H, N, D)[:, :, -1]
    cs = ops.InterChunkScanFn.apply(d(tA), d(fl), N)
    wcs = orc.inter_chunk(tA, fl, N, round_bf16=mask)
    assert rel_err(to_np(cs), wcs) <= tol
    r5 = lambda x: x.reshape(B, NC, *x.shape[1:])
    co = ops.ExactCorrectionFn.apply(d(r5(A)), d(r5(K)), d(r5(beta)), d(wcs), N)
    wco = orc.exact_correction(r5(A), r5(K), r5(beta), wcs, N, round_bf16=mask)
    assert tuple(co.shape) == (B, NC, C, H, N, D)
    assert rel_err(to_np(co), wco) <= tol


@pytest.mark.parametrize("dtype,mask,tol", DT)
@pytest.mark.parametrize("B,L,Dm", [(2, 100, 192), (1, 3, 40), (3, 1, 128)])
def test_conv1d_silu(ops, orc, dtype, mask, tol, B, L, Dm):
    rng = np.random.default_rng(L)
    x = rng.standard_normal((B, L, Dm)).astype(np.float32)
    w = (rng.standard_normal((Dm, 1, 4)) * 0.5).astype(np.float32)
    b = (rng.standard_normal(Dm) * 0.1).astype(np.float32)
    if mask:
        x, w, b = (orc.bf16_round(t) for t in (x, w, b))
    want = orc.conv1d_silu(x, w, b, round_bf16=mask)
    got = ops.CUDAConv1dSiLUOp.apply(to_dev(x, dtype), to_dev(w, dtype), to_dev(b, dtype))
    assert rel_err(to_np(got), want) <= tol


def test_errors_mirror_reference_checks(ops):
    x = torch.zeros(1, 4, 64, device="cuda", dtype=torch.bfloat16)
    with pytest.raises(RuntimeError):                       # conv1d_silu.cu:241
        ops.CUDAConv1dSiLUOp.apply(x, torch.zeros(64, 1, 3, device="cuda"), torch.zeros(64, device="cuda"))
    K = torch.zeros(1, 4, 1, 256, device="cuda", dtype=torch.bfloat16)
    A = torch.zeros(1, 4, 1, 2, device="cuda", dtype=torch.bfloat16)
    with pytest.raises(RuntimeError):                       # intra_chunk_scan.cu:584
        ops.IntraChunkScanFn.apply(A, K, A, A[..., 0], 2)


# What has another rank, an empty last dimension or no batch is an error: nothing is launched on sizes read from the wrong places.
def test_wrong_ranks_are_refused(ops):
    z = lambda *s: torch.zeros(*s, device="cuda", dtype=torch.bfloat16)
    f = lambda *s: torch.zeros(*s, device="cuda")
    dyn = (1.0, 0.1, 0.1, 0.02, 1.0)
    calls = [
        lambda: ops.CUDAConv1dSiLUOp.apply(z(2, 8, 16, 3), z(16, 1, 4), z(16)),
        lambda: ops.CUDAConv1dSiLUOp.apply(z(8, 16), z(16, 1, 4), z(16)),
        lambda: ops.DynamicsFusedFn.apply(z(2, 8, 7 * 3, 2), f(3), f(3), *dyn, 3, 2),
        lambda: ops.IntraChunkScanFn.apply(z(2, 8, 3, 2), z(2, 8, 3, 64, 2), z(2, 8, 3, 2), z(2, 8, 3), 2),
        lambda: ops.InterChunkScanFn.apply(z(2, 4, 3, 2), z(2, 4, 3, 2, 64, 2), 2),
        lambda: ops.ExactCorrectionFn.apply(z(2, 4, 8, 3, 2), z(2, 4, 8, 3, 64, 2), z(2, 4, 8, 3), z(2, 4, 3, 2, 64), 2),
        lambda: ops.NormalizeKQFn.apply(z(2, 3, 0), z(2, 3, 0)),
        lambda: ops.rms_norm(z(2, 0), z(0), 1e-5),
        lambda: ops.groupnorm_gate(z(2, 4, 64, 2), z(64), z(64), z(2, 4, 64, 2), z(64), z(2, 4, 64, 2), 8),
        lambda: ops.conv1d_silu_step(z(2, 16, 2), z(2, 3, 16), z(16, 1, 4), z(16)),
    ]
    for i, call in enumerate(calls):
        with pytest.raises((RuntimeError, ValueError, IndexError)):
            call()
    torch.cuda.synchronize()


def test_wrong_ids_and_weights_are_refused(ops):
    from cdssm_b200.model import CdssmConfig, CdssmLM
    lm = CdssmLM(CdssmConfig(d_model=256, n_layers=2, context_length=128, vocab_size=100, state_dim=2), seed=1)
    ids = torch.zeros(2, 8, dtype=torch.int64, device="cuda")
    logits, cache = lm.prefill(ids)
    with pytest.raises((RuntimeError, ValueError)):
        lm.forward(ids[0])                                 # (L): the batch would be taken for the length
    with pytest.raises((RuntimeError, ValueError, IndexError)):
        lm.prefill(ids[None])
    with pytest.raises((RuntimeError, ValueError)):
        lm.decode(ids[:, :1], cache)
    assert torch.isfinite(lm.forward(ids.tolist())).all()  # a list of lists indexes the embedding, as it always did
    assert torch.isfinite(lm.decode([3, 4], cache)).all()
    for name, shape in (("w_out", (256, 500)), ("w_readout", (512, 8)), ("w_q", (512, 256))):
        good = getattr(lm.blocks[1], name)
        setattr(lm.blocks[1], name, torch.zeros(*shape, device="cuda", dtype=torch.bfloat16))
        with pytest.raises(RuntimeError):
            lm.forward(ids)
        setattr(lm.blocks[1], name, good)
    odd = CdssmLM(CdssmConfig(d_model=48, n_layers=1, context_length=128, vocab_size=100, state_dim=2), seed=1)   # 96 = 1.5 heads
    with pytest.raises(RuntimeError):
        odd.forward(ids)
    torch.cuda.synchronize()


def _step_args(ops, B=2, H=3, N=4, D=64):
    from cdssm_b200.model import CdssmConfig
    g = torch.Generator(device="cuda").manual_seed(1)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    c = CdssmConfig(d_model=128, n_layers=1, context_length=64, vocab_size=64, state_dim=N)
    consts = (c.gating_c, c.omega_thresh, c.adt_delta, c.adt_smoothness, c.adt_eps)
    return (r(B, H, D), r(B, H, D), r(B, H, N), r(B, (N + 5) * H), r(H).float(), torch.ones(H, device="cuda"), *consts, H, N)


def test_outputs_are_seen_by_dispatch_modes(ops):
    """An output's allocation passes the dispatcher where somebody looks on (memory trackers, loggers)."""
    from torch.utils._python_dispatch import TorchDispatchMode

    class Seen(TorchDispatchMode):
        names = []

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            self.names.append(func.name())
            return func(*args, **(kwargs or {}))

    args = _step_args(ops)
    state = torch.zeros(2, 3, 4, 64, device="cuda")
    want = ops.decode_step(state.clone(), *args, 5)
    with Seen() as seen:
        y = ops.decode_step(state, *args, 5)
    assert any(n.startswith("aten::empty") for n in seen.names)
    assert torch.equal(y, want)
