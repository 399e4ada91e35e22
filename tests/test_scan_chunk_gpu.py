"""The whole-chunk tensor-core scan (bf16, chunk = head_dim in {64, 128}, N <= 16) against the CPU oracle and the CUDA-core
kernels: one, two, four and eight pair slots, partly filled ones, ragged lengths, chunk counts on both sides of a hand-off,
each of its three forms (one kernel; local pass; output pass) and decays beyond the range of its scaled unknowns."""
import numpy as np
import pytest
import torch

from test_scan_gpu import oracle_scan, run_fused, unnormalise
from util import BF16_TOL, rel_err, to_np

pytestmark = pytest.mark.gpu
KEEP_SIMT_LOCAL, KEEP_SIMT_OUTPUT = 256, 512

SHAPES = [  # B, H, L, D, N
    (1, 3, 1, 64, 2), (2, 5, 65, 64, 4), (1, 6, 200, 64, 6), (2, 3, 63, 64, 8), (1, 2, 449, 64, 16), (3, 24, 130, 64, 16),
    (1, 6, 129, 128, 2), (2, 3, 255, 128, 4), (1, 4, 300, 128, 8), (1, 2, 385, 128, 10), (1, 3, 128, 128, 16),
]


def _tol(D):
    """Against the oracle with float32 state and the reference's bf16 unit rows: the kernels keep normalised rows in
    float32, up to a bf16 ulp per element of a D-term dot product."""
    return BF16_TOL / 2 if D == 128 else 0.75 * BF16_TOL


def _inputs(orc, B, H, L, D, N, seed):
    inp = unnormalise(orc.make_inputs(B, H, L, D, N=N, seed=seed, bf16=True, context_length=max(L, 2)), np.random.default_rng(seed))
    inp["q"], inp["k"] = orc.bf16_round(inp["q"]), orc.bf16_round(inp["k"])
    return inp


def _close(a, b, tol):
    assert np.abs(to_np(a) - to_np(b)).max() <= tol * max(np.abs(to_np(b)).max(), 1e-3)


@pytest.mark.parametrize("keep", [0, KEEP_SIMT_LOCAL, KEEP_SIMT_OUTPUT])
@pytest.mark.parametrize("B,H,L,D,N", SHAPES)
def test_chunk_scan_matches_oracle_and_simt(ops, orc, B, H, L, D, N, keep):
    inp = _inputs(orc, B, H, L, D, N, seed=L + H)
    h0 = np.random.default_rng(1).standard_normal((B, H, N, D)).astype(np.float32) * 0.3
    kw = dict(h0=h0, shortcut_scale=0.5)
    y, fin, tail = run_fused(ops, inp, torch.bfloat16, N, D, flags=keep, return_tail_state=True, **kw)
    assert ops.scan_fused_status() == 0
    ys, fs, ts = run_fused(ops, inp, torch.bfloat16, N, D, flags=ops.FORCE_SIMT, return_tail_state=True, **kw)
    wy, wf = oracle_scan(orc, inp, N, D, orc.ROUND_FP32_STATE, **kw)
    assert rel_err(to_np(y), wy) <= _tol(D)
    assert rel_err(to_np(y), to_np(ys)) <= BF16_TOL / 2
    _close(fin, fs, 2e-2)
    _close(tail, ts, 2e-2)
    y2, fin2, tail2 = run_fused(ops, inp, torch.bfloat16, N, D, flags=keep, return_tail_state=True, **kw)
    assert torch.equal(y, y2) and torch.equal(fin, fin2) and torch.equal(tail, tail2)


@pytest.mark.parametrize("D,N", [(64, 2), (64, 16), (128, 4)])
@pytest.mark.parametrize("alpha_gate", [None, 2.0])
def test_chunk_scan_strong_decay(ops, orc, D, N, alpha_gate):
    """alpha_gate None: decays still inside the range of the scaled unknowns; 2.0: pairs that take the walk by steps."""
    B, H, L = 1, 3, 320
    inp = _inputs(orc, B, H, L, D, N, seed=11)
    g, NH = inp["gate_raw"].copy(), N // 2
    g[:, 70:250, (N + 4) * H:] += 8.0            # r gate: exponent of the decay magnitude at its maximum
    if alpha_gate is None:
        g[:, 70:250, :NH * H] += 4.0
    else:                                        # the first and the last pair only: mixed column tiles
        for j in {0, NH - 1}:
            g[:, 70:250, j * H:(j + 1) * H] = alpha_gate
            g[:, 70:250, (NH + j) * H:(NH + j + 1) * H] = 0.0
    inp["gate_raw"] = orc.bf16_round(g)
    y, fin, tail = run_fused(ops, inp, torch.bfloat16, N, D, return_tail_state=True, shortcut_scale=0.3)
    assert ops.scan_fused_status() == 0
    ys, fs, ts = run_fused(ops, inp, torch.bfloat16, N, D, flags=ops.FORCE_SIMT, return_tail_state=True, shortcut_scale=0.3)
    wy, _ = oracle_scan(orc, inp, N, D, orc.ROUND_FP32_STATE, shortcut_scale=0.3)
    assert np.isfinite(to_np(y)).all()
    assert rel_err(to_np(y), wy) <= _tol(D)
    assert rel_err(to_np(y), to_np(ys)) <= BF16_TOL / 2
    _close(fin, fs, 2e-2)
    _close(tail, ts, 2e-2)


@pytest.mark.parametrize("keep", [0, KEEP_SIMT_LOCAL, KEEP_SIMT_OUTPUT])
@pytest.mark.parametrize("D,N", [(64, 4), (64, 16), (128, 4), (128, 16)])
@pytest.mark.parametrize("decay", ["every token", "two tokens"])
def test_chunk_scan_decay_on_both_sides_of_a_block_boundary(ops, orc, D, N, decay, keep):
    """A strong decay in the second half of a 32-token block and another in the first half of the next, each inside the range of the
    scaled unknowns (1e-30), their product far below the smallest float32: what one block hands to the next is of order one all the same.
    Each output against the walk: both round y twice, four times 2^-8 of the larger of itself and the typical output."""
    B, H, L = 2, 4, 4 * D - 3
    inp = _inputs(orc, B, H, L, D, N, seed=5)
    NH, r = N // 2, slice((N + 4) * H, None)
    inp["rope_freqs"], inp["log_dt_scale"] = np.zeros(H, np.float32), np.zeros(H, np.float32)
    inp["consts"] = orc.derive_constants(2048)
    g = inp["gate_raw"].copy()
    if decay == "every token":                   # 0.02 each
        g[..., :NH * H], g[..., NH * H:2 * NH * H], g[..., (N + 2) * H:(N + 3) * H] = 4.0, 0.0, 1.0
        g[..., r] = np.random.default_rng(6).uniform(0.7, 0.9, g[..., r].shape)
    else:                                        # 1e-19 once, ordinary ones beside it
        at = (np.arange(L) % 64 == 18) | (np.arange(L) % 64 == 44)
        g[..., r] -= 2.0
        g[:, at, :NH * H], g[:, at, NH * H:2 * NH * H], g[:, at, (N + 2) * H:(N + 3) * H] = 2.0625, 0.0, 0.0
        g[:, at, r] = 8.0
    inp["gate_raw"] = orc.bf16_round(g)
    A, *_ = orc.dynamics(inp["gate_raw"], inp["log_dt_scale"], inp["rope_freqs"], inp["consts"], H, N, round_bf16=orc.ROUND_INPUTS)
    size = np.log10(np.hypot(A[..., 0::2], A[..., 1::2]))[:, :2 * 32].reshape(B, 4, 16, H, NH).sum(2)   # of the first half blocks
    assert size.min() > -29.0 and np.median(size[:, 1] + size[:, 2]) < -40.0
    y, fin, tail = run_fused(ops, inp, torch.bfloat16, N, D, flags=keep, return_tail_state=True, shortcut_scale=0.3)
    assert ops.scan_fused_status() == 0
    ys, fs, ts = run_fused(ops, inp, torch.bfloat16, N, D, flags=ops.FORCE_SIMT, return_tail_state=True, shortcut_scale=0.3)
    for a, b in ((y, ys), (fin, fs), (tail, ts)):
        a, b = to_np(a), to_np(b)
        assert (np.abs(a - b) <= 2.0 ** -6 * np.maximum(np.abs(b), np.sqrt(np.square(b).mean()))).all()
