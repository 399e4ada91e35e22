"""The failure path of the tensor-core scan: every device-side wait is bounded, and a wait that runs out makes
the kernels unwind (status word set, tensor memory freed, context usable) instead of hanging.  The tests make
waits run out on purpose in the only allowed way: a barrier that nothing signals and a short limit."""
import numpy as np
import pytest
import torch

from test_scan_gpu import oracle_scan, run_fused
from util import BF16_TOL, const_args, rel_err, to_np

pytestmark = pytest.mark.gpu


def test_wait_primitive_gives_up_after_its_limit(ops):
    assert ops.selftest_bounded_wait(1_000_000) == 1      # 1 ms: gave up, reported it, returned
    assert ops.selftest_bounded_wait(200_000) == 1
    torch.cuda.synchronize()


@pytest.mark.parametrize("D", [128, 64])
def test_scan_waits_run_out_and_the_next_call_is_correct(ops, orc, D):
    B, H, L, N = 1, 4, 2 * D + 5, 2
    inp = orc.make_inputs(B, H, L, D, N=N, seed=41, bf16=True)
    old = ops.set_wait_limit_ns(2_000_000)                # 2 ms instead of 400 ms
    try:
        run_fused(ops, inp, torch.bfloat16, N, D, flags=ops.TENSOR_CORE_WA | ops.TEST_WITHHOLD)
        code = ops.scan_fused_status()
        assert 200 <= code < 400, code                    # a compute warp (2xx) or the producer (3xx) gave up
        with pytest.raises(ops.CdssmError):
            run_fused(ops, inp, torch.bfloat16, N, D, flags=ops.TENSOR_CORE_WA | ops.TEST_WITHHOLD, strict=True)
    finally:
        ops.set_wait_limit_ns(old)
    # the context is intact and tensor memory was released: the same scan now runs and is right
    y, fin = run_fused(ops, inp, torch.bfloat16, N, D, flags=ops.TENSOR_CORE_WA, strict=True)
    assert ops.scan_fused_status() == 0
    wy, _ = oracle_scan(orc, inp, N, D, orc.ROUND_REFERENCE)
    assert rel_err(to_np(y), wy) <= BF16_TOL


@pytest.mark.parametrize("D,L", [(64, 69), (64, 3000), (128, 133)])
def test_whole_chunk_scan_waits_run_out_too(ops, orc, D, L):
    """Both forms of the whole-chunk scan (a few chunks; a chain of them)."""
    B, H, N = 1, 3, 4
    inp = orc.make_inputs(B, H, L, D, N=N, seed=42, bf16=True)
    old = ops.set_wait_limit_ns(2_000_000)
    try:
        run_fused(ops, inp, torch.bfloat16, N, D, flags=ops.TEST_WITHHOLD)
        assert 200 <= ops.scan_fused_status() < 300
    finally:
        ops.set_wait_limit_ns(old)
    y, _ = run_fused(ops, inp, torch.bfloat16, N, D, strict=True)
    wy, _ = oracle_scan(orc, inp, N, D, orc.ROUND_REFERENCE)
    assert rel_err(to_np(y), wy) <= BF16_TOL


@pytest.mark.parametrize("D,N", [(64, 16), (64, 8), (128, 16)])
@pytest.mark.parametrize("keep", [256, 512])
def test_halves_of_the_whole_chunk_scan_give_up_too(ops, orc, D, N, keep):
    """Its output pass (256: the local results come from the walk) and its local pass (512), two warps or two blocks to a chunk; the
    next call finds the tensor memory free, with a key that is no number among its rows."""
    B, H, L = 2, 5, 3 * D + 7
    inp = orc.make_inputs(B, H, L, D, N=N, seed=43, bf16=True)
    old = ops.set_wait_limit_ns(2_000_000)
    try:
        run_fused(ops, inp, torch.bfloat16, N, D, flags=ops.TEST_WITHHOLD | keep)
        assert 200 <= ops.scan_fused_status() < 300
    finally:
        ops.set_wait_limit_ns(old)
    inp["k"][1, D + 3, 2, 7] = np.nan
    y, _ = run_fused(ops, inp, torch.bfloat16, N, D, strict=True, flags=keep)
    y = to_np(y)
    assert np.isnan(y[1, D + 3:, 2]).all()
    inp["k"][1, D + 3:, 2] = inp["k"][1, D + 2, 2]
    wy, _ = oracle_scan(orc, inp, N, D, orc.ROUND_FP32_STATE)
    y[1, D + 3:, 2] = wy[1, D + 3:, 2]
    assert rel_err(y, wy) <= BF16_TOL


@pytest.mark.parametrize("D,N,H,L", [(64, 16, 24, 523), (64, 12, 3, 69), (128, 8, 12, 1000), (128, 16, 2, 133)])
def test_wide_blocks_give_up_too(ops, orc, D, N, H, L):
    """The form with a warp per column tile (a block per SM at most), with tickets."""
    inp = orc.make_inputs(1, H, L, D, N=N, seed=44, bf16=True)
    old = ops.set_wait_limit_ns(2_000_000)
    try:
        run_fused(ops, inp, torch.bfloat16, N, D, flags=ops.TEST_WITHHOLD)
        assert 200 <= ops.scan_fused_status() < 300
    finally:
        ops.set_wait_limit_ns(old)
    y, _ = run_fused(ops, inp, torch.bfloat16, N, D, strict=True)
    wy, _ = oracle_scan(orc, inp, N, D, orc.ROUND_REFERENCE)
    assert rel_err(to_np(y), wy) <= BF16_TOL


@pytest.mark.parametrize("D,N,H,L", [(64, 16, 24, 523), (64, 10, 24, 700), (128, 8, 12, 1400)])
def test_wide_blocks_of_two_streams_share_the_gpu(ops, orc, D, N, H, L):
    """Two calls whose blocks fill an SM each and are together more than there are SMs: a block that waits for another must find it done or
    running whichever call's blocks started first."""
    inp = orc.make_inputs(1, H, L, D, N=N, seed=45, bf16=True)
    d = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()
    args = [d(inp[k]).bfloat16() for k in ("q", "k", "v", "gate_raw")] + [d(inp["log_dt_scale"]), d(inp["rope_freqs"]), *const_args(inp["consts"]),
                                                                         H, N, D]
    want = ops.scan_fused(*args)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    got = [[], []]
    for i in range(40):
        for s, out in zip(streams, got):
            with torch.cuda.stream(s):
                out.append(ops.scan_fused(*args))
                if i % 10 == 9:
                    assert ops.scan_fused_status() == 0
    torch.cuda.synchronize()
    for out in got:
        for y, fin in out:
            assert torch.equal(y, want[0]) and torch.equal(fin, want[1])
