"""What the tensor-core scans promise beyond closeness: float32 states where a float32 state is handed out, the same bits for a
shard or a piece as for the whole, and no token touched by one behind it."""
import numpy as np
import pytest
import torch

from test_scan_gpu import run_fused, unnormalise
from util import const_args, to_dev, to_np

pytestmark = pytest.mark.gpu


def _inputs(orc, B, H, L, D, N, seed):
    inp = unnormalise(orc.make_inputs(B, H, L, D, N=N, seed=seed, bf16=True, context_length=max(L, 2)), np.random.default_rng(seed))
    inp["q"], inp["k"] = orc.bf16_round(inp["q"]), orc.bf16_round(inp["k"])
    return inp


def _cut(inp, rows=slice(None), tokens=slice(None)):
    return {k: (v[rows, tokens] if getattr(v, "ndim", 0) >= 3 else v) for k, v in inp.items()}


def _state64(ops, inp, N):
    """The recurrent state after a single chunk in float64, from the package's own (bf16) dynamics."""
    c = inp["consts"]
    args = (c["gating_c"], c["omega_thresh"], c["adt_delta"], c["adt_smoothness"], c["adt_eps"])
    k = to_dev(inp["k"], torch.float64)
    B, L, H, D = k.shape
    A, vp, beta, _ = ops.DynamicsFusedFn.apply(to_dev(inp["gate_raw"], torch.bfloat16), to_dev(inp["log_dt_scale"], torch.float32),
                                               to_dev(inp["rope_freqs"], torch.float32), *args, H, N)
    v = (to_dev(inp["v"], torch.bfloat16) * vp.repeat_interleave(2, -1)).double()
    z = torch.zeros(B, H, N, D, dtype=torch.float64, device="cuda")
    for t in range(L):
        kn = (k[:, t] / (k[:, t].square().sum(-1, keepdim=True) + 1e-6).sqrt())[:, :, None]
        b = beta[:, t].double()[..., None, None]
        z = z - b * (z * kn).sum(-1, keepdim=True) * kn
        re, im = (A[:, t].double()[..., i::2, None] for i in (0, 1))
        z = torch.stack([re * z[:, :, 0::2] - im * z[:, :, 1::2], re * z[:, :, 1::2] + im * z[:, :, 0::2]], 3).flatten(2, 3)
        z = z + b * v[:, t][..., None] * kn
    return z


@pytest.mark.parametrize("H,D,N", [(8, 64, 2), (6, 64, 2), (4, 128, 2), (3, 64, 4), (3, 64, 8), (3, 64, 16), (2, 128, 4), (2, 128, 8),
                                   (2, 128, 16)])
def test_tail_state_has_float32_precision(ops, orc, H, D, N):
    """One chunk: nothing between the inputs and the state is rounded, so the state is as near to float64 as the walk's, which is all
    float32.  Measured, times 1e-7 of the state, D 64 / 128: N > 2 1.6 / 1.8, N 2 1.8 / 2.0, the walk 1.2 to 2.1 / 2.0 to 2.2; three bf16
    parts for N > 2 1.7 / 2.3, operands of 22 bits cut off instead of rounded 2.4 / 2.5, products of 16-bit parts 170.  The bound: 3.7
    roundings.  (The median over heads and pairs: where the dynamics of the two sides round one bf16 value differently, a head moves
    by more.)"""
    B, L = 24, D - 3
    inp = _inputs(orc, B, H, L, D, N, seed=D + N)
    want = _state64(ops, inp, N).view(B, H, N // 2, 2 * D)
    err = []
    for flags in (0, ops.FORCE_SIMT):
        tail = run_fused(ops, inp, torch.bfloat16, N, D, return_tail_state=True, flags=flags)[2]
        off = (tail.double().view(B, H, N // 2, 2 * D) - want).norm(dim=-1) / want.norm(dim=-1)
        err.append(float(off.median()))
    assert err[0] <= 3.7 * 2.0 ** -24 and err[0] <= 1.6 * err[1]


@pytest.mark.parametrize("H,D,N", [(8, 64, 2), (6, 64, 2), (4, 128, 2), (8, 64, 4), (8, 64, 16), (4, 128, 8), (4, 128, 16)])
@pytest.mark.parametrize("tail", [False, True])
def test_shards_and_pieces_have_the_bits_of_the_whole(ops, orc, H, D, N, tail):
    """Rows of a batch alone, and chunk-aligned pieces chained through (final_state, pos0), at sizes from one chunk to
    where the GPU is full: the kernel may not go by batch or length."""
    B, L = 24, 12 * D - 5
    inp = _inputs(orc, B, H, L, D, N, seed=H + N)
    h0 = np.random.default_rng(3).standard_normal((B, H, N, D)).astype(np.float32) * 0.3
    run = lambda i, h, **kw: run_fused(ops, i, torch.bfloat16, N, D, h0=h, return_tail_state=tail, **kw)
    whole = run(inp, h0)
    for rows in (slice(0, 1), slice(7, 10)):
        part = run(_cut(inp, rows), h0[rows])
        for w, p in zip(whole, part):
            assert torch.equal(w[rows], p)
    cut = 2 * D
    first = run(_cut(inp, tokens=slice(0, cut)), h0)
    second = run(_cut(inp, tokens=slice(cut, None)), to_np(first[1]), pos0=cut)
    assert torch.equal(torch.cat([first[0], second[0]], 1), whole[0])
    for w, p in zip(whole[1:], second[1:]):
        assert torch.equal(w, p)


@pytest.mark.parametrize("H,D,N", [(8, 64, 2), (8, 64, 4), (3, 64, 16), (4, 128, 4), (2, 128, 16)])
def test_forms_of_a_kernel_have_the_same_bits(ops, orc, H, D, N):
    """With a carry pass, without one and with the carry handed on inside one kernel: 60 chunks in a row, the same in pieces
    of 1, 9 and 50, and beside a batch that fills the GPU."""
    B, L = 1, 60 * D
    inp = _inputs(orc, B, H, L, D, N, seed=N + D)
    run = lambda i, **kw: run_fused(ops, i, torch.bfloat16, N, D, **kw)
    y, fin = run(inp)
    ys, h, at = [], None, 0
    for n in (1, 9, 50):
        piece, f = run(_cut(inp, tokens=slice(at * D, (at + n) * D)), h0=h, pos0=at * D)
        ys.append(piece)
        h, at = to_np(f), at + n
    assert torch.equal(torch.cat(ys, 1), y) and torch.equal(f, fin)
    wide = {k: (np.repeat(v, 16, 0) if getattr(v, "ndim", 0) >= 3 else v) for k, v in inp.items()}
    yw, fw = run(wide)
    assert torch.equal(yw[:1], y) and torch.equal(yw[15:], y) and torch.equal(fw[7:8], fin)


@pytest.mark.parametrize("D,N", [(64, 2), (128, 2), (64, 4), (64, 8), (64, 16), (128, 4), (128, 16)])
@pytest.mark.parametrize("value", [float("nan"), float("inf"), 3e19])
@pytest.mark.parametrize("what", ["k", "v", "beta", "decay"])
def test_tokens_before_a_bad_value_do_not_see_it(ops, orc, D, N, value, what):
    """NaN, infinity and a key whose square overflows, in one token of one head: every other token's output is a number where
    the walk by steps gives one, and the same.  (At the token itself, components that a complex product joins may differ.)"""
    B, H, L, t = 1, 3, 2 * D + 40, D + 21
    inp = _inputs(orc, B, H, L, D, N, seed=N)
    if what == "k":
        inp["k"][0, t, 1, 5] = value
    elif what == "v":
        inp["v"][0, t, 1, 0] = value
    else:
        inp["gate_raw"][0, t, {"beta": (N + 3) * H, "decay": 0}[what] + 1] = value
    y, fin, tail = run_fused(ops, inp, torch.bfloat16, N, D, return_tail_state=True)
    ys, fs, ts = run_fused(ops, inp, torch.bfloat16, N, D, return_tail_state=True, flags=ops.FORCE_SIMT)
    assert ops.scan_fused_status() == 0
    for a, b in ((y, ys), (fin, fs), (tail, ts)):
        a, b = to_np(a), to_np(b)
        if a.shape == tuple(y.shape):
            a, b = np.delete(a, t, 1), np.delete(b, t, 1)
        assert np.array_equal(np.isfinite(a), np.isfinite(b))
        ok = np.isfinite(b)
        assert np.abs(a[ok] - b[ok]).max() <= 2e-2 * np.abs(b[ok]).max()
    assert np.isfinite(to_np(y)[0, :t]).all()


@pytest.mark.parametrize("B,H,NC,D,N,few", [(1, 3, 5, 64, 4, 2), (2, 5, 3, 64, 16, 2), (24, 8, 40, 64, 6, 3), (1, 1, 29, 64, 16, 3), (3, 2, 4, 128, 8, 2),
                                            (2, 3, 2, 128, 16, 2), (1, 2, 60, 64, 8, 3), (1, 1, 70, 128, 4, 3), (1, 3, 13, 64, 10, 2), (1, 5, 1, 64, 12, 2)])
def test_scratch_without_room_for_the_carries_gives_the_same_bits(ops, orc, B, H, NC, D, N, few):
    """The whole-chunk scan hands the carry on inside one kernel where the scratch has room for the words that do it, else between
    two, with a carry pass in between where there are many chunks: full and partly filled column tiles, an odd last head, two blocks
    a chunk, more chunks back than a warp asks for at once."""
    import ctypes
    import cdssm_b200
    lib = cdssm_b200._lib.lib()
    L = NC * D - 3
    inp = _inputs(orc, B, H, L, D, N, seed=N)
    bf = lambda x: to_dev(x, torch.bfloat16)
    f = lambda x: to_dev(x, torch.float32)
    h0 = f(np.random.default_rng(5).standard_normal((B, H, N, D)).astype(np.float32))
    t = [bf(inp[k]) for k in ("q", "k", "v", "gate_raw")] + [f(inp["log_dt_scale"]), f(inp["rope_freqs"]), h0]
    full = ops.scan_fused_workspace_bytes(B, L, H, D, N, D)
    least = full - B * NC * H * (N // 2) * D * 8
    results = []
    for room in (full, least):
        ws = torch.full((room + 256,), 0xa5, dtype=torch.uint8, device="cuda")
        out = [torch.full((B, L, H, N), 3.0, device="cuda", dtype=torch.bfloat16), torch.full((B, H, N, D), 3.0, device="cuda"),
               torch.full((B, H, N, D), 3.0, device="cuda")]
        args = [x.data_ptr() for x in t + out] + [ws.data_ptr() + (-ws.data_ptr()) % 256, room]
        args += [ctypes.c_float(c) for c in const_args(inp["consts"])] + [ctypes.c_float(0.25), B, L, H, D, N, D, 0, 0, 0]
        before = lib.cdssm_b200_launch_count()
        assert lib.cdssm_b200_scan_fused_fwd(*args, torch.cuda.current_stream().cuda_stream) == 0
        passes = lib.cdssm_b200_launch_count() - before - 1   # (behind the records)
        assert passes == (1 if room == full else few)
        torch.cuda.synchronize()
        # (one kernel: a word per gamma and per column of a state, where the passes keep two floats; nothing else is cleared)
        units, up = B * NC * H * (N // 2), lambda n: -(-n // 256) * 256
        at = (-ws.data_ptr()) % 256 + 256
        unused = ws[at + up(4 * units) + 4 * units * D:at + up(8 * units) + up(8 * units * D)]
        assert room < full or bool((unused == 0xa5).all())
        results.append(out)
    for a, b in zip(*results):
        assert torch.equal(a, b)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("L,D,N,C", [(317, 64, 4, 64), (5, 64, 2, 64), (129, 64, 2, 32), (260, 128, 2, 128)])
def test_rows_that_travel_ahead_change_no_bit(ops, orc, dtype, L, D, N, C):
    """The CUDA-core walk takes its rows ahead through shared memory while every SM has a block at most (1 500 units), and one row ahead in
    registers beyond (few units: scan_short.cu): fewer tokens than rows travel ahead, ragged and short chunks, a short chunk first and a longer
    one behind."""
    inp = _inputs(orc, 1, 3, L, D, N, seed=L)
    inp["q"], inp["k"] = inp["q"] * 0.7, inp["k"] * 1.3
    few = run_fused(ops, inp, dtype, N, C, return_tail_state=True, flags=ops.FORCE_SIMT)
    units = -(-L // C) * 3 * (N // 2)
    for times in (1500 // units, 148 * 16 // units + 1):
        wide = {k: (np.repeat(v, times, 0) if getattr(v, "ndim", 0) >= 3 else v) for k, v in inp.items()}
        many = run_fused(ops, wide, dtype, N, C, return_tail_state=True, flags=ops.FORCE_SIMT)
        for f, m in zip(few, many):
            assert torch.equal(m[:1], f) and torch.equal(m[-1:], f)


def test_two_threads_share_a_stream(ops, orc):
    """Scans of two sizes from two threads on one stream: each uses the stream's scratch buffer for itself."""
    import threading
    sizes = [(2, 4, 700, 64, 2), (1, 3, 300, 64, 16)]
    calls, want = [], []
    for B, H, L, D, N in sizes:
        inp = orc.make_inputs(B, H, L, D, N=N, seed=N, bf16=True)
        d = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()
        args = [d(inp[k]).bfloat16() for k in ("q", "k", "v", "gate_raw")] + [d(inp["log_dt_scale"]), d(inp["rope_freqs"]),
                                                                             *const_args(inp["consts"]), H, N, D]
        calls.append(args)
        want.append(ops.scan_fused(*args, return_tail_state=True))
    torch.cuda.synchronize()
    bad = []

    def work(i):
        for _ in range(150):
            got = ops.scan_fused(*calls[i], return_tail_state=True)
            if not all(torch.equal(a, b) for a, b in zip(got, want[i])):
                bad.append(i)

    threads = [threading.Thread(target=work, args=(i,)) for i in (0, 1, 0, 1)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not bad
