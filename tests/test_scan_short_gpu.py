"""The walk for few units (csrc/scan_short.cu) has the bits of the walk for many (csrc/scan_simt.cu)."""
import ctypes

import numpy as np
import pytest
import torch

from test_scan_gpu import unnormalise
from util import const_args, to_dev

pytestmark = pytest.mark.gpu


def _call(lib, t, outs, consts, dims, dt, room=None, flags=1):
    """The scan through the C ABI, by default on the CUDA cores; t: q, k, v, gates, log_dt_scale, rope_freqs, h0."""
    B, L, H, D, N, C = dims
    if room is None:
        room = lib.cdssm_b200_scan_fused_workspace_bytes_for(B, L, H, D, N, C, dt, flags)
    ws = torch.full((room + 256,), 0x5a, dtype=torch.uint8, device="cuda")
    ptr = lambda x: ctypes.c_void_p(0 if x is None else x.data_ptr())
    args = [ptr(x) for x in t + outs] + [ctypes.c_void_p(ws.data_ptr() + (-ws.data_ptr()) % 256), ctypes.c_size_t(room)]
    args += [ctypes.c_float(c) for c in consts] + [ctypes.c_float(0.25), B, L, H, D, N, C, 3, dt, flags]
    assert lib.cdssm_b200_scan_fused_fwd(*args, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    torch.cuda.synchronize()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,L,D,N,C", [(1, 1, 64, 2, 64), (3, 31, 64, 6, 64), (2, 33, 64, 2, 64), (2, 64 * 12 + 1, 64, 2, 64), (1, 64 * 13, 64, 4, 64),
                                       (1, 500, 64, 2, 200), (2, 70, 64, 32, 16), (1, 96, 64, 2, 40), (1, 127, 128, 2, 128), (2, 385, 128, 2, 128),
                                       (1, 300, 128, 6, 256)])
@pytest.mark.parametrize("records", [True, False])
def test_few_units_have_the_bits_of_many(ops, orc, dtype, H, L, D, N, C, records):
    """One sequence alone and beside copies of itself that leave every SM many units: stages of 32 tokens that are full, ragged and
    more than two, chunks added up by the output pass (12 at most) and by the carry pass, units of a warp in chunks of unlike length, an odd
    number of units, records and dynamics formed in place."""
    import cdssm_b200
    lib = cdssm_b200._lib.lib()
    dt = 1 if dtype == torch.float32 else 0
    inp = unnormalise(orc.make_inputs(1, H, L, D, N=N, seed=L + N, context_length=max(L, 2)), np.random.default_rng(L))
    h0 = np.random.default_rng(N).standard_normal((1, H, N, D)).astype(np.float32) * 0.3
    one = [to_dev(inp[n], dtype) for n in ("q", "k", "v", "gate_raw")]
    both = [to_dev(inp[n], torch.float32) for n in ("log_dt_scale", "rope_freqs")]
    state = to_dev(h0, torch.float32)
    copies = 148 * 20 // (-(-L // C) * H * (N // 2)) + 1
    got = []
    for B in (1, copies):
        wide = lambda x: x.expand(B, *x.shape[1:]).contiguous()
        dims = (B, L, H, D, N, C)
        outs = [torch.full((B, L, H, N), 3.0, device="cuda", dtype=dtype), torch.full((B, H, N, D), 3.0, device="cuda"),
                torch.full((B, H, N, D), 3.0, device="cuda")]
        room = None
        if not records:   # (what a call cannot do without)
            room = lib.cdssm_b200_scan_fused_workspace_bytes(B, L, H, D, N, C)
            units = B * -(-L // C) * H * (N // 2)
            if room >= 256 + 8 * units * (1 + D) + B * -(-L // C) * H * C * (16 * (N // 2) + 8):
                pytest.skip("the least scratch has room for the records")
        _call(lib, [wide(x) for x in one] + both + [wide(state)], outs, const_args(inp["consts"]), dims, dt, room=room)
        got.append(outs)
    for few, many in zip(*got):
        assert torch.equal(few[0], many[0]) and torch.equal(few[0], many[-1])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,segments,NC,D,N", [(2, 3, 2, 64, 4), (1, 2, 13, 64, 2), (2, 4, 1, 128, 2)])
@pytest.mark.parametrize("decay", [0, 4096])
def test_segments_of_few_units_have_the_bits_of_many(ops, orc, dtype, H, segments, NC, D, N, decay):
    """Summaries, and scans on the local results that they have left, with positions by segment and with decays in float32: the walk for few
    units, the one whose rows travel ahead, and the one of many."""
    L = segments * NC * D
    inp = unnormalise(orc.make_inputs(1, H, L, D, N=N, seed=L + N, context_length=L), np.random.default_rng(L))
    one = [to_dev(inp[n], dtype) for n in ("q", "k", "v", "gate_raw")]
    both = [to_dev(inp[n], torch.float32) for n in ("log_dt_scale", "rope_freqs")]
    state = to_dev(np.random.default_rng(N).standard_normal((1, H, N, D)).astype(np.float32) * 0.3, torch.float32)
    units = segments * NC * H * (N // 2)
    got = []
    for B in (1, 1500 // units, 148 * 20 // units + 1):
        wide = lambda x: x.expand(B, *x.shape[1:]).contiguous()
        got.append(ops.scan_fused_long(*[wide(x) for x in one], *both, *const_args(inp["consts"]), H, N, D, wide(state), segments=segments,
                                       shortcut_scale=0.25, pos0=5, flags=ops.FORCE_SIMT | decay))
    for few, ring, many in zip(*got):
        for x in (ring, many):
            assert torch.equal(few[0], x[0]) and torch.equal(few[0], x[-1])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_nothing_is_written_beside_the_outputs(ops, orc, dtype):
    import cdssm_b200
    lib = cdssm_b200._lib.lib()
    B, H, L, D, N, C = 1, 3, 100, 64, 6, 64
    es, dt = (4, 1) if dtype == torch.float32 else (2, 0)
    inp = orc.make_inputs(B, H, L, D, N=N, seed=4, context_length=L)
    t = [to_dev(inp[n], dtype) for n in ("q", "k", "v", "gate_raw")] + [to_dev(inp[n], torch.float32) for n in ("log_dt_scale", "rope_freqs")]
    sizes = [B * L * H * N, B * H * N * D, B * H * N * D]
    bufs = [torch.full((n + 9,), 7.0, device="cuda", dtype=d) for n, d in zip(sizes, (dtype, torch.float32, torch.float32))]
    _call(lib, t + [None], [b[5:] for b in bufs], const_args(inp["consts"]), (B, L, H, D, N, C), dt)   # (aligned to a value only)
    want = [torch.empty_like(b[5:5 + n]) for b, n in zip(bufs, sizes)]
    _call(lib, t + [None], want, const_args(inp["consts"]), (B, L, H, D, N, C), dt)
    for b, n, w in zip(bufs, sizes, want):
        assert bool((b[:5] == 7).all()) and bool((b[5 + n:] == 7).all()) and torch.equal(b[5:5 + n], w)


@pytest.mark.parametrize("dtype,H,L,D,N,flags,little", [
    (torch.float32, 3, 50, 64, 2, 0, False), (torch.float32, 4, 128, 64, 6, 0, False), (torch.float32, 2, 64 * 12, 64, 2, 0, False),
    (torch.float32, 2, 300, 128, 2, 0, False), (torch.bfloat16, 2, 500, 64, 4, 1, False),
    (torch.bfloat16, 8, 300, 64, 2, 0, False), (torch.bfloat16, 3, 300, 128, 2, 0, False),    # N = 2 on the tensor cores
    (torch.bfloat16, 3, 300, 64, 8, 0, True), (torch.bfloat16, 2, 300, 128, 4, 0, True),      # whole chunks, two kernels
    (torch.bfloat16, 6, 500, 64, 16, 0, False)])                                              # and one
@pytest.mark.parametrize("which", [1, 2])
def test_states_may_take_the_place_of_h0(ops, orc, dtype, H, L, D, N, flags, little, which):
    """final_state or tail_state in h0's buffer: no block reads what another has written over, whoever adds the carry up."""
    import cdssm_b200
    lib = cdssm_b200._lib.lib()
    B, dt = 2, 1 if dtype == torch.float32 else 0
    inp = unnormalise(orc.make_inputs(B, H, L, D, N=N, seed=L + N, context_length=L), np.random.default_rng(L))
    state = to_dev(np.random.default_rng(N).standard_normal((B, H, N, D)).astype(np.float32) * 0.3, torch.float32)
    t = [to_dev(inp[n], dtype) for n in ("q", "k", "v", "gate_raw")] + [to_dev(inp[n], torch.float32) for n in ("log_dt_scale", "rope_freqs")]
    room = lib.cdssm_b200_scan_fused_workspace_bytes_for(B, L, H, D, N, D, dt, flags)
    room -= B * -(-L // D) * H * (N // 2) * D * 8 if little else 0   # (words that hand the carry on)
    outs = lambda: [torch.full((B, L, H, N), 3.0, device="cuda", dtype=dtype)] + [torch.full((B, H, N, D), 3.0, device="cuda") for _ in range(2)]
    want = outs()
    _call(lib, t + [state], want, const_args(inp["consts"]), (B, L, H, D, N, D), dt, room=room, flags=flags)
    for _ in range(10):
        got = outs()
        got[which] = state.clone()
        _call(lib, t + [got[which]], got, const_args(inp["consts"]), (B, L, H, D, N, D), dt, room=room, flags=flags)
        for w, g in zip(want, got):
            assert torch.equal(w, g)
