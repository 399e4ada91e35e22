"""Kernels that read column slices of wider projections in place: the conv with its history, the fused scan with the value
residual, and the LM's passes over a sequence built on them."""
import pytest
import torch
import torch.nn.functional as F

from util import const_args, rel_err, to_np

pytestmark = pytest.mark.gpu


def _p(t):
    return None if t is None else t.data_ptr()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("B,L,Dm,pad", [(2, 1, 64, 8), (3, 2, 52, 4), (2, 3, 256, 16), (1, 70, 51, 3), (2, 33, 64, 3), (1, 131, 1536, 8)])
def test_conv_strided_with_history(ops, dtype, B, L, Dm, pad):
    """Aligned rows, rows that no vector access fits (odd widths and odd strides), sequences shorter than the history: the bits
    of the dense call, and exactly the last three inputs."""
    g = torch.Generator(device="cuda").manual_seed(L + Dm)
    wide = torch.randn(B, L, Dm + pad, generator=g, device="cuda").to(dtype)
    x = wide[..., :Dm]
    w = (torch.randn(Dm, 4, generator=g, device="cuda") / 2).to(dtype)
    b = torch.randn(Dm, generator=g, device="cuda").to(dtype)
    out, hist = torch.empty(B, L, Dm, device="cuda", dtype=dtype), torch.full((B, 3, Dm), 7.0, device="cuda", dtype=dtype)
    rc = ops._lib.lib().cdssm_b200_conv1d_silu_strided_fwd(_p(x), Dm + pad, _p(w), _p(b), _p(out), _p(hist), B, L, Dm,
                                                           ops._DT[dtype], torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    want = ops.CUDAConv1dSiLUOp.apply(x, w.view(Dm, 1, 4), b)
    # two of the conv's forms may contract a * b + c in a different order: one rounding of the result
    ulp = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -22
    assert (out.float() - want.float()).abs().max() <= ulp * want.float().abs().max()
    assert torch.equal(hist, F.pad(x, (0, 0, 3, 0))[:, L:])


@pytest.mark.parametrize("B,H,L,D,N,flags,dtype", [
    (2, 4, 200, 64, 2, 0, torch.bfloat16),       # two chunks per product
    (1, 3, 130, 64, 2, 0, torch.bfloat16),       # odd head count: whole chunks
    (2, 6, 129, 64, 16, 0, torch.bfloat16), (1, 2, 300, 128, 4, 0, torch.bfloat16),
    (2, 4, 200, 64, 2, None, torch.bfloat16), (1, 3, 65, 64, 6, None, torch.bfloat16),   # None: the CUDA-core kernels
    (1, 3, 90, 64, 4, 0, torch.float32), (1, 2, 50, 40, 2, 0, torch.float32),
])
def test_scan_strided_with_value_residual(ops, orc, B, H, L, D, N, flags, dtype):
    """q, k, v and the gates as slices and the residual mixed in the kernel: the bits of dense copies and an eager lerp."""
    flags = ops.FORCE_SIMT if flags is None else flags
    C = D if D in (64, 128) else 32
    inp = orc.make_inputs(B, H, L, D, N=N, seed=L, bf16=True, context_length=max(L, 2))
    g = torch.Generator(device="cuda").manual_seed(L)
    G, HN, HD = (N + 5) * H, H * N, H * D
    r8 = lambda n: (n + 7) // 8 * 8
    dev = lambda a, n: torch.from_numpy(a).cuda().to(dtype).reshape(B, L, n)
    kv, kv0, qg = (torch.randn(B, L, n, generator=g, device="cuda").to(dtype) for n in (r8(HD + HN), HN + 8, r8(HD + G) + 8))
    kv[..., :HD], kv[..., HD:HD + HN] = dev(inp["k"], HD), dev(inp["v"], HN)
    qg[..., :HD], qg[..., HD:HD + G] = dev(inp["q"], HD), dev(inp["gate_raw"], G)
    k, v, v0, q, gate = kv[..., :HD], kv[..., HD:HD + HN], kv0[..., :HN], qg[..., :HD], qg[..., HD:HD + G]
    mix = torch.sigmoid(torch.randn(H, generator=g, device="cuda") * 2).to(dtype)
    lds, rf = (torch.from_numpy(inp[n]).cuda().float() for n in ("log_dt_scale", "rope_freqs"))
    consts = const_args(inp["consts"])
    y = torch.empty(B, L, H, N, device="cuda", dtype=dtype)
    tail = torch.empty(B, H, N, D, device="cuda")
    lib = ops._lib.lib()
    ws = torch.empty(lib.cdssm_b200_scan_fused_workspace_bytes(B, L, H, D, N, C), device="cuda", dtype=torch.uint8)
    rc = lib.cdssm_b200_scan_fused_strided_fwd(
        _p(q), q.stride(1), _p(k), k.stride(1), _p(v), v.stride(1), _p(v0), v0.stride(1), _p(mix), _p(gate), gate.stride(1),
        _p(lds), _p(rf), None, _p(y), None, _p(tail), _p(ws), ws.numel(), *consts, 0.4, B, L, H, D, N, C, 0, ops._DT[dtype],
        flags, torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    vm = torch.lerp(v0.reshape(B, L, H, N), v.reshape(B, L, H, N), mix.view(1, 1, H, 1))
    wy, _, wt = ops.scan_fused(q.reshape(B, L, H, D), k.reshape(B, L, H, D), vm, gate.contiguous(), lds, rf, *consts, H, N, C,
                               shortcut_scale=0.4, flags=flags, return_tail_state=True)
    assert torch.equal(y, wy) and torch.equal(tail, wt)


def _by_operators(ops, m, ids, cached):
    """The model's pass over a sequence, one public operator and one dense product at a time."""
    cfg, x, v_first, caches = m.cfg, m.embedding[ids], None, []
    B, L = ids.shape
    H, N, D, di = cfg.n_heads, cfg.state_dim, cfg.head_dim, cfg.d_inner
    consts = (cfg.gating_c, cfg.omega_thresh, cfg.adt_delta, cfg.adt_smoothness, cfg.adt_eps)
    for p in m.blocks:
        z, xg, k, v = F.linear(ops.rms_norm(x, p.norm_w, cfg.eps_norm), p.w_in, p.b_in).split([di, di, di, H * N], -1)
        v = v.reshape(B, L, H, N)
        if v_first is None:
            v_first = v
        else:
            v = torch.lerp(v_first, v, torch.sigmoid(p.v_residual_gate).to(v.dtype).view(1, 1, H, 1))
        xc = ops.CUDAConv1dSiLUOp.apply(xg, p.conv_w, p.conv_b)
        y, _, tail = ops.scan_fused(F.linear(xc, p.w_q).view(B, L, H, D), k.reshape(B, L, H, D), v, F.linear(xc, p.w_gate, p.b_gate),
                                    p.log_dt_scale, p.rope_freqs, *consts, H, N, cfg.chunk_size, shortcut_scale=p.shortcut_scale,
                                    flags=ops.FORCE_SIMT, return_tail_state=True)
        caches.append((tail, F.pad(xg, (0, 0, 3, 0))[:, L:]))
        o = ops.groupnorm_gate(F.linear(y.view(B, L, H * N), p.w_readout), p.gn_w, p.gn_b, z, p.D, xc, cfg.ssm_norm_groups,
                               1e-5, per_token=cached)
        x = x + F.linear(o, p.w_out)
    return F.linear(ops.rms_norm(x, m.final_norm_w, cfg.eps_norm), m.embedding), caches


@pytest.mark.parametrize("d_model,state_dim", [(256, 2), (512, 6)])
@pytest.mark.parametrize("B,L", [(1, 1), (3, 2), (2, 70), (2, 576), (1, 577)])   # the last two: both sides of the prompt rule
def test_lm_sequence_equals_operators(ops, d_model, state_dim, B, L):
    """bf16 at the same places, other kernels in the scan: 2e-2 is the model-level bound used elsewhere.  In a state meet k, v,
    the write gate and the decay, and where the scans' sums differ each of them may round to the next bf16, at most 2^-7 of the
    value, without averaging out in the largest element: 4 * 2^-7."""
    from cdssm_b200.model import CdssmConfig, CdssmLM
    m = CdssmLM(CdssmConfig(d_model=d_model, n_layers=2, context_length=256, vocab_size=503, state_dim=state_dim), device="cuda", seed=5)
    for i, p in enumerate(m.blocks):
        p.shortcut_scale = 0.3
        p.D = torch.full_like(p.D, 0.1)
        p.v_residual_gate += 0.5 * i
    ids = torch.randint(0, 503, (B, L), generator=torch.Generator().manual_seed(L)).cuda()
    for cached in (False, True):
        want, caches = _by_operators(ops, m, ids, cached)
        got, cache = m.prefill(ids, last_only=False) if cached else (m.forward(ids), None)
        assert rel_err(to_np(got), to_np(want)) <= 2e-2
        if cached:
            for c, (tail, conv) in zip(cache["layers"], caches):
                assert rel_err(to_np(c["state"]), to_np(tail)) <= 4 * 2.0 ** -7
                assert rel_err(to_np(c["conv"]), to_np(conv)) <= 2e-2


@pytest.mark.parametrize("B,L", [(1, 40), (4, 1100)])     # the kernels of short and of long inputs
def test_kernels_see_what_the_kernel_before_them_wrote(ops, orc, B, L):
    """They are launched while their predecessor drains: every input is rewritten right before the call, by a kernel that is
    still running then, and the result has the bits of a call on settled inputs."""
    H, D, N, di = 4, 64, 4, 512
    g = torch.Generator(device="cuda").manual_seed(L)
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    inp = orc.make_inputs(B, H, L, D, N=N, seed=1, bf16=True)
    lds, rf = (torch.from_numpy(inp[n]).cuda().float() for n in ("log_dt_scale", "rope_freqs"))
    calls = {
        "rms_norm": (lambda x, w: ops.rms_norm(x, w, 1e-5), [rn(B, L, di), rn(di)]),
        "conv": (lambda x, w, b: ops.CUDAConv1dSiLUOp.apply(x, w, b), [rn(B, L, di), rn(di, 1, 4), rn(di)]),
        "gate": (lambda y, w, b, z, s, x: ops.groupnorm_gate(y, w, b, z, s, x, 32), [rn(B, L, di), rn(di), rn(di), rn(B, L, di), rn(di), rn(B, L, di)]),
        "gate, token": (lambda y, w, b, z, s, x: ops.groupnorm_gate(y, w, b, z, s, x, 32, per_token=True),
                        [rn(B, L, di), rn(di), rn(di), rn(B, L, di), rn(di), rn(B, L, di)]),
        "scan": (lambda q, k, v, gate: ops.scan_fused(q, k, v, gate, lds, rf, *const_args(inp["consts"]), H, N, D)[0],
                 [rn(B, L, H, D), rn(B, L, H, D), rn(B, L, H, N), rn(B, L, (N + 5) * H)]),
    }
    busy = torch.randn(1 << 24, device="cuda")
    for name, (call, args) in calls.items():
        want = call(*args).clone()
        for late in range(len(args)):
            work = [a.clone() for a in args]
            work[late].zero_()
            torch.cuda.synchronize()
            busy.mul_(1.0)
            work[late].copy_(args[late])
            assert torch.equal(call(*work), want), (name, late)
