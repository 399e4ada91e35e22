"""The small-batch decode kernels against the library-product path of the same model (taken above 128 sequences at these widths)."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

WIDE = 130   # more sequences than the small-batch kernels take


@pytest.mark.parametrize("d_model,state_dim,batches", [
    (256, 2, (1, 8, 9, 65, 128)),      # groups of 16 channels, K = 16 in the read-out, two batch tiles
    (512, 4, (2, 16, 33)),             # groups of 32
    (768, 16, (5, 17, 85)),            # groups of 48
    (1024, 2, (3, 32)),                # groups of 64
])
def test_small_batch_decode_equals_library_products(ops, d_model, state_dim, batches):
    """Two steps of every batch size against the same rows of a 130-sequence step.  Both round activations to bf16 at the
    same places and differ in the order of 32-bit sums only: a value off by one bf16 ulp (2^-8) in a hidden activation of
    two layers moves logits and states by a few 1e-3 of their largest value; 2e-2 is the model-level bound used elsewhere."""
    from cdssm_b200.model import CdssmConfig, CdssmLM
    cfg = CdssmConfig(d_model=d_model, n_layers=2, context_length=256, vocab_size=1003, state_dim=state_dim)
    lm = CdssmLM(cfg, device="cuda", dtype=torch.bfloat16, seed=3)
    for i, p in enumerate(lm.blocks):
        p.shortcut_scale = 0.3
        p.D = torch.full_like(p.D, 0.1)
        p.v_residual_gate += 0.5 * i
    lib = ops._lib.lib()
    assert lib.cdssm_b200_lm_decode_workspace_bytes(WIDE, d_model, state_dim, 32, 1003, 0) == 0
    g = torch.Generator().manual_seed(1)
    ids = torch.randint(0, 1003, (WIDE, 21), generator=g).cuda()
    tok = torch.randint(0, 1003, (2, WIDE), generator=g).cuda()
    _, wide = lm.prefill(ids)
    copy = lambda n: {"pos": wide["pos"], "layers": [{k: t[:n].clone() for k, t in c.items()} for c in wide["layers"]]}
    caches = {n: copy(n) for n in batches}
    want = [lm.decode(t, wide).float() for t in tok]
    for n, cache in caches.items():
        assert lib.cdssm_b200_lm_decode_workspace_bytes(n, d_model, state_dim, 32, 1003, 0) > 0
        for t, w in zip(tok, want):
            got = lm.decode(t[:n], cache).float()
            assert (got - w[:n]).abs().max() <= 2e-2 * w.abs().max()
        for c, w in zip(cache["layers"], wide["layers"]):
            for k in ("state", "conv"):
                a, b = c[k].float(), w[k][:n].float()
                assert (a - b).abs().max() <= 2e-2 * b.abs().max(), k
        assert cache["pos"] == wide["pos"]


class _Layer(ctypes.Structure):   # cdssm_lm_layer
    _fields_ = ([(n, ctypes.c_void_p) for n in ("norm_w", "w_in", "b_in", "conv_w", "conv_b", "w_qg", "b_qg", "log_dt_scale", "rope_freqs",
                                                "mix", "w_readout", "gn_w", "gn_b", "skip", "w_out")] +
                [("shortcut_scale", ctypes.c_float), ("state", ctypes.c_void_p), ("conv", ctypes.c_void_p)])


def test_step_sees_weights_written_by_the_kernel_before_it(ops):
    """Through the C ABI nothing stands between the caller's last kernel and the step: a one-token scan step, which lets
    its successor start at once, writes the first layer's input bias."""
    from cdssm_b200.model import CdssmConfig, CdssmLM
    cfg = CdssmConfig(d_model=256, n_layers=2, context_length=256, vocab_size=1000, state_dim=2)
    lm = CdssmLM(cfg, device="cuda", dtype=torch.bfloat16, seed=3)
    lib, H, N, B = ops._lib.lib(), cfg.n_heads, 2, 4
    bias = lm.blocks[0].b_in                                          # 1552 values: y of 97 x (8, 2)
    rows = bias.numel() // (H * N)
    rnd = lambda *s: torch.randn(*s, device="cuda").bfloat16()
    q, k, v, g = rnd(rows, H, 64), rnd(rows, H, 64), rnd(rows, H, N), rnd(rows, (N + 5) * H)
    lds, rope = torch.zeros(H, device="cuda"), torch.full((H,), 0.1, device="cuda")
    mix = torch.full((2, H), 0.5, device="cuda", dtype=torch.bfloat16)
    need = lib.cdssm_b200_lm_decode_workspace_bytes(B, 256, N, cfg.ssm_norm_groups, 1000, 0)
    x0 = rnd(B, 256)
    stream = torch.cuda.current_stream().cuda_stream

    def step(apart):
        bias.zero_()
        states = [torch.zeros(B, H, N, 64, device="cuda") for _ in range(2)]
        convs = [torch.zeros(B, 3, 512, device="cuda", dtype=torch.bfloat16) for _ in range(2)]
        ws, x, logits = torch.empty(need + 256, dtype=torch.uint8, device="cuda"), x0.clone(), rnd(B, 1000)
        layers = (_Layer * 2)(*[_Layer(*[t.data_ptr() for t in (p.norm_w, p.w_in, p.b_in, p.conv_w, p.conv_b, p.w_qg, p.b_qg,
                                                                  p.log_dt_scale, p.rope_freqs, mix, p.w_readout, p.gn_w, p.gn_b,
                                                                  p.D, p.w_out)], 0.2, s.data_ptr(), c.data_ptr())
                                for p, s, c in zip(lm.blocks, states, convs)])
        state = torch.ones(rows, H, N, 64, device="cuda")
        torch.cuda.synchronize()
        ops.decode_step(state, q, k, v, g, lds, rope, *cfg.dyn_consts, H, N, 5, out=bias[:rows * H * N].view(rows, H, N))
        if apart:
            torch.cuda.synchronize()
        rc = lib.cdssm_b200_lm_decode(ctypes.addressof(layers), 2, x.data_ptr(), lm.final_norm_w.data_ptr(), lm.embedding.data_ptr(),
                                      logits.data_ptr(), ws.data_ptr() + (-ws.data_ptr()) % 256, need, cfg.eps_norm, 1e-5, 2.0 ** -14,
                                      *cfg.dyn_consts, B, 256, N, cfg.ssm_norm_groups, 1000, 3, None, 0, stream)
        assert rc == 0
        torch.cuda.synchronize()
        return [logits, x] + states + convs

    want = step(True)
    assert float(bias.float().abs().max()) > 0.05
    for _ in range(20):
        assert all(torch.equal(a, b) for a, b in zip(step(False), want))
