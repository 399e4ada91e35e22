"""The small-batch decode kernels against the library-product path of the same model (taken above 128 sequences at these widths)."""
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
