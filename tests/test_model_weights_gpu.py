"""The model's passes read the weights as they are at the time of the call: written in place, assigned, or with other `data`."""
import copy

import pytest
import torch

pytestmark = pytest.mark.gpu


def _model(dtype=torch.bfloat16, n_layers=2, d_model=256, state_dim=4):
    from cdssm_b200.model import CdssmConfig, CdssmLM
    cfg = CdssmConfig(d_model=d_model, n_layers=n_layers, context_length=1024, vocab_size=503, state_dim=state_dim)
    lm = CdssmLM(cfg, device="cuda", dtype=dtype, seed=5)
    for i, p in enumerate(lm.blocks):
        p.shortcut_scale = 0.3
        p.D = torch.full_like(p.D, 0.1)
        p.v_residual_gate += 0.5 * i
    return lm


def _fresh(lm):
    """A model of the same weights that has made no pass."""
    from cdssm_b200.model import CdssmLM
    new = CdssmLM(lm.cfg, device="cuda", dtype=lm.dtype, seed=0)
    new.embedding, new.final_norm_w = lm.embedding.clone(), lm.final_norm_w.clone()
    for a, b in zip(new.blocks, lm.blocks):
        for n in ("norm_w", "w_in", "b_in", "conv_w", "conv_b", "w_gate", "b_gate", "log_dt_scale", "rope_freqs", "w_q", "w_readout",
                  "w_out", "gn_w", "gn_b", "D", "v_residual_gate"):
            setattr(a, n, getattr(b, n).clone())
        a.shortcut_scale = b.shortcut_scale
        a.merge_q_and_gate_projections()
    return new


def _passes(lm, ids, tok):
    """Logits and cached states of a forward, a short and a long prompt, a small and a wide decode step."""
    out = [lm.forward(ids)]
    for L in (40, 600):
        logits, cache = lm.prefill(ids[:, :L])
        out += [logits] + [c["state"] for c in cache["layers"]]
    out.append(lm.decode(tok, cache))
    _, cache = lm.prefill(ids[:1, :20].expand(130, 20).contiguous())
    return out + [lm.decode(tok[:1].expand(130), cache)]


def _other(t, name):
    return t - 5.0 if name == "v_residual_gate" else t * 1.5 + 0.2      # (a gate of 0.5: sigmoid 0.62 -> 0.01)


def _assign(p, name):
    setattr(p, name, _other(getattr(p, name), name))


def _data(p, name):
    t = getattr(p, name)
    t.data = _other(t.detach(), name)


def _in_place(p, name):
    t = getattr(p, name)
    t.copy_(_other(t, name))


def _data_in_place(p, name):
    t = getattr(p, name)
    t.data.copy_(_other(t, name))


@pytest.mark.parametrize("change", [_assign, _data, _in_place, _data_in_place])
@pytest.mark.parametrize("name", ["w_q", "w_gate", "b_gate", "w_in", "b_in", "v_residual_gate"])
def test_changed_weights_are_used_by_every_pass(ops, name, change):
    lm = _model()
    g = torch.Generator().manual_seed(1)
    ids, tok = torch.randint(0, 503, (2, 600), generator=g).cuda(), torch.randint(0, 503, (2,), generator=g).cuda()
    before = _passes(lm, ids, tok)
    change(lm.blocks[1], name)
    got, want = _passes(lm, ids, tok), _passes(_fresh(lm), ids, tok)
    moved = 0
    for b, a, w in zip(before, got, want):
        b, a, w = b.float(), a.float(), w.float()
        assert (a - w).abs().max() <= 2e-2 * w.abs().max()      # one or two products: roundings of bf16 activations only
        moved += bool((b - w).abs().max() > 4e-2 * w.abs().max())
    assert moved >= 3


def test_graph_outlives_a_change_elsewhere(ops):
    """A captured decode step reads nothing that belongs to the layout of the model's weights at the time."""
    lm = _model(n_layers=3)
    g = torch.Generator().manual_seed(2)
    ids = torch.randint(0, 503, (2, 30), generator=g).cuda()
    _, cache = lm.prefill(ids)
    twin = copy.deepcopy(cache)
    graph, tok = lm.make_decode_graph(cache, 2)
    lm.blocks[0].shortcut_scale = 0.3                          # assigned, with the value it had
    lm.forward(ids)
    junk = [torch.full((3, lm.cfg.n_heads), 7.0, device="cuda", dtype=torch.bfloat16) for _ in range(64)]
    tok.copy_(ids[:, 0])
    graph.replay()
    want = lm.decode(ids[:, 0], twin).argmax(-1)
    assert torch.equal(tok, want) and len(junk) == 64
    for a, b in zip(cache["layers"], twin["layers"]):
        assert torch.equal(a["state"], b["state"]) and torch.equal(a["conv"], b["conv"])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_residual_mix_equals_the_eager_operation(ops, dtype):
    H, layers = 150, 70
    gates = [torch.randn(H, device="cuda") * 4 for _ in range(layers)]
    out = torch.empty(layers, H, device="cuda", dtype=dtype)
    import ctypes
    ptrs = (ctypes.c_void_p * layers)(*[t.data_ptr() for t in gates])
    rc = ops._lib.lib().cdssm_b200_residual_mix(ptrs, layers, H, out.data_ptr(), 0 if dtype == torch.bfloat16 else 1,
                                                torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    assert torch.equal(out, torch.stack([torch.sigmoid(t).to(dtype) for t in gates]))


def test_other_threads_run_during_a_pass(ops):
    """A native call does not hold the interpreter's lock while it launches a pass: another thread ticks inside it."""
    import threading
    import time
    lm = _model(n_layers=48)
    ids = torch.randint(0, 503, (1, 40), device="cuda")
    lm.forward(ids)
    ticks, stop = [], threading.Event()

    def tick():
        while not stop.is_set():
            ticks.append(time.perf_counter())
            time.sleep(0)

    t = threading.Thread(target=tick)
    t.start()
    spans = []
    for _ in range(20):
        t0 = time.perf_counter()
        lm.forward(ids)
        spans.append((t0, time.perf_counter()))
    stop.set()
    t.join()
    torch.cuda.synchronize()
    inside = [sum(a < x < b for x in ticks) for a, b in spans]
    assert sorted(inside)[len(inside) // 2] >= 5, inside      # (one may fall between the call and the clock)


@pytest.mark.parametrize("skip,reduced", [(8, True), (8, False), (1, False)])
def test_weights_at_any_address(ops, skip, reduced):
    """Weights 16 bytes off a 256-byte boundary (the library's products are chosen for the alignment they meet) and 2 bytes
    off (other products and kernels), and the program's setting for partial sums.  By 2-norm: single bf16 roundings that fall
    the other way move a state of 600 tokens by 1.5e-2 at most (12 layers; single elements by more)."""
    lm = _model()
    g = torch.Generator().manual_seed(4)
    ids, tok = torch.randint(0, 503, (2, 600), generator=g).cuda(), torch.randint(0, 503, (2,), generator=g).cuda()
    want = _passes(lm, ids, tok)
    for p in lm.blocks:
        for n in ("w_in", "b_in", "w_gate", "b_gate", "w_q", "w_readout", "w_out"):
            t = getattr(p, n)
            room = torch.zeros(t.numel() + 128, device="cuda", dtype=t.dtype)
            moved = room[skip:skip + t.numel()].view(t.shape)
            moved.copy_(t)
            setattr(p, n, moved)
    old = torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction
    torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction = reduced
    try:
        got = _passes(lm, ids, tok)
    finally:
        torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction = old
    for a, w in zip(got, want):
        a, w = a.float(), w.float()
        assert (a - w).norm() <= 2e-2 * w.norm()


def test_used_model_can_be_copied_and_saved(ops, tmp_path):
    """After a pass too, and a model saved before the native path existed has neither plan nor version."""
    lm = _model()
    ids = torch.randint(0, 503, (2, 40), device="cuda")
    want = lm.forward(ids)
    torch.save(lm, tmp_path / "lm.pt")
    for other in (copy.deepcopy(lm), torch.load(tmp_path / "lm.pt", weights_only=False)):
        assert torch.equal(other.forward(ids), want)
        for p in other.blocks:
            p.__dict__.pop("version", None)
        other.__dict__.pop("_plan")
        assert torch.equal(other.forward(ids), want)
        other.blocks[0].w_in.zero_()
        assert not torch.equal(other.forward(ids), want) and torch.equal(lm.forward(ids), want)
