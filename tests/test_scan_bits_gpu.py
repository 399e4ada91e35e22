"""The order in which the tensor-core scans evaluate is kept: a product or a sum taken in another order moves a cached bf16 state of a
twelve-layer model by a percent, so it is a change that users see and not one that happens beside another."""
import zlib

import numpy as np
import pytest
import torch

from test_scan_gpu import run_fused
from util import const_args, to_dev

pytestmark = pytest.mark.gpu

# (H, L, D, N): CRC-32 of y and of the state after the last token.  Gates as a model meets them; "wild": decays that leave the range of a
# block's scaled unknowns, so that pairs of it are walked.
MODEL = {(8, 500, 64, 2): (3704699172, 2960037014), (4, 700, 128, 2): (1125811291, 434316177),
         (5, 381, 64, 4): (2027905606, 1066116165), (24, 1000, 64, 6): (2352845244, 254133680),
         (3, 381, 64, 8): (1354727775, 2107887923), (24, 1277, 64, 12): (1203873897, 415273592),
         (8, 523, 64, 16): (4094638131, 2880548728), (3, 765, 128, 4): (575050562, 3904660780),
         (12, 1000, 128, 6): (143255022, 802764237), (2, 765, 128, 8): (535030354, 2139756516),
         (24, 1500, 128, 16): (2966473696, 1151683306)}
WILD = {(8, 500, 64, 2): (1628976053, 3590081624), (4, 700, 128, 2): (4044209766, 648969707),
        (5, 381, 64, 4): (4013498383, 172472818), (24, 1000, 64, 6): (1437431076, 3742570834),
        (3, 381, 64, 8): (566478194, 676250229), (24, 1277, 64, 12): (3864467463, 195932802),
        (8, 523, 64, 16): (1137290871, 1282402986), (3, 765, 128, 4): (76320381, 709193589),
        (12, 1000, 128, 6): (784751710, 2207710518), (2, 765, 128, 8): (1275000913, 2199383906),
        (24, 1500, 128, 16): (2169433470, 2795242774)}

HUGE = {(5, 165, 64, 4): (566075848, 419627732), (3, 200, 64, 16): (2090349564, 2479583917), (2, 300, 128, 8): (605016733, 4188771241)}


def _inputs(H, L, D, N, wild):
    r = np.random.default_rng(H + L + D + N)
    normal = lambda *s: r.standard_normal(s).astype(np.float32)
    NH = N // 2
    bias = np.zeros((N + 5) * H, np.float32)
    bias[:NH * H] = (2.0 + 2.0 * normal(NH * H)) if wild else (-1.0 + 0.5 * normal(NH * H))
    bias[NH * H:2 * NH * H] = r.uniform(-np.pi, np.pi, NH * H)
    if wild:
        bias[(N + 2) * H:(N + 3) * H], bias[(N + 4) * H:] = 1.0, 3.0
    gates = normal(2, L, (N + 5) * H)
    gates[..., :2 * NH * H] *= 1.0 if wild else 0.1
    return dict(q=normal(2, L, H, D), k=normal(2, L, H, D), v=normal(2, L, H, N), gate_raw=gates + bias, log_dt_scale=0.5 * normal(H),
                rope_freqs=(2048.0 ** (-np.arange(H) / H)).astype(np.float32)), 0.1 * normal(2, H, N, D)


def bits(ops, orc, H, L, D, N, wild, huge=False):
    inp, h0 = _inputs(H, L, D, N, wild)
    if huge:   # (the real part; what is left of the imaginary one beside it is the last bit's)
        inp["v"][0, 29, :, 0] = inp["v"][1, L // 2, :, N - 2] = 3e19
    inp["consts"] = orc.derive_constants(2048)
    y, _, tail = run_fused(ops, inp, torch.bfloat16, N, D, h0=h0, pos0=4 * D, shortcut_scale=0.25, return_tail_state=True)
    return tuple(zlib.crc32(t.contiguous().view(torch.uint8).cpu().numpy().tobytes()) for t in (y, tail))


@pytest.mark.parametrize("H,L,D,N", list(MODEL))
@pytest.mark.parametrize("wild", [False, True])
def test_order_of_evaluation_is_kept(ops, orc, H, L, D, N, wild):
    assert bits(ops, orc, H, L, D, N, wild) == (WILD if wild else MODEL)[H, L, D, N]


@pytest.mark.parametrize("H,L,D,N", list(HUGE))
def test_order_of_evaluation_beside_a_huge_value(ops, orc, H, L, D, N):
    assert bits(ops, orc, H, L, D, N, False, True) == HUGE[H, L, D, N]


def _transition(g, lds, freq, pos, c, off_alpha=0.0, off_tau=0.0, off_ta=0.0, off_tw=0.0):
    """(.., 2): a of the gates (.., 7, H) alpha, omega, sel_B, sel_C, sel_dt, beta, r of one pair.  off: errors of alpha and tau, absolute, of ta and
    tw, relative."""
    softplus, sigmoid = lambda x: torch.nn.functional.softplus(x, threshold=40.0), torch.sigmoid
    w, alpha = g[:, 1] + pos * freq, softplus(g[:, 0]) + off_alpha
    raw, most = softplus(lds) / (alpha + w.abs() + c[4]), (2 - c[2]) / (alpha + c[4])
    blend = sigmoid((c[1] - w.abs()) / c[3])
    tau = 0.5 * (blend * torch.minimum(raw, most) + (1 - blend) * raw + softplus(g[:, 4])) + off_tau
    ta, tw = tau * alpha * (1 + off_ta), tau * w * (1 + off_tw)
    den = (1 + ta) ** 2 + tw ** 2 + 1e-6
    scale = (((1 - ta) ** 2 + tw ** 2) / den).clamp(min=1e-8) ** ((c[0] * sigmoid(g[:, 6]) - 1) / 2)
    return torch.stack([(1 - ta) * (1 + ta) - tw * tw, -2 * tw], -1) / den[..., None] * scale[..., None]


def _transition_of_scan(ops, g, lds, freq, pos, c, D, flags):
    """The transition in float32: a token with k = 0 and state 1 + 0i leaves a."""
    B, H, N = g.shape[0], g.shape[2], 2
    z = torch.zeros(B, 1, H, D, device="cuda", dtype=torch.bfloat16)
    h0 = torch.tensor([1.0, 0.0], device="cuda").view(1, 1, N, 1).expand(B, H, N, D).contiguous()
    return ops.scan_fused(z, z, z[..., :N].contiguous(), to_dev(g.reshape(B, 1, -1).float(), torch.bfloat16), to_dev(lds, torch.float32),
                          to_dev(freq, torch.float32), *c, H, N, D, h0, pos0=pos, return_tail_state=True,
                          flags=ops.FP32_DECAY | flags)[2][..., 0].double().cpu()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("pos", [200, 1000])
def test_angle_of_a_late_token_is_rounded_once(ops, D, pos):
    """N = 2: the angle omega + pos freq where the gate all but cancels the product, from the transition in float32 (a token with k = 0 and
    state 1 + 0i leaves a) against float64.  The bound: some eight results of the special-function unit, 2^-22 each.  With the product rounded
    on its own the angle is off by up to half an ulp of pos freq, and a by 6e-6 at position 1000."""
    B, H, N = 512, 8, 2
    c = tuple(float(np.float32(x)) for x in (np.log(2048.0), 2.0 ** -3.5, 0.125, 2.0 ** -3.5 / 5, 1.0))
    r = np.random.default_rng(D + pos)
    freq = torch.from_numpy(r.uniform(0.2, 0.9, H).astype(np.float32)).double()
    g = torch.from_numpy(r.standard_normal((B, N + 5, H))).bfloat16().double()   # alpha, omega, sel_B, sel_C, sel_dt, beta, r
    g[:, 1] = (-pos * freq * (1 + 2.0 ** -8 * torch.from_numpy(r.uniform(-1, 1, (B, H))))).bfloat16().double()
    lds = torch.from_numpy(r.standard_normal(H).astype(np.float32) * 0.5).double()
    want = _transition(g, lds, freq, pos, c)
    off = (_transition_of_scan(ops, g, lds, freq, pos, c, D, 0) - want).norm(dim=-1) / want.norm(dim=-1)
    assert float(off.median()) <= 8 * 2.0 ** -22


@pytest.mark.parametrize("simt", [0, 1])
@pytest.mark.parametrize("gating_c,smoothness", [(7.6, 0.018), (12.5, 0.018), (40.0, 1.0), (0.0, 1e-4)])
def test_transition_over_the_range_of_the_gates(ops, simt, gating_c, smoothness):
    """Exponentials, logarithms, powers and quotients of the special-function unit from -90 to 90, powers that are subnormal among them, against
    float64.  The bound: a softplus has an absolute error of 2^-22 (the logarithm near one), so alpha and tau have; ta and tw a relative one of 2^-20
    (four results in a row, 2^-22 each), the power and its factors as much again, a logarithm's error times the exponent included; a
    subnormal power has 2^-149."""
    B, H, N, D, pos = 2048, 8, 2, 64, 0
    c = tuple(float(np.float32(x)) for x in (gating_c, 2.0 ** -3.5, 0.125, smoothness, 1.0))   # (as the kernel has them)
    r = np.random.default_rng(int(gating_c) + simt)
    wide = lambda *s: r.uniform(-1, 1, s) * np.exp2(r.uniform(-8, 6.5, s))
    g = torch.from_numpy(wide(B, N + 5, H)).bfloat16().double()
    lds, freq = torch.from_numpy(r.uniform(-3, 20, H).astype(np.float32)).double(), torch.zeros(H).double()
    want = _transition(g, lds, freq, pos, c)
    u = 2.0 ** -20
    room = sum((_transition(g, lds, freq, pos, c, **{n: sign * by}) - want).norm(dim=-1) for n, by in
               (("off_alpha", u / 4), ("off_tau", u / 4), ("off_ta", u), ("off_tw", u)) for sign in (1, -1))
    power = (c[0] * torch.sigmoid(g[:, 6]) - 1).abs() / 2
    got = _transition_of_scan(ops, g, lds, freq, pos, c, D, simt)
    off = (got - want).norm(dim=-1)
    bound = room + want.norm(dim=-1) * u * (1 + power) + 2.0 ** -148
    assert bool((off <= bound).all()), float((off / bound).max())
