"""The tcgen05 attention kernels against 64-bit attention at the sizes where their tiling can go wrong: one row, tile
edges, remainders, key tiles shared by several CTAs, many tiles per CTA, with and without the causal mask."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

# Three roundings to bf16 lie between the operands and a result (P or dS, and the stored value; delta sees the rounded
# output): up to 2^-8 each and 2^-8 / sqrt(3) in the mean square at most, 7e-3 in all if those add up.
TOLERANCE = 1e-2


def _error(x, ref, floor):
    return ((x.double() - ref).norm() / max(ref.norm().item(), floor)).item()


@pytest.mark.parametrize("B,T,H,KV,D,causal", [
    (1, 1, 2, 2, 64, True), (2, 127, 3, 3, 64, True), (1, 128, 2, 1, 128, True), (3, 129, 3, 1, 64, True),
    (2, 255, 6, 2, 128, True), (1, 257, 4, 4, 64, True), (1, 513, 8, 8, 128, True), (2, 777, 12, 12, 64, True),
    (1, 1536, 4, 1, 64, True), (1, 2048, 32, 8, 64, True), (5, 640, 25, 25, 64, True), (1, 4097, 8, 2, 128, True),
    (2, 129, 2, 2, 64, False), (1, 384, 4, 2, 128, False), (1, 1000, 3, 1, 64, False)])
def test_attention_against_64_bits(B, T, H, KV, D, causal):
    from infinitrain_b200 import _ext

    C = _ext.load(required=True)
    torch.manual_seed(B * T + H)
    # scores with a spread of several units: the running maximum moves
    qkv = (1.5 * torch.randn(B, T, H + 2 * KV, D, device="cuda")).bfloat16()
    q, k, v = qkv.split((H, KV, KV), dim=2)
    scale = 1.0 / math.sqrt(D)
    o, lse = C.flash_attn_fwd(q, k, v, scale, causal)
    dout = torch.randn_like(o)
    dqkv = torch.full_like(qkv, float("nan"))
    C.flash_attn_bwd(dout, q, k, v, o, lse, *dqkv.split((H, KV, KV), dim=2), scale, causal)
    torch.cuda.synchronize()
    assert C.kernel_status() == 0

    hidden = torch.ones(T, T, device="cuda", dtype=torch.bool).triu(1) if causal else None
    for b in range(B):
        for g in range(KV):
            heads = slice(g * (H // KV), (g + 1) * (H // KV))
            qr, kr, vr = (t.double().requires_grad_() for t in (q[b, :, heads], k[b, :, g], v[b, :, g]))
            s = torch.einsum("thd,sd->hts", qr, kr) * scale
            if causal:
                s = s.masked_fill(hidden, float("-inf"))
            ref = torch.einsum("hts,sd->thd", s.softmax(-1), vr)
            ref.backward(dout[b, :, heads].double())
            assert (lse[b, heads].double() - s.logsumexp(-1)).abs().max() < 1e-4
            assert _error(o[b, :, heads], ref, 0) < TOLERANCE
            floor = 1e-2 * dout[b, :, heads].double().norm().item()     # of one row dQ and dK are zero
            assert _error(dqkv[b, :, heads], qr.grad, floor) < TOLERANCE
            assert _error(dqkv[b, :, H + g], kr.grad, floor) < TOLERANCE
            assert _error(dqkv[b, :, H + KV + g], vr.grad, 0) < TOLERANCE


def _attend(q, k, v, scale, causal):
    """Output and log-sum-exp in 64 bits, as many KV heads as query heads."""
    s = torch.einsum("bthd,bshd->bhts", q.double(), k.double()) * scale
    if causal:
        T = s.shape[-1]
        s = s.masked_fill(torch.ones(T, T, device="cuda", dtype=torch.bool).triu(1), float("-inf"))
    return torch.einsum("bhts,bshd->bthd", s.softmax(-1), v.double()), s.logsumexp(-1)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("growth", [24, 2, -24])
def test_maximum_that_moves_with_the_keys(D, growth):
    """Every row's maximum grows with each key tile (by 12 to 17 powers of two, by one), or never after the first."""
    from infinitrain_b200 import _ext

    C = _ext.load(required=True)
    torch.manual_seed(D + growth)
    q, k, v = torch.randn(3, 2, 700, 2, D, device="cuda").bfloat16()
    q[..., 0] = 4
    k[..., 0] = (growth * (torch.arange(700, device="cuda") // 128)).bfloat16()[None, :, None]
    scale = 1.0 / math.sqrt(D)
    o, lse = C.flash_attn_fwd(q, k, v, scale, True)
    ref, ref_lse = _attend(q, k, v, scale, True)
    assert C.kernel_status() == 0
    assert (lse.double() - ref_lse).abs().max() < 1e-4
    assert ((o.double() - ref).norm(dim=-1) / ref.norm(dim=-1)).max() < TOLERANCE


def test_probabilities_are_relative_to_the_maximum_so_far():
    """Two keys count, one in each key tile; the first one's value is zero.  Relative to the row's maximum the second
    one's probability is 1 and needs no rounding, so the output is off by its own rounding alone."""
    from infinitrain_b200 import _ext

    C = _ext.load(required=True)
    torch.manual_seed(0)
    H, D = 64, 64
    q, k, v = torch.zeros(3, 1, 256, H, D, device="cuda").bfloat16()
    q[..., 0] = 1
    k[..., 0] = -256                                        # 2^-46 of the first key
    k[:, 0, :, 0] = 0
    k[:, 200, :, 0] = (40 * torch.rand(H, device="cuda")).bfloat16()        # up to 2^7 times the first key
    v[:, 128:] = torch.randn(1, 128, H, D, device="cuda").bfloat16()
    o, _ = C.flash_attn_fwd(q, k, v, 0.125, False)
    ref, _ = _attend(q, k, v, 0.125, False)
    # half a unit in the last place of bf16, and what fp32 leaves: exponents to 2^-21, exp2 and the sum to 2^-22
    unit = torch.ldexp(torch.ones_like(ref), torch.frexp(ref).exponent - 8)
    assert ((o.double() - ref).abs() <= 0.5 * unit + 2.0 ** -19 * ref.abs() + 1e-9).all()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("scale", [0.0, -0.05])
def test_masked_keys_stay_hidden_whatever_the_scale(D, scale):
    from infinitrain_b200 import _ext

    C = _ext.load(required=True)
    torch.manual_seed(D)
    q, k, v = torch.randn(3, 2, 300, 2, D, device="cuda").bfloat16()
    for causal in (True, False):                            # the diagonal tile, the ragged last one
        o, lse = C.flash_attn_fwd(q, k, v, scale, causal)
        ref, ref_lse = _attend(q, k, v, scale, causal)
        assert C.kernel_status() == 0
        assert (lse.double() - ref_lse).abs().max() < 1e-4
        assert ((o.double() - ref).norm(dim=-1) / ref.norm(dim=-1)).max() < TOLERANCE
