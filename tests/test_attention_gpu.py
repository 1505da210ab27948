"""The tcgen05 attention kernels against 64-bit attention at the sizes where their tiling can go wrong: one row, tile
edges, remainders, key tiles shared by several CTAs, many tiles per CTA, with and without the causal mask."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

# Three roundings to bf16 lie between the operands and a result (P or dS, and the stored value; delta sees the rounded
# output): unit roundoff 2^-9 each, 6e-3 in all if they add up.
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
