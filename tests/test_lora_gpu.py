"""LoRALinear where its two products and the base output run on the GPU kernels, against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# Up to six roundings to bf16 lie between the fp32 parameters and a result (operands, x A^T, its multiple, the base
# output, the sum): 2^-8 / sqrt(3) at most in the mean square each, and as independent errors they add up in squares.
TOLERANCE = 2.0 ** -8 * (6 / 3) ** 0.5


@pytest.mark.parametrize("tokens", [96, 5000])               # both sides of the line between small and large output tiles
@pytest.mark.parametrize("rank", [4, 8, 16])                 # 4: no multiple of 8, the second product is a plain one
def test_lora_linear_against_64_bits(rank, tokens):
    from infinitrain_b200 import _ext
    from infinitrain_b200.autocast import AutocastGuard
    from infinitrain_b200.datatype import DataType
    from infinitrain_b200.device import DeviceType
    from infinitrain_b200.nn import lora

    C = _ext.load(required=True)
    torch.manual_seed(rank)
    layer = lora.LoRALinear(256, 200, lora.LoRAConfig(rank=rank, alpha=20.0), device="cuda")      # factor 5, 2.5, 1.25
    with torch.no_grad():
        for p in (layer.weight, layer.bias, layer.lora_A, layer.lora_B):
            p.copy_(0.1 * torch.randn(p.shape, device="cuda"))
    x = torch.randn(2, tokens // 2, 256, device="cuda").bfloat16().requires_grad_()
    dout = torch.randn(2, tokens // 2, 200, device="cuda").bfloat16()
    with AutocastGuard(DeviceType.kCUDA, DataType.kBFLOAT16):
        y = layer(x)
    grads = torch.autograd.grad(y, (x, layer.lora_A, layer.lora_B), dout)
    assert C.kernel_status() == 0

    x64, w, b, a64, b64 = (t.detach().double().requires_grad_() for t in (x, layer.weight, layer.bias, layer.lora_A,
                                                                          layer.lora_B))
    F = torch.nn.functional
    ref = F.linear(x64, w, b) + 20.0 / rank * F.linear(F.linear(x64, a64), b64)
    refs = torch.autograd.grad(ref, (x64, a64, b64), dout.double())
    for got, want in zip((y, *grads), (ref, *refs)):
        assert ((got.double() - want).norm() / want.norm()).item() < TOLERANCE
