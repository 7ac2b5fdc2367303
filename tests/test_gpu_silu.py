"""silu(gate) * up over every bf16 gate there is, the strongly negative ones among them."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _gates(device):
    return torch.arange(-32768, 32768, dtype=torch.int32, device=device).to(torch.int16).view(torch.bfloat16)


@pytest.mark.parametrize("up", [1.0, -0.7734375, 3.0e38, 2.0 ** -120])
def test_silu_mul_over_all_gates(capi, device, up):
    """The two roundings of F.silu(gate) * up on bf16 tensors; torch's silu divides in fp32 as the kernel's expression does."""
    gate = _gates(device).view(64, 1024)
    ups = torch.full_like(gate, up)
    got, want = capi.silu_mul(gate, ups), torch.nn.functional.silu(gate) * ups
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    assert torch.equal(got.nan_to_num(7.0), want.nan_to_num(7.0))
    finite = torch.isfinite(gate)
    exact = gate.double() / (1.0 + torch.exp(-gate.double()))
    silu = capi.silu_mul(gate, torch.ones_like(gate)).double()
    # fp32: exp overflows below about -88.7, where the result is under 3e-37 in size; elsewhere half a unit of the last place of bf16
    # (2^-8) and the errors of fp32, 2^-21
    assert bool(((silu - exact).abs()[finite] <= (2.0 ** -8 + 2.0 ** -21) * exact.abs()[finite] + torch.where(gate.double()[finite] < -88.0, 3e-37, 1e-40)).all())
