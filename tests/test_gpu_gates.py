"""Gates without a branch per element: the sigmoid against 64 bits, and SwiGLU's quotient against IEEE division over every bf16 gate."""
import math

import pytest
import torch

from tests.row_ops import RowOps

pytestmark = pytest.mark.gpu


def test_sigmoid_against_64_bits():
    """In parts of 2^-23, an ulp's largest share of a value: exp 2, the sum a half, the reciprocal a half and what Newton's step leaves of the
    approximation's error, its square."""
    z = torch.cat([torch.linspace(-80.0, 60.0, 1 << 20, device="cuda"), torch.randn(1 << 20, device="cuda")])
    got, want = RowOps().sigmoid(z).to(torch.float64), torch.sigmoid(z.to(torch.float64))
    assert float(((got - want) / want).abs().max()) < 3.01 * 2.0 ** -23


def test_sigmoid_at_its_ends():
    z = torch.tensor([0.0, -0.0, 88.0, 3.0e38, math.inf, -87.0, -88.5, -104.0, -3.0e38, -math.inf, math.nan], device="cuda")
    got = RowOps().sigmoid(z).tolist()
    assert got[:5] == [0.5, 0.5, 1.0, 1.0, 1.0] and got[7:10] == [0.0] * 3 and math.isnan(got[10])
    assert abs(got[5] / math.exp(-87.0) - 1.0) < 1e-5 and 0.0 <= got[6] <= 2.0 ** -126


def test_sigmoid_of_subnormal_values():
    """Between z = -87.3, where the value passes 2^-126, and -88.7, where exp(-z) is infinite: as exact as above, but for a step of 2^-149.  silu of
    these is a normal number."""
    z = torch.linspace(-88.7, -87.3, 1 << 16, device="cuda")
    got, want = RowOps().sigmoid(z).to(torch.float64), torch.sigmoid(z.to(torch.float64))
    assert bool(((got - want).abs() <= 3.01 * 2.0 ** -23 * want + 2.0 ** -149).all())
    silu = (z * got.float()).to(torch.float64)
    assert bool(((silu / (z.to(torch.float64) * want) - 1.0).abs() < 4.01 * 2.0 ** -23 + 2.0 ** -149 / want).all()) and float(silu.max()) < -2.0e-37


@pytest.mark.parametrize("up", [1.0, -3.140625, 2.0 ** -120, 3.0e38])
def test_swiglu_of_every_gate(up):
    gate = torch.arange(65536, dtype=torch.int32, device="cuda").to(torch.int16).view(torch.bfloat16).float()
    ups = torch.full_like(gate, up).to(torch.bfloat16).float()
    got, want = [RowOps().swiglu(gate, ups, divide).view(torch.int32) for divide in (False, True)]
    nan = torch.isnan(want.view(torch.float32))
    assert bool(((got == want) | nan & torch.isnan(got.view(torch.float32))).all())
