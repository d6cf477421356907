"""Products of fp32 rows in three bf16 parts (steps of 512 tokens and more, up to 128 columns), the selective scan's step sizes, with inner sizes at and beside
the parts' 64 columns and the line, against the fp64 restatements within the bounds of the other bf16 tests; and the parts and the product by
themselves, which a whole bf16 model says nothing about."""
import pytest
import torch

from oracle import kinetar_plain
from tests import hybrid_helpers as kin
from tests.row_ops import RowOps

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rank,inner", [(1, 40), (64, 300), (65, 24), (128, 40), (130, 256)])
def test_step_sizes(rank, inner):
    layer = kin.attn_scan(left_scale=0.0, inner=inner, state=16, dt_rank=rank)
    layer["mlp"] = None
    cfg = kin.model_config([layer])
    w = kinetar_plain.random_weights(cfg, 0, 8)
    toks = kin.rand_tokens(515, cfg["vocab"], 3)
    hz = kin.Harness(cfg, w, "bfloat16", num_pages=80, max_step_tokens=640)
    try:
        got = hz.feed("a", toks, [515])
    finally:
        hz.close()
    assert kin.rel_err(got, kin.oracle_logits(cfg, w, toks)) < kin.TOL["bfloat16"]


@pytest.fixture(scope="module")
def ops():
    return RowOps()


@pytest.mark.parametrize("cols", [1, 63, 128])
def test_parts_are_the_whole_number(ops, cols):
    """Every finite fp32 number whose lowest bits a bf16 number can hold is the sum of its parts exactly; what is no number, and infinities, stand in the
    upper part alone."""
    g = torch.Generator(device="cuda").manual_seed(cols)
    a = torch.randn(600, cols, generator=g, device="cuda") * 2.0 ** torch.randint(-90, 120, (600, cols), generator=g, device="cuda").float()
    a[0], a[1], a[2] = float("inf"), -float("inf"), float("nan")
    a[3], a[4], a[5] = 0.0, -0.0, torch.finfo(torch.float32).max
    parts = ops.split_rows(a)
    assert (parts[:, :, cols:] == 0).all()
    low, mid, up = parts[:, :, :cols].to(torch.float64).unbind(1)
    assert torch.equal(low[3:] + mid[3:] + up[3:], a[3:].to(torch.float64))
    assert torch.equal(up[:2], a[:2].to(torch.float64)) and up[2].isnan().all() and (low[:3] == 0).all() and (mid[:3] == 0).all()


@pytest.mark.parametrize("rows,features,cols", [(512, 300, 128), (513, 128, 65), (700, 4096, 16)])
def test_three_parts_hold_fp32(ops, rows, features, cols):
    """A dropped lower part costs 2^-17 of an operand, about 4e-6 of the result's norm, a dropped middle one 2^-9.  The bound: sums of up to 3 x 128 / 16
    blocks, of which each cuts less than 2^-23 off a sum that grows to the result, root mean square of both."""
    g = torch.Generator(device="cuda").manual_seed(rows)
    a, w = torch.randn(rows, cols, generator=g, device="cuda"), torch.randn(features, cols, generator=g, device="cuda").bfloat16()
    want = a.to(torch.float64) @ w.to(torch.float64).T
    got = ops.split_product(a, w).to(torch.float64)
    assert (got - want).norm() < 24 ** 0.5 * 2.0 ** -23 * want.norm()
    # the upper parts cancel: columns in pairs that are equal but for their last 16 bits, with opposite weights; what is left is 2^-8 of the operands
    near = torch.round(a[:, ::2] * 2.0 ** 15) / 2.0 ** 15
    a[:, 1::2] = near[:, :a[:, 1::2].shape[1]] * (1.0 + 2.0 ** -11)
    a[:, ::2] = near
    w[:, 1::2] = -w[:, ::2][:, :w[:, 1::2].shape[1]]
    if cols % 2:
        a[:, -1] = 0.0
    want = a.to(torch.float64) @ w.to(torch.float64).T
    got = ops.split_product(a, w).to(torch.float64)
    whole = a.abs().to(torch.float64) @ w.abs().to(torch.float64).T
    assert (got - want).norm() < 24 ** 0.5 * 2.0 ** -23 * whole.norm() and want.norm() < 2.0 ** -10 * whole.norm()


def test_rows_without_numbers_stay_by_themselves(ops):
    g = torch.Generator(device="cuda").manual_seed(3)
    a, w = torch.randn(520, 64, generator=g, device="cuda"), (torch.rand(64, 64, generator=g, device="cuda") + 0.5).bfloat16()
    clean = ops.split_product(a, w)
    a[7, 5], a[300, 63], a[519, 0] = float("nan"), float("inf"), -float("inf")
    got = ops.split_product(a, w)
    assert got[7].isnan().all() and (got[300] == float("inf")).all() and (got[519] == -float("inf")).all()
    rest = torch.ones(520, dtype=torch.bool)
    rest[[7, 300, 519]] = False
    assert torch.equal(got[rest], clean[rest])
