"""Recurrences whose value columns are spread over blocks, at the edges of their layouts: key sizes at and beside the padded sizes,
value columns that fill a block's eight, miss one or need another block, portions that end at, before and behind a staged
batch, and the size behind which another kernel takes over; the selective scan's lane layouts and the short convolution's
chunks; fp32 build against the plain fp64 restatements, within the
bound of the other fp32 tests (3e-4)."""
import math

import pytest
import torch

from oracle import famepel_plain, kinetar_plain, kisadra_plain, mafalorn_plain
from tests import famepel_helpers as fam
from tests import hybrid_helpers as kin
from tests import kisadra_helpers as kis
from tests import mafalorn_helpers as maf
from tests.row_ops import RowOps

pytestmark = pytest.mark.gpu

CUTS = [31, 1, 33, 2, 32, 8, 64]                               # staged batches hold 32 tokens (16 or fewer at large key sizes)


def _kinetar(layer, cuts=CUTS, width=48, dtype="float32"):
    cfg = kin.model_config([layer], width=width)
    toks = kin.rand_tokens(sum(cuts), cfg["vocab"], 3)
    w = kinetar_plain.random_weights(cfg, 0, 8)
    hz = kin.Harness(cfg, w, dtype=dtype, low=8)
    try:
        got = hz.feed("a", toks, cuts)
    finally:
        hz.close()
    return kin.rel_err(got, kin.oracle_logits(cfg, w, toks))


@pytest.mark.parametrize("dim,vdim,heads,kv", [(16, 8, 4, 2), (17, 7, 2, 1), (32, 9, 2, 2), (33, 1, 3, 1), (64, 16, 1, 1), (128, 24, 2, 1),
                                               (130, 12, 2, 1), (257, 8, 1, 1), (600, 10, 1, 1)])
def test_channel_delta_columns(dim, vdim, heads, kv):
    assert _kinetar(kin.delta(heads=heads, kv_heads=kv, dim=dim, vdim=vdim, ff=0)) < kin.TOL["float32"]


def test_channel_delta_many_wide_key_heads():
    assert _kinetar(kin.delta(heads=52, kv_heads=26, dim=1000, vdim=4, ff=0), cuts=[5, 1, 3], width=16) < kin.TOL["float32"]


@pytest.mark.parametrize("state,inner,rank", [(1, 40, 1), (4, 132, 4), (5, 128, 4), (8, 64, 3), (9, 66, 4), (16, 32, 4), (16, 35, 2), (17, 48, 1), (33, 20, 4),
                                              (65, 16, 2), (128, 12, 4), (129, 8, 4), (256, 5, 4)])
def test_selective_scan_layouts(state, inner, rank):
    """State sizes at and beside what one, two, ... thirty-two lanes hold; channels that fill a block, miss some or leave one over;
    sizes that allow 16-byte copies beside sizes that do not."""
    layer = kin.attn_scan(left_scale=0.0, inner=inner, state=state, dt_rank=rank)
    layer["mlp"] = None
    assert _kinetar(layer) < kin.TOL["float32"]


@pytest.mark.parametrize("conv,width", [(4, 48), (4, 44), (2, 48), (16, 48)])
@pytest.mark.parametrize("cuts", [[1, 2, 1, 15, 16, 17, 3], [33, 1, 48]])
def test_convolution_chunks(conv, width, cuts):
    """Portions shorter than the taps, ending at, before and behind a chunk of 16 tokens; four columns per thread or one."""
    layer = kin.attn_scan(dim=16, conv=conv, sconv=conv, inner=40 if width == 48 else 42)
    assert _kinetar(layer, cuts=cuts, width=width) < kin.TOL["float32"]


@pytest.mark.parametrize("state,vdim,heads,groups", [(1, 3, 2, 1), (10, 8, 4, 2), (16, 9, 2, 2), (33, 12, 4, 1), (64, 8, 2, 1), (128, 20, 2, 1), (130, 4, 1, 1),
                                                     (512, 4, 1, 1)])
def test_state_space_columns(state, vdim, heads, groups):
    cfg = fam.model_config([fam.ssd(heads=heads, vdim=vdim, state=state, groups=groups, norm_groups=1, conv=4, mlp=None)])
    toks = kin.rand_tokens(sum(CUTS), cfg["vocab"], 5)
    w = famepel_plain.random_weights(cfg, 0)
    hz = fam.Harness(cfg, w, "float32")
    try:
        got = hz.feed("a", toks, CUTS)
    finally:
        hz.close()
    assert kin.rel_err(got, fam.oracle_logits(cfg, w, toks)) < fam.TOL["float32"]


@pytest.mark.parametrize("dim,vdim", [(16, 8), (15, 7), (33, 9), (64, 1), (128, 40), (136, 8), (520, 3), (1030, 5)])
def test_forget_gate_columns(dim, vdim):
    cfg = fam.model_config([fam.glr(heads=2, dim=dim, vdim=vdim, mlp=None)])
    toks = kin.rand_tokens(sum(CUTS), cfg["vocab"], 4)
    w = famepel_plain.random_weights(cfg, 0)
    hz = fam.Harness(cfg, w, "float32")
    try:
        got = hz.feed("a", toks, CUTS)
    finally:
        hz.close()
    assert kin.rel_err(got, fam.oracle_logits(cfg, w, toks)) < fam.TOL["float32"]


@pytest.mark.parametrize("dim,vdim,heads", [(64, 120, 16), (100, 113, 16), (128, 8, 120), (33, 232, 8), (128, 15, 119)])
def test_two_columns_per_lane(dim, vdim, heads):
    """bf16 steps with enough heads x columns for two value columns per lane (15 columns x 119 heads stay just below): ragged last blocks and
    odd column counts, against the fp64 restatement within the bound of the other bf16 tests."""
    cfg = fam.model_config([fam.glr(heads=heads, dim=dim, vdim=vdim, mlp=None)])
    toks = kin.rand_tokens(sum(CUTS), cfg["vocab"], 4)
    w = famepel_plain.random_weights(cfg, 0)
    hz = fam.Harness(cfg, w, "bfloat16")
    try:
        got = hz.feed("a", toks, CUTS)
    finally:
        hz.close()
    assert kin.rel_err(got, fam.oracle_logits(cfg, w, toks)) < fam.TOL["bfloat16"]
    assert _kinetar(kin.delta(heads=heads, kv_heads=heads, dim=dim, vdim=vdim, ff=0), dtype="bfloat16") < kin.TOL["bfloat16"]


TWO = [(64, 120, 16), (100, 113, 16), (128, 8, 120), (34, 232, 8), (128, 15, 119), (36, 17, 60), (40, 16, 119)]


@pytest.mark.parametrize("dim,vdim,heads", TWO)
@pytest.mark.parametrize("mode", ["state space", "gated linear", "retention", "head delta"])
def test_two_columns_per_lane_in_the_other_modes(mode, dim, vdim, heads):
    """Heads x blocks of 16 columns at 120 and above (two value columns per lane) and just below, with ragged last blocks and odd column counts: the modes
    that have code of their own per column (step sizes and the skip of the state space, one decay per channel or per head, the delta rule's
    correction), bf16 against the fp64 restatement."""
    plain, helpers = (famepel_plain, fam) if mode == "state space" else (kisadra_plain, kis) if mode == "gated linear" else (mafalorn_plain, maf)
    if mode == "state space":
        cfg = fam.model_config([fam.ssd(heads=heads, vdim=vdim, state=dim, groups=1 if heads % 2 else 2, norm_groups=1, conv=4, mlp=None)])
    elif mode == "gated linear":
        cfg = kis.model_config([kis.gla(heads=heads, dim=dim, vdim=vdim, mlp=None)])
    elif mode == "retention":
        cfg = maf.model_config([maf.ret(heads=heads, dim=dim, vdim=vdim, decay=[1.0 - 2.0 ** (-2.0 - 5.0 * h / heads) for h in range(heads)], mlp=None)])
    else:
        cfg = maf.model_config([maf.par(d_heads=heads, d_kv_heads=heads if heads % 2 else heads // 2, d_dim=dim, d_vdim=vdim, conv=4, mlp=None)])
    toks = kin.rand_tokens(sum(CUTS), cfg["vocab"], 4)
    w = plain.random_weights(cfg, 0)
    hz = helpers.Harness(cfg, w, "bfloat16")
    try:
        got = hz.feed("a", toks, CUTS)
    finally:
        hz.close()
    assert helpers.close(got, helpers.oracle_logits(cfg, w, toks), "bfloat16")


@pytest.mark.parametrize("width,ff,tokens", [(48, 1630, 321), (45, 33, 70), (64, 64, 64), (31, 7, 33), (36, 100, 9)])
def test_fp32_product_tiles(width, ff, tokens):
    """The fp32 build's matrix products at the edges of their tiles of 32 and 64 rows and columns and of their k blocks of 32, with row
    starts that allow four k per load and ones that do not."""
    assert _kinetar(kin.delta(ff=ff), cuts=[tokens], width=width) < kin.TOL["float32"]


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_few_rows_many_columns(dtype):
    """Products of five to eight rows with more columns than four blocks per SM hold at eight a block: warps walk several columns."""
    assert _kinetar(kin.delta(ff=4999), cuts=[5, 8, 7, 6], dtype=dtype) < kin.TOL[dtype]


@pytest.mark.parametrize("low,high", [(1e-30, 1e-3), (1e-3, 1.0), (1.0, 40.0), (40.0, 87.0)])
def test_decays_of_the_selective_scan(low, high):
    """exp(dt a) against 64 bits: the exponential of the hardware is 2^-22 of itself away at most, and three roundings of 2^-24 of a factor near one follow."""
    g = torch.Generator(device="cuda").manual_seed(1)
    n = 1 << 20
    u = torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
    size = torch.exp(math.log(low) + u * math.log(high / low))
    dt = torch.exp(math.log(1e-5) + torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * math.log(1e7)).float()
    a = -(size / dt).float()
    dt, a = dt.repeat_interleave(2), torch.stack([a, a * 0.9], 1).flatten()
    want = torch.exp(dt.to(torch.float64) * a.to(torch.float64))
    got = RowOps().exp_rates(dt, a).to(torch.float64)
    assert ((got - want).abs() / want).max() < 2.0 ** -22 + 3 * 2.0 ** -24


def test_decays_of_the_selective_scan_at_their_ends():
    """Steps of nothing and of more than can be, rates of nothing and beyond counting, results below the smallest normal number, and what is no number."""
    inf, nan, big = float("inf"), float("nan"), torch.finfo(torch.float32).max
    dt = torch.tensor([0.0, 0.0, 1e18, 1e18, big, big, inf, inf, 1.0, 1.0, 1.0, 1.0, nan, nan], device="cuda")
    a = torch.tensor([-1.0, 0.0, -1e-3, -0.0, -1.0, 0.0, -1.0, 0.0, -inf, -1e30, -88.0, -104.0, -1.0, 0.0], device="cuda")
    got = RowOps().exp_rates(dt, a).tolist()
    assert got[:10] == [1.0, 1.0, 0.0, 1.0, 0.0, 1.0, 0.0, 1.0, 0.0, 0.0]
    assert all(0.0 <= g < 1.2e-38 for g in got[10:12]) and all(math.isnan(g) for g in got[12:])
