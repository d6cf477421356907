"""bf16 products of one to eight rows on the tensor cores: features beside the tiles of 16, k beside the blocks of 32 and beside what a batch or a split
holds, sizes that keep the other kernel, and the routed form (experts without a row, experts that every token chose, gated and plain), against the
fp64 restatements within the bounds of the other bf16 tests.  Tokens whose router scores do not compare, beside healthy ones.
The kernel by itself where a model takes the other one."""
import numpy as np
import pytest
import torch

from oracle import famepel_plain, kinetar_plain, mafalorn_plain, vosolorn_plain
from tests import famepel_helpers as fam
from tests import hybrid_helpers as kin
from tests import mafalorn_helpers as maf
from tests import vosolorn_helpers as vos
from tests.row_ops import RowOps

pytestmark = pytest.mark.gpu

CUTS = [5, 1, 8, 2, 7, 1, 4, 3, 6]


@pytest.mark.parametrize("width,ff", [(48, 72), (40, 24), (56, 2040), (264, 4999), (1032, 40), (45, 33)])
def test_dense(width, ff):
    cfg = kin.model_config([kin.delta(heads=2, kv_heads=1, dim=16, vdim=24, ff=ff)], width=width, vocab=83)
    toks = kin.rand_tokens(sum(CUTS), cfg["vocab"], 3)
    w = kinetar_plain.random_weights(cfg, 0, 8)
    hz = kin.Harness(cfg, w, dtype="bfloat16", low=8)
    try:
        got = hz.feed("a", toks, CUTS)
    finally:
        hz.close()
    assert kin.rel_err(got, kin.oracle_logits(cfg, w, toks)) < kin.TOL["bfloat16"]


@pytest.mark.parametrize("width,vocab", [(256, 24000), (1024, 6001)])
def test_one_row_over_many_weights(width, vocab):
    cfg = kin.model_config([kin.delta(heads=2, kv_heads=1, dim=16, vdim=24, ff=0)], width=width, vocab=vocab)
    toks = kin.rand_tokens(9, cfg["vocab"], 3)
    w = kinetar_plain.random_weights(cfg, 0, 8)
    hz = kin.Harness(cfg, w, dtype="bfloat16", low=8)
    try:
        got = hz.feed("a", toks, [1])
    finally:
        hz.close()
    assert kin.rel_err(got, kin.oracle_logits(cfg, w, toks)) < kin.TOL["bfloat16"]


@pytest.mark.parametrize("experts,top,ff,width", [(7, 3, 24, 40), (3, 3, 40, 48), (33, 2, 8, 40), (40, 6, 72, 264)])
def test_gated_experts(experts, top, ff, width):
    """Also all experts chosen by every token (3 of 3)."""
    cfg = maf.model_config([maf.ret(mlp=maf.moe(experts=experts, top=top, ff=ff, identity=None, groups=None))], width=width)
    toks = kin.rand_tokens(sum(CUTS), cfg["vocab"], 4)
    w = maf.settled(mafalorn_plain.random_weights(cfg, 0))
    hz = maf.Harness(cfg, w, "bfloat16")
    try:
        got = hz.feed("a", toks, CUTS)
    finally:
        hz.close()
    assert maf.close(got, maf.oracle_logits(cfg, w, toks), "bfloat16")


@pytest.mark.parametrize("experts,top,ff,shared", [(6, 2, 24, 40), (33, 4, 16, 48)])
def test_plain_experts(experts, top, ff, shared):
    cfg = vos.model_config([vos.mlstm(mlp=vos.moe(experts=experts, top=top, ff=ff, shared=shared))])
    toks = kin.rand_tokens(sum(CUTS), cfg["vocab"], 5)
    w = vosolorn_plain.random_weights(cfg, 0)
    hz = vos.Harness(cfg, w, "bfloat16")
    try:
        got = hz.feed("a", toks, CUTS)
    finally:
        hz.close()
    assert vos.close(got, vos.oracle_logits(cfg, w, toks), "bfloat16")


BROKEN = 7                                                     # the token whose embedding is no number
ROUTED = {"gated, groups": (famepel_plain, fam, fam.model_config([fam.glr(mlp=fam.moe(experts=6, top=4, count=2, keep=2, ff=24))] * 2)),
          "plain, largest": (vosolorn_plain, vos, vos.model_config([vos.mlstm(mlp=vos.moe(experts=6, top=4, ff=24))] * 2)),
          "gated, corrected": (mafalorn_plain, maf, maf.model_config([maf.ret(mlp=maf.moe(experts=6, top=4, ff=24, identity=None, groups=None))] * 2))}


@pytest.mark.parametrize("tokens", [[7, 7, 3], [7, 3, 7, 5, 9, 11, 2, 1], [3, 7, 7, 7, 7, 7, 7, 4], [7, 7, 7, 7, 7, 7, 7, 7]])
@pytest.mark.parametrize("kind", sorted(ROUTED))
def test_a_request_without_numbers_leaves_the_others_alone(kind, tokens):
    """Their logits are those of the same step with another token in the broken one's place, bit by bit."""
    plain, helpers, cfg = ROUTED[kind]
    w = dict(plain.random_weights(cfg, 0))
    w["embed"] = w["embed"].clone()
    w["embed"][BROKEN] = float("nan")
    columns = [c for c in range(cfg["vocab"]) if c != BROKEN]  # an output head that shares the table has one column without numbers
    out = []
    for row in (tokens, [6 if t == BROKEN else t for t in tokens]):
        hz = helpers.Harness(cfg, w, "bfloat16", slots=8)
        try:
            for _ in range(2):                                 # what a step finds in its buffers is what one like it left there
                out.append(hz.step([((len(out), i), [t], [0]) for i, t in enumerate(row)])[:, columns])
                for i in range(len(row)):
                    hz.end((len(out) - 1, i))
        finally:
            hz.close()
    for i, t in enumerate(tokens):
        assert np.isnan(out[0][i]).any() == np.isnan(out[1][i]).any() == (t == BROKEN)
        if t != BROKEN:
            assert np.array_equal(out[0][i], out[2][i]) and np.array_equal(out[1][i], out[2][i]), i


@pytest.mark.parametrize("rows", [4, 5, 8])
def test_fewer_finite_scores_than_choices(rows):
    """A router with one finite score: a token's other choices weigh nothing, and are distinct all the same (an expert takes a token once)."""
    cfg = vos.model_config([vos.mlstm(mlp=vos.moe(experts=6, top=4, ff=24))] * 2)
    w = dict(vosolorn_plain.random_weights(cfg, 0))
    for name in ("l0.mlp.router.b", "l1.mlp.router.b"):
        w[name] = w[name].clone()
        w[name][1:] = -float("inf")
    toks = kin.rand_tokens(3 * rows, cfg["vocab"], 6)
    hz = vos.Harness(cfg, w, "bfloat16")
    try:
        got = hz.feed("a", toks, [rows])
    finally:
        hz.close()
    assert vos.row_errs(got, vos.oracle_logits(cfg, w, toks)).max() < vos.TOL["bfloat16"]


@pytest.fixture(scope="module")
def ops():
    return RowOps()


@pytest.mark.parametrize("features,cols", [(32000, 1024), (2112, 2048), (1024, 7168), (17, 512), (300, 12280), (40, 8), (33, 264)])
@pytest.mark.parametrize("rows", [1, 2, 3, 5, 8])
def test_sums_of_few_rows(ops, rows, features, cols):
    """fp32 sums outside the tensor core: a sum that stayed in it over 1024 columns would be 3.8e-7 of its norm away.  The bound: a lane adds up to
    cols / 32 / 4 products of blocks of 16 one behind the other, each with a rounding of 2^-24 of a sum that grows to the result, root mean square of both; a
    factor of two for what a block's product loses by itself."""
    g = torch.Generator(device="cuda").manual_seed(rows)
    a, w = (torch.randn(n, cols, generator=g, device="cuda").bfloat16() for n in (rows, features))
    want = a.to(torch.float64) @ w.to(torch.float64).T
    err = ((ops.few(a, w).to(torch.float64) - want).norm() / want.norm()).item()
    assert err < min(2.0 * max(cols / 128, 8) ** 0.5 * 2.0 ** -24, 3e-7), err
