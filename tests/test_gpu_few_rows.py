"""bf16 products of one to eight rows on the tensor cores: features beside the tiles of 16, k beside the blocks of 32 and beside what a batch or a split
holds, sizes that keep the other kernel, and the routed form (experts without a row, experts that every token chose, gated and plain), against the
fp64 restatements within the bounds of the other bf16 tests."""
import pytest

from oracle import kinetar_plain, mafalorn_plain, vosolorn_plain
from tests import hybrid_helpers as kin
from tests import mafalorn_helpers as maf
from tests import vosolorn_helpers as vos

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
