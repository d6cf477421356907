"""Products of fp32 rows in three bf16 parts (steps of 512 tokens and more), the selective scan's step sizes, with inner sizes at and beside the parts' 64 columns,
against the fp64 restatements within the bounds of the other bf16 tests."""
import pytest

from oracle import kinetar_plain
from tests import hybrid_helpers as kin

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rank,inner", [(1, 40), (64, 300), (65, 24), (130, 256)])
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
