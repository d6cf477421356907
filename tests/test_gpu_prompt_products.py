"""The prompt products on pairs of SMs where their tiles end: features and tokens at, before and behind 128- and 256-row tiles, k that
is no multiple of 64, more tiles than one wave of pairs (256-row tiles) and fewer (128), grouped products with both tile sizes and
with experts that get no, one or very many rows; every epilogue (squared ReLU, gated pairs, residual with and without norms).
bf16 build against the plain fp64 restatements within the bound of the other bf16 tests (6e-2 per row)."""
import pytest

from oracle import famepel_plain, kinetar_plain, kisadra_plain
from tests import famepel_helpers as fam
from tests import hybrid_helpers as kin

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ff,tokens,width", [(104, 127, 40), (256, 128, 64), (264, 129, 72), (20000, 129, 64), (9800, 257, 72), (9984, 300, 64), (5000, 511, 48)])
def test_squared_relu_tiles(ff, tokens, width):
    """The last four: more than 74 tiles of 256 features x 128 tokens, so 256-token tiles with a remainder."""
    cfg = kin.model_config([kin.delta(heads=2, kv_heads=1, dim=8, vdim=8, ff=ff)], width=width)
    w = kinetar_plain.random_weights(cfg, 0, 8)
    toks = kin.rand_tokens(tokens, cfg["vocab"], 2)
    hz = kin.Harness(cfg, w, dtype="bfloat16", num_pages=40)
    try:
        got = hz.feed("a", toks)
    finally:
        hz.close()
    assert kin.rel_err(got, kin.oracle_logits(cfg, w, toks)) < kin.TOL["bfloat16"]


@pytest.mark.parametrize("experts,top,tokens,ff", [(2, 1, 400, 24), (2, 2, 200, 136), (3, 2, 300, 16), (16, 2, 100, 40), (4, 1, 13, 24)])
def test_grouped_tiles(experts, top, tokens, ff):
    """The first three: 192 rows per expert and more, so 256-row tiles."""
    cfg = fam.model_config([fam.glr(heads=1, dim=4, vdim=4, mlp=fam.moe(experts=experts, top=top, count=1, keep=1, ff=ff))], width=48)
    w = famepel_plain.random_weights(cfg, 0)
    toks = kin.rand_tokens(tokens, cfg["vocab"], 6)
    hz = fam.Harness(cfg, w, "bfloat16", num_pages=40)
    try:
        got = hz.feed("a", toks)
    finally:
        hz.close()
    assert fam.close(got, fam.oracle_logits(cfg, w, toks), "bfloat16")


@pytest.mark.parametrize("tokens", [287, 288, 289])
def test_grouped_tiles_at_the_line_between_their_sizes(tokens):
    """Two experts, one per token: 144 rows per expert and more take 256-row tiles, fewer tiles of 128."""
    test_grouped_tiles(2, 1, tokens, 40)


@pytest.mark.parametrize("ff,tokens", [(40, 65), (10000, 260)])
def test_gated_pairs_beside_plain_columns(ff, tokens):
    layer = {"type": "attention", "mixer": {"heads": 2, "kv_heads": 1, "dim": 16, "vdim": 16, "mask": {"size": 64}, "scale": 0.25},
             "mlp": {"kind": "dense", "ff": ff}}
    cfg = {"architecture": "Kisadra", "layers": [layer], "norm": {"eps": 1e-5}, "vocab": 70, "width": 48}
    w = kisadra_plain.random_weights(cfg, 0)
    toks = kin.rand_tokens(tokens, 70, 7)
    hz = kin.Harness(cfg, w, dtype="bfloat16", num_pages=40)
    try:
        got = hz.feed("a", toks)
    finally:
        hz.close()
    want = kisadra_plain.forward(cfg, w, toks).numpy()
    assert kin.rel_err(got, want) < kin.TOL["bfloat16"]
