"""Latent attention of prompt portions over per-head keys and values: head sizes of every build, rows and keys that end at, before and
behind tiles of 128, portions behind earlier ones, windows shorter and longer than a tile, sinks, gates, several requests in a step,
and portions too short for this form between longer ones.  bf16 build against the plain fp64 restatements (bound of the other bf16
tests, 6e-2 per row; a masked tile or a lost key is of order one)."""
import pytest

from oracle import famepel_plain, mafalorn_plain
from tests import famepel_helpers as fam
from tests import hybrid_helpers as kin
from tests import mafalorn_helpers as maf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,rot,vdim,heads", [(32, 32, 64, 3), (56, 8, 128, 2), (96, 32, 64, 2), (64, 64, 128, 1), (128, 64, 128, 2), (160, 32, 64, 3)])
@pytest.mark.parametrize("cuts", [[64], [127, 65, 128], [129, 1, 130], [300, 64, 20, 100]])
def test_latent_prompt(dim, rot, vdim, heads, cuts):
    cfg = fam.model_config([fam.latent(heads=heads, dim=dim, rot_dim=rot, vdim=vdim, kv_rank=40, q_rank=24, scale=(dim + rot) ** -0.5, mlp=None)], width=64)
    w = famepel_plain.random_weights(cfg, 0)
    toks = kin.rand_tokens(sum(cuts), cfg["vocab"], 8)
    hz = fam.Harness(cfg, w, "bfloat16", num_pages=40)
    try:
        got = hz.feed("a", toks, cuts)
    finally:
        hz.close()
    assert kin.rel_err(got, fam.oracle_logits(cfg, w, toks)) < fam.TOL["bfloat16"]


@pytest.mark.parametrize("size", [1, 50, 128, 200, None])
def test_latent_prompt_window_and_gate(size):
    cfg = maf.model_config([maf.lat(heads=2, dim=64, rot_dim=64, vdim=64, rank=24, size=size, scale=0.1, mlp=None)], width=64)
    w = mafalorn_plain.random_weights(cfg, 0)
    cuts = [140, 129, 66]
    toks = kin.rand_tokens(sum(cuts), cfg["vocab"], 9)
    hz = maf.Harness(cfg, w, "bfloat16", num_pages=40)
    try:
        got = hz.feed("a", toks, cuts)
    finally:
        hz.close()
    assert kin.rel_err(got, maf.oracle_logits(cfg, w, toks)) < maf.TOL["bfloat16"]


def test_latent_prompts_of_several_requests():
    cfg = fam.model_config([fam.latent(heads=2, dim=32, rot_dim=32, vdim=64, kv_rank=40, q_rank=24, mlp=None)], width=64)
    w = famepel_plain.random_weights(cfg, 1)
    toks = {r: kin.rand_tokens(n, cfg["vocab"], 20 + i) for i, (r, n) in enumerate([("a", 300), ("b", 141), ("c", 190)])}
    want = {r: fam.oracle_logits(cfg, w, t) for r, t in toks.items()}
    hz = fam.Harness(cfg, w, "bfloat16", num_pages=60, slots=4)
    try:
        one = hz.step([("a", toks["a"][:170], range(170)), ("b", toks["b"][:1], range(1)), ("c", toks["c"][:100], range(100))])
        two = hz.step([("b", toks["b"][1:], range(140)), ("a", toks["a"][170:], range(130)), ("c", toks["c"][100:], range(90))])
    finally:
        hz.close()
    for got, r, lo, hi in [(one[:170], "a", 0, 170), (one[170:171], "b", 0, 1), (one[171:], "c", 0, 100), (two[:140], "b", 1, 141), (two[140:270], "a", 170, 300),
                           (two[270:], "c", 100, 190)]:
        assert kin.rel_err(got, want[r][lo:hi]) < fam.TOL["bfloat16"]


@pytest.mark.parametrize("scale", [-0.1, 0.0, -2.0])
def test_scales_that_are_not_positive(scale):
    cfg = maf.model_config([maf.lat(heads=2, dim=64, rot_dim=64, vdim=64, rank=24, size=None, scale=scale, mlp=None)], width=64)
    w = mafalorn_plain.random_weights(cfg, 3)
    toks = kin.rand_tokens(300, cfg["vocab"], 12)
    hz = maf.Harness(cfg, w, "bfloat16", num_pages=40)
    try:
        got = hz.feed("a", toks, [170, 130])
    finally:
        hz.close()
    assert kin.rel_err(got, maf.oracle_logits(cfg, w, toks)) < maf.TOL["bfloat16"]


@pytest.mark.parametrize("size", [1, 40, 129, 256])
def test_windows_far_behind_the_first_token(size):
    """Only the keys that a row sees are gathered: portions that begin tiles behind their request's first token, of several requests."""
    cfg = maf.model_config([maf.lat(heads=2, dim=64, rot_dim=64, vdim=64, rank=24, size=size, scale=0.1, mlp=None)], width=64)
    w = mafalorn_plain.random_weights(cfg, 2)
    toks = {r: kin.rand_tokens(n, cfg["vocab"], 40 + i) for i, (r, n) in enumerate([("a", 700), ("b", 420), ("c", 300)])}
    want = {r: maf.oracle_logits(cfg, w, t) for r, t in toks.items()}
    hz = maf.Harness(cfg, w, "bfloat16", num_pages=120, slots=4)
    at = dict.fromkeys(toks, 0)
    try:
        for take in ({"a": 500, "b": 127}, {"b": 129, "a": 70, "c": 257}, {"c": 3, "a": 130, "b": 164}, {"c": 40}):
            got, lo = hz.step([(r, toks[r][at[r]:at[r] + n], range(n)) for r, n in take.items()]), 0
            for r, n in take.items():
                assert kin.rel_err(got[lo:lo + n], want[r][at[r]:at[r] + n]) < maf.TOL["bfloat16"], (r, at[r])
                lo += n
                at[r] += n
        assert at == {r: len(t) for r, t in toks.items()}
    finally:
        hz.close()
