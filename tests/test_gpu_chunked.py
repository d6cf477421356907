"""Matrix-state recurrences of prompt steps in chunks of 64 tokens, against the plain fp64 restatements: portions that end at, before and
behind a chunk, portions too short for chunks between them (the state passes from one form to the other), key and value sizes at and beside
the padded ones (with and without 16-byte rows), several requests of a step, decays of nearly zero and of one."""
import numpy as np
import pytest

from oracle import famepel_plain, kinetar_plain, kisadra_plain, mafalorn_plain
from tests import famepel_helpers as fam
from tests import hybrid_helpers as kin
from tests import kisadra_helpers as kis
from tests import mafalorn_helpers as maf

pytestmark = pytest.mark.gpu

CUTS = [512, 3, 575, 1, 61]                                    # chunks from 512 tokens on


def _model(mode, dim, vdim, heads=2):
    if mode == "state space":
        return famepel_plain, fam, fam.model_config([fam.ssd(heads=heads, vdim=vdim, state=dim, groups=1, norm_groups=1, conv=4, mlp=None)])
    if mode == "forget":
        return famepel_plain, fam, fam.model_config([fam.glr(heads=heads, dim=dim, vdim=vdim, mlp=None)])
    if mode == "gated linear":
        return kisadra_plain, kis, kis.model_config([kis.gla(heads=heads, dim=dim, vdim=vdim, mlp=None)])
    return mafalorn_plain, maf, maf.model_config([maf.ret(heads=heads, dim=dim, vdim=vdim, decay=[1.0 - 2.0 ** (-2.0 - 3.0 * h) for h in range(heads)], mlp=None)])


MODES = ["state space", "forget", "gated linear", "retention"]


def _every_row(helpers, got, want, dtype):
    """These models choose no experts, so that rounding to bf16 has nothing to flip: it makes up to 2e-2 of a row."""
    return helpers.close(got, want, dtype) if dtype == "float32" else helpers.row_errs(got, want).max() < 4e-2


@pytest.mark.parametrize("dim,vdim,dtype", [(33, 35, "float32"), (64, 64, "float32"), (66, 40, "bfloat16"), (128, 64, "bfloat16"), (100, 128, "float32"), (128, 127, "bfloat16")])
@pytest.mark.parametrize("mode", MODES)
def test_chunked_portions(mode, dim, vdim, dtype):
    if mode == "retention" and dim % 2:
        dim += 1
    plain, helpers, cfg = _model(mode, dim, vdim)
    toks = kin.rand_tokens(sum(CUTS), cfg["vocab"], 5)
    w = plain.random_weights(cfg, 0)
    hz = helpers.Harness(cfg, w, dtype, num_pages=80, max_step_tokens=640)
    try:
        got = hz.feed("a", toks, CUTS)
    finally:
        hz.close()
    assert _every_row(helpers, got, helpers.oracle_logits(cfg, w, toks), dtype)


def _delta(kind, dim, vdim, heads, kv):
    if kind == "channel":
        return kinetar_plain, kin, kin.model_config([kin.delta(heads=heads, kv_heads=kv, dim=dim, vdim=vdim, ff=0)])
    return mafalorn_plain, maf, maf.model_config([maf.par(d_heads=heads, d_kv_heads=kv, d_dim=dim, d_vdim=vdim, conv=4, mlp=None)])


def _good(kind, got, want, dtype):
    return kin.rel_err(got, want) < kin.TOL[dtype] if kind == "channel" else _every_row(maf, got, want, dtype)


@pytest.mark.parametrize("dim,vdim,heads,kv,dtype", [(33, 35, 2, 1, "float32"), (64, 64, 1, 1, "bfloat16"), (64, 65, 2, 2, "float32"), (128, 48, 2, 1, "float32"),
                                                     (100, 128, 2, 1, "bfloat16"), (127, 127, 1, 1, "float32")])
@pytest.mark.parametrize("kind", ["channel", "head"])
def test_chunked_delta_rule(kind, dim, vdim, heads, kv, dtype):
    plain, helpers, cfg = _delta(kind, dim, vdim, heads, kv)
    toks = kin.rand_tokens(sum(CUTS), cfg["vocab"], 7)
    w = plain.random_weights(cfg, 0)
    hz = helpers.Harness(cfg, w, dtype, num_pages=80, max_step_tokens=640)
    try:
        got = hz.feed("a", toks, CUTS)
    finally:
        hz.close()
    assert _good(kind, got, helpers.oracle_logits(cfg, w, toks), dtype)


@pytest.mark.parametrize("kind", ["channel", "head"])
def test_chunked_delta_rule_of_equal_keys(kind):
    """One token again and again: every key of the request points the same way, which is as far from independent corrections as they get."""
    plain, helpers, cfg = _delta(kind, 64, 40, 2, 1)
    w = plain.random_weights(cfg, 3)
    toks = [5] * 530
    hz = helpers.Harness(cfg, w, "float32", num_pages=80, max_step_tokens=640)
    try:
        got = hz.feed("a", toks, [530])
    finally:
        hz.close()
    assert _good(kind, got, helpers.oracle_logits(cfg, w, toks), "float32")


@pytest.mark.parametrize("mode", MODES + ["channel delta", "head delta"])
def test_chunked_requests_of_a_step(mode):
    """Requests of 575, 1 and 576 tokens in one step, then again behind themselves."""
    plain, helpers, cfg = _delta(mode[:-6], 64, 36, 2, 1) if mode.endswith("delta") else _model(mode, 64, 36)
    w = plain.random_weights(cfg, 1)
    lens = {"a": 575, "b": 1, "c": 576}
    toks = {k: kin.rand_tokens(2 * n if n < 100 else n + 530, cfg["vocab"], i) for i, (k, n) in enumerate(lens.items())}
    hz = helpers.Harness(cfg, w, "float32", num_pages=160, max_step_tokens=1280)
    try:
        first = hz.step([(k, toks[k][:n], range(n)) for k, n in lens.items()])
        second = hz.step([(k, toks[k][n:], range(len(toks[k]) - n)) for k, n in lens.items()])
    finally:
        hz.close()
    a = b = 0
    for k, n in lens.items():
        m = len(toks[k]) - n
        got = np.concatenate([first[a:a + n], second[b:b + m]], 0)
        a, b = a + n, b + m
        want = helpers.oracle_logits(cfg, w, toks[k])
        assert _good("channel", got, want, "float32") if mode == "channel delta" else helpers.close(got, want, "float32"), k


def test_chunked_forget_gates_of_zero_and_one():
    """Forget gates at their ends: a channel that keeps everything beside one that keeps nothing."""
    plain, helpers, cfg = _model("forget", 64, 64)
    w = plain.random_weights(cfg, 2)
    w["l0.mix.lower"] = w["l0.mix.lower"] * 0
    bias = w["l0.mix.f.b"]
    for i in range(bias.numel()):
        if i % 4 < 2:
            bias.view(-1)[i] = 60.0 if i % 4 else -120.0
    toks = kin.rand_tokens(530, cfg["vocab"], 6)
    hz = helpers.Harness(cfg, w, "float32", num_pages=80, max_step_tokens=640)
    try:
        got = hz.feed("a", toks, [530])
    finally:
        hz.close()
    assert helpers.close(got, helpers.oracle_logits(cfg, w, toks), "float32")


@pytest.mark.parametrize("state,inner,rank", [(1, 300, 1), (5, 128, 4), (16, 64, 4), (17, 33, 2), (130, 8, 4)])
def test_selective_scan_in_segments(state, inner, rank):
    """Portions long enough for segments (three of 96 tokens and more), whole and with a rest, behind and before shorter ones; two requests of unlike
    lengths in a step, of which the shorter has fewer segments."""
    layer = kin.attn_scan(left_scale=0.0, inner=inner, state=state, dt_rank=rank)
    layer["mlp"] = None
    cfg = kin.model_config([layer])
    w = kinetar_plain.random_weights(cfg, 0, 8)
    cuts = [288, 5, 401, 40, 100]
    toks = {k: kin.rand_tokens(n, cfg["vocab"], i) for i, (k, n) in enumerate({"a": sum(cuts), "b": 500, "c": 130}.items())}
    hz = kin.Harness(cfg, w, num_pages=160, max_step_tokens=1280)
    try:
        got = {"a": hz.feed("a", toks["a"], cuts)}
        first = hz.step([("b", toks["b"][:70], range(70)), ("c", toks["c"][:20], range(20))])
        second = hz.step([("b", toks["b"][70:], range(430)), ("c", toks["c"][20:], range(110))])
    finally:
        hz.close()
    got["b"] = np.concatenate([first[:70], second[:430]], 0)
    got["c"] = np.concatenate([first[70:], second[430:]], 0)
    for k in toks:
        assert kin.rel_err(got[k], kin.oracle_logits(cfg, w, toks[k])) < kin.TOL["float32"], k


@pytest.mark.parametrize("dim,vdim", [(64, 40), (128, 128)])
@pytest.mark.parametrize("mode", MODES + ["channel delta", "head delta"])
def test_what_is_no_number_stays_with_the_tokens_from_its_own_on(mode, dim, vdim):
    """A token without numbers, at places of a chunk beside its groups of 4, 8, 16 and 32: the tokens before it come out as they do without it, bit by
    bit, and none behind it comes out at all."""
    plain, helpers, cfg = _delta(mode[:-6], dim, vdim, 2, 1) if mode.endswith("delta") else _model(mode, dim, vdim)
    broken, other = 7, 6
    w = dict(plain.random_weights(cfg, 0))
    w["embed"] = w["embed"].clone()
    w["embed"][broken] = float("nan")
    columns = [c for c in range(cfg["vocab"]) if c != broken]  # an output head that shares the table has one column without numbers
    toks = [other if t == broken else t for t in kin.rand_tokens(520, cfg["vocab"], 5)]
    hz = helpers.Harness(cfg, w, "float32", num_pages=80, max_step_tokens=640)
    try:
        def run(at):
            out = hz.feed("a", toks[:at] + [broken] + toks[at + 1:] if at else toks)[:, columns]
            hz.end("a")
            return out
        clean = run(0)
        for at in (129, 134, 139, 191, 400):
            got = run(at)
            assert np.array_equal(got[:at], clean[:at]) and np.isnan(got[at:]).any(1).all(), at
    finally:
        hz.close()
    assert np.isfinite(clean).all()
