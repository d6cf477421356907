"""Attention of prompt steps over keys and values gathered from their pages (256 or 512 tokens and more), in the layers that take it: temperatures, sinks and
gates; chunks with linear distances; values that are unrotated keys.  Portions at and beside the line and beside the tiles of 128, behind cached tokens,
several requests of a step, sizes of heads with another kernel beside those with this one, windows; bf16 against the fp64 restatements, every row: a
unit of 128 rows that wraps from one head to the next, a border of tiles or of chunks has few of them."""
import numpy as np
import pytest

from oracle import kinetar_plain, kisadra_plain, mafalorn_plain
from tests import hybrid_helpers as kin
from tests import kisadra_helpers as kis
from tests import mafalorn_helpers as maf

pytestmark = pytest.mark.gpu

CUTS = [256, 5, 513, 255]                                      # from 256 tokens on, with one cache for both from 512


def _model(kind, dim, vdim, heads, kv):
    if kind == "temperature":
        return kinetar_plain, kin, kin.model_config([kin.attn_scan(heads=heads, kv_heads=kv, dim=dim, scale=dim ** -0.5, coef=0.4, every=50, right_scale=0.0)])
    if kind == "chunk":
        return kisadra_plain, kis, kis.model_config([kis.attn(heads=heads, kv_heads=kv, dim=dim, vdim=vdim, size=300, scale=0.3, mlp=None)])
    return mafalorn_plain, maf, maf.model_config([maf.par(heads=heads, kv_heads=kv, dim=dim, dims=dim // 2, scale=dim ** -0.5, right_scale=0.0, mlp=None)])


ROW = 2.5e-2                                                   # rounding to bf16 makes up to 1.25e-2 of a row, with this kernel or with the one for shorter steps


def _good(got, want):
    return maf.row_errs(got, want).max() < ROW


@pytest.mark.parametrize("kind,dim,vdim,heads,kv", [("temperature", 64, 64, 4, 2), ("temperature", 128, 128, 3, 1), ("temperature", 32, 32, 4, 2), ("chunk", 64, 64, 4, 4),
                                                    ("chunk", 128, 64, 4, 2), ("chunk", 64, 128, 6, 2), ("chunk", 128, 128, 7, 1), ("chunk", 72, 64, 2, 1), ("side", 64, 64, 4, 2),
                                                    ("side", 128, 128, 2, 2)])
def test_paged_prompts(kind, dim, vdim, heads, kv):
    plain, helpers, cfg = _model(kind, dim, vdim, heads, kv)
    toks = kin.rand_tokens(sum(CUTS), cfg["vocab"], 5)
    w = plain.random_weights(cfg, 0)
    hz = helpers.Harness(cfg, w, "bfloat16", num_pages=80, max_step_tokens=640)
    try:
        got = hz.feed("a", toks, CUTS)
    finally:
        hz.close()
    assert _good(got, helpers.oracle_logits(cfg, w, toks))


@pytest.mark.parametrize("kind", ["temperature", "chunk", "side"])
def test_requests_of_a_step(kind):
    plain, helpers, cfg = _model(kind, 64, 64, 4, 2)
    w = plain.random_weights(cfg, 1)
    toks = {r: kin.rand_tokens(n, cfg["vocab"], i) for i, (r, n) in enumerate([("a", 729), ("b", 480), ("c", 140)])}
    want = {r: helpers.oracle_logits(cfg, w, t) for r, t in toks.items()}
    hz = helpers.Harness(cfg, w, "bfloat16", num_pages=100, max_step_tokens=640)
    at, got = dict.fromkeys(toks, 0), {r: [] for r in toks}
    try:
        for take in ({"a": 300, "b": 259}, {"a": 130, "c": 139, "b": 1}, {"b": 220, "a": 299, "c": 1}):
            out, lo = hz.step([(r, toks[r][at[r]:at[r] + n], range(n)) for r, n in take.items()]), 0
            for r, n in take.items():
                got[r].append(out[lo:lo + n])
                lo, at[r] = lo + n, at[r] + n
    finally:
        hz.close()
    assert at == {r: len(t) for r, t in toks.items()}
    for r in toks:
        assert _good(np.concatenate(got[r], 0), want[r]), r


@pytest.mark.parametrize("window,heads,kv,dim", [(1, 2, 1, 64), (127, 4, 2, 64), (128, 2, 2, 128), (300, 6, 2, 64), (2000, 3, 1, 128)])
def test_windows(monkeypatch, window, heads, kv, dim):
    """Linear distances inside a sliding window, which no model description asks for but a program of the C interface may: the layers of a description
    with the window put in, against the restatement that sees the same."""
    from jacobiforcing_b200.hybrid_config import HybridConfig
    plain = HybridConfig.from_dict

    def windowed(cfg, shapes=None):
        out = plain(cfg, shapes)
        out.layers[0].b_window = window
        return out
    monkeypatch.setattr(HybridConfig, "from_dict", windowed)
    monkeypatch.setattr(kisadra_plain, "sees", lambda i, j, size: j <= i and i - j < window)
    cfg = kis.model_config([kis.attn(heads=heads, kv_heads=kv, dim=dim, vdim=64, size=None, scale=0.3, mlp=None)])
    toks = kin.rand_tokens(sum(CUTS), cfg["vocab"], 5)
    w = kisadra_plain.random_weights(cfg, 0)
    hz = kis.Harness(cfg, w, "bfloat16", num_pages=80, max_step_tokens=640)
    try:
        got = hz.feed("a", toks, CUTS)
    finally:
        hz.close()
    assert _good(got, kis.oracle_logits(cfg, w, toks))
