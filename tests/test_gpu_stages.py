"""Forwards as one kernel per stage (jf_step.cuh) against the persistent kernel: the same bits, so nothing depends on which of the two runs
a forward.  Row counts around the tiles of 16, 128 and 256 rows and where the rings and accumulators change, groups beyond a warp,
odd contexts, contexts of more than 32 chunks, rows behind the last one that a head takes, more rows than one head product takes, commits, hidden rows,
whole Jacobi runs, sampling runs between them; heads of 64 and 128, gate/up with and without k-splits, up to eight k-splits of the others, blocks with several
tiles in turn, chunks of more than one sub-tile; the tiles and k-splits of the 0.5B and 7B shapes."""
import random

import numpy as np
import pytest
import torch

from jacobiforcing_b200.runtime import hf_generate
from tests.gpu_helpers import make_pair

pytestmark = pytest.mark.gpu

# k-splits of query/output/down/gate-up: tiny 1/1/2/1, tiny128 2/2/4/2, mid128 4/4/8/4; six blocks: 16 tiles of the head, 9 of gate and up, in turn
SHAPES = {"tiny": ("tiny", "4", {}), "tiny128": ("tiny128", "4", {}), "mid128": ("mid128", "4", {}), "tiny128-whole-gate": ("tiny128", "1", {}),
          "tiny128-six-blocks": ("tiny128", "4", dict(num_ctas=6)), "tiny128-long-chunks": ("tiny128", "4", dict(attn_chunk=128))}


@pytest.fixture(scope="module", params=list(SHAPES))
def both(request):
    name, gate, more = SHAPES[request.param]
    mp, made = pytest.MonkeyPatch(), []
    mp.setenv("JF_GU_SPLITS", gate)
    for stages in "01":
        mp.setenv("JF_BY_STAGES", stages)
        made.append(make_pair(name, max_rows=640, max_seqs=8, num_kv_pages=40, max_pages_per_seq=12, **more))
    mp.undo()
    yield made[0][0].config, [rt for _, rt in made]
    for _, rt in made:
        rt.close()


def tokens(n, seed, vocab):
    return torch.randint(0, vocab, (n,), generator=torch.Generator().manual_seed(seed)).tolist()


def cached(rt, n, vocab, seed=3):
    """A sequence with n tokens in its pages."""
    s = rt.new_sequence()
    rt.ensure_capacity(s, n + 300)
    toks = tokens(n, seed, vocab)
    for a in range(0, n, 200):
        part = toks[a:a + 200]
        rt.forward(part, [(0, len(part), 0, a)], [s], 0, 0, [(i, 0, a + i) for i in range(len(part))])
    s.ctx = n
    return s


def same(got):
    a, b = got
    assert a.keys() == b.keys()
    for k in a:
        if isinstance(a[k], np.ndarray):
            assert a[k].tobytes() == b[k].tobytes(), k
    return a


@pytest.mark.parametrize("rows", [1, 7, 16, 17, 33, 64, 65, 120, 128, 129, 200, 255, 256, 257, 400, 513])
@pytest.mark.parametrize("ctx", [0, 77])
def test_rows(both, rows, ctx):
    cfg, rts = both
    got = []
    for rt in rts:
        s = cached(rt, ctx, cfg.vocab_size)
        rt.ensure_capacity(s, ctx + rows)
        row0 = (max(0, rows - 256) + 7) // 8 * 8
        launches = rt.launches
        out = rt.forward(tokens(rows, rows, cfg.vocab_size), [(0, rows, 0, ctx)], [s], row0, rows - row0, want_logits=True, want_hidden=True)
        got.append({k: out[k] for k in ("logits", "hidden")})
        got[-1]["greedy"] = np.asarray(out["greedy"])[row0:].copy()
        assert (rt.launches - launches > 1) == (rt is rts[1])
        rt.release(s)
    out = same(got)
    assert (out["logits"][np.arange(rows - row0), out["greedy"]] >= out["logits"].max(1) - 2.0 ** -7 * np.abs(out["logits"]).max(1)).all()      # the first of the largest bf16 values


@pytest.mark.parametrize("rows,first", [(300, 0), (513, 0), (600, 24)])
def test_more_rows_than_a_head_product_takes(both, rows, first):
    cfg, rts = both
    got = []
    for rt in rts:
        s = cached(rt, 77, cfg.vocab_size)
        rt.ensure_capacity(s, 77 + rows)
        out = rt.forward(tokens(rows, rows, cfg.vocab_size), [(0, rows, 0, 77)], [s], first, rows - first)
        got.append({"greedy": np.asarray(out["greedy"])[first:].copy()})
        rt.release(s)
    assert len(set(same(got)["greedy"].tolist())) > 8


def test_groups(both):
    """Forty groups of up to eleven rows over three contexts, then their rows in the pages and what follows them."""
    cfg, rts = both
    got = []
    for rt in rts:
        seqs = [cached(rt, n, cfg.vocab_size, 5 + n) for n in (70, 131, 255)]
        groups, row = [], 0
        for g in range(40):
            n = 1 + g * 7 % 11
            groups.append((row, n, g % 3, seqs[g % 3].ctx))
            row += n
        last = {g[2]: g for g in groups}
        commits = [(g[0] + i, g[2], g[3] + i) for g in last.values() for i in range(g[1])]
        for s in seqs:
            rt.ensure_capacity(s, s.ctx + 40)
        out = rt.forward(tokens(row, 8, cfg.vocab_size), groups, seqs, 0, row, commits, want_logits=True)
        after = rt.forward(tokens(9, 9, cfg.vocab_size), [(0, 9, 1, seqs[1].ctx + last[1][1])], seqs, 0, 9, want_logits=True)
        got.append({"logits": out["logits"], "greedy": np.asarray(out["greedy"])[:row].copy(), "after": after["logits"]})
        for s in seqs:
            rt.release(s)
    same(got)


@pytest.mark.parametrize("ctx", [1985, 2048, 2100])
def test_more_chunks_than_lanes(both, ctx):
    cfg, rts = both
    got = []
    for rt in rts:
        s = cached(rt, ctx, cfg.vocab_size)
        rt.ensure_capacity(s, ctx + 70)
        got.append({"logits": rt.forward(tokens(66, 4, cfg.vocab_size), [(0, 66, 0, ctx)], [s], 0, 66, want_logits=True)["logits"]})
        rt.release(s)
    same(got)


@pytest.mark.parametrize("batch,n,mode", [(1, 8, "single"), (1, 32, "multiblock"), (5, 16, "multiblock"), (8, 24, "single")])
def test_jacobi_runs(both, batch, n, mode):
    cfg, rts = both
    got = []
    for rt in rts:
        prompts = [tokens(20 + 13 * i, 30 + i, cfg.vocab_size) for i in range(batch)]
        seqs, results, run = hf_generate(rt, prompts, n=n, max_new_tokens=70, mode=mode, pad=0, K=2, r=0.85, n_gram_pool_size=4,
                                         rngs=[random.Random(2 + i) for i in range(batch)])
        after = rt.forward(tokens(9, 9, cfg.vocab_size), [(0, 9, 0, 20)], seqs[:1], 0, 9, want_logits=True)["logits"]
        got.append({"after": after, "tokens": np.array([t for r in results for t in r.tokens]), "forwards": np.array([run["forwards"]])})
        for s in seqs:
            rt.release(s)
    same(got)


def test_sampling_between_greedy_calls(both):
    """Sampling runs take the persistent kernel on either engine.  What they leave (argmax keys, tagged words, the plan) is nothing to the forwards and runs by stages
    behind them, nor the other way round."""
    from jacobiforcing_b200.policy import MODES, PolicyKnobs
    cfg, rts = both
    got = []
    for rt in rts:
        mine = {}
        for turn in range(3):
            s = cached(rt, 30, cfg.vocab_size)
            s.tokens, s.ctx = tokens(30, 3, cfg.vocab_size), 29
            knobs = PolicyKnobs(mode=MODES["engine_nongreedy"], n=8, pad=0, max_new_tokens=20, vocab=rt.vocab, temperature=0.3, seed=5 + turn)
            launches = rt.launches
            results, _ = rt.jacobi_run([s], knobs, [0], None, pad_stream=[tokens(512, 6, cfg.vocab_size)])
            assert rt.launches == launches + 1
            mine["sampled%d" % turn] = np.array(results[0].tokens)
            rt.release(s)
            s, launches = cached(rt, 40, cfg.vocab_size, 9), rt.launches
            out = rt.forward(tokens(33, 10 + turn, cfg.vocab_size), [(0, 33, 0, 40)], [s], 0, 33, want_logits=True)
            assert (rt.launches - launches > 1) == (rt is rts[1])
            mine["logits%d" % turn], mine["greedy%d" % turn] = out["logits"], np.asarray(out["greedy"]).copy()
            rt.release(s)
            seqs, results, _ = hf_generate(rt, [tokens(25, 11, cfg.vocab_size)], n=16, max_new_tokens=30, mode="single", pad=0, rngs=[random.Random(turn)])
            mine["run%d" % turn] = np.array(results[0].tokens)
            rt.release(seqs[0])
        got.append(mine)
    same(got)


def test_profiles(both):
    """Of a run's second forward, on either path: nothing comes out otherwise, and the stages' times add up to less than the run's."""
    cfg, rts = both
    got = []
    for rt in rts:
        mine = {}
        for forward in (-1, 1, -1):
            rt.profile_enable(forward)
            seqs, results, run = hf_generate(rt, [tokens(25, 11, cfg.vocab_size)], n=16, max_new_tokens=30, mode="single", pad=0, rngs=[random.Random(4)])
            mine["tokens%d" % len(mine)] = np.array(results[0].tokens)
            rt.release(seqs[0])
            if forward == 1:
                stages = rt.profile_read()["stages"]
                names = [s["stage"] for s in stages]
                for name in ("embed+norm", "L0.attention", "lm_head_argmax"):
                    assert name in names, names
                assert all(s["work_us"] > 0.0 for s in stages if "attention" in s["stage"])
                assert sum(s["work_us"] + s["wait_us"] for s in stages) < 1e3 * run["device_ms"]
        assert mine["tokens0"].tolist() == mine["tokens1"].tolist() == mine["tokens2"].tolist()
        got.append(mine)
    same(got)


@pytest.fixture(scope="module", params=["qwen2-0.5b", "qwen2.5-coder-7b"])
def real(request):
    """Two layers of the real widths: k-splits 3/3/8/3 and 4/5/5/1, a head of 1187 and 1188 tiles for 148 blocks."""
    import bench
    from jacobiforcing_b200.runtime import JacobiRuntime
    if torch.cuda.mem_get_info(0)[0] < 24 << 30:
        pytest.skip("needs 10 GB of free device memory")
    cfg, mp, made = dict(bench.SHAPES[request.param], num_hidden_layers=2), pytest.MonkeyPatch(), []
    for stages in "01":
        mp.setenv("JF_BY_STAGES", stages)
        made.append(JacobiRuntime(cfg, max_rows=512, max_seqs=8, num_kv_pages=24, max_pages_per_seq=4, gen_capacity=1024, max_calls=64))
        bench.load_random_weights(made[-1], cfg, 7, "cuda:0")
    mp.undo()
    yield cfg["vocab_size"], made
    for rt in made:
        rt.close()


@pytest.mark.parametrize("rows", [1, 8, 17, 32, 33, 48, 64, 72, 96, 97, 112, 128, 129, 160, 230, 256, 300])
def test_rows_of_real_widths(real, rows):
    vocab, rts = real
    got = []
    for rt in rts:
        s = cached(rt, 150, vocab)
        rt.ensure_capacity(s, 150 + rows)
        few = rows <= 256
        launches = rt.launches
        out = rt.forward(tokens(rows, rows, vocab), [(0, rows, 0, 150)], [s], 0, rows, want_logits=few, want_hidden=True)
        assert (rt.launches - launches > 1) == (rt is rts[1])
        got.append({"hidden": out["hidden"], "greedy": np.asarray(out["greedy"]).copy()})
        if few:
            got[-1]["logits"] = out["logits"]
        rt.release(s)
    same(got)


@pytest.mark.parametrize("batch,n,mode", [(1, 32, "single"), (1, 8, "multiblock"), (8, 16, "multiblock")])
def test_jacobi_runs_of_real_widths(real, batch, n, mode):
    vocab, rts = real
    got = []
    for rt in rts:
        seqs, results, run = hf_generate(rt, [tokens(20 + 13 * i, 30 + i, vocab) for i in range(batch)], n=n, max_new_tokens=64, mode=mode, pad=0, K=2, r=0.85,
                                         n_gram_pool_size=4, rngs=[random.Random(2 + i) for i in range(batch)])
        got.append({"tokens": np.array([t for r in results for t in r.tokens]), "forwards": np.array([run["forwards"]]), "rows": np.array([run["rows"]])})
        for s in seqs:
            rt.release(s)
    same(got)
