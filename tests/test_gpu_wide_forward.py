"""Prompt chunks that run as one kernel per stage: against the HF fp32 forward (bf16 rounding of the stream, weights and activations:
2e-2 of the logits' norm, as the persistent kernel shows on the same chunks), rows and keys at the edges of tiles of 128 and 256,
chunks behind cached tokens at aligned and odd positions, several sequences in one forward, and the independence of a row's
result of how its prompt was cut (bit for bit)."""
import numpy as np
import pytest
import torch

from oracle.hf_model import teacher_forced_logits
from tests.gpu_helpers import make_pair

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=["tiny", "tiny128"])          # heads of 64 and of 128
def pair(request):
    model, rt = make_pair(request.param, max_rows=1024, max_seqs=4, num_kv_pages=32, max_pages_per_seq=4)
    yield model, rt
    rt.close()


def prompt_of(n, seed, vocab):
    return torch.randint(0, vocab, (n,), generator=torch.Generator().manual_seed(seed)).tolist()


def feed(rt, seq, tokens, cuts):
    """The prompt in chunks, every row committed; the last logits row."""
    rt.ensure_capacity(seq, len(tokens) + 8)
    at = 0
    for n in cuts:
        row0 = (n - 1) // 8 * 8
        r = rt.forward(tokens[at:at + n], [(0, n, 0, at)], [seq], row0, n - row0, [(i, 0, at + i) for i in range(n)], want_logits=True)
        at += n
    seq.ctx = at
    return r["logits"][-1], int(r["greedy"][n - 1])


def verify(rt, seq, tokens):
    """Logits of eight rows behind the committed prompt (the persistent kernel reads the pages that the chunks left)."""
    return rt.forward(tokens, [(0, 8, 0, seq.ctx)], [seq], 0, 8, want_logits=True)["logits"]


@pytest.mark.parametrize("cuts", [[256], [257], [383], [512], [1000], [256, 300], [40, 256], [300, 333], [129, 511, 1]])
def test_prompt_chunks_against_hf(pair, cuts):
    model, rt = pair
    toks = prompt_of(sum(cuts) + 8, 5 + len(cuts), model.config.vocab_size)
    seq = rt.new_sequence()
    try:
        launches = rt.launches
        last, greedy = feed(rt, seq, toks[:-8], cuts)
        assert rt.launches - launches >= sum(8 * model.config.num_hidden_layers if c >= 256 else 1 for c in cuts) - 2     # the stages' own kernels ran
        rows = verify(rt, seq, toks[-8:])
    finally:
        rt.release(seq)
    want = teacher_forced_logits(model, toks).float().numpy()
    n = sum(cuts)
    assert np.linalg.norm(last - want[n - 1]) < 2e-2 * np.linalg.norm(want[n - 1])
    assert np.linalg.norm(rows - want[n:n + 8]) < 2e-2 * np.linalg.norm(want[n:n + 8])
    assert last[greedy] >= last.max() - 2e-2 * np.abs(last).max()


@pytest.mark.parametrize("cuts", [[256, 344], [300, 300], [343, 257]])
def test_cut_of_a_prompt_changes_nothing(pair, cuts):
    model, rt = pair
    toks = prompt_of(608, 9, model.config.vocab_size)
    got = []
    for c in ([600], cuts):
        seq = rt.new_sequence()
        try:
            last, greedy = feed(rt, seq, toks[:600], c)
            got.append((last, greedy, verify(rt, seq, toks[600:])))
        finally:
            rt.release(seq)
    assert np.array_equal(got[0][0], got[1][0]) and got[0][1] == got[1][1] and np.array_equal(got[0][2], got[1][2])


def test_sequences_side_by_side(pair):
    model, rt = pair
    lens = [130, 257, 90]
    toks = [prompt_of(n + 8, 20 + i, model.config.vocab_size) for i, n in enumerate(lens)]
    seqs = [rt.new_sequence() for _ in lens]
    try:
        rows, groups, commits, at = [], [], [], 0
        for i, n in enumerate(lens):
            rt.ensure_capacity(seqs[i], n + 8)
            groups.append((at, n, i, 0))
            commits += [(at + j, i, j) for j in range(n)]
            rows += toks[i][:n]
            at += n
        rt.forward(rows, groups, seqs, 0, 0, commits)
        for i, n in enumerate(lens):
            seqs[i].ctx = n
            want = teacher_forced_logits(model, toks[i]).float().numpy()[n:n + 8]
            got = verify(rt, seqs[i], toks[i][n:])
            assert np.linalg.norm(got - want) < 2e-2 * np.linalg.norm(want)
    finally:
        for s in seqs:
            rt.release(s)


def cached_copy(rt, seq, tokens):
    """A sequence that shares the pages of `seq` for its first `tokens` tokens, as the block manager hands them out on a prefix hit."""
    s = rt.new_sequence()
    s.pages, s.ctx = list(seq.pages[:tokens // 256]), tokens
    return s


@pytest.mark.parametrize("n,cached,draft", [(256, 256, 0), (512, 512, 0), (512, 256, 0), (768, 768, 0), (512, 256, 8), (600, 512, 0), (600, 256, 8)])
def test_prefix_hit_equals_miss(pair, n, cached, draft):
    """Prompts that end inside a page, at its end, with a draft and without: the same tokens, and the same logits behind them bit for bit."""
    model, rt = pair
    toks = prompt_of(n + 8, 31, model.config.vocab_size)
    miss = rt.new_sequence()
    got = [rt.prefill(miss, toks[:n], toks[:draft])[:2], verify(rt, miss, toks[n:])]
    hit = cached_copy(rt, miss, cached)
    own = len(hit.pages)
    try:
        got += [rt.prefill(hit, toks[:n], toks[:draft])[:2], verify(rt, hit, toks[n:])]
    finally:
        hit.pages = hit.pages[own:]
        rt.release(hit)
        rt.release(miss)
    assert got[0] == got[2] and np.array_equal(got[1], got[3])


def test_hit_on_a_page_that_the_end_of_a_prompt_filled(pair):
    """The last page of a 512-token prompt comes from the persistent kernel, the same page of a longer prompt from the stages: a hit on it
    is a miss to bf16 rounding, no more (bound of the comparisons with HF)."""
    model, rt = pair
    toks = prompt_of(608, 33, model.config.vocab_size)
    short, miss = rt.new_sequence(), rt.new_sequence()
    rt.prefill(short, toks[:512], toks[:8])
    rt.prefill(miss, toks[:600], toks[:8])
    hit = cached_copy(rt, short, 512)
    own = len(hit.pages)
    try:
        rt.prefill(hit, toks[:600], toks[:8])
        a, b = verify(rt, hit, toks[600:]), verify(rt, miss, toks[600:])
    finally:
        hit.pages = hit.pages[own:]
        for s in (hit, miss, short):
            rt.release(s)
    assert np.linalg.norm(a - b) < 2e-2 * np.linalg.norm(b)


def test_chunks_whose_rows_nobody_reads(pair):
    """Without logits the last layer ends with its keys and values: the same pages as with them, bit for bit."""
    model, rt = pair
    toks = prompt_of(608, 41, model.config.vocab_size)
    got = []
    for row0, rows in ((0, 0), (248, 8)):
        s = rt.new_sequence()
        rt.ensure_capacity(s, 616)
        for at, n in ((0, 256), (256, 344)):
            rt.forward(toks[at:at + n], [(0, n, 0, at)], [s], row0, rows, [(i, 0, at + i) for i in range(n)])
        s.ctx = 600
        got.append(verify(rt, s, toks[600:]))
        rt.release(s)
    assert np.array_equal(got[0], got[1])
