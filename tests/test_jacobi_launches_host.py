"""Host side of the Jacobi engine's prompt forwards: kernels are set up on every device that an engine is made on, a forward stops at
the first call that fails, and which rows of a prompt run on which kernel."""
import os
import re

import pytest

from tests import fake_cuda

CFG = dict(hidden_size=256, num_hidden_layers=2, num_attention_heads=4, num_key_value_heads=2, head_dim=64, intermediate_size=768, vocab_size=300,
           tie_word_embeddings=False, rope_theta=1e6, max_position_embeddings=2048, rms_norm_eps=1e-6)


@pytest.fixture(scope="module")
def fake():
    from jacobiforcing_b200 import _cabi
    path, mp = fake_cuda.build("jf"), pytest.MonkeyPatch()
    mp.setenv("JF_LIB_PATH", path)
    mp.setattr(_cabi, "_lib", None)
    yield fake_cuda.Fake(path)
    mp.undo()


def engine(head_dim=64, device=0):
    import torch

    from jacobiforcing_b200.runtime import JacobiRuntime
    cfg = dict(CFG, head_dim=head_dim, hidden_size=4 * head_dim)
    rt = JacobiRuntime(cfg, device=device, max_rows=512, max_seqs=4, num_kv_pages=8, max_pages_per_seq=4)
    h, q, kv, inter, v = cfg["hidden_size"], 4 * head_dim, 2 * head_dim, cfg["intermediate_size"], cfg["vocab_size"]
    shapes = {"model.embed_tokens.weight": (v, h), "lm_head.weight": (v, h), "model.norm.weight": (h,)}
    for i in range(cfg["num_hidden_layers"]):
        p = "model.layers.%d." % i
        shapes.update({p + "self_attn.q_proj.weight": (q, h), p + "self_attn.k_proj.weight": (kv, h), p + "self_attn.v_proj.weight": (kv, h),
                       p + "self_attn.q_proj.bias": (q,), p + "self_attn.k_proj.bias": (kv,), p + "self_attn.v_proj.bias": (kv,),
                       p + "self_attn.o_proj.weight": (h, q), p + "mlp.gate_proj.weight": (inter, h), p + "mlp.up_proj.weight": (inter, h),
                       p + "mlp.down_proj.weight": (h, inter), p + "input_layernorm.weight": (h,), p + "post_attention_layernorm.weight": (h,)})
    rt.load_state_dict({k: torch.zeros(s, dtype=torch.bfloat16) for k, s in shapes.items()})
    return rt


def chunk(rt, rows=256):
    s = rt.new_sequence()
    rt.ensure_capacity(s, rows)
    try:
        return rt.forward([1] * rows, [(0, rows, 0, 0)], [s], rows - 8, 8, [(i, 0, i) for i in range(rows)])
    finally:
        rt.release(s)


@pytest.mark.parametrize("head_dim", [64, 128])
def test_prompt_chunks_on_two_devices(fake, head_dim):
    """A kernel's shared-memory limit belongs to a device: an engine on another device of the process launches the same stages."""
    seen = []
    for device in (0, 1):
        rt = engine(head_dim, device)
        fake.reset()
        chunk(rt)
        assert {d for _, d in fake.launches()} == {device}
        seen.append([n for n, _ in fake.launches()])
        rt.close()
    assert seen[0] == seen[1] and sum("pair_kernel" in n for n in seen[0]) == 9 and sum("flash_kernel" in n for n in seen[0]) == 2


@pytest.mark.parametrize("what", ["launch", "tensor map"])
def test_nothing_is_launched_behind_a_failure(fake, what):
    """Whichever launch or tensor map of a prompt chunk fails: an error, and no stage over what another one did not make (the rotary stage
    would leave keys and values of stale rows in the pages).  The engine then works on."""
    kind = fake_cuda.LAUNCH if what == "launch" else fake_cuda.TENSOR_MAP
    rt = engine()
    fake.reset()
    chunk(rt)
    names, calls = [n for n, _ in fake.launches()], fake.count(kind)
    assert len(names) == 2 * 8 + 3 and calls == (len(names) if what == "launch" else 9 * 2 + 2 * 2)
    before = -1
    for at in range(calls):
        fake.reset()
        fake.fail(kind, at)
        with pytest.raises(RuntimeError, match="prompt forward: " + ("launch refused" if what == "launch" else "a tensor map")):
            chunk(rt)
        went = [n for n, _ in fake.launches()]
        assert went == names[:len(went)] and fake.count(kind) == at + 1
        if what == "launch":
            assert len(went) == at
        else:                                                # two maps for each launch that takes some
            assert before <= len(went) < len(names) and ("pair_kernel" in names[len(went)] or "flash_kernel" in names[len(went)])
        before = len(went)
    fake.reset()
    chunk(rt)
    assert [n for n, _ in fake.launches()] == names
    rt.close()


@pytest.mark.parametrize("draft", [0, 8])
@pytest.mark.parametrize("prompt,cached", [(1, 0), (255, 0), (256, 0), (256, 256), (257, 0), (257, 256), (300, 256), (511, 256), (512, 0), (512, 256), (512, 512), (600, 0), (600, 512),
                                           (768, 0), (768, 512), (768, 768)])
def test_the_last_prompt_token_runs_on_the_persistent_kernel(fake, prompt, cached, draft):
    """Whether its pages were cached or not: the two kernels do not agree bit for bit.  Whole pages ahead of it run as stages."""
    rt = engine()
    s = rt.new_sequence()
    s.ctx = cached
    runs, commits, forward, commit_rows = [], [], rt.forward, rt.commit_rows

    def spy(tokens, groups, seqs, lm_row0, lm_rows, com=(), **kw):
        fake.reset()
        out = forward(tokens, groups, seqs, lm_row0, lm_rows, com, **kw)
        runs.append((groups[0][3], len(tokens), lm_rows, ["persistent" in n for n, _ in fake.launches()]))
        commits.extend(c[2] for c in com)
        return out

    def spy_commits(seqs, com):
        commits.extend(c[2] for c in com)
        commit_rows(seqs, com)
    rt.forward, rt.commit_rows = spy, spy_commits
    rt.prefill(s, [1] * prompt, [1] * draft)
    at, rows, lm_rows, kernels = runs[-1]
    assert kernels == [True] and at <= prompt - 1 < at + rows == prompt + draft and lm_rows > draft
    for at, rows, lm_rows, kernels in runs[:-1]:
        assert at % 256 == 0 and rows % 256 == 0 and lm_rows == 0 and len(kernels) == 1 + 8 + 2 and not any(kernels)
    assert sum(r[1] for r in runs[:-1]) == max(0, (prompt - 1) // 256 * 256 - cached)
    assert commits == list(range(min(cached, prompt - 1), prompt))
    rt.release(s)
    rt.close()


@pytest.mark.parametrize("logits,hidden", [(False, False), (True, False), (False, True), (True, True)])
def test_the_last_layer_of_rows_that_nobody_reads(fake, logits, hidden):
    """Only its keys and values are made; hidden rows or logits that are asked for need all of it."""
    rt = engine()
    s = rt.new_sequence()
    rt.ensure_capacity(s, 256)
    fake.reset()
    rt.forward([1] * 256, [(0, 256, 0, 0)], [s], 248 if logits else 0, 8 if logits else 0, [(i, 0, i) for i in range(256)], want_hidden=hidden)
    assert len(fake.launches()) == (1 + 2 * 8 if logits or hidden else 1 + 8 + 2) + 2 * logits
    assert "wide_rope_kernel" in fake.launches()[10][0]
    rt.release(s)
    rt.close()


def test_results_take_page_locked_memory_when_they_are_large(fake):
    """And on the engine's device, whatever the calling thread was on."""
    fake.reset()
    one, other = engine(device=1), engine()
    chunk(other)
    assert fake.pinned() == []
    one._results.empty((64 << 10,))
    assert fake.pinned() == [1]
    one.close()
    other.close()


@pytest.mark.parametrize("what", ["launch", "commit"])
def test_a_forward_by_stages_stops_at_the_first_launch_that_fails(fake, what, monkeypatch):
    """An error, nothing launched behind it, and the engine works on: the next forward finds the argmax keys clean."""
    monkeypatch.setenv("JF_BY_STAGES", "1")
    rt = engine()
    s = rt.new_sequence()
    rt.ensure_capacity(s, 40)
    commits = [(i, 0, i) for i in range(40)] if what == "commit" else []

    def forward():
        fake.reset()
        return rt.forward([1] * 40, [(0, 40, 0, 0)], [s], 0, 40, commits)
    forward()
    names = [n for n, _ in fake.launches()]
    assert len(names) == 1 + 2 * 9 + 2 + (what == "commit") and not any("persistent" in n for n in names) and all(fake.overlaps())
    for at in range(len(names)):
        fake.reset()
        fake.fail(fake_cuda.LAUNCH, at)
        with pytest.raises(RuntimeError, match="forward by stages: launch refused"):
            rt.forward([1] * 40, [(0, 40, 0, 0)], [s], 0, 40, commits)
        assert [n for n, _ in fake.launches()] == names[:at]
    forward()
    assert [n for n, _ in fake.launches()] == names
    rt.release(s)
    rt.close()


@pytest.mark.parametrize("rows,stages", [(256, "0"), (512, "0"), (40, "1"), (40, "0")])
def test_what_is_on_its_way_to_the_device_outlives_the_copy(fake, rows, stages, monkeypatch):
    """A forward waits once, behind its kernels: whatever it copies to the device is still there then, as it was."""
    monkeypatch.setenv("JF_BY_STAGES", stages)
    rt = engine()
    fake.watch(True)
    try:
        for _ in range(2):
            chunk(rt, rows)
        assert fake.changed() == 0
    finally:
        fake.watch(False)
    rt.close()


def test_small_models_keep_the_persistent_kernel(fake):
    """A forward of theirs is one launch; the line is a layer's weights."""
    rt = engine()
    s = rt.new_sequence()
    rt.ensure_capacity(s, 40)
    fake.reset()
    rt.forward([1] * 40, [(0, 40, 0, 0)], [s], 0, 40)
    assert ["persistent" in n for n, _ in fake.launches()] == [True]
    rt.release(s)
    rt.close()


def header(fake, first=0, **fields):
    """What the policy kernel leaves in the header of a run's forward, as the host reads it."""
    source = open(os.path.join(fake_cuda.CSRC, "jf_types.h")).read()
    size, at = 0, {}
    for name, many in re.findall(r"^  int (\w+)(\[kMaxLmTasks\])?;", source[source.index("struct PlanHdr"):source.index("struct SeqSlot")], re.M):
        at[name], size = size, size + 4 * (int(re.search(r"kMaxLmTasks *= (\d+)", source).group(1)) if many else 1)
    for name, value in fields.items():
        fake.plant(size, at[name], value, first)


def run(rt, mode="single", **knobs):
    from jacobiforcing_b200.policy import MODES, PolicyKnobs
    s = rt.new_sequence()
    s.tokens, s.ctx = [1] * 20, 20
    try:
        return rt.jacobi_run([s], PolicyKnobs(mode=MODES[mode], n=8, max_new_tokens=16, max_calls=4, vocab=rt.vocab, **knobs), [1], [[1] * 8])[1]
    finally:
        rt.release(s)


def test_a_run_by_stages_ends_at_the_first_wait_that_ran_out(fake, monkeypatch):
    """The error comes before another forward, and before anything of the stalled one is committed.  The engine works on."""
    monkeypatch.setenv("JF_BY_STAGES", "1")
    rt = engine()

    def names(stalled):
        fake.reset()
        header(fake, T=8, G=1, max_len=8, n_lm_tasks=1, lm_rows=8, n_commit=3)
        header(fake, first=2, stalled=stalled)
        header(fake, first=3, done=1)
        try:
            return run(rt), [n for n, _ in fake.launches()]
        except RuntimeError as e:
            return str(e), [n for n, _ in fake.launches()]
    done, whole = names(0)
    assert isinstance(done, dict) and sum("policy" in n for n in whole) == 4 and sum("commit" in n for n in whole) == 4
    error, short = names(1)
    assert "a wait inside a tensor-core kernel ran out" in error
    ends = [i for i, n in enumerate(whole) if "policy" in n]
    assert short == whole[:ends[2] + 1]
    assert names(0)[1] == whole
    rt.close()


@pytest.mark.parametrize("what", ["launch", "header"])
def test_a_run_by_stages_that_fails_leaves_the_argmax_keys_clean(fake, what, monkeypatch):
    """Whichever launch, or copy of a header, is refused: an error, nothing behind it, and a forward before it has left nothing for the next run."""
    monkeypatch.setenv("JF_BY_STAGES", "1")
    rt = engine()
    keys, kind = 2 * 512 * 8, fake_cuda.LAUNCH if what == "launch" else fake_cuda.TO_HOST

    def plan():
        fake.reset()
        header(fake, T=8, G=1, max_len=8, n_lm_tasks=1, lm_rows=8, n_commit=3)
        header(fake, first=2, done=1)
    plan()
    run(rt)
    whole, calls = [n for n, _ in fake.launches()], fake.count(fake_cuda.LAUNCH) if what == "launch" else 3
    assert fake.cleared(keys) == 1 and sum("policy" in n for n in whole) == 3
    for at in range(calls):
        plan()
        fake.fail(kind, at)
        with pytest.raises(RuntimeError, match="forward by stages: " + ("launch refused" if what == "launch" else "invalid argument")):
            run(rt)
        went = [n for n, _ in fake.launches()]
        assert went == whole[:len(went)] and (what == "header" or len(went) == at) and fake.cleared(keys) == 1
    plan()
    run(rt)
    assert [n for n, _ in fake.launches()] == whole
    rt.close()


def test_a_sampling_run_says_nothing_about_the_calls_behind_it(fake, monkeypatch):
    """It takes the persistent kernel; forwards and greedy runs behind it go by stages as those before it do."""
    monkeypatch.setenv("JF_BY_STAGES", "1")
    rt = engine()

    def kernels(call):
        fake.reset()
        header(fake, T=8, G=1, max_len=8, n_lm_tasks=1, lm_rows=8)
        header(fake, first=1, done=1)
        call()
        return [n for n, _ in fake.launches()]
    forward, greedy = kernels(lambda: chunk(rt, 40)), kernels(lambda: run(rt))
    assert len(forward) > 1 and len(greedy) > 1 and not any("persistent" in n for n in forward + greedy)
    for _ in range(2):
        assert ["persistent" in n for n in kernels(lambda: run(rt, "engine_nongreedy", temperature=0.7))] == [True]
        assert kernels(lambda: chunk(rt, 40)) == forward
    assert kernels(lambda: run(rt)) == greedy and kernels(lambda: chunk(rt, 40)) == forward
    rt.close()


def test_a_profile_shows_the_kernels_that_run(fake, monkeypatch):
    """Profiling a forward by stages changes nothing about which kernels run it; only marks inside the persistent kernel need that one."""
    monkeypatch.setenv("JF_BY_STAGES", "1")
    rt = engine()

    def kernels():
        fake.reset()
        header(fake, T=8, G=1, max_len=8, n_lm_tasks=1, lm_rows=8)
        header(fake, first=1, iter=1)
        header(fake, first=2, done=1)
        run(rt)
        return [n for n, _ in fake.launches()]
    plain = kernels()
    assert rt.profile_read()["stages"] == []
    rt.profile_enable(1)
    assert kernels() == plain
    layer = ["qkv_gemm", "qkv_rope", "attention", "attn_combine", "o_gemm", "o_reduce_norm", "gate_up_gemm", "down_gemm", "down_reduce_norm"]
    assert [s["stage"] for s in rt.profile_read()["stages"]] == ["embed+norm"] + ["L%d.%s" % (i, n) for i in range(2) for n in layer] + ["lm_head_argmax"]
    rt.profile_enable(-1)
    assert kernels() == plain
    rt.close()
    monkeypatch.setenv("JF_PROF_MARKS", "marks.txt")
    rt = engine()
    rt.profile_enable(1)
    assert ["persistent" in n for n in kernels()] == [True]
    rt.close()
