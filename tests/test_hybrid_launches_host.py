"""Host side of the hybrid decoders' steps on a CUDA runtime without a GPU: a step stops at the first call that fails, whichever it is,
says so, and leaves the engine able to run the next; kernels are set up on every device that an engine is made on; the form that latent
attention takes."""
import pytest

from tests import fake_cuda
from tests import famepel_helpers as fam
from tests import hybrid_helpers as kin
from tests import kisadra_helpers as kis
from tests import mafalorn_helpers as maf
from tests import sebavik_helpers as seb
from tests import vosolorn_helpers as vos

FLASH = fam.model_config([fam.latent(heads=2, dim=64, rot_dim=64, vdim=64, kv_rank=40, q_rank=24, mlp=None), fam.glr()])


def weights(cfg):
    import importlib
    plain = importlib.import_module("oracle.%s_plain" % cfg["architecture"].lower())
    return plain.random_weights(cfg, 0, 8) if cfg["architecture"] == "Kinetar" else plain.random_weights(cfg, 0)


CONFIGS = {"kinetar": kin.SMALL, "famepel": fam.SMALL, "flash": FLASH, "mafalorn": maf.SMALL, "kisadra": kis.SMALL, "sebavik": seb.SMALL, "vosolorn": vos.SMALL}


@pytest.fixture(scope="module")
def fake():
    from jacobiforcing_b200 import _hybrid_cabi
    path, mp = fake_cuda.build("hy"), pytest.MonkeyPatch()
    mp.setattr(_hybrid_cabi, "LIB_PATH", path)
    mp.setattr(_hybrid_cabi, "build", lambda force=False: path)
    mp.setattr(_hybrid_cabi, "stale", lambda: False)
    mp.setattr(_hybrid_cabi, "_lib", None)
    yield fake_cuda.Fake(path)
    mp.undo()


def engine(cfg, dtype="bfloat16", device=0):
    from jacobiforcing_b200.hybrid_config import HybridConfig
    from jacobiforcing_b200.hybrid_runtime import HybridRuntime
    w = weights(cfg)
    rt = HybridRuntime(HybridConfig.from_dict(cfg, {k: tuple(t.shape) for k, t in w.items()}), dtype=dtype, device=device, max_step_tokens=256,
                       max_step_entries=4, page_size=16, num_pages=64, max_pages_per_seq=16, num_slots=4, max_want=16)
    rt.load_state_dict(w)
    return rt


def step(rt, tokens, entries=1):
    n = tokens // entries
    return rt.step([([1] * n, 0, e, list(range(16 * e, 16 * e + 16))) for e in range(entries)], [tokens - 1], want_logits=True, sample=True)


@pytest.mark.parametrize("tokens", [3, 150])
@pytest.mark.parametrize("which", sorted(CONFIGS))
@pytest.mark.parametrize("what", ["launch", "tensor map"])
def test_nothing_is_launched_behind_a_failure(fake, what, which, tokens):
    """Were the failure dropped, the step would return what its buffers happened to hold, or rotate the same queries twice."""
    kind = fake_cuda.LAUNCH if what == "launch" else fake_cuda.TENSOR_MAP
    rt = engine(CONFIGS[which])
    step(rt, tokens)
    names = []
    for _ in range(2):                                       # routing counters alternate between two sets: two steps that are alike
        fake.reset()
        step(rt, tokens)
        names.append([n for n, _ in fake.launches()])
    calls, names = fake.count(kind), names[0]
    assert len(names) > 3
    if which == "flash" and tokens > 64:
        assert any("flash_kernel" in n for n in names)
    for at in range(calls):
        fake.reset()
        fake.fail(kind, at)
        with pytest.raises(RuntimeError, match="launch refused" if what == "launch" else "a tensor map of the"):
            step(rt, tokens)
        went = [n for n, _ in fake.launches()]
        assert went == names[:len(went)] and len(went) < len(names) and fake.count(kind) == at + 1
        fake.reset()
        step(rt, tokens)
        assert [n for n, _ in fake.launches()] == names
    rt.close()


def test_nothing_writes_to_the_caller_behind_a_failure(fake):
    """The caller's arrays may be page-locked, so that copies into them go on after the call that made them: a step that fails waits for those."""
    rt = engine(CONFIGS["famepel"])
    fake.reset()
    step(rt, 5)
    copies = fake.count(fake_cuda.TO_HOST)
    assert copies == 3                                       # sampled tokens, logits, the kernels' error word
    for at in range(copies):
        fake.reset()
        fake.fail(fake_cuda.TO_HOST, at)
        with pytest.raises(RuntimeError, match="invalid argument"):
            step(rt, 5)
        assert fake.on_their_way() == 0
        fake.reset()
        step(rt, 5)
    rt.close()


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
@pytest.mark.parametrize("which", sorted(CONFIGS))
def test_steps_on_two_devices(fake, which, dtype):
    """A kernel's shared-memory limit belongs to a device: the fake refuses launches above what was asked for on theirs."""
    seen = []
    for device in (0, 1):
        rt = engine(CONFIGS[which], dtype, device)
        fake.reset()
        for tokens in (1, 4, 150):
            step(rt, tokens)
        step(rt, 152, 4)
        seen.append([n for n, _ in fake.launches()])
        assert {d for _, d in fake.launches()} == {device}
        rt.close()
    assert seen[0] == seen[1]


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
@pytest.mark.parametrize("tokens", [1, 8, 150])
def test_engines_of_unlike_sizes_take_turns(fake, tokens, dtype):
    """The limit of a kernel is one for all engines on a device: what the smaller engine asks for must not take it from the larger one."""
    def layers(dim, vdim, ff):
        return kin.model_config([kin.delta(heads=2, kv_heads=1, dim=dim, vdim=vdim, ff=ff), kin.attn_scan()], width=40)
    large, small = engine(layers(128, 128, 5000), dtype), engine(layers(120, 100, 1200), dtype)
    fake.reset()
    for rt in (large, small, large, small, large):
        step(rt, tokens)
    for rt in (large, small):
        rt.close()


def test_results_take_page_locked_memory_when_they_are_large(fake):
    """And on the engine's device, whatever the calling thread was on."""
    fake.reset()
    cfg = kin.model_config([kin.delta()], vocab=1100)
    one, other = engine(cfg, device=1), engine(cfg)
    step(one, 5)
    step(other, 5)
    assert fake.pinned() == []
    one._results.empty((16, 1100))
    assert fake.pinned() == [1]
    one.close()
    other.close()


def roomy_engine(dtype):
    """An engine whose prompt steps have forms with workspaces of their own: chunks, segments, keys and values out of their pages, rows in three parts."""
    from jacobiforcing_b200.hybrid_config import HybridConfig
    from jacobiforcing_b200.hybrid_runtime import HybridRuntime
    cfg = kin.model_config([kin.attn_scan(heads=2, kv_heads=1, dim=64, inner=64), kin.delta(heads=2, kv_heads=1, dim=64, vdim=64)])
    w = weights(cfg)
    rt = HybridRuntime(HybridConfig.from_dict(cfg, {k: tuple(t.shape) for k, t in w.items()}), dtype=dtype, max_step_tokens=640, max_step_entries=2, page_size=16,
                       num_pages=48, max_pages_per_seq=48, num_slots=2, max_want=8)
    rt.load_state_dict(w)
    return rt


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
def test_workspaces_that_steps_can_do_without(fake, dtype):
    """Without room for them an engine is made all the same, down to the last byte of what it needs, and its steps take the forms that need none."""
    def names(room):
        fake.room(room)
        before = fake.used()
        try:
            rt = roomy_engine(dtype)
            used = fake.used() - before
            fake.reset()
            rt.step([([1] * 600, 0, 0, list(range(48)))], [599], want_logits=True)
            out = [n for n, _ in fake.launches()]
            rt.close()
        finally:
            fake.room()
        return used, out

    def has(out, *kernels):
        return [any(k in n for n in out) for k in kernels]
    held = fake.used()                                       # by engines that other tests left
    with_own = ["delta_chunk_chain_kernel", "page_gather_kernel", "split_rows_kernel"] if dtype == "bfloat16" else ["delta_chunk_chain_kernel"]
    plain = ["delta_head_kernel", "attn_mma_kernel", "gemm_simt_kernel"] if dtype == "bfloat16" else ["delta_head_kernel"]
    most, fast = names(1 << 40)
    assert all(has(fast, *with_own)) and not has(fast, "delta_head_kernel")[0] and sum("scan_kernel" in n for n in fast) == 2
    least, slow = names(held + most)                         # they would leave nothing for kernels that are yet to be loaded
    assert least < most and all(has(slow, *plain)) and not any(has(slow, *with_own)) and sum("scan_kernel" in n for n in slow) == 1
    assert names(held + least) == (least, slow)
    with pytest.raises((RuntimeError, MemoryError)):
        names(held + least - 1)


def test_refused_shared_memory_is_reported(fake):
    rt = engine(FLASH)
    fake.reset()
    fake.fail(fake_cuda.ATTRIBUTE, 0)
    with pytest.raises(RuntimeError, match="invalid argument"):
        step(rt, 150)
    went = fake.launches()
    step(rt, 150)                                            # asked for again
    assert len(fake.launches()) > 2 * len(went)
    rt.close()


ALONE = ("scan_kernel", "gla_kernel", "gla_chunk_", "delta_head_kernel", "delta_chunk_", "attn_mma_kernel", "biased_mma_kernel", "glr_kernel", "attn_sink_kernel", "biased_attn_kernel")


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
@pytest.mark.parametrize("tokens", [1, 8, 9, 63, 64, 65])
def test_which_launches_overlap(fake, tokens, dtype):
    """All in steps of up to 64 tokens, but beyond eight not the folded form of latent attention; beyond 64 not the kernels named in ALONE."""
    rt = engine(fam.model_config([fam.latent(mlp=None), fam.glr(mlp=None)]), dtype)
    fake.reset()
    step(rt, tokens)
    folded = ("latent_query", "attn_", "head_rows", "latent_value")
    for (name, _), overlaps in zip(fake.launches(), fake.overlaps()):
        assert overlaps != (tokens > 8 and any(f in name for f in folded) or tokens > 64 and any(a in name for a in ALONE)), name
    assert sum(any(f in n for f in folded) for n, _ in fake.launches()) >= 3


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
@pytest.mark.parametrize("tokens", [65, 150, 255, 256])
@pytest.mark.parametrize("which", ["kinetar", "famepel", "kisadra", "mafalorn"])
def test_which_launches_of_prompt_steps_overlap(fake, which, tokens, dtype):
    """All but those whose time is their longest block, convolutions among them from 256 tokens on, and the folded form of latent attention."""
    rt = engine(CONFIGS[which], dtype)
    fake.reset()
    step(rt, tokens)
    folded = ("latent_query", "attn_", "head_rows", "latent_value")
    seen = 0
    for (name, _), overlaps in zip(fake.launches(), fake.overlaps()):
        if any(f in name for f in folded) and not any(a in name for a in ALONE):
            continue
        alone = any(a in name for a in ALONE) or ("conv_kernel" in name and tokens >= 256)
        assert overlaps != alone, name
        seen += alone
    assert seen
    rt.close()


def latent_engine(window):
    from jacobiforcing_b200.hybrid_config import HybridConfig
    from jacobiforcing_b200.hybrid_runtime import HybridRuntime
    cfg = maf.model_config([maf.lat(heads=2, dim=64, rot_dim=64, vdim=64, rank=24, size=window, mlp=None)])
    w = weights(cfg)
    rt = HybridRuntime(HybridConfig.from_dict(cfg, {k: tuple(t.shape) for k, t in w.items()}), dtype="bfloat16", max_step_tokens=2048, max_step_entries=8,
                       page_size=64, num_pages=8 * 160, max_pages_per_seq=160, num_slots=8, max_want=16)
    rt.load_state_dict(w)
    return rt


@pytest.mark.parametrize("window,entries,keys", [
    # (tokens, cached tokens) of each request -> keys that are projected (None: the folded form)
    (None, [(64, 0)], 64), (None, [(63, 0)], None), (None, [(64, 8000)], 8064), (None, [(1024, 7168)], 8192), (None, [(1024, 7169)], None),
    (None, [(1, 4000), (127, 0)], 4128), (None, [(1, 7000), (127, 0)], None), (None, [(127, 0), (1, 4095)], 4223), (None, [(127, 0), (1, 4096)], None),
    (None, [(1, 1000)] * 7 + [(512, 0)], 7519), (None, [(40, 0), (600, 10), (3, 700)], 40 + 610 + 703),
    # of a request's keys only the tiles that a row sees through the window
    (128, [(64, 6000)], 6064 - 5760), (128, [(64, 127)], 191), (128, [(64, 254)], 318), (128, [(64, 255)], 319 - 128), (1, [(100, 300)], 400 - 256), (1024, [(64, 6000)], 6064 - 4864),
    (128, [(1, 7000), (127, 0)], 7001 - 6784 + 127), (128, [(2000, 8000)], 10000 - 7808), (50, [(70, 500), (1, 130), (300, 0)], 570 - 384 + 131 + 300)])
def test_form_of_latent_attention(fake, window, entries, keys):
    rt = latent_engine(window)
    fake.reset()
    rt.step([([1] * n, ctx, e, list(range(160 * e, 160 * e + 160))) for e, (n, ctx) in enumerate(entries)], [0])
    assert fake.blocks("latent_gather_kernel") == ([] if keys is None else [keys])
    tiles = sum(-(-n // 128) for n, _ in entries)
    assert fake.blocks("flash_kernel") == ([] if keys is None else [2 * tiles])
    assert bool(fake.blocks("attn_mma") + fake.blocks("attn_wide")) == (keys is None)
    rt.close()


@pytest.mark.parametrize("scale,flash", [(0.4, True), (0.0, False), (-0.4, False)])
def test_flash_takes_positive_scales_only(fake, scale, flash):
    """It looks for the largest score before it scales them."""
    rt = engine(maf.model_config([maf.lat(heads=2, dim=64, rot_dim=64, vdim=64, rank=24, size=None, scale=scale, mlp=None)]))
    fake.reset()
    step(rt, 150)
    assert any("flash_kernel" in n for n, _ in fake.launches()) == flash
    rt.close()


@pytest.mark.parametrize("rank,split", [(128, True), (129, False)])
def test_rows_in_three_parts_are_short(fake, rank, split):
    """The tensor cores' sums lose more with every block of k than fp32 additions do."""
    from jacobiforcing_b200.hybrid_config import HybridConfig
    from jacobiforcing_b200.hybrid_runtime import HybridRuntime
    cfg = kin.model_config([kin.attn_scan(inner=64, dt_rank=rank)])
    w = weights(cfg)
    rt = HybridRuntime(HybridConfig.from_dict(cfg, {k: tuple(t.shape) for k, t in w.items()}), max_step_tokens=512, max_step_entries=1, page_size=16, num_pages=32,
                       max_pages_per_seq=32, num_slots=1, max_want=8)
    rt.load_state_dict(w)
    fake.reset()
    rt.step([([1] * 512, 0, 0, list(range(32)))], [511])
    assert bool(fake.blocks("split_rows_kernel")) == split
    rt.close()


@pytest.mark.parametrize("rows,vocab,few", [(1, 5859, False), (1, 5860, True), (2, 3906, False), (2, 3907, True), (3, 100, True), (8, 100, True)])
def test_which_products_of_few_rows_run_on_the_tensor_cores(fake, rows, vocab, few):
    """The output head over 1024 channels, at both sides of each line."""
    rt = engine(kin.model_config([kin.delta(ff=0)], width=1024, vocab=vocab))
    fake.reset()
    rt.step([([1] * 8, 0, 0, list(range(16)))], list(range(rows)))
    name = fake.launches()[-1][0]
    assert ("gemm_few_kernel" in name) == few and ("gemm_rows_kernel" in name) != few
    rt.close()


@pytest.mark.parametrize("entries,inner,tokens,passes", [(1, 2048, 287, 1), (1, 2048, 288, 2), (3, 2048, 400, 2), (4, 2048, 400, 1), (4, 1024, 383, 1), (4, 1024, 384, 2),
                                                         (3, 4096, 600, 1), (2, 4096, 288, 2)])
def test_which_scans_run_in_segments(fake, entries, inner, tokens, passes):
    """The longest request has so many tokens, the others ten."""
    from jacobiforcing_b200.hybrid_config import HybridConfig
    from jacobiforcing_b200.hybrid_runtime import HybridRuntime
    cfg = kin.model_config([kin.attn_scan(inner=inner, state=16)])
    w = weights(cfg)
    rt = HybridRuntime(HybridConfig.from_dict(cfg, {k: tuple(t.shape) for k, t in w.items()}), max_step_tokens=640, max_step_entries=4, page_size=16,
                       num_pages=160, max_pages_per_seq=40, num_slots=4, max_want=8)
    rt.load_state_dict(w)
    fake.reset()
    rt.step([([1] * (10 if e else tokens), 0, e, list(range(40 * e, 40 * e + 40))) for e in range(entries)], [0])
    assert sum("scan_kernel" in n for n, _ in fake.launches()) == passes
    rt.close()
