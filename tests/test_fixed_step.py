"""Calls over bands and an exact top-k through the single native entry against the general path (masker
by masker, then the attention step) on the same tensors: the same kernels, so the same bits."""

import pytest
import torch

import workloads
from sparse_attention_hub.sparse_attention.research_attention import base
from sparse_attention_hub.sparse_attention.research_attention import fixed_step as fs
from sparse_attention_hub.sparse_attention.utils.mask_attention_utils import (
    attention_wait_errors, get_masked_attention_output, last_union_list)

DEV = "cuda:0"
SINK_LOCAL = [("sink", {"sink_size": 5}), ("local", {"window_size": 37})]
TOPK = SINK_LOCAL + [("oracle_topk", {"heavy_size": 0.05})]


def _inputs(dt, B, Hq, Hkv, Sq, S, D, layout="plain"):
    gen = torch.Generator(device=DEV).manual_seed(S + Sq)
    shape = {"plain": (B, Hkv, S, D), "cache": (B, Hkv, S + 77, D), "rows": (B, S, Hkv, D), "odd": (B, Hkv, S, D + 8)}[layout]
    q = torch.randn((B, Sq, Hq, D), generator=gen, device=DEV).to(dt).transpose(1, 2)
    kv = [torch.randn(shape, generator=gen, device=DEV).to(dt) for _ in range(2)]
    if layout == "rows":
        kv = [t.transpose(1, 2) for t in kv]
    return q, kv[0][:, :, :S, :D], kv[1][:, :, :S, :D]


def _both(ra, q, k, v, am=None, sinks=None):
    out, weights = ra.custom_attention(None, q, k, v, am, 0.125, 0.0, sparse_meta_data={}, layer_idx=0, s_aux=sinks)
    ucols, umemb, counts, _ = (t.clone() if isinstance(t, torch.Tensor) else t for t in last_union_list())
    mask = ra.build_mask(q, k, v, am, 0.125, 0.0, {}, layer_idx=0)
    want = get_masked_attention_output(None, q, k, v, am, sinks, 0.125, 0.0, mask)
    assert weights is None
    ucols_, umemb_, counts_, _ = last_union_list()
    assert torch.equal(counts, counts_)
    for g, n in enumerate(counts.tolist()):
        assert torch.equal(ucols[g, :n], ucols_[g, :n]) and torch.equal(umemb[g, :n], umemb_[g, :n])
    return out, want


@pytest.mark.gpu
@pytest.mark.parametrize("layout", ["plain", "cache", "rows", "odd"])
@pytest.mark.parametrize("dtype,Sq,S,D,stack,served", [
    ("f32", 1, 43, 64, "fixed", True), ("f32", 1, 42, 64, "fixed", True), ("f32", 1, 38, 64, "fixed", False),
    ("bf16", 3, 131, 64, "fixed", True), ("bf16", 1, 32768, 128, "fixed", True), ("bf16", 2, 32769, 64, "fixed", False),
    ("bf16", 1, 50001, 64, "fixed", True),
    ("bf16", 1, 4097, 128, "topk", True), ("f32", 4, 1000, 64, "topk", True), ("bf16", 1, 90000, 64, "topk", False),
    ("bf16", 24, 8191, 128, "topk", True), ("f32", 2, 40000, 64, "topk", True), ("bf16", 1, 19, 64, "topk only", False),
    ("bf16", 2, 260, 64, "topk only", True)])
def test_same_as_the_general_path(dtype, Sq, S, D, stack, served, layout, monkeypatch):
    dt = torch.bfloat16 if dtype == "bf16" else torch.float32
    q, k, v = _inputs(dt, 2, 8, 2, Sq, S, D, layout)
    stack = {"fixed": SINK_LOCAL, "topk": TOPK, "topk only": TOPK[2:]}[stack]
    ra = workloads.research_attention(stack, dtype, DEV)
    results = []

    def noted(*args):
        results.append(fs.fixed_step(*args))
        return results[-1]

    monkeypatch.setattr(base, "fixed_step", noted)
    got, want = _both(ra, q, k, v)
    assert (results[0] is not None) == served
    got, want = got.nan_to_num(), want.nan_to_num()  # (5 % of 19 keys are none, and attention over none is NaN)
    assert torch.equal(got, want)
    assert attention_wait_errors() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["one", "heads", "batches", "longer", "other type", "transposed"])
@pytest.mark.parametrize("dtype", ["f32", "bf16"])
def test_masks_and_sink_logits(dtype, form):
    dt = torch.bfloat16 if dtype == "bf16" else torch.float32
    B, Hq, Sq, S = 2, 8, 3, 700
    q, k, v = _inputs(dt, B, Hq, 2, Sq, S, 64)
    gen = torch.Generator(device=DEV).manual_seed(1)
    shape = {"heads": (1, Hq, Sq, S), "batches": (B, 1, Sq, S), "longer": (1, 1, Sq, S + 9), "transposed": (1, 1, S, Sq)}
    am = torch.randn(shape.get(form, (1, 1, Sq, S)), generator=gen, device=DEV)
    am = torch.where(am > 1.0, torch.finfo(dt).min, am).to(torch.float64 if form == "other type" else dt)
    if form == "transposed":
        am = am.transpose(2, 3)
    sinks = torch.randn(Hq, generator=gen, device=DEV) if form in ("one", "heads") else None
    for stack in (SINK_LOCAL, TOPK):
        got, want = _both(workloads.research_attention(stack, dtype, DEV), q, k, v, am, sinks)
        assert torch.equal(got, want)


@pytest.mark.gpu
def test_wrong_tensors_say_the_same():
    ra = workloads.research_attention(TOPK, "f32", DEV)
    q, k, v = _inputs(torch.float32, 1, 8, 2, 1, 300, 64)

    def call(*args, am=None):
        return ra.custom_attention(None, *args, am, 0.125, 0.0, sparse_meta_data={}, layer_idx=0)

    with pytest.raises(ValueError, match="keys and values"):
        call(q, k, v[:, :, :-1])
    with pytest.raises(ValueError, match="covers"):
        call(q, k, v, am=torch.zeros((1, 1, 1, 299), device=DEV))
    with pytest.raises(ValueError, match="one dtype"):
        call(q, k, v.bfloat16())
    with pytest.raises(Exception, match="cpu"):
        call(q.cpu(), k, v)
    with pytest.raises(NotImplementedError, match="head dim"):
        call(*(torch.randn((1, h, n, 32), device=DEV) for h, n in ((8, 1), (2, 300), (2, 300))))


@pytest.mark.gpu
@pytest.mark.parametrize("Hq,Hkv", [(8, 8), (8, 1), (32, 2)])
@pytest.mark.parametrize("maskers", [
    [("sink", {"sink_size": 1})], [("local", {"window_size": 1})], [("local", {"window_size": 300}), ("sink", {"sink_size": 400})],
    [("sink", {"sink_size": 3}), ("local", {"window_size": 9}), ("sink", {"sink_size": 64}), ("local", {"window_size": 640})]])
@pytest.mark.parametrize("dtype", ["f32", "bf16"])
def test_lists_of_bands(dtype, maskers, Hq, Hkv):
    """Bands that overlap, that come in another order, that are one column; up to sixteen rows per group."""
    q, k, v = _inputs(torch.bfloat16 if dtype == "bf16" else torch.float32, 2, Hq, Hkv, 1, 701, 128)
    got, want = _both(workloads.research_attention(maskers, dtype, DEV), q, k, v)
    assert torch.equal(got, want)


@pytest.mark.gpu
def test_streams_and_capture():
    """Two streams have tickets of their own; a captured call replays on new queries and keys."""
    ra = workloads.research_attention(TOPK, "bf16", DEV)
    q, k, v = _inputs(torch.bfloat16, 1, 8, 2, 1, 5000, 64)
    q, k = q.contiguous(), k.contiguous()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        call = lambda: ra.custom_attention(None, q, k, v, None, 0.125, 0.0, sparse_meta_data={}, layer_idx=0)[0]  # noqa: E731
        warm = call()
    torch.cuda.current_stream().wait_stream(side)
    assert torch.equal(warm, call())
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        out = call()
    q.copy_(torch.randn_like(q))
    k.copy_(torch.randn_like(k))
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, call())


@pytest.mark.gpu
@pytest.mark.parametrize("Hq,Sq,S,stack", [(8, 2, 32769, SINK_LOCAL), (8, 4, 70000, SINK_LOCAL), (8, 1, 40000, TOPK),
                                           (2, 1, 131072, TOPK)])
def test_key_counts_that_are_refused_are_not_tried(Hq, Sq, S, stack, monkeypatch):
    """Nothing of the native entry is prepared for a call that it will not take, and what it would say is known."""
    from sparse_attention_hub.sparse_attention.utils import mask_attention_utils as mau

    q, k, v = _inputs(torch.bfloat16, 1, Hq, 2, Sq, S, 64)
    maskers = workloads.research_attention(stack, "bf16", DEV).maskers
    with monkeypatch.context() as m:
        m.setattr(mau, "merge_tickets", None)
        assert fs.fixed_step(maskers, q, k, v, None, None, 0.125) is None
    monkeypatch.setattr(fs, "_select_fits", lambda *_: 1)
    if stack is TOPK:
        assert fs.fixed_step(maskers, q, k, v, None, None, 0.125) is None


@pytest.mark.gpu
@pytest.mark.parametrize("where", ["masker", "masker class", "score method", "attention", "attention class"])
def test_methods_that_somebody_replaced_are_called(where, monkeypatch):
    """A spy on a masker's or the attention's methods sees the call, on the instance and on the class."""
    ra = workloads.research_attention(TOPK, "bf16", DEV)
    q, k, v = _inputs(torch.bfloat16, 1, 8, 2, 1, 3000, 64)
    owner, name = {"masker": (ra.maskers[1], "add_mask"), "masker class": (type(ra.maskers[0]), "add_mask"),
                   "score method": (ra.maskers[2], "_compute_raw_attention_scores"), "attention": (ra, "build_mask"),
                   "attention class": (type(ra), "build_mask")}[where]

    def call():
        return ra.custom_attention(None, q, k, v, None, 0.125, 0.0, sparse_meta_data={}, layer_idx=0)[0]

    want, original, seen = call(), getattr(owner, name), []

    def spy(*args, **kwargs):
        seen.append(name)
        return original(*args, **kwargs)

    monkeypatch.setattr(owner, name, spy)
    got = call()
    assert seen == [name] and torch.equal(got, want)


@pytest.mark.gpu
@pytest.mark.parametrize("D,S", [(128, 3000), (128, 40000), (64, 3000)])
def test_a_chosen_kernel_is_taken_for_bands(D, S):
    from sparse_attention_hub.sparse_attention.utils import mask_attention_utils as mau

    ra = workloads.research_attention(SINK_LOCAL, "bf16", DEV)
    q, k, v = _inputs(torch.bfloat16, 1, 8, 2, 1, S, D)
    kernels = {}
    for choice in ("auto", "mma", "umma"):
        prev = mau.select_attention_kernel(choice)
        try:
            out = ra.custom_attention(None, q, k, v, None, 0.125, 0.0, sparse_meta_data={}, layer_idx=0)[0]
            kernels[choice] = mau.last_attention_kernel()
        finally:
            mau.select_attention_kernel(prev)
        if choice == "auto":
            want = out
        # rounding P and the output to bfloat16
        assert float((out.double() - want.double()).norm() / want.double().norm()) < 4 * 2.0 ** -9
    mma, umma = "masked_attention_mma_kernel", "masked_attention_umma_kernel"
    assert kernels == {"auto": mma, "mma": mma, "umma": umma if D == 128 else mma}


@pytest.mark.gpu
def test_scores_do_not_outlive_the_call():
    """What is kept for last_union_list() is the list: 32 rows x 8000 scores (0.5 MB) and their bits are given back."""
    ra = workloads.research_attention(TOPK, "bf16", DEV)
    q, k, v = _inputs(torch.bfloat16, 2, 16, 1, 1, 8000, 64)
    call = lambda: ra.custom_attention(None, q, k, v, None, 0.125, 0.0, sparse_meta_data={}, layer_idx=0)[0]  # noqa: E731
    call()
    torch.cuda.synchronize()
    out = call()
    kept = fs.mask_attention_utils._last_plan["step"][0]
    sizes = fs._native.attn_sizes(2, 16, 1, 1, 8000, 64, 0, fs._native.sm_count(q.device))
    assert kept.numel() < sizes.ucols_bytes + sizes.umemb_bytes + sizes.ucount_bytes + sizes.partial_bytes + 4 * 256
    assert torch.equal(out, call())


@pytest.mark.gpu
def test_graphs_have_tickets_of_their_own():
    """Two graphs captured on one stream, the first never replayed before the second, with shapes of their own or
    the same, and eager calls on that stream: nobody relies on another's tickets."""
    from sparse_attention_hub.sparse_attention.research_attention.decode_graph import DecodeStepGraph
    from sparse_attention_hub.sparse_attention.utils import mask_attention_utils as mau

    ra = workloads.research_attention(TOPK, "bf16", DEV)
    side = torch.cuda.Stream()
    calls, graphs, outs = [], [], []
    for S in (3000, 5000, 5000):
        q, k, v = _inputs(torch.bfloat16, 1, 8, 2, 1, S, 64)
        calls.append(lambda q=q, k=k, v=v: ra.custom_attention(None, q, k, v, None, 0.125, 0.0, sparse_meta_data={},
                                                               layer_idx=0)[0])
    want = [call() for call in calls]
    torch.cuda.synchronize()
    assert mau._ticket_cache
    eager = {t.data_ptr() for t in mau._ticket_cache.values()}
    for call in calls:
        graphs.append(torch.cuda.CUDAGraph())
        with torch.cuda.graph(graphs[-1], stream=side):
            outs.append(call())
    with torch.cuda.stream(side):
        assert torch.equal(calls[1](), want[1])
    torch.cuda.synchronize()
    for _ in range(3):
        for g in reversed(range(3)):
            outs[g].zero_()
            graphs[g].replay()
            assert torch.equal(outs[g], want[g])
    own = [t.data_ptr() for t in mau._graph_tickets.values()][-3:]
    assert len(set(own)) == 3 and not eager & set(own)
    held = DecodeStepGraph(ra, q, k, v, None, 0.125, {})
    held_tickets = held._scratch[-1].tickets
    assert len(held_tickets) == 1 and not eager & {t.data_ptr() for t in held_tickets.values()}
    assert torch.equal(held.replay(q), want[2])
    assert attention_wait_errors() == 0


def test_host_module_is_made_anew_for_another_torch(monkeypatch):
    import importlib.util

    spec = importlib.util.spec_from_file_location("sah_b200_build", fs._native.DEFAULT_LIB_DIR.parent / "build.py")
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    build.build_step()
    assert not build.step_is_stale()
    monkeypatch.setattr(build.metadata, "version", lambda _: "1.0")
    assert build.step_is_stale()


@pytest.mark.parametrize("fault", ["missing", "not a module", "other torch"])
def test_without_the_host_module_the_general_path_serves(fault, monkeypatch, tmp_path):
    monkeypatch.setattr(fs, "_module", None)
    if fault == "other torch":
        monkeypatch.setattr(torch, "__version__", "1.0+cu0")
    else:
        monkeypatch.setattr(fs._native, "LIB_PATH", tmp_path / "libsah_b200.so")
        monkeypatch.setattr(fs._native, "DEFAULT_LIB_DIR", tmp_path)
        if fault == "not a module":
            (tmp_path / "_sah_step.so").write_bytes(b"nothing")
    with pytest.warns(RuntimeWarning, match="general path"):
        assert fs._step_module() is False
    assert fs._step_module() is False  # and no second warning


@pytest.mark.gpu
def test_calls_without_the_host_module(monkeypatch):
    ra = workloads.research_attention(TOPK, "bf16", DEV)
    q, k, v = _inputs(torch.bfloat16, 1, 8, 2, 1, 3000, 64)
    call = lambda: ra.custom_attention(None, q, k, v, None, 0.125, 0.0, sparse_meta_data={}, layer_idx=0)[0]  # noqa: E731
    want = call()
    monkeypatch.setattr(fs, "_module", False)
    assert torch.equal(call(), want)


def test_other_stacks_keep_the_general_path():
    """Nothing but plain sink, local and one final top-k masker is taken, whatever the tensors."""
    class Cuda:  # stands in for a CUDA tensor: the maskers are looked at before anything else of it
        pass

    q = torch.zeros((1, 2, 1, 64))
    assert fs.fixed_step([], q, q, q, None, None, 1.0) is None
    assert fs.fixed_step([object()], q, q, q, None, None, 1.0) is None      # not on a CUDA device
    assert fs.fixed_step([object()], Cuda(), q, q, None, None, 1.0) is None
