"""CUDA path vs the numpy restatement and vs the reference's golden outputs.

Every call goes through the Python API, which reaches the kernels through the
C ABI of libsah_b200.so.  Index sets, ptr arrays, mask weights and integer
codes must be bit-exact; attention outputs within 1e-4 (fp32) / 2e-2 (bf16),
absolute and relative.
"""

import numpy as np
import pytest
import torch

from oracle import attention as o_attention
from oracle import hashattention as o_hash
from oracle import mask_ops, qk as o_qk, stacks
import workloads
from sparse_attention_hub.sparse_attention import Mask
from sparse_attention_hub.sparse_attention import _native_ops
from sparse_attention_hub.sparse_attention.utils.mask_attention_utils import (
    get_masked_attention_output,
    native_masked_attention,
)

from conftest import load_golden

pytestmark = pytest.mark.gpu
TOL = {"f32": 1e-4, "bf16": 2e-2}
DEV = "cuda:0"


def _run_native(wl, attention_mask=None, sinks=None, meta=None):
    ra = workloads.research_attention(wl.stack, wl.dtype, DEV)
    q, k, v = (workloads.to_torch(a, wl.dtype, DEV) for a in (wl.q, wl.k, wl.v))
    am = None if attention_mask is None else workloads.to_torch(attention_mask, wl.dtype, DEV)
    meta = {} if meta is None else meta
    mask = ra.build_mask(q, k, v, am, float(wl.scaling), 0.0, meta, layer_idx=0)
    s = None if sinks is None else torch.from_numpy(sinks).to(DEV)
    out = get_masked_attention_output(None, q, k, v, am, s, float(wl.scaling), 0.0, mask)
    torch.cuda.synchronize()
    return mask, out.float().cpu().numpy(), meta


def _assert_mask_equal(mask: Mask, ref_dense=None, golden=None):
    idx, ptr, data = mask.get_index_mask()
    idx, ptr, data = idx.cpu().numpy(), ptr.cpu().numpy(), data.float().cpu().numpy()
    if ref_dense is not None:
        ri, rp, rd = mask_ops.to_csr(ref_dense)
        np.testing.assert_array_equal(idx, ri)
        np.testing.assert_array_equal(ptr, rp)
        np.testing.assert_array_equal(data, rd)
    if golden is not None:
        np.testing.assert_array_equal(idx, golden["idx"])
        np.testing.assert_array_equal(ptr, golden["ptr"])
        np.testing.assert_array_equal(data, golden["data"])


def _close(a, b, dtype, scale=1.0):
    np.testing.assert_allclose(a, b, atol=TOL[dtype] * scale, rtol=TOL[dtype] * scale)


# ---------------------------------------------------------------------------
def test_sink_local_f32_golden_and_oracle():
    g = load_golden("sink_local_f32")
    wl = workloads.sink_local_fp32(seed=11, B=1, Hq=8, Hkv=2, S=640, D=128, sink=16, window=48)
    mask, out, _ = _run_native(wl)
    ref_mask, ref_out, _ = stacks.run_stack(wl.stack, wl.q, wl.k, wl.v, wl.scaling, "f32")
    _assert_mask_equal(mask, ref_mask, g)
    _close(out, ref_out, "f32")
    _close(out, g["out"], "f32")


def test_sink_local_sq3_causal_sinks():
    g = load_golden("sink_local_f32_sq3_causal_sinks")
    wl = workloads.sink_local_fp32(seed=12, B=2, Hq=4, Hkv=2, S=320, D=64, sink=8, window=24, Sq=3)
    mask, out, _ = _run_native(wl, attention_mask=g["attention_mask"], sinks=g["sinks"])
    _assert_mask_equal(mask, golden=g)
    _close(out, g["out"], "f32")


def test_sink_local_bf16_fraction():
    g = load_golden("sink_local_bf16_fraction")
    wl = workloads.sink_local_fp32(seed=13, B=2, Hq=8, Hkv=4, S=512, D=128)
    wl.dtype = "bf16"
    wl.q, wl.k, wl.v = (workloads.to_dtype(a, "bf16") for a in (wl.q, wl.k, wl.v))
    wl.stack = [("sink", {"sink_size": 0.05}), ("local", {"window_size": 0.1})]
    mask, out, _ = _run_native(wl)
    _assert_mask_equal(mask, golden=g)
    _close(out, g["out"], "bf16")


def test_cpu_runnable_config_full_size():
    """Sink(128)+Local(256), fp32, S=4096, 32/8 heads: the first benchmark configuration."""
    wl = workloads.sink_local_fp32(seed=1)
    mask, out, _ = _run_native(wl)
    ref_mask, ref_out, _ = stacks.run_stack(wl.stack, wl.q, wl.k, wl.v, wl.scaling, "f32")
    _assert_mask_equal(mask, ref_mask)
    _close(out, ref_out, "f32")


# ---------------------------------------------------------------------------
def test_hash_codes_bit_exact_vs_oracle_and_golden():
    g = load_golden("hash_bf16")
    wl = workloads.hashattention_bf16(seed=21, B=2, Hq=8, Hkv=2, S=1024, D=128, sink=16, window=32)
    mask, out, meta = _run_native(wl)
    kc = meta["key"][0]
    codes = kc.codes[..., : kc.length].cpu().numpy().view(np.uint32)
    w = wl.stack[2][1]["weights"]
    ref_codes = o_hash.signatures(o_attention.repeat_kv(wl.k, 4), w["key_matrix"], w["key_bias"],
                                  "silu", "bf16")
    np.testing.assert_array_equal(codes, ref_codes)
    np.testing.assert_array_equal(codes, g["kcodes"])  # the reference's own bits
    ref_mask, ref_out, _ = stacks.run_stack(wl.stack, wl.q, wl.k, wl.v, wl.scaling, "bf16")
    _assert_mask_equal(mask, ref_mask, g)
    _close(out, ref_out, "bf16")
    _close(out, g["out"], "bf16")


@pytest.mark.parametrize("act", ["relu", "gelu", "tanh"])
def test_hash_other_activations(act):
    wl = workloads.hashattention_bf16(seed=22, B=1, Hq=4, Hkv=2, S=777, D=128, sink=4, window=9,
                                      heavy=40, bits=32, hidden=64, layers=2, activation=act)
    mask, out, _ = _run_native(wl)
    ref_mask, ref_out, _ = stacks.run_stack(wl.stack, wl.q, wl.k, wl.v, wl.scaling, "bf16")
    _assert_mask_equal(mask, ref_mask)
    _close(out, ref_out, "bf16")


def test_hash_incremental_key_cache():
    """Keys appended between calls are hashed incrementally and give the same codes."""
    wl = workloads.hashattention_bf16(seed=23, B=1, Hq=8, Hkv=2, S=900, D=128, sink=8, window=16)
    ra = workloads.research_attention(wl.stack, "bf16", DEV)
    q, k, v = (workloads.to_torch(a, "bf16", DEV) for a in (wl.q, wl.k, wl.v))
    meta = {}
    ra.build_mask(q, k[:, :, :600], v[:, :, :600], None, wl.scaling, 0.0, meta, layer_idx=0)
    m2 = ra.build_mask(q, k, v, None, wl.scaling, 0.0, meta, layer_idx=0)
    fresh = ra.build_mask(q, k, v, None, wl.scaling, 0.0, {}, layer_idx=0)
    a, b = m2.get_index_mask(), fresh.get_index_mask()
    assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])
    # and both are what the restatement selects on all 900 keys
    ref_mask, _, rmeta = stacks.run_stack(wl.stack, wl.q, wl.k, wl.v, wl.scaling, "bf16")
    _assert_mask_equal(m2, ref_mask)
    kc = meta["key"][0]
    np.testing.assert_array_equal(kc.codes[..., : kc.length].cpu().numpy().view(np.uint32), rmeta["hash_kcodes"])
    with pytest.raises(ValueError):
        ra.build_mask(q, k[:, :, :100], v[:, :, :100], None, wl.scaling, 0.0, meta, layer_idx=0)


def test_hash_with_attention_mask_blocking_keys():
    wl = workloads.hashattention_bf16(seed=24, B=2, Hq=4, Hkv=2, S=640, D=128, sink=8, window=16,
                                      heavy=64)
    am = np.zeros((2, 1, 1, 640), np.float32)
    am[0, :, :, 100:300] = -3.3895313892515355e38  # padded positions of batch 0
    mask, out, _ = _run_native(wl, attention_mask=am)
    ref_mask, ref_out, _ = stacks.run_stack(wl.stack, wl.q, wl.k, wl.v, wl.scaling, "bf16",
                                            attention_mask=am)
    _assert_mask_equal(mask, ref_mask)
    _close(out, ref_out, "bf16")


# ---------------------------------------------------------------------------
@pytest.mark.parametrize("dtype,seed", [("bf16", 31), ("f32", 32)])
def test_oracle_topk(dtype, seed):
    g = load_golden(f"oracle_topk_{dtype}")
    wl = workloads.oracle_topk(seed=seed, dtype=dtype, B=2, Hq=8, Hkv=2, S=1024, D=128, sink=16,
                               window=32, heavy=0.02)
    mask, out, _ = _run_native(wl)
    ref_mask, ref_out, rmeta = stacks.run_stack(wl.stack, wl.q, wl.k, wl.v, wl.scaling, dtype)
    # scores bit-exact against the restatement's fixed summation order
    q, k = (workloads.to_torch(a, dtype, DEV) for a in (wl.q, wl.k))
    s = _native_ops.qk_scores(q, k, None).float().cpu().numpy()
    np.testing.assert_array_equal(s, rmeta["oracle_scores"])
    _assert_mask_equal(mask, ref_mask)
    _close(out, ref_out, dtype)
    _close(out, g["out"], dtype, scale=2.0)
    # selection kernel on the reference's own score tensor reproduces its mask exactly
    prev = workloads.research_attention(wl.stack[:2], dtype, DEV).build_mask(
        q, k, k, None, wl.scaling, 0.0, {}, layer_idx=0)
    sc = workloads.to_torch(g["scores"], dtype, DEV)
    sel = _native_ops.topk_select(sc, prev, int(0.02 * 1024))
    _assert_mask_equal(Mask._from_native(tuple(sc.shape), workloads.torch_dtype(dtype), sel), golden=g)


def test_topk_select_ties_and_short_rows():
    S = 1000
    sc = torch.zeros((1, 3, 1, S), device=DEV)           # all equal: lowest columns win
    sc[0, 1, 0, 500:] = 1.0
    sc[0, 2, 0, ::7] = -0.0
    prev = Mask.create_empty_mask((1, 3, 1, S), torch.float32, torch.device(DEV))
    sel = Mask._from_native((1, 3, 1, S), torch.float32, _native_ops.topk_select(sc, prev, 37))
    dense = sel.get_dense_mask().cpu().numpy()[0, :, 0]
    assert dense[0, :37].all() and dense[0].sum() == 37
    assert dense[1, 500:537].all() and dense[1].sum() == 37
    assert dense[2, :37].all() and dense[2].sum() == 37
    everything = _native_ops.topk_select(sc, prev, 5000)  # k beyond the row: every candidate
    assert Mask._from_native((1, 3, 1, S), torch.float32, everything).get_density() == 1.0


@pytest.mark.parametrize("dtype,S,rows_h,k", [("bf16", 512, 40, 25), ("f32", 700, 9, 60), ("bf16", 5000, 5, 333),
                                              ("f32", 33, 3, 40)])
def test_topk_select_one_cta_per_row_equals_chunked(dtype, S, rows_h, k):
    """Both exact top-k paths give the same bitmap, previous mask and ties included."""
    rng = np.random.default_rng(S + k)
    x = rng.normal(size=(1, rows_h, 1, S)).astype(np.float32)
    x[0, 0, 0, : S // 2] = np.round(x[0, 0, 0, : S // 2])       # many ties
    sc = workloads.to_torch(workloads.to_dtype(x, dtype), dtype, DEV)
    shape = (1, rows_h, 1, S)
    prev_np = np.zeros(shape, np.float32)
    prev_np[..., :5] = 1.0
    tdt = torch.bfloat16 if dtype == "bf16" else torch.float32
    prev = Mask.create_mask_from_dense_mask(shape, torch.from_numpy(prev_np).to(DEV).to(tdt), tdt)
    a = _native_ops.topk_select(sc, prev, k)
    b = _native_ops.topk_select(sc, prev, k, per_row=True)
    assert torch.equal(a.bits, b.bits)
    from oracle import topk as ot
    want = ot.topk_inactive(sc.float().cpu().numpy(), prev_np != 0, k) | (prev_np != 0)
    got = Mask._from_native(shape, tdt, b).get_dense_mask().float().cpu().numpy() != 0
    np.testing.assert_array_equal(got, want)


# ---------------------------------------------------------------------------
def test_mask_conversions_round_trip():
    rng = np.random.default_rng(5)
    dense = (rng.random((2, 3, 2, 333)) < 0.2) * rng.random((2, 3, 2, 333))
    dense = workloads.to_dtype(dense.astype(np.float32), "bf16")
    t = workloads.to_torch(dense, "bf16", DEV)
    m = Mask.create_mask_from_dense_mask(t.shape, t, torch.bfloat16)
    idx, ptr, data = m.get_index_mask()
    ri, rp, rd = mask_ops.to_csr(dense)
    np.testing.assert_array_equal(idx.cpu().numpy(), ri)
    np.testing.assert_array_equal(ptr.cpu().numpy(), rp)
    np.testing.assert_array_equal(data.float().cpu().numpy(), rd)
    nb = m.native_bits()
    back = Mask._from_native(tuple(t.shape), torch.bfloat16, nb).get_dense_mask()
    assert torch.equal(back, t)


def test_weighted_mask_attention_matches_oracle():
    """Non-unit weights (sampling probabilities) enter numerator and denominator."""
    wl = workloads.sink_local_fp32(seed=41, B=2, Hq=8, Hkv=2, S=700, D=128)
    rng = np.random.default_rng(7)
    for dtype in ("f32", "bf16"):
        q, k, v = (workloads.to_dtype(a, dtype) for a in (wl.q, wl.k, wl.v))
        dense = np.where(rng.random((2, 8, 1, 700)) < 0.15, rng.uniform(0.05, 1.0, (2, 8, 1, 700)), 0.0)
        dense[..., :8] = 1.0
        dense = workloads.to_dtype(dense.astype(np.float32), dtype)
        tq, tk, tv = (workloads.to_torch(a, dtype, DEV) for a in (q, k, v))
        m = Mask.create_mask_from_dense_mask(dense.shape, workloads.to_torch(dense, dtype, DEV),
                                             workloads.torch_dtype(dtype))
        out = native_masked_attention(tq, tk, tv, None, None, float(wl.scaling), m)
        ref = o_attention.masked_attention(q, k, v, dense, wl.scaling, dtype)
        _close(out.float().cpu().numpy(), ref, dtype)


def test_full_and_empty_masks_mean_dense_attention():
    wl = workloads.sink_local_fp32(seed=42, B=1, Hq=8, Hkv=8, S=300, D=64)
    tq, tk, tv = (workloads.to_torch(a, "f32", DEV) for a in (wl.q, wl.k, wl.v))
    ref = o_attention.masked_attention(wl.q, wl.k, wl.v, None, wl.scaling, "f32", no_mask=True)
    for m in (Mask.create_full_mask((1, 8, 1, 300), torch.float32, torch.device(DEV)),
              Mask.create_empty_mask((1, 8, 1, 300), torch.float32, torch.device(DEV))):
        out = native_masked_attention(tq, tk, tv, None, None, float(wl.scaling), m)
        _close(out.cpu().numpy(), ref, "f32")


def test_partials_merge_equals_single_pass():
    """Sequence-sharded partials merged by the merge kernel equal the one-shot result."""
    from sparse_attention_hub.sparse_attention.utils.mask_attention_utils import merge_attention_partials

    wl = workloads.sink_local_fp32(seed=43, B=1, Hq=8, Hkv=2, S=1024, D=128, sink=32, window=64)
    tq, tk, tv = (workloads.to_torch(a, "f32", DEV) for a in (wl.q, wl.k, wl.v))
    rng = np.random.default_rng(3)
    dense = (rng.random((1, 8, 1, 1024)) < 0.1).astype(np.float32)
    full = Mask.create_mask_from_dense_mask(dense.shape, torch.from_numpy(dense).to(DEV), torch.float32)
    want = native_masked_attention(tq, tk, tv, None, None, float(wl.scaling), full)
    parts = []
    for lo, hi in ((0, 512), (512, 1024)):
        part = Mask.create_mask_from_dense_mask((1, 8, 1, hi - lo),
                                                torch.from_numpy(dense[..., lo:hi].copy()).to(DEV),
                                                torch.float32)
        _, p = native_masked_attention(tq, tk[:, :, lo:hi].contiguous(),
                                       tv[:, :, lo:hi].contiguous(), None, None,
                                       float(wl.scaling), part, return_partials=True)
        parts.append(p)
    got = merge_attention_partials(torch.stack(parts), 1, 8, 1, torch.float32)
    _close(got.cpu().numpy(), want.cpu().numpy(), "f32")
    # and the restatement's dense computation over all keys
    ref = o_attention.masked_attention(wl.q, wl.k, wl.v, dense, wl.scaling, "f32")
    _close(got.cpu().numpy(), ref, "f32")


def test_hash_topk_degenerate_score_distributions():
    """Rows whose scores are nothing like a binomial: all equal, two levels, all maximal."""
    S, k = 5000, 300
    shape = (1, 4, 1, S)
    rng = np.random.default_rng(9)
    q = np.array([[[0x0F0F0F0F], [0xFFFFFFFF], [0x12345678], [0]]], np.uint32)
    kc = np.empty((1, 4, S), np.uint32)
    kc[0, 0] = ~q[0, 0, 0]                      # every key scores 0 matching bits
    kc[0, 1] = q[0, 1, 0]                       # every key matches all 32 bits
    kc[0, 2] = np.where(rng.random(S) < 0.01, q[0, 2, 0], ~q[0, 2, 0])  # 1 % perfect, rest zero
    kc[0, 3] = rng.integers(0, 2 ** 32, S, dtype=np.uint64).astype(np.uint32)
    tk = torch.from_numpy(kc.view(np.int32)).to(DEV)
    tq = torch.from_numpy(q.view(np.int32)).to(DEV)
    prev = Mask.create_empty_mask(shape, torch.bfloat16, torch.device(DEV))
    sel = _native_ops.hash_topk(tk, S, tq, 32, None, torch.bfloat16, prev, k, shape)
    got = Mask._from_native(shape, torch.bfloat16, sel).get_dense_mask().float().cpu().numpy() != 0
    from oracle import hashattention as oh, topk as ot
    scores = oh.scores(q, kc, 32, "bf16")
    want = ot.topk_inactive(scores, np.zeros(shape, bool), k)
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("S,cap,rows_h,k,nbits,path", [
    (5000, 5003, 4, 300, 32, "row"),      # ragged tail, odd capacity: rows 1.. are not 16-byte aligned
    (5000, 5003, 4, 300, 32, "chunks"),
    (16384, 16384, 3, 512, 32, "row"),    # one word per thread
    (40000, 40960, 2, 1000, 16, "row"),   # two / four words per thread, 16-bit codes
    (40000, 40960, 2, 1000, 16, "chunks"),
    (70001, 70016, 2, 4000, 32, "row"),   # longer than the register-resident kernel takes
    (70001, 70016, 2, 4000, 32, "chunks"),
    (300000, 300000, 1, 9000, 32, "chunks"),
    (300000, 300000, 2, 9000, 32, "pieces"),  # two chunks per row: the byte counters flush several times
    (300000, 300000, 2, 9000, 32, "pieces_scratch"),  # the same with the one-byte score scratch
    (1500, 1500, 2, 0, 32, "row"),
    (1500, 1500, 2, 5000, 32, "chunks"),  # k above the number of candidates
])
def test_hash_topk_kernel_variants(S, cap, rows_h, k, nbits, path):
    """Every Hamming top-k kernel (one CTA per row: register-resident and streaming; chunked
    rows with the plan fused into the emit pass) against the same selection rule, with a
    previous mask in place and score ties cut in column order."""
    from oracle import hashattention as oh, topk as ot
    from sparse_attention_hub import _native
    lib = _native.load()
    rng = np.random.default_rng(S + k + nbits)
    shape = (1, rows_h, 1, S)
    mask_bits = np.uint64((1 << nbits) - 1)
    kc = np.zeros((1, rows_h, cap), np.uint32)
    kc[..., :S] = (rng.integers(0, 2 ** 32, (1, rows_h, S), dtype=np.uint64) & mask_bits).astype(np.uint32)
    kc[0, 0, : S // 2] &= np.uint32(0xFF)   # a row with few distinct scores: long tie runs
    q = (rng.integers(0, 2 ** 32, (1, rows_h, 1), dtype=np.uint64) & mask_bits).astype(np.uint32)
    prev_np = np.zeros(shape, bool)
    prev_np[..., :37] = True
    prev_np[..., S - 70:] = True
    prev_np[0, 0, 0, rng.integers(0, S, 200)] = True
    prev = Mask.create_mask_from_dense_mask(shape, torch.from_numpy(prev_np).to(DEV).to(torch.bfloat16),
                                            torch.bfloat16)
    pb = prev.native_bits()
    tk = torch.from_numpy(kc.view(np.int32)).to(DEV)
    tq = torch.from_numpy(q.view(np.int32)).to(DEV)
    out = torch.empty_like(pb.bits)
    st = _native.stream_of(tk.device)
    if path == "row":
        _native.check(lib.sah_hash_topk(tk.data_ptr(), cap, tq.data_ptr(), nbits, None, _native.SAH_BF16, 0, 0, 0,
                                        1, rows_h, 1, S, pb.words, pb.bits.data_ptr(), k, out.data_ptr(), st),
                      "sah_hash_topk")
    elif path in ("pieces", "pieces_scratch"):
        chunks = 2
        scratch = None
        if path == "pieces_scratch":
            scratch = torch.empty(int(lib.sah_hash_scores_bytes(pb.rows, pb.words)), dtype=torch.uint8, device=DEV)
        sp = None if scratch is None else scratch.data_ptr()
        hist = torch.empty((chunks, pb.rows, 33), dtype=torch.int32, device=DEV)
        thr = torch.empty((chunks, pb.rows), dtype=torch.int32, device=DEV)
        need = torch.empty((chunks, pb.rows), dtype=torch.int64, device=DEV)
        args = (tk.data_ptr(), cap, tq.data_ptr(), nbits, 1, rows_h, 1, S, pb.words, chunks, pb.bits.data_ptr())
        _native.check(lib.sah_hash_hist(*args, hist.data_ptr(), sp, st), "sah_hash_hist")
        _native.check(lib.sah_hash_shard_plan(hist.data_ptr(), 1, 0, chunks, pb.rows, k, thr.data_ptr(),
                                              need.data_ptr(), st), "sah_hash_shard_plan")
        _native.check(lib.sah_hash_emit(*args, thr.data_ptr(), need.data_ptr(), sp, out.data_ptr(), st),
                      "sah_hash_emit")
    else:
        sms = _native.sm_count(tk.device)
        nbytes = int(lib.sah_hash_topk_ws_bytes(pb.rows, pb.words, sms))
        ws = torch.empty(nbytes, dtype=torch.uint8, device=DEV)
        _native.check(lib.sah_hash_topk_ws(tk.data_ptr(), cap, tq.data_ptr(), nbits, 1, rows_h, 1, S, pb.words,
                                           pb.bits.data_ptr(), k, out.data_ptr(), ws.data_ptr(), nbytes, sms,
                                           st), "sah_hash_topk_ws")
    got = Mask._from_native(shape, torch.bfloat16, type(pb)(out, pb.rows, S)).get_dense_mask().float().cpu().numpy() != 0
    scores = oh.scores(q, kc[..., :S], nbits, "bf16")
    want = ot.topk_inactive(scores, prev_np, k) | prev_np
    np.testing.assert_array_equal(got, want)


def test_attention_with_sixteen_rows_per_group():
    """GQA ratio 16: every row of the 16-row tensor-core tile is a real query head."""
    wl = workloads.sink_local_fp32(seed=44, B=1, Hq=16, Hkv=1, S=1500, D=128, sink=8, window=40)
    rng = np.random.default_rng(11)
    for dtype in ("bf16", "f32"):
        q, k, v = (workloads.to_dtype(a, dtype) for a in (wl.q, wl.k, wl.v))
        dense = (rng.random((1, 16, 1, 1500)) < 0.2).astype(np.float32)
        dense[..., :8] = 1.0
        tq, tk, tv = (workloads.to_torch(a, dtype, DEV) for a in (q, k, v))
        m = Mask.create_mask_from_dense_mask(dense.shape, workloads.to_torch(dense, dtype, DEV),
                                             workloads.torch_dtype(dtype))
        out = native_masked_attention(tq, tk, tv, None, None, float(wl.scaling), m)
        ref = o_attention.masked_attention(q, k, v, dense, wl.scaling, dtype)
        _close(out.float().cpu().numpy(), ref, dtype)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["f32", "bf16"])
def test_gpu_mask_interop_from_rows_and_sparse_merge(dtype):
    """`Mask.create_from_row_wise_idx(mode="dense")` and `merge_mask(mode="sparse")` on device
    tensors run the library's scatter / flat-add kernels; both must give the reference's result
    bit for bit (duplicates inside a row: the last one stays; merged entries: summed in the mask
    dtype, clamped, every stored index kept)."""
    g = load_golden(f"mask_interop_{dtype}")
    td = workloads.torch_dtype(dtype)
    shape = tuple(g["row_dense"].shape)
    idx = torch.from_numpy(g["row_idx"]).to(DEV)
    vals = workloads.to_torch(g["row_vals"], dtype, DEV)
    m = Mask.create_from_row_wise_idx(shape, idx, vals, mask_type="dense", dtype=td, mode="dense")
    np.testing.assert_array_equal(m.get_dense_mask().float().cpu().numpy(), g["row_dense"])
    np.testing.assert_array_equal(m.get_dense_mask().float().cpu().numpy(),
                                  mask_ops.from_row_wise_idx(shape, g["row_idx"], g["row_vals"]))

    def index_form(dense):
        d = Mask.create_mask_from_dense_mask(shape, workloads.to_torch(dense, dtype, DEV), td)
        i, p, v = d.get_index_mask()
        return Mask.create_mask_from_indices(shape, i, p, v, td)

    merged = index_form(g["a"]).merge_mask(index_form(g["b"]), inplace=False, mode="sparse")
    mi, mp, md = merged.get_index_mask()
    np.testing.assert_array_equal(mi.cpu().numpy(), g["merged_idx"])
    np.testing.assert_array_equal(mp.cpu().numpy(), g["merged_ptr"])
    np.testing.assert_array_equal(md.float().cpu().numpy(), g["merged_data"])
    oi, op, od = mask_ops.merge_sparse(g["a"], g["b"], dtype)
    np.testing.assert_array_equal(mi.cpu().numpy(), oi)
    np.testing.assert_array_equal(md.float().cpu().numpy(), od)


@pytest.mark.gpu
@pytest.mark.parametrize("hidden,layers,bits,act", [(128, 3, 32, "silu"), (64, 2, 16, "relu"), (32, 3, 32, "gelu")])
def test_hash_signatures_from_tensor_cores_equal_the_fixed_order_kernel(hidden, layers, bits, act,
                                                                        monkeypatch):
    """On request (SAH_HASH_TC=1) ranges of 1024 keys and more are hashed with the layers'
    products on the tensor cores and every output near a bfloat16 rounding midpoint redone in the
    fixed order; shorter ranges take the fixed-order kernel.  Hashing 6000 keys in one call and in
    slices of 1000 must give the same words -- and those are the restatement's codes."""
    monkeypatch.setenv("SAH_HASH_TC", "1")
    S, B, Hkv, Hq, D = 6000, 2, 2, 4, 128
    w = workloads.hat_weights(31 + hidden, Hq, D, hidden, bits, layers)
    rng = np.random.default_rng(3)
    w["key_bias"] = [(rng.standard_normal(b.shape) * 0.1).astype(np.float32) for b in w["key_bias"]]
    k = workloads.to_dtype((rng.standard_normal((B, Hkv, S, D)) * 0.8).astype(np.float32), "bf16")
    tk = workloads.to_torch(k, "bf16", DEV)
    weights = [workloads.to_torch(a, "bf16", DEV).contiguous() for a in w["key_matrix"]]
    biases = [workloads.to_torch(a, "bf16", DEV).contiguous() for a in w["key_bias"]]
    whole = torch.zeros((B, Hq, S), dtype=torch.int32, device=DEV)
    sliced = torch.zeros_like(whole)
    _native_ops.hash_encode(tk, Hq, weights, biases, act, whole, 0, S)
    for s0 in range(0, S, 1000):
        _native_ops.hash_encode(tk, Hq, weights, biases, act, sliced, s0, min(S, s0 + 1000))
    torch.cuda.synchronize()
    assert torch.equal(whole, sliced)
    n = 256
    mats = [workloads.to_dtype(a, "bf16") for a in w["key_matrix"]]
    bias = [workloads.to_dtype(a, "bf16") for a in w["key_bias"]]
    ref = o_hash.signatures(o_attention.repeat_kv(k[:, :, :n], Hq // Hkv), mats, bias, act, "bf16")
    np.testing.assert_array_equal(whole[:, :, :n].cpu().numpy().view(np.uint32), ref)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,widths,n0,n,act", [
    ("bf16", (128, 128, 128, 32), 0, 17, "silu"), ("bf16", (128, 128, 128, 32), 5, 128, "silu"),
    ("bf16", (64, 32, 16), 3, 129, "relu"), ("bf16", (72, 16, 64, 128, 32), 0, 300, "tanh"),
    ("bf16", (128, 128, 128, 128, 32), 0, 257, "gelu"), ("bf16", (128, 128, 128, 32), 0, 12000, "silu"),
    ("f32", (128, 128, 128, 32), 1, 255, "silu"), ("f32", (8, 16), 0, 130, "relu"),
    ("bf16", (128, 128, 128, 32), 2, 592, "silu"), ("bf16", (128, 128, 128, 32), 0, 593, "silu"),
    ("bf16", (128, 128, 128, 128, 32), 3, 700, "relu"), ("bf16", (128, 128, 128, 32), 0, 1153, "silu"),
    ("f32", (64, 32, 16), 0, 1186, "tanh")])
def test_hash_signatures_of_tiles_equal_those_of_single_vectors(dtype, widths, n0, n, act):
    """Ranges of more than 16 vectors go through tiles of 32 (weights of all layers resident in
    shared memory, or layer by layer where they do not fit; one, two or four tiles of a head as the
    unit that CTAs share, and several units per CTA), shorter ones one vector per CTA.  Both walk the channels in the same order: the same words, and words
    outside the range untouched."""
    torch.manual_seed(sum(widths) + n)
    B, Hkv, Hq, S = 2, 2, 4, n0 + n + 3
    dt = torch.bfloat16 if dtype == "bf16" else torch.float32
    k = torch.randn((B, S, Hkv, widths[0]), device=DEV).to(dt).transpose(1, 2)
    weights = [(torch.randn((Hq, a, b), device=DEV) / a ** 0.5).to(dt) for a, b in zip(widths, widths[1:])]
    biases = [(torch.randn((Hq, b), device=DEV) * 0.1).to(dt) for b in widths[1:]]
    whole = torch.full((B, Hq, S + 5), -7, dtype=torch.int32, device=DEV)
    single = whole.clone()
    _native_ops.hash_encode(k, Hq, weights, biases, act, whole, n0, n0 + n)
    for s0 in range(n0, n0 + n, 16):
        _native_ops.hash_encode(k, Hq, weights, biases, act, single, s0, min(n0 + n, s0 + 16))
    assert torch.equal(whole, single)


@pytest.mark.gpu
@pytest.mark.parametrize("rows,S,k,b0,b1,dtype", [
    (1, 131072, 2048, 64, 131072, "bf16"), (3, 16385, 300, 0, 16385, "f32"), (30, 8200, 82, 5, 8190, "bf16"),
    (70, 4097, 1, 0, 4097, "f32"), (200, 519, 26, 0, 519, "bf16"), (2, 33, 32, 31, 33, "bf16"),
    (5, 70000, 70000, 0, 70000, "bf16"), (4, 9000, 0, 0, 9000, "f32"), (2, 700000, 5000, 0, 700000, "bf16")])
def test_topk_select_over_cluster_sizes(rows, S, k, b0, b1, dtype):
    """Rows cut between 8, 4, 2 and 1 CTAs (and, for the longest, over the whole grid or with the
    keys read again in every pass): the restatement's set, ties in column order across the cuts,
    both signs of zero, column bounds inside a byte of the bitmap."""
    from oracle import topk as o_topk

    rng = np.random.default_rng(S + k)
    x = rng.standard_normal((1, rows, 1, S)).astype(np.float32)
    x[0, 0] = np.round(x[0, 0] * 2) / 2                  # a few hundred-fold ties, +0 and -0
    x[0, rows - 1, 0, S // 3:] = 1.5                       # the cut inside one long run
    dt = torch.bfloat16 if dtype == "bf16" else torch.float32
    sc = torch.from_numpy(x).to(DEV).to(dt)
    active = rng.random((1, rows, 1, S)) < 0.05
    prev = Mask.create_mask_from_dense_mask((1, rows, 1, S), torch.from_numpy(active.astype(np.float32)).to(DEV),
                                            torch.float32)
    want = o_topk.topk_inactive(sc.float().cpu().numpy(), active, k, b0, b1) | active
    for per_row in (False, True):
        sel = _native_ops.topk_select(sc, prev, k, b0, b1, per_row=per_row)
        got = Mask._from_native((1, rows, 1, S), torch.float32, sel).get_dense_mask().cpu().numpy() != 0
        np.testing.assert_array_equal(got, want)


@pytest.mark.gpu
@pytest.mark.parametrize("B,Hq,Sq,S,k,dtype", [(1, 4, 1, 20000, 700, "bf16"), (2, 3, 24, 1031, 60, "bf16"),
                                               (1, 5, 2, 260, 9, "f32")])
def test_hash_topk_under_an_additive_mask(B, Hq, Sq, S, k, dtype):
    """Hamming scores plus an additive mask (rounded to the dtype): rows over clusters, ragged
    lengths, a mask shared by the heads with the lowest value, -inf and small offsets."""
    from oracle import topk as o_topk

    rng = np.random.default_rng(S)
    dt = torch.bfloat16 if dtype == "bf16" else torch.float32
    cap = S + 3
    kc = rng.integers(0, 2 ** 32, (B, Hq, cap), dtype=np.uint32)
    kc[..., : S // 2] &= np.uint32(0xFF)
    qc = rng.integers(0, 2 ** 32, (B, Hq, Sq), dtype=np.uint32)
    am = torch.zeros((B, 1, Sq, S))
    am[:, :, 0, S // 2: S // 2 + 50] = torch.finfo(dt).min
    am[..., 7] = -float("inf")
    am[..., 9] = 0.75
    am = am.to(dt).to(DEV)
    pop = np.array([bin(i).count("1") for i in range(65536)], np.int64)
    d = kc[:, :, None, :S] ^ qc[..., None]
    score = (32 - 2 * (pop[d & 0xFFFF] + pop[d >> 16])).astype(np.float32)
    biased = (torch.from_numpy(score).to(DEV) + am.float()).to(dt).float().cpu().numpy()
    active = rng.random((B, Hq, Sq, S)) < 0.1
    prev = Mask.create_mask_from_dense_mask(active.shape, torch.from_numpy(active.astype(np.float32)).to(DEV), dt)
    sel = _native_ops.hash_topk(torch.from_numpy(kc.view(np.int32)).to(DEV), S,
                                torch.from_numpy(qc.view(np.int32)).to(DEV), 32, am, dt, prev, k, (B, Hq, Sq, S))
    got = Mask._from_native(active.shape, dt, sel).get_dense_mask().float().cpu().numpy() != 0
    np.testing.assert_array_equal(got, o_topk.topk_inactive(biased, active, k) | active)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["bf16", "f32"])
@pytest.mark.parametrize("B,Hq,Hkv,Sq,S,D,masked", [
    (1, 4, 1, 1, 1, 128, False), (2, 3, 3, 1, 17, 128, True), (1, 16, 2, 1, 1003, 128, False),
    (1, 6, 2, 3, 333, 64, True), (3, 2, 2, 1, 64, 64, False), (1, 8, 2, 24, 79, 128, True),
    (1, 4, 2, 2, 140, 80, True), (1, 6, 2, 1, 1601, 64, True), (1, 8, 8, 1, 30000, 128, False),
    (1, 32, 8, 1, 19001, 128, False), (1, 32, 8, 1, 19100, 128, True), (2, 32, 8, 1, 9700, 64, False),
    (2, 16, 8, 2, 9770, 64, True), (1, 32, 8, 2, 18945, 128, False)])
def test_score_bits_at_the_edges(dtype, B, Hq, Hkv, Sq, S, D, masked):
    """q.k bit for bit in the fixed order: group sizes that are no multiple of four, key counts
    around the ends of a CTA's tile, more rows than stay in registers, head dims that are and are not
    compiled in, strided keys and queries; and, in the last five in bfloat16, two keys per thread (rows in
    fours, 592 CTAs of 256 keys or more) with a last tile of 1, 42, 57, 156 and 228 keys, of which a thread's
    second one may lie past the end."""
    torch.manual_seed(S + D)
    dt = torch.bfloat16 if dtype == "bf16" else torch.float32
    q = torch.randn((B, Sq, Hq, D), device=DEV).to(dt).transpose(1, 2)
    k = torch.randn((B, S, Hkv, D + 8), device=DEV).to(dt)[..., :D].transpose(1, 2)
    am = None
    if masked:
        am = torch.zeros((B, 1, Sq, S + 3), device=DEV).to(dt)
        am[:, :, 0, S // 2:] = torch.finfo(dt).min
        am[..., 0] = 0.37
    got = _native_ops.qk_scores(q, k, am).float().cpu().numpy()
    n = min(S, 1100)  # the ends of a long row
    cols = np.r_[0:n, S - n:S]
    want = o_qk.qk_scores(q.float().cpu().numpy(), k[:, :, cols].float().cpu().numpy(), dtype,
                          None if am is None else am[..., cols].float().cpu().numpy())
    np.testing.assert_array_equal(got[..., cols], want)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,S,Sq,stack", [
    ("f32", 700, 1, "fixed"), ("bf16", 131, 3, "fixed"), ("bf16", 32768, 1, "fixed"), ("bf16", 33000, 2, "fixed"),
    ("bf16", 4097, 1, "topk"), ("f32", 1000, 4, "topk"), ("bf16", 90000, 1, "topk"), ("bf16", 260, 2, "topk"),
    ("bf16", 20001, 4, "topk"), ("f32", 40000, 2, "topk")])
def test_band_masks_without_a_bitmap(dtype, S, Sq, stack, monkeypatch):
    """A mask of bands alone (sink and window, the future cleared for several query positions) goes
    to the selection and to the attention plan as bands: the same masks and the same output as
    with the bitmap filled first.  The words of the mask that was handed over are written by the
    kernel that took the bands, on its stream: whoever reads them afterwards, on whatever stream
    that waited for the call, finds them without a launch of its own."""
    from sparse_attention_hub import _native
    from sparse_attention_hub.sparse_attention.utils.mask import NativeBits

    taken = []
    pending = NativeBits.pending_bands

    def noted(self):
        bands = pending(self)
        if bands is not None:
            taken.append(self)
        return bands

    monkeypatch.setattr(NativeBits, "pending_bands", noted)

    torch.manual_seed(S)
    dt = torch.bfloat16 if dtype == "bf16" else torch.float32
    q = torch.randn((2, 4, Sq, 64), device=DEV).to(dt)
    k, v = (torch.randn((2, 2, S, 64), device=DEV).to(dt) for _ in range(2))
    maskers = [("sink", {"sink_size": 5}), ("local", {"window_size": 37})]
    if stack == "topk":
        maskers.append(("oracle_topk", {"heavy_size": 0.05}))
    ra = workloads.research_attention(maskers, dtype, DEV)

    def run():
        mask = ra.build_mask(q, k, v, None, 0.125, 0.0, {}, layer_idx=0)
        out = get_masked_attention_output(None, q, k, v, None, None, 0.125, 0.0, mask)
        before = _native.launch_count()
        mask.native_bits().bits
        assert _native.launch_count() == before
        return out, mask.get_dense_mask()

    out, dense = run()
    # longer rows go through a bitmap, as does a selection that is faster over the whole grid
    assert (S in (33000, 90000)) == (not taken)
    monkeypatch.setattr(NativeBits, "pending_bands", lambda self: None)
    want_out, want_dense = run()
    fixed = workloads.research_attention(maskers[:2], dtype, DEV)
    fixed_dense = fixed.build_mask(q, k, v, None, 0.125, 0.0, {}, layer_idx=0).get_dense_mask()
    assert torch.equal(dense, want_dense)
    assert torch.equal(out, want_out)
    for bits in taken:
        before = _native.launch_count()
        words = bits.bits
        assert _native.launch_count() == before
        got = Mask._from_native((2, 4, Sq, S), dt, NativeBits(words, bits.rows, S)).get_dense_mask()
        assert torch.equal(got, fixed_dense)
        assert bool((words[:, (S + 31) // 32:] == 0).all())


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,Hq,Hkv,Sq,S,D,bias", [
    ("bf16", 8, 2, 5, 700, 128, True), ("bf16", 4, 1, 17, 129, 128, False), ("f32", 3, 1, 11, 257, 64, True),
    ("bf16", 2, 2, 33, 40, 64, True), ("f32", 8, 1, 6, 128, 80, False), ("bf16", 8, 1, 2, 300, 128, True),
    ("bf16", 4, 1, 5, 40001, 128, True), ("f32", 1, 1, 17, 30001, 64, False), ("f32", 3, 1, 11, 70000, 128, False)])
def test_scores_of_many_rows_equal_those_of_one_position(dtype, Hq, Hkv, Sq, S, D, bias):
    """Rows per KV head that are cut into blocks (20, 68, 33, 33, 48 and 16 of them), that stay together on a grid of
    more CTAs (20 and 17) and that are cut there too (33): the scores of every position are those of a call for that position alone, bit for bit."""
    import torch
    from sparse_attention_hub import _native

    lib = _native.load()
    dev = torch.device("cuda:0")
    dt = torch.bfloat16 if dtype == "bf16" else torch.float32
    gen = torch.Generator(device=dev).manual_seed(S + Sq)
    q = torch.randn((2, Hq, Sq, D), generator=gen, device=dev).to(dt)
    k = torch.randn((2, Hkv, S, D), generator=gen, device=dev).to(dt)
    am = torch.randn((2, 1, Sq, S), generator=gen, device=dev).to(dt) if bias else None

    def scores(lo, hi):
        out = torch.full((2, Hq, hi - lo, S), float("nan"), dtype=dt, device=dev)
        qs = q[:, :, lo:hi]
        b = (None, 0, 0, 0) if am is None else (am[:, :, lo:hi].data_ptr(), am.stride(0), 0, am.stride(2))
        _native.check(lib.sah_qk_scores(qs.data_ptr(), k.data_ptr(), _native.dtype_code(dt), *qs.stride()[:3],
                                        *k.stride()[:3], 2, Hq, Hkv, hi - lo, S, D, *b, out.data_ptr(),
                                        _native.stream_of(dev)), "sah_qk_scores")
        return out

    together = scores(0, Sq)
    for i in range(Sq):
        assert torch.equal(together[:, :, i:i + 1], scores(i, i + 1))
