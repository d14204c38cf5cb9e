"""PQCache: numpy restatement vs the reference's fixtures (CPU) and CUDA path vs both (GPU).

Integer results (codes, index sets) are compared bit for bit.  k-means is compared in lock
step: from the reference's own initial centres one Lloyd iteration must give the same
assignment and centres within 1e-5; after five iterations a handful of boundary keys may sit
in a different cluster because the reference sums cluster members in fp32 in its own order
(bounded below).  The decode step is compared on the reference-built codebook, where it must
reproduce the reference mask exactly.
"""

import numpy as np
import pytest

from oracle import mask_ops, pq, stacks
import workloads

from conftest import load_golden

N_SUB, CENT, OFF = 16, 16, 4


def _workload():
    return workloads.pqcache(seed=41, dtype="bf16", B=1, Hq=8, Hkv=2, S=600, D=128, sink=4,
                             window=16, heavy=32, group_factor=16, bits=4, kmeans_iter=5,
                             n_clusters=16)


def _check_mask(mask, g, prefix):
    idx, ptr, data = mask_ops.to_csr(mask)
    np.testing.assert_array_equal(idx, g[prefix + "idx"])
    np.testing.assert_array_equal(ptr, g[prefix + "ptr"])
    np.testing.assert_array_equal(data, g[prefix + "data"])


# ------------------------------------------------------------------ CPU: oracle vs reference
def test_kmeans_lock_step_against_reference():
    g = load_golden("pq_kmeans_lockstep")
    wl = _workload()
    X = pq.split_keys(wl.k, OFF, N_SUB)
    init = X[np.arange(X.shape[0])[:, None], g["init_idx"]]
    reseed = [g["reseed"]] * 5  # the draws the reference was handed, one table per iteration
    codes1, cent1 = pq.kmeans(X, init, 1, reseed)
    np.testing.assert_array_equal(codes1, g["codes1"])
    # the reference returns centres cast to the key dtype
    np.testing.assert_allclose(workloads.to_dtype(cent1, "bf16"), g["centers1"], atol=1e-5, rtol=8e-3)
    codes5, cent5 = pq.kmeans(X, init, 5, reseed)
    assert np.mean(codes5 != g["codes5"]) < 5e-3
    np.testing.assert_allclose(workloads.to_dtype(cent5, "bf16"), g["centers5"], atol=2e-2, rtol=2e-2)


def test_pq_decode_exact_on_reference_codebook():
    g = load_golden("pq_stack_bf16")
    wl = _workload()
    n_first = 592 - OFF
    codes = g["codes_first"].transpose(0, 2, 1, 3)  # [B,n,Hkv,n_sub] -> [B,Hkv,n,n_sub]
    meta = {"pq_centroids": g["centroids"], "pq_codes": codes}
    mask, out, _ = stacks.run_stack(wl.stack, wl.q, wl.k[:, :, :592], wl.v[:, :, :592], wl.scaling,
                                    "bf16", meta=meta)
    assert codes.shape[2] == n_first
    _check_mask(mask, g, "first_")
    np.testing.assert_allclose(out, g["first_out"], atol=2e-2, rtol=2e-2)


def test_pq_appended_keys_quantised_like_reference():
    g = load_golden("pq_stack_bf16")
    wl = _workload()
    X_new = pq.split_keys(wl.k[:, :, 592:], 0, N_SUB)
    C = g["centroids"].reshape(-1, CENT, 8)
    new_codes = pq.assign(X_new, C, dtype_math="bf16").reshape(1, 2, N_SUB, 8).transpose(0, 1, 3, 2)
    want = g["codes_after_append"].transpose(0, 2, 1, 3)[:, :, 588:]
    np.testing.assert_array_equal(new_codes, want)
    meta = {"pq_centroids": g["centroids"],
            "pq_codes": g["codes_after_append"].transpose(0, 2, 1, 3)}
    mask, out, _ = stacks.run_stack(wl.stack, wl.q, wl.k, wl.v, wl.scaling, "bf16", meta=meta)
    _check_mask(mask, g, "append_")
    np.testing.assert_allclose(out, g["append_out"], atol=2e-2, rtol=2e-2)


# ------------------------------------------------------------------ GPU: kernels vs oracle / reference
def _native_stack(wl, meta):
    import torch
    from sparse_attention_hub.sparse_attention.utils.mask_attention_utils import get_masked_attention_output

    dev = "cuda:0"
    ra = workloads.research_attention(wl.stack, wl.dtype, dev)
    q, k, v = (workloads.to_torch(a, wl.dtype, dev) for a in (wl.q, wl.k, wl.v))
    mask = ra.build_mask(q, k, v, None, float(wl.scaling), 0.0, meta, layer_idx=0)
    out = get_masked_attention_output(None, q, k, v, None, None, float(wl.scaling), 0.0, mask)
    torch.cuda.synchronize()
    idx, ptr, data = mask.get_index_mask()
    return (idx.cpu().numpy(), ptr.cpu().numpy(), data.float().cpu().numpy()), out.float().cpu().numpy()


@pytest.mark.gpu
def test_gpu_kmeans_build_matches_oracle_bit_for_bit():
    import torch

    wl = _workload()
    groups = 1 * 2 * N_SUB
    init_idx = workloads.pq_init_indices(43, groups, 600 - OFF, CENT)
    reseed = np.random.default_rng(43).integers(0, 600 - OFF, size=(5, groups, CENT)).astype(np.int64)
    meta = {"pq_init_indices": {0: torch.from_numpy(init_idx)},
            "pq_reseed_indices": {0: torch.from_numpy(reseed)}}
    (idx, ptr, data), out = _native_stack(wl, meta)
    ometa = {"pq_init_indices": init_idx, "pq_reseed_indices": reseed}
    ref_mask, ref_out, ometa = stacks.run_stack(wl.stack, wl.q, wl.k, wl.v, wl.scaling, "bf16", meta=ometa)
    got_codes = meta["pq_codebook"][0].codes[:, :, : 600 - OFF].cpu().numpy()
    np.testing.assert_array_equal(got_codes, ometa["pq_codes"])
    np.testing.assert_array_equal(meta["pq_centroids"][0].float().cpu().numpy(), ometa["pq_centroids"])
    ri, rp, rd = mask_ops.to_csr(ref_mask)
    np.testing.assert_array_equal(idx, ri)
    np.testing.assert_array_equal(ptr, rp)
    np.testing.assert_allclose(out, ref_out, atol=2e-2, rtol=2e-2)


@pytest.mark.gpu
def test_gpu_decode_and_append_on_reference_codebook():
    import torch

    g = load_golden("pq_stack_bf16")
    wl = _workload()
    dev = "cuda:0"
    meta = {"pq_centroids": {0: workloads.to_torch(g["centroids"], "bf16", dev)},
            "pq_codebook": {0: torch.from_numpy(g["codes_first"]).to(dev)},  # reference layout
            "pq_ip2l2_phi": {0: None}}
    short = workloads.DecodeWorkload(wl.name, wl.dtype, wl.q, wl.k[:, :, :592], wl.v[:, :, :592],
                                     wl.scaling, wl.stack)
    (idx, ptr, data), out = _native_stack(short, meta)
    np.testing.assert_array_equal(idx, g["first_idx"])
    np.testing.assert_array_equal(ptr, g["first_ptr"])
    np.testing.assert_allclose(out, g["first_out"], atol=2e-2, rtol=2e-2)
    # eight keys appended: quantised against the stored centroids, then the same stack
    (idx, ptr, data), out = _native_stack(wl, meta)
    codes = meta["pq_codebook"][0].to_reference_layout().cpu().numpy()
    np.testing.assert_array_equal(codes, g["codes_after_append"])
    np.testing.assert_array_equal(idx, g["append_idx"])
    np.testing.assert_array_equal(ptr, g["append_ptr"])
    np.testing.assert_allclose(out, g["append_out"], atol=2e-2, rtol=2e-2)


@pytest.mark.gpu
@pytest.mark.parametrize("n_cent,n_keys", [(256, 20000), (16, 3000), (48, 777)])
def test_gpu_assignment_on_tensor_cores_equals_the_fixed_order_kernel(n_cent, n_keys):
    """`sah_pq_assign_tc` (tcgen05 distance contraction, fixed-order argmin among the near-minimal
    centroids) writes the codes of `sah_pq_assign`, including ties (duplicated centroids and keys
    that sit exactly on centroids) -- and those are the restatement's codes."""
    import torch
    from sparse_attention_hub import _native

    lib = _native.load()
    dev = "cuda:0"
    B, Hkv, n_sub, sub_d, off = 2, 2, 16, 8, 5
    D, S = n_sub * sub_d, n_keys + off
    gen = torch.Generator(device=dev).manual_seed(n_cent)
    keys = (torch.randn((B, Hkv, S, D), generator=gen, device=dev) * 1.5).to(torch.bfloat16)
    groups = B * Hkv * n_sub
    cent = torch.randn((groups, n_cent, sub_d), generator=gen, device=dev) * 1.2
    cent[:, 3] = cent[:, 1]                       # a duplicated centroid: the lower index must win
    sub = keys[:, :, off:].reshape(B, Hkv, n_keys, n_sub, sub_d)
    cent.view(B, Hkv, n_sub, n_cent, sub_d)[:, :, :, 5] = sub[:, :, 7].float()   # a key on a centroid
    cent = cent.contiguous()
    cap = n_keys + 11
    want = torch.full((B, Hkv, cap, n_sub), 255, dtype=torch.uint8, device=dev)
    got = torch.full_like(want, 254)
    err = torch.zeros(1, dtype=torch.int32, device=dev)
    st = _native.stream_of(torch.device(dev))
    _native.check(lib.sah_pq_assign(keys.data_ptr(), _native.SAH_BF16, keys.stride(0), keys.stride(1), keys.stride(2),
                                    B, Hkv, off, S, off, n_sub, sub_d, n_cent, cent.data_ptr(), want.data_ptr(), cap,
                                    0, st), "sah_pq_assign")
    _native.check(lib.sah_pq_assign_tc(keys.data_ptr(), keys.stride(0), keys.stride(1), keys.stride(2), B, Hkv, off,
                                       S, off, n_sub, sub_d, n_cent, cent.data_ptr(), got.data_ptr(), cap,
                                       err.data_ptr(), 148, st), "sah_pq_assign_tc")
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    assert torch.equal(got[:, :, :n_keys], want[:, :, :n_keys])
    assert bool((got[:, :, n_keys:] == 254).all())
    # the restatement on a slice
    n = min(n_keys, 400)
    X = pq.split_keys(keys[:, :, : off + n].float().cpu().numpy(), off, n_sub)
    codes = pq.assign(X, cent.cpu().numpy()).reshape(B, Hkv, n_sub, n).transpose(0, 1, 3, 2)
    np.testing.assert_array_equal(got[:, :, :n].cpu().numpy(), codes)


# ------------------------------------------------------------------ metric "ip"
def _ip_workload():
    wl = workloads.pqcache(seed=45, dtype="bf16", B=1, Hq=8, Hkv=2, S=600, D=128, sink=4, window=16,
                           heavy=32, group_factor=N_SUB, bits=4, kmeans_iter=5, n_clusters=16)
    wl.stack[-1][1]["metric"] = "ip"
    return wl


def test_pq_ip_metric_restatement_equals_the_reference():
    """The inner-product metric (utils/pq_utils.py:585-640): augmented clustering, scores on the
    first sub_d centroid columns -- phi, centroids, codes, index sets and output of the reference."""
    g = load_golden("pq_stack_ip_bf16")
    wl = _ip_workload()
    meta = {"pq_init_indices": g["init_idx"],
            "pq_reseed_indices": np.broadcast_to(g["reseed"], (5,) + g["reseed"].shape)}
    mask, out, meta = stacks.run_stack(wl.stack, wl.q, wl.k[:, :, :592], wl.v[:, :, :592], wl.scaling, "bf16",
                                       meta=meta)
    np.testing.assert_array_equal(meta["pq_ip2l2_phi"].reshape(-1), g["phi"].reshape(-1))
    np.testing.assert_array_equal(meta["pq_centroids"], g["centroids"])
    np.testing.assert_array_equal(meta["pq_codes"].transpose(0, 2, 1, 3), g["codes_first"])
    _check_mask(mask, g, "first_")
    np.testing.assert_allclose(out, g["first_out"], atol=2e-2, rtol=2e-2)


def test_pq_two_batches_two_query_positions_against_the_reference():
    """Reference fixture with B = 2 and Sq = 2 (euclidean): centroids, codes, index sets and output
    of the restatement are the reference's."""
    g = load_golden("pq_stack_bf16_sq2")
    wl = workloads.pqcache(seed=47, dtype="bf16", B=2, Hq=4, Hkv=2, S=400, D=128, sink=4, window=16,
                           heavy=24, group_factor=N_SUB, bits=4, kmeans_iter=5, n_clusters=16, Sq=2)
    meta = {"pq_init_indices": g["init_idx"],
            "pq_reseed_indices": np.broadcast_to(g["reseed"], (5,) + g["reseed"].shape)}
    mask, out, meta = stacks.run_stack(wl.stack, wl.q, wl.k, wl.v, wl.scaling, "bf16", meta=meta)
    np.testing.assert_array_equal(meta["pq_centroids"], g["centroids"])
    np.testing.assert_array_equal(meta["pq_codes"].transpose(0, 2, 1, 3), g["codes_first"])
    _check_mask(mask, g, "first_")
    np.testing.assert_allclose(out, g["first_out"], atol=2e-2, rtol=2e-2)


@pytest.mark.gpu
def test_gpu_ip_metric_build_decode_and_append_equal_the_reference():
    import torch

    g = load_golden("pq_stack_ip_bf16")
    wl = _ip_workload()
    reseed = np.broadcast_to(g["reseed"], (5,) + g["reseed"].shape).copy()
    meta = {"pq_init_indices": {0: torch.from_numpy(g["init_idx"])},
            "pq_reseed_indices": {0: torch.from_numpy(reseed)}}
    short = workloads.DecodeWorkload(wl.name, wl.dtype, wl.q, wl.k[:, :, :592], wl.v[:, :, :592],
                                     wl.scaling, wl.stack)
    (idx, ptr, data), out = _native_stack(short, meta)
    np.testing.assert_array_equal(meta["pq_ip2l2_phi"][0].float().cpu().numpy().reshape(-1), g["phi"].reshape(-1))
    np.testing.assert_array_equal(meta["pq_centroids"][0].float().cpu().numpy(), g["centroids"])
    np.testing.assert_array_equal(meta["pq_codebook"][0].to_reference_layout().cpu().numpy(), g["codes_first"])
    np.testing.assert_array_equal(idx, g["first_idx"])
    np.testing.assert_array_equal(ptr, g["first_ptr"])
    np.testing.assert_allclose(out, g["first_out"], atol=2e-2, rtol=2e-2)
    # eight appended keys: a zero column instead of the augmentation (pq_top_k.py:371-383)
    (idx, ptr, data), out = _native_stack(wl, meta)
    np.testing.assert_array_equal(meta["pq_codebook"][0].to_reference_layout().cpu().numpy(),
                                  g["codes_after_append"])
    np.testing.assert_array_equal(idx, g["append_idx"])
    np.testing.assert_array_equal(ptr, g["append_ptr"])
    np.testing.assert_allclose(out, g["append_out"], atol=2e-2, rtol=2e-2)


@pytest.mark.gpu
@pytest.mark.parametrize("n_sub,n_cent,n_keys", [(16, 256, 1), (16, 64, 129), (4, 128, 300), (6, 256, 255), (3, 32, 128),
                                                 (16, 256, 1281), (16, 16, 1200), (8, 64, 2600), (4, 128, 9700)])
def test_gpu_assignment_tile_edges_and_layouts(n_sub, n_cent, n_keys):
    """`sah_pq_assign_tc` at the edges of its tiles (one key, a tile, a tile and one), for every
    padded centroid count and with one sub-vector per CTA or (the last four) four, on integer-valued keys and
    centroids (many exact ties): the codes of `sah_pq_assign`."""
    import torch
    from sparse_attention_hub import _native

    lib = _native.load()
    dev = "cuda:0"
    B, Hkv, off = 1, 2, 3
    gen = torch.Generator(device=dev).manual_seed(n_cent + n_keys)
    keys = torch.randint(-3, 4, (B, Hkv, n_keys + off, n_sub * 8), generator=gen, device=dev).to(torch.bfloat16)
    cent = torch.randint(-3, 4, (B * Hkv * n_sub, n_cent, 8), generator=gen, device=dev).float()
    cap, st = n_keys + 2, _native.stream_of(torch.device(dev))
    want = torch.full((B, Hkv, cap, n_sub), 255, dtype=torch.uint8, device=dev)
    got = want.clone()
    err = torch.zeros(1, dtype=torch.int32, device=dev)
    strides = (keys.stride(0), keys.stride(1), keys.stride(2))
    _native.check(lib.sah_pq_assign(keys.data_ptr(), _native.SAH_BF16, *strides, B, Hkv, off, n_keys + off, off, n_sub, 8,
                                    n_cent, cent.data_ptr(), want.data_ptr(), cap, 0, st), "sah_pq_assign")
    _native.check(lib.sah_pq_assign_tc(keys.data_ptr(), *strides, B, Hkv, off, n_keys + off, off, n_sub, 8, n_cent,
                                       cent.data_ptr(), got.data_ptr(), cap, err.data_ptr(), 148, st), "sah_pq_assign_tc")
    torch.cuda.synchronize()
    assert int(err.item()) == 0 and torch.equal(got, want)


@pytest.mark.gpu
@pytest.mark.parametrize("n_sub,n_cent", [(16, 256), (4, 128), (6, 64), (3, 32)])
def test_gpu_assignment_with_many_near_ties(n_sub, n_cent):
    """Stretches of a few distinct keys (centroids that are their copies, or nearly), of zeros and of keys far from
    0 with little spread, between stretches of ordinary ones, all tiles in two CTAs.  The codes of `sah_pq_assign`."""
    import torch
    from sparse_attention_hub import _native

    lib = _native.load()
    dev = "cuda:0"
    B, Hkv, off, n_keys = 1, 2, 3, 4300
    gen = torch.Generator(device=dev).manual_seed(n_cent)
    keys = torch.randn((B, Hkv, n_keys + off, n_sub * 8), generator=gen, device=dev).to(torch.bfloat16)
    keys[:, :, 600:1900] = keys[:, :, torch.randint(0, 9, (1300,), generator=gen, device=dev)]
    keys[:, :, 2500:3600] = keys[:, :, 2500:3600] * 0.5 + 64.0
    keys[:, :, 3700:3900] = 0.0
    groups = B * Hkv * n_sub
    sub = keys.view(B * Hkv, n_keys + off, n_sub, 8).transpose(1, 2).reshape(groups, n_keys + off, 8).float()
    pick = torch.randint(0, n_keys + off, (groups, n_cent), generator=gen, device=dev)
    pick[:, ::3] = torch.randint(0, 9, (groups, (n_cent + 2) // 3), generator=gen, device=dev)
    cent = torch.gather(sub, 1, pick[..., None].expand(-1, -1, 8)).contiguous()
    cent[:, ::9] *= 1.0 + 2.0 ** -23
    cap, st = n_keys + 2, _native.stream_of(torch.device(dev))
    want = torch.full((B, Hkv, cap, n_sub), 255, dtype=torch.uint8, device=dev)
    got = want.clone()
    err = torch.zeros(1, dtype=torch.int32, device=dev)
    strides = (keys.stride(0), keys.stride(1), keys.stride(2))
    _native.check(lib.sah_pq_assign(keys.data_ptr(), _native.SAH_BF16, *strides, B, Hkv, off, n_keys + off, off, n_sub, 8,
                                    n_cent, cent.data_ptr(), want.data_ptr(), cap, 0, st), "sah_pq_assign")
    _native.check(lib.sah_pq_assign_tc(keys.data_ptr(), *strides, B, Hkv, off, n_keys + off, off, n_sub, 8, n_cent,
                                       cent.data_ptr(), got.data_ptr(), cap, err.data_ptr(), 2, st), "sah_pq_assign_tc")
    torch.cuda.synchronize()
    assert int(err.item()) == 0 and torch.equal(got, want)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,n_sub,sub_d,n_keys,n_cent", [
    ("bf16", 16, 8, 1, 32), ("bf16", 16, 8, 4097, 32), ("bf16", 4, 9, 5000, 32), ("f32", 3, 16, 4096, 32),
    ("f32", 2, 5, 9000, 32), ("bf16", 16, 8, 4200, 256), ("f32", 2, 8, 4099, 129), ("bf16", 2, 8, 5001, 128),
    ("bf16", 4, 8, 4301, 16), ("f32", 2, 6, 4301, 9), ("bf16", 2, 8, 130, 8), ("f32", 1, 3, 4099, 8)])
def test_gpu_cluster_sums_equal_float64_sums(dtype, n_sub, sub_d, n_keys, n_cent):
    """`sah_pq_accumulate`: counts exact, and float64 sums that round to the float32 sums of numpy's
    float64 additions (values are multiples of 2^-8 below 8, so float64 sums are exact in any
    order); one cluster holds half of the keys and one none.  From 129 centroids on a pair of threads has
    a centroid to itself, with 9 to 16 of them a warp has one, with 8 two warps share one."""
    import torch
    from sparse_attention_hub import _native

    lib = _native.load()
    dev = "cuda:0"
    B, Hkv, off = 2, 1, 2
    gen = torch.Generator(device=dev).manual_seed(n_keys)
    keys = (torch.randint(-2047, 2048, (B, Hkv, n_keys + off, n_sub * sub_d), generator=gen, device=dev) / 256.0)
    keys = keys.to(workloads.torch_dtype(dtype))
    cap = n_keys + 3
    codes = torch.randint(0, n_cent - 1, (B, Hkv, cap, n_sub), generator=gen, device=dev)
    codes[:, :, ::2] = 7
    codes = codes.to(torch.uint8)
    groups = B * Hkv * n_sub
    sums = torch.zeros((groups, n_cent, sub_d), dtype=torch.float64, device=dev)
    counts = torch.zeros((groups, n_cent), dtype=torch.int32, device=dev)
    _native.check(lib.sah_pq_accumulate(keys.data_ptr(), _native.dtype_code(keys.dtype), keys.stride(0), keys.stride(1),
                                        keys.stride(2), B, Hkv, n_keys, off, n_sub, sub_d, n_cent, codes.data_ptr(), cap,
                                        sums.data_ptr(), counts.data_ptr(), _native.stream_of(torch.device(dev))),
                  "sah_pq_accumulate")
    x = keys.double().cpu().numpy()[:, :, off:].reshape(B * Hkv, n_keys, n_sub, sub_d)
    c = codes.cpu().numpy()[:, :, :n_keys].reshape(B * Hkv, n_keys, n_sub)
    want, cnt = np.zeros((groups, n_cent, sub_d)), np.zeros((groups, n_cent), np.int64)
    for g in range(groups):
        np.add.at(want[g], c[g // n_sub, :, g % n_sub], x[g // n_sub, :, g % n_sub])
        cnt[g] = np.bincount(c[g // n_sub, :, g % n_sub], minlength=n_cent)
    np.testing.assert_array_equal(counts.cpu().numpy(), cnt)
    np.testing.assert_array_equal(sums.cpu().numpy(), want)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["bf16", "f32"])
@pytest.mark.parametrize("n_sub,sub_d,n_cent,math", [(16, 8, 256, 1), (3, 5, 33, 0), (1, 16, 1, 1), (4, 9, 31, 0)])
def test_gpu_few_appended_keys_equal_the_tile_kernel(dtype, n_sub, sub_d, n_cent, math):
    """Up to 16 keys are quantised by a warp per sub-vector, longer ranges by a thread per key: the
    same codes, equal distances (duplicated centroids) and not-a-number keys included."""
    import torch
    from sparse_attention_hub import _native

    lib = _native.load()
    dev = "cuda:0"
    dt = torch.bfloat16 if dtype == "bf16" else torch.float32
    B, Hkv, S, off = 2, 3, 40, 2
    torch.manual_seed(n_cent)
    x = torch.randn((B, Hkv, S, n_sub * sub_d), device=dev).to(dt)
    x[:, :, 11, :] = float("nan")
    cent = torch.randn((B * Hkv * n_sub, n_cent, sub_d), device=dev).to(dt).float()
    cent[:, n_cent // 2:] = cent[:, :n_cent - n_cent // 2].clone()
    st = _native.stream_of(torch.device(dev))

    def assign(codes, s0, s1):
        _native.check(lib.sah_pq_assign(x.data_ptr(), _native.dtype_code(dt), x.stride(0), x.stride(1), x.stride(2),
                                        B, Hkv, s0, s1, off, n_sub, sub_d, n_cent, cent.data_ptr(), codes.data_ptr(),
                                        S, math, st), "sah_pq_assign")

    whole = torch.full((B, Hkv, S, n_sub), 77, dtype=torch.uint8, device=dev)
    parts = whole.clone()
    assign(whole, off, S)
    for s0, s1 in ((off, off + 1), (off + 1, off + 17), (off + 17, off + 20), (off + 20, off + 36), (off + 36, S)):
        assign(parts, s0, s1)
    assert torch.equal(whole, parts)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,n_sub,sub_d,n_cent,S", [("bf16", 3, 8, 33, 700), ("bf16", 1, 16, 255, 40),
                                                        ("bf16", 5, 5, 1, 300), ("f32", 3, 4, 7, 90)])
def test_gpu_scores_with_odd_tables(dtype, n_sub, sub_d, n_cent, S):
    """`sah_pq_scores` with an odd number of table entries (8 bytes each in bfloat16: the queries
    behind them start on the next 16-byte boundary): table entries summed over ascending channels and
    rounded, an entry per sub-vector added in float32 and rounded once."""
    import torch
    from oracle.bf16 import round_bf16
    from sparse_attention_hub import _native

    lib = _native.load()
    dev = "cuda:0"
    dt = workloads.torch_dtype(dtype)
    rnd = round_bf16 if dtype == "bf16" else (lambda a: a.astype(np.float32))
    B, Hq, Hkv, Sq, off = 2, 6, 2, 1, 3
    gen = torch.Generator(device=dev).manual_seed(n_cent)
    # multiples of 1/8 below 4: every product and partial sum is exact in float32
    q = (torch.randint(-31, 32, (B, Hq, Sq, n_sub * sub_d), generator=gen, device=dev) / 8.0).to(dt)
    cent = (torch.randint(-31, 32, (B * Hkv * n_sub, n_cent, sub_d), generator=gen, device=dev) / 8.0).to(dt)
    codes = torch.randint(0, n_cent, (B, Hkv, S, n_sub), generator=gen, device=dev).to(torch.uint8)
    got = torch.zeros((B, Hq, Sq, S), dtype=dt, device=dev)
    _native.check(lib.sah_pq_scores(q.data_ptr(), _native.dtype_code(dt), q.stride(0), q.stride(1), q.stride(2),
                                    cent.data_ptr(), codes.data_ptr(), S, B, Hq, Hkv, Sq, S - off, off, S, n_sub, sub_d,
                                    n_cent, got.data_ptr(), None, 0, _native.stream_of(torch.device(dev))), "sah_pq_scores")
    qn = q.float().cpu().numpy().reshape(B, Hkv, Hq // Hkv, n_sub, sub_d)
    cn = cent.float().cpu().numpy().reshape(B, Hkv, n_sub, n_cent, sub_d)
    table = rnd(np.einsum("bhgsd,bhscd->bhgsc", qn, cn).astype(np.float32)).astype(np.float32)
    want = np.zeros((B, Hkv, Hq // Hkv, S - off), np.float32)
    c = codes.cpu().numpy()[:, :, :S - off].astype(np.int64)
    for s in range(n_sub):
        want += np.take_along_axis(table[:, :, :, s], np.broadcast_to(c[:, :, None, :, s], want.shape), axis=3)
    np.testing.assert_array_equal(got.float().cpu().numpy()[..., off:].reshape(want.shape), rnd(want))
    assert bool((got[..., :off] == 0).all())


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,n_sub,sub_d,n_cent", [("bf16", 2, 32, 40), ("f32", 3, 17, 33), ("bf16", 4, 16, 256),
                                                      ("f32", 1, 50, 300)])
def test_gpu_centres_of_wide_subvectors(dtype, n_sub, sub_d, n_cent):
    """`sah_pq_accumulate` and `sah_pq_update` with sub-vectors of up to and over 16 channels (and,
    for the sums, more centroids than a byte can name): exact sums and counts; every channel of every
    centre replaced, empty clusters by their key, and the moves of all channels in `shift2`."""
    import torch
    from sparse_attention_hub import _native

    lib = _native.load()
    dev = "cuda:0"
    B, Hkv, n_keys = 1, 2, 4500
    dt = workloads.torch_dtype(dtype)
    gen = torch.Generator(device=dev).manual_seed(sub_d)
    # multiples of 1/16 below 16 (8 significant bits): sums are exact in any order
    keys = (torch.randint(-255, 256, (B, Hkv, n_keys, n_sub * sub_d), generator=gen, device=dev) / 16.0).to(dt)
    used = min(n_cent, 256) - 1                      # the last centroid that a code names stays empty
    codes = torch.randint(0, used, (B, Hkv, n_keys, n_sub), generator=gen, device=dev).to(torch.uint8)
    groups = B * Hkv * n_sub
    sums = torch.zeros((groups, n_cent, sub_d), dtype=torch.float64, device=dev)
    counts = torch.zeros((groups, n_cent), dtype=torch.int32, device=dev)
    st = _native.stream_of(torch.device(dev))
    kargs = (keys.data_ptr(), _native.dtype_code(dt), keys.stride(0), keys.stride(1), keys.stride(2), B, Hkv)
    _native.check(lib.sah_pq_accumulate(*kargs, n_keys, 0, n_sub, sub_d, n_cent, codes.data_ptr(), n_keys,
                                        sums.data_ptr(), counts.data_ptr(), st), "sah_pq_accumulate")
    x = keys.double().cpu().numpy().reshape(B * Hkv, n_keys, n_sub, sub_d)
    c = codes.cpu().numpy().reshape(B * Hkv, n_keys, n_sub)
    want, cnt = np.zeros((groups, n_cent, sub_d)), np.zeros((groups, n_cent), np.int64)
    for g in range(groups):
        np.add.at(want[g], c[g // n_sub, :, g % n_sub], x[g // n_sub, :, g % n_sub])
        cnt[g] = np.bincount(c[g // n_sub, :, g % n_sub], minlength=n_cent)
    np.testing.assert_array_equal(counts.cpu().numpy(), cnt)
    np.testing.assert_array_equal(sums.cpu().numpy(), want)
    if n_cent > 256:
        return
    cent = torch.randn((groups, n_cent, sub_d), generator=gen, device=dev)
    reseed = torch.randint(0, n_keys, (groups, n_cent), generator=gen, device=dev)
    new, shift2 = cent.clone(), torch.zeros(groups, device=dev)
    _native.check(lib.sah_pq_update(*kargs, 0, n_sub, sub_d, n_cent, sums.data_ptr(), counts.data_ptr(),
                                    reseed.data_ptr(), new.data_ptr(), shift2.data_ptr(), st), "sah_pq_update")
    g = np.arange(groups)[:, None]
    seeds = x[g // n_sub, reseed.cpu().numpy(), g % n_sub].astype(np.float32)
    mean = want.astype(np.float32) / np.maximum(cnt, 1).astype(np.float32)[..., None]
    centres = np.where(cnt[..., None] > 0, mean, seeds).astype(np.float32)
    np.testing.assert_array_equal(new.cpu().numpy(), centres)
    moves = np.sqrt(((centres.astype(np.float64) - cent.double().cpu().numpy()) ** 2).sum(-1)).sum(-1) ** 2
    # float32 sums of sub_d squares and of n_cent roots, squared: within (sub_d + 2 n_cent) 2^-23 < 1e-4
    np.testing.assert_allclose(shift2.cpu().numpy(), moves, rtol=1e-4)


@pytest.mark.gpu
@pytest.mark.parametrize("n_cent,scale", [(16, 2.0 ** 52), (48, 2.0 ** 60), (80, 2.0 ** -40), (256, 2.0 ** 60)])
def test_gpu_assignment_of_keys_far_from_one(n_cent, scale):
    """Columns that pad the centroids of `sah_pq_assign_tc` to a power of two lie below every
    centroid's, whatever the keys' magnitude: the codes of `sah_pq_assign`."""
    import torch
    from sparse_attention_hub import _native

    lib = _native.load()
    dev = "cuda:0"
    B, Hkv, n_sub, n_keys = 1, 2, 4, 700
    gen = torch.Generator(device=dev).manual_seed(n_cent)
    keys = (torch.randn((B, Hkv, n_keys, n_sub * 8), generator=gen, device=dev) * scale).to(torch.bfloat16)
    cent = (torch.randn((B * Hkv * n_sub, n_cent, 8), generator=gen, device=dev) + 3.0) * scale
    st = _native.stream_of(torch.device(dev))
    want = torch.full((B, Hkv, n_keys, n_sub), 255, dtype=torch.uint8, device=dev)
    got = want.clone()
    err = torch.zeros(1, dtype=torch.int32, device=dev)
    strides = (keys.stride(0), keys.stride(1), keys.stride(2))
    _native.check(lib.sah_pq_assign(keys.data_ptr(), _native.SAH_BF16, *strides, B, Hkv, 0, n_keys, 0, n_sub, 8, n_cent,
                                    cent.data_ptr(), want.data_ptr(), n_keys, 0, st), "sah_pq_assign")
    _native.check(lib.sah_pq_assign_tc(keys.data_ptr(), *strides, B, Hkv, 0, n_keys, 0, n_sub, 8, n_cent,
                                       cent.data_ptr(), got.data_ptr(), n_keys, err.data_ptr(), 148, st),
                  "sah_pq_assign_tc")
    assert int(err.item()) == 0 and torch.equal(got, want)
    assert len(torch.unique(want)) > 4


@pytest.mark.gpu
@pytest.mark.parametrize("n_cent", [16, 32, 64, 112, 256])
def test_gpu_assignment_of_ties_and_non_finite_keys(n_cent):
    """`sah_pq_assign_tc` where a key's row of the product holds several equal maxima (centroids given
    twice, keys of zero) and where margins are infinite or NaN: the codes of `sah_pq_assign`."""
    import torch
    from sparse_attention_hub import _native

    lib = _native.load()
    dev = "cuda:0"
    B, Hkv, n_sub, n_keys = 1, 2, 8, 515
    gen = torch.Generator(device=dev).manual_seed(n_cent)
    keys = torch.randn((B, Hkv, n_keys, n_sub * 8), generator=gen, device=dev).to(torch.bfloat16)
    keys[:, :, 3] = 0.0
    keys[:, :, 130, 5] = float("nan")
    keys[:, :, 257, 9] = float("inf")
    keys[:, :, 514, 17] = -float("inf")
    cent = torch.randn((B * Hkv * n_sub, n_cent, 8), generator=gen, device=dev)
    cent[:, n_cent // 2:] = cent[:, :n_cent // 2].flip(1)
    cent[1, n_cent // 3, 2] = float("inf")
    cent[2, n_cent - 1, 2] = float("nan")
    cent[3] = 0.0
    st = _native.stream_of(torch.device(dev))
    want = torch.full((B, Hkv, n_keys, n_sub), 255, dtype=torch.uint8, device=dev)
    got = want.clone()
    err = torch.zeros(1, dtype=torch.int32, device=dev)
    strides = (keys.stride(0), keys.stride(1), keys.stride(2))
    _native.check(lib.sah_pq_assign(keys.data_ptr(), _native.SAH_BF16, *strides, B, Hkv, 0, n_keys, 0, n_sub, 8, n_cent,
                                    cent.data_ptr(), want.data_ptr(), n_keys, 0, st), "sah_pq_assign")
    _native.check(lib.sah_pq_assign_tc(keys.data_ptr(), *strides, B, Hkv, 0, n_keys, 0, n_sub, 8, n_cent,
                                       cent.data_ptr(), got.data_ptr(), n_keys, err.data_ptr(), 148, st),
                  "sah_pq_assign_tc")
    assert int(err.item()) == 0 and torch.equal(got, want)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,n_keys,given,iters", [("bf16", 700, True, 6), ("bf16", 40, False, 8), ("f32", 300, False, 3),
                                                      ("bf16", 40, True, 8)])
def test_gpu_lloyd_iterations_launched_together(dtype, n_keys, given, iters):
    """The clustering of a build equals its steps called one after the other with the host's test for
    convergence between them (40 keys for 16 centres converge after a few iterations), and the
    generator has made as many draws."""
    import torch
    from sparse_attention_hub import _native
    from sparse_attention_hub.sparse_attention.research_attention.maskers.fixed import PQCache, PQCacheConfig

    lib = _native.load()
    dev = torch.device("cuda:0")
    B, Hkv, n_sub, n_cent, off = 1, 2, 4, 16, 8
    dt = torch.bfloat16 if dtype == "bf16" else torch.float32
    gen = torch.Generator(device=dev).manual_seed(n_keys)
    keys = torch.randn((B, Hkv, n_keys + off, n_sub * 8), generator=gen, device=dev).to(dt)
    groups, st = B * Hkv * n_sub, _native.stream_of(dev)
    init = torch.rand((groups, n_keys), generator=gen, device=dev).topk(n_cent, dim=1).indices
    draws = [torch.randint(0, n_keys, (groups, n_cent), generator=gen, device=dev) for _ in range(iters)]

    torch.manual_seed(5)
    rows = keys[:, :, off:].reshape(B * Hkv, n_keys, n_sub, 8).transpose(1, 2).reshape(groups, n_keys, 8).float()
    cent = torch.gather(rows, 1, init[..., None].expand(-1, -1, 8)).contiguous()
    codes = torch.zeros((B, Hkv, n_keys, n_sub), dtype=torch.uint8, device=dev)
    args = (keys.data_ptr(), _native.dtype_code(dt), keys.stride(0), keys.stride(1), keys.stride(2), B, Hkv)
    shift2 = torch.empty(groups, device=dev)
    ran = 0
    for it in range(iters):
        _native.check(lib.sah_pq_assign(*args, off, off + n_keys, off, n_sub, 8, n_cent, cent.data_ptr(),
                                        codes.data_ptr(), n_keys, 0, st), "sah_pq_assign")
        sums = torch.zeros((groups, n_cent, 8), dtype=torch.float64, device=dev)
        counts = torch.zeros((groups, n_cent), dtype=torch.int32, device=dev)
        _native.check(lib.sah_pq_accumulate(*args, n_keys, off, n_sub, 8, n_cent, codes.data_ptr(), n_keys,
                                            sums.data_ptr(), counts.data_ptr(), st), "sah_pq_accumulate")
        reseed = draws[it] if given else torch.randint(0, n_keys, (groups, n_cent), device=dev)
        _native.check(lib.sah_pq_update(*args, off, n_sub, 8, n_cent, sums.data_ptr(), counts.data_ptr(),
                                        reseed.data_ptr(), cent.data_ptr(), shift2.data_ptr(), st), "sah_pq_update")
        ran += 1
        if bool((shift2 < 1e-4).all()):
            break
    generator = torch.cuda.get_rng_state(dev)
    assert (ran < iters) == (n_keys == 40)

    torch.manual_seed(5)
    masker = PQCache(PQCacheConfig(heavy_size=8, pq_group_factor=n_sub, pq_bits=4, kmeans_iter=iters, init_offset=off,
                                   metric="euclidean"))
    meta = {"pq_init_indices": {0: init}}
    if given:
        meta["pq_reseed_indices"] = {0: draws[:ran]}  # no more than are needed
    masker._initialize_pq_cache(meta, 0)
    got_cent, got_codes = masker._perform_kmeans_clustering(keys, 0, meta)
    assert torch.equal(got_codes.codes[:, :, :n_keys], codes)
    assert torch.equal(got_cent.reshape(groups, n_cent, 8), cent.to(dt))
    assert torch.equal(torch.cuda.get_rng_state(dev), generator)
    if given:
        meta["pq_reseed_indices"] = {0: draws[:ran - 1]}
        with pytest.raises(IndexError):
            masker._perform_kmeans_clustering(keys, 0, meta)


@pytest.mark.gpu
def test_gpu_clustering_goes_no_further_than_it_has_to(monkeypatch):
    """Forty keys for sixteen centres: the clustering converges after a few of its hundred iterations.  No more
    than one assignment is launched in vain, no index drawn in vain, and the generator is never set back (another
    thread may have drawn from it meanwhile)."""
    import torch
    from sparse_attention_hub import _native
    from sparse_attention_hub.sparse_attention.research_attention.maskers.fixed import PQCache, PQCacheConfig

    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(1)
    keys = torch.randn((1, 2, 48, 32), generator=gen, device=dev).bfloat16()
    masker = PQCache(PQCacheConfig(heavy_size=8, pq_group_factor=4, pq_bits=4, kmeans_iter=100, init_offset=8,
                                   metric="euclidean"))
    init = torch.rand((8, 40), generator=gen, device=dev).topk(16, dim=1).indices
    draw, draws = torch.randint, []

    def counted(*args, **kwargs):
        draws.append(draw(*args, **kwargs))
        return draws[-1]

    def refused(*args, **kwargs):
        raise AssertionError("the generator was set back")

    monkeypatch.setattr(torch, "randint", counted)
    monkeypatch.setattr(torch.cuda, "set_rng_state", refused)
    meta = {"pq_init_indices": {0: init}}
    masker._initialize_pq_cache(meta, 0)
    before = _native.launch_count()
    masker._perform_kmeans_clustering(keys, 0, meta)
    assert 1 <= len(draws) < 20
    assert _native.launch_count() - before <= 3 * (len(draws) + 1)
