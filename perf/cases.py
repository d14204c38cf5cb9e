"""The work that users of this framework have it do, as measurable cases.

A user reaches the framework in two ways.  The Hugging Face adapter hook calls
`ResearchAttention.custom_attention` for every layer and token ("generate" and "step" cases:
plain calls, with the additive mask that the adapter's eager-mask hands over where there is
one); a serving loop captures a decode step once and replays it (`DecodeStepGraph`, "replay"
cases).  Stacks, shapes and key distributions are those of the benchmark configurations, of
`workloads.py` and of the tests: Llama-3-8B's heads (32/8, head dimension 128) and the smaller
and wider GQA layouts that the tests use.

A case is {"kind", "stack", "dtype", "B", "Hq", "Hkv", "D", "S"} and, for "generate", "question"
(query positions of the first call) and "tokens" (decode calls after it).
"""

import os
import sys
from math import ceil, sqrt

import torch

_PACKAGE = os.path.join(os.getcwd(), "sparse-attention-hub_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

from sparse_attention_hub.sparse_attention.research_attention import (  # noqa: E402
    ResearchAttention, ResearchAttentionConfig)
from sparse_attention_hub.sparse_attention.research_attention.decode_graph import (  # noqa: E402
    DecodeStepGraph)
from sparse_attention_hub.sparse_attention.research_attention.maskers import (  # noqa: E402
    fixed, sampling)
from sparse_attention_hub.sparse_attention.research_attention.maskers.fixed import (  # noqa: E402
    implementations as fixed_impl)
from sparse_attention_hub.sparse_attention.research_attention.maskers.sampling import (  # noqa: E402
    implementations as sampling_impl)

_DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16}
_PQ = {"heavy": 2048, "subspaces": 16, "bits": 8, "iterations": 10}
_LSH = {"tables": 75, "bits": 8}
_HASH = {"hidden": 128, "bits": 32}


def _case(name, kind, stack, dtype, B, Hq, Hkv, D, S, question=0, tokens=0):
    c = {"name": name, "kind": kind, "stack": stack, "dtype": dtype, "B": B, "Hq": Hq, "Hkv": Hkv, "D": D, "S": S}
    if kind == "generate":
        c.update(question=question, tokens=tokens)
    return c


def listed():
    return [
        # the smallest call: one fp32 layer of a short context, StreamingLLM-like stack, plain call
        _case("step_sink_local_f32_4k", "step", "sink_local", "f32", 1, 32, 8, 128, 4096),
        # fp32 exact top-k of one sequence, plain call
        _case("step_topk_f32_16k", "step", "oracle_topk", "f32", 1, 32, 8, 128, 16384),
        # batched serving steps, replayed: signatures, pages, exact top-p, sampling with guarantees
        _case("replay_hash_32k_b8", "replay", "hashattention", "bf16", 8, 32, 8, 128, 32768),
        _case("replay_quest_32k_b8", "replay", "quest", "bf16", 8, 32, 8, 128, 32768),
        _case("replay_adaptive_64k_b4", "replay", "oracle_adaptive", "bf16", 4, 32, 8, 128, 65536),
        _case("replay_topp_64k_b4", "replay", "oracle_topp", "bf16", 4, 32, 8, 128, 65536),
        # one long sequence, replayed: product-quantised top-k and LSH sampling at a million keys
        _case("replay_pq_128k", "replay", "pqcache", "bf16", 1, 32, 8, 128, 131072),
        _case("replay_magicpig_1m", "replay", "magicpig", "bf16", 1, 32, 8, 128, 1048576),
        # one layer's share of answering a question over a context, as the adapter does it: fresh
        # state, the question's positions in one call under a causal mask (index build over the
        # prompt), then token by token with the cache growing; a ragged prompt length in the first
        _case("generate_topk_8k", "generate", "oracle_topk", "bf16", 1, 32, 8, 128, 8191, 24, 8),
        _case("generate_hash_16k", "generate", "hashattention", "bf16", 1, 32, 8, 128, 16384, 16, 8),
        _case("generate_pq_64k", "generate", "pqcache", "bf16", 1, 32, 8, 128, 65536, 16, 8),
        _case("generate_magicpig_64k", "generate", "magicpig", "bf16", 1, 32, 8, 128, 65500, 16, 8),
    ]


# (kind, stack) -> (dtypes, smallest keys, largest keys, most B * max(Hq, 4 * Hkv) * keys)
_RANGES = {
    ("step", "sink_local"): (("f32", "bf16"), 1024, 32768, 1 << 22),
    ("step", "oracle_topk"): (("f32",), 2048, 32768, 1 << 20),
    ("replay", "hashattention"): (("bf16",), 4096, 131072, 1 << 23),
    ("replay", "quest"): (("bf16",), 4096, 131072, 1 << 23),
    ("replay", "oracle_adaptive"): (("bf16",), 8192, 131072, 1 << 23),
    ("replay", "oracle_topp"): (("bf16",), 8192, 131072, 1 << 23),
    ("replay", "pqcache"): (("bf16",), 16384, 131072, 1 << 22),
    ("replay", "magicpig"): (("bf16",), 16384, 1048576, 1 << 25),
    ("generate", "oracle_topk"): (("bf16",), 2048, 16384, 1 << 19),
    ("generate", "hashattention"): (("bf16",), 4096, 32768, 1 << 19),
    ("generate", "pqcache"): (("bf16",), 8192, 65536, 1 << 21),
    ("generate", "magicpig"): (("bf16",), 8192, 65536, 1 << 21),
}


def draw(rng):
    while True:
        kind, stack = rng.choice(sorted(_RANGES))
        dtypes, lo, hi, most = _RANGES[kind, stack]
        # Llama-3-8B's heads mostly; multi-head, 2:1 and (where no weights per key are
        # evaluated in the kernel) 8:1 groups, as the tests have them
        heads = [(32, 8), (32, 8), (8, 2), (16, 8), (8, 8)]
        if stack != "magicpig":
            heads.append((64, 8))
        Hq, Hkv = rng.choice(heads)
        B = rng.choice((1, 1, 2, 4, 8)) if kind != "generate" else 1
        S = int(round(lo * (hi / lo) ** rng.random()))
        S -= rng.choice((0, 0, S % 64, S % 1024))
        D = 128 if rng.random() < 0.8 or stack in ("pqcache", "hashattention") else 64
        if B * max(Hq, 4 * Hkv) * S > most or S < lo:
            continue
        c = _case("", kind, stack, rng.choice(dtypes), B, Hq, Hkv, D, S, rng.randint(4, 32), rng.randint(2, 16))
        del c["name"]
        return c


# ---- inputs -----------------------------------------------------------------------------------
def _keys_values(case, gen, total, device):
    """K and V [B, Hkv, total, D]: iid with outlier channels (sink_local), a planted heavy direction
    per KV group (hashattention), Gaussian clusters (the rest); also the query direction if any."""
    B, Hkv, D, dt = case["B"], case["Hkv"], case["D"], _DTYPES[case["dtype"]]
    randn = lambda *s: torch.randn(s, generator=gen, device=device)  # noqa: E731
    k = torch.empty((B, Hkv, total, D), dtype=dt, device=device)
    v = torch.empty_like(k)
    clusters = 256 if case["stack"] == "pqcache" else 64
    centres = randn(2, B, Hkv, clusters, D)
    direction = torch.nn.functional.normalize(randn(B, Hkv, 1, D), dim=-1)
    outliers = torch.randperm(D, generator=gen, device=device)[:4]
    bi = torch.arange(B, device=device)[:, None, None]
    hi = torch.arange(Hkv, device=device)[None, :, None]
    for s in range(0, total, 65536):
        e = min(total, s + 65536)
        kc, vc = randn(B, Hkv, e - s, D), randn(B, Hkv, e - s, D)
        if case["stack"] == "sink_local":
            kc[..., outliers] *= 8.0
        elif case["stack"] == "hashattention":  # one key of a hundred at cosine 0.6 with the queries
            norm = kc.norm(dim=-1, keepdim=True)
            perp = torch.nn.functional.normalize(kc - (kc * direction).sum(-1, keepdim=True) * direction, dim=-1)
            planted = torch.rand((B, Hkv, e - s, 1), generator=gen, device=device) < 0.01
            kc = torch.where(planted, norm * (0.6 * direction + 0.8 * perp), kc)
        else:
            pick = torch.randint(0, clusters, (B, Hkv, e - s), generator=gen, device=device)
            kc = centres[0][bi, hi, pick] + 0.3 * kc
            vc = centres[1][bi, hi, pick] + 0.3 * vc
        k[:, :, s:e], v[:, :, s:e] = kc.to(dt), vc.to(dt)
    return k, v, direction


def _queries(case, gen, n, direction, device):
    B, Hq, Hkv, D = case["B"], case["Hq"], case["Hkv"], case["D"]
    q = torch.randn((B, Hq, n, D), generator=gen, device=device)
    if case["stack"] == "hashattention":
        d = direction.repeat_interleave(Hq // Hkv, dim=1)
        q = sqrt(D) * torch.nn.functional.normalize(d + 0.3 * torch.nn.functional.normalize(q, dim=-1), dim=-1)
    return q.to(_DTYPES[case["dtype"]])


def _hash_weights(case, gen, device):
    D, H, dt = case["D"], case["Hq"], _DTYPES[case["dtype"]]
    dims = [D, _HASH["hidden"], _HASH["hidden"], _HASH["bits"]]
    w = {}
    for side in ("query", "key"):
        w[side + "_matrix"] = [(torch.randn((H, a, b), generator=gen, device=device) / sqrt(a)).to(dt)
                               for a, b in zip(dims, dims[1:])]
        w[side + "_bias"] = [torch.zeros((H, b), dtype=dt, device=device) for b in dims[1:]]
    return {0: w}


def _attention(case, gen, device):
    stack = case["stack"]
    long_ctx = stack in ("pqcache", "magicpig")
    sink, window = (64, 256) if long_ctx else (128, 256 if stack == "sink_local" else 512)
    maskers = [fixed.SinkMaskerConfig(sink_size=sink), fixed.LocalMaskerConfig(window_size=window)]
    if stack == "hashattention":
        maskers.append(fixed.HashAttentionTopKMaskerConfig(
            heavy_size=0.05, hat_bits=_HASH["bits"], hat_mlp_layers=3, hat_mlp_hidden_size=_HASH["hidden"],
            hat_mlp_activation="silu", hat_weights=_hash_weights(case, gen, device)))
    elif stack in ("oracle_topk", "oracle_adaptive"):
        maskers.append(fixed.OracleTopKConfig(heavy_size=0.02))
        if stack == "oracle_adaptive":
            maskers.append(sampling_impl.AdaptiveSamplingMaskerConfig(
                base_rate_sampling=0.05, epsilon=0.05, delta=0.05, init_offset=sink, local_offset=window))
    elif stack == "oracle_topp":
        maskers.append(fixed.OracleTopPMaskerConfig(top_p=0.9))
    elif stack == "quest":
        maskers.append(fixed_impl.QuestTopKMaskerConfig(heavy_size=0.05, page_size=64))
    elif stack == "pqcache":
        maskers.append(fixed.PQCacheConfig(
            heavy_size=_PQ["heavy"], pq_group_factor=_PQ["subspaces"], pq_bits=_PQ["bits"],
            kmeans_iter=_PQ["iterations"], init_offset=sink, metric="euclidean"))
    elif stack == "magicpig":
        maskers.append(sampling.MagicPigConfig(lsh_l=_LSH["tables"], lsh_k=_LSH["bits"], center=True))
    return ResearchAttention.create_from_config(ResearchAttentionConfig(masker_configs=maskers))


def _fresh_meta(state):
    """What a reproducible program hands over for a new sequence: nothing, or the k-means draws."""
    meta = {}
    if state["draws"] is not None:
        meta["pq_init_indices"] = {0: state["draws"][0]}
        meta["pq_reseed_indices"] = {0: state["draws"][1]}
    return meta


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed))
    q_len, tokens = case.get("question", 1), case.get("tokens", 0)
    total = case["S"] + tokens
    k, v, direction = _keys_values(case, gen, total, dev)
    state = {"case": dict(case), "k": k, "v": v, "scaling": 1.0 / sqrt(case["D"]), "draws": None,
             "q": _queries(case, gen, q_len, direction, dev), "attention": _attention(case, gen, dev)}
    if case["stack"] == "pqcache":
        groups, cent, n = case["B"] * case["Hkv"] * _PQ["subspaces"], 1 << _PQ["bits"], case["S"] - 64
        pick = torch.rand((groups, n), generator=gen, device=dev).topk(cent, dim=1).indices
        state["draws"] = (pick, [torch.randint(0, n, (groups, cent), generator=gen, device=dev)
                                 for _ in range(_PQ["iterations"])])
    if case["kind"] == "generate":
        dt = _DTYPES[case["dtype"]]
        state["next_q"] = [_queries(case, gen, 1, direction, dev) for _ in range(tokens)]
        # the adapter's additive masks: causal for the question, nothing forbidden for a token
        ahead = torch.arange(case["S"], device=dev)[None] > torch.arange(q_len, device=dev)[:, None] + (case["S"] - q_len)
        state["causal"] = torch.where(ahead, torch.finfo(dt).min, 0.0).to(dt)[None, None]
        state["open"] = torch.zeros((1, 1, 1, total), dtype=dt, device=dev)
        return state
    # decode: the index over the keys exists (a first call made it); replays also keep the capture
    state["meta"] = _fresh_meta(state)
    if case["kind"] == "replay":
        state["graph"] = DecodeStepGraph(state["attention"], state["q"], k, v, None, state["scaling"],
                                         state["meta"], layer_idx=0)
    else:
        state["attention"].custom_attention(None, state["q"], k, v, None, state["scaling"], 0.0,
                                            sparse_meta_data=state["meta"], layer_idx=0)
    return state


def run(state):
    kind = state["case"]["kind"]
    if kind == "replay":
        return state["graph"].replay(state["q"])
    attention, k, v, scaling = state["attention"], state["k"], state["v"], state["scaling"]
    if kind == "step":
        return attention.custom_attention(None, state["q"], k, v, None, scaling, 0.0,
                                          sparse_meta_data=state["meta"], layer_idx=0)[0]
    meta = _fresh_meta(state)
    S = state["case"]["S"]
    outs = [attention.custom_attention(None, state["q"], k[:, :, :S], v[:, :, :S], state["causal"], scaling, 0.0,
                                       sparse_meta_data=meta, layer_idx=0)[0]]
    for t, q in enumerate(state["next_q"], 1):
        outs.append(attention.custom_attention(None, q, k[:, :, :S + t], v[:, :, :S + t],
                                               state["open"][..., :S + t], scaling, 0.0,
                                               sparse_meta_data=meta, layer_idx=0)[0])
    # the index that the calls built and extended is the sequence's state from here on
    stack, total = state["case"]["stack"], S + len(state["next_q"])
    index = None
    if stack == "hashattention":
        index = meta["key"][0].codes[..., :total]
    elif stack == "pqcache":
        index = [meta["pq_centroids"][0], meta["pq_codebook"][0].codes[:, :, :total - 64]]
    elif stack == "magicpig":
        index = meta["key_signature"][0].codes[:, :, :total]
    return {"outputs": outs, "index": index}


# ---- what a pass cannot do without ------------------------------------------------------------
def _selected(case, S):
    """Keys per query head that the stack selects, at least (K and V rows to read); for the two
    data-dependent ones the share that these key distributions give (top-p 0.9 of a flat softmax,
    LSH matches of one query)."""
    stack = case["stack"]
    if stack in ("hashattention", "quest"):
        return 640 + 0.05 * S
    if stack == "oracle_topk":
        return 640 + 0.02 * S
    if stack == "oracle_adaptive":
        return 640 + 0.07 * S
    if stack == "oracle_topp":
        return 0.6 * S
    if stack == "pqcache":
        return 320 + _PQ["heavy"]
    if stack == "magicpig":
        return 320 + 0.26 * S
    return 384


def _step_work(case, S, q_len=1):
    """One call over S keys with the index in place: the key-side data that the selection reads,
    the selected K and V rows (once per KV head), queries in, outputs out."""
    B, Hq, Hkv, D = case["B"], case["Hq"], case["Hkv"], case["D"]
    e = 4 if case["dtype"] == "f32" else 2
    scan = {"hashattention": B * Hq * S * 4, "quest": 2 * B * Hkv * ceil(S / 64) * D * e,
            "pqcache": B * Hkv * S * _PQ["subspaces"], "magicpig": B * Hkv * S * _LSH["tables"]}.get(case["stack"], 0)
    if case["stack"].startswith("oracle"):
        scan = B * Hkv * S * D * e
    sel = min(S, _selected(case, S))
    bytes_ = scan + B * Hkv * sel * 2 * D * e + 2 * B * Hq * q_len * D * e
    flops = 4.0 * B * Hq * q_len * sel * D
    if case["stack"].startswith("oracle"):
        flops += 2.0 * B * Hq * q_len * S * D
    return bytes_, flops


def work(case):
    S = case["S"]
    if case["kind"] != "generate":
        b, f = _step_work(case, S)
        return {"bytes": b, "flops": f}
    B, Hq, Hkv, D, T = case["B"], case["Hq"], case["Hkv"], case["D"], case["tokens"]
    b, f = _step_work(case, S, case["question"])
    for t in range(1, T + 1):
        x, y = _step_work(case, S + t)
        b, f = b + x, f + y
    n = S + T
    if case["stack"] == "hashattention":  # every key through every query head's MLP, codes out
        b += B * Hkv * n * D * 2 + B * Hq * n * 4
        f += 2.0 * B * Hq * n * (D * _HASH["hidden"] + _HASH["hidden"] ** 2 + _HASH["hidden"] * _HASH["bits"])
    elif case["stack"] == "pqcache":  # ten assignments and centre sums over the keys, codes out
        b += B * Hkv * n * (D * 2 + _PQ["subspaces"])
        f += _PQ["iterations"] * 2.0 * B * Hkv * n * D * (1 << _PQ["bits"])
    elif case["stack"] == "magicpig":  # 600 projections per key, codes out
        b += B * Hkv * n * (D * 2 + 80)
        f += 2.0 * B * Hkv * n * (D + 1) * _LSH["tables"] * _LSH["bits"]
    return {"bytes": b, "flops": f}


def tolerance(case):
    """Four times what one call over each listed stack differs by from float64 attention over the
    same mask: float32 rel 4.8e-7, max 4.1e-6 (sums of 384 terms in another order); bfloat16 rel
    1.6e-3 to 2.3e-3, max 3.8e-3 to 9.3e-3 (probabilities and outputs rounded to bfloat16).
    Codes are whole numbers in a fixed order of operations: none differs."""
    if case["dtype"] == "f32":
        return {"rel": 2e-6, "max": 2e-5}
    return {"rel": 1e-2, "max": 0.04}
