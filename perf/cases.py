"""The work that is timed when this library's speed is compared: calls of its public entry points, in the shapes that a
long-context runtime makes them, from one-thousand-token prompts to a million cached tokens.

A case is a dict of plain values.  ``listed`` gives the standing cases, ``draw`` one more of the same ranges,
``prepare`` the tensors and handles a caller holds before the call (made from the seed on the GPU), ``run`` one call,
``work`` the bytes and operations that call cannot do without, ``tolerance`` how far another correct implementation of the
same precision may be from this one.

Geometries are the two the repository's configurations name: 28 query / 4 KV heads and 32 / 8, head_dim 128.  Keys carry
the outlier channels of the configurations (4 of 128 channels times 8)."""
import math
from types import SimpleNamespace

import torch

from longcontext_sqattn_paddle_b200 import ops
from longcontext_sqattn_paddle_b200.cache_hub import ClusteredKV, RaggedClusteredDecoder, num_clusters_for, segment_k_means
from longcontext_sqattn_paddle_b200.sqattn import attn_causal, attn_unified, mp_triton_wrapper
from longcontext_sqattn_paddle_b200.sqattn.window_search import attention_histograms

D = 128
SINK = 256


def listed():
    return [
        # a short prompt of no round length: five preparation launches and one attention launch, latency counts
        dict(name="prefill_1000", kind="prefill", n=1000, hq=28, hkv=4, dtype="bf16", ratio=0.1, per_head=False, fp8="off"),
        # a document-sized prompt with calibrated windows (every head its own, the outer window wider than the inner)
        dict(name="prefill_20001_per_head", kind="prefill", n=20001, hq=32, hkv=8, dtype="bf16", ratio=0.08, per_head=True, fp8="off"),
        # the headline: the operator on one 128K sequence, the default window of a tenth of the context
        dict(name="prefill_131072", kind="prefill", n=131072, hq=28, hkv=4, dtype="bf16", ratio=0.1, per_head=False, fp8="off"),
        # the operator with P rounded through FP8 everywhere, the scheme's low-precision option
        dict(name="prefill_8192_fp8", kind="prefill", n=8192, hq=28, hkv=4, dtype="bf16", ratio=0.1, per_head=False, fp8="all"),
        # the layers a model keeps dense (its first and last): causal attention on the fused projection's views
        dict(name="dense_32768", kind="dense", n=32768, hq=28, hkv=4, dtype="bf16"),
        # one token of one chat against a short cache: pure latency
        dict(name="decode_4000", kind="decode", batch=1, min_len=4000, max_len=4000, hq=28, hkv=4, dtype="bf16"),
        # a serving batch whose contexts differ by a factor of thirty
        dict(name="decode_ragged_8", kind="decode", batch=8, min_len=2000, max_len=65536, hq=32, hkv=8, dtype="bf16"),
        # one layer of a step at a million tokens of context: pure bandwidth
        dict(name="decode_1048576", kind="decode", batch=1, min_len=1048576, max_len=1048576, hq=28, hkv=4, dtype="bf16"),
        # the launcher with the reference's name and defaults (keys centred on every call)
        dict(name="unified_32000", kind="unified", n=32000, batch=1, hq=28, hkv=4, dtype="fp16"),
        # a step of a ragged batch over clustered caches: select, gather, attend with FP8 P
        dict(name="retrieve_8", kind="retrieve", batch=8, min_len=8192, max_len=65536, hq=32, hkv=8, dtype="bf16", budget=4096),
        # clustering the keys of one 64K-token layer, ten Lloyd iterations, member lists and value sums included
        dict(name="kmeans_65536", kind="kmeans", groups=8, n=65536, dtype="bf16", iters=10),
        # window calibration of one layer, run once per model and layer before the windows above exist
        dict(name="calibrate_8192", kind="calibrate", n=8192, hq=28, hkv=4, dtype="bf16", bins=200),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["prefill", "prefill", "prefill", "dense", "decode", "decode", "unified", "retrieve", "kmeans", "calibrate"])
    hq, hkv = rng.choice([(28, 4), (32, 8)])
    dtype = rng.choice(["bf16", "bf16", "bf16", "fp16"])
    if kind == "prefill":
        return dict(kind=kind, n=_log_uniform(rng, 500, 100000), hq=hq, hkv=hkv, dtype=dtype, ratio=round(rng.uniform(0.05, 0.15), 3),
                    per_head=rng.random() < 0.5, fp8=rng.choice(["off", "off", "off", "all"]))
    if kind == "dense":
        return dict(kind=kind, n=_log_uniform(rng, 500, 40000), hq=hq, hkv=hkv, dtype=dtype)
    if kind == "decode":
        batch = rng.choice([1, 1, 2, 3, 5, 8, 16])
        longest = _log_uniform(rng, 1000, 1000000 // batch)
        return dict(kind=kind, batch=batch, min_len=max(1, longest // rng.choice([1, 4, 30])), max_len=longest, hq=hq, hkv=hkv, dtype=dtype)
    if kind == "unified":
        return dict(kind=kind, n=_log_uniform(rng, 1000, 300000), batch=rng.choice([1, 1, 2]), hq=hq, hkv=hkv, dtype=dtype)
    if kind == "retrieve":
        lo = _log_uniform(rng, 6000, 16000)
        return dict(kind=kind, batch=rng.choice([2, 4, 7, 8]), min_len=lo, max_len=lo * rng.choice([2, 4]), hq=hq, hkv=hkv, dtype=dtype,
                    budget=rng.choice([2048, 4096]))
    if kind == "kmeans":
        return dict(kind=kind, groups=hkv, n=_log_uniform(rng, 4000, 100000), dtype=dtype, iters=10)
    return dict(kind="calibrate", n=_log_uniform(rng, 1000, 12000), hq=hq, hkv=hkv, dtype=dtype, bins=rng.choice([100, 200]))


# ------------------------------------------------------------------------------------------------ inputs
def _dtype(case):
    return torch.bfloat16 if case["dtype"] == "bf16" else torch.float16


def _outliers(k):
    """Four of the head_dim channels times 8, in place."""
    k[..., 5:D:32] *= 8.0
    return k


def _fused(case, g):
    """q, k, v of one layer as the model has them: views [1, n, heads, D] of the fused projection's output."""
    n, hq, hkv = case["n"], case["hq"], case["hkv"]
    qkv = torch.randn(1, n, (hq + 2 * hkv) * D, generator=g, device="cuda", dtype=_dtype(case))
    q, k, v = qkv.split([hq * D, hkv * D, hkv * D], dim=-1)
    q, k, v = q.view(1, n, hq, D), k.view(1, n, hkv, D), v.view(1, n, hkv, D)
    _outliers(k)
    return q, k, v


def _windows(case):
    """Per-head (inner, outer) window ratios: one value for all heads, or what calibration leaves (heads differ by up to
    a factor of three and the outer window is the wider one)."""
    r, hq = case["ratio"], case["hq"]
    if not case["per_head"]:
        return [r] * hq, [r] * hq
    inner = [r * (0.5 + 0.25 * (5 * h % 7)) for h in range(hq)]
    return inner, [min(1.0, 1.5 * w) for w in inner]


def _lengths(case):
    """The batch's context lengths, spread over the logarithm of the range."""
    b, lo, hi = case["batch"], case["min_len"], case["max_len"]
    return [hi if b == 1 else int(round(lo * (hi / lo) ** (i / (b - 1)))) for i in range(b)]


def prepare(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    kind, dt = case["kind"], _dtype(case)

    def randn(*shape):
        return torch.randn(*shape, generator=g, device="cuda", dtype=dt)

    s = {"case": dict(case)}
    if kind == "prefill":
        args = SimpleNamespace(qk_qtype="int", v_qtype="int", use_relative_distance=True)
        inner, outer = _windows(case)
        s["layer"] = SimpleNamespace(num_key_value_groups=case["hq"] // case["hkv"])
        s["attention"] = mp_triton_wrapper(1, bit8_window_sizes=inner, bit4_window_sizes=outer, sink_window_size=SINK, args=args,
                                           p_fp8_mode=case["fp8"])
        s["qkv"] = _fused(case, g)
    elif kind == "dense":
        s["qkv"] = _fused(case, g)
    elif kind == "decode":
        b, hkv = case["batch"], case["hkv"]
        s["lens"] = _lengths(case)
        cap = max(s["lens"]) + 16                        # the cache has room for the tokens still to come
        s["q"] = randn(b, 1, case["hq"], D)
        s["k"], s["v"] = _outliers(randn(b, cap, hkv, D)), randn(b, cap, hkv, D)
    elif kind == "unified":
        b, n = case["batch"], case["n"]
        s["q"] = randn(b, case["hq"], 1, D)
        s["k"], s["v"] = _outliers(randn(b, case["hkv"], n, D)), randn(b, case["hkv"], n, D)
    elif kind == "retrieve":
        caches = [ClusteredKV(_outliers(randn(case["hkv"], n, D)), randn(case["hkv"], n, D)) for n in _lengths(case)]
        s["decoder"] = RaggedClusteredDecoder(caches, budget=case["budget"])
        s["q"] = randn(case["batch"], case["hq"], 1, D)
    elif kind == "kmeans":
        s["k"], s["v"] = _outliers(randn(case["groups"], case["n"], D)), randn(case["groups"], case["n"], D)
        s["clusters"] = num_clusters_for(case["n"])
    else:
        s["q"], s["k"] = randn(case["hq"], case["n"], D), _outliers(randn(case["hkv"], case["n"], D))
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "prefill":
        return state["attention"](state["layer"], *state["qkv"], None)
    if kind == "dense":
        return attn_causal(*state["qkv"], tensor_layout="NHD", output_dtype=state["qkv"][0].dtype)
    if kind == "decode":
        return ops.decode(state["q"], state["k"], state["v"], layout="NHD", out_dtype=state["q"].dtype, kv_lens=state["lens"])
    if kind == "unified":
        return attn_unified(state["q"], state["k"], state["v"], output_dtype=state["q"].dtype, return_lse=True)
    if kind == "retrieve":
        return state["decoder"].step(state["q"])
    if kind == "kmeans":
        centroids, value_sum, clusters, sizes = segment_k_means(state["k"], state["v"], state["clusters"], num_iters=case["iters"])
        # the lists are as wide as the largest cluster: hand back the members themselves, one after another
        members = clusters[torch.arange(clusters.shape[2], device=clusters.device) < sizes[..., None]]
        return {"centroids": centroids, "value_sum": value_sum, "sizes": sizes, "members": members}
    return attention_histograms(state["q"], state["k"], relative=True, num_bins=case["bins"], sink_len=SINK)


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def _window_pairs(n, window):
    """(query, key) pairs one head visits: the sink, the window up to the end of the row's 64-row block, causal."""
    pairs = 0
    for qs in range(0, n, 64):
        rows = min(64, n - qs)
        sink = min(SINK, qs)
        low = max(SINK, qs + 64 - window)
        pairs += rows * (sink + max(0, qs - low)) + rows * (rows + 1) // 2
    return pairs


def work(case):
    kind = case["kind"]
    if kind == "prefill":
        n, hq, hkv = case["n"], case["hq"], case["hkv"]
        inner, outer = _windows(case)
        sizes = [(int(max(a, b) * n) + 127) // 128 * 128 for a, b in zip(inner, outer)]
        pairs = {w: _window_pairs(n, w) for w in set(sizes)}
        return {"bytes": 2 * D * n * (2 * hq + 2 * hkv), "flops": 4 * D * sum(pairs[w] for w in sizes)}
    if kind == "dense":
        n, hq, hkv = case["n"], case["hq"], case["hkv"]
        return {"bytes": 2 * D * n * (2 * hq + 2 * hkv), "flops": 4 * D * hq * n * (n + 1) // 2}
    if kind in ("decode", "unified"):
        keys = sum(_lengths(case)) if kind == "decode" else case["batch"] * case["n"]
        return {"bytes": 4 * D * case["hkv"] * keys, "flops": 4 * D * case["hq"] * keys}
    if kind == "retrieve":
        lens, hq, hkv = _lengths(case), case["hq"], case["hkv"]
        keys = sum(min(n, case["budget"]) for n in lens)
        clusters = sum(num_clusters_for(n) for n in lens)
        return {"bytes": 2 * D * hkv * (2 * keys + clusters), "flops": 4 * D * hq * keys + 2 * D * hkv * clusters}
    if kind == "kmeans":
        g, n, k, it = case["groups"], case["n"], num_clusters_for(case["n"]), case["iters"]
        return {"bytes": 2 * D * g * (2 * n + 2 * k) + 4 * g * n, "flops": it * 2 * D * g * n * k}
    n, hq, hkv = case["n"], case["hq"], case["hkv"]
    return {"bytes": 2 * D * n * (hq + hkv) + 8 * hq * case["bins"], "flops": 2 * D * hq * n * (n + 1) // 2}


def tolerance(case):
    """About four times what this library shows against the same path in fp64 (5001-token prefills, 30000-key decodes,
    4001-token calibration)."""
    kind, bf16 = case["kind"], case["dtype"] == "bf16"
    if kind == "kmeans":
        return "exact"                                       # exact arg-max and order-free sums by construction
    if kind == "calibrate":
        return {"rel": 1e-6}                                 # sums of fp32 weights in any order; seen 5e-8 at 4001 tokens
    if kind == "retrieve" or (kind == "prefill" and case["fp8"] != "off"):
        return {"rel": 6e-2}                                 # P has a 3-bit mantissa; seen 1.2e-2 and 1.5e-2
    if kind == "prefill":
        return {"rel": 6.6e-3, "max": 2e-2}                  # the bf16 rounding of the output; seen 1.7e-3, 5.0e-3
    if kind == "unified":                                    # keys minus their mean may be rounded or not; seen 5.8e-3 / 9.4e-4
        return {"rel": 2.3e-2, "max": 1.9e-1} if bf16 else {"rel": 3.8e-3, "max": 3.3e-2}
    # q times the softmax scale may be rounded or not; seen 3.2e-3, 6.5e-2 / 4.5e-4, 8.6e-3
    return {"rel": 1.3e-2, "max": 2.6e-1} if bf16 else {"rel": 1.8e-3, "max": 3.4e-2}
