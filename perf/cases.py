"""The workloads this framework is timed on, through its public entry points.

Six kinds of work, which together are what a user of the library has it do:

  decode   one generated token of one layer: `hira_decode_attention` (query preparation, threshold,
           search, sparse attention) on a built index, device tensors in and out
  step     the same step behind the one-call entry with host buffers, `HiraDecodeStep`
  search   the reference's own entry point, `CUDASearcher.search`: the dense (query head, slot) score row
  build    prefill: `CUDAIndexer.build` over a prompt's keys and values
  stream   a prefix indexed, keys appended one by one, the index rebuilt at the end
  session  one layer of a model that generates: `HiraCache` layer prefill, then token after token
           `update` + `hira_attention`, with the configuration's defaults

Keys, values and queries come from `hira_b200.workloads` (N(0,1) keys with RoPE by position and four
outlier channels, as Llama-shaped caches look; the anisotropic ones for the fp32 configurations).
"""
from __future__ import annotations

import math

import torch

from hira_b200 import (CacheOutput, CUDAIndexer, CUDASearcher, DeviceMode, HiraCacheLayer, HiraConfig, HiraDecodeStep,
                       hira_attention, hira_decode_attention, sample_kth)
from hira_b200 import workloads as W

DTYPES = {"bf16": torch.bfloat16, "fp32": torch.float32}
KEEP = 0.02          # share of the keys a given threshold keeps (the decode configurations of hira_b200.workloads)
TAU_SAMPLES = 4096   # keys the given threshold is estimated from


def _case(name, kind, *, batch=1, kv=8, group=4, dim=128, dtype="bf16", ctx=32768, levels=3, bf=32, dist="rope_outlier",
          tau="given", queued=0, iters=1, balance=0, tokens=0):
    c = {"kind": kind, "batch": batch, "kv": kv, "group": group, "dim": dim, "dtype": dtype, "ctx": ctx, "levels": levels,
         "bf": bf, "dist": dist, "tau": tau, "queued": queued, "iters": iters, "balance": balance, "tokens": tokens}
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # a short chat turn: everything is latency and launches; the threshold is found in the step
        _case("decode_b1_ctx2048_tau", "decode", ctx=2048, tau="sampled"),
        # the single-sequence configuration of hira_b200.workloads (cfg1), threshold known
        _case("decode_b1_ctx32768", "decode"),
        # the headline step (cfg2): batch 16, 131,072 tokens each
        _case("decode_b16_ctx131072", "decode", batch=16, ctx=131072),
        # one sequence shard of the million-token configuration (cfg4): 64 query heads, branching 64
        _case("decode_b1_ctx131072_q64_tau", "decode", ctx=131072, group=8, bf=64, tau="sampled"),
        # small heads, a two-level index, ragged context, a head group that is no power of two, and keys
        # still waiting in the cache layer's queue
        _case("decode_b3_ctx9001_d64_queue", "decode", batch=3, kv=4, group=3, dim=64, ctx=9001, levels=2, bf=16, queued=5),
        # full precision, one query head per key head, ragged
        _case("decode_b2_ctx20011_fp32", "decode", batch=2, group=1, dtype="fp32", ctx=20011, dist="aniso"),
        # one GPU's share of the headline step on eight GPUs, host buffers in and out
        _case("step_b2_ctx131072", "step", batch=2, ctx=131072),
        # the reference's search call with its default rule: every child of a kept parent, dense scores
        _case("search_dense_b1_ctx32768", "search"),
        # prefill of the single-sequence configuration
        _case("build_b1_ctx32768", "build"),
        # the full-precision configuration (cfg0): two levels, ten k-means iterations
        _case("build_fp32_ctx4096_it10", "build", group=1, dtype="fp32", ctx=4096, levels=2, bf=64, dist="aniso", iters=10),
        # streaming (cfg3): a prefix of 65,536 keys, single-key appends, a rebuild
        _case("stream_ctx65536_append128", "stream", ctx=65536, tokens=128),
        # generation through the cache classes with the defaults of HiraConfig (branching 10, update every token)
        _case("session_prompt3000_gen48", "session", ctx=3000, bf=10, levels=5, tau="sampled", tokens=48),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "decode", "step", "search", "build", "build", "stream", "session"])
    bf = rng.choice([16, 32, 32, 64])
    kv = rng.choice([2, 4, 8, 8])
    if kind in ("decode", "step"):
        dim = rng.choice([64, 128, 128, 128])
        dtype = rng.choice(["bf16", "bf16", "bf16", "fp32"])
        group = rng.choice([1, 2, 3, 4, 4, 5, 8])
        batch = _log_int(rng, 1, 16)
        # no more (head, key) pairs than half of the largest listed case, counted in chunks of four query heads
        most = 16 * 8 * 131072 // 2 // (batch * kv * -(-group // 4) * (2 if dtype == "fp32" else 1))
        ctx = _log_int(rng, 1024, min(131072, most))
        return _case(None, kind, batch=batch, kv=kv, group=group, dim=dim, dtype=dtype, ctx=ctx, levels=rng.choice([2, 3, 3]), bf=bf,
                     dist="rope_outlier" if dtype == "bf16" else "aniso", tau=rng.choice(["given", "sampled"]),
                     queued=rng.choice([0, 0, rng.randint(1, 15)]) if kind == "decode" else 0)
    if kind == "search":
        dtype = rng.choice(["bf16", "fp32"])
        return _case(None, kind, kv=kv, group=rng.choice([1, 2, 4, 8]), dim=rng.choice([64, 128]), dtype=dtype,
                     ctx=_log_int(rng, 1024, 131072), levels=rng.choice([2, 3]), bf=bf,
                     dist="rope_outlier" if dtype == "bf16" else "aniso")
    if kind == "build":
        dtype = rng.choice(["bf16", "bf16", "fp32"])
        return _case(None, kind, batch=rng.choice([1, 1, 2]), kv=kv, dim=rng.choice([64, 128, 128]), dtype=dtype,
                     ctx=_log_int(rng, 1000, 65536 if dtype == "bf16" else 16384), levels=rng.choice([2, 3, 3]), bf=bf,
                     dist="rope_outlier" if dtype == "bf16" else "aniso", iters=rng.choice([1, 1, 4]), balance=rng.choice([0, 0, 2]))
    if kind == "stream":
        return _case(None, kind, kv=kv, ctx=_log_int(rng, 4000, 65536), bf=rng.choice([16, 32]), tokens=rng.randint(16, 128))
    return _case(None, kind, kv=kv, group=rng.choice([1, 2, 4]), dim=rng.choice([64, 128]), ctx=_log_int(rng, 500, 8192),
                 bf=rng.choice([10, 32]), levels=5, tau="sampled", tokens=rng.randint(8, 48))


def _kv(case, n, seed, first_pos=0):
    """keys, values (B, H, n, D)"""
    k, v = W.make_kv(case["batch"] * case["kv"], n, seed, "cuda", dist=case["dist"], dtype=DTYPES[case["dtype"]],
                     first_pos=first_pos, dim=case["dim"])
    shape = (case["batch"], case["kv"], n, case["dim"])
    return k.view(shape), v.view(shape)


def _outliers_fit(case):
    # the outlier channels of the workload generator sit at fixed positions of a 128-wide head
    return case["dist"] != "rope_outlier" or case["dim"] > max(W.OUTLIER_CHANNELS)


def _prompt(case, n, seed, first_pos=0):
    if _outliers_fit(case):
        return _kv(case, n, seed, first_pos)
    # a 64-wide head: the even channels of a 128-wide one (two of the four outliers remain)
    k, v = W.make_kv(case["batch"] * case["kv"], n, seed, "cuda", dist=case["dist"], dtype=DTYPES[case["dtype"]], first_pos=first_pos)
    shape = (case["batch"], case["kv"], n, case["dim"])
    return k[..., ::2].contiguous().view(shape), v[..., ::2].contiguous().view(shape)


def _queries(case, n_sets, seed):
    hq = case["kv"] * case["group"]
    q = torch.stack([W.make_queries(case["batch"] * hq, seed + 13 * i, "cuda", pos=case["ctx"] + i if case["dist"] == "rope_outlier" else None,
                                    dim=case["dim"]) for i in range(n_sets)])
    return q.view(n_sets, case["batch"], hq, 1, case["dim"]).to(DTYPES[case["dtype"]])


def _given_tau(case, keys, q):
    """A threshold that keeps about KEEP of the keys, on the scale of the unit query."""
    n = case["ctx"]
    step = max(1, n // TAU_SAMPLES)
    sample = keys.reshape(-1, n, case["dim"])[:, ::step][:, :TAU_SAMPLES].contiguous()
    qf = q.reshape(-1, case["dim"]).float()
    q_hat = qf / qf.norm(dim=-1, keepdim=True)
    return sample_kth(sample, q_hat, max(1, round(KEEP * sample.shape[1])))


def _indexer(case, **kw):
    return CUDAIndexer(case["levels"], case["iters"], case["bf"], balance_rounds=case["balance"], **kw)


def prepare(case, seed):
    kind, seed = case["kind"], 1000 * int(seed)
    if kind == "session":
        cfg = HiraConfig(device_mode=DeviceMode.CUDA_ONLY, num_levels=case["levels"], branching_factor=case["bf"],
                         max_context=case["ctx"] + case["tokens"])
        keys, vals = _prompt(case, case["ctx"], seed + 1)
        new_k, new_v = _prompt(case, case["tokens"], seed + 2, first_pos=case["ctx"])
        hq = case["kv"] * case["group"]
        prompt_q = torch.randn((1, hq, case["ctx"], case["dim"]), generator=torch.Generator("cuda").manual_seed(seed + 3),
                               device="cuda").to(DTYPES[case["dtype"]])
        layer = HiraCacheLayer(device_mode=cfg.device_mode, update_every=cfg.update_every,
                               indexer_kwargs=cfg.get_indexer_kwargs(), searcher_kwargs=cfg.get_searcher_kwargs())
        return {"kind": kind, "layer": layer, "cfg": cfg, "keys": keys, "vals": vals, "prompt_q": prompt_q,
                "q": _queries(case, case["tokens"], seed + 4),
                "new_k": [new_k[:, :, i:i + 1].contiguous() for i in range(case["tokens"])],
                "new_v": [new_v[:, :, i:i + 1].contiguous() for i in range(case["tokens"])]}
    keys, vals = _prompt(case, case["ctx"], seed + 1)
    if kind == "build":
        return {"kind": kind, "indexer": _indexer(case), "keys": keys, "vals": vals}
    if kind == "stream":
        new_k, new_v = _prompt(case, case["tokens"], seed + 2, first_pos=case["ctx"])
        return {"kind": kind, "indexer": _indexer(case, max_context=case["ctx"] + case["tokens"], reserve_worst_case=True),
                "keys": keys, "vals": vals,
                "new_k": [new_k[:, :, i:i + 1].contiguous() for i in range(case["tokens"])],
                "new_v": [new_v[:, :, i:i + 1].contiguous() for i in range(case["tokens"])]}
    q = _queries(case, 1, seed + 4)[0]
    tau = _given_tau(case, keys, q) if case["tau"] == "given" else None
    s = {"kind": kind, "q": q, "tau": tau}
    if kind == "search":
        s["indexer"] = _indexer(case).build(keys, vals)
        s["searcher"] = CUDASearcher(block_c=case["bf"])
        qf = q.reshape(-1, case["dim"]).float()
        s["q"] = (qf / qf.norm(dim=-1, keepdim=True)).contiguous()
        return s
    if kind == "step":
        s["indexer"] = _indexer(case).build(keys, vals)
        hq = case["batch"] * case["kv"] * case["group"]
        s["step"] = HiraDecodeStep(s["indexer"], hq, q_dtype=q.dtype,
                                   **({"threshold_method": "none"} if tau is not None else {}))
        s["q_host"] = q.reshape(hq, case["dim"]).cpu().pin_memory()
        s["out_host"] = torch.empty((hq, case["dim"]), dtype=torch.float32).pin_memory()
        return s
    indexer = _indexer(case).build(keys, vals)
    # keys not indexed yet: the filled part of the queue of a cache layer that indexes every 16 tokens
    new_k, new_v = _prompt(case, 16, seed + 2, first_pos=case["ctx"])
    s["out"] = CacheOutput(queued_keys=new_k[:, :, :case["queued"]], queued_values=new_v[:, :, :case["queued"]],
                           prefill_keys=None, prefill_values=None, indexer=indexer, searcher=CUDASearcher(block_c=case["bf"]))
    return s


def _index_arrays(ix):
    out = {"children": ix.children, "values": ix.values, "slot2token": ix.slot2token, "parents": ix.parents,
           "parent_radii": ix.parent_radii, "child_counts": ix._child_counts}
    if ix.grand_parents is not None:
        out.update(grand_parents=ix.grand_parents, gp_radii=ix.grand_parent_radii, gp_counts=ix._gp_child_counts)
    return out


def run(s):
    kind = s["kind"]
    if kind == "decode":
        return hira_decode_attention(s["q"], s["out"], threshold=s["tau"])
    if kind == "step":
        s["step"](s["q_host"], s["out_host"], threshold=s["tau"])
        s["step"].synchronize()          # the caller reads its output buffer before the next token
        return s["out_host"]
    if kind == "search":
        return s["searcher"].search(s["q"], s["tau"], s["indexer"])
    if kind == "build":
        return _index_arrays(s["indexer"].build(s["keys"], s["vals"]))
    if kind == "stream":
        ix = s["indexer"].build(s["keys"], s["vals"])
        for k, v in zip(s["new_k"], s["new_v"]):
            ix.update(k, v)
        grown = {"appended_radii": ix.parent_radii.clone(), "appended_counts": ix._child_counts.clone()}
        ix.rebuild()
        return {**_index_arrays(ix), **grown}
    layer, scale = s["layer"], s["q"].shape[-1] ** -0.5
    layer.reset()
    key, _ = layer.update(s["keys"], s["vals"])
    prompt_out, _ = hira_attention(None, s["prompt_q"], key, scaling=scale, hira_config=s["cfg"])
    outs = []
    for i, (k, v) in enumerate(zip(s["new_k"], s["new_v"])):
        key, _ = layer.update(k, v)
        outs.append(hira_attention(None, s["q"][i], key, scaling=scale, hira_config=s["cfg"])[0])
    return {"prompt": prompt_out, "tokens": torch.stack(outs)}


def work(case):
    """What one pass cannot do without.  A search has to look at every key once, in the smallest form the index
    keeps it in (one byte per channel and four of scale where heads are 128 wide, else the keys themselves; all
    of the keys where their scores are the output), and at the values it selects."""
    heads, n, d = case["batch"] * case["kv"], case["ctx"], case["dim"]
    hq, e, bf, kind = heads * case["group"], 2 if case["dtype"] == "bf16" else 4, case["bf"], case["kind"]
    k1 = -(-n // bf)
    centres = k1 + (-(-k1 // bf) if case["levels"] > 2 else 0)
    look = n * ((d + 4) if d == 128 else d * e) + centres * (d * e + 8)
    attend = KEEP * n * d * e
    build_bytes = heads * (n * (4 * d * e + 4) + (n * (d + 4) if d == 128 else 0) + centres * (d * e + 8))
    build_flops = heads * 2.0 * d * (n * k1 + (k1 * -(-k1 // bf) if case["levels"] > 2 else 0)) * (case["iters"] + case["balance"])
    if kind in ("decode", "step"):
        return {"bytes": heads * look + hq * (attend + d * (4 + e)), "flops": 2.0 * hq * d * n * (1 + KEEP)}
    if kind == "search":
        return {"bytes": heads * (n * d * e + centres * (d * e + 8)) + hq * n * 4, "flops": 2.0 * hq * d * n}
    if kind == "build":
        return {"bytes": build_bytes, "flops": build_flops}
    t = case["tokens"]
    append_bytes = heads * centres * (d * e + 4) * t
    if kind == "stream":
        return {"bytes": 2 * build_bytes + append_bytes, "flops": 2 * build_flops + 2.0 * heads * d * centres * t}
    return {"bytes": build_bytes + append_bytes + t * (heads * look + hq * attend),
            "flops": build_flops + 2.0 * hq * d * n * n + 2.0 * hq * d * n * t * (1 + KEEP)}


def tolerance(case):
    kind = case["kind"]
    if kind in ("build", "stream"):
        return "exact"       # rows are moved, not computed; centres, radii and slots follow one stated arithmetic
    if kind == "search":
        return "exact"       # scores are the canonical dot product of the rows
    if kind == "session":
        return {"rel": 1.5e-3}   # outputs rounded to bf16: up to 3.5e-4 against a 64-bit evaluation rounded the same way
    return {"rel": 2.5e-6}       # fp32 sums over the same selected keys: 2.5e-7 to 5.9e-7 against a 64-bit evaluation
