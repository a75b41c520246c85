"""What a user of this framework has it do, as timed cases.

Two kinds of program call it.  One calls an operator layer by layer (``"call"`` cases: one pass is
one eager call of the public wrapper).  The other is a serving engine, which records the decode
step of its model once and replays it (``"step"`` cases: what is once per step -- the plan, the
shared-prefix groups -- and then the calls of several layers with a cache each, recorded in a CUDA
graph when the state is made; one pass is one step).

``listed()`` names the cases, ``draw`` gives more of the same ranges, ``prepare`` makes what the
program holds before the call, ``run`` is one pass, ``exact`` the same result from torch in 64 bits.
"""

from __future__ import annotations

import math

import torch

DEV = "cuda"
PAGE = 16
FP8_MAX = 448.0
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


# ---------------------------------------------------------------------------------- the cases
def _decode(name, q_heads, kv_heads, head_dim, batch, lo, hi, dist, kv="fp8", dtype="bf16", layout="nhd", layers=0,
            append=False):
    """layers 0: one eager call without a plan; more: a recorded step with a plan."""
    return dict(name=name, kind="decode", q_heads=q_heads, kv_heads=kv_heads, head_dim=head_dim, batch=batch, lo=lo, hi=hi,
                dist=dist, kv=kv, dtype=dtype, layout=layout, layers=layers, append=append)


def _prefix(name, batch, groups, alone, prefix, suffix, layers, q_heads=16, kv_heads=2):
    """groups 0: every request shares one prefix whose length the program knows; else the groups are found on the device,
    the i-th sharing ``prefix * (1 + i / 4)`` tokens, and ``alone`` requests belong to none."""
    return dict(name=name, kind="prefix", q_heads=q_heads, kv_heads=kv_heads, head_dim=128, batch=batch, groups=groups,
                alone=alone, prefix=prefix, suffix=suffix, layers=layers, dtype="bf16")


def _append(name, q_heads, kv_heads, head_dim, tokens, rotary, neox, kv, dtype="bf16", table="f32"):
    return dict(name=name, kind="append", q_heads=q_heads, kv_heads=kv_heads, head_dim=head_dim, tokens=tokens, rotary=rotary,
                neox=neox, kv=kv, dtype=dtype, table=table)


def listed():
    return [
        # the smallest call: a handful of chats on a half-billion-parameter model; launches and latency
        _decode("call-d64-b8", 14, 2, 64, 8, 128, 1024, "uniform"),
        # the same model behind a busy endpoint: small heads, many requests
        _decode("call-d64-b256", 14, 2, 64, 256, 512, 4096, "uniform"),
        # a serving engine's recorded decode step of a 3B model, eight of its layers, one plan for all
        _decode("step-d128-b64", 16, 2, 128, 64, 512, 4096, "uniform", layers=8),
        # the step of a recorded model that also rotates, quantises and appends the new token before it attends
        _decode("step-append-b64", 16, 2, 128, 64, 512, 4096, "uniform", layers=2, append=True),
        # a ragged batch of a 7B model: many short requests, a few long ones
        _decode("call-d128-b256-ragged", 28, 4, 128, 256, 1, 8192, "log", layout="hnd"),
        # long documents: few sequences, the largest cache
        _decode("call-d128-b4-long", 32, 8, 128, 4, 131072, 131072, "full"),
        # sixteen query heads to a KV head (heavily grouped attention)
        _decode("call-gqa16-b64", 32, 2, 128, 64, 512, 4096, "uniform", dtype="fp16"),
        # a model whose cache is not quantised
        _decode("call-bf16-b64", 16, 2, 128, 64, 512, 4096, "uniform", kv="same"),
        # one system prompt in front of every chat
        _prefix("step-prefix-b64", 64, 0, 0, 4096, 512, 8),
        # several system prompts at once and requests with none, found in the block table at every step
        _prefix("step-groups-b64", 64, 2, 8, 4096, 512, 8),
        # prefill: rotate and append the tokens of a chunk, FP8 cache
        _append("append-8k-fp8", 28, 4, 128, 8192, 128, True, "fp8"),
        # prefill of a model with interleaved, partial rotation and a 16-bit cache
        _append("append-4k-partial", 32, 8, 128, 4096, 64, False, "same"),
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "step", "long", "prefix", "append"])
    if kind == "append":
        q_heads, kv_heads, d = rng.choice([(14, 2, 64), (16, 2, 128), (28, 4, 128), (32, 8, 128)])
        neox = rng.random() < 0.7
        rotary = d if neox and rng.random() < 0.7 else rng.choice([d // 4, d // 2, d])
        return _append("", q_heads, kv_heads, d, _spread(rng, 1, 8192 if neox and rotary == d else 4096), rotary, neox,
                       rng.choice(["fp8", "same"]), rng.choice(["bf16", "bf16", "fp16"]), rng.choice(["f32", "same"])) | {"name": None}
    if kind == "prefix":
        groups = rng.choice([0, 0, 1, 2, 3])
        batch = _spread(rng, 16, 128) if groups == 0 else _spread(rng, 12 * groups, 96)
        alone = rng.randint(0, batch - 8 * groups) // 2 if groups else 0
        return _prefix(None, batch, groups, alone, PAGE * _spread(rng, 256, 512), _spread(rng, 48, 1024), rng.randint(2, 6))
    if kind == "long":
        q_heads, kv_heads = rng.choice([(16, 2), (28, 4), (32, 8)])
        hi = _spread(rng, 16384, 131072)
        return _decode(None, q_heads, kv_heads, 128, rng.randint(1, 4), hi // 2 if rng.random() < 0.5 else hi, hi, "uniform")
    q_heads, kv_heads, d = rng.choice([(14, 2, 64), (16, 2, 128), (28, 4, 128), (32, 8, 128), (32, 2, 128)])
    batch = _spread(rng, 1, 256)
    kv = "fp8" if d == 64 or q_heads // kv_heads > 8 else rng.choice(["fp8", "fp8", "same"])
    # at most 160 MB of keys and values a layer
    most = 160e6 / (batch * kv_heads * d * 2 * (1 if kv == "fp8" else 2))
    hi = _spread(rng, 24, max(25, min(8192, most)))
    lo = max(1, hi // rng.choice([1, 2, 8, 64, 8192]))
    layers = rng.randint(2, 4) if kind == "step" else 0
    return _decode(None, q_heads, kv_heads, d, batch, lo, hi, rng.choice(["uniform", "log"]), kv, rng.choice(["bf16", "bf16", "fp16"]),
                   rng.choice(["nhd", "hnd"]), layers, bool(layers) and kv == "fp8" and rng.random() < 0.4)


# ---------------------------------------------------------------------------------- inputs, from the seed alone
def _lengths(batch, lo, hi, dist, gen):
    """Lengths of the distribution, one from each of ``batch`` equal parts of it, in random order: every seed's batch has
    other lengths and nearly the same sum.  Without a generator: the longest that each part can give."""
    if gen is None:
        u = torch.arange(1, batch + 1, dtype=torch.float64) / batch
    else:
        u = (torch.randperm(batch, generator=gen) + torch.rand(batch, generator=gen, dtype=torch.float64)) / batch
    if dist == "log":
        x = torch.exp(math.log(lo) + u * (math.log(hi) - math.log(lo)))
    else:
        x = lo + u * (hi - lo)
    return x.round().clamp(1, hi).to(torch.int64)


def _case_lengths(case, gen):
    if case["kind"] == "decode":
        return _lengths(case["batch"], case["lo"], case["hi"], case["dist"], gen)
    own = _lengths(case["batch"], 0, case["suffix"], "uniform", gen)
    return own + _prefix_lengths(case)


def _prefix_lengths(case):
    """Tokens of each request that it shares (requests in no group share none; theirs are as long as the first prefix)."""
    batch, groups, alone = case["batch"], case["groups"], case["alone"]
    if groups == 0:
        return torch.full((batch,), case["prefix"], dtype=torch.int64)
    shares = [g * (batch - alone) // groups for g in range(groups + 1)]
    n = torch.full((batch,), case["prefix"], dtype=torch.int64)
    for g in range(groups):
        n[shares[g]:shares[g + 1]] = int(case["prefix"] * (1 + g / 4)) // PAGE * PAGE
    return n


def _group_of(case):
    """Group of each request, -1 for none."""
    batch, groups, alone = case["batch"], case["groups"], case["alone"]
    g_of = torch.full((batch,), -1 if groups else 0, dtype=torch.int64)
    for g in range(groups):
        g_of[g * (batch - alone) // groups:(g + 1) * (batch - alone) // groups] = g
    return g_of


def _block_table(case, lens, gen):
    """Pages of every request in random places; the requests of a group start with the same ones.  (table, pages)"""
    pages = (lens + PAGE - 1) // PAGE
    shared, g_of = torch.zeros_like(lens), torch.full_like(lens, -1)
    if case["kind"] == "prefix":
        g_of = _group_of(case)
        shared = torch.where(g_of >= 0, _prefix_lengths(case) // PAGE, shared)
    first = {}
    total = int((pages - shared).sum()) + sum(int(shared[(g_of == g).nonzero()[0]]) for g in set(g_of.tolist()) - {-1})
    if case["kind"] == "decode":  # an engine's pool: what the case can need at most, whatever the seed
        total = int(((_lengths(case["batch"], case["lo"], case["hi"], case["dist"], None) + PAGE - 1) // PAGE).sum())
    free = torch.randperm(total, generator=gen).to(torch.int32)
    table, at = torch.zeros(len(lens), int(pages.max()), dtype=torch.int32), 0
    for b in range(len(lens)):
        g, s, n = int(g_of[b]), int(shared[b]), int(pages[b])
        if g >= 0:
            if g not in first:
                first[g], at = free[at:at + s], at + s
            table[b, :s] = first[g]
        table[b, s:n] = free[at:at + n - s]
        at += n - s
    return table.to(DEV), total


def _cache(pages, case, gen):
    """(cache [pages, 16, Hkv, D], scale [Hkv]): N(0, 1) values, quantised with amax / 448 per head where the cache is FP8."""
    hkv, d = case["kv_heads"], case["head_dim"]
    hnd = case.get("layout") == "hnd"
    x = torch.randn((pages, hkv, PAGE, d) if hnd else (pages, PAGE, hkv, d), generator=gen, device=DEV)
    if hnd:
        x = x.transpose(1, 2)
    if case.get("kv", "fp8") != "fp8":
        return x.to(DTYPES[case["dtype"]]), torch.ones(hkv, device=DEV)
    scale = x.abs().amax(dim=(0, 1, 3)) / FP8_MAX
    return (x / scale[None, None, :, None]).clamp_(-FP8_MAX, FP8_MAX).to(torch.float8_e4m3fn), scale


def _rotary_table(rows, rotary):
    freq = 10000.0 ** (-torch.arange(0, rotary, 2, device=DEV, dtype=torch.float64) / rotary)
    angle = torch.arange(rows, device=DEV, dtype=torch.float64)[:, None] * freq
    return torch.cat([angle.cos(), angle.sin()], 1)


def _split_qkv(qkv, case):
    """Query, key and value as the views of the projection's output that an engine hands on."""
    hq, hkv, d = case["q_heads"], case["kv_heads"], case["head_dim"]
    rows = qkv.view(qkv.shape[0], hq + 2 * hkv, d)
    return rows[:, :hq], rows[:, hq:hq + hkv], rows[:, hq + hkv:]


def _inputs(case, seed):
    """Everything the program is given, in plain torch."""
    cpu = torch.Generator().manual_seed(seed)
    gen = torch.Generator(device=DEV).manual_seed(seed)
    hq, hkv, d = case["q_heads"], case["kv_heads"], case["head_dim"]
    dtype = DTYPES[case["dtype"]]
    x = {}
    if case["kind"] == "append":
        tokens = case["tokens"]
        x["positions"] = torch.arange(tokens, device=DEV) + int(torch.randint(0, 512, (1,), generator=cpu))
        table = _rotary_table(tokens + 512, case["rotary"])
        x["cos_sin"] = table.float() if case["table"] == "f32" else table.to(dtype)
        pages = -(-tokens // PAGE)
        ids = torch.randperm(pages, generator=cpu).to(DEV)
        at = torch.arange(tokens, device=DEV)
        x["slots"] = ids[at // PAGE] * PAGE + at % PAGE
        x["qkv"] = torch.randn(tokens, (hq + 2 * hkv) * d, generator=gen, device=DEV).to(dtype)
        cache_dtype = torch.float8_e4m3fn if case["kv"] == "fp8" else dtype
        x["k_cache"] = torch.zeros(pages, PAGE, hkv, d, device=DEV, dtype=cache_dtype)
        x["v_cache"] = torch.zeros_like(x["k_cache"])
        x["k_scale"] = torch.rand(hkv, generator=gen, device=DEV) * 0.01 + 0.005
        x["v_scale"] = torch.rand(hkv, generator=gen, device=DEV) * 0.01 + 0.005
        return x
    lens = _case_lengths(case, cpu)
    table, pages = _block_table(case, lens, cpu)
    x["max_len"] = int(lens.max())
    x["lens"], x["table"] = lens.to(torch.int32).to(DEV), table
    x["layers"] = []
    for _ in range(max(1, case["layers"])):
        k, ks = _cache(pages, case, gen)
        v, vs = _cache(pages, case, gen)
        layer = {"k": k, "v": v, "ks": ks, "vs": vs}
        if case.get("append"):
            layer["qkv"] = torch.randn(len(lens), (hq + 2 * hkv) * d, generator=gen, device=DEV).to(dtype)
        else:
            layer["q"] = torch.randn(len(lens), hq, d, generator=gen, device=DEV).to(dtype)
        x["layers"].append(layer)
    if case.get("append"):
        last = (lens - 1).to(DEV)
        x["positions"] = last
        x["slots"] = table.gather(1, (last // PAGE)[:, None])[:, 0].to(torch.int64) * PAGE + last % PAGE
        x["cos_sin"] = _rotary_table(x["max_len"], d).float()
    return x


# ---------------------------------------------------------------------------------- the program
def prepare(case, seed):
    from single_gpu_inference_lab_b200 import l20_paged_decode as ops
    from single_gpu_inference_lab_b200 import l20_paged_split_kv as split_kv
    from single_gpu_inference_lab_b200 import l20_rope_kv
    from single_gpu_inference_lab_b200 import l20_shared_prefix_decode_dispatch as prefix

    x = _inputs(case, seed)
    if case["kind"] == "append":
        work = torch.empty_like(x["qkv"])
        q, k, v = _split_qkv(work, case)
        scales = dict(k_scale=x["k_scale"], v_scale=x["v_scale"]) if case["kv"] == "fp8" else {}

        def append():
            work.copy_(x["qkv"])  # stands for the projection that fills it: the rotation is in place
            l20_rope_kv.l20_rope_and_cache(q, k, v, x["positions"], x["cos_sin"], case["neox"], x["k_cache"], x["v_cache"],
                                           x["slots"], **scales)
            return work, x["k_cache"].view(torch.uint8), x["v_cache"].view(torch.uint8)

        return append

    layers, table, lens, max_len = x["layers"], x["table"], x["lens"], x["max_len"]
    q0 = layers[0]["q"] if "q" in layers[0] else torch.empty(case["batch"], case["q_heads"], case["head_dim"], device=DEV,
                                                             dtype=DTYPES[case["dtype"]])
    outs = [torch.empty_like(q0) for _ in layers]

    if case["kind"] == "prefix":
        if case["groups"] == 0:
            split = prefix.choose_suffix_split_size(case["batch"], case["kv_heads"], max_len - case["prefix"])
            ws = prefix.allocate_shared_prefix_workspace(q0, max_len, case["prefix"], suffix_split_size=split)

            def step():
                for layer, out in zip(layers, outs):
                    prefix.shared_paged_prefix_paged_suffix_gqa_decode_attention_fp8(
                        layer["q"], layer["k"], layer["v"], table, lens, case["prefix"], k_scale=layer["ks"], v_scale=layer["vs"],
                        max_seq_len=max_len, suffix_split_size=split, output=out, workspace=ws)
                return outs
        else:
            max_suffix = max(max_len - case["prefix"], PAGE)
            split = prefix.choose_suffix_split_size(case["batch"], case["kv_heads"], max_suffix)
            slots = -(-max_len // 256) + -(-max_suffix // split)
            shape = (case["batch"], case["q_heads"], slots)
            ws = [torch.empty(s, device=DEV, dtype=torch.float32) for s in ((*shape, 128), shape, shape)]
            max_groups = 4
            buffer = torch.empty(torch.ops.l20_stack.prefix_groups_bytes(case["batch"], max_groups) // 4, dtype=torch.int32, device=DEV)

            def step():
                groups = ops.group_shared_prefixes(table, seq_lens=lens, min_batch=4, min_prefix_len=case["prefix"],
                                                   max_groups=max_groups, buffer=buffer)
                for layer, out in zip(layers, outs):
                    ops.shared_prefix_decode_grouped_fp8_e4m3(
                        layer["q"], layer["k"], layer["v"], table, lens, *ws, out, layer["ks"], layer["vs"], max_len, split, groups,
                        max_suffix_len=max_suffix)
                return outs
        return _record(step)

    ws = split_kv.allocate_l20_paged_split_kv_workspace(q0, max_len, num_kv_heads=case["kv_heads"])
    fp8 = case["kv"] == "fp8"
    attend = split_kv.l20_paged_split_kv_attention_fp8 if fp8 else split_kv.l20_paged_split_kv_attention

    if case["layers"] == 0:
        layer, out = layers[0], outs[0]
        scales = dict(k_scale=float(layer["ks"][0]), v_scale=float(layer["vs"][0])) if case["layout"] == "nhd" \
            else dict(k_scale=layer["ks"], v_scale=layer["vs"])  # one float for the layer, or one for each head

        def call():
            return attend(layer["q"], layer["k"], layer["v"], table, lens, max_seq_len=max_len, output=out, workspace=ws,
                          **(scales if fp8 else {}))

        return call

    views = []
    for layer in layers:
        if case["append"]:
            layer["work"] = torch.empty_like(layer["qkv"])
            views.append(_split_qkv(layer["work"], case))
    plan = split_kv.plan_l20_paged_split_kv(q0, layers[0]["k"], layers[0]["v"], table, lens, max_seq_len=max_len, workspace=ws)

    def step():
        if plan is not None:
            split_kv.plan_l20_paged_split_kv(q0, layers[0]["k"], layers[0]["v"], table, lens, max_seq_len=max_len, workspace=ws,
                                             plan=plan)
        for i, (layer, out) in enumerate(zip(layers, outs)):
            scales = dict(k_scale=layer["ks"], v_scale=layer["vs"]) if fp8 else {}
            q = layer.get("q")
            if case["append"]:
                layer["work"].copy_(layer["qkv"])  # stands for the projection
                q, k, v = views[i]
                l20_rope_kv.l20_rope_and_cache(q, k, v, x["positions"], x["cos_sin"], True, layer["k"], layer["v"], x["slots"], **scales)
            attend(q, layer["k"], layer["v"], table, lens, max_seq_len=max_len, output=out, workspace=ws, plan=plan,
                   metadata_stable=i > 0 or case["append"], **scales)
        if case["append"]:
            return outs, [layer["work"] for layer in layers], [layer[c].view(torch.uint8) for layer in layers for c in "kv"]
        return outs

    return _record(step)


def _record(step):
    """A callable that replays `step` from a CUDA graph."""
    step()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        outputs = step()

    def replay(keep=step):  # the graph reads and writes the tensors that `step` holds: they live as long as it does
        graph.replay()
        return outputs

    return replay


def run(state):
    return state()


# ---------------------------------------------------------------------------------- what a pass cannot do without
def work(case):
    hq, hkv, d = case["q_heads"], case["kv_heads"], case["head_dim"]
    if case["kind"] == "append":
        t = case["tokens"]
        cache = 1 if case["kv"] == "fp8" else 2
        row = (hq + 2 * hkv) * d * 2
        # the projection's stand-in reads and writes the rows, the rotation reads them and writes query and key back
        return {"bytes": t * (3 * row + (hq + hkv) * d * 2 + 2 * hkv * d * cache + case["rotary"] * (4 if case["table"] == "f32" else 2) + 16),
                "flops": t * 3 * (hq + hkv) * case["rotary"]}
    lens = _case_lengths(case, torch.Generator().manual_seed(0))
    attended = int(lens.sum())
    tokens = attended
    if case["kind"] == "prefix":
        g_of, shared = _group_of(case), _prefix_lengths(case)
        for g in set(g_of.tolist()) - {-1}:
            members = (g_of == g).nonzero()[:, 0]
            tokens -= int(shared[members].sum()) - int(shared[members[0]])
    layers = max(1, case["layers"])
    elem = 1 if case.get("kv", "fp8") == "fp8" else 2
    per_layer = tokens * hkv * d * 2 * elem + 2 * len(lens) * hq * d * 2 + 4 * int((lens + PAGE - 1).sum() // PAGE)
    if case.get("append"):
        per_layer += len(lens) * (3 * (hq + 2 * hkv) + (hq + hkv)) * d * 2
    return {"bytes": layers * per_layer, "flops": layers * 4 * attended * hq * d}


def tolerance(case):
    if case["kind"] == "append":
        return "exact"
    # 16-bit outputs and 16-bit probabilities: two right implementations differ by flipped roundings (the rounded output is
    # 1.7e-3 in bf16 and 2.6e-4 in fp16 from the exact one)
    if case["dtype"] == "fp16":
        return {"rel": 1e-3, "max": 5e-3}
    return {"rel": 5e-3, "max": 3e-2}


# ---------------------------------------------------------------------------------- the same in 64 bits
def _rotated(x, positions, cos_sin, neox):
    """[T, H, D] rotated in 64 bits."""
    half = cos_sin.shape[1] // 2
    cs = cos_sin.double()[positions][:, None, :]
    c, s = cs[..., :half], cs[..., half:]
    y = x.double().clone()
    first, second = (slice(0, half), slice(half, 2 * half)) if neox else (slice(0, 2 * half, 2), slice(1, 2 * half, 2))
    a, b = x[..., first].double(), x[..., second].double()
    y[..., first], y[..., second] = a * c - b * s, b * c + a * s
    return y


def _attention(q, k_cache, v_cache, table, lens, ks, vs):
    out = torch.empty(q.shape, dtype=torch.float64, device=DEV)
    hkv, d = k_cache.shape[2], q.shape[2]
    as_rows = (lambda t: t.view(torch.uint8)) if k_cache.dtype == torch.float8_e4m3fn else (lambda t: t)
    for b, n in enumerate(lens.tolist()):
        pages = table[b, :-(-n // PAGE)].long()

        def rows(cache, scale):
            x = as_rows(cache)[pages].view(cache.dtype).float().reshape(-1, hkv, d)[:n]
            return x.double().transpose(0, 1) * scale.double()[:, None, None]

        k = rows(k_cache, ks)
        p = torch.softmax(q[b].double().view(hkv, -1, d) @ k.transpose(1, 2) * d ** -0.5, -1)
        del k
        out[b] = (p @ rows(v_cache, vs)).reshape(-1, d)
    return out


def exact(case, seed):
    x = _inputs(case, seed)
    if case["kind"] == "append":
        q, k, v = _split_qkv(x["qkv"], case)
        both = [_rotated(t, x["positions"], x["cos_sin"], case["neox"]) for t in (q, k)]
        return torch.cat([*both, v.double()], 1).reshape(x["qkv"].shape), None, None
    outs, rows = [], []
    for layer in x["layers"]:
        ks, vs = layer["ks"], layer["vs"]
        if case["kind"] == "decode" and case["layers"] == 0 and case["kv"] == "fp8" and case["layout"] == "nhd":
            ks, vs = ks[:1].expand_as(ks), vs[:1].expand_as(vs)
        q = layer.get("q")
        if case.get("append"):
            q, k, v = _split_qkv(layer["qkv"], case)
            q64, k64 = (_rotated(t, x["positions"], x["cos_sin"], True) for t in (q, k))
            rows.append(torch.cat([q64, k64, v.double()], 1).reshape(layer["qkv"].shape))
            q, k = q64.to(q.dtype), k64.to(k.dtype)
            at = (x["slots"] // PAGE, x["slots"] % PAGE)
            for cache, new, scale in ((layer["k"], k, ks), (layer["v"], v, vs)):
                stored = (new.float() / scale[:, None]).clamp(-FP8_MAX, FP8_MAX).to(torch.float8_e4m3fn)
                cache.view(torch.uint8)[at] = stored.view(torch.uint8)
        outs.append(_attention(q, layer["k"], layer["v"], x["table"], x["lens"], ks, vs))
    return (outs, rows, [None] * (2 * len(outs))) if case.get("append") else outs if case["layers"] else outs[0]
