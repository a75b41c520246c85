"""The producer step (rotary embedding + paged KV append, optionally quantised to FP8):
the CPU oracle against the reference's own outputs, and the CUDA kernel against the oracle --
bit for bit -- and against the decode operator that consumes what it wrote."""

import pytest
import torch

from oracle import paged_decode_oracle as decode_oracle
from oracle import rope_kv_oracle as oracle

from helpers import assert_within_gate

DEV = "cuda:0"


def golden_inputs(case):
    """The seeded inputs tests/golden/make_golden.py fed to the reference's rope_kv_reference."""
    tokens, hkv, d, rot = case["tokens"], case["kv_heads"], case["head_dim"], case["rotary_dim"]
    dtype = getattr(torch, case["dtype"])
    gen = torch.Generator().manual_seed(41)
    k = torch.randn(tokens, hkv, d, generator=gen).to(dtype)
    v = torch.randn(tokens, hkv, d, generator=gen).to(dtype)
    angle = torch.rand(tokens, rot // 2, generator=gen) * 6.2831853
    slots = torch.randperm(4 * tokens, generator=gen)[:tokens]
    return k, v, torch.cos(angle), torch.sin(angle), slots, dtype


def test_oracle_reproduces_reference_rope_kv_outputs_bit_for_bit(golden):
    for name, case in golden["rope"].items():
        k, v, cos, sin, slots, dtype = golden_inputs(case)
        tokens, hkv, d = k.shape
        # the reference writes a flat [slots, Hkv, D] cache from per-token cos / sin rows: the same thing
        # as a one-token-per-block paged cache and a cos_sin table indexed by the token number
        table = torch.cat([cos, sin], dim=1)
        kc = torch.zeros(4 * tokens, 1, hkv, d, dtype=dtype)
        _, _, kc2, vc2 = oracle.rope_and_cache(
            torch.zeros(tokens, hkv, d, dtype=dtype), k, v, torch.arange(tokens), table, True, kc, torch.zeros_like(kc), slots
        )
        assert torch.equal(kc2[:, 0].view(torch.int16), case["key_cache"].view(torch.int16)), name
        assert torch.equal(vc2[:, 0].view(torch.int16), case["value_cache"].view(torch.int16)), name


def paged_golden_inputs(case):
    """The seeded inputs tests/golden/make_golden.py fed to the reference's paged_rope_kv_reference
    (src/l20_stack/ops/triton_rope_kv.py:176-205): same recipe as paged_rope_inputs there."""
    seqs, tokens, hkv, d, rot = case["seqs"], case["tokens"], case["kv_heads"], case["head_dim"], case["rotary_dim"]
    dtype = getattr(torch, case["dtype"])
    gen = torch.Generator().manual_seed(43)
    k = torch.randn(tokens, hkv, d, generator=gen).to(dtype)
    v = torch.randn(tokens, hkv, d, generator=gen).to(dtype)
    angle = torch.rand(tokens, rot // 2, generator=gen) * 6.2831853
    max_blocks = 6
    table = torch.randperm(seqs * max_blocks, generator=gen).reshape(seqs, max_blocks)
    flat = torch.randperm(seqs * max_blocks * 16, generator=gen)[:tokens]
    sequence_ids, positions = flat // (max_blocks * 16), flat % (max_blocks * 16)
    # what an engine hands the operator: the slot of every token, resolved through the block table
    slots = table[sequence_ids, positions // 16] * 16 + positions % 16
    cos_sin = torch.cat([torch.cos(angle), torch.sin(angle)], dim=1)  # one row per token, indexed by token number
    return k, v, cos_sin, slots, table.numel(), dtype


def check_against_paged_golden(case, kc, vc, slots, name):
    from helpers import digest

    assert torch.equal(kc[slots // 16, slots % 16].view(torch.int16), case["key_rows"].view(torch.int16)), name
    assert torch.equal(vc[slots // 16, slots % 16].view(torch.int16), case["value_rows"].view(torch.int16)), name
    assert digest(kc) == case["key_cache_sha256"] and digest(vc) == case["value_cache_sha256"], name


def test_oracle_reproduces_reference_paged_rope_kv_outputs_bit_for_bit(golden):
    for name, case in golden["rope_paged"].items():
        k, v, cos_sin, slots, blocks, dtype = paged_golden_inputs(case)
        tokens, hkv, d = k.shape
        kc = torch.zeros(blocks, 16, hkv, d, dtype=dtype)
        _, _, kc2, vc2 = oracle.rope_and_cache(torch.zeros(tokens, hkv, d, dtype=dtype), k, v, torch.arange(tokens), cos_sin,
                                               True, kc, torch.zeros_like(kc), slots)
        check_against_paged_golden(case, kc2, vc2, slots, name)


@pytest.mark.gpu
def test_kernel_reproduces_reference_paged_rope_kv_outputs_bit_for_bit(built_libs, golden):
    from single_gpu_inference_lab_b200 import l20_rope_kv

    for name, case in golden["rope_paged"].items():
        k, v, cos_sin, slots, blocks, dtype = paged_golden_inputs(case)
        tokens, hkv, d = k.shape
        kc = torch.zeros(blocks, 16, hkv, d, dtype=dtype, device=DEV)
        vc = torch.zeros_like(kc)
        q = torch.zeros(tokens, hkv, d, dtype=dtype, device=DEV)
        l20_rope_kv.l20_rope_and_cache(q, k.to(DEV), v.to(DEV), torch.arange(tokens, device=DEV), cos_sin.to(DEV), True,
                                       kc, vc, slots.to(DEV))
        torch.cuda.synchronize()
        check_against_paged_golden(case, kc.cpu(), vc.cpu(), slots, name)


def make_step(seed, tokens, hq, hkv, d, rot, dtype, cache_dtype, table_dtype, block_size=16):
    gen = torch.Generator().manual_seed(seed)
    q = torch.randn(tokens, hq, d, generator=gen).to(dtype)
    k = torch.randn(tokens, hkv, d, generator=gen).to(dtype)
    v = torch.randn(tokens, hkv, d, generator=gen).to(dtype)
    max_pos = 512
    angle = torch.rand(max_pos, rot // 2, generator=gen) * 6.2831853
    cos_sin = torch.cat([torch.cos(angle), torch.sin(angle)], dim=1).to(table_dtype)
    positions = torch.randint(0, max_pos, (tokens,), generator=gen)
    blocks = 2 * tokens // block_size + 3
    slots = torch.randperm(blocks * block_size, generator=gen)[:tokens]
    slots[tokens // 2] = -1  # a padded token: rotated, not stored
    if cache_dtype == torch.float8_e4m3fn:
        kc = torch.full((blocks, block_size, hkv, d), 0x11, dtype=torch.uint8).view(torch.float8_e4m3fn)
        vc = torch.full((blocks, block_size, hkv, d), 0x22, dtype=torch.uint8).view(torch.float8_e4m3fn)
        ks = torch.rand(hkv, generator=gen) * 0.02 + 0.003
        vs = torch.rand(hkv, generator=gen) * 0.02 + 0.003
    else:
        kc = torch.full((blocks, block_size, hkv, d), 7.0, dtype=dtype)
        vc = torch.full((blocks, block_size, hkv, d), -7.0, dtype=dtype)
        ks = vs = None
    return q, k, v, positions, cos_sin, kc, vc, slots, ks, vs


@pytest.mark.gpu
@pytest.mark.parametrize("is_neox", [True, False])
@pytest.mark.parametrize("cache", ["same", "fp8"])
def test_kernel_matches_oracle_bit_for_bit(built_libs, is_neox, cache):
    from single_gpu_inference_lab_b200 import l20_rope_kv

    for seed, (tokens, hq, hkv, d, rot, dtype, table_dtype) in enumerate([
        (64, 16, 2, 128, 128, torch.bfloat16, torch.float32),
        (5, 28, 4, 128, 64, torch.float16, torch.float16),
        (256, 14, 2, 64, 64, torch.bfloat16, torch.bfloat16),
        (1, 32, 8, 128, 32, torch.float16, torch.float32),
        (33, 8, 8, 128, 128, torch.float16, torch.float16),  # the vectorised kernel in fp16 with an fp16 table
        (700, 16, 2, 128, 128, torch.bfloat16, torch.float32),
    ]):
        cache_dtype = torch.float8_e4m3fn if cache == "fp8" else dtype
        q, k, v, pos, cs, kc, vc, slots, ks, vs = make_step(seed, tokens, hq, hkv, d, rot, dtype, cache_dtype, table_dtype)
        eq, ek, ekc, evc = oracle.rope_and_cache(q, k, v, pos, cs, is_neox, kc, vc, slots, ks, vs)
        g = [t.to(DEV) for t in (q, k, v, pos, cs, kc, vc, slots)]
        gq, gk, gv, gpos, gcs, gkc, gvc, gslots = g
        l20_rope_kv.l20_rope_and_cache(gq, gk, gv, gpos, gcs, is_neox, gkc, gvc, gslots,
                                       k_scale=None if ks is None else ks.to(DEV), v_scale=None if vs is None else vs.to(DEV))
        torch.cuda.synchronize()
        what = f"tokens={tokens} hq={hq} hkv={hkv} d={d} rot={rot} {dtype} neox={is_neox} cache={cache}"
        assert torch.equal(gq.cpu().view(torch.int16), eq.view(torch.int16)), "query " + what
        assert torch.equal(gk.cpu().view(torch.int16), ek.view(torch.int16)), "key " + what
        as_bits = (lambda t: t.view(torch.uint8)) if cache == "fp8" else (lambda t: t.view(torch.int16))
        assert torch.equal(as_bits(gkc.cpu()), as_bits(ekc)), "key cache " + what
        assert torch.equal(as_bits(gvc.cpu()), as_bits(evc)), "value cache " + what


@pytest.mark.gpu
def test_append_then_decode_equals_the_oracles(built_libs):
    """One decode step of a small model layer: append the new token of every sequence with the
    producer kernel, then attend with the FP8 decode operator; compare with the two CPU oracles
    chained the same way."""
    from single_gpu_inference_lab_b200 import l20_paged_split_kv, l20_rope_kv
    from single_gpu_inference_lab_b200.workloads import make_inputs

    w = make_inputs("qwen2.5-coder-3b-b64", seed=12, batch=12, shrink=0.2)
    batch, hq, d = w.query.shape
    hkv = w.key_cache.shape[2]
    gen = torch.Generator().manual_seed(3)
    # the new token of each sequence overwrites its last position
    positions = (w.seq_lens.long() - 1)
    slots = w.block_table[torch.arange(batch), positions // 16].long() * 16 + positions % 16
    q = torch.randn(batch, hq, d, generator=gen).to(torch.bfloat16)
    k = torch.randn(batch, hkv, d, generator=gen).to(torch.bfloat16)
    v = torch.randn(batch, hkv, d, generator=gen).to(torch.bfloat16)
    angle = torch.arange(int(positions.max()) + 1)[:, None] * (1e4 ** (-torch.arange(0, d, 2) / d))[None, :]
    cos_sin = torch.cat([torch.cos(angle), torch.sin(angle)], dim=1).float()
    eq, _, ekc, evc = oracle.rope_and_cache(q, k, v, positions, cos_sin, True, w.key_cache, w.value_cache, slots,
                                            w.k_scale, w.v_scale)
    exp = decode_oracle.reference(eq, ekc, evc, w.block_table.long(), w.seq_lens, w.k_scale, w.v_scale)
    g = w.to(DEV)
    gq, gk, gv = q.to(DEV), k.to(DEV), v.to(DEV)
    l20_rope_kv.l20_rope_and_cache(gq, gk, gv, positions.to(DEV), cos_sin.to(DEV), True, g.key_cache, g.value_cache,
                                   slots.to(DEV), k_scale=g.k_scale, v_scale=g.v_scale)
    out = l20_paged_split_kv.l20_paged_split_kv_attention_fp8(
        gq, g.key_cache, g.value_cache, g.block_table, g.seq_lens, k_scale=g.k_scale, v_scale=g.v_scale,
        max_seq_len=w.max_seq_len, split_size=256)
    torch.cuda.synchronize()
    assert torch.equal(g.key_cache.cpu().view(torch.uint8), ekc.view(torch.uint8))
    assert_within_gate(out, exp, "append + decode")
    # The same step with a plan and the caller's word that the kernel in front of the decode call
    # writes K/V only at each sequence's last position (kv_stable): the balanced kernel may then
    # fetch older pages before the append has completed, and must still see the new token.
    w2 = make_inputs("qwen2.5-coder-3b-b64", seed=12, batch=64, shrink=0.5)
    batch = w2.query.shape[0]
    positions = (w2.seq_lens.long() - 1)
    slots = w2.block_table[torch.arange(batch), positions // 16].long() * 16 + positions % 16
    q = torch.randn(batch, hq, d, generator=gen).to(torch.bfloat16)
    k = torch.randn(batch, hkv, d, generator=gen).to(torch.bfloat16)
    v = torch.randn(batch, hkv, d, generator=gen).to(torch.bfloat16)
    angle = torch.arange(int(positions.max()) + 1)[:, None] * (1e4 ** (-torch.arange(0, d, 2) / d))[None, :]
    cos_sin = torch.cat([torch.cos(angle), torch.sin(angle)], dim=1).float()
    eq, _, ekc, evc = oracle.rope_and_cache(q, k, v, positions, cos_sin, True, w2.key_cache, w2.value_cache, slots,
                                            w2.k_scale, w2.v_scale)
    exp = decode_oracle.reference(eq, ekc, evc, w2.block_table.long(), w2.seq_lens, w2.k_scale, w2.v_scale)
    g = w2.to(DEV)
    kc0, vc0 = g.key_cache.clone(), g.value_cache.clone()
    ws = l20_paged_split_kv.allocate_l20_paged_split_kv_workspace(g.query, w2.max_seq_len, split_size=512)
    plan = l20_paged_split_kv.plan_l20_paged_split_kv(g.query, g.key_cache, g.value_cache, g.block_table, g.seq_lens,
                                                      max_seq_len=w2.max_seq_len, split_size=512, workspace=ws)
    cs, pos, sl = cos_sin.to(DEV), positions.to(DEV), slots.to(DEV)
    for rep in range(8):
        g.key_cache.copy_(kc0)
        g.value_cache.copy_(vc0)
        gq, gk, gv = q.to(DEV), k.to(DEV), v.to(DEV)
        l20_rope_kv.l20_rope_and_cache(gq, gk, gv, pos, cs, True, g.key_cache, g.value_cache, sl,
                                       k_scale=g.k_scale, v_scale=g.v_scale)
        out = l20_paged_split_kv.l20_paged_split_kv_attention_fp8(
            gq, g.key_cache, g.value_cache, g.block_table, g.seq_lens, k_scale=g.k_scale, v_scale=g.v_scale,
            max_seq_len=w2.max_seq_len, split_size=512, workspace=ws, plan=plan, metadata_stable=True, kv_stable=True)
        torch.cuda.synchronize()
        assert_within_gate(out, exp, f"append + planned decode with early K/V, repetition {rep}")


@pytest.mark.gpu
@pytest.mark.parametrize("kv_stable", [False, True])
def test_recorded_producer_and_decode_read_what_the_step_wrote(built_libs, kv_stable):
    """Plan, append and decode recorded, then replayed behind one another with new lengths, rows and slots: the decode kernel,
    resident while the append kernel runs, reads this replay's plan, rotated queries and new tokens."""
    from single_gpu_inference_lab_b200 import l20_paged_split_kv, l20_rope_kv
    from single_gpu_inference_lab_b200.workloads import make_inputs

    w = make_inputs("qwen2.5-coder-3b-b64", seed=13, batch=16, shrink=0.25)
    batch, hq, d = w.query.shape
    hkv, replays = w.key_cache.shape[2], 6
    gen = torch.Generator().manual_seed(14)
    angle = torch.arange(w.max_seq_len)[:, None] * (1e4 ** (-torch.arange(0, d, 2) / d))[None, :]
    cos_sin = torch.cat([torch.cos(angle), torch.sin(angle)], dim=1).float()
    lens = torch.stack([(w.seq_lens - i).clamp_min(1) for i in range(replays)])
    rows = torch.randn(replays, batch, hq + 2 * hkv, d, generator=gen).to(torch.bfloat16)
    positions = lens.long() - 1
    slots = w.block_table[torch.arange(batch), positions // 16].long() * 16 + positions % 16
    g = w.to(DEV)
    g_lens, g_rows, g_positions, g_slots, g_cs = (t.to(DEV) for t in (lens, rows, positions, slots, cos_sin))
    now_lens, now_rows, now_positions, now_slots = (t[0].clone() for t in (g_lens, g_rows, g_positions, g_slots))
    ws = l20_paged_split_kv.allocate_l20_paged_split_kv_workspace(g.query, w.max_seq_len, split_size=512)
    shape = dict(max_seq_len=w.max_seq_len, split_size=512, workspace=ws)
    caches = g.key_cache, g.value_cache, g.block_table
    plan = l20_paged_split_kv.plan_l20_paged_split_kv(g.query, *caches, now_lens, **shape)
    out, work = torch.empty_like(g.query), torch.empty_like(now_rows)

    def step():
        l20_paged_split_kv.plan_l20_paged_split_kv(g.query, *caches, now_lens, plan=plan, **shape)
        work.copy_(now_rows)
        q, k, v = work[:, :hq], work[:, hq:hq + hkv], work[:, hq + hkv:]
        l20_rope_kv.l20_rope_and_cache(q, k, v, now_positions, g_cs, True, g.key_cache, g.value_cache, now_slots,
                                       k_scale=g.k_scale, v_scale=g.v_scale)
        l20_paged_split_kv.l20_paged_split_kv_attention_fp8(q, *caches, now_lens, k_scale=g.k_scale, v_scale=g.v_scale, plan=plan,
                                                            output=out, metadata_stable=True, kv_stable=kv_stable, **shape)

    kc, vc = w.key_cache, w.value_cache
    kc0, vc0 = g.key_cache.clone(), g.value_cache.clone()
    step()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        step()
    g.key_cache.copy_(kc0)
    g.value_cache.copy_(vc0)
    got = []
    for r in range(replays):
        for now, new in ((now_lens, g_lens), (now_rows, g_rows), (now_positions, g_positions), (now_slots, g_slots)):
            now.copy_(new[r])
        graph.replay()
        got.append(out.clone())
    torch.cuda.synchronize()
    for r in range(replays):
        q, k, v = rows[r][:, :hq], rows[r][:, hq:hq + hkv], rows[r][:, hq + hkv:]
        q, _, kc, vc = oracle.rope_and_cache(q, k, v, positions[r], cos_sin, True, kc, vc, slots[r], w.k_scale, w.v_scale)
        exp = decode_oracle.reference(q, kc, vc, w.block_table.long(), lens[r], w.k_scale, w.v_scale)
        assert_within_gate(got[r], exp, f"replay {r} kv_stable={kv_stable}")


def test_wrapper_argument_errors_without_a_gpu():
    from single_gpu_inference_lab_b200 import l20_rope_kv

    q = torch.zeros(2, 4, 128, dtype=torch.bfloat16)
    with pytest.raises(RuntimeError, match="requires an SM100 GPU"):
        l20_rope_kv.l20_rope_and_cache(q, q, q, torch.zeros(2, dtype=torch.long), torch.zeros(8, 128), True,
                                       torch.zeros(1, 16, 4, 128, dtype=torch.bfloat16),
                                       torch.zeros(1, 16, 4, 128, dtype=torch.bfloat16), torch.zeros(2, dtype=torch.long))


@pytest.mark.gpu
@pytest.mark.parametrize("is_neox", [True, False])
@pytest.mark.parametrize("cache", ["same", "fp8"])
def test_chunk_kernel_edges_bit_for_bit(built_libs, is_neox, cache):
    """The kernel of 16-byte chunks where it can go wrong: every number of threads per token with a ragged last CTA,
    partial rotation, frequency groups that do not divide a token's threads, more heads than the threads take at once,
    scales that are powers of two (ties) and that are not; and rotary_dim 24, which the scalar kernel takes."""
    from single_gpu_inference_lab_b200 import l20_rope_kv

    for seed, (tokens, hq, hkv, d, rot, dtype, table_dtype) in enumerate([
        (256, 5, 1, 128, 64, torch.bfloat16, torch.float32),
        (257, 28, 4, 128, 128, torch.bfloat16, torch.bfloat16),
        (1027, 3, 3, 80, 48, torch.float16, torch.float32),
        (1030, 40, 8, 64, 16, torch.bfloat16, torch.float32),
        (2, 71, 9, 128, 96, torch.float16, torch.float16),
        (1201, 16, 2, 128, 128, torch.bfloat16, torch.float32),
        (2401, 6, 2, 64, 64, torch.float16, torch.float32),
        (301, 14, 2, 256, 256, torch.bfloat16, torch.float32),
        (300, 4, 2, 64, 24, torch.bfloat16, torch.float32),
    ]):
        cache_dtype = torch.float8_e4m3fn if cache == "fp8" else dtype
        q, k, v, pos, cs, kc, vc, slots, ks, vs = make_step(100 + seed, tokens, hq, hkv, d, rot, dtype, cache_dtype, table_dtype)
        if ks is not None and seed % 2:
            ks, vs = torch.full_like(ks, 0.25), torch.full_like(vs, 2.0)
        want = oracle.rope_and_cache(q, k, v, pos, cs, is_neox, kc, vc, slots, ks, vs)
        # rows of one projection output, as an engine hands them on
        rows = torch.cat([q, k, v], 1).to(DEV)
        gq, gk, gv = rows[:, :hq], rows[:, hq:hq + hkv], rows[:, hq + hkv:]
        gkc, gvc = kc.to(DEV), vc.to(DEV)
        l20_rope_kv.l20_rope_and_cache(gq, gk, gv, pos.to(DEV), cs.to(DEV), is_neox, gkc, gvc, slots.to(DEV),
                                       k_scale=None if ks is None else ks.to(DEV), v_scale=None if vs is None else vs.to(DEV))
        as_bytes = lambda t: t.cpu().contiguous().view(torch.uint8)
        for name, got, exp in zip(("query", "key", "key cache", "value cache"), (gq, gk, gkc, gvc), want):
            assert torch.equal(as_bytes(got), as_bytes(exp)), f"{name}: case {seed} neox={is_neox} cache={cache}"
        assert torch.equal(as_bytes(gv), as_bytes(v))


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_every_finite_value_quantised_as_by_a_division(built_libs, dtype):
    """All finite 16-bit values as V, at 75 scales (powers of two, where quotients tie, their neighbours, and others): the bytes
    of x / scale rounded, saturated, without a division per value."""
    from single_gpu_inference_lab_b200 import l20_rope_kv

    bits = torch.arange(-(1 << 15), 1 << 15, dtype=torch.int32).to(torch.int16)
    x = bits.view(dtype)
    x = torch.where(x.float().abs() <= torch.finfo(dtype).max, x, torch.zeros_like(x))  # (NaN compares false)
    d, hkv = 128, 4
    tokens = x.numel() // (d * hkv)
    v = x.view(tokens, hkv, d)
    zeros = torch.zeros_like(v)
    pos, slots = torch.zeros(tokens, dtype=torch.long), torch.arange(tokens)
    cs = torch.zeros(1, d)
    gen = torch.Generator().manual_seed(17)
    powers = [2.0 ** e for e in range(-12, 13)]
    near = [p * (1 + s * 2.0 ** -23) for p in powers[::5] for s in (-1, 1)]
    others = torch.exp(torch.rand(75 - len(powers) - len(near), generator=gen) * 16 - 11).tolist()
    g = [t.to(DEV) for t in (zeros, zeros, v, pos, cs, slots)]
    kc = torch.zeros(tokens // 16, 16, hkv, d, dtype=torch.float8_e4m3fn, device=DEV)
    vc = torch.zeros_like(kc)
    one = torch.ones(hkv, device=DEV)
    for scale in powers + near + others:
        s = torch.full((hkv,), scale, dtype=torch.float32)
        l20_rope_kv.l20_rope_and_cache(g[0], g[1], g[2], g[3], g[4], True, kc, vc, g[5], k_scale=one, v_scale=s.to(DEV))
        got = vc.view(torch.uint8).cpu().view(tokens, hkv, d)
        want = oracle.quantize(v, s).view(torch.uint8)
        assert torch.equal(got, want), f"scale {scale!r}: {int((got != want).sum())} bytes differ"
