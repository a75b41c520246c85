"""Parity of the CUDA path against the CPU oracle, through the C ABI (ctypes).

Gate (on bf16 / fp16 outputs): |a - b| <= 2e-3 + 1e-2 * |b| element-wise; gather indices
bit-exact.  Every test here needs a B200.
"""

import math

import pytest
import torch

from oracle import paged_decode_oracle as oracle
from single_gpu_inference_lab_b200.workloads import make_inputs

from helpers import assert_within_gate, smoke_recipe

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


@pytest.fixture(scope="module")
def cabi(built_libs):
    from single_gpu_inference_lab_b200 import cabi as module

    module.load()
    return module


PATH_LDG, PATH_TMA, PATH_BALANCED, PATH_FUSED = 1, 2, 3, 5
EARLY = 32  # PFD_FLAG_EARLY_METADATA: what the benchmark and the vLLM hook pass
SINGLE = 64  # PFD_FLAG_SINGLE_LAUNCH: pieces combined inside the balanced kernel (needs a plan)
EARLY_KV = 256  # PFD_FLAG_EARLY_KV: with EARLY and a plan, pages other than a sequence's last are streamed before the wait
PLAN = 1 << 20  # not a library flag: the test helpers call pfd_plan_decode first and pass the plan
FUSED = PLAN | SINGLE


def workspace(q, max_seq_len, split_size, dtype=torch.float32, kv_start=0, poison=True, min_rows=0):
    """(partial_output, partial_max, partial_sum, None) with one slot per split, or as many as
    it takes to hold ``min_rows`` rows (the capacity the balanced persistent kernel asks for)."""
    b, hq, d = q.shape
    s = max(1, -(-(max_seq_len - kv_start) // split_size), -(-min_rows // (b * hq)))
    fill = float("nan") if poison else 0.0
    return (
        torch.full((b, hq, s, d), fill, device=q.device, dtype=dtype),
        torch.full((b, hq, s), fill, device=q.device, dtype=torch.float32),
        torch.full((b, hq, s), fill, device=q.device, dtype=torch.float32),
        None,
    )


def expected_path(cabi, q, num_kv_heads, flags, partial_dtype=torch.float32):
    """Which kernels a call must have launched.  flags 0: the library's choice, i.e. the balanced
    persistent kernel for head_dim 128 with at most 8 query heads per kv head and an f32 workspace
    that is large enough (PLAN: both kernels read a plan; FUSED: the balanced kernel alone); 8:
    fixed-split grid with TMA; 1: with plain loads."""
    _, hq, d = q.shape
    if flags & 1 or d != 128:
        return PATH_LDG
    if flags & (8 | 2) or partial_dtype != torch.float32 or hq // num_kv_heads > 8:
        return PATH_TMA
    return PATH_FUSED if (flags & FUSED) == FUSED else PATH_BALANCED


def balanced(path):
    return path in (PATH_BALANCED, PATH_FUSED)


def make_plan(cabi, want, flags, q, kc, vc, table, lens, ws, msl, split_size, kv_start=0):
    """The plan of a call that asks for one (PLAN) and runs the balanced kernel (None otherwise)."""
    if not (flags & PLAN) or not balanced(want):
        return None
    return cabi.plan_decode(q, kc, vc, table, lens, max_seq_len=msl, split_size=split_size, workspace=ws, kv_start=kv_start)


def run(cabi, w, split_size, *, flags=0, kv_start=0, partial_dtype=torch.float32, packed=False,
        k_scale=None, v_scale=None, max_seq_len=None):
    """w: PagedDecodeInputs on the GPU. Returns output (and packed partial if asked)."""
    q = w.query
    hkv = w.key_cache.shape[2]
    msl = w.max_seq_len if max_seq_len is None else max_seq_len
    want = expected_path(cabi, q, hkv, flags, partial_dtype)
    rows = cabi.balanced_workspace_rows(q.shape[1], hkv) if balanced(want) else 0
    ws = workspace(q, msl, split_size, partial_dtype, kv_start, min_rows=rows)
    out = torch.full_like(q, float("nan"))
    pk = torch.full((q.shape[0], q.shape[1], q.shape[2] + 2), float("nan"), device=q.device) if packed else None
    plan = make_plan(cabi, want, flags, q, w.key_cache, w.value_cache, w.block_table, w.seq_lens, ws, msl, split_size, kv_start)
    flags &= ~PLAN
    cabi.paged_decode_fp8_e4m3_split_out(
        q, w.key_cache, w.value_cache, w.block_table, w.seq_lens,
        k_scale=w.k_scale if k_scale is None else k_scale,
        v_scale=w.v_scale if v_scale is None else v_scale,
        max_seq_len=msl, split_size=split_size, output=None if packed else out, packed_output=pk,
        workspace=ws, kv_start=kv_start, flags=flags, plan=plan,
    )
    torch.cuda.synchronize()
    assert cabi.device_status() == 0, "a bounded device-side wait gave up"
    assert cabi.last_path() == want, f"flags={flags}: path {cabi.last_path()}, expected {want}"
    return pk if packed else out


def expected(w, **kw):
    return oracle.reference(w.query, w.key_cache, w.value_cache, w.block_table.long(), w.seq_lens, w.k_scale, w.v_scale, **kw)


# ---------------------------------------------------------------- golden fixtures
@pytest.mark.parametrize(
    "name", ["cfg1-qwen0.5b-b8", "cfg2-coder3b-b4", "cfg3-qwen7b-b24", "cfg4-llama8b-b2", "cfg5-prefix-b8"]
)
@pytest.mark.parametrize("flags", [PLAN, FUSED, 8, 1, 0, PLAN | EARLY, FUSED | EARLY, PLAN | EARLY | EARLY_KV, FUSED | EARLY | EARLY_KV])
def test_against_committed_reference_outputs(cabi, golden, name, flags):
    case = golden["cases"][name]
    w = make_inputs(case["workload"], seed=0, device="cpu", batch=case["batch"], shrink=case["shrink"])
    for split in (64, 512):
        out = run(cabi, w.to(DEV), split, flags=flags)
        assert_within_gate(out, case["output"], f"{name} split={split}")


def test_reference_smoke_recipe_fp16_query_scalar_scales(cabi, golden):
    for key, case in golden["smoke"].items():
        q, kc, vc, table, lens, ks, vs = smoke_recipe(
            case["batch"], case["context"], case["q_heads"], case["kv_heads"], oracle.quantize_fp8_e4m3
        )
        q, kc, vc, table, lens = (t.to(DEV) for t in (q, kc, vc, table, lens))
        out = torch.empty_like(q)
        ws = workspace(q, case["context"], 128)
        cabi.paged_decode_fp8_e4m3_split_out(
            q, kc, vc, table, lens, k_scale=ks, v_scale=vs, max_seq_len=case["context"], split_size=128,
            output=out, workspace=ws,
        )
        torch.cuda.synchronize()
        assert_within_gate(out, case["output"], key)


# ---------------------------------------------------------------- the five configurations
def test_config1_full_size(cabi):
    w = make_inputs("qwen2.5-0.5b-b8", seed=0)
    exp = expected(w)
    for split in (16, 128, 1024):
        for flags in (0, EARLY):
            assert_within_gate(run(cabi, w.to(DEV), split, flags=flags), exp, f"cfg1 split={split} flags={flags}")


def test_config2_full_size(cabi):
    w = make_inputs("qwen2.5-coder-3b-b64", seed=0)
    exp = expected(w)
    for split, flags in ((256, PLAN), (512, 0), (896, 0), (512, 8), (1024, 1), (512, EARLY), (896, EARLY | 8), (256, EARLY | 1), (512, PLAN | EARLY), (512, FUSED), (256, FUSED | EARLY), (512, PLAN | EARLY | EARLY_KV), (256, EARLY | EARLY_KV)):
        assert_within_gate(run(cabi, w.to(DEV), split, flags=flags), exp, f"cfg2 split={split} flags={flags}")


def test_config3_full_size_log_uniform_lengths(cabi):
    w = make_inputs("qwen2.5-7b-b256", seed=0)
    assert int(w.seq_lens.min()) <= 4
    exp = expected(w)
    for flags in (0, PLAN, FUSED, 8, EARLY, EARLY | 8, PLAN | EARLY, FUSED | EARLY, PLAN | EARLY | EARLY_KV):
        assert_within_gate(run(cabi, w.to(DEV), 512, flags=flags), exp, f"cfg3 flags={flags}")


def test_config4_long_context_sampled_rows_and_split_invariance(cabi):
    """Full 4 x 131072 tokens on the GPU.  The oracle is run on one sequence compacted to its
    own pages (the whole-cache dequantisation of the reference function would need ~10 GB);
    split invariance covers the rest."""
    w = make_inputs("llama3-8b-long-b4", seed=0, device=DEV)
    out_a = run(cabi, w, 2048, flags=PLAN)
    out_b = run(cabi, w, 512, flags=8)
    out_c = run(cabi, w, 16384)
    out_d = run(cabi, w, 2048, flags=EARLY)
    out_f = run(cabi, w, 2048, flags=PLAN | EARLY)
    out_h = run(cabi, w, 2048, flags=PLAN | EARLY | EARLY_KV)
    assert_within_gate(out_f, out_a, "planned, early metadata vs not")
    assert_within_gate(out_h, out_a, "planned, early metadata and early K/V vs not")
    out_g = run(cabi, w, 2048, flags=FUSED | EARLY)
    assert_within_gate(out_g, out_a, "pieces combined inside the balanced kernel vs the merge kernel")
    out_e = run(cabi, w, 1024, flags=EARLY | 8)
    assert_within_gate(out_d, out_a, "early metadata vs not")
    assert_within_gate(out_e, out_a, "early metadata, fixed split 1024 vs 2048")
    assert_within_gate(out_b, out_a, "split 512 vs 2048")
    assert_within_gate(out_c, out_a, "split 8192 vs 2048")
    b = 2
    pages = w.block_table[b].long().cpu()
    kc = w.key_cache[pages.to(DEV)].cpu()
    vc = w.value_cache[pages.to(DEV)].cpu()
    table = torch.arange(pages.numel(), dtype=torch.int64)[None]
    exp = oracle.reference(
        w.query[b : b + 1].cpu(), kc, vc, table, w.seq_lens[b : b + 1].cpu(), w.k_scale.cpu(), w.v_scale.cpu()
    )
    assert_within_gate(out_a[b : b + 1], exp, "cfg4 row 2")


def test_config5_shared_prefix_full_size(cabi):
    w = make_inputs("shared-prefix-b64", seed=0)
    exp = expected(w)
    for flags in (0, PLAN, FUSED, 8, EARLY, EARLY | 8, PLAN | EARLY):
        assert_within_gate(run(cabi, w.to(DEV), 512, flags=flags), exp, f"cfg5 flags={flags}")


# ---------------------------------------------------------------- edge cases
@pytest.mark.parametrize("d,hq,hkv", [(128, 16, 2), (64, 14, 2), (128, 28, 4), (128, 32, 8), (128, 16, 16), (128, 16, 1)])
def test_every_short_context_length(cabi, d, hq, hkv):
    """ctx = 1 .. 70 in one batch: ragged tails, single page, page boundary +-1."""
    torch.manual_seed(11)
    lens = torch.arange(1, 71, dtype=torch.int32)
    b = lens.numel()
    pages_per = 5
    table = torch.randperm(b * pages_per).to(torch.int32).reshape(b, pages_per)
    kc, ks = oracle.quantize_fp8_e4m3_per_head(torch.randn(b * pages_per, 16, hkv, d))
    vc, vs = oracle.quantize_fp8_e4m3_per_head(torch.randn(b * pages_per, 16, hkv, d))
    q = torch.randn(b, hq, d).to(torch.bfloat16)
    exp = oracle.reference(q, kc, vc, table.long(), lens, ks, vs)
    for split in (16, 32, 64, 512):
        for flags in (PLAN, FUSED, 0, 8, 1, 2, EARLY, EARLY | 8, EARLY | 1, PLAN | EARLY, FUSED | EARLY):
            out = torch.full_like(q, float("nan"), device=DEV)
            want = expected_path(cabi, q, hkv, flags)
            rows = cabi.balanced_workspace_rows(hq, hkv) if balanced(want) else 0
            ws = workspace(q.to(DEV), 70, split, min_rows=rows)
            g = [t.to(DEV) for t in (q, kc, vc, table, lens)]
            plan = make_plan(cabi, want, flags, *g, ws, 70, split)
            cabi.paged_decode_fp8_e4m3_split_out(
                *g, k_scale=ks.to(DEV), v_scale=vs.to(DEV),
                max_seq_len=70, split_size=split, output=out, workspace=ws, flags=flags & ~PLAN, plan=plan,
            )
            torch.cuda.synchronize()
            assert cabi.last_path() == want, f"flags={flags}"
            assert_within_gate(out, exp, f"d={d} hq={hq} hkv={hkv} split={split} flags={flags}")


def test_unused_slots_may_hold_nan_bytes(cabi):
    """Slots past seq_len inside the last page (and unused pages) are never trusted: fill
    them with the e4m3 NaN pattern."""
    w = make_inputs("qwen2.5-coder-3b-b64", seed=5, batch=6, shrink=0.1)
    exp = expected(w)
    kc = w.key_cache.clone().view(torch.uint8)
    vc = w.value_cache.clone().view(torch.uint8)
    for b in range(6):
        n = int(w.seq_lens[b])
        if n % 16:
            page = int(w.block_table[b, n // 16])
            kc[page, n % 16 :] = 0x7F
            vc[page, n % 16 :] = 0xFF
    w.key_cache, w.value_cache = kc.view(torch.float8_e4m3fn), vc.view(torch.float8_e4m3fn)
    for flags in (PLAN, FUSED, 0, 8, 1):
        assert_within_gate(run(cabi, w.to(DEV), 64, flags=flags), exp, "nan slots")


def test_max_seq_len_larger_than_every_sequence_and_empty_splits(cabi):
    w = make_inputs("qwen2.5-0.5b-b8", seed=2, shrink=0.25)
    exp = expected(w)
    wide = torch.zeros(8, 40, dtype=torch.int32)
    wide[:, : w.block_table.shape[1]] = w.block_table
    w.block_table = wide
    out = run(cabi, w.to(DEV), 64, max_seq_len=640)
    assert_within_gate(out, exp, "msl=640")


def test_consumer_right_behind_the_call_sees_finished_rows(cabi):
    """Stream order without a host synchronisation: a kernel enqueued right behind the call (here a
    copy of the output) must see finished rows.  The merge grid is a programmatic dependent of the
    partial grid; when every one of its rows is already final it must still not complete early.
    Cases: one short sequence (one warp group, nothing to merge), and lengths that all fit one
    split while max_seq_len asks for several."""
    torch.manual_seed(3)
    hq, hkv, d, pages = 16, 2, 128, 8
    for batch, ctx, msl, flags in ((1, 64, 64, 0), (1, 64, 64, EARLY), (3, 60, 640, 8), (3, 60, 640, EARLY | 8), (1, 64, 64, FUSED), (2, 640, 640, FUSED | EARLY), (2, 640, 640, PLAN | EARLY)):
        lens = torch.full((batch,), ctx, dtype=torch.int32)
        table = torch.randperm(batch * 40).to(torch.int32).reshape(batch, 40)
        kc, ks = oracle.quantize_fp8_e4m3_per_head(torch.randn(batch * 40, 16, hkv, d))
        vc, vs = oracle.quantize_fp8_e4m3_per_head(torch.randn(batch * 40, 16, hkv, d))
        q = torch.randn(batch, hq, d).to(torch.bfloat16)
        exp = oracle.reference(q, kc, vc, table.long(), lens, ks, vs)
        g = [t.to(DEV) for t in (q, kc, vc, table, lens, ks, vs)]
        want = expected_path(cabi, q, hkv, flags)
        rows = cabi.balanced_workspace_rows(hq, hkv) if balanced(want) else 0
        ws = workspace(g[0], msl, 64, min_rows=rows)
        plan = make_plan(cabi, want, flags, *g[:5], ws, msl, 64)
        torch.cuda.synchronize()
        out = torch.empty_like(g[0])
        copies = []
        for _ in range(200):
            out.fill_(float("nan"))
            cabi.paged_decode_fp8_e4m3_split_out(
                g[0], g[1], g[2], g[3], g[4], k_scale=g[5], v_scale=g[6], max_seq_len=msl, split_size=64,
                output=out, workspace=ws, flags=flags & ~PLAN, plan=plan)
            copies.append(out.clone())
        torch.cuda.synchronize()
        assert cabi.last_path() == want
        for c in copies:
            assert_within_gate(c, exp, f"batch={batch} ctx={ctx} max_seq_len={msl} flags={flags}")


def test_zero_length_sequence_gives_zeros(cabi):
    w = make_inputs("qwen2.5-0.5b-b8", seed=2, shrink=0.25)
    lens = w.seq_lens.clone()
    lens[3] = 0
    w.seq_lens = lens
    exp = expected(w)  # softmax over nothing is NaN in torch; the operator writes zeros there
    out = run(cabi, w.to(DEV), 64)
    assert (out[3] == 0).all()
    keep = [0, 1, 2, 4, 5, 6, 7]
    assert_within_gate(out[keep], exp[keep], "others")


@pytest.mark.parametrize("layout", ["hnd", "interleaved_kv", "padded_pages"])
def test_strided_cache_layouts(cabi, layout):
    """The reference's Triton path honours cache strides (l20_paged_split_kv.py:665-668);
    vLLM hands it `kv_cache.unbind(1)` views.  Same logical [pages,16,Hkv,D] view, other memory."""
    w = make_inputs("qwen2.5-coder-3b-b64", seed=7, batch=5, shrink=0.1)
    exp = expected(w)
    g = w.to(DEV)
    if layout == "hnd":
        g.key_cache = g.key_cache.permute(0, 2, 1, 3).contiguous().permute(0, 2, 1, 3)
        g.value_cache = g.value_cache.permute(0, 2, 1, 3).contiguous().permute(0, 2, 1, 3)
    elif layout == "interleaved_kv":
        both = torch.stack([g.key_cache.view(torch.uint8), g.value_cache.view(torch.uint8)], dim=1)
        k, v = both.view(torch.float8_e4m3fn).unbind(1)
        g.key_cache, g.value_cache = k, v
    else:
        pages, _, hkv, d = g.key_cache.shape
        big = torch.zeros(pages, 16, hkv + 1, d, dtype=torch.uint8, device=DEV).view(torch.float8_e4m3fn)
        big2 = big.clone()
        big[:, :, :hkv] = g.key_cache
        big2[:, :, :hkv] = g.value_cache
        g.key_cache, g.value_cache = big[:, :, :hkv], big2[:, :, :hkv]
    assert not g.key_cache.is_contiguous()
    for flags in (PLAN, FUSED, 0, 8, 1):
        assert_within_gate(run(cabi, g, 64, flags=flags), exp, layout)


@pytest.mark.parametrize("pdtype", [torch.float32, torch.float16, torch.bfloat16])
def test_partial_workspace_dtypes(cabi, pdtype):
    """The reference keeps partial outputs in the query dtype (l20_paged_split_kv.py:24-26);
    callers that pass such a workspace still work (looser: one extra rounding per split)."""
    w = make_inputs("qwen2.5-coder-3b-b64", seed=3, batch=4, shrink=0.25)
    exp = expected(w)
    out = run(cabi, w.to(DEV), 128, partial_dtype=pdtype)
    if pdtype == torch.float32:
        assert_within_gate(out, exp, str(pdtype))
    else:
        assert torch.allclose(out.float().cpu(), exp.float(), atol=2e-2, rtol=2e-2)


def test_kv_start_suffix_pass_and_packed_partials_merge(cabi):
    """Prefix part + suffix part, each returned as packed (o, m, l), merged by pfd_merge_packed
    == attention over the whole range.  kv_start both page-aligned and not."""
    w = make_inputs("shared-prefix-b64", seed=4, batch=9, shrink=0.125)
    exp = expected(w)
    g = w.to(DEV)
    for cut in (w.prefix_len, w.prefix_len - 5, 3):
        head = g.to(DEV)
        head.seq_lens = torch.clamp(g.seq_lens, max=cut)
        p0 = run(cabi, head, 128, packed=True, max_seq_len=cut, flags=FUSED if cut == 3 else 0)
        p1 = run(cabi, g, 128, packed=True, kv_start=cut, flags=(FUSED if cut == 3 else PLAN) if cut % 2 else 8)
        out = torch.empty_like(g.query)
        cabi.merge_packed(torch.stack([p0, p1]).contiguous(), out)
        torch.cuda.synchronize()
        assert_within_gate(out, exp, f"cut={cut}")
        # the suffix alone equals the oracle restricted to [cut, len)
        has_suffix = (w.seq_lens > cut).nonzero().flatten().tolist()
        if has_suffix:
            sub = oracle.reference_fp32(
                w.query, w.key_cache, w.value_cache, w.block_table.long(), w.seq_lens, w.k_scale, w.v_scale, kv_start=cut
            )
            o, m, l = p1[..., :-2], p1[..., -2], p1[..., -1]
            got = (o / l[..., None]).cpu()
            assert torch.allclose(got[has_suffix], sub[has_suffix], atol=2e-3, rtol=1e-2)
        empty = (w.seq_lens <= cut).nonzero().flatten().tolist()
        for b in empty:
            assert (p1[b, :, :-2] == 0).all() and torch.isneginf(p1[b, :, -2]).all() and (p1[b, :, -1] == 0).all()


def test_partials_match_oracle_split_semantics(cabi):
    """partial_max (natural log units), partial_sum and un-normalised partial_output of every
    live split equal the oracle's restatement of the reference partial kernel."""
    w = make_inputs("qwen2.5-0.5b-b8", seed=6, batch=4, shrink=0.5)
    split = 64
    ns = -(-w.max_seq_len // split)
    o, m, l = oracle.split_partials(
        w.query, w.key_cache, w.value_cache, w.block_table.long(), w.seq_lens, w.k_scale, w.v_scale,
        split_size=split, num_splits=ns,
    )
    g = w.to(DEV)
    ws = workspace(g.query, w.max_seq_len, split, poison=False)
    out = torch.empty_like(g.query)
    cabi.paged_decode_fp8_e4m3_split_out(
        g.query, g.key_cache, g.value_cache, g.block_table, g.seq_lens, k_scale=g.k_scale, v_scale=g.v_scale,
        max_seq_len=w.max_seq_len, split_size=split, output=out, workspace=ws, flags=2,
    )
    torch.cuda.synchronize()
    po, pm, ps = (t.cpu() for t in ws[:3])
    for b in range(4):
        live = -(-int(w.seq_lens[b]) // split)
        assert torch.allclose(pm[b, :, :live], m[b, :, :live], atol=2e-3, rtol=1e-3)
        # rescale both to a common max before comparing sums / outputs
        c = torch.exp(pm[b, :, :live] - m[b, :, :live])
        assert torch.allclose(ps[b, :, :live] * c, l[b, :, :live], atol=1e-3, rtol=5e-3)
        assert torch.allclose(po[b, :, :live] * c[..., None], o[b, :, :live], atol=5e-3, rtol=1e-2)


def test_gather_indices_bit_exact(cabi):
    for name, kw in [("qwen2.5-0.5b-b8", {}), ("qwen2.5-7b-b256", {}), ("shared-prefix-b64", {})]:
        w = make_inputs(name, seed=0, shrink=0.25 if name != "qwen2.5-0.5b-b8" else 1.0)
        want = oracle.resolve_slots(w.block_table, w.seq_lens, w.max_seq_len)
        got = cabi.resolve_slots(w.block_table.to(DEV), w.seq_lens.to(DEV), w.max_seq_len)
        torch.cuda.synchronize()
        assert got.dtype == torch.int64 and torch.equal(got.cpu(), want), name


def test_block_table_permutation_invariance_and_idempotence(cabi):
    """Relocating every page (new permutation, caches moved accordingly) must not change a bit
    of the output; neither must running the same step twice into a reused workspace."""
    w = make_inputs("qwen2.5-coder-3b-b64", seed=8, batch=8, shrink=0.2).to(DEV)
    a = run(cabi, w, 128, flags=8)
    a2 = run(cabi, w, 128, flags=8)
    assert torch.equal(a.view(torch.int16), a2.view(torch.int16))
    pages = w.key_cache.shape[0]
    perm = torch.randperm(pages, device=DEV)
    moved = w.to(DEV)
    kc = torch.empty_like(w.key_cache.view(torch.uint8))
    vc = torch.empty_like(kc)
    kc[perm] = w.key_cache.view(torch.uint8)
    vc[perm] = w.value_cache.view(torch.uint8)
    moved.key_cache, moved.value_cache = kc.view(torch.float8_e4m3fn), vc.view(torch.float8_e4m3fn)
    moved.block_table = perm[w.block_table.long()].to(torch.int32)
    b = run(cabi, moved, 128, flags=8)
    assert torch.equal(a.view(torch.int16), b.view(torch.int16))
    # the balanced path sums warps in a fixed order too: same bits run to run and after relocation
    c1, c2, c3 = run(cabi, w, 128, flags=0), run(cabi, w, 128, flags=0), run(cabi, moved, 128, flags=0)
    assert torch.equal(c1.view(torch.int16), c2.view(torch.int16))
    assert torch.equal(c1.view(torch.int16), c3.view(torch.int16))
    # combined inside the balanced kernel the pieces of a cut sequence are folded in a fixed order as well
    c1, c2, c3 = run(cabi, w, 128, flags=FUSED), run(cabi, w, 128, flags=FUSED), run(cabi, moved, 128, flags=FUSED)
    assert torch.equal(c1.view(torch.int16), c2.view(torch.int16))
    assert torch.equal(c1.view(torch.int16), c3.view(torch.int16))


def test_linearity_in_v_scale_and_scale_folding(cabi):
    w = make_inputs("qwen2.5-0.5b-b8", seed=9, batch=4, shrink=0.5).to(DEV)
    a = run(cabi, w, 64)
    b = run(cabi, w, 64, v_scale=w.v_scale * 2)
    assert torch.equal((a.float() * 2).to(torch.bfloat16).view(torch.int16), b.view(torch.int16))


def test_a_wait_that_nothing_satisfies_runs_out_and_sets_the_status_word(cabi):
    """Every device-side wait is bounded in time.  The self-test kernel arms a barrier for bytes
    that no copy delivers: the wait gives up after the limit, the kernel finishes, the error word
    reads 1 once and then 0 again, and the next decode call runs as usual."""
    assert cabi.device_status() == 0
    for limit_ns in (200_000, 3_000_000):
        waited = cabi.selftest_bounded_wait(limit_ns)
        assert limit_ns <= waited < limit_ns + 2_000_000, (limit_ns, waited)
        assert cabi.device_status() == 1
        assert cabi.device_status() == 0
    w = make_inputs("qwen2.5-coder-3b-b64", seed=12, batch=4, shrink=0.25)
    assert_within_gate(run(cabi, w.to(DEV), 128), expected(w), "decode after an expired wait")


# ---------------------------------------------------------------- dispatcher op (torch.ops) surface
def test_torch_op_reference_signature_and_wrapper_module(built_libs, golden):
    from single_gpu_inference_lab_b200 import l20_paged_decode, l20_paged_split_kv

    key, case = next(iter(golden["smoke"].items()))
    q, kc, vc, table, lens, ks, vs = smoke_recipe(
        case["batch"], case["context"], case["q_heads"], case["kv_heads"], oracle.quantize_fp8_e4m3
    )
    q, kc, vc, table, lens = (t.to(DEV) for t in (q, kc, vc, table, lens))
    splits = -(-case["context"] // 128)
    # exactly the call of scripts/smoke_cuda_paged_fp8_decode_op.py:89-111 (fp16 partial workspace)
    partial = torch.empty(case["batch"], case["q_heads"], splits, 128, device=DEV, dtype=torch.float16)
    maxima = torch.empty(case["batch"], case["q_heads"], splits, device=DEV)
    sums = torch.empty_like(maxima)
    output = torch.empty_like(q)
    actual = torch.ops.l20_stack.paged_decode_fp8_e4m3_split_out(
        q, kc, vc, table, lens, partial, maxima, sums, output, ks, vs, case["context"], 128
    )
    torch.cuda.synchronize()
    assert actual.data_ptr() == output.data_ptr()
    torch.testing.assert_close(actual.cpu(), case["output"], rtol=2e-2, atol=2e-2)  # the reference smoke's own gate
    # module-level wrapper with allocator, fp32 partials, bf16 query, per-head scales
    w = make_inputs("qwen2.5-coder-3b-b64", seed=0, batch=4, shrink=0.25)
    exp = expected(w)
    g = w.to(DEV)
    out = l20_paged_split_kv.l20_paged_split_kv_attention_fp8(
        g.query, g.key_cache, g.value_cache, g.block_table, g.seq_lens, k_scale=g.k_scale, v_scale=g.v_scale,
        max_seq_len=w.max_seq_len, split_size=256,
    )
    torch.cuda.synchronize()
    assert_within_gate(out, exp, "wrapper")
    with pytest.raises(RuntimeError, match="workspace shape does not match"):
        l20_paged_split_kv.l20_paged_split_kv_attention_fp8(
            g.query, g.key_cache, g.value_cache, g.block_table, g.seq_lens, k_scale=1.0, v_scale=1.0,
            max_seq_len=w.max_seq_len, split_size=256,
            workspace=l20_paged_split_kv.allocate_l20_paged_split_kv_workspace(g.query[:2], 16, split_size=256),
        )
    with pytest.raises(RuntimeError, match="split_size must be a multiple of 16"):
        l20_paged_decode.paged_decode_fp8_e4m3_split_out(
            q, kc, vc, table, lens, partial, maxima, sums, output, ks, vs, case["context"], 100
        )
    assert l20_paged_decode.resolve_slots(table, lens, case["context"]).shape == (case["batch"], case["context"])


def test_cuda_graph_capture_and_replay(built_libs):
    """The op makes no host sync and no allocation, so it captures (the reference switches its
    hook off while capturing, install_l20_fp8_paged_decode.py:72; its fp16 sibling is graph
    tested in scripts/stress_cuda_paged_decode.py:129-167)."""
    from single_gpu_inference_lab_b200 import l20_paged_split_kv as m

    w = make_inputs("qwen2.5-coder-3b-b64", seed=1, batch=4, shrink=0.25)
    exp = expected(w)
    g = w.to(DEV)
    ws = m.allocate_l20_paged_split_kv_workspace(g.query, w.max_seq_len, split_size=128)
    m.l20_paged_split_kv_attention_fp8(
        g.query, g.key_cache, g.value_cache, g.block_table, g.seq_lens, k_scale=g.k_scale, v_scale=g.v_scale,
        max_seq_len=w.max_seq_len, split_size=128, workspace=ws,
    )
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    ws[3].zero_()
    with torch.cuda.graph(graph):
        m.l20_paged_split_kv_attention_fp8(
            g.query, g.key_cache, g.value_cache, g.block_table, g.seq_lens, k_scale=g.k_scale, v_scale=g.v_scale,
            max_seq_len=w.max_seq_len, split_size=128, workspace=ws,
        )
    for _ in range(3):
        ws[3].zero_()
        graph.replay()
    torch.cuda.synchronize()
    assert_within_gate(ws[3], exp, "graph replay")


# ---------------------------------------------------------------- balanced kernel, head_dim 64
@pytest.mark.parametrize("layout,dtype", [("nhd", torch.bfloat16), ("hnd", torch.bfloat16), ("nhd", torch.float16)])
@pytest.mark.parametrize("d,hq,hkv", [(64, 14, 2), (64, 8, 1), (64, 8, 8), (64, 6, 3), (64, 9, 1)])
def test_balanced_kernel_with_head_dim_64(cabi, d, hq, hkv, layout, dtype):
    """Batches large enough for the balanced kernel: every length around a page and a page pair, empty and long sequences,
    unaligned kv_start, packed output, NaN bytes in the unused slots, a workspace with room for all warp groups and for
    three quarters of them; and what the grid keeps: less room, nine heads per KV head, the fixed-split flag."""
    gen = torch.Generator().manual_seed(d + hq)
    batch, longest = 200, 700
    lens = torch.cat([torch.arange(0, 70), torch.randint(1, longest + 1, (batch - 72,), generator=gen),
                      torch.tensor([longest, longest - 1])]).to(torch.int32)
    pages_of = (lens + 15) // 16
    total = int(pages_of.sum()) + 1
    table = torch.full((batch, -(-longest // 16)), total - 1, dtype=torch.int32)
    free = torch.randperm(total - 1, generator=gen).to(torch.int32)
    at = 0
    for b, n in enumerate(pages_of.tolist()):
        table[b, :n] = free[at:at + n]
        at += n
    kc, ks = oracle.quantize_fp8_e4m3_per_head(torch.randn(total, 16, hkv, d, generator=gen))
    vc, vs = oracle.quantize_fp8_e4m3_per_head(torch.randn(total, 16, hkv, d, generator=gen))
    q = torch.randn(batch, hq, d, generator=gen).to(dtype)
    for c in (kc, vc):  # what no sequence owns: NaN
        for b, n in enumerate(lens.tolist()):
            if n % 16:
                c.view(torch.uint8)[table[b, n // 16], n % 16:] = 0x7F
        c.view(torch.uint8)[total - 1] = 0x7F
    g = [t.to(DEV) for t in (q, kc, vc, table, lens)]
    if layout == "hnd":
        g[1:3] = [t.permute(0, 2, 1, 3).contiguous().permute(0, 2, 1, 3) for t in g[1:3]]
    all_groups = torch.cuda.get_device_properties(DEV).multi_processor_count * 16 // hkv
    all_rows = 2 * all_groups * hq
    for kv_start in (0, 21):
        live = lens > kv_start
        exp = torch.zeros(batch, hq, d)
        for b in live.nonzero()[:, 0].tolist():
            one = slice(b, b + 1)
            exp[b] = oracle.reference_fp32(q[one], kc, vc, table[one].long(), lens[one], ks, vs, kv_start=kv_start)[0]
        for rows, flags, packed in ((all_rows + 2 * hq, 0, False), (3 * all_rows // 4 + 2 * hq, EARLY, False), (all_rows + 2 * hq, 0, True), (0, 0, False),
                                    (all_rows, 8, False)):
            ws = workspace(g[0], longest, 512, kv_start=kv_start, min_rows=rows)
            out = torch.full_like(g[0], float("nan"))
            pk = torch.full((batch, hq, d + 2), float("nan"), device=DEV) if packed else None
            cabi.paged_decode_fp8_e4m3_split_out(
                *g, k_scale=ks.to(DEV), v_scale=vs.to(DEV), max_seq_len=longest, split_size=512, output=None if packed else out,
                packed_output=pk, workspace=ws, kv_start=kv_start, flags=flags)
            torch.cuda.synchronize()
            assert cabi.device_status() == 0
            what = f"d={d} hq={hq} hkv={hkv} {layout} {dtype} kv_start={kv_start} rows={rows} flags={flags} packed={packed}"
            room = batch * ws[0].shape[2] // 2
            grid = flags & 8 or hq // hkv > 8 or 4 * room < 3 * all_groups
            assert cabi.last_path() == (PATH_LDG if grid else PATH_BALANCED), what
            if packed:
                o, m, l = pk[..., :d], pk[..., d], pk[..., d + 1]
                assert torch.equal(l.cpu() > 0, live[:, None].expand(batch, hq)), what
                out = torch.where(l[..., None] > 0, o / l[..., None], 0.0).to(q.dtype)
            assert_within_gate(out, exp.to(q.dtype), what)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows_per_sm,longest", [(6, 2100), (10, 4100)])
def test_head_dim_64_rows_merged_by_four_warps(cabi, rows_per_sm, longest, dtype):
    """The merge kernel gives a row four warps at up to eight rows per SM, and up to sixteen where sequences can be longer
    than 4096 tokens: sequences of many pieces, of one, and of none, packed and final."""
    sms = torch.cuda.get_device_properties(DEV).multi_processor_count
    d, hq, hkv = 64, 14, 2
    batch = max(rows_per_sm * sms // hq, -(-(1 << 17) // longest))
    gen = torch.Generator().manual_seed(longest)
    lens = torch.randint(1, 200, (batch,), generator=gen).to(torch.int32)
    lens[:4] = torch.tensor([longest, 0, longest - 1, 33])
    pages = 400
    table = torch.randint(0, pages, (batch, -(-longest // 16)), generator=gen).to(torch.int32)
    kc, ks = oracle.quantize_fp8_e4m3_per_head(torch.randn(pages, 16, hkv, d, generator=gen))
    vc, vs = oracle.quantize_fp8_e4m3_per_head(torch.randn(pages, 16, hkv, d, generator=gen))
    q = torch.randn(batch, hq, d, generator=gen).to(dtype)
    live = lens > 0
    exp = torch.zeros_like(q)
    exp[live] = oracle.reference(q[live], kc, vc, table[live].long(), lens[live], ks, vs)
    g = [t.to(DEV) for t in (q, kc, vc, table, lens)]
    ws = workspace(g[0], longest, 512, min_rows=2 * (sms * 16 // hkv) * hq + 2 * hq)
    for packed in (False, True):
        out = torch.full_like(g[0], float("nan"))
        pk = torch.full((batch, hq, d + 2), float("nan"), device=DEV) if packed else None
        cabi.paged_decode_fp8_e4m3_split_out(*g, k_scale=ks.to(DEV), v_scale=vs.to(DEV), max_seq_len=longest, split_size=512,
                                             output=None if packed else out, packed_output=pk, workspace=ws)
        torch.cuda.synchronize()
        assert cabi.device_status() == 0 and cabi.last_path() == PATH_BALANCED
        if packed:
            o, l = pk[..., :d], pk[..., d + 1:]
            out = torch.where(l > 0, o / l, 0.0).to(q.dtype)
        assert_within_gate(out, exp, f"batch={batch} longest={longest} {dtype} packed={packed}")


@pytest.mark.parametrize("what", ["d64 partials", "d128 partials", "d64 packed", "d128 packed", "kv16 packed", "kv16 packed fused"])
def test_buffers_aligned_to_four_bytes_only(cabi, what):
    """A workspace that a one-split call does not need, and packed rows, may lie at any float: the balanced kernel, which
    stores 16 and 8 bytes at a time, leaves such calls to the grid (16-bit caches: stored by element)."""
    gen = torch.Generator().manual_seed(3)
    d, kv16, packed = 64 if "d64" in what else 128, "kv16" in what, "packed" in what
    batch, longest, hq, hkv = 260, 512, 8, 8
    lens = torch.randint(1, longest + 1, (batch,), generator=gen).to(torch.int32)
    lens[:2] = torch.tensor([longest, longest - 1])
    pages = 900
    table = torch.randint(0, pages, (batch, longest // 16), generator=gen).to(torch.int32)
    k, v = torch.randn(pages, 16, hkv, d, generator=gen), torch.randn(pages, 16, hkv, d, generator=gen)
    q = torch.randn(batch, hq, d, generator=gen).to(torch.bfloat16)
    if kv16:
        kc, vc, scales = k.to(q.dtype), v.to(q.dtype), {}
        exp = oracle.reference_kv16(q, kc, vc, table.long(), lens)
    else:
        (kc, ks), (vc, vs) = oracle.quantize_fp8_e4m3_per_head(k), oracle.quantize_fp8_e4m3_per_head(v)
        scales = dict(k_scale=ks.to(DEV), v_scale=vs.to(DEV))
        exp = oracle.reference(q, kc, vc, table.long(), lens, ks, vs)
    g = [t.to(DEV) for t in (q, kc, vc, table, lens)]
    split = 256 if packed else 512
    at_float = lambda *shape: torch.full((math.prod(shape) + 1,), float("nan"), device=DEV)[1:].view(shape)
    ws = list(workspace(g[0], longest, split, min_rows=cabi.balanced_workspace_rows(hq, hkv) * (2 if d == 64 else 1)))
    if not packed:
        ws[0] = at_float(*ws[0].shape)
    out = torch.full_like(g[0], float("nan"))
    pk = at_float(batch, hq, d + 2) if packed else None
    assert (pk if packed else ws[0]).data_ptr() % 8 == 4
    plan = cabi.plan_decode(*g, max_seq_len=longest, split_size=split, workspace=ws) if "fused" in what else None
    call = cabi.paged_decode_kv16_split_out if kv16 else cabi.paged_decode_fp8_e4m3_split_out
    call(*g, max_seq_len=longest, split_size=split, output=None if packed else out, packed_output=pk, workspace=ws, plan=plan,
         flags=64 if plan is not None else 0, **scales)
    torch.cuda.synchronize()
    assert cabi.device_status() == 0
    assert cabi.last_path() == (4 if kv16 else PATH_LDG if d == 64 else PATH_TMA)
    if packed:
        o, l = pk[..., :d], pk[..., d + 1:]
        out = (o / l).to(q.dtype)
    assert_within_gate(out, exp, what)


# ---------------------------------------------------------------- the running maximum and the sign of the scale
KERNELS = {  # head_dim, 16-bit cache, flags, path
    "balanced": (128, False, 0, PATH_BALANCED), "balanced d64": (64, False, 0, PATH_BALANCED), "kv16": (128, True, 0, 4),
    "grid tma": (128, False, 8, PATH_TMA), "grid loads": (128, False, 1, PATH_LDG), "grid d64": (64, False, 8, PATH_LDG),
}


def _exact(q, kc, vc, table, lens, ks=1.0, vs=1.0, sm_scale=None):
    """Attention in 64 bits.  (The oracle rounds the dequantised cache to fp16, by up to 2^-11 of a value: of no account at
    ordinary scores, but 0.13 of a score of 260 (log2), 9 % of a weight where the gate allows 1 %.)"""
    batch, hq, d = q.shape
    hkv = kc.shape[2]
    scale = d ** -0.5 if sm_scale is None else sm_scale
    per_head = lambda s: (s.double() if isinstance(s, torch.Tensor) else torch.full((hkv,), s, dtype=torch.float64))[:, None, None]
    out = torch.empty(batch, hq, d, dtype=torch.float64)
    for b, n in enumerate(lens.tolist()):
        rows = lambda c, s: c[table[b].long()].double().reshape(-1, hkv, d)[:n].transpose(0, 1) * per_head(s)
        w = torch.softmax(q[b].double().view(hkv, hq // hkv, d) @ rows(kc, ks).transpose(1, 2) * scale, -1)
        out[b] = (w @ rows(vc, vs)).reshape(hq, d)
    return out.to(q.dtype)


def _one_direction(kernel, dtype, log2_scores, sm_scale=None, k_sign=1.0, seed=0):
    """A batch in which every key is a multiple of one vector: score (log2) of token t for query head h of sequence b is
    ``log2_scores(t) * (1, -1, 0.5, 0)[h % 4]`` or, the keys being quantised, nearly that.  (operands, expected)"""
    d, kv16, _, _ = KERNELS[kernel]
    gen = torch.Generator().manual_seed(seed)
    batch, longest, hq, hkv = 256 if d == 64 else 12, 520, 8, 2  # (head_dim 64: enough work for the balanced kernel)
    lens = torch.randint(1, longest + 1, (batch,), generator=gen).to(torch.int32)
    lens[:5] = torch.tensor([longest, longest - 1, 33, 17, 1])
    width, pages = -(-longest // 16), 200
    u = torch.nn.functional.normalize(torch.randn(d, generator=gen), dim=0) * d ** 0.5
    t = torch.arange(width * 16, dtype=torch.float64)
    scale = d ** -0.5 if sm_scale is None else sm_scale
    # pages of the table in token order, so that page p holds tokens 16 p .. 16 p + 15 of every sequence
    rows = log2_scores(t) / (1.4426950408889634 * scale * k_sign * float(u.double() @ u.double()))
    k = (rows[:, None].float() * u).view(width, 16, 1, d).expand(width, 16, hkv, d).contiguous()
    v = torch.randn(width, 16, hkv, d, generator=gen)
    table = torch.arange(width).expand(batch, width).contiguous().to(torch.int32)
    q = (u * torch.tensor([1.0, -1.0, 0.5, 0.0]).repeat(hq // 4)[:, None]).expand(batch, hq, d).to(dtype).contiguous()
    if kv16:
        kc, vc, scales = k.to(dtype), v.to(dtype), {}
        assert sm_scale is None and k_sign == 1.0
    else:
        (kc, ks), (vc, vs) = oracle.quantize_fp8_e4m3_per_head(k), oracle.quantize_fp8_e4m3_per_head(v)
        ks = ks * k_sign
        scales = dict(k_scale=ks, v_scale=vs)
    return (q, kc, vc, table, lens), scales, longest, _exact(q, kc, vc, table, lens, *scales.values(), sm_scale=sm_scale)


def _attend(cabi, kernel, operands, scales, longest, **kw):
    d, kv16, flags, path = KERNELS[kernel]
    g = [t.to(DEV) for t in operands]
    ws = workspace(g[0], longest, 512, min_rows=2 * cabi.balanced_workspace_rows(g[0].shape[1], g[1].shape[2]))
    out = torch.full_like(g[0], float("nan"))
    call = cabi.paged_decode_kv16_split_out if kv16 else cabi.paged_decode_fp8_e4m3_split_out
    call(*g, max_seq_len=longest, split_size=512, output=out, workspace=ws, flags=flags,
         **{n: s.to(DEV) for n, s in scales.items()}, **kw)
    torch.cuda.synchronize()
    assert cabi.device_status() == 0 and cabi.last_path() == path
    return out


def _normal_scores(kernel, dtype, sharp, seed):
    """Normal queries and keys, scores of a standard deviation of ``sharp`` (natural units)."""
    d, kv16, _, _ = KERNELS[kernel]
    gen = torch.Generator().manual_seed(seed)
    batch, longest, hq, hkv = 256 if d == 64 else 48, 1024 if d == 128 else 520, 8, 2
    lens = torch.randint(longest // 2, longest + 1, (batch,), generator=gen).to(torch.int32)
    pages = 400
    table = torch.randint(0, pages, (batch, -(-longest // 16)), generator=gen).to(torch.int32)
    q = (sharp * torch.randn(batch, hq, d, generator=gen)).to(dtype)
    k, v = torch.randn(pages, 16, hkv, d, generator=gen), torch.randn(pages, 16, hkv, d, generator=gen)
    if kv16:
        kc, vc, scales = k.to(dtype), v.to(dtype), {}
    else:
        (kc, ks), (vc, vs) = oracle.quantize_fp8_e4m3_per_head(k), oracle.quantize_fp8_e4m3_per_head(v)
        scales = dict(k_scale=ks, v_scale=vs)
    return (q, kc, vc, table, lens), scales, longest, _exact(q, kc, vc, table, lens, *scales.values())


@pytest.mark.parametrize("kernel", [k for k in KERNELS if k != "kv16"])  # (whose bf16 probabilities have 16 bits)
def test_probabilities_are_relative_to_the_true_maximum(cabi, kernel):
    """The largest probability is then 1, exact in f16, and a bf16 output shows it: of outputs whose error before the last
    rounding is r (relative, rms), about 0.8 r / (2^-8 / 1.44) are not the rounded 64-bit result.  At scores of a standard
    deviation of 3, r is 0.6e-4 .. 0.9e-4 with the true maximum (measured here: 2.7 % .. 3.5 % of the outputs) and 1.5e-4 ..
    2e-4 with one up to 8 (log2) behind (5.2 % .. 6.7 %)."""
    operands, scales, longest, exp = _normal_scores(kernel, torch.bfloat16, 3.0, seed=0)
    out = _attend(cabi, kernel, operands, scales, longest).cpu()
    assert float((out != exp).float().mean()) < 0.043
    assert_within_gate(out, exp, kernel)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("kernel", list(KERNELS))
def test_scores_that_rise_along_the_sequence(cabi, kernel, dtype):
    """The maximum moves in every step, by a little or by a lot, late, or never: falling and constant scores, a step of a
    page, a jump far above everything before it.  (Half the heads see the scores with the other sign.)"""
    rises = {
        "slowly": lambda t: 0.0625 * t, "by 7.9 a page pair": lambda t: 7.9 * (t // 32), "by 8.1 a page": lambda t: 8.1 * (t // 16),
        "falling": lambda t: -0.5 * t, "constant": lambda t: torch.zeros_like(t), "a late jump": lambda t: 40.0 * (t >= 500),
    }
    for what, scores in rises.items():
        operands, scales, longest, exp = _one_direction(kernel, dtype, scores, seed=len(what))
        assert_within_gate(_attend(cabi, kernel, operands, scales, longest), exp, f"{kernel} {dtype} {what}")


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("kernel", [k for k in KERNELS if k != "kv16"])
def test_scales_below_and_at_zero(cabi, kernel, dtype):
    """A negative softmax scale or K scale (its sign goes into the query), both, and a K scale of zero (all tokens alike)."""
    rising = lambda t: 0.05 * t
    for sm_scale, k_sign in ((-0.07, 1.0), (None, -1.0), (-0.07, -1.0), (0.11, 1.0)):
        operands, scales, longest, exp = _one_direction(kernel, dtype, rising, sm_scale, k_sign)
        out = _attend(cabi, kernel, operands, scales, longest, **({} if sm_scale is None else {"sm_scale": sm_scale}))
        assert_within_gate(out, exp, f"{kernel} {dtype} sm_scale={sm_scale} k_sign={k_sign}")
    operands, scales, longest, _ = _one_direction(kernel, dtype, rising)
    scales["k_scale"] = torch.zeros_like(scales["k_scale"])
    exp = _exact(*operands, *scales.values())
    assert_within_gate(_attend(cabi, kernel, operands, scales, longest), exp, f"{kernel} {dtype} k_scale=0")


@pytest.mark.parametrize("kernel", list(KERNELS))
def test_an_infinite_query_value_spoils_its_own_head_only(cabi, kernel):
    operands, scales, longest, exp = _one_direction(kernel, torch.bfloat16, lambda t: 0.05 * t)
    operands[0][1, 3, 7] = float("inf")
    out = _attend(cabi, kernel, operands, scales, longest)
    assert out[1, 3].isnan().all()
    out[1, 3] = exp[1, 3].to(DEV)
    assert_within_gate(out, exp, kernel)
