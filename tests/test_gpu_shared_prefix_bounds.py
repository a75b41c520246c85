"""Shared-prefix decode of a request that is longer than the caller's max_seq_len says: nothing behind the block-table row
is read, the request is attended up to there, and a grouped call reports it."""

import pytest
import torch

from oracle import paged_decode_oracle as oracle

from helpers import assert_within_gate

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


@pytest.fixture(scope="module")
def cabi(built_libs):
    from single_gpu_inference_lab_b200 import cabi as module

    module.load()
    return module


@pytest.mark.parametrize("grouped,batch,hq,hkv,prefix,max_len,member,alone", [
    (True, 20, 16, 2, 512, 612, 640, 700),  # within the last split, behind the last page; a request in no group behind all
    (True, 20, 16, 2, 512, 512, 520, 520),  # no room for any token behind the prefix
    (False, 40, 32, 4, 4096, 4324, 4350, None),
])
def test_a_request_longer_than_the_bound_stays_inside_its_row(cabi, grouped, batch, hq, hkv, prefix, max_len, member, alone):
    from single_gpu_inference_lab_b200.workloads import quantize_per_head

    gen = torch.Generator().manual_seed(7)
    d, pages, split = 128, 900, 64
    cols = -(-max_len // 16)
    kc, ks = quantize_per_head(torch.randn(pages, 16, hkv, d, generator=gen))
    vc, vs = quantize_per_head(torch.randn(pages, 16, hkv, d, generator=gen))
    # the rows that are passed are the first columns of wider ones, whose rest names pages that must not count
    wide = torch.randint(0, pages, (batch, cols + 8), generator=gen, dtype=torch.int32)
    members = batch - 2 if grouped else batch
    wide[:members, :prefix // 16] = wide[0, :prefix // 16]
    lens = torch.randint(prefix, max_len + 1, (batch,), generator=gen, dtype=torch.int32)
    lens[0] = lens[batch - 3] = member
    if grouped:
        lens[-1] = alone
    q = torch.randn(batch, hq, d, generator=gen).to(torch.bfloat16)
    table = wide[:, :cols]
    exp = oracle.reference(q, kc, vc, table.long(), lens.clamp(max=cols * 16), ks, vs)
    gq, gkc, gvc, gw, gl, gks, gvs = (t.to(DEV) for t in (q, kc, vc, wide, lens, ks, vs))
    gt = gw[:, :cols]
    suffix = 100 if grouped else max_len - prefix
    slots = -(-prefix // 256) + -(-suffix // split)
    ws = tuple(torch.full(s, float("nan"), device=DEV) for s in ((batch, hq, slots, d), (batch, hq, slots), (batch, hq, slots)))
    out = torch.full_like(gq, float("nan"))
    common = dict(k_scale=gks, v_scale=gvs, max_seq_len=max_len, split_size=split, output=out, workspace=ws)
    if grouped:
        shared = torch.tensor([prefix if r < members else 0 for r in range(batch)], dtype=torch.int32)
        groups, max_groups = cabi.group_shared_prefixes(gt, prefix_lengths=shared.to(DEV), min_batch=8, min_prefix_len=256, max_groups=2)
        torch.cuda.synchronize()
        assert groups[3:5].tolist() == [1, members]
    before = cabi.launch_count()
    if grouped:
        cabi.shared_prefix_decode_grouped_fp8_e4m3(gq, gkc, gvc, gt, gl, groups=groups, max_groups=max_groups, max_prefix_len=prefix,
                                                   max_suffix_len=suffix, **common)
    else:
        cabi.shared_prefix_decode_fp8_e4m3(gq, gkc, gvc, gt, gl, prefix_len=prefix, **common)
    torch.cuda.synchronize()
    assert cabi.launch_count() - before == 2  # (the fused kernel and the merge)
    assert cabi.device_status() == (5 if grouped else 0)
    assert_within_gate(out, exp, f"grouped={grouped} max_seq_len={max_len}")
