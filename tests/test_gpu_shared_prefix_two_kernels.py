"""Grouped shared-prefix decode by the dense pass and the split-KV pass behind it: what the fused kernel does not take by
itself, or is told not to.  The launches of a call (2 with the fused kernel, 3 without) pin which one ran."""

import pytest
import torch

import test_gpu_shared_prefix as base
from oracle import paged_decode_oracle as oracle

from helpers import assert_within_gate

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


class Counted:
    """The binding, with the launches of each grouped decode written down."""

    def __init__(self, cabi):
        self._cabi, self.launches = cabi, []

    def __getattr__(self, name):
        return getattr(self._cabi, name)

    def shared_prefix_decode_grouped_fp8_e4m3(self, *args, **kw):
        before = self._cabi.launch_count()
        self._cabi.shared_prefix_decode_grouped_fp8_e4m3(*args, **kw)
        self.launches.append(self._cabi.launch_count() - before)


@pytest.fixture(scope="module")
def cabi(built_libs):
    from single_gpu_inference_lab_b200 import cabi as module

    module.load()
    return module


@pytest.fixture
def two_kernels(cabi):
    """The split-KV pass behind the dense pass, whatever the library would choose; the choice is restored."""
    cabi.set_suffix_form(0)
    yield Counted(cabi)
    cabi.set_suffix_form(-1)


def _decode(counted, batch, hq, hkv, groups_of, prefix, own, split, alone, flags=0):
    """Groups of `groups_of` requests behind `prefix` + 16 g tokens, the rest in none with the lengths `alone`, in turn; own
    tokens of the members as listed in turn."""
    from single_gpu_inference_lab_b200.workloads import quantize_per_head

    gen = torch.Generator().manual_seed(batch + hq)
    pages, d, n_groups = 2500, 128, batch // groups_of
    kc, ks = quantize_per_head(torch.randn(pages, 16, hkv, d, generator=gen))
    vc, vs = quantize_per_head(torch.randn(pages, 16, hkv, d, generator=gen))
    of = [prefix + 16 * (r // groups_of) if r < n_groups * groups_of else 0 for r in range(batch)]
    lens = torch.tensor([of[r] + own[r % len(own)] if of[r] else alone[r % len(alone)] for r in range(batch)], dtype=torch.int32)
    longest = int(lens.max())
    table = torch.randint(0, pages, (batch, -(-longest // 16)), generator=gen, dtype=torch.int32)
    for g in range(n_groups):
        shared = of[g * groups_of] // 16
        table[g * groups_of:(g + 1) * groups_of, :shared] = table[g * groups_of, :shared]
    q = torch.randn(batch, hq, d, generator=gen).to(torch.bfloat16)
    exp = oracle.reference(q, kc, vc, table.long(), lens, ks, vs)
    gq, gkc, gvc, gt, gl, gks, gvs = (t.to(DEV) for t in (q, kc, vc, table, lens, ks, vs))
    groups, max_groups = counted.group_shared_prefixes(gt, prefix_lengths=torch.tensor(of, dtype=torch.int32, device=DEV),
                                                       min_batch=groups_of, min_prefix_len=256, max_groups=n_groups)
    torch.cuda.synchronize()
    assert groups[3:5].tolist() == [n_groups, n_groups * groups_of]
    cap = max(of)
    slots = -(-cap // 256) + -(-max(own) // split)
    ws = tuple(torch.full(s, float("nan"), device=DEV) for s in ((batch, hq, slots, d), (batch, hq, slots), (batch, hq, slots)))
    for step in range(2):
        out = torch.full_like(gq, float("nan"))
        counted.shared_prefix_decode_grouped_fp8_e4m3(
            gq, gkc, gvc, gt, gl, groups=groups, max_groups=max_groups, max_prefix_len=cap, max_suffix_len=max(own),
            k_scale=gks, v_scale=gvs, max_seq_len=longest, split_size=split, output=out, workspace=ws, flags=flags)
        torch.cuda.synchronize()
        assert counted.device_status() == 0
        assert_within_gate(out, exp, f"step {step}")


@pytest.mark.parametrize("hinted", [False, True])
def test_a_long_context_in_no_group_sends_the_call_to_the_two_kernels(cabi, hinted):
    """One request of 30000 tokens beside 39 behind a prefix: three launches, two if the caller (mistakenly, here) says that
    every request is in a group; the same result."""
    counted = Counted(cabi)
    _decode(counted, 40, 32, 4, 39, 4096, (5, 512), 128, (30000,), cabi.PFD_FLAG_ALL_IN_GROUPS if hinted else 0)
    assert counted.launches == ([2, 2] if hinted else [3, 3])


@pytest.mark.parametrize("batch,hq,hkv,prefix,own,split,launches", [
    (40, 32, 4, 4096, (0, 1, 31, 32, 33, 64, 65, 512), 128, 2),   # more tiles than SMs, the last row tile of 64 rows
    (20, 64, 8, 5136, (17, 300, 301), 304, 2),                    # a last chunk of one page, one piece to a suffix
    (32, 16, 2, 4096, (0, 1, 31, 32, 33, 64, 65, 512), 128, 3),   # fewer tiles than SMs
    (40, 32, 4, 4096, (0, 1, 16), 64, 3),                         # hardly any own tokens
])
def test_one_prefix_on_either_side_of_the_rule(cabi, batch, hq, hkv, prefix, own, split, launches):
    from single_gpu_inference_lab_b200.workloads import quantize_per_head

    gen = torch.Generator().manual_seed(batch)
    pages, d = 1500, 128
    kc, ks = quantize_per_head(torch.randn(pages, 16, hkv, d, generator=gen))
    vc, vs = quantize_per_head(torch.randn(pages, 16, hkv, d, generator=gen))
    lens = torch.tensor([prefix + own[r % len(own)] for r in range(batch)], dtype=torch.int32)
    max_len = prefix + max(own)
    table = torch.randint(0, pages, (batch, -(-max_len // 16)), generator=gen, dtype=torch.int32)
    table[:, :prefix // 16] = table[0, :prefix // 16]
    q = torch.randn(batch, hq, d, generator=gen).to(torch.bfloat16)
    exp = oracle.reference(q, kc, vc, table.long(), lens, ks, vs)
    gq, gkc, gvc, gt, gl, gks, gvs = (t.to(DEV) for t in (q, kc, vc, table, lens, ks, vs))
    slots = -(-prefix // 256) + -(-max(own) // split)
    ws = tuple(torch.full(s, float("nan"), device=DEV) for s in ((batch, hq, slots, d), (batch, hq, slots), (batch, hq, slots)))
    for step in range(2):
        out = torch.full_like(gq, float("nan"))
        before = cabi.launch_count()
        cabi.shared_prefix_decode_fp8_e4m3(gq, gkc, gvc, gt, gl, prefix_len=prefix, k_scale=gks, v_scale=gvs, max_seq_len=max_len,
                                           split_size=split, output=out, workspace=ws)
        torch.cuda.synchronize()
        assert cabi.launch_count() - before == launches and cabi.device_status() == 0
        assert_within_gate(out, exp, f"step {step}")


@pytest.mark.parametrize("shape", [
    (150, 16, 2, 8, 1500, 40),    # many requests in none: the scan takes two rounds, items are taken in several turns
    (12, 32, 8, 8, 4000, 16),     # a few long ones: as many splits as their slots allow
    (40, 8, 8, 0, 700, 100),      # no group at all
    (16, 28, 4, 15, 900, 300),    # one request in none
])
def test_requests_in_no_group_on_the_two_kernels(two_kernels, shape):
    base.test_requests_in_no_group_have_ctas_of_their_own(two_kernels, *shape)
    assert two_kernels.launches == [3, 3]


@pytest.mark.parametrize("hint", [False, True])
def test_more_tiles_than_tile_slots_on_the_two_kernels(two_kernels, hint):
    base.test_grouped_decode_with_more_tiles_than_tile_slots(two_kernels, hint)
    assert two_kernels.launches == [3, 3]


@pytest.mark.parametrize("batch,hq,hkv,groups_of,prefix,own,split,alone", [
    (64, 32, 2, 17, 2304, (1, 64, 100), 64, (2400, 1, 300)),  # 16 heads: nine row tiles for eight slots, the ninth in a second turn
    (100, 24, 2, 9, 272, (17, 33), 48, (500,)),               # 12 heads, eleven groups: more than are looked up at once
    (30, 18, 2, 29, 256, (3, 90), 64, (257,)),                # 9 heads: rows of one request in two tiles
])
def test_more_heads_than_the_fused_kernel_takes(cabi, batch, hq, hkv, groups_of, prefix, own, split, alone):
    counted = Counted(cabi)
    _decode(counted, batch, hq, hkv, groups_of, prefix, own, split, alone)
    assert counted.launches == [3, 3]
