"""The kernels that ``bench.py`` names beside a time are the ones that the step launched."""

import importlib.util
from pathlib import Path
from types import SimpleNamespace

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def bench():
    spec = importlib.util.spec_from_file_location("bench_under_test", ROOT / "bench.py")
    module = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(module)
    return module


@pytest.mark.parametrize("launches,kernels", [
    (2, ["shared_prefix_fused_kernel", "paged_decode_merge_kernel"]),
    (3, ["shared_prefix_dense_kernel", "paged_decode_fp8_partial_tma_kernel", "paged_decode_merge_kernel"]),
])
def test_a_shared_prefix_step_names_the_kernels_it_launched(bench, launches, kernels):
    named = bench.Case.kernel_name(SimpleNamespace(shared_prefix=True), {"path": 2, "launches_per_step": launches})
    assert named.split(" + ") == kernels


def test_other_steps_are_named_by_their_path(bench):
    assert bench.Case.kernel_name(SimpleNamespace(shared_prefix=False), {"path": 3, "launches_per_step": 2}) == "paged_decode_fp8_chunk_kernel"
