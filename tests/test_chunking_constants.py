"""The host model of the balanced kernel's work split (chunking_model) has the constants that the library is built with."""

import re
from pathlib import Path

import chunking_model as model

CSRC = Path(__file__).resolve().parents[1] / "single_gpu_inference_lab_b200/csrc"


def _constant(name):
    found = {int(m) for f in CSRC.glob("*.cu*") for m in re.findall(rf"constexpr int {name} = (\d+);", f.read_text())}
    assert len(found) == 1, (name, found)
    return found.pop()


def test_the_model_restates_the_librarys_constants():
    assert model.PIECE_COST == _constant("kChunkPieceCost")
    assert model.MIN_CHUNK_COST == _constant("kMinChunkCost")
    assert model.WARPS_PER_SM == _constant("kChunkWarps")
    assert model.PAGE == _constant("kPage")
