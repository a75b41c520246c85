"""The smoke entry point passes on the library as it is built."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")
def test_smoke_passes(capsys):
    import __graft_entry__

    __graft_entry__.smoke()
    assert capsys.readouterr().out.count("ok=True") == 3
