"""Two copies of the library in one process (an application that links it and loads a package that brings its own): each keeps its own
state, so every kind of call works in both, whichever came first."""
import shutil

import pytest
import torch

from tests import datagen
from tests import gpu_util as gu

pytestmark = pytest.mark.gpu


def test_every_call_works_in_both_copies(tmp_path):
    copy = tmp_path / "libmlops_attention_copy.so"
    shutil.copy(gu.OURS, copy)
    results = []
    for path in (gu.OURS, str(copy)):
        lib = gu.CLib(path)
        q, k, v = (gu.bf16_tensor(x) for x in datagen.uneven_case(5, 1, 4, 1, 400, q_rows=400))
        c = lib.encode(k[:, :, :200].contiguous(), v[:, :, :200].contiguous(), "4+2", capacity=512)
        outs = [lib.prefill(c, k[:, :, 200:].contiguous(), v[:, :, 200:].contiguous(), q[:, :, 200:].contiguous())]  # tensor-core pass
        outs.append(lib.prefill(c, k[:, :, :3].contiguous(), v[:, :, :3].contiguous(), q[:, :, :3].contiguous()))   # few-row pass
        for tau in (0.0, 1.0):  # two sweeps, one
            outs.append(lib.decode(c, q[:, :, 0].contiguous(), tau=tau))
        torch.cuda.synchronize()
        results.append(outs)
    assert all(torch.equal(a, b) for a, b in zip(*results))
