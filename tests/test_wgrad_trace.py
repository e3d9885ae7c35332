"""The trace of a weight gradient names the product that is launched: operands, transposed store and tile width of the plan (host code)."""
import types

import pytest
import torch

from terra_b200 import _ext
from terra_b200.ops import _flags as F
from terra_b200.ops import blocks


@pytest.mark.parametrize("M,N,K,sums,swapped", [(450001, 384, 2304, True, True), (200000, 376, 2296, False, True), (139264, 384, 1536, True, False),
                                                (512, 96, 288, False, False)])
def test_the_product_that_is_launched(monkeypatch, capsys, M, N, K, sums, swapped):
    ext = _ext.load()
    assert ext.wgrad_swapped(N, K, M, sums) == swapped
    launched = types.SimpleNamespace(wgrad_plan=ext.wgrad_plan, wgrad_swapped=ext.wgrad_swapped, wgrad=lambda *args: None)
    monkeypatch.setattr(blocks, "TRACE", True)
    monkeypatch.setattr(blocks._ext, "load", lambda: launched)
    dy, x, gw = (torch.empty(1, 1).expand(*s) for s in ((M, N), (M, K), (N, K)))
    blocks.wgrad_accumulate(dy, x, gw, torch.empty(N) if sums else None)
    line = capsys.readouterr().err
    a, b = ((M, K), (M, N)) if swapped else ((M, N), (M, K))
    flags = F.EPI_OUT_F32 | F.EPI_ATOMIC | (F.EPI_TRANSPOSE if swapped else 0)
    bn, _, split = ext.wgrad_plan(N, K, M, sums)
    assert f"gemm a={a}/" in line and f" b={b}/" in line and f"flags={flags} split_k={split} bn={bn} " in line


def test_an_empty_operand_is_refused():
    with pytest.raises(RuntimeError):
        _ext.load().wgrad_swapped(384, 0, 1000, True)
