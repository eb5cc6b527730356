"""What the op layer refuses, and how (no GPU: every case ends before a plan is built)."""
from types import SimpleNamespace

import pytest
import torch

from tileccl_b200.ops import torch_ops


@pytest.mark.parametrize("op", ["_gemm", "_gemm_rs", "_ag_gemm"])
@pytest.mark.parametrize("shape", [(), (64,), (2, 256, 64), (2, 2, 256, 64)])
def test_a_weight_that_is_no_matrix_is_a_value_error(monkeypatch, op, shape):
    monkeypatch.setitem(torch_ops._ctx, "heap", SimpleNamespace(world=1, rank=0))
    monkeypatch.setitem(torch_ops._ctx, "plans", {})
    with pytest.raises(ValueError):
        getattr(torch_ops, op)(torch.zeros(256, 64, dtype=torch.bfloat16), torch.zeros(shape, dtype=torch.bfloat16))
    assert not torch_ops._ctx["plans"]
