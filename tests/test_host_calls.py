"""The native front ends of the operators: arguments they do not accept give None (the Python operator then names the
argument), whatever their number and type; no GPU."""
from __future__ import annotations

import pytest
import torch

from flaggems_vllm import _native

FRONT_ENDS = [n for n in dir(_native.host_calls()) if not n.startswith("_") and n != "bind"]


@pytest.mark.parametrize("name", FRONT_ENDS)
@pytest.mark.parametrize("args", [(), (None,) * 10, (torch.zeros(2, 4, 512, dtype=torch.bfloat16),) * 10, (torch.zeros(0),) * 10, ("x",) * 3,
                                  (1 << 80,) * 10, (float("nan"),) * 10])
def test_refuses_without_raising(name, args):
    assert getattr(_native.host_calls(), name)(*args) is None
