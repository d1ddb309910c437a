"""The native front ends of the operators: arguments they do not accept give None (the Python operator then names the
argument), whatever their number and type; no GPU."""
from __future__ import annotations

import pytest
import torch

from flaggems_vllm import _native, build

FRONT_ENDS = [n for n in dir(_native.host_calls()) if not n.startswith("_") and n != "bind"]


@pytest.mark.parametrize("name", FRONT_ENDS)
@pytest.mark.parametrize("args", [(), (None,) * 10, (torch.zeros(2, 4, 512, dtype=torch.bfloat16),) * 10, (torch.zeros(0),) * 10, ("x",) * 3,
                                  (1 << 80,) * 10, (float("nan"),) * 10])
def test_refuses_without_raising(name, args):
    assert getattr(_native.host_calls(), name)(*args) is None


def test_another_torch_makes_the_build_stale(monkeypatch):
    """The module calls torch's C++ interface: built for another version, it may not even load."""
    assert _native.host_calls().__doc__ == build.built_for()
    assert build.up_to_date(build.HOST_OUT, build.HOST_SOURCES)
    monkeypatch.setattr(torch, "__version__", torch.__version__ + "1")
    assert not build.up_to_date(build.HOST_OUT, build.HOST_SOURCES)
    assert build.up_to_date(build.OUT, build.SOURCES)  # the operator library knows nothing of torch
