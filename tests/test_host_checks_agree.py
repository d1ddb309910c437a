"""The native front ends and the Python assertions behind them accept the same arguments.  Every operator is given a call that
both accept, changed in one argument at a time: another type, number of dimensions, size, stride or device, another number.
No GPU and no memory: the tensors are CUDA tensors in name only, made from an address that nothing may read, and a call that the
native front end accepts ends at the missing driver.  Not run where there is a driver."""
from __future__ import annotations

import ctypes
import importlib

import pytest
import torch

import flaggems_vllm as fg
from flaggems_vllm import _native

pytestmark = pytest.mark.skipif(torch.cuda.is_available(), reason="accepted calls would launch on addresses that are not memory")

BF16, F16, F32, I64, I32, U8 = torch.bfloat16, torch.float16, torch.float32, torch.int64, torch.int32, torch.uint8
DLPACK = {BF16: (4, 16), F16: (2, 16), F32: (2, 32), I64: (0, 64), I32: (0, 32), U8: (1, 8)}


class _Device(ctypes.Structure):
    _fields_ = [("type", ctypes.c_int32), ("index", ctypes.c_int32)]


class _Type(ctypes.Structure):
    _fields_ = [("code", ctypes.c_uint8), ("bits", ctypes.c_uint8), ("lanes", ctypes.c_uint16)]


class _Tensor(ctypes.Structure):
    _fields_ = [("data", ctypes.c_void_p), ("device", _Device), ("ndim", ctypes.c_int32), ("dtype", _Type),
                ("shape", ctypes.POINTER(ctypes.c_int64)), ("strides", ctypes.POINTER(ctypes.c_int64)), ("offset", ctypes.c_uint64),
                ("context", ctypes.c_void_p), ("deleter", ctypes.c_void_p)]


class Spec:
    """A tensor by its properties; `make` gives one on cuda:`device` (`None`: an ordinary tensor of the CPU)."""

    def __init__(self, dtype, *shape, strides=None, device=0):
        if strides is None:
            strides, n = [], 1
            for size in reversed(shape):
                strides.insert(0, n)
                n *= max(size, 1)
        self.dtype, self.shape, self.strides, self.device = dtype, tuple(shape), tuple(strides), device

    def make(self, keep):
        if self.device is None:
            return torch.empty_strided(self.shape, self.strides, dtype=self.dtype)
        n = len(self.shape)
        shape, strides = (ctypes.c_int64 * n)(*self.shape), (ctypes.c_int64 * n)(*self.strides)
        t = _Tensor(1 << 32, _Device(2, self.device), n, _Type(*DLPACK[self.dtype], 1), shape, strides, 0, None, None)
        keep += [shape, strides, t]
        capsule = ctypes.pythonapi.PyCapsule_New
        capsule.restype, capsule.argtypes = ctypes.py_object, [ctypes.c_void_p, ctypes.c_char_p, ctypes.c_void_p]
        return torch.utils.dlpack.from_dlpack(capsule(ctypes.addressof(t), b"dltensor", None))

    def changed(self):
        d, s, st = self.dtype, self.shape, self.strides
        for other in DLPACK:
            if other != d:
                yield Spec(other, *s, strides=st)
        yield Spec(d, 1, *s)
        yield Spec(d, *s, 1)
        yield Spec(d, *s[1:])
        for i in range(len(s)):
            for size in (s[i] + 1, s[i] - 1):
                yield Spec(d, *s[:i], size, *s[i + 1 :])
        yield Spec(d, *s, strides=[2 * x for x in st])
        if len(s) > 1:
            yield Spec(d, *s, strides=[st[0] + 32, *st[1:]])
            yield Spec(d, *s, strides=[*st[:-1], 2])
            yield Spec(d, *reversed(s), strides=tuple(reversed(st)))
        if len(s) > 2:
            yield Spec(d, *s, strides=[s[1] * (st[1] + 32), st[1] + 32, *st[2:]])
        yield Spec(d, *s, strides=st, device=1)
        yield Spec(d, *s, strides=st, device=None)

    def __repr__(self):
        return f"{str(self.dtype)[6:]}{list(self.shape)} strides {list(self.strides)} on {'cpu' if self.device is None else f'cuda:{self.device}'}"


def changed_number(v):
    return ["x", None] if isinstance(v, float) else [0, -1, v + 1, v - 1, 2 * v, 3, 64, 128, 1 << 40, "x", str(v), None]


OPS = {
    "prologue": (fg.fused_deepseek_v4_qnorm_rope_kv_rope_quant_insert,
                 (Spec(BF16, 5, 4, 512), Spec(BF16, 5, 512), Spec(U8, 3, 64 * 584), Spec(I64, 5), Spec(I64, 5), Spec(F32, 99, 64), 1e-6, 64)),
    "q_kv_rmsnorm": (fg.fused_q_kv_rmsnorm, (Spec(BF16, 5, 1536), Spec(BF16, 5, 512), Spec(BF16, 1536), Spec(BF16, 512), 1e-6)),
    "group_quant": (fg.per_token_group_quant_fp8, (Spec(BF16, 6, 512), 128, 1e-10, None, False, True)),
    "group_quant, column-major scales": (fg.per_token_group_quant_fp8, (Spec(BF16, 6, 512), 128, 1e-10, None, True, True)),
    "act_quant": (fg.act_quant_triton, (Spec(BF16, 6, 512), 128, None)),
    "inv_rope": (fg.fused_inv_rope_fp8_quant, (Spec(BF16, 5, 16, 512), Spec(I64, 5), Spec(F32, 99, 64), 4, 4, 448, 64, 128, 1e-10, None, False)),
    "inv_rope, packed scales": (fg.fused_inv_rope_fp8_quant,
                                (Spec(BF16, 5, 16, 512), Spec(I64, 5), Spec(F32, 99, 64), 4, 4, 448, 64, 128, 1e-10, None, True)),
    "indexer_q": (fg.fused_indexer_q_rope_quant, (Spec(I64, 5), Spec(BF16, 5, 8, 128), Spec(F32, 99, 64), Spec(BF16, 5, 8), 0.1, 0.1, False)),
    "indexer_q, mxfp4": (fg.fused_indexer_q_rope_quant, (Spec(I64, 5), Spec(BF16, 5, 8, 128), Spec(F32, 99, 64), Spec(BF16, 5, 8), 0.1, 0.1, True)),
    "indexer_k": (fg.indexer_k_quant_and_cache, (Spec(BF16, 5, 128), Spec(U8, 3, 64, 132), Spec(I64, 5), 128, "ue8m0")),
    "cp_gather": (fg.cp_gather_indexer_k_quant_cache, (Spec(U8, 3, 64, 132), Spec(U8, 7, 128), Spec(U8, 7, 4), Spec(I32, 2, 3), Spec(I32, 3))),
    "global_topk": (fg.compute_global_topk_indices_and_lens, (Spec(I32, 5, 32), Spec(I32, 5), Spec(I32, 2, 9), 64, Spec(I32, 5))),
    "combine_topk": (fg.combine_topk_swa_indices, (Spec(I32, 5, 32), Spec(I32, 3), Spec(I32, 2), Spec(I32, 2), 128, 4, 32, 100, 50)),
    "dequantize_and_gather": (fg.dequantize_and_gather_k_cache,
                              (Spec(BF16, 2, 9, 512), Spec(U8, 3, 64 * 584), Spec(I32, 2), Spec(I32, 2), Spec(I32, 2, 3), 64, 0, 64, None, None)),
    "top_k_decode": (fg.top_k_per_row_decode, (Spec(F32, 4, 900), 2, Spec(I32, 2), Spec(I32, 4, 64), 4, 900, 1, 64)),
    "top_k_prefill": (fg.top_k_per_row_prefill, (Spec(F32, 4, 900), Spec(I32, 4), Spec(I32, 4), Spec(I32, 4, 64), 4, 900, 1, 64)),
    "persistent_topk": (fg.persistent_topk, (Spec(F32, 4, 900), Spec(I32, 4), Spec(I32, 4, 512), Spec(U8, 64), 512, 900)),
}


# Accepted by the assertions, refused by the front end, which says why: sizes the library cannot take.  So are numbers that are none.
LIMITS = {("group_quant", 1, -1), ("group_quant, column-major scales", 1, -1), ("act_quant", 1, -1), ("dequantize_and_gather", 7, -1),
          ("dequantize_and_gather", 7, 1 << 40), ("top_k_decode", 1, 1 << 40)}


def accepts(op, args, native):
    """Whether the native front end, or else the assertions behind it, accept the call, and the message if not."""
    module, keep, answers = importlib.import_module(op.__module__), [], []
    call = module._bind()

    def watched(*a):
        answers.append(call(*a) if native else None)
        return answers[-1]

    module._call = watched
    try:
        op(*[a.make(keep) if isinstance(a, Spec) else a for a in args])
        return True, ""  # nothing to do: an empty batch
    except _native.Dsv4Error as e:  # (a code of the library itself: the front end had accepted)
        return (not native or "refused" not in str(e)), str(e)
    except (AssertionError, TypeError, ValueError, IndexError, AttributeError, ArithmeticError) as e:
        return False, f"{type(e).__name__} {e}"
    except RuntimeError as e:
        return native and "driver" in str(e), str(e)
    finally:
        module._call = call


@pytest.mark.parametrize("name", OPS)
def test_both_accept_the_same(name, monkeypatch):
    monkeypatch.setattr(torch.cuda, "_lazy_init", lambda: None)
    op, args = OPS[name]
    assert accepts(op, args, True)[0] and accepts(op, args, False)[0]
    refused = 0
    for i, a in enumerate(args):
        if isinstance(a, (bool, str, type(None))):
            continue
        for c in a.changed() if isinstance(a, Spec) else changed_number(a):
            changed = args[:i] + (c,) + args[i + 1 :]
            (native, why), (python, _) = accepts(op, changed, True), accepts(op, changed, False)
            if python and (c in ("x", None) or (name, i, c) in LIMITS):
                assert not native or (name, i) == ("persistent_topk", 5), (i, c)
                assert native or "the call was refused (" in why, (i, c, why)
            else:
                assert native == python, (i, c, why)
            refused += not native
    assert refused > 20
