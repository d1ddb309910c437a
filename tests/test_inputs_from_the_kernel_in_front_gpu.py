"""Operators whose inputs the kernel directly in front of them in the stream has just written.

A kernel asks L2 for its inputs while the kernel in front still runs, and waits for that kernel before it loads them.  A chain in which
every input comes from the launch in front, over buffers that held other values a moment before, has to give what the same calls give
with a synchronisation between them - bit for bit, at sizes whose last tile is ragged and at sizes of several waves."""
from __future__ import annotations

import pytest
import torch

import flaggems_vllm as fg
from flaggems_vllm.testing import workloads

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
EPS, BS, HEADS = 1e-6, 64, 16


def chain(s, between):
    """norms -> quantiser -> key insert -> prologue (twice, in place) -> indexer query -> epilogue; `between` runs after every call."""
    qr, kv = fg.fused_q_kv_rmsnorm(s["qr"], s["kv"], s["wq"], s["wkv"], EPS)
    between()
    qr8, qr_scale = fg.per_token_group_quant_fp8(qr, 128, scale_ue8m0=True)
    between()
    fg.indexer_k_quant_and_cache(qr[:, :128], s["icache"], s["slots"], 128, "ue8m0")
    between()
    for _ in range(2):
        fg.fused_deepseek_v4_qnorm_rope_kv_rope_quant_insert(s["q"], kv, s["cache"], s["slots"], s["pos"], s["cs"], EPS, BS)
        between()
    out = [qr, kv, qr8, qr_scale, s["icache"], s["cache"], s["q"]]
    n = s["q"].shape[0]
    for fp4 in (False, True):
        iq, iw = fg.fused_indexer_q_rope_quant(s["pos"], s["q"].view(n, 4 * HEADS, 128), s["cs"], s["iw"], 0.1, 0.2, use_fp4=fp4)
        between()
        out += [*(iq if fp4 else [iq]), iw]
        # the next consumer's input: the same buffer, written again by the launch in front of it
        fg.fused_deepseek_v4_qnorm_rope_kv_rope_quant_insert(s["q"], kv, s["cache"], s["slots"], s["pos"], s["cs"], EPS, BS)
        between()
    o8, o_scale = fg.fused_inv_rope_fp8_quant(s["q"], s["pos"], s["cs"], 8, HEADS // 8, tma_aligned_scales=True)
    between()
    return [t.clone() for t in out + [o8, o_scale]]


@pytest.mark.parametrize("n", [1, 3, 61, 257, 1100, 4097])
def test_chain_equals_the_synchronised_chain(n):
    g = torch.Generator(device=DEV).manual_seed(n)
    act = lambda *shape: torch.empty(shape, dtype=torch.bfloat16, device=DEV).normal_(generator=g)  # noqa: E731
    blocks = -(-n // BS)
    s = {
        "wq": act(1536), "wkv": act(512), "cs": workloads.cos_sin_table(4096).to(DEV), "iw": act(n, 4 * HEADS),
        "pos": torch.randint(0, 4096, (n,), generator=g, device=DEV), "slots": torch.randperm(blocks * BS, generator=g, device=DEV)[:n].contiguous(),
        "qr": act(n, 1536), "kv": act(n, 512), "q": act(n, HEADS, 512),
        "cache": torch.zeros(blocks, BS * 584, dtype=torch.uint8, device=DEV), "icache": torch.zeros(blocks, BS, 132, dtype=torch.uint8, device=DEV),
    }
    for repeat in range(4):
        fresh = {k: act(*s[k].shape) for k in ("qr", "kv", "q")}
        results = []
        for between in (lambda: None, torch.cuda.synchronize):
            for k, v in fresh.items():
                s[k].copy_(v)
            torch.cuda.synchronize()
            results.append(chain(s, between))
        torch.cuda.synchronize()
        for i, (a, b) in enumerate(zip(*results)):
            a, b = a.contiguous().view(torch.uint8), b.contiguous().view(torch.uint8)
            assert torch.equal(a, b), f"output {i} of pass {repeat}"
