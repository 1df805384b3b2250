"""Into how many parts of K an engine cuts a dense product of a prompt-sized step."""
import types

import pytest
import torch

from cuteafd_b200.engine import engine as E
from cuteafd_b200.engine.engine import Engine
from cuteafd_b200.ops import KIND_BF16, KIND_FP8B, KIND_MXFP4, KIND_NVFP4


def parts(monkeypatch, kind, T, tn, N, K, out) -> int:
    """The `splits` that reach the kernel for T rows of an operand in token tiles of `tn`."""
    seen = []
    monkeypatch.setattr(E.ops, "tc_linear", lambda *a, **kw: seen.append(kw["splits"]))
    eng = types.SimpleNamespace(sm_count=148, status=None, launches_per_step=0)
    eng._splits, eng._tiling = (lambda *a: Engine._splits(eng, *a)), (lambda *a: Engine._tiling(eng, *a))
    Engine._dense(eng, types.SimpleNamespace(kind=kind, N=N, K=K), types.SimpleNamespace(tn=tn), torch.empty(0, dtype=out), T)
    return seen[0]


@pytest.mark.parametrize("tn", [128, 256])
@pytest.mark.parametrize("T", [65, 128, 300, 2048, 4096])
@pytest.mark.parametrize("N,K", [(128, 4096), (256, 7168)])
def test_router_logits_keep_the_parts_that_idle_sms_give(monkeypatch, tn, T, N, K):
    tiles = -(-N // 128) * -(-T // tn)
    want = max(1, min(8, 148 // tiles))
    assert parts(monkeypatch, KIND_BF16, T, tn, N, K, torch.float32) == want
    assert parts(monkeypatch, KIND_BF16, T, tn, N, K, torch.bfloat16) == 1
    assert parts(monkeypatch, KIND_BF16, T, tn, N, 2048, torch.float32) == 1


@pytest.mark.parametrize("kind", [KIND_NVFP4, KIND_MXFP4])
def test_fp4_products_keep_their_parts_and_fp8_ones_have_none(monkeypatch, kind):
    assert parts(monkeypatch, kind, 130, 128, 4096, 8192, torch.bfloat16) == 2
    assert parts(monkeypatch, kind, 65, 128, 4096, 4096, torch.bfloat16) == 4
    assert parts(monkeypatch, kind, 300, 128, 4096, 8192, torch.bfloat16) == 1
    assert parts(monkeypatch, KIND_FP8B, 130, 128, 1536, 7168, torch.bfloat16) == 1
