"""The token tiles and K splits that an engine's dense products take, at the borders of the rule, against the oracle."""
import types

import pytest
import torch

from cuteafd_b200 import ops
from cuteafd_b200.engine.engine import Engine
from cuteafd_b200.ops import ActBuffer, TcWeight, KIND_BF16, KIND_FP8B
from cuteafd_b200.ref import quant

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("kind", [KIND_BF16, KIND_FP8B])
@pytest.mark.parametrize("T", [17, 32, 33, 64, 65, 200])
@pytest.mark.parametrize("N,K", [(256, 1024), (2048, 512), (20480, 256)])            # K split over a cluster; in one piece; more tiles than SMs
def test_dense_products_of_every_tiling(kind, T, N, K):
    eng = types.SimpleNamespace(sm_count=148)
    eng._splits = lambda *a: Engine._splits(eng, *a)
    cap = 64 if T <= 64 else 256
    g = torch.Generator(device=DEV).manual_seed(T + N)
    x = torch.randn(cap, K, generator=g, device=DEV).to(torch.bfloat16)
    act = ActBuffer.wrap_bf16(x, min(cap, 128)) if kind == KIND_BF16 else ops.quant_fp4_rows(x, ActBuffer.alloc(kind, cap, K, min(cap, 128), DEV))
    w, st = TcWeight.random(1, N, K, kind, DEV, seed=N), torch.zeros(4, dtype=torch.int32, device=DEV)
    operand, splits = Engine._tiling(eng, w, act, T)
    assert operand.tn <= max(act.tn, 32) and (operand.tn < 128 or splits == 1)
    y = torch.zeros(cap, N, dtype=torch.float32, device=DEV)
    ops.tc_linear(w, operand, y, rows=T, splits=splits, status=st)
    torch.cuda.synchronize()
    assert int(st[0]) == 0 and bool((y[T:] == 0).all())
    if kind == KIND_BF16:
        xd = x.double()
    else:
        xd = (quant.e4m3_decode(act.data.cpu()).reshape(cap, -1, 128) * act.sf.cpu()[:, :, None]).reshape(cap, K).double().to(DEV)
    ref = xd[:T] @ w.dequantize()[0].double().to(DEV).T
    assert float((y[:T].double() - ref).norm() / ref.norm()) < 1e-6 * K ** 0.5       # fp32 sums of K products


@pytest.mark.parametrize("kind", [KIND_BF16, KIND_FP8B])
def test_the_narrow_tiles_of_an_operand_come_with_it(kind):
    """A new shape's first step allocates and copies nothing for them."""
    acts = [ActBuffer.alloc(kind, 64, 512, 64, DEV)] + ([ActBuffer.wrap_bf16(torch.zeros(64, 512, dtype=torch.bfloat16, device=DEV), 64)] if kind == KIND_BF16 else [])
    torch.cuda.synchronize()
    before = torch.cuda.memory_stats()["allocation.all.allocated"]
    narrow = [a.retiled(32) for a in acts]
    assert torch.cuda.memory_stats()["allocation.all.allocated"] == before
    for a, b in zip(acts, narrow):
        assert b.tn == 32 and b.data is a.data and b.sf is a.sf and b is a.retiled(32) and a.retiled(64) is a
        assert torch.equal(b.tmap, ops.encode_tmap(a.data, 32)) and torch.equal(a.tmap, ops.encode_tmap(a.data, 64))
