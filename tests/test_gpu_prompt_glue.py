"""The glue kernels' forms for prompt-sized steps, at the sizes where they are chosen and at their edges."""
import pytest
import torch

from cuteafd_b200 import ops
from cuteafd_b200.ops import ActBuffer, KIND_FP8B, KIND_MXFP4, KIND_NVFP4
from cuteafd_b200.ref import ops as rops, quant

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def status_word():
    return torch.zeros(4, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("interleaved", [False, True])
@pytest.mark.parametrize("norms", [False, True])
@pytest.mark.parametrize("T,Hq,Hkv", [(3, 5, 1), (700, 64, 4), (1500, 13, 3)])      # a head per warp; several, not dividing the heads
def test_rotation_of_several_heads_per_warp(interleaved, norms, T, Hq, Hkv):
    g = torch.Generator().manual_seed(T)
    qkv = torch.randn(T, (Hq + 2 * Hkv) * 128, generator=g).to(torch.bfloat16)
    pos = torch.randint(0, 9000, (T,), generator=g)
    slots = torch.randperm(T + 5, generator=g)[:T]
    wq, wk = (torch.rand(128, generator=g) + 0.5 if norms else None for _ in range(2))
    d = lambda t: None if t is None else t.to(DEV)
    x, kv, st = d(qkv.clone()), torch.full((T + 5, 2, Hkv, 128), 7.0, dtype=torch.bfloat16, device=DEV), status_word()
    ops.qk_norm_rope_kvwrite(x, d(pos.int()), d(slots.int()), d(wq), d(wk), kv, T, Hq, Hkv, 128, 1e6, interleaved, 1e-6, st)
    torch.cuda.synchronize()
    assert int(st[0]) == 0
    heads = qkv.float().reshape(T, Hq + 2 * Hkv, 128)
    q, k, v = heads[:, :Hq], heads[:, Hq:Hq + Hkv], heads[:, Hq + Hkv:]
    if norms:
        q, k = rops.rmsnorm(q, wq, 1e-6), rops.rmsnorm(k, wk, 1e-6)
    # fp32 angles of up to 9000 are good to 5e-4, the result is rounded to bf16
    near = lambda a, b: float((a.float().cpu() - b).abs().max()) < 2 ** -8 * float(b.abs().max()) + 1e-3 * float(b.abs().max())
    assert near(x[:, :Hq * 128].reshape(T, Hq, 128), rops.apply_rope(q, pos, 1e6, interleaved))
    assert near(kv[slots.to(DEV), 0], rops.apply_rope(k, pos, 1e6, interleaved))
    assert torch.equal(kv[slots.to(DEV), 1].float().cpu(), v)
    bad = slots.clone().int()
    bad[T // 2] = T + 5
    ops.qk_norm_rope_kvwrite(x, d(pos.int()), d(bad), d(wq), d(wk), kv, T, Hq, Hkv, 128, 1e6, interleaved, 1e-6, st)
    assert int(st[0]) != 0                                                  # reported, not written


@pytest.mark.parametrize("rows,K", [(33, 16384), (700, 1536), (4097, 144)])        # from 4097 groups on; groups that do not fill a block; a short last group
def test_fp8_rows_of_whole_words(rows, K):
    x = (torch.randn(rows, K, generator=torch.Generator().manual_seed(K)) * 3).to(torch.bfloat16)
    x[1] = 0
    x[2, :] *= 1e-6
    act = ActBuffer.alloc(KIND_FP8B, rows, K, 128, DEV)
    ops.quant_fp4_rows(x.to(DEV), act)
    torch.cuda.synchronize()
    pad = torch.nn.functional.pad(x.float(), (0, -K % 128))
    q, s = quant.act_quant_fp8_block(pad)
    assert torch.equal(act.data.cpu(), q[:, :K]) and torch.equal(act.sf.cpu(), s)


@pytest.mark.parametrize("kind", [KIND_NVFP4, KIND_MXFP4])
def test_four_bit_codes_of_every_bf16_value(kind):
    """Every bf16 pattern beside a fixed largest value of its block: ties, both zeros, subnormals."""
    bits = torch.arange(1 << 16, dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    vals = bits[torch.isfinite(bits.float()) & (bits.float().abs() <= 6)]
    n = (15 if kind == KIND_NVFP4 else 31)
    vals = vals[:vals.numel() // (32 * n) * 32 * n].reshape(-1, n)
    x = torch.cat([torch.full((vals.shape[0], 1), 6.0, dtype=torch.bfloat16), vals], 1).reshape(-1, 32 * (n + 1))
    act = ActBuffer.alloc(kind, x.shape[0], x.shape[1], 128, DEV)
    ops.quant_fp4_rows(x.to(DEV), act, inv_gs=torch.tensor([1.0], device=DEV) if kind == KIND_NVFP4 else None)
    torch.cuda.synchronize()
    p, s = quant.nvfp4_quantize(x.float(), 1.0)[:2] if kind == KIND_NVFP4 else quant.mxfp4_quantize(x.float())
    assert torch.equal(act.data.cpu(), p) and torch.equal(act.sf.cpu()[:, :s.shape[1]], s)


@pytest.mark.parametrize("kind", [KIND_NVFP4, KIND_MXFP4])
def test_rows_gathered_quantised_equal_rows_quantised_gathered(kind):
    T, H, rows = 700, 1024, 5000
    g = torch.Generator(device=DEV).manual_seed(1)
    x = torch.randn(T, H, generator=g, device=DEV).to(torch.bfloat16)
    src = torch.randint(0, T, (rows,), generator=g, device=DEV, dtype=torch.int32)
    n = torch.tensor([rows - 37], dtype=torch.int32, device=DEV)
    gs, st = torch.tensor([64.0], device=DEV), status_word()
    a, t, b = (ActBuffer.alloc(kind, r, H, 128, DEV) for r in (rows, T, rows))
    ops.quant_fp4_rows(x, a, src_rows=src, n_rows_dev=n, inv_gs=gs)
    ops.route_gather(ops.quant_fp4_rows(x, t, inv_gs=gs).data, t.sf, src, n, b, rows, status=st)
    torch.cuda.synchronize()
    assert int(st[0]) == 0 and torch.equal(a.data, b.data) and torch.equal(a.sf, b.sf)


@pytest.mark.parametrize("T,H", [(5, 8192), (5, 8200), (3, 9216), (2, 16384), (2, 16392), (2, 32768)])
def test_combine_with_next_norm_of_wide_rows(T, H):
    """Rows of one, two and four vectors per thread, at the edges: a block of 1024 threads has 64 registers for each."""
    k, g = 4, torch.Generator(device=DEV).manual_seed(H)
    y, w = torch.randn(T * k, H, generator=g, device=DEV).to(torch.bfloat16), torch.rand(H, generator=g, device=DEV) + 0.5
    slot, wts = torch.randperm(T * k, generator=g, device=DEV).view(T, k).int(), torch.rand(T, k, generator=g, device=DEV)
    slot[0, 1] = -1
    x = torch.randn(T, H, generator=g, device=DEV).to(torch.bfloat16)
    want, got, xn = x.clone(), x.clone(), torch.zeros_like(x)
    ops.moe_combine(y, slot, wts, None, want, want, T, k)
    ops.moe_combine(y, slot, wts, None, got, got, T, k, norm_w=w, eps=1e-6, xn=xn)
    torch.cuda.synchronize()
    assert torch.equal(want, got)
    ref = rops.rmsnorm(want.float().cpu(), w.cpu(), 1e-6)
    assert bool(((xn.float().cpu() - ref).abs() <= 2 ** -8 * ref.abs()).all())              # half a last place of bf16, and fp32 sums
