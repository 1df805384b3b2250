"""The wide GEMM (128 tokens x 256 weight rows) at the edges of its tiles: against the oracle, and bit for bit against the narrow kernel,
which sums the same products in the same order."""
import pytest
import torch

from cuteafd_b200 import ops
from cuteafd_b200.ops import ActBuffer, TcWeight, KIND_BF16, KIND_FP8B, KIND_MXFP4, KIND_NVFP4, KIND_W4A8
from cuteafd_b200.ref import quant

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def operand(kind, x, tn):
    if kind == KIND_BF16:
        return ActBuffer.wrap_bf16(x, tn)
    act = ActBuffer.alloc(kind, x.shape[0], x.shape[1], tn, DEV)
    return ops.quant_fp4_rows(x, act, inv_gs=torch.tensor([64.0], device=DEV) if kind == KIND_NVFP4 else None)


def retiled(act, tn):
    return ActBuffer(act.kind, act.rows, act.K, tn, act.data, ops.encode_tmap(act.data, tn), act.sf)


def dequantised(act):
    n = act.K // (16 if act.kind == KIND_NVFP4 else 32)
    if act.kind == KIND_BF16:
        return act.data.double().cpu()
    if act.kind == KIND_FP8B:
        return (quant.e4m3_decode(act.data.cpu()).reshape(act.rows, -1, 128) * act.sf.cpu()[:, :, None]).reshape(act.rows, -1).double()
    return (quant.nvfp4_dequantize(act.data.cpu(), act.sf.cpu()[:, :n], 1 / 64) if act.kind == KIND_NVFP4 else quant.mxfp4_dequantize(act.data.cpu(), act.sf.cpu()[:, :n])).double()


# (rows, N, K): whole tiles; one row and one column block over; a last tile of one row; K of one stage and of an unfinished one
SHAPES = [(2048, 1280, 1024), (1153, 2432, 512), (1025, 2208, 288), (640, 4096, 128), (129, 9600, 640)]


@pytest.mark.parametrize("kind", [KIND_BF16, KIND_NVFP4, KIND_MXFP4, KIND_FP8B])
@pytest.mark.parametrize("T,N,K", SHAPES)
def test_wide_products_equal_narrow_ones(kind, T, N, K):
    if kind == KIND_FP8B:
        K = -(-K // 128) * 128
    g = torch.Generator(device=DEV).manual_seed(T + N)
    x = torch.randn(T, K, generator=g, device=DEV).to(torch.bfloat16)
    w = TcWeight.random(1, N, K, kind, DEV, seed=K)
    act, st = operand(kind, x, 128), torch.zeros(4, dtype=torch.int32, device=DEV)
    r = torch.randn(T, N, generator=g, device=DEV).to(torch.bfloat16)
    for dtype, residual in ((torch.float32, None), (torch.bfloat16, None), (torch.bfloat16, r)):
        wide, narrow = (torch.full((T, N), 7.0, dtype=dtype, device=DEV) for _ in range(2))
        ops.tc_linear(w, act, wide, residual=residual, status=st)
        ops.tc_linear(w, retiled(act, 64), narrow, residual=residual, status=st)
        torch.cuda.synchronize()
        assert int(st[0]) == 0
        assert torch.equal(wide, narrow)
        if dtype == torch.float32:
            ref = dequantised(act) @ w.dequantize()[0].double().T * (1.0 / 64 * 64)
            # fp32 sums of K products, in the tensor core's order
            assert float((wide.double().cpu() - ref).norm() / ref.norm()) < 1e-6 * K ** 0.5
    out = r.clone()
    ops.tc_linear(w, act, out, residual=out, status=st)                 # in place, as the residual stream is
    assert torch.equal(out, wide)


@pytest.mark.parametrize("kind", [KIND_BF16, KIND_NVFP4, KIND_MXFP4])
@pytest.mark.parametrize("counts,N,K", [((128, 1, 0, 127, 129, 300, 64), 768, 512), ((5, 256, 31, 400), 1312, 1024), ((700,) * 3, 512, 288)])
def test_wide_expert_products_equal_narrow_ones(kind, counts, N, K):
    """Grouped by expert: gate and up with the fused activation, quantised for the next product or not, and plain."""
    T, G = sum(counts), len(counts)
    g = torch.Generator(device=DEV).manual_seed(T)
    x = torch.randn(T, K, generator=g, device=DEV).to(torch.bfloat16)
    gate, up = (TcWeight.random(G, N, K, kind, DEV, seed=s) for s in (1, 2))
    act, st = operand(kind, x, 128), torch.zeros(4, dtype=torch.int32, device=DEV)

    def tiled(tn):
        rows, at = [], 0
        for e, n in enumerate(counts):
            rows += [[e, at + o, min(tn, n - o), 0] for o in range(0, n, tn)]
            at += n
        i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
        # a launch is sized for the most tiles a step can have
        return retiled(act, tn), dict(tiles=i32(rows), n_tiles=i32([len(rows)]), max_tiles=max(len(rows) + 3, 80), status=st)

    results = []
    for tn in (128, 32):
        a, tiles = tiled(tn)
        plain, both = (torch.full((T, N), 7.0, dtype=torch.bfloat16, device=DEV) for _ in range(2))
        ops.tc_linear(gate, a, plain, **tiles)
        ops.tc_linear(gate, a, both, w_up=up, **tiles)
        got = [plain, both]
        if kind != KIND_BF16:
            q = ActBuffer.alloc(kind, T, N, tn, DEV)
            ops.tc_linear(gate, a, None, w_up=up, quant_out=q, inv_gs_out=torch.tensor([64.0], device=DEV) if kind == KIND_NVFP4 else None, **tiles)
            got += [q.data, q.sf]
        results.append(got)
    torch.cuda.synchronize()
    assert int(st[0]) == 0
    for a, b in zip(*results):
        assert torch.equal(a, b)
    dense = [w.dequantize()[counts.index(max(counts))].double() for w in (gate, up)]
    s = sum(counts[:counts.index(max(counts))])
    xe = dequantised(act)[s:s + max(counts)]
    ref = torch.nn.functional.silu(xe @ dense[0].T) * (xe @ dense[1].T)
    err = (results[0][1][s:s + max(counts)].double().cpu() - ref).norm() / ref.norm()
    assert float(err) < 2 ** -8                                          # the output's rounding to bf16


# (rows, N, K, parts): even and uneven parts, one row and one column block over, K of an unfinished stage, many small parts, an eighth of the SMs and one unit
PARTS = [(130, 4096, 2048, 2), (65, 512, 4096, 8), (257, 768, 1280, 3), (300, 100, 2336, 4), (129, 288, 1824, 5), (2048, 256, 7168, 4), (1, 256, 1024, 2)]


@pytest.mark.parametrize("kind", [KIND_BF16, KIND_NVFP4, KIND_MXFP4])
@pytest.mark.parametrize("T,N,K,parts", PARTS)
def test_parts_of_k_are_added_as_a_split_adds_them(kind, T, N, K, parts):
    """Bit for bit the narrow kernel's fix-up over CTAs (which a limit on the CTAs selects), with every epilogue, and the 64-bit product."""
    g = torch.Generator(device=DEV).manual_seed(T + N)
    x = torch.randn(T, K, generator=g, device=DEV).to(torch.bfloat16)
    w = TcWeight.random(1, N, K, kind, DEV, seed=K)
    act, st = operand(kind, x, 128), torch.zeros(4, dtype=torch.int32, device=DEV)
    r = torch.randn(T, N, generator=g, device=DEV).to(torch.bfloat16)
    for dtype, residual in ((torch.float32, None), (torch.bfloat16, None), (torch.bfloat16, r)):
        wide, split = (torch.full((T, N), 7.0, dtype=dtype, device=DEV) for _ in range(2))
        ops.tc_linear(w, act, wide, residual=residual, splits=parts, status=st)
        ops.tc_linear(w, act, split, residual=residual, splits=parts, max_ctas=148, status=st)
        torch.cuda.synchronize()
        assert int(st[0]) == 0
        assert torch.equal(wide, split)
        if dtype == torch.float32:
            ref = dequantised(act) @ w.dequantize()[0].double().T
            assert float((wide.double().cpu() - ref).norm() / ref.norm()) < 1e-6 * (K / parts) ** 0.5       # fp32 sums of a part's products


def test_more_parts_than_stages():
    """K of three stages in eight parts: five of them are empty."""
    x = torch.randn(200, 192, device=DEV).to(torch.bfloat16)
    w, st, y = TcWeight.random(1, 320, 192, KIND_BF16, DEV, seed=3), torch.zeros(4, dtype=torch.int32, device=DEV), torch.zeros(200, 320, device=DEV)
    ops.tc_linear(w, operand(KIND_BF16, x, 128), y, splits=8, status=st)
    torch.cuda.synchronize()
    ref = x.double() @ w.dequantize()[0].double().to(DEV).T
    assert int(st[0]) == 0 and float((y.double() - ref).norm() / ref.norm()) < 1e-6 * 192 ** 0.5


@pytest.mark.parametrize("kind,tn,K", [(KIND_BF16, 32, 192), (KIND_BF16, 64, 128), (KIND_BF16, 256, 320), (KIND_NVFP4, 64, 512), (KIND_MXFP4, 256, 768), (KIND_W4A8, 64, 256), (KIND_W4A8, 128, 640)])
def test_more_parts_than_stages_in_narrow_tiles(kind, tn, K):
    """The same through the fix-up over CTAs, whose empty parts must not add what an earlier product left in tensor memory."""
    rows = min(tn, 200)
    w, st = TcWeight.random(1, 320, K, kind, DEV, seed=3), torch.zeros(4, dtype=torch.int32, device=DEV)
    x = torch.randn(rows, K, device=DEV).to(torch.bfloat16)
    act, loud, whole, parts = operand(kind, x, tn), operand(kind, x * 50, tn), torch.zeros(rows, 320, device=DEV), torch.zeros(rows, 320, device=DEV)
    ops.tc_linear(w, act, whole, status=st)
    for _ in range(3):
        ops.tc_linear(w, loud, parts, status=st)
        ops.tc_linear(w, act, parts, splits=8, status=st)
        torch.cuda.synchronize()
        assert int(st[0]) == 0 and float((parts - whole).norm() / whole.norm()) < 1e-6 * K ** 0.5       # fp32 sums of K products in another order
