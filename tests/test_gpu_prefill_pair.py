"""Prompt attention with one or two query tiles per CTA: steps with tiles enough for two against the fp32 oracles of the one-tile kernels' tests, and both
bit for bit against the kernel for windows, given one that hides nothing (all of a row's values are added in the same order)."""
import pytest
import torch

from cuteafd_b200 import ops
from cuteafd_b200.ops.native import call, ptr, stream
from test_gpu_kernels import test_gqa_prefill_attention as check_gqa
from test_gpu_latent_stack import test_expanding_prefill_attention as check_latent

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("Hq,Hkv,use_sink", [(128, 8, False), (128, 16, True), (48, 48, False)])
def test_paged_against_oracle(Hq, Hkv, use_sink):
    check_gqa(Hq, Hkv, 0, use_sink)


@pytest.mark.parametrize("H,d,dv,r,gate", [(60, 128, 128, 128, False), (60, 192, 80, 64, True), (60, 40, 24, 72, True)])
def test_expanded_against_oracle(H, d, dv, r, gate):
    check_latent(H, d, dv, r, gate)


# a lone tile, a ragged pair, a pair whose second tile is one token; over contexts that end inside, at and just behind a key tile
@pytest.mark.parametrize("q,before", [(8, 0), (9, 119), (16, 112), (17, 240), (300, 0), (130, 1000), (257, 383)])
@pytest.mark.parametrize("copies", [1, 40])
def test_paged_same_bits_as_window_kernel(q, before, copies):
    """One sequence takes a tile per CTA, many copies of it take two; a sliding window as long as the sequence takes the one-tile kernel."""
    Hq, Hkv, kv = 64, 4, q + before
    g = torch.Generator().manual_seed(q)
    pages = -(-kv // 64)
    cache = torch.randn(1, pages * 64, 2, Hkv, 128, generator=g).to(torch.bfloat16).to(DEV)
    maps, rows = ops.encode_kv_tmaps(cache), (torch.randn(q, Hq * 128, generator=g) * 2).to(torch.bfloat16).to(DEV)

    def run(n, window):
        x, out = rows.repeat(n, 1).contiguous(), torch.zeros(n * q, Hq * 128, dtype=torch.bfloat16, device=DEV)
        status, table = torch.zeros(4, dtype=torch.int32, device=DEV), i32([list(range(pages))] * n)
        lens, qs, ql = i32([kv] * n), i32([i * q for i in range(n)]), i32([q] * n)
        call("cuteafd_gqa_prefill_attention", ptr(x), ptr(maps[0]), ptr(table), ptr(lens), ptr(qs), ptr(ql), None, ptr(out), n * q, n, q, Hq * 128, Hq, Hkv, pages, window, 128 ** -0.5,
             ptr(status), stream())
        torch.cuda.synchronize()
        assert int(status[0]) == 0
        return out.view(n, q, -1)
    want, got = run(1, kv), run(copies, 0)
    assert float(want.float().abs().max()) > 0
    for i in range(copies):
        assert torch.equal(got[i], want[0]), i

