"""Decode attention that cuts every sequence by its length, against the form with one part per sequence, and against the oracle."""
import pytest
import torch

from cuteafd_b200 import ops
from cuteafd_b200.ops import ActBuffer, KIND_NVFP4
from cuteafd_b200.ref import ops as rops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
PAGE = 64


# even lengths (left whole); uneven ones; one long sequence among short ones; lengths around page borders; more than 32 sequences
LENGTHS = {"even": [1024] * 6, "uneven": [37 + 211 * i for i in range(12)], "one-long": [3] * 9 + [9000] + [130] * 5, "borders": [63, 64, 65, 127, 128, 129],
           "many": [1 + (97 * i) % 1500 for i in range(45)]}


@pytest.mark.parametrize("name", list(LENGTHS))
@pytest.mark.parametrize("rows,Hq,Hkv", [(1, 64, 4), (4, 64, 4), (13, 16, 2)])
def test_cut_by_length_matches_one_part(name, rows, Hq, Hkv):
    lens = [max(n, rows) for n in LENGTHS[name]]
    n, T = len(lens), len(lens) * rows
    g = torch.Generator(device=DEV).manual_seed(T + Hq)
    per = [-(-l // PAGE) for l in lens]
    pages = torch.randperm(sum(per), generator=torch.Generator().manual_seed(n))
    table, at = torch.zeros(n, max(per), dtype=torch.int32), 0
    for s, p in enumerate(per):
        table[s, :p] = pages[at:at + p]
        at += p
    kv = torch.randn(1, sum(per) * PAGE, 2, Hkv, 128, generator=g, device=DEV).to(torch.bfloat16)
    q = torch.randn(T, (Hq + 2 * Hkv) * 128, generator=g, device=DEV).to(torch.bfloat16)
    sink = torch.randn(Hq, generator=g, device=DEV)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    meta = (table.to(DEV), i32(lens), i32([rows * s for s in range(n)]), i32([rows] * n))
    status, maps = torch.zeros(4, dtype=torch.int32, device=DEV), ops.encode_kv_tmaps(kv)
    kw = dict(T=T, n_seq=n, max_q_len=rows, q_stride=q.shape[1], Hq=Hq, Hkv=Hkv, sink=sink, status=status)
    want, got = (torch.zeros(T, Hq * 128, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    ops.paged_attention_tc(q, maps[0], *meta, want, **kw)
    slots = ops.attn_slots(n, rows, Hq, Hkv, 1)
    assert slots > n and ops.attn_slots(n, rows, Hq, Hkv, 2) == ops.attn_slots(1, rows, Hq, Hkv, 1) == 0
    po, pml = torch.full((slots * rows * Hq * 128,), float("nan"), device=DEV), torch.full((slots * rows * Hq * 2,), float("nan"), device=DEV)
    quant = ActBuffer.alloc(KIND_NVFP4, T, Hq * 128, 128, DEV)
    gs = torch.tensor([64.0], device=DEV)
    assert ops.paged_attention_slots(q, maps[0], *meta, got, **kw, slots=slots, part_o=po, part_ml=pml,
                                     slot_of_row=torch.zeros(T, 4, dtype=torch.int32, device=DEV), quant=quant, inv_gs=gs)
    torch.cuda.synchronize()
    assert int(status[0]) == 0
    # probabilities are rounded against the same reference maximum: only the order of fp32 sums differs, a last place of bf16 here and there
    assert float((got.float() - want.float()).norm() / want.float().norm()) < 2 ** -11
    again = ops.quant_fp4_rows(got, ActBuffer.alloc(KIND_NVFP4, T, Hq * 128, 128, DEV), inv_gs=gs)
    assert torch.equal(quant.data, again.data) and torch.equal(quant.sf, again.sf)
    for s in (0, n - 1):
        slot = (table[s, torch.arange(lens[s]) // PAGE].long() * PAGE + torch.arange(lens[s]) % PAGE)
        k, v = (kv[0, slot.to(DEV), i].float().cpu() for i in (0, 1))
        pos = torch.arange(lens[s])
        ref = rops.attention(q[s * rows:(s + 1) * rows, :Hq * 128].float().cpu().reshape(rows, Hq, 128), k, v, pos[-rows:], pos, sink=sink.cpu()).reshape(rows, -1)
        assert float((got[s * rows:(s + 1) * rows].float().cpu() - ref).norm() / ref.norm()) < 1e-2
