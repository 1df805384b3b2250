"""Decode attention that cuts every sequence by its length, against the form with one part per sequence, and against the oracle."""
import pytest
import torch

from cuteafd_b200 import ops
from cuteafd_b200.ref import ops as rops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
PAGE = 64


def i32(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


class Step:
    """Sequences of `lens` keys with runs of `runs` query rows each (at the end of their keys), pages in any order, room for `room` pages a sequence."""

    def __init__(self, lens, runs, Hq, Hkv, room=0, spare_rows=0):
        self.lens, self.runs, self.Hq, self.Hkv, self.n = list(lens), list(runs), Hq, Hkv, len(lens)
        self.rows, self.T = max(runs), sum(runs) + spare_rows
        g = torch.Generator(device=DEV).manual_seed(self.T + Hq)
        per = [max(room, -(-l // PAGE)) for l in lens]
        pages, at = torch.randperm(sum(per), generator=torch.Generator().manual_seed(self.n)), 0
        self.table = torch.zeros(self.n, max(per), dtype=torch.int32)
        for s, p in enumerate(per):
            self.table[s, :p] = pages[at:at + p]
            at += p
        self.kv = torch.randn(1, sum(per) * PAGE, 2, Hkv, 128, generator=g, device=DEV).to(torch.bfloat16)
        self.q = torch.randn(self.T, (Hq + 2 * Hkv) * 128, generator=g, device=DEV).to(torch.bfloat16)
        self.sink = torch.randn(Hq, generator=g, device=DEV)
        self.start = [sum(self.runs[:s]) for s in range(self.n)]
        self.kv_len, self.meta = i32(lens), (i32(self.start), i32(self.runs))
        self.status, self.maps = torch.zeros(4, dtype=torch.int32, device=DEV), ops.encode_kv_tmaps(self.kv)
        self.dev_table = self.table.to(DEV)
        self.slots = ops.attn_slots(self.n, self.rows, Hq, Hkv, 1)
        self.part_o, self.part_ml = (torch.full((self.slots * self.rows * Hq * k,), float("nan"), device=DEV) for k in (128, 2))
        self.arrived = torch.zeros(self.n * Hq, dtype=torch.int32, device=DEV)

    def run(self, cut: bool, out=None):
        out = torch.full((self.T, self.Hq * 128), 7.0, dtype=torch.bfloat16, device=DEV) if out is None else out
        kw = dict(T=self.T, n_seq=self.n, max_q_len=self.rows, q_stride=self.q.shape[1], Hq=self.Hq, Hkv=self.Hkv, sink=self.sink, status=self.status)
        if cut:
            ops.paged_attention_slots(self.q, self.maps[0], self.dev_table, self.kv_len, *self.meta, out, **kw, slots=self.slots, part_o=self.part_o, part_ml=self.part_ml,
                                      arrived=self.arrived)
        else:
            ops.paged_attention_tc(self.q, self.maps[0], self.dev_table, self.kv_len, *self.meta, out, **kw)
        return out

    def done(self):
        torch.cuda.synchronize()
        assert int(self.status[0]) == 0 and not bool(self.arrived.any())

    def slots_of(self, s):
        t = torch.arange(self.lens[s])
        return (self.table[s, t // PAGE].long() * PAGE + t % PAGE).to(DEV)

    def oracle(self, s):
        k, v = (self.kv[0, self.slots_of(s), i].float().cpu() for i in (0, 1))
        n, pos = self.runs[s], torch.arange(self.lens[s])
        q = self.q[self.start[s]:self.start[s] + n, :self.Hq * 128].float().cpu().reshape(n, self.Hq, 128)
        return rops.attention(q, k, v, pos[-n:], pos, sink=self.sink.cpu()).reshape(n, -1)

    def check(self, got, some=None):
        for s in some or (0, self.n - 1):
            ref, rows = self.oracle(s), slice(self.start[s], self.start[s] + self.runs[s])
            assert float((got[rows].float().cpu() - ref).norm() / ref.norm()) < 1e-2, s


def rel(a, b):
    return float((a.float() - b.float()).norm() / b.float().norm())


# lengths (of up to 45 sequences) by the step's number of sequences: even (left whole); uneven; one long sequence among short ones; around page borders
LENGTHS = {"even": lambda i, n: 1024, "uneven": lambda i, n: 37 + 211 * i, "one-long": lambda i, n: 9000 if i == n // 2 else 130 - 97 * (i % 2),
           "borders": lambda i, n: (63, 64, 65, 127, 128, 129, 1500)[i % 7], "many": lambda i, n: 1 + (97 * i) % 1500}


@pytest.mark.parametrize("name", list(LENGTHS))
@pytest.mark.parametrize("n,rows,Hq,Hkv", [(40, 1, 64, 4), (38, 4, 64, 4), (24, 13, 64, 4), (80, 13, 16, 2), (19, 16, 64, 4), (20, 1, 8, 8)])
def test_cut_by_length_matches_one_part(name, n, rows, Hq, Hkv):
    """Rows of one query tile and of two (9 to 16 rows of 16 heads per KV head)."""
    st = Step([max(LENGTHS[name](i, n), rows) for i in range(n)], [rows] * n, Hq, Hkv)
    assert st.slots > n
    want, got = st.run(False), st.run(True)
    st.done()
    # probabilities are rounded against the same reference maximum: only the order of fp32 sums differs, a last place of bf16 here and there
    assert rel(got, want) < 2 ** -11
    if name == "even":       # whole sequences take the one-part form's path, and leave no partials
        assert torch.equal(got, want) and bool(st.part_o.isnan().all())
    st.check(got)


def test_runs_of_unequal_length_and_rows_outside_the_sequences():
    """Prompt tails and decode rows in one step: query tiles that some sequences do not have, and rows behind the last sequence, which stay as they were."""
    n = 30
    st = Step([16 + 313 * i % 4000 for i in range(n)], [(1, 16, 3, 9)[i % 4] for i in range(n)], 64, 4, spare_rows=5)
    want, got = st.run(False), st.run(True)
    st.done()
    assert rel(got, want) < 2 ** -11 and bool((got[-5:] == 7).all())
    st.check(got, range(4))


def test_a_captured_step_replays_with_other_lengths():
    """The plan is made on the device, from the lengths of the moment: whole sequences, cut ones, and whole ones again."""
    n = 40
    st = Step([4096] * n, [1] * n, 64, 4)
    got = st.run(True)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        st.run(True, got)
    for lens in ([4096] * n, [1 + (409 * i) % 4096 for i in range(n)], [64] * n, [4000] + [1] * (n - 1), [4096] * n):
        st.lens = lens
        st.kv_len.copy_(i32(lens))
        graph.replay()
        st.done()
        assert rel(got, st.run(False)) < 2 ** -11
        st.check(got)


def test_a_score_far_above_the_first_page():
    """A key in a middle piece that lifts that piece's reference, not the others': their probabilities round against other references than an uncut sequence's
    (a place of bf16 each, 2^-9), no more."""
    n = 40
    st = Step([6000] + [70] * (n - 1), [1] * n, 64, 4)
    st.sink.fill_(-30.0)
    key = st.slots_of(0)[3000]
    st.kv[0, key, 0] = st.q[0, :64 * 128].reshape(4, 16, 128)[:, 0] * 1.5             # scores of about 17 / 0.69 binary orders for the first head of each group
    want, got = st.run(False), st.run(True)
    st.done()
    assert rel(got[:1], want[:1]) < 2 ** -9 and rel(got[1:], want[1:]) < 2 ** -11
    st.check(got)


def test_steps_that_get_no_slots():
    assert ops.attn_slots(40, 1, 64, 4, 2) == 0                                           # cut evenly
    assert ops.attn_slots(37, 1, 64, 4, 1) == 0 and ops.attn_slots(38, 1, 64, 4, 1) > 38      # SMs without a block: contexts of one page
    assert ops.attn_slots(1, 16, 64, 4, 1) == ops.attn_slots(40, 17, 64, 4, 1) == 0
    assert ops.attn_slots(18, 16, 64, 4, 1) == 0 and ops.attn_slots(19, 16, 64, 4, 1) > 19    # two query tiles
