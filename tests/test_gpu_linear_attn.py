"""Gated delta-rule linear attention (GDN: one decay per head; KDA: one per key channel) and the width-4 causal convolution in
front of it, against the fp32 statements in `ref.ops`: decode steps that continue a prefilled state, verify runs with
per-token state snapshots, ragged batches over state slots."""
import pytest
import torch

from cuteafd_b200.ops.native import call, ptr, stream
from cuteafd_b200.ref import ops as rops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("per_channel", [False, True])
def test_gated_delta_rule_matches_reference(per_channel):
    g = torch.Generator().manual_seed(8 + per_channel)
    H, n_slots = 3, 5
    lens = [9, 1, 4]                      # a short prefill run, a decode token, a verify run
    slots = [4, 0, 2]
    T = sum(lens)
    q = torch.nn.functional.normalize(torch.randn(T, H, 128, generator=g), dim=-1) * 128 ** -0.5
    k = torch.nn.functional.normalize(torch.randn(T, H, 128, generator=g), dim=-1)
    v = torch.randn(T, H, 128, generator=g)
    gate = torch.rand(T, H, 128, generator=g) * 0.3 + 0.7 if per_channel else torch.rand(T, H, generator=g) * 0.3 + 0.7
    beta = torch.rand(T, H, generator=g)
    state0 = torch.randn(n_slots, H, 128, 128, generator=g) * 0.1
    b16 = lambda t: t.to(torch.bfloat16)
    d = lambda t: t.to(DEV).contiguous()
    qd, kd, vd = d(b16(q)), d(b16(k)), d(b16(v))
    state = d(state0.clone())
    out = torch.zeros(T, H, 128, dtype=torch.bfloat16, device=DEV)
    snaps = torch.zeros(T, H, 128, 128, device=DEV)
    status = torch.zeros(4, dtype=torch.int32, device=DEV)
    starts = [0, lens[0], lens[0] + lens[1]]
    i32 = lambda v_: torch.tensor(v_, dtype=torch.int32, device=DEV)
    d_slots, d_starts, d_lens = i32(slots), i32(starts), i32(lens)
    gd, bd = d(gate), d(beta)
    call("cuteafd_gated_delta_step", ptr(qd), ptr(kd), ptr(vd), ptr(gd), ptr(bd), ptr(state), ptr(d_slots), ptr(d_starts), ptr(d_lens),
         ptr(out), ptr(snaps), len(lens), H, 1 if per_channel else 0, n_slots, ptr(status), stream())
    torch.cuda.synchronize()
    assert status.tolist() == [0, 0, 0, 0]
    for s, (t0, n, slot) in enumerate(zip(starts, lens, slots)):
        rows = slice(t0, t0 + n)
        want, final, sn = rops.gated_delta_rule(b16(q[rows]).float(), b16(k[rows]).float(), b16(v[rows]).float(), gate[rows], beta[rows], state0[slot])
        got = out[rows].float().cpu()
        assert float((got - want).abs().max()) < 2e-2 * float(want.abs().max()) + 1e-3, f"sequence {s}"
        assert torch.allclose(state[slot].cpu(), final, atol=1e-4, rtol=1e-4)
        assert torch.allclose(snaps[t0 + n - 1].cpu(), final, atol=1e-4, rtol=1e-4) and torch.allclose(snaps[t0].cpu(), sn[0], atol=1e-4, rtol=1e-4)
    untouched = [i for i in range(n_slots) if i not in slots]
    assert torch.equal(state[untouched].cpu(), state0[untouched])


def test_short_conv4_carries_its_history():
    g = torch.Generator().manual_seed(3)
    C, n_slots = 384, 3
    x1, x2 = torch.randn(7, C, generator=g), torch.randn(2, C, generator=g)
    w = torch.randn(C, 4, generator=g) * 0.5
    b16 = lambda t: t.to(torch.bfloat16)
    carry = torch.zeros(n_slots, 3, C, dtype=torch.bfloat16, device=DEV)
    status = torch.zeros(4, dtype=torch.int32, device=DEV)
    i32 = lambda v_: torch.tensor(v_, dtype=torch.int32, device=DEV)
    wd = w.to(DEV)
    want1, c1 = rops.short_conv4(b16(x1).float(), w)
    want2, _ = rops.short_conv4(b16(x2).float(), w, b16(c1).float())
    for x, want in ((x1, want1), (x2, want2)):       # two calls on slot 1: the second continues from the carried inputs
        xd = b16(x).to(DEV)
        y = torch.zeros(x.shape[0], C, dtype=torch.bfloat16, device=DEV)
        d_slot, d_start, d_len = i32([1]), i32([0]), i32([x.shape[0]])
        call("cuteafd_short_conv4", ptr(xd), ptr(wd), ptr(carry), ptr(d_slot), ptr(d_start), ptr(d_len), ptr(y), 1, C, C, n_slots, ptr(status), stream())
        torch.cuda.synchronize()
        assert status.tolist() == [0, 0, 0, 0]
        assert float((y.float().cpu() - want).abs().max()) < 2e-2
    assert bool((carry[0] == 0).all()) and bool((carry[2] == 0).all())


@pytest.mark.parametrize("per_channel", [False, True])
@pytest.mark.parametrize("lens", [(8, 7, 17), (64, 1, 200)])
def test_long_runs_of_the_delta_rule_match_reference(per_channel, lens):
    """Runs around the eight tokens that are staged at a time, with and without the state written back: the fp32 recurrence in the reference's order of
    tokens; sums over 128 rows in another order."""
    g = torch.Generator().manual_seed(sum(lens))
    H, n_slots, T = 4, 3, sum(lens)
    b16 = lambda t: t.to(torch.bfloat16)
    q = b16(torch.nn.functional.normalize(torch.randn(T, H, 128, generator=g), dim=-1) * 128 ** -0.5)
    k = b16(torch.nn.functional.normalize(torch.randn(T, H, 128, generator=g), dim=-1))
    v = b16(torch.randn(T, H, 128, generator=g))
    gate = torch.rand(T, H, 128, generator=g) * 0.2 + 0.8 if per_channel else torch.rand(T, H, generator=g) * 0.2 + 0.8
    beta, state0 = torch.rand(T, H, generator=g), torch.randn(n_slots, H, 128, 128, generator=g) * 0.1
    d = lambda t: t.to(DEV).contiguous()
    i32 = lambda v_: torch.tensor(v_, dtype=torch.int32, device=DEV)
    starts, slots = [0, lens[0], lens[0] + lens[1]], [1, 2, 0]
    args = [d(t) for t in (q, k, v, gate, beta)]
    meta, status = [i32(x) for x in (slots, starts, lens)], torch.zeros(4, dtype=torch.int32, device=DEV)
    for keep, max_len in ((2, max(lens)), (0, max(lens)), (0, 0)):       # outputs only, with the state, length not known
        state, out = d(state0.clone()), torch.zeros(T, H, 128, dtype=torch.bfloat16, device=DEV)
        call("cuteafd_gated_delta_run", *map(ptr, args), ptr(state), *map(ptr, meta), ptr(out), None, 3, H, int(per_channel) | keep, n_slots, max_len, ptr(status), stream())
        torch.cuda.synchronize()
        assert status.tolist() == [0, 0, 0, 0]
        for t0, n, slot in zip(starts, lens, slots):
            rows = slice(t0, t0 + n)
            want, final, _ = rops.gated_delta_rule(q[rows].float(), k[rows].float(), v[rows].float(), gate[rows], beta[rows], state0[slot])
            # bf16 outputs: half a last place of the largest, 2^-9
            assert float((out[rows].float().cpu() - want).abs().max()) < 2 ** -8 * float(want.abs().max())
            assert torch.equal(state[slot].cpu(), state0[slot]) if keep else torch.allclose(state[slot].cpu(), final, atol=1e-5, rtol=1e-5)


@pytest.mark.parametrize("per_channel", [False, True])
def test_short_runs_of_many_sequences_equal_the_long_form(per_channel):
    """Decode-sized steps of more sequences than one wave of the four-block form: the one-block form, against the other one."""
    g = torch.Generator(device=DEV).manual_seed(5)
    H, n, rows = 8, 20, 3
    T = n * rows
    b16 = lambda t: t.to(torch.bfloat16).contiguous()
    unit = lambda: b16(torch.nn.functional.normalize(torch.randn(T, H, 128, generator=g, device=DEV), dim=-1))
    args = [unit(), unit(), b16(torch.randn(T, H, 128, generator=g, device=DEV)),
            torch.rand(*((T, H, 128) if per_channel else (T, H)), generator=g, device=DEV) * 0.3 + 0.7, torch.rand(T, H, generator=g, device=DEV)]
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    meta = [i32(list(range(n))), i32([rows * s for s in range(n)]), i32([rows - s % 2 for s in range(n)])]
    state0, status, got = torch.randn(n, H, 128, 128, generator=g, device=DEV) * 0.1, torch.zeros(4, dtype=torch.int32, device=DEV), []
    for max_len in (rows, 0):
        state, out = state0.clone(), torch.zeros(T, H, 128, dtype=torch.bfloat16, device=DEV)
        call("cuteafd_gated_delta_run", *map(ptr, args), ptr(state), *map(ptr, meta), ptr(out), None, n, H, int(per_channel), n, max_len, ptr(status), stream())
        got.append((state, out.float()))
    torch.cuda.synchronize()
    assert status.tolist() == [0, 0, 0, 0]
    assert torch.allclose(got[0][0], got[1][0], atol=1e-5, rtol=1e-5)
    assert float((got[0][1] - got[1][1]).abs().max()) <= 2 ** -8 * float(got[1][1].abs().max())      # a last place of bf16


@pytest.mark.parametrize("C,ldx", [(384, 512), (130, 131)])          # 8-byte words, and odd rows
@pytest.mark.parametrize("lens", [(1, 2, 3), (16, 17, 50), (4, 200, 33)])
def test_short_conv4_in_token_blocks_matches_reference(C, ldx, lens):
    """Sequences cut into blocks of 16 tokens, fewer blocks than the longest needs, the carry read and replaced by the same launch."""
    g = torch.Generator().manual_seed(C + sum(lens))
    T, n_slots = sum(lens), 4
    b16 = lambda t: t.to(torch.bfloat16)
    x, w, carry0 = b16(torch.randn(T, ldx, generator=g)), torch.randn(C, 4, generator=g) * 0.5, b16(torch.randn(n_slots, 3, C, generator=g))
    i32 = lambda v_: torch.tensor(v_, dtype=torch.int32, device=DEV)
    starts, slots = [0, lens[0], lens[0] + lens[1]], [3, 0, 2]
    xd, wd, meta, status = x.to(DEV), w.to(DEV), [i32(t) for t in (slots, starts, lens)], torch.zeros(4, dtype=torch.int32, device=DEV)
    for update, max_len in ((1, max(lens)), (1, 40), (0, max(lens)), (1, 0)):
        carry, y = carry0.to(DEV), torch.zeros(T, C, dtype=torch.bfloat16, device=DEV)
        call("cuteafd_short_conv4_run", ptr(xd), ptr(wd), ptr(carry), *map(ptr, meta), ptr(y), 3, C, ldx, n_slots, max_len, update, ptr(status), stream())
        torch.cuda.synchronize()
        assert status.tolist() == [0, 0, 0, 0]
        for t0, n, slot in zip(starts, lens, slots):
            want, after = rops.short_conv4(x[t0:t0 + n, :C].float(), w, carry0[slot].float())
            assert float((y[t0:t0 + n].float().cpu() - want).abs().max()) < 2 ** -7 * float(want.abs().max())
            assert torch.equal(carry[slot].cpu(), b16(after) if update else carry0[slot])
        assert torch.equal(carry[1].cpu(), carry0[1])


@pytest.mark.parametrize("lens", [(1, 2, 3), (16, 17, 50), (4, 200, 33)])
def test_outputs_may_take_the_place_of_inputs(lens):
    """The convolution over its own rows, and the delta rule's output over its queries, keys or values: as into rows of their own."""
    g = torch.Generator(device=DEV).manual_seed(sum(lens))
    H, C, n, T = 4, 384, 3, sum(lens)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    meta, status = [i32(t) for t in ((2, 0, 1), (0, lens[0], lens[0] + lens[1]), lens)], torch.zeros(4, dtype=torch.int32, device=DEV)
    x, w, carry0 = (torch.randn(*s, generator=g, device=DEV) for s in ((T, C), (C, 4), (n, 3, C)))
    for max_len in (0, max(lens)):
        got = []
        for same in (False, True):
            rows, carry = x.to(torch.bfloat16), carry0.to(torch.bfloat16)
            y = rows if same else torch.zeros_like(rows)
            call("cuteafd_short_conv4_run", ptr(rows), ptr(w), ptr(carry), *map(ptr, meta), ptr(y), n, C, C, n, max_len, 1, ptr(status), stream())
            got.append((y, carry))
        torch.cuda.synchronize()
        assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    unit = lambda: torch.nn.functional.normalize(torch.randn(T, H, 128, generator=g, device=DEV), dim=-1).to(torch.bfloat16)
    qkv, gate, beta = [unit(), unit(), unit()], torch.rand(T, H, generator=g, device=DEV) * 0.3 + 0.7, torch.rand(T, H, generator=g, device=DEV)
    for over in (None, 0, 1, 2):
        args, state = [t.clone() for t in qkv], torch.zeros(n, H, 128, 128, device=DEV)
        out = torch.zeros_like(qkv[0]) if over is None else args[over]
        call("cuteafd_gated_delta_run", *map(ptr, args), ptr(gate), ptr(beta), ptr(state), *map(ptr, meta), ptr(out), None, n, H, 0, n, max(lens), ptr(status), stream())
        torch.cuda.synchronize()
        want = (out.float(), state) if over is None else want
        assert float((out.float() - want[0]).abs().max()) <= 2 ** -8 * float(want[0].abs().max())      # a last place of bf16
        assert torch.allclose(state, want[1], atol=1e-5, rtol=1e-5)
    assert status.tolist() == [0, 0, 0, 0]


@pytest.mark.parametrize("n,rows", [(9, 3), (10, 3), (10, 4), (19, 4), (19, 5), (28, 6), (28, 7)])
def test_runs_on_both_sides_of_the_line_between_the_forms(n, rows):
    """8 heads: one wave and just more, two and three waves, with the longest run that still takes the short form there and one more."""
    g = torch.Generator(device=DEV).manual_seed(n * rows)
    H, T = 8, n * rows
    unit = lambda: torch.nn.functional.normalize(torch.randn(T, H, 128, generator=g, device=DEV), dim=-1).to(torch.bfloat16)
    args = [unit(), unit(), unit(), torch.rand(T, H, generator=g, device=DEV) * 0.3 + 0.7, torch.rand(T, H, generator=g, device=DEV)]
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    meta, status = [i32(list(range(n))), i32([rows * s for s in range(n)]), i32([rows] * n)], torch.zeros(4, dtype=torch.int32, device=DEV)
    state0, out = torch.randn(n, H, 128, 128, generator=g, device=DEV) * 0.1, torch.zeros(T, H, 128, dtype=torch.bfloat16, device=DEV)
    state = state0.clone()
    call("cuteafd_gated_delta_run", *map(ptr, args), ptr(state), *map(ptr, meta), ptr(out), None, n, H, 0, n, rows, ptr(status), stream())
    torch.cuda.synchronize()
    assert status.tolist() == [0, 0, 0, 0]
    q, k, v, gate, beta = (t.float().cpu() for t in args)
    for s in (0, n - 1):
        at = slice(s * rows, (s + 1) * rows)
        want, final, _ = rops.gated_delta_rule(q[at], k[at], v[at], gate[at], beta[at], state0[s].cpu())
        assert float((out[at].float().cpu() - want).abs().max()) < 2 ** -8 * float(want.abs().max()) and torch.allclose(state[s].cpu(), final, atol=1e-5, rtol=1e-5)
