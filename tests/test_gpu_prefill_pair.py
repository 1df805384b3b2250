"""Prompt attention with one or two query tiles per CTA: steps with tiles enough for two against the fp32 oracles of the one-tile kernels' tests, both
bit for bit against the kernel for windows, given one that hides nothing (all of a row's values are added in the same order), and every width and mask against a
softmax in 64 bits."""
import pytest
import torch

from cuteafd_b200 import ops
from cuteafd_b200.ops.native import call, lib, ptr, stream
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



# ------------------------------------------------------------------ steps of sequences (rows, rows in the cache before them) and their outputs in 64 bits
def attended(q, k, v, scale, before, bidir=False, sink=None):
    """q [n, H, d] at positions before .. over k, v [m, H, .]: [n, H, dv]."""
    s = torch.einsum("qhd,khd->hqk", q.double(), k.double()) * scale
    if not bidir:
        s.masked_fill_(torch.arange(k.shape[0], device=DEV)[None] > before + torch.arange(q.shape[0], device=DEV)[:, None], -float("inf"))
    if sink is not None:
        s = torch.cat([s, sink.double()[:, None, None].expand(-1, q.shape[0], 1)], -1)
    return torch.einsum("hqk,khd->qhd", torch.softmax(s, -1)[..., :k.shape[0]], v.double())


class Step:
    def __init__(self, seqs):
        self.seqs, self.n, self.T, self.max_q = seqs, len(seqs), sum(q for q, _ in seqs), max(q for q, _ in seqs)
        self.starts = [sum(q for q, _ in seqs[:i]) for i in range(len(seqs))]
        self.q_start, self.q_len, self.kv_len = i32(self.starts), i32([q for q, _ in seqs]), i32([q + b for q, b in seqs])
        self.gen, self.status = torch.Generator(device=DEV).manual_seed(self.T), torch.zeros(4, dtype=torch.int32, device=DEV)

    def randn(self, *shape):
        return torch.randn(*shape, generator=self.gen, device=DEV).to(torch.bfloat16)

    def rows(self, i):
        return slice(self.starts[i], self.starts[i] + self.seqs[i][0])

    def done(self, out):
        torch.cuda.synchronize()
        assert int(self.status[0]) == 0
        return out


class PagedStep(Step):
    """Key and value heads of dk and dv columns (in the store: whole 64-wide chunks) on scattered pages."""
    def __init__(self, seqs, Hq, Hkv, dk=128, dv=128):
        super().__init__(seqs)
        self.Hq, self.Hkv, self.dp, self.dvp, self.dv = Hq, Hkv, -(-dk // 64) * 64, -(-dv // 64) * 64, dv
        pages = [-(-(q + b) // 64) for q, b in seqs]
        order = torch.randperm(sum(pages), generator=torch.Generator().manual_seed(1)).tolist()
        tables = [[order.pop() for _ in range(p)] for p in pages]
        self.table = i32([t + [0] * (max(pages) - len(t)) for t in tables])
        self.q = torch.nn.functional.pad(self.randn(self.T, Hq, dk), (0, self.dp - dk)).contiguous()
        self.store = torch.zeros(sum(pages) * 64, Hkv * (self.dp + self.dvp), dtype=torch.bfloat16, device=DEV)
        self.k, self.v = [], []
        for (q, b), t in zip(seqs, tables):
            k, v = self.randn(q + b, Hkv, dk), self.randn(q + b, Hkv, dv)
            at = torch.tensor([t[j // 64] * 64 + j % 64 for j in range(q + b)], device=DEV)
            self.store[at] = torch.cat([torch.nn.functional.pad(k, (0, self.dp - dk)).flatten(1), torch.nn.functional.pad(v, (0, self.dvp - dv)).flatten(1)], 1)
            self.k.append(k), self.v.append(v)
            self.slots = getattr(self, "slots", []) + [at]

    def run(self, scale, window=0, extras=None):
        """window < 0: bidirectional."""
        out = torch.full((self.T, self.Hq * self.dv), 7.0, dtype=torch.bfloat16, device=DEV)
        if window < 0:
            maps = ops.encode_kv_tmaps(self.store.view(1, -1, 2, self.Hkv, 128))
            call("cuteafd_gqa_prefill_attention", ptr(self.q), ptr(maps[0]), ptr(self.table), ptr(self.kv_len), ptr(self.q_start), ptr(self.q_len), None, ptr(out), self.T, self.n, self.max_q,
                 self.Hq * 128, self.Hq, self.Hkv, self.table.shape[1], window, scale, ptr(self.status), stream())
        else:
            maps = ops.encode_window_maps(self.store, self.Hkv, self.dp, self.dvp)
            ops.window_attention(self.q.flatten(1), maps, self.table, self.kv_len, self.q_start, self.q_len, out, T=self.T, n_seq=self.n, max_q_len=self.max_q, Hq=self.Hq, Hkv=self.Hkv,
                                 dp=self.dp, dvp=self.dvp, dv=self.dv, window=window, scale=scale, prefill=True, extras=extras, status=self.status)
        return self.done(out).view(self.T, self.Hq, self.dv)

    def want(self, i, scale, bidir=False, sink=None):
        group = lambda t: t.repeat_interleave(self.Hq // self.Hkv, 1)
        return attended(self.q[self.rows(i), :, :self.k[i].shape[2]], group(self.k[i]), group(self.v[i]), scale, self.seqs[i][1], bidir, sink)


class LatentStep(Step):
    """Keys of 64 kn columns per head and, with kr, 64 shared ones; values of 64 nv."""
    def __init__(self, seqs, H, kn, kr, nv):
        super().__init__(seqs)
        self.H, self.kn, self.kr, self.nv, ctx, tot = H, kn, kr, nv, [], 0
        for q, b in seqs:
            ctx.append(tot)
            tot += -(-(q + b) // 64) * 64
        self.ctx, self.ctx_start, self.cap = ctx, i32(ctx), tot + 64
        self.q, self.q_rope = self.randn(H, self.T, kn * 64), self.randn(H, self.T, 64)
        self.kvb, self.lat = self.randn(self.cap, H, (kn + nv) * 64), self.randn(self.cap, 128)

    def run(self, scale, heads=None):
        """`heads`: of these alone, as a step of its own."""
        q, qr, kvb = self.q, self.q_rope, self.kvb
        if heads is not None:
            q, qr, kvb = q[heads].contiguous(), qr[heads].contiguous(), kvb[:, heads].contiguous()
        H, dv = q.shape[0], self.nv * 64
        out = torch.full((self.T, H * dv), 7.0, dtype=torch.bfloat16, device=DEV)
        rope = (ptr(qr), ptr(self.lat), 128, 64) if self.kr else (None, None, 0, 0)
        call("cuteafd_latent_prefill_attention", ptr(q), rope[0], ptr(kvb), *rope[1:], None, self.cap, ptr(self.ctx_start), ptr(self.kv_len), ptr(self.q_start), ptr(self.q_len), None, ptr(out),
             self.T, self.T, self.n, self.max_q, H, self.kn * 64, dv, dv, H * dv, scale, ptr(self.status), stream())
        return self.done(out).view(self.T, H, dv)

    def want(self, i, scale):
        at = slice(self.ctx[i], self.ctx[i] + sum(self.seqs[i]))
        k, q, d = self.kvb[at, :, :self.kn * 64], self.q[:, self.rows(i)].transpose(0, 1), self.kn * 64
        if self.kr:
            k, q = torch.cat([k, self.lat[at, None, 64:].expand(-1, self.H, -1)], -1), torch.cat([q, self.q_rope[:, self.rows(i)].transpose(0, 1)], -1)
        return attended(q, k, self.kvb[at, :, d:], scale, self.seqs[i][1])


# outputs are sums of values of about 1 with weights of 8 bits: errors of 2^-8 of the values' mean size, and the output's rounding
def close(got, want):
    return bool(torch.isfinite(got).all()) and torch.allclose(got.double(), want, atol=1e-2, rtol=2 ** -7)


@pytest.mark.parametrize("scale", [0.0, -0.02])
@pytest.mark.parametrize("form", ["one tile", "pairs", "bidirectional", "wide keys", "latent", "latent pairs"])
def test_scales_that_are_not_positive(form, scale):
    """Hidden keys have no weight whatever the scale: rows average what they see at 0 and turn from the keys they resemble below."""
    seqs = [(300, 20), (17, 0), (64, 200)]
    if form.startswith("latent"):
        step, bidir = LatentStep(seqs, *((3, 1, 1, 2) if form == "latent" else (48, 2, 1, 2))), False
    else:
        step, bidir = PagedStep(seqs, *((8, 8) if form == "one tile" else (128, 16)), *((192, 128) if form == "wide keys" else (128, 128))), form == "bidirectional"
    got = step.run(scale, -1) if bidir else step.run(scale)
    for i in range(len(seqs)):
        want = step.want(i, scale, True) if bidir else step.want(i, scale)
        assert close(got[step.rows(i)], want), (i, float((got[step.rows(i)].double() - want).abs().max()))


@pytest.mark.parametrize("form", ["one tile", "pairs", "bidirectional", "window", "latent", "latent pairs", "wide latent"])
def test_rows_whose_keys_all_score_minus_infinity_are_nan(form):
    """As a softmax over nothing else is; rows that see one more key, or none of these, are not."""
    seqs, low = [(300, 0), (64, 200), (17, 0)], [(0, 150), (0, 130), (0, 1)]
    if "latent" in form:
        step = LatentStep(seqs, *{"latent": (3, 1, 1, 2), "latent pairs": (48, 2, 1, 2), "wide latent": (3, 3, 1, 2)}[form])
        step.q[..., 0] = 1
        for at, (lo, hi) in zip(step.ctx, low):
            step.kvb[at + lo:at + hi, :, 0] = -float("inf")
    else:
        step = PagedStep(seqs, *((8, 8) if form == "one tile" else (128, 16)))
        step.q[..., 0] = 1
        for k, slots, (lo, hi) in zip(step.k, step.slots, low):
            k[lo:hi, :, 0] = -float("inf")
            step.store[slots[lo:hi, None], torch.arange(step.Hkv, device=DEV) * 128] = -float("inf")
    bidir = form == "bidirectional"
    got = step.run(0.1, -1) if bidir else step.run(0.1, 300) if form == "window" else step.run(0.1)
    for i in range(len(seqs)):
        want = step.want(i, 0.1, True) if bidir else step.want(i, 0.1)
        out, none = got[step.rows(i)], want.isnan()
        assert bool(none.any()) == (not bidir and i != 1) and torch.equal(out.isnan(), none)
        assert close(out[~none], want[~none])


# contexts of more than eight key tiles: with 192 columns of keys and 128 of values the ring's eight chunks go round every 1.6 of them
LATENT = [(kn, kr, nv) for kr in (0, 1) for kn in (1, 2, 3) if kn + kr <= 3 for nv in (1, 2)]


@pytest.mark.parametrize("kn,kr,nv", LATENT)
def test_latent_pairs(kn, kr, nv):
    """Against the 64-bit softmax, and bit for bit what few heads give, which take one tile per CTA here or the one-tile kernel."""
    seqs, H, scale = [(250, 900), (257, 383), (20, 1300)], 64, 0.7 * ((kn + kr) * 64) ** -0.5
    step, tiles = LatentStep(seqs, H, kn, kr, nv), lib().cuteafd_latent_prefill_tiles
    assert tiles(kn, kr, nv, H, step.n, step.T, step.max_q) == 2 and tiles(kn, kr, nv, 2, step.n, step.T, step.max_q) < 2
    got = step.run(scale)
    for heads in ([0, 41], [63]):
        assert torch.equal(got[:, heads], step.run(scale, heads))
    for i in range(len(seqs)):
        assert close(got[step.rows(i)], step.want(i, scale))


@pytest.mark.parametrize("heads", [(4, 4), (16, 2), (64, 64), (128, 16)])
def test_bidirectional_sequences_of_unequal_lengths(heads):
    """The first two: one tile per CTA; the others: pairs."""
    step = PagedStep([(300, 0), (129, 0), (100, 60), (17, 0), (256, 0), (1, 0)], *heads)
    got = step.run(0.06, -1)
    for i in range(step.n):
        assert close(got[step.rows(i)], step.want(i, 0.06, True))


@pytest.mark.parametrize("heads", [(6, 2), (160, 80)])
@pytest.mark.parametrize("dk,dv", [(64, 64), (40, 128), (128, 24), (100, 65), (192, 64), (160, 128)])
@pytest.mark.parametrize("gate", ["head", "value", None])
def test_sinks_gates_and_factors_without_a_window(heads, dk, dv, gate):
    """Few heads: one tile per CTA (with 192 columns of keys: the one-tile kernel); many: pairs."""
    (Hq, Hkv), scale = heads, 1.3 * dk ** -0.5
    step = PagedStep([(250, 0), (250, 640)], Hq, Hkv, dk, dv)
    sink, logits = torch.randn(Hq, generator=step.gen, device=DEV) + 2, step.randn(step.T, 3 + Hq * dv)[:, 3:]
    x = ops.attn_extras(sink=sink, gate=None if gate is None else logits, per_value=gate == "value", out_scale=0.6)
    got = step.run(scale, 0, x)
    for i in range(step.n):
        g = logits[step.rows(i)].double().sigmoid()
        factor = {"head": lambda: g[:, :Hq, None], "value": lambda: g.view(-1, Hq, dv), None: lambda: 1.0}[gate]()
        assert close(got[step.rows(i)], step.want(i, scale, sink=sink) * factor * 0.6)
