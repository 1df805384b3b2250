"""Scratch of split attention: how it grows, what stays for captured steps, and that it is on the memory ledger."""
import types

import torch

from cuteafd_b200.engine import engine as E
from cuteafd_b200.engine.engine import Engine
from cuteafd_b200.utils.memory_ledger import LEDGER


def test_a_growing_batch_outgrows_few_buffers(monkeypatch):
    """One sequence more per step, from 38 to 64 of 8 rows: few buffers, together no larger than the last one, all kept and charged."""
    monkeypatch.setattr(E.ops, "attn_slots", lambda n, rows, Hq, Hkv, splits: n + 112 if splits == 1 else 0)
    a = types.SimpleNamespace(kind="gqa", n_heads=64, n_kv_heads=4, head_dim=2)
    eng = types.SimpleNamespace(spec=types.SimpleNamespace(attn=a), kv_tmaps=(), max_seqs=64, device="cpu")
    for name in ("_grown", "_attn_slots"):
        setattr(eng, name, getattr(Engine, name).__get__(eng))
    charged, seen = LEDGER.by_scope["workspace/attention"], []
    for n in range(38, 65):
        Engine._ensure_attn_scratch(eng, E.StepShape(T=8 * n, n_seq=n, max_q_len=8, n_logits=8 * n, attn_splits=1))
        rows = (n + 112) * 8 * 64
        assert eng.part_o.numel() >= rows * 2 and eng.part_ml.numel() >= rows * 2
        if not any(b is eng.part_o for b in seen):
            seen.append(eng.part_o)
    done = eng.part_done
    Engine._ensure_attn_scratch(eng, E.StepShape(T=64, n_seq=4, max_q_len=16, n_logits=64, attn_splits=8))
    assert 1 < len(seen) <= 3 and all(any(b is k for k in eng._outgrown) for b in seen[:-1])
    assert sum(b.numel() for b in seen[:-1]) <= seen[-1].numel() and eng.part_o is seen[-1] and eng.part_done is done and done.numel() == 64 * 64
    held = seen + [eng.part_ml] + [b for b in eng._outgrown if not any(b is k for k in seen)]
    assert LEDGER.by_scope["workspace/attention"] - charged == 4 * sum(b.numel() for b in held)


def test_latent_engines_grow_theirs_the_same_way():
    """A captured step holds the address of the scratch that it was captured with, so nothing that a larger step outgrew is given back."""
    eng = types.SimpleNamespace(device="cpu")
    first = Engine._grown(eng, "mla_part_o", 1000)
    assert Engine._grown(eng, "mla_part_o", 900) is first
    second = Engine._grown(eng, "mla_part_o", 1001)
    assert second.numel() == 2000 and eng._outgrown == [first] and eng.mla_part_o is second
    import inspect
    from cuteafd_b200.engine import mla
    assert "self.mla_part_o =" not in inspect.getsource(mla)
