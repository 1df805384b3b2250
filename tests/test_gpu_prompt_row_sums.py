"""The order in which prompt attention adds up a row's probabilities: key after key, tile after tile, also where two threads share a row.  Layers
behind it choose experts and quantise from these bits."""
import numpy as np
import pytest
import torch

from cuteafd_b200 import ops
from cuteafd_b200.ops.native import call, ptr, stream

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
TILE = 128


def unit_scale() -> float:
    """An fp32 scale whose product with the kernels' fp32 log2(e) rounds to 1: scores are then powers of two."""
    near = np.float32(np.log(2)).view(np.int32) + np.arange(-4, 5, dtype=np.int32)
    return float(next(f for f in near.view(np.float32) if f * np.float32(1.4426950408889634) == np.float32(1)))


def row(n_tiles: int, at: int):
    """Scores and values of one query row over n_tiles of keys, in tile `at`: key 0 has probability 1 and value 1 + 2^-7, keys 64 .. 127 probability 2^-25
    and value 2^11, the others probability 0.  Their products sum to 1 + 3 2^-8 exactly, halfway between two bf16 values.  Added key after key every
    pair 2^-24 is rounded off, the sum stays 1 and the output rounds to the even neighbour, 1 + 2^-6; summed apart, the second half's 64 add
    2^-19 and the output rounds down."""
    score, value = torch.full((n_tiles * TILE,), -200.0), torch.zeros(n_tiles * TILE)
    score[at * TILE], value[at * TILE] = 0.0, 1 + 2 ** -7
    score[at * TILE + 64:(at + 1) * TILE], value[at * TILE + 64:(at + 1) * TILE] = -25.0, 2.0 ** 11
    return score, value


@pytest.mark.parametrize("n_tiles,at", [(1, 0), (2, 0), (2, 1), (3, 1), (4, 3)])
@pytest.mark.parametrize("form", ["paged", "window", "latent"])
def test_row_sum_is_taken_key_after_key(form, n_tiles, at):
    score, value = row(n_tiles, at)
    n = n_tiles * TILE
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    st, out = torch.zeros(4, dtype=torch.int32, device=DEV), torch.zeros(1, 128, dtype=torch.bfloat16, device=DEV)
    q = torch.zeros(1, 128, dtype=torch.bfloat16, device=DEV)
    q[0, 0] = 1
    kv_len, q_start, q_len = i32([n]), i32([0]), i32([1])
    if form != "latent":                                                 # without a window one thread has the row, with one two share it, as in the latent form
        kv = torch.zeros(1, n, 2, 1, 128, dtype=torch.bfloat16, device=DEV)
        kv[0, :, 0, 0, 0], kv[0, :, 1, 0] = score.to(DEV), value[:, None].to(DEV)
        maps, table = ops.encode_kv_tmaps(kv), i32([list(range(n // 64))])
        call("cuteafd_gqa_prefill_attention", ptr(q), ptr(maps[0]), ptr(table), ptr(kv_len), ptr(q_start), ptr(q_len), None, ptr(out), 1, 1, 1, 128, 1, 1,
             table.shape[1], n if form == "window" else 0, unit_scale(), ptr(st), stream())
    else:
        kvb = torch.zeros(n + 64, 256, dtype=torch.bfloat16, device=DEV)
        kvb[:n, 0], kvb[:n, 128:] = score.to(DEV), value[:, None].to(DEV)
        lat, rope = torch.zeros(n + 64, 576, dtype=torch.bfloat16, device=DEV), torch.zeros(1, 64, dtype=torch.bfloat16, device=DEV)
        starts = i32([0])
        call("cuteafd_mla_prefill_attention", ptr(q), ptr(rope), ptr(kvb), ptr(lat), n + 64, ptr(starts), ptr(kv_len), ptr(q_start), ptr(q_len), ptr(out), 1, 1, 1,
             1, unit_scale(), ptr(st), stream())
    torch.cuda.synchronize()
    assert int(st[0]) == 0
    assert torch.equal(out, torch.full_like(out, 1 + 2 ** -6))
