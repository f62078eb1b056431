"""The tensor-core and chunked forms of single kernels at the sizes where they can go wrong (edges of tiles, remainders, the
smallest and the largest sizes that take them), against the same in 64 bits (needs a B200)."""
import math
from types import SimpleNamespace

import pytest
import torch

from questwend_b200.kernels import ops

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")
BF, F64 = torch.bfloat16, torch.float64


def paged(lens, rows_of, width):
    """Sequences of these lengths in pages of 64 dealt out in reverse order: (page table, pools filled by ``rows_of(shape)``
    for each of ``width``).  The rows behind a sequence's end hold large numbers: nothing may read them."""
    pages = [-(-n // 64) for n in lens]
    order = list(range(sum(pages)))[::-1]
    table = torch.zeros(len(lens), max(pages), dtype=torch.int32, device=DEV)
    pools = [rows_of((sum(pages), heads, 64, size)) for heads, size in width]
    for b, (n, p) in enumerate(zip(lens, pages)):
        mine, order = order[:p], order[p:]
        table[b, :p] = torch.tensor(mine, dtype=torch.int32)
        for pool in pools:
            pool[mine[-1], :, n - 64 * (p - 1):] = 1e4
    return table, pools


def rows(pool, table, n):
    return pool[table[:-(-n // 64)].long()].double().permute(1, 0, 2, 3).reshape(pool.shape[1], -1, pool.shape[3])[:, :n]


def softmax(q, k, v, scale, pos, window=0, softcap=0.0, sink=None):
    """q [n, d] at positions ``pos`` [n] over k, v [m, .], one head."""
    s = q @ k.T * scale
    if softcap:
        s = softcap * torch.tanh(s / softcap)
    back = pos[:, None] - torch.arange(len(k), device=DEV)[None, :]
    s = s.masked_fill((back < 0) | ((back >= window) if window else False), -math.inf)
    if sink is not None:
        s = torch.cat([s, sink.expand(len(s), 1)], 1)
    return torch.softmax(s, 1)[:, :len(k)] @ v


# ----------------------------------------------------------------------------- latent attention, single tokens
@pytest.mark.parametrize("H, L, R", [(16, 512, 64), (1, 8, 0), (17, 128, 64), (3, 136, 8), (16, 256, 64), (33, 264, 56), (2, 512, 0), (5, 64, 128)])
@pytest.mark.parametrize("window", [0, 1, 65, 700])
def test_latent_single_tokens_on_the_tensor_cores(H, L, R, window):
    """Queries and probabilities are held to 32-bit there, so what is left against 64 bits is the rounding of the bfloat16
    results, half a unit in the last of 8 bits, and a little for sums of 32-bit products."""
    torch.manual_seed(H + L + R + window)
    lens = [1, 31, 32, 33, 64, 65, 127, 1000, 2048, 2049, 4161]
    B = len(lens)
    table, (pool,) = paged(lens, lambda s: torch.randn(s, device=DEV).to(BF), [(1, L + R)])
    q_abs, q_rot = torch.randn(H, B, L, device=DEV), torch.randn(B, H, R, device=DEV)
    sink = torch.randn(H, device=DEV) if window != 65 else None
    scale = (L + R) ** -0.5
    alone = []
    for pick in (list(range(B)), [1], [9], [10]):
        ctx = SimpleNamespace(single_token=True, n_seqs=len(pick), max_len=max(lens[b] for b in pick), max_new=1,
                              pos0=torch.tensor([lens[b] - 1 for b in pick], device=DEV).int(),
                              cu_seqlens=torch.arange(len(pick) + 1, device=DEV).int())
        out = ops.latent_attention(q_abs[:, pick].contiguous(), q_rot[pick].contiguous(), pool, table[pick].contiguous(), ctx, sink, scale, window)
        alone.append(out)
        for i, b in enumerate(pick):
            k = rows(pool, table[b], lens[b])[0]
            q = torch.cat([q_abs[:, b], q_rot[b]], 1).double()
            ref = torch.cat([softmax(q[h:h + 1], k, k[:, :L], scale, torch.tensor([lens[b] - 1], device=DEV), window,
                                     sink=None if sink is None else sink[h].double()) for h in range(H)])
            err = (out[:, i].double() - ref).abs()
            assert (err <= 2.0 ** -8 * ref.abs() + 2e-5).all(), (lens[b], err.max())
    for i, b in enumerate([1, 9, 10]):                      # a sequence's result does not depend on the batch
        assert torch.equal(alone[0][:, b], alone[i + 1][:, 0])
