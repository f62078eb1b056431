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


def paged(lens, rows_of, width, behind=math.nan):
    """Sequences of these lengths in pages of 64 dealt out in reverse order: (page table, pools filled by ``rows_of(shape)``
    for each of ``width``).  The rows behind a sequence's end hold no numbers (or ``behind``): nothing of them may reach a result."""
    pages = [-(-n // 64) for n in lens]
    order = list(range(sum(pages)))[::-1]
    table = torch.zeros(len(lens), max(pages), dtype=torch.int32, device=DEV)
    pools = [rows_of((sum(pages), heads, 64, size)) for heads, size in width]
    for b, (n, p) in enumerate(zip(lens, pages)):
        mine, order = order[:p], order[p:]
        table[b, :p] = torch.tensor(mine, dtype=torch.int32)
        for pool in pools:
            pool[mine[-1], :, n - 64 * (p - 1):] = behind
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


# ----------------------------------------------------------------------------- prompts with two softmax streams a block (tcgen05)
def prompt_step(lens, before=None):
    before = before or [0] * len(lens)
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    return SimpleNamespace(single_token=False, n_seqs=len(lens), max_new=max(lens), max_len=max(n + p for n, p in zip(lens, before)),
                           cu_seqlens=torch.tensor(cu, device=DEV).int(), pos0=torch.tensor(before, device=DEV).int())


def bf16_close(got, ref, spread):
    """Probabilities and results are bfloat16 (half a unit in the last of 8 bits each): a result's error is at most 2^-8 of
    itself and 2^-8 of what its probabilities weigh, of which ``spread``, the largest |value|, is a bound that a row's
    average of rounding errors stays well below."""
    err = (got.double() - ref).abs()
    assert torch.isfinite(got).all() and (err <= 2.0 ** -8 * ref.abs() + 2.0 ** -9 * spread).all(), err.max()
    assert err.square().mean().sqrt() <= 2.0 ** -8 * ref.square().mean().sqrt()


@pytest.mark.parametrize("dim, rot, vdim", [(128, 64, 128), (64, 0, 64), (32, 16, 72), (8, 8, 8), (128, 0, 120), (72, 24, 128)])
@pytest.mark.parametrize("window", [0, 1, 64, 200])
def test_latent_prompts_with_two_streams(dim, rot, vdim, window):
    """Prompts at the edges of 64-key tiles, of 128-row streams and of 256-row blocks; a value that is infinite in one
    sequence stays there."""
    assert ops.latent_prefill_tc_fits(dim, rot, vdim)
    torch.manual_seed(dim + rot + window)
    lens, H = [1, 63, 64, 65, 128, 129, 256, 257, 511], 3
    T = sum(lens)
    q, k, rows_, v = (torch.randn(s, device=DEV).to(BF) for s in ((T, H, dim + rot), (T, H * dim), (T, 16 + rot), (T, H * vdim)))
    sink = torch.randn(H, device=DEV) if window != 64 else None
    gate = torch.randn(T, H, device=DEV) if window else None
    scale = (dim + rot) ** -0.5
    for copies in (1, 8):                                   # 8: enough blocks that one takes 256 rows
        pick = lens * copies
        step = prompt_step(pick)
        rep = lambda t: t.repeat(copies, *([1] * (t.dim() - 1)))
        vv = rep(v)
        at = sum(lens[:4])                                  # the first token of the fifth sequence
        vv[at] = math.inf
        got = ops.latent_prefill(rep(q), rep(k), rep(rows_), vv, step, sink, scale, window, H, dim, rot, vdim,
                                 gate=None if gate is None else rep(gate)).view(copies, T, H, vdim)
        start = 0
        for i, n in enumerate(lens):
            pos = torch.arange(n, device=DEV)
            part = slice(start, start + n)
            for h in range(H):
                keys = torch.cat([k[part].view(n, H, dim)[:, h], rows_[part, 16:]], 1).double()
                ref = softmax(q[part, h].double(), keys, v[part].view(n, H, vdim)[:, h].double(), scale, pos, window,
                              sink=None if sink is None else sink[h].double())
                ref = ref if gate is None else ref * torch.sigmoid(gate[part, h:h + 1].double())
                for c in range(copies):
                    if i != 4 or c:
                        bf16_close(got[c, part, h], ref, 4.0)
            start += n
        ops.gemm_tc_check(DEV)


@pytest.mark.parametrize("H, G, dim, vdim", [(16, 4, 64, 128), (2, 2, 8, 8), (6, 2, 40, 72), (4, 1, 128, 128), (3, 1, 72, 64)])
@pytest.mark.parametrize("softcap, window, chunk, gated", [(0.0, 0, 0, False), (50.0, 0, 0, True), (3.0, 100, 0, False), (0.0, 65, 128, True), (20.0, 0, 96, False)])
def test_two_map_prompts_with_a_stream_a_map(H, G, dim, vdim, softcap, window, chunk, gated):
    """Whole prompts and portions behind cached tokens; caps far above the scores (the series) and among them (ex2 and rcp)."""
    assert ops.maps_prefill_tc_fits(BF, 2, dim, vdim, H // G)
    torch.manual_seed(H + dim + window + chunk)
    lens, before = [1, 63, 64, 130, 300, 33, 64], [0, 0, 0, 0, 0, 70, 191]
    T = sum(lens)
    table, (k_pool, v_pool) = paged([n + b for n, b in zip(lens, before)], lambda s: torch.randn(s, device=DEV).to(BF), [(G, 2 * dim), (G, vdim)])
    q = (2.0 * torch.randn(T, H, 2 * dim, device=DEV)).to(BF)
    gate = torch.randn(T, H + 3, device=DEV) if gated else None
    kw = dict(softcap=softcap, window=window, chunk=chunk, lam=0.4, norm_out=True, eps=1e-5, out_scale=0.3, gate=gate, gate_col0=2 if gated else 0)
    got = ops.maps_attention(q, k_pool, v_pool, table, prompt_step(lens, before), 2, dim ** -0.5, impl="tc", **kw).view(T, H, vdim)
    start = 0
    for b, (n, p) in enumerate(zip(lens, before)):
        ks, vs = rows(k_pool, table[b], n + p), rows(v_pool, table[b], n + p)
        pos = p + torch.arange(n, device=DEV)
        for h in range(H):
            part, g = slice(start, start + n), h // (H // G)
            a = []
            for m in (0, 1):
                ref = torch.empty(n, vdim, dtype=F64, device=DEV)
                qs, kk = q[part, h, m * dim:(m + 1) * dim].double(), ks[g, :, m * dim:(m + 1) * dim]
                for c in (range(0, n + p, chunk) if chunk else [0]):      # chunk by chunk
                    mine = (pos >= c) & (pos < c + chunk) if chunk else torch.ones_like(pos, dtype=torch.bool)
                    if mine.any():
                        ref[mine] = softmax(qs[mine], kk[c:], vs[g][c:], dim ** -0.5, pos[mine] - c, window, softcap)
                a.append(ref)
            ref = a[0] - 0.4 * a[1]
            size = ref.square().mean(1, keepdim=True).add(1e-5).rsqrt()
            ref = ref * size * 0.3
            size = size * 0.3 * (1.4 * 4.0)
            if gated:
                ref, size = ref * torch.sigmoid(gate[part, h + 2:h + 3].double()), size * torch.sigmoid(gate[part, h + 2:h + 3].double())
            bf16_close(got[part, h], ref, size)
        start += n
    ops.gemm_tc_check(DEV)


@pytest.mark.parametrize("dim, vdim", [(64, 64), (64, 128), (128, 64), (72, 120)])
def test_prompts_on_two_streams_where_the_kernel_was_built_otherwise(dim, vdim, monkeypatch):
    """As built here every uncapped kernel for two maps has its registers; without them the mma.sync kernel takes the same calls."""
    assert ops._streams_built(dim, vdim)
    torch.manual_seed(3)
    lens, H = [200, 65], 4
    table, (k_pool, v_pool) = paged(lens, lambda s: torch.randn(s, device=DEV).to(BF), [(2, 2 * dim), (2, vdim)])
    q = torch.randn(sum(lens), H, 2 * dim, device=DEV).to(BF)
    run = lambda: ops.maps_attention(q, k_pool, v_pool, table, prompt_step(lens, [0, 0]), 2, dim ** -0.5, lam=0.4)
    here, names, call = run(), [], ops._call
    monkeypatch.setattr(ops, "_streams_built", lambda *sizes: False)
    monkeypatch.setattr(ops, "_call", lambda module, name, *args, **kw: (names.append(name), call(module, name, *args, **kw))[1])
    bf16_close(run(), here.double(), 8.0)
    assert len(names) == 1 and names[0] in ("qwb_maps_prefill_mma", "qwb_maps_prefill")


def rounded_by_running_maxima(q, k, v, scale):
    """Causal attention as the tensor cores are given it: tiles of 64 keys, probabilities relative to the largest score so far (which
    is 1 then, and exact) in bfloat16, all else in 64 bits; the result in bfloat16."""
    n = len(q)
    m, l, o = torch.full((n, 1), -math.inf, dtype=F64, device=DEV), 0.0, 0.0
    for at in range(0, n, 64):
        s = (q @ k[at:at + 64].T * scale).masked_fill(torch.arange(n, device=DEV)[:, None] < at + torch.arange(len(k[at:at + 64]), device=DEV)[None, :], -math.inf)
        top = torch.maximum(m, s.amax(1, keepdim=True))
        p, fade = torch.exp(s - top), torch.exp(m - top)
        l, o, m = l * fade + p.sum(1, keepdim=True), o * fade + p.float().to(BF).double() @ v[at:at + 64], top
    return (o / l).float().to(BF).double()


@pytest.mark.parametrize("sharp", [1.0, 2.0, 4.0])
def test_probabilities_of_two_streams_are_relative_to_the_largest(sharp):
    """A row's largest probability is 1, which costs no rounding: errors are those of the running maximum, also where few keys weigh."""
    torch.manual_seed(int(sharp))
    T, H, dim = 600, 4, 64
    q, k, v = (torch.randn(T, H, n, device=DEV) for n in (dim, dim, 128))
    q = (sharp * q).to(BF)
    k, v = k.to(BF), v.to(BF)
    got = ops.latent_prefill(q, k.view(T, -1), torch.zeros(T, 16, dtype=BF, device=DEV), v.view(T, -1), prompt_step([T]), None, dim ** -0.5, 0, H, dim, 0, 128).view(T, H, 128)
    table, (k_pool, v_pool) = paged([T], lambda s: torch.randn(s, device=DEV).to(BF), [(H, 2 * dim), (H, 128)])
    at = torch.arange(T, device=DEV)
    k_pool[table[0, at // 64].long(), :, at % 64] = torch.cat([k, k], 2)
    v_pool[table[0, at // 64].long(), :, at % 64] = v
    two = ops.maps_attention(torch.cat([q, q], 2), k_pool, v_pool, table, prompt_step([T]), 2, dim ** -0.5, lam=0.0, impl="tc").view(T, H, 128)
    exact, same = (torch.stack([f(q[:, h].double(), k[:, h].double(), v[:, h].double()) for h in range(H)], 1) for f in (
        lambda a, b, c: softmax(a, b, c, dim ** -0.5, at), lambda a, b, c: rounded_by_running_maxima(a, b, c, dim ** -0.5)))
    allowed = 1.02 * float((same - exact).norm())           # what 32-bit sums and exponentials move across a rounding is far less
    for out in (got, two):
        assert float((out.double() - exact).norm()) <= allowed
    ops.gemm_tc_check(DEV)


@pytest.mark.parametrize("softcap", [0.0, 3.0, 50.0])
def test_two_map_prompts_see_nothing_behind_a_row(softcap):
    """The same bits whatever stands behind the sequence's end in its last page, and whatever tokens follow."""
    H, G, dim, vdim, lens = 16, 4, 64, 128, [1, 33, 70, 130, 300]
    results = []
    for behind, later in ((math.nan, 0), (1e4, 0), (0.0, 0), (0.0, 100)):
        torch.manual_seed(1)                                # the first tokens of a sequence are the same, however many there are
        ks, vs, qs = ([torch.randn(400, *size, device=DEV).to(BF) for _ in lens] for size in ((G, 2 * dim), (G, vdim), (H, 2 * dim)))
        counts = [n + later for n in lens]
        table, pools = paged(counts, lambda s: torch.zeros(s, dtype=BF, device=DEV), [(G, 2 * dim), (G, vdim)], behind)
        for b, n in enumerate(counts):
            at = torch.arange(n, device=DEV)
            for pool, seq in zip(pools, (ks, vs)):
                pool[table[b, (at // 64).long()].long(), :, (at % 64).long()] = seq[b][:n]
        q = torch.cat([x[:n] for x, n in zip(qs, counts)])
        out = ops.maps_attention(q, *pools, table, prompt_step(counts), 2, dim ** -0.5, softcap=softcap, lam=0.4, impl="tc")
        results.append(torch.cat([x[:n] for x, n in zip(out.split(counts), lens)]))
    assert torch.isfinite(results[0]).all() and all(torch.equal(results[0], r) for r in results[1:])
    ops.gemm_tc_check(DEV)


# ----------------------------------------------------------------------------- recurrences in chunks
class Steps(SimpleNamespace):
    """What a recurrence reads of a step: sequences with these numbers of tokens, in these slots."""

    def __init__(self, counts, slots):
        cu = [0]
        for n in counts:
            cu.append(cu[-1] + n)
        seq = [b for b, n in enumerate(counts) for _ in range(n)]
        super().__init__(cu_seqlens=torch.tensor(cu, device=DEV).int(), slots=torch.tensor(slots, device=DEV).int(), n_seqs=len(counts),
                         max_new=max(counts), single_token=all(n == 1 for n in counts), tok_seq=torch.tensor(seq, device=DEV).int())


def sums_close(got, ref, terms=2 ** -15):
    """32-bit sums of a few hundred terms of either sign: far below 2^-15 of the largest."""
    err = (got.double() - ref).abs().max()
    assert torch.isfinite(got).all() and err <= terms * ref.abs().max(), err / ref.abs().max()


@pytest.mark.parametrize("H, P, N, G", [(2, 64, 128, 1), (4, 4, 4, 2), (3, 68, 132, 3), (8, 32, 64, 2), (2, 128, 256, 1)])
@pytest.mark.parametrize("pace", [0.01, 1.0, 40.0])
def test_mamba2_in_chunks(H, P, N, G, pace, monkeypatch):
    """Sequences at the edges of the chunks of 128, from a state, with slow, usual and immediate decays; the scan, which takes
    shorter steps, gives the same; slots of others stay as they are."""
    torch.manual_seed(H + P + N)
    monkeypatch.setattr(ops, "SSM_CHUNKED_FROM", 2)        # all but the shortest
    lens, slots = [1, 64, 127, 128, 129, 300], [4, 2, 7, 1, 5, 3]
    T, inner = sum(lens), H * P
    step = Steps(lens, slots)
    xbc, dt = torch.randn(T, inner + 2 * G * N, device=DEV), torch.randn(T, H + 5, device=DEV)
    bias, a_log, d = torch.randn(H, device=DEV), torch.log(pace * (1 + torch.rand(H, device=DEV))), torch.randn(H, device=DEV)
    start = torch.randn(9, H, P, N, device=DEV)
    state, again = start.clone(), start.clone()
    y = ops.ssm_scan(xbc, dt, 3, bias, a_log, d, state, step, H, P, N, G)
    step.max_new = 1                                        # taken for a short step: the scan
    y_scan = ops.ssm_scan(xbc, dt, 3, bias, a_log, d, again, step, H, P, N, G)
    t = 0
    for n, slot in zip(lens, slots):
        S = start[slot].double()
        ref = torch.empty(n, inner, dtype=F64, device=DEV)
        for i in range(n):
            row = xbc[t + i].double()
            x, (b, c) = row[:inner].view(H, P), (row[inner + k * G * N:inner + (k + 1) * G * N].view(G, N).repeat_interleave(H // G, 0) for k in (0, 1))
            s = torch.nn.functional.softplus(dt[t + i, 3:3 + H].double() + bias.double(), threshold=100.0)
            S = torch.exp(-torch.exp(a_log.double()) * s)[:, None, None] * S + (s[:, None] * x)[:, :, None] * b[:, None, :]
            ref[i] = ((S @ c[:, :, None])[..., 0] + d.double()[:, None] * x).reshape(-1)
        for got, st in ((y, state), (y_scan, again)):
            sums_close(got[t:t + n], ref)
            sums_close(st[slot], S)
        t += n
    assert torch.equal(state[[0, 6, 8]], start[[0, 6, 8]])
    step.max_new, before = max(lens), state.clone()
    ops.ssm_scan(xbc, dt, 3, bias, a_log, d, state, step, H, P, N, G, write_state=False)
    assert torch.equal(state, before)


@pytest.mark.parametrize("rate", [10.0, 80.0, 100.0])
def test_mamba2_in_chunks_with_decays_of_nothing(rate):
    """Rates so large that a token leaves nothing of the state (e^100 is no 32-bit number: its log decay is -infinity), in all heads or
    only with large steps: as the scan, which multiplies by a token's own decay."""
    torch.manual_seed(int(rate))
    H, P, N, G, T = 4, 64, 128, 2, 300
    step = Steps([T], [0])
    xbc, dt = torch.randn(T, H * P + 2 * G * N, device=DEV), torch.randn(T, H, device=DEV) - 3.0
    dt[:, 1] = -40.0                                        # a step of 4e-18: little of e^40, much of e^50
    dt[5::9, 1] = 3.0
    a_log = torch.tensor([rate, rate / 2, 0.0, 1.0], device=DEV)
    bias, d, start = torch.zeros(H, device=DEV), torch.randn(H, device=DEV), torch.randn(1, H, P, N, device=DEV)
    results = []
    for longest in (T, 1):
        step.max_new, state = longest, start.clone()
        results.append((ops.ssm_scan(xbc, dt, 0, bias, a_log, d, state, step, H, P, N, G), state))
    for got, want in zip(*results):
        sums_close(got, want.double(), 2 ** -18)


def matrix_memory(row, at, H, K, P, i_b, f_b, cap, S, top):
    """The mLSTM in 64 bits over one sequence's rows from a memory [H, P + 1, K] and its maxima [H]: (read-outs, divisors, both after it)."""
    row, n, n_qkv, S, top = row.double(), len(row), H * (2 * K + P), S.double().transpose(1, 2), top.double()
    q, k, v = (row[:, a:b].reshape(n, H, -1) for a, b in ((0, H * K), (H * K, 2 * H * K), (2 * H * K, n_qkv)))
    v = torch.cat([v, torch.ones(n, H, 1, dtype=F64, device=DEV)], 2)
    li, lf = (cap * torch.tanh((row[:, c:c + H] + b.double()) / cap) for c, b in ((at, i_b), (at + H, f_b)))
    lf = torch.nn.functional.logsigmoid(lf)
    raw, div = torch.empty(n, H * P, dtype=F64, device=DEV), torch.empty(n, H, dtype=F64, device=DEV)
    for i in range(n):
        new = torch.maximum(top + lf[i], li[i])
        S = torch.exp(top + lf[i] - new)[:, None, None] * S + torch.exp(li[i] - new)[:, None, None] * k[i][:, :, None] * v[i][:, None, :]
        top = new
        read = torch.einsum("hk,hkp->hp", q[i], S) * K ** -0.5
        raw[i], div[i] = read[:, :P].reshape(-1), torch.maximum(read[:, P].abs(), torch.exp(-top)) + 1e-6
    return raw, div, S.transpose(1, 2), top


@pytest.mark.parametrize("lens", [[1025, 31, 1], [2100, 1024, 33], [3, 1, 20]])
@pytest.mark.parametrize("forget", [2.0, 9.0])
def test_exponential_gates_over_several_passes(lens, forget):
    """Running maxima, decays and write strengths of sequences at the edges of a warp and of a pass of 1,024 tokens."""
    torch.manual_seed(sum(lens))
    H, K, P, cap = 2, 4, 4, 15.0
    T, at, step = sum(lens), H * (2 * K + P), Steps(lens, [2, 0, 1])
    proj = torch.randn(T, at + 2 * H, device=DEV)
    proj[:, at + H:] += forget
    i_b, f_b = 0.3 * torch.randn(H, device=DEV), 0.3 * torch.randn(H, device=DEV)
    start, m_start = 0.5 * torch.randn(3, H, P + 1, K, device=DEV), (2 * torch.rand(3, H, 1, device=DEV)).repeat(1, 1, P + 1)
    for chunked in (False, True):
        st, m, t = start.clone(), m_start.clone(), 0
        raw, div = ops.mlstm_scan(proj, at, at + H, i_b, f_b, cap, st, m, step, H, K, P, K ** -0.5, 1e-6, chunked=chunked)
        for n, slot in zip(lens, [2, 0, 1]):
            ref, div_ref, S, top = matrix_memory(proj[t:t + n], at, H, K, P, i_b, f_b, cap, start[slot], m_start[slot, :, 0])
            for got, want in ((raw[t:t + n], ref), (div[t:t + n], div_ref), (st[slot], S)):
                sums_close(got, want)
            assert (m[slot].double() - top[:, None]).abs().max() <= 2 ** -20 * (1 + top.abs().max())
            t += n


@pytest.mark.parametrize("H, K, P", [(1, 4, 4), (2, 64, 128), (3, 20, 68), (2, 132, 60), (2, 256, 512)])
@pytest.mark.parametrize("forget", [-4.0, 2.0, 9.0])
def test_matrix_memory_in_chunks_of_128(H, K, P, forget, monkeypatch):
    """Sequences at the edges of the chunks of 128, from a memory, that fade, last and mix; rows shifted by one float take the
    general form, which gives the same; slots of others stay as they are."""
    torch.manual_seed(H + K + P)
    monkeypatch.setattr(ops, "mlstm_tiles_pay", lambda *sizes: True)
    lens, slots, cap = [1, 64, 127, 128, 129, 300], [4, 2, 7, 1, 5, 3], 15.0
    T, n_qkv, step = sum(lens), H * (2 * K + P), Steps(lens, slots)
    wide = torch.randn(T, -(-(n_qkv + 2 * H) // 4) * 4 + 4, device=DEV)
    at, ld = n_qkv, wide.shape[1]
    wide[:, at + H:at + 2 * H] += forget
    flat = torch.empty(T * ld + 1, device=DEV)
    shifted = flat[1:].view(T, ld)
    shifted.copy_(wide)
    i_b, f_b = 0.3 * torch.randn(H, device=DEV), 0.3 * torch.randn(H, device=DEV)
    start, m_start = 0.5 * torch.randn(9, H, P + 1, K, device=DEV), (2 * torch.rand(9, H, 1, device=DEV)).repeat(1, 1, P + 1)
    forms = []
    for proj in (wide, shifted):
        st, m = start.clone(), m_start.clone()
        raw, div = ops.mlstm_scan(proj, at, at + H, i_b, f_b, cap, st, m, step, H, K, P, K ** -0.5, 1e-6)
        forms.append((raw, div, st, m))
    t = 0
    for n, slot in zip(lens, slots):
        ref, div_ref, S, top = matrix_memory(wide[t:t + n], at, H, K, P, i_b, f_b, cap, start[slot], m_start[slot, :, 0])
        for raw, div, st, m in forms:
            sums_close(raw[t:t + n], ref)
            sums_close(div[t:t + n], div_ref)
            sums_close(st[slot], S)
            assert (m[slot].double() - top[:, None]).abs().max() <= 2 ** -20 * (1 + top.abs().max())
        t += n
    raw, div, st, m = forms[0]
    assert torch.equal(st[[0, 6, 8]], start[[0, 6, 8]]) and torch.equal(m[[0, 6, 8]], m_start[[0, 6, 8]])
    before, m_before = st.clone(), m.clone()
    ops.mlstm_scan(wide, at, at + H, i_b, f_b, cap, st, m, step, H, K, P, K ** -0.5, 1e-6, write_state=False)
    assert torch.equal(st, before) and torch.equal(m, m_before)


@pytest.mark.parametrize("lens", [[1] * 33 + [300, 1, 128, 129, 127] + [1] * 34 + [257], [400] + [1] * 70, [1] * 64 + [130], [5, 1, 700]])
def test_matrix_memory_in_chunks_of_128_among_many_sequences(lens, monkeypatch):
    """Chunks of sequences anywhere among more than a warp's worth of others, against the chunks of 64."""
    torch.manual_seed(len(lens))
    H, K, P, T = 2, 20, 36, sum(lens)
    at, slots = H * (2 * K + P), [(7 * i + 3) % len(lens) for i in range(len(lens))] if len(lens) % 7 else list(range(len(lens)))[::-1]
    proj, zero = torch.randn(T, at + 2 * H, device=DEV), torch.zeros(H, device=DEV)
    start, m_start = 0.5 * torch.randn(len(lens), H, P + 1, K, device=DEV), torch.rand(len(lens), H, 1, device=DEV).repeat(1, 1, P + 1)
    forms = []
    for tiles in (False, True):
        monkeypatch.setattr(ops, "mlstm_tiles_pay", lambda *sizes: tiles)
        st, m = start.clone(), m_start.clone()
        forms.append((*ops.mlstm_scan(proj, at, at + H, zero, zero, 15.0, st, m, Steps(lens, slots), H, K, P, K ** -0.5, 1e-6), st, m))
    for got, want in zip(forms[1], forms[0]):
        sums_close(got, want.double(), 2 ** -18)


@pytest.mark.parametrize("kind", ["mamba2", "delta", "mlstm"])
def test_a_long_prompt_beside_many_single_tokens_costs_what_it_has_to_do(kind, monkeypatch):
    """Twice what the two cost alone at most: no grid is as long as the longest sequence and as wide as all of them (6 times, then).
    The delta rule's chain through the prompt's chunks has its SMs for itself (1.28 times where it shares them, 0.98 where it does not)."""
    H, K, P, G, prompt, others = (64, 128, 64, 8, 8192, 63) if kind == "mamba2" else (16, 128, 128, 16, 8192, 63)
    monkeypatch.setattr(ops, "_mlstm_tiles", lambda *sizes: True)

    def call(lens):
        T, step = sum(lens), Steps(lens, list(range(len(lens))))
        step.min_new, rows, zero = min(lens), torch.randn(T, H * (2 * K + P) + 2 * H, device=DEV), torch.zeros(H * K, device=DEV)
        if kind == "mamba2":
            xbc, state = rows[:, :H * P + 2 * G * K].contiguous(), torch.zeros(len(lens), H, P, K, device=DEV)
            return lambda: ops.ssm_scan(xbc, rows, 0, zero[:H].contiguous(), zero[:H].contiguous(), zero[:H].contiguous(), state, step, H, P, K, G)
        if kind == "delta":
            qkv, side, state = rows[:, :H * (2 * K + P)].contiguous(), rows[:, :H].contiguous(), torch.zeros(len(lens), H, P, K, device=DEV)
            return lambda: ops.delta_rule(qkv, side, 0, side, zero[:H].contiguous(), zero[:H].contiguous(), state, step, H, H, K, P, 1e-6, K ** -0.5, per_head=True)
        state, m, n = torch.zeros(len(lens), H, P + 1, K, device=DEV), torch.zeros(len(lens), H, P + 1, device=DEV), H * (2 * K + P)
        return lambda: ops.mlstm_scan(rows, n, n + H, zero[:H].contiguous(), zero[:H].contiguous(), 15.0, state, m, step, H, K, P, K ** -0.5, 1e-6)

    def took(f):
        best = math.inf
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            f()
            a.record()
            f()
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        return best

    alone, rest, both = took(call([prompt])), took(call([1] * others)), took(call([prompt] + [1] * others))
    torch.cuda.empty_cache()                                # large blocks that a test of little memory would find room in
    assert both <= (1.15 if kind == "delta" else 2.0) * (alone + rest), (alone, rest, both)


@pytest.mark.parametrize("kind", ["mamba2", "mlstm"])
@pytest.mark.parametrize("H, K, P", [(2, 36, 20), (4, 128, 64), (2, 260, 132)])
def test_products_of_three_parts_keep_32_bits(kind, H, K, P, monkeypatch):
    """Sequences at the edges of the eights, stages and chunks.  Without cancellation every digit of a sum can be compared: six products of
    parts leave 2^-23 of a term, cut sums of two and rounded ones of up to 13 about 2^-22, gates and decays (of at most 4) about 2^-21; a part
    less would be off by 2^-17."""
    torch.manual_seed(H + K + P)
    lens, slots = [7, 8, 9, 31, 32, 33, 96, 97, 160], [4, 2, 7, 1, 5, 3, 0, 6, 8]
    T, step, near = sum(lens), Steps(lens, slots), lambda got, ref: ((got.double() - ref).abs() / ref.abs()).max().item() <= 2.0 ** -19
    if kind == "mamba2":
        monkeypatch.setattr(ops, "SSM_CHUNKED_FROM", 2)
        G, inner = 2, H * P
        xbc, dt = 0.1 + torch.rand(T, inner + 2 * G * K, device=DEV), torch.randn(T, H, device=DEV)
        bias, a_log, d, start = torch.zeros(H, device=DEV), torch.full((H,), -4.0, device=DEV), torch.rand(H, device=DEV), torch.rand(9, H, P, K, device=DEV)
        state = start.clone()
        y = ops.ssm_scan(xbc, dt, 0, bias, a_log, d, state, step, H, P, K, G)
    else:
        monkeypatch.setattr(ops, "mlstm_tiles_pay", lambda *sizes: True)
        n_qkv = H * (2 * K + P)
        proj = 0.1 + torch.rand(T, -(-(n_qkv + 2 * H) // 4) * 4, device=DEV)
        proj[:, n_qkv + H:n_qkv + 2 * H] += 5.0
        zero, start, m_start = torch.zeros(H, device=DEV), torch.rand(9, H, P + 1, K, device=DEV), torch.rand(9, H, 1, device=DEV).repeat(1, 1, P + 1)
        state, m = start.clone(), m_start.clone()
        y, div = ops.mlstm_scan(proj, n_qkv, n_qkv + H, zero, zero, 15.0, state, m, step, H, K, P, K ** -0.5, 1e-6)
    t = 0
    for n, slot in zip(lens, slots):
        if kind == "mamba2":
            S, ref = start[slot].double(), torch.empty(n, inner, dtype=F64, device=DEV)
            for i in range(n):
                row = xbc[t + i].double()
                x, (b, c) = row[:inner].view(H, P), (row[inner + k * G * K:inner + (k + 1) * G * K].view(G, K).repeat_interleave(H // G, 0) for k in (0, 1))
                s = torch.nn.functional.softplus(dt[t + i].double(), threshold=100.0)
                S = torch.exp(-math.exp(-4.0) * s)[:, None, None] * S + (s[:, None] * x)[:, :, None] * b[:, None, :]
                ref[i] = ((S @ c[:, :, None])[..., 0] + d.double()[:, None] * x).reshape(-1)
        else:
            ref, div_ref, S, _ = matrix_memory(proj[t:t + n], n_qkv, H, K, P, zero, zero, 15.0, start[slot], m_start[slot, :, 0])
            ref = ref.reshape(n, -1)
            assert near(div[t:t + n], div_ref.reshape(n, H))
        assert near(y[t:t + n], ref) and near(state[slot], S.reshape(state[slot].shape))
        t += n
    ops.gemm_tc_check(DEV)


@pytest.mark.parametrize("forget", [3.0, 5.0])
def test_chunks_of_128_round_as_little_as_those_of_64(forget, monkeypatch):
    """Against 64 bits the mLSTM's two chunked forms are off by the same: their sums and weights have about as many roundings."""
    torch.manual_seed(int(forget))
    H, K, P, T = 4, 128, 128, 1024
    step, at = Steps([T], [0]), H * (2 * K + P)
    proj = torch.randn(T, at + 2 * H, device=DEV)
    proj[:, at + H:] += forget
    zero, errors = torch.zeros(H, device=DEV), []
    ref = matrix_memory(proj, at, H, K, P, zero, zero, 15.0, torch.zeros(H, P + 1, K, device=DEV), torch.zeros(H, device=DEV))[0]
    for tiles in (False, True):
        monkeypatch.setattr(ops, "mlstm_tiles_pay", lambda *sizes: tiles)
        raw = ops.mlstm_scan(proj, at, at + H, zero, zero, 15.0, torch.zeros(1, H, P + 1, K, device=DEV), torch.zeros(1, H, P + 1, device=DEV), step, H, K, P, K ** -0.5, 1e-6)[0]
        errors.append(float((raw.view(ref.shape).double() - ref).norm() / ref.norm()))
    assert errors[1] <= 1.03 * errors[0], errors


@pytest.mark.parametrize("taps, C", [(2, 4), (3, 20), (4, 516), (4, 24)])
@pytest.mark.parametrize("mode", ["silu", "plain", "plus", "bf16"])
def test_convolutions_of_four_channels_a_thread(taps, C, mode):
    """Sequences that begin and end inside a block of eight tokens, against the kernel of one channel a thread (a row that is
    shifted by one float takes it): the same bits."""
    torch.manual_seed(taps + C)
    lens, slots = [3, 1, 9, 8, 40, 2], [1, 0, 5, 3, 2, 6]
    step, T = Steps(lens, slots), sum(lens)
    wide = torch.randn(T, C + 8, device=DEV)
    shifted = torch.zeros(T, C + 8, device=DEV)
    shifted[:, 1:] = wide[:, :-1]
    w, bias, in_bias = torch.randn(C, taps, device=DEV), torch.randn(C, device=DEV), torch.randn(C, device=DEV)
    tail = torch.randn(7, taps - 1, C, device=DEV)
    kw = dict(activation=mode == "silu", plus_input=mode == "plus", out_dtype=BF if mode == "bf16" else torch.float32,
              in_bias=in_bias if mode != "silu" else None)
    a, b = tail.clone(), tail.clone()
    got = ops.short_conv(wide, 4, C, w, bias if mode != "plain" else None, a, step, **kw)
    one = ops.short_conv(shifted, 5, C, w, bias if mode != "plain" else None, b, step, **kw)
    assert torch.equal(got, one) and torch.equal(a, b)


@pytest.mark.parametrize("H, Hk, K, P, per_head", [(2, 2, 128, 128, False), (4, 1, 128, 128, True), (2, 1, 4, 4, False), (3, 3, 36, 20, False), (2, 2, 100, 260, True)])
@pytest.mark.parametrize("pace", [0.01, 1.0, 60.0])
def test_delta_rule_in_chunks(H, Hk, K, P, per_head, pace, monkeypatch):
    """Sequences at the edges of the chunks of 64 and their sub-blocks of 16, from a state, with slow, usual and immediate
    decays; the scan gives the same; slots of others stay as they are."""
    torch.manual_seed(H + K + P)
    monkeypatch.setattr(ops, "DELTA_CHUNKED_FROM", 2)      # all but the shortest
    lens, slots = [1, 15, 16, 17, 63, 64, 65, 200], [4, 2, 7, 1, 5, 3, 8, 9]
    T, n_decay = sum(lens), H if per_head else H * K
    step = Steps(lens, slots)
    C = 2 * Hk * K + H * P
    qkv, b_raw, a_raw = torch.randn(T, C, device=DEV), torch.randn(T, H + 3, device=DEV), torch.randn(T, n_decay + (5 if per_head else 0), device=DEV)
    bias, a_log = torch.randn(n_decay, device=DEV), torch.log(pace * (1 + torch.rand(H, device=DEV)))
    start = 0.3 * torch.randn(11, H, P, K, device=DEV)
    col, scale = 2 if per_head else 0, K ** -0.5

    def run(state, **kw):
        return ops.delta_rule(qkv.clone(), b_raw, 1, a_raw, bias, a_log, state, step, H, Hk, K, P, 1e-6, scale, per_head=per_head, a_col0=col, **kw)

    state, again = start.clone(), start.clone()
    o = run(state)
    step.max_new = 1                                        # taken for a short step: the scan
    o_scan = run(again)
    t = 0
    for n, slot in zip(lens, slots):
        S = start[slot].double()
        ref = torch.empty(n, H * P, dtype=F64, device=DEV)
        for i in range(n):
            row = qkv[t + i].double()
            q, k = (x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6) for x in (row[m * Hk * K:(m + 1) * Hk * K].view(Hk, K).repeat_interleave(H // Hk, 0) for m in (0, 1)))
            raw = torch.nn.functional.softplus(a_raw[t + i, col:col + n_decay].double() + bias.double(), threshold=100.0).view(H, -1)
            S = S * torch.exp(-torch.exp(a_log.double())[:, None] * raw)[:, None, :]
            u = torch.sigmoid(b_raw[t + i, 1:1 + H].double())[:, None] * (row[2 * Hk * K:].view(H, P) - (S @ k[:, :, None])[..., 0])
            S = S + u[:, :, None] * k[:, None, :]
            ref[i] = (S @ (q * scale)[:, :, None]).reshape(-1)
        for got, st in ((o, state), (o_scan, again)):
            sums_close(got[t:t + n], ref)
            sums_close(st[slot], S)
        t += n
    assert torch.equal(state[[0, 6, 10]], start[[0, 6, 10]])
    step.max_new, before = max(lens), state.clone()
    run(state, write_state=False)
    assert torch.equal(state, before)


def test_mamba2_adds_a_token_s_own_value_with_one_rounding():
    """Outputs that are D x but for little: the sum's error is that of the multiply-add, 2^-25 to 2^-24 of it, 2.9e-8 on average (a third of
    2^-24 squared, over the numbers between two powers of two); what is given back for the tensor cores' cuts must not reach it."""
    torch.manual_seed(8)
    H, P, N, G, T = 4, 64, 128, 2, 300
    xbc, dt = torch.randn(T, H * P + 2 * G * N, device=DEV), torch.randn(T, H, device=DEV) - 12.0
    d, zero, state = 1.0 + torch.rand(H, device=DEV), torch.zeros(H, device=DEV), torch.zeros(1, H, P, N, device=DEV)
    step, x, S, ref = Steps([T], [0]), xbc[:, :H * P].double().view(T, H, P), torch.zeros(H, P, N, dtype=F64, device=DEV), torch.empty(T, H, P, dtype=F64, device=DEV)
    y = ops.ssm_scan(xbc, dt, 0, zero, zero, d, state, step, H, P, N, G).view(T, H, P)
    for i in range(T):
        b, c = (xbc[i, H * P + k * G * N:H * P + (k + 1) * G * N].double().view(G, N).repeat_interleave(H // G, 0) for k in (0, 1))
        s = torch.nn.functional.softplus(dt[i].double())
        S = torch.exp(-s)[:, None, None] * S + (s[:, None] * x[i])[:, :, None] * b[:, None, :]
        ref[i] = (S @ c[:, :, None])[..., 0] + d.double()[:, None] * x[i]
    assert (y.double() - ref).norm() <= 2.9e-8 * ref.norm()


@pytest.mark.parametrize("kind", ["mamba2", "mlstm", "delta", "delta_per_head"])
@pytest.mark.parametrize("where", ["value", "key", "query"])
@pytest.mark.parametrize("number", [math.inf, -math.inf, math.nan, 3.4e38])
def test_chunks_keep_what_is_not_finite_to_those_who_see_it(kind, where, number, monkeypatch):
    """One number of a token that is not finite, or nearly so, in a sequence of positive ones.  Tokens before it, other sequences and
    other heads hold what they held without it (the same bits, but in its own chunk and head, whose sums are formed in another way);
    it and those after it hold the infinity that a sum of products gives, or the finite sum."""
    delta = kind.startswith("delta")
    if delta and (where != "value" or number == 3.4e38):
        pytest.skip("unit keys and queries; the bound of a value's product is not of this form")
    torch.manual_seed(5)
    H, K, P, slots = 4, 68, 72, [1, 0, 2]
    lens, at, head, column = [130, 300, 40], 70, 2, 37
    T, hit, tiny = sum(lens), lens[0] + 128 + at, 1e-4
    chunk, step = lens[0] + 128 + (64 if delta else 0), Steps(lens, slots)              # where its chunk begins
    if kind == "mamba2":
        monkeypatch.setattr(ops, "SSM_CHUNKED_FROM", 2)
        G, inner = 2, H * P
        rows, dt = 0.1 + torch.rand(T, inner + 2 * G * K, device=DEV), torch.randn(T, H, device=DEV) - 10.0
        rows[:, inner:] *= tiny
        bias, a_log, d, start = torch.zeros(H, device=DEV), torch.zeros(H, device=DEV), tiny * torch.rand(H, device=DEV), tiny * torch.rand(3, H, P, K, device=DEV)
        place = {"value": head * P + column, "key": inner + head // 2 * K + 5, "query": inner + (G + head // 2) * K + 5}[where]
        heads = [head] if where == "value" else [2, 3]
        run = lambda x, state: (ops.ssm_scan(x, dt, 0, bias, a_log, d, state, step, H, P, K, G),)
    elif kind == "mlstm":
        monkeypatch.setattr(ops, "mlstm_tiles_pay", lambda *sizes: True)
        n_qkv = H * (2 * K + P)
        rows = 0.1 + torch.rand(T, -(-(n_qkv + 2 * H) // 4) * 4, device=DEV)
        rows[:, :2 * H * K] *= tiny
        rows[:, n_qkv + H:n_qkv + 2 * H] += 5.0
        zero, start = torch.zeros(H, device=DEV), tiny * torch.rand(3, H, P + 1, K, device=DEV)
        place = {"value": 2 * H * K + head * P + column, "key": (H + head) * K + 5, "query": head * K + 5}[where]
        heads = [head]
        run = lambda x, state: ops.mlstm_scan(x, n_qkv, n_qkv + H, zero, zero, 15.0, state, torch.zeros(3, H, P + 1, device=DEV), step, H, K, P, K ** -0.5, 1e-6)
    else:
        monkeypatch.setattr(ops, "DELTA_CHUNKED_FROM", 2)
        per_head = kind == "delta_per_head"
        n_decay = H if per_head else H * K
        rows = 0.1 + torch.rand(T, 2 * H * K + H * P, device=DEV)
        b_raw, a_raw, bias, a_log, start = torch.zeros(T, H, device=DEV), torch.randn(T, n_decay, device=DEV) - 3.0, torch.zeros(n_decay, device=DEV), torch.zeros(H, device=DEV), torch.rand(3, H, P, K, device=DEV)
        place, heads = 2 * H * K + head * P + column, [head]
        run = lambda x, state: (ops.delta_rule(x.clone(), b_raw, 0, a_raw, bias, a_log, state, step, H, H, K, P, 1e-6, K ** -0.5, per_head=per_head),)
    results = []
    for plant in (False, True, "scan"):
        x, state = rows.clone(), start.clone()
        if plant:
            x[hit, place] = number
        step.max_new = max(lens) if plant != "scan" else 1
        y = run(x, state)[0] if kind != "mlstm" or plant != "scan" else None
        results.append((None if y is None else y.view(T, H, P), state))
    (clean, clean_state), (got, state), (scan, _) = results
    mine = torch.zeros(H, dtype=torch.bool, device=DEV)
    mine[heads] = True
    before, after = slice(0, hit), slice(hit, lens[0] + lens[1])
    assert torch.equal(got[:, ~mine], clean[:, ~mine]) and torch.equal(state[[1, 2]], clean_state[[1, 2]]) and torch.equal(state[0][~mine], clean_state[0][~mine])
    assert torch.equal(got[:chunk], clean[:chunk]) and torch.equal(got[after.stop:], clean[after.stop:])
    assert ((got[before] - clean[before]).abs() <= 2.0 ** -19 * clean[before].abs()).all()
    seen = got[after][:, mine]
    if where == "value":
        other = torch.arange(P, device=DEV) != column
        assert ((seen[..., other] - clean[after][:, mine][..., other]).abs() <= 2.0 ** -19 * clean[after][:, mine][..., other].abs()).all()
        seen = seen[..., column]
    if where == "query":
        behind = got[hit + 1:after.stop]
        assert ((behind - clean[hit + 1:after.stop]).abs() <= 2.0 ** -19 * clean[hit + 1:after.stop].abs()).all() and torch.equal(state, clean_state)
        seen = seen[:1]
    if number == 3.4e38:
        assert torch.isfinite(seen).all() and (seen > 1e25).all()
        if scan is not None:
            want = scan[after][:, mine]
            want = want[..., column] if where == "value" else want[:1] if where == "query" else want
            # up to 300 tokens of the scan, each of which rounds its decay and the state: 600 half units of the last place
            assert ((seen - want).abs() <= 600 * 2.0 ** -25 * want.abs()).all()
    elif math.isnan(number):
        assert torch.isnan(seen).all()
    elif delta:
        assert (seen[0] == number).all() and not torch.isfinite(seen).any()
    else:
        assert (seen == number).all()
    ops.gemm_tc_check(DEV)


@pytest.mark.parametrize("per_head", [False, True])
@pytest.mark.parametrize("rate, forget", [(16.0, 10.0), (1.0, 1000.0), (1.0, 1e5), (2.0, math.inf)])
def test_delta_rule_in_chunks_with_tokens_that_forget(per_head, rate, forget):
    """Tokens that clear most of the memory among tokens that keep it.  The scan multiplies by a token's own decay, an error of a
    rounding or two a token whatever came before; the chunks' error is of that size."""
    torch.manual_seed(int(rate))
    H, Hk, K, P, T = 2, 2, 128, 64, 400
    n_decay, C, col = H if per_head else H * K, 2 * Hk * K + H * P, 3 if per_head else 0
    step = Steps([T], [1])
    qkv, b_raw, a_raw = torch.randn(T, C, device=DEV), torch.randn(T, H, device=DEV), torch.randn(T, n_decay + col, device=DEV) - 8.0
    bias, a_log = torch.zeros(n_decay, device=DEV), torch.full((H,), math.log(rate), device=DEV)
    if per_head:
        a_raw[3::8, col:] = forget
    else:
        a_raw[3::8, torch.rand(n_decay, device=DEV) < 0.7] = forget
    start = 0.3 * torch.randn(2, H, P, K, device=DEV)
    S, ref = start[1].double(), torch.empty(T, H * P, dtype=F64, device=DEV)
    for i in range(T):
        row = qkv[i].double()
        q, k = (x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6) for x in (row[m * Hk * K:(m + 1) * Hk * K].view(Hk, K).repeat_interleave(H // Hk, 0) for m in (0, 1)))
        raw = torch.nn.functional.softplus(a_raw[i, col:].double(), threshold=100.0).view(H, -1)
        S = S * torch.exp(-torch.exp(a_log.double())[:, None] * raw)[:, None, :]
        u = torch.sigmoid(b_raw[i].double())[:, None] * (row[2 * Hk * K:].view(H, P) - (S @ k[:, :, None])[..., 0])
        S = S + u[:, :, None] * k[:, None, :]
        ref[i] = (S @ (q * K ** -0.5)[:, :, None]).reshape(-1)
    errors = []
    for longest in (T, 1):                                  # the chunks, the scan
        step.max_new, state = longest, start.clone()
        o = ops.delta_rule(qkv.clone(), b_raw, 0, a_raw, bias, a_log, state, step, H, Hk, K, P, 1e-6, K ** -0.5, per_head=per_head, a_col0=col)
        assert torch.isfinite(o).all() and torch.isfinite(state).all()
        errors.append([float((got.double() - want).norm() / want.norm()) for got, want in ((o, ref), (state[1], S))])
    for chunks, scan in zip(*errors):
        assert chunks <= 2 * scan + 2.0 ** -23, errors


@pytest.mark.parametrize("kind", ["mamba2", "delta", "delta_per_head"])
@pytest.mark.parametrize("lens", [[200, 1, 1, 1], [1] * 40 + [96, 1, 144, 143, 95, 2, 500] + [1] * 30, [300, 96, 144, 600], [90, 1, 30]])
def test_recurrences_do_not_look_at_the_rest_of_the_batch(kind, lens):
    """Whether a sequence goes through the scan or through chunks follows from its own length: its outputs and its state are the same
    bits alone and beside others, short and long."""
    torch.manual_seed(len(lens))
    H, P, K, G, T, B = 4, 64, 64, 2, sum(lens), len(lens)
    inner, n_decay = H * P, H if kind == "delta_per_head" else H * K
    xbc, side, a_raw = torch.randn(T, inner + 2 * G * K, device=DEV), torch.randn(T, H, device=DEV), torch.randn(T, n_decay, device=DEV) - 3.0
    qkv, vec, bias = torch.randn(T, 2 * H * K + inner, device=DEV), torch.randn(H, device=DEV), torch.randn(n_decay, device=DEV)
    start = 0.3 * torch.randn(B, H, P, K, device=DEV)

    def run(picked, rows_, slots):
        step, state = Steps(picked, slots), start.clone()
        step.min_new = min(picked)
        if kind == "mamba2":
            out = ops.ssm_scan(xbc[rows_].contiguous(), side[rows_].contiguous(), 0, vec, vec, vec, state, step, H, P, K, G)
        else:
            out = ops.delta_rule(qkv[rows_].clone(), side[rows_].contiguous(), 0, a_raw[rows_].contiguous(), bias, vec, state, step, H, H, K, P, 1e-6, K ** -0.5,
                                 per_head=kind == "delta_per_head")
        return out, state

    out, state = run(lens, slice(0, T), list(range(B)))
    seen, at = set(), 0
    for b, n in enumerate(lens):
        if n not in seen:
            alone, after = run([n], slice(at, at + n), [b])
            assert torch.equal(out[at:at + n], alone) and torch.equal(state[b], after[b]), n
        seen.add(n)
        at += n


@pytest.mark.parametrize("kind", ["mamba2", "delta", "mixed"])
def test_recurrences_without_memory_for_chunks(kind):
    """Where the scratch memory of the chunks cannot be had, a prompt goes through the scan, as it would without them."""
    torch.manual_seed(5)
    H, P, K, G, lens = 16, 64, 256 if kind == "mamba2" else 64, 2, [3000, 1] if kind == "mixed" else [3000]
    T, B = sum(lens), len(lens)
    step = Steps(lens, list(range(B)))
    xbc, side, a_raw = torch.randn(T, H * P + 2 * G * K, device=DEV), torch.randn(T, H, device=DEV), torch.randn(T, H * K, device=DEV) - 3.0
    qkv, vec, bias = torch.randn(T, 2 * H * K + H * P, device=DEV), torch.randn(H, device=DEV), torch.randn(H * K, device=DEV)
    start = 0.3 * torch.randn(B, H, P, K, device=DEV)

    def run(x, state):
        if kind == "mamba2":
            return ops.ssm_scan(x, side, 0, vec, vec, vec, state, step, H, P, K, G)
        return ops.delta_rule(x, side, 0, a_raw, bias, vec, state, step, H, H, K, P, 1e-6, K ** -0.5)

    inputs = xbc if kind == "mamba2" else qkv
    states, xs, outs = [start.clone() for _ in range(3)], [inputs.clone() for _ in range(3)], []
    outs.append(run(xs[0], states[0]))                      # with chunks
    step.max_new = 1                                        # the scan
    outs.append(run(xs[1], states[1]))
    step.max_new, total = max(lens), torch.cuda.get_device_properties(DEV).total_memory
    torch.cuda.empty_cache()
    room = torch.cuda.memory_reserved() + (16 << 20 if kind == "mamba2" else 32 << 20)      # y, or o and the decays: 12 MB each; the scratch is more
    try:
        torch.cuda.set_per_process_memory_fraction(room / total, DEV)
        outs.append(run(xs[2], states[2]))
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0, DEV)
    assert torch.equal(outs[1], outs[2]) and torch.equal(states[1], states[2])
    sums_close(outs[0], outs[1].double())


# ----------------------------------------------------------------------------- score maps, single tokens
@pytest.mark.parametrize("maps, H, G, dim, vdim", [(2, 16, 4, 64, 128), (2, 2, 2, 8, 8), (2, 15, 3, 40, 72), (1, 10, 1, 128, 128), (2, 4, 1, 128, 120), (1, 3, 3, 24, 16)])
@pytest.mark.parametrize("softcap, window, chunk, gated", [(0.0, 0, 0, False), (5.0, 0, 0, True), (3.0, 100, 0, False), (2.0, 1, 0, True), (20.0, 0, 96, False)])
def test_score_maps_of_single_tokens_on_the_tensor_cores(maps, H, G, dim, vdim, softcap, window, chunk, gated):
    """Scores are exact products, probabilities 32-bit, so what is left is the rounding of the bfloat16 results (and of sums of
    32-bit products, which the norm of a small difference enlarges)."""
    if maps == 1 and not softcap and not gated and not chunk:
        pytest.skip("plain grouped-query attention: its own kernel")
    torch.manual_seed(H + dim + window + chunk)
    lens = [1, 15, 16, 17, 63, 64, 65, 130, 1000, 2049, 4500]
    B = len(lens)
    table, (k_pool, v_pool) = paged(lens, lambda s: torch.randn(s, device=DEV).to(BF), [(G, maps * dim), (G, vdim)])
    q = (2.0 * torch.randn(B, H, maps * dim, device=DEV)).to(BF)
    gate = torch.randn(B, H + 3, device=DEV) if gated else None
    alone = []
    for pick in (list(range(B)), [1], [9], [10]):
        ctx = SimpleNamespace(single_token=True, n_seqs=len(pick), max_new=1, max_len=max(lens[b] for b in pick),
                              seq_len=torch.tensor([lens[b] for b in pick], device=DEV).int())
        out = ops.maps_attention(q[pick].contiguous(), k_pool, v_pool, table[pick].contiguous(), ctx, maps, dim ** -0.5, softcap=softcap, window=window,
                                 chunk=chunk, lam=0.4, norm_out=maps == 2, eps=1e-5, out_scale=0.3, gate=None if gate is None else gate[pick].contiguous(),
                                 gate_col0=2 if gated else 0).view(len(pick), H, vdim)
        alone.append(out)
        for i, b in enumerate(pick):
            n = lens[b]
            ks, vs = rows(k_pool, table[b], n), rows(v_pool, table[b], n)
            c = (n - 1) // chunk * chunk if chunk else 0
            pos = torch.tensor([n - 1 - c], device=DEV)
            for h in range(H):
                g = h // (H // G)
                a = [softmax(q[b, h:h + 1, m * dim:(m + 1) * dim].double(), ks[g, c:, m * dim:(m + 1) * dim], vs[g, c:], dim ** -0.5, pos, window, softcap)[0] for m in range(maps)]
                ref, grown = a[0], 1.0
                if maps == 2:
                    ref = a[0] - 0.4 * a[1]
                    grown = 0.3 * float(ref.square().mean().add(1e-5).rsqrt())
                    ref = ref * grown
                if gated:
                    ref = ref * torch.sigmoid(gate[b, h + 2].double())
                err = (out[i, h].double() - ref).abs()
                assert (err <= 2.0 ** -8 * ref.abs() + 2e-5 * max(1.0, grown)).all(), (n, h, err.max())
    for i, b in enumerate([1, 9, 10]):                      # a sequence's result does not depend on the batch
        assert torch.equal(alone[0][b], alone[i + 1][0])


@pytest.mark.parametrize("maps, H, G, dim, vdim", [(2, 16, 4, 64, 128), (2, 6, 3, 40, 72)])
def test_score_maps_of_single_tokens_from_any_address(maps, H, G, dim, vdim):
    """Queries that do not lie at a multiple of 16 bytes take the form that reads them one by one, with runs of its own."""
    torch.manual_seed(H + dim)
    lens = [1, 65, 300, 6000]
    table, (k_pool, v_pool) = paged(lens, lambda s: torch.randn(s, device=DEV).to(BF), [(G, maps * dim), (G, vdim)])
    q = torch.randn(len(lens), H, maps * dim, device=DEV).to(BF)
    flat = torch.empty(q.numel() + 1, dtype=BF, device=DEV)
    shifted = flat[1:].view(q.shape)
    shifted.copy_(q)
    ctx = SimpleNamespace(single_token=True, n_seqs=len(lens), max_new=1, max_len=max(lens), seq_len=torch.tensor(lens, device=DEV).int())
    a, b = (ops.maps_attention(x, k_pool, v_pool, table, ctx, maps, dim ** -0.5, lam=0.4) for x in (q, shifted))
    assert ((a.double() - b.double()).abs() <= 2.0 ** -7 * a.double().abs() + 2e-5).all()      # two roundings of nearly the same numbers


# ----------------------------------------------------------------------------- experts
@pytest.mark.parametrize("T, E, top, D, F, Fs, activation", [(1, 3, 1, 8, 8, 0, "relu2"), (7, 64, 6, 264, 40, 72, "gelu"), (9, 5, 5, 72, 24, 16, "silu"), (17, 130, 8, 2048, 136, 0, "gated_silu"),
                                                            (40, 2, 1, 136, 264, 520, "relu2"), (33, 4, 2, 40, 8, 0, "gated_silu"), (140, 6, 16 // 4, 64, 72, 8, "relu2"), (600, 9, 4, 24, 16, 40, "silu")])
@pytest.mark.parametrize("on_input", [False, True])
def test_experts_read_once_for_all_their_tokens(T, E, top, D, F, Fs, activation, on_input, monkeypatch):
    """Experts with no token, one eight, more than four eights and all tokens; rows, features and contractions that end inside a tile; a
    shared expert with a gate; more tokens than a launch takes.  The form that reads the weights for each copy gives the same."""
    torch.manual_seed(T + E + F)
    gated, r16 = activation == "gated_silu", lambda x: x.to(torch.bfloat16).double()
    x, up, down = (torch.randn(*s, device=DEV).mul(f).to(torch.bfloat16) for s, f in (((T, D), 1.0), ((E, (2 if gated else 1) * F, D), D ** -0.5), ((E, D, F), F ** -0.5)))
    su, sd, gate = (None, None, None) if not Fs else (torch.randn(Fs, D, device=DEV).mul(D ** -0.5).to(torch.bfloat16), torch.randn(D, Fs, device=DEV).mul(Fs ** -0.5).to(torch.bfloat16), torch.rand(T, device=DEV))
    logits = torch.randn(T, E, device=DEV)
    logits[:, 0] += 3.0                                     # most tokens choose the first one, few the last
    logits[:, -1] -= 3.0 * (E > top)
    chosen, weight = ops.moe_route(logits, top)
    act = {"relu2": lambda z: torch.relu(z).square(), "gelu": lambda z: torch.nn.functional.gelu(z, approximate="tanh"), "silu": torch.nn.functional.silu}
    ref = torch.zeros(T, D, dtype=F64, device=DEV)
    for k in range(top):
        w = weight[:, k].double()[:, None]
        z = torch.einsum("tfd,td->tf", up[chosen[:, k].long()].double(), x.double()) * (w if on_input else 1.0)
        a = torch.nn.functional.silu(z[:, :F]) * z[:, F:] if gated else act[activation](z)
        ref += torch.einsum("tdf,tf->td", down[chosen[:, k].long()].double(), r16(a)) * (1.0 if on_input else w)
    if Fs:
        ref += gate.double()[:, None] * (r16(act[activation](x.double() @ su.double().T)) @ sd.double().T)
    base = torch.randn(T, D, device=DEV)
    for least in (1, 10 ** 6):                              # every step in that form; none that brings fewer choices than experts
        monkeypatch.setattr(ops, "MOE_STREAM_MIN_TOKENS", least)
        if least > 1:
            monkeypatch.setattr(ops, "moe_stream_fits", lambda *sizes: False)
        for out in (None, base.clone()):
            got = ops.moe_experts(x, up, down, chosen, weight, activation, su, sd, gate, out=out, weight_on_input=on_input)
            want = ref + base.double() if out is not None else ref
            # an activation that lies at the border of two bfloat16 numbers may be rounded the other way: 2^-8 of one of F terms
            assert torch.isfinite(got).all() and (got.double() - want).norm() <= 2 ** -9 * ref.norm() and (got.double() - want).abs().max() <= 2 ** -6 * (1 + ref.abs().max())


@pytest.mark.parametrize("T, E", [(3, 1025), (17, 1024), (17, 1025), (40, 1500)])
def test_any_number_of_experts(T, E):
    """More experts than the lists of the form that reads them once hold: the rows for each copy."""
    torch.manual_seed(E + T)
    D, F, top = 16, 8, 2
    x, up, down = (torch.randn(*s, device=DEV).to(torch.bfloat16) for s in ((T, D), (E, F, D), (E, D, F)))
    chosen, weight = torch.randint(0, E, (T, top), device=DEV).int(), torch.rand(T, top, device=DEV)
    chosen[-1, 0] = E - 1
    got = ops.moe_experts(x, up, down, chosen, weight, "relu2")
    z = torch.relu(torch.einsum("tkfd,td->tkf", up[chosen.long()].double(), x.double())).square().to(torch.bfloat16).double()
    want = torch.einsum("tkdf,tkf,tk->td", down[chosen.long()].double(), z, weight.double())
    assert (got.double() - want).norm() <= 2 ** -9 * want.norm()         # an activation at the border of two bfloat16 numbers: 2^-8 of one of F terms
    with pytest.raises(ops.KernelError):
        ops.moe_experts(x, up, down, chosen[:, :0].contiguous(), weight[:, :0].contiguous(), "relu2")


@pytest.mark.parametrize("dtype, classes", [(torch.float32, [(1, 2, 3, 8, 40)]), (torch.bfloat16, [(1, 2, 3, 5, 7), (8, 9, 24, 130, 500)])])
@pytest.mark.parametrize("Fs", [0, 24, 72, 136])
@pytest.mark.parametrize("skew", [0.0, 3.0, 1e3])
def test_a_token_s_experts_are_the_same_bits_beside_others(dtype, classes, Fs, skew):
    """Within a form (the rows for each copy; an expert's rows once for all of its tokens) a token's sums have one order, whatever the
    number of tokens and whoever else chose its experts: most of them the same ones, or all, in many slots an expert."""
    torch.manual_seed(Fs)
    E, top, D, F = 64, 6, 264, 40
    x, up, down = (torch.randn(*s, device=DEV).mul(f).to(dtype) for s, f in (((500, D), 1.0), ((E, F, D), D ** -0.5), ((E, D, F), F ** -0.5)))
    su, sd = (torch.randn(Fs, D, device=DEV).mul(D ** -0.5).to(dtype), torch.randn(D, Fs, device=DEV).mul(Fs ** -0.5).to(dtype)) if Fs else (None, None)
    logits = torch.randn(500, E, device=DEV)
    logits[:, 5:5 + top] += skew
    chosen, weight = ops.moe_route(logits, top)
    gate = torch.rand(500, device=DEV) if Fs else None
    for sizes in classes:
        outs = [ops.moe_experts(x[:n], up, down, chosen[:n], weight[:n], "relu2", su, sd, gate[:n] if Fs else None) for n in sizes]
        for small, large in zip(outs, outs[1:]):
            assert torch.equal(small, large[:len(small)])
