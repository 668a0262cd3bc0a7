"""Attention without a softmax in registers (attention_quads.cu) against float64: every instance, groups of fewer than four
query heads, several sequences with pasts, key ranges, rows at the edges of blocks, tiles and pages."""
from types import SimpleNamespace

import pytest
import torch

from burn_lm_b200 import kernels as K

pytestmark = pytest.mark.gpu

SHAPES = [(32, 8, 64, 64), (24, 8, 64, 128), (16, 8, 128, 64), (32, 8, 128, 128), (8, 8, 64, 64), (20, 5, 48, 72), (6, 2, 16, 8),
          (12, 3, 112, 128), (32, 8, 48, 64)]
STEPS = [([33, 1, 16, 70], [0, 100, 63, 129], 1), ([300], [700], 3), ([1, 1, 1], [0, 63, 1090], 1), ([1], [1500], 5), ([2], [64], 1),
         ([1, 0, 1], [15, 9, 640], 4)]


@pytest.mark.parametrize("lens,starts,ranges", STEPS)
@pytest.mark.parametrize("H,G,dk,dv", SHAPES)
def test_weights_mix_and_values(H, G, dk, dv, lens, starts, ranges):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(H * 1000 + dk + sum(lens))
    rnd = lambda *shape: torch.randn(shape, generator=gen, device="cuda")
    assert K.sigmoid_attention_in_registers(torch.bfloat16, H, G, dk, dv)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    n, each = cu[-1], max(-(-(a + b) // K.PAGE) for a, b in zip(lens, starts))
    pages = torch.randperm(each * len(lens) + 1, generator=torch.Generator().manual_seed(1))[: each * len(lens)].to(torch.int32)
    table = pages.reshape(len(lens), each).cuda()
    pool = torch.full((each * len(lens) + 1, G * K.PAGE * (dk + dv)), float("nan"), dtype=torch.bfloat16, device="cuda")
    step = SimpleNamespace(n_tokens=n + 3, n_seqs=len(lens), max_q_len=max(lens), max_kv_len=each * K.PAGE, cu_seqlens=i32(cu),
                           token_seq=i32([s for s, m in enumerate(lens) for _ in range(m)] + [-1] * 3),
                           slot_of_seq=i32(list(range(len(lens)))), start_pos=i32(starts))
    q = rnd(n + 3, H * dk).bfloat16()
    talk, bias, scale, cap = rnd(H, H) * H ** -0.5, rnd(H) - 1, 2.0 * dk ** -0.5, 6.0
    keys, values = [], []
    for s, (m, start) in enumerate(zip(lens, starts)):
        total = start + m
        keys.append(rnd(total, G, dk).bfloat16())
        values.append(rnd(total, G, dv).bfloat16())
        for j in range(0, total, K.PAGE):
            page, rows = pool[int(table[s, j // K.PAGE])], min(K.PAGE, total - j)
            page[: G * K.PAGE * dk].view(G, K.PAGE, dk)[:, :rows] = keys[-1][j:j + rows].transpose(0, 1)
            page[G * K.PAGE * dk:].view(G, K.PAGE, dv)[:, :rows] = values[-1][j:j + rows].transpose(0, 1)
    for cut, mixed in ((cap, talk), (0.0, None)):
        out = torch.zeros((n + 3, H * dv), dtype=torch.bfloat16, device="cuda")
        partial = torch.full((ranges * (n + 3) * H * dv,), float("nan"), device="cuda") if ranges > 1 else None
        K.sigmoid_attention(q, pool, table, step, out, H, G, dk, dv, scale, softcap=cut, talk=mixed, head_bias=bias, ranges=ranges,
                            partial=partial)
        for s, (m, start) in enumerate(zip(lens, starts)):
            if m == 0:
                continue
            sl = slice(cu[s], cu[s + 1])
            sc = torch.einsum("nhd,thd->hnt", q[sl].double().view(m, H, dk), keys[s].double().repeat_interleave(H // G, 1)) * scale
            sc = cut * torch.tanh(sc / cut) if cut else sc
            w = torch.sigmoid(sc + bias.double()[:, None, None])
            w = w * (torch.arange(start + m, device="cuda")[None] <= start + torch.arange(m, device="cuda")[:, None])
            terms = torch.einsum("hg,gnt->hnt", mixed.double().abs(), w) if mixed is not None else w
            w = torch.einsum("hg,gnt->hnt", mixed.double(), w) if mixed is not None else w
            v = values[s].double().repeat_interleave(H // G, 1)
            want = torch.einsum("hnt,thd->nhd", w, v)
            # mixed weights and outputs are rounded to bfloat16 once each (2^-8 of either); a weight carries the errors of two
            # exponentials and quotients of fp32 scores of up to 30 (2^-17 of the terms it is mixed from, which may cancel)
            room = 2.0 ** -7 * torch.einsum("hnt,thd->nhd", w.abs(), v.abs()) + 2.0 ** -17 * torch.einsum("hnt,thd->nhd", terms, v.abs())
            assert ((out[sl].double().view(m, H, dv) - want).abs() <= room).all()
        assert not out[n:].any()


@pytest.mark.parametrize("lens", [[1], [2, 1]])                               # the kernel of single tokens, and that of portions
@pytest.mark.parametrize("H,G,dk,dv", [(32, 8, 64, 64), (20, 5, 48, 72), (6, 2, 16, 8)])
def test_the_mix_keeps_every_bit_of_the_weights(H, G, dk, dv, lens):
    """Scores of zero give weights of exactly a half; every head takes two others' weights with factors that differ in their last
    bits, so that what is left of the two is those bits."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(H)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    cu = [0]
    for m in lens:
        cu.append(cu[-1] + m)
    n = cu[-1]
    step = SimpleNamespace(n_tokens=n, n_seqs=len(lens), max_q_len=max(lens), max_kv_len=max(lens), cu_seqlens=i32(cu),
                           token_seq=i32([s for s, m in enumerate(lens) for _ in range(m)]), slot_of_seq=i32(list(range(len(lens)))),
                           start_pos=i32([0] * len(lens)))
    assert K.sigmoid_attention_in_registers(torch.bfloat16, H, G, dk, dv)
    pool = torch.zeros((len(lens), G * K.PAGE * (dk + dv)), dtype=torch.bfloat16, device="cuda")
    pool[:, G * K.PAGE * dk:].view(-1, G, K.PAGE, dv)[:, :, 0] = 1.0          # the first position's values: one
    talk = torch.zeros((H, H), device="cuda")
    for h in range(H):
        a, b = torch.randperm(H, generator=torch.Generator().manual_seed(h))[:2].tolist()
        bits = int(torch.randint(1 << 23, (1,), generator=torch.Generator().manual_seed(h + 100)))
        talk[h, a] = (1 << 23 | bits) * 2.0 ** -23                            # (24 bits, between one and two)
        talk[h, b] = -((1 << 23 | bits) - 1 - h % 7) * 2.0 ** -23
    out = torch.zeros((n, H * dv), dtype=torch.bfloat16, device="cuda")
    K.sigmoid_attention(torch.zeros((n, H * dk), dtype=torch.bfloat16, device="cuda"), pool, i32([[s] for s in range(len(lens))]), step, out,
                        H, G, dk, dv, 1.0, talk=talk)
    want = (talk.double().sum(1) * 0.5)[:, None].expand(H, dv).reshape(-1)     # every position sees the first one's value; the others' are zero
    assert ((out.double() - want).abs() <= 2.0 ** -7 * want.abs()).all()      # (bfloat16 rounds what is left, twice)


@pytest.mark.parametrize("H,G,dk,dv", [(32, 8, 64, 64), (12, 3, 16, 24), (16, 4, 64, 8)])
@pytest.mark.parametrize("lens,starts,ranges", [([15, 16, 17], [0, 0, 0], 1), ([2, 31, 33], [47, 48, 49], 1), ([5], [60], 1),       # four and five tiles
                                                ([18, 1], [1006, 2030], 8), ([400, 0, 9], [113, 7, 1], 2)])
def test_portions_at_the_edges_of_rings_and_blocks(H, G, dk, dv, lens, starts, ranges):
    """Blocks of sixteen rows, a ring of four tiles of sixteen keys (passed several times), a last tile that is full, ragged or all the
    sequence has, fewer lanes than a box of the copies."""
    test_weights_mix_and_values(H, G, dk, dv, lens, starts, ranges)


@pytest.mark.parametrize("most", [1, 20])
def test_several_ranges_write_every_row(most):
    """Where a query's keys are cut into ranges, rows of no sequence come out as zeros whatever lay there."""
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    gen = torch.Generator(device="cuda")
    gen.manual_seed(most)
    n, pages = most + 2, 12
    step = SimpleNamespace(n_tokens=n, n_seqs=1, max_q_len=most, max_kv_len=pages * K.PAGE, cu_seqlens=i32([0, most]),
                           token_seq=i32([0] * most + [-1] * 2), slot_of_seq=i32([0]), start_pos=i32([pages * K.PAGE - most]))
    pool = torch.randn((pages, 8 * K.PAGE * 128), generator=gen, device="cuda").bfloat16()
    q = torch.randn((n, 32 * 64), generator=gen, device="cuda").bfloat16()
    table, outs = i32([list(range(pages))]), []
    for ranges, fill in ((1, 0.0), (3, float("nan"))):
        out = torch.full((n, 32 * 64), fill, dtype=torch.bfloat16, device="cuda")
        partial = torch.full((ranges * n * 32 * 64,), float("nan"), device="cuda")
        K.sigmoid_attention(q, pool, table, step, out, 32, 8, 64, 64, 0.125, ranges=ranges, partial=partial)
        outs.append(out.float())
    assert not outs[1][most:].any()
    # sums of some 800 products of about one in another order (800 * 2^-20 is generous), each rounded once to the eight bits of a
    # bfloat16 number: by up to 2^-8 of it, so that two differ by up to 2^-7 of the larger
    room = 2.0 ** -7 * torch.maximum(outs[0].abs(), outs[1].abs()) + 800 * 2.0 ** -20
    diff = (outs[0] - outs[1]).abs()
    assert (diff <= room).all(), (diff - room).max()
