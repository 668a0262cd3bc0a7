"""The tcgen05 prompt attention with kept first positions and a sink, against float64: windows and kept positions on both sides of
pages and of the rows' own beginnings, portions behind a past, several sequences."""
from types import SimpleNamespace

import pytest
import torch

from burn_lm_b200 import kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,G,dk,dv", [(4, 2, 64, 64), (2, 1, 96, 80), (4, 1, 128, 128), (2, 2, 64, 128), (2, 1, 128, 200)])
@pytest.mark.parametrize("window,keep", [(1, 0), (1, 1), (64, 64), (65, 70), (200, 4), (200, 130), (4000, 3)])
@pytest.mark.parametrize("sink", ["none", "zero", "numbers"])
@pytest.mark.parametrize("lens,starts", [([300], [0]), ([130, 1, 64], [190, 70, 0])])
def test_window_kept_positions_and_sink(H, G, dk, dv, window, keep, sink, lens, starts):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(dk + dv + window + keep)
    rnd = lambda *shape: torch.randn(shape, generator=gen, device="cuda")
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    n, each = cu[-1], max(-(-(a + b) // K.PAGE) for a, b in zip(lens, starts))
    perm = torch.randperm(each * len(lens) + 1, generator=torch.Generator().manual_seed(2))[: each * len(lens)].to(torch.int32)
    table = perm.reshape(len(lens), each).cuda()
    pool = torch.full((each * len(lens) + 1, G * K.PAGE * (dk + dv)), float("nan"), dtype=torch.bfloat16, device="cuda")
    step = SimpleNamespace(n_tokens=n + 2, n_seqs=len(lens), max_q_len=max(lens), max_kv_len=each * K.PAGE, cu_seqlens=i32(cu),
                           token_seq=i32([s for s, m in enumerate(lens) for _ in range(m)] + [-1, -1]),
                           token_pos=i32([a + t for m, a in zip(lens, starts) for t in range(m)] + [0, 0]),
                           slot_of_seq=i32(list(range(len(lens)))), start_pos=i32(starts))
    q, gate, logits = rnd(n + 2, H * dk).bfloat16(), rnd(n + 2, H), 3.0 * rnd(H)
    keys, values = [], []
    for s, (m, start) in enumerate(zip(lens, starts)):
        keys.append(rnd(start + m, G, dk).bfloat16())
        values.append(rnd(start + m, G, dv).bfloat16())
        for j in range(0, start + m, K.PAGE):
            page, rows = pool[int(table[s, j // K.PAGE])], min(K.PAGE, start + m - j)
            page[: G * K.PAGE * dk].view(G, K.PAGE, dk)[:, :rows] = keys[-1][j:j + rows].transpose(0, 1)
            page[G * K.PAGE * dk:].view(G, K.PAGE, dv)[:, :rows] = values[-1][j:j + rows].transpose(0, 1)
    if dk == dv:
        pool = pool.view(-1, 2, G, K.PAGE, dk)
    out = torch.full((n + 2, H * dv), float("nan"), dtype=torch.bfloat16, device="cuda")
    K.attention_sink(q, step, pool, table, out, H, G, dk, dv, dk ** -0.5, window, keep, sink=sink != "none", gate=gate, gate_stride=H,
                     max_q_len=step.max_q_len, sink_logit=logits if sink == "numbers" else None)
    for s, (m, start) in enumerate(zip(lens, starts)):
        sl = slice(cu[s], cu[s + 1])
        sc = torch.einsum("nhd,thd->hnt", q[sl].double().view(m, H, dk), keys[s].double().repeat_interleave(H // G, 1)) * dk ** -0.5
        i, j = start + torch.arange(m, device="cuda")[:, None], torch.arange(start + m, device="cuda")[None]
        sc = torch.where((j <= i) & ((i - j < window) | (j < keep)), sc, -torch.inf)
        if sink != "none":
            extra = logits.double() if sink == "numbers" else torch.zeros(H, dtype=torch.float64, device="cuda")
            p = torch.softmax(torch.cat([sc, extra[:, None, None].expand(H, m, 1)], -1), -1)[..., :-1]
        else:
            p = torch.softmax(sc, -1)
        v, g = values[s].double().repeat_interleave(H // G, 1), torch.sigmoid(gate[sl].double())[:, :, None]
        want = torch.einsum("hnt,thd->nhd", p, v) * g
        # probabilities and outputs are rounded to bfloat16 once each (2^-8 of either)
        room = 2.0 ** -7 * torch.einsum("hnt,thd->nhd", p, v.abs()) * g + 1e-4
        assert ((out[sl].double().view(m, H, dv) - want).abs() <= room).all()
    assert not out[n:].any()                                                  # rows of no sequence hold zeros
    K.check_status(torch.device("cuda"))


@pytest.mark.parametrize("dk,dv", [(64, 64), (128, 128), (64, 200)])
def test_the_largest_probability_is_not_rounded(dk, dv):
    """Rows whose largest score comes late and exceeds what came before by less than 2^8: their probabilities are taken against that
    score itself, so that it enters the sum over the values as exactly one."""
    tops = torch.linspace(0.5, 5.4, 24).bfloat16()
    n_seqs, m, at = len(tops), 256, 200
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    step = SimpleNamespace(n_tokens=n_seqs * m, n_seqs=n_seqs, max_q_len=m, max_kv_len=m, cu_seqlens=i32([m * s for s in range(n_seqs + 1)]),
                           token_seq=i32([s for s in range(n_seqs) for _ in range(m)]), token_pos=i32(list(range(m)) * n_seqs),
                           slot_of_seq=i32(list(range(n_seqs))), start_pos=i32([0] * n_seqs))
    pages = m // K.PAGE
    pool = torch.zeros((n_seqs * pages, K.PAGE * (dk + dv)), dtype=torch.bfloat16, device="cuda")
    of_top = pool.view(n_seqs, pages, -1)[:, at // K.PAGE]                    # the page of the one key that is not zero
    of_top[:, : K.PAGE * dk].view(n_seqs, K.PAGE, dk)[:, at % K.PAGE, 0] = tops.cuda()
    of_top[:, K.PAGE * dk:].view(n_seqs, K.PAGE, dv)[:, at % K.PAGE] = 1.0     # ... nor its values
    if dk == dv:
        pool = pool.view(-1, 2, 1, K.PAGE, dk)
    q = torch.zeros((n_seqs * m, dk), dtype=torch.bfloat16, device="cuda")
    q[:, 0] = 1.0
    out = torch.zeros((n_seqs * m, dv), dtype=torch.bfloat16, device="cuda")
    K.attention_sink(q, step, pool, i32(list(range(n_seqs * pages))).view(n_seqs, pages), out, 1, 1, dk, dv, 1.0, 4000, 3, sink=True,
                     max_q_len=m)
    e = torch.exp(tops.double().cuda())[:, None]
    others = torch.arange(at, m, device="cuda", dtype=torch.float64)[None] + 1.0      # the keys before and after it, and the sink: exp(0) each
    want = (e / (e + others))[:, :, None]
    got = out.double().view(n_seqs, m, dv)
    assert not got[:, :at].any()
    # half a place of a bfloat16 output, and 2^-14 for the fp32 sums of some two hundred exponentials
    assert ((got[:, at:] - want).abs() <= 2.0 ** (torch.floor(torch.log2(want)) - 8) + 2.0 ** -14 * want).all()
    K.check_status(torch.device("cuda"))
