"""Row kernels that move 16-byte pieces, against float64 and at sizes and alignments on both sides of their rules (the general
kernels serve the others): the norm over groups, the token shift, the rotation and the norm in front of the attentions."""
from types import SimpleNamespace

import pytest
import torch

from burn_lm_b200 import kernels as K

pytestmark = pytest.mark.gpu


def i32(v):
    return torch.tensor(v, dtype=torch.int32, device="cuda")


def rng(seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return lambda *shape: torch.randn(shape, generator=gen, device="cuda")


def step_of(lens, starts, padding=2):
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    seqs, pos = [s for s, n in enumerate(lens) for _ in range(n)], [a + t for n, a in zip(lens, starts) for t in range(n)]
    return SimpleNamespace(cu_seqlens=i32(cu), slot_of_seq=i32([len(lens) - s for s in range(len(lens))]), start_pos=i32(starts),
                           token_seq=i32(seqs + [-1] * padding), token_pos=i32(pos + [0] * padding), n_tokens=cu[-1] + padding,
                           n_seqs=len(lens), max_q_len=max(lens))


def close(got, want, dtype):
    # one rounding to the result's type on top of a few units of 2^-23 of the row's largest value
    unit = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -21
    return ((got.double() - want).abs() <= unit * want.abs() + 2.0 ** -19 * want.abs().amax(-1, keepdim=True)).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("group,n_groups", [(4, 3), (12, 5), (64, 7), (100, 3), (128, 32), (516, 2), (1024, 2), (1028, 1), (6, 4)])
@pytest.mark.parametrize("shared,col0", [(True, 0), (False, 4), (False, 3)])
def test_norm_over_groups(dtype, group, n_groups, shared, col0):
    rnd = rng(group * 10 + n_groups)
    n, c = 37, group * n_groups
    y, wide, w = rnd(n, c), rnd(n, c + 8 + (-c) % 4), rnd(group if shared else c)
    gate = wide[:, col0:col0 + c].double()
    u = y.double()
    unit = lambda t: (t.view(n, n_groups, group) / torch.sqrt((t.view(n, n_groups, group) ** 2).mean(-1, keepdim=True) + 1e-5)).view(n, c)
    ww = w.double().repeat(n_groups) if shared else w.double()
    want = {K.GATE_FIRST: unit(u * gate * torch.sigmoid(gate)) * ww, K.GATE_LAST: unit(u) * ww * torch.sigmoid(gate),
            K.GATE_SILU_LAST: unit(u) * ww * gate * torch.sigmoid(gate), K.GATE_NONE: unit(u) * ww}
    for mode, expected in want.items():
        out = torch.zeros((n, c), dtype=dtype, device="cuda")
        K.gated_group_norm(y, None if mode == K.GATE_NONE else wide, col0, w, group, mode, 1e-5, out)
        assert close(out, expected, dtype), mode


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("channels", [4, 132, 516, 33])
@pytest.mark.parametrize("lens,starts", [([33], [0]), ([8, 1, 40, 7], [3, 0, 6, 1]), ([31], [2])])
def test_token_shift(dtype, channels, lens, starts):
    rnd = rng(channels + len(lens))
    st, S = step_of(lens, starts), 3
    n = st.n_tokens
    x, mu, state = rnd(n, channels), rnd(S, channels), rnd(len(lens) + 1, 2, channels + 5)
    before, out = state.clone(), torch.zeros((S, n, channels), dtype=dtype, device="cuda")
    K.shift_mix(x, mu, out, st, state, 5)
    at = 0
    for s, (m, start) in enumerate(zip(lens, starts)):
        slot = len(lens) - s
        carried = before[slot, start & 1, 5:].double() if start else torch.zeros(channels, dtype=torch.float64, device="cuda")
        rows = x[at:at + m].double()
        prev = torch.cat([carried[None], rows[:-1]])
        want = rows[None] + (prev - rows)[None] * mu.double()[:, None]
        assert close(out[:, at:at + m], want, dtype)
        assert torch.equal(state[slot, (start + m) & 1, 5:], x[at + m - 1])
        at += m
    assert not out[:, at:].any()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,G,dk,dv,rot,biased", [(4, 2, 64, 64, 64, True), (3, 3, 24, 20, 8, False), (2, 1, 16, 12, 12, True), (5, 1, 12, 8, 0, True),
                                                  (2, 2, 10, 6, 4, True), (32, 8, 128, 64, 96, True)])
def test_rotation_and_append(dtype, H, G, dk, dv, rot, biased):
    rnd = rng(H * 100 + dk)
    st = step_of([5, 66, 1], [0, 60, 127])
    n, width, half = st.n_tokens, (H + G) * dk + G * dv, rot // 2
    proj, bias = rnd(n, width), rnd(width) if biased else None
    freq = torch.tensor([500.0 ** (-2.0 * i / max(rot, 1)) for i in range(half)], dtype=torch.float64, device="cuda") if rot else None
    table = i32([[0, 1, 2], [3, 4, 5], [6, 7, 8], [9, 10, 11]])
    pool = torch.full((12, G * K.PAGE * (dk + dv)), 7.0, dtype=dtype, device="cuda")
    q = torch.zeros((n, H * dk), dtype=dtype, device="cuda")
    K.bias_rope_append(proj, bias, freq, rot, q, pool, table, st, H, G, dk, dv)
    full = proj.double() + (bias.double() if biased else 0.0)
    heads = full[:, :(H + G) * dk].view(n, H + G, dk).clone()
    if rot:
        ang = st.token_pos.double()[:, None, None] * freq
        a, b = heads[..., :half].clone(), heads[..., half:rot].clone()
        heads[..., :half], heads[..., half:rot] = a * torch.cos(ang) - b * torch.sin(ang), b * torch.cos(ang) + a * torch.sin(ang)
    assert close(q, heads[:, :H].reshape(n, -1), dtype)
    expected = torch.full((12, G * K.PAGE * (dk + dv)), 7.0, dtype=torch.float64, device="cuda")
    keys, values = expected[:, :G * K.PAGE * dk].view(12, G, K.PAGE, dk), expected[:, G * K.PAGE * dk:].view(12, G, K.PAGE, dv)
    for t in range(n - 2):
        pos, slot = int(st.token_pos[t]), int(st.slot_of_seq[int(st.token_seq[t])])
        keys[int(table[slot, pos // K.PAGE]), :, pos % K.PAGE] = heads[t, H:]
        values[int(table[slot, pos // K.PAGE]), :, pos % K.PAGE] = full[t, (H + G) * dk:].view(G, dv)
    assert close(pool, expected, dtype)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,G,dk,dv,blend,left", [(4, 2, 64, 80, True, True), (32, 8, 128, 128, False, False), (64, 16, 128, 64, True, False),
                                                  (3, 1, 12, 20, False, True), (2, 1, 6, 10, True, True), (80, 8, 128, 8, False, False)])
def test_norms_over_whole_projections_and_append(dtype, H, G, dk, dv, blend, left):
    rnd = rng(H + dk)
    st = step_of([3, 65], [1, 62])
    n, width = st.n_tokens, (H + G) * dk + G * dv
    proj, wq, wk, lam, earlier = rnd(n, width + 4), rnd(H * dk), rnd(G * dk), rnd(1), rnd(n, G * dv)
    table = i32([[0, 1], [2, 3], [4, 5]])
    pool = torch.full((6, G * K.PAGE * (dk + dv)), 7.0, dtype=dtype, device="cuda")
    q, kept = torch.zeros((n, H * dk), dtype=dtype, device="cuda"), torch.zeros((n, G * dv), device="cuda") if left else None
    K.qk_norm_append(proj, st, pool, table, q, H, G, dk, dv, q_weight=wq, k_weight=wk, eps=1e-6, blend=lam if blend else None,
                     values_in=earlier if blend else None, values_out=kept)
    x = proj.double()
    unit = lambda t: t / torch.sqrt((t * t).mean(-1, keepdim=True) + 1e-6)
    qs, ks, vs = x[:, :H * dk], x[:, H * dk:(H + G) * dk], x[:, (H + G) * dk:width]
    vs = (1 - lam.double()) * vs + lam.double() * earlier.double() if blend else vs
    assert close(q, unit(qs) * wq.double(), dtype)
    if left:
        assert close(kept, vs, torch.float32)
    expected = torch.full((6, G * K.PAGE * (dk + dv)), 7.0, dtype=torch.float64, device="cuda")
    keys, values = expected[:, :G * K.PAGE * dk].view(6, G, K.PAGE, dk), expected[:, G * K.PAGE * dk:].view(6, G, K.PAGE, dv)
    for t in range(n - 2):
        pos, slot = int(st.token_pos[t]), int(st.slot_of_seq[int(st.token_seq[t])])
        page = int(table[slot, pos // K.PAGE])
        keys[page, :, pos % K.PAGE] = (unit(ks) * wk.double())[t].view(G, dk)
        values[page, :, pos % K.PAGE] = vs[t].view(G, dv)
    assert close(pool, expected, dtype)
