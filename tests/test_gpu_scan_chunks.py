"""The recurrences in chunks of sixteen tokens (scan_chunks.cu) against the walk in float64, at the edges of chunks, of row
and column tiles, through used states, and beside single tokens in one step."""
from types import SimpleNamespace

import pytest
import torch

from burn_lm_b200 import kernels as K

pytestmark = pytest.mark.gpu


def step_of(lens, starts):
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    return SimpleNamespace(cu_seqlens=i32(cu), slot_of_seq=i32([len(lens) + 1 - s for s in range(len(lens))]), start_pos=i32(starts),
                           n_tokens=cu[-1], n_seqs=len(lens), max_q_len=max(lens))


def state_of(step, heads, rows, dv, offset, gen):
    """A state block per slot whose unused rows hold zeros, as the scans leave them; everything else is drawn."""
    floats = K.scan_state_floats(heads, rows, dv)
    slots = step.n_seqs + 2
    state = torch.randn((slots, 2, offset + floats), generator=gen, device="cuda")
    padded = floats // heads // dv
    lanes = state[:, :, offset:].view(slots, 2, heads, padded // 8, dv, 8)
    lanes *= (torch.arange(padded, device="cuda").view(padded // 8, 1, 8) < rows)
    return state


def read_state(state, slot, copy, offset, heads, dv):
    lanes = state[slot, copy, offset:].view(heads, -1, dv, 8)
    return lanes.permute(0, 1, 3, 2).reshape(heads, -1, dv)


def walk(q, k, v, w, beta, bonus, S):
    """float64, token by token: (outputs [T, H, dv], the state behind the last token)."""
    out = []
    for t in range(q.shape[0]):
        if bonus is not None:
            kv = k[t][:, :, None] * v[t][:, None, :]
            out.append(torch.einsum("hrv,hr->hv", S + bonus[:, :, None] * kv, q[t]))
            S = w[t][:, :, None] * S + kv
            continue
        S = w[t][:, :, None] * S
        u = v[t] if beta is None else beta[t][:, None] * (v[t] - torch.einsum("hrv,hr->hv", S, k[t]))
        S = S + k[t][:, :, None] * u[:, None, :]
        out.append(torch.einsum("hrv,hr->hv", S, q[t]))
    return torch.stack(out), S


STEPS = [([33], [0]), ([160, 1, 47], [0, 5, 64]), ([16, 32, 17, 15], [1, 0, 2, 3]), ([513], [7])]
SIZES = [(2, 20, 5), (3, 64, 64), (4, 128, 100), (1, 200, 33), (40, 48, 48)]      # heads, rows, columns: every instance and its edges


@pytest.mark.parametrize("lens,starts", STEPS)
@pytest.mark.parametrize("heads,rows,dv", SIZES)
@pytest.mark.parametrize("kind", ["ssm", "wkv", "lower", "delta"])
def test_chunks_against_the_walk_in_float64(kind, heads, rows, dv, lens, starts):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(heads * 1000 + rows + len(lens))
    rnd = lambda *shape: torch.randn(shape, generator=gen, device="cuda")
    step, n, offset = step_of(lens, starts), sum(lens), 7                    # (an odd offset: the state is not 16-byte aligned)
    assert K._scan_route(K._SCAN_SSM, heads, rows, step, "cuda")[2] == 1      # every sequence in chunks
    state = state_of(step, heads, rows, dv, offset, gen)
    before = state.double()
    out = torch.zeros((n, heads * dv), device="cuda")
    f64 = lambda t, *shape: t.double().reshape(n, *shape)
    beta = bonus = None
    if kind == "ssm":
        groups = 2 if heads % 2 == 0 else 1
        odd = 1 if heads == 2 else 0                                          # (rows that cannot be copied in 16-byte pieces)
        b0 = (heads * dv + 3) // 4 * 4 + odd
        x, dt = rnd(n, b0 + 2 * groups * rows), rnd(n, heads)
        dt_bias, a_log, skip = rnd(heads) - 2, rnd(heads), rnd(heads)
        K.ssm_scan(x, 0, b0, b0 + groups * rows, dt, 0, dt_bias, a_log, skip, out, heads, groups, rows, dv, step, state, offset)
        d = torch.nn.functional.softplus(dt.double() + dt_bias.double())
        v = f64(x[:, :heads * dv], heads, dv)
        k = f64(x[:, b0:b0 + groups * rows], groups, rows).repeat_interleave(heads // groups, 1) * d[..., None]
        q = f64(x[:, b0 + groups * rows:], groups, rows).repeat_interleave(heads // groups, 1)
        w = torch.exp(-torch.exp(a_log.double()) * d)[..., None].expand(n, heads, rows)
    else:
        qr, kr, v32, a = rnd(n, heads * rows), rnd(n, heads * rows), rnd(n, heads * dv), rnd(n, heads * rows)
        bias, v = rnd(heads * rows), f64(v32, heads, dv)
        if kind == "delta":
            b, a_log = rnd(n, heads), rnd(heads)
            K.delta_scan(qr, 0, kr, 0, v32, 0, b, 0, a, 0, bias, a_log, out, heads, heads, rows, dv, step, state, offset)
            unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)
            q, k, beta = unit(f64(qr, heads, rows)) * rows ** -0.5, unit(f64(kr, heads, rows)), torch.sigmoid(b.double())
            w = torch.exp(-torch.exp(a_log.double())[:, None] * torch.nn.functional.softplus((a.double() + bias.double()).view(n, heads, rows)))
        elif kind == "wkv":
            extra = rnd(heads * rows)
            K.decay_scan(qr, 0, kr, 0, v32, 0, a, 0, bias, extra, out, heads, rows, dv, K.DECAY_EXP_EXP, True, step, state, offset)
            q, k, bonus = f64(qr, heads, rows), f64(kr, heads, rows), extra.double().view(heads, rows)
            w = torch.exp(-torch.exp(a.double() + bias.double())).view(n, heads, rows)       # (from one to none left in a token)
        else:
            low = torch.rand(heads * rows, generator=gen, device="cuda")
            K.decay_scan(qr, 0, None, 0, v32, 0, a, 0, bias, low, out, heads, rows, dv, K.DECAY_LOWER_BOUND, False, step, state, offset)
            w = (low.double() + (1 - low.double()) * torch.sigmoid(a.double() + bias.double())).view(n, heads, rows)
            q, k = torch.nn.functional.silu(f64(qr, heads, rows)), 1 - w
    at = 0
    for s, (m, start) in enumerate(zip(lens, starts)):
        slot = int(step.slot_of_seq[s])
        S = read_state(before, slot, start & 1, offset, heads, dv)[:, :rows]
        if start == 0:
            S = torch.zeros_like(S)
        sl = slice(at, at + m)
        want, S = walk(q[sl], k[sl], v[sl], w[sl], None if beta is None else beta[sl], bonus, S)
        if kind == "ssm":
            want = want + skip.double()[:, None] * v[sl]
        got = read_state(state, slot, (start + m) & 1, offset, heads, dv).double()
        # fp32 sums of a few hundred terms and decays of at most sixteen factors: a few units of 2^-23 of the largest value;
        # the lower bound's written row 1 - w is formed in fp32 from a w close to 1
        tol = 2e-5 if kind == "lower" else 1e-5
        assert (out[sl].double().view(m, heads, dv) - want).abs().max() <= tol * want.abs().max()
        assert (got[:, :rows] - S).abs().max() <= tol * S.abs().max()
        assert not got[:, rows:].any()
        if (start + m) & 1 != start & 1:                                     # the other copy, what lies in front, and other slots stay
            assert torch.equal(state[slot, start & 1], before[slot, start & 1].float())
        assert torch.equal(state[slot, :, :offset], before[slot, :, :offset].float())
        at += m
    for slot in set(range(state.shape[0])) - set(step.slot_of_seq.tolist()):
        assert torch.equal(state[slot], before[slot].float())


@pytest.mark.parametrize("heads,rows,dv", [(2, 20, 5), (3, 64, 64), (2, 128, 100)])      # 8, 16 and 32 row groups
@pytest.mark.parametrize("kind,where", [("ssm", "value"), ("ssm", "key"), ("wkv", "value"), ("wkv", "key"), ("lower", "value"), ("delta", "value"),
                                        ("delta", "key"), ("delta", "beta")])
def test_a_value_that_is_not_finite_leaves_earlier_tokens_alone(kind, where, heads, rows, dv):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(heads + rows)
    rnd = lambda *shape: torch.randn(shape, generator=gen, device="cuda")
    lens, starts, bad = [40, 35], [0, 3], 40 + 22                             # (in the middle of a chunk of the second sequence)
    step, n = step_of(lens, starts), sum(lens)
    state = state_of(step, heads, rows, dv, 0, gen)
    q, k, v, a, b = rnd(n, heads * rows), rnd(n, heads * rows), rnd(n, heads * dv), rnd(n, heads * rows), rnd(n, heads)
    bias, extra, per_head = rnd(heads * rows), torch.rand(heads * rows, generator=gen, device="cuda"), [rnd(heads) for _ in range(3)]

    def run(value, key, beta):
        out, own = torch.zeros((n, heads * dv), device="cuda"), state.clone()
        if kind == "ssm":
            x = torch.cat([value, key, q], 1)
            K.ssm_scan(x, 0, heads * dv, heads * (dv + rows), b, 0, *per_head, out, heads, heads, rows, dv, step, own, 0)
        elif kind == "delta":
            K.delta_scan(q, 0, key, 0, value, 0, beta, 0, a, 0, bias, per_head[0], out, heads, heads, rows, dv, step, own, 0)
        else:
            K.decay_scan(q, 0, key if kind == "wkv" else None, 0, value, 0, a, 0, bias, extra, out, heads, rows, dv,
                         K.DECAY_EXP_EXP if kind == "wkv" else K.DECAY_LOWER_BOUND, kind == "wkv", step, own, 0)
        return out, own

    clean, _ = run(v, k, b)
    for wrong in (float("nan"), float("inf"), float("-inf")):
        spoilt = dict(value=v.clone(), key=k.clone(), beta=b.clone())
        spoilt[where][bad] = float("nan") if where == "beta" else wrong      # (beta passes through a sigmoid)
        out, own = run(spoilt["value"], spoilt["key"], spoilt["beta"])
        assert torch.equal(out[:bad], clean[:bad])
        assert not torch.isfinite(out[bad]).any()
        assert torch.isfinite(own[int(step.slot_of_seq[0])]).all() and not torch.isfinite(own[int(step.slot_of_seq[1]), (3 + 35) & 1]).all()


def scan_of(kind, heads, rows, dv, n, gen):
    """run(rows of the inputs, out, step, state) of a recurrence on drawn inputs of n tokens."""
    rnd = lambda *shape: torch.randn(shape, generator=gen, device="cuda")
    q, k, v, a, b = rnd(n, heads * rows), rnd(n, heads * rows), rnd(n, heads * dv), rnd(n, heads * rows), rnd(n, heads)
    bias, extra, per_head = rnd(heads * rows), torch.rand(heads * rows, generator=gen, device="cuda"), [rnd(heads) for _ in range(3)]
    x = torch.cat([v, k, q], 1)
    if kind == "ssm":
        return lambda sl, out, step, state: K.ssm_scan(x[sl], 0, heads * dv, heads * (dv + rows), b[sl], 0, *per_head, out, heads, heads, rows,
                                                       dv, step, state, 0)
    if kind == "delta":
        return lambda sl, out, step, state: K.delta_scan(q[sl], 0, k[sl], 0, v[sl], 0, b[sl], 0, a[sl], 0, bias, per_head[0], out, heads, heads,
                                                         rows, dv, step, state, 0)
    exp = kind == "wkv"
    return lambda sl, out, step, state: K.decay_scan(q[sl], 0, k[sl] if exp else None, 0, v[sl], 0, a[sl], 0, bias, extra, out, heads, rows, dv,
                                                     K.DECAY_EXP_EXP if exp else K.DECAY_LOWER_BOUND, exp, step, state, 0)


@pytest.mark.parametrize("heads,rows,dv", [(2, 20, 5), (3, 64, 64), (2, 128, 100)])
@pytest.mark.parametrize("kind", ["ssm", "wkv", "delta"])
def test_an_infinite_state_stays_in_its_column(kind, heads, rows, dv):
    """Where products are formed of parts it comes out as not a number rather than as an infinity; no other column sees it, and without
    the delta rule no other row of the state."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(rows)
    step, h, r, c = step_of([40, 35], [0, 3]), 1, 3, 2
    state, slot = state_of(step, heads, rows, dv, 0, gen), int(step.slot_of_seq[1])
    run = scan_of(kind, heads, rows, dv, 75, gen)
    outs, states = [], []
    for value in (1.0, float("inf")):
        own, out = state.clone(), torch.zeros((75, heads, dv), device="cuda")
        own[slot, 1].view(heads, -1, dv, 8)[h, r // 8, c, r % 8] = value
        run(slice(0, 75), out.view(75, -1), step, own)
        outs.append(out)
        states.append(read_state(own, slot, (3 + 35) & 1, 0, heads, dv))
    assert not torch.isfinite(outs[1][40:, h, c]).any() and not torch.isfinite(states[1][h, r, c])
    outs[1][40:, h, c] = outs[0][40:, h, c]
    states[1][h, r if kind != "delta" else slice(None), c] = states[0][h, r if kind != "delta" else slice(None), c]
    assert torch.equal(*outs) and torch.equal(*states)


@pytest.mark.parametrize("lens", [[1, 1, 1, 40, 1, 13, 0, 35, 0], [15, 16, 17, 31], [1] * 15 + [4], [0, 64, 1]])
@pytest.mark.parametrize("heads,rows,dv", [(3, 64, 64), (2, 128, 100)])
@pytest.mark.parametrize("kind", ["ssm", "wkv", "lower", "delta"])
def test_a_sequence_runs_by_its_own_length_whatever_shares_the_step(kind, heads, rows, dv, lens):
    """In a step of a captured size (rows and sequences behind the real ones, a longest run that is rounded up), every sequence's
    outputs and state are the bits that it has alone: short ones walked, long ones in chunks."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(len(lens) + rows)
    starts = [(5 * s) % 7 for s in range(len(lens))]
    real, n = step_of(lens, starts), -(-sum(lens) // 64) * 64
    run = scan_of(kind, heads, rows, dv, n, gen)
    state = state_of(real, heads, rows, dv, 0, gen)
    pad = lambda t, m, v: torch.cat([t, torch.full((m,), v, dtype=torch.int32, device="cuda")])
    more = 16 - len(lens)
    step = SimpleNamespace(cu_seqlens=pad(real.cu_seqlens, more, sum(lens)), slot_of_seq=pad(real.slot_of_seq, more, int(real.slot_of_seq[-1])),
                           start_pos=pad(real.start_pos, more, starts[-1]), n_tokens=n, n_seqs=16, max_q_len=min(n, 128),
                           scan_runs=(True, True))
    scratch, _, least, below = K._scan_route(K._SCAN_SSM, heads, rows, step, "cuda")
    assert scratch is not None and least == below == K.SCAN_CHUNK_TOKENS
    got, got_state = torch.full((n, heads * dv), 7.0, device="cuda"), state.clone()
    run(slice(0, n), got, step, got_state)
    want_state, at = state.clone(), 0
    for s, m in enumerate(lens):
        if m == 0:
            continue
        own = step_of([m], [starts[s]])
        own.slot_of_seq, own.scan_runs = real.slot_of_seq[s:s + 1], K.scan_runs([m])
        assert (K._scan_route(K._SCAN_SSM, heads, rows, own, "cuda")[0] is not None) == (m >= K.SCAN_CHUNK_TOKENS)
        out = torch.empty((m, heads * dv), device="cuda")
        run(slice(at, at + m), out, own, want_state)
        assert torch.equal(got[at:at + m], out), s
        at += m
    assert torch.equal(got_state, want_state)
    assert (got[at:] == 7.0).all()                                            # rows of no sequence are left alone


def test_the_engine_launches_the_scans_that_have_work(tmp_path, monkeypatch):
    from burn_lm_b200 import StepEntry
    from nufolix_tiny import NUF_D, make_folder
    from burn_lm_b200.engine.engine import Engine
    folder, calls, plain = make_folder(tmp_path, "nuf_d"), [], K._call

    def watching(module, name, *args, **kw):
        calls.append(name)
        return plain(module, name, *args, **kw)

    monkeypatch.setattr(K, "_call", watching)
    engine = Engine.from_folder(folder, "bfloat16", max_tokens=64 * 64, max_seqs=20)
    slots = [engine.acquire() for _ in range(16)]
    engine.step([StepEntry(s, [1, 2, 3, 4, 5], [0]) for s in slots])          # (another bucket than those below)
    chunked = lambda: [n for n in calls if n.startswith("blm_scan_chunks_")]
    walked = lambda: [n for n in calls if n in ("blm_ssm_scan", "blm_delta_scan")]
    for lengths, in_chunks, by_walk in (([1] * 15 + [4], False, True), ([15], False, True), ([1] * 15 + [300], True, True), ([40, 16], True, False),
                                        ([1] * 15 + [4], False, True)):
        calls.clear()
        logits = engine.step([StepEntry(s, [t % NUF_D["vocab"] for t in range(m)], [m - 1]) for s, m in zip(slots, lengths)])
        assert bool(chunked()) == in_chunks and bool(walked()) == by_walk, lengths
        assert bool(torch.isfinite(logits).all())


@pytest.mark.parametrize("kind,heads,rows,dv,lens", [("wkv", 32, 128, 16, [2100, 1700]), ("delta", 32, 128, 16, [900, 1800]),
                                                     ("ssm", 2048, 32, 1, [500, 33, 400])])
def test_passes_change_no_bit(kind, heads, rows, dv, lens):
    """Steps whose scratch would be larger than one pass may take: the bits of two of the heads are those of a step of the two."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(heads + rows)
    rnd = lambda *shape: torch.randn(shape, generator=gen, device="cuda")
    starts, n, few = list(range(len(lens))), sum(lens), 2
    step = step_of(lens, starts)
    route = lambda h: K._scan_route({"wkv": K._SCAN_DECAY, "delta": K._SCAN_DELTA, "ssm": K._SCAN_SSM}[kind], h, rows, step, "cuda")
    assert route(heads)[0].numel() <= 32 << 20 and route(heads)[1] > 2 and route(few)[1] == 2
    state = state_of(step, heads, rows, dv, 0, gen)
    own = state.view(state.shape[0], 2, heads, -1)[:, :, :few].reshape(state.shape[0], 2, -1).contiguous()
    b, bias, extra, per_head = rnd(n, heads), rnd(heads * rows), rnd(heads * rows), [rnd(heads) for _ in range(3)]
    v = rnd(n, heads * dv)
    if kind == "ssm":
        x = torch.cat([v, rnd(n, 2 * rows)], 1)
        run = lambda h, out, st: K.ssm_scan(x, 0, heads * dv, heads * dv + rows, b, 0, *[t[:h].contiguous() for t in per_head], out, h, 1, rows, dv,
                                            step, st, 0)
    else:
        q, k, a = rnd(n, heads * rows), rnd(n, heads * rows), rnd(n, heads * rows)
        part = lambda t, h: t[:h * rows].contiguous()
        if kind == "delta":
            run = lambda h, out, st: K.delta_scan(q, 0, k, 0, v, 0, b, 0, a, 0, part(bias, h), per_head[0][:h].contiguous(), out, h, h, rows, dv,
                                                  step, st, 0)
        else:
            run = lambda h, out, st: K.decay_scan(q, 0, k, 0, v, 0, a, 0, part(bias, h), part(extra, h), out, h, rows, dv, K.DECAY_EXP_EXP, True,
                                                  step, st, 0)
    out, two = torch.empty((n, heads * dv), device="cuda"), torch.empty((n, few * dv), device="cuda")
    run(heads, out, state)
    run(few, two, own)
    assert torch.equal(out[:, :few * dv], two)
    assert torch.equal(state.view(state.shape[0], 2, heads, -1)[:, :, :few].reshape(own.shape), own)


def test_more_sequences_than_a_grid_holds_are_walked():
    step = SimpleNamespace(n_tokens=300000, n_seqs=70000, max_q_len=64)
    assert K._scan_route(K._SCAN_SSM, 2, 64, step, "cuda") == (None, 0, 0, K._NO_LIMIT)
