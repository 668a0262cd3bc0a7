"""The state-space scan in chunks of 64 tokens on the tensor cores (scan_long.cu) against the walk in float64, at the edges of its chunks
and groups of chunks, beside shorter sequences, with rows that cannot be copied in 16-byte pieces, and with values that are not finite."""
import pytest
import torch

from burn_lm_b200 import kernels as K
from test_gpu_scan_chunks import read_state, state_of, step_of, walk

pytestmark = pytest.mark.gpu
BORDERS = K.SCAN_LONG_TOKENS, K.SCAN_LONG_TOKENS_FEW_HEADS


@pytest.fixture(autouse=True)
def from_64_tokens_on(monkeypatch):
    monkeypatch.setattr(K, "SCAN_LONG_TOKENS", 64)
    monkeypatch.setattr(K, "SCAN_LONG_TOKENS_FEW_HEADS", 64)


def inputs(heads, groups, rows, dv, n, gen, odd=0):
    rnd = lambda *shape: torch.randn(shape, generator=gen, device="cuda")
    b0 = (heads * dv + 3) // 4 * 4 + odd
    return rnd(n, b0 + 2 * groups * rows), b0, rnd(n, heads), rnd(heads) - 2, rnd(heads), rnd(heads)


def scan(x, b0, dt, dt_bias, a_log, skip, heads, groups, rows, dv, step, state, offset):
    out = torch.zeros((step.n_tokens, heads * dv), device="cuda")
    K.ssm_scan(x, 0, b0, b0 + groups * rows, dt, 0, dt_bias, a_log, skip, out, heads, groups, rows, dv, step, state, offset)
    return out


@pytest.mark.parametrize("lens,starts", [([64], [0]), ([65], [5]), ([127, 40, 1, 576], [2, 0, 9, 1]), ([512, 513], [0, 3]), ([1153], [1])])
@pytest.mark.parametrize("heads,groups,rows,dv", [(2, 1, 128, 64), (8, 2, 100, 36), (12, 3, 66, 63), (36, 1, 128, 64)])
def test_long_sequences_against_the_walk_in_float64(heads, groups, rows, dv, lens, starts):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(heads + rows + sum(lens))
    step, n, offset = step_of(lens, starts), sum(lens), 7
    route = K._long_route(heads, groups, rows, dv, step, "cuda")
    assert route is not None and route[2] == 64 and route[3] == (len(lens) == 1)
    state = state_of(step, heads, rows, dv, offset, gen)
    before = state.double()
    x, b0, dt, dt_bias, a_log, skip = args = inputs(heads, groups, rows, dv, n, gen, odd=heads % 8 == 2)
    out = scan(*args, heads, groups, rows, dv, step, state, offset)
    f64 = lambda t, *shape: t.double().reshape(n, *shape)
    d = torch.nn.functional.softplus(dt.double() + dt_bias.double())
    v = f64(x[:, :heads * dv], heads, dv)
    k = f64(x[:, b0:b0 + groups * rows], groups, rows).repeat_interleave(heads // groups, 1) * d[..., None]
    q = f64(x[:, b0 + groups * rows:], groups, rows).repeat_interleave(heads // groups, 1)
    w = torch.exp(-torch.exp(a_log.double()) * d)[..., None].expand(n, heads, rows)
    at = 0
    for s, (m, start) in enumerate(zip(lens, starts)):
        slot, sl = int(step.slot_of_seq[s]), slice(at, at + m)
        S = read_state(before, slot, start & 1, offset, heads, dv)[:, :rows]
        want, S = walk(q[sl], k[sl], v[sl], w[sl], None, None, torch.zeros_like(S) if start == 0 else S)
        want = want + skip.double()[:, None] * v[sl]
        got = read_state(state, slot, (start + m) & 1, offset, heads, dv).double()
        # as for the chunks of sixteen tokens: fp32 sums, decays of at most 64 factors, operands with all 24 bits
        assert (out[sl].double().view(m, heads, dv) - want).abs().max() <= 1e-5 * want.abs().max()
        assert (got[:, :rows] - S).abs().max() <= 1e-5 * S.abs().max()
        assert not got[:, rows:].any()
        at += m
    assert torch.equal(state[:, :, :offset], before[:, :, :offset].float())
    assert K.check_status("cuda") is None


def test_groups_in_any_order_read_the_state_the_sequence_brings(monkeypatch):
    """An even number of tokens: the state is written where it was read.  With more blocks than the chip holds at a time the last
    sequences' groups start one after another."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(6)
    heads, groups, rows, dv, lens, starts = 64, 2, 128, 64, [512, 194, 512, 512, 514], [2, 4, 3, 6, 8]
    step, n = step_of(lens, starts), sum(lens)
    state = state_of(step, heads, rows, dv, 0, gen)
    x, b0, dt, dt_bias, a_log, skip = args = inputs(heads, groups, rows, dv, n, gen)
    step.scan_runs = (False, True)                                            # walked token by token; then as long sequences
    walked, run = state.clone(), state.clone()
    monkeypatch.setattr(K, "SCAN_LONG_TOKENS", K._NO_LIMIT)
    want = scan(*args, heads, groups, rows, dv, step, walked, 0)
    monkeypatch.setattr(K, "SCAN_LONG_TOKENS", 64)
    step.scan_runs = K.scan_runs(lens)
    route = K._long_route(heads, groups, rows, dv, step, "cuda")
    assert route is not None and route[3] and K.sm_count("cuda") < heads // 2 * 4 * len(lens)
    got = scan(*args, heads, groups, rows, dv, step, run, 0)
    assert (got - want).abs().max() <= 2e-5 * want.abs().max()                # both within 1e-5 of 64 bits
    assert (run - walked).abs().max() <= 2e-5 * walked.abs().max()


def test_a_sequence_has_the_bits_it_has_alone():
    gen = torch.Generator(device="cuda")
    gen.manual_seed(3)
    heads, groups, rows, dv, lens = 8, 2, 128, 64, [70, 30, 700, 64]
    step = step_of(lens, [0, 0, 4, 1])
    step.scan_runs = K.scan_runs(lens)
    state = state_of(step, heads, rows, dv, 0, gen)
    args = x, b0, dt, dt_bias, a_log, skip = inputs(heads, groups, rows, dv, sum(lens), gen)
    together, own, at = state.clone(), state.clone(), 0
    out = scan(*args, heads, groups, rows, dv, step, together, 0)
    for s, m in enumerate(lens):
        alone = step_of([m], [[0, 0, 4, 1][s]])
        alone.slot_of_seq, alone.scan_runs = step.slot_of_seq[s:s + 1], K.scan_runs([m])
        got = scan(x[at:at + m], b0, dt[at:at + m], dt_bias, a_log, skip, heads, groups, rows, dv, alone, own, 0)
        assert torch.equal(got, out[at:at + m]), s
        at += m
    assert torch.equal(own, together)


def test_scratch_is_bounded_and_heads_in_passes_change_no_bit(monkeypatch):
    monkeypatch.setattr(K, "SCAN_LONG_TOKENS", 1536)                            # (sums are kept for every so many tokens of a step)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(4)
    heads, groups, rows, dv, n = 64, 4, 128, 64, 12000
    step = step_of([n], [0])
    scratch, launches, _, _ = K._long_route(heads, groups, rows, dv, step, "cuda")
    assert scratch.numel() <= 64 << 20 and launches > 3
    state = state_of(step, heads, rows, dv, 0, gen)
    x, b0, dt, dt_bias, a_log, skip = inputs(heads, groups, rows, dv, n, gen)
    few = heads // groups                                                     # the heads of the first group, in one pass
    part = torch.cat([x[:, :few * dv], x[:, b0:b0 + rows], x[:, b0 + groups * rows:b0 + (groups + 1) * rows]], 1).contiguous()
    own = state.view(state.shape[0], 2, heads, -1)[:, :, :few].reshape(state.shape[0], 2, -1).contiguous()
    out = scan(x, b0, dt, dt_bias, a_log, skip, heads, groups, rows, dv, step, state, 0)
    got = scan(part, few * dv, dt[:, :few].contiguous(), dt_bias[:few].contiguous(), a_log[:few].contiguous(), skip[:few].contiguous(), few, 1, rows, dv,
               step, own, 0)
    assert torch.equal(out[:, :few * dv], got)
    assert torch.equal(state.view(state.shape[0], 2, heads, -1)[:, :, :few].reshape(own.shape), own)


@pytest.mark.parametrize("m", [1, 63, 64, 130, 700])
def test_a_lone_sequence_among_rows_of_none(m):
    """A step that knows no lengths but the bounds of a captured size: its one sequence is run however short it is."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(m)
    heads, groups, rows, dv, n = 4, 2, 128, 64, 4500
    step, real = step_of([m], [3]), step_of([m], [3])
    step.n_tokens = step.max_q_len = n
    state = state_of(step, heads, rows, dv, 0, gen)
    x, b0, dt, dt_bias, a_log, skip = args = inputs(heads, groups, rows, dv, n, gen)
    assert K._long_route(heads, groups, rows, dv, step, "cuda")[3]
    own, walked, real.scan_runs = state.clone(), state.clone(), (False, True)
    out = scan(*args, heads, groups, rows, dv, step, own, 0)
    want = scan(x[:m], b0, dt[:m], dt_bias, a_log, skip, heads, groups, rows, dv, real, walked, 0)
    assert not out[m:].any()
    assert (out[:m] - want).abs().max() <= 2e-5 * want.abs().max() and (own - walked).abs().max() <= 2e-5 * walked.abs().max()


@pytest.mark.parametrize("heads,lens,long,alone", [(36, [4095], False, None), (36, [4096], True, True), (38, [1535], False, None), (38, [1536], True, True),
                                                   (36, [4096, 2000], True, False), (38, [1536, 2000], True, True), (38, [1536, 1], True, False)])
def test_where_the_long_scans_begin(heads, lens, long, alone, monkeypatch):
    """Thirty-six heads of 64 columns are one block a multiprocessor in chunks of sixteen, thirty-eight more."""
    monkeypatch.setattr(K, "SCAN_LONG_TOKENS", BORDERS[0])
    monkeypatch.setattr(K, "SCAN_LONG_TOKENS_FEW_HEADS", BORDERS[1])
    step = step_of(lens, [0] * len(lens))
    step.scan_runs = K.scan_runs(lens)
    route = K._long_route(heads, 1, 128, 64, step, "cuda")
    assert (route is not None) == long and (not long or route[3] == alone)


LARGEST = 256 << 20                                                           # bytes of scratch


@pytest.mark.parametrize("heads,groups", [(64, 1), (64, 4), (64, 8), (64, 32), (128, 8), (24, 1), (8, 4)])
@pytest.mark.parametrize("n_seqs,longest", [(1, 2048), (1, 16384), (1, 131072), (4, 2048), (3, 20000), (200, 2000), (20, 65536)])
def test_scratch_does_not_grow_with_the_tokens(heads, groups, n_seqs, longest):
    least, n = 1536, n_seqs * longest
    used = K._ask("scan_long", "blm_scan_long_scratch", heads, heads // groups, 128, 64, n, n_seqs, longest, least)
    launches = K._ask("scan_long", "blm_scan_long_launches", heads, heads // groups, 128, 64, n, n_seqs, longest, least)
    assert 0 < used <= LARGEST and launches % 3 == 0 and 0 < launches <= 3 * (2 if heads == 128 or groups == 32 else 1) * (-(-n // 2048) + n_seqs + 1)


@pytest.mark.parametrize("lens,starts", [([4096], [2]), ([4097], [1]), ([8256], [4]), ([9000, 70, 2, 4160, 4096, 100], [2, 0, 3, 6, 1, 8])])
def test_segments_against_the_walk(lens, starts, monkeypatch):
    """Sequences of several segments, whose edges fall between those of others, in passes of their own."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(sum(lens))
    heads, groups, rows, dv = 4, 1, 128, 64
    step, n = step_of(lens, starts), sum(lens)
    state = state_of(step, heads, rows, dv, 0, gen)
    x, b0, dt, dt_bias, a_log, skip = args = inputs(heads, groups, rows, dv, n, gen)
    step.scan_runs = K.scan_runs(lens)
    assert K._long_route(heads, groups, rows, dv, step, "cuda")[1] >= (3 if n <= 4096 else 6)
    run, own, walked = state.clone(), state.clone(), state.clone()
    got, at = scan(*args, heads, groups, rows, dv, step, run, 0), 0
    for s, m in enumerate(lens):                                              # the bits it has alone
        alone = step_of([m], [starts[s]])
        alone.slot_of_seq, alone.scan_runs = step.slot_of_seq[s:s + 1], K.scan_runs([m])
        assert torch.equal(got[at:at + m], scan(x[at:at + m], b0, dt[at:at + m], dt_bias, a_log, skip, heads, groups, rows, dv, alone, own, 0)), s
        at += m
    assert torch.equal(run, own)
    monkeypatch.setattr(K, "SCAN_LONG_TOKENS", K._NO_LIMIT)
    step.scan_runs = (False, True)
    want = scan(*args, heads, groups, rows, dv, step, walked, 0)
    assert (got - want).abs().max() <= 2e-5 * want.abs().max()                # both within 1e-5 of 64 bits
    assert (run - walked).abs().max() <= 2e-5 * walked.abs().max()


def test_an_infinite_state_stays_in_its_column():
    gen = torch.Generator(device="cuda")
    gen.manual_seed(9)
    heads, rows, dv, h, r, c = 4, 128, 64, 1, 70, 33
    step = step_of([70, 640], [0, 3])
    state, slot = state_of(step, heads, rows, dv, 0, gen), int(step.slot_of_seq[1])
    args, outs, states = inputs(heads, 1, rows, dv, 710, gen), [], []
    for value in (1.0, float("inf")):
        own = state.clone()
        own[slot, 1].view(heads, -1, dv, 8)[h, r // 8, c, r % 8] = value
        outs.append(scan(*args, heads, 1, rows, dv, step, own, 0).view(710, heads, dv))
        states.append(read_state(own, slot, (3 + 640) & 1, 0, heads, dv))
    assert not torch.isfinite(outs[1][70:, h, c]).any() and not torch.isfinite(states[1][h, r, c])
    outs[1][70:, h, c], states[1][h, r, c] = outs[0][70:, h, c], states[0][h, r, c]
    assert torch.equal(*outs) and torch.equal(*states)


@pytest.mark.parametrize("where", ["value", "key", "dt"])
def test_a_value_that_is_not_finite_leaves_earlier_tokens_alone(where):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(5)
    heads, rows, dv, lens, bad = 4, 128, 64, [70, 640], 70 + 100              # (in the second chunk of the second sequence's first group)
    step = step_of(lens, [0, 3])
    state = state_of(step, heads, rows, dv, 0, gen)
    x, b0, dt, *per_head = inputs(heads, 1, rows, dv, sum(lens), gen)
    clean = scan(x, b0, dt, *per_head, heads, 1, rows, dv, step, state.clone(), 0)
    for wrong in (float("nan"), float("inf"), float("-inf")):
        x2, dt2, own = x.clone(), dt.clone(), state.clone()
        if where == "value":
            x2[bad, 5] = wrong                                                # one column of one head
        elif where == "key":
            x2[bad, b0:b0 + rows] = wrong
        else:
            dt2[bad] = float("nan")
        out = scan(x2, b0, dt2, *per_head, heads, 1, rows, dv, step, own, 0)
        assert torch.equal(out[:bad], clean[:bad])
        last = own[int(step.slot_of_seq[1]), (3 + 640) & 1]
        assert torch.isfinite(own[int(step.slot_of_seq[0])]).all() and not torch.isfinite(last).all()
        if where == "value":
            assert not torch.isfinite(out[bad, 5])
            others = [c for c in range(heads * dv) if c != 5]
            assert torch.equal(out[:, others], clean[:, others])
        else:
            assert not torch.isfinite(out[bad]).any()
