"""Sums of one sign: what the tensor cores cut off, and the products of parts that are left out, add up instead of cancelling.  The products in
parts against the walk, token by token in multiply-adds, and the float32 product: both from float64."""
import pytest
import torch

from burn_lm_b200 import kernels as K
from test_gpu_scan_chunks import read_state, state_of, step_of, walk

pytestmark = pytest.mark.gpu
CUT = 2.0 ** -24                                                              # of a sum, on average, when its last place is cut off


def relative(got, want):
    return float((got.double() - want).norm() / want.norm())


@pytest.mark.parametrize("kind,heads,rows,dv,n", [("long", 8, 128, 64, 2048), ("long", 8, 66, 40, 1600), ("ssm", 8, 128, 64, 1024), ("ssm", 8, 64, 40, 500),
                                                  ("wkv", 4, 128, 64, 1024), ("wkv", 4, 64, 64, 1024), ("delta", 4, 128, 64, 1024)])
@pytest.mark.parametrize("sign", [True, False])
def test_scans_are_as_exact_as_the_walk(kind, heads, rows, dv, n, sign, monkeypatch):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(rows + n)
    rnd = lambda *shape: torch.randn(shape, generator=gen, device="cuda")
    drawn = lambda *shape: rnd(*shape).abs() if sign else rnd(*shape)
    f64 = lambda t, *shape: t.double().reshape(n, *shape)
    step = step_of([n], [2])
    state = state_of(step, heads, rows, dv, 0, gen)
    state = state.abs() if sign else state
    q, k, v, a, b = drawn(n, heads * rows), drawn(n, heads * rows), drawn(n, heads * dv), rnd(n, heads * rows), rnd(n, heads)
    bias, extra, a_log = rnd(heads * rows), drawn(heads * rows), rnd(heads)
    beta = bonus = None
    k64, q64 = f64(k, heads, rows), f64(q, heads, rows)
    if kind in ("long", "ssm"):
        groups, dt_bias, skip = 2, rnd(heads) - 2, drawn(heads)
        x = torch.cat([v, k[:, :groups * rows], q[:, :groups * rows]], 1)
        d = torch.nn.functional.softplus(b.double() + dt_bias.double())
        k64 = f64(k[:, :groups * rows], groups, rows).repeat_interleave(heads // groups, 1) * d[..., None]
        q64 = f64(q[:, :groups * rows], groups, rows).repeat_interleave(heads // groups, 1)
        w = torch.exp(-torch.exp(a_log.double()) * d)[..., None].expand(n, heads, rows)
    elif kind == "delta":
        unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)
        q64, k64, beta = unit(q64) * rows ** -0.5, unit(k64), torch.sigmoid(b.double())
        w = torch.exp(-torch.exp(a_log.double())[:, None] * torch.nn.functional.softplus((a.double() + bias.double()).view(n, heads, rows)))
    else:
        bonus, w = extra.double().view(heads, rows), torch.exp(-torch.exp(a.double() + bias.double())).view(n, heads, rows)
    slot = int(step.slot_of_seq[0])
    want, S = walk(q64, k64, f64(v, heads, dv), w, beta, bonus, read_state(state.double(), slot, 0, 0, heads, dv)[:, :rows])
    if kind in ("long", "ssm"):
        want = want + skip.double()[:, None] * f64(v, heads, dv)

    def run(runs, least):
        monkeypatch.setattr(K, "SCAN_LONG_TOKENS", least)
        monkeypatch.setattr(K, "SCAN_LONG_TOKENS_FEW_HEADS", least)
        step.scan_runs, own, out = runs, state.clone(), torch.zeros((n, heads * dv), device="cuda")
        if kind in ("long", "ssm"):
            at = heads * dv
            K.ssm_scan(x, 0, at, at + groups * rows, b, 0, dt_bias, a_log, skip, out, heads, groups, rows, dv, step, own, 0)
        elif kind == "delta":
            K.delta_scan(q, 0, k, 0, v, 0, b, 0, a, 0, bias, a_log, out, heads, heads, rows, dv, step, own, 0)
        else:
            K.decay_scan(q, 0, k, 0, v, 0, a, 0, bias, extra, out, heads, rows, dv, K.DECAY_EXP_EXP, True, step, own, 0)
        return relative(out.view(n, heads, dv), want), relative(read_state(own, slot, n & 1, 0, heads, dv)[:, :rows], S)

    in_parts = run((True, False, kind == "long", kind == "long"), 64 if kind == "long" else K._NO_LIMIT)
    walked = run((False, True), K._NO_LIMIT)
    # an output is cut where a chunk's sums leave the tensor cores; a state once more for what a group of chunks adds to it
    assert in_parts[0] <= walked[0] + CUT and in_parts[1] <= walked[1] + 2 * CUT


@pytest.mark.parametrize("n,m,k", [(64, 512, 1024), (317, 2048, 2048), (3, 4096, 256), (70, 900, 8192)])
def test_the_product_is_as_exact_with_one_sign(n, m, k):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(k)
    x, w = (torch.rand(shape, generator=gen, device="cuda") for shape in ((n, k), (m, k)))
    # a step of 64 places is cut four times at its full size and rounded once where it joins the others
    assert relative(K.gemm_f32(x, w), x.double() @ w.double().T) <= 2 * CUT
