"""The float32 product on the tensor cores at the edges of its tiles, steps and shares, with infinities, and with weights that lie so that
the other kernel takes them."""
import pytest
import torch

from burn_lm_b200 import kernels as K

pytestmark = pytest.mark.gpu


def _operands(n, m, k, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return [torch.randn(shape, generator=gen, device="cuda") for shape in ((n, k), (m, k))]


@pytest.mark.parametrize("n", [1, 31, 64, 65, 97, 159, 161, 321])
@pytest.mark.parametrize("m,k", [(1, 64), (127, 68), (129, 1020), (128, 1028), (257, 2112), (2700, 196)])
def test_edges(n, m, k):
    x, w = _operands(n, m, k, n * 7 + m)
    want = x.double() @ w.double().T
    err = (K.gemm_f32(x, w).double() - want).norm() / want.norm()
    # operands exact, products left out below 2^-21 of a term and random; the large products meet four at a time: below what a chain of
    # 1,024 multiply-adds shows (5.7e-7)
    assert err <= 4e-7
    assert K.check_status("cuda") is None


def test_one_block_adds_the_shares_as_planes_do():
    x, w = _operands(300, 9000, 4096, 5)                     # many tiles: a block adds a tile's four shares up
    y = K.gemm_f32(x, w)
    assert torch.equal(y[:, 128:256], K.gemm_f32(x, w[128:256].contiguous()))      # few: planes


def test_weights_that_lie_otherwise():
    x, w = _operands(40, 70, 256, 6)
    wide = torch.zeros((70, 257), device="cuda")
    wide[:, :256] = w
    y = K.batched_product(x[None], wide[None, :, :256])      # rows not at multiples of 16 bytes: FFMA
    assert (y[0] - K.gemm_f32(x, w)).abs().max() <= 2 * 4 * 256 * 2.0 ** -24


def test_what_is_not_finite():
    x, w = _operands(70, 200, 256, 7)
    inf = float("inf")
    x[3, 5], x[4, 7], x[6] = inf, float("nan"), 3e38
    w[10, 3], w[20] = -inf, 3e38
    y, want = K.gemm_f32(x, w), (x[:, None] * w[None]).sum(-1)
    assert torch.equal(y.isnan(), want.isnan()) and torch.equal(y.isinf(), want.isinf())
    assert torch.equal(y[y.isinf()], want[want.isinf()])


@pytest.mark.parametrize("m,k,tensor", [(512, 64, 0), (513, 64, 1), (64, 512, 0), (65, 512, 1), (1, 516, 1), (64, 64, 0), (200, 160, 0), (200, 66, 0)])
def test_small_weights_take_one_launch(m, k, tensor):
    """A weight's size says which kernel forms its products, and a row has the bits it has alone, on either side of the border."""
    x, w = _operands(1700, m, k, m + k)
    assert K._ask("gemm", "blm_gemm_f32_tensor", w.data_ptr(), m, k, k, 0) == tensor
    scratch, launches = K._gemm_f32_scratch(1, 1700, m, k, "cuda", w, k)
    assert launches == 1 + tensor and (scratch is None) == (not tensor)
    y, want = K.gemm_f32(x, w), x.double() @ w.double().T
    # FFMA: roundings of partial sums that grow with the square root of their length, 32 places at a time where rows come in 16-byte pieces;
    # the tensor cores: four additions a step of 64 places
    chain = k if k % 4 else 32
    assert (y.double() - want).norm() / want.norm() <= (1.5e-7 if tensor else (chain / 2 + k / chain / 2) ** 0.5 * 2.0 ** -24 / 3 ** 0.5)
    for n in (1, 16, 17, 40, 130, 700):                      # tiles of every size
        assert torch.equal(K.gemm_f32(x[:n].contiguous(), w), y[:n]), n


def test_scratch_is_that_of_the_kernel_that_runs():
    parts = 600 * 2048 * 3 // 2                              # x in three bfloat16 numbers a float
    w = torch.empty((16384, 2052), device="cuda")
    assert K._gemm_f32_scratch(1, 600, 16384, 2048, "cuda", w, 2052)[0].numel() == parts
    assert K._gemm_f32_scratch(1, 600, 16384, 2048, "cuda", w.view(-1)[1:], 2052)[0].numel() == 2 * 600 * 16384      # FFMA's planes
    # one row of a wider matrix says it is contiguous, whatever its stride
    x, wide = _operands(5, 1, 2048, 8)[0], torch.randn((3, 2049), device="cuda")
    w = wide[1:2, 3:2051 - 2].as_strided((1, 2048), (2049, 1), 2052)
    assert w.is_contiguous() and (K.gemm_f32(x, w).double() - x.double() @ w.double().T).abs().max() <= 1e-3
