"""The float32 product at the edges of its tiles and of its shares of K, against float64; a row's bits depend on nothing but
the row and the weights."""
import pytest
import torch

from burn_lm_b200 import kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 16, 17, 32, 33, 65, 130])
@pytest.mark.parametrize("m,k", [(33, 5), (128, 1023), (129, 1024), (300, 1025), (64, 2600), (40, 4096)])
def test_product_at_the_edges(n, m, k):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n * 100003 + m * 31 + k)
    x, w = (torch.randn(shape, generator=gen, device="cuda") for shape in ((n, k), (m, k)))
    want = x.double() @ w.double().T
    y = K.gemm_f32(x, w)
    # sums of K products of unit normals: rounding errors of at most sqrt(K) 2^-24 times partial sums of size sqrt(K)
    assert (y.double() - want).abs().max() <= 4 * k * 2.0 ** -24
    assert torch.equal(K.gemm_f32(x[:1].contiguous(), w), y[:1])
    assert torch.equal(K.gemm_f32(x, w[3:20].contiguous()), y[:, 3:20])
    # the same as one of a batch of strided operands
    wide = torch.zeros((n, 2, k + 3), device="cuda")
    wide[:, 1, :k] = x
    both = K.batched_product(wide[:, :, :k].transpose(0, 1), torch.stack([w, w]), out=torch.empty((n, 2, m), device="cuda").transpose(0, 1))
    assert torch.equal(both[1], y) and not both[0].any()


@pytest.mark.parametrize("of", ["x", "w"])
def test_rows_further_apart_than_an_int_can_tell(of):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(2)
    apart = (1 << 31) // 63 // 4 * 4 + 4                                      # the 64th row of a tile lies 2^31 places behind the first
    wide = torch.empty(63 * apart + 8, device="cuda").as_strided((1, 64, 8), (0, apart, 1))
    wide.copy_(torch.randn((1, 64, 8), generator=gen, device="cuda"))
    near = torch.randn((1, 60, 8), generator=gen, device="cuda")
    x, w = (wide, near) if of == "x" else (near, wide)
    assert torch.equal(K.batched_product(x, w), K.batched_product(x.contiguous(), w.contiguous()))


def test_batches_whose_shares_fill_more_than_one_grid():
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1)
    x, w = (torch.randn(shape, generator=gen, device="cuda") for shape in ((40000, 1, 1030), (40000, 3, 1030)))
    y = K.batched_product(x, w)                                               # two shares each: 80,000 blocks deep
    for b in (0, 1, 32766, 32767, 32768, 39999):
        assert torch.equal(y[b], K.gemm_f32(x[b], w[b])), b
    want = torch.einsum("bnk,bmk->bnm", x.double(), w.double())
    assert (y.double() - want).abs().max() <= 4 * 1030 * 2.0 ** -24


@pytest.mark.parametrize("n,m,k", [(1030, 20000, 4096), (9000, 300, 30000), (270, 20000, 16384)])
def test_passes_change_no_bit(n, m, k):
    """Products whose planes of sums would be larger than one pass may take, cut along their columns and along their rows."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(3)
    x, w = (torch.randn(shape, generator=gen, device="cuda") for shape in ((n, k), (m, k)))
    scratch, launches = K._gemm_f32_scratch(1, n, m, k, "cuda")
    assert scratch.numel() <= 64 << 20 and launches > 2
    y = K.gemm_f32(x, w)
    rows, cols = [0, n // 2, n - 1], slice(m // 2 - 20, m // 2 + 20)
    assert torch.equal(y[rows], K.gemm_f32(x[rows].contiguous(), w))
    assert torch.equal(y[:, cols], K.gemm_f32(x, w[cols].contiguous()))
    assert torch.equal(y[:, -1:], K.gemm_f32(x, w[-1:].contiguous()))


@pytest.mark.parametrize("batch,n,m,k", [(1, 2048, 128256, 4096), (1, 128256, 2048, 14336), (32, 2048, 512, 2048), (1, 4000000, 3, 4096)])
def test_scratch_is_bounded(batch, n, m, k):
    assert 0 < int(K._lib("gemm").blm_gemm_f32_scratch(batch, n, m, k)) <= 64 << 20
