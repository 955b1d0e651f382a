"""The product of a decode step's few rows over weights held in registers (``csrc/gemm_rows.cu``) against 64 bits."""
import pytest
import torch

from roost_b200.kernels import library

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def kernels():
    return library.load()


def _rand(shape, seed, scale=1.0):
    return (torch.randn(shape, generator=torch.Generator().manual_seed(seed)) * scale).bfloat16().cuda()


# every number of k blocks a warp, one, two and four groups of rows a CTA, the last CTA with rows beyond the matrix
SIZES = [(1, 256), (64, 512), (250, 768), (1024, 1024), (4104, 1024), (9472, 512), (8000, 1024), (512, 1536), (2048, 2048), (4700, 2048), (1030, 3072), (1024, 4096)]


@pytest.mark.parametrize("m", [1, 7, 8, 9, 16])
@pytest.mark.parametrize("n,k", SIZES)
def test_against_64_bits_and_rows_alone(kernels, m, n, k):
    x, w = _rand((m, k), 1), _rand((n, k), 2, 0.05)
    assert kernels.gemm_rows_supported(x, w), "sizes that a form serves"
    want, size = x.double() @ w.double().T, x.abs().double() @ w.abs().double().T
    got = kernels.gemm_rows(x, w, torch.float32)
    # chains of k / 128 products a warp whose sums are cut off (2^-23 of the terms' magnitude each, a product of 16 k), nine additions to nearest
    bound = (k / 128 * 2 + 10) * 2.0 ** -23 * size
    assert ((got.double() - want).abs() <= bound).all()
    rounded = kernels.gemm_rows(x, w)
    assert ((rounded.double() - want).abs() <= bound + 2.0 ** -8 * want.abs()).all()
    assert torch.equal(rounded, got.bfloat16()), "one rounding of the same sums"
    i = m // 2
    assert torch.equal(kernels.gemm_rows(x[i : i + 1], w, torch.float32), got[i : i + 1]), "a row alone"
    wide = torch.zeros((m, k + 8), dtype=torch.bfloat16, device="cuda")
    wide[:, 8:] = x
    assert torch.equal(kernels.gemm_rows(wide[:, 8:], w, torch.float32), got), "strided rows"


@pytest.mark.parametrize("m", [1, 8, 13])
@pytest.mark.parametrize("inter,k", [(128, 256), (256, 768), (1536, 2048), (3072, 1024)])
def test_with_the_activation(kernels, m, inter, k):
    x, w = _rand((m, k), 3), _rand((2 * inter, k), 4, 0.05)
    if not kernels.gemm_rows_supported(x, w, swiglu=True):
        pytest.fail("sizes that a form serves")
    y = (x.double() @ w.double().T).reshape(m, inter // 128, 2, 128)
    g, u = y[:, :, 0].reshape(m, inter), y[:, :, 1].reshape(m, inter)
    want = g / (1.0 + torch.exp(-g)) * u
    got = kernels.gemm_rows(x, w, swiglu=True)
    # one rounding to bfloat16; the sums' own error (see above) passes a factor of at most |u| + 1.1 |g|, which 2^-12 covers by far
    assert ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -12 * (u.abs() + 1.1 * g.abs() + 1)).all()


def test_what_is_not_served(kernels):
    w = _rand((64, 256), 5)
    assert not kernels.gemm_rows_supported(_rand((17, 256), 6), w)
    assert not kernels.gemm_rows_supported(_rand((4, 264), 6), _rand((64, 264), 6))
    assert not kernels.gemm_rows_supported(_rand((4 * 256 + 1,), 6)[1:].reshape(4, 256), w), "rows that do not start on 16 bytes"
    assert not kernels.gemm_rows_supported(_rand((1, 1024), 6), _rand((151936, 1024), 6))
    assert not kernels.gemm_rows_supported(_rand((1, 1024), 6), _rand((9480, 1024), 6)), "a row more than the processors hold"
    assert not kernels.gemm_rows_supported(_rand((1, 1280), 6), _rand((64, 1280), 6)), "five pieces a warp"
    with pytest.raises(Exception):
        kernels.gemm_rows(_rand((17, 256), 6), w)
