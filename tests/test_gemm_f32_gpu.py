"""The float32 product on the tensor cores (``csrc/gemm_f32_tc.cu``) against 64 bits: edges of its tiles and blocks, every form, any row alone, what is not
finite."""
import pytest
import torch

from roost_b200.kernels import library

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def kernels():
    return library.load()


def _rand(shape, seed):
    return torch.randn(shape, generator=torch.Generator().manual_seed(seed)).cuda()


def _bound(a, w):
    """A chain of 12 products of 32 k cuts its sum off at most 12 times, 2^-23 of it each (24 units of 2^-24); k / 128 chains and three parts are added to nearest;
    the products of parts that are left out are each below 2^-24 of a term, two of them of one sign. All of the sum of the terms' magnitudes."""
    return (24 + a.shape[1] / 128 + 8) * 2.0 ** -24 * (a.abs().double() @ w.abs().double().T)


@pytest.mark.parametrize("m", [1, 15, 16, 17, 33, 64, 65, 97, 129, 400])
@pytest.mark.parametrize("n,k", [(1, 512), (127, 516), (129, 1028), (1000, 3072), (2500, 608)])
def test_against_64_bits_and_any_row_alone(kernels, m, n, k):
    a, w = _rand((m, k), 1), _rand((n, k), 2) * torch.exp(_rand((n, 1), 3))
    got = kernels.gemm_simt(a, w)
    assert ((got.double() - a.double() @ w.double().T).abs() <= _bound(a, w)).all()
    wide = torch.zeros((m, k + 1), device="cuda")
    wide[:, 1:] = a
    assert torch.equal(kernels.gemm_simt(wide[:, 1:], w), got), "rows that do not start on 16 bytes"
    assert torch.equal(kernels.gemm_simt(a[m // 2 : m // 2 + 1], w), got[m // 2 : m // 2 + 1]), "a row alone"
    big = torch.cat([a, _rand((700, k), 4)])
    assert torch.equal(kernels.gemm_simt(big, w)[:m], got), "among other rows"
    assert kernels._lib.roost_gemm_tcgen05_status() == 0


def test_persistent_ctas_take_several_tiles(kernels):
    a, w = _rand((70, 544), 5), _rand((40000, 544), 6)
    got = kernels.gemm_simt(a, w)
    assert ((got.double() - a.double() @ w.double().T).abs() <= _bound(a, w)).all()
    assert torch.equal(kernels.gemm_simt(a[:9], w), got[:9])


def test_clusters_of_narrow_tiles_in_several_rounds(kernels):
    a, w = _rand((300, 2048), 15), _rand((24700, 2048), 16)             # 193 tiles by 16 rows or fewer, 772 CTAs
    got = kernels.gemm_simt(a, w)
    assert ((got.double() - a.double() @ w.double().T).abs() <= _bound(a, w)).all()
    assert torch.equal(kernels.gemm_simt(a[:16], w), got[:16]) and torch.equal(kernels.gemm_simt(a[299:], w), got[299:])


def test_what_is_not_finite_comes_out_as_a_chain_of_sums_has_it(kernels):
    """Infinities, NaN and numbers whose rounding to bfloat16 overflows reach the outputs of their row and column, and no others."""
    k = 512
    a, w = _rand((20, k), 7), _rand((40, k), 8)
    clean = kernels.gemm_simt(a, w)
    a[3, 5], a[7, 1], a[9, 2] = float("inf"), float("nan"), 3.4e38
    w[:, 2] = 0.25
    w[4, 17], w[6] = float("-inf"), 0.0
    w[8, 5] = 0.0                                                   # inf times zero
    got, want = kernels.gemm_simt(a, w), a.double() @ w.double().T
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isinf(got), torch.isinf(want))
    assert torch.equal(got[torch.isinf(want)].double(), want[torch.isinf(want)])
    fine = torch.isfinite(want)
    assert ((got.double() - want).abs()[fine] <= _bound(a, w).nan_to_num(0.0, 0.0)[fine] + 2.0 ** -20 * want.abs()[fine]).all()
    assert got[9, 0].item() == pytest.approx(0.85e38, rel=1e-5) and torch.isfinite(clean).all()


def test_rows_that_are_not_finite_do_not_hold_up_the_other_tiles(kernels):
    """Half the rows of every tile NaN, several tiles a CTA and a long reduction: the chains of FFMAs that those outputs become run when nobody waits for them, and
    what is finite is what it is without them."""
    m, n, k = 1920, 1280, 24576
    a, w = _rand((m, k), 11), _rand((n, k), 12)
    clean = kernels.gemm_simt(a, w)
    bad = torch.arange(m, device="cuda") % 2 == 1
    a[bad, 3] = float("nan")
    w[7, 100] = float("inf")
    got = kernels.gemm_simt(a, w)
    assert kernels._lib.roost_gemm_tcgen05_status() == 0
    assert torch.isnan(got[bad]).all()
    others = torch.arange(n, device="cuda") != 7
    assert torch.equal(got[~bad][:, others], clean[~bad][:, others])
    assert torch.equal(got[~bad][:, 7], torch.where(a[~bad, 100] > 0, float("inf"), float("-inf")))


@pytest.mark.parametrize("m,n,k", [(5, 130, 512), (100, 257, 1028), (40, 20000, 512)])      # clusters, narrow and wide tiles, several tiles a CTA
@pytest.mark.parametrize("of_a,of_w", [(0, -115), (-118, 0), (60, -126), (-126, 100), (0, -138), (-70, -70), (100, -100), (110, -60)])
def test_operands_of_any_size_keep_their_24_bits(kernels, m, n, k, of_a, of_w):
    """Operands down to the smallest numbers that there are and up to where sums no longer fit, as accurate as ordinary ones: relative to the sum of the
    terms' magnitudes, and half a unit of the smallest number."""
    a, w = _rand((m, k), 13) * 2.0 ** of_a, (_rand((n, k), 14).double() * 2.0 ** of_w).float()
    got, want = kernels.gemm_simt(a, w), a.double() @ w.double().T
    assert ((got.double() - want).abs() <= _bound(a, w) + 2.0 ** -149).all()
    assert torch.equal(kernels.gemm_simt(a[m // 2 : m // 2 + 1], w), got[m // 2 : m // 2 + 1]), "a row alone"
