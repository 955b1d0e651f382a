"""Attention of a decode step's few rows (``csrc/attention_rows.cu``) against 64 bits."""
import math

import pytest
import torch

from roost_b200.kernels import library

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def kernels():
    return library.load()


def _rand(shape, seed):
    return torch.randn(shape, generator=torch.Generator().manual_seed(seed)).bfloat16().cuda()


def _i32(v):
    return torch.tensor(v, dtype=torch.int32, device="cuda")


def _cache(lens, kv_heads, page, width, seed):
    """A pool whose pages lie shuffled, NaN beyond the rows' keys, and the tables that name them."""
    need = [-(-n // page) for n in lens]
    total = sum(need) + 2
    pool = torch.full((total, kv_heads, page, width), float("nan"), dtype=torch.bfloat16, device="cuda")
    order = torch.randperm(total, generator=torch.Generator().manual_seed(seed)).tolist()
    indptr, indices, keys = [0], [], []
    for r, n in enumerate(lens):
        mine = order[indptr[-1] : indptr[-1] + need[r]]
        x = _rand((max(n, 1), kv_heads, width), seed + r)
        for j in range(n):
            pool[mine[j // page], :, j % page] = x[j]
        indptr.append(indptr[-1] + need[r])
        indices += mine
        keys.append(x[:n])
    return pool, _i32(indptr), _i32(indices or [0]), keys


# one key, edges of a block of 16, of a warp's turn, of a cluster's; padding rows; a group that fills the tile of heads and ones that do not
ROWS = [[1], [16, 17, 1000], [129, 0, 1023, 15], [300] * 9, [2000]]


@pytest.mark.parametrize("lens", ROWS)
@pytest.mark.parametrize("heads,kv_heads,dim,page", [(16, 8, 128, 16), (4, 4, 64, 32), (16, 1, 64, 16), (24, 2, 128, 64)])
def test_softmax(kernels, lens, heads, kv_heads, dim, page):
    k_pool, indptr, indices, keys = _cache(lens, kv_heads, page, dim, 1)
    v_pool, _, _, values = _cache(lens, kv_heads, page, dim, 1)
    v_pool, values = v_pool * -1.5, [v * -1.5 for v in values]
    q, cap = _rand((len(lens), heads, dim), 7), 1024 * (-(-max(lens) // 1024))
    if not kernels.attention_rows_supported(q, k_pool, kv_heads, cap):
        assert len(lens) == 9 and kv_heads == 8, "sizes that the kernel serves: all but these, whose warps would have four blocks of keys"
        return
    out = kernels.attention_rows(q, k_pool, v_pool, _i32(lens), indptr, indices, dim ** -0.5, cap).reshape(len(lens), heads, dim)
    for r, n in enumerate(lens):
        if n == 0:
            continue
        for h in range(heads):
            k, v = keys[r][:, h * kv_heads // heads].double(), values[r][:, h * kv_heads // heads].double()
            p = torch.softmax(k @ q[r, h].double() * dim ** -0.5, 0)
            # weights to 2^-17 and 32-bit sums, one rounding to bfloat16
            assert ((out[r, h].double() - p @ v).abs() <= 2.0 ** -15 * (p @ v.abs()) + 2.0 ** -8 * (p @ v).abs()).all(), (r, h)


@pytest.mark.parametrize("lens", ROWS)
@pytest.mark.parametrize("heads,kv_heads,dim,two", [(16, 4, 64, True), (8, 8, 128, False), (16, 1, 64, False)])
@pytest.mark.parametrize("gated", [False, True])
def test_sigmoid(kernels, lens, heads, kv_heads, dim, two, gated):
    page = 16
    pool, indptr, indices, both = _cache(lens, kv_heads, page, 2 * dim, 3)
    k_pool, v_pool = (pool[..., :dim].contiguous(), pool[..., dim:].contiguous()) if two else (pool, None)
    T = len(lens)
    q, slopes, bias = _rand((T, heads, dim), 8), torch.rand(heads).cuda() * 0.1, torch.randn(heads).cuda()
    gate = _rand((T, 8 + heads * dim), 9)
    cap = 1024 * (-(-max(lens) // 1024))
    positions = _i32([n - 1 for n in lens])
    before = kernels.launches
    out = kernels.sigmoid_attention(q, k_pool, v_pool, gate, 8 if gated else None, slopes, bias, positions, _i32(list(range(T))), indptr, indices, kv_heads, dim,
                                    dim ** -0.5, kv_cap=cap)
    if kernels.attention_rows_supported(q, k_pool, kv_heads, cap, sigmoid=True):
        assert kernels.launches == before + 1
    for r, n in enumerate(lens):
        if n == 0:
            continue
        for h in range(heads):
            x = both[r][:, h * kv_heads // heads].double()
            w = torch.sigmoid(x[:, :dim] @ q[r, h].double() * dim ** -0.5 - slopes[h].double() * torch.arange(n - 1, -1, -1, device="cuda") + bias[h].double())
            scale = torch.sigmoid(gate[r, 8 + h * dim : 8 + (h + 1) * dim].double()) if gated else 1.0
            want, size = w @ x[:, dim:] * scale, w @ x[:, dim:].abs() * scale
            # 32-bit weights and sums (products cut off, 2^-23 of the sum each, at most 3 a block of 16 keys and warp), one rounding
            assert ((out[r, h * dim : (h + 1) * dim].double() - want).abs() <= (2.0 ** -20 + n / 16 * 3 * 2.0 ** -23) * size + 2.0 ** -8 * want.abs()).all(), (r, h)


def _softmax_64(q, keys, values, heads, kv_heads):
    """[rows, heads, dim] of softmax(q k^T / sqrt(dim)) v in 64 bits."""
    out = torch.empty(q.shape, dtype=torch.float64, device="cuda")
    for r in range(q.shape[0]):
        for h in range(heads):
            k, v = keys[r][:, h * kv_heads // heads].double(), values[r][:, h * kv_heads // heads].double()
            out[r, h] = torch.softmax(k @ q[r, h].double() * q.shape[2] ** -0.5, 0) @ v
    return out


# one block of keys and one warp; a warp a block; several CTAs a row
@pytest.mark.parametrize("lens", [[9, 16, 12, 10], [100, 128, 40, 90], [300, 1000, 700, 513]])
@pytest.mark.parametrize("heads,kv_heads,dim", [(16, 4, 64), (16, 8, 128)])
def test_a_score_that_is_not_finite_reaches_the_output(kernels, lens, heads, kv_heads, dim):
    """A NaN score makes its row and head NaN, and so does one of +inf; -inf is a weight of zero. No other row or head sees them."""
    page, group = 16, heads // kv_heads
    k_pool, indptr, indices, keys = _cache(lens, kv_heads, page, dim, 1)
    v_pool, values = k_pool * -1.5, [k * -1.5 for k in keys]
    q = _rand((len(lens), heads, dim), 7)
    starts = indptr.tolist()

    def set_key(r, j, head, d, value):
        keys[r][j, head, d] = value
        k_pool[indices[starts[r] + j // page], head, j % page, d] = value

    q[0, 1] = float("nan")                                     # every score of a head
    set_key(1, 7, 1, 3, float("nan"))                          # a score of a group of heads
    q[2, :, 5] = -q[2, :, 5].abs() - 0.1
    set_key(2, 4, 0, 5, float("inf"))                          # a score of -inf
    q[3, :, 5] = q[3, :, 5].abs() + 0.1
    set_key(3, 8, 2, 5, float("inf"))                          # a score of +inf
    cap = 1024
    assert kernels.attention_rows_supported(q, k_pool, kv_heads, cap)
    out = kernels.attention_rows(q, k_pool, v_pool, _i32(lens), indptr, indices, dim ** -0.5, cap).reshape(len(lens), heads, dim)
    want = _softmax_64(q, keys, values, heads, kv_heads)
    assert torch.equal(torch.isnan(out), torch.isnan(want))
    assert torch.isnan(want[0, 1]).all() and torch.isnan(want[1, group : 2 * group]).all() and not torch.isnan(want[2]).any() and torch.isnan(want[3, 2 * group]).all()
    fine = torch.isfinite(want)
    # as above; what |v| a weight meets is below 8 here
    assert ((out.double() - want).abs()[fine] <= 2.0 ** -15 * 8 + 2.0 ** -8 * want.abs()[fine]).all()


@pytest.mark.parametrize("lens", [[9, 16], [300, 1000]])
def test_a_sigmoid_weight_that_is_not_a_number_reaches_the_output(kernels, lens):
    heads, kv_heads, dim, page = 8, 4, 64, 16
    k_pool, indptr, indices, _ = _cache(lens, kv_heads, page, dim, 1)
    v_pool = k_pool * -1.5
    q, T = _rand((len(lens), heads, dim), 7), len(lens)
    q[0, 3] = float("nan")
    k_pool[indices[indptr[1]], 1, 2, 9] = float("nan")          # key 2 of row 1, head 1
    out = kernels.sigmoid_attention(q, k_pool, v_pool, None, None, torch.zeros(heads, device="cuda"), torch.zeros(heads, device="cuda"), _i32([n - 1 for n in lens]),
                                    _i32(list(range(T))), indptr, indices, kv_heads, dim, dim ** -0.5, kv_cap=1024).reshape(T, heads, dim)
    want = torch.zeros((T, heads), dtype=torch.bool, device="cuda")
    want[0, 3], want[1, 2:4] = True, True
    assert torch.equal(torch.isnan(out), want[:, :, None].expand_as(out))


@pytest.mark.parametrize("lens", [[16, 9], [300, 1000]])
@pytest.mark.parametrize("sigmoid", [False, True])
def test_an_infinite_value_makes_its_column_infinite(kernels, lens, sigmoid):
    """A weight is the sum of two or three numbers, of which the small ones may be zero or negative: an infinite value meets the largest alone."""
    heads, kv_heads, dim, page = 8, 4, 64, 16
    k_pool, indptr, indices, keys = _cache(lens, kv_heads, page, dim, 1)
    v_pool, values = k_pool * -1.5, [k * -1.5 for k in keys]
    q, T = _rand((len(lens), heads, dim), 7), len(lens)
    for r, j, head, d, x in ((0, 2, 0, 5, "inf"), (0, 7, 1, 60, "-inf"), (1, 4, 2, 0, "inf"), (1, 3, 3, 9, "inf"), (1, 8, 3, 9, "-inf")):
        values[r][j, head, d] = float(x)
        v_pool[indices[indptr[r]], head, j, d] = float(x)
    if sigmoid:
        zeros = torch.zeros(heads, device="cuda")
        out = kernels.sigmoid_attention(q, k_pool, v_pool, None, None, zeros, zeros, _i32([n - 1 for n in lens]), _i32(list(range(T))), indptr, indices, kv_heads, dim,
                                        dim ** -0.5, kv_cap=1024).reshape(T, heads, dim)
        want = torch.stack([torch.stack([torch.sigmoid(keys[r][:, h // 2].double() @ q[r, h].double() * dim ** -0.5) @ values[r][:, h // 2].double()
                                         for h in range(heads)]) for r in range(T)])
    else:
        out = kernels.attention_rows(q, k_pool, v_pool, _i32(lens), indptr, indices, dim ** -0.5, 1024).reshape(T, heads, dim)
        want = _softmax_64(q, keys, values, heads, kv_heads)
    assert torch.equal(torch.isnan(out), torch.isnan(want)) and torch.isinf(want).any() and torch.isnan(want).any()
    assert torch.equal(out[torch.isinf(want)].double(), want[torch.isinf(want)])
    fine = torch.isfinite(want)
    # one rounding; 32-bit weights (2^-15 of the sum of |v|, which is below 2 a key here) and sums
    assert ((out.double() - want).abs()[fine] <= 2.0 ** -15 * 2 * max(lens) + 2.0 ** -8 * want.abs()[fine]).all()


def test_rows_longer_than_the_bound_that_was_told(kernels):
    """More blocks of keys than a warp reads table entries for at a time: slower, and right all the same."""
    lens, heads, kv_heads, dim, page = [5000, 17], 4, 2, 64, 16
    k_pool, indptr, indices, keys = _cache(lens, kv_heads, page, dim, 1)
    q = _rand((len(lens), heads, dim), 7)
    out = kernels.attention_rows(q, k_pool, k_pool * -1.5, _i32(lens), indptr, indices, dim ** -0.5, 16).reshape(len(lens), heads, dim)
    want = _softmax_64(q, keys, [k * -1.5 for k in keys], heads, kv_heads)
    # as above; what |v| a weight meets is below 8 here
    assert ((out.double() - want).abs() <= 2.0 ** -15 * 8 + 2.0 ** -8 * want.abs()).all()
