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
        assert len(lens) * kv_heads > 18, "sizes that the kernel serves"
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
