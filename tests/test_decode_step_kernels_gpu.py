"""Kernels of a step of few rows whose inputs are in registers ahead of the kernel in front, against 64 bits: the rotation of few tokens, the norms over a
32-bit stream, the states that begin at zero."""
import math

import pytest
import torch

from roost_b200.kernels import library

pytestmark = pytest.mark.gpu
F64 = torch.float64


@pytest.fixture(scope="module")
def kernels():
    return library.load()


def _rand(shape, seed, dtype=torch.float32):
    return torch.randn(shape, generator=torch.Generator().manual_seed(seed)).to(dtype).cuda()


@pytest.mark.parametrize("hidden", [4, 1020, 2048, 2052, 4100, 8192])
@pytest.mark.parametrize("form", ["norm", "add", "extra", "rows", "gate", "sum"])
def test_norm_over_a_32_bit_stream(kernels, hidden, form):
    n = 5
    stream, w = _rand((n, hidden), 1), 1 + 0.1 * _rand((hidden,), 2)
    addend, extra, gate, bias = _rand((n, hidden), 3, torch.bfloat16), _rand((n, hidden), 4), _rand((n, hidden), 5), _rand((hidden,), 6)
    rows = torch.tensor([4, 0], dtype=torch.int32, device="cuda") if form == "rows" else None
    s = stream.to(F64)
    if form == "gate":
        s = s + addend.to(F64) * torch.sigmoid(gate.to(F64) + bias.to(F64))
        kept = stream.clone()
        out = kernels.wide_rms_norm_gated(kept, w, 1e-6, torch.bfloat16, addend, gate, bias)
    else:
        if form in ("add", "extra", "rows", "sum"):
            s = s + addend.to(F64)
        if form == "extra":
            s = s + extra.to(F64)
        kept = stream.clone()
        out = kernels.wide_rms_norm(kept, None if form == "sum" else w, 1e-6, torch.bfloat16, None if form == "norm" else addend, extra if form == "extra" else None, rows)
    assert torch.equal(kept, stream) if form in ("norm", "rows") else (kept.to(F64) - s).abs().max() <= 2.0 ** -21 * s.abs().max()
    want = s if form == "sum" else s / torch.sqrt((s * s).mean(-1, keepdim=True) + 1e-6) * w.to(F64)
    want = want if rows is None else want[rows.long()]
    # one rounding to bfloat16 beside sums in 32 bits
    assert ((out.to(F64) - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -18).all()


# where long rows change to the kernel for any sizes: one, two, four pieces a thread
@pytest.mark.parametrize("hidden,gated,n", [(1024, True, 1025), (1028, True, 1024), (1028, True, 1025), (4096, True, 512), (4096, True, 513), (4096, False, 700),
                                            (4100, False, 256), (4100, False, 257), (8192, True, 148), (8192, True, 149)])
def test_norm_over_a_32_bit_stream_of_many_rows(kernels, hidden, gated, n):
    stream, w = _rand((n, hidden), 1), 1 + 0.1 * _rand((hidden,), 2)
    addend, gate, bias = _rand((n, hidden), 3, torch.bfloat16), _rand((n, hidden), 5), _rand((hidden,), 6)
    s = stream.to(F64) + addend.to(F64) * (torch.sigmoid(gate.to(F64) + bias.to(F64)) if gated else 1.0)
    out = kernels.wide_rms_norm_gated(stream, w, 1e-6, torch.bfloat16, addend, gate, bias) if gated else kernels.wide_rms_norm(stream, w, 1e-6, torch.bfloat16, addend)
    want = s / torch.sqrt((s * s).mean(-1, keepdim=True) + 1e-6) * w.to(F64)
    assert (stream.to(F64) - s).abs().max() <= 2.0 ** -21 * s.abs().max()
    # one rounding to bfloat16 beside sums in 32 bits
    assert ((out.to(F64) - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -18).all()


@pytest.mark.parametrize("dim", [64, 128, 256])
@pytest.mark.parametrize("tokens,heads,kv_heads", [(1, 1, 1), (7, 5, 1), (63, 8, 4)])
@pytest.mark.parametrize("normed", [True, False])
def test_rotation_of_few_tokens(kernels, dim, tokens, heads, kv_heads, normed):
    page, pages, half = 16, 6, dim // 2
    qkv = _rand((tokens, (heads + 2 * kv_heads) * dim), 7, torch.bfloat16)
    qw, kw = ((1 + 0.1 * _rand((dim,), s)).bfloat16() for s in (8, 9))
    positions = torch.arange(tokens, dtype=torch.int32) * 997
    slots = torch.randperm(page * pages, generator=torch.Generator().manual_seed(1))[:tokens].int()
    slots[tokens // 2] = -1 if tokens > 1 else slots[0]
    inv = torch.pow(torch.tensor(1e6, dtype=F64), -2.0 * torch.arange(half, dtype=F64) / dim).cuda()
    kp, vp = (torch.full((pages, kv_heads, page, dim), 7.0, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    q = kernels.qk_norm_rope_cache(qkv, heads, kv_heads, dim, q_w=qw if normed else None, k_w=kw if normed else None, eps=1e-6, inv_freq=inv, rotary_dim=dim,
                                   positions=positions.cuda(), k_pool=kp, v_pool=vp, slot_mapping=slots.cuda(), page_size=page)
    x = qkv.to(F64).reshape(tokens, heads + 2 * kv_heads, dim)
    ang = (positions.to(F64).cuda()[:, None] * inv)[:, None]

    def turned(y, w):
        if normed:
            y = y / torch.sqrt((y * y).mean(-1, keepdim=True) + 1e-6) * w.to(F64)
        a, b = y[..., :half], y[..., half:]
        return torch.cat([a * torch.cos(ang) - b * torch.sin(ang), b * torch.cos(ang) + a * torch.sin(ang)], -1)

    def close(got, want):      # one rounding; angles of 32 bits after their reduction
        assert ((got.to(F64) - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -18 * want.abs().max()).all()

    close(q.reshape(tokens, heads, dim), turned(x[:, :heads], qw))
    keys = turned(x[:, heads : heads + kv_heads], kw)
    for t, slot in enumerate(slots.tolist()):
        if slot >= 0:
            close(kp[slot // page, :, slot % page], keys[t])
            assert torch.equal(vp[slot // page, :, slot % page], qkv.reshape(tokens, -1, dim)[t, heads + kv_heads :])
    written = {s for s in slots.tolist() if s >= 0}
    for s in set(range(page * pages)) - written:
        assert (kp[s // page, :, s % page] == 7).all() and (vp[s // page, :, s % page] == 7).all()


@pytest.mark.parametrize("dtype,width", [(torch.float32, 5000), (torch.float32, 3), (torch.bfloat16, 7)])
def test_states_that_begin_are_zero_and_no_other(kernels, dtype, width):
    state = _rand((3, 6, width), 10, dtype)
    state[:, 2] = float("nan")                                  # what a finished request left
    before = state.clone()
    slots, fresh = (torch.tensor(v, dtype=torch.int32, device="cuda") for v in ([4, 2, 0, 6, -1], [0, 1, 1, 1, 1]))
    kernels.zero_slots(state, slots, fresh)
    assert (state[:, [0, 2]] == 0).all() and torch.equal(state[:, [1, 3, 4, 5]], before[:, [1, 3, 4, 5]])
