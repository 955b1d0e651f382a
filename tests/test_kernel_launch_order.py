"""What the order of dependent kernels rests on, read from their sources: a grid launched with programmatic serialisation orders the kernels
behind it only if it has itself waited for the ones ahead."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "roost_b200" / "csrc"


def _kernels(path):
    """(name, body) of every kernel, comments blanked."""
    src = re.sub(r"//[^\n]*", "", path.read_text())
    for m in re.finditer(r"__global__", src):
        start = src.index("{", m.end())
        if ";" in src[m.end() : start]:
            continue                                    # a declaration
        depth, at = 0, start
        while True:
            depth += {"{": 1, "}": -1}.get(src[at], 0)
            if depth == 0:
                break
            at += 1
        head = re.sub(r"__launch_bounds__\s*\((?:[^()]|\([^()]*\))*\)", "", src[m.end() : start])
        yield re.search(r"(\w+)\s*\(", head).group(1), src[start : at + 1]


def _returns_without_waiting(body):
    """Bare returns ahead of the kernel's own wait that do not wait themselves."""
    body = re.sub(r"pdl_wait\(\d*\)\s*;\s*return\s*;", "", body)
    own = re.search(r"pdl_wait\(\d*\)", body)
    return re.findall(r"[^\n]*\breturn\s*;", body[: own.start()] if own else body)


FILES = sorted(CSRC.glob("*.cu")) + sorted(CSRC.glob("*.cuh"))


@pytest.mark.parametrize("path", FILES, ids=lambda p: p.name)
def test_no_block_of_a_dependent_kernel_returns_before_it_has_waited(path):
    """All blocks of a first walk return at once where no row has a second segment. Were they not to wait, the grid would be over before the
    kernels ahead of it, and the wait of the kernel behind it, which covers that grid alone, would order nothing."""
    for name, body in _kernels(path):
        if "pdl_wait(" in body:
            assert not _returns_without_waiting(body), f"{path.name}: {name} returns before pdl_wait()"


def _recurrent_layer(kind):
    from roost_b200.config.spec import GatedLinearAttentionSpec, Mamba1Spec, Mamba2Spec
    return {"mamba2": lambda: Mamba2Spec(hidden=1024, num_heads=32, head_dim=64, state=128, groups=1, conv_taps=4, norm_groups=1, eps=1e-6),
            "mamba1": lambda: Mamba1Spec(hidden=1024, inner=2048, state=16, dt_rank=64, conv_taps=4),
            "gla": lambda: GatedLinearAttentionSpec(hidden=1024, num_heads=8, head_dim=64, v_dim=128, tau=16.0, decay_rank=16, eps=1e-6)}[kind]()


@pytest.mark.gpu
@pytest.mark.parametrize("kind,rows,tokens", [("mamba2", 8, 200), ("mamba2", 2, 250), ("mamba1", 40, 60), ("gla", 24, 60)])
def test_a_layer_whose_rows_are_one_segment_each_gives_the_same_bits_with_and_without_overlap(kernels, kind, rows, tokens):
    """The first walk and the carry have nothing to do there; the layer's outputs and states must not depend on whether kernels overlap. Another
    input every time: what a kernel read too early would be the values of the pass before."""
    import torch

    from roost_b200.cache.manager import CacheManager, build_groups
    from roost_b200.cache.storage import CacheStorage
    from roost_b200.engine.batch import BatchBuilder
    from roost_b200.parts import Runtime
    from roost_b200.parts.base import MIXERS
    spec = _recurrent_layer(kind)
    part = MIXERS.build(spec, Runtime(torch.bfloat16, "cuda", kernels))
    g = torch.Generator().manual_seed(rows)
    draw = lambda d: (torch.empty(d.shape).uniform_(d.init[1], d.init[2], generator=g) if d.init and d.init[0] == "uniform" else   # noqa: E731
                      torch.randn(d.shape, generator=g) * (d.init[2] if d.init else 0.02 if d.role == "matrix" else 0.1) +
                      (d.init[1] if d.init else 0.0 if d.role == "matrix" else 1.0)).to(torch.bfloat16).cuda()
    part.load({k: draw(d) for k, d in sorted(MIXERS.get(spec.kind).parameters(spec).items())})
    groups = build_groups([part.cache_need()], 16)
    manager = CacheManager(groups, [rows])
    storage = CacheStorage(groups, [p.capacity for p in manager.pools], torch.bfloat16, "cuda")
    batch = BatchBuilder("cuda", manager).build([(manager.extend(r, tokens), 0, [0] * tokens, []) for r in range(rows)], 1)
    cache = storage.view(0)
    inputs = [torch.randn(rows * tokens, 1024, generator=g).to(torch.bfloat16).cuda() for _ in range(6)]
    got, was = {}, kernels.pdl
    try:
        for pdl in (False, True):
            kernels.set_pdl(pdl)
            cache.state.zero_()
            got[pdl] = [(part(x, batch, cache).clone(), cache.state[:-1].clone()) for x in inputs]
            torch.cuda.synchronize()
    finally:
        kernels.set_pdl(was)
    for (y, s), (y2, s2) in zip(got[False], got[True]):
        assert torch.isfinite(y).all() and torch.equal(y, y2) and torch.equal(s, s2)


def test_the_header_names_the_tables_that_are_read_ahead_of_the_wait():
    """A caller's kernel must not be writing them: the ABI's contract of programmatic launch has to name each."""
    header = (CSRC / "roost_kernels.h").read_text()
    contract = re.search(r"/\* Programmatic dependent launch.*?\*/", header, re.S).group(0)
    early = set()
    for path in FILES:
        src = re.sub(r"//[^\n]*", "", path.read_text())
        for name, body in _kernels(path):
            wait = re.search(r"pdl_wait\(\d*\)", body)
            if not wait:
                continue
            head = src[: src.index(body)][-2000:]
            for table in re.findall(r"const int32_t\*\s*(?:__restrict__\s*)?(\w+)", head[head.rindex(name) :]):
                if re.search(rf"\b{table}\[", body[: wait.start()]):
                    early.add((path.name, name, table))
    assert any(table == "positions" for _, _, table in early)
    assert not {e for e in early if e[2] not in contract}
