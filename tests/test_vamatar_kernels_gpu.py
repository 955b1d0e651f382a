"""The kernels of the Vamatar parts on the device, each against the plain formula, and the forms a step chooses between
against one another (split keys against one block a token, a warp an output against tiles of rows); sizes of every
register class of the scan kernel; the replay tool on a Vamatar folder."""
import json
import subprocess
import sys

import numpy as np
import pytest
import torch

from roost_b200.engine.executor import StepEntry, StepExecutor
from roost_b200.kernels import library
from tests import helpers as H
from tests import vamatar_models as VM
from tests.conftest import ROOT
from tests.plain import vamatar_plain as P

pytestmark = pytest.mark.gpu
DTYPES = [torch.float32, torch.bfloat16]


def close(got, want, dtype, what, f32=2e-5, bf16=2e-2):
    err = H.scaled_error(got.float(), want)
    print(f"MEASURED {what} {dtype}: {err:.3e}")
    assert err < (f32 if dtype == torch.float32 else bf16), (what, err)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("hidden", [20, 352, 4096])
def test_layer_norm_over_a_32_bit_stream(kernels, dtype, hidden):
    g = torch.Generator().manual_seed(hidden)
    stream = (torch.randn(9, hidden, generator=g) * 3 + 1).cuda()
    addend = torch.randn(9, hidden, generator=g).to(dtype).cuda()
    w, b = torch.randn(hidden, generator=g).cuda(), torch.randn(hidden, generator=g).cuda()
    want_sum = stream.double().cpu() + addend.double().cpu()
    want = P.layer_norm(want_sum, w.double().cpu(), b.double().cpu(), 1e-5)
    rows = torch.tensor([7, 0, 3], dtype=torch.int32).cuda()
    before = stream.clone()
    gathered = kernels.layer_norm(stream, w, b, 1e-5, dtype, addend, rows)
    assert torch.equal(stream, before)                  # gathered rows leave the stream as it is
    close(gathered, want[[7, 0, 3]], dtype, "layer norm of gathered rows")
    out = kernels.layer_norm(stream, w, b, 1e-5, dtype, addend)
    close(out, want, dtype, "add + layer norm")
    assert H.scaled_error(stream, want_sum) < 1e-6      # the stream holds the 32-bit sum, not a rounded one
    close(kernels.layer_norm(stream, w, b, 1e-5, dtype), want, dtype, "layer norm alone")


def test_scaled_embedding_and_capped_logits(kernels):
    table = torch.randn(30, 24).to(torch.bfloat16).cuda()
    ids = torch.tensor([3, 29, 0, 3], dtype=torch.int32).cuda()
    out = kernels.embedding_scaled(table, ids, 0.3)
    assert out.dtype == torch.float32 and torch.equal(out.cpu(), table.float().cpu()[ids.long().cpu()] * torch.tensor(0.3))
    z = (torch.randn(5, 77) * 30).cuda()
    want = 12.0 * torch.tanh(z.double().cpu() / 12.0)
    assert H.scaled_error(kernels.softcap_(z.clone(), 12.0), want) < 1e-6


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("window", [None, 37])
def test_latent_attention_with_split_keys_against_the_plain_sum(kernels, dtype, window):
    """Three rows of unequal length, one token each at the end of 5, 130 and 260 cached entries on pages of 8 handed out in
    a scrambled order; the keys of a token dealt to several blocks (a decode step of few rows) and to one."""
    heads, nope, rope, rank, page = 5, 8, 6, 20, 8
    g = torch.Generator().manual_seed(3)
    lens = [5, 130, 260]
    n_pages = sum(-(-n // page) for n in lens)
    order = torch.randperm(n_pages, generator=g).tolist()
    pool = torch.zeros(n_pages, 1, page, rank + rope)
    entries, tables = [], []
    for n in lens:
        e = torch.randn(n, rank + rope, generator=g)
        mine = [order.pop() for _ in range(-(-n // page))]
        for j in range(n):
            pool[mine[j // page], 0, j % page] = e[j]
        entries.append(e)
        tables.append(mine)
    pool = pool.to(dtype).cuda()
    T = len(lens)
    q_latent = torch.randn(heads, T, rank, generator=g).to(dtype).cuda()
    q = torch.randn(T, heads * (nope + rope), generator=g).to(dtype).cuda()
    positions = torch.tensor([n - 1 for n in lens], dtype=torch.int32).cuda()
    token_row = torch.arange(T, dtype=torch.int32).cuda()
    indptr = torch.tensor([0] + list(np.cumsum([len(t) for t in tables])), dtype=torch.int32).cuda()
    indices = torch.tensor([p for t in tables for p in t], dtype=torch.int32).cuda()
    scale = 0.21
    want = torch.zeros(heads, T, rank, dtype=torch.float64)
    for t, n in enumerate(lens):
        lo = 0 if window is None else max(0, n - window)
        e = pool[:, 0].reshape(-1, rank + rope).double().cpu()
        rows = torch.stack([e[tables[t][j // page] * page + j % page] for j in range(lo, n)])
        qr = q[t].double().cpu().reshape(heads, nope + rope)[:, nope:]
        s = (q_latent[:, t].double().cpu() @ rows[:, :rank].T + qr @ rows[:, rank:].T) * scale
        want[:, t] = torch.softmax(s, -1) @ rows[:, :rank]
    args = (q_latent, q, pool, positions, token_row, indptr, indices, heads, nope, rope, rank, scale, window)
    one = kernels.latent_attention(*args, 0)
    split = kernels.latent_attention(*args, 1024, True)
    assert kernels.latent_splits_for(T, heads, window, 1024) > 1
    close(one, want, dtype, "latent attention, one block a token", bf16=1e-2)
    close(split, want, dtype, "latent attention, split keys", bf16=1e-2)
    # more splits than this library's caller asks for, as the entry point takes them: another merge
    for splits in (32, 33, 70):
        out, part = torch.empty_like(one), torch.empty(T * heads * splits * (rank + 2), device="cuda")
        ptr, stream = library._ptr, library._stream()
        kernels._call("roost_latent_attention", ptr(q_latent), ptr(q), ptr(out), ptr(part), ptr(pool), ptr(positions), ptr(token_row), ptr(indptr), ptr(indices), T, heads,
                      nope, rope, rank, page, scale, window or 0, splits, None, library.dtype_code(dtype), stream, launches=2)
        close(out, want, dtype, f"latent attention, {splits} splits", bf16=1e-2)


@pytest.mark.parametrize("rank", [32, 80, 272])
@pytest.mark.parametrize("window", [None, 37])
def test_latent_attention_on_the_tensor_cores_against_the_plain_sum(kernels, rank, window):
    """Portions of three requests in one step (77 tokens after 60 cached ones, 5 from the start, 140 after 3), five heads, so
    that the packed (token, head) rows of a tile span several tokens with windows of their own; pages of 8 in a scrambled
    order; with a window the pages it has passed are gone from the block tables (-1)."""
    heads, nope, rope, page = 5, 8, 8, 8
    g = torch.Generator().manual_seed(rank)
    spans = [(60, 77), (0, 5), (3, 140)]
    totals = [a + n for a, n in spans]
    n_pages = sum(-(-n // page) for n in totals)
    order = torch.randperm(n_pages, generator=g).tolist()
    pool = torch.zeros(n_pages, 1, page, rank + rope)
    tables, entries = [], []
    for (start, n), total in zip(spans, totals):
        e = torch.randn(total, rank + rope, generator=g)
        mine = [order.pop() for _ in range(-(-total // page))]
        for j in range(total):
            pool[mine[j // page], 0, j % page] = e[j]
        if window:            # pages wholly before the first query's window are given back
            for i in range(max(0, start - window + 1) // page):
                pool[mine[i]] = float("nan")
                mine[i] = -1
        entries.append(e)
        tables.append(mine)
    pool = pool.to(torch.bfloat16).cuda()
    T = sum(n for _, n in spans)
    q_latent = torch.randn(heads, T, rank, generator=g)
    if window:
        # two queries of the first request made to score one key far above the rest: the oldest key its window keeps (position
        # 100 sees 64..100), and the first key its window has dropped (position 110 sees 74..110, not 73); a window one off
        # turns either result into another
        q_latent[:, 40] = 2.0 * entries[0][100 - window + 1, :rank]
        q_latent[:, 50] = 2.0 * entries[0][110 - window, :rank]
    q_latent = q_latent.to(torch.bfloat16).cuda()
    q = torch.randn(T, heads * (nope + rope), generator=g).to(torch.bfloat16).cuda()
    positions = torch.tensor([start + i for start, n in spans for i in range(n)], dtype=torch.int32).cuda()
    token_row = torch.tensor([b for b, (_, n) in enumerate(spans) for _ in range(n)], dtype=torch.int32).cuda()
    q_indptr = torch.tensor([0] + list(np.cumsum([n for _, n in spans])), dtype=torch.int32).cuda()
    indptr = torch.tensor([0] + list(np.cumsum([len(t) for t in tables])), dtype=torch.int32).cuda()
    indices = torch.tensor([p for t in tables for p in t], dtype=torch.int32).cuda()
    scale = 0.3
    want = torch.zeros(heads, T, rank, dtype=torch.float64)
    t = 0
    for b, (start, n) in enumerate(spans):
        e = entries[b].to(torch.bfloat16).double()
        for i in range(n):
            pos = start + i
            lo = 0 if window is None else max(0, pos - window + 1)
            rows = e[lo : pos + 1]
            qr = q[t].double().cpu().reshape(heads, nope + rope)[:, nope:]
            sc = (q_latent[:, t].double().cpu() @ rows[:, :rank].T + qr @ rows[:, rank:].T) * scale
            want[:, t] = torch.softmax(sc, -1) @ rows[:, :rank]
            t += 1
    got = kernels.latent_attention(q_latent, q, pool, positions, token_row, indptr, indices, heads, nope, rope, rank, scale, window, 1024,
                                   False, q_indptr)
    assert kernels._lib.roost_latent_attention_tc_supported(nope, rope, rank) and T * heads >= kernels.LATENT_TC_MIN_ROWS
    close(got, want, torch.bfloat16, f"latent attention on the tensor cores, rank {rank}", bf16=1.5e-2)
    slow = kernels.latent_attention(q_latent, q, pool, positions, token_row, indptr, indices, heads, nope, rope, rank, scale, window, 0)
    close(slow, want, torch.bfloat16, "the 32-bit form on the same step", bf16=1e-2)


@pytest.mark.parametrize("dtype", DTYPES)
def test_routing_chooses_the_largest_scores_and_sorts_the_pairs_by_expert(kernels, dtype):
    T, E, top, hidden, ff = 50, 9, 3, 24, 16
    g = torch.Generator().manual_seed(9)
    logits = torch.randn(T, E, generator=g) * 3
    logits[4, 2] = logits[4, 6] = logits[4].max() + 1          # a tie goes to the lower index
    route = kernels.moe_route(logits.cuda(), top)
    token, expert, weight, inverse = route.token.cpu(), route.expert.cpu(), route.weight.cpu(), route.inverse.cpu().long()
    assert torch.equal(expert, expert.sort().values)            # sorted by expert
    offsets = route.offsets.cpu()
    assert int(offsets[-1]) == T * top and all(int((expert == e).sum()) == int(offsets[e + 1] - offsets[e]) for e in range(E))
    for t in range(T):
        want = sorted(range(E), key=lambda e: (-float(logits[t, e]), e))[:top]
        assert [int(expert[inverse[t * top + k]]) for k in range(top)] == want
        assert all(int(token[inverse[t * top + k]]) == t for k in range(top))
        for k, e in enumerate(want):
            assert abs(float(weight[inverse[t * top + k]]) - float(torch.sigmoid(logits[t, e].double()))) < 1e-6
    tiles = route.tiles.cpu().reshape(-1, 3)
    covered = sorted((int(a), int(b)) for e, a, b in tiles if e >= 0)
    assert covered[0][0] == 0 and covered[-1][1] == T * top and all(x[1] == y[0] for x, y in zip(covered, covered[1:]))
    # the expert products in both forms, and the sum
    x = torch.randn(T, hidden, generator=g).to(dtype).cuda()
    wg, wu = (torch.randn(E, ff, hidden, generator=g) * 0.3).to(dtype).cuda(), (torch.randn(E, ff, hidden, generator=g) * 0.3).to(dtype).cuda()
    wd = (torch.randn(E, hidden, ff, generator=g) * 0.3).to(dtype).cuda()
    shared = torch.randn(T, hidden, generator=g).to(dtype).cuda()
    xs = kernels.moe_gather_scale(x, route)
    outs = []
    for form in (0, 1):
        a = torch.empty(T * top, ff, dtype=dtype, device="cuda")
        kernels._call("roost_moe_expert_gemm", xs.data_ptr(), wg.data_ptr(), wu.data_ptr(), a.data_ptr(), route.tiles.data_ptr(), route.max_tiles,
                      route.expert.data_ptr(), T * top, ff, hidden, form, 0, 0, 0.0, 1 << 30, 0 if dtype == torch.float32 else 1, torch.cuda.current_stream().cuda_stream)
        y = torch.empty(T * top, hidden, dtype=dtype, device="cuda")
        kernels._call("roost_moe_expert_gemm", a.data_ptr(), wd.data_ptr(), None, y.data_ptr(), route.tiles.data_ptr(), route.max_tiles,
                      route.expert.data_ptr(), T * top, hidden, ff, form, 0, 0, 0.0, 1 << 30, 0 if dtype == torch.float32 else 1, torch.cuda.current_stream().cuda_stream)
        outs.append(kernels.moe_combine(y, route, shared))
    want = shared.double().cpu().clone()
    xd = x.double().cpu()
    for t in range(T):
        for e in sorted(range(E), key=lambda e: (-float(logits[t, e]), e))[:top]:
            xin = (torch.sigmoid(logits[t, e].double()) * xd[t])[None]
            w = {"gate": wg[e].double().cpu(), "up": wu[e].double().cpu(), "down": wd[e].double().cpu()}
            want[t] += P.gated_ff(xin, w, "")[0]
    close(outs[0], want, dtype, "experts on tiles of rows", bf16=4e-2)
    close(outs[1], want, dtype, "experts, a warp an output", bf16=4e-2)


def test_experts_on_tcgen05_for_steps_of_many_rows(kernels):
    """1,230 sorted rows over 9 experts of unequal load (one expert gets no row at all): the grouped tcgen05 product with the
    activation on its accumulator, and the down product, against the tiles on mma.sync and against the plain formula."""
    from roost_b200.kernels.library import MOE_TCGEN05_MIN_ROWS
    T, E, top, hidden, ff = 410, 9, 3, 192, 256
    g = torch.Generator().manual_seed(12)
    logits = torch.randn(T, E, generator=g) * 2
    logits[:, 4] = -50.0                                    # nobody chooses expert 4
    logits[:200, 7] += 6.0                                  # and many choose expert 7: several tiles of one expert
    route = kernels.moe_route(logits.cuda(), top)
    assert T * top >= MOE_TCGEN05_MIN_ROWS and route.wide_tiles is not None
    x = torch.randn(T, hidden, generator=g).to(torch.bfloat16).cuda()
    wg = (torch.randn(E, ff, hidden, generator=g) * 0.15).to(torch.bfloat16).cuda()
    wu = (torch.randn(E, ff, hidden, generator=g) * 0.15).to(torch.bfloat16).cuda()
    wd = (torch.randn(E, hidden, ff, generator=g) * 0.15).to(torch.bfloat16).cuda()
    gate_up = torch.stack([wg.reshape(E, ff // 128, 128, hidden), wu.reshape(E, ff // 128, 128, hidden)], dim=2).reshape(E, 2 * ff, hidden).contiguous()
    xs = kernels.moe_gather_scale(x, route)
    act_tc = kernels.moe_expert_gate_up(xs, wg, wu, route, gate_up)
    act_mma = kernels._moe_gemm(xs, wg, wu, route)
    assert H.scaled_error(act_tc.float(), act_mma.double().cpu()) < 2e-2
    # the interleaved tensor read by the other forms: tiles on mma.sync, tiles on FFMA, a warp an output (few rows)
    assert torch.equal(kernels._moe_gemm(xs, gate_up, None, route, block=128), act_mma)
    few = kernels.moe_route(logits[:10].cuda(), top)
    xs_few = kernels.moe_gather_scale(x[:10], few)
    assert H.scaled_error(kernels._moe_gemm(xs_few, gate_up, None, few, block=128).float(), kernels._moe_gemm(xs_few, wg, wu, few).double().cpu()) < 1e-6
    f32 = lambda t: t.float()
    assert H.scaled_error(kernels._moe_gemm(f32(xs_few), f32(gate_up), None, few, block=128), kernels._moe_gemm(f32(xs_few), f32(wg), f32(wu), few).double().cpu()) < 1e-6
    y_tc = kernels.moe_expert_down(act_mma, wd, route)
    y_mma = kernels._moe_gemm(act_mma, wd, None, route)
    assert H.scaled_error(y_tc.float(), y_mma.double().cpu()) < 2e-2
    kernels.check_device_status()
    expert, xs_c = route.expert.cpu(), xs.double().cpu()
    for row in (0, 1, 127, 128, 129, 700, T * top - 1):
        e = int(expert[row])
        w = {"gate": wg[e].double().cpu(), "up": wu[e].double().cpu(), "down": wd[e].double().cpu()}
        gv, uv = xs_c[row] @ w["gate"].T, xs_c[row] @ w["up"].T
        assert H.scaled_error(act_tc[row].float(), P.silu(gv) * uv) < 2e-2, row


@pytest.mark.parametrize("state,vdim", [(100, 24), (200, 40), (3, 128)])
def test_the_recurrence_at_sizes_of_every_register_class(tmp_path, state, vdim):
    cfg = VM.config([(VM.mamba(heads=2, vdim=vdim, state=state, groups=2, conv=4, norm_groups=1), None)], width=48, vocab=31, cap=None)
    tensors = VM.draw_tensors(cfg, state)
    folder = VM.write_model(tmp_path, cfg, tensors)
    model = H.make_model(folder, torch.float32, "gpu")
    ex = StepExecutor(model, page_size=4, num_pages=8, max_requests=2)
    ids = H.random_ids(45, cfg["vocab"], 1)
    got = torch.cat([ex.step([StepEntry("r", ids[:20], list(range(20)))]), ex.step([StepEntry("r", ids[20:22], [0, 1])])] +
                    [ex.step([StepEntry("r", [t], [0])]) for t in ids[22:]])
    want = P.forward(cfg, VM.plain_weights(tensors), ids)
    assert H.scaled_error(got, want) < 2e-4 and H.rms_error(got, want) < 3e-5


@pytest.mark.parametrize("dtype", DTYPES)
def test_long_rows_cut_into_chunks_that_run_side_by_side(tmp_path, kernels, dtype):
    """A step of 700 + 41 + 130 tokens (three requests, the second and third continuing earlier portions) is long enough for
    the recurrence to cut its rows into chunks: the states the chunks start from, the carried state of each request and the
    decoding that follows must be those of a walk token by token."""
    cfg = VM.config([(VM.mamba(heads=4, vdim=32, state=64, groups=2, conv=4, norm_groups=2), None),
                     (VM.mamba(heads=2, vdim=16, state=16, groups=1, conv=3, norm_groups=1), VM.dense(ff=32))], width=64, vocab=90, cap=None)
    tensors = VM.draw_tensors(cfg, 31)
    folder = VM.write_model(tmp_path, cfg, tensors)
    model = H.make_model(folder, dtype, "gpu")
    ex = StepExecutor(model, page_size=16, num_pages=8, max_requests=3)
    a, b, c = H.random_ids(703, cfg["vocab"], 1), H.random_ids(60, cfg["vocab"], 2), H.random_ids(140, cfg["vocab"], 3)
    assert sum(map(len, (a[:700], b[16:57], c[7:137]))) >= kernels.SCAN_CHUNKED_MIN_TOKENS
    ex.step([StepEntry("b", b[:16], []), StepEntry("c", c[:7], [])])
    out = ex.step([StepEntry("a", a[:700], [0, 127, 128, 699]), StepEntry("b", b[16:57], [40]), StepEntry("c", c[7:137], [0, 129])])
    tail = [ex.step([StepEntry("a", [a[700 + i]], [0]), StepEntry("b", [b[57 + i]], [0]), StepEntry("c", [c[137 + i]], [0])]) for i in range(3)]
    w = VM.plain_weights(tensors)
    wa, wb, wc = P.forward(cfg, w, a), P.forward(cfg, w, b), P.forward(cfg, w, c)
    want = torch.cat([wa[[0, 127, 128, 699]], wb[[56]], wc[[7, 136]]] + [torch.stack([wa[700 + i], wb[57 + i], wc[137 + i]]) for i in range(3)])
    got = torch.cat([out] + tail)
    err, rms = H.scaled_error(got, want), H.rms_error(got, want)
    print(f"MEASURED chunked recurrence {dtype}: worst {err:.3e}, rms {rms:.3e}")
    assert (err < 1e-4 and rms < 1e-5) if dtype == torch.float32 else (err < 0.25 and rms < 0.04)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_the_replay_tool_on_a_vamatar_folder(tmp_path, dtype):
    cfg = VM.WIDE
    tensors = VM.draw_tensors(cfg, 8)
    folder = VM.write_model(tmp_path / "model", cfg, tensors)
    a, b = H.random_ids(70, cfg["vocab"], 1), H.random_ids(41, cfg["vocab"], 2)
    steps = [{"step": 0, "entries": [{"id": "a", "tokens": a[:33], "want": [0, 32]}], "end": []},
             {"step": 1, "entries": [{"id": "b", "tokens": b[:2], "want": []}], "end": []},
             {"step": 2, "entries": [{"id": "a", "tokens": a[33:69], "want": [35]}, {"id": "b", "tokens": b[2:], "want": [38]}], "end": ["b"]},
             {"step": 3, "entries": [{"id": "a", "tokens": a[69:], "want": [0]}], "end": ["a"]}]
    out = tmp_path / "out"
    r = subprocess.run([sys.executable, str(ROOT / "bin" / "trace_run"), "--model", str(folder), "--dtype", dtype, "--out", str(out),
                        "--max-tokens", "192"], input="".join(json.dumps(s) + "\n" for s in steps), capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    assert [line for line in r.stdout.splitlines() if line.startswith("done")] == ["done 0", "done 1", "done 2", "done 3"]
    assert not (out / "1.f32").exists()
    read = lambda n, rows: torch.from_numpy(np.fromfile(out / f"{n}.f32", dtype="<f4").reshape(rows, cfg["vocab"]))
    w = VM.plain_weights(tensors)
    wa, wb = P.forward(cfg, w, a), P.forward(cfg, w, b)
    bound = 2e-4 if dtype == "float32" else 0.25
    assert H.scaled_error(read(0, 2), wa[[0, 32]]) < bound
    assert H.scaled_error(read(2, 2), torch.stack([wa[68], wb[40]])) < bound
    assert H.scaled_error(read(3, 1), wa[69:70]) < bound


def test_the_command_line_writes_a_vamatar_folder_and_generates_from_it(tmp_path):
    """random-weights draws the folder from the configuration alone (decay rates and step biases by their declarations' hints),
    generate runs it through the entry point; the greedy tokens are the plain implementation's wherever its choice is clear."""
    roost = lambda *a: subprocess.run([sys.executable, str(ROOT / "bin" / "roost"), *a], capture_output=True, text=True, timeout=600)
    (tmp_path / "config.json").write_text(json.dumps(VM.MIXED))
    r = roost("random-weights", "--config", str(tmp_path / "config.json"), "--out", str(tmp_path / "model"), "--seed", "4", "--std", "0.2",
              "--norm-std", "0.1")
    assert r.returncode == 0, r.stderr
    cfg, w = P.load_model_dir(tmp_path / "model")
    assert -3.0 <= float(w["l1.mix.A_log"].min()) and float(w["l1.mix.A_log"].max()) <= -0.5
    prompt = H.random_ids(21, cfg["vocab"], 6)
    r = roost("generate", "--model", str(tmp_path / "model"), "--dtype", "float32", "--prompt-ids", ",".join(map(str, prompt)),
              "--max-output-tokens", "8", "--ignore-eos", "--attention-blocks", "16", "--max-sequences", "2")
    assert r.returncode == 0, r.stderr
    out = json.loads(r.stdout.strip().splitlines()[-1])
    assert out["finish_reason"] == "length" and len(out["token_ids"]) == 8
    logits = P.forward(cfg, w, prompt + out["token_ids"][:-1])
    for j, tok in enumerate(out["token_ids"]):
        top = logits[len(prompt) - 1 + j].topk(2)
        if float(top.values[0] - top.values[1]) > 1e-3:
            assert tok == int(top.indices[0]), (j, tok, int(top.indices[0]))


def _recurrence_in_64_bits(xbc, dt, dt_bias, a_log, d, state, lengths, heads, N, groups):
    """y and the states after the rows, token by token; ``state`` [rows, heads, 64, N]."""
    H, S, at, ys = heads, state.double().cpu().clone(), 0, []
    x, B, C = xbc.double().cpu().split([H * 64, groups * N, groups * N], -1)
    x, (B, C) = x.reshape(-1, H, 64), (t.reshape(-1, groups, N).repeat_interleave(H // groups, 1) for t in (B, C))
    dt = torch.nn.functional.softplus(dt.double().cpu() + dt_bias.double().cpu())
    fade = torch.exp(-torch.exp(a_log.double().cpu()) * dt)
    for r, n in enumerate(lengths):
        for t in range(at, at + n):
            S[r] = fade[t][:, None, None] * S[r] + (dt[t][:, None] * x[t])[:, :, None] * B[t][:, None]
            ys.append(torch.einsum("hpn,hn->hp", S[r], C[t]) + d.double().cpu()[:, None] * x[t])
        at += n
    return torch.stack(ys).reshape(at, -1), S


@pytest.mark.parametrize("odd", [None, "late", "early"])
@pytest.mark.parametrize("H,N,groups,lengths", [(4, 64, 1, [64, 65]), (4, 128, 2, [1, 300, 17]), (4, 128, 4, [63, 128]), (4, 64, 2, [8, 9, 1, 200]),
                                                (4, 128, 1, [1300, 70]), (4, 64, 4, [2100]), (64, 128, 8, [1700, 1320])])
def test_recurrence_in_chunks_on_the_tensor_cores(kernels, H, N, groups, lengths, odd):
    """Edges of chunks, rows of one token, rows of six and nine segments (the carry takes four at a time), a step whose segments are longer than
    the shortest, carried states, decays from none to complete; against 64 bits, and no further from it than the walk in 32 bits over the same
    numbers. A value that is not finite, in a row's last segment or in its first, shows from its own token on and not before."""
    T = sum(lengths)
    g = torch.Generator().manual_seed(N + len(lengths))
    xbc = torch.randn(T, H * 64 + 2 * groups * N, generator=g).to(torch.bfloat16)
    u = torch.zeros(T, 8 + H)
    u[:, 8:] = torch.randn(T, H, generator=g)
    u = u.to(torch.bfloat16)
    dt_bias, d = torch.randn(H, generator=g), torch.randn(H, generator=g)
    a_log = torch.tensor([-3.0, -1.0, 1.0, 4.0]).repeat(H // 4)
    state = torch.randn(len(lengths), H * 64 * N, generator=g)
    if odd:
        t = T - 6 if odd == "late" else min(100, T - 6)
        xbc[t, 70], u[t, 9] = float("inf"), float("inf")
    want, S = _recurrence_in_64_bits(xbc, u[:, 8:].float(), dt_bias, a_log, d, state.reshape(len(lengths), H, 64, N), lengths, H, N, groups)
    q_indptr = torch.tensor([0] + list(np.cumsum(lengths)), dtype=torch.int32).cuda()
    slots = torch.arange(len(lengths), dtype=torch.int32).cuda()
    got = {}
    for dtype in DTYPES:
        s = state.cuda()
        y = kernels.mamba2_scan(xbc.to(dtype).cuda(), u.to(dtype).cuda(), 8, dt_bias.cuda(), a_log.cuda(), d.cuda(), s, q_indptr, slots, H, 64, N, groups)
        got[dtype] = (y.double().cpu(), s.double().cpu().reshape(S.shape))
    for name, w, k in (("y", want, 0), ("state", S, 1)):
        fine = torch.isfinite(w)
        assert torch.equal(torch.isfinite(got[torch.bfloat16][k]), fine) and torch.equal(torch.isfinite(got[torch.float32][k]), fine), name
        off = {t: float((got[t][k] - w)[fine].norm() / w[fine].norm()) for t in DTYPES}
        print(f"MEASURED recurrence in chunks {name}: tensor cores {off[torch.bfloat16]:.2e}, walk {off[torch.float32]:.2e}")
        # no further off than the walk, whose sums of N and 64 terms leave it within a unit of 2^-23 or two
        assert off[torch.bfloat16] < max(1.1 * off[torch.float32], 2.0 ** -23), (name, off)


# lists of 76, 77, 78 entries (all of them take a tile of w together on 148 processors), of 75, 79 and 81 (two do, a last one by itself), 128 + 24
@pytest.mark.parametrize("E,T,top", [(64, 256, 6), (64, 266, 6), (64, 290, 6), (64, 220, 6), (64, 320, 6), (64, 350, 6), (128, 380, 8), (16, 80, 16)])
@pytest.mark.parametrize("n", [256, 768, 520])
def test_every_order_of_the_grouped_product_takes_every_tile(kernels, E, T, top, n):
    hidden = 64
    g = torch.Generator().manual_seed(T)
    logits = torch.randn(T, E, generator=g)
    logits[:, 3] -= 20.0                                    # an expert without rows
    if E < 128:
        logits[: T // 2, 5] += 20.0                         # and one of several tiles
    route = kernels.moe_route(logits.cuda(), top)
    assert route.wide_tiles is not None
    x, w = torch.randn(route.rows, hidden, generator=g).to(torch.bfloat16).cuda(), (torch.randn(E, n, hidden, generator=g) * 0.15).to(torch.bfloat16).cuda()
    want = torch.empty((route.rows, n), dtype=torch.float64, device="cuda")
    for e in range(E):
        mine = route.expert == e
        want[mine] = x[mine].double() @ w[e].double().T
    assert ((kernels._moe_gemm_tcgen05(x, w, route, False).double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -16).all()
    if n % 256 == 0:
        gate, up = want.reshape(route.rows, n // 256, 2, 128).unbind(2)
        act = (gate / (1.0 + torch.exp(-gate)) * up).reshape(route.rows, n // 2)
        assert ((kernels._moe_gemm_tcgen05(x, w, route, True).double() - act).abs() <= 2.0 ** -8 * act.abs() + 2.0 ** -16).all()
    kernels.check_device_status()


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("lengths,channels", [([1, 2, 3, 4, 37], 24), ([600, 1, 2, 3, 414], 1032), ([100, 1, 2, 78], 6144), ([3000, 1, 2000], 1032)])
def test_convolution_forms_agree_bit_for_bit(kernels, dtype, lengths, channels):
    """Sixteen tokens a thread, four (token counts that are no multiple of four, rows that begin inside a thread's), and a number at a time (columns that start off a
    whole piece): the same sums."""
    T = sum(lengths)
    g = torch.Generator().manual_seed(T)
    u = torch.randn(T, channels + 16, generator=g).to(dtype).cuda()
    shifted = torch.zeros_like(u)
    shifted[:, 9 : 9 + channels] = u[:, 8 : 8 + channels]
    w, bias = torch.randn(channels, 4, generator=g).cuda(), torch.randn(channels, generator=g).cuda()
    state = torch.randn(len(lengths) + 1, 8 + 3 * channels, generator=g).cuda()
    rows = torch.tensor([r for r, n in enumerate(lengths) for _ in range(n)], dtype=torch.int32).cuda()
    q_indptr = torch.tensor([0] + list(np.cumsum(lengths)), dtype=torch.int32).cuda()
    slots = torch.arange(len(lengths), 0, -1, dtype=torch.int32).cuda()
    args = (channels, w, bias, state, 8, rows, q_indptr, slots)
    assert torch.equal(kernels.mamba2_conv(u, 8, *args), kernels.mamba2_conv(shifted, 9, *args))


GATES = (-88.0, -87.5, -87.0, -60.0, -20.0, -1.0)      # exp(88) is still a number, and so is what a gate of -88 leaves
# one rounding of the result; the 32-bit gate itself, below the smallest normal number, is a multiple of 2^-149
FAR_BELOW_ZERO = {torch.bfloat16: 2.0 ** -8, torch.float32: 2.0 ** -19}


def within_a_rounding(got, want, dtype):
    assert ((got.double() - want).abs() <= FAR_BELOW_ZERO[dtype] * want.abs()).all() and (got != 0).all()


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("tokens,channels", [(7, 24), (600, 1032), (1100, 1032), (5000, 1032)])
def test_the_convolution_of_sums_far_below_zero(kernels, dtype, tokens, channels):
    bias = torch.tensor(GATES).repeat(-(-channels // 6))[:channels].cuda()
    u, w = torch.zeros(tokens, channels, dtype=dtype, device="cuda"), torch.zeros(channels, 4, device="cuda")
    state, one = torch.zeros(1, 3 * channels, device="cuda"), torch.zeros(tokens, dtype=torch.int32, device="cuda")
    q_indptr, slots = torch.tensor([0, tokens], dtype=torch.int32).cuda(), one[:1].contiguous()
    got = kernels.mamba2_conv(u, 0, channels, w, bias, state, 0, one, q_indptr, slots)
    z = bias.double()
    within_a_rounding(got, (z / (1.0 + torch.exp(-z))).expand_as(got), dtype)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("tokens,heads,vdim", [(9, 1, 96), (9, 4, 30), (9, 4, 96)])      # a row a block, a number a lane, a head a warp
@pytest.mark.parametrize("gate", ["sigmoid", "silu"])
def test_the_head_norm_behind_gates_far_below_zero(kernels, dtype, tokens, heads, vdim, gate):
    width = heads * vdim
    g = torch.tensor(GATES).repeat(width)[:width].expand(tokens, width)
    o, w = torch.ones(tokens, width, device="cuda"), torch.full((width,), 1e25, device="cuda")
    got = kernels.head_norm_gate(o, g.to(dtype).cuda(), 0, w, heads, 1e-12, dtype, gate=gate)
    z = g.double().cuda()
    within_a_rounding(got, float(torch.tensor(1e25)) / (1.0 + torch.exp(-z)) * (z if gate == "silu" else 1.0), dtype)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("tokens,size", [(5, 30), (5, 96), (1536, 96)])                  # a number at a time, a group a block, a group a warp
def test_the_gated_norm_behind_gates_far_below_zero(kernels, dtype, tokens, size):
    z = torch.tensor([-88.0, -87.5]).repeat(size)[:size].expand(tokens, size)
    y, w = torch.full((tokens, size), 1e36, device="cuda"), torch.ones(size, device="cuda")
    got = kernels.gated_group_norm(y, z.to(dtype).cuda(), w, 1, 1e-12, dtype)
    v = (float(torch.tensor(1e36)) * z.double() / (1.0 + torch.exp(-z.double()))).cuda()
    within_a_rounding(got, v / torch.sqrt((v * v).mean(-1, keepdim=True) + 1e-12), dtype)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("tokens", [5, 1536])        # a group a block, a group a warp
@pytest.mark.parametrize("size,groups", [(4, 3), (36, 2), (256, 2), (512, 8), (1024, 1), (1028, 3), (2048, 1), (4100, 1), (8192, 1), (8196, 1), (50, 1)])
def test_gated_group_norm_at_every_width(kernels, dtype, size, groups, tokens):
    g = torch.Generator().manual_seed(size)
    y, w = torch.randn(tokens, size * groups, generator=g).cuda() * 3, torch.randn(size * groups, generator=g).cuda()
    u = torch.randn(tokens, size * groups + 4, generator=g).to(dtype).cuda()
    z = u.double().cpu()[:, : size * groups]
    v = y.double().cpu() * z * torch.sigmoid(z)
    want = P.unit_rms(v.reshape(tokens, groups, size), 1e-6).reshape(tokens, -1) * w.double().cpu()
    close(kernels.gated_group_norm(y, u, w, groups, 1e-6, dtype), want, dtype, "gated group norm")


@pytest.mark.parametrize("T,E,top", [(1, 1, 1), (700, 3, 3), (2049, 700, 1), (900, 701, 5), (1500, 64, 6)])
def test_pairs_sorted_by_one_block_and_by_a_cluster(kernels, T, E, top):
    """Ranges, tiles of both widths and the sorted rows from the choices alone, twice (the counts are left at zero), experts that nobody chose."""
    g = torch.Generator().manual_seed(E)
    logits = torch.randn(T, E, generator=g)
    logits[:, : E // 2] -= 3.0 * (E > 8)
    for _ in range(2):
        route = kernels.moe_route(logits.cuda(), top)
    chosen = torch.topk(logits, top, dim=1).indices
    counts = torch.bincount(chosen.flatten(), minlength=E)
    offsets = torch.cat([torch.zeros(1, dtype=torch.long), counts.cumsum(0)])
    assert torch.equal(route.offsets.cpu().long(), offsets)
    inverse = route.inverse.cpu().long().reshape(T, top)
    assert torch.equal(inverse.flatten().sort().values, torch.arange(T * top))
    assert torch.equal(route.expert.cpu().long()[inverse].sort(1).values, chosen.sort(1).values)
    assert torch.equal(route.token.cpu().long()[inverse], torch.arange(T)[:, None].expand(T, top))
    want = torch.sigmoid(logits.double())[torch.arange(T)[:, None], route.expert.cpu().long()[inverse]]
    assert float((route.weight.cpu().double()[inverse] - want).abs().max()) < 1e-6
    for tiles, width in ((route.tiles, 64), (route.wide_tiles, 128)):
        if tiles is None:
            continue
        rows = [(e, r, min(r + width, int(offsets[e + 1]))) for e in range(E) for r in range(int(offsets[e]), int(offsets[e + 1]), width)]
        got = tiles.cpu().reshape(-1, 3)
        assert [tuple(t) for t in got[: len(rows)].tolist()] == rows and (got[len(rows):, 0] == -1).all()


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("hidden", [4, 36, 264, 2048])
def test_rows_gathered_and_combined_at_every_width(kernels, dtype, hidden):
    g = torch.Generator().manual_seed(hidden)
    T, E, top = 37, 5, 3
    logits, x = torch.randn(T, E, generator=g), torch.randn(T, hidden, generator=g).to(dtype)
    route = kernels.moe_route(logits.cuda(), top)
    token, weight, inverse = route.token.cpu().long(), route.weight.cpu(), route.inverse.cpu().long().reshape(T, top)
    assert torch.equal(kernels.moe_gather_scale(x.cuda(), route, scale=False).cpu(), x[token])
    assert torch.equal(kernels.moe_gather_scale(x.cuda(), route).cpu(), (weight[:, None] * x[token].float()).to(dtype))
    ys, shared = torch.randn(T * top, hidden, generator=g).to(dtype), torch.randn(T, hidden, generator=g).to(dtype)
    total = torch.zeros(T, hidden)
    for k in range(top):
        total += ys[inverse[:, k]].float()
    assert torch.equal(kernels.moe_combine(ys.cuda(), route, None).cpu(), total.to(dtype))
    assert torch.equal(kernels.moe_combine(ys.cuda(), route, shared.cuda()).cpu(), (total + shared.float()).to(dtype))
