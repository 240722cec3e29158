"""Forms of kernels chosen by size, each at the sizes where it can go wrong, against 64-bit products and sums.

Tolerances: a float32 sum of k products of numbers of order one and 1 / sqrt(k) differs from the exact one by a few 2^-24 times
sqrt(k) of its own size at most, i.e. below 1e-5 for the sizes here; a result rounded to bfloat16 by 2^-9 of itself."""
import math
import os
import subprocess
import sys
import types

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from wick_b200 import ops  # noqa: E402
from wick_b200.engine.batch import BatchLayout, StepBatch, fill_host  # noqa: E402

DEV = "cuda"
PAGE = 64
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def batch_of(q_lens, starts):
    """Sequences of these many new tokens behind these many cached ones, on pages in no order; and their pages."""
    n_pages = sum((s + q + PAGE - 1) // PAGE for s, q in zip(starts, q_lens))
    order, pages = list(np.random.RandomState(3).permutation(n_pages) + 1), []
    for s, q in zip(starts, q_lens):
        pages.append([int(order.pop()) for _ in range((s + q + PAGE - 1) // PAGE)])
    layout = BatchLayout(len(q_lens), sum(q_lens), max(len(p) for p in pages), len(q_lens))
    host = np.zeros(layout.size, dtype=np.int32)
    fill_host(layout, host, tokens=[[0] * q for q in q_lens], starts=starts, slots=[1 + i for i in range(len(q_lens))], pages=pages,
              want=[[q - 1] for q in q_lens])
    return StepBatch(layout, torch.from_numpy(host).to(DEV), q_lens=q_lens, starts=starts), pages, n_pages + 1


def unwritten_as_nan(monkeypatch):
    """What torch.empty gives on the device holds NaN until a kernel writes it."""
    real = torch.empty

    def empty(*a, **k):
        t = real(*a, **k)
        return t.fill_(float("nan")) if t.is_cuda and t.is_floating_point() else t
    monkeypatch.setattr(torch, "empty", empty)


def gated(y):
    g, u = y.chunk(2, dim=1)
    return g / (1 + torch.exp(-g)) * u


@pytest.mark.parametrize("n, k", [(8, 4), (130, 100), (72, 128), (200, 132), (513, 1028), (64, 640), (2400, 2052)])
@pytest.mark.parametrize("pair", [False, True])
def test_float32_products_of_every_form_give_the_same_bits(n, k, pair):
    """1 to 32 rows stream the weights, more rows take tiles whose slices of the inner dimension a cluster joins, or whole tiles
    of 128 x 128 (the last size at 2,500 rows); all of them add in one order.  k: less than a slice, remainders of one, two
    slices' worth, five slices (a cluster of five), eight with a remainder."""
    g = torch.Generator().manual_seed(n + k)
    rows = 2500 if n == 2400 else 300
    x = torch.randn(rows, k, generator=g).to(DEV)
    w = (torch.randn(2 * n if pair else n, k, generator=g) / math.sqrt(k)).to(DEV)
    got = ops.gemm_simt(x, w, torch.float32, gated=pair)
    ref = x.double() @ w.double().T
    ref = gated(ref) if pair else ref
    assert (got.double() - ref).abs().max() < 1e-5 * max(1.0, float(ref.abs().max()))
    for m in (1, 2, 3, 5, 8, 9, 16, 17, 32, 33, 64, 65, 129, 300):
        assert torch.equal(ops.gemm_simt(x[:m].contiguous(), w, torch.float32, gated=pair, w_static=m % 2 == 0), got[:m]), m


@pytest.mark.parametrize("m", [1, 32, 33, 300])
def test_float32_products_read_a_matrix_that_the_kernel_before_wrote(m):
    """Without ``w_static`` the second operand may be the result of the kernel launched just before, which need not have finished
    when the product's blocks start: nothing of it may be read early."""
    x, src = torch.randn(m, 2048).to(DEV), torch.randn(2048, 2048).to(DEV)
    delta, one = torch.randn(8, 2048, 2048).to(DEV), torch.ones(2048, device=DEV)
    for _ in range(5):
        w = torch.full((2048, 2048), float("nan"), device=DEV)        # (what an early load would find)
        ops.rmsnorm(src.clone(), one, 1e-5, torch.float32, delta=delta, out=w)
        got = ops.gemm_simt(x, w, torch.float32)
        torch.cuda.synchronize()
        assert torch.equal(got, ops.gemm_simt(x, w, torch.float32))


@pytest.mark.parametrize("n, k, pair", [(2049, 64, False), (16385, 100, False), (4097, 128, True), (12300, 128, True), (4096, 132, False), (4100, 256, True), (300, 64, True),
                                        (37900, 64, False), (18950, 260, True)])
def test_float32_products_of_wide_matrices_give_the_same_bits(n, k, pair):
    """Wide matrices of few inputs: the general form (a single slice), tiles instead of streamed weights, tiles of 64 rows where the
    large ones would be half empty."""
    g = torch.Generator().manual_seed(n + k)
    x = torch.randn(300, k, generator=g).to(DEV)
    w = (torch.randn(2 * n if pair else n, k, generator=g) / math.sqrt(k)).to(DEV)
    got = ops.gemm_simt(x, w, torch.float32, gated=pair, w_static=True)
    ref = x.double() @ w.double().T
    ref = gated(ref) if pair else ref
    assert (got.double() - ref).abs().max() < 1e-5 * max(1.0, float(ref.abs().max()))
    for m in (1, 8, 9, 16, 17, 32, 33, 64, 65, 128, 129):
        assert torch.equal(ops.gemm_simt(x[:m].contiguous(), w, torch.float32, gated=pair, w_static=True), got[:m]), m


@pytest.mark.parametrize("n, k, pair", [(8192, 132, True), (2100, 192, True), (1500, 256, True), (6200, 100, True), (16400, 48, True), (4100, 176, True),
                                        (8192, 132, False), (4100, 160, False), (6200, 224, False), (6200, 100, False), (9500, 60, False), (2048, 132, False), (24600, 132, False), (32800, 384, False), (16400, 320, True)])
def test_float32_products_of_few_inputs_give_the_same_bits(n, k, pair):
    """One or two slices: the general form takes the slices as the others do, gated tiles of 64 rows both one after the other.  The rows
    cross the sizes at which the forms change."""
    g = torch.Generator().manual_seed(n + k)
    x = torch.randn(600, k, generator=g).to(DEV)
    w = (torch.randn(2 * n if pair else n, k, generator=g) / math.sqrt(k)).to(DEV)
    got = ops.gemm_simt(x, w, torch.float32, gated=pair, w_static=True)
    ref = x.double() @ w.double().T
    ref = gated(ref) if pair else ref
    assert (got.double() - ref).abs().max() < 1e-5 * max(1.0, float(ref.abs().max()))
    for m in (1, 4, 8, 9, 16, 17, 32, 33, 64, 65, 128, 129, 193, 257, 321):
        assert torch.equal(ops.gemm_simt(x[:m].contiguous(), w, torch.float32, gated=pair, w_static=m % 2 == 0), got[:m]), m


def test_float32_products_of_misaligned_rows_take_the_general_form():
    x, w = torch.randn(5 * 64 + 1).to(DEV)[1:].view(5, 64), torch.randn(24, 64).to(DEV)
    assert x.data_ptr() % 16 != 0
    assert (ops.gemm_simt(x, w, torch.float32).double() - x.double() @ w.double().T).abs().max() < 1e-4


@pytest.mark.parametrize("H, R, r, q_lens, starts, window, sink", [
    (32, 576, 512, [1, 1, 1], [0, 700, 2100], 2048, False),          # runs of keys, a window's edge
    (40, 576, 512, [1], [33], 0, False),                             # a second, partial group of heads
    (16, 320, 256, [1, 1], [31, 32], 20, True),                      # one group of 16 heads, a window that starts inside a tile
    (7, 80, 64, [3, 70], [62, 0], 0, True),                          # few heads, the smallest value, new tokens of one sequence
    (5, 64, 64, [200], [5], 50, False),                              # many tokens: one run each, the value is the whole row
    (33, 144, 128, [2], [127], 64, True),
])
def test_attention_over_rows_on_the_tensor_cores(H, R, r, q_lens, starts, window, sink):
    """float32 queries as three bfloat16 numbers each: no further from 64 bits than float32 arithmetic is."""
    g = torch.Generator().manual_seed(H)
    assert ops.attention_latent_supported(R, r)
    batch, pages, n_pages = batch_of(q_lens, starts)
    store = torch.full((n_pages, PAGE, R), float("nan")).bfloat16()
    rows = []
    for b, (q, s) in enumerate(zip(q_lens, starts)):
        rows.append(torch.randn(s + q, R, generator=g).bfloat16())
        for p in range(s + q):
            store[pages[b][p // PAGE], p % PAGE] = rows[b][p]
    n = sum(q_lens)
    q = torch.randn(n, H, R, generator=g)
    sinks = torch.randn(H, generator=g) if sink else None
    scale = R ** -0.5
    out = ops.attention_multi(q.to(DEV), store.to(DEV), batch, scale, maps=1, kv_heads=1, v_dim=r, window=window,
                              sink=sinks.to(DEV) if sink else None, rows_of=R, out_dtype=torch.float32).double().cpu()
    t = 0
    for b, (ql, s) in enumerate(zip(q_lens, starts)):
        k = rows[b].double()
        for p in range(s, s + ql):
            lo = max(0, p - window + 1) if window else 0
            z = q[t].double() @ k[lo:p + 1].T * scale
            e = torch.exp(z - 20.0)                     # (scores of order one to ten: no maximum is needed in 64 bits)
            den = e.sum(1, keepdim=True) + (torch.exp(sinks.double()[:, None] - 20.0) if sink else 0.0)
            ref = (e / den) @ k[lo:p + 1, :r]
            assert (out[t] - ref).abs().max() < 1e-5 * float(ref.abs().max()), (b, p)
            t += 1


def test_attention_over_rows_of_queries_near_the_largest_float():
    """Queries beyond bfloat16's largest number are still the sum of their three parts."""
    batch, pages, n_pages = batch_of([1, 1], [40, 3])
    store = torch.randn(n_pages, PAGE, 80, generator=torch.Generator().manual_seed(1)).bfloat16()
    store[:, :, 79] = ((1 + torch.arange(PAGE) / 64) * 2.0 ** -126).bfloat16()
    q = torch.randn(2, 5, 80, generator=torch.Generator().manual_seed(2))
    q[0, 1, 79], q[0, 3, 79] = 3.4e38, -torch.finfo(torch.float32).max
    out = ops.attention_multi(q.to(DEV), store.to(DEV), batch, 0.3, maps=1, kv_heads=1, v_dim=64, rows_of=80, out_dtype=torch.float32).double().cpu()
    for t, n in ((0, 41), (1, 4)):
        k = torch.cat([store[p] for p in pages[t]])[:n].double()
        ref = torch.softmax(q[t].double() @ k.T * 0.3, -1) @ k[:, :64]
        assert (out[t] - ref).abs().max() < 1e-5 * float(ref.abs().max())


@pytest.mark.parametrize("H, R, r, q_lens, starts, window, keep", [
    (16, 80, 64, [1, 1], [500, 90], 64, 10),                        # kept keys end inside a tile, runs of keys
    (4, 80, 64, [70], [300], 100, 40),                              # beyond one tile, few runs
    (5, 80, 64, [200], [5], 50, 7),                                 # many tokens: one run each, some before the window's start
    (32, 576, 512, [1, 2], [2000, 31], 512, 33),
])
def test_attention_over_rows_with_kept_first_keys_on_the_tensor_cores(H, R, r, q_lens, starts, window, keep):
    g = torch.Generator().manual_seed(H)
    batch, pages, n_pages = batch_of(q_lens, starts)
    store = torch.randn(n_pages, PAGE, R, generator=g).bfloat16()
    q = torch.randn(sum(q_lens), H, R, generator=g)
    out = ops.attention_multi(q.to(DEV), store.to(DEV), batch, R ** -0.5, maps=1, kv_heads=1, v_dim=r, window=window, keep_first=keep, rows_of=R,
                              out_dtype=torch.float32).double().cpu()
    t = 0
    for b, (ql, s) in enumerate(zip(q_lens, starts)):
        k = torch.cat([store[p] for p in pages[b]])[:s + ql].double()
        for p in range(s, s + ql):
            j = torch.arange(p + 1)
            seen = k[:p + 1][(p - j < window) | (j < keep)]
            ref = torch.softmax(q[t].double() @ seen.T * R ** -0.5, -1) @ seen[:, :r]
            assert (out[t] - ref).abs().max() < 1e-5 * float(ref.abs().max()), (b, p)
            t += 1


def test_attention_over_rows_of_a_token_alone_and_among_others():
    """How many runs a token's keys are cut into follows the number of tokens and the step's bound: what differs is the order of float32
    sums, a few 2^-24 of a result that is an average of its values."""
    g = torch.Generator().manual_seed(8)
    starts = [700, 33, 1500, 64] * 6
    batch, pages, n_pages = batch_of([1] * 24, starts)
    store, q = torch.randn(n_pages, PAGE, 144, generator=g).bfloat16().to(DEV), torch.randn(24, 20, 144, generator=g).to(DEV)
    args = dict(maps=1, kv_heads=1, v_dim=128, rows_of=144, out_dtype=torch.float32)
    many = ops.attention_multi(q, store, batch, 0.08, **args)
    for i in range(4):
        layout = BatchLayout(1, 1, len(pages[i]), 1)
        host = np.zeros(layout.size, dtype=np.int32)
        fill_host(layout, host, tokens=[[0]], starts=starts[i:i + 1], slots=[1], pages=pages[i:i + 1], want=[[0]])
        one = StepBatch(layout, torch.from_numpy(host).to(DEV), q_lens=[1], starts=starts[i:i + 1])
        alone = ops.attention_multi(q[i:i + 1].contiguous(), store, one, 0.08, **args)[0]
        assert (alone - many[i]).abs().max() < 2e-6 * float(many[i].abs().max())


@pytest.mark.parametrize("H, R, tensor_cores", [(1, 80, False), (1, 192, False), (2, 80, False), (2, 128, True), (3, 80, True)])
def test_attention_over_rows_of_few_heads_stays_on_the_cuda_cores(H, R, tensor_cores, monkeypatch):
    batch, pages, n_pages = batch_of([150], [30])
    store = torch.randn(n_pages, PAGE, R, generator=torch.Generator().manual_seed(H)).bfloat16()
    q = torch.randn(150, H, R, generator=torch.Generator().manual_seed(9))
    form, taken = ops._attention_latent, []
    monkeypatch.setattr(ops, "_attention_latent", lambda *a: taken.append(1) or form(*a))
    out = ops.attention_multi(q.to(DEV), store.to(DEV), batch, 0.1, maps=1, kv_heads=1, v_dim=64, rows_of=R, out_dtype=torch.float32)
    assert bool(taken) == tensor_cores
    k = torch.cat([store[p] for p in pages[0]])[:180].double()
    for t in (0, 77, 149):
        ref = torch.softmax(q[t].double() @ k[:31 + t].T * 0.1, -1) @ k[:31 + t, :64]
        assert (out[t].double().cpu() - ref).abs().max() < 1e-5 * float(ref.abs().max())


@pytest.mark.parametrize("bn", [16, 48, 80, 112])
@pytest.mark.parametrize("rows, runs, dtype", [(100, 1, torch.float32), (131, 2, torch.float32), (100, 1, torch.bfloat16)])
def test_products_whose_tokens_take_several_tiles_of_an_odd_width(bn, rows, runs, dtype):
    """Weights on the 128-row side, the tokens in more than one tile of a width that is no multiple of 32: a tile writes its own
    columns only."""
    from wick_b200.ops import gemm_tc as G
    n, k = 200, 320
    g = torch.Generator().manual_seed(bn + rows)
    w = (torch.randn(n, k, generator=g) / math.sqrt(k)).bfloat16().to(DEV)
    x = torch.randn(rows, k, generator=g).bfloat16().to(DEV)
    ref = x.double() @ w.double().T
    for _ in range(20):
        out = torch.full((runs, rows, n), float("nan"), dtype=dtype, device=DEV)
        G.gemm_tc(w, n, x, rows, bn=bn, out=out, ldo=n, transposed=True, splits=runs, split_stride=rows * n, a_static=True)
        assert (out.double().sum(0) - ref).abs().max() < (1e-5 if dtype == torch.float32 else 2 ** -8) * float(ref.abs().max())
    if runs == 1 and dtype == torch.bfloat16:
        w2 = (torch.randn(2 * 128, k, generator=g) / math.sqrt(k)).bfloat16().to(DEV)
        out = torch.full((rows, 128), float("nan"), dtype=dtype, device=DEV)
        G.gemm_tc(w2, 128, x, rows, bn=bn, out=out, ldo=128, gated=3, pair_offset=128, transposed=True, a_static=True)
        ref = gated(x.double() @ w2.double().T)
        assert (out.double() - ref).abs().max() < 2 ** -8 * max(1.0, float(ref.abs().max()))
    G.check_status()


@pytest.mark.parametrize("ff, width, t", [(64, 512, 1), (200, 1024, 16), (320, 2048, 17), (65, 576, 128), (1000, 264, 5)])
def test_gated_products_of_few_tokens_joined_over_a_cluster(ff, width, t):
    """Few tiles of a gated pair: runs of the inner dimension meet inside the kernel; a token's bits do not depend on the others."""
    from wick_b200.ops import gemm_tc as G
    g = torch.Generator().manual_seed(ff)
    w = (torch.randn(2 * ff, width, generator=g) / math.sqrt(width)).bfloat16().to(DEV)
    x = torch.randn(t, width, generator=g).bfloat16().to(DEV)
    plan = G.plan_for(w, gated=True)
    assert plan.joined_splits == {512: 2, 1024: 4, 2048: 8, 576: 2, 264: 1}[width]
    got = plan.forward(x, torch.bfloat16)
    ref = gated(x.double() @ w.double().T)
    G.check_status()
    assert (got.double() - ref).abs().max() < 2 ** -8 * max(1.0, float(ref.abs().max()))
    if t <= G.SMALL:
        assert torch.equal(plan.forward(x[:1].contiguous(), torch.bfloat16), got[:1])


@pytest.mark.parametrize("ff, width, runs", [(66, 768, 3), (130, 640, 2), (257, 1280, 5), (70, 1536, 6)])
@pytest.mark.parametrize("t", [1, 31, 128])
def test_gated_products_joined_with_rows_that_are_no_whole_groups(ff, width, runs, t):
    """Up to four runs four neighbours a thread are finished at once, or one by one at a row's end."""
    from wick_b200.ops import gemm_tc as G
    g = torch.Generator().manual_seed(ff)
    w = (torch.randn(2 * ff, width, generator=g) / math.sqrt(width)).bfloat16().to(DEV)
    x = torch.randn(t, width, generator=g).bfloat16().to(DEV)
    plan = G.plan_for(w, gated=True)
    assert plan.joined_splits == runs
    got, ref = plan.forward(x, torch.bfloat16), gated(x.double() @ w.double().T)
    G.check_status()
    assert (got.double() - ref).abs().max() < 2 ** -8 * max(1.0, float(ref.abs().max()))


@pytest.mark.parametrize("E, top, ff, width, shared", [(5, 3, 136, 264, 0), (8, 2, 192, 1024, 64), (1, 1, 64, 128, 0), (16, 2, 72, 512, 0), (5, 2, 520, 264, 1000)])
@pytest.mark.parametrize("n", [1, 2, 17, 64, 65, 128, 129])
def test_table_experts_of_few_tokens(E, top, ff, width, shared, n, monkeypatch):
    """Experts that no token uses are left alone; results beyond a token's own experts are never read (they hold NaN before), nor, beyond
    128 tokens, rows between the sorted experts' and tiles beyond the last one's (without the host's token ids there are the most rows
    that there can be)."""
    from wick_b200.models.spec import PartSpec
    from wick_b200.parts.base import BuildContext, build_part
    from wick_b200.parts import feedforward  # noqa: F401
    g = torch.Generator().manual_seed(E + n)
    part = build_part("ffn", PartSpec("table_moe", dict(width=width, vocab=50, experts=E, top=top, intermediate=ff,
                                                        shared=PartSpec("gated_mlp", dict(width=width, intermediate=shared, activation="silu",
                                                                                          names=dict(gate="gate_proj.weight", up="up_proj.weight", down="down_proj.weight"))) if shared else None)),
                      BuildContext(dtype=torch.bfloat16, device=torch.device(DEV)))
    tensors = {}

    def get(name):
        if name == "table":
            return torch.rand(50, E, generator=g).argsort(1)[:, :top].int()
        inner = shared if "shared" in name else ff
        rows, cols = (width, inner) if "down" in name else (inner, width)
        return tensors.setdefault(name, (torch.randn(rows, cols, generator=g) / math.sqrt(cols)).bfloat16().to(DEV))
    part.load(get)
    x = torch.randn(n, width, generator=g).bfloat16().to(DEV)
    tok = torch.randint(0, 50, (n,), generator=g).int().to(DEV)
    unwritten_as_nan(monkeypatch)
    got = part.forward(x, types.SimpleNamespace(tokens=tok, host=None)).sum(0)
    ops.check_status()

    def expert(pre, h):
        a = gated(torch.cat([h @ tensors[pre + "gate_proj.weight"].double().T, h @ tensors[pre + "up_proj.weight"].double().T], 1))
        return a @ tensors[pre + "down_proj.weight"].double().T
    ref = expert("shared.", x.double()) if shared else torch.zeros(n, width, dtype=torch.float64, device=DEV)
    for t in range(n):
        for e in part.table[int(tok[t])].tolist():
            ref[t] += expert(f"experts.{e}.", x[t:t + 1].double())[0] / top
    assert (got.double() - ref).norm() < 5e-3 * ref.norm()             # (the inner activations are rounded to bfloat16)
    if n <= 64:
        one = part.forward(x[:1].contiguous(), types.SimpleNamespace(tokens=tok[:1].contiguous(), host=None)).sum(0)
        assert torch.equal(one, got[:1]), "a token's bits do not depend on the others"


@pytest.mark.parametrize("E, top", [(40, 3), (300, 2), (320, 5), (1024, 1), (1025, 1)])
@pytest.mark.parametrize("n", [1, 25, 26, 60, 61, 128])
def test_table_experts_of_which_a_step_names_a_few(E, top, n):
    """Blocks for as many experts as the step can name where those are few of many (up to 1,024 experts), the i-th slot's expert being the
    i-th that it names; otherwise blocks for all."""
    from wick_b200.ops import gemm_tc as G
    g, f, w = torch.Generator().manual_seed(E + n), 72, 64
    mats = (torch.randn(E, f, w, generator=g) / math.sqrt(w)).bfloat16()
    table = torch.stack([torch.randperm(E, generator=g)[:top] for _ in range(50)]).int()
    table[7], table[8] = torch.arange(top), torch.arange(E - top, E)        # (the first and the last)
    tiles = torch.cat([G.pack(m.to(DEV)) for m in mats], 0)
    x = torch.randn(n, w, generator=g).bfloat16()
    tok = torch.randint(0, 50, (n,), generator=g).int()
    tok[0], tok[-1] = 7, 8
    y = G.gemm_tc_experts(tiles, E, f, x.to(DEV), tok.to(DEV), table.to(DEV), gated=False, per_expert_b=False, k=w)[0].cpu()
    G.check_status()
    for t in range(n):
        for e in table[int(tok[t])].tolist():
            ref = mats[e].double() @ x[t].double()
            assert (y[e, t].double() - ref).abs().max() < 1e-5, (t, e)


@pytest.mark.parametrize("width", [4, 132, 4096, 4100, 5120, 5124, 6144, 6148])
@pytest.mark.parametrize("splits", [0, 1, 7, 9])
def test_norm_forms_give_the_same_bits(width, splits):
    """A warp per row (600 rows, up to 5,120 numbers), a block with the row in registers, a block with the row in shared memory."""
    g = torch.Generator().manual_seed(width + splits)
    x, w = torch.randn(600, width, generator=g).to(DEV), (1 + 0.1 * torch.randn(width, generator=g)).to(DEV)
    delta = torch.randn(splits, 600, width, generator=g).to(DEV) if splits else None
    ref = x.double() + (delta.double().sum(0) if splits else 0)
    ref = ref / torch.sqrt((ref * ref).mean(1, keepdim=True) + 1e-5) * w.double()
    for dtype, tol in ((torch.float32, 2e-6), (torch.bfloat16, 2 ** -8)):
        many = ops.rmsnorm(x.clone(), w, 1e-5, dtype, delta=delta)
        assert (many.double() - ref).abs().max() < tol * float(ref.abs().max())
        few_x = x[:9].clone()
        few = ops.rmsnorm(few_x, w, 1e-5, dtype, delta=delta[:, :9].contiguous() if splits else None)
        assert torch.equal(few, many[:9])
        if splits:
            assert (few_x.double() - (x[:9].double() + delta[:, :9].double().sum(0))).abs().max() < 1e-5


@pytest.mark.parametrize("width", [4096, 4100, 5120])
def test_norms_of_long_rows_among_many_give_the_same_bits(width):
    """Up to two partial sums of long rows take a warp a row from 512 rows on, more a block a row."""
    g = torch.Generator().manual_seed(width)
    w = (1 + 0.1 * torch.randn(width, generator=g)).to(DEV)
    for splits in (1, 2, 3, 8):
        x, delta = torch.randn(513, width, generator=g).to(DEV), torch.randn(splits, 513, width, generator=g).to(DEV)
        many_x, few_x = x.clone(), x[:511].clone()
        many = ops.rmsnorm(many_x, w, 1e-5, torch.float32, delta=delta)
        few = ops.rmsnorm(few_x, w, 1e-5, torch.float32, delta=delta[:, :511].contiguous())
        assert torch.equal(few, many[:511]) and torch.equal(few_x, many_x[:511])


@pytest.mark.parametrize("width", [4, 260, 2048, 4096, 4100, 8192, 8196])
@pytest.mark.parametrize("n", [3, 65])
@pytest.mark.parametrize("splits", [0, 1, 3, 9])
def test_scaled_sum_and_norm_forms(width, n, splits):
    g = torch.Generator().manual_seed(width + n)
    x, w = torch.randn(n, width, generator=g).to(DEV), (1 + 0.1 * torch.randn(width, generator=g)).to(DEV)
    delta = torch.randn(splits, n, width, generator=g).to(DEV) if splits else None
    ref = 1.7 * x.double() + (delta.double().sum(0) if splits else 0)
    ref = ref / torch.sqrt((ref * ref).mean(1, keepdim=True) + 1e-5) * w.double()
    xd = x.clone()
    out = ops.scaled_add_rmsnorm(xd, delta, 1.7, w, 1e-5, torch.bfloat16)
    assert (xd.double() - ref).abs().max() < 2e-6 * float(ref.abs().max())
    assert torch.equal(out, xd.bfloat16())


@pytest.mark.parametrize("width", [4, 132, 2048, 2052, 4096, 4100, 8192])
@pytest.mark.parametrize("splits", [0, 1, 3, 9])
def test_a_row_of_the_scaled_sum_and_norm_does_not_depend_on_the_number_of_rows(width, splits):
    """The block's size follows the number of rows (64 and 65), the order of a row's sum of squares does not."""
    g = torch.Generator().manual_seed(width + splits)
    x, w = torch.randn(300, width, generator=g).to(DEV), (1 + 0.1 * torch.randn(width, generator=g)).to(DEV)
    delta = torch.randn(splits, 300, width, generator=g).to(DEV) if splits else None
    many = x.clone()
    ops.scaled_add_rmsnorm(many, delta, 1.7, w, 1e-5, torch.float32)
    for n in (1, 3, 64, 65):
        few = x[:n].clone()
        ops.scaled_add_rmsnorm(few, delta[:, :n].contiguous() if splits else None, 1.7, w, 1e-5, torch.float32)
        assert torch.equal(few, many[:n]), n


@pytest.mark.parametrize("H, G, d, e, rot, n, splits", [(4, 2, 16, 24, 8, 3, 1), (32, 8, 128, 128, 128, 70, 1), (32, 8, 128, 128, 64, 8, 8),
                                                        (10, 2, 20, 4, 20, 66, 3), (48, 8, 128, 64, 0, 65, 2), (1, 1, 4, 4, 4, 1, 9)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("mode", [0, 1, 2])
def test_projection_finish_in_registers_is_the_general_form(H, G, d, e, rot, n, splits, dtype, mode):
    """The same call with a further column in every row of partial sums, so that rows are no multiple of four numbers, takes the
    general form, element by element."""
    g = torch.Generator().manual_seed(H * d + n)
    W = (H + G) * d + G * e
    parts = torch.randn(splits, n, W, generator=g).to(DEV)
    odd = torch.cat([parts, torch.zeros(splits, n, 1, device=DEV)], 2).contiguous()
    assert W % 4 == 0 and odd.shape[2] % 4 != 0
    bias, qw, kw = ((s + 0.1 * torch.randn(m, generator=g)).to(DEV) for s, m in ((0.0, W), (1.0, H * d), (1.0, G * d)))
    batch, pages, n_pages = batch_of([n], [37])
    cos = sin = None
    if rot:
        inv = torch.tensor([100.0 ** (-2.0 * i / rot) for i in range(rot // 2)]).to(DEV)
        cos, sin = ops.rope_table(batch.positions, inv)
    keep0 = torch.randn(n, G * e, generator=g).to(DEV)
    got = []
    for p in (parts, odd):
        keep = keep0.clone()
        kv = torch.zeros((n_pages, G * PAGE * (d + e)), dtype=dtype, device=DEV)
        q = ops.qkv_finish(p, H, G, d, e, dtype=dtype, bias=bias, q_weight=qw, k_weight=kw, eps=1e-5, cos=cos, sin=sin, rot_dims=rot,
                           v_keep=keep if mode else None, v_mode=mode, blend=torch.tensor([0.3], device=DEV) if mode == 2 else None, kv=kv,
                           page_table=batch.page_table, seq_of_token=batch.seq_of_token, positions=batch.positions)
        got.append((q, kv, keep))
    tol = 1e-5 if dtype == torch.float32 else 2 ** -7              # (the sums of squares run in another order: the last bit of 32, or one of bfloat16)
    for a, b in zip(*got):
        assert (a.double() - b.double()).abs().max() <= tol * max(1.0, float(b.double().abs().max()))


@pytest.mark.parametrize("H, G, d, e, rot, splits", [(4, 2, 16, 24, 8, 1), (16, 4, 128, 128, 128, 8), (32, 8, 128, 128, 64, 3), (48, 8, 128, 128, 128, 2), (1, 1, 4, 4, 4, 9)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_a_row_of_the_projections_finish_does_not_depend_on_the_number_of_rows(H, G, d, e, rot, splits, dtype):
    """The block's size follows the number of rows (64 and 65), a row's bits do not."""
    g = torch.Generator().manual_seed(H * d)
    W, start = (H + G) * d + G * e, 37
    parts, keep0 = torch.randn(splits, 200, W, generator=g).to(DEV), torch.randn(200, G * e, generator=g).to(DEV)
    bias, qw, kw = ((s + 0.1 * torch.randn(m, generator=g)).to(DEV) for s, m in ((0.0, W), (1.0, H * d), (1.0, G * d)))
    inv = torch.tensor([100.0 ** (-2.0 * i / rot) for i in range(rot // 2)]).to(DEV)
    got = {}
    for n in (200, 65, 64, 3, 1):
        batch, pages, n_pages = batch_of([n], [start])
        cos, sin = ops.rope_table(batch.positions, inv)
        kv = torch.zeros((n_pages, G * PAGE * (d + e)), dtype=dtype, device=DEV)
        q = ops.qkv_finish(parts[:, :n].contiguous(), H, G, d, e, dtype=dtype, bias=bias, q_weight=qw, k_weight=kw, eps=1e-5, cos=cos, sin=sin,
                           rot_dims=rot, v_keep=keep0[:n].contiguous(), v_mode=2, blend=torch.tensor([0.3], device=DEV), kv=kv,
                           page_table=batch.page_table, seq_of_token=batch.seq_of_token, positions=batch.positions)
        k = kv[:, :G * PAGE * d].view(n_pages, G, PAGE, d)
        v = kv[:, G * PAGE * d:].view(n_pages, G, PAGE, e)
        at = [(pages[0][p // PAGE], p % PAGE) for p in range(start, start + n)]
        got[n] = (q, torch.stack([k[a, :, r] for a, r in at]), torch.stack([v[a, :, r] for a, r in at]))
        for one, many in zip(got[n], got[200]):
            assert torch.equal(one, many[:n]), n


@pytest.mark.parametrize("qr, r, dr, gates", [(24, 40, 8, 3), (96, 300, 64, 0), (1536, 512, 64, 0), (512, 256, 32, 5), (3840, 512, 64, 0), (23, 41, 8, 2)])
@pytest.mark.parametrize("splits", [1, 3, 8, 12])
def test_a_latents_finish_does_not_depend_on_the_number_of_rows(qr, r, dr, gates, splits):
    """Few rows take larger blocks and their partial sums' loads together; a row's bits are the same.  The last sizes cannot be read four
    numbers at a time."""
    g = torch.Generator().manual_seed(qr)
    W, start, n_all = qr + r + dr + gates, 50, 200
    parts = torch.randn(splits, n_all, W + (-W % 4 if qr % 4 == 0 else 0), generator=g).to(DEV)
    wq, wkv = torch.randn(qr, generator=g).to(DEV), torch.randn(r, generator=g).to(DEV)
    s = parts.double().sum(0)
    unit = lambda x: x / torch.sqrt((x * x).mean(1, keepdim=True) + 1e-5)  # noqa: E731
    got = {}
    for n in (n_all, 65, 64, 1):
        batch, pages, n_pages = batch_of([n], [start])
        cos, sin = ops.rope_table(batch.positions, torch.tensor([100.0 ** (-2.0 * i / dr) for i in range(dr // 2)]).to(DEV))
        rows = torch.zeros(n_pages, PAGE, r + dr, device=DEV)
        cq, gate = ops.latent_finish(parts[:, :n].contiguous(), qr, r, dr, gates, dtype=torch.float32, q_weight=wq, kv_weight=wkv, eps=1e-5, cos=cos,
                                     sin=sin, rows=rows, page_table=batch.page_table, seq_of_token=batch.seq_of_token, positions=batch.positions)
        own = torch.stack([rows[pages[0][p // PAGE], p % PAGE] for p in range(start, start + n)])
        got[n] = [cq, own] + ([gate] if gates else [])
        for one, many in zip(got[n], got[n_all]):
            assert torch.equal(one, many[:n]), n
    # (a float32 sum of a few numbers of order one, a norm and a product: a few 2^-24 of the largest, below 3e-6 of it)
    for a, ref in ((got[n_all][0], unit(s[:, :qr]) * wq.double()), (got[n_all][1][:, :r], unit(s[:, qr:qr + r]) * wkv.double())):
        assert (a.double() - ref).abs().max() < 3e-6 * float(ref.abs().max())


@pytest.mark.parametrize("ff", [8196, 15360, 16384])
@pytest.mark.parametrize("splits", [1, 3])
def test_a_long_row_of_poly_norm_does_not_depend_on_the_number_of_rows(ff, splits):
    parts = (0.7 * torch.randn(splits, 300, ff, generator=torch.Generator().manual_seed(ff))).to(DEV)
    co = torch.tensor([0.5, -1.2, 0.8, 0.3], device=DEV)
    many = ops.poly_norm(parts, co, 1e-5, torch.float32)
    for n in (1, 148, 149, 296, 297):
        assert torch.equal(ops.poly_norm(parts[:, :n].contiguous(), co, 1e-5, torch.float32), many[:n]), n


@pytest.mark.parametrize("hd", [16, 48, 64, 128])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H, G", [(4, 4), (10, 2), (12, 4), (34, 2)])
def test_short_form_of_the_decode_attention_among_few_and_many(hd, dtype, H, G):
    """Few blocks have a warp per page and head, many a warp per page for four heads: the same bits."""
    g = torch.Generator().manual_seed(hd + H)
    lens = [1, 63, 64, 65, 300, 777, 1025] + [130] * 60
    store, n_pages = torch.randn(160, 2, G, PAGE, hd, generator=g).to(dtype).to(DEV), 160
    q = torch.randn(len(lens), H, hd, generator=g).to(dtype).to(DEV)

    def run(which):
        pages, at = [], 1
        for i, n in enumerate(lens):
            k = (n + PAGE - 1) // PAGE
            pages.append([1 + (at + j) % (n_pages - 1) for j in range(k)])
            at += k
        ls = [lens[i] for i in which]
        layout = BatchLayout(len(ls), len(ls), max(len(pages[i]) for i in which), len(ls))
        host = np.zeros(layout.size, dtype=np.int32)
        fill_host(layout, host, tokens=[[0]] * len(ls), starts=[n - 1 for n in ls], slots=[1 + i for i in range(len(ls))],
                  pages=[pages[i] for i in which], want=[[0]] * len(ls))
        batch = StepBatch(layout, torch.from_numpy(host).to(DEV), q_lens=[1] * len(ls), starts=[n - 1 for n in ls])
        scratch = torch.empty(ops.attention_decode_scratch_floats(len(ls), H, hd, max(ls), dtype), device=DEV)
        return ops.attention_decode(q[which].contiguous(), store, batch, hd ** -0.5, scratch), pages
    many, pages = run(list(range(len(lens))))
    for i in range(8):
        assert torch.equal(run([i])[0][0], many[i]), lens[i]
        k, v = (torch.cat([store[p, a] for p in pages[i]], 1)[:, :lens[i]].double() for a in (0, 1))
        z = torch.softmax(torch.einsum("ghd,gkd->ghk", q[i].double().view(G, H // G, hd), k) * hd ** -0.5, -1)
        ref = (z @ v).reshape(H, hd)
        # (float32 sums of at most 1,025 terms: below 1e-5; the result's own rounding to bfloat16 2^-9)
        assert (many[i].double() - ref).abs().max() < (1e-5 if dtype == torch.float32 else 2 ** -8) * max(1.0, float(ref.abs().max()))
    ops.check_status()


def test_a_prompt_product_in_three_runs():
    """Few tiles for the pairs of SMs, an inner dimension of three runs of 32 steps at most."""
    from wick_b200.ops import gemm_tc as G
    g = torch.Generator().manual_seed(3)
    w, x = (torch.randn(1000, 6144, generator=g) / 78).bfloat16().to(DEV), torch.randn(300, 6144, generator=g).bfloat16().to(DEV)
    plan = G.plan_for(w)
    assert plan.prompt_splits(300) == 3
    parts = plan.forward_delta(x)
    G.check_status()
    assert parts.shape == (3, 300, 1000)
    assert (parts.sum(0).double() - x.double() @ w.double().T).abs().max() < 1e-5 * 5


@pytest.mark.parametrize("t, k, out, pair", [(4357, 7400, 300, False), (2305, 14000, 513, True), (4096, 7688, 257, False)])
def test_prompt_products_in_slabs_of_rows_are_those_of_fewer_rows(t, k, out, pair):
    """More than 60 MB of activations: the tiles come in slabs of rows, every tile computed as it is in a product of fewer rows."""
    from wick_b200.ops import gemm_tc
    g = torch.Generator().manual_seed(t)
    plan = gemm_tc.plan_for((torch.randn(2 * out if pair else out, k, generator=g) / math.sqrt(k)).bfloat16().to(DEV), gated=pair)
    x = torch.randn(t, k, generator=g).bfloat16().to(DEV)
    assert x.numel() * 2 > 60 << 20
    got = plan.forward(x, torch.bfloat16)
    for a in (0, 1024, t - 700):
        assert torch.equal(got[a:a + 700], plan.forward(x[a:a + 700].contiguous(), torch.bfloat16))
    ops.check_status()


@pytest.mark.parametrize("ff", [8192, 8196, 16384, 16388])
@pytest.mark.parametrize("n", [1, 148, 149])
@pytest.mark.parametrize("splits", [1, 3])
def test_poly_norm_forms(ff, n, splits):
    g = torch.Generator().manual_seed(ff + n)
    parts = (0.7 * torch.randn(splits, n, ff, generator=g)).to(DEV)
    z = parts.double().sum(0)
    co = torch.tensor([0.5, -1.2, 0.8, 0.3], device=DEV)
    ref = sum(c * z ** (i + 1) / torch.sqrt((z ** (2 * i + 2)).mean(1, keepdim=True) + 1e-5) for i, c in enumerate(co.tolist()[:3])) + 0.3
    got = ops.poly_norm(parts, co, 1e-5, torch.float32)
    assert (got.double() - ref).abs().max() < 5e-6 * float(ref.abs().max())
    assert torch.equal(ops.poly_norm(parts, co, 1e-5, torch.bfloat16), got.bfloat16())


# Decode attention and the product that reads it, one behind the other without a look in between, over several caches in turn.
_ATTENTION_THEN_PRODUCT = """
import sys
sys.path[:0] = [{root!r}, {tests!r}]
import torch
from wick_b200 import ops
from wick_b200.ops import gemm_tc as G
from test_gpu_forms import DEV, batch_of
lens, mask, size, heads, kv = {case!r}
batch, pages, n_pages = batch_of([1] * len(lens), [n - 1 for n in lens])
g = torch.Generator().manual_seed(5)
store = [torch.randn(n_pages, 2, kv, 64, 64, generator=g).bfloat16().to(DEV) for _ in range(4)]
q = [torch.randn(len(lens), heads, 64, generator=g).bfloat16().to(DEV) for _ in range(4)]
plan = G.plan_for(torch.randn(256, heads * 64, generator=g).bfloat16().to(DEV))
scratch = torch.empty(max(1, ops.attention_decode_parts_scratch(len(lens), heads, kv, 64, 4096)), device=DEV)
att = torch.zeros(len(lens), heads, 64, dtype=torch.bfloat16, device=DEV)
got = []
torch.cuda.synchronize()
for i in range(16):
    if mask:
        a = ops.attention_masked(q[i % 4], store[i % 4], batch, 0.2, n_kv=kv, v_dim=64, mask=mask, mask_size=size, kind="bulk")
    else:
        a = ops.attention_decode_parts(q[i % 4], store[i % 4], batch, 0.2, scratch, out=att, max_kv_len=4096)    # (sized as in a captured step)
    got.append(plan.forward_delta(a.view(len(lens), -1)))
ops.check_status()
torch.save([x.cpu() for x in got], sys.argv[1])
"""


@pytest.mark.parametrize("case", [
    ([700 + i for i in range(40)], "window", 64, 8, 4), ([64 + 65 * (i % 20) for i in range(40)], "window", 65, 8, 4),
    ([1025 + i for i in range(40)], "block", 1024, 8, 4), ([100] * 64, None, 0, 16, 8)])
def test_what_follows_a_decode_attention_with_nothing_to_merge_waits_for_it(case, tmp_path):
    """More pairs of sequence and key head than multiprocessors, every pair in one part (its rows are written by the parts' kernel, the
    merge behind it has nothing to do): the product that reads the rows gives the same bits with dependent launch and without."""
    got = []
    for off in ("0", "1"):
        out = str(tmp_path / off)
        run = subprocess.run([sys.executable, "-c", _ATTENTION_THEN_PRODUCT.format(root=ROOT, tests=os.path.join(ROOT, "tests"), case=case), out],
                             env=dict(os.environ, WICK_B200_NO_PDL=off, WICK_B200_PAIR_DECODE="0"), capture_output=True, text=True, timeout=300)
        assert run.returncode == 0, run.stderr[-2000:]
        got.append(torch.load(out))
    assert all(torch.equal(a, b) for a, b in zip(*got))
    assert all(torch.isfinite(a).all() for a in got[0])


@pytest.mark.parametrize("d, heads, kv", [(64, 20, 4), (128, 16, 16)])
@pytest.mark.parametrize("start, mask, size, pos, clean", [(0, "causal", 0, 200, (0, 128)), (64, "window", 16, 100, (128, 256)), (64, "block", 128, 300, (0, 128))])
def test_prompt_rows_do_not_show_values_of_key_blocks_they_see_nothing_of(d, heads, kv, start, mask, size, pos, clean):
    """Two tiles of 128 tokens a block: a value that is no number lies in a key block (128 positions) that only one of them sees."""
    lens, starts = [256] * 16, [start] * 16
    batch, pages, n_pages = batch_of(lens, starts)
    g = torch.Generator().manual_seed(d + start)
    store = torch.randn(n_pages, 2, kv, PAGE, d, generator=g).bfloat16()
    for b, bad in ((0, float("nan")), (7, float("inf")), (15, -float("inf"))):
        store[pages[b][pos // PAGE], 1, :, pos % PAGE] = bad
    q = torch.randn(sum(lens), heads, d, generator=g).bfloat16()
    out = ops.attention_masked(q.to(DEV), store.to(DEV), batch, 0.2, n_kv=kv, v_dim=d, mask=mask, mask_size=size, kind="tc").cpu()
    ref = ops.attention_masked(q.to(DEV), store.to(DEV), batch, 0.2, n_kv=kv, v_dim=d, mask=mask, mask_size=size, kind="warp").cpu()
    ops.check_status()
    for b in range(16):
        a, z = 256 * b + clean[0], 256 * b + clean[1]
        assert torch.isfinite(ref[a:z].float()).all() and torch.isfinite(out[a:z].float()).all(), b
        assert (out[a:z].float() - ref[a:z].float()).abs().max() < 0.02
    assert not torch.isfinite(out[:256].float()).all(), "and those that see it show it"


@pytest.mark.parametrize("heads, kv", [(64, 16), (64, 8), (40, 8)])
def test_prompt_rows_of_a_step_of_few_tokens_do_not_depend_on_the_other_sequences(heads, kv):
    """Up to 64 tokens in a step: a sequence's rows are the same bits alone and among others, however many items the step makes."""
    d, lens, starts = 64, [33] + [1] * 31, [500] + [130 + 7 * i for i in range(31)]
    batch, pages, n_pages = batch_of(lens, starts)
    g = torch.Generator().manual_seed(heads)
    store = torch.randn(n_pages, 2, kv, PAGE, d, generator=g).bfloat16().to(DEV)
    q = torch.randn(sum(lens), heads, d, generator=g).bfloat16().to(DEV)
    full = ops.attention_prompt(q, store, batch, 0.2)
    at = 0
    for b, n in enumerate(lens[:3]):
        one, own, _ = batch_of([n], [starts[b]])
        one.page_table.copy_(torch.tensor([pages[b]], dtype=torch.int32))
        assert torch.equal(ops.attention_prompt(q[at:at + n].contiguous(), store, one, 0.2), full[at:at + n]), b
        at += n
    ops.check_status()


def prompt_case(lens, starts, d, heads, kv, seed):
    """Sequences whose caches hold NaN behind their ends; queries; the step."""
    batch, pages, n_pages = batch_of(lens, starts)
    g = torch.Generator().manual_seed(seed)
    store = torch.full((n_pages, 2, kv, PAGE, d), float("nan"))
    for n, s, own in zip(lens, starts, pages):
        for i, page in enumerate(own):
            rows = min(PAGE, n + s - i * PAGE)
            store[page, :, :, :rows] = torch.randn(2, kv, rows, d, generator=g)
    q = torch.randn(sum(lens), heads, d, generator=g)
    return q.bfloat16().to(DEV), store.bfloat16().to(DEV), batch


def prompt_items(lens, heads, kv, tokens):
    """Work items of a prompt step whose items are ``tokens`` tokens of 128 rows each: (items, those a multiprocessor gets)."""
    group = heads // kv
    gs = max(g for g in range(1, group + 1) if group % g == 0 and 128 % g == 0)
    items = sum(-(-n // (tokens * (128 // gs))) for n in lens) * (heads // gs)
    return items, items / torch.cuda.get_device_properties(0).multi_processor_count


# 40 sequences (more than a warp's lanes), a few of more than eight blocks of 128 keys
MANY = ([5 + 37 * (i % 23) for i in range(36)] + [700, 128, 129, 1], [(61 * i) % 300 for i in range(36)] + [1100, 1500, 0, 2000])


@pytest.mark.parametrize("d, heads, kv, lens, starts, a_block", [
    (128, 32, 8, *MANY, 4), (64, 16, 2, *MANY, 2), (128, 10, 2, *MANY, 1), (64, 6, 6, *MANY, 1),
    (64, 64, 16, [400 + i for i in range(64)], [0] * 64, 16), (64, 6, 2, [300] * 100 + [1000], [0] * 100 + [300], 4)])
@pytest.mark.parametrize("mask, size", [("causal", 0), ("block", 500), ("window", 300), ("window", 129)])
def test_prompt_attention_of_two_tiles_a_block_item_behind_item(d, heads, kv, lens, starts, a_block, mask, size):
    """Steps whose items are two tiles a block and several a block (more than 16: several rounds of blocks), one, two, four and eight
    heads to a tile, of more than 32 sequences, of up to eight key blocks and of more, with masks and sinks; against the kernel that
    takes row by row in float32.  A rounding to bfloat16 (8 bits) is off by at most 2^-8 of the number: the
    probabilities' by 2^-8 of the largest value together, the two results' by 2^-8 of themselves each."""
    one, each = prompt_items(lens, heads, kv, 1)
    two, _ = prompt_items(lens, heads, kv, 2)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert one > 2 * sms and two > 2 * sms and two / sms > a_block, (one, two)
    q, store, batch = prompt_case(lens, starts, d, heads, kv, heads + size)
    sink = torch.randn(heads, generator=torch.Generator().manual_seed(1)).to(DEV)
    for sk in (sink, None):
        kw = dict(n_kv=kv, v_dim=d, mask=mask, mask_size=size, sink=sk)
        out = ops.attention_masked(q, store, batch, d ** -0.5, kind="tc", **kw).float()
        ref = ops.attention_masked(q, store, batch, d ** -0.5, kind="warp", **kw).float()
        ops.check_status()
        assert torch.isfinite(out).all()
        assert ((out - ref).abs() <= 2 ** -8 * 6 + 2 ** -7 * ref.abs()).all()          # (values are normal: none is beyond 6)


@pytest.mark.parametrize("d, heads, kv", [(64, 16, 4), (128, 6, 6), (64, 10, 2)])
@pytest.mark.parametrize("window, block, cap", [(200, 16, 30.0), (130, 1, None), (0, 0, 5.0)])
def test_prompt_attention_beside_blocks_of_two_tiles_a_block_item_behind_item(d, heads, kv, window, block, cap):
    """The form with blocks of positions before the window, capped scores and a factor of the result, at the same kinds of steps."""
    lens = [5 + 37 * (i % 23) for i in range(36)] + [1700, 128, 129, 1]
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    lens = lens * (1 if prompt_items(lens, heads, kv, 2)[0] > 2 * sms else 4)
    assert prompt_items(lens, heads, kv, 2)[0] > 2 * sms
    q, store, batch = prompt_case(lens, [0] * len(lens), d, heads, kv, window + block)
    flat = store.view(store.shape[0], -1)
    gate = torch.rand(q.shape[0], heads, generator=torch.Generator().manual_seed(2)).to(DEV)
    got = {}
    for kind in ("tc", "rows"):
        means = torch.full((store.shape[0], kv * ops.block_rows(block) * 2 * d), float("nan"), dtype=torch.bfloat16, device=DEV) if block else None
        got[kind] = ops.attention_pooled(q, flat, batch, d ** -0.5, n_kv=kv, v_dim=d, window=window, store=means, block=block, soft_cap=cap,
                                         gate=gate, kind=kind).float()
    ops.check_status()
    assert torch.isfinite(got["tc"]).all()
    assert ((got["tc"] - got["rows"]).abs() <= 2 ** -8 * 6 + 2 ** -7 * got["rows"].abs()).all()


@pytest.mark.parametrize("lens, starts", [([400], [0]), ([70, 1, 130], [900, 500, 800])])
def test_prompt_rows_do_not_depend_on_the_width_of_the_page_table(lens, starts):
    """A table of up to 16 pages (1,024 positions) takes the kernel without the code for long items, a wider one the kernel with it."""
    d, heads, kv = 128, 8, 2
    q, store, batch = prompt_case(lens, starts, d, heads, kv, 12)
    assert batch.table_width <= 16
    layout = BatchLayout(len(lens), sum(lens), 40, 0)
    host = np.zeros(layout.size, dtype=np.int32)
    fill_host(layout, host, tokens=[[0] * n for n in lens], starts=starts, slots=[1 + i for i in range(len(lens))],
              pages=[[int(p) for p in row] for row in batch.page_table.cpu()], want=[[]] * len(lens))
    wide = StepBatch(layout, torch.from_numpy(host).to(DEV), q_lens=lens, starts=starts)
    assert torch.equal(ops.attention_prompt(q, store, batch, 0.1), ops.attention_prompt(q, store, wide, 0.1))
    ops.check_status()
