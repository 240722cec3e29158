"""Forms of kernels chosen by size, each at the sizes where it can go wrong, against 64-bit products and sums.

Tolerances: a float32 sum of k products of numbers of order one and 1 / sqrt(k) differs from the exact one by a few 2^-24 times
sqrt(k) of its own size at most, i.e. below 1e-5 for the sizes here; a result rounded to bfloat16 by 2^-9 of itself."""
import math
import types

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from wick_b200 import ops  # noqa: E402
from wick_b200.engine.batch import BatchLayout, StepBatch, fill_host  # noqa: E402

DEV = "cuda"
PAGE = 64


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
