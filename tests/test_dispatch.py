"""The rules that send a call to one kernel or another, as far as they can be looked at without a GPU."""
import os
import re

import pytest
import torch

from wick_b200 import ops
from wick_b200.ops.build import CSRC


@pytest.mark.parametrize("hd", [64, 128])
def test_decode_attention_by_parts_is_offered_only_what_its_library_takes(hd):
    """The kernel holds a step's lengths in shared memory and refuses more sequences than fit there; a step of more has to
    go to the other decode kernels, not to an error."""
    lib = ops._attn(hd)._lib
    for n in (0, 1, 512, 1023, 1024, 1025, 1500, 2048, 2049):
        for heads, kv in ((8, 2), (8, 1), (9, 1), (18, 2), (7, 2), (4, 0)):
            want = bool(lib.wick_attn_decode_parts_supported(n, heads, kv))
            assert ops.attention_decode_parts_supported(n, heads, kv, hd, torch.bfloat16) == want, (n, heads, kv)
    assert ops.attention_decode_parts_supported(1024, 8, 2, hd, torch.bfloat16)
    assert not ops.attention_decode_parts_supported(1025, 8, 2, hd, torch.bfloat16)
    assert not ops.attention_decode_parts_supported(1, 8, 2, hd, torch.float32)
    assert not ops.attention_decode_parts_supported(1, 8, 2, 32, torch.bfloat16)


def test_decode_attention_by_parts_refuses_query_rows_it_cannot_read():
    """Rows are read two numbers at a time: an address that is no multiple of 4 is an error of the call, not of the device."""
    lib = ops._attn(64)
    for at, message in ((1 << 20, None), ((1 << 20) + 2, "multiple of 4 bytes")):
        try:
            lib.call("wick_attn_decode_parts_masked_bf16", "pplpplpiipiiifpiipp", at, 1 << 20, 4, 1 << 20, 1 << 20, 0 if message is None else 1 << 20,
                     1 << 20, 1, 64, 1 << 20, 1, 4, 2, 0.1, 1 << 20, 2, 64, None, 0)
            got = ""
        except ops.KernelError as e:
            got = str(e)
        assert got and (message is None) == ("multiple of 4 bytes" not in got), got       # (the first call is refused for its scratch)


def _enclosed(text, at, pair="{}"):
    """The text from the bracket that opens at or behind ``at`` to the one that closes it."""
    begin = at = text.index(pair[0], at)
    depth = 0
    while True:
        depth += {pair[0]: 1, pair[1]: -1}.get(text[at], 0)
        if depth == 0:
            return text[begin:at + 1]
        at += 1


def _kernels():
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, f)) as fh:
                text = re.sub(r"//[^\n]*", "", fh.read())
            for m in re.finditer(r"__global__", text):
                name = re.compile(r"\w+_kernel(?=\()").search(text, m.end())
                args = _enclosed(text, name.end(), "()")
                yield f, name.group(), _enclosed(text, name.end() + len(args))


def test_no_kernel_that_lets_its_successor_start_ends_before_it_has_waited():
    """A kernel waits for the one before it only (griddepcontrol.wait), so that one must not have ended before ITS predecessor has: no
    thread may leave ahead of the wait.  (Were every thread to leave there, nothing would order the kernel behind it and the kernel
    ahead of it.)"""
    found = 0
    for f, name, body in _kernels():
        if "pdl_trigger" not in body:
            continue
        found += 1
        while True:                                    # a lambda's own returns leave the lambda only
            m = re.search(r"\[[&=]?\]\s*\([^()]*\)\s*(?:->\s*\w+\s*)?(?=\{)", body)
            if not m:
                break
            body = body[:m.start()] + body[m.end() + len(_enclosed(body, m.end())):]
        first = body.find("return")
        if name == "attn_decode_parts_kernel":         # its warps without a part leave, where there are warps with one
            assert "if (before == 0) pdl_wait();" in body[:first]
            first = body.find("return", first + 1)
        assert "pdl_wait()" in body[:first if first >= 0 else len(body)], f"{name} ({f}) may end before its wait"
    assert found > 40, "the kernels' sources are not where they were"
