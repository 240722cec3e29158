"""The rules that send a call to one kernel or another, as far as they can be looked at without a GPU."""
import pytest
import torch

from wick_b200 import ops


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
