"""Which kernel decodes a batch (ops/kv_cache.py decode_impl), and the scratch of its splits."""
import pytest
import torch

from vllm_omni_b200.ops import kv_cache as KC


def test_split_scratch_is_the_calls_own():
    a, b = (KC._scratch_for(torch.device("cpu"), 12, 128) for _ in range(2))
    assert [t.numel() for t in a] == [12 * 128, 24] and not {t.data_ptr() for t in a} & {t.data_ptr() for t in b}
