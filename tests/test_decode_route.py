"""Which kernel decodes a batch (ops/kv_cache.py decode_impl), and the scratch of its splits."""
import pytest
import torch

from vllm_omni_b200.ops import kv_cache as KC


def test_split_scratch_is_the_calls_own():
    a, b = (KC._scratch_for(torch.device("cpu"), 12, 128) for _ in range(2))
    assert [t.numel() for t in a] == [12 * 128, 24] and not {t.data_ptr() for t in a} & {t.data_ptr() for t in b}


@pytest.mark.parametrize("H,Hkv", [(8, 8), (16, 8), (28, 4), (32, 4), (36, 3), (64, 4), (40, 2), (256, 1)])
@pytest.mark.parametrize("bs", [4, 8, 16, 24, 48, 64, 128, 256])
def test_route(H, Hkv, bs):
    """Weights stay in fp32 where they were: pages that the tensor-core kernel does not take, group sizes of the fp32 kernel."""
    G, tiles = H // Hkv, bs % 8 == 0 and 128 % bs == 0
    for n in (1, 3, 16, 64, 300):
        impl = KC.decode_impl(n, H, Hkv, 128, bs, None, H * 128, H * 128)
        if not tiles and G in (1, 2, 4, 8):
            assert impl == "simt"
        elif tiles and G <= 128:
            assert impl in (("stream", "tc") if G <= 16 else ("tc",))
        assert impl != "stream" or (bs % 8 == 0 and G <= 16)                  # what csrc/decode_attn.cu takes
        assert impl != "tc" or (tiles and G <= 128)
        assert KC.decode_impl(n, H, Hkv, 128, bs, 4, H * 128, H * 128) == ("tc" if tiles and G <= 128 else "simt")
    assert KC.decode_impl(4, H, Hkv, 64, bs, None, H * 64, H * 64) == "simt"


@pytest.mark.parametrize("H,Hkv,n,impl", [(64, 4, 4, "stream"), (64, 4, 5, "tc"), (64, 4, 37, "tc"), (64, 4, 38, "stream"), (64, 4, 66, "stream"),
                                          (64, 4, 67, "tc"), (64, 4, 74, "tc"), (64, 4, 75, "stream"), (32, 2, 8, "stream"), (32, 2, 9, "tc"),
                                          (16, 1, 148, "tc"), (16, 1, 149, "stream"), (36, 3, 2, "tc"), (36, 3, 200, "tc"), (32, 4, 40, "stream")])
def test_groups_of_9_to_16_heads(H, Hkv, n, impl):
    assert KC.decode_impl(n, H, Hkv, 128, 16, None, H * 128, H * 128) == impl
