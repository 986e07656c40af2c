"""Scratch of the experts: one set for the layers of a decoder, none in common between decoders, whose steps run in threads and on
streams of their own."""
import copy

import pytest
import torch

from vllm_omni_b200.ops.moe import MoEWorkspace


def _qwen():
    from vllm_omni_b200.models.qwen_decoder import DecoderConfig, QwenDecoderModel
    return QwenDecoderModel(DecoderConfig(vocab_size=16, hidden_size=16, num_hidden_layers=2, num_attention_heads=2, num_key_value_heads=1, head_dim=8,
                                          intermediate_size=16, num_experts=4, num_experts_per_tok=2, moe_intermediate_size=8))


def _hunyuan():
    from vllm_omni_b200.diffusion.models.hunyuan_image_3.transformer import HunyuanImage3Config, HunyuanImage3Model
    return HunyuanImage3Model(HunyuanImage3Config(vocab_size=16, hidden_size=16, num_hidden_layers=2, num_attention_heads=2, num_key_value_heads=1,
                                                  head_dim=8, intermediate_size=8, moe_intermediate_size=8, num_experts=4, moe_topk=2))


def _milivik():
    from vllm_omni_b200.models.milivik import MilivikConfig, MilivikDecoder, tiny_config_dict
    return MilivikDecoder(MilivikConfig.from_dict(tiny_config_dict()))


def _nidilix():
    from vllm_omni_b200.models.nidilix import NidilixConfig, NidilixDecoder, tiny_config_dict
    return NidilixDecoder(NidilixConfig.from_dict(tiny_config_dict()))


def _buffers(decoder):
    ws = [v for m in decoder.modules() for v in vars(m).values() if isinstance(v, MoEWorkspace)]
    assert ws
    return [{n: t.data_ptr() for n, t in vars(w.get(5, 2, 4, 16, 8, "cpu", torch.bfloat16)).items() if isinstance(t, torch.Tensor) and t.numel()}
            for w in ws]


@pytest.mark.parametrize("make", [_qwen, _hunyuan, _milivik, _nidilix])
def test_layers_share_and_decoders_do_not(make):
    one = make()
    a, b, c = _buffers(one), _buffers(make()), _buffers(copy.deepcopy(one))
    for bufs in (a, b, c):
        assert all(x == bufs[0] for x in bufs)
    pools = [set(x[0].values()) for x in (a, b, c)]
    assert "xp" in a[0] and not (pools[0] & pools[1]) and not (pools[0] & pools[2])


def test_workspaces_of_their_own():
    a, b = (MoEWorkspace().get(5, 2, 4, 16, 8, "cpu", torch.bfloat16) for _ in range(2))
    assert a.y.data_ptr() != b.y.data_ptr()
    assert a.get(3, 2, 4, 16, 8, "cpu", torch.bfloat16).y.data_ptr() == a.get(64, 2, 4, 16, 8, "cpu", torch.bfloat16).y.data_ptr()   # a bucket keeps them
