"""Channels-last execution of the image VAE decoder on the sm_100a kernels.

Built from a ``Decoder2d`` (same parameters, repacked once): every convolution is an implicit
GEMM on the tcgen05 kernel with bias / residual in its epilogue, RMS-norm + SiLU ride in it too where a tile holds all
channels (192 and 96 of the published decoder) and are one fused kernel per pixel row elsewhere, a doubled image is read as the small one, activations stay NHWC bf16 from the latent to the image.  The single
mid-block attention (one head of width C, outside the flash kernel's head sizes) is one launch at 384 channels and two GEMMs
around a row-softmax kernel at other widths (``ops.conv.wide_head_attention``).  Replaces the cuDNN path the
reference takes through diffusers (vllm_omni/diffusion/models/qwen_image/
autoencoder_kl_qwenimage.py).
"""
from __future__ import annotations

import torch

from ....ops import conv as C


class _Conv:
    def __init__(self, m: torch.nn.Conv2d, dtype):
        self.k = m.kernel_size[0]
        self.cin, self.cout = m.in_channels, m.out_channels
        self.w, self.b = C.pack_conv_weight(m.weight.data, m.bias.data if m.bias is not None else None, dtype)

    def __call__(self, x, act=None, residual=None):
        return C.conv2d_nhwc(x, self.w, self.b, self.k, self.cin, act=act, residual=residual)

    def then_norm(self, x, norm, residual=None, up=False, keep=True):
        """(result, its norm): ``norm`` is (gamma, SiLU or not), or None where no norm follows."""
        gamma, silu = norm or (None, False)
        return C.conv3x3_norm_nhwc(x, self.w, self.b, self.cin, residual=residual, up=up, gamma=gamma, silu=silu, keep=keep)


class NHWCDecoder:
    def __init__(self, decoder, post_quant_conv=None, dtype=torch.bfloat16):
        d = decoder
        g = lambda n: n.gamma.data.to(dtype).contiguous()
        self.dtype = dtype
        self.post_quant = _Conv(post_quant_conv, dtype) if post_quant_conv is not None else None
        self.conv_in = _Conv(d.conv_in, dtype)
        self.stages = []
        for m in list(d.mid) + [m for blk in d.up_blocks for m in blk]:
            name = type(m).__name__
            if name == "ResBlock":
                self.stages.append(("res", g(m.norm1), _Conv(m.conv1, dtype), g(m.norm2), _Conv(m.conv2, dtype),
                                    _Conv(m.shortcut, dtype) if m.shortcut is not None else None))
            elif name == "AttnBlock":
                self.stages.append(("attn", g(m.norm), _Conv(m.to_qkv, dtype), _Conv(m.proj, dtype)))
            elif name == "Upsample":
                self.stages.append(("up", _Conv(m.conv, dtype)))
            else:
                raise TypeError(f"unexpected decoder block {name}")
        self.norm_out = g(d.norm_out)
        # the norm that reads the result of conv_in, then of every stage
        self.norms = [(st[1], st[0] == "res") if st[0] != "up" else None for st in self.stages] + [(self.norm_out, True)]
        self.conv_out = _Conv(d.conv_out, dtype)

    @torch.no_grad()
    def __call__(self, z: torch.Tensor, uint8: bool = False) -> torch.Tensor:
        """z: [B, z_dim, h, w] de-normalised latents -> [B, 3, 8h, 8w] fp32 in [-1, 1] (or uint8 NHWC)."""
        x = C.nchw_to_nhwc(z, dtype=self.dtype)
        if self.post_quant is not None:
            x = self.post_quant(x)
        x, n = self.conv_in.then_norm(x, self.norms[0])
        for i, st in enumerate(self.stages):
            norm = self.norms[i + 1]
            if st[0] == "res":
                _, _, c1, g2, c2, sc = st
                skip = x if sc is None else sc(x)
                x, n = c2.then_norm(c1.then_norm(n, (g2, True), keep=False)[1], norm, residual=skip, keep=i + 1 < len(self.stages))
            elif st[0] == "attn":
                _, _, qkv, proj = st
                B, H, W, ch = x.shape
                t = qkv(n).view(B, H * W, 3, ch)
                o = C.wide_head_attention(t[:, :, 0], t[:, :, 1], t[:, :, 2])
                x = proj(o.reshape(B, H, W, ch).contiguous(), residual=x)
                n = None if norm is None else C.rmsnorm_silu_nhwc(x, norm[0], silu=norm[1])
            else:
                x, n = st[1].then_norm(x, norm, up=True)
        x = self.conv_out(n)
        return C.nhwc_to_image(x, uint8=uint8)
