"""Attention of one 384-channel head (csrc/attn_wide_sm100.cu) against softmax(q k^T) v in 64 bits."""
import pytest
import torch

from vllm_omni_b200.ops import _native as nv
from vllm_omni_b200.ops import conv as C

pytestmark = pytest.mark.gpu


def _exact(q, k, v):
    q, k, v = q.double(), k.double(), v.double()
    return torch.softmax(q @ k.transpose(1, 2) * q.shape[2] ** -0.5, -1) @ v


# rows below, at and past a tile of 256 and a step of 128 keys; runs of work that begin and end inside tiles (workers not a multiple of the tiles)
@pytest.mark.parametrize("B,N,workers", [(1, 1, 0), (1, 63, 0), (1, 64, 0), (1, 127, 0), (1, 128, 0), (1, 129, 2), (2, 256, 0), (2, 257, 7), (1, 1000, 0), (1, 1024, 5),
                                         (3, 700, 33), (1, 4099, 74), (1, 4099, 17), (1, 4099, 0), (2, 9999, 0)])
def test_wide_attention(B, N, workers):
    g = torch.Generator(device="cuda").manual_seed(N)
    t = torch.randn(B, N, 3, 384, device="cuda", generator=g).bfloat16()
    t[..., :2, :] *= 3.0                                   # scores of several units: row maxima grow, weights are uneven
    q, k, v = t[:, :, 0], t[:, :, 1], t[:, :, 2]
    out = C._wide_head_flash(q, k, v, 384 ** -0.5, workers)
    torch.cuda.synchronize()
    nv.check_status(q.device)
    ref = _exact(q, k, v)
    # probabilities and results are bf16 (2^-9 each, at worst aligned), the exponentials 2^-22
    assert (out.double() - ref).norm() <= 2 ** -8 * ref.norm()
    assert (out.double() - ref).abs().max() <= 2 ** -7 * v.abs().max()


def test_wide_attention_growing_maxima():
    """Keys sorted by their score: every step raises the maximum by more than the kernel lets pass without rescaling."""
    N = 640
    g = torch.Generator(device="cuda").manual_seed(1)
    d = torch.randn(384, device="cuda", generator=g)
    q = (d + 0.1 * torch.randn(1, N, 384, device="cuda", generator=g)).bfloat16()
    k = (torch.linspace(-6, 6, N, device="cuda")[None, :, None] * d).bfloat16()
    v = torch.randn(1, N, 384, device="cuda", generator=g).bfloat16()
    ref = _exact(q, k, v)
    for workers in (0, 11):
        out = C._wide_head_flash(q, k, v, 384 ** -0.5, workers)
        torch.cuda.synchronize()
        nv.check_status(q.device)
        assert (out.double() - ref).norm() <= 2 ** -8 * ref.norm()


@pytest.mark.parametrize("N,workers,launches", [(256, 1, 1), (512, 2, 1), (512, 3, 2), (300, 2, 1), (300, 6, 2)])
def test_launches_are_counted(N, workers, launches):
    q = torch.zeros(1, N, 384, device="cuda", dtype=torch.bfloat16)
    before = nv.launch_count
    C._wide_head_flash(q, q, q, 1.0, workers)
    assert nv.launch_count - before == launches


def test_wide_attention_of_shared_keys():
    """Two batch entries with the same keys and values (a batch stride of zero)."""
    g = torch.Generator(device="cuda").manual_seed(6)
    q, k, v = (torch.randn(n, 264, 384, device="cuda", generator=g).bfloat16() for n in (2, 1, 1))
    out = C.wide_head_attention(q, k.expand(2, -1, -1), v.expand(2, -1, -1))
    nv.check_status(q.device)
    assert torch.equal(out, C.wide_head_attention(q, k.repeat(2, 1, 1), v.repeat(2, 1, 1)))


@pytest.mark.parametrize("workers", [0, 1, 5])
def test_scores_of_minus_infinity(workers):
    """Rows whose first keys score -inf (products past the range of fp32) beside rows of the same warp whose maxima grow: those keys weigh nothing."""
    N, dead = 640, 300
    g = torch.Generator(device="cuda").manual_seed(4)
    q, k, v = (torch.randn(1, N, 384, device="cuda", generator=g).bfloat16() for _ in range(3))
    k *= torch.linspace(1, 12, N, device="cuda")[None, :, None].bfloat16()
    q[..., 0], k[..., 0] = 0.0, 0.0
    q[:, ::3, 0], k[:, :dead, 0] = -1e30, 1e30
    out = C._wide_head_flash(q, k, v, 384 ** -0.5, workers)
    torch.cuda.synchronize()
    nv.check_status(q.device)
    s = q.double() @ k.double().transpose(1, 2) * 384 ** -0.5
    s[:, ::3, :dead] = float("-inf")
    ref = torch.softmax(s, -1) @ v.double()
    # probabilities and results are bf16, the exponentials 2^-22
    assert torch.isfinite(out).all() and (out.double() - ref).norm() <= 2 ** -8 * ref.norm()


def test_wide_attention_width_outside_the_kernel():
    """512 channels stay with the two GEMMs around the row softmax, whose scores pass through bf16 as well."""
    g = torch.Generator(device="cuda").manual_seed(2)
    q, k, v = (torch.randn(1, 520, 512, device="cuda", generator=g).bfloat16() for _ in range(3))
    out, ref = C.wide_head_attention(q, k, v, chunk_rows=256), _exact(q, k, v)
    nv.check_status(q.device)
    assert (out.double() - ref).norm() <= 2 ** -7 * ref.norm()
