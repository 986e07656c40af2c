"""Row kernels at the sizes where their layout changes: norms of more than 1024 channels (a block per row, or some warps per row), head
norms with rotation of few and of many rows, with and without pages."""
import pytest
import torch

from vllm_omni_b200.ops import fused, kv_cache as KC

pytestmark = pytest.mark.gpu


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


@pytest.mark.parametrize("width", [1024, 1032, 2048, 3072, 4096, 6152, 8192])
@pytest.mark.parametrize("rows", [1, 6, 1183, 1184, 5002])
@pytest.mark.parametrize("rms", [True, False])
def test_norm_modulate(width, rows, rms):
    _norm(width, rows, rms)


@pytest.mark.parametrize("width", [1032, 2048, 2056, 2560, 2568, 3072, 3080, 4096, 4104, 5120, 5128, 6144, 6152, 8192])
@pytest.mark.parametrize("per_sm", [1, 2, 4, 5, 12, 16])
def test_norm_layouts(width, per_sm):
    """Both sides of every limit, in rows per SM, at which the number of warps per row changes, at the widths where the chunks per lane do."""
    rows = per_sm * torch.cuda.get_device_properties(0).multi_processor_count
    for r in (rows, rows + 1):
        _norm(width, r, r % 2 == 0)


def _norm(width, rows, rms):
    g = _gen(width + rows)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    b = 1 if rows % 2 else 2
    x, out = rnd(b, rows // b, width + 8)[..., :width], torch.full((b, rows // b, width + 16), 3.0, device="cuda", dtype=torch.bfloat16)
    mods = rnd(b, 3 * width)
    for kw in (dict(weight=rnd(width)), dict(shift=mods[:, :width], scale=mods[:, width:2 * width]), dict(weight=rnd(width), bias=rnd(width)), {}):
        x = x.contiguous() if x.shape[0] > 1 else x
        y = fused.norm_modulate(x, rms=rms, eps=1e-6, out=out[..., :width].clone(), **kw)
        f = x.double()
        f = f if rms else f - f.mean(-1, keepdim=True)
        ref = f * torch.rsqrt((f * f).mean(-1, keepdim=True) + 1e-6)
        if "weight" in kw:
            ref = ref * kw["weight"].double()
        if "bias" in kw:
            ref = ref + kw["bias"].double()
        if "scale" in kw:
            ref = ref * (1 + kw["scale"].double()[:, None]) + kw["shift"].double()[:, None]
        # half an ulp of bf16, and fp32 arithmetic before it (sums of up to 8192 squares, cancellation against a shift)
        assert ((y.double() - ref).abs() <= ref.abs() * 2.0 ** -8 + 2e-5).all()


@pytest.mark.parametrize("rows", [1, 5, 64, 700, 1300, 2400])
@pytest.mark.parametrize("heads,kv", [(32, 4), (3, 1), (24, 24)])
@pytest.mark.parametrize("interleaved", [False, True])
def test_head_norm_rotation_and_pages(rows, heads, kv, interleaved):
    _heads_and_pages(rows, heads, kv, interleaved)


# rows enough for a warp per row with every count: heads and pages that leave 0, 1, 2 and 6 of a step of 8 over (without pages
# heads + kv, with them heads + 2 kv)
@pytest.mark.parametrize("heads,kv", [(7, 1), (8, 1), (3, 1), (4, 2), (32, 1)])
@pytest.mark.parametrize("interleaved,gains", [(False, True), (True, False)])
def test_many_rows_and_head_counts_within_a_step(heads, kv, interleaved, gains):
    _heads_and_pages(9501, heads, kv, interleaved, gains)


def _heads_and_pages(rows, heads, kv, interleaved, gains=True):
    D, g = 128, _gen(rows + heads)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    qkv = rnd(1, rows, (heads + 2 * kv) * D).bfloat16()
    wq, wk = (1 + 0.1 * rnd(2, D)).bfloat16() if gains else (None, None)
    ang = rnd(rows * 64 + 1) * 3
    cos, sin = ang[1:].cos().view(rows, 64), ang[:-1].sin().view(rows, 64).clone()
    if not interleaved:                                     # tables at an offset that no 16-byte load can take
        flat = torch.empty(rows * 64 + 1, device="cuda")
        flat[1:] = cos.reshape(-1)
        cos = flat[1:].view(rows, 64)
    blocks = (rows + 15) // 16 + 1
    kc, vc = (torch.full((blocks, 16, kv, D), 9.0, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    slots = torch.randperm(blocks * 16, generator=_gen(1), device="cuda")[:rows].int()
    slots[rows // 2] = -1
    ref = fused.qk_norm_rope_reference(qkv, heads, kv, D, wq, wk, None, None, 1 << 30, cos, sin, interleaved, 1e-6)
    plain, paged = qkv.clone(), qkv.clone()
    fused.qk_norm_rope_(plain, heads, kv, D, wq=wq, wk=wk, cos=cos, sin=sin, interleaved=interleaved)
    fused.qk_norm_rope_(paged, heads, kv, D, wq=wq, wk=wk, cos=cos, sin=sin, interleaved=interleaved, pages=(kc, vc, slots))
    assert torch.equal(plain, paged)
    # reference and kernel round once to bf16 from fp32 values a few ulps of fp32 apart
    assert ((plain.float() - ref.float()).abs() <= ref.float().abs() * 2.0 ** -7 + 1e-5).all()
    k2, v2 = torch.full_like(kc, 9.0), torch.full_like(vc, 9.0)
    r = plain.view(rows, -1)
    KC.kv_write(r[:, heads * D:(heads + kv) * D].view(rows, kv, D), r[:, (heads + kv) * D:].view(rows, kv, D), k2, v2, slots)
    assert torch.equal(kc, k2) and torch.equal(vc, v2)


def test_more_slots_than_rows():
    """A slot mapping may be longer than the batch, as the page-writing kernel takes it."""
    D, g, rows = 128, _gen(3), 5
    qkv = torch.randn(1, rows, 4 * D, generator=g, device="cuda").bfloat16()
    slots = torch.tensor([3, -1, 0, 17, 9, 30, 31], dtype=torch.int32, device="cuda")
    pages = [torch.full((2, 16, 1, D), 9.0, device="cuda", dtype=torch.bfloat16) for _ in range(2)]
    fused.qk_norm_rope_(qkv, 2, 1, D, pages=(*pages, slots))
    want = [torch.full((2, 16, 1, D), 9.0, device="cuda", dtype=torch.bfloat16) for _ in range(2)]
    r = qkv.view(rows, 4, D)
    KC.kv_write(r[:, 2:3], r[:, 3:], *want, slots)
    assert torch.equal(pages[0], want[0]) and torch.equal(pages[1], want[1])
