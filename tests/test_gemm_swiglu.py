"""Gated layers in one launch (``gemm.linear_swiglu``) and the epilogue kernels of the general linear layers, against 64-bit sums."""
import pytest
import torch
import torch.nn.functional as F

from vllm_omni_b200.ops import _native as nv, gemm

pytestmark = pytest.mark.gpu


def _rnd(seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()


# rows of the few-row kernels (1 to 16), of the two-launch form (17 to 128) and of both general kernels; widths that end inside a group of 8, a chunk and a tile
@pytest.mark.parametrize("M", [1, 7, 8, 9, 16, 17, 64, 128, 129, 300, 700, 2500])
@pytest.mark.parametrize("F_,K", [(8, 64), (24, 200), (136, 72), (768, 512), (1000, 2048), (6144, 256)])
def test_swiglu(M, F_, K):
    rnd = _rnd(M + F_)
    x, w = rnd(M, K), (rnd(2 * F_, K).float() * K ** -0.5 * 1.5).bfloat16()
    y = gemm.linear_swiglu(x, w)
    nv.check_status(x.device)
    g, u = (x.double() @ w.double().T).split(F_, 1)
    ref = F.silu(g) * u
    # fp32 sums of K / 16 MMA steps, each off by at most an ulp of the terms' magnitudes so far; silu's slope is at most 1.1
    mass = (x.double().abs() @ w.double().abs().T).split(F_, 1)
    sums = 1.1 * (mass[0] * u.abs() + mass[1] * g.abs()) * (K / 16 + 1) * 2.0 ** -24
    # result to bf16; tanh.approx in silu; where it takes two launches both halves pass through bf16 first
    halves = (2.0 ** -8 * (g.abs() * u.abs()) * 2.2 if 16 < M <= 128 else 0.0)
    assert torch.isfinite(y).all() and ((y.double() - ref).abs() <= ref.abs() * 2.0 ** -8 + g.abs() * u.abs() * 2.0 ** -10 + sums + halves + 1e-5).all()


def test_swiglu_takes_views():
    rnd = _rnd(3)
    x, w = rnd(2, 150, 96)[:, :, 8:72], rnd(80, 64)
    a, b = gemm.linear_swiglu(x, w), gemm.linear_swiglu(x.contiguous(), w)
    assert a.shape == (2, 150, 40) and torch.equal(a, b)


@pytest.mark.parametrize("M", [4, 64, 300])
def test_swiglu_of_rows_narrower_than_the_weights(M):
    """As in ``linear``, rows of fewer channels meet the first columns of the weights; each row stays a row."""
    rnd = _rnd(M)
    x, w = rnd(M, 512), (rnd(2 * 96, 1024).float() * 512 ** -0.5).bfloat16()
    g, u = (x.double() @ w[:, :512].double().T).split(96, 1)
    ref = F.silu(g) * u
    y = gemm.linear_swiglu(x, w)
    nv.check_status(x.device)
    # both halves and the result rounded to bf16; tanh.approx in silu, whose slope is at most 1.1
    assert y.shape == ref.shape and ((y.double() - ref).abs() <= ref.abs() * 2.0 ** -8 + g.abs() * u.abs() * (2.2 * 2.0 ** -8 + 2.0 ** -10) + 1e-4).all()


def _gated(x, w, F_, halves):
    """SwiGLU in 64 bits and how far the kernels may be from it; ``halves``: gate and lift pass through bf16."""
    K = x.shape[1]
    g, u = (x.double() @ w.double().T).split(F_, 1)
    mass = (x.double().abs() @ w.double().abs().T).split(F_, 1)
    # fp32 sums of K / 16 MMA steps, each off by at most an ulp of the terms' magnitudes so far; silu's slope is at most 1.1; tanh.approx in silu; result to bf16
    sums = 1.1 * (mass[0] * u.abs() + mass[1] * g.abs()) * (K / 16 + 1) * 2.0 ** -24
    ref, size = F.silu(g) * u, g.abs() * u.abs()
    return ref, ref.abs() * 2.0 ** -8 + size * 2.0 ** -10 + sums + (2.2 * 2.0 ** -8 * size if halves else 0.0) + 1e-5


# tiles of 128, 192 and 256 columns on single CTAs and on pairs: rows of one and of several tiles, widths that end inside a group of 8, a chunk and a tile
@pytest.mark.parametrize("bn", [128, 192, 256, 384, 448, 576])
@pytest.mark.parametrize("M,F_,K", [(1, 8, 64), (129, 100 * 8, 136), (257, 1000, 72), (700, 136, 512)])
def test_swiglu_of_every_kernel(bn, M, F_, K):
    rnd = _rnd(M + bn)
    x, w = rnd(M, K), (rnd(2 * F_, K).float() * K ** -0.5 * 1.5).bfloat16()
    y = gemm.linear_swiglu(x, w, force_bn=bn)
    nv.check_status(x.device)
    ref, bound = _gated(x, w, F_, False)
    assert ((y.double() - ref).abs() <= bound).all()


# the three-tile form of the rows kernel and the rows past it: every split of its columns over the SMs
@pytest.mark.parametrize("M", [17, 23, 24, 25])
@pytest.mark.parametrize("per_sm,K", [(0.5, 9216), (1, 136), (1.5, 4096), (2.5, 512), (3.5, 264), (4.5, 1024)])
def test_swiglu_of_17_to_25_rows(M, per_sm, K):
    F_ = int(per_sm * torch.cuda.get_device_properties(0).multi_processor_count) * 8 - 8
    rnd = _rnd(M + K)
    x, w = rnd(M, K), (rnd(2 * F_, K).float() * K ** -0.5 * 1.5).bfloat16()
    y = gemm.linear_swiglu(x, w)
    nv.check_status(x.device)
    ref, bound = _gated(x, w, F_, M > 24)
    assert ((y.double() - ref).abs() <= bound).all()


# both problems of a launch with the same activation, which has a kernel of its own, residual and gate
@pytest.mark.parametrize("act", [None, "gelu_tanh"])
@pytest.mark.parametrize("force", [False, True])
@pytest.mark.parametrize("S,T,N,K", [(300, 40, 1544, 136), (1024, 64, 3072, 256), (64, 8, 520, 64)])
def test_epilogues_of_two_problems(act, force, S, T, N, K):
    rnd = _rnd(S + N)
    ws = [(rnd(N, K).float() * K ** -0.5).bfloat16() for _ in range(2)]
    ops = [dict(x=rnd(2, s, K), w=w, bias=rnd(N), act=act, residual=rnd(2, s, N), gate=rnd(2, N)) for s, w in zip((S, T), ws)]
    outs = [o["residual"].clone() for o in ops]                      # in place
    gemm.linear_pair(*(dict(o, residual=y, out=y) for o, y in zip(ops, outs)), force_pair=force)
    nv.check_status(outs[0].device)
    for o, y in zip(ops, outs):
        z = o["x"].double() @ o["w"].double().T + o["bias"].double()
        slack = z.abs() * 2.0 ** -10                                 # tanh.approx; fp32 sums
        z = F.gelu(z, approximate="tanh") if act else z
        g = o["gate"].double()[:, None]
        ref = z * g + o["residual"].double()
        assert ((y.double() - ref).abs() <= ref.abs() * 2.0 ** -8 + slack * g.abs() + 2e-5).all()


# every kernel (pair of 256 / 192 / 128 columns, automatic choice) with every epilogue; ragged rows and columns; rows of a tile in two batches
@pytest.mark.parametrize("bn", [0, 384, 448, 576])
@pytest.mark.parametrize("act", [None, "gelu_tanh", "xielu", "silu", "relu2"])
@pytest.mark.parametrize("B,S,N,K", [(2, 100, 200, 136), (2, 333, 520, 64), (1, 257, 8, 72)])
@pytest.mark.parametrize("operands", ["", "bias", "bias residual", "bias gate residual"])
def test_epilogues(bn, act, B, S, N, K, operands):
    rnd = _rnd(S + N)
    x, w = rnd(B, S, K), (rnd(N, K).float() * K ** -0.5).bfloat16()
    kw = dict(bias=rnd(N) if "bias" in operands else None, residual=rnd(B, S, N) if "residual" in operands else None,
              gate=rnd(B, N) if "gate" in operands else None, coef=(0.8, 0.6))
    y = gemm.linear(x, w, act=act, force_bn=bn, **kw)
    nv.check_status(x.device)
    up = lambda t: None if t is None else t.double()
    z = x.double() @ w.double().T
    ref = z if kw["bias"] is None else z + up(kw["bias"])
    size = ref.abs()
    ref = {None: lambda t: t, "gelu_tanh": lambda t: F.gelu(t, approximate="tanh"), "silu": F.silu, "relu2": lambda t: F.relu(t).square(),
           "xielu": lambda t: gemm.xielu(t, (0.8, 0.6))}[act](ref)
    slack = size * 2.0 ** -10 + (ref.abs() * 2.0 ** -13 if act in ("relu2", "xielu") else 0.0)      # tanh.approx, ex2.approx; fp32 sums
    if kw["gate"] is not None:
        ref, slack = ref * up(kw["gate"])[:, None], slack * up(kw["gate"]).abs()[:, None]
    if kw["residual"] is not None:
        ref = ref + up(kw["residual"])
    assert ((y.double() - ref).abs() <= ref.abs() * 2.0 ** -8 + slack + 2e-5).all()
    buf = None if kw["residual"] is None else kw["residual"].clone()
    if buf is not None:                                              # in place: the residual is the output
        assert torch.equal(gemm.linear(x, w, act=act, force_bn=bn, **{**kw, "residual": buf}, out=buf), y)


# tiles of 128, 192 and 256 columns on single CTAs, whose epilogues are kernels of their own
@pytest.mark.parametrize("bn", [128, 192, 256])
@pytest.mark.parametrize("act", [None, "gelu_tanh", "xielu", "silu", "relu2"])
@pytest.mark.parametrize("B,S,N,K", [(2, 100, 200, 136), (2, 333, 520, 64), (1, 257, 8, 72)])
@pytest.mark.parametrize("operands", ["", "bias", "bias residual", "bias gate residual"])
def test_epilogues_of_single_ctas(bn, act, B, S, N, K, operands):
    test_epilogues(bn, act, B, S, N, K, operands)
