"""Linear layers of at most 128 rows (csrc/gemm_skinny.cuh): edges of the row tiles (16, 32, 64, 128), of the 128-column tiles and of
the split contraction, with every epilogue, against 64-bit products."""
import pytest
import torch

from vllm_omni_b200.ops import _native as nv, gemm

pytestmark = pytest.mark.gpu


def _check(y, ref, mass, act_err=0.0):
    # bf16 result: half an ulp; fp32 sums: K / 16 additions of at most 2^-23 of the products' mass each, K <= 12288; the
    # activations are 1.13-Lipschitz and use tanh.approx (2^-11 relative)
    bound = 1.2 * (ref.abs() * 2.0 ** -8 + mass * (12288 / 16) * 2.0 ** -23) + act_err
    assert torch.isfinite(y).all()
    assert ((y.double() - ref).abs() <= bound + 1e-6).all()


@pytest.mark.parametrize("rows", [1, 15, 16, 17, 32, 33, 64, 65, 127, 128])
@pytest.mark.parametrize("n,k", [(8, 8), (136, 72), (2048, 64), (2048, 2048), (1000, 12288), (5120, 136), (40000, 128)])
def test_plain(rows, n, k):
    g = torch.Generator(device="cuda").manual_seed(rows * 7 + n + k)
    x = torch.randn(rows, k + 8, generator=g, device="cuda").bfloat16()[:, :k]          # a row pitch wider than the row
    w = torch.randn(n, k, generator=g, device="cuda").bfloat16()
    buf = torch.full((rows + 1, n + 8), 7.0, device="cuda", dtype=torch.bfloat16)
    y = gemm.linear(x, w, out=buf[:rows, :n])
    _check(y, x.double() @ w.double().T, x.double().abs() @ w.double().abs().T)
    assert (buf[rows] == 7).all() and (buf[:, n:] == 7).all()
    nv.check_status()


@pytest.mark.parametrize("rows", [2, 16, 48, 128])
@pytest.mark.parametrize("act", [None, "gelu_tanh", "silu", "relu2", "xielu"])
def test_epilogue(rows, act):
    n, k = 264, 1024
    g = torch.Generator(device="cuda").manual_seed(rows)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    x, w, b, res, gate = rnd(rows, k), rnd(n, k) * 0.03, rnd(n), rnd(rows, n), rnd(2, n)
    coef = (0.4, 0.7)
    z = x.double() @ w.double().T + b.double()
    ref = {None: lambda t: t, "gelu_tanh": lambda t: torch.nn.functional.gelu(t, approximate="tanh"), "silu": torch.nn.functional.silu,
           "relu2": lambda t: t.clamp(min=0) ** 2, "xielu": lambda t: gemm.xielu(t, coef)}[act](z)
    y = (ref.view(2, rows // 2, n) * gate.double()[:, None]).view(rows, n) + res.double()
    slope = {None: 1.0, "relu2": 2 * z.abs(), "xielu": z.abs() + 1}.get(act, 1.0)
    err = z.abs() * 2.0 ** -11 * (act in ("gelu_tanh", "silu")) + 1e-5 * (act == "xielu")
    mass = (x.double().abs() @ w.double().abs().T) * slope
    big = gate.double().abs().max()
    out = gemm.linear(x, w, b, act=act, residual=res, gate=gate, coef=coef)
    _check(out, y, mass * big, err * big)
    inplace = res.clone()
    gemm.linear(x, w, b, act=act, residual=inplace, gate=gate, coef=coef, out=inplace)
    assert torch.equal(inplace, out)
    # rows of two batches into one joint buffer
    joint = torch.zeros(2, rows // 2 + 3, n, device="cuda", dtype=torch.bfloat16)
    gemm.linear(x, w, b, act=act, residual=res, gate=gate, coef=coef, out=joint[:, 1:], out_rows_per_batch=rows // 2,
                out_batch_stride=joint.stride(0))
    assert torch.equal(joint[:, 1:1 + rows // 2].reshape(rows, n), out) and (joint[:, 0] == 0).all() and (joint[:, 1 + rows // 2:] == 0).all()
    nv.check_status()


@pytest.mark.parametrize("rows", [1, 8, 9, 16])
@pytest.mark.parametrize("per_sm", [1, 2, 3, 3.5, 4, 4.5, 6, 8])
def test_splits_of_at_most_16_rows(rows, per_sm):
    """Every split of csrc/gemm_skinny.cuh's launch_rows, at and just past its limits in 16-column tiles per SM."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for n in (int(per_sm * sms) * 16, int(per_sm * sms) * 16 + 8):
        for k in (72, 1032):
            g = torch.Generator(device="cuda").manual_seed(rows + n + k)
            rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
            x, w, b, res = rnd(rows, k), rnd(n, k), rnd(n), rnd(rows, n)
            y = gemm.linear(x, w, b, residual=res)
            _check(y, x.double() @ w.double().T + b.double() + res.double(), x.double().abs() @ w.double().abs().T)
    nv.check_status()


@pytest.mark.parametrize("rows,n,k", [(8, 14400, 8192), (9, 14208, 6912), (9, 14216, 6912), (16, 14216, 3840), (16, 14216, 3912), (16, 14208, 4096),
                                      (16, 9480, 12288), (16, 9472, 12288), (17, 9480, 136), (32, 12808, 1032), (32, 18944, 200), (32, 18952, 200), (48, 4736, 520), (64, 4608, 1024), (64, 9472, 72), (64, 9480, 72),
                                      (65, 2048, 1016), (65, 2048, 960), (65, 2056, 1024), (128, 2688, 1032), (128, 2824, 1024), (128, 2824, 1096),
                                      (128, 6272, 2304), (128, 6272, 2240), (128, 6280, 3200)])
def test_edges_of_the_rules(rows, n, k):
    """Both sides of every limit of few_rows() and of the widest layout that is one cluster short of a round (37 tiles)."""
    g = torch.Generator(device="cuda").manual_seed(rows + n + k)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    x, w, b, res = rnd(rows, k), rnd(n, k), rnd(n), rnd(rows, n)
    y = gemm.linear(x, w, b, residual=res)
    _check(y, x.double() @ w.double().T + b.double() + res.double(), x.double().abs() @ w.double().abs().T)
    nv.check_status()


@pytest.mark.parametrize("rows", [17, 23, 24, 25])
@pytest.mark.parametrize("per_sm,k", [(0.5, 9216), (1, 136), (1.5, 4096), (2, 72), (2.5, 512), (3.5, 264), (4.5, 1024), (5.5, 64)])
def test_splits_of_17_to_24_rows(rows, per_sm, k):
    """Every split of the three-tile form, and the rows and widths past it."""
    n = int(per_sm * torch.cuda.get_device_properties(0).multi_processor_count) * 16 - 8
    g = torch.Generator(device="cuda").manual_seed(rows + k)
    x, w, r = (torch.randn(*s, generator=g, device="cuda").bfloat16() for s in ((rows, k), (n, k), (rows, n)))
    y = gemm.linear(x, w, residual=r)
    _check(y, x.double() @ w.double().T + r.double(), x.double().abs() @ w.double().abs().T)
    nv.check_status()


# both sides of every limit of the rule for 17 to 24 rows: rounds of blocks that are four fifths full and not, the longest contraction of each
@pytest.mark.parametrize("rows", [17, 24])
@pytest.mark.parametrize("n,k", [(1888, 2048), (1888, 2056), (1904, 9216), (1904, 9224), (3776, 2048), (3776, 2056), (3800, 4096), (3800, 4104), (5680, 3072),
                                 (5680, 3080), (5696, 4096), (5696, 4104), (9472, 2560), (9472, 2568), (12432, 2048), (12432, 2056), (12440, 2048)])
def test_edges_of_17_to_24_rows(rows, n, k):
    test_edges_of_the_rules(rows, n, k)
