"""Experts of few tokens (csrc/moe.cu, tiles of 16 rows gathered in place) and of more (csrc/moe_gemm.cuh, tiles of up to 64, 128 or 256
rows): one row to several tiles per expert, experts of another rank, ragged widths, both activations; and the plans of tiles."""
import pytest
import torch

from vllm_omni_b200.ops import _native as nv
from vllm_omni_b200.ops.moe import MoEWorkspace, Router, _few, _tile_rows, expert_rows, moe_forward

pytestmark = pytest.mark.gpu


def _problem(T, E, k, D, F, crowd, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed + T * 31 + E)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    x, w13, w2 = rnd(T, D).bfloat16(), (rnd(E, 2 * F, D) * D ** -0.5).bfloat16(), (rnd(E, D, F) * F ** -0.5).bfloat16()
    # distinct logits (no ties to break); with ``crowd`` every token wants expert 1
    logits = torch.stack([torch.randperm(E, generator=g, device="cuda") for _ in range(T)]).float() / 16
    if crowd:
        logits[:, 1] = E / 16 + 1
    return x, logits.bfloat16(), w13, w2


def _expected(x, ids, w, up, down, act, lo=0, hi=1 << 30):
    """(result, bound): bf16 rounding of h, of every pair's row and of the result, tanh.approx in silu, fp32 sums."""
    T, F = x.shape[0], down.shape[2]
    y, bound = torch.zeros(T, down.shape[1], dtype=torch.float64, device="cuda"), 0
    bound = torch.zeros_like(y)
    for t in range(T):
        for j in range(ids.shape[1]):
            e = int(ids[t, j])
            if not lo <= e < hi:
                continue
            a = x[t].double() @ up[e - lo].double().T
            if act == "swiglu":
                h = torch.nn.functional.silu(a[:F]) * a[F:]
                eh = h.abs() * 2.0 ** -8 + (a[:F] * a[F:]).abs() * 2.0 ** -11 + 1e-4
            else:
                h = a.clamp(min=0) ** 2
                eh = h * 2.0 ** -8 + 1e-4
            d = down[e - lo].double()
            y[t] += w[t, j].double() * (h @ d.T)
            bound[t] += w[t, j].double() * (eh @ d.abs().T + (h @ d.T).abs() * 2.0 ** -8 + 1e-4)
    return y, 1.2 * bound + y.abs() * 2.0 ** -8


@pytest.mark.parametrize("T,E,k,D,F,crowd", [(1, 128, 8, 2048, 768, False), (16, 128, 8, 256, 96, False), (8, 8, 1, 72, 40, True),
                                              (8, 16, 2, 1032, 136, True), (16, 128, 8, 128, 64, True), (32, 256, 4, 64, 1096, True)])
def test_moe_forward(T, E, k, D, F, crowd):
    assert _few(T, k, E, False)
    _check_forward(T, E, k, D, F, crowd)


@pytest.mark.parametrize("T,E,k,D,F,crowd,tile", [(5, 4, 2, 72, 40, False, 64), (100, 16, 4, 256, 136, False, 64), (130, 16, 2, 64, 64, True, 64),
                                                  (200, 16, 4, 136, 72, True, 128), (300, 8, 2, 128, 200, True, 256), (700, 8, 2, 64, 96, False, 256)])
def test_moe_forward_more_tokens(T, E, k, D, F, crowd, tile):
    assert not _few(T, k, E, False) and _tile_rows(T, k, E) == tile
    _check_forward(T, E, k, D, F, crowd)


def _check_forward(T, E, k, D, F, crowd):
    x, logits, w13, w2 = _problem(T, E, k, D, F, crowd)
    p = torch.softmax(logits.double(), -1)
    w, ids = p.topk(k, -1)
    w = w / w.sum(-1, keepdim=True)
    res = torch.randn(T, D, device="cuda").bfloat16()
    ref, bound = _expected(x, ids, w, w13, w2, "swiglu")
    y = moe_forward(x, logits, w13, w2, k, ws=MoEWorkspace(), residual=res)
    assert ((y.double() - ref - res.double()).abs() <= bound + res.double().abs() * 2.0 ** -8).all()
    half = E // 2
    parts = [moe_forward(x, logits, w13[a:b], w2[a:b], k, e_lo=a, e_hi=b).double() for a, b in ((0, half), (half, E))]
    for (a, b), got in zip(((0, half), (half, E)), parts):
        ref, bound = _expected(x, ids, w, w13[a:b], w2[a:b], "swiglu", a, b)
        assert ((got - ref).abs() <= bound).all()
    nv.check_status()


@pytest.mark.parametrize("T", [18, 90])
@pytest.mark.parametrize("act", ["relu2", "swiglu"])
def test_expert_rows(act, T):
    E, k, D, F = 72, 4, 200, 72
    x, logits, up, down = _problem(T, E, k, D, F, False)
    up = up if act == "swiglu" else up[:, :F].contiguous()
    router = Router(E, k)
    rw = torch.randn(E, D, device="cuda").bfloat16()
    got = expert_rows(x, rw, None, router, up, down, act, MoEWorkspace())
    ids, w = router.choose(x.double() @ rw.double().T)
    y = torch.zeros(T, D, dtype=torch.float64, device="cuda")
    for t in range(T):
        for j in range(k):
            y[t] += got.weights[t, j].double() * got.y[got.row_of_pair[t * k + j]].double()
    ref, bound = _expected(x, ids, w, up, down, act)
    same = (got.weights.double() - w.double()).abs().max(1).values < 1e-3      # rows whose choice is not a rounding
    assert same.sum() >= T - 4 and ((y - ref).abs() <= bound + 0.01 * ref.abs())[same].all()


@pytest.mark.parametrize("act", [0, 3, 5])                             # none, squared ReLU, SwiGLU
@pytest.mark.parametrize("tile", [64, 128, 256])
@pytest.mark.parametrize("pitch,base", [(3, 0), (0, 1), (8, 4), (5, 7)])
def test_expert_gemm_into_any_rows(act, tile, pitch, base):
    """C of any pitch and base gets the bits of one whose rows lie on 16 bytes, and nothing beside them is written."""
    from ctypes import c_int
    E, N, K, rows = 3, 136, 72, [tile, 0, tile - 15, 1]
    g = torch.Generator(device="cuda").manual_seed(tile)
    a, w = (torch.randn(*s, generator=g, device="cuda").bfloat16() for s in ((sum(rows), K), (E, (2 if act == 5 else 1) * N, K)))
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    used = [i for i, r in enumerate(rows) if r]
    te, t0, tn = i32([i % E for i in used] + [-1]), i32([sum(rows[:i]) for i in used] + [0]), i32([rows[i] for i in used] + [0])
    def run(ld, at):
        c = torch.full((sum(rows) * ld + 16,), 7.0, device="cuda", dtype=torch.bfloat16)
        nv.check_rc(nv.lib("gemm_sm100").omni_gemm_bf16_experts(nv.ptr(a), c_int(K), nv.ptr(w), c_int(E), nv.ptr(c[at:]), c_int(ld), c_int(sum(rows)), c_int(N), c_int(K),
                                                                nv.ptr(te), nv.ptr(t0), nv.ptr(tn), c_int(len(te)), c_int(tile), c_int(act),
                                                                nv.ptr(nv.status_word(a.device)), nv.stream_ptr()), "experts")
        nv.check_status(a.device)
        body = c[at:at + sum(rows) * ld].view(-1, ld)
        assert (c[:at] == 7).all() and (c[at + sum(rows) * ld:] == 7).all() and (body[:, N:] == 7).all()
        return body[:, :N]
    assert torch.equal(run(N + pitch, base), run(N, 0))


@pytest.mark.parametrize("n_pairs,E,lo,hi,tile", [(1, 1, 0, 1, 64), (5000, 128, 0, 128, 64), (5000, 128, 0, 128, 128), (3000, 7, 2, 5, 128), (2048, 1024, 0, 1024, 128),
                                                     (70001, 64, 0, 64, 256), (70001, 64, 0, 64, 128), (1300, 4, 1, 4, 256),
                                                     (8192, 128, 0, 128, 128), (8193, 128, 0, 128, 128), (16385, 1024, 100, 900, 256)])
def test_even_plan(n_pairs, E, lo, hi, tile):
    g = torch.Generator(device="cuda").manual_seed(n_pairs)
    ids = (torch.rand(n_pairs, generator=g, device="cuda") ** 2 * E).int().clamp(max=E - 1)
    tiles = min(E, n_pairs) + n_pairs // tile
    row, te, t0, tn, n = (torch.full((m,), -7, dtype=torch.int32, device="cuda") for m in (n_pairs, tiles, tiles, tiles, 1))
    from ctypes import c_int
    nv.check_rc(nv.lib("moe").omni_moe_plan_tiles(nv.ptr(ids), c_int(n_pairs), c_int(E), c_int(lo), c_int(hi), c_int(tile), c_int(tiles), nv.ptr(row),
                                                  nv.ptr(te), nv.ptr(t0), nv.ptr(tn), nv.ptr(n), nv.stream_ptr()), "plan")
    local = (ids >= lo) & (ids < hi)
    assert int(n) == int(local.sum()) and (row[~local] == -1).all()
    assert torch.equal(row[local].sort().values, torch.arange(int(n), device="cuda", dtype=torch.int32))
    of_row = torch.empty(int(local.sum()), dtype=torch.int32, device="cuda")
    of_row[row[local].long()] = ids[local] - lo
    assert torch.equal(of_row, of_row.sort().values)                            # experts in order, rows back to back
    at, used = 0, True
    for e, r0, rn in zip(te.tolist(), t0.tolist(), tn.tolist()):
        used = used and e >= 0
        assert used == (e >= 0)                                                 # used tiles first
        if used:
            assert r0 == at and 1 <= rn <= tile and (of_row[r0:r0 + rn] == e).all()
            at += rn
    assert at == of_row.numel() == int(n)


@pytest.mark.parametrize("T,D", [(1, 2048), (3, 72), (70, 264), (5, 8192), (2, 8184)])
def test_norm_of_the_result(T, D):
    """The combining launch with the next norm: the same rows, and their norm against 64 bits."""
    from vllm_omni_b200.ops import fused
    E, k, Fd = 8, 2, 40
    x, logits, w13, w2 = _problem(T, E, k, D, Fd, False)
    res, gain = torch.randn(T, D, device="cuda").bfloat16(), torch.randn(D, device="cuda").bfloat16()
    plain = moe_forward(x, logits, w13, w2, k, residual=res)
    xn = x.clone()
    y = moe_forward(xn, logits, w13, w2, k, residual=res, norm=(gain, 1e-6, xn))         # into its own input
    assert torch.equal(y, plain)
    ref = y.double() * torch.rsqrt(y.double().pow(2).mean(-1, keepdim=True) + 1e-6) * gain.double()
    # one rounding to bf16; fp32 sums of at most 8192 squares and rsqrtf (2 ulp)
    assert ((xn.double() - ref).abs() <= ref.abs() * (2.0 ** -8 + 1e-4) + 1e-30).all()
    nv.check_status()
