"""Attention of all prompt segments of a step in one launch, and decoded tokens on any rows of it, against softmax in 64 bits."""
import pytest
import torch

from vllm_omni_b200.ops import _native as nv, kv_cache as KC

pytestmark = pytest.mark.gpu
PAGE = 16


def _exact(q, k, v, context):
    H, G = q.shape[1], q.shape[1] // k.shape[1]
    k, v = (t.double().repeat_interleave(G, 1) for t in (k, v))
    s = torch.einsum("qhd,khd->hqk", q.double(), k) * q.shape[2] ** -0.5
    n = q.shape[0]
    s = s.masked_fill(torch.arange(k.shape[0], device=q.device)[None] > context + torch.arange(n, device=q.device)[:, None], float("-inf"))
    return torch.einsum("hqk,khd->qhd", s.softmax(-1), v)


# one row, edges of a query tile (128) and block (256), contexts that end inside a page and a key tile; more than eight segments; two launches' worth of blocks
@pytest.mark.parametrize("segs,H,Hkv,D", [
    ([(1, 0)], 4, 1, 128), ([(257, 0), (128, 0), (129, 5)], 8, 2, 128), ([(1, 300), (256, 128), (40, 0), (700, 129)], 4, 4, 128),
    ([(3 * i + 2, 17 * (i % 3)) for i in range(19)], 4, 2, 128), ([(130, 0), (64, 0)], 8, 8, 64), ([(66000, 0)], 1, 1, 128)])
def test_segments(segs, H, Hkv, D):
    g = torch.Generator(device="cuda").manual_seed(len(segs))
    T = sum(n for n, _ in segs) + 3                                  # three rows of no segment
    qkv = torch.randn(T, (H + 2 * Hkv) * D, device="cuda", generator=g).bfloat16()
    q, k, v = qkv[:, :H * D].view(T, H, D), qkv[:, H * D:(H + Hkv) * D].view(T, Hkv, D), qkv[:, (H + Hkv) * D:].view(T, Hkv, D)
    need = [-(-(n + c) // PAGE) for n, c in segs]
    perm = torch.randperm(sum(need), generator=torch.Generator().manual_seed(3))
    kc, vc = (torch.randn(sum(need), PAGE, Hkv, D, device="cuda", generator=g).bfloat16() for _ in range(2))
    out = torch.full((T, H, D), 7.0, device="cuda", dtype=torch.bfloat16)
    work, keys, at, pg = [], [], 2, 0
    for (n, c), m in zip(segs, need):
        table = perm[pg:pg + m].int().cuda()
        rows = table.long()[torch.arange(n + c, device="cuda") // PAGE] * PAGE + torch.arange(n + c, device="cuda") % PAGE
        for cache, x in ((kc, k), (vc, v)):
            cache.view(-1, Hkv, D)[rows[c:]] = x[at:at + n]
        work.append((at, n, c, table))
        keys.append(rows)
        at, pg = at + n, pg + m
    assert KC.prefill_segments_ok(q, kc, [c for _, c in segs])
    KC.prefill_segments(q, k, v, kc, vc, work, out=out)
    torch.cuda.synchronize()
    nv.check_status(q.device)
    for (a, n, c, _), rows in zip(work, keys):
        pick = torch.arange(n, device="cuda") if n < 2000 else torch.tensor([0, 255, 256, n // 2, n - 1], device="cuda")
        kk, vv = kc.view(-1, Hkv, D)[rows], vc.view(-1, Hkv, D)[rows]
        for r in ([pick] if n < 2000 else pick[:, None]):
            last = int(r[-1]) + c + 1
            ref = _exact(q[a + r], kk[:last], vv[:last], last - len(r)) if n >= 2000 else _exact(q[a:a + n], kk, vv, c)
            got = out[a + r] if n >= 2000 else out[a:a + n]
            # probabilities and results are bf16, a quarter of the exponentials a polynomial to 7.5e-5
            assert (got.double() - ref).norm() <= 2.0 ** -8 * ref.norm()
    assert (out[:2] == 7).all() and (out[at:] == 7).all()


# a lone segment of one round of blocks, which goes to the kernel of a single sequence, and just past its limits
@pytest.mark.parametrize("segs,H,Hkv,D", [([(1000, 0)], 4, 2, 128), ([(999, 0)], 4, 2, 128), ([(300, 700)], 8, 2, 128), ([(17, 1300)], 16, 4, 128), ([(1027, 0)], 2, 2, 64),
                                          ([(1300, 33)], 24, 4, 128), ([(1300, 33)], 25, 5, 128)])
def test_lone_segment(segs, H, Hkv, D):
    test_segments(segs, H, Hkv, D)


@pytest.mark.parametrize("lengths,launches", [([5] * 8, 1), ([5] * 9, 2), ([300] * 19, 3), ([64000], 1), ([65536], 1), ([65537], 2), ([0] * 9, 0)])
def test_launches_are_counted(lengths, launches):
    T = max(1, sum(lengths))
    q = torch.zeros(T, 1, 64, device="cuda", dtype=torch.bfloat16)
    segs = [(sum(lengths[:i]), n, 0, None) for i, n in enumerate(lengths)]
    before = nv.launch_count
    KC.prefill_segments(q, q, q, None, None, segs, out=torch.empty_like(q))
    assert nv.launch_count - before == launches
    nv.check_status(q.device)


# Rows 192 to 199 of the first prompt share a warp with the second one's, whose scores against the first one's keys then grow in the second key tile only
@pytest.mark.parametrize("context", [0, 130])
@pytest.mark.parametrize("D", [64, 128])
def test_results_do_not_depend_on_the_next_segment(context, D):
    if context and D == 64:
        pytest.skip("pages have 128 channels")
    g = torch.Generator(device="cuda").manual_seed(D)
    n, H = 200, 8
    q, k, v = (torch.randn(n + 60, H, D, device="cuda", generator=g).bfloat16() for _ in range(3))
    m = -(-(n + context) // PAGE)
    table = torch.arange(m, dtype=torch.int32, device="cuda")
    kc, vc = (torch.randn(m, PAGE, H, D, device="cuda", generator=g).bfloat16() for _ in range(2))
    for cache, x in ((kc, k), (vc, v)):
        cache.view(-1, H, D)[context:context + n] = x[:n]
    segs = [(0, n, context, table if context else None), (n, 60, 0, None)]
    got = []
    for scale in (0.0, 8.0):
        q[n:] = scale * k[150]
        got.append(KC.prefill_segments(q, k, v, kc, vc, segs, out=torch.empty_like(q))[:n])
    torch.cuda.synchronize()
    nv.check_status(q.device)
    assert torch.equal(*got)


def test_steps_past_the_launch_limit_go_segment_by_segment():
    q = torch.empty(1 << 20, 1, 64, device="cuda", dtype=torch.bfloat16)
    assert KC.prefill_segments_ok(q, None, [0])
    assert not KC.prefill_segments_ok(torch.empty((1 << 20) + 1, 1, 64, device="cuda", dtype=torch.bfloat16), None, [0])


@pytest.mark.parametrize("n,H,Hkv", [(1, 8, 2), (5, 32, 4), (3, 16, 1)])
def test_decode_on_rows_of_a_step(n, H, Hkv):
    g = torch.Generator(device="cuda").manual_seed(n)
    T, L = 40, 333
    q = torch.randn(T, H, 128, device="cuda", generator=g).bfloat16()
    kc, vc = (torch.randn(n * 21, PAGE, Hkv, 128, device="cuda", generator=g).bfloat16() for _ in range(2))
    bt = torch.randperm(n * 21, generator=torch.Generator().manual_seed(1)).view(n, 21).int().cuda()
    lens = torch.tensor([L - 50 * i for i in range(n)], dtype=torch.int32, device="cuda")
    rows = torch.tensor([-1, 3, 17, 8, 0][:n], device="cuda")
    want = KC.paged_decode(q[rows].contiguous(), kc, vc, bt, lens)
    out = torch.full_like(q, 7.0)
    assert KC.paged_decode(q, kc, vc, bt, lens, out=out, rows=rows) is out
    torch.cuda.synchronize()
    nv.check_status(q.device)
    assert torch.equal(out[rows], want)
    rest = torch.ones(T, dtype=torch.bool, device="cuda")
    rest[rows] = False
    assert (out[rest] == 7).all()


# more sequences than one early launch takes, groups of 12 heads, rows from both ends, every length down to one key
@pytest.mark.parametrize("n,H,Hkv", [(40, 32, 4), (20, 48, 4), (17, 12, 1)])
def test_many_decoded_rows_of_a_step(n, H, Hkv):
    g = torch.Generator(device="cuda").manual_seed(n)
    T, L = 2 * n + 5, 900
    q = torch.randn(T, H, 128, device="cuda", generator=g).bfloat16()
    m = -(-L // PAGE)
    kc, vc = (torch.randn(n * m, PAGE, Hkv, 128, device="cuda", generator=g).bfloat16() for _ in range(2))
    bt = torch.randperm(n * m, generator=torch.Generator().manual_seed(1)).view(n, m).int().cuda()
    lens = [max(1, L - i * i * 7) if i % 2 else max(1, 40 - i) for i in range(n)]
    rows = torch.randperm(T, generator=torch.Generator().manual_seed(2))[:n].cuda()
    rows[::3] -= T
    out = torch.full_like(q, 7.0)
    KC.paged_decode(q, kc, vc, bt, torch.tensor(lens, dtype=torch.int32, device="cuda"), out=out, rows=rows, impl="stream")
    torch.cuda.synchronize()
    nv.check_status(q.device)
    for i in range(n):
        keys = bt[i].long().repeat_interleave(PAGE)[:lens[i]] * PAGE + torch.arange(lens[i], device="cuda") % PAGE
        ref = _exact(q[rows[i]][None], kc.view(-1, Hkv, 128)[keys], vc.view(-1, Hkv, 128)[keys], lens[i] - 1)
        # probabilities and results are bf16
        assert (out[rows[i]][None].double() - ref).norm() <= 2.0 ** -8 * ref.norm()
    rest = torch.ones(T, dtype=torch.bool, device="cuda")
    rest[rows] = False
    assert (out[rest] == 7).all()


@pytest.mark.parametrize("impl", ["stream", "tc", "simt"])
def test_rows_of_a_step_take_the_kernel_asked_for(impl):
    g = torch.Generator(device="cuda").manual_seed(5)
    q = torch.randn(9, 8, 128, device="cuda", generator=g).bfloat16()
    kc, vc = (torch.randn(30, PAGE, 2, 128, device="cuda", generator=g).bfloat16() for _ in range(2))
    bt = torch.arange(30, dtype=torch.int32, device="cuda").view(3, 10)
    lens = torch.tensor([150, 90, 33], dtype=torch.int32, device="cuda")
    rows = torch.tensor([7, 0, -3], device="cuda")
    out = KC.paged_decode(q, kc, vc, bt, lens, out=torch.zeros_like(q), rows=rows, impl=impl)
    assert torch.equal(out[rows], KC.paged_decode(q[rows].contiguous(), kc, vc, bt, lens, impl=impl))
    nv.check_status(q.device)
