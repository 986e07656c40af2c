"""Paged attention of single tokens straight from the pages (csrc/decode_attn.cu): group sizes, head counts that do not fill a block,
page sizes, lengths around tiles of 16 keys, one and many shares; page rows past a sequence's end hold NaN."""
import pytest
import torch

from vllm_omni_b200.ops import kv_cache as KC

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,Hkv", [(8, 1), (32, 4), (32, 8), (12, 3), (20, 10), (16, 1), (36, 3), (5, 5)])
@pytest.mark.parametrize("bs", [8, 16, 48, 128])
@pytest.mark.parametrize("lens", [[1], [7, 8, 9, 16, 17, 33], [1000, 1, 333, 2047] * 5])
def test_against_64_bits(H, Hkv, bs, lens):
    D, n, G = 128, len(lens), H // Hkv
    g = torch.Generator(device="cuda").manual_seed(H * 100 + bs + n)
    per = [-(-l // bs) for l in lens]
    width = max(per) + 1
    order = torch.randperm(sum(per), generator=torch.Generator().manual_seed(n)).tolist()
    k, v = (torch.full((sum(per), bs, Hkv, D), float("nan"), device="cuda", dtype=torch.bfloat16) for _ in range(2))
    tables, at = torch.zeros(n, width, dtype=torch.int32), 0
    q = torch.randn(n, H * D + 16, generator=g, device="cuda").bfloat16()[:, :H * D].view(n, H, D)
    ref, bound = torch.empty(n, H, D, dtype=torch.float64, device="cuda"), torch.empty(n, H, D, dtype=torch.float64, device="cuda")
    for s, l in enumerate(lens):
        pages = order[at:at + per[s]]
        at += per[s]
        tables[s, :per[s]] = torch.tensor(pages)
        ks, vs = (torch.randn(l, Hkv, D, generator=g, device="cuda").bfloat16() for _ in range(2))
        for cache, rows in ((k, ks), (v, vs)):
            for i, pg in enumerate(pages):
                part = rows[i * bs:(i + 1) * bs]
                cache[pg, :part.shape[0]] = part
        kk, vv = (t.double().repeat_interleave(G, 1) for t in (ks, vs))
        w = torch.softmax(torch.einsum("hd,khd->hk", q[s].double(), kk) * D ** -0.5, -1)
        ref[s] = torch.einsum("hk,khd->hd", w, vv)
        # weights rounded to bf16 (half an ulp, 2^-9, of each), ex2.approx and fp32 scores far below that; result rounded once
        bound[s] = torch.einsum("hk,khd->hd", w, vv.abs()) * 2.0 ** -8 + ref[s].abs() * 2.0 ** -8 + 1e-5
    out = torch.empty(n, H, D, device="cuda", dtype=torch.bfloat16)
    KC.paged_decode(q, k, v, tables.cuda(), torch.tensor(lens, dtype=torch.int32, device="cuda"), out=out, impl="stream")
    assert ((out.double() - ref).abs() <= bound).all()


@pytest.mark.parametrize("H,Hkv", [(8, 1), (16, 1)])
@pytest.mark.parametrize("dead", [1, 16, 40, 99])
def test_scores_of_minus_infinity(H, Hkv, dead):
    """Keys whose scores are -inf at the head of a sequence, whole tiles and shares of them too, weigh nothing."""
    D, n, L = 128, 3, 100
    g = torch.Generator(device="cuda").manual_seed(dead)
    q = torch.randn(n, H, D, generator=g, device="cuda").bfloat16()
    q[..., 0] = q[..., 0].abs() + 0.25
    k, v = (torch.randn(n * 7, 16, Hkv, D, generator=g, device="cuda").bfloat16() for _ in range(2))
    k.view(n, 112, Hkv, D)[:, :dead, :, 0] = float("-inf")
    tables = torch.arange(n * 7, dtype=torch.int32, device="cuda").view(n, 7)
    out = KC.paged_decode(q, k, v, tables, torch.full((n,), L, dtype=torch.int32, device="cuda"))
    kk, vv = (t.view(n, 112, Hkv, D)[:, :L].double().repeat_interleave(H // Hkv, 2) for t in (k, v))
    w = torch.softmax(torch.einsum("nhd,nkhd->nhk", q.double(), kk) * D ** -0.5, -1)
    ref = torch.einsum("nhk,nkhd->nhd", w, vv)
    # as above: weights and result rounded to bf16
    bound = torch.einsum("nhk,nkhd->nhd", w, vv.abs()) * 2.0 ** -8 + ref.abs() * 2.0 ** -8 + 1e-5
    assert ((out.double() - ref).abs() <= bound).all()


@pytest.mark.parametrize("bs", [24, 48, 256])
@pytest.mark.parametrize("H,Hkv", [(8, 1), (8, 4)])
def test_pages_of_other_sizes_keep_fp32_weights(bs, H, Hkv):
    """Pages the tensor-core kernel does not take are decoded with weights in fp32."""
    D, n, L = 128, 3, 500
    g = torch.Generator(device="cuda").manual_seed(bs)
    per = -(-L // bs)
    q = torch.randn(n, H, D, generator=g, device="cuda").bfloat16()
    k, v = (torch.randn(n * per, bs, Hkv, D, generator=g, device="cuda").bfloat16() for _ in range(2))
    tables = torch.arange(n * per, dtype=torch.int32, device="cuda").view(n, per)
    out = KC.paged_decode(q, k, v, tables, torch.full((n,), L, dtype=torch.int32, device="cuda"))
    kk, vv = (t.view(n, per * bs, Hkv, D)[:, :L].double().repeat_interleave(H // Hkv, 2) for t in (k, v))
    w = torch.softmax(torch.einsum("nhd,nkhd->nhk", q.double(), kk) * D ** -0.5, -1)
    ref = torch.einsum("nhk,nkhd->nhd", w, vv)
    # the result's rounding to bf16 alone; fp32 scores, weights and sums are 2^-14 and below
    bound = ref.abs() * 2.0 ** -8 + torch.einsum("nhk,nkhd->nhd", w, vv.abs()) * 2.0 ** -14
    assert ((out.double() - ref).abs() <= bound).all()


# shares of very different and of like lengths (as many as make one round of warps), sequences without keys, more sequences than add up their lengths, a block each
@pytest.mark.parametrize("H,Hkv,lens", [(32, 4, [4000, 3, 0, 70] + [17] * 40 + [900]), (8, 1, [2500] + [1] * 200), (16, 8, [0, 0, 5]), (32, 8, [33] * 700),
                                        (12, 3, [16 * i for i in range(50)]), (16, 1, [5000, 0, 40]), (8, 8, [1] * 450), (4, 1, [7000]),
                                        (32, 4, [3500] * 8), (32, 4, [700] * 20), (32, 4, [3500] * 7 + [1])])          # a round's room used up, and not
def test_shares_by_the_lengths(H, Hkv, lens):
    D, bs, n = 128, 16, len(lens)
    g = torch.Generator(device="cuda").manual_seed(n)
    per = [-(-l // bs) for l in lens]
    k, v = (torch.randn(max(1, sum(per)), bs, Hkv, D, generator=g, device="cuda").bfloat16() for _ in range(2))
    order = torch.randperm(sum(per), generator=torch.Generator().manual_seed(n)).tolist()
    tables, at = torch.zeros(n, max(per) + 3, dtype=torch.int32), 0
    for s in range(n):
        tables[s, :per[s]] = torch.tensor(order[at:at + per[s]], dtype=torch.int32)
        at += per[s]
    q = torch.randn(n, H, D, generator=g, device="cuda").bfloat16()
    out = KC.paged_decode(q, k, v, tables.cuda(), torch.tensor(lens, dtype=torch.int32, device="cuda"), out=torch.full_like(q, 9.0), impl="stream")
    for s, l in enumerate(lens):
        if l == 0:
            assert (out[s] == 0).all()
            continue
        kk, vv = (t[order[sum(per[:s]):sum(per[:s + 1])]].reshape(-1, Hkv, D)[:l].double().repeat_interleave(H // Hkv, 1) for t in (k, v))
        w = torch.softmax(torch.einsum("hd,khd->hk", q[s].double(), kk) * D ** -0.5, -1)
        ref = torch.einsum("hk,khd->hd", w, vv)
        bound = torch.einsum("hk,khd->hd", w, vv.abs()) * 2.0 ** -8 + ref.abs() * 2.0 ** -8 + 1e-5          # as above
        assert ((out[s].double() - ref).abs() <= bound).all(), (s, l)


# batches of less and of more than a round of warps, both group sizes; one block of tables throughout
@pytest.mark.parametrize("H,Hkv,n,length", [(32, 4, 64, 1800), (32, 8, 8, 3500), (32, 8, 48, 2600), (16, 1, 40, 700), (32, 4, 3, 2000)])
def test_neighbours_leave_a_sequence_alone(H, Hkv, n, length):
    """A sequence's result has the same bits whatever the lengths of the others in its batch."""
    D, bs, width = 128, 16, 256
    g = torch.Generator(device="cuda").manual_seed(n)
    k, v = (torch.randn(2 * width, bs, Hkv, D, generator=g, device="cuda").bfloat16() for _ in range(2))
    q = torch.randn(n, H, D, generator=g, device="cuda").bfloat16()
    tables = torch.arange(width, 2 * width, dtype=torch.int32, device="cuda").repeat(n, 1)         # the others share their pages
    tables[0] -= width
    def first(others):
        lens = torch.tensor([length] + [others(i) for i in range(1, n)], dtype=torch.int32, device="cuda")
        return KC.paged_decode(q, k, v, tables, lens, impl="stream")[0]
    want = first(lambda i: length)
    for others in (lambda i: 1, lambda i: 4096, lambda i: 1 + 997 * i % 4096, lambda i: 0):
        assert torch.equal(first(others), want)
