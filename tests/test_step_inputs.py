"""One-launch step inputs (csrc/step_inputs.cu) against the PyTorch forms they stand for."""
import pytest
import torch

from vllm_omni_b200.engine.graph_runner import DecodeGraphRunner
from vllm_omni_b200.models.qwen_decoder import DecoderConfig, ModelBatch, QwenDecoderModel
from vllm_omni_b200.models.seq_table import SeqTable

pytestmark = pytest.mark.gpu


def _decoder(mrope, interleaved=False):
    cfg = DecoderConfig(vocab_size=100, hidden_size=136, num_hidden_layers=1, num_attention_heads=2, num_key_value_heads=1, head_dim=128,
                        intermediate_size=64, mrope_section=(24, 20, 20) if mrope else None, mrope_interleaved=interleaved)
    return QwenDecoderModel(cfg, torch.bfloat16, "cuda")


@pytest.mark.parametrize("T", [1, 5, 300])
@pytest.mark.parametrize("axes", ["one", "sections", "interleaved", "one position for all"])
@pytest.mark.parametrize("overlay", [None, "mask", "all"])
def test_rows_and_rotation(T, axes, overlay):
    m = _decoder(axes != "one", axes == "interleaved")
    g = torch.Generator(device="cuda").manual_seed(T)
    ids = torch.randint(-3, 110, (T,), generator=g, device="cuda")              # outside the table too: held inside
    pos = torch.randint(0, 40000, (3, T) if axes in ("sections", "interleaved") else (T,), generator=g, device="cuda")
    kw = {}
    if overlay:
        kw["input_embeds"] = torch.randn(T, 136, generator=g, device="cuda").bfloat16()
        kw["embeds_mask"] = torch.rand(T, generator=g, device="cuda") < 0.5 if overlay == "mask" else None
    b = ModelBatch(ids, pos, None, **kw)
    x, cos, sin = m.rows_and_rotation(b)
    c, s = m.rope.cos_sin_for(pos, m.cfg.mrope_section, m.cfg.mrope_interleaved)
    assert torch.equal(x, m.embed(b))
    # the same fp32 angle; two correct cosines of it differ by an ulp of 1 at most
    assert (cos - c).abs().max() <= 2.0 ** -23 and (sin - s).abs().max() <= 2.0 ** -23 and cos.is_contiguous() and sin.is_contiguous()


@pytest.mark.parametrize("n", [1, 3, 4, 7])
@pytest.mark.parametrize("mrope,overlay,seqs", [(False, False, False), (True, True, False), (False, True, True), (True, False, True)])
def test_fill(n, mrope, overlay, seqs, monkeypatch):
    m = _decoder(mrope)
    m.uses_seq_table = seqs
    kv = [tuple(torch.zeros(8, 16, 1, 128, device="cuda", dtype=torch.bfloat16) for _ in range(2)) + ((torch.zeros(1, device="cuda"),) if seqs else ())]
    runners = [DecodeGraphRunner(m, kv, max_blocks=5, buckets=(1, 4, 8)) for _ in range(2)]
    g = torch.Generator(device="cuda").manual_seed(n)
    i32 = lambda *s: torch.randint(0, 50, s, generator=g, device="cuda", dtype=torch.int32)
    pos = torch.randint(0, 99, (3, n) if mrope and n != 3 else (n,), generator=g, device="cuda")
    b = ModelBatch(torch.randint(0, 99, (n,), generator=g, device="cuda"), pos, i32(n), [],
                   decode_rows=torch.randperm(n, generator=g, device="cuda"), decode_block_tables=i32(n, 6)[:, :3], decode_seq_lens=i32(n))
    if overlay:
        b.input_embeds, b.embeds_mask = torch.randn(n, 136, generator=g, device="cuda").bfloat16(), torch.rand(n, generator=g, device="cuda") < 0.5
    if seqs:
        b.seqs = SeqTable(None, i32(n), None, None, None, n, n, 0, i32(n), i32(n))
    states = []
    for r, once in zip(runners, (True, False)):
        if not once:
            monkeypatch.setattr(DecodeGraphRunner, "_fill_once", lambda *a: False)
        st = r._bucket(n)
        for name in ("ids", "pos", "slots", "tables", "lens"):
            getattr(st, name).fill_(77)                      # what an earlier step left
        st.emask.fill_(True)
        if once:
            assert r._fill_once(st, b)
        else:
            r._fill(st, b)
        states.append(st)
    a, c = states
    for name in ("ids", "pos", "slots", "tables", "lens", "emask") + (("embeds",) if overlay else ()) + (("ctx",) if seqs else ()):
        assert torch.equal(getattr(a, name), getattr(c, name)), name
    if seqs:
        assert torch.equal(a.seqs.state_in, c.seqs.state_in) and torch.equal(a.seqs.state_out, c.seqs.state_out)


def test_rows_on_another_device_are_left_to_the_general_form():
    """Given rows, their mask or positions in host memory: refused by the general form, never read by the kernel."""
    from vllm_omni_b200.ops.step_inputs import token_rows
    m, T = _decoder(False), 3
    ids = pos = torch.arange(T, device="cuda")
    given, mask, freq = torch.zeros(T, 136, dtype=torch.bfloat16), torch.ones(T, dtype=torch.bool), m.rope.freq_on(ids.device)
    assert token_rows(ids, m.embed_tokens, pos, freq, None, given.cuda(), mask.cuda()) is not None
    for kw in (dict(given=given), dict(given=given, mask=mask.cuda()), dict(given=given.cuda(), mask=mask)):
        assert token_rows(ids, m.embed_tokens, pos, freq, None, **kw) is None
    assert token_rows(ids, m.embed_tokens, pos.cpu(), freq) is None and token_rows(ids, m.embed_tokens, pos, freq.cpu()) is None
    with pytest.raises(RuntimeError):
        m.rows_and_rotation(ModelBatch(ids, pos, None, input_embeds=given, embeds_mask=mask))


def test_rotation_tables_are_fp32_whatever_the_default_type():
    m, pos = _decoder(False), torch.arange(5, device="cuda")
    want = m.rows_and_rotation(ModelBatch(pos, pos, None))
    torch.set_default_dtype(torch.bfloat16)
    try:
        got = m.rows_and_rotation(ModelBatch(pos, pos, None))
    finally:
        torch.set_default_dtype(torch.float32)
    assert all(a.dtype == b.dtype and torch.equal(a, b) for a, b in zip(want, got)) and got[1].dtype == torch.float32


def test_fill_takes_whole_rows_only():
    """Only block tables may be narrower than the static tensor; narrower embeddings are refused as before."""
    m, n = _decoder(False), 2
    r = DecodeGraphRunner(m, [tuple(torch.zeros(8, 16, 1, 128, device="cuda", dtype=torch.bfloat16) for _ in range(2))], max_blocks=5, buckets=(2,))
    i32 = lambda *s: torch.zeros(s, device="cuda", dtype=torch.int32)
    b = ModelBatch(torch.zeros(n, device="cuda", dtype=torch.long), torch.zeros(n, device="cuda", dtype=torch.long), i32(n), [],
                   decode_rows=torch.arange(n, device="cuda"), decode_block_tables=i32(n, 3), decode_seq_lens=i32(n))
    st = r._bucket(n)
    assert r._fill_once(st, b)
    b.input_embeds = torch.zeros(n, 72, device="cuda", dtype=torch.bfloat16)
    assert not r._fill_once(st, b)
    with pytest.raises(RuntimeError):
        r._fill(st, b)


def test_positions_of_two_axes_keep_the_general_form():
    """Sections of two axes (the one-launch form has three): the tables of the general form, as before there was another."""
    m = _decoder(False)
    m.cfg.mrope_section = (40, 24)
    pos = torch.arange(10, device="cuda").view(2, 5)
    ids = torch.arange(5, device="cuda")
    x, cos, sin = m.rows_and_rotation(ModelBatch(ids, pos, None))
    c, s = m.rope.cos_sin_for(pos, m.cfg.mrope_section, False)
    assert torch.equal(x, m.embed_tokens[ids]) and torch.equal(cos, c) and torch.equal(sin, s)


@pytest.mark.parametrize("experts,per_token", [(0, 8), (8, 5), (8, 6)])         # 3 sequences: 15 and 18 choices of 8 experts
@pytest.mark.parametrize("once", [True, False])
def test_padding_rows_of_a_step(experts, per_token, once, monkeypatch):
    """Without experts, or with two choices per expert, they see one key, else row 0's; either way its pages, and they write nothing."""
    long = experts and per_token == 5
    m = _decoder(False)
    m.cfg.num_experts, m.cfg.num_experts_per_tok, m.uses_seq_table = experts, per_token, True
    kv = [tuple(torch.zeros(8, 16, 1, 128, device="cuda", dtype=torch.bfloat16) for _ in range(2))]
    r = DecodeGraphRunner(m, kv, max_blocks=5, buckets=(8,))
    i32 = lambda *v: torch.tensor(v, dtype=torch.int32, device="cuda")
    b = ModelBatch(torch.arange(3, device="cuda"), torch.arange(3, device="cuda"), i32(4, 5, 6), [], decode_rows=torch.arange(3, device="cuda"),
                   decode_block_tables=i32(7, 8, 9)[:, None], decode_seq_lens=i32(20, 30, 40))
    b.seqs = SeqTable(None, i32(19, 29, 39), None, None, None, 3, 3, 0, None, None)
    if not once:
        monkeypatch.setattr(DecodeGraphRunner, "_fill_once", lambda *a: False)
    st = r._bucket(3)
    r._fill(st, b)
    assert st.lens.tolist() == [20, 30, 40] + [20 if long else 1] * 5
    assert st.ctx.tolist() == [19, 29, 39] + [19 if long else 0] * 5
    assert st.slots.tolist() == [4, 5, 6] + [-1] * 5 and st.tables[:, 0].tolist() == [7, 8, 9] + [7] * 5
