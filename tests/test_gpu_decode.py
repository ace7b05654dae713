"""Decode kernels and the decode engine against fp32 torch references (one GPU)."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _pools(b, max_pages, page_size, nkv, h, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    n_pages = b * max_pages + 3
    k = torch.randn(n_pages, page_size, nkv, h, device="cuda", generator=g).bfloat16()
    v = torch.randn(n_pages, page_size, nkv, h, device="cuda", generator=g).bfloat16()
    # A scrambled page table: sequences own arbitrary pages.
    perm = torch.randperm(n_pages, device="cuda", generator=g)[:b * max_pages].to(torch.int32)
    return k, v, perm.reshape(b, max_pages).contiguous()


@pytest.mark.parametrize("nq,nkv", [(4, 4), (8, 2), (8, 1), (6, 3), (8, 4), (16, 4), (32, 8)])
@pytest.mark.parametrize("splits", [1, 3])
def test_paged_decode_attention_matches_reference(nq, nkv, splits):
    from axlearn_b200.ops import cuda_ops, decode_ops

    b, page_size, max_pages, h = 5, 16, 9, 128
    k, v, table = _pools(b, max_pages, page_size, nkv, h)
    lengths = torch.tensor([1, 16, 17, 100, 144], dtype=torch.int32, device="cuda")
    q = torch.randn(b, nq, h, device="cuda").bfloat16()
    out = decode_ops.paged_decode_attention(q, k, v, table, lengths, splits=splits)
    ref = decode_ops.reference_paged_attention(q, k, v, table, lengths)
    torch.cuda.synchronize()
    cuda_ops.check_status()
    err = (out.float() - ref).abs().max().item()
    assert err < 2e-2 * max(1.0, ref.abs().max().item()), err


@pytest.mark.parametrize("nq,nkv", [(3, 3), (12, 4), (16, 2), (12, 1), (20, 2)])
@pytest.mark.parametrize("page_size,splits", [(4, 1), (12, 2), (16, 5), (16, 8), (20, 9)])
def test_paged_decode_attention_at_tile_and_split_edges(nq, nkv, page_size, splits):
    """Lengths around the 16-token tiles and the four warps' stride, rows that leave splits empty, up to eight and more
    than eight query heads per KV head, cluster merges (2 to 8 splits) and the merge launch (9)."""
    from axlearn_b200.ops import decode_ops

    lens = [0, 1, 15, 16, 17, 63, 64, 65, 129, 240]
    b, max_pages, h = len(lens), 240 // page_size, 128
    k, v, table = _pools(b, max_pages, page_size, nkv, h, seed=splits)
    lengths = torch.tensor(lens, dtype=torch.int32, device="cuda")
    q = (2 * torch.randn(b, nq, h, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))).bfloat16()
    out = decode_ops.paged_decode_attention(q, k, v, table, lengths, splits=splits)
    ref = decode_ops.reference_paged_attention(q[1:], k, v, table[1:], lengths[1:])
    assert not out[0].any()  # nothing cached
    # The output's rounding to bf16 (8 significant bits: half a unit is up to 2^-8 of a value), and sums of values of
    # size max|v| in 32 bits with P to 2^-15.
    bound = 2.0 ** -8 * ref.abs() + 2.0 ** -14 * v.abs().max().float()
    assert ((out[1:].float() - ref).abs() <= bound).all()


@pytest.mark.parametrize("nq,nkv", [(4, 4), (8, 4), (12, 4), (16, 4), (20, 4), (32, 4), (36, 4)])
def test_paged_decode_attention_keeps_32_bit_probabilities(nq, nkv):
    """The splits' 32-bit partials, merged here in 64 bits, for every number of copies of the heads in a tile.  Scores of up
    to 32 (in powers of two) are rounded by up to 2^-20 in 32 bits, and their probabilities with them; 16-bit terms of P
    would show as 2^-17 a probability, 1.4e-6 of the result."""
    from axlearn_b200.ops import decode_ops

    b, t, h, splits = 3, 1500, 128, 9
    k, v, table = _pools(b, (t + 15) // 16, 16, nkv, h, seed=nq)
    lengths = torch.tensor([1500, 777, 130], dtype=torch.int32, device="cuda")
    q = (2 * torch.randn(b, nq, h, device="cuda", generator=torch.Generator(device="cuda").manual_seed(2))).bfloat16()
    scratch = torch.empty(b * nq * splits * (h + 2), device="cuda")
    decode_ops.paged_decode_attention(q, k, v, table, lengths, splits=splits, scratch=scratch)
    sums = scratch[:b * nq * splits * h].view(b, nq, splits, h).double()
    top, total = scratch[b * nq * splits * h:].view(b, nq, splits, 2).double().unbind(-1)
    weight = torch.exp2(top - top.amax(-1, keepdim=True))
    got = (sums * weight[..., None]).sum(2) / (total * weight).sum(-1)[..., None]
    for i in range(b):
        n = int(lengths[i])
        kk, vv = (x[table[i].long()].reshape(-1, nkv, h)[:n].double().repeat_interleave(nq // nkv, 1) for x in (k, v))
        p = (torch.einsum("nh,snh->ns", q[i].double(), kk) * h ** -0.5).softmax(-1)
        want = torch.einsum("ns,snh->nh", p, vv)
        assert (got[i] - want).norm() <= 2.0 ** -20 * want.norm()


def test_paged_decode_attention_keeps_infinite_values():
    from axlearn_b200.ops import decode_ops

    k, v, table = _pools(2, 3, 16, 2, 128, seed=3)
    v[table[0, 1].long(), 5, 1, 7] = float("inf")
    lengths = torch.tensor([40, 33], dtype=torch.int32, device="cuda")
    q = torch.randn(2, 4, 128, device="cuda").bfloat16()
    for splits in (1, 3):
        out = decode_ops.paged_decode_attention(q, k, v, table, lengths, splits=splits).float()
        bad = ~torch.isfinite(out)
        assert (out[0, 2:, 7] == float("inf")).all() and bad.sum() == 2


def test_chained_step_sees_new_weights_and_matches_separate_launches():
    """A captured step reads its first weight tiles ahead of the kernels before it: new weights written right before a
    replay have to show, and the logits are those of separately launched kernels bit for bit."""
    from axlearn_b200.inference.decode_engine import DecodeEngine, FujiDims, LayerWeights

    d, f, vocab, nq, nkv, b = 256, 512, 1024, 4, 2, 3
    g = torch.Generator(device="cuda").manual_seed(0)

    def w(*shape):
        return (torch.randn(*shape, device="cuda", generator=g) * shape[0] ** -0.5).bfloat16()

    layers = [LayerWeights(attn_norm=1 + 0.1 * w(d), wqkv=w(d, (nq + 2 * nkv) * 128), wo=w(nq * 128, d),
                           ffn_norm=1 + 0.1 * w(d), wgu=w(d, 2 * f), wdown=w(f, d)) for _ in range(3)]
    weights = {"layers": layers, "emb": w(vocab, d) * 16, "head": w(vocab, d), "final_norm": 1 + 0.1 * w(d)}
    dims = FujiDims(num_layers=3, hidden_dim=d, num_heads=nq, num_kv_heads=nkv, head_dim=128, ffn_dim=f, vocab_size=vocab)
    engines = [DecodeEngine(weights, dims, batch=b, max_len=64, use_graph=use) for use in (True, False)]
    ids = torch.randint(0, vocab, (b, 9), device="cuda", generator=g)
    for e in engines:
        e.prefill(ids)
    tokens = ids[:, 0]
    for _ in range(6):
        for lw in layers:
            for t in (lw.wqkv, lw.wo, lw.wgu, lw.wdown):
                t.copy_(w(*t.shape))
        chained, plain = (e.step_logits(tokens).clone() for e in engines)
        assert torch.equal(chained, plain)
        tokens = plain.argmax(dim=-1)


@pytest.mark.parametrize("d,f,vocab,nq,nkv,b", [(2048, 5632, 4096, 16, 16, 1), (4096, 14336, 8192, 32, 8, 16)])
def test_chained_steps_at_serving_widths(d, f, vocab, nq, nkv, b):
    """Kernels that overlap for long: replays of the chained step against separate launches, bit for bit."""
    from axlearn_b200.inference.decode_engine import DecodeEngine, FujiDims, LayerWeights

    g = torch.Generator(device="cuda").manual_seed(1)

    def w(*shape):
        return (torch.randn(*shape, device="cuda", generator=g) * shape[0] ** -0.5).bfloat16()

    layers = [LayerWeights(attn_norm=1 + 0.1 * w(d), wqkv=w(d, (nq + 2 * nkv) * 128), wo=w(nq * 128, d),
                           ffn_norm=1 + 0.1 * w(d), wgu=w(d, 2 * f), wdown=w(f, d)) for _ in range(4)]
    weights = {"layers": layers, "emb": w(vocab, d) * 16, "head": w(vocab, d), "final_norm": 1 + 0.1 * w(d)}
    dims = FujiDims(num_layers=4, hidden_dim=d, num_heads=nq, num_kv_heads=nkv, head_dim=128, ffn_dim=f, vocab_size=vocab)
    engines = [DecodeEngine(weights, dims, batch=b, max_len=512, use_graph=use) for use in (True, False)]
    ids = torch.randint(0, vocab, (b, 300), device="cuda", generator=g)
    lengths = torch.randint(1, 301, (b,), device="cuda", generator=g)
    for e in engines:
        e.prefill(ids, lengths=lengths)
    for i in range(24):
        chained, plain = (e.step_logits(ids[:, i]).clone() for e in engines)
        assert torch.equal(chained, plain), i


@pytest.mark.parametrize("b", [1, 5])
@pytest.mark.parametrize("family,name", [("sagisun", "wide"), ("sagisun", "mixed"), ("zukitar", "wide"),
                                         ("zukitar", "small")])
def test_chained_module_steps_see_new_weights_and_match_separate_launches(family, name, b, tmp_path):
    """Mixers on a side stream, gates, routing and states inside the chain, with weights changed before each replay."""
    import importlib

    from axlearn_b200.common.utils import flatten_items
    from axlearn_b200.inference.decode_engine import ModuleDecodeEngine
    from axlearn_b200.inference.model_loader import load_model

    ckpt = importlib.import_module(f"tests.{family}_checkpoints")
    cfg = ckpt.CONFIGS[name]
    loaded = load_model(ckpt.save(tmp_path, cfg, ckpt.random_tensors(cfg, seed=3)), dtype=torch.bfloat16, device="cuda")
    params = loaded.parameters["decoder"]
    engines = [ModuleDecodeEngine(loaded.decoder, params, batch=b, max_len=200, device="cuda", use_graph=use)
               for use in (True, False)]
    g = torch.Generator().manual_seed(b)
    ids = torch.randint(0, cfg["vocab"], (b, 70), generator=g).cuda()
    lengths = torch.randint(1, 71, (b,), generator=g)
    for e in engines:
        e.prefill(ids, lengths=lengths)
    matrices = [t for _, t in flatten_items(params) if t.dim() >= 2]
    assert matrices
    for i in range(20):
        if i % 4 == 0:
            for t in matrices:
                t.mul_(1.0 + 0.25 * (-1) ** (i // 4))
        active = torch.ones(b, dtype=torch.int32)
        active[i % b] = int(b == 1 or i % 3 > 0)
        for e in engines:
            e.set_active(active)
        chained, plain = (e.step_logits(ids[:, i]).clone() for e in engines)
        assert torch.equal(chained, plain), i
        for (_, x), (_, y) in zip(flatten_items(engines[0].states), flatten_items(engines[1].states)):
            assert torch.equal(x, y)


def _fuji_engine(use_graph, batch=3):
    from axlearn_b200.inference.decode_engine import DecodeEngine, FujiDims, LayerWeights

    d, f, vocab, nq, nkv = 256, 512, 1000, 4, 2
    g = torch.Generator(device="cuda").manual_seed(0)

    def w(*shape):
        return (torch.randn(*shape, device="cuda", generator=g) * shape[0] ** -0.5).bfloat16()

    layers = [LayerWeights(attn_norm=1 + 0.1 * w(d), wqkv=w(d, (nq + 2 * nkv) * 128), wo=w(nq * 128, d),
                           ffn_norm=1 + 0.1 * w(d), wgu=w(d, 2 * f), wdown=w(f, d)) for _ in range(2)]
    weights = {"layers": layers, "emb": w(vocab, d) * 16, "head": w(vocab, d), "final_norm": 1 + 0.1 * w(d)}
    dims = FujiDims(num_layers=2, hidden_dim=d, num_heads=nq, num_kv_heads=nkv, head_dim=128, ffn_dim=f, vocab_size=vocab)
    return DecodeEngine(weights, dims, batch=batch, max_len=64, use_graph=use_graph), vocab, -vocab, vocab


def _module_engine(use_graph, tmp_path, batch=3):
    from axlearn_b200.inference.decode_engine import ModuleDecodeEngine
    from axlearn_b200.inference.model_loader import load_model
    from tests import sagisun_checkpoints as ckpt

    cfg = ckpt.CONFIGS["odd"]
    loaded = load_model(ckpt.save(tmp_path, cfg, ckpt.random_tensors(cfg)), dtype=torch.bfloat16, device="cuda")
    engine = ModuleDecodeEngine(loaded.decoder, loaded.parameters["decoder"], batch=batch, max_len=64, device="cuda",
                                use_graph=use_graph)
    return engine, cfg["vocab"], 0, (cfg["vocab"] + 31) // 32 * 32  # rows of the padded table


@pytest.mark.parametrize("use_graph", [True, False])
@pytest.mark.parametrize("kind", ["fuji", "module"])
def test_step_logits_refuses_ids_outside_the_table(kind, use_graph, monkeypatch, tmp_path):
    """On the host before anything runs; on the GPU by the operator's way, an assertion on the device: a stand-in for it
    records here which flag it is given (in the captured step, or by every separate one)."""
    from axlearn_b200.ops import cuda_ops

    engine, vocab, low, high = _fuji_engine(use_graph) if kind == "fuji" else _module_engine(use_graph, tmp_path)
    asserted = []
    monkeypatch.setattr(torch, "_assert_async", lambda ok, message: asserted.append(ok))
    ids = torch.randint(0, vocab, (3, 5), device="cuda")
    engine.prefill(ids)
    lengths = engine.lengths.clone()
    for bad in (high, low - 1, 1 << 40, -(1 << 40)):
        with pytest.raises(IndexError, match="outside"):
            engine.step_logits(torch.tensor([0, bad, 1]))
        assert torch.equal(engine.lengths, lengths)
        logits = engine.step_logits(torch.tensor([0, bad, 1], device="cuda"))
        assert not engine._ids_ok  # pylint: disable=protected-access
        assert logits.isfinite().all()  # the step itself has not seen the id
        engine.prefill(ids)
    cuda_ops.check_status()
    given = torch.tensor([low, high - 1, 0], device="cuda")
    for feed in (given, given.cpu(), given.int(), given[:, None]):
        engine.prefill(ids)
        got = engine.step_logits(feed).clone()
        engine.prefill(ids)
        assert engine._ids_ok  # pylint: disable=protected-access
        assert torch.equal(got, engine.step_logits(given)) and got.isfinite().all()
    assert len(asserted) == (1 if use_graph else 12)
    assert all(ok is engine._ids_ok for ok in asserted)  # pylint: disable=protected-access


def test_a_layer_call_with_one_token_keeps_the_embedding_operator(monkeypatch, tmp_path):
    """The gather that only marks bad ids is for captured steps, whose engine has looked at them."""
    from axlearn_b200.ops import step_ops

    engine = _module_engine(False, tmp_path)[0]
    engine.prefill(torch.randint(0, 60, (3, 4), device="cuda"))

    def refuse(*_, **__):
        raise AssertionError("the marking gather outside of a captured step")

    monkeypatch.setattr(step_ops, "embed_rows", refuse)
    engine.extend(torch.randint(0, 60, (3, 1), device="cuda"))
    engine.step_logits(torch.randint(0, 60, (3,), device="cuda"))


@pytest.mark.parametrize("b,v,ld", [(1, 1, 4), (3, 33, 40), (2, 4096, 4096), (5, 32768, 32768), (2, 32772, 32776)])
def test_step_end_picks_as_torch_and_keeps(b, v, ld):
    """Vector and element paths around one pass of the block; ties go to the first, NaN above all."""
    from axlearn_b200.ops import step_ops

    g = torch.Generator(device="cuda").manual_seed(v)
    logits = torch.randint(-50, 50, (b, ld), device="cuda", generator=g).float()[:, :v]
    if v > 1:
        logits[0] = float("-inf")
    if b > 2:
        logits[1, [v // 3, v // 2]] = float("nan")
    tokens = torch.full((b,), -1, dtype=torch.int64, device="cuda")
    lengths, active = (torch.arange(b, dtype=torch.int32, device="cuda") + i for i in range(2))
    kept = [(torch.zeros(b, dtype=torch.int32, device="cuda"), lengths + 10 * i) for i in range(3)]
    copy = torch.empty((b, v), device="cuda")
    want_lengths = lengths + active
    step_ops.step_end(logits, tokens, logits_out=copy, lengths=lengths, active=active, kept=kept)
    # numpy names the first of equals, and the first NaN.
    assert tokens.tolist() == logits.cpu().numpy().argmax(axis=-1).tolist()
    assert torch.equal(copy.nan_to_num(99.0), logits.nan_to_num(99.0))
    assert torch.equal(lengths, want_lengths) and all(torch.equal(x, y) for x, y in kept)


@pytest.mark.parametrize("b", [1, 3, 256, 300])
def test_advance_in_a_captured_chain(b):
    from axlearn_b200.ops import cuda_ops, step_ops

    counts = torch.arange(b, dtype=torch.int32, device="cuda")
    by = torch.arange(b, dtype=torch.int32, device="cuda") % 2
    assert torch.equal(step_ops.advance(counts, by), counts + by) and torch.equal(step_ops.advance(counts, 2), counts + 2)
    graph = torch.cuda.CUDAGraph()
    before = cuda_ops.launch_count
    with torch.cuda.graph(graph), cuda_ops.chained_launches():
        out = step_ops.advance(step_ops.advance(counts, by), by)
        plain = step_ops.advance(counts, 2)
    assert cuda_ops.launch_count == before + 2
    counts += 5
    graph.replay()
    assert torch.equal(out, counts + 2 * by) and torch.equal(plain, counts + 2)


@pytest.mark.parametrize("width", [8, 264, 2048, 4104])
def test_embed_rows_gathers_and_marks_bad_ids(width):
    from axlearn_b200.ops import cuda_ops, step_ops

    table = torch.randn(7, width, device="cuda").bfloat16()
    ids = torch.tensor([[6], [0], [-2]], device="cuda")
    lengths = torch.tensor([3, 8, 9], dtype=torch.int32, device="cuda")
    out = step_ops.embed_rows(table, ids, wrap=True, lengths=lengths, max_len=9)
    assert torch.equal(out, table[ids]) and lengths.tolist() == [4, 9, 9]
    cuda_ops.check_status()
    out = step_ops.embed_rows(table, ids)
    assert torch.equal(out[:2], table[ids[:2]]) and out[2].isnan().all()
    with pytest.raises(RuntimeError, match="status 5"):
        cuda_ops.check_status()


def test_rope_append_writes_page_slot_and_rotates():
    from axlearn_b200.ops import decode_ops, reference

    b, nq, nkv, h, page_size, max_pages = 3, 4, 2, 128, 16, 4
    k, v, table = _pools(b, max_pages, page_size, nkv, h, seed=1)
    k0, v0 = k.clone(), v.clone()
    lengths = torch.tensor([1, 16, 40], dtype=torch.int32, device="cuda")
    qkv = torch.randn(b, (nq + 2 * nkv) * h, device="cuda").bfloat16()
    q = decode_ops.rope_append_paged(qkv, k, v, table, lengths, num_q_heads=nq, theta=5e5)
    x = qkv.reshape(b, 1, nq + 2 * nkv, h)
    for i in range(b):
        pos = torch.tensor([int(lengths[i]) - 1], device="cuda")
        ref_q = reference.rope(x[i:i + 1, :, :nq].float(), pos, 5e5)[0, 0]
        ref_k = reference.rope(x[i:i + 1, :, nq:nq + nkv].float(), pos, 5e5)[0, 0]
        assert (q[i].float() - ref_q).abs().max() < 3e-2
        page = int(table[i, (int(lengths[i]) - 1) // page_size])
        off = (int(lengths[i]) - 1) % page_size
        assert (k[page, off].float() - ref_k).abs().max() < 3e-2
        assert torch.equal(v[page, off], x[i, 0, nq + nkv:])
        k0[page, off], v0[page, off] = k[page, off], v[page, off]
    # Nothing else was touched.
    assert torch.equal(k, k0) and torch.equal(v, v0)


@pytest.mark.parametrize("nq,nkv", [(3, 3), (4, 2), (12, 4), (16, 2), (12, 1), (20, 2)])
@pytest.mark.parametrize("page_size,splits", [(4, 1), (12, 2), (16, 5), (16, 8), (20, 9)])
def test_rope_decode_attention_equals_append_and_attention(nq, nkv, page_size, splits):
    """Bit for bit, attention and pools: new tokens at the edges of tiles, pages, warps' strides and splits, alone in their
    tile or not, up to eight and more than eight query heads per KV head."""
    from axlearn_b200.ops import decode_ops

    lens = [1, 2, 15, 16, 17, 33, 63, 64, 65, 129, 224, 240]
    b, max_pages, h = len(lens), 240 // page_size, 128
    k, v, table = _pools(b, max_pages, page_size, nkv, h, seed=splits)
    lengths = torch.tensor(lens, dtype=torch.int32, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(nq)
    qkv = (2 * torch.randn(b, (nq + 2 * nkv) * h, device="cuda", generator=g)).bfloat16()
    k1, v1 = k.clone(), v.clone()
    q = decode_ops.rope_append_paged(qkv, k1, v1, table, lengths, num_q_heads=nq, theta=1e4)
    want = decode_ops.paged_decode_attention(q, k1, v1, table, lengths, splits=splits)
    out = decode_ops.rope_decode_attention(qkv, k, v, table, lengths, num_q_heads=nq, theta=1e4, softmax_scale=h ** -0.5,
                                           splits=splits)
    assert torch.equal(out, want) and torch.equal(k, k1) and torch.equal(v, v1)


@pytest.mark.parametrize("b,t,nq,nkv", [(1, 1, 4, 4), (2, 127, 6, 2), (3, 129, 16, 1), (1, 300, 40, 8)])
def test_prompt_attention_equals_rotation_copies_and_attention(b, t, nq, nkv):
    """Bit for bit what separate rotations, copies into the cache and attention on contiguous tensors give; rows of the
    cache beyond the prompts stay."""
    from axlearn_b200.ops import attention_ops, cuda_ops, decode_ops

    h, rows = 128, t + 5
    qkv = torch.randn(b, t, (nq + 2 * nkv) * h, device="cuda").bfloat16()
    kp, vp = (torch.full((b, rows, nkv, h), 7.0, device="cuda").bfloat16() for _ in range(2))
    x, pos = qkv.clone().reshape(b, t, nq + 2 * nkv, h), torch.arange(t, device="cuda")
    q, k = cuda_ops.rope(x[:, :, :nq], pos, 5e5), cuda_ops.rope(x[:, :, nq:nq + nkv], pos, 5e5)
    v = x[:, :, nq + nkv:].contiguous()
    want = attention_ops.flash_attention(q, k, v, causal=True, softmax_scale=0.1)
    got = decode_ops.prompt_attention(qkv, kp, vp, decode_ops.rope_table(t, h, 5e5, "cuda"), num_q_heads=nq,
                                      softmax_scale=0.1)
    cuda_ops.check_status()
    assert torch.equal(kp[:, :t], k) and torch.equal(vp[:, :t], v) and (kp[:, t:] == 7).all() and (vp[:, t:] == 7).all()
    assert torch.equal(got.reshape(want.shape), want)


@pytest.mark.parametrize("variant", ["v1", "v2"])
def test_prompt_attention_follows_the_chosen_forward_kernel(variant, monkeypatch):
    """Bit for bit that kernel on separate tensors, where it was always v3."""
    from axlearn_b200.ops import cuda_ops, decode_ops, flash_sm100

    b, t, nq, nkv, h = 2, 150, 6, 2, 128
    qkv = torch.randn(b, t, (nq + 2 * nkv) * h, device="cuda").bfloat16()
    kp, vp = (torch.zeros((b, t + 5, nkv, h), device="cuda").bfloat16() for _ in range(2))
    table = decode_ops.rope_table(t, h, 5e5, "cuda")
    v3 = decode_ops.prompt_attention(qkv.clone(), kp, vp, table, num_q_heads=nq, softmax_scale=0.1)
    q = cuda_ops.rope(qkv.reshape(b, t, nq + 2 * nkv, h)[:, :, :nq], torch.arange(t, device="cuda"), 5e5)
    monkeypatch.setattr(flash_sm100, "FORWARD_VARIANT", variant)
    want, _ = flash_sm100.forward(q.contiguous(), kp[:, :t].contiguous(), vp[:, :t].contiguous(), causal=True, scale=0.1)
    calls, forward = [], flash_sm100.forward
    monkeypatch.setattr(flash_sm100, "forward", lambda *a, **k: calls.append(1) or forward(*a, **k))
    got = decode_ops.prompt_attention(qkv, kp, vp, table, num_q_heads=nq, softmax_scale=0.1)
    cuda_ops.check_status()
    assert calls and torch.equal(got.reshape(want.shape), want)
    # Each is within bf16 roundings of P and the output (2^-8 each) of the same sums of values of size max|v|.
    assert ((got.float() - v3.float()).abs() <= 2.0 ** -6 * vp.abs().max().float()).all()


@pytest.mark.parametrize("rows,f", [(1, 8), (3, 98), (2, 4096), (5, 4104), (70000, 16)])
def test_swiglu_packed_sizes(rows, f):
    """Vector and pairwise paths, around a block's 512 vectors, and more rows than a grid is high."""
    from axlearn_b200.ops import decode_ops

    gu = torch.randn(rows, 2 * f, device="cuda").bfloat16()
    ref = torch.nn.functional.silu(gu[:, :f].double()) * gu[:, f:].double()
    # Rounding to bf16, and a 32-bit sigmoid to about 2^-20 of itself.
    assert ((decode_ops.swiglu_packed(gu).double() - ref).abs() <= (2.0 ** -8 + 2.0 ** -18) * ref.abs() + 1e-30).all()


def test_swiglu_packed():
    from axlearn_b200.ops import decode_ops

    gu = torch.randn(7, 2 * 96, device="cuda").bfloat16()
    out = decode_ops.swiglu_packed(gu)
    ref = torch.nn.functional.silu(gu[:, :96].float()) * gu[:, 96:].float()
    assert (out.float() - ref).abs().max() < 3e-2


def test_one_shot_all_reduce_emulated():
    """Four emulated ranks on one GPU: every rank pushes first (separate launches), then every
    rank finishes -- no launch waits on a later one."""
    from axlearn_b200.ops import cuda_ops, decode_ops

    world, n, sites = 4, 4096, 2
    ranks = [decode_ops.OneShotAllReduce(n, sites, device="cuda", peers=[None] * world, rank=r) for r in range(world)]
    for r in ranks:
        r.connect(ranks)
    for step in range(2):
        xs = [torch.randn(n, device="cuda").bfloat16() for _ in range(world)]
        res = torch.randn(n, device="cuda").bfloat16()
        for r in ranks:
            r.begin_step()
        for site in range(sites):
            for r, x in zip(ranks, xs):
                r.push(x, site)
            for r in ranks:
                out = r.finish(site, residual=res)
                ref = res.float() + sum(x.float() for x in xs)
                assert (out.float() - ref).abs().max() < 5e-2, (step, site)
    torch.cuda.synchronize()
    cuda_ops.check_status()


@pytest.mark.parametrize("world,m,k,n", [(2, 64, 256, 512), (2, 4096, 512, 1024), (4, 2048, 256, 2048)])
def test_gemm_with_all_reduce_push_epilogue_emulated(world, m, k, n):
    """Emulated ranks: each rank's GEMM stores its rows into every staging buffer and raises the
    flags itself; the finish kernels then see residual + the sum of the products.  The small case
    runs on the single-CTA kernel, the large ones on the CTA-pair kernel (TMA stores per peer)."""
    from axlearn_b200.ops import cuda_ops, decode_ops

    ranks = [decode_ops.OneShotAllReduce(m * n, 2, device="cuda", peers=[None] * world, rank=r) for r in range(world)]
    for r in ranks:
        r.connect(ranks)
    a = [torch.randn(m, k, device="cuda").bfloat16() for _ in range(world)]
    b = [(torch.randn(k, n, device="cuda") * 0.1).bfloat16() for _ in range(world)]
    res = torch.randn(m * n, device="cuda").bfloat16()
    for step in range(2):
        for r in ranks:
            r.begin_step()
        for r in range(world):
            ranks[r].gemm_push(a[r], b[r], 0)
        ref = res.float() + sum((x.float() @ y.float()).reshape(-1) for x, y in zip(a, b))
        for r in ranks:
            out = r.finish(0, residual=res)
            assert (out.float() - ref).abs().max() < 3e-2 * ref.abs().max(), step
    torch.cuda.synchronize()
    cuda_ops.check_status()


def _tiny_model(num_kv_heads):
    from axlearn_b200.common import prng
    from axlearn_b200.experiments.text.gpt import fuji

    cfg = fuji.model_config(num_layers=2, hidden_dim=256, num_heads=2, num_kv_heads=num_kv_heads, vocab_size=512,
                            rope_theta=1e4, shared_lm_head=False, ffn_dim=512)
    model = cfg.set(name="model").instantiate(parent=None)
    params = model.initialize_parameters_recursively(prng.PRNGKey(0))
    return model, params


@pytest.mark.parametrize("num_kv_heads,use_graph", [(None, True), (1, False)])
def test_decode_engine_matches_model_forward(num_kv_heads, use_graph):
    from axlearn_b200.common import prng
    from axlearn_b200.common.module import functional
    from axlearn_b200.inference.decode_engine import DecodeEngine, FujiDims, weights_from_fuji_state
    from axlearn_b200.ops import cuda_ops

    model, params = _tiny_model(num_kv_heads)
    dims = FujiDims(num_layers=2, hidden_dim=256, num_heads=2, num_kv_heads=num_kv_heads or 2, head_dim=128,
                    ffn_dim=512, vocab_size=512, rope_theta=1e4)
    weights = weights_from_fuji_state(params, dims, device="cuda")
    batch, t, new = 3, 128, 12
    engine = DecodeEngine(weights, dims, batch=batch, max_len=t + new + 4, device=torch.device("cuda"),
                          use_graph=use_graph)
    g = torch.Generator().manual_seed(0)
    prompts = torch.randint(2, 512, (batch, t), generator=g)
    tokens = engine.generate(prompts.cuda(), new).cpu()
    torch.cuda.synchronize()
    cuda_ops.check_status()
    assert engine.launches_per_step > 0
    # Teacher-forced fp32 logits of the reference model over prompt + generated tokens.
    from axlearn_b200.common.utils import tree_leaves

    full = torch.cat([prompts, tokens], dim=1).to(tree_leaves(params)[0].device)
    logits, _ = functional(model, prng.PRNGKey(1), params, dict(input_batch={"input_ids": full}),
                           is_training=False, method="extract_logits")
    for b in range(batch):
        for i in range(new):
            row = logits[b, t + i - 1].float().cpu()
            # The engine's pick is the reference argmax up to bf16 noise between near-ties.
            assert row.max() - row[tokens[b, i]] < 0.1 * max(1.0, row.std().item()), (b, i)


def test_sample_decode_api_runs_on_the_engine_and_matches_the_eager_path(monkeypatch):
    """``Model.sample_decode`` on a Fuji-shaped bf16 model on one GPU goes through the CUDA-graph
    engine; with deterministic sampling (top-k = 1) its tokens are those of the eager
    ``prefill_states`` / ``extend_step`` path, ragged prompts and two decodes per prompt included."""
    from axlearn_b200.common import decoding, logit_modifiers, prng
    from axlearn_b200.common.module import functional
    from axlearn_b200.common.utils import tree_map
    from axlearn_b200.inference import decode_engine
    from axlearn_b200.ops import cuda_ops

    model, params = _tiny_model(1)
    params = tree_map(lambda t: t.cuda().bfloat16() if t.is_floating_point() else t.cuda(), params)
    g = torch.Generator().manual_seed(3)
    prefix = torch.randint(2, 512, (3, 24), generator=g)
    prefix[1, 17:] = 0            # shorter prompts are right-padded with the pad id
    prefix[2, 9:] = 0
    calls = {"n": 0}
    real = decode_engine.DecodeEngine.step_logits

    def counted(self, tokens):
        calls["n"] += 1
        return real(self, tokens)

    monkeypatch.setattr(decode_engine.DecodeEngine, "step_logits", counted)
    kwargs = dict(input_batch={"prefix": prefix.cuda()}, num_decodes=2, max_sequence_length=40,
                  logits_modifier=logit_modifiers.top_k_logits(1),
                  stop_decoding_condition=decoding.StopOnSubsequence([[511]]))
    fast, _ = functional(model, prng.PRNGKey(5), params, kwargs, is_training=False, method="sample_decode")
    assert calls["n"] > 0, "the engine was not used"
    torch.cuda.synchronize()
    cuda_ops.check_status()
    monkeypatch.setenv("AXB200_DECODE_ENGINE", "0")
    before = calls["n"]
    slow, _ = functional(model, prng.PRNGKey(5), params, kwargs, is_training=False, method="sample_decode")
    assert calls["n"] == before
    assert fast.sequences.shape == slow.sequences.shape == (3, 2, 39)
    assert torch.equal(fast.sequences[:, :, :8], slow.sequences[:, :, :8])          # the prompts
    # With top-k = 1 every generated token must be the argmax of the model's own logits for the
    # sequence so far, up to bf16 noise between near-ties (a random model has many of those, so
    # the two paths may part ways at a tie and are therefore not compared token by token).
    lengths = (prefix != 0).sum(-1)
    for out in (fast, slow):
        full = torch.cat([prefix[:, :1].cuda().repeat_interleave(2, dim=0), out.sequences.reshape(6, 39)], dim=1)
        logits, _ = functional(model, prng.PRNGKey(1), params, dict(input_batch={"input_ids": full}),
                               is_training=False, method="extract_logits")
        for row in range(6):
            start = int(lengths[row // 2])
            for t in range(start, 40):
                tok = int(full[row, t])
                if tok == 0:
                    break
                ref = logits[row, t - 1].float()
                assert ref.max() - ref[tok] < 0.15 * max(1.0, ref.std().item()), (row, t)
    same = (fast.sequences == slow.sequences).float().mean().item()
    assert same > 0.5, same
