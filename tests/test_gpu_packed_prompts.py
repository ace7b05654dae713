"""Prompts without their padding against the padded ones: the mixers alone, and whole served models."""

import pytest
import torch

from axlearn_b200.ops import gla_ops, latent_ops, packed_ops, ssd_ops, window_ops

pytestmark = pytest.mark.gpu

# Sequences of one token, of none, at the edges of the kernels' chunks and tiles, and of all of T.
_LENGTHS = [[300, 1, 64, 65, 128, 255], [40, 40, 17], [1100, 700, 1], [129, 0, 256, 3]]


def _packed(lengths, width, seed):
    t = max(lengths)
    live = torch.tensor(lengths, dtype=torch.int32, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(seed)
    proj = torch.randn(len(lengths), t, width, device="cuda", generator=g).bfloat16()
    return packed_ops.PackedRows(live, t), live, proj


def _alike(packed, out, padded):
    """Bit by bit: a row's arithmetic does not know where the row lies."""
    assert torch.equal(out, packed.pack(padded)) and out.shape[1] == packed.rows


@pytest.mark.parametrize("lengths", _LENGTHS)
@pytest.mark.parametrize("groups,segments", [(1, None), (2, 2)])
def test_state_space(lengths, groups, segments):
    spec = ssd_ops.SsdSpec(heads=4, vdim=64, state=64, groups=groups, taps=4, norm_groups=2, eps=1e-6)
    cols = ssd_ops.SsdColumns(z=0, xbc=spec.inner, dt=spec.inner + spec.channels)
    packed, live, proj = _packed(lengths, spec.inner + spec.channels + 8, 1)
    w = ssd_ops.SsdWeights(*(torch.randn(n, device="cuda") * 0.3 for n in (
        (4, spec.channels), (spec.channels,), (4,), (4,), (4,), (spec.inner,))))

    def run(x, **more):
        state = {"ssm": torch.zeros(len(lengths), 4, 64, 64, device="cuda"),
                 "conv": torch.zeros(len(lengths), 4, spec.channels, device="cuda", dtype=torch.bfloat16)}
        cut = segments and (segments, -(-max(lengths) // segments // 64) * 64 + 64)
        return ssd_ops._cuda_ssd_mix(  # pylint: disable=protected-access
            x, w, spec, cols, start=None, state=state, segments=cut or None, **more)

    padded, want = run(proj, live=live)
    out, state = run(packed.pack(proj), live=live, packed=packed)
    _alike(packed, out, padded)
    assert torch.equal(state["ssm"], want["ssm"]) and torch.equal(state["conv"], want["conv"])


@pytest.mark.parametrize("lengths", _LENGTHS)
@pytest.mark.parametrize("segments", [None, (3, 384)])
def test_linear_attention(lengths, segments):
    spec = gla_ops.GlaSpec(heads=4, dim=64, vdim=128, rank=16, tau=16.0, q_scale=0.125, eps=1e-6)
    widths = [("q", 256), ("k", 256), ("v", 512), ("g", 512), ("a1", 16)]
    cols, at = {}, 0
    for name, n in widths:
        cols[name], at = at, at + n
    packed, live, proj = _packed(lengths, at, 2)
    a2, bias, norm = (torch.randn(*n, device="cuda") * 0.2 for n in ((256, 16), (256,), (128,)))

    def run(x, **more):
        state = torch.zeros(len(lengths), 4, 64, 128, device="cuda")
        return gla_ops._cuda_gla(x, a2.bfloat16(), bias, norm, spec, gla_ops.GlaColumns(**cols), start=None,  # pylint: disable=protected-access
                                 state=state, segments=segments, **more)

    padded, want = run(proj, live=live)
    out, state = run(packed.pack(proj), live=live, packed=packed)
    _alike(packed, out, padded)
    assert torch.equal(state, want)


@pytest.mark.parametrize("lengths", _LENGTHS)
@pytest.mark.parametrize("dim,window", [(64, 100), (128, 33)])
def test_window_attention(lengths, dim, window):
    spec = window_ops.WindowSpec(heads=4, kv_heads=2, dim=dim, vdim=dim, window=window, scale=dim ** -0.5,
                                 distance_bias=True, gated=True, q_temp=(0.1, 50))
    cols = window_ops.WindowColumns(q=0, k=4 * dim, v=6 * dim, g=8 * dim)
    packed, live, proj = _packed(lengths, 12 * dim, 3)

    def run(x, **more):
        cache = {n: torch.zeros(len(lengths), window, 2, dim, device="cuda", dtype=torch.bfloat16) for n in ("key", "value")}
        return window_ops.window_attention(x, spec, cols, live=live, cache=cache, **more)

    with torch.no_grad():
        padded, want = run(proj)
        out, cache = run(packed.pack(proj), packed=packed)
    _alike(packed, out, padded)
    assert torch.equal(cache["key"], want["key"]) and torch.equal(cache["value"], want["value"])


@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("bad", [float("nan"), float("inf"), float("-inf")])
def test_window_attention_keeps_sequences_apart(dim, bad):
    """Last tiles of 1, 127 and 128 keys, neighbours shorter than a tile, more than one bad neighbour in a tile: nothing that
    one sequence holds reaches another."""
    lengths = [129, 300, 5, 3, 255, 128, 1, 40]
    spec = window_ops.WindowSpec(heads=4, kv_heads=2, dim=dim, vdim=dim, window=100, scale=dim ** -0.5, distance_bias=True,
                                 gated=True)
    cols = window_ops.WindowColumns(q=0, k=4 * dim, v=6 * dim, g=8 * dim)
    packed, live, proj = _packed(lengths, 12 * dim, 4)

    def run(x):
        cache = {n: torch.zeros(len(lengths), 100, 2, dim, device="cuda", dtype=torch.bfloat16) for n in ("key", "value")}
        with torch.no_grad():
            return window_ops.window_attention(packed.pack(x), spec, cols, live=live, cache=cache, packed=packed)

    want, want_cache = run(proj)
    for spoilt in ([1], [2, 3], [0, 5, 7], [6]):
        x = proj.clone()
        x[spoilt] = bad
        got, cache = run(x)
        kept = [i for i in range(len(lengths)) if i not in spoilt]
        for i in kept:
            rows = slice(packed.first[i].item(), packed.first[i].item() + lengths[i])
            assert torch.equal(got[:, rows], want[:, rows]), (spoilt, i)
        assert all(torch.equal(cache[n][kept], want_cache[n][kept]) for n in cache)


@pytest.mark.parametrize("width", [1, 7, 8, 264, 2048, 4104])
def test_unpacked_padding_is_zero(width):
    lengths = [3, 0, 300, 256, 1]
    packed, _, x = _packed(lengths, width, 5)
    got = packed.unpack(packed.pack(x))
    want = x.clone()
    for i, n in enumerate(lengths):
        want[i, n:] = 0
    assert torch.equal(got, want)
    rows = packed.pack(x)
    rows[:, 0] = float("nan")
    assert not packed.unpack(rows)[1:].isnan().any()


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_latent_attention_keeps_sequences_apart(bad):
    """The first sequence as well, whose rows padding must not hold."""
    lengths, heads, dim, rot, vdim, rank = [129, 300, 5, 255, 128, 40], 4, 64, 32, 64, 128
    spec = latent_ops.LatentSpec(heads, dim, rot, vdim, rank, rot, 1000.0, 0.1, 1e-5)
    cols = latent_ops.LatentColumns(q=0, c=heads * (dim + rot), r=heads * (dim + rot) + rank)
    packed, live, proj = _packed(lengths, cols.r + rot, 6)
    g = torch.Generator(device="cuda").manual_seed(7)
    norm = torch.ones(rank, device="cuda")
    uk, uv = (0.1 * torch.randn(*n, device="cuda", generator=g).bfloat16() for n in ((rank, heads * dim), (heads * vdim, rank)))

    def run(x):
        cache = {"latent": torch.zeros(len(lengths), max(lengths), spec.row_width, device="cuda", dtype=torch.bfloat16)}
        with torch.no_grad():
            out, cache = latent_ops.latent_attention(packed.unpack(packed.pack(x)), norm, uk, uv, spec, cols, live=live, cache=cache)
        return packed.pack(out), cache["latent"]

    want, want_cache = run(proj)
    for spoilt in (0, 2, 4):
        x = proj.clone()
        x[spoilt] = bad
        got, cache = run(x)
        for i, n in enumerate(lengths):
            if i != spoilt:
                rows = slice(packed.first[i].item(), packed.first[i].item() + n)
                assert torch.equal(got[:, rows], want[:, rows]) and torch.equal(cache[i], want_cache[i]), (spoilt, i)


@pytest.mark.parametrize("family", ["sagisun", "zukitar"])
def test_served_prompts(family, monkeypatch):
    """The engine's logits after ragged prompts and its steps behind them, packed and padded: the same up to products of
    another number of rows, whose kernels sum in another order."""
    from perf import cases
    from axlearn_b200.ops import cuda_ops

    case = dict(kind="serve", family=family, size="1B", layers=2 if family == "sagisun" else 3, batch=5, prompt=1011)
    used = []
    plain = packed_ops.pack_prompts

    def pack(*args):
        used.append(plain(*args))
        return used[-1]

    monkeypatch.setattr(packed_ops, "pack_prompts", pack)
    got = cases.run(cases.prepare(case, 5))
    assert used and all(p is not None and p.rows < 5 * 1011 for p in used)
    monkeypatch.setattr(packed_ops, "pack_prompts", lambda *args: None)
    want = cases.run(cases.prepare(case, 5))
    for a, b in zip([got["prompt_logits"], *got["logits"]], [want["prompt_logits"], *want["logits"]]):
        assert (a - b).norm() <= 2e-2 * b.norm()
    cuda_ops.check_status()


def test_where_packing_does_not_pay():
    def pack(lengths, t):
        return packed_ops.pack_prompts(torch.tensor(lengths, dtype=torch.int32, device="cuda"), t)

    assert pack([4000], 8000) is None and pack([100, 40], 200) is None and pack([4000, 3990], 4000) is None
    assert pack([4000, 8000], 4000) is None  # more tokens than rows: all of them
    p = pack([0, 600, 700, -3], 2000)
    assert p.rows == 1300 and p.first.tolist() == [0, 0, 600, 1300] and p.live.tolist() == [0, 600, 700, 0]
    x = torch.arange(8000, device="cuda").reshape(4, 2000, 1)
    y = p.pack(x)
    assert y.flatten().tolist() == list(range(2000, 2600)) + list(range(4000, 4700))
    assert torch.equal(p.pack(p.unpack(y)), y)


@pytest.mark.parametrize("family", ["sagisun", "zukitar"])
def test_served_prompt_without_tokens(family, monkeypatch):
    """Among ragged prompts: its logits are still those of the padding in its first place, bit for bit."""
    from perf import cases
    from axlearn_b200.ops import cuda_ops

    case = dict(kind="serve", family=family, size="1B", layers=2 if family == "sagisun" else 3, batch=5, prompt=1011)
    state = cases.prepare(case, 5)
    state["lengths"][1:3] = torch.tensor([0, 400])
    engine = state["engine"]
    engine.prefill(state["ids"], lengths=state["lengths"])
    got = engine.logits.clone()
    monkeypatch.setattr(packed_ops, "pack_prompts", lambda *args: None)
    engine.prefill(state["ids"], lengths=state["lengths"])
    assert torch.equal(got, engine.logits)
    cuda_ops.check_status()


@pytest.mark.parametrize("lengths,t", [([4000, 4000], 4000), ([4000, 3990, 4000], 4000), ([4000, 8000], 4000), ([600, 700, 90], 2000),
                                       ([0, 600, 700, -3], 2000), ([100, 2, 3], 2000), ([100, 40], 200)])
def test_known_lengths_decide_without_a_wait(lengths, t):
    known = torch.tensor(lengths, dtype=torch.int32)
    live = known.cuda()
    want = packed_ops.pack_prompts(live, t)
    torch.cuda.set_sync_debug_mode("error")
    try:
        with packed_ops.lengths_known(live, known):
            got = packed_ops.pack_prompts(live, t)
        if want is not None:  # those of another batch are not this one's
            with packed_ops.lengths_known(live[:1], known[:1]), pytest.raises(RuntimeError, match="synchroniz"):
                packed_ops.pack_prompts(live, t)
    finally:
        torch.cuda.set_sync_debug_mode("default")
    assert (got is None) == (want is None)
    if got is not None:
        assert (got.rows, got.some_empty) == (want.rows, want.some_empty)
        assert torch.equal(got.first, want.first) and torch.equal(got.live, want.live)


@pytest.mark.parametrize("more", [1, -50, 400])
def test_known_lengths_are_not_those_that_a_model_makes_of_them(more):
    """A prefix that a model puts ahead of the prompts, say."""
    known = torch.tensor([600, 700, 90], dtype=torch.int32)
    live = known.cuda()
    made = live + more
    want = packed_ops.pack_prompts(made, 2000)
    with packed_ops.lengths_known(live, known):
        got = packed_ops.pack_prompts(made, 2000)
    assert got.rows == want.rows == 1390 + 3 * more and torch.equal(got.live, made)


def test_engine_tells_the_lengths_it_knows(monkeypatch):
    from perf import cases

    case = dict(kind="serve", family="sagisun", size="1B", layers=2, batch=5, prompt=1011)
    state = cases.prepare(case, 5)
    engine, ids, lengths = state["engine"], state["ids"], state["lengths"]
    used, plain = [], packed_ops.pack_prompts

    def pack(*args):
        used.append((plain(*args), getattr(packed_ops._known, "lengths", None)))  # pylint: disable=protected-access
        return used[-1][0]

    monkeypatch.setattr(packed_ops, "pack_prompts", pack)
    logits = []
    for given in (lengths, lengths.cpu(), lengths.cpu().long(), None):
        engine.prefill(ids, lengths=given)
        logits.append(engine.logits.clone())
    assert torch.equal(logits[0], logits[1]) and torch.equal(logits[0], logits[2])
    assert [p is not None for p, _ in used] == [True, True, True, False]
    assert used[0][1] is None and all(torch.equal(k, lengths.cpu()) for _, k in used[1:3])
    assert used[3][1].tolist() == [1011] * 5
    assert getattr(packed_ops._known, "lengths", None) is None  # pylint: disable=protected-access


@pytest.mark.parametrize("family", ["sagisun", "zukitar"])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_served_prompts_keep_sequences_apart(family, bad):
    """A token whose embedding is spoilt, in one prompt of a packed batch: the others' logits and states keep their bits."""
    from perf import cases
    from axlearn_b200.common.utils import flatten_items
    from axlearn_b200.ops import cuda_ops

    case = dict(kind="serve", family=family, size="1B", layers=2 if family == "sagisun" else 3, batch=5, prompt=1011)
    state = cases.prepare(case, 5)
    engine, ids, lengths = state["engine"], state["ids"].clone(), state["lengths"]
    table, token = engine.params["emb"]["token_emb"]["weight"], 77
    row = table[token].clone()
    ids[ids == token] = 78
    for spoilt in (0, 2):
        x = ids.clone()
        x[spoilt, 5] = token

        def run():
            engine.prefill(x, lengths=lengths)
            kept = [i for i in range(5) if i != spoilt]
            columns = torch.arange(engine.logits.shape[1], device="cuda") != token  # the table is the output product's, too
            states = [t[kept] for _, t in flatten_items(engine.states) if t.shape[0] == 5]
            return [engine.logits[kept][:, columns].clone()] + states, engine.logits[spoilt].clone()

        want, _ = run()
        table[token] = bad
        got, own = run()
        table[token] = row
        assert not own.isfinite().any()
        assert all(torch.equal(a, b) for a, b in zip(got, want)), spoilt
    cuda_ops.check_status()


@pytest.mark.parametrize("short", [False, True])
def test_prompts_behind_a_capture_find_their_memory(short, monkeypatch):
    """The capture of the step leaves the allocator's cache alone unless memory is short."""
    from perf import cases

    case = dict(kind="serve", family="sagisun", size="1B", layers=2, batch=5, prompt=1011)
    state = cases.prepare(case, 5)
    engine, want = state["engine"], cases.run(state)
    engine._graph = None  # pylint: disable=protected-access
    engine.prefill(state["ids"], lengths=state["lengths"])
    if short:
        monkeypatch.setattr(torch.cuda, "mem_get_info", lambda device=None: (1 << 20, 1 << 37))
    torch.cuda.synchronize()
    freed = torch.cuda.memory_stats()["segment.all.freed"]
    engine.step_logits(state["continuation"][:, 0])
    assert (torch.cuda.memory_stats()["segment.all.freed"] > freed) == short
    made = torch.cuda.memory_stats()["segment.all.allocated"]
    engine.prefill(state["ids"], lengths=state["lengths"])
    assert (torch.cuda.memory_stats()["segment.all.allocated"] > made) == short
    got = cases.run(state)
    assert torch.equal(got["prompt_logits"], want["prompt_logits"])
    assert all(torch.equal(a, b) for a, b in zip(got["logits"], want["logits"]))
