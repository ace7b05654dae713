"""The work that users of this framework run on one GPU, as measurable cases: training steps of Fuji decoders through
``SpmdTrainer``, prompts and decoding steps of Fuji decoders through ``DecodeEngine``, and whole served batches (prompts,
then decoding steps) of the Sagisun and Zukitar designs through ``ModuleDecodeEngine``.

``listed()`` names the cases, ``draw(rng)`` gives another one of the same ranges; ``prepare`` builds what a program holds
before the call, ``run`` is one pass, ``work`` what a pass cannot do without, ``exact`` the outputs in 64 bits.  Layers
repeat in these models, so a case has a few of them; widths are those of the named sizes.
"""

from __future__ import annotations

import math
import os
import tempfile

import torch

# ------------------------------------------------------------------------------------------
# Cases.
# ------------------------------------------------------------------------------------------

# Fuji decoders (head size 128 unless a head count says otherwise): widths of the sizes of that name.
_FUJI = {
    "1B": dict(hidden=2048, heads=16, kv=16, ffn=8192, theta=1e4),
    "1B-gqa": dict(hidden=2048, heads=16, kv=4, ffn=5632, theta=5e5),
    "7B": dict(hidden=4096, heads=32, kv=32, ffn=11008, theta=1e4),
    "8B": dict(hidden=4096, heads=32, kv=8, ffn=14336, theta=5e5),
}
_STEPS = 8          # decoding steps of a "decode" pass
_SERVE_STEPS = 16   # decoding steps after the prompts of a "serve" pass


def _fuji(size: str, layers: int, vocab: int = 32768, **more) -> dict:
    return dict(_FUJI[size], size=size, layers=layers, vocab=vocab, **more)


def listed() -> list:
    return [
        # A smoke test or a debugging run: everything is small, launches and host work count.
        dict(name="train small", kind="train", hidden=512, heads=4, kv=4, ffn=1536, theta=1e4, layers=2, vocab=4096,
             batch=2, seq=333, remat=False),
        # Grouped-query 1B (32 heads of 64, 8 KV heads) at a sequence length of 2048, activations kept.
        dict(name="train 1B gqa", kind="train", hidden=2048, heads=32, kv=8, ffn=8192, theta=5e5, layers=2, vocab=32768,
             batch=2, seq=2048, remat=False),
        # The headline configuration (7B widths, sequences of 4096, full rematerialisation) cut to two layers.
        dict(name="train 7B", kind="train", hidden=4096, heads=32, kv=32, ffn=11008, theta=1e4, layers=2, vocab=32768,
             batch=2, seq=4096, remat=True),
        # One chat message into a small model, and a batch of full prompts into the 8B widths.
        dict(_fuji("1B-gqa", 4), name="prefill 1B one", kind="prefill", batch=1, prompt=333),
        dict(_fuji("8B", 2), name="prefill 8B batch", kind="prefill", batch=8, prompt=2048),
        # Interactive decoding for one user; a ragged batch on a grouped-query cache; a full batch on a cache with one
        # KV head per query head.
        dict(_fuji("1B", 4), name="decode 1B one", kind="decode", batch=1, prompt=300),
        dict(_fuji("8B", 4), name="decode 8B ragged", kind="decode", batch=16, prompt=2048),
        dict(_fuji("7B", 2), name="decode 7B full", kind="decode", batch=64, prompt=2000),
        # Served batches of the two other designs: one short conversation, and a ragged batch.
        dict(name="serve sagisun one", kind="serve", family="sagisun", size="1B", layers=2, batch=1, prompt=200),
        dict(name="serve sagisun batch", kind="serve", family="sagisun", size="1B", layers=2, batch=8, prompt=1500),
        dict(name="serve zukitar one", kind="serve", family="zukitar", size="1B", layers=3, batch=1, prompt=200),
        dict(name="serve zukitar batch", kind="serve", family="zukitar", size="1B", layers=3, batch=16, prompt=1000),
    ]


def _log_uniform(rng, low: float, high: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng) -> dict:
    kind = rng.choice(["train", "prefill", "decode", "decode", "serve"])
    if kind == "train":
        hidden = rng.choice([512, 1024, 2048])
        heads = hidden // rng.choice([64, 128])
        seq = _log_uniform(rng, 100, 3000)
        return dict(kind=kind, hidden=hidden, heads=heads, kv=heads // rng.choice([1, 2, 4]),
                    ffn=hidden * rng.choice([2, 3, 4]), theta=rng.choice([1e4, 5e5]), layers=rng.choice([1, 2, 3]),
                    vocab=rng.choice([4096, 32768]), batch=_log_uniform(rng, 1, max(1.0, 6000 / seq)), seq=seq,
                    remat=rng.random() < 0.5)
    if kind == "serve":
        prompt = _log_uniform(rng, 40, 1600)
        family = rng.choice(["sagisun", "zukitar"])
        return dict(kind=kind, family=family, size="1B", layers=2 if family == "sagisun" else 3,
                    batch=_log_uniform(rng, 1, max(1.0, min(32.0, 12000 / prompt))), prompt=prompt)
    size = rng.choice(sorted(_FUJI))
    layers = rng.choice([1, 2, 3]) if size in ("7B", "8B") else rng.choice([2, 4, 6])
    if kind == "prefill":
        prompt = _log_uniform(rng, 60, 4000)
        batch = _log_uniform(rng, 1, max(1.0, min(64.0, 15000 / prompt)))
        return dict(_fuji(size, min(layers, 3)), kind=kind, batch=batch, prompt=prompt)
    prompt = _log_uniform(rng, 60, 4000)
    batch = _log_uniform(rng, 1, max(1.0, min(64.0, 60000 / prompt)))
    return dict(_fuji(size, layers), kind=kind, batch=batch, prompt=prompt)


def tolerance(case: dict) -> dict:
    """bf16 operands and activations with 32-bit sums.  Against 64 bits the gradients of a training step were measured to
    be off by 0.014 at most, the logits of prompts and decoding steps by 0.008 (0.003-0.008 for cached keys and values);
    about four times that is stated."""
    return {"rel": 5e-2 if case["kind"] == "train" else 3e-2}


# ------------------------------------------------------------------------------------------
# What a program has in hand before the call.
# ------------------------------------------------------------------------------------------


def _generator(seed: int, salt: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(seed * 1000 + salt)


def _normal(gen, *shape, std: float = 1.0, dtype=torch.bfloat16) -> torch.Tensor:
    return (torch.randn(*shape, device="cuda", generator=gen) * std).to(dtype)


def _token_ids(case: dict, seed: int, *shape) -> torch.Tensor:
    return torch.randint(0, case.get("vocab", 32768), shape, device="cuda", generator=_generator(seed, 7))


def _lengths(case: dict, seed: int) -> torch.Tensor:
    """Prompt lengths of a batch: the longest first, the others between a quarter of it and all of it."""
    b, t = case["batch"], case["prompt"]
    part = 0.25 + 0.75 * torch.rand(b, device="cuda", generator=_generator(seed, 8))
    out = (part * t).to(torch.int32).clamp(min=1)
    out[0] = t
    return out


def _fuji_weights(case: dict, seed: int) -> dict:
    from axlearn_b200.inference.decode_engine import LayerWeights

    gen = _generator(seed, 1)
    d, h, f, v = case["hidden"], 128, case["ffn"], case["vocab"]
    nq, nkv = case["heads"], case["kv"]
    layers = [LayerWeights(
        attn_norm=1 + _normal(gen, d, std=0.1), wqkv=_normal(gen, d, (nq + 2 * nkv) * h, std=d ** -0.5),
        wo=_normal(gen, nq * h, d, std=(nq * h) ** -0.5), ffn_norm=1 + _normal(gen, d, std=0.1),
        wgu=_normal(gen, d, 2 * f, std=d ** -0.5), wdown=_normal(gen, f, d, std=f ** -0.5))
        for _ in range(case["layers"])]
    return {"layers": layers, "emb": _normal(gen, v, d), "head": _normal(gen, v, d, std=d ** -0.5),
            "final_norm": 1 + _normal(gen, d, std=0.1)}


def _fuji_engine(case: dict, seed: int):
    from axlearn_b200.inference.decode_engine import DecodeEngine, FujiDims

    dims = FujiDims(num_layers=case["layers"], hidden_dim=case["hidden"], num_heads=case["heads"],
                    num_kv_heads=case["kv"], head_dim=128, ffn_dim=case["ffn"], vocab_size=case["vocab"],
                    rope_theta=case["theta"])
    return DecodeEngine(_fuji_weights(case, seed), dims, batch=case["batch"], max_len=case["prompt"] + 2 * _STEPS,
                        device="cuda")


def _family(case: dict):
    from axlearn_b200.experiments.text.gpt import sagisun, zukitar

    module = {"sagisun": sagisun, "zukitar": zukitar}[case["family"]]
    config = module.size_config(case["size"])
    config["layers"] = config["layers"][:case["layers"]]
    return module, config


def _checkpoint(case: dict, config: dict, seed: int) -> dict:
    """Random tensors under the names of a checkpoint of the design."""
    gen = _generator(seed, 1)
    d = config["width"]
    out = {"embed": _normal(gen, config["vocab"], d, std=1.0)}
    topics = None
    routers = [layer["mlp"]["router"] for layer in config["layers"] if layer["mlp"]["kind"] == "moe"]
    if routers:
        # A trained router knows its tokens: every token carries the directions of the experts it goes to, so that the
        # choice does not hang on the last bit of a score.
        count, top = routers[0]["experts"], routers[0]["top"]
        topics = _normal(gen, count, d, std=d ** -0.5, dtype=torch.float32)
        chosen = torch.rand(config["vocab"], count, device="cuda", generator=gen).argsort(dim=1)[:, :top]
        member = torch.zeros(config["vocab"], count, device="cuda").scatter_(1, chosen, 14.0)
        out["embed"] = (out["embed"].float() + member @ topics).to(torch.bfloat16)

    def matrix(name, rows, cols):
        out[name] = _normal(gen, rows, cols, std=cols ** -0.5)

    def vector(name, n, mean=0.0, std=0.1):
        out[name] = mean + _normal(gen, n, std=std, dtype=torch.float32)

    one = 0.0 if case["family"] == "sagisun" else 1.0  # Sagisun stores offsets from one
    vector("final.norm", d, one)
    for i, layer in enumerate(config["layers"]):
        pre, m = f"l{i}.", layer["mixer"]
        vector(pre + "norm1", d, one)
        vector(pre + "norm2", d, one)
        if case["family"] == "sagisun":
            n = config["streams"]
            for q in ("hc1.", "hc2."):
                vector(pre + q + "in", n, 1 / n, 0.05)
                vector(pre + q + "out", n, 1.0)
                out[pre + q + "mix"] = torch.eye(n, device="cuda") + _normal(gen, n, n, std=0.05, dtype=torch.float32)
            a, r = m["left"], m["right"]
            left, right = pre + "mix.left.", pre + "mix.right."
            matrix(left + "q", a["heads"] * a["dim"], d)
            matrix(left + "k", a["kv_heads"] * a["dim"], d)
            matrix(left + "v", a["kv_heads"] * a["vdim"], d)
            matrix(left + "g", a["heads"] * a["vdim"], d)
            matrix(left + "o", d, a["heads"] * a["vdim"])
            matrix(right + "q", r["heads"] * r["dim"], d)
            matrix(right + "k", r["heads"] * r["dim"], d)
            matrix(right + "v", r["heads"] * r["vdim"], d)
            matrix(right + "g", r["heads"] * r["vdim"], d)
            matrix(right + "a1", 16, d)
            matrix(right + "a2", r["heads"] * r["dim"], 16)
            vector(right + "a2.b", r["heads"] * r["dim"], 1.0, 0.5)
            vector(right + "norm", r["vdim"], 1.0)
            matrix(right + "o", d, r["heads"] * r["vdim"])
            vector(left + "out", d, 1.0)
            vector(right + "out", d, 1.0)
        elif layer["type"] == "mamba2":
            inner, gn = m["heads"] * m["vdim"], m["groups"] * m["state"]
            mix = pre + "mix."
            matrix(mix + "in", 2 * inner + 2 * gn + m["heads"], d)
            matrix(mix + "conv", inner + 2 * gn, m["conv"])
            vector(mix + "conv.b", inner + 2 * gn)
            vector(mix + "dt_bias", m["heads"], -3.0, 0.5)
            vector(mix + "A_log", m["heads"], 1.0, 0.5)
            vector(mix + "D", m["heads"], 1.0)
            vector(mix + "norm", inner, 1.0)
            matrix(mix + "o", d, inner)
        else:
            mix = pre + "mix."
            matrix(mix + "q", m["heads"] * (m["dim"] + m["rot_dim"]), d)
            matrix(mix + "dkv", m["kv_rank"] + m["rot_dim"], d)
            vector(mix + "dkv.norm", m["kv_rank"], 1.0)
            matrix(mix + "uk", m["heads"] * m["dim"], m["kv_rank"])
            matrix(mix + "uv", m["heads"] * m["vdim"], m["kv_rank"])
            matrix(mix + "o", d, m["heads"] * m["vdim"])
        mlp, pre = layer["mlp"], pre + "mlp."
        if mlp["kind"] == "dense":
            matrix(pre + "gate", mlp["ff"], d)
            matrix(pre + "up", mlp["ff"], d)
            matrix(pre + "down", d, mlp["ff"])
        else:
            out[pre + "router"] = (0.4 * topics).to(torch.bfloat16)
            for e in range(mlp["router"]["experts"]):
                matrix(f"{pre}e{e}.gate", mlp["expert"]["ff"], d)
                matrix(f"{pre}e{e}.up", mlp["expert"]["ff"], d)
                matrix(f"{pre}e{e}.down", d, mlp["expert"]["ff"])
    return out


def _train_state(case: dict, seed: int) -> dict:
    from axlearn_b200.common import prng
    from axlearn_b200.common.base_layer import RematSpec, nothing_saveable
    from axlearn_b200.experiments.text.gpt import fuji
    from axlearn_b200.experiments.text.gpt.common import (
        adamw_decoupled_learner_config,
        get_trainer_config_fn,
        mesh_shape_from_axes,
    )

    model = fuji.model_config(
        num_layers=case["layers"], hidden_dim=case["hidden"], num_heads=case["heads"],
        num_kv_heads=None if case["kv"] == case["heads"] else case["kv"], vocab_size=case["vocab"],
        rope_theta=case["theta"], shared_lm_head=True, ffn_dim=case["ffn"], scan_chunk=8192, flash_attention=True)
    if case["remat"]:
        model.decoder.transformer.layer.remat_spec = RematSpec(prevent_cse=False, policy=nothing_saveable)
    cfg = get_trainer_config_fn(
        model_cfg=model, learner_cfg=adamw_decoupled_learner_config(peak_lr=3e-4, max_step=100_000, weight_decay=0.1),
        max_step=100_000, train_batch_size=case["batch"], max_sequence_length=case["seq"], vocab_size=case["vocab"],
        mesh_shape=mesh_shape_from_axes(), train_dtype=torch.bfloat16)()
    cfg.dir = os.path.join(tempfile.gettempdir(), f"axb200_cases_{os.getpid()}")
    cfg.device = "cuda:0"
    trainer = cfg.instantiate(parent=None)
    trainer.init(prng.PRNGKey(seed % (1 << 31)))
    tokens = torch.randint(0, case["vocab"], (case["batch"], case["seq"] + 1), dtype=torch.int32,
                           generator=torch.Generator().manual_seed(seed))
    batch = {"input_ids": tokens[:, :-1].contiguous().pin_memory(),
             "target_labels": tokens[:, 1:].contiguous().pin_memory(),
             "target_num_bytes": torch.ones(case["batch"], dtype=torch.int32).pin_memory()}
    return dict(kind="train", trainer=trainer, batch=batch)


@torch.no_grad()
def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    if kind == "train":
        with torch.enable_grad():
            return _train_state(case, seed)
    b, t = case["batch"], case["prompt"]
    state = dict(kind=kind, ids=_token_ids(case, seed, b, t))
    if kind == "prefill":
        state["engine"] = _fuji_engine(case, seed)
        return state
    if kind == "decode":
        engine = state["engine"] = _fuji_engine(case, seed)
        state["lengths"] = _lengths(case, seed)
        state["continuation"] = _token_ids(case, seed + 1, b, _STEPS)
        engine.prefill(state["ids"], lengths=state["lengths"])
        engine.step_logits(state["continuation"][:, 0])  # the captured step: once per engine
        return state
    from axlearn_b200.inference.decode_engine import ModuleDecodeEngine

    module, config = _family(case)
    model = module.model_config(config).set(name="model", dtype=torch.bfloat16).instantiate(parent=None)
    params = module.parameters(model, _checkpoint(case, config, seed), dtype=torch.bfloat16, device="cuda")
    engine = state["engine"] = ModuleDecodeEngine(model.decoder, params["decoder"], batch=b,
                                                  max_len=t + 2 * _SERVE_STEPS, device="cuda")
    state["lengths"] = _lengths(case, seed)
    state["continuation"] = _token_ids(case, seed + 1, b, _SERVE_STEPS)
    engine.prefill(state["ids"], lengths=state["lengths"])
    engine.step_logits(state["continuation"][:, 0])
    return state


# ------------------------------------------------------------------------------------------
# One pass.
# ------------------------------------------------------------------------------------------


def run(state: dict):
    kind = state["kind"]
    if kind == "train":
        # One optimisation step from a pinned host batch; gradients show in the first moments.
        trainer = state["trainer"]
        loss = trainer.train_step(state["batch"])["loss"]
        now = trainer.trainer_state
        return {"loss": loss, "first_moments": _leaves(now["learner"]["optimizer"][1][0].mu),
                "weights": _leaves(now["model"])}
    engine = state["engine"]
    if kind == "prefill":
        first = engine.prefill(state["ids"])
        return {"first": first, "logits": engine.logits, "keys": engine.k_pools, "values": engine.v_pools}
    out = {}
    if kind == "serve":
        engine.prefill(state["ids"], lengths=state["lengths"])
        out["prompt_logits"] = engine.logits.clone()
    else:
        # Another continuation of the same prompts: back to their ends, then token by token.
        engine.lengths.copy_(state["lengths"])
    tokens = state["continuation"]
    out["logits"] = [engine.step_logits(tokens[:, i]).clone() for i in range(tokens.shape[1])]
    return out


def _leaves(tree) -> dict:
    out = {}

    def visit(node, path):
        if isinstance(node, dict):
            for key in node:
                visit(node[key], f"{path}/{key}" if path else str(key))
        else:
            out[path] = node

    visit(tree, "")
    return out


# ------------------------------------------------------------------------------------------
# What a pass cannot do without.
# ------------------------------------------------------------------------------------------


def _layer_params(case: dict, head: int) -> int:
    d = case["hidden"]
    return d * (2 * case["heads"] + 2 * case["kv"]) * head + 3 * d * case["ffn"]


def _mean_length(case: dict) -> float:
    """Expected prompt length of a ragged batch (one row of full length, the others at 5/8 of it on average)."""
    return case["prompt"] * (1 + 0.625 * (case["batch"] - 1)) / case["batch"]


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "train":
        head = case["hidden"] // case["heads"]
        tokens, table = case["batch"] * case["seq"], case["vocab"] * case["hidden"]
        params = case["layers"] * _layer_params(case, head) + table
        # Masters and both moments are read and written, the bf16 weights written; tokens read.
        return {"bytes": params * (3 * 8 + 2) + tokens * 8,
                "flops": 6.0 * tokens * params + 6.0 * case["layers"] * tokens * case["seq"] * case["hidden"]}
    b, t = case["batch"], case["prompt"]
    if kind == "serve":
        return _serve_work(case)
    params = case["layers"] * _layer_params(case, 128)
    table = case["vocab"] * case["hidden"]
    kv_row = case["layers"] * 2 * case["kv"] * 128
    if kind == "prefill":
        return {"bytes": 2 * (params + table + b * t * (case["hidden"] + kv_row)) + 4 * b * case["vocab"],
                "flops": 2.0 * b * t * params + 2.0 * b * table
                + 2.0 * case["layers"] * b * t * t * case["heads"] * 128}
    context = b * (_mean_length(case) + _STEPS / 2)
    step_bytes = 2 * (params + table + context * kv_row) + 4 * b * case["vocab"]
    step_flops = 2.0 * b * (params + table) + 4.0 * case["layers"] * context * case["heads"] * 128
    return {"bytes": _STEPS * step_bytes, "flops": _STEPS * step_flops}


def _serve_work(case: dict) -> dict:
    _, config = _family(case)
    b, d = case["batch"], config["width"]
    rows = b * _mean_length(case)
    table = config["vocab"] * d
    flops = 2.0 * b * table * (1 + _SERVE_STEPS)
    prompt_bytes = step_bytes = 2.0 * table + 4.0 * b * config["vocab"]
    seen = case["prompt"] * 0.7
    for layer in config["layers"]:
        m, mlp = layer["mixer"], layer["mlp"]
        if case["family"] == "sagisun":
            a, r = m["left"], m["right"]
            dense = d * (3 * a["heads"] * a["dim"] + 2 * a["kv_heads"] * a["dim"]
                         + r["heads"] * (2 * r["dim"] + 3 * r["vdim"]) + 16) + 16 * r["heads"] * r["dim"]
            window = min(seen, a["mask"]["size"])
            pair = 4.0 * a["heads"] * a["dim"] * window / 2
            token = pair + 6.0 * r["heads"] * r["dim"] * r["vdim"]
            state = 2.0 * 4 * r["heads"] * r["dim"] * r["vdim"] + 4.0 * window * a["kv_heads"] * a["dim"]
        elif layer["type"] == "mamba2":
            inner, gn = m["heads"] * m["vdim"], m["groups"] * m["state"]
            dense = d * (3 * inner + 2 * gn + m["heads"])
            token = 6.0 * inner * m["state"]
            state = 2.0 * 4 * inner * m["state"]
        else:
            dense = (d * (m["heads"] * (m["dim"] + m["rot_dim"]) + m["kv_rank"] + m["rot_dim"] + m["heads"] * m["vdim"])
                     + m["kv_rank"] * m["heads"] * (m["dim"] + m["vdim"]))
            token = m["heads"] * (2.0 * (m["dim"] + m["rot_dim"]) + 2.0 * m["vdim"]) * seen / 2
            state = 2.0 * seen * (m["kv_rank"] + m["rot_dim"])
        if mlp["kind"] == "dense":
            used, read = 3 * d * mlp["ff"], 3 * d * mlp["ff"]
            step_read = read
        else:
            experts, top, one = mlp["router"]["experts"], mlp["router"]["top"], 3 * d * mlp["expert"]["ff"]
            used = top * one + d * experts
            read = one * experts * (1 - (1 - top / experts) ** rows)
            step_read = one * experts * (1 - (1 - top / experts) ** b)
        flops += (rows + b * _SERVE_STEPS) * (2.0 * (dense + used) + token)
        prompt_bytes += 2.0 * (dense + read) + b * state / 2
        step_bytes += 2.0 * (dense + step_read) + b * state
    return {"bytes": prompt_bytes + 2.0 * rows * d + _SERVE_STEPS * step_bytes, "flops": flops}


# ------------------------------------------------------------------------------------------
# The outputs in 64 bits, without this repository's kernels.
# ------------------------------------------------------------------------------------------


def _d(t: torch.Tensor) -> torch.Tensor:
    return t.double()


def _rms64(x, eps):
    return x * torch.rsqrt((x * x).mean(dim=-1, keepdim=True) + eps)


def _rope64(x, theta, dims=None):
    """``x [B, T, N, H]``: pairs (2i, 2i + 1) of the first ``dims`` entries turn by ``position * theta^(-2i / dims)``."""
    dims = x.shape[-1] if dims is None else dims
    freq = theta ** (-torch.arange(0, dims, 2, device=x.device, dtype=torch.float64) / dims)
    angle = torch.arange(x.shape[1], device=x.device, dtype=torch.float64)[:, None] * freq
    c, s = angle.cos()[:, None], angle.sin()[:, None]
    u, v = x[..., 0:dims:2], x[..., 1:dims:2]
    turned = torch.stack([u * c - v * s, v * c + u * s], dim=-1).flatten(-2)
    return torch.cat([turned, x[..., dims:]], dim=-1)


def _attention64(q, k, v, scale, bias=None):
    """``q [B, T, N, H]``, ``k, v [B, T, G, ...]``; ``bias(head) [T, T]`` or None for the causal mask; head by head."""
    b, t, n, _ = q.shape
    group = n // k.shape[2]
    mask = None if bias is not None else torch.full((t, t), -math.inf, device=q.device, dtype=q.dtype).triu(1)
    outs = []
    for head in range(n):
        s = torch.einsum("bth,bsh->bts", q[:, :, head], k[:, :, head // group]) * scale
        p = torch.softmax(s + (mask if bias is None else bias(head)), dim=-1)
        outs.append(torch.einsum("bts,bsv->btv", p, v[:, :, head // group]))
    return torch.stack(outs, dim=2)


def _fuji_layer64(x, w, *, heads, kv, head, theta, eps=1e-5):
    b, t, _ = x.shape
    qkv = ((_rms64(x, eps) * w["attn_norm"]) @ w["wqkv"]).reshape(b, t, heads + 2 * kv, head)
    q, k, v = _rope64(qkv[:, :, :heads], theta), _rope64(qkv[:, :, heads:heads + kv], theta), qkv[:, :, heads + kv:]
    x = x + _attention64(q, k, v, head ** -0.5).reshape(b, t, -1) @ w["wo"]
    gate, up = ((_rms64(x, eps) * w["ffn_norm"]) @ w["wgu"]).chunk(2, dim=-1)
    return x + (torch.nn.functional.silu(gate) * up) @ w["wdown"], k, v


def _sequences(case: dict, state_ids, lengths, continuation):
    """Each row's prompt with its continuation behind it, right-padded with token 0."""
    b, t = state_ids.shape
    steps = continuation.shape[1]
    ids = torch.zeros(b, t + steps, dtype=torch.int64, device="cuda")
    ids[:, :t] = state_ids
    at = lengths.long()[:, None] + torch.arange(steps, device="cuda")
    return ids.scatter(1, at, continuation), at


@torch.no_grad()
def _fuji_exact(case: dict, seed: int):
    w = _fuji_weights(case, seed)
    b, t = case["batch"], case["prompt"]
    ids, lengths = _token_ids(case, seed, b, t), None
    if case["kind"] == "decode":
        lengths = _lengths(case, seed)
        ids, at = _sequences(case, ids, lengths, _token_ids(case, seed + 1, b, _STEPS))
    last, caches = [], [([], []) for _ in w["layers"]]
    rows = max(1, 16384 // ids.shape[1])
    for b0 in range(0, b, rows):
        x = _d(w["emb"][ids[b0:b0 + rows]])
        for i, layer in enumerate(w["layers"]):
            x, k, v = _fuji_layer64(x, {n: _d(p) for n, p in vars(layer).items()}, heads=case["heads"], kv=case["kv"],
                                    head=128, theta=case["theta"])
            if lengths is None:
                for parts, new in zip(caches[i], (k, v)):
                    parts.append(new)
        last.append(x[:, -1:] if lengths is None else torch.stack([r[a] for r, a in zip(x, at[b0:b0 + rows])]))
    hidden = torch.cat(last)
    logits = (_rms64(hidden, 1e-5) * _d(w["final_norm"])) @ _d(w["head"]).t()
    if lengths is not None:
        return {"logits": list(logits.unbind(1))}
    max_len = -(-(t + 2 * _STEPS) // 16) * 16

    def pool(parts):
        whole = torch.zeros(b, max_len, case["kv"], 128, dtype=torch.float64, device="cuda")
        whole[:, :t] = torch.cat(parts)
        return whole.reshape(b * max_len // 16, 16, case["kv"], 128)

    return {"first": None, "logits": logits[:, 0], "keys": [pool(k) for k, _ in caches],
            "values": [pool(v) for _, v in caches]}


def _train_exact(case: dict, seed: int):
    from torch.utils.checkpoint import checkpoint

    state = _train_state(case, seed)
    masters = {k: v.detach().clone() for k, v in _leaves(state["trainer"].trainer_state["model"]).items()}
    ids, labels = state["batch"]["input_ids"].cuda().long(), state["batch"]["target_labels"].cuda().long()
    del state
    # The model reads the weights in bf16.
    w = {k: _d(v.to(torch.bfloat16)).requires_grad_() for k, v in masters.items()}
    pre = "decoder/transformer/repeat/layer/"
    heads, kv, d = case["heads"], case["kv"], case["hidden"]
    head = d // heads

    def weights(i):
        qkv = w[pre + "self_attention/attention/i_proj/i_proj/qkv_proj/weight"][i]
        qkv = torch.cat(list(qkv), dim=1) if qkv.dim() == 4 else qkv      # [3, D, N, H] or [D, N + 2 Nkv, H]
        up = [w[pre + f"feed_forward/linear1_{j}/weight"][i] for j in (0, 1)]
        return {"wqkv": qkv.reshape(d, -1), "attn_norm": w[pre + "self_attention/norm/scale"][i],
                "wo": w[pre + "self_attention/attention/o_proj/weight"][i].reshape(d, -1).t(),
                "ffn_norm": w[pre + "feed_forward/norm/scale"][i], "wgu": torch.cat(up, dim=1),
                "wdown": w[pre + "feed_forward/linear2/weight"][i]}

    def layer(x, i):
        return _fuji_layer64(x, weights(i), heads=heads, kv=kv, head=head, theta=case["theta"])[0]

    table = w["decoder/emb/token_emb/weight"]
    x = table[ids]
    for i in range(case["layers"]):
        x = checkpoint(layer, x, i, use_reentrant=False)
    x = (_rms64(x, 1e-5) * w["decoder/output_norm/scale"]).reshape(-1, d)
    loss = 0.0
    for h, y in zip(x.split(2048), labels.reshape(-1).split(2048)):
        loss = loss + checkpoint(lambda a, c: torch.nn.functional.cross_entropy(a @ table.t(), c, reduction="sum"), h, y,
                                 use_reentrant=False)
    loss = loss / labels.numel()
    loss.backward()
    # Clip to a global norm of 1, first AdamW step, both learning rate and decay scaled by 1 / 2000 (the warm-up).
    norm = math.sqrt(sum(float((v.grad ** 2).sum()) for v in w.values()))
    moments, updated = {}, {}
    for k, v in w.items():
        g = v.grad * min(1.0, 1.0 / norm)
        moments[k] = 0.1 * g
        updated[k] = _d(masters[k]) - (3e-4 * g / (g.abs() + 1e-8) + 0.1 * _d(masters[k])) / 2000
    return {"loss": loss.detach(), "first_moments": moments, "weights": updated}


def _window64(h, w, m):
    b, t, _ = h.shape
    heads, groups, dim, vdim = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    temp, pos = m["q_temp"], torch.arange(t, device=h.device)
    q = (h @ w["q"].t()).reshape(b, t, heads, dim)
    q = q * (1 + temp["coef"] * torch.log(((pos + 1) // temp["every"] + 1).double()))[:, None, None]
    k = (h @ w["k"].t()).reshape(b, t, groups, dim)
    v = (h @ w["v"].t()).reshape(b, t, groups, vdim)
    dist = (pos[:, None] - pos[None]).double()
    hidden = (dist < 0) | (dist >= m["mask"]["size"])
    o = _attention64(q, k, v, m["scale"],
                     lambda n: (-(2.0 ** (-8.0 * (n + 1) / heads)) * dist).masked_fill(hidden, -math.inf))
    return (o.reshape(b, t, -1) * torch.sigmoid(h @ w["g"].t())) @ w["o"].t()


def _linear_attention64(h, w, m, eps):
    b, t, _ = h.shape
    heads, dim, vdim = m["heads"], m["dim"], m["vdim"]
    q = (h @ w["q"].t()).reshape(b, t, heads, dim) * dim ** -0.5
    k = (h @ w["k"].t()).reshape(b, t, heads, dim)
    v = (h @ w["v"].t()).reshape(b, t, heads, vdim)
    z = (h @ w["a1"].t()) @ w["a2"].t() + w["a2.b"]
    decay = torch.exp(torch.nn.functional.logsigmoid(z) / m["tau"]).reshape(b, t, heads, dim)
    s = torch.zeros(b, heads, dim, vdim, dtype=h.dtype, device=h.device)
    out = []
    for i in range(t):
        s = decay[:, i, :, :, None] * s + k[:, i, :, :, None] * v[:, i, :, None, :]
        out.append(torch.einsum("bhd,bhdv->bhv", q[:, i], s))
    o = (_rms64(torch.stack(out, dim=1), eps) * w["norm"]).reshape(b, t, -1)
    return (o * torch.nn.functional.silu(h @ w["g"].t())) @ w["o"].t()


def _sagisun64(config, w, ids):
    eps, n = config["norm"]["eps"], config["streams"]
    streams = [w("embed")[ids]] * n
    for i, layer in enumerate(config["layers"]):
        for q in (1, 2):
            pre = f"l{i}.hc{q}."
            u = sum(w(pre + "in")[s] * streams[s] for s in range(n))
            u = _rms64(u, eps) * (1 + w(f"l{i}.norm{q}"))
            if q == 1:
                m = layer["mixer"]
                left = _window64(u, w.part(f"l{i}.mix.left."), m["left"])
                right = _linear_attention64(u, w.part(f"l{i}.mix.right."), m["right"], eps)
                y = 0.5 * (_rms64(left, eps) * w(f"l{i}.mix.left.out") + _rms64(right, eps) * w(f"l{i}.mix.right.out"))
            else:
                p = w.part(f"l{i}.mlp.")
                y = (torch.nn.functional.silu(u @ p["gate"].t()) * (u @ p["up"].t())) @ p["down"].t()
            mix, write = w(pre + "mix"), w(pre + "out") * config["residual_mult"]
            streams = [sum(mix[s, to] * streams[s] for s in range(n)) + write[to] * y for to in range(n)]
    return _rms64(sum(streams), eps) * (1 + w("final.norm"))


def _mamba64(h, w, m, eps):
    b, t, _ = h.shape
    heads, p, n, groups = m["heads"], m["vdim"], m["state"], m["groups"]
    inner, taps = heads * p, m["conv"]
    z, xbc, dt = (h @ w["in"].t()).split([inner, inner + 2 * groups * n, heads], dim=-1)
    before = torch.nn.functional.pad(xbc, (0, 0, taps - 1, 0))
    xbc = torch.nn.functional.silu(w["conv.b"] + sum(w["conv"][:, j] * before[:, j:j + t] for j in range(taps)))
    x, bb, cc = xbc.split([inner, groups * n, groups * n], dim=-1)
    x = x.reshape(b, t, heads, p)
    bb = bb.reshape(b, t, groups, n).repeat_interleave(heads // groups, dim=2)
    cc = cc.reshape(b, t, groups, n).repeat_interleave(heads // groups, dim=2)
    dt = torch.nn.functional.softplus(dt + w["dt_bias"])
    decay = torch.exp(-torch.exp(w["A_log"]) * dt)
    s = torch.zeros(b, heads, n, p, dtype=h.dtype, device=h.device)
    out = []
    for i in range(t):
        s = decay[:, i, :, None, None] * s + (dt[:, i, :, None] * bb[:, i])[..., None] * x[:, i, :, None, :]
        out.append(torch.einsum("bhn,bhnp->bhp", cc[:, i], s))
    y = torch.stack(out, dim=1) + w["D"][:, None] * x
    v = (y.reshape(b, t, inner) * torch.nn.functional.silu(z)).reshape(b, t, m["norm_groups"], -1)
    return (_rms64(v, eps).reshape(b, t, inner) * w["norm"]) @ w["o"].t()


def _latent64(h, w, m, eps):
    b, t, _ = h.shape
    heads, dim, rdim, rank, rot = m["heads"], m["dim"], m["rot_dim"], m["kv_rank"], m["rot"]
    q = (h @ w["q"].t()).reshape(b, t, heads, dim + rdim)
    q = torch.cat([q[..., :dim], _rope64(q[..., dim:], rot["base"], rot["dims"])], dim=-1)
    both = h @ w["dkv"].t()
    c = _rms64(both[..., :rank], eps) * w["dkv.norm"]
    shared = _rope64(both[..., None, rank:], rot["base"], rot["dims"]).expand(b, t, heads, rdim)
    k = torch.cat([(c @ w["uk"].t()).reshape(b, t, heads, dim), shared], dim=-1)
    v = (c @ w["uv"].t()).reshape(b, t, heads, m["vdim"])
    return _attention64(q, k, v, m["scale"]).reshape(b, t, -1) @ w["o"].t()


def _experts64(h, w, mlp):
    x = h.reshape(-1, h.shape[-1])
    scores, ids = torch.sigmoid(x @ w["router"].t()).topk(mlp["router"]["top"], dim=-1)
    out, limit = torch.zeros_like(x), mlp["expert"]["limit"]
    for e in range(mlp["router"]["experts"]):
        row, choice = torch.nonzero(ids == e, as_tuple=True)
        u = x[row] * scores[row, choice][:, None]
        gate = (u @ w[f"e{e}.gate"].t()).clamp(max=limit)
        up = (u @ w[f"e{e}.up"].t()).clamp(-limit, limit)
        out.index_add_(0, row, (gate * torch.sigmoid(1.702 * gate) * (up + 1)) @ w[f"e{e}.down"].t())
    return out.reshape(h.shape)


def _zukitar64(config, w, ids):
    eps = config["norm"]["eps"]
    x = w("embed")[ids]
    for i, layer in enumerate(config["layers"]):
        mix = {"latent_attention": _latent64, "mamba2": _mamba64}[layer["type"]]
        x = x + mix(_rms64(x, eps) * w(f"l{i}.norm1"), w.part(f"l{i}.mix."), layer["mixer"], eps)
        h, p = _rms64(x, eps) * w(f"l{i}.norm2"), w.part(f"l{i}.mlp.")
        if layer["mlp"]["kind"] == "dense":
            gate = torch.nn.functional.gelu(h @ p["gate"].t(), approximate="tanh")
            x = x + (gate * (h @ p["up"].t())) @ p["down"].t()
        else:
            x = x + _experts64(h, p, layer["mlp"])
    return _rms64(x, eps) * w("final.norm") * config["logit_scale"]


class _Weights64:
    """A checkpoint's tensors in 64 bits, one at a time or by prefix."""

    def __init__(self, tensors: dict):
        self._tensors = tensors

    def __call__(self, name: str) -> torch.Tensor:
        return _d(self._tensors[name])

    def part(self, prefix: str) -> dict:
        return {k[len(prefix):]: _d(v) for k, v in self._tensors.items() if k.startswith(prefix)}


@torch.no_grad()
def _serve_exact(case: dict, seed: int):
    _, config = _family(case)
    tensors = _checkpoint(case, config, seed)
    lengths = _lengths(case, seed)
    ids, at = _sequences(case, _token_ids(case, seed, case["batch"], case["prompt"]), lengths,
                         _token_ids(case, seed + 1, case["batch"], _SERVE_STEPS))
    at = torch.cat([at[:, :1] - 1, at], dim=1)
    forward = {"sagisun": _sagisun64, "zukitar": _zukitar64}[case["family"]]
    hidden = []
    rows = max(1, 8192 // ids.shape[1])
    for b0 in range(0, case["batch"], rows):
        x = forward(config, _Weights64(tensors), ids[b0:b0 + rows])
        hidden.append(torch.stack([r[a] for r, a in zip(x, at[b0:b0 + rows])]))
    logits = torch.cat(hidden) @ _d(tensors["embed"]).t()
    return {"prompt_logits": logits[:, 0], "logits": list(logits[:, 1:].unbind(1))}


def exact(case: dict, seed: int):
    if case["kind"] == "train":
        return _train_exact(case, seed)
    return _serve_exact(case, seed) if case["kind"] == "serve" else _fuji_exact(case, seed)
