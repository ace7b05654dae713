"""Captured training steps against steps run one launch after the other."""

import pytest
import torch

from axlearn_b200.common import prng
from axlearn_b200.common.base_layer import RematSpec, nothing_saveable
from axlearn_b200.common.utils import flatten_items
from axlearn_b200.experiments.text.gpt import fuji
from axlearn_b200.experiments.text.gpt.common import (
    adamw_decoupled_learner_config,
    get_trainer_config_fn,
    mesh_shape_from_axes,
)

pytestmark = pytest.mark.gpu
_VOCAB = 512


def _trainer(tmp_path, *, kv=None, remat=False, seed=0):
    model = fuji.model_config(num_layers=2, hidden_dim=256, num_heads=4, num_kv_heads=kv, vocab_size=_VOCAB, rope_theta=1e4,
                              shared_lm_head=True, ffn_dim=512, scan_chunk=1024, flash_attention=True)
    if remat:
        model.decoder.transformer.layer.remat_spec = RematSpec(prevent_cse=False, policy=nothing_saveable)
    learner = adamw_decoupled_learner_config(peak_lr=1e-2, max_step=1000, weight_decay=0.1, lr_warmup_steps=4)
    cfg = get_trainer_config_fn(
        model_cfg=model, learner_cfg=learner, max_step=1000, train_batch_size=2, max_sequence_length=128,
        vocab_size=_VOCAB, mesh_shape=mesh_shape_from_axes(), train_dtype=torch.bfloat16)()
    cfg.dir, cfg.device = str(tmp_path), "cuda:0"
    trainer = cfg.instantiate(parent=None)
    trainer.init(prng.PRNGKey(seed))
    return trainer


def _batch(seed, rows=2, length=128):
    tokens = torch.randint(0, _VOCAB, (rows, length + 1), dtype=torch.int32, generator=torch.Generator().manual_seed(seed))
    return {"input_ids": tokens[:, :-1].contiguous(), "target_labels": tokens[:, 1:].contiguous(),
            "target_num_bytes": torch.ones(rows, dtype=torch.int32)}


def _captured(trainer) -> bool:
    return trainer._step_graphs._captured is not None  # pylint: disable=protected-access


def _eager(trainer):
    trainer._step_graphs._capturable = False  # pylint: disable=protected-access
    return trainer


def _same(a, b, rel):
    """Both trainers' parameters, moments and shadows: off by the order of sums in the gradients at most."""
    for pick in (lambda t: t.trainer_state["model"], lambda t: t.trainer_state["learner"]["optimizer"][1][0].mu,
                 lambda t: t.trainer_state["learner"]["optimizer"][1][0].nu, lambda t: t._shadows):
        for (path, x), (_, y) in zip(flatten_items(pick(a)), flatten_items(pick(b))):
            x, y = x.detach().double(), y.detach().double()
            assert (x - y).norm() <= rel * y.norm() + 1e-12, path


@pytest.mark.parametrize("kv,remat", [(None, True), (2, False)])
def test_captured_steps_are_the_steps(tmp_path, kv, remat):
    from axlearn_b200.ops import cuda_ops

    a, b = _trainer(tmp_path, kv=kv, remat=remat), _eager(_trainer(tmp_path, kv=kv, remat=remat))
    kept = []
    for step in range(6):
        before = cuda_ops.launch_count
        x = a.train_step(_batch(step))
        middle = cuda_ops.launch_count
        y = b.train_step(_batch(step))
        launches = cuda_ops.launch_count - middle
        assert _captured(a) == (step >= 1) and not _captured(b)
        # As many kernels, plus the one that stores the scalars in a replay.
        assert middle - before == launches + (1 if step >= 1 else 0)
        kept.append((x, y))
    for x, y in kept:  # outputs of earlier steps are not those of later ones
        torch.testing.assert_close(x["loss"], y["loss"], rtol=2e-3, atol=0)
        assert list(x["summaries"]) == list(y["summaries"])
        for part in x["summaries"]:
            assert list(x["summaries"][part]) == list(y["summaries"][part])
        for name in ("lr/schedule_scale", "lr/schedule_step", "update/schedule_scale", "update/schedule_step"):
            assert x["summaries"]["learner"][name] == y["summaries"]["learner"][name]
        torch.testing.assert_close(x["summaries"]["learner"]["gradient_norm"],
                                   y["summaries"]["learner"]["gradient_norm"], rtol=2e-2, atol=0)
    assert len({float(x["loss"]) for x, _ in kept}) == len(kept)
    _same(a, b, 2e-2)
    for (_, x), (_, y) in zip(flatten_items(a.trainer_state["learner"]), flatten_items(b.trainer_state["learner"])):
        if isinstance(x, torch.Tensor) and x.dim() == 0:
            assert torch.equal(x, y)
    assert torch.equal(a.trainer_state["prng_key"], b.trainer_state["prng_key"])
    cuda_ops.check_status()


def test_captured_steps_share_no_scratch(tmp_path):
    """Tables of rotations are a graph's own: later, larger calls on the capture's stream and steps of another trainer whose
    capture got the same stream do not touch them."""
    from axlearn_b200.ops import cuda_ops

    a, b = _trainer(tmp_path), _eager(_trainer(tmp_path))
    a.train_step(_batch(0)), b.train_step(_batch(0))
    tables = dict(cuda_ops._rope_tables)  # pylint: disable=protected-access
    streams, plain = [], torch.cuda.Stream

    def stream(*args, **kwargs):
        streams.append(plain(*args, **kwargs))
        return streams[-1]

    torch.cuda.Stream = stream
    try:
        a.train_step(_batch(1))
    finally:
        torch.cuda.Stream = plain
    b.train_step(_batch(1))
    assert _captured(a) and streams
    assert {k: t.data_ptr() for k, t in cuda_ops._rope_tables.items()} == {k: t.data_ptr() for k, t in tables.items()}  # pylint: disable=protected-access
    positions = torch.arange(40_000, device="cuda")[None]
    x = torch.randn(1, 40_000, 1, 64, device="cuda").bfloat16()
    with torch.cuda.stream(streams[-1]):
        cuda_ops.rope(x, positions, 1e4)
    torch.cuda.synchronize()
    for step in range(2, 5):
        x, y = a.train_step(_batch(step)), b.train_step(_batch(step))
        torch.testing.assert_close(x["loss"], y["loss"], rtol=2e-3, atol=0)
    _same(a, b, 2e-2)


def test_other_shapes_hooks_and_states(tmp_path):
    a, b = _trainer(tmp_path), _eager(_trainer(tmp_path))

    def both(batch):
        x, y = a.train_step(batch), b.train_step(batch)
        torch.testing.assert_close(x["loss"], y["loss"], rtol=2e-3, atol=0)

    for step in range(3):
        both(_batch(step))
    assert _captured(a)
    graph = a._step_graphs._captured
    for step, shape in enumerate([(1, 128), (2, 100), (2, 128), (2, 128)]):  # one of each: not captured
        both(_batch(10 + step, *shape))
        assert a._step_graphs._captured is graph
    # A hook on a parameter runs, and the step with it.
    seen = []
    leaf = next(t for _, t in flatten_items(a._shadows) if t.requires_grad and t.dim() == 1)
    handle = leaf.register_hook(lambda g: seen.append(g.shape))
    both(_batch(20))
    assert seen == [leaf.shape]
    handle.remove()
    with torch.autograd.graph.saved_tensors_hooks(lambda t: (seen.append(0), t)[1], lambda t: t):
        both(_batch(21))
    assert len(seen) > 2
    both(_batch(22))
    _same(a, b, 3e-2)
    # New parameters in the trainer: not those of the graph.
    for t in (a, b):
        t.init(prng.PRNGKey(7))
    assert not _captured(a)
    for step in range(3):
        both(_batch(30 + step))
    assert _captured(a) and a._step_graphs._captured is not graph
    _same(a, b, 2e-2)


def test_not_captured(tmp_path, monkeypatch):
    """Dropout, a subclass of a layer, too much memory."""
    from axlearn_b200.common import layers, step_graph

    a = _trainer(tmp_path)
    assert step_graph.capturable(a)
    a.model.decoder.output_dropout._config.rate = 0.1  # pylint: disable=protected-access
    assert not step_graph.capturable(a)
    b = _trainer(tmp_path)
    b.model.decoder.output_norm.__class__ = type("Norm", (layers.RMSNorm,), {})
    assert not step_graph.capturable(b)
    monkeypatch.setattr(step_graph, "_MEMORY_SHARE", 1 << 40)
    c = _trainer(tmp_path)
    d = _eager(_trainer(tmp_path))
    for step in range(3):
        torch.testing.assert_close(c.train_step(_batch(step))["loss"], d.train_step(_batch(step))["loss"], rtol=2e-3, atol=0)
        assert not _captured(c)
    _same(c, d, 2e-2)


def test_gradients_beyond_the_bound_are_not_allocated_twice(tmp_path, monkeypatch):
    """A model whose gradients do not fit the bound is not captured to find that out."""
    from axlearn_b200.common import step_graph

    tried = []
    plain = step_graph._capture
    monkeypatch.setattr(step_graph, "_capture", lambda *args: (tried.append(0), plain(*args))[1])
    a = _trainer(tmp_path)
    held = step_graph._gradient_bytes(a)
    assert held == sum(2 * t.numel() for _, t in flatten_items(a._shadows))
    monkeypatch.setattr(step_graph, "_most_memory", lambda device: held - 1)
    for step in range(3):
        a.train_step(_batch(step))
    assert not tried and not _captured(a)
    monkeypatch.setattr(step_graph, "_most_memory", lambda device: 1 << 30)
    a.train_step(_batch(3))
    assert tried and _captured(a)


def test_a_capture_that_fails_is_tried_again(tmp_path, monkeypatch):
    import gc

    from axlearn_b200.common import step_graph

    monkeypatch.setattr(step_graph, "_PAUSES", (2, 3))
    a, b = _trainer(tmp_path), _eager(_trainer(tmp_path))
    failures, collects = [], []
    plain, update = step_graph._capture, a._apply_update

    def capture(*args):
        if len(failures) < 2:
            failures.append(0)
            raise RuntimeError("out of memory")
        return plain(*args)

    def apply_update(*args):
        collects.append(gc.isenabled())
        return update(*args)

    monkeypatch.setattr(step_graph, "_capture", capture)
    a._apply_update = apply_update
    seen = []
    for step in range(10):
        x, y = a.train_step(_batch(step)), b.train_step(_batch(step))
        torch.testing.assert_close(x["loss"], y["loss"], rtol=2e-3, atol=0)
        seen.append((len(failures), _captured(a)))
    # Steps 1 and 4 fail, 8 succeeds.
    assert seen == [(0, False)] + [(1, False)] * 3 + [(2, False)] * 4 + [(2, True)] * 2
    assert collects == [True] * 8 + [False] and gc.isenabled()
    _same(a, b, 3e-2)
    # What will not pass is not tried again, other parameters are.
    c = _trainer(tmp_path)
    monkeypatch.setattr(step_graph, "_capture", lambda *args: (failures.append(0), (_ for _ in ()).throw(step_graph.Refused("no")))[1])
    for step in range(6):
        c.train_step(_batch(step))
    assert len(failures) == 3
    for _ in range(6):
        a.init(prng.PRNGKey(1))
        assert a._step_graphs._captures == 0


@pytest.mark.parametrize("error", ["Refused", "RuntimeError"])
def test_a_capture_given_up_is_tried_for_other_parameters(tmp_path, monkeypatch, error):
    from axlearn_b200.common import step_graph

    monkeypatch.setattr(step_graph, "_PAUSES", ())
    a, plain = _trainer(tmp_path), step_graph._capture
    kind = step_graph.Refused if error == "Refused" else RuntimeError

    def fail(*args):
        raise kind("no memory today")

    monkeypatch.setattr(step_graph, "_capture", fail)
    for step in range(3):
        a.train_step(_batch(step))
    monkeypatch.setattr(step_graph, "_capture", plain)
    a.train_step(_batch(3))
    assert not _captured(a)
    a.init(prng.PRNGKey(1))
    for step in range(2):
        a.train_step(_batch(step))
    assert _captured(a)


def test_settings_changed_after_the_capture(tmp_path):
    """A rate, a constant of a norm, a weight of the loss, a list changed in place, a method of its own: as step by step."""
    a, b = _trainer(tmp_path), _eager(_trainer(tmp_path))

    def both(step, captured):
        x, y = a.train_step(_batch(step)), b.train_step(_batch(step))
        torch.testing.assert_close(x["loss"], y["loss"], rtol=2e-3, atol=0)
        assert _captured(a) == captured
        return float(x["loss"])

    def change(fn):
        fn(a), fn(b)

    for step in range(3):
        both(step, step >= 1)
    change(lambda t: setattr(t.model.decoder.output_norm._config, "eps", 3.0))
    before = both(3, False)
    assert abs(both(4, True) - before) < 2
    graph = a._step_graphs._captured
    change(lambda t: t.learner._config.update_rules.append((".*never.*", None)))
    both(5, False)
    both(6, True)
    assert a._step_graphs._captured is not graph
    a.model.decoder.output_dropout._config.rate = 0.5
    losses = [float(a.train_step(_batch(7))["loss"]) for _ in range(2)]
    assert not _captured(a) and losses[0] != losses[1]
    a.model.decoder.output_dropout._config.rate = 0.0
    a.train_step(_batch(8)), a.train_step(_batch(8))
    assert _captured(a)
    calls = []
    plain = a.model.forward
    a.model.forward = lambda *args, **kwargs: (calls.append(0), plain(*args, **kwargs))[1]
    a.train_step(_batch(9))
    assert not _captured(a) and calls


def test_layers_are_looked_over_in_place(tmp_path, monkeypatch):
    """What decides about a capture copies no configuration and asks for no field that is not there (either took longer than
    half a small step)."""
    from axlearn_b200.common import config, step_graph

    a = _trainer(tmp_path)

    def refuse(*args, **kwargs):
        raise AssertionError(args)

    monkeypatch.setattr(config.ConfigBase, "clone", refuse)
    monkeypatch.setattr(config.ConfigBase, "_unknown", refuse)
    assert step_graph.capturable(a)


@pytest.mark.parametrize("train_dtype", [None, torch.float32])
def test_training_in_32_bits(tmp_path, train_dtype):
    """The model reads the masters themselves, which the fused update changes in place; no step of it is captured.

    Sums of up to 1024 terms in another order than the CPU's, 1e-5 of a gradient; AdamW's first steps turn a gradient into
    little more than its sign, so a weight may differ by two learning rates (1e-2 in all) where a gradient is next to zero."""
    from tests.helpers import tiny_fuji_trainer_config

    trainers = []
    for device in ("cuda:0", "cpu"):
        cfg = tiny_fuji_trainer_config(tmp_path / device, device=device, train_dtype=train_dtype, hidden=128, heads=2, ffn=256,
                                       vocab=512, seq=64, layers=2, max_step=10)
        trainer = cfg.instantiate(parent=None)
        trainer.init(prng.PRNGKey(0))
        trainers.append((trainer, iter(trainer.input.dataset())))
    for (_, x), (_, y) in zip(*(flatten_items(t.trainer_state["model"]) for t, _ in trainers)):
        y.copy_(x)  # random numbers are a device's own
    for _ in range(4):
        x, y = (t.train_step(next(data))["loss"] for t, data in trainers)
        torch.testing.assert_close(x.cpu(), y, rtol=1e-3, atol=0)
    assert not _captured(trainers[0][0])
    for (path, x), (_, y) in zip(*(flatten_items(t.trainer_state["model"]) for t, _ in trainers)):
        assert (x.cpu() - y).norm() <= 1e-2 * y.norm(), path
