"""A training step as one CUDA graph.

The reference traces and compiles its step (axlearn/common/trainer.py:1000-1090) and launches it as one program.  Run
eagerly, a step of a small decoder is some 240 launches behind 8 ms of Python, of which the GPU is busy for one (two
layers of 512, 2 x 333 tokens: 8.7 ms; two layers of 2048, 2 x 2048 tokens: 8.8 ms, 6.5 ms of work on the GPU).  So a
step that repeats is captured -- forward, backward, clipping, update -- and replayed; what changes from step to step
on the host (schedules, bias corrections, counters, keys) is computed there each time and handed over in device
memory.  The two steps take 0.8 and 7.1 ms then, 0.4 ms of it on the host.  Capturing takes some 15 ms once, in the
second step.

When a step is captured: one GPU, weights that the model reads in bf16, nothing in the model that draws random numbers,
every layer of a type that is known to put the same work on the GPU whatever the values (``_LAYERS``), the learner's
closed-form AdamW, and a step of the same signature just before it: shapes of the batch, addresses of parameters,
moments and shadows, and the switches that choose kernels.  The configurations that a step reads are compared each time.
Everything else runs step by step as before, and so does a step under autograd hooks, function transforms, dispatch or
function modes, anomaly detection, autocast, a running profiler trace or a caller's own capture.  A model whose gradients
alone take more than a sixteenth of the GPU's memory is not tried, and a capture that would keep more than that is given
up.  One that fails is tried again later, twice, and says so in the log.  With other parameters or settings all begins anew.

A graph keeps its activations' memory for as long as it lives; a trainer has one at a time and captures a few times at
most for the same parameters.  Steps of two shapes in turn are not captured.
"""

from __future__ import annotations

import dataclasses
import gc
import logging
from typing import Any, Callable, Optional

import torch

from axlearn_b200.common import remat
from axlearn_b200.common.utils import flatten_items, tree_map

Tensor = torch.Tensor

_MAX_CAPTURES = 4
_MEMORY_SHARE = 16
# Steps to wait after the first, the second, ... capture that failed for a reason that may pass (memory that somebody else
# held); behind them no more is tried.
_PAUSES = (100, 1000)

_COMMON = "axlearn_b200.common."
# Exact types: a subclass may do anything in its forward.
_LAYERS = frozenset(_COMMON + name for name in (
    "causal_lm.Model", "causal_lm.CompositeLossMetrics", "causal_lm.CrossEntropyLossMetrics",
    "causal_lm.AuxLossMetrics", "decoder.Decoder", "decoder.DecodingLayer", "embedding.TransformerTextEmbeddings",
    "layers.Embedding", "layers.Dropout", "layers.RMSNorm", "layers.StochasticDepth", "layers.Linear",
    "attention.RepeatedTransformerLayer", "attention._TransformerRepeat", "attention.TransformerLayer",
    "attention.TransformerAttentionLayer", "attention.RoFormerQKVLinear",
    "attention.RoFormerSinusoidalPositionalEmbedding", "attention.FusedQKVLinear", "attention._FusedQKVProj",
    "attention.FusedGroupedQKVLinear", "attention.MultiheadInputLinear", "attention.MultiheadOutputLinear",
    "attention.ScaleQuery", "attention.ScaleKey", "attention.TransformerFeedForwardLayer",
    "flash_attention.layer.FlashAttention", "kv_cache.kv_cache.KVCache"))


class Refused(RuntimeError):
    """A step that cannot be captured."""


def map_tensors(tree: Any, fn: Callable) -> Any:
    """``tree`` (dicts, sequences, named tuples, dataclasses, tensors, plain values) with ``fn`` applied to its tensors."""
    if isinstance(tree, Tensor):
        return fn(tree)
    if tree is None or isinstance(tree, (bool, int, float, str)):
        return tree
    if isinstance(tree, dict):
        return type(tree)((k, map_tensors(v, fn)) for k, v in tree.items())
    if isinstance(tree, tuple) and hasattr(tree, "_fields"):
        return type(tree)(*(map_tensors(v, fn) for v in tree))
    if isinstance(tree, (list, tuple)):
        return type(tree)(map_tensors(v, fn) for v in tree)
    if dataclasses.is_dataclass(tree) and not isinstance(tree, type):
        return dataclasses.replace(tree, **{f.name: map_tensors(getattr(tree, f.name), fn)
                                            for f in dataclasses.fields(tree)})
    raise Refused(f"an output of type {type(tree)}")


def _layers_known(module) -> bool:
    name = f"{type(module).__module__}.{type(module).__qualname__}"
    if name not in _LAYERS or "forward" in vars(module):
        return False
    # (Read in place and asked for what it has: `config` copies, and a missing field makes up the text of an error, together
    # 5 ms for a small model's layers.)
    cfg = module._config  # pylint: disable=protected-access
    if "rate" in cfg and cfg.rate:  # drops something at random
        return False
    spec = cfg.remat_spec if "remat_spec" in cfg else None
    if spec is not None:
        policy = remat.as_policy(spec.policy)
        if policy is not None and (policy.offload_pattern is not None or policy.dots == remat.OFFLOAD):
            return False
    return all(_layers_known(child) for child in module._children.values())  # pylint: disable=protected-access


def _settings(trainer) -> tuple:
    """What an eager step reads from configurations each time and a captured one does not."""

    def values(cfg):
        # (Lists by value: they may be changed in place.)
        return [list(v) if type(v) is list else v for v in cfg._values.values()]  # pylint: disable=protected-access

    def visit(module):
        out.append((type(module), "forward" in vars(module), values(module._config)))  # pylint: disable=protected-access
        for child in module._children.values():  # pylint: disable=protected-access
            visit(child)

    out: list = []
    visit(trainer.model)
    learner, cfg = trainer.learner, trainer._config  # pylint: disable=protected-access
    out.append((type(trainer), cfg.grad_accumulation_steps, trainer._has_param_noise, type(learner),  # pylint: disable=protected-access
                "update" in vars(learner), learner.ema, values(learner._config)))  # pylint: disable=protected-access
    return tuple(out)


def capturable(trainer) -> bool:
    """Whether the trainer's configuration allows a captured step (what a single call adds: ``_call_allows``)."""
    from axlearn_b200.common.learner import Learner
    from axlearn_b200.common.trainer import SpmdTrainer

    cfg, learner = trainer._config, trainer.learner  # pylint: disable=protected-access
    fused = getattr(getattr(learner, "optimizer", None), "fused", None)
    return (
        type(trainer) is SpmdTrainer and type(learner) is Learner and "update" not in vars(learner)
        and trainer._device.type == "cuda" and trainer._mesh is not None  # pylint: disable=protected-access
        and all(size == 1 for size in trainer._mesh.shape.values())  # pylint: disable=protected-access
        and cfg.grad_accumulation_steps <= 1 and not trainer._has_param_noise  # pylint: disable=protected-access
        and learner.ema is None and fused is not None and fused.per_param_scale is None
        and learner._config.allow_fused_update  # pylint: disable=protected-access
        and not learner._config.enable_per_variable_summaries  # pylint: disable=protected-access
        and _layers_known(trainer.model))


def _call_allows(trainer, leaves: list) -> bool:
    from axlearn_b200.ops import cuda_ops

    try:
        # pylint: disable=protected-access
        modes = (torch._C._len_torch_function_stack() or torch._C._len_torch_dispatch_stack()
                 or torch._C._autograd._top_saved_tensors_default_hooks(False) is not None)
    except AttributeError:  # not a name that torch promises: unknown counts as on
        modes = True
    return not (
        modes or cuda_ops._transformed() or not torch.is_grad_enabled()  # pylint: disable=protected-access
        or torch.is_anomaly_enabled() or torch.is_autocast_enabled() or torch.is_inference_mode_enabled()
        or torch.cuda.is_current_stream_capturing() or trainer._profiler is not None  # pylint: disable=protected-access
        or any(t._backward_hooks or getattr(t, "_post_accumulate_grad_hooks", None) for t in leaves))


def _switches() -> tuple:
    from axlearn_b200.ops import cuda_ops, dispatch, flash_sm100

    return (cuda_ops.GEMM_VARIANT, cuda_ops.RMSNORM_VARIANT, cuda_ops.COMM_RESERVED_SMS, flash_sm100.FORWARD_VARIANT,
            flash_sm100.BACKWARD_VARIANT, dispatch._flags.force_reference,  # pylint: disable=protected-access
            torch.are_deterministic_algorithms_enabled(), torch.get_float32_matmul_precision(),
            torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction, torch.get_default_dtype(),
            torch.cuda.current_device())


class _Captured:
    """One captured step and what its replays need."""

    def __init__(self, signature, graph, inputs, outputs, grads, scalars, launches, kept):
        self.signature, self.graph, self.inputs, self.outputs = signature, graph, inputs, outputs
        self.grads, self.scalars, self.launches, self.kept = grads, scalars, launches, kept


class StepGraphs:
    """The captured step of one trainer."""

    def __init__(self):
        self._capturable: Optional[bool] = None
        self._settings: Optional[tuple] = None  # with which that was found
        self._captured: Optional[_Captured] = None
        self._last: Optional[tuple] = None
        self._given_up = False
        self._captures = self._failures = self._pause = 0

    def forget(self) -> None:
        """Gives the captured step up, with what it holds: the trainer has got other parameters."""
        self._captured = self._last = None
        self._given_up = False
        self._captures = self._failures = self._pause = 0

    def run(self, trainer, batch: Any) -> Optional[dict]:
        """The step's outputs, or None where the caller has to run it."""
        settings = _settings(trainer)
        if self._capturable is None or (self._settings is not None and self._settings != settings):
            self._capturable, self._settings = capturable(trainer), settings
            self._captured = self._last = None
            self._given_up = False
        if not self._capturable or self._given_up:
            return None
        signature = self._signature(trainer, batch)
        if signature is not None and (self._captured is None or self._captured.signature != signature):
            device = trainer._device  # pylint: disable=protected-access
            if (signature == self._last and self._captures < _MAX_CAPTURES and _gradient_bytes(trainer) <= _most_memory(device)
                    and torch.cuda.mem_get_info(device)[0] > _most_memory(device)):
                self._captured = None  # its memory is given back first
                if self._pause:
                    self._pause -= 1
                    return None
                try:
                    self._captured = _capture(trainer, batch, signature)
                    self._captures += 1
                except Refused as e:
                    logging.info("training step not captured: %s", e)
                    self._given_up = True
                    return None
                except Exception as e:  # pylint: disable=broad-except
                    self._failures += 1
                    self._given_up = self._failures > len(_PAUSES)
                    self._pause = 0 if self._given_up else _PAUSES[self._failures - 1]
                    logging.warning("training step not captured (attempt %d), %s: %s", self._failures,
                                    "given up" if self._given_up else f"tried again in {self._pause} steps", e)
                    return None
        self._last = signature
        if signature is None or self._captured is None or self._captured.signature != signature:
            return None
        return _replay(self._captured, trainer, batch)

    @staticmethod
    def _signature(trainer, batch: Any) -> Optional[tuple]:
        state = trainer.trainer_state
        inputs = flatten_items(batch)
        shadows = flatten_items(trainer._shadows)  # pylint: disable=protected-access
        leaves = [t for _, t in shadows if isinstance(t, Tensor)]
        if not _call_allows(trainer, leaves) or not all(isinstance(t, Tensor) and t.is_cuda for _, t in inputs):
            return None
        if any(t.is_floating_point() and t.dtype != torch.bfloat16 for t in leaves):
            return None
        adam = trainer.learner.optimizer.fused.locate(state["learner"]["optimizer"])[0]
        held = leaves + [t for tree in (state["model"], adam.mu, adam.nu) for _, t in flatten_items(tree)]
        if not all(isinstance(t, Tensor) and t.is_cuda for t in held):
            return None
        fused = trainer.learner.optimizer.fused
        return (tuple((p, tuple(t.shape), t.stride(), t.dtype) for p, t in inputs),
                tuple((t.data_ptr(), tuple(t.shape), t.dtype, t.requires_grad) for t in held),
                (fused.b1, fused.b2, fused.eps, fused.clip_max_norm, fused.clip_eps), _switches())


@torch.no_grad()
def _copy(dst: list, src: list) -> None:
    by_type: dict = {}
    for d, s in zip(dst, src):
        by_type.setdefault(d.dtype, ([], []))
        by_type[d.dtype][0].append(d)
        by_type[d.dtype][1].append(s)
    for d, s in by_type.values():
        torch._foreach_copy_(d, s)  # pylint: disable=protected-access


def _gradient_bytes(trainer) -> int:
    """What a captured step holds at least: gradients of its own."""
    return sum(t.numel() * t.element_size() for _, t in flatten_items(trainer._shadows)  # pylint: disable=protected-access
               if isinstance(t, Tensor) and t.requires_grad)


def _most_memory(device: torch.device) -> int:
    return torch.cuda.get_device_properties(device).total_memory // _MEMORY_SHARE


def _capture(trainer, batch: Any, signature: tuple) -> _Captured:
    from axlearn_b200.ops import cuda_ops
    from axlearn_b200.parallel import fsdp

    device = trainer._device  # pylint: disable=protected-access
    inputs = [torch.empty_like(t) for _, t in flatten_items(batch)]
    order = {id(t): i for i, (_, t) in enumerate(flatten_items(batch))}
    static = map_tensors(batch, lambda t: inputs[order[id(t)]])
    scalars = cuda_ops.AdamwScalars(device)
    # Other leaves on the shadows' memory: outputs of an earlier step that a caller still holds keep that step's nodes of
    # the shadows alive, which belong to its stream and would be met again here.
    shadows = trainer._shadows  # pylint: disable=protected-access
    leaves = tree_map(lambda t: t.detach().requires_grad_(t.requires_grad), shadows)
    reserved = torch.cuda.memory_reserved(device)
    before = cuda_ops.launch_count
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream(device)
    stream.wait_stream(torch.cuda.current_stream(device))
    collects = gc.isenabled()
    gc.disable()  # garbage with CUDA objects in it would be destroyed in the middle, which ends a capture
    try:
        trainer._shadows = leaves  # pylint: disable=protected-access
        # (Not `torch.cuda.graph`, which empties the allocator's cache: what runs next would pay for its memory again.)
        with torch.cuda.stream(stream):
            graph.capture_begin(capture_error_mode="thread_local")
            try:
                loss, aux, collected = trainer._forward_backward(static, None)  # pylint: disable=protected-access
                if any(True for _ in flatten_items(collected.state_updates)):
                    raise Refused("a layer updates its state")
                with cuda_ops.adamw_scalars(scalars):
                    _, learner_summaries = trainer._apply_update(collected)  # pylint: disable=protected-access
            finally:
                graph.capture_end()
    finally:
        if collects:
            gc.enable()
        trainer._shadows = shadows  # pylint: disable=protected-access
        launches, cuda_ops.launch_count = cuda_ops.launch_count - before, before
        for _, leaf in flatten_items(leaves):
            fsdp.reset_grad_slices(leaf)
    if torch.cuda.memory_reserved(device) - reserved > _most_memory(device):
        raise Refused("its activations would stay in too much memory")
    outputs = {"loss": loss, "aux": aux, "model": collected.summaries, "learner": learner_summaries}
    results: list = []

    def note(t):
        if not t.is_cuda:
            raise Refused("an output in host memory")
        results.append(t)
        return t

    map_tensors({k: v for k, v in outputs.items() if k != "learner"}, note)
    for name, value in learner_summaries.items():
        if isinstance(value, Tensor) and value.is_cuda:
            results.append(value)
        elif name not in _host_summaries(trainer)[2]:
            raise Refused(f"a learner summary {name}")
    grads = [(t, leaf.grad) for (_, t), (_, leaf) in zip(flatten_items(shadows), flatten_items(leaves))]
    # Held as long as the graph has their addresses (inputs, gradients and scalars are, too).
    learner_state = trainer.trainer_state["learner"]
    kept = [static, trainer.trainer_state["model"], shadows,
            trainer.learner.optimizer.fused.locate(learner_state["optimizer"])[0]]
    return _Captured(signature, graph, inputs, (outputs, results), grads, scalars, launches, kept)


def _host_summaries(trainer) -> tuple:
    from axlearn_b200.common.learner import fused_scalars

    fused = trainer.learner.optimizer.fused
    return fused_scalars(fused, trainer.trainer_state["learner"]["optimizer"])


def _replay(captured: _Captured, trainer, batch: Any) -> dict:
    from axlearn_b200.common.learner import rebuild_fused_state
    from axlearn_b200.ops import cuda_ops

    learner_state = trainer.trainer_state["learner"]
    fused = trainer.learner.optimizer.fused
    count, values, host = _host_summaries(trainer)
    _copy(captured.inputs, [t for _, t in flatten_items(batch)])
    captured.scalars.store(b1=fused.b1, b2=fused.b2, **values)
    for leaf, grad in captured.grads:
        if leaf.grad is not grad:
            leaf.grad = grad
    captured.graph.replay()
    cuda_ops.launch_count += captured.launches
    new_state = dict(learner_state)
    new_state["optimizer"] = rebuild_fused_state(learner_state["optimizer"], fused, count)
    trainer.trainer_state["learner"] = new_state
    outputs, results = captured.outputs
    # The graph's own outputs change with the next step.
    fresh = {id(t): torch.empty_like(t) for t in results}
    _copy([fresh[id(t)] for t in results], results)

    def pick(t):
        return fresh[id(t)]

    learner = {name: pick(v) if isinstance(v, Tensor) and v.is_cuda else host[name]
               for name, v in outputs["learner"].items()}
    return {"loss": pick(outputs["loss"]), "aux": map_tensors(outputs["aux"], pick),
            "summaries": {"model": map_tensors(outputs["model"], pick), "learner": learner}}
