"""Kernels of chained launches (``csrc/chain.cuh``), by their sources: a chained kernel is resident before its input is
written, so it waits before anything else and reads with ordinary loads."""

import os
import re

import pytest

from axlearn_b200.csrc import build

_KERNEL = re.compile(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\s*\(([^)]*(?:\(\)[^)]*)*)\)\s*\{")
# Parameters that no step writes.
_CONSTANT = {"table"}


def _kernels() -> dict:
    """``{name: (parameters, body)}`` of all kernels in the sources."""
    out = {}
    for path in build.sources():
        with open(path, encoding="utf-8") as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        for m in _KERNEL.finditer(text):
            depth, at = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[at], 0)
                at += 1
            out[m.group(1)] = (m.group(2), text[m.end():at - 1])
    return out


def _chained() -> dict:
    return {name: k for name, k in _kernels().items() if "chain_link()" in k[1] or "chain_wait()" in k[1]}


def test_every_chained_launch_has_a_kernel_that_waits():
    launched = set()
    for path in build.sources():
        with open(path, encoding="utf-8") as f:
            text = f.read()
        launched |= set(re.findall(r"launch_chained\(\s*(?:axb::)?(\w+)", text))
        launched |= set(re.findall(r"kernel = chain_launches \? (\w+)", text))
    launched -= {"kernel"}  # a variable: set as in the second pattern, or (hyper.cu) to hyper_step_kernel
    assert launched and "hyper_step_kernel" in _chained() and launched <= set(_chained())


@pytest.mark.parametrize("name", sorted(_chained()))
def test_chained_kernel_waits_first_and_reads_in_order(name):
    params, body = _chained()[name]
    if name != "gemm_skinny_kernel":  # fills its stages with resident weights ahead of the wait
        assert body.lstrip().startswith("chain_link();")
    for param in params.split(","):
        assert "__restrict__" not in param or param.split()[-1] in _CONSTANT, param
    for call in ("__ldg(", "ld_nc(", ".nc."):
        for at in re.finditer(re.escape(call), body):
            assert re.match(r"\s*(\w+)", body[at.end():]).group(1) in _CONSTANT, body[at.start():at.end() + 40]
