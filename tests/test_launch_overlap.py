"""Kernels whose launch overlaps the kernel before them (`launch_after`): each waits for it
before anything else, and reads what other launches write by coherent loads only."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "wellbalanced_b200" / "csrc"
#: element types of the tables that the host uploads and no launch writes
TABLES = {"PatchDesc", "Tile", "CopyOp", "InterpOp", "RestrictOp", "FaceFluxOp", "RefluxOp"}
KERNEL = re.compile(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\((?:[^()]|\([^()]*\))*\))*\)\s*)?(\w+)\(([^)]*)\)\s*\{\s*([^\n]*)")


def _sources():
    return {path.name: path.read_text() for path in sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")])}


def _kernels():
    return {name: (params, first) for text in _sources().values() for name, params, first in KERNEL.findall(text)}


def _overlapping():
    names = {name for text in _sources().values() for name in re.findall(r"launch_after\((\w+)<", text)}
    assert {"stage2d_kernel", "stage3d_kernel", "stable_dt_kernel", "copy_ops_kernel", "reflux_apply_kernel"} <= names
    return sorted(names)


@pytest.mark.parametrize("name", _overlapping())
def test_an_overlapping_kernel_waits_first(name):
    _, first = _kernels()[name]
    assert first.startswith("after_previous();")


@pytest.mark.parametrize("name", _overlapping())
def test_an_overlapping_kernel_marks_tables_only_as_read_only(name):
    """A `const T* __restrict__` parameter may be read through the non-coherent path and ahead
    of the wait; the kernel before may still be writing a pool, a dt or a flux buffer."""
    params, _ = _kernels()[name]
    marked = re.findall(r"const\s+(\w+)\s*\*\s*__restrict__\s*(\w+)", params)
    assert all(kind in TABLES for kind, _ in marked), marked


@pytest.mark.parametrize("name", ["ops.cuh", "ratecell.cuh", "stage2d.cu", "stage3d.cu", "reflux.cu"])
def test_helpers_of_these_kernels_mark_tables_only(name):
    """The bodies that the kernels share with the op programs, whose phases write what later
    ones read: no read-only pointer to a state or a dt there either."""
    text = _sources()[name]
    helpers = [params for _, params in re.findall(r"__device__ __forceinline__ \w+ (\w+)\(([^{;]*)\)\s*\{", text)]
    assert helpers
    marked = [m for params in helpers for m in re.findall(r"const\s+(\w+)\s*\*\s*__restrict__\s*(\w+)", params)]
    assert all(kind in TABLES for kind, _ in marked), marked
    assert not re.search(r"const\s+(?:S|R|double)\s*\*\s*__restrict__\s*\w+\s*=", text)
