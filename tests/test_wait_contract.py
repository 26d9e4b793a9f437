"""The contract of the kernels that work ahead of their dependency wait (``common.cuh``), read off the sources: what they mark
``__restrict__`` is a model's own or the step's plan, never an operand that an earlier kernel of the step may have written."""

import pathlib
import re

import pytest

CSRC = pathlib.Path(__file__).resolve().parents[1] / "mini_infer_b200" / "csrc"

# weights, and what is uploaded before a step's first kernel
CONSTANT = {"W", "w", "uk_t", "uv", "sinks", "slopes", "freq", "block_table", "table_rows", "q_start", "kv_len", "positions", "slice_chunks"}


def kernels_that_wait_themselves():
    for path in sorted(CSRC.glob("*.cu")):
        text = path.read_text()
        starts = [m.start() for m in re.finditer(r"__global__", text)]
        for begin, end in zip(starts, starts[1:] + [len(text)]):
            body = text[begin:end]
            if "mi_pdl_wait()" in body:
                name, params = re.search(r"(\w+)\s*\(((?:[^()]|\([^()]*\))*)\)\s*\{", body[body.index("void"):]).groups()
                yield pytest.param(params, id=f"{path.stem}:{name}")


@pytest.mark.parametrize("params", list(kernels_that_wait_themselves()))
def test_only_constants_are_marked_restrict(params):
    marked = set(re.findall(r"__restrict__\s+(\w+)", params))
    assert marked <= CONSTANT, sorted(marked - CONSTANT)


def test_the_kernels_are_found():
    assert len(list(kernels_that_wait_themselves())) >= 10
