"""Guards around the integer form: memory that an early-resident pass reads, what a failed call
leaves behind, which form a plan runs, and the calls of an integer plan that run in FP64."""
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "gpulucas_gb300", "csrc")


def _code(name):
    """A source file without its comments."""
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def test_early_resident_passes_read_written_memory_with_ordinary_loads():
    """A programmatic dependent is resident while the pass before it still writes the
    products and work arrays, so it may not read them through the non-coherent path."""
    nc = re.compile(r"__ldg\s*\((?:[^()]|\([^()]*\))*\ba\.(?:ll|Z|Z2|digit|hi)\b")
    for name in ("gl_dice.cuh", "gl_int_kernels.cu"):
        assert not nc.search(_code(name)), name
    k = _code("gl_int_kernels.cu")
    # every pass that may be launched as a dependent (P == 0) asks for the ordinary loads
    assert re.findall(r"load_point<([^>]*)>", k) == ["FROM_STATE, NC, P == 0"]
    assert "dependent) after_previous_pass()" in k
