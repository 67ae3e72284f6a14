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


@pytest.mark.gpu
def test_batch_gives_row_units_room_for_the_stage_values(gl):
    """A plan with row_pass = 2 reads its stage values through L1; the batch's row kernel
    copies them behind the line buffers all the same."""
    p, N = 1257787, 65536
    o = {"fft_h": 128, "max_radix_row": 4}
    with gl.Plan(p, N, row_pass=2, **o) as a, gl.Plan(p, N, row_pass=1, **o) as b, gl.Plan(p, N) as want:
        assert a.info.row_variant == 2 and b.info.row_variant == 1
        assert a.info.smem_row < b.info.smem_row
        with gl.Batch(plans=[a]) as batch:
            assert batch.info.smem_row >= b.info.smem_row
            batch.iterate(70)
        want.iterate(70)
        assert (a.products() == want.products()).all()
