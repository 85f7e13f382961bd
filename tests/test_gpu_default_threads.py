"""kyn_tuned_threads states what a step of few beams runs with: 256 threads where
two such CTAs fit an SM, else 512; dense models 128, condensed ones 256."""
import pytest

from openturbine_b200 import workloads as W
from tests.workloads_ref import four_element_cantilever_model, two_long_beams_model

pytestmark = pytest.mark.gpu


def test_default_threads_by_kind():
    from openturbine_b200.runtime import Context
    from tests.test_gpu_bordered import _chain
    ctx = Context(0)
    small = ctx.create_model(W.cantilever_model().pack())
    long = ctx.create_model(W.cantilever_model(21, 10., 23).pack())
    dense = ctx.create_model(_chain(4, True)[0].pack())
    condensed = [ctx.create_model(f()[0].pack()) for f in (four_element_cantilever_model, two_long_beams_model)]
    assert all(ctx.info(c).condensed_dofs > 0 for c in condensed)
    for precision in (0, 1):
        assert ctx.tuned_threads(small, precision) == 256
        assert ctx.tuned_threads(dense, precision) == 128
        assert [ctx.tuned_threads(c, precision) for c in condensed] == [256, 256]
    assert ctx.tuned_threads(long, 0) == 512 and ctx.tuned_threads(long, 1) == 256
    ctx.close()
