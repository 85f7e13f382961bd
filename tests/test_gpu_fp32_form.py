"""Tip states of the FP32 form (with one closing correction) on beams whose
corrections contract least, against the record of its arithmetic: 3xTF32
integration, FP32 panel LU.  Another order of the integration or of the
factorisation draws the form's rounding errors anew, which moved these tips by
2e-11 to 8e-11 m in one step; the last bits of the FP64 parts flip at most a few
of the 1e4 and more FP32 roundings behind a state, a hundredth of that or less."""
import numpy as np
import pytest

from openturbine_b200 import workloads as W
from openturbine_b200.model import StepParameters
from tests.workloads_ref import load_golden

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("copies", [1, 100])  # a small step, and one that fills the GPU
def test_fp32_form_states_match_record(copies):
    from openturbine_b200.runtime import Context
    gold = load_golden("fp32_form.json")
    tips = gold["tip_q_after_one_step"]
    draws = [W.draw_batch(1, int(i))[0] for i in tips]
    ctx = Context(0)
    first = [ctx.create_model(W.batch_cantilever_model(d).pack()) for d in draws]
    fz = gold["load_scale"] * W.tip_loads(draws, 0)
    for m, d, f in zip(first, draws, fz):
        ctx.set_node_fx(m, W.node_fx_for(d, f))
    ids = np.array([i for m in first for i in [m] + [ctx.clone_model(m) for _ in range(copies - 1)]], dtype=np.int32)
    st, _ = ctx.step(ids, StepParameters(True, 10, 0.01, 0.9, a_tol=1e-7, r_tol=1e-3, precision=1, refine_iters=1))
    assert (st == 0).all()
    for k, (d, tip) in enumerate(zip(draws, tips.values())):
        for i in ids[k * copies:(k + 1) * copies]:
            assert np.abs(ctx.state(int(i), "q")[-1] - tip).max() <= 1e-12, d
    ctx.close()
