"""The Gauss-Jordan solver in a step of more beams than fill the GPU twice over:
such a step runs small beams on 128 threads each, but not beams whose free block
the 128-thread register grid does not hold, which keep the solver that the caller
asked for.  FP32 form: 64 rows in that grid, 128 at 256 threads (clamped beams of
12 to 14 nodes have 66 to 78); FP64 form: 56 and 96 rows (an unconstrained beam of
10 nodes has 60)."""
import numpy as np
import pytest

from openturbine_b200 import workloads as W
from openturbine_b200.model import GaussLegendreQuadrature, Model

pytestmark = pytest.mark.gpu

STAT_SOLVES_CHECKED = 4  # KYN_STAT_SOLVES_CHECKED


def _beam(nodes, clamped):
    m = Model()
    ids = [m.AddNode().SetElemLocation(s).SetPosition(20. * s, 0., 0., 1., 0., 0., 0.).Build()
           for s in W.gll_node_locations(nodes)]
    m.AddBeamElement(ids, W.tapered_sections(W.rng_for(9_100 + nodes), 5), GaussLegendreQuadrature(nodes + 2))
    if clamped:
        m.AddFixedBC(ids[0])
    return m.pack()


@pytest.mark.parametrize("nodes, clamped, precision", [
    (5, True, 1), (11, True, 1), (12, True, 1), (13, True, 1), (14, True, 1), (9, True, 0), (10, True, 0), (10, False, 0)])
def test_gauss_jordan_alone_and_in_a_large_step(nodes, clamped, precision):
    from openturbine_b200.runtime import SOLVER_GAUSS_JORDAN, Context
    ctx = Context(0)
    ctx.set_linear_solver(SOLVER_GAUSS_JORDAN)
    pm = _beam(nodes, clamped)
    alone = ctx.create_model(pm)
    many = [ctx.create_model(pm)]
    many += [ctx.clone_model(many[0]) for _ in range(319)]
    p = W.batch_params()
    p.precision = precision
    fx = np.zeros((nodes, 6))
    for step in range(3):
        fx[-1] = np.array([200., 300., 400., 10., 20., 30.]) * np.cos(0.3 * step)
        for i in [alone] + many:
            ctx.set_node_fx(i, fx)
        before = ctx.stat(STAT_SOLVES_CHECKED)
        st, it = ctx.step([alone], p)
        assert int(st[0]) == 0 and ctx.stat(STAT_SOLVES_CHECKED) - before == int(it[0])
        before = ctx.stat(STAT_SOLVES_CHECKED)
        sm, im = ctx.step(many, p)
        assert (sm == 0).all() and (im == it[0]).all()
        assert ctx.stat(STAT_SOLVES_CHECKED) - before == int(im.sum())
    q = ctx.state(alone, "q")
    for i in (many[0], many[-1]):
        assert np.abs(ctx.state(i, "q") - q).max() <= 1e-10 * np.abs(q).max()
    ctx.close()


@pytest.mark.parametrize("nodes", [5, 12, 16, 18])
def test_tuned_fp32_gauss_jordan_keeps_its_refinement(nodes):
    """The autotuner trades no refinement for speed: every solve of the FP32 form
    with the solver is still checked."""
    from openturbine_b200.runtime import SOLVER_GAUSS_JORDAN, Context
    ctx = Context(0)
    ctx.set_linear_solver(SOLVER_GAUSS_JORDAN)
    ids = [ctx.create_model(_beam(nodes, True))]
    ids += [ctx.clone_model(ids[0]) for _ in range(319)]
    p = W.batch_params()
    p.precision = 1
    fx = np.zeros((nodes, 6))
    fx[-1] = [200., 300., 400., 10., 20., 30.]
    for i in ids:
        ctx.set_node_fx(i, fx)
    ctx.autotune(ids, p)
    before = ctx.stat(STAT_SOLVES_CHECKED)
    st, it = ctx.step(ids, p)
    assert (st == 0).all()
    assert ctx.stat(STAT_SOLVES_CHECKED) - before == int(it.sum())
    ctx.close()
