"""The step kernel's block elimination at the sizes where its tiles can go wrong:
free blocks of one 8-row panel, of whole panels and of a last panel of 2, 4 and
6 rows (6 unknowns per free node), and unconstrained beams, each in both forms
against the FP64 oracle."""
import numpy as np
import pytest

from openturbine_b200 import workloads as W
from openturbine_b200.model import GaussLegendreQuadrature, Model

pytestmark = pytest.mark.gpu


def _beam(nodes, points, clamped):
    rng = W.rng_for(9_000 + nodes)
    m = Model()
    ids = [m.AddNode().SetElemLocation(s).SetPosition(20. * s, 0., 0., 1., 0., 0., 0.).Build()
           for s in W.gll_node_locations(nodes)]
    m.AddBeamElement(ids, W.tapered_sections(rng, 5), GaussLegendreQuadrature(points))
    if clamped:
        m.AddFixedBC(ids[0])
    return m


# nodes, clamped; clamped free blocks of 6 (n - 1) rows: 6, 12, 18, 24, 30, 48, 60, 84, 96, 120
@pytest.mark.parametrize("nodes, clamped", [(2, True), (3, True), (4, True), (5, True), (6, True), (9, True),
                                            (11, True), (15, True), (17, True), (21, True), (4, False), (7, False)])
@pytest.mark.parametrize("precision", [0, 1])
def test_elimination_matches_oracle(nodes, clamped, precision):
    from openturbine_b200.runtime import Context
    from oracle.oracle_py import OracleModel
    pm = _beam(nodes, nodes + 1, clamped).pack()
    ctx = Context(0)
    mid = ctx.create_model(pm)
    orc = OracleModel(pm)
    p, po = W.batch_params(), W.batch_params()
    p.precision = precision
    fx = np.zeros((nodes, 6))
    for step in range(3):
        fx[-1] = np.array([200., 300., 400., 10., 20., 30.]) * np.cos(0.3 * step)
        ctx.set_node_fx(mid, fx)
        orc.set_node_fx(fx)
        st, it = ctx.step([mid], p)
        ost, oit = orc.step(po)
        assert int(st[0]) == ost == 0
        if precision == 0:
            assert int(it[0]) == oit
    # FP64: the parity bar on q; FP32: the worst-beam bar of the form (1e-5) on the motion
    q, oq = ctx.state(mid, "q"), orc.state("q")
    d, od = (q - [0., 0., 0., 1., 0., 0., 0.]), (oq - [0., 0., 0., 1., 0., 0., 0.])
    tol = 1e-10 * np.abs(oq).max() if precision == 0 else 1e-5 * np.abs(od).max()
    assert np.abs(d - od).max() <= tol
    ctx.close()



@pytest.mark.parametrize("precision", [0, 1])
def test_many_small_beams_match_few(precision):
    """A step of more beams than fill the GPU twice over runs small beams on
    fewer threads each: the same Newton decisions and states as alone, at the
    smallest size and at the largest that fits four to an SM."""
    from openturbine_b200.runtime import Context
    p = W.batch_params()
    p.precision = precision
    ctx = Context(0)
    sizes = (2, 5, 10)
    alone, many = [], []
    for nodes in sizes:
        pm = _beam(nodes, nodes + 1, True).pack()
        alone.append(ctx.create_model(pm))
        many.append([ctx.create_model(pm)])
        many[-1] += [ctx.clone_model(many[-1][0]) for _ in range(109)]
    fx = [np.zeros((n, 6)) for n in sizes]
    for step in range(2):
        for f, a, ms in zip(fx, alone, many):
            f[-1] = np.array([200., 300., 400., 10., 20., 30.]) * np.cos(0.3 * step)
            for i in [a] + ms:
                ctx.set_node_fx(i, f)
        sa, ia = ctx.step(alone, p)
        sm, im = ctx.step([i for ms in many for i in ms], p)
        assert (sa == 0).all() and (sm == 0).all()
        assert (im.reshape(len(sizes), -1) == ia[:, None]).all()
    for a, ms in zip(alone, many):
        q = ctx.state(a, "q")
        for i in (ms[0], ms[-1]):
            assert np.abs(ctx.state(i, "q") - q).max() <= 1e-13 * np.abs(q).max()
    ctx.close()
