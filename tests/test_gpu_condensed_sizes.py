"""Condensed beam elements at the sizes where their tiles and passes can go
wrong: interior unknowns that need 0, 2, 4 and 6 rows of padding to whole
tiles, all quadrature points in one pass, in passes of sixteen and eight with a
remainder, and the packed rows of the largest elements, against the oracle's
dense solve."""
import numpy as np
import pytest

from openturbine_b200.model import BeamSection, Model, StepParameters
from tests.workloads_ref import COMPOSITE_MASS, COMPOSITE_STIFF, chain_beam, chain_tip_loads

pytestmark = pytest.mark.gpu


# (elements, order, points): the last element's tip is interior too, so that a
# chain has elements of order - 1 and of order interior nodes.  A single element
# carries a two-node beam on a rigid joint (one pair of nodes with the packed
# rows' largest element).
@pytest.mark.parametrize("elements, order, points", [
    (8, 3, 5), (7, 3, 17), (6, 4, 6), (5, 5, 7), (3, 10, 12), (2, 17, 41), (2, 19, 21), (2, 19, 53), (2, 20, 34),
    (1, 21, 23)])
def test_condensed_elements_match_oracle(elements, order, points):
    from openturbine_b200.runtime import Context
    from oracle.oracle_py import OracleModel
    m = Model()
    m.SetGravity(0., 0., -9.81)
    secs = [BeamSection(0., COMPOSITE_MASS, COMPOSITE_STIFF), BeamSection(1., COMPOSITE_MASS, COMPOSITE_STIFF)]
    rule = [[x, w] for x, w in zip(*np.polynomial.legendre.leggauss(points))]
    along, elems = chain_beam(m, elements, order, 10. * elements, [1., 0., 0., 0.], secs, rule)
    m.AddFixedBC(along[0])
    if elements == 1:
        tail, more = chain_beam(m, 1, 1, 1., [1., 0., 0., 0.], secs, rule, origin=(10., 0., 0.))
        m.AddRigidJointConstraint([along[-1], tail[0]])
        elems = elems + more
    pm = m.pack()
    ctx = Context(0)
    mid = ctx.create_model(pm)
    assert ctx.info(mid).condensed_dofs > 0
    orc = OracleModel(pm)
    p = StepParameters(True, 8, 0.005, 0.2)
    for step in range(3):
        fx = chain_tip_loads(elems, along[-1], step)
        ctx.set_node_fx(mid, fx)
        orc.set_node_fx(fx)
        st, it = ctx.step([mid], p)
        assert (int(st[0]), int(it[0])) == orc.step(p)
        assert int(st[0]) == 0
    for f in ("q", "v"):
        a, b = ctx.state(mid, f), orc.state(f)
        assert np.abs(a - b).max() <= 1e-10 * max(1., np.abs(b).max())
    ctx.close()
