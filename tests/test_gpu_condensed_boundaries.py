"""Condensed beam elements with many boundary nodes (point masses along the
element, its clamped root, a joint at its tip): the eliminated system's boundary
and right-hand-side columns take more tiles than the CTA has warps from eleven
boundary nodes on at 256 threads, from six on at 128.  And an element whose root
alone is a boundary node, of 22 interior nodes: more rows than 128 threads.
With the default threads and with the tuned ones, against the oracle's dense
solve."""
import numpy as np
import pytest

from openturbine_b200.model import BeamSection, Model, StepParameters
from tests.workloads_ref import COMPOSITE_MASS, COMPOSITE_STIFF, chain_beam

pytestmark = pytest.mark.gpu


def _model(order, points, masses):
    """A clamped element of `order` with point masses at its first `masses`
    interior nodes, and a second beam on a rigid joint at its tip; without
    masses, a beam of two nodes on a rigid joint at its root."""
    m = Model()
    m.SetGravity(0., 0., -9.81)
    secs = [BeamSection(0., COMPOSITE_MASS, COMPOSITE_STIFF), BeamSection(1., COMPOSITE_MASS, COMPOSITE_STIFF)]

    def rule(n):
        return [[x, w] for x, w in zip(*np.polynomial.legendre.leggauss(n))]

    along, _ = chain_beam(m, 1, order, 10., [1., 0., 0., 0.], secs, rule(points))
    joint, rest = (along[-1], 12) if masses else (along[0], 1)
    tail, _ = chain_beam(m, 1, rest, 6., [1., 0., 0., 0.], secs, rule(rest + 1),
                         origin=(10. if masses else 0., 0., 1.))
    for k in range(masses):
        m.AddMassElement(along[1 + k], np.diag([0.02] * 3 + [1e-4, 2e-4, 2e-4]) * (1. + 0.1 * k))
    m.AddFixedBC(along[0])
    m.AddRigidJointConstraint([joint, tail[0]])
    return m, along, tail


# (order, points, masses, boundary nodes of the first element)
@pytest.mark.parametrize("tuned", [False, True])
@pytest.mark.parametrize("order, points, masses, boundary", [
    (20, 21, 4, 6), (20, 21, 8, 10), (20, 21, 9, 11), (20, 21, 10, 12), (20, 21, 14, 16), (12, 13, 10, 12),
    (22, 12, 0, 1)])
def test_condensed_boundaries_match_oracle(order, points, masses, boundary, tuned):
    from openturbine_b200.runtime import Context
    from oracle.oracle_py import OracleModel
    m, along, tail = _model(order, points, masses)
    pm = m.pack()
    ctx = Context(0)
    mid = ctx.create_model(pm)
    # boundary nodes, the second beam's root, the clamp and the joint
    assert ctx.info(mid).condensed_dofs == 6 * (boundary + 1) + 12
    orc = OracleModel(pm)
    p = StepParameters(True, 8, 0.005, 0.2)
    fx = np.zeros((m.NumNodes(), 6))
    for step in range(3):
        fx[tail[-1], 1:3] = [9. * np.cos(0.4 * step), 15.]
        fx[along[1], 2] = 6.
        ctx.set_node_fx(mid, fx)
        orc.set_node_fx(fx)
        if step == 0 and tuned:
            ctx.autotune([mid], p)
        st, it = ctx.step([mid], p)
        assert (int(st[0]), int(it[0])) == orc.step(p)
        assert int(st[0]) == 0
    for f in ("q", "v"):
        a, b = ctx.state(mid, f), orc.state(f)
        assert np.abs(a - b).max() <= 1e-10 * max(1., np.abs(b).max())
    ctx.close()
