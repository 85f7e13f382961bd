"""Copies of one hub model in one step: every copy takes the same Newton
iterations to the same bits, which needs all threads of a CTA to form the
model's convergence error from the same hub record."""
import numpy as np
import pytest

from openturbine_b200 import workloads as W
from openturbine_b200.model import Model, RotationVectorToQuaternion, StepParameters
from openturbine_b200.model import GaussLegendreQuadrature

pytestmark = pytest.mark.gpu

OMEGA, H = 0.8, 0.01


def _rotor(nodes, drive):
    """Three spinning blades on a hub node that follows a prescribed rotation, or
    on a drive train (revolute joint from a fixed base)."""
    m = Model()
    m.SetGravity(0., 0., -9.81)
    spin = [0., 0., 0., 0., 0., OMEGA]
    sections = W.tapered_sections(W.rng_for(31), 5)
    roots = []
    for b in range(3):
        ids = [m.AddNode().SetElemLocation(s).SetPosition(2. + 30. * s, 0., 0., 1., 0., 0., 0.).Build()
               for s in W.gll_node_locations(nodes)]
        e = m.AddBeamElement(ids, sections, GaussLegendreQuadrature(nodes + 1))
        m.RotateBeamAboutPoint(e, RotationVectorToQuaternion([0., 0., 2. * np.pi * b / 3.]), [0., 0., 0.])
        m.SetBeamVelocityAboutPoint(e, spin, [0., 0., 0.])
        roots.append(ids[0])
    hub = m.AddNode().SetPosition(0., 0., 0., 1., 0., 0., 0.).SetVelocity(*spin).Build()
    if drive:
        base = m.AddNode().SetPosition(0., 0., -1., 1., 0., 0., 0.).Build()
        m.AddFixedBC(base)
        held = m.AddRevoluteJointConstraint([base, hub], [0., 0., 1.], np.zeros(1))
    else:
        held = m.AddPrescribedBC(hub)
    for r in roots:
        m.AddRigidJointConstraint([hub, r])
    return m, held


@pytest.mark.parametrize("nodes, drive", [(5, False), (9, False), (5, True), (9, True)])
def test_hub_copies_take_the_same_steps(nodes, drive):
    from openturbine_b200.runtime import Context
    m, held = _rotor(nodes, drive)
    ctx = Context(0)
    ids = [ctx.create_model(m.pack())]
    ids += [ctx.clone_model(ids[0]) for _ in range(63)]
    p = StepParameters(True, 10, H, 0.9)
    for step in range(6):
        if not drive:
            a = 0.5 * OMEGA * H * (step + 1)
            for i in ids:
                ctx.set_prescribed(i, held, [0., 0., 0., np.cos(a), 0., 0., np.sin(a)])
        st, it = ctx.step(ids, p)
        assert (st == 0).all() and (it == it[0]).all()
    for f in ("q", "v", "lambda"):
        first = ctx.state(ids[0], f)
        assert np.isfinite(first).all()
        for i in ids[1:]:
            assert (ctx.state(i, f) == first).all()
    ctx.close()
