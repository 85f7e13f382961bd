"""The pivoted panel LU of the dense models at the sizes where its panels and
tiles can go wrong: chains of rigidly jointed point masses (12 unknowns a mass,
joint rows included) with and without a position-only node carried by the last
one (6 more), from a single short panel to the largest dense system, against
the oracle's dense solve."""
import numpy as np
import pytest

from openturbine_b200.model import Model, StepParameters

pytestmark = pytest.mark.gpu


def _chain(masses, light):
    m = Model()
    m.SetGravity(0., 0., -9.81)
    ids = [m.AddNode().SetPosition(1.3 * k, 0.2 * k, 0., 1., 0., 0., 0.).Build() for k in range(masses)]
    for k, n in enumerate(ids):
        m.AddMassElement(n, np.diag([20. + k] * 3 + [1. + 0.1 * k, 2., 3.]))
    base = m.AddPrescribedBC(ids[0])
    for a, b in zip(ids, ids[1:]):
        m.AddRigidJointConstraint([a, b])
    if light:
        f = m.AddNode().SetPosition(1.3 * masses, 0., 0.5, 1., 0., 0., 0.).Build()
        m.AddRigidJoint6DOFsTo3DOFs([ids[-1], f])
    return m, base


# unknowns 12 n (+ 6): 24, 30, 48, 54, 60, 66, 72, 96, 102, 120
@pytest.mark.parametrize("masses, light", [(2, False), (2, True), (4, False), (4, True), (5, False), (5, True),
                                           (6, False), (8, False), (8, True), (10, False)])
def test_bordered_solve_matches_oracle(masses, light):
    from openturbine_b200.runtime import Context
    from oracle.oracle_py import OracleModel
    m, base = _chain(masses, light)
    pm = m.pack()
    ctx = Context(0)
    mid = ctx.create_model(pm)
    orc = OracleModel(pm)
    assert ctx.info(mid).num_dofs == 12 * masses + (6 if light else 0)
    p = StepParameters(True, 8, 0.01, 0.5)
    for step in range(4):
        a = 0.05 * (step + 1)
        u = [0.02 * step, 0., 0.01 * step, np.cos(a / 2.), 0., np.sin(a / 2.), 0.]
        ctx.set_prescribed(mid, base, u)
        orc.set_prescribed(base, u)
        st, it = ctx.step([mid], p)
        assert (int(st[0]), int(it[0])) == orc.step(p)
        assert int(st[0]) == 0
    for f in ("q", "v"):
        a, b = ctx.state(mid, f), orc.state(f)
        assert np.abs(a - b).max() <= 1e-10 * max(1., np.abs(b).max())
    ctx.close()
