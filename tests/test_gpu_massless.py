"""A beam whose sections have stiffness but no mass: eta, the offset of the mass
centre, is a quotient by the mass (calculate_quadrature_point_values.hpp), so a
step of such a beam is refused as singular, as a beam system and as the element
of a dense or condensed model."""
import numpy as np
import pytest

from openturbine_b200 import workloads as W
from openturbine_b200.model import BeamSection, GaussLegendreQuadrature, Model, StepParameters
from tests.workloads_ref import COMPOSITE_STIFF, chain_beam

pytestmark = pytest.mark.gpu


def _beam(nodes):
    m = Model()
    ids = [m.AddNode().SetElemLocation(s).SetPosition(20. * s, 0., 0., 1., 0., 0., 0.).Build()
           for s in W.gll_node_locations(nodes)]
    m.AddBeamElement(ids, [BeamSection(x, np.zeros((6, 6)), W.BASE_STIFFNESS) for x in (0., 1.)],
                     GaussLegendreQuadrature(nodes + 1))
    m.AddFixedBC(ids[0])
    return m


def _pair(order):
    m = Model()
    secs = [BeamSection(x, np.zeros((6, 6)), COMPOSITE_STIFF) for x in (0., 1.)]
    rule = [[x, w] for x, w in zip(*np.polynomial.legendre.leggauss(order + 2))]
    a, _ = chain_beam(m, 1, order, 10., [1., 0., 0., 0.], secs, rule)
    b, _ = chain_beam(m, 1, order, 10., [1., 0., 0., 0.], secs, rule, origin=(10., 0., 0.))
    m.AddFixedBC(a[0])
    m.AddRigidJointConstraint([a[-1], b[0]])
    return m


@pytest.mark.parametrize("kind, size, precision", [("beam", 2, 0), ("beam", 9, 0), ("beam", 9, 1),
                                                   ("dense", 4, 0), ("condensed", 12, 0)])
def test_massless_sections_are_refused(kind, size, precision):
    from openturbine_b200.runtime import Context
    m = _beam(size) if kind == "beam" else _pair(size)
    ctx = Context(0)
    mid = ctx.create_model(m.pack())
    assert (ctx.info(mid).condensed_dofs > 0) == (kind == "condensed")
    fx = np.zeros((m.NumNodes(), 6))
    fx[-1, 2] = 10.
    ctx.set_node_fx(mid, fx)
    st, _ = ctx.step([mid], StepParameters(True, 8, 0.01, 0.9, precision=precision))
    assert int(st[0]) == -6
    ctx.close()
