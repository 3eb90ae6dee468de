"""The 2D line kernels above N = 1, on meshes large enough to run by lines (15,000
lines per direction), against the CPU oracle (marked gpu): sheared and
re-oriented elements, each boundary type alone, every physics on each branch of
the logarithmic means, and Runge-Kutta steps.

Tolerances as in the other parity tests: 1e-12 of each field's maximum for one
right-hand side, 1e-14 relative for the largest characteristic speed (the same
sums of the same state), 1e-12 for the blending coefficient, 1e-10 for steps."""
import os
import sys

import numpy as np
import pytest

from conftest import normalized_error
from prandtl_b200 import cases
from prandtl_b200.mesh import periodic_box, read_mesh

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(HERE, "golden"))
import make_golden  # noqa: E402

pytestmark = pytest.mark.gpu

N_LARGE = {2: (101, 53), 3: (61, 67), 4: (59, 53), 5: (53, 49)}
SHEAR = np.array([[1.0, 0.2], [0.1, 1.1]])
PHYS = [dict(), dict(blending=True), dict(parabolic=True), dict(parabolic=True, blending=True)]


def box(order, bcs=None):
    n = N_LARGE[order]
    mesh = periodic_box(2, n, order, 0.0, tuple(0.5 * c for c in n), affine=SHEAR, bcs=bcs)
    assert mesh.num_elements * mesh.Np >= 15000
    return mesh


def state(mesh, amp, seed):
    return cases.perturbed(mesh, cases.free_stream(mesh, rho=1.1, vel=[0.3, 0.2], p=2.0), amp=amp, seed=seed)


def compare(oracle_mod, mesh, u, quirks, **kw):
    from prandtl_b200.operator import DGSEMOperator
    okw = {k: int(v) if isinstance(v, bool) else v for k, v in kw.items()}
    ref = oracle_mod.Oracle(mesh, quirks=int(quirks == "fixed"), **okw).rhs(u, want_alpha=True)
    op = DGSEMOperator(mesh, quirks=quirks, **kw)
    d = op.Mult(u, np.empty_like(u))
    assert normalized_error(d, ref["dudt"], 4) <= 1e-12, (quirks, kw)
    assert op.GetMaxCharSpeed() == pytest.approx(ref["lambda_max"], rel=1e-14)
    if kw.get("blending"):
        np.testing.assert_allclose(op.alpha(), ref["alpha"], rtol=0, atol=1e-12)
    op.close()


@pytest.mark.parametrize("amp", [0.003, 0.1, 0.4])   # the means' short series, the long one, the logarithm
@pytest.mark.parametrize("order", [2, 3, 4, 5])
def test_sheared(oracle_mod, order, amp):
    mesh = box(order)
    u = state(mesh, amp, order)
    for phys in PHYS:
        for quirks in ("fixed", "reference"):
            compare(oracle_mod, mesh, u, quirks, **phys, **(make_golden.PHYS if phys.get("parabolic") else {}))


@pytest.mark.parametrize("order", [2, 3, 4, 5])
def test_reoriented_elements_and_boundaries(oracle_mod, order):
    """A Gmsh mesh of 96 x 80 quadrilaterals, frames turned element by element, in Hilbert order."""
    from test_mesh_io import CAVITY_EULER, CAVITY_NS, MESHES
    mesh = read_mesh(os.path.join(MESHES, "cavity_6x5.msh"), order, refine=4, hilbert=True)
    assert mesh.affine and mesh.num_elements * mesh.Np >= 15000
    u = state(mesh, 0.1, order)
    for phys in PHYS:
        for quirks in ("fixed", "reference"):
            kw = dict(bcs=CAVITY_NS, mu=0.01, R_gas=287.05) if phys.get("parabolic") else dict(bcs=CAVITY_EULER)
            compare(oracle_mod, mesh, u, quirks, **phys, **kw)


@pytest.mark.parametrize("blending", [False, True])
@pytest.mark.parametrize("order", [3, 4])
@pytest.mark.parametrize("parabolic,kind",
                         [(False, k) for k in ("state", "outflow", "slip_wall", "symmetry", "pressure_outflow", "riemann",
                                               "riemann_supersonic", "inflow_rv", "inflow_pttt")] +
                         [(True, k) for k in ("noslip_adiabatic", "noslip_isothermal", "outflow", "state",
                                              "pressure_outflow", "riemann", "inflow_rv")])
def test_each_boundary_type_alone(oracle_mod, parabolic, kind, order, blending):
    mesh = box(order, bcs=[0] * 4)
    kw = dict(parabolic=parabolic, blending=blending, bcs=[make_golden.bc_example(kind, 2)])
    if parabolic:
        kw.update(make_golden.PHYS)
    compare(oracle_mod, mesh, state(mesh, 0.2, order), "fixed", **kw)


@pytest.mark.parametrize("scheme", ["RK3SSP", "LSRK45"])
@pytest.mark.parametrize("order", [2, 3, 4, 5])
def test_steps(oracle_mod, order, scheme):
    from prandtl_b200.operator import DGSEMOperator
    for phys in PHYS:
        for sides in (None, [0, 1, 1, 0]):
            bcs = None if sides is None else [make_golden.bc_example("noslip_adiabatic" if phys.get("parabolic") else
                                                                     "slip_wall", 2), ("outflow",)]
            mesh = box(order, bcs=sides)
            u0 = state(mesh, 0.05, order)
            kw = dict(bcs=bcs, **(make_golden.PHYS if phys.get("parabolic") else {}))
            orc = oracle_mod.Oracle(mesh, quirks=1, **{k: int(v) for k, v in phys.items()}, **kw)
            dt = 0.1 * mesh.hmin / (orc.rhs(u0)["lambda_max"] * mesh.Np ** 2)
            ref = orc.step(u0, dt, scheme=0 if scheme == "RK3SSP" else 1, nsteps=2)
            op = DGSEMOperator(mesh, quirks="fixed", **phys, **kw)
            u = op.Step(u0.copy(), dt, scheme=scheme, nsteps=2)
            assert normalized_error(u, ref, 4) <= 1e-10, (phys, sides)
            op.close()
