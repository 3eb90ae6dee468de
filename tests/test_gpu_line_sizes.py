"""Right-hand sides on both sides of the mesh sizes from which kernels by lines
take over from the general form (marked gpu): 2D reference-mode Navier-Stokes and
viscous walls in FP64 against the oracle at 1e-12 of each field's maximum."""
import numpy as np
import pytest

from conftest import normalized_error
from prandtl_b200 import cases
from prandtl_b200.mesh import periodic_box

pytestmark = pytest.mark.gpu

# lines per direction just below and above 13,000 (N=3) and 10,000
REFERENCE = [(1, (3, 2)), (2, (5, 4)), (3, (57, 57)), (3, (50, 65)), (4, (40, 49)), (4, (40, 51)), (5, (40, 41)), (5, (40, 43))]
# ... below 15,000, between and above 21,000
WALLS = [(2, (70, 71)), (2, (70, 73)), (3, (59, 63)), (3, (63, 67)), (3, (72, 73)), (4, (61, 67)), (4, (65, 65)),
         (5, (50, 59)), (5, (59, 60))]


def state(mesh, order):
    return cases.perturbed(mesh, cases.free_stream(mesh, p=1.5), amp=0.1, seed=order)


@pytest.mark.parametrize("order,n", REFERENCE)
def test_reference_mode(oracle_mod, order, n):
    from prandtl_b200.operator import DGSEMOperator
    mesh = periodic_box(2, n, order, 0.0, tuple(0.5 * c for c in n), affine=np.array([[1.0, 0.2], [0.1, 1.1]]))
    u = state(mesh, order)
    r = oracle_mod.Oracle(mesh, quirks=0, parabolic=1, mu=0.01).rhs(u)
    op = DGSEMOperator(mesh, quirks="reference", parabolic=True, mu=0.01)
    assert normalized_error(op.Mult(u, np.empty_like(u)), r["dudt"], 4) <= 1e-12
    assert op.GetMaxCharSpeed() == pytest.approx(r["lambda_max"], rel=1e-14)
    op.close()


@pytest.mark.parametrize("blending", [False, True])
@pytest.mark.parametrize("order,n", WALLS)
def test_walls(oracle_mod, order, n, blending):
    from prandtl_b200.operator import DGSEMOperator
    bcs = [("noslip_adiabatic", dict(wall_vel=(0.1, 0.0), heat_flux=0.02)), ("noslip_isothermal", dict(wall_T=1.6))]
    mesh = periodic_box(2, n, order, 0.0, tuple(0.5 * c for c in n), bcs=[None, None, 0, 1])
    u = state(mesh, order)
    kw = dict(mu=0.01, R_gas=1.0, bcs=bcs)
    r = oracle_mod.Oracle(mesh, quirks=1, parabolic=1, blending=int(blending), **kw).rhs(u)
    op = DGSEMOperator(mesh, quirks="fixed", parabolic=True, blending=blending, **kw)
    assert normalized_error(op.Mult(u, np.empty_like(u)), r["dudt"], 4) <= 1e-12
    op.close()


# FP32-bulk lifting: just below and above 21,000 lines (2D N=5: 10,000), and N <= 2 by lines;
# with walls 70,000 (N=2 and 2D N=5: 20,000)
FP32 = [(2, 1, (185, 189)), (2, 1, (187, 189)), (2, 2, (80, 83)), (2, 2, (80, 84)), (2, 3, (130, 134)), (2, 3, (130, 135)),
        (2, 5, (55, 60)), (2, 5, (55, 61)), (3, 2, (13, 13, 13)), (3, 2, (13, 13, 14)), (3, 3, (16, 16, 17)), (3, 3, (16, 17, 17)),
        (2, 2, (9, 7)), (2, 3, (70, 74)), (2, 3, (71, 75)), (2, 4, (60, 69)), (2, 4, (60, 71)), (2, 5, (40, 41)),
        (2, 5, (40, 43)), (3, 1, (3, 3, 2)), (3, 2, (3, 3, 2)), (3, 3, (10, 11, 11)), (3, 3, (11, 11, 11)),
        (3, 4, (9, 9, 10)), (3, 4, (9, 10, 10)), (3, 5, (8, 8, 9)), (3, 5, (8, 9, 9))]


@pytest.mark.parametrize("walls", [False, True])
@pytest.mark.parametrize("dim,order,n", FP32)
def test_fp32_lifting(dim, order, n, walls):
    """Within the FP32-bulk form's bound of the FP64 right-hand side, 2e-3 in relative L2."""
    from prandtl_b200.operator import DGSEMOperator
    from test_gpu_fp32 import rel_l2
    kw = dict(mu=0.01, R_gas=1.0, parabolic=True, quirks="fixed")
    if walls:
        kw["bcs"] = [("noslip_adiabatic", dict(wall_vel=(0.1,) + (0.0,) * (dim - 1), heat_flux=0.02)), ("outflow",)]
    mesh = periodic_box(dim, n, order, 0.0, tuple(0.5 * c for c in n), bcs=[None] * (2 * dim - 2) + [0, 1] if walls else None)
    u = cases.perturbed(mesh, cases.free_stream(mesh, p=1.5), amp=0.1, seed=order)
    out = []
    for precision in ("fp64", "fp32"):
        op = DGSEMOperator(mesh, precision=precision, **kw)
        out.append(op.Mult(u, np.empty_like(u)))
        op.close()
    assert max(rel_l2(out[1], out[0], mesh.num_fields)) <= 2e-3
