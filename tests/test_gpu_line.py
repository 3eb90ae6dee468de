"""The line form of the FP64 right-hand side (dgsem_line.cuh) against the CPU
oracle where its packing and its branches change: element counts that leave
lane groups and CTAs partly filled, neighbouring states on each side of the
logarithmic mean's branches, blended and plain elements side by side, and
boundary faces of every element position.

Tolerance: the FP64 parity bound of the other tests (1e-12 of each field's
maximum); the states are O(1) with O(1) variation, so no large terms cancel."""
import numpy as np
import pytest

from conftest import normalized_error
from prandtl_b200 import cases
from prandtl_b200.mesh import periodic_box

pytestmark = pytest.mark.gpu

# elements per direction: one warp's groups partly filled, one CTA and a bit
SHAPES = {2: [(2, 1), (3, 3), (13, 5)], 3: [(1, 1, 2), (3, 2, 1), (3, 3, 5)]}


def state(mesh, amp, seed):
    """Free stream with node-wise noise: amp 0.003 keeps every logarithmic mean
    on its short series, 0.1 reaches the long one, 0.4 the logarithm."""
    return cases.perturbed(mesh, cases.free_stream(mesh, p=1.5), amp=amp, seed=seed)


@pytest.mark.parametrize("amp", [0.003, 0.1, 0.4])
@pytest.mark.parametrize("order", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("dim", [2, 3])
def test_packing_and_mean_branches(oracle_mod, dim, order, amp):
    from prandtl_b200.operator import DGSEMOperator
    for k, n in enumerate(SHAPES[dim]):
        mesh = periodic_box(dim, n, order, 0.0, tuple(0.5 * c for c in n))
        u = state(mesh, amp, 10 * order + k)
        for phys in (dict(), dict(blending=True), dict(parabolic=True, mu=0.01)):
            for quirks in (("reference", "fixed") if not phys.get("parabolic") else ("fixed",)):
                r = oracle_mod.Oracle(mesh, quirks=int(quirks == "fixed"), **{a: (int(b) if isinstance(b, bool) else b)
                                                                            for a, b in phys.items()}).rhs(u)
                op = DGSEMOperator(mesh, quirks=quirks, **phys)
                d = op.Mult(u, np.empty_like(u))
                assert normalized_error(d, r["dudt"], mesh.num_fields) <= 1e-12, (n, phys, quirks)
                assert op.GetMaxCharSpeed() == pytest.approx(r["lambda_max"], rel=1e-14)
                op.close()


@pytest.mark.parametrize("blending", [False, True])
@pytest.mark.parametrize("order", [1, 3, 4])
@pytest.mark.parametrize("dim", [2, 3])
def test_boundaries(oracle_mod, dim, order, blending):
    """Walls and an outflow on every side, inviscid and viscous."""
    from prandtl_b200.operator import DGSEMOperator
    n = (3, 2) if dim == 2 else (2, 1, 3)
    for parabolic in (False, True):
        kinds = [("slip_wall",), ("outflow",)]
        if parabolic:
            kinds = [("noslip_adiabatic", dict(wall_vel=(0.1,) * dim, heat_flux=0.02)),
                     ("noslip_isothermal", dict(wall_vel=(0.0,) * dim, wall_T=1.6)), ("outflow",)]
        bcs = [k % len(kinds) for k in range(2 * dim)]
        mesh = periodic_box(dim, n, order, 0.0, tuple(0.5 * c for c in n), bcs=bcs)
        u = state(mesh, 0.1, order)
        phys = dict(parabolic=parabolic, blending=blending, mu=0.01, R_gas=1.0, bcs=kinds)
        r = oracle_mod.Oracle(mesh, quirks=1, **{a: (int(b) if isinstance(b, bool) else b) for a, b in phys.items()}).rhs(u)
        op = DGSEMOperator(mesh, quirks="fixed", **phys)
        d = op.Mult(u, np.empty_like(u))
        assert normalized_error(d, r["dudt"], mesh.num_fields) <= 1e-12
        op.close()


@pytest.mark.parametrize("scale", [1.0, 1.0 + 1e-6])
@pytest.mark.parametrize("order", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("dim", [2, 3])
def test_reference_mode_navier_stokes(oracle_mod, dim, order, scale):
    """The reference's own viscous terms by lines, on each branch of the means;
    with normals that are not the adjugate rows (scale) by the general form."""
    from prandtl_b200.operator import DGSEMOperator
    for k, (n, amp) in enumerate(zip(SHAPES[dim], (0.003, 0.1, 0.4))):
        mesh = periodic_box(dim, n, order, 0.0, tuple(0.5 * c for c in n))
        mesh.face_nor = mesh.face_nor * scale
        u = state(mesh, amp, 20 * order + k)
        r = oracle_mod.Oracle(mesh, quirks=0, parabolic=1, mu=0.01).rhs(u)
        op = DGSEMOperator(mesh, quirks="reference", parabolic=True, mu=0.01)
        d = op.Mult(u, np.empty_like(u))
        assert normalized_error(d, r["dudt"], mesh.num_fields) <= 1e-12, (n, amp)
        op.close()


# 2D meshes above the size from which lines run (15,000 lines per direction), odd
LARGE_2D = {2: (101, 53), 3: (61, 67), 4: (59, 53), 5: (53, 49)}


@pytest.mark.parametrize("walls", [False, True])
@pytest.mark.parametrize("order", [2, 3, 4, 5])
def test_large_2d(oracle_mod, order, walls):
    """2D by lines: partly filled last groups, each branch of the means, blending
    and boundaries."""
    from prandtl_b200.operator import DGSEMOperator
    n = LARGE_2D[order]
    kinds = [("slip_wall",), ("outflow",)] if walls else None
    mesh = periodic_box(2, n, order, 0.0, tuple(0.5 * c for c in n), bcs=[0, 1, 1, 0] if walls else None)
    for k, phys in enumerate((dict(), dict(blending=True), dict(parabolic=True, mu=0.01))):
        u = state(mesh, (0.003, 0.4, 0.1)[k], 30 * order + k)
        if walls and phys.get("parabolic"):
            kinds = [("noslip_adiabatic", dict(wall_vel=(0.1, 0.0), heat_flux=0.02)), ("outflow",)]
        r = oracle_mod.Oracle(mesh, quirks=1, bcs=kinds, **{a: (int(b) if isinstance(b, bool) else b)
                                                            for a, b in phys.items()}).rhs(u)
        op = DGSEMOperator(mesh, quirks="fixed", bcs=kinds, **phys)
        d = op.Mult(u, np.empty_like(u))
        assert normalized_error(d, r["dudt"], mesh.num_fields) <= 1e-12, phys
        op.close()
