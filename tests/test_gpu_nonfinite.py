"""Where a state has no right-hand side the operator returns NaN, as the oracle
does: negative pressures have no speed of sound and no entropy.  An infinite
energy gives an infinite characteristic speed (marked gpu).

The finite values beside them are held to the FP64 parity bound, 1e-12 of each
field's maximum over the finite entries."""
import numpy as np
import pytest

from prandtl_b200 import cases
from prandtl_b200.mesh import periodic_box

pytestmark = pytest.mark.gpu

# a small and a larger mesh each (2D: on both sides of the size from which lines run)
MESHES = [(2, (4, 3), 1), (2, (4, 3), 3), (2, (67, 61), 3), (2, (53, 59), 4), (3, (3, 2, 2), 1), (3, (3, 2, 2), 2),
          (3, (3, 2, 2), 3), (3, (2, 2, 3), 4), (3, (2, 2, 2), 5)]
PHYS = {"euler": dict(quirks="fixed"), "euler-reference": dict(quirks="reference"),
        "blended": dict(quirks="fixed", blending=True),
        "viscous": dict(quirks="fixed", parabolic=True, mu=0.01),
        "viscous-reference": dict(quirks="reference", parabolic=True, mu=0.01)}


def both(oracle_mod, mesh, u, **phys):
    from prandtl_b200.operator import DGSEMOperator
    kw = {k: int(v) if isinstance(v, bool) else v for k, v in phys.items()}
    kw["quirks"] = int(phys["quirks"] == "fixed")
    r = oracle_mod.Oracle(mesh, **kw).rhs(u)
    op = DGSEMOperator(mesh, **phys)
    d = op.Mult(u, np.empty_like(u))
    lam = op.GetMaxCharSpeed()
    op.close()
    return d.reshape(mesh.num_fields, -1), lam, r["dudt"].reshape(mesh.num_fields, -1), r["lambda_max"]


def same_where_finite(d, r):
    np.testing.assert_array_equal(np.isnan(d), np.isnan(r))
    for f in range(len(r)):
        ok = ~np.isnan(r[f])
        if ok.any():
            assert np.abs(d[f][ok] - r[f][ok]).max() <= 1e-12 * np.abs(r[f][ok]).max()


@pytest.mark.parametrize("dim,n,order", MESHES)
def test_reference_mode_at_low_density(oracle_mod, dim, n, order):
    """The reference's face flux reads velocities in the momentum slots: at
    rho = 0.1 the pressure it forms there is negative."""
    mesh = periodic_box(dim, n, order, 0.0, tuple(0.5 * c for c in n))
    u = cases.perturbed(mesh, cases.free_stream(mesh, rho=0.1, vel=[1.0, 0.5, 0.2][:dim], p=1.0), amp=0.01, seed=order)
    d, _, r, _ = both(oracle_mod, mesh, u, quirks="reference", parabolic=True, mu=0.01)
    assert np.isnan(r).any()
    same_where_finite(d, r)


@pytest.mark.parametrize("where", ["all", "one"])
@pytest.mark.parametrize("phys", sorted(PHYS))
@pytest.mark.parametrize("dim,n,order", MESHES)
def test_negative_pressure_of_whole_elements(oracle_mod, dim, n, order, phys, where):
    """Every surface flux of such an element needs its speed of sound; without
    blending (whose switch between two NaNs differs) the NaNs are the oracle's."""
    mesh = periodic_box(dim, n, order, 0.0, tuple(0.5 * c for c in n))
    u = cases.perturbed(mesh, cases.free_stream(mesh, p=1.5), amp=0.01, seed=order).reshape(mesh.num_fields, mesh.num_elements, -1)
    e = slice(None) if where == "all" else mesh.num_elements // 2
    kinetic = 0.5 * (u[1:-1, e] ** 2).sum(axis=0) / u[0, e]
    u[-1, e] = 2.0 * kinetic - u[-1, e]   # p -> -p
    d, _, r, _ = both(oracle_mod, mesh, u.reshape(-1), **PHYS[phys])
    at = np.unravel_index(np.arange(mesh.nodes_per_elem), (order + 1,) * dim)
    on_face = np.any([(x == 0) | (x == order) for x in at], axis=0)
    assert not np.isfinite(d.reshape(u.shape)[:, e][..., on_face]).all(axis=0).any()
    if where == "all" and phys != "blended":
        same_where_finite(d, r)


@pytest.mark.parametrize("phys", sorted(PHYS))
@pytest.mark.parametrize("dim,n,order", MESHES)
def test_infinite_energy(oracle_mod, dim, n, order, phys):
    mesh = periodic_box(dim, n, order, 0.0, tuple(0.5 * c for c in n))
    u = cases.perturbed(mesh, cases.free_stream(mesh, p=1.5), amp=0.01, seed=order)
    at = mesh.ndof // 2
    u.reshape(mesh.num_fields, -1)[-1, at] = np.inf
    d, lam, _, lam_ref = both(oracle_mod, mesh, u, **PHYS[phys])
    assert np.isinf(lam_ref) and np.isinf(lam)
    assert not np.isfinite(d[:, at]).all()
