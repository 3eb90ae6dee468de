"""The batch's walk over elements by lines (marked gpu): solves whose element
counts leave a work item, a chunk of 64 or a CTA partly filled, against the same
solves alone through the operator; and that a solve's result is the same bit for
bit whatever the launch shape and whatever else the batch holds, in FP64 as in
FP32 and with blended and bounded solves beside it.

Tolerances of the batch tests: FP64 1e-12, FP32 1e-5, normalised per field."""
import numpy as np
import pytest

from conftest import normalized_error
from prandtl_b200 import cases
from prandtl_b200.batch import Batch
from prandtl_b200.ensemble import fixed_dt
from prandtl_b200.mesh import periodic_box

pytestmark = pytest.mark.gpu
EULER, NS = dict(quirks="fixed"), dict(quirks="fixed", parabolic=True, mu=0.01, R_gas=1.0)
WALLS = {False: [("slip_wall",), ("outflow",)], True: [("noslip_adiabatic", dict(heat_flux=0.0)), ("outflow",)]}
# elements of one work item: those of a warp where that fills 30 of its 32 lanes, else of a CTA
PER_ITEM = {(2, 1): 16, (2, 2): 10, (2, 3): 8, (2, 4): 6, (2, 5): 25,
            (3, 1): 8, (3, 2): 14, (3, 3): 2, (3, 4): 5, (3, 5): 7}


def solve(dim, count, order, phys, sides=None, amp=0.1):
    """A row of `count` elements."""
    mesh = periodic_box(dim, (count,) + (1,) * (dim - 1), order, 0.0, (0.5 * count,) + (0.5,) * (dim - 1), bcs=sides)
    u = cases.perturbed(mesh, cases.free_stream(mesh, p=1.5), amp=amp, seed=count + order)
    return mesh, u, dict(phys, dt=fixed_dt(mesh, u, 0.2), nsteps=3)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("parabolic", [False, True])
@pytest.mark.parametrize("dim,order", sorted(PER_ITEM))
def test_element_counts(dim, order, parabolic, precision):
    from prandtl_b200.operator import DGSEMOperator
    k = PER_ITEM[dim, order]
    phys = NS if parabolic else EULER
    solves = [solve(dim, c, order, phys) for c in sorted({1, k - 1, k, k + 1, 63, 64, 65})]
    b = Batch(precision, "LSRK45", arena_bytes=1 << 28)
    ids = b.add_many(solves)
    b.advance(3)
    for sid, (mesh, u, kw) in zip(ids, solves):
        op = DGSEMOperator(mesh, precision=precision, **phys)
        ref = op.Step(u.copy(), kw["dt"], scheme="LSRK45", nsteps=3)
        op.close()
        assert normalized_error(b.read(sid), ref, mesh.num_fields) <= (1e-12 if precision == "fp64" else 1e-5)
    b.close()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("parabolic", [False, True])
@pytest.mark.parametrize("dim,order", sorted(PER_ITEM))
def test_same_bits_alone_tuned_and_beside_others(dim, order, parabolic, precision):
    phys = NS if parabolic else EULER
    sides = [0, 1] + [None] * (2 * dim - 2)
    for amp in (0.003, 0.1, 0.4):
        mine = solve(dim, 21, order, phys, amp=amp)
        others = [solve(dim, 9, order, dict(phys, blending=True)), solve(dim, 70, order, phys, amp=0.3),
                  solve(dim, 5, order, dict(phys, bcs=WALLS[parabolic]), sides=sides)]
        states = []
        for beside, tune, graph in ((False, False, True), (False, True, True), (True, False, True), (True, True, True),
                                    (True, False, False)):
            b = Batch(precision, "LSRK45", arena_bytes=1 << 28, use_graph=graph)
            if beside:
                b.add_many(others[:2])
            sid = b.add_many([mine])[0]
            if tune:   # each of the three launch shapes in a step of its own
                b.tune_in_steps()
            b.advance(1)
            if beside:   # one more joins between the steps
                b.add_many(others[2:])
            b.advance(2)
            states.append(b.read(sid))
            b.close()
        for s in states[1:]:
            np.testing.assert_array_equal(s, states[0])


def test_class_info_covers_plain_and_featured_solves():
    """Solves of one class that launch apart are reported together: with a few
    blended elements beside many plain ones and the other way round."""
    info = []
    for few, many in ((dict(EULER, blending=True), EULER), (EULER, dict(EULER, blending=True))):
        b = Batch("fp32", "LSRK45", arena_bytes=1 << 28)
        b.add_many([solve(2, 4, 3, few)])
        b.tune(reps=2)
        v, alone, _ = b.class_info(2, 3, False)
        assert alone[v] == min(alone) > 0
        b.add_many([solve(2, 3000, 3, many)] * 4)
        b.tune(reps=2)
        v, both, lift = b.class_info(2, 3, False)
        assert min(both) > 1.5 * max(alone) and lift < 0
        b.close()
        info.append(both)
    assert max(info[0] + info[1]) < 4 * min(info[0] + info[1])
