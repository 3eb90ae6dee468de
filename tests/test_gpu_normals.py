"""Meshes whose scaled normals differ from their elements' adjugate rows by more
than rounding and less than the 1e-9 that the fixed mode admits: the FP64 lifting
takes the normals it was given, on every path (marked gpu).

The same mesh handed over with per-node geometry runs the node-by-node kernels,
which read the normal of every face node; both are within the FP64 parity bound
of the exact sums, 1e-12 of each field's maximum.  Normals 5e-10 off change the
lifted gradients, and with them the result, by some 1e-10 of it."""
import copy
import ctypes as C

import numpy as np
import pytest

from conftest import normalized_error
from prandtl_b200 import cases
from prandtl_b200.mesh import periodic_box

pytestmark = pytest.mark.gpu
OFF = 1.0 + 5e-10
# 2D: a mesh above the size from which lines run, and a small one
MESHES = [(2, (7, 5), 3), (2, (67, 61), 3), (2, (53, 59), 4), (2, (3, 4), 1), (3, (3, 3, 2), 1), (3, (3, 3, 2), 2),
          (3, (3, 3, 2), 3), (3, (2, 2, 3), 4), (3, (2, 2, 2), 5)]
PHYS = dict(parabolic=True, mu=1.0, Pr=0.71, quirks="fixed")


def setup(dim, n, order):
    mesh = periodic_box(dim, n, order, 0.0, tuple(0.1 * c for c in n))
    mesh.face_nor = mesh.face_nor * OFF
    by_node = copy.copy(mesh)
    nd = (order + 1) ** dim
    by_node.node_adj = np.repeat(mesh.elem_adj[:, None], nd, axis=1)
    by_node.node_detj = np.repeat(mesh.elem_detj[:, None], nd, axis=1)
    by_node.face_node_nor = np.repeat(mesh.face_nor[:, None], nd // (order + 1), axis=1)
    u = cases.perturbed(mesh, cases.free_stream(mesh, p=1.5), amp=0.1, seed=order)
    return mesh, by_node, u


def mult(mesh, u):
    from prandtl_b200.operator import DGSEMOperator
    op = DGSEMOperator(mesh, **PHYS)
    d = op.Mult(u, np.empty_like(u))
    op.close()
    return d


@pytest.mark.parametrize("dim,n,order", MESHES)
def test_operator(dim, n, order):
    mesh, by_node, u = setup(dim, n, order)
    assert normalized_error(mult(mesh, u), mult(by_node, u), mesh.num_fields) <= 1e-12


@pytest.mark.parametrize("dim,n,order", MESHES)
def test_batch(dim, n, order):
    """One step, so short that the stages hardly differ: the state's change."""
    from prandtl_b200.batch import Batch
    from prandtl_b200.operator import DGSEMOperator
    mesh, by_node, u = setup(dim, n, order)
    dt = 0.05 * np.abs(u).max() / np.abs(mult(by_node, u)).max()
    b = Batch("fp64", "RK3SSP", arena_bytes=1 << 28)
    sid = b.add(mesh, u, dt=dt, nsteps=1, **PHYS)
    b.advance(1)
    got = b.read(sid)
    b.close()
    op = DGSEMOperator(by_node, **PHYS)
    ref = op.Step(u.copy(), dt, scheme="RK3SSP", nsteps=1)
    op.close()
    assert normalized_error(got, ref, mesh.num_fields) <= 1e-12


@pytest.mark.parametrize("dim,n,order", MESHES)
def test_noalloc(dim, n, order):
    import torch

    from prandtl_b200 import _lib
    from test_zz_no_alloc import _config, _device_desc
    mesh, by_node, u = setup(dim, n, order)
    L, keep = _lib.load(), []
    desc, cfg = _device_desc(torch, mesh, keep), _config(L, parabolic=1, mu=PHYS["mu"], Pr=PHYS["Pr"], quirks=1)
    ut = torch.from_numpy(u).cuda()
    out = torch.empty_like(ut)
    torch.cuda.synchronize()
    assert L.prandtl_rhs_noalloc(C.byref(desc), C.byref(cfg), C.c_void_p(ut.data_ptr()), C.c_void_p(out.data_ptr()),
                                 None) == _lib.PRANDTL_OK
    torch.cuda.synchronize()
    assert normalized_error(out.cpu().numpy(), mult(by_node, u), mesh.num_fields) <= 1e-12
