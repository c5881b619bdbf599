"""The tensor-core stage at the edges of its tiles.

A tile holds 20, 6, 4, 2 or 2 whole cubes (1, 3, 5, 6 or 9 components), taken
two cubes at a time; meshes of 1 .. 9 cubes leave every remainder of a tile
and of a pair, with interior, wall, inflow / outflow and one-sided boundary
faces meeting in one pair.  The right-hand side is compared with the FP64
oracle.  Bound: the operands carry 16 (split-BF16) or 22 (split-TF32)
significant bits, 2^-16 and 2^-22 relative, times a cancellation of up to 3
between the volume and lift terms; the FP32 fluxes add a few 2^-24 of the
flux over the element's flux variation, here O(1)."""
import numpy as np
import pytest

import mojoxm_b200 as M
from tests import dgcases as C

CUBES = [(1, 1, 1), (2, 1, 1), (3, 1, 1), (1, 5, 1), (1, 1, 7), (3, 3, 1), (2, 2, 2)]
CASES = [("advection", 2, "mixed"), ("shallow_water", 3, "mixed"), ("euler_rusanov", 2, "mixed"),
         ("euler_rusanov", 3, "mixed"), ("euler_hlle", 4, "mixed"), ("euler_hllec", 5, "mixed"),
         ("maxwell", 4, "mixed"), ("mhd", 3, "mixed"), ("euler_hllec_fix", 3, "tf32"), ("maxwell", 4, "tf32"),
         ("mhd", 4, "tf32")]


@pytest.mark.gpu
@pytest.mark.parametrize("name,P,prec", CASES)
@pytest.mark.parametrize("bcs", ["periodic", "inflow_outflow", "mixed_lo_only"])
def test_rhs_on_partial_tiles(oracle_mod, name, P, prec, bcs):
    ph, L = C.PHYSICS_3D[name](), (1.0, 0.8, 0.6)
    for n in CUBES:
        s = M.Solver(M.Mesh(*n, *L, bcs=M.BoundaryConditions(*C.BCS_3D[bcs])), ph, P=P, precision=prec)
        o = oracle_mod.Oracle3D(P, n, L, M.physics_dict(ph), C.BCS_3D[bcs])
        q = C.random_state(s.shape, ph, seed=sum(n)).astype(np.float32).astype(np.float64)
        err = C.rel_err(s.rhs(q), o.rhs(q))
        s.close()
        assert err < (5e-5 if prec == "mixed" else 5e-6), (n, err)


@pytest.mark.gpu
@pytest.mark.parametrize("name,P,prec", [("euler_rusanov", 3, "mixed"), ("euler_hllec", 4, "mixed"),
                                         ("maxwell", 4, "tf32"), ("mhd", 5, "mixed")])
def test_steps_over_many_tiles(oracle_mod, name, P, prec):
    """More tiles than resident blocks, so that every block reuses its tile
    buffers (one or two of them) while its epilogue still reads the state.
    Three steps; the states differ by their FP32 rounding (2^-24 a stage, nine
    stages, random) and dt times the operator's error."""
    ph, n, L = C.PHYSICS_3D[name](), (15, 11, 13), (1.0, 0.8, 0.6)
    s = M.Solver(M.Mesh(*n, *L), ph, P=P, precision=prec)
    f = M.Solver(M.Mesh(*n, *L), ph, P=P, precision="f64")
    xyz = f.node_xyz()
    w = np.sin(2 * np.pi * (xyz / np.array(L)).sum(-1))
    q = C.random_state((1, 1, s.NC), ph, seed=3) * np.ones(f.shape)
    q *= 1.0 + 0.05 * w[..., None]
    q = q.astype(np.float32).astype(np.float64)
    for x in (s, f):
        x.upload_state(q)
        x.step_n(1e-4, 3)
    a, b = s.download_state().astype(np.float64), f.download_state()
    s.close()
    f.close()
    assert np.sqrt(((a - b) ** 2).sum() / (b ** 2).sum()) < 1e-6
