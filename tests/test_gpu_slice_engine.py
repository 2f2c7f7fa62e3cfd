"""The slice engine at lattice sides where its tiling changes: against the
numpy oracle where that is quick, else against the double-precision engine."""
import math

import numpy as np
import pytest
import torch

from oracle import qedf_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _case(L, Nt, bs, seed, level=0.1):
    """Angles [bs, Nt, 2 L^2] around the pi-flux saddle point and Gaussian vectors."""
    rng = np.random.default_rng(seed)
    y, x = np.meshgrid(np.arange(L), np.arange(L), indexing="ij")
    sg = (1 - 2 * ((x + y) % 2)) * (math.pi / 4)
    phi = np.stack([sg, -sg], axis=-1).reshape(1, 1, -1) + level * rng.standard_normal((bs, Nt, 2 * L * L))
    v = rng.standard_normal((bs, Nt * L * L)) + 1j * rng.standard_normal((bs, Nt * L * L))
    return phi.astype(np.float32).astype(np.float64), v


@pytest.mark.parametrize("L", [16, 32, 64])
def test_operator_rows_that_fill_a_warp(L):
    """Sides whose rows of tiles fill a power of two of lanes, over enough
    slices that the warps of a block drift apart (complex64 against the
    complex128 engine, whose kernel is the general one)."""
    from qed_fermion_b200 import ops
    phi, v = _case(L, 60, 2, seed=L)
    p64 = torch.tensor(phi.reshape(2, -1), device=DEV)
    x64 = torch.tensor(v, device=DEV)
    for op in ("m", "mh", "mhm"):
        want = ops.apply_operator(op, p64, x64, L, 0.1)
        for slab in (0, 13):
            got = ops.apply_operator(op, p64.float(), x64.to(torch.complex64), L, 0.1, slab=slab)
            assert ((got - want).abs().max() / want.abs().max()).item() < 1e-6


@pytest.mark.parametrize("L,Nt", [(16, 160), (32, 64)])
def test_mixed_solve_takes_the_double_solves_iterations(L, Nt):
    """A float engine that is wrong now and then still ends at the true
    residual, by reliable updates, but takes many more iterations."""
    from qed_fermion_b200.solver import PcgSolver, System
    phi, v = _case(L, Nt, 2, seed=3 * L)
    its = {}
    for mode in ("fp64", "mixed"):
        s = PcgSolver([System(L, Nt, 2)], mode=mode, rtol=1e-8, max_iter=20000, device=DEV)
        res = s.solve(torch.tensor(phi.reshape(2, -1), dtype=s.angle_dtype, device=DEV), torch.tensor(v, device=DEV))
        assert int(res.status.max()) == 0
        its[mode] = int(res.iters.max())
    assert its["mixed"] <= 1.2 * its["fp64"] + 10
