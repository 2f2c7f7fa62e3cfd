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


@pytest.mark.parametrize("prec", ["c64", "c128"])
@pytest.mark.parametrize("L,Nt,bs", [(2, 5, 2000), (4, 7, 1500), (18, 5, 700), (28, 3, 301)])
def test_runs_across_right_hand_sides_match_slabs(L, Nt, bs, prec):
    """More slices than the GPU holds blocks: a block's run of slices ends one
    right-hand side and begins the next.  The same arithmetic per slice as with
    one slab per block, so the results are equal bit for bit."""
    from qed_fermion_b200 import ops
    cdt, rdt = (torch.complex64, torch.float32) if prec == "c64" else (torch.complex128, torch.float64)
    g = torch.Generator(device=DEV).manual_seed(L)
    phi = torch.randn((bs, 2 * L * L * Nt), device=DEV, dtype=rdt, generator=g)
    x = torch.randn((bs, L * L * Nt), device=DEV, dtype=cdt, generator=g)
    for op in ("m", "mh", "mhm"):
        assert torch.equal(ops.apply_operator(op, phi, x, L, 0.1), ops.apply_operator(op, phi, x, L, 0.1, slab=Nt))
    assert torch.equal(ops.fermion_force(phi, x, L, 0.1), ops.fermion_force(phi, x, L, 0.1, slab=2))


@pytest.mark.parametrize("L,by", [(20, 2), (20, 4), (24, 2), (24, 4), (24, 6), (52, 4), (54, 6), (56, 4), (60, 4), (60, 6)])
@pytest.mark.parametrize("prec,tol", [("c64", 1e-6), ("c128", 1e-13)])
def test_tile_heights_match_oracle(L, by, prec, tol):
    """Every tile height that a side allows, the operators and the force."""
    from qed_fermion_b200 import ops
    phi, v = _case(L, 5, 2, seed=L + by)
    w = v.reshape(2, 5, L * L)
    cdt, rdt = (torch.complex64, torch.float32) if prec == "c64" else (torch.complex128, torch.float64)
    p, x = torch.tensor(phi.reshape(2, -1), dtype=rdt, device=DEV), torch.tensor(v, dtype=cdt, device=DEV)
    for op, f in (("m", O.m_vec), ("mh", O.mh_vec), ("mhm", O.mhm_vec)):
        want = f(phi, w, L, 0.1).reshape(2, -1)
        got = ops.apply_operator(op, p, x, L, 0.1, by=by).cpu().numpy()
        assert np.abs(got - want).max() < tol * np.abs(want).max()
    want = O.force_f_from_xi(phi, w, L, 0.1).reshape(2, -1)
    got = ops.fermion_force(p, x, L, 0.1, by=by).cpu().numpy()
    # the force's tolerances of the parity tests
    assert np.abs(got - want).max() < (2e-5 if prec == "c64" else 1e-12) * np.abs(want).max()


@pytest.mark.parametrize("L,Nt,nrhs,mode", [(38, 300, 3, "mixed"), (42, 340, 2, "mixed_f16"), (48, 251, 2, "mixed"),
                                            (66, 260, 1, "mixed"), (66, 670, 1, "mixed")])
def test_wide_elementwise_units(L, Nt, nrhs, mode):
    """Shapes whose 16-site units take two rounds and 32-site ones a single
    round, with ragged last units: the solver's choice and both widths' solutions
    meet the true residual, formed by the complex128 operator, in the double-
    precision solves' iterations."""
    from qed_fermion_b200 import ops
    from qed_fermion_b200.solver import PcgSolver, System
    phi, v = _case(L, Nt, nrhs, seed=L + Nt, level=0.05)
    p = torch.tensor(phi.reshape(nrhs, -1), device=DEV)
    R = torch.tensor(v, device=DEV)
    b = ops.apply_operator("mh", p, R, L, 0.1)
    its = []
    for chunk in (0, 16):
        s = PcgSolver([System(L, Nt, nrhs)], mode=mode, rtol=1e-10, max_iter=20000, chunk=chunk, device=DEV)
        res = s.solve(p.float(), b)
        assert int(res.status.max()) == 0
        x = res.x.view(nrhs, -1)
        r = b - ops.apply_operator("mhm", p, x, L, 0.1)
        assert (torch.linalg.vector_norm(r, dim=1) / torch.linalg.vector_norm(b, dim=1)).max().item() < 1.01e-10
        its.append(int(res.iters.max()))
    # sums in another order move the last iteration by one or two in a hundred
    assert abs(its[0] - its[1]) <= 2 + 0.02 * its[1]
