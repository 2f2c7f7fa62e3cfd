"""How the operators' and the force's slices are cut into runs and tiled, at the edges of the rules."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
DT = {"c64": (torch.complex64, torch.float32), "c128": (torch.complex128, torch.float64)}


def _inputs(L, Nt, bs, prec):
    cdt, rdt = DT[prec]
    g = torch.Generator(device=DEV).manual_seed(L + Nt)
    return (torch.randn((bs, 2 * L * L * Nt), device=DEV, dtype=rdt, generator=g),
            torch.randn((bs, L * L * Nt), device=DEV, dtype=cdt, generator=g))


@pytest.mark.parametrize("prec,tol", [("c64", 1e-6), ("c128", 1e-13)])
@pytest.mark.parametrize("L,Nt", [(2, 2), (4, 3), (18, 5)])
def test_runs_of_every_length(L, Nt, prec, tol):
    """M^dag (and M, M^dag M) over runs from one slice to all of tau, with the
    antiperiodic wrap at either end: the same slices bit for bit, and the oracle's."""
    from oracle import qedf_oracle as O
    from qed_fermion_b200 import ops
    phi, x = _inputs(L, Nt, 2, prec)
    for op, f in (("m", O.m_vec), ("mh", O.mh_vec), ("mhm", O.mhm_vec)):
        z = [ops.apply_operator(op, phi, x, L, 0.1, slab=s) for s in range(Nt + 1)]
        assert all(torch.equal(z[0], w) for w in z[1:])
        want = f(phi.double().cpu().numpy().reshape(2, Nt, -1), x.to(torch.complex128).cpu().numpy().reshape(2, Nt, -1), L, 0.1)
        want = torch.from_numpy(want.reshape(2, -1))
        assert (z[0].cpu().to(torch.complex128) - want).abs().max() < tol * want.abs().max()


@pytest.mark.parametrize("L,prec", [(10, "c64"), (26, "c128"), (28, "c64"), (48, "c64")])
@pytest.mark.parametrize("num,den,more", [(3, 1, 1), (7, 2, 0), (4, 1, -1), (9, 2, 0), (9, 2, 1), (6, 1, 3)])
def test_a_few_more_slices_than_block_places(L, prec, num, den, more):
    """Slices a little above a multiple of the SMs, where runs are of two slices
    each: the results of one slice to a block, bit for bit."""
    from qed_fermion_b200 import ops
    W = torch.cuda.get_device_properties(0).multi_processor_count * num // den + more
    for bs in (1, 3):
        phi, x = _inputs(L, W // bs, bs, prec)
        for op in ("m", "mh", "mhm"):
            assert torch.equal(ops.apply_operator(op, phi, x, L, 0.1), ops.apply_operator(op, phi, x, L, 0.1, slab=1))
        assert torch.equal(ops.fermion_force(phi, x, L, 0.1), ops.fermion_force(phi, x, L, 0.1, slab=1))


@pytest.mark.parametrize("L,prec", [(12, "c64"), (18, "c64"), (30, "c64"), (32, "c64"), (36, "c64"), (16, "c128"), (20, "c128"),
                                    (28, "c128"), (32, "c128"), (36, "c128")])
@pytest.mark.parametrize("bs", [1, 2, 8])
def test_choice_is_one_of_the_tile_heights(L, prec, bs):
    """Sides where the tile height follows the number of slices: the operators'
    results are those of a height that can be asked for, the force's of all."""
    from qed_fermion_b200 import ops
    phi, x = _inputs(L, 8 * L, bs, prec)
    heights = [h for h in (2, 4, 6) if L % h == 0]
    for op in ("m", "mh", "mhm"):
        z = ops.apply_operator(op, phi, x, L, 0.1)
        assert any(torch.equal(z, ops.apply_operator(op, phi, x, L, 0.1, by=h)) for h in heights)
    F = ops.fermion_force(phi, x, L, 0.1)
    # (one site's terms are added in the order of its own tile)
    for h in heights:
        G = ops.fermion_force(phi, x, L, 0.1, by=h)
        assert (F - G).abs().max() <= (1e-5 if prec == "c64" else 1e-13) * F.abs().max()
