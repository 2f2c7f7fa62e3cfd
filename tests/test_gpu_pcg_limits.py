"""The solver's longest lattices in tau, with as many right-hand sides as a solve takes."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("mode,Nt", [("fp64", 833), ("fp64", 807), ("mixed", 1539), ("mixed_f16", 1530), ("fp32", 1539)])
@pytest.mark.parametrize("nrhs", [3, 256])
def test_longest_tau_column(mode, Nt, nrhs):
    """2 x 2 lattices, whose blocks have the fewest threads and so the longest
    columns: solved to the true residual, formed by the complex128 operator."""
    from qed_fermion_b200 import ops
    from qed_fermion_b200.solver import PcgSolver, System
    L = 2
    g = torch.Generator(device=DEV).manual_seed(Nt)
    sign = torch.tensor([[1.0, -1.0], [-1.0, 1.0]], dtype=torch.float64, device=DEV) * (math.pi / 4)
    phi = torch.stack([sign, -sign], dim=-1) + 0.05 * torch.randn((nrhs, Nt, L, L, 2), dtype=torch.float64, device=DEV, generator=g)
    phi = phi.float().double().reshape(nrhs, -1)
    b = ops.apply_operator("mh", phi, torch.randn((nrhs, Nt * L * L), dtype=torch.complex128, device=DEV, generator=g), L, 0.1)
    rtol = 1e-4 if mode == "fp32" else 1e-9
    s = PcgSolver([System(L, Nt, nrhs)], mode=mode, rtol=rtol, max_iter=20000, device=DEV)
    res = s.solve(phi.to(s.angle_dtype), b.to(s.vec_dtype))
    assert int(res.status.max()) == 0
    r = b - ops.apply_operator("mhm", phi, res.x.view(nrhs, -1).to(torch.complex128), L, 0.1)
    # fp64's iterated residual and fp32's vectors carry roundings of the solve
    slack = 1e-3 if mode == "fp32" else 1e-11
    assert (torch.linalg.vector_norm(r, dim=1) / torch.linalg.vector_norm(b, dim=1)).max().item() < rtol * 1.01 + slack


@pytest.mark.parametrize("mode,Nt", [("fp64", 834), ("mixed", 1540)])
def test_longer_columns_are_refused(mode, Nt):
    from qed_fermion_b200 import _lib
    from qed_fermion_b200.solver import PcgSolver, System
    s = PcgSolver([System(2, Nt, 1)], mode=mode, device=DEV)
    with pytest.raises(_lib.QedfError) as e:
        s.solve(torch.zeros(s.angle_len, dtype=s.angle_dtype, device=DEV), torch.zeros(s.vec_len, dtype=s.vec_dtype, device=DEV))
    assert e.value.status == _lib.QEDF_ERR_SIZE
