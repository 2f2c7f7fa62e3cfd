"""The tau-space preconditioner's row forms: shifted middle rows and rows run over their CSR entries."""

import numpy as np
import pytest
import torch

from qed_fermion_b200 import ops

pytestmark = pytest.mark.gpu


def _matrix(Nt, rng):
    """A 13-tap band with rows that differ from it: by a value, a column, their length; one row is dense."""
    taps = rng.standard_normal(13)
    rows = [[(t + d, taps[d + 6]) for d in range(-6, 7) if 0 <= t + d < Nt] for t in range(Nt)]
    if Nt > 13:
        rows[7][4] = (rows[7][4][0], 0.5)
        rows[9] = []
        rows[Nt - 8] = [(c, 0.25 * (c + 1)) for c in range(Nt)]
        rows[10][3] = (Nt + 2, 3.0)  # outside the matrix: does not count
    return rows


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("L,Nt,bs", [(2, 1, 1), (4, 7, 2), (6, 13, 1), (10, 31, 3), (6, 64, 1), (8, 65, 2), (10, 129, 1)])
def test_precon_rows(L, Nt, bs, dtype):
    rng = np.random.default_rng(Nt)
    rows = _matrix(Nt, rng)
    r = (rng.standard_normal((bs, Nt, L * L)) + 1j * rng.standard_normal((bs, Nt, L * L)))
    r = torch.from_numpy(r).to(dtype)
    exact, bound = np.zeros((bs, Nt, L * L), complex), np.zeros((bs, Nt, L * L))
    for t, row in enumerate(rows):
        for c, v in row:
            if c < Nt:
                x = r[:, c].to(torch.complex128).numpy()
                exact[:, t] += v * x
                bound[:, t] += abs(v) * np.abs(x)
    dev = "cuda"
    csr = (
        torch.tensor(np.cumsum([0] + [len(q) for q in rows]), dtype=torch.int32, device=dev),
        torch.tensor([c for q in rows for c, _ in q], dtype=torch.int32, device=dev),
        torch.tensor([v for q in rows for _, v in q], dtype=torch.float64, device=dev),
    )
    z = ops.precon_apply(r.reshape(bs, -1).to(dev), csr, L).cpu().to(torch.complex128).numpy().reshape(exact.shape)
    eps = np.finfo(np.float32 if dtype == torch.complex64 else np.float64).eps
    # n rounded products and sums, and the value's own rounding
    assert np.all(np.abs(z - exact) <= (Nt + 3) * eps * bound + 1e-300)
