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


def _forms(Nt, rng):
    """Rows of every form next to one another: subsets of the band with values of their own, the
    same out of order, an entry twice, entries just outside the band, 33 entries, none."""
    rows = []
    for t in range(Nt):
        near = [c for c in range(max(0, t - 6), min(Nt, t + 7)) if rng.random() < 0.6]
        row = {0: near, 1: near[::-1], 2: near + near[:1], 3: near + [min(t + 7, Nt - 1)], 4: [max(t - 7, 0)] + near,
               5: list(range(0, Nt, 3))[:33], 6: [], 7: near + [-1]}.get(int(rng.integers(0, 16)), near)
        rows.append([(int(c), float(rng.standard_normal())) for c in row])
    return rows


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("L,Nt,bs", [(2, 2, 3), (4, 14, 2), (6, 15, 1), (6, 16, 1), (6, 17, 2), (10, 63, 3), (6, 130, 1)])
def test_precon_row_forms(L, Nt, bs, dtype):
    """Against sums in complex128; an infinity or NaN in r reaches the rows that have
    an entry there and no other."""
    rng = np.random.default_rng(100 + Nt)
    rows = _forms(Nt, rng)
    r = (rng.standard_normal((bs, Nt, L * L)) + 1j * rng.standard_normal((bs, Nt, L * L)))
    r = torch.from_numpy(r).to(dtype)
    bad = Nt // 3
    r[-1, bad, 0], r[-1, bad, 1] = complex(float("inf"), 0), complex(0, float("nan"))
    dev = "cuda"
    csr = (
        torch.tensor(np.cumsum([0] + [len(q) for q in rows]), dtype=torch.int32, device=dev),
        torch.tensor([c for q in rows for c, _ in q], dtype=torch.int32, device=dev),
        torch.tensor([v for q in rows for _, v in q], dtype=torch.float64, device=dev),
    )
    z = ops.precon_apply(r.reshape(bs, -1).to(dev), csr, L).cpu().to(torch.complex128).numpy().reshape(bs, Nt, L * L)
    eps = np.finfo(np.float32 if dtype == torch.complex64 else np.float64).eps
    x = r.to(torch.complex128).numpy()
    for t, row in enumerate(rows):
        row = [(c, v) for c, v in row if 0 <= c < Nt]
        hit = any(c == bad for c, _ in row)
        for s in range(L * L):
            for b in range(bs):
                if b == bs - 1 and s < 2 and hit:
                    assert not np.isfinite(z[b, t, s])
                    continue
                exact = sum(v * x[b, c, s] for c, v in row)
                bound = sum(abs(v) * abs(x[b, c, s]) for c, v in row)
                # n rounded products and sums, and the value's own rounding
                assert abs(z[b, t, s] - exact) <= (len(row) + 3) * eps * bound + 1e-300
