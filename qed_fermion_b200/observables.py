"""Bond-bond correlators of the stochastic estimator on the GPU.

These are the observables the reference computes from the noise vectors eta
and G_eta = (M^dag M)^-1 M^dag eta of one gauge field
(``qed_fermion/stochastic_estimator.py``: ``T1`` :1393, ``T21`` :1447, ``T2``
:1504, ``T4`` :1561, ``Tvv`` :1612, ``get_bond_bond_per_b2`` :2594,
``bond_corr`` :2643), with the same names, arguments and return values.

Each ``T`` averages, over all noise pairs s < s' (``torch.combinations``
order) and over tau, the spatial correlation of two bond products,
    C(d) = (1 / Vs) sum_r a(r) b(r + d),
evaluated with 2-D FFTs over (y, x).  Because the inverse transform is linear,
the products of the transforms are summed over pairs and tau first and only
one inverse FFT per observable remains; the reference instead transforms back
per batch.  One kernel forms both fields of a pair and slice, transforms them
and adds their product into a double-precision k-space sum (``ops.bb_corr``; for
the sum of all four, from transforms that they share, ``ops.bb_corr_sum``).
On sides that it is not compiled for, or with ``fused=False``, pairs are
processed in chunks sized by ``chunk_bytes``: per chunk one kernel writes both
fields of every pair (``ops.bb_pair_fields``), cuFFT transforms them, and one
kernel adds the products of the transforms to the sum (``ops.bb_kspace_acc``).

Layouts as in the reference: eta, G_eta ``[Nrv, Ltau * Ly * Lx]`` (index
tau Vs + x + Lx y); boson ``[1, 2, Lx, Ly, Ltau]``.  Inputs must be CUDA
tensors; the transforms are cuFFT's (through torch).
"""
from __future__ import annotations

import torch

from . import ops


class BondBond:
    def __init__(self, Lx: int, Ltau: int, chunk_bytes: int = 1 << 30, fused: bool | None = None):
        self.Lx = self.Ly = Lx
        self.Ltau = Ltau
        self.chunk_bytes = int(chunk_bytes)
        # pair sums in one pass on the sides where that is faster; False: on none
        # (complex128, L = 48, 12 vectors, one correlator: 3.2 ms in two passes, 9.9 in
        # one with the kernel for any side)
        self.fused = fused is None or bool(fused)

    # ---- helpers ----------------------------------------------------------
    def _chunk(self, ec, n_arrays=4):
        per = ec[0].numel() * ec.element_size() * n_arrays
        return max(1, self.chunk_bytes // max(1, per))

    def _pair_mean(self, kind, eta, G_eta, boson):
        return self._mean_of(kind, self._pair_inputs(eta, G_eta, boson))

    def _mean_of(self, kind, inputs):
        """mean over pairs s < t and tau of ifft2(a_st) * fft2(b_st), transformed
        back to real space; a_st, b_st are the fields of correlator ``kind``."""
        e, g, ep, pairs, S = inputs
        dt, nrv, Vs = e.dtype, e.shape[0], self.Lx * self.Ly
        one = self.fused and ops.bb_corr_lines(self.Lx, dt)
        if one and ops.bb_corr(kind, e, g, ep, pairs[:, 0].contiguous(), pairs[:, 1].contiguous(), self.Lx, S):
            S = S.view(self.Ly, self.Lx) / (Vs * Vs)
            return (torch.fft.ifft2(S, norm="forward") / (len(pairs) * self.Ltau)).to(dt)
        chunk = min(65535, self._chunk(e.reshape(nrv, self.Ltau, self.Ly, self.Lx)), len(pairs))
        fa = torch.empty((chunk, self.Ltau, self.Ly, self.Lx), dtype=dt, device=e.device)
        fb = torch.empty_like(fa)
        for ch in pairs.split(chunk):
            n = len(ch)
            a, b = fa[:n], fb[:n]
            ops.bb_pair_fields(kind, e, g, ep, ch[:, 0].contiguous(), ch[:, 1].contiguous(), self.Lx, a, b)
            # unnormalised transforms; the 1 / Vs of each is applied to S once
            ops.bb_kspace_acc(torch.fft.ifft2(a, norm="forward"), torch.fft.fft2(b, norm="backward"), S)
        S = S.view(self.Ly, self.Lx) / (Vs * Vs)
        return (torch.fft.ifft2(S, norm="forward") / (len(pairs) * self.Ltau)).to(dt)

    def _pair_inputs(self, eta, G_eta, boson):
        """The kernels' inputs, the noise pairs and the zeroed k-space sum."""
        nrv = eta.shape[0]
        if nrv < 2:
            raise RuntimeError("bond-bond correlators need at least two noise vectors")
        e, g, ep = self._inputs(eta, G_eta, boson)
        pairs = torch.combinations(torch.arange(nrv, device=e.device), r=2, with_replacement=False).to(torch.int32)
        return e, g, ep, pairs, torch.zeros(self.Lx * self.Ly, dtype=torch.complex128, device=e.device)

    def _inputs(self, eta, G_eta, boson):
        """eta, G_eta as contiguous [Nrv, N] of one dtype and e^{i phi_x} [Ltau, Ly, Lx]."""
        dt = eta.dtype
        nrv = eta.shape[0]
        e = eta.resolve_conj().reshape(nrv, -1).contiguous()
        g = G_eta.to(dt).resolve_conj().reshape(nrv, -1).contiguous()
        ph = boson.permute(0, 1, 4, 3, 2)[0, 0].to(e.real.dtype)
        return e, g, torch.exp(1j * ph).to(dt).contiguous()

    def _diag(self, eta, G_eta, boson):
        """The three short-distance terms as means (kernel ``bb_diag``)."""
        e, g, ep = self._inputs(eta, G_eta, boson)
        return ops.bb_diag(e, g, ep, self.Lx) / e.numel()

    # ---- the correlators ----------------------------------------------------
    def T1(self, eta, G_eta, boson):
        out = -self._pair_mean("T1", eta, G_eta, boson)
        out[0, -1] += self._diag(eta, G_eta, boson)[0].to(out.dtype)
        return out

    def T21(self, eta, G_eta, boson):
        out = -self._pair_mean("T21", eta, G_eta, boson)
        out[0, 0] += self._diag(eta, G_eta, boson)[1].to(out.dtype)
        return out

    @staticmethod
    def _reflect(a):
        """a at -d: element (-dy mod Ly, -dx mod Lx) at (dy, dx)"""
        return torch.roll(torch.flip(a, dims=(-2, -1)), shifts=(1, 1), dims=(-2, -1))

    def T2(self, eta, G_eta, boson):
        """T2's two pair fields are T21's with a and b exchanged:
        (ec_s g_t(r+x) + ec_t g_s(r+x)) e/2 is T21's b, and (g_s ec_t(r+x) +
        g_t ec_s(r+x)) e*/2 is T21's a.  Its pair correlation is therefore T21's
        at -d, and both add the same term at d = 0, so T2 is T21 reflected."""
        return self._reflect(self.T21(eta, G_eta, boson))

    def T2_direct(self, eta, G_eta, boson):
        """T2 from its own pair fields (the reference's computation)."""
        out = -self._pair_mean("T2", eta, G_eta, boson)
        out[0, 0] += self._diag(eta, G_eta, boson)[1].to(out.dtype)
        return out

    def T4(self, eta, G_eta, boson):
        out = -self._pair_mean("T4", eta, G_eta, boson)
        out[0, 1] += self._diag(eta, G_eta, boson)[2].to(out.dtype)
        return out

    def Tvv(self, eta, G_eta, boson):
        """The current-current correlation and the mean current: each vector's
        field v (kernel ``bb_vfield``, which also sums it), the products of its
        transforms summed in k-space (``bb_kspace_acc``), one inverse FFT."""
        e, g, ep = self._inputs(eta, G_eta, boson)
        nrv = e.shape[0]
        Vs = self.Lx * self.Ly
        S = torch.zeros(Vs, dtype=torch.complex128, device=e.device)
        Tv = torch.zeros(Vs, dtype=torch.complex128, device=e.device)
        per = max(1, self.chunk_bytes // max(1, 3 * e[0].numel() * e.element_size()))
        v = torch.empty((min(per, nrv), self.Ltau, self.Ly, self.Lx), dtype=e.dtype, device=e.device)
        for lo in range(0, nrv, per):
            n = min(per, nrv - lo)
            vb = v[:n]
            ops.bb_vfield(e[lo:lo + n], g[lo:lo + n], ep, self.Lx, vb, Tv)
            # the reference's ifft2(v, "backward") * fft2(v, "forward"): unnormalised
            # transforms here, their two 1 / Vs applied to the sum once
            ops.bb_kspace_acc(torch.fft.ifft2(vb, norm="forward"), torch.fft.fft2(vb, norm="backward"), S)
        S = S.view(self.Ly, self.Lx) / (Vs * Vs)
        dt = eta.dtype
        return ((torch.fft.ifft2(S, norm="forward") / (nrv * self.Ltau)).to(dt),
                (Tv.view(self.Ly, self.Lx) / (nrv * self.Ltau)).to(dt))

    def _T_sum(self, eta, G_eta, boson):
        """T1 + T21 + T2 + T4.  One pass over the pairs where its kernel is
        compiled for the side (and ``fused`` is not False): the four share their fields' transforms (20
        vectors, L = 30, Ltau = 300, complex128: 3.6 -> 1.57 ms; L = 48, 12
        vectors, complex64: 5.2 -> 1.5)."""
        e, g, ep, pairs, S = inputs = self._pair_inputs(eta, G_eta, boson)
        dt, Vs = e.dtype, self.Lx * self.Ly
        if self.fused and ops.bb_corr_sum(e, g, ep, pairs[:, 0].contiguous(), pairs[:, 1].contiguous(), self.Lx, S):
            S = S.view(self.Ly, self.Lx) / (Vs * Vs)
            out = -(torch.fft.ifft2(S, norm="forward") / (len(pairs) * self.Ltau)).to(dt)
        else:
            t21 = self._mean_of("T21", inputs)
            out = -(self._mean_of("T1", (*inputs[:-1], torch.zeros_like(S))) + t21 + self._reflect(t21)
                    + self._mean_of("T4", (*inputs[:-1], torch.zeros_like(S))))
        diag = (ops.bb_diag(e, g, ep, self.Lx) / e.numel()).to(dt)
        out[0, -1] += diag[0]
        out[0, 0] += 2 * diag[1]  # T21's and T2's
        out[0, 1] += diag[2]
        return out

    def get_bond_bond_per_b2(self, eta, G_eta, boson):
        """BB0_r, BB_r, B_r and BB_k (real parts; BB_k in ascending momentum order)."""
        T = self._T_sum(eta, G_eta, boson)
        Tvv, Tv = self.Tvv(eta, G_eta, boson)
        BB_r = T * 2 + Tvv * 4
        BB_k = torch.fft.ifft2(BB_r, norm="forward")
        BB_k = torch.roll(BB_k, shifts=(self.Ly // 2, self.Lx // 2), dims=(-2, -1))
        return {"BB0_r": (T * 2).real, "BB_r": BB_r.real, "B_r": Tv.real, "BB_k": BB_k.real}

    def bond_corr(self, BB_r_mean, B_r_mean):
        """BB_r minus the disconnected part 4 (B_r correlated with itself)."""
        vF_neg = torch.fft.ifftn(B_r_mean, (self.Ly, self.Lx), norm="backward")
        vF = torch.fft.fftn(B_r_mean, (self.Ly, self.Lx), norm="forward")
        return BB_r_mean - 4 * torch.fft.ifftn(vF_neg * vF, (self.Ly, self.Lx), norm="forward")
