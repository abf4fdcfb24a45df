"""H*psi, the filter and the density on grids whose lengths have no compiled
kernel: unequal lengths, factors 7, 11, 13 and every prime factor the
register path takes, single primes, and a length it leaves to the generic
passes (2 * 2 * 61), against the oracle.  Bars: those of the other parity
tests (FP64 1e-12, FP32 2e-5 relative max-norm; 1e-4 after the filter).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

import pspw_oracle as O  # noqa: E402
from helpers import oracle_cell, relmax  # noqa: E402
from pspw import PREC_F32, PREC_F64, Cell, basis_gamma, synth  # noqa: E402

TOL64, TOL32, TOL32_FILTER = 1e-12, 2e-5, 1e-4

GRIDS = [
    (13, 14, 16), (16, 24, 18), (22, 21, 26), (28, 33, 20), (30, 32, 45), (36, 25, 49),
    (34, 24, 38), (46, 40, 34), (58, 62, 24), (74, 22, 74), (82, 20, 26), (24, 86, 94),
    (53, 24, 59), (20, 61, 16), (17, 18, 19), (72, 90, 24), (96, 75, 20), (64, 100, 12),
    (122, 24, 15), (24, 24, 22), (26, 26, 74),
]


def _cell(nr, nb):
    lat, pos = synth.si_diamond(1)
    b = basis_gamma(lat, 5.0, nr, [3], [pos[:3] + 0.1])
    pkg_a, wnl = synth.kb_form_factors(b, lat)
    b.update(pkg_a=pkg_a, wnl=wnl, lm_end=[4], na=[3])
    veff = synth.local_potential(b["nr"], lat, pos)
    psi = synth.wavefunctions(b, lat, nb, 7).astype(np.complex64).astype(complex)
    cell = Cell.from_arrays(b)
    cell.set_veff(veff)
    return b, cell, veff, np.asfortranarray(psi)


def _dev(cell, psi, prec):
    ngw, nb = psi.shape
    dt = torch.complex64 if prec == PREC_F32 else torch.complex128
    d_in = torch.from_numpy(np.ascontiguousarray(psi.T)).to(dt).cuda()
    d_out = torch.zeros_like(d_in)
    torch.cuda.synchronize()
    cell.apply_ham_block_dev(d_in, d_out, ngw, ngw, nb, prec)
    torch.cuda.synchronize()
    return d_out.cpu().numpy().T.astype(complex)


@pytest.mark.parametrize("nr", GRIDS)
def test_hpsi_and_filter(nr):
    b, cell, veff, psi = _cell(nr, 5)
    oc = oracle_cell(b)
    ref = O.apply_ham_block(oc, psi, veff)
    assert relmax(_dev(cell, psi, PREC_F64), ref) < TOL64
    assert relmax(_dev(cell, psi, PREC_F32), ref) < TOL32
    flt = O.chebyfilt(oc, psi, 4, 0.5, 8.0, veff)
    assert relmax(cell.chebyfilt(psi, 4, 0.5, 8.0, PREC_F64), flt) < TOL64
    assert relmax(cell.chebyfilt(psi, 4, 0.5, 8.0, PREC_F32), flt) < TOL32_FILTER


@pytest.mark.parametrize("nr", GRIDS[::2] + [(26, 26, 74), (38, 38, 38)])
def test_density(nr):
    b, cell, _, _ = _cell(nr, 1)
    lat, _ = synth.si_diamond(1)
    nx, ngw = 7, b["ngw"]
    psi = synth.wavefunctions(b, lat, nx, 9)
    focc = np.linspace(2.0, 0.1, nx)
    flat = np.concatenate([psi.T.reshape(-1), np.zeros(b["ngwx"])])
    rho, ekin = cell.eval_rho_psi(np.zeros(cell.nnr), flat, ngw, ngw, nx, focc, 1.0, b["omega"])
    ref, ekin_ref, _ = O.eval_rho_psi(oracle_cell(b), flat, ngw, ngw, nx, focc, 1.0, b["omega"],
                                      b["ngwx"])
    assert relmax(rho, ref) < TOL64
    assert abs(ekin - ekin_ref) < TOL64 * abs(ekin_ref)
