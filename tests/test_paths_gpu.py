"""Paths of H*psi, the filter and the density that the usual cells do not take:

- planes around the sizes where the register FFT stops fitting in a block's
  shared memory, in FP32, in FP64 and for the FP64 density with its accumulator
  (each cell may be on either side of each), the compiled square lengths 100 to
  128 among them;
- the five generic passes, on a length without a register split (125) and where
  PSPW_GENERIC_FFT asks for them, the allocation-free call included;
- FP32 tensor-core projectors over single G, which arrays without the symmetry of
  G and -G take: one and several species, projector counts 1-4, bands around the
  128-column tile, part of the sphere, the filter.

Bars of the other parity tests: FP64 1e-12, FP32 2e-5 relative max-norm, 1e-4
after the filter."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

import pspw_oracle as O  # noqa: E402
from helpers import oracle_cell, relmax  # noqa: E402
from pspw import NL_SIMT, NL_TENSOR_CORE, PREC_F32, PREC_F64, Cell, basis_gamma, synth  # noqa: E402
from pspw._lib import check, lib, ptr  # noqa: E402

TOL64, TOL32, TOL32_FILTER = 1e-12, 2e-5, 1e-4


def _arrays(nr, na, lm_end, ecut=5.0):
    lat, sites = synth.si_diamond(1)
    rng = np.random.default_rng(sum(na))
    pos = rng.uniform(0.0, 10.26, (sum(na), 3))
    b = basis_gamma(lat, ecut, nr, na, np.split(pos, np.cumsum(na)[:-1]))
    pkg_a, wnl = synth.kb_form_factors(b, lat, nsp=len(na),
                                       rc=[1.0 + 0.1 * s for s in range(len(na))])
    for s, lm in enumerate(lm_end):
        wnl[s, :4] = np.array([1.5 - 0.3 * s, -0.8 + 0.2 * s, 0.7, -0.6]) / (3 * sum(na))
        pkg_a[lm:, :, s] = 0.0
    b.update(pkg_a=pkg_a, wnl=wnl, lm_end=lm_end, na=na)
    b["veff"] = synth.local_potential(b["nr"], lat, sites)
    return b, lat


def _cell(b):
    cell = Cell.from_arrays(b)
    cell.set_veff(b["veff"])
    return cell


def _psi(b, lat, nb):
    return synth.wavefunctions(b, lat, nb, 7).astype(np.complex64).astype(complex)


def _hpsi(cell, psi, prec, noalloc=False):
    ngw, nb = psi.shape
    dt = torch.complex64 if prec == PREC_F32 else torch.complex128
    d_in = torch.from_numpy(np.ascontiguousarray(psi.T)).to(dt).cuda()
    d_out = torch.full_like(d_in, float("nan"))
    torch.cuda.synchronize()
    call = lib().pspw_apply_ham_block_dev_noalloc if noalloc else lib().pspw_apply_ham_block_dev
    check(call(cell.handle, prec, ptr(d_in), ptr(d_out), ngw, ngw, nb))
    check(lib().pspw_cell_synchronize(cell.handle))
    return d_out.cpu().numpy().T.astype(complex)


def _check_hpsi_filter_density(b, lat, noalloc):
    cell, oc = _cell(b), oracle_cell(b)
    psi = _psi(b, lat, 5)
    ref = O.apply_ham_block(oc, psi, b["veff"])
    for prec, tol in ((PREC_F64, TOL64), (PREC_F32, TOL32)):
        assert relmax(_hpsi(cell, psi, prec), ref) < tol
        for _ in range(2 if noalloc else 0):  # the scratch keeps the first call's contents
            assert relmax(_hpsi(cell, psi, prec, noalloc=True), ref) < tol
    flt = O.chebyfilt(oc, psi, 4, 0.5, 8.0, b["veff"])
    assert relmax(cell.chebyfilt(psi, 4, 0.5, 8.0, PREC_F64), flt) < TOL64
    assert relmax(cell.chebyfilt(psi, 4, 0.5, 8.0, PREC_F32), flt) < TOL32_FILTER
    nx, ngw = 5, b["ngw"]
    focc = np.linspace(2.0, 0.1, nx)
    # normalised over the plane waves that the density sums (all but the last)
    q = synth.wavefunctions(b, lat, nx, 9)
    q = q / np.linalg.norm(q[:-1], axis=0)
    flat = np.concatenate([q.T.reshape(-1), np.zeros(b["ngwx"])])
    rho, ekin = cell.eval_rho_psi(np.zeros(cell.nnr), flat, ngw, ngw, nx, focc, 1.0, b["omega"])
    rho_ref, ekin_ref, _ = O.eval_rho_psi(oc, flat, ngw, ngw, nx, focc, 1.0, b["omega"], b["ngwx"])
    assert relmax(rho, rho_ref) < TOL64
    assert abs(ekin - ekin_ref) < TOL64 * abs(ekin_ref)


# compiled squares; 96 x 98 and 96 x 100 (density), 112 x 124 and 112 x 128
# (FP64), 160 x 176 and 160 x 180 (FP32): the last that fits, one that does not
@pytest.mark.parametrize("n1,n2", [(96, 96), (100, 100), (108, 108), (120, 120), (128, 128),
                                   (96, 98), (96, 100), (112, 124), (112, 128), (160, 176),
                                   (160, 180)])
def test_planes_around_the_limits(n1, n2):
    b, lat = _arrays((n1, n2, 12), [3], [4])
    _check_hpsi_filter_density(b, lat, noalloc=False)


@pytest.mark.parametrize("nr", [(20, 125, 20), (22, 21, 26), (24, 24, 24)])
@pytest.mark.parametrize("na,lm_end", [([3], [4]), ([2, 3], [4, 1])])
def test_generic_passes(nr, na, lm_end, monkeypatch):
    monkeypatch.setenv("PSPW_GENERIC_FFT", "1")
    b, lat = _arrays(nr, na, lm_end)
    _check_hpsi_filter_density(b, lat, noalloc=True)


@pytest.mark.parametrize("nr", [(20, 20, 24), (20, 125, 20)])
@pytest.mark.parametrize("na,lm_end,nb", [
    ([8], [4], 1), ([17], [3], 17), ([5], [2], 65), ([256], [1], 9), ([6, 19], [4, 1], 11),
    ([2, 2, 3], [4, 2, 3], 33),
])
def test_projectors_over_single_g(na, lm_end, nb, nr):
    b, lat = _arrays(nr, na, lm_end)
    b["eigr"] = np.array(b["eigr"], order="F")
    b["eigr"][57, 0, 0] *= np.exp(0.3j)  # no longer the conjugate of its partner's
    cell, oc = _cell(b), oracle_cell(b)
    psi = _psi(b, lat, nb)
    for ngw in (psi.shape[0], psi.shape[0] - 45):
        x = np.asfortranarray(psi[:ngw])
        ref = O.apply_ham_block(oc, x, b["veff"])
        outs = []
        for path in (NL_TENSOR_CORE, NL_SIMT):
            cell.set_nl_path(path)
            outs.append(_hpsi(cell, x, PREC_F32))
            assert relmax(outs[-1], ref) < TOL32
            assert relmax(_hpsi(cell, x, PREC_F32, noalloc=True), ref) < TOL32
        assert not np.array_equal(outs[0], outs[1])
        assert relmax(_hpsi(cell, x, PREC_F64), ref) < TOL64
        cell.set_nl_path(NL_TENSOR_CORE)
        flt = O.chebyfilt(oc, x, 4, 0.5, 10.0, b["veff"])
        assert relmax(cell.chebyfilt(x, 4, 0.5, 10.0, PREC_F32), flt) < TOL32_FILTER
