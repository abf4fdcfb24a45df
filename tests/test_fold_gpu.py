"""FP64 projector products over pairs (+G, -G) against the oracle, at band
counts around the tile widths (1, 2, 16, 17, 32, 33, 64, 65), projector counts
that leave ragged tiles, and arrays that have the symmetry or lack it in one
value only (those take the complex products).  Bar: FP64 1e-12 relative
max-norm, as every FP64 parity test."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

import pspw_oracle as O  # noqa: E402
from helpers import oracle_cell, relmax  # noqa: E402
from pspw import PREC_F64, Cell, basis_gamma, synth  # noqa: E402

TOL = 1e-12


def _arrays(na, lm_end, seed=3, nr=(24, 24, 24), ecut=9.0):
    lat, pos = synth.si_diamond(1)
    rng = np.random.default_rng(seed)
    pos = pos[:sum(na)] + rng.uniform(-0.3, 0.3, (sum(na), 3))
    tau = np.split(pos, np.cumsum(na)[:-1])
    b = basis_gamma(lat, ecut, nr, na, tau)
    pkg_a, wnl = synth.kb_form_factors(b, lat, nsp=len(na), rc=[1.0 + 0.1 * s for s in range(len(na))])
    for s, lm in enumerate(lm_end):
        wnl[s, :4] = [1.5 - 0.3 * s, -0.8 + 0.2 * s, 0.7, -0.6]
        pkg_a[lm:, :, s] = 0.0
    b.update(pkg_a=pkg_a, wnl=wnl, lm_end=lm_end, na=na)
    b["veff"] = synth.local_potential(b["nr"], lat, pos)
    return b, lat


def _break(b, how):
    b = dict(b)
    if how == "eigr":  # one phase of one atom, off the axis of its conjugate
        b["eigr"] = b["eigr"].copy(order="F")
        b["eigr"][57, 1, 0] *= np.exp(0.3j)
    elif how == "pkg":  # one form factor neither even nor odd
        b["pkg_a"] = b["pkg_a"].copy(order="F")
        b["pkg_a"][2, 91, 0] += 0.125
    elif how == "origin":  # a p projector that does not vanish at G = 0
        b["pkg_a"] = b["pkg_a"].copy(order="F")
        b["pkg_a"][1, 0, 0] = 0.5
    return b


def _hpsi(b, psi, ld=None):
    cell = Cell.from_arrays(b)
    cell.set_veff(b["veff"])
    ngw, nb = psi.shape
    ld = ld or ngw
    d_in = torch.zeros(nb, ld, dtype=torch.complex128)
    d_in[:, :ngw] = torch.from_numpy(np.ascontiguousarray(psi.T))
    d_in = d_in.cuda()
    d_out = torch.zeros_like(d_in)
    torch.cuda.synchronize()
    cell.apply_ham_block_dev(d_in, d_out, ld, ngw, nb, PREC_F64)
    torch.cuda.synchronize()
    return cell, d_out.cpu().numpy()[:, :ngw].T


@pytest.mark.parametrize("nb", [1, 2, 16, 17, 32, 33, 64, 65])
@pytest.mark.parametrize("na,lm_end", [([8], [4]), ([3], [1]), ([5, 3], [4, 3])])
def test_bands_and_projectors(nb, na, lm_end):
    b, lat = _arrays(na, lm_end)
    psi = synth.wavefunctions(b, lat, nb, 5)
    _, out = _hpsi(b, psi, ld=psi.shape[0] + 3)
    assert relmax(out, O.apply_ham_block(oracle_cell(b), psi, b["veff"])) < TOL


@pytest.mark.parametrize("how", ["eigr", "pkg", "origin"])
@pytest.mark.parametrize("nb", [1, 20])
def test_arrays_without_the_symmetry(how, nb):
    b, lat = _arrays([8], [4])
    b = _break(b, how)
    psi = synth.wavefunctions(b, lat, nb, 5)
    cell, out = _hpsi(b, psi)
    assert relmax(out, O.apply_ham_block(oracle_cell(b), psi, b["veff"])) < TOL
    ref = O.chebyfilt(oracle_cell(b), psi, 3, 0.5, 12.0, b["veff"])
    assert relmax(cell.chebyfilt(psi, 3, 0.5, 12.0, PREC_F64), ref) < TOL


@pytest.mark.parametrize("nr", [(24, 24, 24), (24, 30, 26), (64, 16, 122)])
@pytest.mark.parametrize("nx", [1, 9])
def test_filter_and_projections(nr, nx):
    b, lat = _arrays([5, 3], [4, 3], nr=nr, ecut=4.0)
    psi = synth.wavefunctions(b, lat, nx, 5)
    cell = Cell.from_arrays(b)
    cell.set_veff(b["veff"])
    oc = oracle_cell(b)
    flt = O.chebyfilt(oc, psi, 4, 0.5, 8.0, b["veff"])
    assert relmax(cell.chebyfilt(psi, 4, 0.5, 8.0, PREC_F64), flt) < TOL
    focc = np.linspace(2.0, 0.5, nx)
    e, fnl = cell.eval_enl(psi, nx, focc, 1.0)
    e_ref, fnl_ref = O.eval_enl(oc, psi, b["ngw"], nx, focc, 1.0)
    assert relmax(fnl, fnl_ref) < TOL
    assert abs(e - e_ref) < TOL * abs(e_ref)
