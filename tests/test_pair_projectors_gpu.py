"""FP32 tensor-core projector GEMMs over pairs (+G, -G): projector counts 1-4
(s, s + p parts: even and odd form factors), several species, atoms around the
16-atom operand tiles, bands around the 128-column tile, both grid paths and
the recurrence of the filter, against the oracle, at the parity tests' bars
(2e-5 relative max-norm, 1e-4 after the filter).  The SIMT kernels, which sum
over G, are held to the same values."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

import pspw_oracle as O  # noqa: E402
from helpers import oracle_cell, relmax  # noqa: E402
from pspw import NL_SIMT, NL_TENSOR_CORE, PREC_F32, Cell, basis_gamma, synth  # noqa: E402

TOL, TOL_FILTER = 2e-5, 1e-4


def _arrays(na, lm_end, nr):
    lat, _ = synth.si_diamond(1)
    rng = np.random.default_rng(sum(na))
    pos = rng.uniform(0.0, 10.26, (sum(na), 3))
    tau = np.split(pos, np.cumsum(na)[:-1])
    b = basis_gamma(lat, 6.0, nr, na, tau)
    pkg_a, wnl = synth.kb_form_factors(b, lat, nsp=len(na), rc=[1.0 + 0.1 * s for s in range(len(na))])
    for s, lm in enumerate(lm_end):
        wnl[s, :4] = np.array([1.5 - 0.3 * s, -0.8 + 0.2 * s, 0.7, -0.6]) / 24.0
        pkg_a[lm:, :, s] = 0.0
    b.update(pkg_a=pkg_a, wnl=wnl, lm_end=lm_end, na=na)
    b["veff"] = synth.local_potential(b["nr"], lat, pos[:8])
    return b, lat


@pytest.mark.parametrize("nr", [(24, 24, 24), (20, 125, 20)])  # 125: generic passes
@pytest.mark.parametrize("na,lm_end,nb", [
    ([8], [4], 1), ([15], [4], 16), ([16], [4], 17), ([17], [4], 33), ([33], [3], 7),
    ([5], [2], 65), ([1], [1], 20), ([6, 19], [4, 1], 11), ([2, 2, 3], [4, 2, 3], 5),
])
def test_pairs(na, lm_end, nb, nr):
    b, lat = _arrays(na, lm_end, nr)
    psi = synth.wavefunctions(b, lat, nb, 5).astype(np.complex64).astype(complex)
    cell = Cell.from_arrays(b)
    cell.set_veff(b["veff"])
    oc = oracle_cell(b)
    ref = O.apply_ham_block(oc, psi, b["veff"])
    ngw = psi.shape[0]
    ld = ngw + 1
    d_in = torch.zeros(nb, ld, dtype=torch.complex64)
    d_in[:, :ngw] = torch.from_numpy(np.ascontiguousarray(psi.T)).to(torch.complex64)
    d_in = d_in.cuda()
    for path in (NL_TENSOR_CORE, NL_SIMT):
        cell.set_nl_path(path)
        d_out = torch.zeros_like(d_in)
        torch.cuda.synchronize()
        cell.apply_ham_block_dev(d_in, d_out, ld, ngw, nb, PREC_F32)
        torch.cuda.synchronize()
        assert relmax(d_out.cpu().numpy()[:, :ngw].T, ref) < TOL
    cell.set_nl_path(NL_TENSOR_CORE)
    flt = O.chebyfilt(oc, psi, 4, 0.5, 12.0, b["veff"])
    assert relmax(cell.chebyfilt(psi, 4, 0.5, 12.0, PREC_F32), flt) < TOL_FILTER
