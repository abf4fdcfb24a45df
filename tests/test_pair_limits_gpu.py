"""FP32 tensor-core projectors over pairs (+G, -G) at the largest atom counts
they take (256 per species, 16 operand rows per step), where the operand slots
and the psi slots share a block's 227 KB, against the oracle.  Bars: 2e-5
relative max-norm, 1e-4 after the filter, as the other FP32 parity tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

import pspw_oracle as O  # noqa: E402
from helpers import oracle_cell, relmax  # noqa: E402
from pspw import NL_TENSOR_CORE, PREC_F32, Cell, basis_gamma, synth  # noqa: E402


@pytest.mark.parametrize("na,lm", [(240, 1), (241, 1), (256, 1), (256, 2), (256, 4)])
def test_most_atoms(na, lm):
    lat, _ = synth.si_diamond(1)
    pos = np.random.default_rng(na).uniform(0.0, 10.26, (na, 3))
    b = basis_gamma(lat, 6.0, (20, 20, 20), [na], [pos])
    pkg_a, wnl = synth.kb_form_factors(b, lat)
    pkg_a[lm:] = 0.0
    wnl[0, :4] = np.array([1.5, -0.8, 0.7, -0.6]) / (3 * na)
    b.update(pkg_a=pkg_a, wnl=wnl, lm_end=[lm], na=[na])
    veff = synth.local_potential(b["nr"], lat, pos[:8])
    psi = synth.wavefunctions(b, lat, 9, 5).astype(np.complex64).astype(complex)
    cell = Cell.from_arrays(b)
    cell.set_veff(veff)
    cell.set_nl_path(NL_TENSOR_CORE)
    oc = oracle_cell(b)
    d_in = torch.from_numpy(np.ascontiguousarray(psi.T)).to(torch.complex64).cuda()
    d_out = torch.zeros_like(d_in)
    torch.cuda.synchronize()
    ngw, nb = psi.shape
    cell.apply_ham_block_dev(d_in, d_out, ngw, ngw, nb, PREC_F32)
    torch.cuda.synchronize()
    assert relmax(d_out.cpu().numpy().T, O.apply_ham_block(oc, psi, veff)) < 2e-5
    ref = O.chebyfilt(oc, psi, 4, 0.5, 12.0, veff)
    assert relmax(cell.chebyfilt(psi, 4, 0.5, 12.0, PREC_F32), ref) < 1e-4
