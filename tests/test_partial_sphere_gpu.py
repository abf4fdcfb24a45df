"""Calls over the first ngw G of a cell, fewer than its sphere, where the
projector products run over pairs (+G, -G): ngw from 1 over the 8-pair groups
to one less than the sphere, G ordered so that partners are neighbours or all
of them come after the first half, one band and several, both precisions,
H*psi, filter and projections, against the oracle.  Bars: FP64 1e-12, FP32 2e-5
relative max-norm, 1e-4 after the filter.  The allocation-free call keeps the
kernels of the selected path whatever calls came before it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

import pspw_oracle as O  # noqa: E402
from helpers import oracle_cell, relmax  # noqa: E402
from pspw import (NL_SIMT, NL_TENSOR_CORE, PREC_F32, PREC_F64, Cell, basis_gamma,  # noqa: E402
                  synth)
from pspw._lib import check, lib, ptr  # noqa: E402

TOL64, TOL32, TOL32_FILTER = 1e-12, 2e-5, 1e-4


def _arrays(order="sphere"):
    lat, pos = synth.si_diamond(1)
    na, lm_end = [5, 3], [4, 3]
    pos = pos + np.random.default_rng(4).uniform(-0.3, 0.3, pos.shape)
    b = basis_gamma(lat, 6.0, (20, 20, 24), na, [pos[:5], pos[5:]])
    pkg_a, wnl = synth.kb_form_factors(b, lat, nsp=2, rc=[1.0, 1.1])
    for s, lm in enumerate(lm_end):
        wnl[s, :4] = [1.5 - 0.3 * s, -0.8 + 0.2 * s, 0.7, -0.6]
        pkg_a[lm:, :, s] = 0.0
    b.update(pkg_a=pkg_a, wnl=wnl, lm_end=lm_end, na=na)
    b["veff"] = synth.local_potential(b["nr"], lat, pos)
    if order == "halves":  # every partner in the second half
        n, n1, n2 = b["ngw"], b["nr"][0], b["nr"][1]
        i = np.asarray(b["n123"][:n], dtype=np.int64) - 1
        g = np.stack([i % n1, i // n1 % n2, i // (n1 * n2)], 1)
        g = np.where(g > np.array(b["nr"]) // 2, g - np.array(b["nr"]), g)
        first = np.array([tuple(v) >= (0, 0, 0) for v in g])
        perm = np.concatenate([np.flatnonzero(first), np.flatnonzero(~first)])
        for k, axis in (("n123", 0), ("xkg", 0), ("eigr", 0), ("pkg_a", 1)):
            a = np.array(b[k], order="F")
            head = np.take(a, perm, axis=axis)
            if axis == 0:
                a[:n] = head
            else:
                a[:, :n] = head
            b[k] = np.asfortranarray(a)
    return b, lat


def _cell(b):
    cell = Cell.from_arrays(b)
    cell.set_veff(b["veff"])
    return cell


def _hpsi(cell, psi, prec, noalloc=False):
    ngw, nb = psi.shape
    dt = torch.complex64 if prec == PREC_F32 else torch.complex128
    d_in = torch.from_numpy(np.ascontiguousarray(psi.T)).to(dt).cuda()
    d_out = torch.zeros_like(d_in)
    torch.cuda.synchronize()
    call = lib().pspw_apply_ham_block_dev_noalloc if noalloc else lib().pspw_apply_ham_block_dev
    check(call(cell.handle, prec, ptr(d_in), ptr(d_out), ngw, ngw, nb))
    check(lib().pspw_cell_synchronize(cell.handle))
    return d_out.cpu().numpy().T


@pytest.mark.parametrize("order", ["sphere", "halves"])
@pytest.mark.parametrize("nb", [1, 17])
def test_partial_sphere(order, nb):
    b, lat = _arrays(order)
    n = b["ngw"]
    psi = synth.wavefunctions(b, lat, nb, 5).astype(np.complex64).astype(complex)
    cell, oc = _cell(b), oracle_cell(b)
    for ngw in (1, 2, 15, 16, 17, 129, n // 2, n // 2 + 1, n - 1, n):
        x = np.asfortranarray(psi[:ngw])
        ref = O.apply_ham_block(oc, x, b["veff"])
        assert relmax(_hpsi(cell, x, PREC_F64), ref) < TOL64, ngw
        for path in (NL_TENSOR_CORE, NL_SIMT):
            cell.set_nl_path(path)
            assert relmax(_hpsi(cell, x, PREC_F32), ref) < TOL32, ngw
        cell.set_nl_path(NL_TENSOR_CORE)
        focc = np.linspace(2.0, 0.5, nb)
        e, fnl = cell.eval_enl(x, nb, focc, 1.0)
        e_ref, fnl_ref = O.eval_enl(oc, x, ngw, nb, focc, 1.0)
        assert relmax(fnl, fnl_ref) < TOL64, ngw
        assert abs(e - e_ref) < TOL64 * abs(e_ref)
    ngw = n // 2 + 1
    x = np.asfortranarray(psi[:ngw])
    ref = O.chebyfilt(oc, x, 4, 0.5, 12.0, b["veff"])
    assert relmax(cell.chebyfilt(x, 4, 0.5, 12.0, PREC_F64), ref) < TOL64
    assert relmax(cell.chebyfilt(x, 4, 0.5, 12.0, PREC_F32), ref) < TOL32_FILTER


@pytest.mark.parametrize("path", [NL_TENSOR_CORE, NL_SIMT])
def test_noalloc_does_not_depend_on_earlier_calls(path):
    b, lat = _arrays()
    n, nb = b["ngw"], 11
    psi = synth.wavefunctions(b, lat, nb, 5).astype(np.complex64).astype(complex)
    x = np.asfortranarray(psi[:n - 100])
    cell = _cell(b)
    cell.set_nl_path(path)
    ref = O.apply_ham_block(oracle_cell(b), x, b["veff"])
    first = _hpsi(cell, x, PREC_F32, noalloc=True)
    assert relmax(first, ref) < TOL32
    _hpsi(cell, x, PREC_F32)  # an ordinary call may build tables of its own
    assert np.array_equal(_hpsi(cell, x, PREC_F32, noalloc=True), first)
    cell.set_nl_path(NL_SIMT if path == NL_TENSOR_CORE else NL_TENSOR_CORE)
    assert not np.array_equal(_hpsi(cell, x, PREC_F32, noalloc=True), first)
