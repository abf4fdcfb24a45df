"""The start of the SCF loop: Lanczos bounds that do not exist are an error and
not a filter window, and the start block of pspw_system_cheby_scf is glibc's
rand() after srand(1) (ChebySCFLoop.cpp:100-106, 201-208), as the C library
draws it."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from helpers import write_input, write_synthetic_fhi  # noqa: E402
from pspw import PREC_F32, PREC_F64, PspwError, synth  # noqa: E402
from pspw.system import System  # noqa: E402

LAPACK = 7


@pytest.fixture(scope="module")
def system(tmp_path_factory):
    d = tmp_path_factory.mktemp("scf")
    write_synthetic_fhi(str(d / "X.fhi"))
    _, pos = synth.si_diamond(1)
    write_input(str(d / "INPUT"), "X.fhi", pos, 10.26, ecut_ry=8.0, idiag=-1, imix=3, max_scf=2)
    return System(str(d))


def _loop(system, v0, X, prec, **kw):
    p = system.params()
    p.update(kw)
    return system.scf().cheby_scf(
        system.array("focc"), system.array("rho_start"), v0, X, nx=p["nx"], nempty=p["nempty"],
        degree=p["degree"], max_scf_iter=p["max_scf_iter"], conv=p["conv"], imix=p["imix"],
        mixdim=p["mixdim"], mix_beta=p["mix_beta"], pulay_beta=p["pulay_beta"],
        kerker_q0=p["kerker_q0"], idiag=p["idiag"], max_diag_iter=p["max_diag_iter"],
        filter_prec=prec)


def _rand(n):
    libc = ctypes.CDLL("libc.so.6")
    libc.srand(1)
    return np.array([libc.rand() for _ in range(n)], dtype=float) / 2147483647.0


@pytest.mark.parametrize("prec", [PREC_F64, PREC_F32])
@pytest.mark.parametrize("bad", ["zero", "nan"])
def test_no_bounds_is_an_error(system, prec, bad):
    ngw, nx2 = system.dims["ngw"], system.dims["nx"] + 2
    v0 = np.zeros(ngw, dtype=complex)
    if bad == "nan":
        v0[:] = 1.0
        v0[5] = np.nan
    X = np.random.default_rng(1).uniform(0, 1, (ngw, nx2)) + 0j
    with pytest.raises(PspwError) as e:
        _loop(system, v0, X, prec)
    assert e.value.code == LAPACK


def test_start_block_is_libc_rand(system):
    ngw, ngwx, nx2 = system.dims["ngw"], system.dims["ngwx"], system.dims["nx"] + 2
    r = _rand(2 * ngwx + 2 * ngw * nx2)
    v0 = r[0:2 * ngwx:2] + 1j * r[1:2 * ngwx:2]
    x = r[2 * ngwx:]
    X = (x[0::2] + 1j * x[1::2]).reshape((ngw, nx2), order="F")
    a = system.cheby_scf(PREC_F64)
    b = _loop(system, v0[:ngw], X, PREC_F64)
    # the same arithmetic on the same numbers
    assert np.array_equal(a["hist"][:, :3], b["hist"][:, :3])
    assert np.array_equal(a["eig"], b["eig"])
    c = _loop(system, v0[:ngw], X[:, ::-1], PREC_F64)
    assert not np.array_equal(a["hist"][:, :3], c["hist"][:, :3])
