"""The SCF loop's orthonormalisation (pspw_ortho_span_dev) where its passes
branch: a second Gram matrix that is the identity to 1e-9 (inverted to first
order) or not (factored), columns of very different norms, norms outside the
factorisation's range and a zero column (Householder), at orders around the
8-column panels.  Q^H Q = I and X = Q (Q^H X) within 1e-12: CholeskyQR2 and
Householder leave n eps = 3e-14 at most, times a margin."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from helpers import engine_cell_args, golden  # noqa: E402
from pspw import Cell  # noqa: E402

TOL = 1e-12


@pytest.fixture(scope="module")
def cell():
    return Cell.from_arrays(engine_cell_args(golden("si8_8ry")))


def _block(m, n, cond, seed):
    rng = np.random.default_rng(seed)
    z = lambda a, b: rng.standard_normal((a, b)) + 1j * rng.standard_normal((a, b))  # noqa: E731
    q = np.linalg.qr(z(m, n))[0]
    u = np.linalg.qr(z(n, n))[0]
    return (q * np.geomspace(1.0, 1.0 / cond, n)) @ u


@pytest.mark.parametrize("n", [1, 7, 8, 9, 33, 146, 150])
@pytest.mark.parametrize("case", ["well", "ill", "scaled", "tiny", "zero"])
def test_span(cell, n, case):
    m = 437
    X = _block(m, n, 1e5 if case == "ill" else 30.0, n)
    if case == "scaled":
        X = X * np.geomspace(1e-6, 1e6, n)[None]
    elif case == "tiny":
        X[:, n // 2] *= 1e-130
    elif case == "zero":
        X[:, n // 2] = 0.0
    d = torch.from_numpy(np.ascontiguousarray(X.T)).cuda()
    torch.cuda.synchronize()
    cell.ortho_span_dev(d, m, n)
    torch.cuda.synchronize()
    Q = d.cpu().numpy().T
    if case == "zero":  # the basis of the other columns, whatever fills the gap
        if n == 1:
            return
        keep = np.arange(n) != n // 2
        X = X[:, keep]
    else:
        assert np.abs(Q.conj().T @ Q - np.eye(n)).max() < TOL
    Xn = X / np.linalg.norm(X, axis=0)
    assert np.abs(Xn - Q @ (Q.conj().T @ Xn)).max() < TOL
