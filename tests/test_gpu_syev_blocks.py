"""The block Jacobi eigensolver at the edges of its 32-index blocks and on
matrices whose rotations take its special cases: diagonal, zero, repeated
levels, equal diagonals and very large or small elements."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def matrix(kind, n):
    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n))
    a = a + a.T
    if kind == "diagonal":
        return np.diag(rng.standard_normal(n))
    if kind == "zero":
        return np.zeros((n, n))
    if kind == "repeated":
        q = np.linalg.qr(a)[0]
        return (q * np.repeat([1.0, -2.0], [n // 2, n - n // 2])) @ q.T
    if kind == "equal":   # every rotation starts from app == aqq
        return a - np.diag(np.diag(a)) + 3.0 * np.eye(n)
    return a * {"random": 1.0, "tiny": 1e-150, "large": 1e150}[kind]


@pytest.mark.parametrize("n", [1, 31, 32, 33, 64, 65, 128, 193])
@pytest.mark.parametrize("kind", ["random", "diagonal", "zero", "repeated", "equal"])
def test_syev_blocks(cuda, built_lib, kind, n):
    check(matrix(kind, n), n)


@pytest.mark.parametrize("kind", ["tiny", "large"])
def test_syev_element_range(cuda, built_lib, kind):
    check(matrix(kind, 40), 40)


def check(a, n):
    from rspacedist_b200 import kukan as K
    a = 0.5 * (a + a.T)
    w, Z, _ = K.syev(torch.tensor(a, device="cuda"))
    w, Z = w.cpu().numpy(), Z.cpu().numpy()
    # Jacobi: backward error of a few n eps of the norm, and orthogonal to a few n eps
    eps, nrm = np.finfo(float).eps, np.abs(a).max() * n
    assert np.all(np.diff(w) >= 0)
    assert np.abs(w - np.linalg.eigvalsh(a)).max() <= 8 * n * eps * nrm
    assert np.abs(a @ Z - Z * w).max() <= 8 * n * eps * nrm
    assert np.abs(Z.T @ Z - np.eye(n)).max() <= 8 * n * eps
    top = np.abs(Z).argmax(0)
    assert np.all(Z[top, np.arange(n)] > 0)
