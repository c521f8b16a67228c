"""rs_chol_inv_t: entries of L rounded once per division, and the inverse at the
edges of its two forms (blocks of 64 rows up to 3000, a warp per column above)."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


def chol_inv(n, seed=0):
    """(G, L, L^-1) of a seeded positive definite G of order n."""
    from rspacedist_b200 import lib
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed + n)
    a = torch.randn((n, n), generator=gen, device="cuda", dtype=torch.float64)
    G = a @ a.T / n + torch.eye(n, device="cuda", dtype=torch.float64)
    L, W = G.T.contiguous().clone(), torch.empty_like(G)   # column-major
    lib.call("rs_chol_inv_t", n, C.c_void_p(L.data_ptr()), C.c_void_p(W.data_ptr()), None)
    torch.cuda.synchronize()
    return G, L.T.tril(), W   # W is L^-T by columns: L^-1 by rows


@pytest.mark.parametrize("n", [2, 64, 65, 150])
def test_first_column(cuda, built_lib, n):
    G, L, _ = chol_inv(n)
    # IEEE root and quotient, in the diagonal block and in the panels below it
    assert torch.equal(L[:, 0].cpu(), torch.cat([G[:1, 0].sqrt(), G[1:, 0] / G[0, 0].sqrt()]).cpu())


@pytest.mark.parametrize("n", [1, 63, 64, 65, 200, 3000, 3001])
def test_factor_and_inverse(cuda, built_lib, n):
    G, L, X = chol_inv(n)
    eps = 2.0 ** -53
    # |L L^T - G| <= (n + 1) eps |L| |L^T| and |L X - 1| <= n eps |L| |X| (Higham), with a
    # factor of two for the checking products' own rounding
    assert bool(((L @ L.T - G).abs() <= 2 * (n + 1) * eps * (L.abs() @ L.abs().T)).all())
    one = torch.eye(n, device="cuda", dtype=torch.float64)
    assert bool(((L @ X - one).abs() <= 2 * (n + 1) * eps * (L.abs() @ X.abs())).all())
    assert float(X.triu(1).abs().max()) == 0.0
