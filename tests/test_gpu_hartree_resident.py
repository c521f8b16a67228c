"""The one-launch Hartree solves at the edges of their block layouts: FP64 bit
for bit against the oracle (iterates, count, residual) on grids that end inside
a chunk, on one chunk and with a restart; the mixed solve against FP64 on ragged
tiles, z runs that end inside a block and every block shape."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def density(shape, seed):
    rng = np.random.default_rng(seed)
    nx, ny, nz = shape
    r = rng.standard_normal((nz, ny, nx))
    k = [np.fft.fftfreq(n) for n in (nz, ny, nx)]
    k2 = k[0][:, None, None] ** 2 + k[1][:, None] ** 2 + k[2] ** 2
    return np.ascontiguousarray(np.fft.ifftn(np.fft.fftn(r) * np.exp(-60 * k2)).real).ravel()


@pytest.mark.parametrize("shape,nfh,ncgmax,ncgres", [
    ((16, 16, 16), 4, 800, 801), ((18, 20, 22), 4, 800, 7), ((10, 64, 14), 4, 3, 801),
    ((14, 16, 18), 6, 800, 801), ((12, 9, 11), 2, 800, 801), ((40, 34, 26), 4, 800, 801)])
def test_fp64_bits(oracle, cuda, built_lib, shape, nfh, ncgmax, ncgres):
    from rspacedist_b200 import kukan as K
    xmax = tuple(0.08 * n for n in shape)
    rho = density(shape, 1)
    v0 = 0.01 * density(shape, 2)
    ref, it, dp = oracle.hartree_cg(shape, nfh, xmax, 1e-12, 1, ncgmax, ncgres, rho, v0)
    vh = torch.tensor(v0, device="cuda")
    got = K.scf_hartree(shape, nfh, xmax, torch.tensor(rho, device="cuda"), vh, 1e-12, 1, ncgmax,
                        ncgres)
    assert got == (it, dp)
    assert np.array_equal(vh.cpu().numpy(), ref)


# (the launch's own state takes 448 doubles: grids of fewer points keep the plain
# launches, 8 x 7 x 8 is the first that does not)
@pytest.mark.parametrize("entry", ["rs_hartree_cg", "rs_hartree_cg_noalloc"])
@pytest.mark.parametrize("shape", [(6, 5, 5), (6, 6, 6), (8, 7, 6), (8, 7, 7), (8, 7, 8)])
def test_fp64_bits_smallest_grids(oracle, cuda, built_lib, shape, entry):
    from rspacedist_b200 import lib
    xmax = tuple(0.15 * n for n in shape)
    rho, v0 = density(shape, 5), density(shape, 6)
    ref, it, dp = oracle.hartree_cg(shape, 2, xmax, 1e-12, 1, 800, 801, rho, v0)
    d_rho, vh = torch.tensor(rho, device="cuda"), torch.tensor(v0, device="cuda")
    n, d = C.c_int(0), C.c_double(0.0)
    lib.call(entry, *shape, 2, *xmax, 1e-12, 1, 800, 801, C.c_void_p(d_rho.data_ptr()),
             C.c_void_p(vh.data_ptr()), C.byref(n), C.byref(d), None)
    assert (n.value, d.value) == (it, dp)
    assert np.array_equal(vh.cpu().numpy(), ref)


@pytest.mark.parametrize("shape", [(64, 64, 64), (20, 36, 14), (68, 34, 30), (128, 96, 20),
                                   (100, 100, 90), (128, 128, 126)])
def test_mixed_matches_fp64(cuda, built_lib, shape):
    from rspacedist_b200 import kukan as K
    xmax = tuple(0.08 * n for n in shape)
    rho = torch.tensor(density(shape, 3), device="cuda")
    out = []
    for mixed in (False, True):
        vh = torch.zeros_like(rho)
        it, dp = K.scf_hartree(shape, 4, xmax, rho, vh, epsvh=1e-10, mixed=mixed)
        assert dp <= 1e-10 and it < 800
        out.append(vh)
    # both residuals are below epsvh in FP64: up to a constant (the null space of
    # the operator) the potentials agree to epsvh over the smallest nonzero
    # eigenvalue of -1/2 lap, (pi / xmax)^2 / 2
    lam = 0.5 * (np.pi / max(xmax)) ** 2
    diff = out[0] - out[1]
    assert float((diff - diff.mean()).square().mean().sqrt()) <= 3e-10 / lam


def test_mixed_iteration_limit(cuda, built_lib):
    """A solve cut off by ncgmax stops there and returns the norm of the FP64
    residual of its potential (rounded to FP32 per point: 2^-24 of it)."""
    from rspacedist_b200 import kukan as K
    shape, xmax = (64, 48, 32), (5.0, 4.0, 2.5)
    h = [2 * x / n for x, n in zip(xmax, shape)]
    rho = torch.tensor(density(shape, 4), device="cuda")
    vh = torch.zeros_like(rho)
    it, dp = K.scf_hartree(shape, 4, xmax, rho, vh, ncgmax=7, mixed=True)
    r = 2 * np.pi * (rho - rho.mean()) - K.scf_hartee_laplacian(shape, 4, h, vh)
    ref = float(r.square().mean().sqrt())
    assert it == 7
    assert abs(dp - ref) <= 1e-6 * ref


@pytest.mark.parametrize("shape", [(32, 24, 20), (22, 24, 20)])
def test_mixed_start_off_a_boundary(cuda, built_lib, shape):
    """A vh eight bytes past a 16-byte boundary is solved by the FP64 iteration."""
    from rspacedist_b200 import kukan as K
    xmax = tuple(0.08 * n for n in shape)
    rho = torch.tensor(density(shape, 3), device="cuda")
    ref, vh = torch.zeros_like(rho), torch.zeros(rho.numel() + 1, device="cuda",
                                                 dtype=torch.float64)[1:]
    want = K.scf_hartree(shape, 4, xmax, rho, ref)
    assert K.scf_hartree(shape, 4, xmax, rho, vh, mixed=True) == want
    assert torch.equal(vh, ref)
