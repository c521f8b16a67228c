"""The projector forces are additive over the bands: one call over nb bands
equals the sum of its parts, at band counts around the adjoint pass's 32-band
blocks and the force sum's 128 threads, and the projector sums it hands out
equal <p|psi>."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("which,nb", [("si_paw", 1), ("si_paw", 33), ("c_nc", 130)])
def test_force_sums(cuda, built_lib, which, nb):
    import conftest
    from rspacedist_b200 import forces as F, kukan as K, system as S
    cell = conftest.make_si8(20, 0.05, 4) if which == "si_paw" else conftest.make_c8(20)
    T = lambda a: torch.tensor(np.ascontiguousarray(a), device="cuda")
    psi = T(S.random_bands(cell, nb, 3))
    sval, occ = np.linspace(-0.3, 0.5, nb), np.where(np.arange(nb) % 3 == 0, 0.0, 1.7)
    occ[0] = 2.0
    sss = None if cell.sss is None else T(cell.sss)
    rp = torch.empty((nb, cell.natom, cell.nprjmx), dtype=torch.float64, device="cuda")
    f = F.projector_forces(cell, psi, sval, occ, T(cell.dij), sss, rp_out=rp)
    cut = max(1, nb // 2)
    parts = sum(F.projector_forces(cell, psi[a:b], sval[a:b], occ[a:b], T(cell.dij), sss)
                for a, b in ((0, cut), (cut, nb)) if b > a)
    np.testing.assert_allclose(f, parts, atol=1e-12 * np.abs(parts).max())
    ref = K.nonlocaloperation_01(K.Geometry(cell), psi)
    assert float((rp - ref).abs().max()) <= 1e-12 * float(ref.abs().max())
