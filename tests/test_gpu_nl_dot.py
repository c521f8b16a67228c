"""<p|psi> in FP64 at the edges of its launch rules, bit for bit against the
oracle's sequential chain: few (atom, band) pairs (one band per chain), enough
for 32-band blocks, a remainder block, an odd number of projectors, an atom
with fewer projectors than the others, and more projectors than the staged
kernel takes."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def widened(cell, P):
    """cell with P projectors per atom (its own, repeated with other weights);
    the first atom uses one fewer."""
    v = cell.vnlocp
    w = np.stack([v[:, j % v.shape[1]] * (1.0 + 0.1 * j) for j in range(P)], axis=1)
    w[0, P - 1] = 0.0
    nprj = np.full(cell.natom, P, np.int32)
    nprj[0] = P - 1

    class Widened(type(cell)):
        @property
        def nprj(self):
            return nprj

    out = Widened(**{f: getattr(cell, f) for f in cell.__dataclass_fields__})
    out.vnlocp, out.nprjmx = np.ascontiguousarray(w), P
    return out


@pytest.mark.parametrize("P,nb", [(12, 1), (12, 23), (12, 611), (5, 2), (32, 600), (33, 3),
                                  (130, 1)])
def test_nl_dot_f64_chains(oracle, cuda, built_lib, P, nb):
    import conftest
    from rspacedist_b200 import kukan as K
    cell = widened(conftest.make_si8(20, 0.05, 4), P)
    rng = np.random.default_rng(P + nb)
    psi = rng.standard_normal((nb, cell.N))
    geo = dict(natom=cell.natom, nprjmx=P, num_list=cell.num_list, nprj=cell.nprj,
               natinf=cell.natinf, lst=cell.lst, v=cell.vnlocp.ravel())
    ref = oracle.nl_dot(geo, psi, cell.N)
    got = K.nonlocaloperation_01(K.Geometry(cell), torch.tensor(psi, device="cuda"))
    assert np.array_equal(got.cpu().numpy().reshape(ref.shape), ref)
