"""FP32 H psi on grids of even nx, the plane-marching stencil against the
per-point gather that serves arrays off the vectors' boundary (16 bytes for nx =
0 mod 4, else 8), and the batched call against the single-cell one, at the edges
of their tiles and thread layouts."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def cell_of(shape, natom=3):
    from rspacedist_b200 import system as S
    ds = S.load_dataset("c_ncps")
    edge = 0.3 * np.array(shape)
    pos = np.random.default_rng(1).uniform(-0.5, 0.5, (natom, 3)) * edge
    c = S.make_cell(edge, shape, pos, ds)
    return c


def inputs(cell, nb):
    from rspacedist_b200 import kukan as K, system as S
    g = K.Geometry(cell)
    psi = torch.tensor(S.random_bands(cell, nb, nb), dtype=torch.float32, device="cuda")
    veff = torch.tensor(S.smooth_veff(cell, 1), dtype=torch.float32, device="cuda")
    dij = torch.tensor(cell.dij, dtype=torch.float64, device="cuda")
    return g, veff, dij, K.nonlocaloperation_01(g, psi), psi


def shifted(t):
    """t one element past a 16-byte boundary"""
    buf = torch.empty(t.numel() + 1, dtype=t.dtype, device="cuda")
    out = buf[1:].view(t.shape)
    out.copy_(t)
    return out


@pytest.mark.parametrize("shape,nb", [((62, 62, 16), 3), ((66, 34, 10), 2), ((130, 30, 12), 1),
                                      ((10, 64, 70), 5), ((18, 66, 22), 17),
                                      ((64, 64, 16), 3), ((36, 10, 12), 5)])
def test_even_rows_match_the_gather(cuda, built_lib, shape, nb):
    from rspacedist_b200 import kukan as K
    g, veff, dij, rp, psi = inputs(cell_of(shape), nb)
    out = K.hpsi(g, veff, dij, rp, psi)
    ref = K.hpsi(g, shifted(veff), dij, rp, shifted(psi), out=shifted(psi))
    # 25 + 4 terms of the size of the diagonal one, rounded at 2^-24 each
    assert float((out - ref).abs().max()) <= 2e-6 * float(ref.abs().max())


@pytest.mark.parametrize("shapes", [[(10, 10, 10), (64, 10, 12), (40, 40, 18)],
                                    [(32, 32, 32), (34, 34, 34), (22, 22, 22), (11, 12, 13)],
                                    [(64, 64, 12), (24, 20, 30)]])
def test_batch_equals_single_cell_call(cuda, built_lib, shapes):
    """Cells whose planes fit one CTA, and beside them an odd grid and one too
    large (per-point gather)."""
    from rspacedist_b200 import kukan as K, system as S
    cells = []
    for sh in shapes:
        c = cell_of([n + n % 2 for n in sh])
        if any(n % 2 for n in sh):   # odd grids come through the C ABI only
            c.shape = tuple(sh)
            c.natinf = np.zeros_like(c.natinf)
        cells.append(c)
    ins = [inputs(c, 5 + 9 * k) for k, c in enumerate(cells)]
    outs = [torch.full_like(i[4], float("nan")) for i in ins]
    plan = K.HpsiBatch([i[0] for i in ins], [len(i[4]) for i in ins])
    cols = list(zip(*[i[1:] for i in ins]))
    plan.set(cols[0], cols[1], cols[2], cols[3], outs)
    plan.run()
    for c, i, o in zip(cells, ins, outs):
        ref = K.hpsi(*i)
        nx, ny = c.shape[:2]
        cols, threads = (nx + 3) // 4, (nx + 3) // 4 * (ny // 2)
        same = nx % 2 or (threads <= 256 and 4 * ny + 16 * cols <= 4 * threads)
        assert torch.equal(o, ref) if same else \
            float((o - ref).abs().max()) <= 2e-6 * float(ref.abs().max()), c.shape
    plan.close()


def test_many_bands_equal_few(cuda, built_lib):
    """The nonlocal pass over several hundred thousand CTAs gives the bits of the
    pass over a few."""
    from rspacedist_b200 import kukan as K
    cell = cell_of((20, 20, 20), 16)
    g, veff, dij, rp, psi = inputs(cell, 20)
    few = K.hpsi(g, veff, dij, rp, psi)
    lists = np.reshape(cell.lst, (16, -1))
    covered = np.unique(np.concatenate([l[:n] for l, n in zip(lists, cell.natinf)])).size
    # (at least half of the listed points have a nonzero projector value)
    rep = 16 * (200000 // (covered // 128) + 2) // 20 + 1
    many = K.hpsi(g, veff, dij, rp.repeat((rep,) + (1,) * (rp.dim() - 1)),
                  psi.repeat((rep,) + (1,) * (psi.dim() - 1)))
    assert torch.equal(many.view(rep, -1), few.view(1, -1).expand(rep, -1))


def test_two_batch_plans(cuda, built_lib):
    """Plans of different cells that are alive together, run in both orders and
    captured: each keeps the shared memory its own launch needs."""
    from rspacedist_b200 import kukan as K
    plans = []
    for shape, nb in (((22, 22, 22), 7), ((34, 34, 34), 2), ((22, 22, 22), 1)):
        cols = inputs(cell_of(shape), nb)
        out = torch.full_like(cols[4], float("nan"))
        plan = K.HpsiBatch([cols[0]], [nb])
        plan.set(*[[c] for c in cols[1:]], [out])
        plans.append((plan, cols, out, K.hpsi(*cols)))
    st = torch.cuda.Stream()
    for order in (plans, plans[::-1]):
        for graph in (False, True):
            for plan, cols, out, ref in order:
                out.fill_(float("nan"))
                st.wait_stream(torch.cuda.current_stream())
                with torch.cuda.stream(st):
                    plan.run(graph=graph)
                st.synchronize()
                assert torch.equal(out, ref)
    for plan, *_ in plans:
        plan.close()


def test_batch_tunes_when_cells_leave_the_march(cuda, built_lib):
    """A plan first run on cells that march, then set to arrays off the march's
    8-byte boundary: its gather still times its launch shapes."""
    from rspacedist_b200 import kukan as K
    g, veff, dij, rp, psi = inputs(cell_of((34, 34, 34)), 20)
    plan = K.HpsiBatch([g], [20])
    out = torch.empty_like(psi)
    plan.set([veff], [dij], [rp], [psi], [out])
    plan.run()
    before = plan.info()
    out = shifted(psi)
    plan.set([shifted(veff)], [dij], [rp], [shifted(psi)], [out])
    plan.run()
    # (128 threads, 4 bands, 4 CTAs per SM is what a plan holds before it has timed
    # its shapes, and none of those it times)
    assert before == {"threads_per_cta": 128, "bands_per_item": 4, "ctas_per_sm": 4}
    assert plan.info() != before
    assert float((out - K.hpsi(g, veff, dij, rp, psi)).abs().max()) <= 2e-6 * float(out.abs().max())
    plan.close()


def test_f64_off_a_boundary(cuda, built_lib):
    """FP64 H psi of arrays eight bytes past a 16-byte boundary takes the gather, which
    has the march's bits; each array alone is enough."""
    from rspacedist_b200 import kukan as K
    g, veff, dij, rp, psi = inputs(cell_of((18, 12, 10)), 3)
    veff, psi = veff.double(), psi.double()
    ref = K.hpsi(g, veff, dij, rp, psi)
    assert torch.equal(K.hpsi(g, shifted(veff), dij, rp, psi), ref)
    assert torch.equal(K.hpsi(g, veff, dij, rp, shifted(psi)), ref)
    assert torch.equal(K.hpsi(g, veff, dij, rp, psi, out=shifted(psi)), ref)


def test_reported_shape(cuda, built_lib):
    """The FP32 H psi has one launch shape, reported before and after its calls."""
    import ctypes as C
    from rspacedist_b200 import kukan as K, lib
    g, *ins = inputs(cell_of((10, 10, 10)), 64)
    for _ in range(2):
        chunk, bands = C.c_int(0), C.c_int(0)
        lib.call("rs_hpsi_f32_tuning", g.handle, C.byref(chunk), C.byref(bands))
        assert (chunk.value, bands.value) == (-1, 16)
        K.hpsi(g, *ins)


def test_s_psi_band_limit(cuda, built_lib):
    """More bands than a launch's grid can count are refused before anything runs."""
    from rspacedist_b200 import kukan as K, lib
    g = K.Geometry(cell_of((10, 10, 10)))
    assert built_lib.rs_spsi_f64(g.handle, None, None, None, None, 262141, None) == -1
    assert "262140" in lib.last_error()
