"""Host threads with sizes of their own at work at once: the dynamic shared memory
a kernel may take is the device's, not the call's, so no call may lower it."""
import ctypes as C
import threading

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def nl_dot(P, nb):
    import conftest
    from rspacedist_b200 import kukan as K
    from test_gpu_nl_dot import widened
    cell = widened(conftest.make_si8(20, 0.05, 4), P)
    g, psi = K.Geometry(cell), torch.ones((nb, cell.N), dtype=torch.float64, device="cuda")
    return lambda: K.nonlocaloperation_01(g, psi)


def chol(n, _):
    from rspacedist_b200 import lib
    G = 2.0 * torch.eye(n, dtype=torch.float64, device="cuda")
    A, W = torch.empty_like(G), torch.empty_like(G)

    def call():
        A.copy_(G)
        lib.call("rs_chol_inv_t", n, C.c_void_p(A.data_ptr()), C.c_void_p(W.data_ptr()),
                 C.c_void_p(torch.cuda.current_stream().cuda_stream))
        return W.clone()
    return call


def diis(nx, f64):
    from rspacedist_b200 import kukan as K, lib, system as S
    cell = S.make_cell(0.3 * np.array([nx, 12, 12]), (nx, 12, 12), np.zeros((1, 3)),
                       S.load_dataset("c_ncps"))
    dtype = torch.float64 if f64 else torch.float32
    psi = torch.tensor(S.random_bands(cell, 2, 1), dtype=dtype, device="cuda")
    veff = torch.tensor(S.smooth_veff(cell, 1), dtype=dtype, device="cuda")
    dij = torch.tensor(cell.dij, dtype=torch.float64, device="cuda")
    g = K.Geometry(cell)

    def call():
        b = K.Bands(g, psi.clone())
        K.ksdiis(b, veff, dij, lib.solver_prm(ndiismax=2), l_hsv=0)
        return b.psi
    return call


@pytest.mark.parametrize("make,large,small,times", [(nl_dot, (32, 600), (5, 600), 6000),
                                                    (chol, (1000, 0), (40, 0), 2000),
                                                    (diis, (512, True), (20, True), 400)])
def test_sizes_of_threads(cuda, built_lib, make, large, small, times):
    """One thread calls with a large size, three with a small one for as long as it
    does."""
    jobs = [make(*large)] + [make(*small) for _ in range(3)]
    refs = [job() for job in jobs]
    wrong, over = [], threading.Event()

    def work(k):
        with torch.cuda.stream(torch.cuda.Stream()):
            n = 0
            try:
                while n < times if k == 0 else not over.is_set():
                    got, n = jobs[k](), n + 1
                    if n % 100 == 0:
                        torch.cuda.current_stream().synchronize()
                if not torch.equal(got, refs[k]):
                    wrong.append("another result")
            except Exception as e:
                wrong.append(str(e))
            finally:
                if k == 0:
                    over.set()

    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


def test_hartree_solves_of_two_threads(cuda, built_lib):
    """One-launch Poisson solves of nearly all SMs from two threads: each launch gets
    its CTAs together, so the barriers of neither wait for the other's."""
    from rspacedist_b200 import kukan as K
    jobs = []
    for shape, mixed in (((84, 84, 84), False), ((128, 128, 120), True)):
        gen = torch.Generator(device="cuda")
        gen.manual_seed(3)
        rho = torch.randn(int(np.prod(shape)), generator=gen, dtype=torch.float64, device="cuda")

        def job(shape=shape, mixed=mixed, rho=rho):
            vh = torch.zeros_like(rho)
            return K.scf_hartree(shape, 4, (6.0, 6.0, 6.0), rho, vh, ncgmax=60, mixed=mixed), vh
        jobs.append(job)
    refs, wrong = [job() for job in jobs], []

    def work(job, ref):
        with torch.cuda.stream(torch.cuda.Stream()):
            try:
                for _ in range(40):
                    got = job()
                    if got[0] != ref[0] or not torch.equal(got[1], ref[1]):
                        wrong.append("another result")
            except Exception as e:
                wrong.append(str(e))

    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=a) for a in zip(jobs, refs)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
