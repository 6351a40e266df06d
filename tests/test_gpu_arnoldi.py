"""The Arnoldi step's kernels (bw_arnoldi_step) on the GPU (-m gpu) against the
same Gmres on CPU tensors: basis, Hessenberg matrix and solutions, for vectors
shorter than a warp, around a CTA's slice and longer than the CTAs' threads,
the three kinds of preconditioner, and an exhausted Krylov space.  Cycles that
go over to vector operations at a later step, and no slower cycle than with
those alone."""
import numpy as np
import pytest

from bigwham_dev_b200.solve import Gmres

pytestmark = pytest.mark.gpu


def _pair(op_matrix, n, m, minv, seed):
    import torch

    out = []
    for dev in ("cpu", "cuda"):
        A = op_matrix.to(dev)
        d = minv.to(dev) if torch.is_tensor(minv) else minv
        g = Gmres(lambda x, y, A=A: torch.mul(A, x, out=y) if A.dim() == 1 else torch.mv(A, x, out=y), n, m, d,
                  device=dev, use_graph=dev == "cuda")
        b = torch.randn(n, dtype=torch.float64, generator=torch.Generator().manual_seed(seed)).to(dev)
        g.V[0].copy_(b / torch.linalg.vector_norm(b))
        g._run_cycle()
        V, H = g.V.cpu().clone(), g.H.cpu().clone()  # solve() writes them again
        out.append((V, H, g.solve(b, tol=1e-10, maxiter=5 * m)[0].cpu()))
    return out


@pytest.mark.parametrize("kind", ["none", "vector", "callable"])
@pytest.mark.parametrize("n,m", [(1, 1), (5, 3), (31, 8), (64, 20), (700, 33), (9473, 12), (90000, 6), (700, 70),
                                 (700000, 9)])
def test_cycle_equals_the_cpu_cycle(n, m, kind):
    import torch

    g = torch.Generator().manual_seed(n + m)
    if n <= 1000:
        M = torch.eye(n, dtype=torch.float64) + 0.5 / n ** 0.5 * torch.randn(n, n, dtype=torch.float64, generator=g)
    else:  # a diagonal operator: its Krylov spaces are as deep as its distinct values
        M = 1.0 + torch.rand(n, dtype=torch.float64, generator=g)
    minv = None if kind == "none" else 0.5 + torch.rand(n, dtype=torch.float64, generator=g)
    if kind == "callable":
        minv = lambda v, out: torch.mul(v, 0.75, out=out)  # noqa: E731
    (Vc, Hc, xc), (Vg, Hg, xg) = _pair(M, n, m, minv, n)
    # rounding grows with the steps as the Krylov vectors become dependent:
    # 1e-16 n^(1/2) a product, amplified by the subdiagonal's decay
    assert torch.linalg.norm(Hg - Hc) <= 1e-9 * torch.linalg.norm(Hc)
    assert torch.linalg.norm(Vg - Vc) <= 1e-7 * torch.linalg.norm(Vc)
    assert torch.linalg.norm(xg - xc) <= 1e-8 * torch.linalg.norm(xc)
    live = Vg.abs().sum(1) > 0
    gram = Vg[live] @ Vg[live].t()
    assert torch.linalg.norm(gram - torch.eye(int(live.sum()), dtype=torch.float64)) <= 1e-12 * m


def test_exhausted_space_gives_zero_vectors():
    import torch

    n = 500
    d = torch.ones(n, dtype=torch.float64)
    d[::2] = 2.0  # two distinct values: the space has dimension two
    (Vc, Hc, xc), (Vg, Hg, xg) = _pair(d, n, 5, None, 3)
    assert float(Hg[2, 1]) == 0.0 == float(Hc[2, 1])
    assert not Vg[2:].any() and np.allclose(xg, xc, rtol=1e-12)


@pytest.mark.parametrize("n,m", [(20000, 300), (196608, 100), (531111, 30), (2000000, 6)])
def test_long_cycles_are_no_slower_than_vector_operations(n, m):
    """Steps of long vectors or deep cycles: the kernels alone took 1.3 to 2.5
    times the vector operations' time; a quarter is allowed for noise."""
    import torch

    ms = []
    for work in (True, False):
        d = 1.0 + torch.rand(n, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
        g = Gmres(lambda x, y, d=d: torch.mul(d, x, out=y), n, m, 1.0 / d + 0.1)
        if not work:
            g._work = None
        g.V[0].fill_(n ** -0.5)
        for _ in range(3):
            g._run_cycle()
        ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        ev[0].record()
        for _ in range(5):
            g._run_cycle()
        ev[1].record()
        torch.cuda.synchronize()
        ms.append(ev[0].elapsed_time(ev[1]))
    assert ms[0] <= 1.25 * ms[1], ms
