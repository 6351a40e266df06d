"""Products issued back to back (-m gpu): the launches of a product overlap
one another, so every vector must be the one just written.  A sequence of
products of changing vectors, operators, precisions and numbers of columns on
one stream, without a wait between them, equals the same products one by one
bit for bit.  Overlapped launches take no longer than one after the other.
"""
import numpy as np
import pytest
from synth import synthetic_hmat

from bigwham_dev_b200 import HmatGpu

pytestmark = pytest.mark.gpu


# unstaged launches alone (teams of warps), both kernels, the CTA-wide one alone
@pytest.mark.parametrize("npr,npc,dof,leaf,tuning", [(300, 300, 2, 20, {}), (400, 260, 3, 16, {"narrow_rows": 16}),
                                                     (600, 600, 2, 32, {"narrow_rows": 0})])
def test_back_to_back_equals_one_by_one(npr, npc, dof, leaf, tuning):
    import torch

    arr = synthetic_hmat(npr, npc, dof, seed=npr + npc + leaf, leaf=leaf, rank0_share=0.2)
    h = HmatGpu.from_flat(arr.dof, arr.n_rows, arr.n_cols, arr.fr, arr.lr, arr.fr_data, arr.lr_data, arr.perm0,
                          arr.perm1, device=0, precisions=("fp64", "fp32", "bf16"), transpose=True, matmat=True,
                          tuning=tuning)
    rng = np.random.default_rng(0)
    calls = []
    for k in range(60):
        tr, cols = bool(rng.integers(2)), int(rng.choice([1, 1, 3, 8]))
        X = torch.from_numpy(rng.uniform(-1, 1, (cols, arr.n_rows if tr else arr.n_cols))).cuda()
        calls.append((("fp64", "fp32", "bf16")[k % 3], tr, X))

    def run(prec, tr, X):
        return h.matvec(X[0], prec, transpose=tr) if len(X) == 1 else h.matmat(X.t(), prec, transpose=tr)

    want = []
    for c in calls:
        want.append(run(*c).clone())
        h.sync()
    for _ in range(3):
        got = [run(*c) for c in calls]
        h.sync()
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    h.close()


def _long_items(n, k, prec, rng):
    """k rank-1 blocks of 8 rows side by side: k items of n columns in phase 1."""
    A, B = rng.uniform(-1, 1, (k, 8)), rng.uniform(-1, 1, (k, n))
    h = HmatGpu(1, 8, k * n, np.arange(8), np.arange(k * n), device=0)
    for j in range(k):
        h.add_lowrank(0, j * n, A[j][:, None], B[j][None, :])
    return h.finalize(precisions=(prec,)), A, B


@pytest.mark.parametrize("prec,tol", [("fp64", 1e-13), ("fp32", 2e-6), ("bf16", 1e-2)])
@pytest.mark.parametrize("chunks", [5, 6, 7, 31, 32, 33, 65])
def test_long_items_around_the_stages_and_batches(prec, tol, chunks):
    """First items of as many chunks as the stages (6) and the descriptor
    batches (32) hold, more or less, on fewer and on more items than CTAs."""
    import torch

    rng = np.random.default_rng(chunks)
    for k in (1, 5, 200):
        n = chunks * (256 if prec == "fp64" else 512) - 3
        h, A, B = _long_items(n, k, prec, rng)
        for _ in range(3):
            x = rng.uniform(-1, 1, (k, n))
            y = h.matvec(torch.from_numpy(x.ravel()).cuda(), prec).cpu().numpy()
            want = A.T @ (B * x).sum(1)
            # against the size of what is summed: |A| (|B| |x|), which the sums cancel from
            assert np.linalg.norm(y - want) <= tol * np.linalg.norm(abs(A).T @ np.linalg.norm(B * x, axis=1))
        h.sync()
        h.close()


@pytest.mark.parametrize("n", [70_000, 80_000])
def test_one_long_item_among_short_ones(n):
    """FP64 phases whose longest item takes over 4.8 MB of 8 rows keep their SMs
    to themselves (the 80,000 columns), the short items' launch after them."""
    import torch

    rng = np.random.default_rng(n)
    k, m, r = 400, 300, 3
    A, B = rng.uniform(-1, 1, (8, 1)), rng.uniform(-1, 1, (1, n))
    h = HmatGpu(1, 8, n + k * m, np.arange(8), np.arange(n + k * m), device=0)
    h.add_lowrank(0, 0, A, B)
    short = [(rng.uniform(-1, 1, (8, r)), rng.uniform(-1, 1, (r, m))) for _ in range(k)]
    for j, (a, b) in enumerate(short):
        h.add_lowrank(0, n + j * m, a, b)
    h.finalize(precisions=("fp64",))
    p = h.plan_export("fp64", 1, with_data=False)
    assert (p["n_wide"], len(p["item_ptr"]) - 1) == (1, 1 + k)
    for _ in range(3):
        x = rng.uniform(-1, 1, n + k * m)
        y = h.matvec(torch.from_numpy(x).cuda()).cpu().numpy()
        want = A @ (B @ x[:n]) + sum(a @ (b @ x[n + j * m:n + (j + 1) * m]) for j, (a, b) in enumerate(short))
        assert np.linalg.norm(y - want) <= 1e-13 * np.linalg.norm(abs(A) @ (abs(B) @ abs(x[:n])))
    h.close()


@pytest.mark.parametrize("prec", ["fp64", "fp32", "bf16"])
def test_long_items_go_to_ctas_of_their_own(prec):
    """One long item per CTA (148 of 20,000 columns) and a gather of 3 million
    values, beside which the CTAs of phase 1 start one after the other: each
    item is some CTA's first, so phase 1 takes one item's time as it does after
    the gather (launch by launch timing).  When the first CTAs took three each,
    FP64 took 122 us against 101 launch by launch; one each, 64 against 87."""
    import torch

    n, k = 20_000, 148
    rng = np.random.default_rng(0)
    h, _, _ = _long_items(n, k, prec, rng)
    x = torch.from_numpy(rng.uniform(-1, 1, k * n)).cuda()
    y = torch.empty(8, dtype=torch.float64, device="cuda")
    for _ in range(3):
        h.matvec(x, prec, out=y)
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    ev[0].record()
    for _ in range(20):
        h.matvec(x, prec, out=y)
    ev[1].record()
    h.sync()
    h.set_timing(True)
    for _ in range(20):
        h.matvec(x, prec, out=y)
    h.sync()
    ms, count = h.timing_read_launches()
    assert count == 20 and ev[0].elapsed_time(ev[1]) < sum(ms)
    h.close()


def test_64_columns_deal_their_items_evenly():
    """The tensor-core product's phase 1, whose CTAs also start one after the
    other beside the gather of X: an item per CTA takes half the time of two
    (0.185 and 0.365 ms; 0.213 and 0.359 when the first CTAs took three each)."""
    import torch

    ms = []
    for k in (148, 296):
        n = 8_000
        rng = np.random.default_rng(0)
        h = HmatGpu(1, 8, k * n, np.arange(8), np.arange(k * n), device=0)
        for j in range(k):
            h.add_lowrank(0, j * n, rng.uniform(-1, 1, (8, 1)), rng.uniform(-1, 1, (1, n)))
        h.finalize(precisions=("bf16",), matmat=True)
        X = torch.from_numpy(rng.uniform(-1, 1, (64, k * n))).cuda().t()
        Y = torch.empty((64, 8), dtype=torch.float64, device="cuda").t()
        for _ in range(3):
            h.matmat(X, "bf16", out=Y)
        ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        ev[0].record()
        for _ in range(10):
            h.matmat(X, "bf16", out=Y)
        ev[1].record()
        h.sync()
        ms.append(ev[0].elapsed_time(ev[1]) / 10)
        h.close()
    assert ms[1] > 1.8 * ms[0]
