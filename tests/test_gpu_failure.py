"""Failure detection on the GPU without faulting it (-m gpu).

bw_test_withhold_chunk makes CTA 0 of the next streaming launch skip staging
one chunk: a barrier that nothing completes.  With a 20 ms wait limit
(bw_set_wait_limit) the wait for it runs out.  The timed-out kernel:
* writes an error word;
* lets its bulk copies and tensor-core work finish (those waits keep a fixed
  2 s bound);
* frees its TMEM and returns.
The next sync reports BW_ERR_DEVICE.  With the default limit restored the same
handle gives the bitwise-same results as before: no state is left behind
(error word, work-queue counters, TMEM).  The limit counts from the end of the
launch before: a product whose phase 1 takes longer than the limit is healthy.
"""
import numpy as np
import pytest

from bigwham_dev_b200 import BigWhamError, HmatGpu
from bigwham_dev_b200 import _capi as A
from bigwham_dev_b200.meshes import square_crack_3d
from oracle import RefHmat

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def handle():
    coor, conn = square_crack_3d(48)
    arr = RefHmat("3DR0-H", coor, conn, [1.0, 0.25], 32, 3.0, 1e-5, n_threads=16).arrays()
    return HmatGpu.from_flat(arr.dof, arr.n_rows, arr.n_cols, arr.fr, arr.lr, arr.fr_data, arr.lr_data, arr.perm0,
                             arr.perm1, device=0, precisions=("fp64", "bf16"), matmat=True)


def test_timeout_reported_and_handle_recovers(handle):
    import torch

    h = handle
    x = torch.from_numpy(np.random.default_rng(0).uniform(-1, 1, h.n_cols)).cuda()
    X = torch.from_numpy(np.random.default_rng(1).uniform(-1, 1, (h.n_cols, 8))).cuda()
    good = {p: h.matvec(x, p).clone() for p in ("fp64", "bf16")}
    good_mm = h.matmat(X, "bf16").clone()
    h.sync()
    h.set_wait_limit(20_000_000)
    for run in (lambda: h.matvec(x, "fp64"), lambda: h.matvec(x, "bf16"), lambda: h.matmat(X, "bf16")):
        A.check(A.lib().bw_test_withhold_chunk(h._h, 1), h._h)
        run()
        with pytest.raises(BigWhamError) as e:
            h.sync()
        assert e.value.status == A.BW_ERR_DEVICE
        assert "error word" in str(e.value)
    h.set_wait_limit(2_000_000_000)
    for p in ("fp64", "bf16"):
        assert torch.equal(h.matvec(x, p), good[p])
    assert torch.equal(h.matmat(X, "bf16"), good_mm)
    h.sync()


def test_wait_limit_range_checked(handle):
    for bad in (0, -5, 10 ** 12):
        with pytest.raises(BigWhamError) as e:
            handle.set_wait_limit(bad)
        assert e.value.status == A.BW_ERR_ARG


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_timeout_of_several_columns(prec):
    """The same for the products of several columns (passes of 8 and 4): some
    nine items per CTA in phase 1, all of them CTA-wide."""
    import torch

    nb, bs, r = 64, 64, 8
    n = nb * bs
    rng = np.random.default_rng(0)
    h = HmatGpu(1, n, n, np.arange(n), np.arange(n), device=0).set_tuning(narrow_rows=0)
    fr = np.zeros((0, 4), np.int64)
    lr = np.array([(i * bs, j * bs, (i + 1) * bs, (j + 1) * bs, r) for i in range(nb) for j in range(nb)], np.int64)
    h.add_flat(fr, lr, np.zeros(0), rng.standard_normal(nb * nb * 2 * r * bs))
    h.finalize(precisions=(prec,))
    X, other = (torch.from_numpy(rng.uniform(-1, 1, (8, n))).cuda().t() for _ in range(2))
    good = {k: h.matmat(X[:, :k], prec).clone() for k in (8, 3)}
    h.sync()
    for k in good:
        h.set_wait_limit(20_000_000)
        h.matmat(other[:, :k], prec)  # what the lost chunk's products are then replaced by
        A.check(A.lib().bw_test_withhold_chunk(h._h, 1), h._h)
        Y = h.matmat(X[:, :k], prec)
        with pytest.raises(BigWhamError) as e:
            h.sync()
        assert e.value.status == A.BW_ERR_DEVICE and "error word" in str(e.value)
        # one pass holds all columns, so the chunk is lost to each of them
        assert not any(torch.equal(Y[:, j], good[k][:, j]) for j in range(k))
        h.set_wait_limit(2_000_000_000)
        for q in good:
            assert torch.equal(h.matmat(X[:, :q], prec), good[q])
        h.sync()
    h.close()


@pytest.mark.parametrize("prec", ["fp64", "fp32", "bf16"])
def test_timeout_of_long_items(prec):
    """The same where the CTAs take their first items one by one: long items,
    the withheld chunk in a CTA's first one (before or after it has its next)."""
    import torch

    n, k = 20_000, 200
    rng = np.random.default_rng(0)
    h = HmatGpu(1, 8, k * n, np.arange(8), np.arange(k * n), device=0)
    for j in range(k):
        h.add_lowrank(0, j * n, rng.uniform(-1, 1, (8, 1)), rng.uniform(-1, 1, (1, n)))
    h.finalize(precisions=(prec,))
    x = torch.from_numpy(rng.uniform(-1, 1, k * n)).cuda()
    good = h.matvec(x, prec).clone()
    h.sync()
    for chunk in (0, 5, 6, 38):
        h.set_wait_limit(20_000_000)
        A.check(A.lib().bw_test_withhold_chunk(h._h, chunk), h._h)
        h.matvec(x, prec)
        with pytest.raises(BigWhamError) as e:
            h.sync()
        assert e.value.status == A.BW_ERR_DEVICE and "error word" in str(e.value)
        h.set_wait_limit(2_000_000_000)
        assert torch.equal(h.matvec(x, prec), good)
        h.sync()
    h.close()


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_the_limit_is_a_stage_s_not_the_launch_before_s(prec):
    """A phase-2 CTA may get its SM while phase 1 still runs elsewhere (here on
    one CTA: a single item of a million columns) and waits for it.  That wait
    does not count: a limit well below the phase's time, and well above any
    stage's, reports nothing."""
    import torch

    n, m, k, limit_us = 1 << 20, 64, 8, 300
    rng = np.random.default_rng(0)
    h = HmatGpu(1, m, n, np.arange(m), np.arange(n), device=0).set_tuning(narrow_rows=0)
    h.add_lowrank(0, 0, rng.uniform(-1, 1, (m, 1)), rng.uniform(-1, 1, (1, n)))
    h.finalize(precisions=(prec,))
    X = torch.from_numpy(rng.uniform(-1, 1, (k, n))).cuda().t()
    want, want1 = h.matmat(X, prec).clone(), h.matvec(X[:, 0], prec).clone()
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    h.sync()
    ev[0].record()
    h.matmat(X, prec)
    ev[1].record()
    h.sync()
    assert ev[0].elapsed_time(ev[1]) > 2e-3 * limit_us  # else the limit tests nothing
    h.set_wait_limit(1000 * limit_us)
    for _ in range(5):
        Y, y = h.matmat(X, prec), h.matvec(X[:, 0], prec)
        h.sync()
        assert torch.equal(Y, want) and torch.equal(y, want1)
    h.close()
