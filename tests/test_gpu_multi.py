"""FP64 / FP32 products of several columns (bw_matmat, passes of 8 and 4
columns) on the GPU (-m gpu).

The multi-column kernels keep the matvec's arithmetic order in every column,
so each column must equal the matvec of that column bit for bit; the matvec
itself is checked against the oracle elsewhere.  Counts of columns around the
passes' edges (a single one left over, up to 4, up to 8), both kernels of the
phase split (with narrow_coop 1 units run CTA-cooperatively, and the columns go
one by one through the matvec), ragged partitions, rank-0 blocks, H and H^T, both orderings and
padded leading dimensions.
"""
import numpy as np
import pytest
from synth import synthetic_hmat

from bigwham_dev_b200 import HmatGpu

pytestmark = pytest.mark.gpu


def _check(h, prec, k, transpose, permuted, seed, pad=0):
    import torch

    nin, nout = (h.n_rows, h.n_cols) if transpose else (h.n_cols, h.n_rows)
    g = torch.Generator(device="cuda").manual_seed(seed)
    buf = torch.randn(k, nin + pad, dtype=torch.float64, device="cuda", generator=g)
    X = buf[:, :nin].t()
    Y = torch.full((k, nout + pad), float("nan"), dtype=torch.float64, device="cuda")
    h.matmat(X, prec, permuted=permuted, transpose=transpose, out=Y[:, :nout].t())
    h.sync()
    for j in range(k):
        y = h.matvec(X[:, j].contiguous(), prec, permuted=permuted, transpose=transpose)
        assert torch.equal(Y[j, :nout], y), (prec, k, j, transpose, permuted)
    assert torch.isnan(Y[:, nout:]).all()  # nothing written past a column


@pytest.mark.parametrize("tuning", [{}, {"narrow_rows": 0}, {"narrow_rows": 16, "chunk_bytes": 4096},
                                    {"narrow_coop": 1}], ids=str)
@pytest.mark.parametrize("npr,npc,dof,leaf", [(600, 600, 2, 32), (400, 260, 3, 16)])
def test_columns_equal_matvecs(npr, npc, dof, leaf, tuning):
    arr = synthetic_hmat(npr, npc, dof, seed=npr + npc + leaf, leaf=leaf, rank0_share=0.2)
    h = HmatGpu.from_flat(arr.dof, arr.n_rows, arr.n_cols, arr.fr, arr.lr, arr.fr_data, arr.lr_data, arr.perm0,
                          arr.perm1, device=0, precisions=("fp64", "fp32"), transpose=True, tuning=tuning)
    for i, k in enumerate((1, 2, 4, 5, 8, 9, 11, 17)):
        for prec in ("fp64", "fp32"):
            _check(h, prec, k, bool(i & 1), bool(i & 2), 10 * k, pad=3 * (i & 1))
            _check(h, prec, k, not (i & 1), bool(i & 2), 10 * k + 1)
    h.close()


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_thin_long_and_tall_items(prec):
    """Items of 8 padded rows with thousands of columns (the widest vector
    windows) and of 512 rows (the smallest chunks), one full block each."""
    for m, n in ((5, 3001), (1500, 7), (1, 1)):
        h = HmatGpu(1, m, n, np.arange(m), np.arange(n), device=0)
        h.add_full(0, 0, np.random.default_rng(m).standard_normal((m, n)))
        h.finalize(precisions=(prec,), transpose=True)
        for k in (3, 8):
            _check(h, prec, k, False, False, k)
            _check(h, prec, k, True, True, k)
        h.close()
