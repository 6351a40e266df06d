"""Products issued back to back (-m gpu): the launches of a product overlap
one another, so every vector must be the one just written.  A sequence of
products of changing vectors, operators, precisions and numbers of columns on
one stream, without a wait between them, equals the same products one by one
bit for bit.
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
