"""Phase 2's slices of G2 as the device reads them (bw_plan_slices): the row
parts of a panel that are cut alike share theirs, everything else is apart, and
all stay inside G2.  Replays of the same plan against the oracle are in
test_layout.py and test_narrow_cpu.py (planreplay.device_phase2)."""
import numpy as np
import pytest
from planreplay import decode, gather_runs, slices
from synth import synthetic_hmat

from bigwham_dev_b200 import HmatGpu


def _check(h, precision, tr):
    """Checks the slices of one operator; returns how many chunks share."""
    g_len, sl, runs = slices(h, precision, tr)
    ds = [decode(w) for w in h.plan_export(precision, 2, tr, with_data=False)["chunks"]]
    assert len(ds) == len(sl)
    cols = (runs[:, 2].view(np.uint32) & 0x7FFFFFFF).astype(np.int64)
    every = gather_runs(h, precision, tr)  # the same runs, chunk by chunk
    at, used, places = 0, np.zeros(len(runs), np.int64), {}
    for d, (g, first, n) in zip(ds, sl.astype(np.int64)):
        own = runs[first:first + n].copy()
        # the runs fill the slice in order, and are those shown for the chunk
        assert list(own[:, 0] - g) == list(np.cumsum(cols[first:first + n]) - cols[first:first + n])
        assert cols[first:first + n].sum() == d["ncols"] and 0 <= g and g + d["ncols"] <= g_len
        own[:, 0] += d["g_off"] - g
        assert np.array_equal(own, every[at:at + n])
        at += n
        if d["ncols"] == 0:
            continue
        # one place, one content: shared slices are those of equal cuts
        assert places.setdefault(g, (d["ncols"], first, n, d["hpad"])) == (d["ncols"], first, n, d["hpad"])
        used[first:first + n] += 1
    assert at == len(every) and np.all(used > 0)
    ends = sorted((g, g + v[0]) for g, v in places.items())
    assert all(a[1] <= b[0] for a, b in zip(ends, ends[1:]))  # no slices overlap
    written = np.zeros(g_len, np.int64)
    for r, c in zip(runs[:, 0].astype(np.int64), cols):
        written[r:r + c] += 1
    assert written.max(initial=0) <= 1  # no place is gathered twice
    return len(ds) - len(places)


CASES = [(40, 25, 2, 4), (17, 60, 3, 8), (200, 130, 1, 32), (90, 70, 3, 32), (600, 600, 2, 32)]


@pytest.mark.parametrize("precision", ["fp64", "fp32", "bf16"])
def test_slices_of_synthetic_partitions(precision):
    shared = 0
    for npr, npc, dof, leaf in CASES:
        arr = synthetic_hmat(npr, npc, dof, seed=npr + npc + leaf, leaf=leaf, rank0_share=0.2)
        for tuning in ({}, {"chunk_bytes": 4096, "items_per_cta_phase2": 1}):
            h = HmatGpu.from_flat(arr.dof, arr.n_rows, arr.n_cols, arr.fr, arr.lr, arr.fr_data, arr.lr_data,
                                  arr.perm0, arr.perm1, device=-1, plan_only=True, precisions=(precision,),
                                  transpose=True, tuning=tuning)
            shared += _check(h, precision, False) + _check(h, precision, True)
    assert shared > 0  # some panels are cut into parts


@pytest.mark.parametrize("precision", ["fp64", "fp32", "bf16"])
def test_slices_of_the_golden_cases(golden, precision):
    arr, _ = golden
    h = HmatGpu.from_flat(arr.dof, arr.n_rows, arr.n_cols, arr.fr, arr.lr, arr.fr_data, arr.lr_data, arr.perm0,
                          arr.perm1, device=-1, plan_only=True, precisions=(precision,), transpose=True)
    _check(h, precision, False)
    _check(h, precision, True)
