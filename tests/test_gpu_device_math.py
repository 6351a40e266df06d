"""Field and block-compression kernels on the GPU (-m gpu) against the host
builds of the same headers, at the sizes where the kernels' divisions of the
work have edges.

* Fields: points around a CTA's and a warp's share for every number of lanes
  per point, elements around the tile, each combination of outputs.
* Block ACA: blocks smaller and larger than the CTA and with sides that are
  not multiples of a warp, ranks on both sides of the 32 rank blocks one
  Frobenius pass takes, and a capacity too small.  The crack's spacing varies,
  so no pivots tie; the product A B then agrees to far below the compression's eps.
"""
import numpy as np
import pytest
from test_aca_cpu import lib  # noqa: F401
from test_fields_cpu import E, G, NU, host_fields, probe  # noqa: F401

pytestmark = pytest.mark.gpu


def _graded(nx, ny, bend, seed=0):
    """Records of a rectangle crack of uneven spacing; bend > 0 tilts each
    column of elements about its own axis (entries off the element plane)."""
    r = np.random.default_rng(seed)
    out = []
    gx, gy = (np.concatenate([[0.0], np.cumsum(r.uniform(0.8, 1.2, n))]) for n in (nx, ny))
    for j in range(ny):
        for i in range(nx):
            x, y = 0.5 * (gx[i] + gx[i + 1]), 0.5 * (gy[j] + gy[j + 1])
            t = bend * x
            R = np.array([[np.cos(t), 0, np.sin(t)], [0, 1.0, 0], [-np.sin(t), 0, np.cos(t)]])
            out.append(np.concatenate([[x, y, 0.1 * bend * x * x], R.ravel(), R[2],
                                       [0.45 * (gx[i + 1] - gx[i]), 0.45 * (gy[j + 1] - gy[j])]]))
    return np.ascontiguousarray(out)


@pytest.mark.parametrize("n_elems", [1, 31, 128, 129, 300])
@pytest.mark.parametrize("n_pts", [1, 3, 129, 9472, 9473, 40000, 310000])
def test_fields_lanes_and_tiles(probe, n_pts, n_elems):
    import torch

    from bigwham_dev_b200.fields import R0Fields, S0Fields

    rng = np.random.default_rng(n_pts + n_elems)
    pick = np.unique(np.concatenate([[0, n_pts - 1], rng.integers(0, n_pts, 40)]))
    x = np.linspace(-1, 1, n_elems + 1)
    coor, conn = np.column_stack([x, 0.2 * np.sin(3 * x)]), np.column_stack([np.arange(n_elems), np.arange(1, n_elems + 1)])
    rec = _graded(n_elems, 1, 0.05)
    for f, dim in ((S0Fields(coor, conn, E, NU), 2), (R0Fields(rec, E, NU), 3)):
        pts = rng.uniform(-2, 2, (n_pts, dim))
        dd = rng.uniform(-1, 1, dim * n_elems)
        p, d = torch.from_numpy(pts).cuda(), torch.from_numpy(dd).cuda()
        s, u = f.fields(p, d)
        s1, none = f.fields(p, d, want_disp=False)
        none2, u1 = f.fields(p, d, want_stress=False)
        assert none is None and none2 is None
        if dim == 2:
            ws, wu = host_fields(probe, coor, conn, dd, pts[pick])
        else:
            ws, wu = np.empty((len(pick), 6)), np.empty((len(pick), 3))
            probe.probe_r0_fields(n_elems, rec, dd, G, NU, len(pick), np.ascontiguousarray(pts[pick]), ws, wu)
        for got, want in ((s, ws), (s1, ws), (u, wu), (u1, wu)):
            got = got.cpu().numpy()
            assert np.isfinite(got).all()
            # host and device differ in the last bits of each element's terms;
            # close points amplify them by the cancellation between corners
            assert np.abs(got[pick] - want).max() <= 1e-11 * np.abs(want).max(), (n_pts, n_elems, dim)


@pytest.mark.parametrize("bend", [0.0, 0.02])
def test_aca_equals_the_host_build(lib, bend):
    from bigwham_dev_b200.devbuild import DeviceKernels, factor_layout

    rec = _graded(40, 30, bend)
    n = rec.shape[0]
    perm = np.arange(n, dtype=np.int64)
    # the last two touch: high ranks, over 32 rank blocks
    blocks = np.array([[0, 900, 5, 903], [10, 700, 41, 733], [0, 600, 128, 729], [0, 800, 300, 1200],
                       [100, 240, 233, 373], [0, 45, 45, 90]], np.int64)
    k = DeviceKernels()
    for cap in (48, 4):
        fa, fb, ranks, errs = k.aca(rec, G, NU, blocks, perm, 1e-5, cap)
        fa, fb = fa.cpu().numpy(), fb.cpu().numpy()
        n0, n1, capk, a_off, b_off = factor_layout(blocks, cap)
        for q, (i0, j0, i1, j1) in enumerate(blocks):
            m, c, w = 3 * int(n0[q]), 3 * int(capk[q]), 3 * int(n1[q])
            A, B, err = np.zeros(m * c), np.zeros(c * w), np.zeros(1)
            r = lib.probe_r0_aca(rec, G, NU, perm, i0, j0, i1, j1, 1e-5, int(capk[q]), A, B, err)
            assert ranks[q] == (3 * r if r > 0 else r), (cap, q, r, ranks[q])
            if r <= 0:
                continue
            dA, hA = fa[a_off[q]:a_off[q] + m * 3 * r].reshape(3 * r, m), A[:m * 3 * r].reshape(3 * r, m)
            dB, hB = fb[b_off[q]:b_off[q + 1]].reshape(w, c)[:, :3 * r], B.reshape(w, c)[:, :3 * r]
            want = hA.T @ hB.T
            assert np.linalg.norm(dA.T @ dB.T - want) <= 1e-9 * np.linalg.norm(want)
            # the first pivots and rank blocks, before the amplification
            assert np.linalg.norm(dA[:3] - hA[:3]) <= 1e-11 * np.linalg.norm(hA[:3])
            # the last rank block is eps of the norm: the entries' rounding
            # (1e-10 of the largest one, off the element plane) shows 1 / eps larger
            assert errs[q] == pytest.approx(err[0], rel=1e-4)
    assert (ranks == -1).any()
