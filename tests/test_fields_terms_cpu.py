"""The element fields of bw_s0.h and bw_r0_fields.h against their closed forms
taken term by term (end by end, corner by corner) in extended precision.

The headers combine the ends and corners before they divide or take a
logarithm or an angle; near an end or an edge, close to the element's plane
and far away the combined forms must lose nothing.  Bar: four times the largest
error that the term-by-term forms show in double precision on the same points
(over a dozen draws the ratio is at most 2.9, mostly below 1.5), or 2e-15.
"""
import numpy as np
import pytest
from test_fields_cpu import G, NU, probe  # noqa: F401

LD = np.longdouble
PI = LD("3.14159265358979323846264338327950288")


def s0_terms(rec, dd, pts, T=LD):
    rec, dd, pts = rec.astype(T), dd.astype(T), pts.astype(T)
    nu, g = T(NU), T(G)
    c = 1 / (4 * T(PI) * (1 - nu))
    S, U = np.zeros((len(pts), 3), T), np.zeros((len(pts), 2), T)
    for (cx, cy, a, tx, ty), (ds, dn) in zip(rec, dd.reshape(-1, 2)):
        nx, ny = -ty, tx
        dx, dy = pts[:, 0] - cx, pts[:, 1] - cy
        x, y = tx * dx + ty * dy, nx * dx + ny * dy
        xm, xp = x - a, x + a
        r1, r2 = xm * xm + y * y, xp * xp + y * y
        ys = np.where(y == 0, T(-0.0), y)  # on the line, from below
        fx, fy = c / 2 * (np.log(r1) - np.log(r2)), -c * (np.arctan2(ys, xm) - np.arctan2(ys, xp))
        fxy, fyy = c * (y / r1 - y / r2), -c * (xm / r1 - xp / r2)
        fxyy = c * ((xm * xm - y * y) / r1 ** 2 - (xp * xp - y * y) / r2 ** 2)
        fyyy = 2 * c * y * (xm / r1 ** 2 - xp / r2 ** 2)
        sxx = 2 * g * (ds * (2 * fxy + y * fxyy) + dn * (fyy + y * fyyy))
        syy = 2 * g * (-ds * y * fxyy + dn * (fyy - y * fyyy))
        sxy = 2 * g * (ds * (fyy + y * fyyy) - dn * y * fxyy)
        ux = ds * (2 * (1 - nu) * fy + y * fyy) - dn * ((1 - 2 * nu) * fx + y * fxy)
        uy = ds * ((1 - 2 * nu) * fx - y * fxy) + dn * (2 * (1 - nu) * fy - y * fyy)
        S += np.stack([sxx * tx * tx + syy * nx * nx + 2 * sxy * tx * nx,
                       sxx * ty * ty + syy * ny * ny + 2 * sxy * ty * ny,
                       sxx * tx * ty + syy * nx * ny + sxy * (tx * ny + nx * ty)], 1)
        U += np.stack([ux * tx + uy * nx, ux * ty + uy * ny], 1)
    return S, U


def r0_terms(rec, dd, pts, T=LD):
    rec, dd, pts = rec.astype(T), dd.astype(T), pts.astype(T)
    nu, g = T(NU), T(G)
    S, U = np.zeros((len(pts), 6), T), np.zeros((len(pts), 3), T)
    for el, (d0, d1, d2) in zip(rec, dd.reshape(-1, 3)):
        R = el[3:12].reshape(3, 3)
        x, y, z = ((pts - el[:3]) @ R.T).T
        a, b = el[15], el[16]
        d = {}
        for sx in (1, -1):
            for sy in (1, -1):
                s, X, Y = sx * sy, x + sx * a, y + sy * b
                r = np.sqrt(X * X + Y * Y + z * z)
                terms = {"z": -np.arctan(X * Y / (z * r)), "xy": 1 / r, "xxy": -X / r ** 3, "xyy": -Y / r ** 3,
                         "xyz": -z / r ** 3,
                         "zz": X * Y * (X * X + Y * Y + 2 * z * z) / (r * (X * X + z * z) * (Y * Y + z * z))}
                for k, (P, Q) in {"x": (X, Y), "y": (Y, X)}.items():
                    w = np.where(Q >= 0, r + Q, (P * P + z * z) / (r - Q))
                    terms.update({k: np.log(w), k * 2: P / (r * w), k + "z": z / (r * w),
                                  k * 3: (r * w - P * P * (2 * r + Q) / r) / (r * w) ** 2,
                                  k * 2 + "z": -P * z * (2 * r + Q) / (r ** 3 * w * w),
                                  k + "zz": (r * w - z * z * (2 * r + Q) / r) / (r * w) ** 2})
                for k, v in terms.items():
                    d[k] = d.get(k, 0) + s * v
        zzz = -(d["xxz"] + d["yyz"])
        Cs, c, k1, k2 = g / (4 * T(PI) * (1 - nu)), 1 / (8 * T(PI) * (1 - nu)), 2 * (1 - nu), 1 - 2 * nu
        xx = d0 * (2 * d["xz"] - z * d["xxx"]) + d1 * (2 * nu * d["yz"] - z * d["xxy"])
        xx = xx + d2 * (d["zz"] + k2 * d["yy"] - z * d["xxz"])
        yy = d0 * (2 * nu * d["xz"] - z * d["xyy"]) + d1 * (2 * d["yz"] - z * d["yyy"])
        yy = yy + d2 * (d["zz"] + k2 * d["xx"] - z * d["yyz"])
        zz = -d0 * z * d["xzz"] - d1 * z * d["yzz"] + d2 * (d["zz"] - z * zzz)
        xy = d0 * ((1 - nu) * d["yz"] - z * d["xxy"]) + d1 * ((1 - nu) * d["xz"] - z * d["xyy"])
        xy = xy - d2 * (k2 * d["xy"] + z * d["xyz"])
        xz = d0 * (d["zz"] + nu * d["yy"] - z * d["xxz"]) - d1 * (nu * d["xy"] + z * d["xyz"]) - d2 * z * d["xzz"]
        yz = -d0 * (nu * d["xy"] + z * d["xyz"]) + d1 * (d["zz"] + nu * d["xx"] - z * d["yyz"]) - d2 * z * d["yzz"]
        T = Cs * np.stack([xx, xy, xz, xy, yy, yz, xz, yz, zz], -1).reshape(-1, 3, 3)
        T = np.einsum("ki,pkl,lj->pij", R, T, R)
        S += np.stack([T[:, 0, 0], T[:, 1, 1], T[:, 2, 2], T[:, 0, 1], T[:, 0, 2], T[:, 1, 2]], 1)
        U += c * np.stack([
            d0 * (k1 * d["z"] - z * d["xx"]) - d1 * z * d["xy"] - d2 * (k2 * d["x"] + z * d["xz"]),
            -d0 * z * d["xy"] + d1 * (k1 * d["z"] - z * d["yy"]) - d2 * (k2 * d["y"] + z * d["yz"]),
            d0 * (k2 * d["x"] - z * d["xz"]) + d1 * (k2 * d["y"] - z * d["yz"]) + d2 * (k1 * d["z"] - z * d["zz"])],
            -1) @ R
    return S, U


def _off(a, b):
    b = b.astype(np.float64)
    return float(np.max(np.linalg.norm(a - b, axis=1) / np.linalg.norm(b, axis=1)))


def _no_worse(got, terms, want):
    """Largest relative error of a point's vector against the term-by-term form's."""
    return _off(got, want) < max(4 * _off(terms, want), 2e-15)


# points around one element of half length 1 (half sides 1 and 0.8)
WHERE = {
    "around": lambda r, n, k: r.uniform(-2, 2, (n, k)),
    "close": lambda r, n, k: np.column_stack([r.uniform(-2, 2, (n, k - 1)),
                                              10.0 ** r.uniform(-6, -1, n) * r.choice([-1, 1], n)]),
    "end": lambda r, n, k: np.eye(k)[0] + 1e-4 * r.standard_normal((n, k)),
    # far away the ends and corners cancel by (size / distance)^2 or more
    "far": lambda r, n, k: 30.0 * r.uniform(-2, 2, (n, k)),
}


@pytest.mark.parametrize("where", WHERE)
def test_s0_combined_ends(probe, where):
    pts = np.ascontiguousarray(WHERE[where](np.random.default_rng(3), 400, 2))
    rec, dd = np.array([[0.0, 0.0, 1.0, 1.0, 0.0]]), np.array([0.7, 1.3])
    s, u = np.empty((400, 3)), np.empty((400, 2))
    probe.probe_s0_fields(1, rec, dd, G, NU, 400, pts, s, u)
    S, U = s0_terms(rec, dd, pts)
    Sd, Ud = s0_terms(rec, dd, pts, np.float64)
    assert _no_worse(s, Sd, S) and _no_worse(u, Ud, U)


@pytest.mark.parametrize("x", [0.3, -0.7, 1.5, -2.0])
def test_s0_on_the_line(probe, x):
    """The limit from below on the element's line, inside and beyond it."""
    rec, dd, pts = np.array([[0.0, 0.0, 1.0, 1.0, 0.0]]), np.array([0.7, 1.3]), np.array([[x, 0.0]])
    s, u = np.empty((1, 3)), np.empty((1, 2))
    probe.probe_s0_fields(1, rec, dd, G, NU, 1, pts, s, u)
    S, U = s0_terms(rec, dd, pts)
    assert _off(s, S) < 1e-14 and _off(u, U) < 1e-14


@pytest.mark.parametrize("where", WHERE)
def test_r0_combined_corners(probe, where):
    pts = np.ascontiguousarray(WHERE[where](np.random.default_rng(4), 400, 3))
    rec = np.hstack([np.zeros(3), np.eye(3).ravel(), [0, 0, 1.0], [1.0, 0.8]])[None, :].copy()
    dd = np.array([0.7, -0.4, 1.3])
    s, u = np.empty((400, 6)), np.empty((400, 3))
    probe.probe_r0_fields(1, rec, dd, G, NU, 400, pts, s, u)
    S, U = r0_terms(rec, dd, pts)
    Sd, Ud = r0_terms(rec, dd, pts, np.float64)
    assert _no_worse(s, Sd, S) and _no_worse(u, Ud, U)
