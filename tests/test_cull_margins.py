"""The cone test of the traversal (may_hit) may drop no leaf that the exact test hits: both restated in FP32 on
the CPU, a tile of rays around the rim of a flat or long Gaussian whose axes differ by up to 1e5, near and
far, with wide and narrow tiles.  The kernel's reciprocal square roots and divisions are a few ulps off; the
restatement moves each by up to 3 ulps at random."""
import numpy as np
import pytest

F = np.float32
ULP = F(2.0 ** -23)


def _dot(a, b):
    return a[..., 0] * b[..., 0] + a[..., 1] * b[..., 1] + a[..., 2] * b[..., 2]


def _norm(a):
    return np.sqrt(_dot(a, a))


def _scene(rng, n, scales, dist, px, density):
    """Rotations, eye, mean, camera axes and the directions (dx, dy) of one 8x4 tile per Gaussian, which looks at
    a point at 0.9 to 1.02 of its threshold ellipsoid's silhouette."""
    q = rng.normal(size=(n, 4))
    w, x, y, z = (q / np.linalg.norm(q, axis=1)[:, None]).T
    R = np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y), 2 * (x * y + w * z),
                  1 - 2 * (x * x + z * z), 2 * (y * z - w * x), 2 * (x * z - w * y), 2 * (y * z + w * x),
                  1 - 2 * (x * x + y * y)], 1).reshape(-1, 3, 3)
    s = np.asarray(scales)
    M = np.swapaxes(R, 1, 2) / s[None, :, None]
    k = np.sqrt(2 * np.log(density / 0.1))
    D = rng.normal(size=(n, 3))
    # half of the discs edge-on: the view direction within the plane of the longer axes, or nearly
    flat = R[:, :, int(np.argmin(s))]
    edge = rng.random(n) < 0.5
    D[edge] -= (flat * (D * flat).sum(1)[:, None])[edge] * (1 - 10.0 ** rng.uniform(-6, -1, n))[edge, None]
    D /= np.linalg.norm(D, axis=1)[:, None]
    C = np.einsum("nij,nj->ni", M, D)
    e = C / np.linalg.norm(C, axis=1)[:, None]
    t = rng.normal(size=(n, 3))
    t -= e * (t * e).sum(1)[:, None]
    t *= (k * rng.uniform(0.9, 1.02, n) / np.linalg.norm(t, axis=1))[:, None]
    rim = np.einsum("nij,nj->ni", R * s[None, None, :], t)
    mu = rng.uniform(-3, 3, (n, 3))
    eye = mu + rim - dist * D
    u = np.cross(rng.normal(size=(n, 3)), D)
    u /= np.linalg.norm(u, axis=1)[:, None]
    v = np.cross(D, u)
    ang = rng.uniform(-0.3, 0.3, n)
    fwd = D * np.cos(ang)[:, None] + u * np.sin(ang)[:, None]
    right = u * np.cos(ang)[:, None] - D * np.sin(ang)[:, None]
    h = 2 * np.tan(np.radians(22.5)) / px
    dx = (-np.tan(ang) + rng.uniform(-3, 3, n) * h)[:, None, None] + ((np.arange(8) - 3.5) * h)[None, None, :]
    dy = (rng.uniform(-2, 2, n) * h)[:, None, None] + ((np.arange(4) - 1.5) * h)[None, :, None]
    dx, dy = (a.reshape(n, -1).astype(F) for a in np.broadcast_arrays(dx, dy))
    return M.astype(F), F(1 / k), eye.astype(F), mu.astype(F), right.astype(F), v.astype(F), fwd.astype(F), dx, dy


def _off(rng, a):
    return (a * (F(1) + ULP * rng.integers(-3, 4, a.shape).astype(F))).astype(F)


def _may_hit(rng, sc):
    """False where the cone test drops the leaf (its `miss`), in the kernel's operations."""
    M, k, eye, mu, right, v, fwd, dx, dy = sc
    x0, x1, y0, y1 = dx.min(1), dx.max(1), dy.min(1), dy.max(1)
    half = F(0.5)
    dc = right * (half * (x0 + x1))[:, None] + (v * (half * (y0 + y1))[:, None] + fwd)
    du, dv = right * (half * (x1 - x0))[:, None], v * (half * (y1 - y0))[:, None]
    d = mu - eye
    O, C, U, V = (np.stack([_dot(M[:, i], a) for i in range(3)], 1) for a in (d, dc, du, dv))
    c2 = _dot(C, C)
    ic = _off(rng, 1 / np.sqrt(c2))
    c1, e = c2 * ic, C * ic[:, None]
    b = _dot(O, e)
    P = O - e * b[:, None]
    rho2 = _dot(P, P)
    ir = _off(rng, 1 / np.sqrt(rho2))
    rho = rho2 * ir
    eu, ev = _dot(e, U), _dot(e, V)
    spread = np.abs(eu) + np.abs(ev)
    width = (np.abs(_dot(P, U - e * eu[:, None])) + np.abs(_dot(P, V - e * ev[:, None]))) * ir + F(4e-7) * (
        _norm(U) + _norm(V))
    along = c1 * F(0.99999) - spread
    m2 = _dot(M[:, 0], M[:, 0]) + _dot(M[:, 1], M[:, 1]) + _dot(M[:, 2], M[:, 2])
    R = _off(rng, F(1) / k * np.ones_like(b)) * F(1.001) + F(1e-5) * (rho + np.abs(b)) + F(1e-6) * np.sqrt(m2 * _dot(d, d))
    return ~((along > 0) & (rho * along - b * width > R * np.sqrt(along * along + width * width)))


def _any_hit(sc):
    """Whether a ray of the tile hits the ellipsoid in front of the eye (roots_exact, roots_fast)."""
    M, k, eye, mu, right, v, fwd, dx, dy = sc
    d = right[:, None] * dx[:, :, None] + v[:, None] * dy[:, :, None] + fwd[:, None]
    d = (d / _norm(d)[..., None]).astype(F)
    o = (eye - mu)[:, None, :]
    rows = [(M[:, i] * k).astype(F)[:, None, :] for i in range(3)]
    Oe, De = (np.stack([_dot(r, a) for r in rows], -1) for a in (o, d))
    Dn = De * (F(1) / _norm(De))[..., None]
    b = -_dot(Oe, Dn)
    p = Oe + Dn * b[..., None]
    return ((F(1) - _dot(p, p) > F(1e-7)) & (b > 0)).any(1)


@pytest.mark.parametrize("px", [1000, 64])
@pytest.mark.parametrize("dist", [1.0, 8.0, 50.0])
def test_no_hit_leaf_is_dropped(dist, px):
    rng = np.random.default_rng(int(dist) + px)
    culled = hit = 0
    with np.errstate(all="ignore"):
        for ratio in (1, 10, 100, 1e3, 1e4, 1e5):
            for scales in ((0.3 / ratio, 0.3, 0.3), (0.3, 0.3, 0.3 * ratio), (0.1, 0.1 / ratio, 0.01)):
                sc = _scene(rng, 8000, np.minimum(scales, 3.0), dist, px, rng.choice([0.2, 1.0, 30.0]))
                may, h = _may_hit(rng, sc), _any_hit(sc)
                assert not (h & ~may).any(), (ratio, scales)
                culled, hit = culled + int((~may).sum()), hit + int(h.sum())
    assert hit > 10_000 and culled > 0
