"""Periodic native walks where the images matter: positions over several boxes,
groups wider than half a box, tight pairs beside the origin and across the
box's boundary. Against FP64 sums over the minimum images, within the error of
FP32 pair differences, row by row."""
import math

import numpy as np
import pytest

import sbh_b200 as B

pytestmark = pytest.mark.gpu


def _minimum_image_sums(p, m, w, box, eps, cut):
    """Force, query + source gradient and mass gradient in FP64, and a bound of
    each row's FP32 error: d = fl(q - p) is off by what that rounds away (0 for
    close neighbours), a moved image by another 2^-24 of the box; a pair's
    force changes by at most 4 m h^-3/2 per unit of d, its gradient terms by 20
    h^-2 |w|. The rest (reciprocal square roots, the attenuation's 1.5e-7, sums
    of at most 1,000 terms) stays below 4e-6 of the unattenuated magnitudes."""
    p32 = p.astype(np.float32)
    p, m, w = p.astype(np.float64), m.astype(np.float64), w.astype(np.float64)
    d = p[:, None] - p[None]
    k = np.floor(d / box + 0.5)
    off = np.abs((p32[:, None] - p32[None]).astype(np.float64) - d) + (k != 0) * box * 2.0 ** -24
    r = d - box * k
    off = np.linalg.norm(off, axis=-1) + 2.0 ** -24 * np.linalg.norm(r, axis=-1)
    r2 = (r * r).sum(-1)
    ir = (r2 + eps * eps + 1e-12) ** -0.5
    dist = np.sqrt(r2 + 1e-12)
    att, cc = np.ones_like(dist), np.zeros_like(dist)
    if cut:
        u = dist / (2.0 * cut)
        e = np.exp(-u * u)
        att = np.vectorize(math.erfc)(u) + 2.0 / math.sqrt(math.pi) * u * e
        cc = ir ** 3 * dist * e / (2.0 * math.sqrt(math.pi) * cut ** 3)
    for a in (att, cc, off):
        np.fill_diagonal(a, 0.0)
    lin, rw = att * ir ** 3, (r * w[:, None]).sum(-1)
    q = m[None, :, None] * (((3.0 * att * ir ** 5 + cc) * rw)[..., None] * r - lin[..., None] * w[:, None])
    f, gx, gm = -(lin * m[None])[..., None] * r, q.sum(1) - q.sum(0), -(lin * rw).sum(0)
    one = 1.0 - np.eye(len(p))
    wn = np.linalg.norm(w, axis=-1)[:, None]
    bf = m[None] * ir ** 3 * (4.0 * off + 4e-6 * dist * one)
    bq = m[None] * wn * (20.0 * ir ** 4 * off + 2e-5 * ir ** 3 * one)
    bm = wn * ir ** 3 * (4.0 * off + 4e-6 * dist * one)
    return (f.sum(1), gx, gm), (bf.sum(1)[:, None], (bq.sum(1) + bq.sum(0))[:, None], bm.sum(0))


def _points(kind, box, rng):
    if kind == "several boxes":
        return rng.uniform(0.0, 3.0 * box, (100, 3))
    if kind == "far from the origin":  # small groups, each some boxes away from the others
        return rng.uniform(0.0, 0.2 * box, (300, 3)) + 5.0 * box * rng.integers(-1, 2, (300, 1))
    if kind == "tight pair":
        p = rng.uniform(-0.5 * box, 0.5 * box, (100, 3))
        p[1] = p[0] = box * np.array([1e-4, -2e-4, 1.5e-4])
        p[1, 0] += 1e-5 * box
        return p
    if kind == "wide group by the boundary":  # groups in the last quarter, far sources in their batches
        p = rng.uniform(0.0, box, (300, 3))
        p[:150] = rng.uniform(0.77 * box, box, (150, 3))
        p[150:160] = p[:10] + rng.uniform(-1e-4, 1e-4, (10, 3)) * box
        return np.minimum(p, box * (1.0 - 1e-6))
    p = rng.uniform(0.0, box, (1000, 3))  # a tight cluster across the boundary
    p[:20] = np.mod(p[0] * [0, 1, 1] + rng.uniform(-2e-3, 2e-3, (20, 3)) * box, box)
    return p


@pytest.mark.parametrize("kind", ["several boxes", "far from the origin", "tight pair",
                                  "wide group by the boundary", "across"])
@pytest.mark.parametrize("box,cut", [(1.0, 0.0), (1.0, 0.1), (0.7, 0.07), (128.0, 6.4)])
@pytest.mark.parametrize("eps", [1e-2, 1e-3])
def test_periodic_walks_match_minimum_image_sums(cuda, kind, box, cut, eps):
    rng = np.random.default_rng(int(10 * box) + len(kind))
    p = _points(kind, box, rng).astype(np.float32)
    n = len(p)
    m, w = np.full(n, 1.0 / n, np.float32), rng.normal(size=(n, 3)).astype(np.float32)
    eps *= box
    t = B.NativeTree().build(p, m, leaf_size=8, group_size=64 if kind == "far from the origin" else 128)
    kw = dict(beta=1e4, softening=eps, cutoff=cut, quadrupole=False, periodic=True, box_length=box)  # every pair
    alone = t.force(**kw).cpu().numpy()
    got = [v.cpu().numpy() for v in t.force_vjp(w, **kw)]
    want, bound = _minimum_image_sums(p, m, w, box, eps, cut)
    for g, x, b in zip([alone] + got, (want[0],) + want, (bound[0],) + bound):
        assert (np.abs(g - x) <= b).all(), float((np.abs(g - x) / b).max())
