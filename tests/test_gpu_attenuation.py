"""The erfc attenuation of the native walks against FP64, in the scalar and the
packed slots, and where u^2 = (r / 2 cutoff)^2 would leave FP32's range."""
import math

import numpy as np
import pytest

import sbh_b200 as B

pytestmark = pytest.mark.gpu

CUT, EPS = 0.5, 1e-2


# one slot (scalar), two (a packed pair), three (both), four (two pairs)
@pytest.mark.parametrize("n", [20, 60, 90, 120])
@pytest.mark.parametrize("periodic", [False, True])
def test_attenuation_over_u(cuda, n, periodic):
    """One source and n massless targets at u from 0 to 10: att to 1.5e-7 (the
    published bound of its approximation of erfc) and a few ulps of the pair, the
    gradient's att and cc terms, each at most 3 h^-3/2 |w|, to the same share."""
    u = np.linspace(0.0, 10.0, n)
    p = np.zeros((n + 1, 3), np.float32)
    p[1:, 0] = 2.0 * CUT * u
    p[1:, 1] = 1e-3
    m = np.zeros(n + 1, np.float32)
    m[0] = 1.0
    rng = np.random.default_rng(n)
    w = rng.normal(size=p.shape).astype(np.float32)
    w[0] = 0.0
    t = B.NativeTree().build(p, m, leaf_size=8)
    kw = dict(beta=1e4, softening=EPS, cutoff=CUT, quadrupole=False)
    if periodic:
        kw.update(periodic=True, box_length=64.0)
    alone = t.force(**kw).cpu().numpy()[1:]
    f, gx, _ = (v.cpu().numpy()[1:] for v in t.force_vjp(w, **kw))
    r = p[1:].astype(np.float64)
    W = w[1:].astype(np.float64)
    r2 = (r * r).sum(1)
    ir, d = (r2 + EPS * EPS + 1e-12) ** -0.5, np.sqrt(r2 + 1e-12)
    x = d / (2.0 * CUT)
    e = np.exp(-x * x)
    att = np.array([math.erfc(v) for v in x]) + 2.0 / math.sqrt(math.pi) * x * e
    cc = ir ** 3 * d * e / (2.0 * math.sqrt(math.pi) * CUT ** 3)
    want = -(att * ir ** 3)[:, None] * r
    bound = (ir ** 3 * d * (2e-7 + 1e-6 * att))[:, None]
    assert (np.abs(f - want) <= bound).all() and (np.abs(alone - want) <= bound).all()
    rw = (r * W).sum(1)
    want = ((3.0 * att * ir ** 5 + cc) * rw)[:, None] * r - (att * ir ** 3)[:, None] * W
    bound = (ir ** 3 * np.linalg.norm(W, axis=1) * (4 * 2e-7 + 2e-6 * (4.0 * att + cc / ir ** 3 * d * d)))[:, None]
    assert (np.abs(gx - want) <= bound).all(), float((np.abs(gx - want) / bound).max())


@pytest.mark.parametrize("cut", [1e-3, 1e-10, 1e-18, 1e-20, 1e-30])
def test_everything_beyond_a_tiny_cutoff_is_zero(cuda, cut):
    rng = np.random.default_rng(1)
    p = rng.random((300, 3)).astype(np.float32) * 10.0
    m, w = np.ones(300, np.float32), rng.normal(size=(300, 3)).astype(np.float32)
    t = B.NativeTree().build(p, m, leaf_size=8)
    for per in (dict(), dict(periodic=True, box_length=10.0)):
        kw = dict(softening=1e-2, cutoff=cut, quadrupole=False, **per)
        for v in (t.force(**kw), *t.force_vjp(w, **kw)):
            assert not v.cpu().numpy().any()
