"""States and grids outside the range of the branch-free division (lare_div.cuh)
fall back to IEEE division point by point: still the checker's bits (every NaN
taken as one value: its sign and payload are the machine's)."""
import numpy as np
import pytest

from sams_b200 import lare
from tests.golden.make_golden import STATE

pytestmark = pytest.mark.gpu


def _tiny_velocity(F, rng):
    for f in (3, 4, 5):  # vanishing, denormal and ordinary velocities side by side
        F[f] *= 10.0 ** rng.choice([0, 0, -150, -280, -310], size=F[f].shape)
        F[f][rng.random(F[f].shape) < 0.2] = -0.0


def _thin_density(F, rng):
    F[0][...] *= 1e-36  # mass per cell below 2^-120
    for f in (9, 10, 11):
        F[f] *= 1e-20


def _no_field(F, rng):
    for f in (9, 10, 11):
        F[f][...] = -0.0


@pytest.mark.parametrize("case,n,scale,change", [
    ("rf", (9, 8, 26), 1e-12, None),   # cell volumes below 2^-120
    ("rf", (9, 8, 26), 1e14, None),    # ... above 2^119
    ("rf", (16, 8, 8), 1.0, _tiny_velocity),   # a power-of-two grid
    ("rf", (9, 10, 11), 1.0, _tiny_velocity),
    ("rf", (9, 10, 11), 1.0, _thin_density),
    ("harris", (9, 10, 6), 1.0, _tiny_velocity),
    ("ot", (12, 10, 4), 1.0, _no_field),
])
@pytest.mark.parametrize("batched", [False, True])
def test_fallback_matches_checker(case, n, scale, change, batched, oracle_lib):
    lo = oracle_lib

    def setup(mod):
        p, b = mod.case_setup(case, *n)
        for d in "xyz":
            for e in ("min", "max"):
                setattr(p, f"{d}_{e}", getattr(p, f"{d}_{e}") * scale)
        return p, b

    p, b = setup(lare)
    q, _ = lare.case_setup(case, *n)
    F = [np.array(a) for a in lare.case_fields(case, q, seed=5)]
    if change:
        change(F, np.random.default_rng(3))
    po, bo = setup(lo)
    o = lo.Oracle(po, bo, [a.copy() for a in F])
    o.step(2)
    if batched:
        bt = lare.Batch()
        i = bt.add(p, b, F)
        bt.step(2)
        bt.synchronize()
        got = {f: bt.download(i, f) for f in STATE}
        if all(np.isfinite(o.field(f)).all() for f in STATE):
            dt = bt.state(i)[0]
        else:  # (a batch reports such a solve instead of its dt)
            with pytest.raises(lare.LareError):
                bt.state(i)
            dt = o.dt
    else:
        s = lare.LARE3D(p, b)
        s.upload_all(F)
        s.step(2)
        dt, got = s.dt, {f: s.download(f) for f in STATE}
    assert dt == o.dt and np.isfinite(dt)
    for f in STATE:
        sl = lare.field_slices(f, *n)
        a, b = (np.where(np.isnan(x), np.nan, x).view(np.int64) for x in (got[f][sl], o.field(f)[sl]))
        assert np.array_equal(a, b), f
