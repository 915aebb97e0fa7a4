"""Batched solves whose rows are padded: host boxes pass through a scratch
array of the solve, whose contents no step may read."""
import numpy as np
import pytest

from sams_b200 import lare

pytestmark = pytest.mark.gpu

STATE = ["rho", "energy_electron", "energy_ion", "vx", "vy", "vz", "bx", "by", "bz"]


@pytest.mark.parametrize("case,n", [("ot", (9, 8, 64)), ("rf", (8, 11, 63)), ("harris", (12, 10, 70)),
                                    ("rf", (2, 9, 66)), ("ot", (5, 4, 284)), ("rf", (4, 3, 300))])
def test_transfers_leave_nothing_for_a_step(case, n):
    p, b = lare.case_setup(case, *n)
    fields = lare.case_fields(case, p, seed=7)
    solo, bt = lare.LARE3D(p, b), lare.Batch()
    solo.upload_all(fields)
    sid = bt.add(p, b, fields)
    # a field that every step overwrites comes last: the scratch array holds its NaN when the step begins
    junk = np.full(tuple(q + 5 for q in n), np.nan)
    solo.upload("dm", junk)
    bt.upload(sid, "dm", junk)
    for _ in range(3):
        solo.step(1)
        bt.step(1)
        bt.synchronize()
        for f in STATE:
            sl = lare.field_slices(f, *n)
            want = solo.download(f)[sl]
            assert np.isfinite(want).all()
            assert np.array_equal(bt.download(sid, f)[sl], want), f
        solo.upload("dm", junk)
        bt.upload(sid, "dm", junk)
    solo.close()
    bt.close()
