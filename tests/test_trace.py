"""The timeline reader on records made by hand: a launch with all stamps, and one whose vector is staged in one pass (no points 6 to 8: their places hold zero or
what an earlier launch left)."""
import numpy as np
import pytest

from slai_b200 import trace


def record(kid, stamps):
    return [kid] + list(stamps) + [0] * (trace.SLOTS - 1 - len(stamps))


@pytest.mark.parametrize("left", [(0, 0, 0), (400, 450, 500), (400, 9_000, 9_500)])
def test_launches_without_the_points_of_staging(left):
    full = [1000 * i for i in range(1, 15)]
    plain = [20_000 + s for s in full]
    plain[6:9] = left
    rows = {r[0]: r[2:] for r in trace.summarise(np.array([record(16 * 1000 + 100 + 20, full), record(16 * 1000 + 100 + 1, plain)], dtype=np.int64))}
    names = [c for c, _, _ in trace.COLS]
    whole = dict(zip(names, rows["gemv K=4096 ln+store"]))
    one_pass = dict(zip(names, rows["gemv K=4096 resid"]))
    assert all(abs(whole[n] - 1.0) < 1e-9 for n in names)
    assert one_pass["load"] == one_pass["stats"] == one_pass["bar"] == 0 and abs(one_pass["digits"] - 4.0) < 1e-9
    assert all(one_pass[n] >= 0 for n in names) and abs(sum(one_pass[n] for n in names) - 13.0) < 1e-9
