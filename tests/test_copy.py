"""Staged host transfers (gale_b200/csrc/gg_copy.cu; needs a B200): points written and read
back unchanged around the sizes where the split changes, and from two threads at once."""
import threading

import numpy as np
import pytest

from gale_b200.stokes import Mesh, StokesProblem

pytestmark = pytest.mark.gpu


def round_trip(n, seed, repeat=1):
    rng = np.random.default_rng(seed)
    G = StokesProblem(Mesh(2, (4, 4)))
    for _ in range(repeat):
        x, m, ps = rng.random((n, 2)), rng.integers(0, 5, n, dtype=np.int32), rng.random(n)
        G.set_points(x, m, ps)
        gx, gm, gps = G.points()
        assert np.array_equal(gx, x) and np.array_equal(gm, m) and np.array_equal(gps, ps)


# coordinates of 16 bytes: 1 MB, one more and one less, a ragged last chunk, full slots
@pytest.mark.parametrize("n", [1, 65535, 65536, 65537, 262143, 1_000_003, 2_097_153])
def test_round_trip(n):
    round_trip(n, n)


def test_two_threads():
    fails = []

    def work(seed):
        try:
            round_trip(700_001, seed, repeat=6)
        except BaseException as e:  # noqa: BLE001
            fails.append(e)
    ts = [threading.Thread(target=work, args=(s,)) for s in (1, 2, 3)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not fails


# coordinates of 16 bytes: 12 MB up, one more and one less, and full large slots; four round trips
# each, so that the slots are there
@pytest.mark.parametrize("n", [786_431, 786_432, 786_433, 3_000_001])
def test_round_trip_staged_both_ways(n):
    round_trip(n, n, repeat=4)


def test_threads_with_staged_uploads():
    fails = []

    def work(seed):
        try:
            round_trip(1_000_001 + seed, seed, repeat=6)
        except BaseException as e:  # noqa: BLE001
            fails.append(e)
    ts = [threading.Thread(target=work, args=(s,)) for s in (1, 2, 3, 4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not fails
