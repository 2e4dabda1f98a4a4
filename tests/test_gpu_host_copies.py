"""Host arrays of sizes around the ones where their copies change: the least
shared size of each direction, whole and broken chunks (512 KB), one half and
the whole of the staging buffer.  An identity map with nearest-neighbour
sampling returns the input, so every byte has to come back as it went in."""
import threading

import numpy as np
import pytest

import mirorr_b200 as mb

pytestmark = pytest.mark.gpu

MB = 1 << 20


def round_trip(ctx, nbytes, seed):
    n = nbytes // 4
    img = np.random.default_rng(seed).random(n, dtype=np.float32).reshape(1, 1, n)
    out, _ = mb.resample(ctx, img, None, (n, 1, 1), np.eye(3), np.zeros(3), nearest=True)
    np.testing.assert_array_equal(out.reshape(-1), img.reshape(-1))


@pytest.mark.parametrize("nbytes", [
    4096, 5 * MB - 4, 5 * MB, 5 * MB + 4, 8 * MB, 8 * MB + 4, 16 * MB - 4, 16 * MB + 4,
    24 * MB - 4, 24 * MB, 24 * MB + 4, 56 * MB + 512 * 1024 + 12, 64 * MB])
def test_round_trip(nbytes):
    ctx = mb.Context()
    for k in range(2):  # the second pass reuses staging that the first has filled
        round_trip(ctx, nbytes, nbytes + k)
    ctx.close()


def test_two_threads_one_context():
    errors = []

    def run(ctx, seed):
        try:
            for k in range(3):
                round_trip(ctx, 50 * MB, seed + k)
        except Exception as e:  # noqa: BLE001 - reported by the main thread
            errors.append(e)

    ctx = mb.Context()
    ts = [threading.Thread(target=run, args=(ctx, 10 * i)) for i in range(2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    ctx.close()
    assert not errors, errors
