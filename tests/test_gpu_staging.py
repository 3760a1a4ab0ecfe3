"""Copies of large pageable buffers through a context's staging threads (staging.hpp): the
samples a scene holds and the matched filter's output are the caller's, bit for bit, at
sizes around a slot and the staging threshold, from pinned memory (no staging), and with
several threads on one context and on contexts of their own."""
import threading

import numpy as np
import pytest

import bsar

pytestmark = pytest.mark.gpu

N = 4096      # 65536 bytes a row


def _roundtrip(ctx, rows, seed, pinned=False):
    import torch

    rng = np.random.default_rng(seed)
    x = rng.normal(size=(rows, N)) + 1j * rng.normal(size=(rows, N))
    if pinned:
        t = torch.empty((rows, N), dtype=torch.complex128, pin_memory=True)
        t.numpy()[:] = x
        x = t.numpy()
    dem = bsar.DemArrays(np.arange(4.0), np.arange(4.0), np.zeros((4, 4)))
    tx = np.zeros((rows, 3)) + [0.0, 0.0, 30.0]
    sid = ctx.scene_upload(dem, tx, tx, x, kind="compressed")
    try:
        back = ctx.scene_read_samples(sid, rows, N)
    finally:
        ctx.scene_release(sid)
    assert np.array_equal(back, x)


@pytest.mark.parametrize("rows", [1, 31, 32, 33, 40, 71, 257, 511, 513, 700])
def test_round_trip(ctx, rows):
    _roundtrip(ctx, rows, rows)
    _roundtrip(ctx, rows, rows + 1, pinned=True)


@pytest.mark.parametrize("own", [False, True])
def test_threads(ctx, own):
    errors = []

    def run(k):
        try:
            c = bsar.Context(0) if own else ctx
            for i in range(4):
                _roundtrip(c, 50 + 13 * k + i, 100 * k + i)
            if own:
                c.close()
        except Exception as e:      # noqa: BLE001
            errors.append(e)

    ts = [threading.Thread(target=run, args=(k,)) for k in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors
