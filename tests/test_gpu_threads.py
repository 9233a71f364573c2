"""Engines of their own in threads of their own: films of different depths synthesized at the same time."""
import threading

import numpy as np
import pytest

import fgrain_gb300 as fg

pytestmark = pytest.mark.gpu


def test_films_of_different_depths_at_once(engine):
    depths, rounds = (3.0, 60.0), 1500  # 10 and 87 cells: 20 and 81 KB of shared memory a column
    want = [np.sort(synthesize(engine, d), axis=0) for d in depths]
    failed = []

    def work(k):
        try:
            e = fg.GpuEngine(0)
            for _ in range(rounds):
                np.testing.assert_array_equal(np.sort(synthesize(e, depths[k]), axis=0), want[k])
            e.close()
        except Exception as x:  # noqa: BLE001 - reported below
            failed.append((k, x))

    threads = [threading.Thread(target=work, args=(k,)) for k in (0, 1, 0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed


def synthesize(e, depth):
    em = fg.VirtualEmulsionLayer.synthesize(fg.EmulsionConfig((12.0, 10.0, depth), 1.2, 0.5, 0.3), 5, e)
    pos = em.crystals()["pos"]
    em.close()
    return pos
