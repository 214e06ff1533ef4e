"""Large pageable boxes of batches through the shared pinned bands.

Whatever way a box crosses (the driver's own staging for a batch's first bytes,
the shared bands after, the driver's again while another thread holds the
bands), it arrives bit for bit, with ghost cells and padding of the caller's box
left alone.  Batches alive share one set of host threads, and one that moves
little makes none."""
import ctypes as C
import os
import threading

import numpy as np
import pytest

from amrex_euler_allmach_explicit_imex_b200 import _lib, api, workloads

pytestmark = pytest.mark.gpu


def _states(grids, seed):
    cfgs, states = workloads.riemann_batch(len(grids), seed=seed, grids=grids)
    return cfgs, [u + 1.0e-3 * np.random.default_rng(k).standard_normal(u.shape) for k, u in enumerate(states)]


def _round_trips(batch, states, n):
    for _ in range(n):
        for k, u in enumerate(states):
            batch.upload(k, u)
        for k, u in enumerate(states):
            assert np.array_equal(batch.download(k), u)


def _threads():
    return len(os.listdir("/proc/self/task"))


# rows of a band: all of a plane, a part, one; a row that no band holds; one column
@pytest.mark.parametrize("grid", [(256, 128), (1023, 701), (32769, 3), (65536, 2), (65537, 2), (1, 40000)])
def test_boxes_cross_unchanged(gpu, grid):
    cfgs, states = _states([grid, (256, 256)], 3)
    with api.Batch(cfgs) as b:
        _round_trips(b, states, 1 + (72 << 20) // sum(2 * u.nbytes for u in states))
        _round_trips(b, states, 2)


def test_boxes_with_ghosts_and_padding(gpu):
    """The caller's box: two ghost cells below, three columns and a row more
    above, planes apart; only its own cells are read and written."""
    (nx, ny), lo = (601, 500), 2
    cfgs, (u,) = _states([(nx, ny)], 5)
    js, rows = nx + lo + 3, ny + lo + 1
    lib, box = _lib.load(), np.full((4, rows, js), 7.0)
    with api.Batch(cfgs) as b:
        for _ in range(6):  # 9.6 MB each way
            box[:] = 7.0
            box[:, lo:lo + ny, lo:lo + nx] = u
            _lib.check(lib.ecg_batch_upload(b._h, 0, C.c_void_p(box.ctypes.data), -lo, -lo, js, js * rows), "upload")
            box[:] = -5.0
            _lib.check(lib.ecg_batch_download(b._h, 0, C.c_void_p(box.ctypes.data), -lo, -lo, js, js * rows), "download")
            assert np.array_equal(box[:, lo:lo + ny, lo:lo + nx], u)
            box[:, lo:lo + ny, lo:lo + nx] = -5.0
            assert (box == -5.0).all()


def test_two_threads_share_the_bands(gpu):
    """Two batches transferring at once: one has the bands, the other goes
    without; both arrive."""
    fails = []

    def work(seed):
        try:
            cfgs, states = _states([(700, 701)] * 2, seed)
            with api.Batch(cfgs) as b:
                _round_trips(b, states, 6)
        except BaseException as e:  # noqa: BLE001 - reported below
            fails.append(e)

    ts = [threading.Thread(target=work, args=(s,)) for s in (1, 2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not fails


def test_batches_share_the_threads_and_give_them_back(gpu):
    cfgs, states = _states([(512, 512)] * 3, 9)
    with api.Batch(cfgs) as b:  # the CUDA runtime's own threads
        b.upload(0, states[0])
        b.run(1)
    base = _threads()
    one = api.Batch(cfgs)
    one.upload(0, states[0])  # 8 MB
    one.download(0)
    assert _threads() == base
    _round_trips(one, states, 2)  # 100 MB
    shared = _threads()
    more = [api.Batch(cfgs) for _ in range(4)]
    for b in more:
        _round_trips(b, states, 2)
    assert _threads() == shared
    for b in [one] + more:
        b.close()
    assert _threads() == base
