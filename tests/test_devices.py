"""What the host side asks of the devices (no GPU: fake_device): on several
devices of one process every kernel is launched with the shared memory it was
allowed on its own; the traceback arena stays within its bound."""
import ctypes

import numpy as np
import pytest

import fake_device
import test_launch_errors

u64, i64 = ctypes.c_uint64, ctypes.c_int64


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return fake_device.load(tmp_path_factory.mktemp("fake"))


def _p(a):
    return ctypes.c_void_p(a.ctypes.data)


def _pairwise(lib, h, weight):
    seq = np.frombuffer(b"ACGTTGCA", np.uint8).repeat(500)
    out, n = np.zeros(3000, np.int64), u64(0)
    return lib.mvg_pairwise_matches(h, _p(seq), u64(len(seq)), _p(seq), u64(len(seq)),
                                    u64(lib.mvg_get_seed(weight, 3)), _p(out), u64(1000), ctypes.byref(n))


def _gap_search(lib, h, _):
    seq = np.frombuffer(b"ACGTTGCA", np.uint8).repeat(500)
    gaps, out = np.array([[0, 3000, 0, 3000]], np.int64), np.zeros(3000, np.int64)
    off, n = np.zeros(2, np.uint64), u64(0)
    return lib.mvg_gap_anchor_search(h, _p(seq), u64(len(seq)), _p(seq), u64(len(seq)), _p(gaps), u64(1), _p(out),
                                     u64(1000), _p(off), ctypes.byref(n))


def _banded(lib, h, ring):
    # one band in the strip kernel (ring off) or the ring's; both are rejected
    # by a device that does nothing and run whole
    lib.mvg_set_band_ring(h, ring)
    seq, off = np.zeros(9000, np.uint8), np.array([0, 9000], np.uint64)
    delta, half = np.zeros(1, np.int32), np.full(1, 100, np.int32)
    score, path, plen = np.zeros(1, np.int32), np.zeros(18000, np.uint8), np.zeros(1, np.int64)
    used, poff = np.zeros(1, np.uint8), np.array([0, 18000], np.uint64)
    return lib.mvg_gapdp_banded(h, _p(seq), _p(off), _p(seq), _p(off), i64(1), _p(delta), _p(half), _p(score),
                                _p(path), _p(poff), _p(plen), _p(used), None)


@pytest.mark.parametrize("call,arg", [(_pairwise, 11), (_pairwise, 15), (_pairwise, 17), (_gap_search, None),
                                      (_banded, 0), (_banded, 1)])
def test_second_device(lib, call, arg):
    for device in (0, 1, 0, 2):
        h = ctypes.c_void_p()
        assert lib.mvg_create(ctypes.byref(h), device) == 0
        lib.fake_reset(1 << 40)
        assert call(lib, h, arg) == 0, lib.mvg_last_error()
        assert lib.fake_refused() == 0
        lib.mvg_destroy(h)


@pytest.mark.parametrize("call", test_launch_errors.CALLS)
def test_every_call_on_a_second_device(lib, call):
    for device in (0, 1):
        h = ctypes.c_void_p()
        assert lib.mvg_create(ctypes.byref(h), device) == 0
        lib.fake_reset(1 << 40)
        assert call(lib, h) == 0, lib.mvg_last_error()
        assert lib.fake_refused() == 0
        lib.mvg_destroy(h)


def _least(la, lb, checkpoints=True):
    """The least arena bound at which the gap DP takes a problem."""
    strips = -(-la // 256)
    if not checkpoints:
        return strips * (lb + 31) * 128
    return ((strips - 1) * lb + strips * (-(-lb // 128) - 1) * 256) * 16


# Slots that the shape chosen for speed would make larger than the bound:
# stored bits, half-height strips, one strip of many states, many strips of few
# columns, bits by request.
@pytest.mark.parametrize("la,lb,checkpoints", [(5900, 700, True), (5000, 1500, True), (200, 40000, True),
                                               (200000, 120, True), (5900, 690, False)])
def test_arena_bound(lib, la, lb, checkpoints):
    h = ctypes.c_void_p()
    assert lib.mvg_create(ctypes.byref(h), 0) == 0
    least = _least(la, lb, checkpoints)
    bound = max(least // 256 * 256 + 256, 1 << 20)
    lib.mvg_set_dp_checkpoint(h, int(checkpoints))
    a, b = np.zeros(la, np.uint8), np.zeros(lb, np.uint8)
    oa, ob, po = (np.array([0, n], np.uint64) for n in (la, lb, la + lb))
    score, path, plen = np.zeros(1, np.int32), np.zeros(la + lb, np.uint8), np.zeros(1, np.int64)

    def call():
        return lib.mvg_gapdp_batch(h, _p(a), _p(oa), _p(b), _p(ob), i64(1), _p(score), _p(path), _p(po), _p(plen))

    for by_free_memory in (False, True):  # the bound asked for, then 60% of free memory
        assert lib.mvg_set_tb_arena(h, u64(2**64 - 1 if by_free_memory else bound)) == 0
        lib.fake_reset(int(bound / 0.6) + 2 if by_free_memory else 1 << 40)
        assert call() == 0, lib.mvg_last_error()
        assert lib.fake_largest() <= bound + bound // 8 + 512  # a buffer is made an eighth larger than asked for
        lib.mvg_destroy(h)
        assert lib.mvg_create(ctypes.byref(h), 0) == 0
        lib.mvg_set_dp_checkpoint(h, int(checkpoints))
    lib.fake_reset(1 << 40)
    if lib.mvg_set_tb_arena(h, u64(least - 1)) == 0:
        assert call() == 5  # MVG_ERR_CAPACITY
    lib.mvg_destroy(h)
