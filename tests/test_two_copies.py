"""Two copies of the library in one process, as two installed versions or a
plugin's own make: neither relies on what the other has set up (no GPU:
fake_device)."""
import ctypes

import numpy as np

import fake_device


def _p(a):
    return ctypes.c_void_p(a.ctypes.data)


def test_small_sorts(tmp_path_factory):
    libs = [fake_device.load(tmp_path_factory.mktemp("copy")) for _ in range(2)]
    seq = np.frombuffer(b"ACGTTGCA", np.uint8).repeat(2000)
    out, n = np.zeros(3000, np.int64), ctypes.c_uint64(0)
    # segment ends, pairs, buckets left over: the ends of 3,500 segments are
    # sorted in one CTA, with more than 48 KB of shared memory
    counts = np.array([7000, 9000, 0], np.uint32)
    for lib in libs:
        for device in (0, 1):
            h = ctypes.c_void_p()
            assert lib.mvg_create(ctypes.byref(h), device) == 0
            lib.fake_reset(1 << 40)
            lib.fake_reply(_p(counts), counts.nbytes)
            rc = lib.mvg_pairwise_matches(h, _p(seq), ctypes.c_uint64(len(seq)), _p(seq), ctypes.c_uint64(len(seq)),
                                          ctypes.c_uint64(lib.mvg_get_seed(15, 3)), _p(out), ctypes.c_uint64(1000),
                                          ctypes.byref(n))
            assert rc == 0, lib.mvg_last_error()
            stats = np.zeros(4, np.uint64)
            assert lib.mvg_pairwise_stats(h, _p(stats)) == 0 and stats[0] == 9000  # the counts were read
            assert lib.fake_refused() == 0
            lib.mvg_destroy(h)
