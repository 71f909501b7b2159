"""A launch that CUDA refuses, or an allocation, makes the call it belongs to
fail, whichever of the call's it is, and leaves nothing for the next call (no
GPU: fake_device)."""
import ctypes

import numpy as np
import pytest

import fake_device

u64, i64 = ctypes.c_uint64, ctypes.c_int64


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return fake_device.load(tmp_path_factory.mktemp("fake"))


def _p(a):
    p = ctypes.c_void_p(a.ctypes.data)
    p.array = a  # alive as long as the pointer
    return p


SEQ = np.frombuffer(b"ACGTTGCA", np.uint8).repeat(1000)
N = len(SEQ)
CODES = np.arange(600, dtype=np.uint8) % 4
OFF = np.array([0, 250, 600], np.uint64)


def _pairwise(lib, h, weight=15):
    out, n = np.zeros(3000, np.int64), u64(0)
    counts, comps = np.array([300, 9000, 0], np.uint32), np.array([20, 0], np.uint32)
    lib.fake_reply(_p(counts), 12)  # segment ends, pairs, buckets left over
    lib.fake_reply(_p(comps), 8)  # components, flagged buckets
    return lib.mvg_pairwise_matches(h, _p(SEQ), u64(N), _p(SEQ), u64(N), u64(lib.mvg_get_seed(weight, 3)), _p(out),
                                    u64(1000), ctypes.byref(n))


def _pairwise_sorted(lib, h):
    return _pairwise(lib, h, 23)


def _gap_search(lib, h):
    gaps, out = np.array([[0, 7000, 0, 7000]], np.int64), np.zeros(3000, np.int64)
    off, n = np.zeros(2, np.uint64), u64(0)
    counts, comps = np.array([300, 9000, 0], np.uint32), np.array([20, 0], np.uint32)
    lib.fake_reply(_p(counts), 12)
    lib.fake_reply(_p(comps), 8)
    return lib.mvg_gap_anchor_search(h, _p(SEQ), u64(N), _p(SEQ), u64(N), _p(gaps), u64(1), _p(out), u64(1000),
                                     _p(off), ctypes.byref(n))


def _dp_out():
    return np.zeros(2, np.int32), np.zeros(1200, np.uint8), 2 * OFF, np.zeros(2, np.int64)


def _batch(lib, h):
    return lib.mvg_gapdp_batch(h, _p(CODES), _p(OFF), _p(CODES), _p(OFF), i64(2), *map(_p, _dp_out()))


def _banded(lib, h):
    delta, half, used = np.zeros(2, np.int32), np.full(2, 9, np.int32), np.zeros(2, np.uint8)
    return lib.mvg_gapdp_banded(h, _p(CODES), _p(OFF), _p(CODES), _p(OFF), i64(2), _p(delta), _p(half),
                                *map(_p, _dp_out()), _p(used), None)


def _banded_strips(lib, h):
    lib.mvg_set_band_ring(h, 0)
    return _banded(lib, h)


def _sml(lib, h):
    pos, mer, n = np.zeros(N, np.uint32), np.zeros(N, np.uint64), u64(0)
    return lib.mvg_sml_build(h, _p(SEQ), u64(N), u64(lib.mvg_get_seed(15, 3)), _p(pos), _p(mer), u64(N),
                             ctypes.byref(n))


def _lut(lib, h):
    one, off, lut = np.array([1], np.int64), np.array([0, N], np.uint64), np.zeros(N, np.int32)
    return lib.mvg_build_index_lut(h, _p(one), _p(one), _p(off), _p(SEQ), _p(SEQ), u64(1), _p(SEQ), u64(N), _p(SEQ),
                                   u64(N), 1, 300, 1, 20, _p(lut), u64(N))


def _xmfa(lib, h):
    starts, lens, off = np.array([1, 1], np.int64), np.array([N, N], np.int64), np.array([0, N], np.uint64)
    out, n = np.zeros(4 * N, np.uint8), u64(0)
    return lib.mvg_xmfa_write(h, b"a", b"b", b"", i64(1), _p(starts), _p(lens), _p(SEQ), _p(SEQ), _p(off), _p(out),
                              u64(len(out)), ctypes.byref(n))


def _rows(lib, h):
    path, off, plen = np.full(600, ord("M"), np.uint8), OFF, np.array([250, 350], np.int64)
    ra, rb = np.zeros(600, np.uint8), np.zeros(600, np.uint8)
    return lib.mvg_path_rows(h, _p(CODES), _p(off), _p(CODES), _p(off), i64(2), _p(path), _p(off), _p(plen), _p(ra),
                             _p(rb))


def _gradient(lib, h):
    lib.mvg_mlp_num_params.restype = ctypes.c_int64
    w = np.zeros(lib.mvg_mlp_num_params(), np.float32)
    if rc := lib.mvg_mlp_set_params(h, _p(w)):
        return rc
    x, t, g, loss = np.zeros(100 * 528, np.uint16), np.zeros(200, np.float32), np.zeros_like(w), ctypes.c_float(0)
    return lib.mvg_mlp_grad_dev(h, _p(x), _p(t), i64(100), _p(g), ctypes.byref(loss))


def _train(lib, h):
    lib.mvg_mlp_num_params.restype = ctypes.c_int64
    if rc := lib.mvg_mlp_set_params(h, _p(np.zeros(lib.mvg_mlp_num_params(), np.float32))):
        return rc
    x, t, loss = np.zeros(100 * 528, np.uint16), np.zeros(200, np.float32), ctypes.c_float(0)
    return lib.mvg_mlp_train_step_dev(h, _p(x), _p(t), i64(100), ctypes.c_float(0.1), 1, ctypes.byref(loss))


def _propose(lib, h):
    lib.mvg_mlp_num_params.restype = ctypes.c_int64
    lib.mvg_set_band_gate(h, 20)
    if rc := lib.mvg_mlp_set_params(h, _p(np.zeros(lib.mvg_mlp_num_params(), np.float32))):
        return rc
    delta, half = np.zeros(2, np.int32), np.zeros(2, np.int32)
    return lib.mvg_band_propose_dev(h, _p(CODES), _p(OFF), _p(CODES), _p(OFF), i64(2), ctypes.c_float(1),
                                    ctypes.c_float(8), _p(delta), _p(half))


def _gapped(lib, h):
    off, out_off = np.array([0, 3000, N], np.uint64), np.zeros(3, np.uint64)
    out = [np.zeros(2 * N, np.uint8) for _ in range(2)]
    return lib.mvg_gapped_alignment(h, _p(SEQ), _p(SEQ), _p(off), i64(2), ctypes.c_double(20000), 3, _p(out[0]),
                                    _p(out[1]), _p(out_off), u64(2 * N))


def _outside_lcbs(lib, h):
    regions, out, n, w = np.array([1, 4000], np.int64), np.zeros(3000, np.int64), u64(0), ctypes.c_uint32(0)
    return lib.mvg_search_lcb_gaps(h, _p(SEQ), u64(N), _p(SEQ), u64(N), _p(regions), u64(2), _p(regions), u64(2),
                                   _p(out), u64(1000), ctypes.byref(n), ctypes.byref(w))


CALLS = [_pairwise, _pairwise_sorted, _gap_search, _batch, _banded, _banded_strips, _sml, _lut, _xmfa, _rows, _gradient,
         _train, _propose, _gapped, _outside_lcbs]


@pytest.mark.parametrize("call", CALLS)
def test_every_launch(lib, call):
    h = ctypes.c_void_p()
    assert lib.mvg_create(ctypes.byref(h), 0) == 0
    lib.fake_reset(1 << 40)
    assert call(lib, h) == 0, lib.mvg_last_error()
    count = lib.fake_launches()
    assert count >= 1
    silent = []
    for k in range(count):
        lib.fake_reset(1 << 40)
        lib.fake_fail_at(k)
        if call(lib, h) == 0:
            silent.append(k)
        lib.fake_reset(1 << 40)
        rc = call(lib, h)
        assert rc == 0 or k in silent, (k, lib.mvg_last_error())
    lib.mvg_destroy(h)
    assert not silent, (silent, count)


@pytest.mark.parametrize("call", CALLS)
def test_every_allocation(lib, call):
    def fresh():
        h = ctypes.c_void_p()
        lib.fake_reset(1 << 40)
        assert lib.mvg_create(ctypes.byref(h), 0) == 0
        lib.fake_reset(1 << 40)
        return h

    h = fresh()
    assert call(lib, h) == 0
    count = lib.fake_allocations()
    lib.mvg_destroy(h)
    assert count >= 1
    for k in range(count):
        h = fresh()
        lib.fake_no_memory_at(k)
        # the staging and read-back buffers have a way round
        assert call(lib, h) in ((0, 6) if call in (_batch, _banded, _banded_strips, _xmfa, _gapped) else (6,)), k
        for _ in range(2):
            lib.fake_reset(1 << 40)
            assert call(lib, h) == 0, (k, lib.mvg_last_error())
        lib.mvg_destroy(h)
