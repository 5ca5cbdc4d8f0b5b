"""The C-ABI library loads and exports every function include/gsq.h and include/gsq_debug.h declare (no compute calls)."""

import ctypes
import os
import re

from gsq_b200 import _cabi

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _declared():
    src = open(os.path.join(ROOT, "include", "gsq.h")).read() + open(os.path.join(ROOT, "include", "gsq_debug.h")).read()
    src = re.sub(r"/\*.*?\*/", "", src, flags=re.S)
    return sorted(set(re.findall(r"\b(gsq_[a-z0-9_]+)\s*\(", src)))


def test_header_functions_are_exported():
    names = _declared()
    assert len(names) >= 14
    lib = ctypes.CDLL(_cabi.LIB_PATH)
    missing = [n for n in names if not hasattr(lib, n)]
    assert not missing, missing
    assert set(_cabi.EXPORTS) <= set(names)


def test_host_only_entry_points():
    lib = _cabi.lib
    assert lib.gsq_abi_version() >= 1
    assert [lib.gsq_type_block_bytes(t) for t in (12, 14, 21, 23, 2)] == [144, 210, 110, 136, 0]
    assert lib.gsq_strerror(0) == b"ok" and b"guard" in lib.gsq_strerror(-1)
    assert lib.gsq_q8_layout_for_type(12) == _cabi.LAYOUT_DS4 and lib.gsq_q8_layout_for_type(21) == _cabi.LAYOUT_D4
    # zero-size work returns before any CUDA call
    assert lib.gsq_mul_mat_vec_q8(None, 0, 0, 21, 1, None, 0, 5120, None, 0, 0, None) == 0
    assert lib.gsq_quantize_q8_1(None, 1, 0, 512, 512, None, None) == 0
    assert lib.gsq_iq3s_repack(None, 0, 220, 0, None) == 0


def test_pairs_that_one_launch_serves():
    """Two weights of a fused layer: the listed pairs of types, at the rows of the small-batch kernel, repacked where that reads
    repacked weights; everything else is refused before the GPU is touched."""
    lib, first = _cabi.lib, {12: 2, 21: 1, 23: 4}      # fewest rows of Q4_K, IQ3_S, IQ4_XS

    def weight(t, rows=64, k=512):
        return _cabi.Weight(1, k // 256 * lib.gsq_type_block_bytes(t), rows, t, int(t in (14, 21)), 1)

    for ta in (10, 12, 14, 21, 23):
        for tb in (10, 12, 14, 21, 23):
            for m in range(0, 10):
                want = (tb == 14 and ta in first or (ta, tb) == (21, 23)) and max(first[ta], first.get(tb, 1)) <= m <= 8
                a, b = weight(ta), weight(tb)
                assert lib.gsq_linear_vec_pair_serves(a, b, m) == int(want), (ta, tb, m)
                if not want:
                    assert lib.gsq_linear_vec_pair(a, b, 1, -1, m, 512, 0, 0, 128, None) == _cabi.ERR_UNSUPPORTED
    for bad in (weight(14, rows=40), weight(14, k=768)):
        assert lib.gsq_linear_vec_pair(weight(21), bad, 1, -1, 4, 512, 0, 0, 128, None) == _cabi.ERR_UNSUPPORTED
    unpacked = weight(21)
    unpacked.packed = 0
    assert lib.gsq_linear_vec_pair_serves(unpacked, weight(14), 4) == 0


def test_repacked_weights_of_ragged_rows_are_refused():
    """Repacked IQ3_S / Q6_K are records of 16 rows. gsq_linear and gsq_linear_vec refuse any other row count before they
    touch the device, at every number of activation rows (from 25 on the weights used to be expanded record by record,
    past the last row)."""
    lib = _cabi.lib
    buf = ctypes.create_string_buffer(1 << 20)
    at = (ctypes.addressof(buf) + 255) // 256 * 256
    for t, bs in ((21, 110), (14, 210)):
        for rows in (1, 15, 24, 40, 17400):
            for m in (1, 8, 9, 24, 25, 32, 48, 97, 128, 300):
                k = 1024
                args = (at, k // 256 * bs, rows, t, 1, at, 2, m, k, k, at, 2, rows)
                assert lib.gsq_linear_workspace_bytes(rows, m, k, t, 1) == 0 and lib.gsq_linear_scratch_bytes(rows, m, k, t, 1) == 0
                assert lib.gsq_linear(*args, at, 1 << 30, None) == _cabi.ERR_UNSUPPORTED, (t, rows, m)
                assert lib.gsq_linear_vec(*args, None) == _cabi.ERR_UNSUPPORTED, (t, rows, m)
                assert lib.gsq_linear_allreduce(*args, at, 1 << 30, ctypes.byref(_cabi.PeerReduce()), None) != 0
        assert lib.gsq_linear_workspace_bytes(32, 128, 1024, t, 1) > 0


def test_packed_flag_means_nothing_for_types_of_one_layout():
    lib = _cabi.lib
    for t in (12, 23):
        for rows in (16, 24, 5120, 17408):
            for m in (1, 8, 9, 40, 100, 200, 256, 777):
                assert lib.gsq_linear_workspace_bytes(rows, m, 2048, t, 1) == lib.gsq_linear_workspace_bytes(rows, m, 2048, t, 0), (t, rows, m)


def test_which_pairs_one_launch_serves():
    """The size of the smaller product decides, whichever of the two it is."""
    def weight(t, rows, k):
        bs = {12: 144, 14: 210, 21: 110, 23: 136}[t]
        return _cabi.Weight(4096, k // 256 * bs, rows, t, int(t in (14, 21)), 4096)

    for a, b in ((12, 14), (21, 14), (23, 14), (21, 23)):
        for ra, rb, k, served in ((5120, 1024, 5120, 1), (34816, 1024, 17408, 1), (1024, 34816, 17408, 1), (12288, 60000, 8192, 1),
                                  (60000, 12288, 8192, 1), (12304, 60000, 8192, 0), (60000, 12304, 8192, 0)):
            assert _cabi.lib.gsq_linear_vec_pair_serves(weight(a, ra, k), weight(b, rb, k), 4) == served, (a, b, ra, rb, k)
