"""The C-ABI library loads and exports every symbol include/*.h declares.  No GPU needed."""
import ctypes
import glob
import os
import re
import threading

from conftest import ROOT
from hingetreefortorch_b200 import _build, _cabi


def declared_symbols():
    names = set()
    for header in glob.glob(os.path.join(ROOT, "include", "*.h")):
        text = open(header).read()
        text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
        names |= set(re.findall(r"\b(ht_[a-z0-9_]+)\s*\(", text))
    return names


def test_library_exports_every_declared_symbol():
    lib = ctypes.CDLL(_build.library_path())
    declared = declared_symbols()
    assert declared, "no declarations found"
    for name in declared:
        assert hasattr(lib, name), name
    assert declared == set(_cabi.SYMBOLS)


def test_status_strings_and_version():
    lib = _cabi.library()
    assert lib.ht_version() >= 100
    for status in range(0, -6, -1):
        assert lib.ht_status_string(status)
    assert b"unknown" in lib.ht_status_string(-99)


def test_workspace_query_and_argument_screening():
    lib = _cabi.library()
    p = _cabi.ForestProblem(0, 8, 1024, 128, 1, 1024, 1, 0, 0)
    need = lib.ht_forest_workspace_bytes(ctypes.byref(p))
    assert need >= 1024 * 255 * 4
    bad_depth = _cabi.ForestProblem(0, 32, 1, 1, 1, 1, 1, 0, 0)
    assert lib.ht_forest_workspace_bytes(ctypes.byref(bad_depth)) == 0
    # bad arguments are refused before anything touches a device
    rc = lib.ht_forest_forward_f32(ctypes.byref(bad_depth), None, None, None, None, None, None, ctypes.c_size_t(0), None, None)
    assert rc == -2
    rc = lib.ht_forest_forward_f32(ctypes.byref(p), None, None, None, None, None, None, ctypes.c_size_t(0), None, None)
    assert rc == -1
    rc = lib.ht_forest_forward_f32(None, None, None, None, None, None, None, ctypes.c_size_t(0), None, None)
    assert rc == -1


def test_image_shaped_forwards_run_without_room_for_tile_records():
    """The packed ordinals are enough where no tile kernel is needed, and room for what a backward keeps where that is asked for.  (The
    workspace's size is looked at before the missing output; nothing here is read.)"""
    lib = _cabi.library()
    host = (ctypes.c_char * 256)()
    for kind, B, C, K, T, depth, M in [(0, 8, 16, 64, 4096, 8, 2), (0, 135, 152, 2500, 527, 3, 3), (1, 228, 47, 576, 466, 5, 2),
                                       (0, 9, 200, 1000, 200, 10, 1)]:
        for flags in (0, 2):  # HT_WORKSPACE_FOR_BACKWARD
            p = _cabi.ForestProblem(kind, depth, B, C, K, T, M, flags, 0)
            ordinals = (T * (depth if kind else 2 ** depth - 1) * 4 + 255) // 256 * 256 + 256
            backward = 0
            if flags and M > 1:
                backward = lib.ht_forest_workspace_bytes(ctypes.byref(p))
                p.flags = 0
                backward -= lib.ht_forest_workspace_bytes(ctypes.byref(p))
                p.flags = flags
                assert backward >= T * B * K * 6
            elif flags:
                continue

            def call(workspace_bytes):
                at = ctypes.c_void_p((ctypes.addressof(host) + 255) // 256 * 256)
                some = ctypes.c_void_p(ctypes.addressof(host))
                return lib.ht_forest_forward_f32(ctypes.byref(p), some, some, some, some, None, at, ctypes.c_size_t(workspace_bytes), None, None)

            assert call(ordinals + backward) == -1  # the missing output
            assert call(ordinals - 257) == -4
            assert lib.ht_forest_workspace_bytes(ctypes.byref(p)) >= ordinals + backward


def test_backward_workspace_counts_records_only_where_they_are_used():
    """One output per leaf on more features than the tile kernels take: the gradients are scattered, in either mode of the workspace."""
    lib = _cabi.library()

    def size(flags, kind, B, C, K, T, depth):
        return lib.ht_forest_workspace_bytes(ctypes.byref(_cabi.ForestProblem(kind, depth, B, C, K, T, 1, flags, 0)))

    for shape in [(1, 601, 914, 64, 35, 7), (0, 64, 1000, 4096, 256, 8), (0, 40000, 1800, 1, 64, 6)]:
        evaluations = shape[1] * shape[3] * shape[4]
        assert size(2, *shape) == size(0, *shape)  # HT_WORKSPACE_FOR_BACKWARD
        if evaluations <= 1 << 26:
            assert size(3, *shape) >= size(0, *shape) + 22 * evaluations  # fixed order: paths and lists
    for shape in [(1, 601, 91, 64, 35, 7), (0, 40000, 180, 1, 64, 6)]:
        assert size(2, *shape) >= size(0, *shape) + 10 * shape[1] * shape[3] * shape[4]


def test_convolution_plans_at_hand_are_those_of_the_question():
    """Sizes asked for in turn, and each in a thread of its own, which has no earlier plan at hand: the same answers."""
    lib = _cabi.library()
    lib.ht_conv_saved_bytes.restype = lib.ht_conv_workspace_bytes.restype = ctypes.c_size_t
    t = _cabi._triple
    problems = [_cabi.ConvProblem(kind, depth, 2, 0, 4, ci, co, 1, t((h, h), 1), t((k, k), 1), t((1, 1), 1), t((p, p), 0), t((1, 1), 1))
                for kind, depth, ci, co, h, k, p in [(0, 5, 64, 128, 64, 3, 1), (1, 5, 64, 128, 64, 3, 1), (0, 7, 8, 16, 128, 3, 1),
                                                     (0, 4, 3, 64, 224, 5, 2), (0, 7, 8, 16, 128, 5, 2), (0, 5, 2, 2, 8, 3, 1)]]

    def sizes(p):
        return lib.ht_conv_saved_bytes(ctypes.byref(p)), lib.ht_conv_workspace_bytes(ctypes.byref(p))

    alone = []
    for p in problems:
        thread = threading.Thread(target=lambda p=p: alone.append(sizes(p)))
        thread.start()
        thread.join()
    assert [a[0] > 0 for a in alone] == [True, True, True, True, False, False]
    for order in (range(len(problems)), reversed(range(len(problems)))):
        for k in order:
            assert sizes(problems[k]) == alone[k] == sizes(problems[k])
