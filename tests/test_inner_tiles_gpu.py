"""Forwards of inputs with inner positions through resident tiles of samples: every form of the weights and of the outputs, rows that
end inside a warp and inside a tile, last groups of trees that are short."""
import ctypes

import numpy as np
import pytest
import torch

import hingetreefortorch_b200._cabi as _cabi
from conftest import grad_close
from oracle import hinge_oracle as ho
from test_forest_gpu import dev, random_forest_inputs

THREADS, TILES = 0, 1

# B, C, inner, T, depth, M
SHAPES = [
    (40, 8, (33,), 401, 5, 2),      # rows of a warp and one position more
    (200, 8, (7,), 403, 4, 3),      # several rows per warp; scalar staging
    (2, 8, (20, 30), 517, 1, 4),
    (3, 9, (516,), 530, 9, 5),      # dealt out one by one
    (3, 9, (516,), 530, 7, 6),      # ... in twos
    (3, 9, (516,), 530, 3, 8),      # ... in fours
    (6, 300, (700,), 300, 6, 2),    # two-byte feature indices
    (9, 20, (900,), 130, 9, 3),     # wide paths
    (11, 16, (900,), 130, 10, 2),   # weights that leave no room for two trees at a time stay in global memory
    (9, 12, (1000,), 60, 12, 7),
    (5, 24, (1001,), 200, 8, 1),    # one output: weights in the records
    (9, 200, (1000,), 200, 10, 1),  # ... in global memory
    (60, 5, (85,), 70, 3, 1),
]


def taken(kind, x, w, keep=False):
    p = _cabi.forest_problem(kind, x, w)
    p.flags |= 4 if keep else 0  # HT_SAVE_FOR_BACKWARD
    return _cabi.library().ht_forest_forward_kernel(ctypes.byref(p))


def inputs(kind, shape):
    B, C, inner, T, depth, M = shape
    return random_forest_inputs(700 + SHAPES.index(shape), kind, B, C, inner, T, depth, (M,), quantise=True)


@pytest.mark.parametrize("shape, want", [((2796, 284, (169,), 8, 4, 1), THREADS), ((228, 47, (576,), 466, 5, 1), TILES),
                                         ((26, 1561, (3249,), 25, 4, 2), THREADS), ((135, 152, (2500,), 527, 3, 3), TILES)])
def test_choice_between_tiles_and_threads(shape, want):
    B, C, inner, T, depth, M = shape
    assert taken("tree", torch.empty((B, C) + inner, device="meta"), torch.empty(T, 2 ** depth, M, device="meta")) == want


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["tree", "fern"])
@pytest.mark.parametrize("shape", SHAPES, ids=[str(s) for s in SHAPES])
def test_tiles_match_oracle(kind, shape):
    x, thr, ord_, w = inputs(kind, shape)
    want = ho.forward(kind, x, thr, ord_, w)
    dx, dthr, dord, dw = dev(x, thr, ord_, w)
    if kind == "tree":
        assert taken(kind, dx, dw) == TILES
    f = _cabi.Forest(kind, dx, dw)
    assert np.array_equal(f.forward(dx, dthr, dord, dw).cpu().numpy(), want)
    g = np.random.default_rng(5).standard_normal(want.shape).astype(np.float32)
    ref, sizes = ho.backward(kind, x, thr, ord_, w, g), ho.backward_magnitudes(kind, x, thr, ord_, w, g)
    dg, = dev(g)
    assert np.array_equal(f.forward(dx, dthr, dord, dw, save=True).cpu().numpy(), want)
    for got, r, s in zip(f.backward(dx, dthr, dord, dw, dg, saved=True), ref, sizes):
        assert grad_close(got, r, s)
    for got, r, s in zip(f.backward(dx, dthr, dord, dw, dg), ref, sizes):  # walked again
        assert grad_close(got, r, s)
    x.reshape(-1)[:3] = [np.inf, -np.inf, np.nan]
    got = f.forward(dev(x)[0], dthr, dord, dw).cpu().numpy()
    assert np.array_equal(got, ho.forward(kind, x, thr, ord_, w), equal_nan=True)
    assert f.ordinal_flags() == 0


def test_choice_against_the_times_of_both_kernels():
    """profiles/inner_forward_choice.csv: forwards of random sizes, timed both ways."""
    import csv
    import math
    import os
    chosen = better = 0.0
    logs = []
    with open(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "profiles", "inner_forward_choice.csv")) as table:
        for row in csv.DictReader(table):
            B, C, K, T, depth, M = (int(row[c]) for c in ("B", "C", "K", "T", "depth", "M"))
            p = _cabi.ForestProblem(_cabi.HT_KIND[row["kind"]], depth, B, C, K, T, M, 4 if row["keeps_paths"] == "1" else 0, 0)
            takes = _cabi.library().ht_forest_forward_kernel(ctypes.byref(p))
            tiles, threads = float(row["tiles_us"]), float(row["threads_us"])
            chosen += tiles if takes == TILES else threads
            better += min(tiles, threads)
            logs.append(math.log((tiles if takes == TILES else threads) / min(tiles, threads)))
    assert chosen <= 1.02 * better and math.exp(sum(logs) / len(logs)) <= 1.03


def test_choice_on_forwards_that_the_estimates_were_not_fitted_to():
    """The rows of profiles/inner_forward_choice.csv that were kept out of the fit."""
    import csv
    import os
    chosen = better = 0.0
    with open(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "profiles", "inner_forward_choice.csv")) as table:
        for row in csv.DictReader(table):
            if row["held_out"] == "0":
                continue
            B, C, K, T, depth, M = (int(row[c]) for c in ("B", "C", "K", "T", "depth", "M"))
            p = _cabi.ForestProblem(_cabi.HT_KIND[row["kind"]], depth, B, C, K, T, M, 4 if row["keeps_paths"] == "1" else 0, 0)
            takes = _cabi.library().ht_forest_forward_kernel(ctypes.byref(p))
            times = {TILES: float(row["tiles_us"]), THREADS: float(row["threads_us"])}
            chosen += times[takes]
            better += min(times.values())
            assert times[takes] <= 1.15 * min(times.values()) or min(times.values()) < 100.0, row
    assert better > 0.0 and chosen <= 1.01 * better


# sizes at which tiles are taken for trees and for ferns, with and without kept paths
FORMS = [
    (96, 9, (33,), 131, 5, 2),
    (96, 9, (5, 6), 131, 2, 3),
    (6, 9, (500,), 131, 1, 4),
    (16, 9, (516,), 131, 9, 5),     # dealt out one by one
    (6, 9, (515,), 131, 7, 6),      # ... in twos
    (6, 9, (516,), 131, 3, 8),      # ... in fours
    (256, 9, (45,), 131, 6, 10),    # rows that end inside a warp
    (6, 9, (515,), 131, 10, 2),     # weights in global memory
    (24, 9, (515,), 131, 12, 7),
]


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["tree", "fern"])
@pytest.mark.parametrize("shape", FORMS, ids=[str(s) for s in FORMS])
def test_every_form_of_the_tiles(kind, shape):
    B, C, inner, T, depth, M = shape
    x, thr, ord_, w = random_forest_inputs(800 + FORMS.index(shape), kind, B, C, inner, T, depth, (M,), quantise=True)
    dx, dthr, dord, dw = dev(x, thr, ord_, w)
    assert taken(kind, dx, dw) == TILES and taken(kind, dx, dw, keep=True) == TILES
    f = _cabi.Forest(kind, dx, dw)
    want = ho.forward(kind, x, thr, ord_, w)
    assert np.array_equal(f.forward(dx, dthr, dord, dw).cpu().numpy(), want)
    assert np.array_equal(f.forward(dx, dthr, dord, dw, save=True).cpu().numpy(), want)
    g = np.random.default_rng(5).standard_normal(want.shape).astype(np.float32)
    dg, = dev(g)
    for got, r, s in zip(f.backward(dx, dthr, dord, dw, dg, saved=True), ho.backward(kind, x, thr, ord_, w, g),
                         ho.backward_magnitudes(kind, x, thr, ord_, w, g)):
        assert grad_close(got, r, s)
    assert f.ordinal_flags() == 0
