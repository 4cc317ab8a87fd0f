"""Convolution backwards of any shape: which kernel takes a call, and both kernels at padded, strided and dilated windows, whole and
partial slices of 256 and 1024 evaluations, in either precision.

Bars: forward bit-exact; gradients against the oracle (single precision) within 1e-5 of the summed term magnitudes.  In double precision
against the sums of numpy: fewer than 2^13 terms per element in either order are within 2 * 2^13 * 2^-53 = 2e-12 of the magnitudes.
"""
import csv
import ctypes
import itertools
import os

import numpy as np
import pytest
import torch

from conftest import grad_close
from hingetreefortorch_b200 import _cabi
from oracle import hinge_oracle as ho

SCATTERED, SORTED, TILES = 0, 1, 2


def route(kind, depth, x_shape, Co, M, kernel, stride, padding, dilation, real_bytes):
    dims = len(kernel)
    p = _cabi.ConvProblem(_cabi.HT_KIND[kind], depth, dims, 0, x_shape[0], x_shape[1], Co, M, _cabi._triple(x_shape[2:], 1),
                          _cabi._triple(kernel, 1), _cabi._triple(stride, 1), _cabi._triple(padding, 0), _cabi._triple(dilation, 1))
    return _cabi.library().ht_conv_backward_kernel(ctypes.byref(p), real_bytes)


def table(held_out):
    with open(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "profiles", "conv_backward_choice.csv")) as f:
        for row in csv.DictReader(f):
            if row["held_out"] == held_out:
                n = {k: int(row[k]) for k in ("dims", "B", "Ci", "Co", "size", "window", "stride", "padding", "depth", "M", "real_bytes")}
                d = n["dims"]
                takes = route(row["kind"], n["depth"], (n["B"], n["Ci"]) + (n["size"],) * d, n["Co"], n["M"], (n["window"],) * d,
                              (n["stride"],) * d, (n["padding"],) * d, (1,) * d, n["real_bytes"])
                yield n["real_bytes"], takes, {SORTED: float(row["sorted_us"]), SCATTERED: float(row["scatters_us"])}


@pytest.mark.parametrize("real_bytes", [4, 8])
@pytest.mark.parametrize("held_out", ["0", "1"])
def test_choice_against_the_times_of_both_kernels(real_bytes, held_out):
    chosen = better = 0.0
    for bytes_, takes, times in table(held_out):
        if bytes_ == real_bytes:
            chosen += times[takes]
            better += min(times.values())
            assert times[takes] <= 1.3 * min(times.values()) or min(times.values()) < 100.0
    assert better > 0.0 and chosen <= 1.02 * better


def test_route_of_calls_that_a_kernel_of_their_own_serves_better():
    # 3-D, one output per leaf, few leaves in all: scattered 695 us, sorted 982
    assert route("tree", 3, (35, 30, 7, 7, 7), 75, 1, (2,) * 3, (1,) * 3, (1,) * 3, (1,) * 3, 4) == SCATTERED
    assert route("tree", 4, (64, 8, 64, 64), 16, 4, (3, 3), (1, 1), (1, 1), (1, 1), 4) == SORTED
    assert route("tree", 5, (64, 64, 64, 64), 128, 1, (3, 3), (1, 1), (1, 1), (1, 1), 4) == TILES
    assert route("tree", 11, (1, 2, 300), 2, 2, (9,), (1,), (0,), (1,), 4) == SCATTERED  # more bins than the sorted kernel takes


# x shape, Co, depth, outputs, kernel, stride, padding, dilation, single precision's and double precision's route
CASES = [
    ((3, 4, 11, 10, 9), 40, 3, 1, (2, 3, 2), (1, 1, 1), (1, 1, 1), (1, 1, 1), SORTED, SORTED),    # 4 per thread, last slice of 1024 partial
    ((5, 7, 29, 31), 25, 4, 3, (3, 3), (1, 1), (1, 1), (1, 1), SORTED, SORTED),                   # ... three outputs (a chunk and more in double)
    ((6, 6, 35, 33), 27, 5, 5, (3, 2), (1, 2), (2, 1), (2, 1), SORTED, SORTED),                   # ... strided, dilated, wide padding
    ((1, 3, 700), 5, 6, 2, (5,), (2,), (2,), (3,), SORTED, SORTED),                               # 1 per thread
    ((2, 5, 9, 9, 9), 3, 2, 1, (3, 3, 3), (2, 2, 2), (1, 1, 1), (1, 1, 1), SORTED, SORTED),
    ((4, 8, 9, 9, 9), 120, 6, 1, (2, 2, 2), (1, 1, 1), (1, 1, 1), (1, 1, 1), SCATTERED, SCATTERED),
]


def inputs(kind, case, dtype):
    shape, Co, depth, M, kernel = case[:5]
    rng = np.random.default_rng(CASES.index(case))
    N = 2 ** depth - 1 if kind == "tree" else depth
    x = rng.standard_normal(shape).astype(dtype)
    thr = rng.uniform(-1, 1, (Co, shape[1], N)).astype(dtype)
    ord_ = rng.integers(0, int(np.prod(kernel)), (Co, shape[1], N)).astype(np.int64)
    w = rng.standard_normal((Co, shape[1], 2 ** depth, M)).astype(dtype)
    return x, thr, ord_, w


def numpy_step(kind, x, thr, ord_, w, g, kernel, stride, padding, dilation):
    """Forward and gradients in double precision, each gradient with the sum of its terms' magnitudes."""
    dims, (B, Ci), (Co, _, L, M) = len(kernel), x.shape[:2], w.shape
    depth, size = L.bit_length() - 1, x.shape[2:]
    image = np.pad(x, [(0, 0), (0, 0)] + [(p, p) for p in padding])
    places = np.arange(np.prod(image.shape[2:])).reshape(image.shape[2:])
    osize = [(s + 2 * p - d * (k - 1) - 1) // t + 1 for s, p, d, k, t in zip(size, padding, dilation, kernel, stride)]
    origins = places[np.ix_(*[np.arange(o) * t for o, t in zip(osize, stride)])].reshape(-1)
    cells = np.array([np.ravel_multi_index([q * d for q, d in zip(cell, dilation)], image.shape[2:])
                      for cell in itertools.product(*[range(k) for k in kernel])])
    flat = image.reshape(B, Ci, -1)
    out = np.zeros((B, Co, origins.size, M))
    g = g.reshape(out.shape)
    sums = [[np.zeros_like(flat), np.zeros_like(thr), np.zeros_like(w)] for _ in range(2)]
    rows, at = np.arange(B)[:, None], origins[None, :]
    for j in range(Co):
        for c in range(Ci):
            v = np.zeros((B, origins.size), dtype=np.int64)
            key, best, vertex = v.copy(), np.full(v.shape, np.inf), v.copy()
            for level in range(depth):
                here = v if kind == "tree" else np.full_like(v, level)
                margin = flat[rows, c, at + cells[ord_[j, c, here]]] - thr[j, c, here]
                nearer = np.abs(margin) < np.abs(best)
                best, vertex = np.where(nearer, margin, best), np.where(nearer, here, vertex)
                key |= (margin > 0).astype(np.int64) << level
                v = 2 * v + 1 + (margin > 0)
            out[:, j] += np.abs(best)[..., None] * w[j, c, key]
            products = np.sign(best)[..., None] * w[j, c, key] * g[:, j]
            for (gx, gthr, gw), of in zip(sums, (lambda t: t, np.abs)):
                terms = of(products).sum(-1)
                np.add.at(gx, (rows, c, at + cells[ord_[j, c, vertex]]), terms)
                np.add.at(gthr[j, c], vertex, -terms)
                np.add.at(gw[j, c], key, of(np.abs(best)[..., None] * g[:, j]))
    inside = (slice(None), slice(None)) + tuple(slice(p, p + s) for p, s in zip(padding, size))
    grads, scales = [[s[0].reshape(image.shape)[inside], s[1], s[2]] for s in sums]
    return out.reshape([B, Co] + osize + [M]), grads, [np.abs(s) for s in scales]


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["tree", "fern"])
@pytest.mark.parametrize("case", CASES, ids=[str(c[:4]) for c in CASES])
def test_single_precision(kind, case):
    geometry = case[4:8]
    x, thr, ord_, w = inputs(kind, case, np.float32)
    if kind == "tree":
        assert route(kind, case[2], case[0], case[1], case[3], *geometry, 4) == case[8]
    want = ho.conv_forward(kind, x, thr, ord_, w, *geometry)
    g = np.random.default_rng(1).standard_normal(want.shape).astype(np.float32)
    dx, dthr, dord, dw, dg = [torch.from_numpy(a).cuda() for a in (x, thr, ord_, w, g)]
    conv = _cabi.Conv(kind, dx, dw, *geometry)
    assert np.array_equal(conv.forward(dx, dthr, dord, dw).cpu().numpy(), want)
    refs = ho.conv_backward(kind, x, thr, ord_, w, g, *geometry)
    scales = ho.magnitudes(ho.conv_backward, kind, x, thr, ord_, w, g, *geometry)
    for got, ref, scale in zip(conv.backward(dx, dthr, dord, dw, dg), refs, scales):
        assert grad_close(got, ref, scale)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["tree", "fern"])
@pytest.mark.parametrize("case", CASES, ids=[str(c[:4]) for c in CASES])
def test_double_precision(kind, case):
    from hingetreefortorch_b200._ext import hingetree_cpp
    geometry = case[4:8]
    x, thr, ord_, w = inputs(kind, case, np.float64)
    if kind == "tree":
        assert route(kind, case[2], case[0], case[1], case[3], *geometry, 8) == case[9]
    name = "%s_conv%dd_" % (kind, len(case[4]))
    dx, dthr, dord, dw = [torch.from_numpy(a).cuda() for a in (x, thr, ord_, w)]
    lists = [list(v) for v in geometry]
    out = getattr(hingetree_cpp, name + "forward")(dx, dthr, dord, dw, *lists)
    g = np.random.default_rng(1).standard_normal(tuple(out.shape))
    want, refs, scales = numpy_step(kind, x, thr, ord_, w, g, *geometry)
    assert np.allclose(out.cpu().numpy(), want, rtol=0, atol=1e-12 * np.abs(want).max())
    gx, gthr, _, gw = getattr(hingetree_cpp, name + "backward")(dx, True, dthr, True, dord, False, dw, True, torch.from_numpy(g).cuda(), *lists)
    for got, ref, scale in zip((gx, gthr, gw), refs, scales):
        assert grad_close(got, ref, scale, rel=2e-12)
