"""The convolution's backward through one walk: codes for the whole batch, for a part of it at a time, and for none (each
kernel walks); single rows of outputs, rows and columns off the tiles, odd channel counts, the widest and deepest codes."""
import numpy as np
import pytest
import torch

import hingetreefortorch_b200._cabi as _cabi
from conftest import grad_close, requested_bytes
from oracle import hinge_oracle as ho
from test_conv_gpu import dev

pytestmark = pytest.mark.gpu

CASES = [
    # dims, x shape, Co, depth, kernel, stride, padding, dilation
    (2, (5, 3, 33, 65), 40, 5, (3, 3), (1, 1), (1, 1), (1, 1)),
    (2, (3, 5, 50, 47), 37, 3, (5, 3), (2, 1), (0, 2), (1, 2)),
    (2, (2, 4, 40, 40), 24, 7, (11, 11), (1, 1), (5, 5), (1, 1)),
    (1, (3, 7, 1501), 35, 4, (5,), (1,), (2,), (1,)),
    (1, (9, 2, 700), 100, 1, (2,), (2,), (0,), (3,)),
]


@pytest.mark.parametrize("kind", ["tree", "fern"])
@pytest.mark.parametrize("case", CASES, ids=[str(c[:4]) for c in CASES])
def test_backward_through_codes(kind, case):
    dims, xs, Co, depth, kernel, stride, padding, dilation = case
    rng = np.random.default_rng(70 + CASES.index(case))
    Ci, N = xs[1], (2 ** depth - 1 if kind == "tree" else depth)
    x = (np.round(rng.standard_normal(xs) * 4) / 4).astype(np.float32)  # margins of zero among them
    thr = (np.round(rng.uniform(-1, 1, (Co, Ci, N)) * 4) / 4).astype(np.float32)
    ord_ = rng.integers(0, int(np.prod(kernel)), (Co, Ci, N)).astype(np.int64)
    w = rng.standard_normal((Co, Ci, 2 ** depth)).astype(np.float32)
    geometry = (kernel, stride, padding, dilation)
    want = ho.conv_forward(kind, x, thr, ord_, w, *geometry)
    g = rng.standard_normal(want.shape).astype(np.float32)
    ref = ho.conv_backward(kind, x, thr, ord_, w, g, *geometry)
    sizes = ho.magnitudes(ho.conv_backward, kind, x, thr, ord_, w, g, *geometry)
    tensors = dev(x, thr, ord_, w, g)
    for share in (1.0, 0.5, 0.0):
        conv = _cabi.Conv(kind, tensors[0], tensors[3], *geometry, code_share=share)
        for got, r, s in zip(conv.backward(*tensors), ref, sizes):
            assert grad_close(got, r, s)
        assert int(conv.status.item()) == 0


@pytest.mark.parametrize("samples", [5, 2, 0])
def test_backward_within_the_scratch_limit(samples):
    """The operator's codes stay within the limit that the caller set: the whole batch, two samples at a time, none."""
    from hingetreefortorch_b200._ext import hingetree_cpp as ext
    dims, xs, Co, depth, kernel, stride, padding, dilation = CASES[0]
    rng = np.random.default_rng(80)
    x = rng.standard_normal(xs).astype(np.float32)
    thr = rng.uniform(-1, 1, (Co, xs[1], 2 ** depth - 1)).astype(np.float32)
    ord_ = rng.integers(0, int(np.prod(kernel)), thr.shape).astype(np.int64)
    w = rng.standard_normal((Co, xs[1], 2 ** depth)).astype(np.float32)
    g = rng.standard_normal((xs[0], Co, 33, 65)).astype(np.float32)
    ref = ho.conv_backward("tree", x, thr, ord_, w, g, kernel, stride, padding, dilation)
    sizes = ho.magnitudes(ho.conv_backward, "tree", x, thr, ord_, w, g, kernel, stride, padding, dilation)
    dx, dthr, dord, dw, dg = dev(x, thr, ord_, w, g)
    ext.tree_conv2d_forward(dx, dthr, dord, dw, kernel, stride, padding, dilation)  # checks the ordinals
    code_bytes = 2 * Co * xs[1] * 36 * 68 + 65536  # of a sample: rows and columns rounded up to groups; tree records
    limit = samples * code_bytes
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = requested_bytes()
    ext.set_backward_scratch_limit(limit)
    try:
        grads = ext.tree_conv2d_backward(dx, True, dthr, True, dord, False, dw, True, dg, kernel, stride, padding, dilation)
    finally:
        ext.set_backward_scratch_limit(2 ** 62)
    assert requested_bytes(peak=True) - before <= x.nbytes + thr.nbytes + w.nbytes + max(limit, 16 * thr.size + 4 * w.size + 65536)
    for got, r, s in zip((grads[0], grads[1], grads[3]), ref, sizes):
        assert grad_close(got, r, s)
