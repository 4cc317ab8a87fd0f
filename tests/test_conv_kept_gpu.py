"""Convolution: the forward that takes four rows at a time, the codes that it keeps, and the gradients formed from them.  Trees
fewer than a CTA's warps and more, the shallowest and deepest, codes that use every spare bit, windows off the image, strides,
dilations, rows and columns off the tiles, input channels staged in several lots, single rows of outputs."""
import numpy as np
import pytest
import torch

import hingetreefortorch_b200._cabi as _cabi
from conftest import grad_close, grad_same, requested_bytes
from oracle import hinge_oracle as ho
from test_conv_gpu import dev

pytestmark = pytest.mark.gpu

CASES = [
    # dims, x shape, Co, depth, kernel, stride, padding, dilation
    (2, (5, 3, 33, 65), 40, 5, (3, 3), (1, 1), (1, 1), (1, 1)),
    (2, (16, 11, 37, 41), 4, 4, (3, 3), (1, 1), (1, 1), (1, 1)),
    (2, (40, 37, 9, 11), 33, 2, (2, 2), (1, 1), (0, 0), (1, 1)),
    (2, (3, 5, 50, 47), 67, 6, (5, 5), (2, 1), (2, 2), (1, 2)),
    (2, (2, 70, 40, 100), 8, 5, (5, 5), (1, 1), (2, 2), (1, 1)),
    (2, (2, 4, 61, 60), 130, 7, (4, 4), (1, 2), (0, 3), (2, 1)),
    (1, (3, 7, 1501), 35, 4, (5,), (1,), (2,), (1,)),
    (1, (9, 2, 3000), 100, 3, (2,), (2,), (0,), (3,)),
    (1, (2, 66, 4100), 3, 6, (3,), (1,), (1,), (1,)),
]


def inputs(kind, case):
    dims, xs, Co, depth, kernel, stride, padding, dilation = case
    rng = np.random.default_rng(90 + CASES.index(case))
    Ci, N = xs[1], (2 ** depth - 1 if kind == "tree" else depth)
    x = (np.round(rng.standard_normal(xs) * 4) / 4).astype(np.float32)  # margins of zero among them
    thr = (np.round(rng.uniform(-1, 1, (Co, Ci, N)) * 4) / 4).astype(np.float32)
    ord_ = rng.integers(0, int(np.prod(kernel)), (Co, Ci, N)).astype(np.int64)
    w = rng.standard_normal((Co, Ci, 2 ** depth)).astype(np.float32)
    return x, thr, ord_, w, (kernel, stride, padding, dilation), rng


@pytest.mark.parametrize("kind", ["tree", "fern"])
@pytest.mark.parametrize("case", CASES, ids=[str(c[:5]) for c in CASES])
def test_forward_and_backward_from_kept_codes(kind, case):
    x, thr, ord_, w, geometry, rng = inputs(kind, case)
    want = ho.conv_forward(kind, x, thr, ord_, w, *geometry)
    g = rng.standard_normal(want.shape).astype(np.float32)
    ref = ho.conv_backward(kind, x, thr, ord_, w, g, *geometry)
    sizes = ho.magnitudes(ho.conv_backward, kind, x, thr, ord_, w, g, *geometry)
    tensors = dev(x, thr, ord_, w, g)
    conv = _cabi.Conv(kind, tensors[0], tensors[3], *geometry)
    assert np.array_equal(conv.forward(*tensors[:4]).cpu().numpy(), want)
    assert conv.saved_bytes() > 0
    out, kept = conv.forward_saving(*tensors[:4])
    assert np.array_equal(out.cpu().numpy(), want)
    for need in ((True, True, True), (True, False, False), (False, True, False), (False, False, True), (True, True, True)):
        for wanted, got, r, s in zip(need, conv.backward_saved(*tensors, kept, need=need), ref, sizes):
            assert (got is None) if not wanted else grad_close(got, r, s)
    assert int(conv.status.item()) == 0
    # infinite pixels and one that is no number, in the first channels; the upstream gradient too
    x.reshape(-1)[:3] = [np.inf, -np.inf, np.nan]
    g.reshape(-1)[[0, 5]] = [np.inf, np.nan]
    dx, dg = dev(x, g)
    with np.errstate(all="ignore"):
        want = ho.conv_forward(kind, x, thr, ord_, w, *geometry)
        ref = ho.conv_backward(kind, x, thr, ord_, w, g, *geometry)
        sizes = ho.magnitudes(ho.conv_backward, kind, x, thr, ord_, w, g, *geometry)
    assert not all(np.isfinite(r).all() for r in ref) and all(np.isfinite(r).any() for r in ref)
    assert np.array_equal(conv.forward(dx, *tensors[1:4]).cpu().numpy(), want, equal_nan=True)
    out, kept = conv.forward_saving(dx, *tensors[1:4])
    assert np.array_equal(out.cpu().numpy(), want, equal_nan=True)
    for grads in (conv.backward_saved(dx, *tensors[1:4], dg, kept), conv.backward(dx, *tensors[1:4], dg)):
        for got, r, s in zip(grads, ref, sizes):
            assert grad_same(got, r, s)
    assert int(conv.status.item()) == 0


def test_codes_without_room_for_the_height_are_not_kept():
    x = torch.empty(4, 4, 64, 64)
    assert _cabi.Conv("tree", x.cuda(), torch.empty(32, 4, 128, device="cuda"), (5, 5), (1, 1), (2, 2), (1, 1)).saved_bytes() == 0


@pytest.mark.parametrize("setting", ["kept", "switched off", "limited"])
def test_autograd_keeps_the_codes_by_the_callers_settings(setting):
    """Two backwards through one graph, with and without what the forward may keep."""
    from hingetreefortorch_b200._ext import hingetree_cpp as ext
    x, thr, ord_, w, geometry, rng = inputs("tree", CASES[0])
    want = ho.conv_forward("tree", x, thr, ord_, w, *geometry)
    g = rng.standard_normal(want.shape).astype(np.float32)
    ref = ho.conv_backward("tree", x, thr, ord_, w, g, *geometry)
    sizes = ho.magnitudes(ho.conv_backward, "tree", x, thr, ord_, w, g, *geometry)
    dx, dthr, dord, dw, dg = dev(x, thr, ord_, w, g)
    leaves = [t.requires_grad_() for t in (dx, dthr, dw)]
    ext.tree_conv2d_forward(dx.detach(), dthr.detach(), dord, dw.detach(), *geometry)  # checks the ordinals
    codes = _cabi.Conv("tree", dx, dw, *geometry).saved_bytes()
    ext.set_save_forward(setting != "switched off")
    ext.set_backward_scratch_limit(codes - 1 if setting == "limited" else 2 ** 62)
    try:
        torch.cuda.synchronize()
        before = torch.cuda.memory_allocated()
        out = ext.tree_conv2d_apply(dx, dthr, dord, dw, *geometry)
        held = torch.cuda.memory_allocated() - before - out.numel() * 4
        assert (held >= codes) if setting == "kept" else held < codes
        assert np.array_equal(out.detach().cpu().numpy(), want)
        for _ in range(2):
            for got, r, s in zip(torch.autograd.grad(out, leaves, dg, retain_graph=True), ref, sizes):
                assert grad_close(got, r, s)
    finally:
        ext.set_save_forward(True)
        ext.set_backward_scratch_limit(2 ** 62)


def layer(x_shape=(4, 32, 32, 64), Co=32, depth=5):
    """The call of a 3 x 3 convolution, what it is differentiated by, an upstream gradient, and the bytes that a forward keeps."""
    from hingetreefortorch_b200._ext import hingetree_cpp as ext
    geometry = ((3, 3), (1, 1), (1, 1), (1, 1))
    x, w = torch.randn(x_shape, device="cuda"), torch.randn(Co, x_shape[1], 2 ** depth, device="cuda")
    thr = torch.rand(Co, x_shape[1], 2 ** depth - 1, device="cuda") - 0.5
    ord_ = torch.randint(0, 9, thr.shape, device="cuda")
    g = torch.randn_like(ext.tree_conv2d_forward(x, thr, ord_, w, *geometry))  # (which checks the ordinals)
    leaves = [t.requires_grad_() for t in (x, thr, w)]
    return lambda: ext.tree_conv2d_apply(x, thr, ord_, w, *geometry), leaves, g, _cabi.Conv("tree", x, w, *geometry).saved_bytes()


def test_a_backward_gives_back_what_the_forward_kept():
    """The output still referenced, as a training loop holds it until the next step's forward has run: of both steps' codes only
    one is ever there.  A graph that is retained holds on to them until the backward that does not retain it."""
    call, leaves, g, codes = layer()
    before = requested_bytes()
    out = call()
    assert requested_bytes() - before >= codes + out.numel() * 4
    torch.autograd.grad(out, leaves, g)
    assert requested_bytes() - before <= out.numel() * 4
    torch.cuda.reset_peak_memory_stats()
    second = call()
    assert requested_bytes(peak=True) - before < 2 * codes
    first = torch.autograd.grad(second, leaves, g, retain_graph=True)
    held = requested_bytes() - before
    again = torch.autograd.grad(second, leaves, g, retain_graph=True)
    assert requested_bytes() - held - before == sum(t.numel() * 4 for t in again)
    del again
    torch.autograd.grad(second, leaves, g)
    assert requested_bytes() - before <= 2 * out.numel() * 4 + sum(t.numel() * 4 for t in first)


def test_layers_together_keep_no_more_than_the_limit():
    from hingetreefortorch_b200._ext import hingetree_cpp as ext
    call, leaves, g, codes = layer()
    expected = torch.autograd.grad(call(), leaves, g)
    ext.set_backward_scratch_limit(2 * codes + codes // 2)
    try:
        before = requested_bytes()
        stack = [call() for _ in range(4)]
        assert 2 * codes <= requested_bytes() - before - 4 * g.numel() * 4 < 3 * codes
        for out in stack + [call()]:  # the last one keeps its codes again
            for a, b in zip(torch.autograd.grad(out, leaves, g), expected):
                assert (a - b).norm() <= 1e-5 * b.norm()
        before = requested_bytes()
        out = call()
        assert requested_bytes() - before >= codes
        del out, stack
    finally:
        ext.set_backward_scratch_limit(2 ** 62)


def within(room, what):
    """The call under a limit of that much more device memory than is in use."""
    torch.cuda.empty_cache()
    room += torch.cuda.memory_reserved()
    torch.cuda.set_per_process_memory_fraction(room / torch.cuda.get_device_properties(0).total_memory)
    try:
        return what()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)


def test_codes_give_way_to_the_forwards_scratch():
    """4.7 MB, from a segment of 20 MB, under a limit that results and codes alone would fill."""
    call, leaves, g, codes = layer((32, 16, 32, 32), 128, 7)
    before, segment = requested_bytes(), 2 ** 21
    out = within((-(-g.numel() * 4 // segment) - (-codes // segment)) * segment + 2 ** 20, call)
    assert requested_bytes() - before < codes
    assert torch.equal(out, call())


def test_codes_give_way_to_the_gradients():
    """The image's gradient, 17 MB, under a limit that leaves no room beside the codes; after that a second backward, which walks."""
    torch.cuda.empty_cache()
    call, leaves, g, codes = layer((64, 16, 64, 64), 16, 5)
    expected = torch.autograd.grad(call(), leaves, g)
    torch.cuda.empty_cache()
    out = call()
    torch.cuda.empty_cache()
    held = requested_bytes()
    assert torch.cuda.memory_reserved() - held < leaves[0].numel() * 4  # (else the gradient fits into what is cached)
    got = within(2 ** 20, lambda: torch.autograd.grad(out, leaves, g, retain_graph=True))
    assert requested_bytes() < held  # the codes are gone
    for grads in (got, torch.autograd.grad(out, leaves, g)):
        for a, b in zip(grads, expected):  # sums in another order, the bar of the module's cases
            assert (a - b).norm() <= 1e-5 * b.norm()
