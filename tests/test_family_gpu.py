"""Image+vector fusion forests and forests followed by a linear layer, against the CPU oracle.

Bars: the fusion forward and the fused-linear forward are bit-exact (the fused-linear forward adds
its terms in the reference CPU order); gradients match within 1e-5 of the summed term magnitudes
(these backwards scatter with atomics, so their summation order is free)."""
import numpy as np
import pytest
import torch

from conftest import grad_close, grad_same, random_forest_inputs, requested_bytes
from oracle import hinge_oracle as ho

pytestmark = pytest.mark.gpu


def dev(*arrays):
    return [None if a is None else torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in arrays]


CASES = [
    # kind, B, C, inner, T, depth, extra, O, Cv
    ("tree", 64, 12, (), 10, 4, (), 5, 0),
    ("fern", 33, 9, (3,), 7, 5, (2,), 4, 0),
    ("tree", 40, 6, (2, 2), 9, 3, (2,), 3, 5),
    ("fern", 50, 8, (), 11, 6, (), 6, 4),
    ("tree", 257, 20, (), 33, 7, (), 10, 0),
]


@pytest.mark.parametrize("case", CASES, ids=[str(c) for c in CASES])
def test_fused_linear_and_fusion(case):
    from hingetreefortorch_b200 import _cabi
    kind, B, C, inner, T, depth, extra, O, Cv = case
    rng = np.random.default_rng(CASES.index(case))
    x, thr, ord_, w = random_forest_inputs(50 + CASES.index(case), kind, B, C, inner, T, depth, extra)
    vec = rng.standard_normal((B, Cv)).astype(np.float32) if Cv else None
    if Cv:
        ord_ = rng.integers(0, C + Cv, ord_.shape).astype(np.int64)
    lin = rng.standard_normal((O, T)).astype(np.float32)
    bias = rng.standard_normal(O).astype(np.float32)
    dx, dvec, dthr, dord, dw, dlin, dbias = dev(x, vec, thr, ord_, w, lin, bias)
    fam = _cabi.ForestFamily(kind, dx, dw, vec=dvec, lin=dlin)

    out = fam.linear_forward(dx, dvec, dthr, dord, dw, dlin, dbias)
    want = ho.linear_forward(kind, x, thr, ord_, w, lin, bias, vec=vec)
    assert out.shape == want.shape and np.array_equal(out.cpu().numpy(), want)
    g = rng.standard_normal(want.shape).astype(np.float32)
    dg, = dev(g)
    gx, gvec, gthr, gw, glin = fam.linear_backward(dx, dvec, dthr, dord, dw, dlin, dg)
    ref = ho.linear_backward(kind, x, thr, ord_, w, lin, g, vec=vec)
    mag = ho.magnitudes(ho.linear_backward, kind, x, thr, ord_, w, lin, g, vec=vec)
    if Cv:
        rx, rvec, rthr, rw, rlin, _ = ref
        ax, avec, athr, aw, alin, _ = mag
        assert grad_close(gvec, rvec, avec)
    else:
        rx, rthr, rw, rlin, _ = ref
        ax, athr, aw, alin, _ = mag
    assert grad_close(gx, rx, ax) and grad_close(gthr, rthr, athr) and grad_close(gw, rw, aw) and grad_close(glin, rlin, alin)
    assert fam.status.item() == 0

    if Cv:
        plain = _cabi.ForestFamily(kind, dx, dw, vec=dvec)
        out = plain.fusion_forward(dx, dvec, dthr, dord, dw)
        want = ho.forward(kind, x, thr, ord_, w, vec=vec)
        assert np.array_equal(out.cpu().numpy(), want)
        g2 = rng.standard_normal(want.shape).astype(np.float32)
        dg2, = dev(g2)
        gimg, gvec, gthr, gw = plain.fusion_backward(dx, dvec, dthr, dord, dw, dg2)
        rimg, rvec, rthr, rw = ho.backward(kind, x, thr, ord_, w, g2, vec=vec)
        aimg, avec, athr, aw = ho.magnitudes(ho.backward, kind, x, thr, ord_, w, g2, vec=vec)
        assert grad_close(gimg, rimg, aimg) and grad_close(gvec, rvec, avec)
        assert grad_close(gthr, rthr, athr) and grad_close(gw, rw, aw)


@pytest.mark.parametrize("setting", ["keep", "limit", "off"])
def test_fused_linear_keeps_its_paths_as_the_caller_allows(setting):
    """The forward's scratch stays until the backward, unless the scratch limit or the switch for keeping rules it out; the
    gradients are the same sums either way."""
    from hingetreefortorch_b200._ext import hingetree_cpp as ext
    from hingetreefortorch_b200.HingeTree import HingeTreeFusedLinear
    B, C, T, depth, O = 900, 24, 40, 6, 7
    rng = np.random.default_rng(3)
    x, thr, ord_, w = random_forest_inputs(60, "tree", B, C, (), T, depth, ())
    lin, bias, g = [rng.standard_normal(s).astype(np.float32) for s in ((O, T), O, (B, O))]
    ref = ho.linear_backward("tree", x, thr, ord_, w, lin, g)
    sizes = ho.magnitudes(ho.linear_backward, "tree", x, thr, ord_, w, lin, g)
    dx, dthr, dord, dw, dlin, dbias, dg = dev(x, thr, ord_, w, lin, bias, g)
    ext.tree_fused_linear_forward(dx, dthr, dord, dw, dlin, dbias)  # checks the ordinals
    wrt = [t.requires_grad_(True) for t in (dx, dthr, dw, dlin, dbias)]
    before = requested_bytes()
    try:
        if setting == "limit":
            ext.set_backward_scratch_limit(10 * B * T)
        elif setting == "off":
            ext.set_save_forward(False)
        out = HingeTreeFusedLinear.apply(dx, dthr, dord, dw, dlin, dbias)
        held = requested_bytes() - before - 4 * out.numel()
        grads = torch.autograd.grad(out, wrt, dg)
    finally:
        ext.set_backward_scratch_limit(2 ** 62)
        ext.set_save_forward(True)
    assert held >= 10 * B * T if setting == "keep" else held == 0
    for got, r, s in zip(grads, ref, sizes):
        assert grad_close(got, r, s)


@pytest.mark.parametrize("kind,depth", [("tree", 6), ("tree", 9), ("fern", 8), ("fern", 11)])
@pytest.mark.parametrize("offset_then", ["aligned", "moved"])
def test_fused_linear_on_data_off_the_copies_alignment(offset_then, kind, depth):
    """x that starts between two 16-byte boundaries, and a backward whose x is a copy elsewhere (saved-tensor hooks): the paths
    that the forward kept mean the same wherever x lies."""
    from hingetreefortorch_b200.HingeTree import HingeFernFusedLinear, HingeTreeFusedLinear
    B, C, T, O = 300, 24, 40, 7
    function = HingeTreeFusedLinear if kind == "tree" else HingeFernFusedLinear
    rng = np.random.default_rng(4)
    x, thr, ord_, w = random_forest_inputs(61, kind, B, C, (), T, depth, ())
    lin, bias, g = [rng.standard_normal(s).astype(np.float32) for s in ((O, T), O, (B, O))]
    ref = ho.linear_backward(kind, x, thr, ord_, w, lin, g)
    sizes = ho.magnitudes(ho.linear_backward, kind, x, thr, ord_, w, lin, g)
    dthr, dord, dw, dlin, dbias, dg = dev(thr, ord_, w, lin, bias, g)
    dx = torch.empty(B * C + 1, device="cuda")[1:].view(B, C).copy_(torch.from_numpy(x))
    assert dx.is_contiguous() and dx.data_ptr() % 16 == 4

    def elsewhere(t):  # a contiguous copy at another alignment
        start = 0 if t.data_ptr() % 16 else 1
        return torch.empty(t.numel() + start, dtype=t.dtype, device=t.device)[start:].view(t.shape).copy_(t)

    if offset_then == "aligned":  # the other way round: aligned in the forward, not in the backward
        dx = dx.clone()
    wrt = [t.requires_grad_(True) for t in (dx, dthr, dw, dlin, dbias)]
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t.detach(), elsewhere):
        out = function.apply(dx, dthr, dord, dw, dlin, dbias)
        grads = torch.autograd.grad(out, wrt, dg)
    assert np.array_equal(out.detach().cpu().numpy(), ho.linear_forward(kind, x, thr, ord_, w, lin, bias))
    for got, r, s in zip(grads, ref, sizes):
        assert grad_close(got, r, s)


# kind, B, C, T, depth, O of tabular calls with one output per leaf.  Linear outputs up to the last that the row kernels take and one
# beyond; more than 592 blocks of 256 samples (a block of threads takes several); records of 16 + 16 bits; last rows, and trees
# split among blocks; the narrowest x, an odd one, the widest whose gradient rows fit and one beyond.
LINEAR = [
    ("tree", 1000, 24, 33, 7, 16),
    ("fern", 1000, 24, 33, 7, 13),
    ("tree", 700, 24, 20, 6, 17),
    ("tree", 593 * 256 + 1, 6, 9, 4, 3),
    ("fern", 2 * 592 * 256 + 77, 5, 3, 3, 1),
    ("tree", 515, 40, 12, 9, 4),
    ("fern", 515, 40, 12, 12, 5),
    ("tree", 333, 1, 100, 5, 10),
    ("tree", 257, 783, 50, 7, 8),
    ("tree", 70, 1815, 17, 6, 2),
    ("tree", 70, 1900, 17, 6, 2),
    ("tree", 31, 10, 1, 1, 1),
]


@pytest.mark.parametrize("case", LINEAR, ids=[str(c) for c in LINEAR])
def test_fused_linear_on_tabular_data(case):
    """Through the operators (the backward walks again), through autograd from the forward's paths, and some gradients only."""
    from hingetreefortorch_b200 import HingeTree as F, _cabi
    kind, B, C, T, depth, O = case
    rng = np.random.default_rng(90 + LINEAR.index(case))
    x, thr, ord_, w = random_forest_inputs(90 + LINEAR.index(case), kind, B, C, (), T, depth, (), quantise=True)
    lin, bias, g = [rng.standard_normal(s).astype(np.float32) for s in ((O, T), O, (B, O))]
    ref = ho.linear_backward(kind, x, thr, ord_, w, lin, g)
    sizes = ho.magnitudes(ho.linear_backward, kind, x, thr, ord_, w, lin, g)
    tensors = dev(x, thr, ord_, w, lin, bias)
    dx, dthr, dord, dw, dlin, dbias = tensors
    dg, = dev(g)
    fam = _cabi.ForestFamily(kind, dx, dw, lin=dlin)
    want = ho.linear_forward(kind, x, thr, ord_, w, lin, bias)
    assert np.array_equal(fam.linear_forward(dx, None, dthr, dord, dw, dlin, dbias).cpu().numpy(), want)
    gx, _, gthr, gw, glin = fam.linear_backward(dx, None, dthr, dord, dw, dlin, dg)
    for got, r, s in zip((gx, gthr, gw, glin), ref, sizes):
        assert grad_close(got, r, s)
    assert fam.status.item() == 0
    function = F.HingeTreeFusedLinear if kind == "tree" else F.HingeFernFusedLinear
    for wanted in ((0, 1, 3, 4, 5), (0,), (4,), (1, 3)):
        wrt = [tensors[n].detach().requires_grad_(True) if n in wanted else tensors[n] for n in range(6)]
        out = function.apply(*wrt)
        assert np.array_equal(out.detach().cpu().numpy(), want)
        grads = torch.autograd.grad(out, [wrt[n] for n in wanted], dg)
        for n, got in zip(wanted, grads):
            at = n - (n > 2)  # the ordinals have none
            assert grad_close(got, ref[at], sizes[at])


# Rows of x streaming past resident trees: pitches that are padded and that are not, 16, 8 and 4 rows at a time, from fewer sets of
# trees than warps to several rounds of them, several groups of trees, more steps than row buffers and a last step that is short.
ROWS = [
    ("tree", 16 * 148 * 10 + 5, 64, 100, 7),
    ("tree", 16 * 148 * 3 + 16, 41, 9, 3),
    ("fern", 5000, 90, 113, 8),
    ("tree", 2400, 24, 250, 2),
    ("tree", 700, 1500, 65, 6),
    ("tree", 600, 3004, 40, 6),
    ("tree", 150, 5002, 70, 9),
    ("fern", 300, 6008, 20, 10),
]


@pytest.mark.parametrize("case", ROWS, ids=[str(c) for c in ROWS])
def test_rows_past_resident_trees(case):
    from hingetreefortorch_b200 import _cabi
    kind, B, C, T, depth = case
    rng = np.random.default_rng(190 + ROWS.index(case))
    x, thr, ord_, w = random_forest_inputs(190 + ROWS.index(case), kind, B, C, (), T, depth, (), quantise=True)
    x[0, :] = np.nan
    x[B - 1, ::2] = np.inf
    lin, bias = [rng.standard_normal(s).astype(np.float32) for s in ((2, T), 2)]
    dx, dthr, dord, dw, dlin, dbias = dev(x, thr, ord_, w, lin, bias)
    fam = _cabi.ForestFamily(kind, dx, dw, lin=dlin)
    got = fam.linear_forward(dx, None, dthr, dord, dw, dlin, dbias).cpu().numpy()
    with np.errstate(all="ignore"):
        assert np.array_equal(got, ho.linear_forward(kind, x, thr, ord_, w, lin, bias), equal_nan=True)
    assert fam.status.item() == 0
    # Gradients, the upstream one infinite and no number in places.  One linear output: with several their gradients are summed before
    # they meet the margin, and an infinite margin stays one where the reference's terms of opposite signs leave no number.
    lin, g = lin[:1].copy(), rng.standard_normal((B, 1)).astype(np.float32)
    g[B // 2], g[B // 3] = np.inf, np.nan
    dlin, dg = dev(lin, g)
    with np.errstate(all="ignore"):
        ref = ho.linear_backward(kind, x, thr, ord_, w, lin, g)
        sizes = ho.magnitudes(ho.linear_backward, kind, x, thr, ord_, w, lin, g)
    assert not np.isfinite(ref[0]).all() and np.isfinite(ref[0]).any()
    fam = _cabi.ForestFamily(kind, dx, dw, lin=dlin)
    gx, _, gthr, gw, glin = fam.linear_backward(dx, None, dthr, dord, dw, dlin, dg)
    for grad, r, s in zip((gx, gthr, gw, glin), ref, sizes):
        assert grad_same(grad, r, s)
    assert fam.status.item() == 0


def test_modules_fused_linear_and_fusion():
    from hingetreefortorch_b200 import RandomHingeForest as R
    torch.manual_seed(1)
    m = R.RandomHingeForestFusedLinear(16, 12, 5, 4, extra_outputs=2).cuda()
    x = torch.randn(32, 16, device="cuda", requires_grad=True)
    y = m(x)
    assert y.shape == (32, 5, 2)
    y.square().sum().backward()
    args = [t.detach().cpu().numpy() for t in (x, m.thresholds, m.ordinals, m.weights, m.linear_weights, m.linear_bias)]
    assert np.array_equal(y.detach().cpu().numpy(), ho.linear_forward("tree", *args))
    g = (2 * y).detach().cpu().numpy()
    gx, gthr, gw, glin, gbias = ho.linear_backward("tree", args[0], args[1], args[2], args[3], args[4], g)
    ax, athr, aw, alin, abias = ho.magnitudes(ho.linear_backward, "tree", args[0], args[1], args[2], args[3], args[4], g)
    assert grad_close(x.grad, gx, ax) and grad_close(m.thresholds.grad, gthr, athr) and grad_close(m.weights.grad, gw, aw)
    assert grad_close(m.linear_weights.grad, glin, alin) and grad_close(m.linear_bias.grad, gbias, abias)

    f = R.RandomHingeFernFusion(6, 3, 8, 4).cuda()
    img = torch.randn(5, 6, 4, 4, device="cuda", requires_grad=True)
    vec = torch.randn(5, 3, device="cuda", requires_grad=True)
    y = f(img, vec)
    assert y.shape == (5, 8, 4, 4)
    y.sum().backward()
    want = ho.forward("fern", img.detach().cpu().numpy(), f.thresholds.detach().cpu().numpy(), f.ordinals.cpu().numpy(),
                      f.weights.detach().cpu().numpy(), vec=vec.detach().cpu().numpy())
    assert np.array_equal(y.detach().cpu().numpy(), want)
    assert img.grad is not None and vec.grad is not None and vec.grad.shape == (5, 3)

    ff = R.RandomHingeForestFusionFusedLinear(6, 3, 8, 2, 3).cuda()
    y = ff(img.detach(), vec.detach().requires_grad_(True))
    assert y.shape == (5, 2, 4, 4)
    y.sum().backward()
