"""The convolution kernels for any shape at the edges of their slices, lots and bins, against the CPU oracle.

Bars: forward bit-exact (input channels are added in the reference's order, also where several warps walk them); gradients within
1e-5 of the summed term magnitudes, and where terms are infinite or no number the oracle's.
"""
import numpy as np
import pytest
import torch

from conftest import grad_same
from oracle import hinge_oracle as ho

pytestmark = pytest.mark.gpu

CASES = [
    # x shape, Co, depth, extra, kernel (1-D to 3-D by its length)
    ((1, 3, 34), 1, 3, (), (3,)),               # 32 outputs: one warp of positions, three channels for eight warps
    ((1, 9, 35), 1, 4, (2,), (3,)),             # a position and a channel more than a whole lot
    ((3, 17, 11), 5, 1, (5,), (2,)),            # depth 1, a chunk of four outputs and one more
    ((1, 8, 9, 10, 4), 2, 5, (6,), (2, 2, 2)),  # 3-D, outputs that are no multiple of four
    ((2, 2, 129), 3, 7, (4,), (2,)),            # slice of 256 evaluations exactly
    ((1, 2, 258), 3, 7, (4,), (2,)),            # ... and one more
    ((5, 20, 514), 32, 3, (), (3,)),            # four evaluations per thread, slices of 1024: 2560 evaluations
    ((4, 300, 18, 18), 2, 2, (4,), (3, 3)),     # ... 1024 exactly
    ((1, 2, 700), 2, 10, (), (9,)),             # as many bins as the sorted kernel takes
    ((1, 2, 300), 2, 11, (2,), (9,)),           # ... and more
    ((2, 3, 200), 2, 3, (66,), (3,)),           # more outputs than the shared forward adds up
    ((2, 32, 12, 12, 12), 32, 7, (), (2, 2, 2)),   # many leaves, enough outputs: the scatters
    ((2, 32, 12, 12, 12), 32, 6, (), (2, 2, 2)),   # half as many
]


def inputs(kind, case, seed, dtype=np.float32):
    xs, Co, depth, extra, kernel = case
    rng = np.random.default_rng(seed)
    N = 2 ** depth - 1 if kind == "tree" else depth
    x = rng.standard_normal(xs).astype(dtype)
    thr = rng.uniform(-1, 1, (Co, xs[1], N)).astype(dtype)
    ord_ = rng.integers(0, int(np.prod(kernel)), (Co, xs[1], N)).astype(np.int64)
    w = rng.standard_normal((Co, xs[1], 2 ** depth) + extra).astype(dtype)
    return x, thr, ord_, w


@pytest.mark.parametrize("special", [False, True], ids=["numbers", "infinite"])
@pytest.mark.parametrize("kind", ["tree", "fern"])
@pytest.mark.parametrize("case", CASES, ids=[str(c[:4]) for c in CASES])
def test_any_shape_kernels_match_oracle(kind, case, special):
    from hingetreefortorch_b200 import _cabi
    kernel = case[4]
    one = (1,) * len(kernel)
    geometry = (kernel, one, (0,) * len(kernel), one)
    x, thr, ord_, w = inputs(kind, case, CASES.index(case))
    if special:
        x.reshape(-1)[:3] = [np.inf, -np.inf, np.nan]
        x.reshape(-1)[5:9] = thr.reshape(-1)[0]  # margins of zero
    want = ho.conv_forward(kind, x, thr, ord_, w, *geometry)
    g = np.random.default_rng(1).standard_normal(want.shape).astype(np.float32)
    if special:
        g.reshape(-1)[[0, g.size // 2]] = [np.inf, np.nan]
    dx, dthr, dord, dw, dg = [torch.from_numpy(a).cuda() for a in (x, thr, ord_, w, g)]
    conv = _cabi.Conv(kind, dx, dw, *geometry)
    out = conv.forward(dx, dthr, dord, dw).cpu().numpy()
    assert np.array_equal(out, want, equal_nan=True)
    grads = conv.backward(dx, dthr, dord, dw, dg)
    with np.errstate(invalid="ignore"):
        refs = ho.conv_backward(kind, x, thr, ord_, w, g, *geometry)
        scales = ho.magnitudes(ho.conv_backward, kind, x, thr, ord_, w, g, *geometry)
    for got, ref, scale in zip(grads, refs, scales):
        assert grad_same(got, ref, scale)


@pytest.mark.parametrize("wanted", [(True, False, False), (False, True, False), (False, False, True), (False, True, True)])
def test_gradients_that_are_not_asked_for_are_left_out(wanted):
    from hingetreefortorch_b200.HingeTree import HingeTreeConv1d
    case = ((3, 5, 120), 4, 4, (6,), (3,))
    tensors = [torch.from_numpy(a).cuda() for a in inputs("tree", case, 3)]
    x, thr, ord_, w = tensors
    for t, need in zip((x, thr, w), wanted):
        t.requires_grad_(need)
    out = HingeTreeConv1d.apply(x, thr, ord_, w, (3,), (1,), (0,), (1,))
    g = np.random.default_rng(2).standard_normal(tuple(out.shape)).astype(np.float32)
    grads = torch.autograd.grad(out, [t for t, need in zip((x, thr, w), wanted) if need], torch.from_numpy(g).cuda())
    host = [t.detach().cpu().numpy() for t in tensors]
    geometry = ((3,), (1,), (0,), (1,))
    refs = ho.conv_backward("tree", *host, g, *geometry)
    scales = ho.magnitudes(ho.conv_backward, "tree", *host, g, *geometry)
    for got, (ref, scale) in zip(grads, [p for p, need in zip(zip(refs, scales), wanted) if need]):
        assert grad_same(got, ref, scale)


@pytest.mark.parametrize("kind", ["tree", "fern"])
def test_double_precision_sorted(kind):
    """Against the single-precision kernels on the same (single) numbers, whose terms differ by a few roundings."""
    from hingetreefortorch_b200 import RandomHingeForest as R
    torch.manual_seed(0)
    cls = getattr(R, "HingeTreeConv2d" if kind == "tree" else "HingeFernConv2d")
    m = cls(3, 4, 5, 3, padding=1, extra_outputs=5).cuda().double()
    x = torch.randn(3, 3, 21, 17, device="cuda").double().requires_grad_()
    out = m(x)
    g = torch.randn(out.shape, device="cuda").double()
    grads = torch.autograd.grad(out, [x, m.thresholds, m.weights], g)
    single = cls(3, 4, 5, 3, padding=1, extra_outputs=5).cuda()
    single.load_state_dict({k: v for k, v in m.state_dict().items()})
    xs = x.detach().float().requires_grad_()
    near = torch.autograd.grad(single(xs), [xs, single.thresholds, single.weights], g.float())
    for a, b in zip(grads, near):
        assert a.dtype == torch.float64 and torch.norm(a - b.double()) <= 1e-5 * torch.norm(a)
