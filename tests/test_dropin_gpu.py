"""The reference-facing surface on a GPU: the `hingetree_cpp` operators, the autograd
Functions and the nn.Modules, checked against the CPU oracle."""
import copy

import numpy as np
import pytest
import torch

from conftest import grad_close, random_forest_inputs, requested_bytes
from oracle import hinge_oracle as ho

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ext():
    from hingetreefortorch_b200._ext import hingetree_cpp
    return hingetree_cpp


def dev(*arrays):
    return [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in arrays]


@pytest.mark.parametrize("kind", ["tree", "fern"])
def test_operators_match_oracle(ext, kind):
    x, thr, ord_, w = random_forest_inputs(21, kind, 40, 12, (3,), 10, 4, (2,))
    g = np.random.default_rng(0).standard_normal((40, 10, 3, 2)).astype(np.float32)
    dx, dthr, dord, dw, dg = dev(x, thr, ord_, w, g)
    out = getattr(ext, kind + "_forward")(dx, dthr, dord, dw)
    assert out.shape == (40, 10, 3, 2) and np.array_equal(out.cpu().numpy(), ho.forward(kind, x, thr, ord_, w))
    leaf, margin, mord, reach = ho.maps(kind, x, thr, ord_, w)
    got_leaf = getattr(ext, kind + "_leafmap")(dx, dthr, dord, dw)
    assert got_leaf.dtype == torch.int64 and np.array_equal(got_leaf.cpu().numpy(), leaf)
    got_margin, got_mord = getattr(ext, kind + "_marginmap")(dx, dthr, dord, dw)
    assert np.array_equal(got_margin.cpu().numpy(), margin) and np.array_equal(got_mord.cpu().numpy(), mord)
    got_reach = getattr(ext, kind + "_reachability")(dx, dthr, dord, dw)
    assert got_reach.dtype == torch.int64 and np.array_equal(got_reach.cpu().numpy(), reach)
    want = ho.backward(kind, x, thr, ord_, w, g)
    grads = getattr(ext, kind + "_backward_deterministic")(dx, True, dthr, True, dord, False, dw, True, dg)
    assert grads[2] is None
    for got, ref in zip((grads[0], grads[1], grads[3]), want):
        assert np.array_equal(got.cpu().numpy(), ref)
    grads = getattr(ext, kind + "_backward")(dx, True, dthr, False, dord, False, dw, True, dg)
    assert grads[1] is None and grads[2] is None
    mags = ho.backward_magnitudes(kind, x, thr, ord_, w, g)
    assert grad_close(grads[0], want[0], mags[0]) and grad_close(grads[3], want[2], mags[2])
    assert getattr(ext, kind + "_backward")(dx, False, dthr, False, dord, False, dw, False, dg) == [None] * 4


def test_module_training_step_keeps_the_forward_traversal(ext):
    """A module large enough for the tile kernel: the autograd Function keeps the forward's traversal and the
    backward uses it (ext.tree_forward_saving returns a non-empty scratch); results match the oracle at the
    usual bars, in default and in deterministic mode, and equal those with keeping switched off."""
    from hingetreefortorch_b200 import RandomHingeForest as R
    torch.manual_seed(3)
    m = R.RandomHingeForest(128, 64, 6, extra_outputs=1).cuda()
    x = torch.randn(1024, 128, device="cuda", requires_grad=True)
    w2 = m.weights.detach().reshape(64, 64)
    assert ext.tree_forward_saving(x.detach(), m.thresholds.detach(), m.ordinals, w2)[1].numel() > 0
    results = {}
    for keep in (True, False):
        ext.set_save_forward(keep)
        try:
            for p in (x, m.thresholds, m.weights):
                p.grad = None
            y = m(x)
            (y * y).sum().backward()
            results[keep] = [t.detach().clone() for t in (y, x.grad, m.thresholds.grad, m.weights.grad)]
        finally:
            ext.set_save_forward(True)
    xn, thr, ord_, w = x.detach().cpu().numpy(), m.thresholds.detach().cpu().numpy(), m.ordinals.cpu().numpy(), m.weights.detach().cpu().numpy()
    want = ho.forward("tree", xn, thr, ord_, w)
    g = 2 * want
    ref = ho.backward("tree", xn, thr, ord_, w, g)
    mags = ho.backward_magnitudes("tree", xn, thr, ord_, w, g)
    for keep in (True, False):
        assert np.array_equal(results[keep][0].cpu().numpy(), want)
        for t, r, mg in zip(results[keep][1:], ref, mags):
            assert grad_close(t, r, mg)
    assert torch.equal(results[True][1], results[False][1])  # the x gradient is added in tree order either way
    prev = torch.are_deterministic_algorithms_enabled()
    torch.use_deterministic_algorithms(True)
    try:
        for p in (x, m.thresholds, m.weights):
            p.grad = None
        y = m(x)
        (y * y).sum().backward()
    finally:
        torch.use_deterministic_algorithms(prev)
    for t, r in zip((x.grad, m.thresholds.grad, m.weights.grad), ref):
        assert np.array_equal(t.cpu().numpy(), r)


def test_error_contract_on_device(ext):
    x, thr, ord_, w = random_forest_inputs(22, "tree", 8, 5, (), 3, 3, ())
    dx, dthr, dord, dw = dev(x, thr, ord_, w)
    bad = dord.clone()
    bad[0, 0] = 5
    with pytest.raises(RuntimeError, match="ordinal"):
        ext.tree_forward(dx, dthr, bad, dw)
    with pytest.raises(RuntimeError, match="ordinal"):
        ext.tree_backward(dx, True, dthr, True, bad, False, dw, True, torch.ones(8, 3, device="cuda"))
    with pytest.raises(ValueError, match="same device"):
        ext.tree_forward(dx, dthr.cpu(), dord, dw)
    with pytest.raises(RuntimeError, match="tree depth"):
        ext.tree_forward(dx, dthr[:, :6].contiguous(), dord[:, :6].contiguous(), dw)
    with pytest.raises(ValueError, match="outDataGrad.shape"):
        ext.tree_backward(dx, True, dthr, True, dord, False, dw, True, torch.ones(8, 4, device="cuda"))
    with pytest.raises(ValueError):  # mixed real types
        ext.tree_forward(dx.double(), dthr, dord, dw)
    with pytest.raises(ValueError):  # half precision is taken by no operator
        ext.tree_forward(dx.half(), dthr.half(), dord, dw.half())
    # a valid ordinals tensor that is later corrupted in place is re-validated (version changed)
    ext.tree_forward(dx, dthr, dord, dw)
    dord[1, 1] = -3
    with pytest.raises(RuntimeError, match="ordinal"):
        ext.tree_forward(dx, dthr, dord, dw)


@pytest.mark.parametrize("module_name,kind", [("RandomHingeForest", "tree"), ("RandomHingeFern", "fern")])
def test_modules_forward_backward(module_name, kind):
    from hingetreefortorch_b200 import RandomHingeForest as R
    torch.manual_seed(0)
    m = getattr(R, module_name)(20, 16, 5, extra_outputs=3).cuda()
    x = torch.randn(64, 20, device="cuda", requires_grad=True)
    y = m(x)
    assert y.shape == (64, 16, 3)
    y.backward(torch.ones_like(y))
    xn, thr, ord_, w = x.detach().cpu().numpy(), m.thresholds.detach().cpu().numpy(), m.ordinals.cpu().numpy(), m.weights.detach().cpu().numpy()
    assert np.array_equal(y.detach().cpu().numpy(), ho.forward(kind, xn, thr, ord_, w))
    gx, gthr, gw = ho.backward(kind, xn, thr, ord_, w, np.ones(y.shape, np.float32))
    ax, athr, aw = ho.backward_magnitudes(kind, xn, thr, ord_, w, np.ones(y.shape, np.float32))
    assert grad_close(x.grad, gx, ax) and grad_close(m.thresholds.grad, gthr, athr) and grad_close(m.weights.grad, gw, aw)
    assert m.ordinals.grad is None
    # deterministic mode selects the fixed-order backward: bit-exact against the oracle
    prev = torch.are_deterministic_algorithms_enabled()
    torch.use_deterministic_algorithms(True)
    try:
        for p in (x, m.thresholds, m.weights):
            p.grad = None
        m(x).backward(torch.ones_like(y))
    finally:
        torch.use_deterministic_algorithms(prev)
    assert np.array_equal(x.grad.cpu().numpy(), gx)
    assert np.array_equal(m.thresholds.grad.cpu().numpy(), gthr)
    assert np.array_equal(m.weights.grad.cpu().numpy(), gw)
    # analysis helpers
    leaf = m.leafmap(x.detach())
    assert leaf.shape == (64, 16) and m.reachability(x.detach()).sum() == 64 * 16
    assert m.pathmap(x.detach()).shape == (64, 16, 5)


def test_kernels_run_on_the_current_stream(ext):
    x, thr, ord_, w = random_forest_inputs(23, "tree", 512, 64, (), 32, 6, ())
    dx, dthr, dord, dw = dev(x, thr, ord_, w)
    ext.tree_forward(dx, dthr, dord, dw)  # validates the ordinals once
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        out = ext.tree_forward(dx, dthr, dord, dw)
    side.synchronize()
    assert np.array_equal(out.cpu().numpy(), ho.forward("tree", x, thr, ord_, w))


def test_training_step_is_cuda_graph_capturable():
    """Once an ordinals tensor has been validated no operator synchronises or reads back, so a whole
    forward + backward of a module can be captured in a CUDA graph and replayed on new data."""
    from hingetreefortorch_b200 import RandomHingeForest as R
    torch.manual_seed(3)
    m = R.RandomHingeForest(40, 12, 5, extra_outputs=2).cuda()
    x = torch.rand(64, 40, device="cuda", requires_grad=True)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(2):  # validates the ordinals, warms the allocator
            m(x).sum().backward()
    torch.cuda.current_stream().wait_stream(side)
    m.zero_grad(set_to_none=True)
    x.grad = None
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = m(x)
        y.sum().backward()
    with torch.no_grad():
        x.copy_(torch.rand(64, 40, device="cuda"))  # new data in the captured input
    graph.replay()
    torch.cuda.synchronize()
    got_y, got_gx, got_gw = y.clone(), x.grad.clone(), m.weights.grad.clone()
    m.zero_grad(set_to_none=True)
    x.grad = None
    want = m(x)
    want.sum().backward()
    assert torch.equal(got_y, want)
    assert torch.allclose(got_gx, x.grad, rtol=1e-5, atol=1e-6) and torch.allclose(got_gw, m.weights.grad, rtol=1e-5, atol=1e-6)


def test_backward_scratch_limit_switches_to_scatters(ext):
    """With the per-evaluation records ruled out the default-mode backward still matches within tolerance."""
    rng = np.random.default_rng(8)
    B, C, T, depth = 1200, 64, 40, 6
    x = rng.standard_normal((B, C)).astype(np.float32)
    thr = rng.uniform(-3, 3, (T, 63)).astype(np.float32)
    ord_ = rng.integers(0, C, (T, 63)).astype(np.int64)
    w = rng.standard_normal((T, 64)).astype(np.float32)
    g = rng.standard_normal((B, T)).astype(np.float32)
    dx, dthr, dord, dw, dg = [torch.from_numpy(a).cuda() for a in (x, thr, ord_, w, g)]
    with_records = ext.tree_backward(dx, True, dthr, True, dord, False, dw, True, dg)
    ext.set_backward_scratch_limit(0)
    try:
        scattered = ext.tree_backward(dx, True, dthr, True, dord, False, dw, True, dg)
    finally:
        ext.set_backward_scratch_limit(2 ** 62)
    want = ho.backward("tree", x, thr, ord_, w, g)
    mags = ho.backward_magnitudes("tree", x, thr, ord_, w, g)
    for got in (with_records, scattered):  # both paths against the oracle at the stated bar
        for t, ref, mag in zip((got[0], got[1], got[3]), want, mags):
            assert grad_close(t, ref, mag)
    with pytest.raises(ValueError):
        ext.set_backward_scratch_limit(-1)


# B, C, T, depth, outputs per leaf: one output with and without tile records, several
@pytest.mark.parametrize("shape", [(4096, 64, 32, 6, 1), (7000, 20, 4, 7, 1), (3000, 30, 20, 6, 3)], ids=str)
@pytest.mark.parametrize("room", ["all", "records", "none"])
def test_scratch_limit_in_fixed_order_mode(ext, shape, room):
    """The fixed-order mode stays within the limit, and its sums keep their order with any scratch: with the lists, with the
    default mode's records (one output per leaf) and with none."""
    from hingetreefortorch_b200.HingeTree import HingeTree
    B, C, T, depth, M = shape
    x, thr, ord_, w = random_forest_inputs(33, "tree", B, C, (), T, depth, (M,))
    g = np.random.default_rng(10).standard_normal((B, T, M)).astype(np.float32)
    ref = ho.backward("tree", x, thr, ord_, w, g)
    dx, dthr, dord, dw, dg = dev(x, thr, ord_, w, g)
    ext.tree_forward(dx, dthr, dord, dw)  # the ordinals' check takes memory of its own
    for t in (dx, dthr, dw):
        t.requires_grad_(True)
    parameters = 16 * thr.size + 8 * w.size + 65536  # packed ordinals, tree records
    limit = {"all": 2 ** 62, "records": 12 * B * T + parameters, "none": parameters}[room]
    results = x.nbytes + thr.nbytes + w.nbytes + g.nbytes + 65536
    torch.use_deterministic_algorithms(True)
    ext.set_backward_scratch_limit(limit)
    try:
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        before = requested_bytes()
        out = HingeTree.apply(dx, dthr, dord, dw)
        assert requested_bytes() - before <= g.nbytes + limit
        grads = torch.autograd.grad(out, (dx, dthr, dw), dg)
        peak = requested_bytes(peak=True) - before
    finally:
        ext.set_backward_scratch_limit(2 ** 62)
        torch.use_deterministic_algorithms(False)
    assert np.array_equal(out.detach().cpu().numpy(), ho.forward("tree", x, thr, ord_, w))
    for got, r in zip(grads, ref):
        assert np.array_equal(got.cpu().numpy(), r)
    assert peak <= results + limit if room != "all" else peak > results + 16 * B * T


def test_fixed_order_mode_without_memory_for_its_lists(ext):
    """An allocation that fails is like a limit: the step goes on without the lists."""
    B, C, T, depth, M = 40000, 20, 100, 4, 2
    x, thr, ord_, w = random_forest_inputs(34, "tree", B, C, (), T, depth, (M,))
    g = np.random.default_rng(11).standard_normal((B, T, M)).astype(np.float32)
    ref = ho.backward("tree", x, thr, ord_, w, g)
    dx, dthr, dord, dw, dg = dev(x, thr, ord_, w, g)
    ext.tree_forward(dx, dthr, dord, dw)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + 40 * 2 ** 20) / total)  # the lists take 88 MB
    try:
        grads = ext.tree_backward_deterministic(dx, True, dthr, True, dord, False, dw, True, dg)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    for got, r in zip((grads[0], grads[1], grads[3]), ref):
        assert np.array_equal(got.cpu().numpy(), r)


# B, C, T, depth, outputs per leaf: the forward keeps its paths in fixed-order mode only (too few evaluations; more than 64
# outputs), in both modes (several outputs; one), in neither
SWITCHED = [(100, 1000, 100, 7, 10), (700, 20, 50, 4, 70), (1100, 40, 31, 6, 3), (2048, 64, 32, 6, 1), (200, 16, 6, 3, 1)]


@pytest.mark.parametrize("shape", SWITCHED, ids=[str(s) for s in SWITCHED])
@pytest.mark.parametrize("forward_mode", [False, True], ids=["off_then_on", "on_then_off"])
def test_fixed_order_switched_between_forward_and_backward(shape, forward_mode):
    """torch.use_deterministic_algorithms changed between the two: the backward runs in the mode that is set when it runs."""
    from hingetreefortorch_b200.HingeTree import HingeTree
    B, C, T, depth, M = shape
    x, thr, ord_, w = random_forest_inputs(31, "tree", B, C, (), T, depth, (M,))
    g = np.random.default_rng(9).standard_normal((B, T, M)).astype(np.float32)
    ref, mags = ho.backward("tree", x, thr, ord_, w, g), ho.backward_magnitudes("tree", x, thr, ord_, w, g)
    dx, dthr, dord, dw, dg = dev(x, thr, ord_, w, g)
    for t in (dx, dthr, dw):
        t.requires_grad_(True)
    try:
        torch.use_deterministic_algorithms(forward_mode)
        out = HingeTree.apply(dx, dthr, dord, dw)
        torch.use_deterministic_algorithms(not forward_mode)
        grads = torch.autograd.grad(out, (dx, dthr, dw), dg)
    finally:
        torch.use_deterministic_algorithms(False)
    assert np.array_equal(out.detach().cpu().numpy(), ho.forward("tree", x, thr, ord_, w))
    for got, r, m in zip(grads, ref, mags):
        assert np.array_equal(got.cpu().numpy(), r) if not forward_mode else grad_close(got, r, m)


@pytest.mark.parametrize("call", ["tile", "several", "ordered", "linear", "conv"])
def test_second_backward_through_the_same_node(call):
    """retain_graph: the first backward uses up what the forward kept, the second walks the trees again."""
    from hingetreefortorch_b200 import HingeTree as F
    rng = np.random.default_rng(12)
    B, C, T, depth, M = 1030, 48, 32, 6, {"tile": 1, "several": 3, "ordered": 2}.get(call, 1)
    if call == "conv":
        x = rng.standard_normal((9, 4, 40, 41)).astype(np.float32)
        thr, w = rng.uniform(-1, 1, (20, 4, 31)).astype(np.float32), rng.standard_normal((20, 4, 32)).astype(np.float32)
        ord_ = rng.integers(0, 9, thr.shape).astype(np.int64)
        geometry = ((3, 3), (1, 1), (1, 1), (1, 1))
        g = rng.standard_normal((9, 20, 40, 41)).astype(np.float32)
        inputs, extra, function = (x, thr, ord_, w), [list(v) for v in geometry], F.HingeTreeConv2d
        ref, sizes = ho.conv_backward("tree", *inputs, g, *geometry), ho.magnitudes(ho.conv_backward, "tree", *inputs, g, *geometry)
    else:
        inputs = random_forest_inputs(35, "tree", B, C, (), T, depth, () if call == "linear" else (M,))
        if call == "linear":
            lin, bias, g = [rng.standard_normal(s).astype(np.float32) for s in ((5, T), 5, (B, 5))]
            inputs, extra, function = (*inputs, lin, bias), [], F.HingeTreeFusedLinear
            ref = ho.linear_backward("tree", *inputs[:5], g)
            sizes = ho.magnitudes(ho.linear_backward, "tree", *inputs[:5], g)
        else:
            g = rng.standard_normal((B, T, M)).astype(np.float32)
            extra, function = [], F.HingeTree
            ref, sizes = ho.backward("tree", *inputs, g), ho.backward_magnitudes("tree", *inputs, g)
    tensors = dev(*inputs)
    dg, = dev(g)
    wrt = [t.requires_grad_(True) for t in tensors if t.is_floating_point()]
    torch.use_deterministic_algorithms(call == "ordered")
    try:
        out = function.apply(*tensors, *extra)
        for again in (True, False):
            grads = torch.autograd.grad(out, wrt, dg, retain_graph=again)
            for got, r, s in zip(grads, ref, sizes):
                assert np.array_equal(got.cpu().numpy(), r) if call == "ordered" else grad_close(got, r, s)
    finally:
        torch.use_deterministic_algorithms(False)


def _small_modules():
    from hingetreefortorch_b200 import RandomHingeForest as R
    torch.manual_seed(5)
    tabular = torch.randn(12, 8, device="cuda")
    front = R.LinearBatchNorm1d(8, 4 * 7)
    return {
        "forest": (R.RandomHingeForest(8, 6, 3).cuda(), tabular),
        "linear": (R.RandomHingeFernFusedLinear(8, 6, 3, 4).cuda(), tabular),
        "conv": (R.HingeTreeConv1d(2, 3, 3, 3).cuda(), torch.randn(2, 2, 9, device="cuda")),
        "pipeline": (R.LinearBatchNormForest(front, R.RandomHingeForest(28, 4, 3, init_type="sequential")).cuda(), tabular),
    }


@pytest.mark.parametrize("name", ["forest", "linear", "conv", "pipeline"])
@pytest.mark.parametrize("grad", [True, False])
def test_forward_mode_and_vmap_are_refused(name, grad):
    """The operators have neither; a call that is not differentiated backward must not drop a tangent."""
    from torch.autograd import forward_ad
    m, x = _small_modules()[name]
    m(x)
    m.requires_grad_(False)
    with torch.set_grad_enabled(grad):
        with forward_ad.dual_level(), pytest.raises((RuntimeError, NotImplementedError), match="jvp"):
            m(forward_ad.make_dual(x, torch.ones_like(x)))
        with pytest.raises(RuntimeError):
            torch.func.vmap(m)(torch.stack([x, x + 1]))
        with pytest.raises(RuntimeError):
            torch.func.jvp(m, (x,), (x,))


@pytest.mark.parametrize("name", ["forest", "linear", "conv", "pipeline"])
@pytest.mark.parametrize("grad", [True, False])
def test_a_traced_module_computes_on_new_data(name, grad):
    """torch.jit.trace records the operators (as Python operations), not what they gave on the example."""
    m, x = _small_modules()[name]
    m(x)

    class Around(torch.nn.Module):
        def __init__(self):
            super().__init__()
            self.inner = m

        def forward(self, v):
            return 3 * self.inner(v + 1)

    net = Around()
    with torch.set_grad_enabled(grad):
        traced = torch.jit.trace(net, x, check_trace=False)
        eager = copy.deepcopy(net)
        y = torch.randn_like(x).requires_grad_(grad)
        got, want = traced(y), eager(y)
        assert torch.allclose(got, want, atol=1e-5) and not torch.allclose(got, eager(x), atol=1e-2)
    traced(x)
    for a, b in zip(net.state_dict().values(), eager.state_dict().values()):  # running statistics, too
        assert torch.allclose(a.double(), b.double(), atol=1e-6)
    if grad:
        g = torch.randn_like(want)
        grads = [torch.autograd.grad(out, [y] + [p for p in n.parameters() if p.requires_grad], g) for out, n in ((got, net), (want, eager))]
        for a, b in zip(*grads):
            assert torch.allclose(a, b, rtol=1e-4, atol=1e-4 * float(b.abs().max()) + 1e-6)


def test_scratch_of_no_saving_forward_is_refused(ext):
    x, thr, ord_, w = random_forest_inputs(32, "tree", 100, 30, (), 20, 5, (4,))
    dx, dthr, dord, dw = dev(x, thr, ord_, w)
    g = torch.ones(100, 20, 4, device="cuda")
    for scratch in (torch.empty(0, dtype=torch.uint8, device="cuda"), torch.empty(1 << 20, device="cuda"), torch.empty(1 << 20, dtype=torch.uint8)):
        with pytest.raises(ValueError, match="saving forward"):
            ext.tree_backward_saved(dx, True, dthr, True, dord, False, dw, True, g, scratch, False)


def test_speedtest_sweeps_like_the_reference(ext, capfd):
    """The reference's own benchmark operator: trees 1..512 by powers of two, depth 1..12, rows = trees, depth,
    forward ms, backward ms (hingetree.cpp:1361-1438)."""
    x = torch.rand(100, 1000, device="cuda")
    timings = ext.tree_speedtest(x, False)
    assert timings.shape == (4, 120) and timings.device.type == "cpu"
    assert timings[0].tolist() == [float(2 ** s) for s in range(10) for _ in range(12)]
    assert timings[1].tolist() == [float(d) for _ in range(10) for d in range(1, 13)]
    assert bool((timings[2:] > 0).all()) and float(timings[2:].max()) < 50.0
    assert "hingetree_forward: numBatches = 100" in capfd.readouterr().out


def test_a_wait_that_runs_out_reaches_the_caller(ext):
    """The error path of the tile kernels without a lost copy: the library's self-test kernel waits a few tries on
    a barrier nothing arrives on, sets HT_FLAG_PIPELINE_TIMEOUT and returns; the C ABI shows the flag in the
    caller's status word, the extension raises RuntimeError at its next status read and clears the word, and the
    device keeps working."""
    from hingetreefortorch_b200 import _cabi
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    _cabi.selftest_bounded_wait(status)
    assert int(status.item()) & _cabi.HT_FLAG_PIPELINE_TIMEOUT
    assert ext.pipeline_status() == 0
    ext.selftest_bounded_wait()
    with pytest.raises(RuntimeError, match="bounded wait"):
        ext.pipeline_status()
    assert ext.pipeline_status() == 0
    x, thr, ord_, w = random_forest_inputs(3, "tree", 16, 8, (), 4, 3, ())
    dx, dthr, dord, dw = dev(x, thr, ord_, w)
    assert np.array_equal(ext.tree_forward(dx, dthr, dord, dw).cpu().numpy(), ho.forward("tree", x, thr, ord_, w))
