"""The layers' native host path (``binding/cgnn_torch.cpp``) where it meets torch: tracing, saved tensors, gradients of
gradients, precision switches, streams, devices and graph capture."""
import numpy as np
import pytest
import torch

from compressgnn_b200 import runtime as rt


# ---------------------------------------------------------------------------------------------
# torch.jit.trace
# ---------------------------------------------------------------------------------------------
class _Scaled(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, factor):
        ctx.factor = factor
        out = torch.empty_like(x)
        out.numpy()[...] = x.numpy() * factor  # as a native operator: written past the dispatcher
        return out

    @staticmethod
    def backward(ctx, grad):
        return grad * ctx.factor, None


def _native_like(x, factor, _plan):
    return _Scaled.apply(x, factor)


@pytest.mark.filterwarnings("ignore")
def test_a_trace_calls_the_operator_again():
    for grad in (False, True):
        traced = torch.jit.trace(lambda x: rt.differentiable(_native_like, x, 3.0, None) + 1,
                                 (torch.randn(4, 5, requires_grad=grad),))
        x = torch.randn(4, 5, requires_grad=True)
        out = traced(x)
        torch.testing.assert_close(out, 3 * x + 1)
        upstream = torch.randn(4, 5)
        out.backward(upstream, retain_graph=True)
        torch.testing.assert_close(x.grad, 3 * upstream)
        out.backward(upstream)
        torch.testing.assert_close(x.grad, 6 * upstream)
        with pytest.raises(RuntimeError, match="second time"):
            out.backward(upstream)


class _Holding(torch.nn.Module):
    def __init__(self, layer, graph):
        super().__init__()
        self.layer, self.graph = layer, graph

    def forward(self, x):
        return self.layer(x, self.graph)


def _graph(width=8, n=600, **kw):
    from test_layers_gpu import make_data
    data = make_data(n=n, width=width, **kw)
    data.to("cuda")
    return data.edge_index


@pytest.mark.gpu
@pytest.mark.filterwarnings("ignore")
def test_traced_layers_replay():
    from compressgnn_b200.layer import Compressgnn_Reconstruct, Compressgnn_SPMM, _Mean
    from compressgnn_b200.model import GNNLayer
    graph = _graph()
    nodes = graph.vertex_cnt
    index = torch.randint(0, 7, (nodes,), device="cuda")
    counts = torch.bincount(index, minlength=7).int()
    spmm, reconstruct = Compressgnn_SPMM(), Compressgnn_Reconstruct()
    layer = GNNLayer(8, 5, 4, use_transformation=True, activation="relu", refresh_interval=5).cuda()
    layer.set_epoch(0)
    layer(torch.randn(nodes, 8, device="cuda"), graph)  # the assignment that is kept
    bias = torch.randn(8, device="cuda")
    for f in (lambda x: 2 * spmm(graph, x), lambda x: reconstruct(_Mean.apply(x, index, counts), index, bias, "relu"),
              _Holding(layer, graph)):
        x = torch.randn(nodes, 8, device="cuda", requires_grad=True)
        want = f(x)
        traced = torch.jit.trace(f, (torch.randn(nodes, 8, device="cuda", requires_grad=True),))
        torch.full((1 << 20,), float("nan"), device="cuda")  # what a fresh buffer would hold
        got = traced(x)
        assert torch.equal(got, want)
        upstream = torch.randn_like(want)
        assert torch.equal(torch.autograd.grad(got, x, upstream)[0], torch.autograd.grad(want, x, upstream)[0])


# ---------------------------------------------------------------------------------------------
# a layer's transformation
# ---------------------------------------------------------------------------------------------
@pytest.mark.gpu
@pytest.mark.filterwarnings("ignore:Initializing zero-element")
@pytest.mark.parametrize("nodes, activation", [(600, None), (600, "relu"), (0, "relu")])
def test_features_without_columns(nodes, activation):
    """[N, 0] features: the output is the bias, its gradient the column sums, the weight's gradient is empty."""
    layer = _layer(0, 5, activation)
    x = torch.randn(nodes, 0, device="cuda", requires_grad=True)
    out = layer(x, None)
    want = layer.lin.bias.detach().expand(nodes, 5)
    want = want.relu() if activation else want
    assert torch.equal(out, want)
    upstream = torch.randn(nodes, 5, device="cuda")
    out.backward(upstream)
    masked = upstream * (want > 0) if activation else upstream
    torch.testing.assert_close(layer.lin.bias.grad, masked.double().sum(0).float())
    assert layer.lin.weight.grad.shape == (5, 0) and x.grad.shape == (nodes, 0)


@pytest.mark.gpu
@pytest.mark.parametrize("switch", ["allow_tf32", "set_float32_matmul_precision", "matmul.fp32_precision", "fp32_precision",
                                    "ieee"])
def test_precision_switches(switch):
    """Each of torch's ways to allow TF32 products sends the weight gradient to the library, none makes it raise."""
    matmul = torch.backends.cuda.matmul
    layer = _layer(24, 12)
    x = torch.randn(600, 24, device="cuda")
    a, b = torch.randn(3000, 48, device="cuda"), torch.randn(3000, 65, device="cuda")
    layer(x, None).square().sum().backward()
    want, full = layer.lin.weight.grad.clone(), rt.ops().matmul_tn(a, b)
    layer.lin.weight.grad = None
    try:
        if switch == "allow_tf32":
            matmul.allow_tf32 = True
        elif switch == "set_float32_matmul_precision":
            torch.set_float32_matmul_precision("high")
        elif switch == "matmul.fp32_precision":
            matmul.fp32_precision = "tf32"
        elif switch == "fp32_precision":
            torch.backends.fp32_precision = "tf32"
        else:
            matmul.fp32_precision = "ieee"
        layer(x, None).square().sum().backward()
        assert torch.equal(rt.ops().matmul_tn(a, b), full if switch == "ieee" else a.t() @ b)
    finally:
        torch.backends.fp32_precision = matmul.fp32_precision = "none"
        torch.set_float32_matmul_precision("highest")
        matmul.fp32_precision = "none"
    assert not matmul.allow_tf32
    # three products of operands rounded to 11 bits, against sums of some hundred terms
    error = (layer.lin.weight.grad.double() - want.double()).norm() / want.double().norm()
    assert error <= 4 * 2.0 ** -11
    assert torch.equal(rt.ops().matmul_tn(a, b), full)


def _layer(width, out, activation=None):
    """A GNNLayer whose propagation is the identity."""
    from compressgnn_b200.model import GNNLayer
    layer = GNNLayer(width, out, 4, use_transformation=True, activation=activation).cuda()
    layer.P.forward = lambda x, **_: x
    return layer


# ---------------------------------------------------------------------------------------------
# gradients of gradients
# ---------------------------------------------------------------------------------------------
def _operators():
    """(function of one differentiable matrix, its shape) of every first-order operator."""
    from compressgnn_b200.layer import Compressgnn_Reconstruct, _Mean
    index = torch.randint(0, 7, (60,), device="cuda")
    counts = torch.bincount(index, minlength=7).int()
    rt.index_plan(index, 7)  # the reconstruction's plan is known, as it is inside a layer
    reconstruct, layer = Compressgnn_Reconstruct(), _layer(6, 4, "relu")
    return [(lambda x: _Mean.apply(x, index, counts), (60, 6)),
            (lambda x: reconstruct(x, index), (7, 6)),
            (lambda x: reconstruct(x, index, activation="relu"), (7, 6)),
            (lambda x: layer(x, None), (60, 6))]


@pytest.mark.gpu
@pytest.mark.parametrize("which", range(4))
def test_gradients_of_first_order_operators(which):
    """With create_graph: a gradient taken with a constant upstream gradient is a constant, one taken with a
    differentiable upstream gradient refuses to be differentiated."""
    f, shape = _operators()[which]
    x = torch.randn(shape, device="cuda", requires_grad=True)
    w = torch.randn(shape, device="cuda", requires_grad=True)
    out = f(x)
    (plain,) = torch.autograd.grad(out, x, torch.ones_like(out), retain_graph=True)
    (grad,) = torch.autograd.grad(out, x, torch.ones_like(out), create_graph=True)
    assert torch.equal(grad, plain) and not grad.requires_grad
    (grad * w).sum().backward()
    assert torch.equal(w.grad, grad)
    upstream = torch.ones_like(out, requires_grad=True)
    (grad,) = torch.autograd.grad(f(x), x, upstream, create_graph=True)
    assert torch.equal(grad, plain)
    with pytest.raises(RuntimeError, match="once_differentiable"):
        grad.sum().backward()


@pytest.mark.gpu
@pytest.mark.parametrize("which", range(4))
def test_a_second_backward_needs_the_graph_retained(which):
    f, shape = _operators()[which]
    out = f(torch.randn(shape, device="cuda", requires_grad=True))
    out.sum().backward(retain_graph=True)
    out.sum().backward()
    with pytest.raises(RuntimeError, match="second time"):
        out.sum().backward()


@pytest.mark.gpu
def test_saved_tensors_modified_in_place():
    """Whatever a node saved, a change between forward and backward is refused, also of what this backward can do
    without."""
    from compressgnn_b200.layer import Compressgnn_Reconstruct, _Mean
    index = torch.randint(0, 7, (60,), device="cuda")
    counts = torch.bincount(index, minlength=7).int()
    rt.index_plan(index, 7)
    x = torch.randn(60, 6, device="cuda")
    reps = torch.randn(7, 6, device="cuda")
    for f, changed in ((lambda: _Mean.apply(x.clone().requires_grad_(), index, counts), counts),
                       (lambda: Compressgnn_Reconstruct()(reps.clone().requires_grad_(), index), index)):
        out = f()
        changed += 0
        with pytest.raises(RuntimeError, match="inplace"):
            out.sum().backward()
    for activation in (None, "relu"):
        layer = _layer(6, 4, activation)
        out = layer(x, None)  # takes no gradient itself: the weight is saved, and not needed
        with torch.no_grad():
            layer.lin.weight += 0
        with pytest.raises(RuntimeError, match="inplace"):
            out.sum().backward()
        out = layer(x, None)
        layer.cluster.vertex_index += 0
        with pytest.raises(RuntimeError, match="inplace"):
            out.sum().backward()


class _NoGradient(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x):
        return x.clone()

    @staticmethod
    def backward(ctx, grad):
        return None


@pytest.mark.gpu
def test_no_gradient_from_the_consumer_is_a_zero_gradient():
    from compressgnn_b200.layer import Compressgnn_SPMM
    graph, spmm = _graph(), Compressgnn_SPMM()
    for f, shape in _operators() + [(lambda x: spmm(graph, x), (graph.vertex_cnt, 8))]:
        x = torch.randn(shape, device="cuda", requires_grad=True)
        _NoGradient.apply(f(x)).sum().backward()
        assert x.grad is not None and x.grad.shape == shape and not x.grad.any()


# ---------------------------------------------------------------------------------------------
# the propagation's launch tables
# ---------------------------------------------------------------------------------------------
def _tables(plan, graph):
    """The launches of ``graph`` as the native propagation takes them: (forward, backward)."""
    forward = [(plan.r2v.native, [graph.r2v_graph.value])] + \
        [(p.native, [b.value]) for p, b in zip(plan.levels, graph.r2r_graph)] + \
        [(plan.out.native, [graph.v2r_graph.value, graph.v2v_graph.value])]
    backward = [(plan.v2r_t.native, [graph.v2r_graph.csc()[2]])] + \
        [(p.native, [b.csc()[2]]) for p, b in reversed(list(zip(plan.levels_t, graph.r2r_graph)))] + \
        [(plan.out_t.native, [graph.v2v_graph.csc()[2], graph.r2v_graph.csc()[2]])]
    return forward, backward


@pytest.mark.gpu
def test_a_failed_first_pass_can_be_repeated():
    """A value array that does not match its plan fails each call, not only the first."""
    graph = _graph()
    plan = graph.propagation_plan()
    forward, backward = _tables(plan, graph)
    forward[-1] = (forward[-1][0], [forward[-1][1][0], forward[-1][1][1][:-1].contiguous()])
    native = rt.ops().Propagation(graph.vertex_cnt, graph.rule_cnt, forward, backward)
    x = torch.randn(graph.vertex_cnt, 8, device="cuda")
    for _ in range(3):
        with pytest.raises(RuntimeError, match="values do not match"):
            native.run(x, False)
    assert torch.equal(native.run(x, True), plan.native.run(x, True))


@pytest.mark.gpu
def test_first_passes_on_two_streams():
    """The value arrays are shared: a pass on a second stream right after the first one, on a busy stream, reads them
    complete."""
    x = torch.randn(3000, 40, device="cuda")
    busy = torch.randn(2048, 2048, device="cuda")
    graph = _graph(n=3000)
    plan = graph.propagation_plan()
    want = plan.native.run(x, False), plan.native.run(x, True)
    for _ in range(3):
        native = rt.ops().Propagation(graph.vertex_cnt, graph.rule_cnt, *_tables(plan, graph))
        first, second = torch.cuda.Stream(), torch.cuda.Stream()
        torch.cuda.synchronize()
        got = []
        for stream in (first, second):
            with torch.cuda.stream(stream):
                if stream is first:
                    for _ in range(40):
                        busy @ busy
                got.append([native.run(x, backward) for backward in (False, True)])
        torch.cuda.synchronize()
        for pair in got:
            assert torch.equal(pair[0], want[0]) and torch.equal(pair[1], want[1])


@pytest.mark.gpu
def test_first_pass_inside_a_capture():
    """A first pass of a value type and width while a graph is captured: what the graph object keeps of it (values in
    plan order, scratch) is complete without a replay."""
    graph = _graph(n=3000)
    plan = graph.propagation_plan()
    x = torch.randn(3000, 40, device="cuda", dtype=torch.float64)
    want = [plan.native.run(x, backward) for backward in (False, True)]
    side = torch.cuda.Stream()
    for replays in (0, 2):
        graph._plan = None
        plan = graph.propagation_plan()
        native = plan.native
        assert any(p.long_rows for p in [plan.out, plan.out_t])  # scratch is used
        torch.cuda.synchronize()
        recorded, again = torch.cuda.CUDAGraph(), torch.cuda.CUDAGraph()
        with torch.cuda.graph(recorded, stream=side):
            outs = [native.run(x, backward) for backward in (False, True)]
        with torch.cuda.stream(side):
            for backward in (False, True):
                assert torch.equal(native.run(x, backward), want[backward])
        torch.cuda.synchronize()
        with torch.cuda.graph(again, stream=side):
            outs_again = [native.run(x, backward) for backward in (False, True)]
        for _ in range(replays):
            for graph_of, results in ((again, outs_again), (recorded, outs)):
                for out in results:
                    out.zero_()
                graph_of.replay()
                assert all(torch.equal(a, b) for a, b in zip(results, want))
        del recorded, again, outs, outs_again


@pytest.mark.gpu
def test_values_of_a_plan_are_ordered_per_stream():
    """``spmm_func`` with values a busy stream has yet to bring into plan order, at once on a second stream, inside a
    capture, and after a capture that was never replayed."""
    rng = np.random.default_rng(0)
    rows = rng.integers(0, 9, 2000)
    vlist = torch.from_numpy(np.concatenate([[0], np.cumsum(rows)])).cuda()
    elist = torch.from_numpy(rng.integers(0, 2000, rows.sum())).cuda()
    mat = torch.randn(2000, 24, device="cuda")
    busy = torch.randn(2048, 2048, device="cuda")

    def product(value):
        return rt.spmm_func(vlist, elist, value, mat, "rowbalance_rowcache", None)

    for _ in range(3):
        value = torch.randn(elist.numel(), device="cuda")
        want = product(value.clone())
        first, second, third = (torch.cuda.Stream() for _ in range(3))
        torch.cuda.synchronize()
        recorded = torch.cuda.CUDAGraph()
        with torch.cuda.graph(recorded, stream=third):
            inside = product(value)
        with torch.cuda.stream(first):
            for _ in range(40):
                busy @ busy
            got = [product(value)]
        with torch.cuda.stream(second):
            got.append(product(value))
        with torch.cuda.stream(third):
            got.append(product(value))
        torch.cuda.synchronize()
        assert all(torch.equal(g, want) for g in got)
        again = torch.cuda.CUDAGraph()
        with torch.cuda.graph(again, stream=third):
            twice = product(value)
        inside.zero_(), twice.zero_()
        again.replay(), recorded.replay()
        assert torch.equal(inside, want) and torch.equal(twice, want)
        del recorded, again


@pytest.mark.gpu
def test_operands_of_a_pass_are_checked_on_the_host():
    """A matrix on another device, or one that is no dense matrix, is refused before anything is launched.  (Plans said
    to lie on a second GPU stand in for a graph there.)"""
    import ctypes
    from compressgnn_b200.layer import spmm

    def plan_on(device):
        handle, rowptr = ctypes.c_void_p(0), torch.zeros(5, dtype=torch.int64, device="cuda")
        rt.check(rt.lib().cgnn_plan_create(ctypes.byref(handle), 4, 8, rowptr.data_ptr(), None, 0, None, None, 0, 0,
                                           torch.cuda.current_stream().cuda_stream))
        return rt.ops().Plan(handle.value, device), [torch.empty(0, device="cuda")]

    graph = _graph()
    x = torch.randn(graph.vertex_cnt, 8, device="cuda")
    want = spmm._forward(graph, x)
    wide = torch.empty(graph.rule_cnt, 16, device="cuda")
    for bad in (torch.empty(graph.rule_cnt, 8), wide[:, :8], wide[:, ::2], torch.empty(8, graph.rule_cnt, device="cuda").t()):
        with pytest.raises(RuntimeError, match="rule buffer does not match"):
            spmm._forward(graph, x, rule_out=bad)
        for detail in (dict(record=[]), dict(per_block=True)):
            with pytest.raises(RuntimeError, match="rule buffer does not match"):
                spmm._forward(graph, x, rule_out=bad, **detail)
    for bad in (torch.empty(graph.vertex_cnt, 8), torch.empty(8, graph.vertex_cnt, device="cuda").t()):
        with pytest.raises(RuntimeError, match="out does not match"):
            spmm._forward(graph, x, out=bad)
        with pytest.raises(RuntimeError, match="contiguous matrices on the plan's device"):
            spmm._forward(graph, x, out=bad, per_block=True)
    elsewhere = rt.ops().Propagation(graph.vertex_cnt, 4, [plan_on(1), plan_on(1)], [plan_on(1), plan_on(1)])
    for call in (elsewhere.run, elsewhere.apply):
        with pytest.raises(RuntimeError, match="on cuda:0 and the graph on cuda:1"):
            call(x, False)
    with pytest.raises(RuntimeError, match="one device"):
        rt.ops().Propagation(graph.vertex_cnt, 4, [plan_on(0), plan_on(0)], [plan_on(0), plan_on(1)])
    assert torch.equal(spmm._forward(graph, x), want)


@pytest.mark.gpu
def test_fake_tensors_leave_nothing_behind():
    """A pass under a fake tensor mode is refused, and what it asked for is not kept for real ones."""
    from torch._subclasses.fake_tensor import FakeTensorMode
    graph = _graph(n=3000)
    native = graph.propagation_plan().native
    x = torch.randn(3000, 40, device="cuda")
    native.run(torch.randn(3000, 8, device="cuda"), False)  # the value arrays are known, the scratch of 40 columns is not
    with FakeTensorMode(allow_non_fake_inputs=True):
        with pytest.raises(RuntimeError):
            native.run(x, False)
        with pytest.raises(RuntimeError):
            native.run(torch.empty(3000, 40, device="cuda"), False)
    per_launch = torch.empty_like(x)
    rule = rt.empty_row_aligned(graph.rule_cnt, x)
    for i in range(graph.propagation_plan().launches):
        native.run(x, False, per_launch, rule, i, i)
    assert torch.equal(native.run(x, False), per_launch)
    from conftest import assert_close_rel
    from oracle import oracle
    from test_layers_gpu import oracle_blocks
    assert_close_rel(per_launch.cpu().numpy(), oracle.propagate_forward(oracle_blocks(graph), x.cpu().numpy()))
