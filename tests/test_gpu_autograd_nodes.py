"""The native autograd nodes: what autograd promises of any operator (one backward per graph, in-place checks, absent
cotangents, other weight types) and the weight gather at the edges of its launches."""
import pytest
import torch

from oracle import ncn_oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ncn():
    import ncn_cuda_b200 as m
    return m


def _case(kind, L, n=None):
    # fused: one feature per position; chain, ctx: several features, stage by stage
    B, N, E, C, n = (3, 64, 1, 1, n or 4) if kind == "fused" else (2, 64, 16, 2, n or 8)
    x, xa, ws, dy, dya = O.make_inputs(11, B, N, E, L, 0.2, dya_zero=False)
    net = (B, N, E, C, n)
    return net, x, xa, ws, dy, dya


def _run(ncn, case, train=True, wdtype=torch.float32):
    (B, N, E, C, n), x, xa, ws, dy, dya = case
    xd, xad = (t.cuda().requires_grad_(train) for t in (x, xa))
    wd = [w.cuda().to(wdtype).requires_grad_(train) for w in ws]
    net = ncn.NCNNetTestCuda(0.9, "tanh", n, C, len(ws), wd)
    return xd, xad, wd, net, dy.cuda(), dya.cuda()


@pytest.mark.parametrize("kind", ["fused", "chain"])
@pytest.mark.parametrize("L", [1, 3, 33])  # 33: one more than a gather launch takes
def test_against_oracle_and_without_gradients(ncn, kind, L):
    case = _case(kind, L)
    (B, N, E, C, n), x, xa, ws, dy, dya = case
    xd, xad, wd, net, dyd, dyad = _run(ncn, case)
    y, ya = net(xd, xad)
    got = [y, ya, *torch.autograd.grad((y, ya), (xd, xad, *wd), (dyd, dyad))]
    want = O.net_fwd_bwd(x, xa, ws, dy, dya, 0.9, "tanh", n, C)
    # both sides round in every one of the n * L steps that a value passes, each by a few units of 2^-24 at most: a sum that
    # grows at worst linearly in the steps, above 1e-5 from 42 steps on (the 132 steps of L = 33)
    tol = max(1e-5, 4 * n * L * 2.0 ** -24)
    for a, b in zip(got, [*want[:4], *want[4]]):
        assert O.rel_err(a.detach(), b) < tol
    with torch.no_grad():  # nothing stored, the same numbers
        y2, ya2 = net(xd, xad)
    assert not y2.requires_grad and torch.equal(y, y2) and torch.equal(ya, ya2)


@pytest.mark.parametrize("kind", ["fused", "chain"])
def test_autograd_semantics(ncn, kind):
    case = _case(kind, 3)
    xd, xad, wd, net, dyd, dyad = _run(ncn, case)
    ins = (xd, xad, *wd)
    y, ya = net(xd, xad)
    # a cotangent that never arrives is zero
    a = torch.autograd.grad(y, ins, dyd, retain_graph=True)
    b = torch.autograd.grad((y, ya), ins, (dyd, torch.zeros_like(dyad)))
    assert all(torch.equal(p, q) for p, q in zip(a, b))
    with pytest.raises(RuntimeError, match="second time"):
        torch.autograd.grad(y, ins, dyd)
    # the backward starts from the output: changing it in place is noticed
    y, ya = net(xd, xad)
    y.data_ptr()
    with torch.no_grad():
        y.mul_(2.0)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        torch.autograd.grad(y, ins, dyd)
    # expanded cotangents and non-contiguous inputs
    xt = xd.detach().transpose(0, 1).contiguous().transpose(0, 1).requires_grad_()
    y, ya = net(xt, xad)
    (y.sum() + ya.sum()).backward()
    ref = torch.autograd.grad(net(xd, xad), (xd,), (torch.ones_like(y), torch.ones_like(y)))[0]
    assert torch.equal(xt.grad, ref)


def test_bf16_weights_get_bf16_gradients(ncn):
    case = _case("fused", 3)
    xd, xad, wd, net, dyd, dyad = _run(ncn, case, wdtype=torch.bfloat16)
    y, ya = net(xd, xad)
    g = torch.autograd.grad((y, ya), wd, (dyd, dyad))
    net32 = ncn.NCNNetTestCuda(0.9, "tanh", 4, 1, 3, [w.detach().float().requires_grad_() for w in wd])
    y, ya = net32(xd, xad)
    g32 = torch.autograd.grad((y, ya), net32.weights, (dyd, dyad))
    assert all(p.dtype == torch.bfloat16 and torch.equal(p, q.to(torch.bfloat16)) for p, q in zip(g, g32))


def test_residual_stack_is_one_node_of_all_layers(ncn):
    """Layer by layer (fused_ncn_net on slices of the weight) gives the same numbers."""
    B, N, n, L, layers = 5, 1024, 4, 3, 3
    x, xa, _, dy, dya = (t if not torch.is_tensor(t) else t.cuda() for t in O.make_inputs(12, B, N, 1, L, 0.25, dya_zero=False))
    stack = ncn.NCNResidualStack(layers, 0.9, "tanh", n, 1, L, 1, w_std=0.5).cuda()
    for mode in ("tape", "recompute"):
        stack.backward_mode = mode
        xs, xas = x.clone().requires_grad_(), xa.clone().requires_grad_()
        one = torch.autograd.grad(stack(xs, xas), (xs, xas, stack.weight), (dy, dya))
        y, ya = xs, xas
        for k in range(layers):
            y, ya = ncn.fused_ncn_net(y, ya, stack.weight[k], 0.9, 0, n, 1, 0, mode, True)
        many = torch.autograd.grad((y, ya), (xs, xas, stack.weight), (dy, dya))
        assert all(torch.equal(p, q) for p, q in zip(one, many))


def _calls(ncn, kind, case):
    """The call under test on (x, xa, *ws), and the same through the Function's own forward and backward."""
    (B, N, E, C, n), *_ = case

    def general(f):
        return type("Subclass", (f,), {})

    ctx = torch.tensor([B, N - 3] + [N] * (B - 2), dtype=torch.int32)
    if kind == "fused":
        return (lambda x, xa, *ws: ncn.NCNNetTestCuda(0.9, "tanh", n, C, len(ws), ws)(x, xa),
                lambda x, xa, *ws: general(ncn.NCNNetFunction).apply(x, xa, torch.stack(ws), 0.9, 0, n, C, 0, "auto", False))
    if kind == "ctx":
        return (lambda x, xa, *ws: ncn.fused_ncn_cuda_ctxlen(x, xa, ws[0], ctx, 0.9, "tanh", n, C, 1),
                lambda x, xa, *ws: general(ncn.NCNContextFunction).apply(x, xa, ws[0], ctx, 0.9, 0, n, C, 1))

    def stages(x, xa, *ws):
        for l, w in enumerate(ws):
            x, xa = general(ncn.NCNFunction).apply(x, xa, w, 0.9, "tanh", n, C, l)
        return x, xa

    return lambda x, xa, *ws: ncn.NCNNetTestCuda(0.9, "tanh", n, C, len(ws), ws)(x, xa), stages


@pytest.mark.parametrize("kind,keep", [("fused", "auto"), ("chain", "output"), ("chain", "input"), ("chain", "mid"), ("ctx", "auto")])
def test_functions_have_a_forward_and_a_backward_of_their_own(ncn, kind, keep):
    """NCNFunction and its like are autograd Functions; what `apply` answers natively is what they compute."""
    case = _case(kind, 1 if kind == "ctx" else 3, n=32 if keep != "auto" else None)
    _, x, xa, ws, dy, dya = case
    prev = ncn.set_stage_backward(keep)
    try:
        out = []
        for call in _calls(ncn, kind, case):
            leaves = [t.cuda().requires_grad_() for t in (x, xa, *ws)]
            y, ya = call(*leaves)
            out.append([y, ya, *torch.autograd.grad((y, ya), leaves, (dy.cuda(), dya.cuda()))])
    finally:
        ncn.set_stage_backward(prev)
    assert all(torch.equal(p, q) for p, q in zip(*out))


@pytest.mark.parametrize("kind", ["fused", "chain", "ctx", "stack"])
def test_a_traced_module_computes(ncn, kind):
    """torch.jit.trace records the operators: the traced module gives other inputs' results, not the memory of the tracing."""
    case = _case("fused" if kind == "stack" else kind, 1 if kind == "ctx" else 3)
    _, x, xa, ws, dy, dya = case
    if kind == "stack":
        net = ncn.NCNResidualStack(2, 0.9, "tanh", 4, 1, 3, 1, w_std=0.5).cuda()
    else:
        class Net(torch.nn.Module):
            def __init__(self):
                super().__init__()
                self.ws = torch.nn.ParameterList(w.cuda() for w in ws)

            def forward(self, a, b):
                return _calls(ncn, kind, case)[0](a, b, *self.ws)

        net = Net()
    traced = torch.jit.trace(net, (x.cuda(), xa.cuda()))
    for p, q in zip(traced(dy.cuda(), dya.cuda()), net(dy.cuda(), dya.cuda())):
        assert torch.equal(p, q)


@pytest.mark.parametrize("kind", ["fused", "chain", "ctx", "stack"])
def test_transforms_are_refused(ncn, kind):
    """No forward-mode rule and no vmap rule: a dual tensor or a functorch transform is an error, never a lost tangent."""
    import torch.autograd.forward_ad as fwAD

    case = _case("fused" if kind == "stack" else kind, 1 if kind == "ctx" else 3)
    _, x, xa, ws, *_ = case
    args = [t.cuda() for t in (x, xa, *ws)]
    if kind == "stack":
        net = ncn.NCNResidualStack(2, 0.9, "tanh", 4, 1, 3, 1).cuda()
        args, call = args[:2], lambda a, b: net(a, b)
    else:
        call = _calls(ncn, kind, case)[0]
    for i in range(len(args)):  # every input and every weight
        with fwAD.dual_level(), pytest.raises(NotImplementedError, match="jvp"):
            call(*[fwAD.make_dual(t, torch.ones_like(t)) if i == k else t for k, t in enumerate(args)])
    first, rest = args[0], args[1:]
    for transformed in (lambda: torch.func.grad(lambda a: call(a, *rest)[0].sum())(first),
                        lambda: torch.func.vmap(lambda a: call(a, *rest))(torch.stack([first, first])),
                        lambda: torch.func.grad(lambda s: (s * call(*args)[0]).sum())(torch.ones((), device="cuda"))):
        with pytest.raises(RuntimeError, match="setup_context"):
            transformed()
    with torch.no_grad():  # with the level left, the same tensors are taken
        call(*args)


@pytest.mark.parametrize("n,keep", [(8, "auto"), (32, "auto"), (32, "input")])
def test_a_chain_is_walked_as_far_as_gradients_are_asked_for(ncn, n, keep):
    """Frozen stages before the first trainable one store nothing and have no backward; a gradient of late weights
    alone walks the late stages alone.  Counted by the tensors saved and unpacked."""
    case = _case("chain", 3, n)
    _, x, xa, ws, dy, dya = case
    call = _calls(ncn, "chain", case)[0]

    def run(trainable, wanted, x_grad=False):
        packed, unpacked = [], []
        xd = x.cuda().requires_grad_(x_grad)
        wd = [w.cuda().requires_grad_(t) for w, t in zip(ws, trainable)]
        with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t) or t, lambda t: unpacked.append(t) or t):
            y, ya = call(xd, xa.cuda(), *wd)
        ins = [wd[i] for i in wanted] + ([xd] if x_grad else [])
        return torch.autograd.grad((y, ya), ins, (dy.cuda(), dya.cuda())), len(packed), len(unpacked)

    prev = ncn.set_stage_backward(keep)
    try:
        full, saved, read = run([True] * 3, [0, 1, 2])
        late, _, read_late = run([True] * 3, [2])
        frozen, saved_one, read_one = run([False, False, True], [2])
        gap, saved_gap, read_gap = run([False, True, False], [1])
        through, _, read_all = run([False, False, False], [], x_grad=True)
    finally:
        ncn.set_stage_backward(prev)
    assert torch.equal(full[2], late[0]) and torch.equal(full[2], frozen[0]) and torch.equal(full[1], gap[0])
    extra = 2 if keep == "input" else 0  # the input of the first stage, beside each stage's own tensors
    assert saved_one - extra == (saved - extra) // 3 and saved_gap - extra == (saved - extra) * 2 // 3
    assert read_one == read_late == read // 3 and read_gap == read * 2 // 3 and read_all == read


@pytest.mark.parametrize("kind", ["chain", "stack"])
def test_the_walk_back_releases_what_it_has_used(ncn, kind):
    """The states of a stage (a layer) are freed behind it, so that the next one's results take their memory."""
    if kind == "chain":  # 32 steps: each stage keeps its output (2 tensors) and the state half way (2)
        B, N, E, C, n, L = 64, 256, 64, 2, 32, 4
        ws = [(torch.randn(2 * E, device="cuda") * 0.1).requires_grad_() for _ in range(L)]
        net = ncn.NCNNetTestCuda(0.9, "tanh", n, C, L, ws)
    else:  # each layer keeps two states of 2 tensors
        B, N, E, n, L = 4096, 1024, 1, 8, 4
        net = ncn.NCNResidualStack(L, 0.9, "tanh", n, 1, 3, E, w_std=0.2).cuda()
        ws = [net.weight]
    one = 4 * B * N * E
    x, xa, dy, dya = (torch.randn(B, N, E, device="cuda") * s for s in (1.0, 0.25, 1.0, 0.25))
    x.requires_grad_()

    def rise(**kw):
        y, ya = net(x, xa)
        base = torch.cuda.memory_allocated()
        torch.cuda.reset_peak_memory_stats()
        torch.autograd.grad((y, ya), [x, *ws], (dy, dya), **kw)
        return (torch.cuda.max_memory_allocated() - base) / one

    rise()
    # the results of two stages are alive at a time (4 tensors), and workspace of less than one; against that stands
    # what the first of the two had kept and nobody else holds
    assert rise() < 3.5 < 4 < rise(retain_graph=True)


def test_gradients_of_a_chain_have_memory_of_their_own(ncn):
    """Keeping (or saving) one stage's gradient keeps that one alone."""
    case = _case("chain", 3)
    xd, xad, wd, net, dyd, dyad = _run(ncn, case)
    grads = torch.autograd.grad(net(xd, xad), wd, (dyd, dyad))
    assert [g.untyped_storage().nbytes() for g in grads] == [4 * w.numel() for w in wd]


def test_errors_of_the_native_nodes(ncn):
    """Through the operators and modules: the library's status as NCNError, bad tensors by type."""
    (_, _, _, C, n), x, xa, ws, _, _ = _case("chain", 2)
    x, xa, ws = x.cuda(), xa.cuda(), [w.cuda() for w in ws]
    from ncn_cuda_b200._lib import NCNError

    for bad_n, bad_heads in ((7, C), (n, 3)):
        with pytest.raises(NCNError, match="bad shape"):
            ncn.fused_ncn_cuda_v2(x, xa, ws[0], 0.9, 0, bad_n, bad_heads, 0)
    with pytest.raises(NCNError, match="does not cover"):
        ncn.fused_ncn_net(x, xa, torch.stack(ws), 0.9, 0, n, C)
    with pytest.raises(ValueError, match="elements"):
        ncn.NCNNetTestCuda(0.9, "tanh", n, C, 2, [ws[0], ws[1][:3]])(x, xa)
    with pytest.raises(ValueError, match="agree"):
        ncn.fused_ncn_cuda_v2(x, xa[:1], ws[0], 0.9, 0, n, C, 0)
    with pytest.raises(ValueError, match="entries"):
        ncn.fused_ncn_cuda_ctxlen(x, xa, ws[0], torch.ones(3), 0.9, 0, n, C, 0)
    with pytest.raises(TypeError, match="float32 or bfloat16"):
        ncn.fused_ncn_cuda_v2(x.half(), xa.half(), ws[0], 0.9, 0, n, C, 0)
    with pytest.raises(RuntimeError, match="CUDA tensors only"):
        ncn.fused_ncn_cuda_v2(x.cpu(), xa.cpu(), ws[0], 0.9, 0, n, C, 0)
