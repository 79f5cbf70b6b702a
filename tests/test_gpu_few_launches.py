"""Nets whose kernels take the stages' weights one by one, and chains of stages whose weight gradients are summed by one
launch: the same numbers as through the calls these stand for."""
import pytest
import torch

pytestmark = pytest.mark.gpu

ALPHA = 0.9
NCN_ERR_WORKSPACE = 6


# up to 32 vectors travel with the kernel's parameters; rows of 16 * 15 and 4 * 129 positions run in other kernels
@pytest.mark.parametrize("n,N,L", [(2, 1024, 1), (2, 1024, 10), (8, 4096, 32), (8, 4096, 33), (16, 240, 3), (4, 516, 3), (16, 240, 33)])
def test_weights_one_by_one_are_the_gathered_ones(n, N, L):
    import ncn_cuda_b200 as ncn

    g = torch.Generator().manual_seed(N + L)
    x, xa, dy, dya = (torch.randn(5, N, 1, generator=g).cuda().requires_grad_(k < 2) for k in range(4))
    net = ncn.NCNNetCuda(ALPHA, "tanh", n, 1, L, 1).cuda()
    W = torch.stack([m.weight.detach() for m in net.ncn_modules]).requires_grad_()
    got = net(x, xa)
    want = ncn.fused_ncn_net(x, xa, W, ALPHA, 0, n, 1)
    for a, b in zip(got, want):
        assert torch.equal(a, b)
    ga = torch.autograd.grad(got, (x, xa, *net.parameters()), (dy, dya))
    gb = torch.autograd.grad(want, (x, xa, W), (dy, dya))
    for a, b in zip((ga[0], ga[1], torch.stack(ga[2:])), gb):
        assert torch.equal(a, b)


# (2500, 64, 8, 8, 4): twenty stages fill the room for partial sums more than once; (1, 32, 2, 8, 4): they are summed by one call, two
# launches of up to 16; heads of 20: the shared-memory kernels
@pytest.mark.parametrize("B,N,heads,d,n,L", [(3, 96, 2, 32, 32, 1), (3, 96, 2, 32, 32, 3), (2500, 64, 8, 8, 4, 20), (1, 32, 2, 8, 4, 20),
                                             (2, 64, 2, 20, 16, 3)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_weight_gradients_of_a_chain_are_those_of_its_stages(B, N, heads, d, n, L, dtype):
    import ncn_cuda_b200 as ncn

    E = heads * d
    g = torch.Generator().manual_seed(E + L)
    x, xa, dy, dya = (torch.randn(B, N, E, generator=g).cuda().to(dtype) for _ in range(4))
    net = ncn.NCNNetCuda(ALPHA, "tanh", n, heads, L, E).cuda()
    with torch.no_grad():
        for m in net.ncn_modules:
            m.weight.copy_(torch.randn(2 * E, generator=g) * d**-0.5)
    leaves = (x.requires_grad_(), xa.requires_grad_(), *net.parameters())
    got = torch.autograd.grad(net(x, xa), leaves, (dy, dya))
    a, b = x, xa
    for l, m in enumerate(net.ncn_modules):
        a, b = ncn.fused_ncn_cuda_v2(a, b, m.weight, ALPHA, 0, n, heads, l)  # a node, and a reduction, per stage
    want = torch.autograd.grad((a, b), leaves, (dy, dya))
    for p, q in zip(got, want):
        assert torch.equal(p, q)


def test_a_chain_takes_one_workspace():
    import ncn_cuda_b200 as ncn
    from ncn_cuda_b200 import _lib

    B, N, E, n, L = 1, 32, 1024, 4, 3
    x, xa = (torch.randn(B, N, E, device="cuda").requires_grad_() for _ in range(2))
    net = ncn.NCNNetCuda(ALPHA, "tanh", n, 32, L, E).cuda()
    y = net(x, xa)
    one = _lib.load().ncn_bwd_workspace_bytes(B, N, E, n, 32, 1, 0)
    before = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    torch.autograd.grad(y, (x, xa, *net.parameters()), (x.detach(), xa.detach()))
    # beside the workspace: a few gradients of 128 KB each
    assert torch.cuda.max_memory_allocated() - before < one + 32 * x.numel() * 4


@pytest.mark.parametrize("keep", ["output", "ctx"])
def test_partial_sums_want_room_for_their_rows(keep):
    """ncn_stage_bwd_partial: refused without a launch where its rows do not fit; where they just do, the sums of ncn_stage_bwd."""
    import ctypes

    from ncn_cuda_b200 import _lib, ops

    lib = _lib.load()
    B, N, E, n, heads = 6, 96, 64, 32, 2
    g = torch.Generator(device="cuda").manual_seed(3)
    y, ya, dy, dya = (torch.randn(B, N, E, generator=g, device="cuda") for _ in range(4))
    W = torch.randn(2 * E, generator=g, device="cuda") * 0.2
    cl = torch.full((B,), N, dtype=torch.int32, device="cuda")
    dx, dxa = torch.zeros_like(y), torch.zeros_like(y)
    ws = torch.zeros(lib.ncn_bwd_workspace_bytes(B, N, E, n, heads, 1, 0) // 4, device="cuda")
    rows = ctypes.c_int(0)

    def call(nbytes):
        return lib.ncn_stage_bwd_partial(
            0 if keep == "output" else 3, None, None, y.data_ptr(), ya.data_ptr(), None, 0, cl.data_ptr(), dy.data_ptr(), dya.data_ptr(),
            W.data_ptr(), dx.data_ptr(), dxa.data_ptr(), ws.data_ptr(), nbytes, ctypes.byref(rows), B, N, E, n, heads, 1, ALPHA, 0, 0,
            torch.cuda.current_stream().cuda_stream)

    assert call(ws.numel() * 4) == 0 and rows.value > 0
    need = rows.value * 2 * E * 4
    whole = ws[: rows.value * 2 * E].clone()
    ws.zero_()
    dx.zero_()
    assert call(need - 4) == NCN_ERR_WORKSPACE
    assert dx.abs().max() == 0 and ws.abs().max() == 0
    assert call(need) == 0 and torch.equal(ws[: rows.value * 2 * E], whole)
    dW = torch.empty(2 * E, device="cuda")
    arr = lambda t, v: (t * 1)(v)
    assert lib.ncn_reduce_partials(arr(ctypes.c_void_p, ws.data_ptr()), arr(ctypes.c_int, rows.value), arr(ctypes.c_void_p, dW.data_ptr()), 1,
                                   2 * E, torch.cuda.current_stream().cuda_stream) == 0
    want = (ops.stage_bwd(y, ya, dy, dya, W, ALPHA, 0, n, heads, 1) if keep == "output"
            else ops.stage_bwd_ctx(y, ya, dy, dya, W, cl, ALPHA, 0, n, heads, 1))
    assert torch.equal(dW, want[2] if keep == "output" else want[-1])
