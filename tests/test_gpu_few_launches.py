"""Nets whose kernels take the stages' weights one by one, and chains of stages whose weight gradients are summed by one
launch: the same numbers as through the calls these stand for."""
import pytest
import torch

pytestmark = pytest.mark.gpu

ALPHA = 0.9


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


# (2500, 64, 8, 8, 4): twenty stages fill the room for partial sums more than once; heads of 20: the shared-memory kernels
@pytest.mark.parametrize("B,N,heads,d,n,L", [(3, 96, 2, 32, 32, 1), (3, 96, 2, 32, 32, 3), (2500, 64, 8, 8, 4, 20), (2, 64, 2, 20, 16, 3)])
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
