"""NaN, infinities and huge values in the fused row kernels: the forward has them where the plain step formula has them, and
the other rows of a batch keep their values to the bit.  Rows of each family that takes fp32 tanh and sigmoid nets:
register-resident rows (n, N) of a power of two of blocks, ragged ones, one row per CTA, one group per thread."""
import pytest
import torch

from oracle import ncn_oracle as O

pytestmark = pytest.mark.gpu

ALPHA = 0.9
PLAIN = [(2, 1024), (4, 1024), (8, 1024), (4, 8192)]
RAGGED = [(2, 1044), (4, 3000), (8, 3008)]
ONE_GROUP = [(8, 1048), (16, 240), (16, 1840)]


def _close(got, want):
    """NaN and infinities where the oracle has them; the rest to 1e-5 of the larger of the value and 1 (the bound of the
    parity tests on values of order 1; large ones are rounded relative to themselves)."""
    got = got.float().cpu()
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    assert torch.equal(torch.isinf(got), torch.isinf(want))
    inf = torch.isinf(want)
    assert torch.equal(got[inf], want[inf])
    ok = torch.isfinite(want)
    assert ((got[ok] - want[ok]).abs() <= 1e-5 * want[ok].abs().clamp(min=1.0)).all()


def _inputs(B, N, L, seed):
    g = torch.Generator().manual_seed(seed)
    return torch.randn(B, N, 1, generator=g), torch.randn(B, N, 1, generator=g) * 0.3, torch.randn(L, 2, generator=g)


def _fwd(x, xa, W, n, act):
    import ncn_cuda_b200 as ncn

    with torch.no_grad():
        return ncn.fused_ncn_net(x.cuda(), xa.cuda(), W.cuda(), ALPHA, ncn.ops.ACTIVATION_CODES[act], n, 1)


@pytest.mark.parametrize("n,N,L", [(n, N, L) for n, N in PLAIN + ONE_GROUP for L in (1, 3)] + [(n, N, 3) for n, N in RAGGED])
@pytest.mark.parametrize("act", ["tanh", "sigmoid"])
def test_a_nan_goes_where_the_formula_takes_it(n, N, L, act):
    x, xa, W = _inputs(9, N, L, N + n)
    W *= n ** -0.5
    clean = _fwd(x, xa, W, n, act)
    x[1, 5 * n + n - 1] = float("nan")  # the last member of a group
    xa[2, 3 * n] = float("nan")         # a group's first member: it is x_j before the NaN reaches x
    xa[4, N - 1] = float("nan")
    x[6, 0] = xa[6, N // 2 + 1] = float("nan")
    got = _fwd(x, xa, W, n, act)
    for a, b, c in zip(got, O.net_forward(x, xa, W, ALPHA, act, n, 1), clean):
        _close(a, b)
        for row in (0, 3, 5, 7, 8):
            assert torch.equal(a[row], c[row])


@pytest.mark.parametrize("n,N,L", [(n, N, L) for n, N in PLAIN + ONE_GROUP for L in (1, 2)] + [(n, N, 2) for n, N in RAGGED])
@pytest.mark.parametrize("act", ["tanh", "sigmoid"])
@pytest.mark.parametrize("wi,wj", [(0.5, -0.25), (-0.5, 0.25), (0.5, 0.25), (-0.25, -0.5)])
def test_infinities_and_huge_values(n, N, L, act, wi, wj):
    """(Up to values whose squares are fp32 numbers: beyond, T = inf - inf is a matter of the order of its terms.)"""
    x, xa, _ = _inputs(9, N, L, 3 * N + n)
    W = torch.tensor([[wi, wj]]).repeat(L, 1)
    x[1, 0] = float("inf")
    x[2, 2 * n + 1] = float("-inf")
    xa[3, 4 * n] = float("inf")
    xa[5, N - 1] = float("-inf")
    x[6, n], x[6, 7 * n + n - 1] = 1e12, -3e15
    x[7, 1], xa[7, 2 * n] = 1e15, -1e14
    for a, b in zip(_fwd(x, xa, W, n, act), O.net_forward(x, xa, W, ALPHA, act, n, 1)):
        _close(a, b)


@pytest.mark.parametrize("n,N", PLAIN + RAGGED + ONE_GROUP)
@pytest.mark.parametrize("act", ["tanh", "sigmoid"])
@pytest.mark.parametrize("bad", [(1, 0, float("nan")), (0, 1, float("nan")), (1, 1, float("inf")), (0, 0, float("-inf")), (1, 0, 1e20)])
def test_weights(n, N, act, bad):
    x, xa, W = _inputs(5, N, 2, N)
    W[bad[0], bad[1]] = bad[2]
    for a, b in zip(_fwd(x, xa, W, n, act), O.net_forward(x, xa, W, ALPHA, act, n, 1)):
        _close(a, b)


@pytest.mark.parametrize("n,N,B,act", [(4, 1024, 9001, "tanh"), (8, 3008, 2500, "sigmoid"), (16, 240, 9001, "tanh")])
def test_rows_in_many_tiles_of_a_cta(n, N, B, act):
    x, xa, W = _inputs(B, N, 2, B)
    W *= n ** -0.5
    clean = _fwd(x, xa, W, n, act)
    bad = torch.arange(0, B, 61)
    x[bad, N - 3] = float("nan")
    got = _fwd(x, xa, W, n, act)
    ok = torch.ones(B, dtype=torch.bool)
    ok[bad] = False
    for a, b, c in zip(got, O.net_forward(x[bad], xa[bad], W, ALPHA, act, n, 1), clean):
        _close(a[bad.cuda()], b)
        assert torch.equal(a[ok.cuda()], c[ok.cuda()])


@pytest.mark.parametrize("n,N", [(4, 1024), (4, 3000), (16, 1840)])
def test_a_training_step_with_a_nan_row(n, N):
    """Rows are independent: the gradients of the other rows are those without it, the row's own group and dW are NaN."""
    import ncn_cuda_b200 as ncn

    x, xa, W = _inputs(7, N, 3, N)
    W *= n ** -0.5
    dy, dya, _ = _inputs(7, N, 3, N + 1)

    def step(x):
        leaves = [t.cuda().requires_grad_() for t in (x, xa, W)]
        y = ncn.fused_ncn_net(*leaves, ALPHA, 0, n, 1)
        return torch.autograd.grad(y, leaves, (dy.cuda(), dya.cuda()))

    clean = step(x)
    x[3, 2 * n + 1] = float("nan")
    got = step(x)
    for a, b in zip(got[:2], clean[:2]):
        for row in (0, 1, 2, 4, 5, 6):
            assert torch.equal(a[row], b[row])
    assert torch.isnan(got[0][3, 2 * n : 3 * n]).all() and torch.isnan(got[2]).all()
