"""Register-tiled kernels for several features per position: every team size (warps per group), rows of 6 features per
lane, several small groups per warp, ragged group counts, context lengths and leaky-relu, against the fp64 oracle."""
import pytest
import torch

from oracle import ncn_oracle as O

from .kernels_util import kernels_of, launched

pytestmark = pytest.mark.gpu

ALPHA = 0.9
# (B, N, heads, d, n): teams of 4, 2 and 1 warps (small to larger batches of the same shape), eight rows per group, groups
# side by side in a warp with a last warp that is partly empty, heads of 24 and 48 features
SHAPES = [
    (3, 256, 4, 32, 32),
    (12, 256, 4, 32, 32),
    (160, 96, 4, 32, 32),
    (2, 96, 2, 64, 32),
    (40, 96, 8, 48, 32),
    (5, 80, 1, 128, 16),
    (5, 96, 2, 24, 32),
    (5, 72, 2, 24, 8),
    (5, 60, 3, 8, 4),
    (5, 10, 2, 2, 2),
    (300, 48, 5, 4, 16),
]


def _case(B, N, heads, d, seed=0):
    g = torch.Generator().manual_seed(seed)
    E = heads * d

    def r(s):
        return torch.randn(B, N, E, generator=g) * s

    return r(1.0), r(0.25), torch.randn(2 * E, generator=g) * d**-0.5, r(1.0), r(0.25)


def _oracle(fn, x, xa, W, dy, dya):
    leaves = [t.double().requires_grad_(True) for t in (x, xa, W)]
    y, ya = fn(*leaves)
    return [y.detach(), ya.detach(), *torch.autograd.grad((y, ya), leaves, (dy.double(), dya.double()))]


def _check(got, want, tol):
    for name, a, b in zip(("y", "ya", "dx", "dxa", "dW"), got, want):
        err = (a.double().cpu() - b).abs().max() / b.abs().max()
        assert err <= tol, f"{name}: {err:.2e} > {tol:.0e}"


@pytest.mark.parametrize("activation", ["tanh", "linear"])
@pytest.mark.parametrize("B,N,heads,d,n", SHAPES)
def test_stage(B, N, heads, d, n, activation):
    import ncn_cuda_b200 as ncn

    x, xa, W, dy, dya = _case(B, N, heads, d)
    want = _oracle(lambda a, b, w: O.stage_forward(a, b, w, ALPHA, activation, n, heads, 2), x, xa, W, dy, dya)
    leaves = [t.cuda().requires_grad_(True) for t in (x, xa, W)]
    y, ya = ncn.fused_ncn_cuda_v2(*leaves, ALPHA, ncn.ops.ACTIVATION_CODES[activation], n, heads, 2)
    grads = torch.autograd.grad((y, ya), leaves, (dy.cuda(), dya.cuda()))
    _check((y, ya, *grads), want, 1e-5)  # no inverse chain is longer than 16 steps


# One warp per group with four, two and one rows per lane, teams of two warps with two rows, heads of 24 and 48, several
# groups per warp: what a call keeps for its backward chooses among the kernels of each.
@pytest.mark.parametrize("keep", ["auto", "input", "mid"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("B,N,heads,d,n", [(160, 96, 4, 32, 32), (12, 256, 4, 32, 32), (160, 96, 4, 16, 32), (40, 96, 8, 48, 32),
                                           (5, 96, 2, 24, 32), (5, 72, 2, 24, 8), (160, 48, 4, 64, 16), (160, 96, 4, 8, 32),
                                           (160, 48, 4, 16, 16), (300, 48, 5, 4, 16), (40, 72, 4, 8, 8), (40, 60, 4, 16, 4)])
def test_kernels_of_a_call(B, N, heads, d, n, dtype, keep):
    import ncn_cuda_b200 as ncn

    x, xa, W, dy, dya = _case(B, N, heads, d, seed=6)
    x, xa, dy, dya = (t.to(dtype) for t in (x, xa, dy, dya))
    want = _oracle(lambda a, b, w: O.stage_forward(a, b, w, ALPHA, "tanh", n, heads, 1), x, xa, W, dy, dya)
    prev = ncn.set_stage_backward(keep)
    try:
        leaves = [t.cuda().requires_grad_(True) for t in (x, xa, W)]
        y, ya = ncn.fused_ncn_cuda_v2(*leaves, ALPHA, 0, n, heads, 1)
        got = (y, ya, *torch.autograd.grad((y, ya), leaves, (dy.cuda(), dya.cuda())))
    finally:
        ncn.set_stage_backward(prev)
    if keep != "mid" or n >= 16:  # (the states of shorter groups are stored by the shared-memory kernels, with the exact tanh)
        with torch.no_grad():  # stored states change no result
            assert torch.equal(y, ncn.fused_ncn_cuda_v2(*leaves, ALPHA, 0, n, heads, 1)[0])
    # bf16: results rounded to 2^-9; the weight gradient sums terms that carry the rounding and largely cancel
    _check(got[:4], want[:4], 1e-5 if dtype == torch.float32 else 2e-2)
    _check([got[4]], [want[4]], 1e-5 if dtype == torch.float32 else 3e-2)


@pytest.mark.parametrize("B,N,heads,d,n", SHAPES)
def test_context_lengths(B, N, heads, d, n):
    import ncn_cuda_b200 as ncn

    x, xa, W, dy, dya = _case(B, N, heads, d, seed=1)
    ctx = torch.randint(0, N + 3, (B,), generator=torch.Generator().manual_seed(2), dtype=torch.int32)
    ctx[0] = 0
    ctx[-1] = N
    want = _oracle(lambda a, b, w: O.stage_forward_ctxlen(a, b, w, ctx, ALPHA, "tanh", n, heads, 1), x, xa, W, dy, dya)
    leaves = [t.cuda().requires_grad_(True) for t in (x, xa, W)]
    y, ya = ncn.fused_ncn_cuda_ctxlen(*leaves, ctx.cuda(), ALPHA, 0, n, heads, 1)
    grads = torch.autograd.grad((y, ya), leaves, (dy.cuda(), dya.cuda()))
    # the walk back from the output: rounding grows by 1 / 0.9 per step, 29-fold over 32 steps
    _check((y, ya, *grads), want, 1e-5 if n <= 16 else 3e-5)


@pytest.mark.parametrize("activation", ["tanh", "linear", "relu", "sigmoid", "leaky-relu"])
@pytest.mark.parametrize("B,N,heads,d,n", [(160, 96, 4, 32, 32), (320, 80, 1, 64, 16), (700, 32, 2, 32, 16)])
def test_context_lengths_dealt_out_evenly(B, N, heads, d, n, activation):
    """More than eight groups per SM: kernels of their own (the last template argument), in every activation."""
    import ncn_cuda_b200 as ncn

    x, xa, W, dy, dya = _case(B, N, heads, d, seed=4)
    ctx = torch.randint(0, N + 3, (B,), generator=torch.Generator().manual_seed(5), dtype=torch.int32)
    want = _oracle(lambda a, b, w: O.stage_forward_ctxlen(a, b, w, ctx, ALPHA, activation, n, heads, 1), x, xa, W, dy, dya)
    leaves = [t.cuda().requires_grad_(True) for t in (x, xa, W)]

    def step():
        y, ya = ncn.fused_ncn_cuda_ctxlen(*leaves, ctx.cuda(), ALPHA, ncn.ops.ACTIVATION_CODES[activation], n, heads, 1)
        return (y, ya, *torch.autograd.grad((y, ya), leaves, (dy.cuda(), dya.cuda())))

    got, names = kernels_of(step)
    assert launched(names, r"feat_fwd_kernel<.*5>") and launched(names, r"feat_bwd_kernel<.*5>"), names
    _check(got[:2], want[:2], 1e-5)
    if "relu" in activation:
        # the derivative jumps at 0: a pre-activation of order 1 carries 1e-7 of rounding, 1 / 0.9^n times that at the end of a walk back, so a
        # share of `flips` of them (0.4: the density at 0) has the other sign; each changes its element's gradient by up to a tenth
        # and a term of dW, (1 - alpha) c x_j x_i gT, by up to 1e-2
        flips = 2 * 0.4 * 1e-7 / 0.9**n
        for a, b in zip(got[2:4], want[2:4]):
            assert (a.double().cpu() - b).norm() / b.norm() < 1e-5 + 0.1 * (n * flips) ** 0.5
        assert (got[4].double().cpu() - want[4]).norm() < 1e-5 * want[4].norm() + 1e-2 * (x.numel() * n * flips) ** 0.5
    else:
        _check(got[2:], want[2:], 1e-5 if n <= 16 else 3e-5)


@pytest.mark.parametrize("n,d", [(4, 8), (16, 24)])
def test_padding_is_not_read_into_the_results(n, d):
    """Groups beyond a row's length take no step: what stands there (NaN, as in memory never written) stays there."""
    import ncn_cuda_b200 as ncn

    B, N, heads = 3, 8 * n, 2
    x, xa, W, dy, dya = _case(B, N, heads, d, seed=3)
    ctx = torch.tensor([n, 3 * n, 8 * n], dtype=torch.int32)
    w = W.cuda().requires_grad_(True)
    out = []
    for fill in (0.0, float("nan")):
        a, b = x.clone(), xa.clone()
        for i in range(B):
            a[i, ctx[i] :] = fill
            b[i, ctx[i] :] = fill
        a, b = a.cuda().requires_grad_(True), b.cuda().requires_grad_(True)
        y, ya = ncn.fused_ncn_cuda_ctxlen(a, b, w, ctx.cuda(), ALPHA, 0, n, heads, 0)
        gx, gxa, gw = torch.autograd.grad((y, ya), (a, b, w), (dy.cuda(), dya.cuda()))
        out.append((y, gx, gxa, gw))
    for i in range(B):
        for p, q in zip(out[0][:3], out[1][:3]):
            assert torch.equal(p[i, : ctx[i]], q[i, : ctx[i]])
    assert torch.equal(out[0][3], out[1][3])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n,d", [(8, 16), (16, 32)])
def test_leaky_relu(n, d, dtype):
    from ncn_cuda_b200 import ops

    B, N, heads = 4, 6 * n, 2
    x, xa, W, _, _ = _case(B, N, heads, d, seed=4)
    x, xa = x.to(dtype), xa.to(dtype)
    y, ya = ops.stage_fwd(x.cuda(), xa.cuda(), W.cuda(), ALPHA, 3, n, heads, 1)
    Y, YA = O.stage_forward(x.double(), xa.double(), W.double(), ALPHA, "leaky-relu", n, heads, 1)
    _check((y, ya), (Y, YA), 1e-5 if dtype == torch.float32 else 2e-2)


@pytest.mark.parametrize("activation", ["tanh", "sigmoid"])
@pytest.mark.parametrize("B,N,heads,d,n,ctx", [(2, 96, 2, 32, 32, False), (600, 96, 2, 32, 32, False), (2, 96, 2, 24, 32, False),
                                               (2, 96, 2, 48, 16, False), (2, 96, 2, 64, 32, False), (2, 64, 2, 32, 8, False),
                                               (2, 128, 2, 32, 32, True), (2, 64, 2, 8, 4, True), (2, 64, 2, 2, 2, False)])
def test_nan_goes_where_the_arithmetic_takes_it(B, N, heads, d, n, ctx, activation):
    """A NaN in a token reaches its whole group (head by head) and nothing else; one in the second stream of the group's
    first token, which is x_j before it is touched, stays with that token."""
    import ncn_cuda_b200 as ncn

    act = ncn.ops.ACTIVATION_CODES[activation]
    x, xa, W, dy, dya = _case(B, N, heads, d, seed=5)
    x[0, n + 1, 3 % d] = float("nan")
    xa[1, 2 * n, (5 % d) + d] = float("nan")
    # (the groups that hold a NaN are complete: the oracle selects between a step and none, and 0 * NaN is NaN there)
    cl = torch.full((B,), 3 * n + 1, dtype=torch.int32)

    def oracle(a, b, w):
        if ctx:
            return O.stage_forward_ctxlen(a, b, w, cl, ALPHA, activation, n, heads, 0)
        return O.stage_forward(a, b, w, ALPHA, activation, n, heads, 0)

    want = _oracle(oracle, x, xa, W, dy, dya)
    leaves = [t.cuda().requires_grad_(True) for t in (x, xa, W)]
    if ctx:
        y, ya = ncn.fused_ncn_cuda_ctxlen(*leaves, cl.cuda(), ALPHA, act, n, heads, 0)
    else:
        y, ya = ncn.fused_ncn_cuda_v2(*leaves, ALPHA, act, n, heads, 0)
    got = (y, ya, *torch.autograd.grad((y, ya), leaves, (dy.cuda(), dya.cuda())))
    for name, p, q in zip(("y", "ya", "dx", "dxa", "dW"), got, want):
        assert torch.equal(p.isnan().cpu(), q.isnan()), name


@pytest.mark.parametrize("n,heads,d", [(8, 2, 24), (8, 1, 1), (24, 2, 5), (20, 1, 16), (32, 1, 40)])
def test_stored_end_state_of_any_number_of_steps(n, heads, d):
    """bf16 storage with stored states: the backward starts from the fp32 state after the last step, also where the
    number of steps is no multiple of 16."""
    from ncn_cuda_b200 import ops

    B, N = 6, 3 * n
    x, xa, W, dy, dya = _case(B, N, heads, d, seed=7)
    x, xa, dy, dya = (t.bfloat16() for t in (x, xa, dy, dya))
    want = _oracle(lambda a, b, w: O.stage_forward(a, b, w, ALPHA, "tanh", n, heads, 1), x, xa, W, dy, dya)
    y, ya, mid = ops.stage_fwd_mid(x.cuda(), xa.cuda(), W.cuda(), ALPHA, 0, n, heads, 1)
    got = (y, ya, *ops.stage_bwd_mid(y, ya, mid, dy.cuda(), dya.cuda(), W.cuda(), ALPHA, 0, n, heads, 1))
    # results rounded to 2^-9; the weight gradient is not rounded, and its terms start from unrounded states
    _check(got, want, 2e-2)


@pytest.mark.parametrize("activation", ["tanh", "linear"])
@pytest.mark.parametrize("B,d,ctx", [(4, 32, False), (64, 32, False), (16, 64, False), (16, 24, False), (64, 32, True)])
def test_forward_error_over_32_steps_is_that_of_roundings(B, d, ctx, activation):
    """Each of 32 steps rounds a value a few times by 2^-25 of its size on average, independently: sqrt(32) * 2^-25 * 2 = 3.4e-7
    in the mean.  The fp32 value of 0.9 alone, 2.6e-8 off in every step, would add 8e-7."""
    import ncn_cuda_b200 as ncn

    N, heads, n = 96, 2, 32
    x, xa, W, dy, dya = _case(B, N, heads, d, seed=8)
    cl = torch.full((B,), N, dtype=torch.int32)
    Y, YA = O.stage_forward(x.double(), xa.double(), W.double(), ALPHA, activation, n, heads, 1)
    act = ncn.ops.ACTIVATION_CODES[activation]
    args = (x.cuda(), xa.cuda(), W.cuda())
    y, ya = ncn.fused_ncn_cuda_ctxlen(*args, cl.cuda(), ALPHA, act, n, heads, 1) if ctx else ncn.fused_ncn_cuda_v2(*args, ALPHA, act, n, heads, 1)
    for got, want in ((y, Y), (ya, YA)):
        assert (got.double().cpu() - want).norm() / want.norm() < 3.5e-7


@pytest.mark.parametrize("n,d,heads,m", [(32, 32, 2, 3), (16, 32, 1, 5), (16, 64, 1, 4), (32, 24, 1, 2)])
def test_a_padded_batch_is_dealt_out_without_loss(n, d, heads, m):
    """Up to 1024 rows the groups that take steps are shared out evenly among the teams; a longer batch goes row by row.
    Rows are independent, so the same rows give the same values either way."""
    import ncn_cuda_b200 as ncn

    B, N, E = 1025, m * n, heads * d
    g = torch.Generator().manual_seed(n + d)
    x, xa, dy, dya = (torch.randn(B, N, E, generator=g).cuda() for _ in range(4))
    W = torch.randn(2 * E, generator=g).cuda() * d**-0.5
    ctx = torch.randint(-2, N + 3, (B,), generator=g, dtype=torch.int32)
    ctx[:3] = 0
    ctx[1021:1024] = torch.tensor([N, 0, 1], dtype=torch.int32)

    def run(rows):
        ys = ncn.ops.stage_fwd_ctx(x[rows], xa[rows], W, ctx[rows], ALPHA, 0, n, heads, 1)
        return (*ys, *ncn.ops.stage_bwd_ctx(*ys, dy[rows], dya[rows], W, ctx[rows], ALPHA, 0, n, heads, 1))

    whole = run(slice(0, B))
    for rows in (slice(0, 1024), slice(1, 8), slice(1023, 1025), slice(0, 3)):  # (smaller teams sum in another order)
        for k, (p, q) in enumerate(zip(run(rows)[:4], whole[:4])):
            # 1e-5 forward; gradients over up to 32 rebuilt steps 5e-5, as for the walk from the output alone
            assert (p - q[rows]).abs().max() <= (1e-5 if k < 2 else 5e-5) * q.abs().max()
    parts = [run(slice(0, 512))[4], run(slice(512, 1025))[4]]
    # the weight gradient is a sum over at most 1025 m groups in another order
    assert ((parts[0] + parts[1]) - whole[4]).abs().max() <= 2e-5 * whole[4].abs().max()
