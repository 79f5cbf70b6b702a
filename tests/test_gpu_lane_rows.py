"""Row kernels around the line between the register-resident ones (rows that do not fill their warps, rows of 8192 positions, one
group per thread) and the shared-memory ones: where a warp's share ends inside a thread's blocks, inside a warp and just behind one,
halos as long as a warp's share, shifts through the tile buffer, several rows per CTA, several tiles per CTA, a last tile that is not
full.  The short rows of SHAPES lie on the other side of the line; the tests that name a family ask which kernels ran.  Tolerances are those of test_gpu_sweep.py: 1e-5 (fp32) of
the largest value, 2e-5 for the gradients of a walk back over more than 16 steps, 2e-2 (bf16)."""
import pytest
import torch

from oracle import ncn_oracle as O

from .kernels_util import kernels_of, launched

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ncn():
    import ncn_cuda_b200

    return ncn_cuda_b200


def _data(B, N, n, L, dtype, seed):
    x, xa, ws, dy, dya = O.make_inputs(seed, B, N, 1, L, 1.0 / n, dya_zero=False)
    xa = torch.randn(B, N, 1, generator=torch.Generator().manual_seed(seed)) * 0.3
    if dtype != torch.float32:
        x, xa, dy, dya = (t.bfloat16().float() for t in (x, xa, dy, dya))
    return x, xa, ws, dy, dya


def _step(ncn, x, xa, ws, dy, dya, act, n, mode, dtype, first=0):
    xd, xad = (t.cuda().to(dtype).requires_grad_() for t in (x, xa))
    W = torch.stack(ws).cuda().requires_grad_()
    y, ya = ncn.fused_ncn_net(xd, xad, W, 0.9, ncn.ops.ACTIVATION_CODES[act], n, 1, first_module=first, backward_mode=mode)
    torch.autograd.backward([y, ya], [dy.cuda().to(dtype), dya.cuda().to(dtype)])
    ncn.ops.device_status()
    return [t.float().cpu() for t in (y.detach(), ya.detach(), xd.grad, xad.grad, W.grad)]


def _against_oracle(got, x, xa, ws, dy, dya, act, n, first):
    ry, rya, rdx, rdxa, rdW = O.net_fwd_bwd(x, xa, ws, dy, dya, 0.9, act, n, 1, first_module=first)
    for name, a, b in zip(("y", "ya", "dx", "dxa"), got, (ry, rya, rdx, rdxa)):
        if act == "relu" and name[0] == "d":
            # the derivative jumps at 0: a pre-activation of order 1 carries 2e-7 of rounding, five times that at the end of a walk back
            # over 16 steps, so 16 * 1e-6 * 0.4 (the density at 0) of the elements have one of the other sign, and each changes its
            # element's gradient by up to a tenth: 0.1 * sqrt(6e-6) = 2.5e-4 of the 2-norm
            assert (a - b).norm() / b.norm() < 3e-4, name
        else:
            assert O.rel_err(a, b) < 1e-5, name
    # the weight gradient sums B N terms that largely cancel, the oracle's in fp32 as well: 1e-5 of the terms' size per sqrt(count)
    got_w, want_w = got[4], torch.stack(list(rdW))
    assert (got_w - want_w).abs().max() < 1e-4 * max(1.0, want_w.abs().max().item(), (x.numel() ** 0.5)), "dW"


def _bf16_against_oracle(got, want):
    """Activations and their gradients to 2e-2 of the largest value.  The weight gradient is in fp32, a sum of B N terms of order 0.03 that
    largely cancel, each off by up to 2^-11 of itself (tanh.approx): 2e-5 per sqrt(count), or of the result where that is more (measured
    up to 3e-7).  A tile of rows left out or taken twice is ten times that and more."""
    for name, a, b in zip(("y", "ya", "dx", "dxa"), got, want):
        assert O.rel_err(a, b) < 2e-2, name
    dW = torch.stack(list(want[4]))
    assert (got[4].float().cpu() - dW).abs().max() < 2e-5 * max(1.0, dW.abs().max().item(), got[0].numel() ** 0.5), "dW"


# (n, N): blocks per row m = N / n in the comment
SHAPES = [
    (2, 248), (2, 264), (2, 1040), (2, 4088), (2, 8184), (2, 8192),  # m = 124, 132, 520, 2044, 4092, 4096
    (4, 240), (4, 520), (4, 1032), (4, 3000), (4, 4104), (4, 8184), (4, 8192),  # m = 60, 130, 258, 750, 1026, 2046, 2048
    (8, 256), (8, 272), (8, 528), (8, 1040), (8, 3008), (8, 8176), (8, 8192),  # m = 32, 34, 66, 130, 376, 1022, 1024
]
STAGES = {2: 9, 4: 6, 8: 4}


@pytest.mark.parametrize("n,N", SHAPES)
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_rows_of_any_even_number_of_blocks(ncn, n, N, dtype):
    L = STAGES[n]
    while 2 ** (L - 2) >= N // n:
        L -= 1
    x, xa, ws, dy, dya = _data(7, N, n, L, dtype, N + n)
    ry, rya, rdx, rdxa, rdW = O.net_fwd_bwd(x, xa, ws, dy, dya, 0.9, "tanh", n, 1)
    got = _step(ncn, x, xa, ws, dy, dya, "tanh", n, "auto", dtype)
    for name, a, b in zip(("y", "ya", "dx", "dxa", "dW"), got, (ry, rya, rdx, rdxa, torch.stack(list(rdW)))):
        assert O.rel_err(a, b) < (1e-5 if dtype == torch.float32 else 2e-2), name


@pytest.mark.parametrize("n,N,B,act,mode,first", [
    (4, 1048, 1, "linear", "checkpoint", 0), (4, 1048, 300, "sigmoid", "tape", 0), (4, 2984, 3, "relu", "invert", 2),
    (8, 1040, 65, "tanh", "tape", 1), (2, 1044, 5, "tanh", "checkpoint", 3), (8, 8192, 2, "tanh", "invert", 0),
])
def test_modes_and_first_stages(ncn, n, N, B, act, mode, first):
    L = {2: 5, 4: 3, 8: 2}[n]
    x, xa, ws, dy, dya = _data(B, N, n, L, torch.float32, 3 * N + B)
    ry, rya, rdx, rdxa, rdW = O.net_fwd_bwd(x, xa, ws, dy, dya, 0.9, act, n, 1, first_module=first)
    got = _step(ncn, x, xa, ws, dy, dya, act, n, mode, torch.float32, first)
    for name, a, b in zip(("y", "ya", "dx", "dxa", "dW"), got, (ry, rya, rdx, rdxa, torch.stack(list(rdW)))):
        assert O.rel_err(a, b) < 1e-5, name


# Ragged rows in every mode and activation, with more tiles than CTAs (2 to 5 CTAs per SM); (2, 1044) and (8, 1008) have several rows
# to a tile and a last tile that is not full.
@pytest.mark.parametrize("n,N,B,act,mode,first", [
    (4, 3000, 800, "linear", "checkpoint", 0), (4, 4112, 700, "sigmoid", "tape", 0), (8, 3008, 800, "relu", "invert", 1),
    (2, 1044, 3001, "sigmoid", "checkpoint", 0), (2, 1044, 3001, "tanh", "tape", 2), (8, 1008, 3003, "tanh", "checkpoint", 0),
    (8, 1008, 3003, "linear", "tape", 0), (4, 3000, 800, "tanh", "invert", 0),
])
def test_ragged_rows_in_many_tiles(ncn, n, N, B, act, mode, first):
    L = {2: 5, 4: 3, 8: 2}[n]
    x, xa, ws, dy, dya = _data(B, N, n, L, torch.float32, N + B)
    got, names = kernels_of(lambda: _step(ncn, x, xa, ws, dy, dya, act, n, mode, torch.float32, first))
    assert launched(names, rf"lane_fwd_kernel<{n}, .*true>") and launched(names, rf"lane_bwd_kernel<{n}, .*true>"), names
    _against_oracle(got, x, xa, ws, dy, dya, act, n, first)


# What the backward fetches a tile ahead, rows that fill their warps and ragged ones: from the output (1), with the end state stored alone (2) or behind
# others (3); one tile, several rows to a tile and a last one that is not full, many tiles per CTA, first stages whose last shift is not 0.
@pytest.mark.parametrize("n,N,B,L,act,mode,dtype,first,ahead", [
    (8, 2048, 1, 4, "tanh", "tape", torch.bfloat16, 0, 2), (8, 1024, 2003, 3, "tanh", "tape", torch.bfloat16, 1, 2), (2, 8192, 500, 3, "sigmoid", "tape", torch.bfloat16, 0, 2),
    (8, 4096, 700, 2, "linear", "tape", torch.float32, 0, 2), (8, 4096, 700, 4, "tanh", "tape", torch.float32, 0, 3), (2, 1024, 2001, 10, "tanh", "tape", torch.float32, 0, 0),
    (4, 4096, 700, 5, "tanh", "tape", torch.float32, 0, 3), (4, 4096, 700, 3, "tanh", "tape", torch.bfloat16, 1, 2), (4, 8192, 301, 5, "tanh", "checkpoint", torch.float32, 0, 1),
    (4, 1024, 3001, 4, "sigmoid", "invert", torch.float32, 0, 1), (4, 4096, 601, 6, "tanh", "checkpoint", torch.float32, 0, 0), (4, 512, 2003, 4, "linear", "tape", torch.float32, 1, 2),
    (8, 8192, 301, 3, "tanh", "checkpoint", torch.float32, 0, 1), (2, 4096, 901, 8, "relu", "checkpoint", torch.float32, 0, 1),
    (4, 3000, 800, 5, "tanh", "checkpoint", torch.float32, 0, 1), (8, 5008, 500, 4, "tanh", "checkpoint", torch.float32, 0, 1), (2, 5000, 700, 6, "tanh", "tape", torch.float32, 0, 2), (4, 4000, 500, 5, "tanh", "tape", torch.float32, 0, 3),
    (2, 8184, 400, 7, "tanh", "tape", torch.bfloat16, 1, 2), (8, 3008, 700, 3, "tanh", "tape", torch.float32, 0, 0),
    (8, 4096, 601, 2, "sigmoid", "invert", torch.float32, 1, 1), (2, 512, 3001, 5, "tanh", "checkpoint", torch.float32, 1, 1),
])
def test_rows_a_tile_ahead(ncn, n, N, B, L, act, mode, dtype, first, ahead):
    x, xa, ws, dy, dya = _data(B, N, n, L, dtype, N + B)
    got, names = kernels_of(lambda: _step(ncn, x, xa, ws, dy, dya, act, n, mode, dtype, first))
    assert launched(names, rf"lane_bwd_kernel<{n},.* {ahead}, (true|false|0|1)>") or launched(names, rf"lanep_bwd_kernel<{n},.* {ahead}>"), names
    if dtype == torch.float32:
        _against_oracle(got, x, xa, ws, dy, dya, act, n, first)
    else:
        _bf16_against_oracle(got, O.net_fwd_bwd(x, xa, ws, dy, dya, 0.9, act, n, 1, first_module=first))


# Residual layers: dy of a tile is read a second time, for its end, and counted on a barrier of its own.  Many tiles per CTA, a last one that
# is not full, one stored state (2) and several (3).
@pytest.mark.parametrize("n,N,B,L,dtype,ahead", [
    (4, 4096, 1001, 6, torch.float32, 3), (4, 1024, 4003, 3, torch.bfloat16, 2), (8, 4096, 701, 4, torch.float32, 3), (8, 1024, 4003, 4, torch.bfloat16, 2),
    (2, 8192, 501, 3, torch.bfloat16, 2), (2, 5000, 701, 6, torch.float32, 2), (4, 4000, 701, 5, torch.float32, 3),
])
def test_residual_layers_a_tile_ahead(ncn, n, N, B, L, dtype, ahead):
    from ncn_cuda_b200.ncn_pytorch_wrapper_v2 import plan_backward

    x, xa, ws, dy, dya = _data(B, N, n, L, dtype, N + B)
    W = torch.stack(ws).cuda()
    xd, xad, dyd, dyad = (t.cuda().to(dtype) for t in (x, xa, dy, dya))
    _, every, _ = plan_backward(dtype, n, L, True, "tape")

    def calls():
        y, ya, ck = ncn.ops.net_fwd(xd, xad, W, 0.9, 0, n, 1, 0, every, True, True)
        return y, ya, *ncn.ops.net_bwd(None, None, dyd, dyad, W, 0.9, 0, n, 1, 0, ckpt=ck, ckpt_every=every, residual=True, tape=True)

    got, names = kernels_of(calls)
    ncn.ops.device_status()
    assert launched(names, rf"lane_bwd_kernel<{n},.* {ahead}, (true|false|0|1)>") or launched(names, rf"lanep_bwd_kernel<{n},.* {ahead}>"), names
    want = O.stack_fwd_bwd(x, xa, [ws], dy, dya, 0.9, "tanh", n, 1)
    got, want = [t.float().cpu() for t in got], (*want[:4], want[4][0])
    if dtype == torch.bfloat16:
        _bf16_against_oracle(got, want)
    else:
        for name, a, b in zip(("y", "ya", "dx", "dxa"), got, want):
            assert O.rel_err(a, b) < 1e-5, name
        dW = torch.stack(list(want[4]))  # (bound as in _against_oracle)
        assert (got[4] - dW).abs().max() < 1e-4 * max(1.0, dW.abs().max().item(), x.numel() ** 0.5), "dW"


# A backward that is asked for the rebuilt input reads the states as the forward of the same arguments wrote them: where all of them fit
# into shared memory, where they do not (groups of 4: read from global memory, form 4), behind an output and behind a stored end state.
@pytest.mark.parametrize("n,N,L,tape,residual,dtype,form", [
    (4, 512, 5, True, False, torch.float32, 0), (4, 512, 5, True, True, torch.float32, 4), (4, 512, 6, True, False, torch.float32, 4),
    (4, 1024, 6, True, True, torch.bfloat16, 4), (4, 2048, 6, True, False, torch.float32, 4), (4, 2048, 5, True, True, torch.bfloat16, 0),
    (4, 4096, 5, True, False, torch.float32, 0), (4, 4096, 5, True, True, torch.float32, 4), (4, 4096, 6, True, False, torch.float32, 4),
    (4, 4096, 6, True, True, torch.float32, 4), (4, 4096, 6, True, False, torch.bfloat16, 4), (4, 8192, 2, True, False, torch.float32, 4),
    (4, 8192, 4, True, True, torch.bfloat16, 4), (4, 8192, 4, False, False, torch.float32, 4), (4, 4096, 7, False, False, torch.float32, None),
    (2, 1024, 9, True, False, torch.float32, None), (8, 4096, 4, True, True, torch.float32, None), (16, 1040, 3, True, False, torch.float32, None),
])
def test_rebuilt_input_from_the_same_states(ncn, n, N, L, tape, residual, dtype, form):
    B = 37
    x, xa, ws, dy, dya = _data(B, N, n, L, dtype, N + L)
    W = torch.stack(ws).cuda()
    xd, xad, dyd, dyad = (t.cuda().to(dtype) for t in (x, xa, dy, dya))

    def calls():
        y, ya, ck = ncn.ops.net_fwd(xd, xad, W, 0.9, 0, n, 1, 0, 1, residual, tape)
        s0, s1 = (None, None) if tape else (y, ya)
        return [ncn.ops.net_bwd(s0, s1, dyd, dyad, W, 0.9, 0, n, 1, 0, ckpt=ck, ckpt_every=1, residual=residual, tape=tape, want_inputs=want)
                for want in (False, True)]

    (got, rec), names = kernels_of(calls)
    ncn.ops.device_status()
    fp32 = dtype == torch.float32
    for name, a, b in zip(("x", "xa"), rec[3:], (x, xa)):
        assert O.rel_err(a.float(), b) < (1e-5 if fp32 else 2 ** -8), name
    want = O.stack_fwd_bwd(x, xa, [ws], dy, dya, 0.9, "tanh", n, 1) if residual else O.net_fwd_bwd(x, xa, ws, dy, dya, 0.9, "tanh", n, 1)
    dW = torch.stack(list(want[4][0] if residual else want[4]))
    for res in (got, rec):
        for name, a, b in zip(("dx", "dxa"), res, want[2:4]):
            assert O.rel_err(a.float(), b) < (1e-5 if fp32 else 2e-2), name
        assert O.rel_err(res[2], dW) < (2e-5 if fp32 else 2e-2), "dW"
    if form is not None:
        assert launched(names, rf"lanep_bwd_kernel<{n},.* {form}>"), names


@pytest.mark.parametrize("n,N,B,act,mode", [
    (16, 240, 5003, "tanh", "checkpoint"), (16, 1840, 700, "sigmoid", "tape"), (8, 1048, 2001, "linear", "checkpoint"),
    (8, 1048, 2001, "tanh", "tape"), (16, 2048, 600, "relu", "checkpoint"),
])
def test_one_group_per_thread_in_many_tiles(ncn, n, N, B, act, mode):
    L = 2
    x, xa, ws, dy, dya = _data(B, N, n, L, torch.float32, N + B)
    got, names = kernels_of(lambda: _step(ncn, x, xa, ws, dy, dya, act, n, mode, torch.float32))
    assert launched(names, rf"solo_fwd_kernel<{n},") and launched(names, rf"solo_bwd_kernel<{n},"), names
    _against_oracle(got, x, xa, ws, dy, dya, act, n, 0)


@pytest.mark.parametrize("n,N", [(16, 16), (16, 48), (16, 240), (16, 512), (16, 528), (16, 1840), (16, 2048), (16, 2080), (16, 8176),
                                 (16, 8192), (8, 8), (8, 1048), (8, 2968), (8, 4088)])  # 1, 3, 15, 32, 33, 115 ... 512 blocks
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_one_group_per_thread(ncn, n, N, dtype):
    L = 4 if n == 16 else 5  # strides 0, 1, 2, 4 (8) mod m: rows of a few blocks wrap
    x, xa, ws, dy, dya = _data(11, N, n, L, dtype, N)
    ry, rya, rdx, rdxa, rdW = O.net_fwd_bwd(x, xa, ws, dy, dya, 0.9, "tanh", n, 1)
    got = _step(ncn, x, xa, ws, dy, dya, "tanh", n, "auto", dtype)
    for name, a, b in zip(("y", "ya", "dx", "dxa", "dW"), got, (ry, rya, rdx, rdxa, torch.stack(list(rdW)))):
        assert O.rel_err(a, b) < (1e-5 if dtype == torch.float32 else 2e-2), name


# What the backward fetches a tile ahead: with the end state stored (2) or from the output (1); one tile per CTA, many, several rows to
# a tile and a last tile that is not full.  fp32 rows of 4096 positions from the output have no room for it (0).
@pytest.mark.parametrize("n,N,B,act,mode,dtype,ahead", [
    (16, 8192, 1, "tanh", "tape", torch.float32, 2), (16, 8192, 500, "tanh", "tape", torch.bfloat16, 2), (16, 240, 5003, "sigmoid", "tape", torch.float32, 2),
    (16, 16, 9, "tanh", "tape", torch.bfloat16, 2), (8, 1048, 2001, "linear", "tape", torch.float32, 2), (8, 2968, 700, "tanh", "checkpoint", torch.float32, 1),
    (16, 6000, 301, "relu", "checkpoint", torch.float32, 1), (16, 4096, 700, "tanh", "checkpoint", torch.float32, 0),
])
def test_one_group_per_thread_a_tile_ahead(ncn, n, N, B, act, mode, dtype, ahead):
    x, xa, ws, dy, dya = _data(B, N, n, 2, dtype, N + B)
    got, names = kernels_of(lambda: _step(ncn, x, xa, ws, dy, dya, act, n, mode, dtype))
    assert launched(names, rf"solo_bwd_kernel<{n},.* {ahead}>"), names
    if dtype == torch.float32:
        _against_oracle(got, x, xa, ws, dy, dya, act, n, 0)
    else:
        _bf16_against_oracle(got, O.net_fwd_bwd(x, xa, ws, dy, dya, 0.9, act, n, 1))


@pytest.mark.parametrize("n,N,B,act,mode,first,L", [
    (16, 1840, 1, "linear", "checkpoint", 0, 3), (16, 240, 700, "sigmoid", "tape", 0, 2), (16, 2048, 3, "relu", "checkpoint", 2, 2),
    (16, 1040, 5, "tanh", "invert", 1, 1), (16, 1040, 5, "tanh", "invert", 0, 2), (8, 1048, 5, "sigmoid", "checkpoint", 1, 3),
])
def test_one_group_per_thread_modes(ncn, n, N, B, act, mode, first, L):
    x, xa, ws, dy, dya = _data(B, N, n, L, torch.float32, 5 * N + B)
    ry, rya, rdx, rdxa, rdW = O.net_fwd_bwd(x, xa, ws, dy, dya, 0.9, act, n, 1, first_module=first)
    got = _step(ncn, x, xa, ws, dy, dya, act, n, mode, torch.float32, first)
    tol = 2e-5 if mode == "invert" and n * L > 16 else 1e-5
    for name, a, b in zip(("y", "ya", "dx", "dxa", "dW"), got, (ry, rya, rdx, rdxa, torch.stack(list(rdW)))):
        assert O.rel_err(a, b) < tol, name


def test_long_walks_back_stay_stage_by_stage(ncn):
    """8192 fp32 positions: fused where stored states keep a walk back to 16 steps, else a kernel per stage."""
    x = torch.empty(2, 8192, 1, device="cuda")
    for n in (2, 4, 8, 16):
        assert ncn.ops.net_supported(x, n, 1, 4, 0, 16 // n)
        assert not ncn.ops.net_supported(x, n, 1, 16 // n + 1, 0, 0)
        assert ncn.ops.net_supported(x, n, 1, 16 // n, 0, 0)


@pytest.mark.parametrize("n,N", [(2, 8192), (4, 8192), (8, 8192), (16, 8192), (4, 3000), (2, 1024)])
def test_what_is_called_covered_is(ncn, n, N):
    """Stage strides that wrap (2^(stage - 1) >= N / n) leave the register-resident kernels; whole rows of 8192 fp32 positions
    have no others in groups of 2, 4 and 8."""
    from ncn_cuda_b200 import _lib

    lib = _lib.load()
    x = torch.randn(2, N, 1, device="cuda")
    W = torch.randn(2, 2, device="cuda") * n**-0.5
    every = 1 if n == 16 else 0
    for first in (0, 1, 9, 13):
        covered = ncn.ops.net_supported(x, n, 1, 2, 0, every, first_module=first)
        wraps = first > 0 and 2**first >= N // n
        assert covered == (not (wraps and N == 8192 and n < 16))
        if lib.ncn_net_supported(2, N, 1, n, 1, 2, 0, 0, every):
            assert covered
        if covered:
            y, ya, ck = ncn.ops.net_fwd(x, x, W, 0.9, 0, n, 1, first, every)
            ncn.ops.net_bwd(y, ya, x, x, W, 0.9, 0, n, 1, first, ckpt=ck, ckpt_every=every)
    assert lib.ncn_net_supported(2, N, 1, n, 1, 2, 0, 0, every) == (not (N == 8192 and n < 16))


@pytest.mark.parametrize("n,N", [(8, 1040), (16, 1840)])
def test_residual_layers_on_such_rows(ncn, n, N):
    B, layers, L = 9, 3, 3 if n == 8 else 2
    stack = ncn.NCNResidualStack(layers, 0.9, "tanh", n, 1, L, 1).cuda()
    W = torch.randn(layers, L, 2, generator=torch.Generator().manual_seed(5)) * n ** -0.5
    with torch.no_grad():
        stack.weight.copy_(W.cuda())
    x, xa, _, dy, dya = _data(B, N, n, L, torch.float32, 77)
    want = O.stack_fwd_bwd(x, xa, [list(w) for w in W], dy, dya, 0.9, "tanh", n, 1)
    xd, xad = x.cuda().requires_grad_(), xa.cuda().requires_grad_()
    y, ya = stack(xd, xad)
    g = torch.autograd.grad((y, ya), (xd, xad, stack.weight), (dy.cuda(), dya.cuda()))
    for a, b in zip((y, ya, g[0], g[1]), want[:4]):
        assert O.rel_err(a.detach().cpu(), b) < 1e-5


@pytest.mark.parametrize("n,N", [(4, 3000), (16, 1840)])
def test_the_weight_gradient_is_bitwise_repeatable(ncn, n, N):
    x, xa, ws, dy, dya = _data(70, N, n, 4, torch.float32, 11)
    a, b = (_step(ncn, x, xa, ws, dy, dya, "tanh", n, "auto", torch.float32) for _ in range(2))
    assert all(torch.equal(p, q) for p, q in zip(a, b))


@pytest.mark.parametrize("n,N", [(4, 1024), (4, 1048), (8, 1024), (8, 1040), (8, 1048), (2, 1048), (16, 1840)])
def test_a_nan_reaches_the_groups_that_read_it_and_no_others(ncn, n, N):
    L = 3
    x, xa, ws, dy, dya = _data(3, N, n, L, torch.float32, 21)
    x[1, 37] = float("nan")
    xa[1, N - 2] = float("nan")
    want = O.net_forward(x, xa, ws, 0.9, "tanh", n, 1)
    W = torch.stack(ws).cuda()
    with torch.no_grad():
        got = ncn.fused_ncn_net(x.cuda(), xa.cuda(), W, 0.9, 0, n, 1)
    for a, b in zip(got, want):
        assert torch.equal(torch.isnan(a).cpu(), torch.isnan(b))
