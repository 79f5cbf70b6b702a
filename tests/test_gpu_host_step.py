"""The host-buffer call in one chunk and in many: every backward mode, chunks shorter than the buffers, more chunks than buffers, and
what it refuses.  Tolerance: 1e-5 of the largest value (fp32), as for the device call; 2e-5 for the gradients of `recompute`, whose walk
back over 24 steps multiplies rounding by 1/0.9 each; the rows themselves do not depend on the chunk they are in."""
import pytest
import torch

from oracle import ncn_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["auto", "tape", "recompute", "checkpoint"])
def test_chunks(mode):
    from ncn_cuda_b200.host import net_fwd_bwd_host

    B, N, n, L = 61, 512, 4, 6
    x, xa, ws, dy, dya = O.make_inputs(5, B, N, 1, L, 0.25, dya_zero=False)
    W = torch.stack(ws)
    call = lambda rows: net_fwd_bwd_host(x, xa, W, dy, dya, 0.9, "tanh", n, 1, chunk_rows=rows, backward_mode=mode)
    whole, cut = call(B), call(8)
    want = O.net_fwd_bwd(x, xa, ws, dy, dya, 0.9, "tanh", n, 1)
    for a, b, c in zip(whole, cut, want[:4]):
        assert torch.equal(a, b) and O.rel_err(a, c) < (2e-5 if mode == "recompute" else 1e-5)
    for g in (whole[4], cut[4]):
        assert O.rel_err(g, torch.stack(list(want[4]))) < 2e-5


def test_refusals_leave_the_call_usable():
    from ncn_cuda_b200 import _lib
    from ncn_cuda_b200.host import net_fwd_bwd_host

    x = torch.randn(40, 96, 1)
    W = torch.randn(2, 2)
    with pytest.raises(ValueError):
        net_fwd_bwd_host(x[:, :, 0], x[:, :, 0], W, x[:, :, 0], x[:, :, 0], 0.9, "tanh", 4, 1)
    with pytest.raises(ValueError):
        net_fwd_bwd_host(x, x, torch.randn(2, 3), x, x, 0.9, "tanh", 4, 1)
    with pytest.raises(_lib.NCNError):
        net_fwd_bwd_host(x, x, W, x, x, 0.9, "tanh", 5, 1, chunk_rows=3)
    y = net_fwd_bwd_host(x, x, W, x, x, 0.9, "tanh", 4, 1)[0]
    assert O.rel_err(y, O.net_forward(x, x, list(W), 0.9, "tanh", 4, 1)[0]) < 1e-5
