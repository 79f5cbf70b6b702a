"""How far a long walk back from the output stands from 64 bits.  Each rebuilt step multiplies what went before by 1/0.9, so 18 to 32 steps
show what the rounding of a step does: the backward takes its reciprocals in the batches that LaneBatch and SoloBwd name, near those
of the forward, so that the two errors cancel.

The kernels are deterministic to the bit, and so are the inputs and the oracle.  Mean relative error (2-norm) over the seeds, measured with
those batches / with a reciprocal per position (groups of 16: half of them) and two roundings into gx_j instead of one:
  groups of 2, dx 6.544e-7 / 6.623e-7;  4, dx 9.884e-7 / 1.0025e-6;  8, dxa 1.0452e-6 / 1.0554e-6;
  one group per thread: 8, dxa 1.0449e-6 / 1.0496e-6;  16, dxa 1.3379e-6 / 1.3399e-6.
The bounds lie between the two."""
import pytest
import torch

from oracle import ncn_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,N,L,which,most", [
    (2, 1024, 10, "dx", 6.58e-7), (4, 1024, 6, "dx", 9.93e-7), (8, 1024, 4, "dxa", 1.049e-6),
    (8, 1048, 4, "dxa", 1.047e-6), (16, 1024, 2, "dxa", 1.3389e-6),
])
def test_error_of_a_long_walk(n, N, L, which, most):
    import ncn_cuda_b200 as ncn

    total, seeds = 0.0, 6
    for seed in range(seeds):
        x, xa, ws, dy, dya = O.make_inputs(seed, 64, N, 1, L, 0.01, dya_zero=False)
        want = O.net_fwd_bwd(x.double(), xa.double(), [w.double() for w in ws], dy.double(), dya.double(), 0.9, "tanh", n, 1)
        xd, xad = x.cuda().requires_grad_(), xa.cuda().requires_grad_()
        y = ncn.fused_ncn_net(xd, xad, torch.stack(ws).cuda(), 0.9, ncn.ops.ACTIVATION_CODES["tanh"], n, 1, backward_mode="invert")
        got = torch.autograd.grad(y, (xd, xad), (dy.cuda(), dya.cuda()))
        k = ("dx", "dxa").index(which)
        total += ((got[k].double().cpu() - want[2 + k]).norm() / want[2 + k].norm()).item()
    assert total / seeds < most
