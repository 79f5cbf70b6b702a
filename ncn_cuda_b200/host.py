"""Host-buffer entry: forward + backward of a fused net on tensors that live in (pinned) host memory.

Rows are independent, so the batch is cut into chunks that flow through three streams
(host->device copies, kernels, device->host copies; `host_step` of csrc/ncn_torch.cpp); the
weight gradient is accumulated chunk after chunk in a fixed order, so it stays bitwise
reproducible.  This is the call a host-side caller of the reference's operator would make
when its activations are not resident on the GPU.
"""
from __future__ import annotations

import math
from typing import Optional, Tuple

import torch

from . import _lib, ops
from .ncn_pytorch_wrapper_v2 import plan_backward


def chunk_bounds(B: int, rows: int):
    """[begin, end) of the chunks: `rows` rows each, with shorter ones at both ends of a long batch
    (quarter, quarter, half) so that the first copy in and the last copy out, which nothing
    overlaps, are short."""
    if B < 6 * rows or rows < 4:
        return [(r0, min(B, r0 + rows)) for r0 in range(0, B, rows)]
    ramp = [rows // 4, rows // 4, rows // 2]
    sizes = list(ramp)
    left = B - 2 * sum(ramp)
    sizes += [rows] * (left // rows)
    if left % rows:
        sizes.append(left % rows)
    sizes += ramp[::-1]
    out, r0 = [], 0
    for n in sizes:
        out.append((r0, r0 + n))
        r0 += n
    assert r0 == B
    return out


def rows_per_chunk(B: int, tensor_bytes: int, chunk_rows: int) -> int:
    """Rows of a chunk, at most `chunk_rows`.  c chunks leave 1/c of the copies without overlap and cost 75 us each (eight copies,
    three launches, events), so the sum is smallest at c = sqrt(copies / 75 us); four tensors each way at 47 GB/s make that
    sqrt(tensor / 0.9 MB).  (From six on chunk_bounds cuts the first and the last up. That adds four, 300 us, and
    takes three quarters off the first copy in and the last out, which at six chunks are 0.46 ms each.)  Measured with 1, 2, 4, 8, 16 chunks, us: tensors of 2.1 MB 429 436 474 788 1134; 8.4 MB 1354 1149 1148 -
    1623; 33.6 MB 5040 4050 3641 3662 4145; 134 MB 20045 15900 14225 13161 13033."""
    c = max(1, round(math.sqrt(tensor_bytes / 0.9e6)))
    return min(chunk_rows, B, -(-B // c))


def net_fwd_bwd_host(
    x: torch.Tensor, xa: torch.Tensor, W: torch.Tensor, dy: torch.Tensor, dya: torch.Tensor,
    alpha: float, activation, n_cache: int, n_head: int,
    out: Optional[Tuple[torch.Tensor, ...]] = None, chunk_rows: int = 4096, backward_mode: str = "auto",
    device: Optional[torch.device] = None,
):
    """x, xa, dy, dya: CPU tensors [B, N, E] (pinned for full copy bandwidth); W: [L, 2E].  `chunk_rows`: most rows
    on the device at a time per buffer.  Returns (y, ya, dx, dxa, dW) on the host; `out` may supply the four pinned result tensors."""
    B = x.shape[0]
    if B < 1 or chunk_rows < 1:
        raise ValueError(f"no rows to take: {B} rows in chunks of {chunk_rows}")
    device = device or torch.device("cuda", torch.cuda.current_device())
    L = W.shape[0]
    if out is None:
        out = tuple(torch.empty_like(x).pin_memory() for _ in range(4))
    y_h, ya_h, dx_h, dxa_h = out
    Wd = W.to(device=device, dtype=torch.float32).contiguous()
    dW = torch.zeros(L, W.shape[1], dtype=torch.float32, device=device)
    recompute, every, tape = plan_backward(x.dtype, n_cache, L, False, backward_mode)
    act = ops.activation_code(activation)

    rows = rows_per_chunk(B, x.numel() * x.element_size(), chunk_rows)
    _lib.native().host_step(
        [x, xa, dy, dya], list(out), Wd, dW, alpha, act, n_cache, n_head, recompute, every, tape, chunk_bounds(B, rows)
    )
    dW_h = dW.to("cpu")
    return y_h, ya_h, dx_h, dxa_h, dW_h
