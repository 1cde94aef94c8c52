"""What the launches of a step promise beside their results: SMs that stay free, errors that do not outlive their call."""
import numpy as np
import pytest
import torch

import soklyn_b200 as sk
from soklyn_b200 import log

pytestmark = pytest.mark.gpu


def _chain(ctx, width, blocks, rows, prec):
    cfg = sk.LayerInitConfig(sk.Normalisation.Disabled, sk.Activation.Identity, sk.Regularisation.none(), 0.0)
    net = sk.FeedForwardNetwork([sk.DenseBlock(ctx, False, width, width, rows, sk.InitZeroFunc(), cfg, prec)
                                 for _ in range(blocks)], width)
    return net, sk.Tensor.zeros(ctx, (rows, width), prec)


def test_reserved_sms_are_free_while_products_follow_each_other(gpu_ctx):
    """A kernel on another stream, issued while the first of two long products runs, finishes beside it: the blocks of
    the second product do not wait on the reserved SMs for the first one's end. The products' blocks take an SM's
    whole register file, so the kernel has no other place to run."""
    net, x = _chain(gpu_ctx, 8192, 2, 8192, sk.Precision.FP16)   # about 0.8 ms each, several times the host's part of the test
    side, word = torch.cuda.Stream(), torch.zeros(1, device=gpu_ctx.device)
    try:
        gpu_ctx.set_reserve_sms(16)
        for _ in range(2):   # the first round loads the kernels
            start, end, done = (torch.cuda.Event(enable_timing=True) for _ in range(3))
            torch.cuda.synchronize()
            start.record(gpu_ctx.stream)
            net.forward(gpu_ctx, x, 8192, False, 1)
            end.record(gpu_ctx.stream)
            with torch.cuda.stream(side):
                word.add_(1.0)
                done.record(side)
            torch.cuda.synchronize()
    finally:
        gpu_ctx.set_reserve_sms(0)
    assert start.elapsed_time(done) < 0.4 * start.elapsed_time(end)


def test_a_refused_launch_is_reported_once(gpu_ctx):
    """More rows than a grid of 128-row tiles has: the launch is refused, and the calls after it are not blamed for it."""
    rows = 65536 * 128 + 1
    net, x = _chain(gpu_ctx, 8, 1, rows, sk.Precision.FP32)
    with pytest.raises(log.DriverError, match="gemm"):
        net.forward(gpu_ctx, x, rows, False, 1)
    assert np.all(sk.Tensor.fill(gpu_ctx, (3, 5), 2.0).download(gpu_ctx) == 2.0)
    net.forward(gpu_ctx, x, 1000, False, 1)
    gpu_ctx.synchronize()
