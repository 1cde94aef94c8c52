"""Sums of 16-bit products whose operands are copied to a pitch the tensor cores can fetch: no further from 64 bits than
the FFMA kernel's chain of round-to-nearest adds, whatever their length and sign."""
import numpy as np
import pytest

import soklyn_b200 as sk
from soklyn_b200.configs import _GivenWeights

pytestmark = pytest.mark.gpu


def _gradient_error(ctx, k, n, batch, prec, positive, ffma):
    """2-norm error of dW = X^T . dY of a block, against its own 16-bit operands in 64 bits."""
    rng = np.random.default_rng(7)
    w = rng.standard_normal((k, n)).astype(np.float32) / np.float32(np.sqrt(k))
    draw = (lambda s: rng.random(s, np.float32)) if positive else (lambda s: rng.standard_normal(s).astype(np.float32))
    cfg = sk.LayerInitConfig(sk.Normalisation.Disabled, sk.Activation.Identity, sk.Regularisation.none(), 0.0)
    blk = sk.DenseBlock(ctx, True, k, n, batch, _GivenWeights(w), cfg, prec)
    x = sk.Tensor.from_cpu_vector(ctx, draw((batch, k)), (batch, k), prec)
    target = draw((batch, n))
    t = sk.Tensor.from_cpu_vector(ctx, -8 - target if positive else target, (batch, n), prec)   # deltas all positive
    try:
        ctx.set_gemm_engine(ffma)
        blk.forward(ctx, x, batch, False, 1)
        blk.compute_loss(ctx, t, sk.LossConfig(sk.LossFunc.MeanSquareLoss, sk.Activation.Identity))
        blk.backward_output(ctx, x, sk.TrainContext(sk.Optimiser.SGD(), sk.Optimiser.SGD(), batch, 0.0), 1)
        ctx.synchronize()
    finally:
        ctx.set_gemm_engine(False)
    # the 16-bit deltas are stored at 1/16, the loss scale is 512
    exact = x.data.double().T @ blk.d_prenorm_lp.data.double() * (16.0 / (512.0 * batch))
    return float((blk.get_dv_weights().data.double() - exact).norm() / exact.norm())


@pytest.mark.parametrize("prec", [sk.Precision.FP16, sk.Precision.BF16], ids=["f16", "bf16"])
@pytest.mark.parametrize("positive", [False, True], ids=["signed", "one_sided"])
@pytest.mark.parametrize("k,n,batch", [(333, 417, 300), (777, 1001, 1024), (333, 416, 4096), (1001, 2003, 4099), (65, 131, 16384)])
def test_odd_width_sums_are_no_less_exact_than_the_ffma_kernels(gpu_ctx, k, n, batch, positive, prec):
    """The tensor pipe truncates when it adds into its accumulator: left in it, one-sided sums of this length are 3 to 10
    times further off than the chain. The tenth is for the two kernels' different order of the same sum."""
    ours, chain = (_gradient_error(gpu_ctx, k, n, batch, prec, positive, ffma) for ffma in (False, True))
    assert ours <= 1.1 * chain, f"{ours:.2e} against {chain:.2e}"
