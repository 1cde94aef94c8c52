"""One training step against the CPU oracle at the sizes where the kernel choice changes or a tile, cluster or copy has a
ragged end. Tolerances as in test_parity_gpu.py: 1e-5 of a tensor's largest value in f32 (5e-5 with the tensor-core
option: its products are within 2e-6 element by element, the norm backward amplifies them), 1e-2 in 16 bits, whose
storage rounds every tensor of the chain to 2^-12 in f16. bf16 rounds to 2^-9: the two operands of a product put
sqrt(2) 2^-9 of its spread (1.4, normal inputs, He weights) on every element, 4e-3, and the largest of 3e4 elements is
4.5 standard deviations out, 1.8e-2; the deltas carry two such roundings: 4e-2."""
import pytest

import harness as H
from soklyn_b200 import configs
from soklyn_b200.configs import NetSpec

pytestmark = pytest.mark.gpu


def _spec(name, dims, norm, act, prec, batch, optimiser="adam", dropout=0.0):
    n = len(dims) - 2
    return NetSpec(11, name, dims, (norm,) * n + ("disabled",), (act,) * n + ("identity",), (dropout,) * n + (0.0,), prec, "mse",
                   "identity", optimiser, 1e-3, batch, "he_normal", "normal", "normal", dropout > 0)


CASES = [
    _spec("one_row_tile_cluster_of_8", (1024, 512, 256), "rms", "silu", "f16", 16),
    _spec("k_steps_not_a_multiple_of_the_cluster", (456, 136, 72), "layer", "mish", "f16", 130, dropout=0.1),
    _spec("two_row_tiles_one_row_in_the_last", (192, 264, 128), "disabled", "tanh", "bf16", 129, "sgd"),
    _spec("odd_widths_copied", (333, 417, 203, 10), "layer", "mish", "f16", 301),
    _spec("odd_widths_copied_rms", (515, 266, 1001, 7), "rms", "silu", "f16", 257, dropout=0.3),
    _spec("odd_widths_persistent_tiles", (77, 2557, 130), "disabled", "sigmoid", "f16", 1950, "sgd"),
    _spec("pairs_odd_row_tiles", (1896, 2296, 136), "rms", "silu", "f16", 1900),
    _spec("pairs_half_empty_last_pair", (72, 2296, 128), "layer", "mish", "bf16", 1801, "sgd"),
    _spec("pairs_ten_rows_in_the_last_block", (72, 2296, 128), "rms", "silu", "f16", 1930, "sgd"),
    _spec("pairs_element_by_element", (72, 2301, 136), "disabled", "tanh", "f16", 1900),
    _spec("batchnorm_five_rows", (64, 40, 16), "batch", "tanh", "f32", 5, "sgd"),
    _spec("batchnorm_uneven_cluster", (128, 136, 10), "batch", "tanh", "f16", 1001),
    _spec("batchnorm_scalar_columns", (77, 133, 10), "batch", "tanh", "f32", 65),
    _spec("batchnorm_uncached_rows", (16, 64, 8), "batch", "sigmoid", "f32", 20011, "sgd"),
    _spec("few_long_rows", (40, 4104, 24), "layer", "silu", "f16", 3),
    _spec("head_over_many_rows", (48, 33, 10), "rms", "relu", "f32", 4099),
    _spec("ffma_cluster_uneven_panels", (1000, 70, 34), "layer", "silu", "f16", 33),
]


def _unheld(spec):
    """Not held to the tolerance of a gradient: with Adam dv is its square, which doubles the relative error (dm holds the
    gradient then); with SGD dv is the gradient."""
    return ("mask",) + (("dv_w", "dv_b", "dv_nw", "dv_nb") if spec.optimiser == "adam" else ())


def _pairs(m, n, sms=148):
    """Does a product of m x n outputs run on pairs of SMs? 256-wide tiles have to take at most 5/4 of the time of 128-wide
    ones by waves, leave no cluster of two a place, and come in an even number of rows or in 15 and more."""
    rows, tiles = -(-m // 128), lambda bn: -(-m // 128) * -(-n // bn)
    cost = lambda bn: -(-tiles(bn) // sms) * bn
    return n > 128 and cost(256) * 4 <= cost(128) * 5 and 2 * tiles(256) > sms and (rows % 2 == 0 or rows >= 15)


@pytest.mark.parametrize("spec", [s for s in CASES if s.name.startswith("pairs")], ids=lambda s: s.name)
def test_the_pair_cases_run_pairs(spec):
    assert _pairs(spec.batch, spec.dims[1])                                        # forward and the hidden delta
    assert spec.name != "pairs_odd_row_tiles" or _pairs(spec.dims[0], spec.dims[1])   # and the weight gradient


@pytest.mark.parametrize("spec", CASES, ids=lambda s: s.name)
def test_step_matches_oracle_at_the_edges(gpu_ctx, spec):
    w = configs.make_weights(spec)
    x, t, _ = configs.make_data(spec)
    onet, _ = H.run_oracle(spec, w, x, t, 1)
    dnet, _ = H.run_device(gpu_ctx, spec, w, x, t, 1)
    H.compare_states(gpu_ctx, spec, dnet, onet, {"f32": 1e-5, "f16": 1e-2, "bf16": 4e-2}[spec.precision], skip=_unheld(spec))


def test_f32_tensor_core_option_takes_odd_widths(gpu_ctx):
    spec = _spec("f32_tensor_cores_odd", (515, 1030, 333), "rms", "silu", "f32", 601, "sgd")
    w = configs.make_weights(spec)
    x, t, _ = configs.make_data(spec)
    onet, _ = H.run_oracle(spec, w, x, t, 1)
    try:
        gpu_ctx.set_f32_tensor_cores(True)
        dnet, _ = H.run_device(gpu_ctx, spec, w, x, t, 1)
    finally:
        gpu_ctx.set_f32_tensor_cores(False)
    H.compare_states(gpu_ctx, spec, dnet, onet, 5e-5, skip=_unheld(spec))
