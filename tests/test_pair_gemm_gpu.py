"""Linears of more than 128 rows on pairs of CTAs against float64: one step and rings that wrap, K that ends inside a tile, tiles without rows or
columns, one wave of pairs and several, both tile widths, every form of the epilogue."""
import numpy as np
import pytest
import torch

from seq2seqsharp_b200 import _native as N
from tests.test_cluster_linears_gpu import check, linear
from tests import layered_models as LM, test_layered_gpu as LG
from tests.test_fused_gpu import dev, host

pytestmark = pytest.mark.gpu


# 257: a tile of one row; 1040, 72: a last step of one k tile; 2050, 300, 5: columns that do not exist; 3000 x 4608: several waves
@pytest.mark.parametrize("M,K,n", [(129, 8, 5), (130, 72, 300), (256, 64, 128), (257, 1040, 256), (385, 520, 2050), (700, 2048, 768), (3000, 136, 4608), (1281, 4104, 384)])
def test_rows(cuda, M, K, n):
    check(M, K, n, torch.float16, (0, 1))


@pytest.mark.parametrize("M,n", [(129, 96), (300, 2080)])
def test_outputs_with_other_companions(cuda, M, n):
    """A residual under a 16-bit output, fp32 without a residual, activations before either."""
    K = 200
    rng = np.random.default_rng(M + n)
    x, W = dev(rng.standard_normal((M, K)).astype(np.float32), torch.float16), dev((rng.standard_normal((K, n)) * 0.05).astype(np.float32), torch.float16)
    b, res = dev((rng.standard_normal(n) * 0.1).astype(np.float32), torch.float16), dev(rng.standard_normal((M, n)).astype(np.float32))
    ref = host(x).astype(np.float64) @ host(W).astype(np.float64) + host(b)
    tol = K * 2.0 ** -23 * float(np.abs(host(x)).max() * np.abs(host(W)).max()) + 1e-6      # fp32 sums, every rounding at its largest
    half = 2.0 ** -11 * max(1.0, float(np.abs(ref).max() + np.abs(host(res)).max()))
    np.testing.assert_allclose(host(linear(x, W, b, N.ACT_NONE, residual=res)), ref + host(res), atol=tol + half)
    np.testing.assert_allclose(host(linear(x, W, b, N.ACT_NONE, f32_out=True)), ref, atol=tol)
    np.testing.assert_allclose(host(linear(x, W, b, N.ACT_RELU, residual=res, f32_out=True)), np.maximum(ref, 0) + host(res), atol=tol + 1e-6)
    got = host(linear(x, W, b, N.ACT_GLU_NOACT, f32_out=True))
    big = max(1.0, float(np.abs(ref).max()))
    np.testing.assert_allclose(got, ref[:, 0::2] * ref[:, 1::2], atol=2 * tol * big + 1e-6)


# chunks of 32 columns with the gate's activation (a loop of its own), and the element-wise form
@pytest.mark.parametrize("M,K,n", [(130, 72, 320), (515, 264, 4096), (129, 40, 50)])
def test_gated_products(cuda, M, K, n):
    rng = np.random.default_rng(M)
    x, W = dev(rng.standard_normal((M, K)).astype(np.float32), torch.float16), dev((rng.standard_normal((K, n)) * 0.05).astype(np.float32), torch.float16)
    b = dev((rng.standard_normal(n) * 0.1).astype(np.float32), torch.float16)
    ref = host(x).astype(np.float64) @ host(W).astype(np.float64) + host(b)
    a, g = ref[:, 0::2], ref[:, 1::2]
    want = a / (1.0 + np.exp(-a)) * g
    tol = K * 2.0 ** -23 * float(np.abs(host(x)).max() * np.abs(host(W)).max()) + 1e-6      # of a sum; silu's slope is below 1.1, expf and the divide add 2^-21
    big = max(1.0, float(np.abs(ref).max()))
    np.testing.assert_allclose(host(linear(x, W, b, N.ACT_SWIGLU)), want, atol=(2.2 * tol + 2.0 ** -11 * big + 2.0 ** -21 * big) * big)


@pytest.mark.parametrize("keep", ["attention", "gate", "experts"])
def test_bf16_rows_of_one_layer(cuda, keep):
    """One bf16 layer whose weights leave one mechanism: its projections, the gate times output plus residual, the experts' clamped gated products; 300 rows at once
    and in portions that other kernels take."""
    cfg = LM.config([LM.layer(3, 16, 8, 16, 24, scale=1.5, experts=5 if keep == "experts" else None, top=2, ff=96, limit=0.5)], 256, 67, groups=4, taps=4)
    w = LM.weights(cfg, 5)
    w["l0.canon1"][:] = 0.0
    if keep != "gate":
        w["l0.rg1"][:] = 0.0
        w["l0.rg1.b"][:] = 8.0
    if keep == "experts":
        w["l0.mix.o"][:] = 0.0
    ids = LM.tokens(cfg, 300)
    want = LM.oracle(cfg, w).forward(ids)
    g = LG.engine(cfg, w, "bfloat16")
    for cuts in (None, [129, 171], [64] * 5, [100] * 3):
        assert LM.rel(LG.score(g, ids, cuts=cuts), want) < LM.TOL["bfloat16"], cuts
    g.CheckGuards()
    g.close()
