"""The linears whose K ranges lie on the CTAs of a cluster against float64, at the edges of their rules: odd widths and unaligned rows (scalar
epilogues), one to eight ranks, several groups of four columns per thread, K that ends inside a tile, rings that wrap."""
import numpy as np
import pytest
import torch

from seq2seqsharp_b200 import _native as N
from tests.test_fused_gpu import dev, host, stream

pytestmark = pytest.mark.gpu


def linear(x, W, bias, act, residual=None, f32_out=False, shift=0):
    """shift: elements between a 16-byte boundary and the packed weights (first) / the output and the residual (second)."""
    (M, K), n = x.shape, W.shape[1]
    code = N.F16 if x.dtype == torch.float16 else N.F32
    w_shift, y_shift = shift if isinstance(shift, tuple) else (0, shift)
    raw = torch.zeros(N.lib().TSB200_PackedWeightBytes(code, K, n) // x.element_size() + w_shift, device="cuda", dtype=x.dtype)
    Wp = raw[w_shift:]
    N.call("TSB200_PackWeight", 0, code, Wp.data_ptr(), W.data_ptr(), code, K, n, stream())
    No = n // 2 if act in (N.ACT_GLU_NOACT, N.ACT_SWIGLU) else n
    out = torch.full((M * No + y_shift + 1,), -7.0, device="cuda", dtype=torch.float32 if f32_out else x.dtype)
    y = out[y_shift:y_shift + M * No]
    if residual is not None:
        r = torch.zeros(M * No + y_shift, device="cuda")
        r[y_shift:] = residual.reshape(-1)
        residual = r[y_shift:]
    ws = torch.empty(N.lib().TSB200_LinearPackedWorkspaceBytes(code, M, K, n), dtype=torch.uint8, device="cuda")
    N.call("TSB200_LinearPacked", 0, code, None if f32_out else y.data_ptr(), y.data_ptr() if f32_out else None, x.data_ptr(), None, None, None, -1, 0.0, Wp.data_ptr(),
           bias.data_ptr() if bias is not None else None, residual.data_ptr() if residual is not None else None, M, K, n, act, ws.data_ptr(), ws.numel(), stream())
    torch.cuda.synchronize()
    assert (out[:y_shift] == -7.0).all() and out[y_shift + M * No] == -7.0       # nothing beside the output
    return y.reshape(M, No)


def check(M, K, n, dtype, shifts):
    rng = np.random.default_rng(M * 7919 + K * 31 + n)
    x, W = dev(rng.standard_normal((M, K)).astype(np.float32), dtype), dev((rng.standard_normal((K, n)) * 0.05).astype(np.float32), dtype)
    b, res = dev((rng.standard_normal(n) * 0.1).astype(np.float32), dtype), dev(rng.standard_normal((M, n)).astype(np.float32))
    ref = host(x).astype(np.float64) @ host(W).astype(np.float64) + host(b)
    # fp32 sums of K products, every rounding at its largest; a 16-bit output is rounded once more
    tol = K * 2.0 ** -23 * float(np.abs(host(x)).max() * np.abs(host(W)).max()) + 1e-6
    half = 2.0 ** -11 if dtype == torch.float16 else 0.0
    big = max(1.0, float(np.abs(ref).max()))
    for s in shifts:
        got = host(linear(x, W, b, N.ACT_NONE, shift=s))
        np.testing.assert_allclose(got, ref, atol=tol + half * big)
        np.testing.assert_array_equal(host(linear(x, W, b, N.ACT_NONE, shift=s)), got)
        np.testing.assert_allclose(host(linear(x, W, None, N.ACT_NONE, residual=res, f32_out=True, shift=s)), ref - host(b) + host(res), atol=tol + 1e-6)
        np.testing.assert_allclose(host(linear(x, W, b, N.ACT_RELU, shift=s)), np.maximum(ref, 0), atol=tol + half * big)
        if n % 2 == 0:
            np.testing.assert_allclose(host(linear(x, W, b, N.ACT_GLU_NOACT, shift=s)), ref[:, 0::2] * ref[:, 1::2], atol=2 * tol * big + half * big * big)


# 8 k: one step of one rank; 264 and 4104: a last pair with one tile; 1024 columns and fewer: eight ranks; 20000: one
@pytest.mark.parametrize("M,K,n", [(5, 8, 5), (8, 264, 130), (16, 4104, 1024), (17, 72, 516), (31, 1024, 127), (33, 512, 128), (48, 4096, 260), (64, 64, 64), (64, 136, 20000),
                                   (64, 2048, 2050), (63, 11008, 384)])
def test_fp16_rows(cuda, M, K, n):
    check(M, K, n, torch.float16, (0, 1))


# 8 rows of 11008: one CTA per SM; 33, 100, 4097: K ends inside a tile; 4096 -> 130: eight ranks, the ring of five tiles wraps
@pytest.mark.parametrize("M", [5, 6, 7, 8])
@pytest.mark.parametrize("K,n", [(4, 5), (33, 127), (100, 130), (4097, 128), (4096, 130), (512, 2000), (96, 20000), (11008, 260)])
def test_fp32_rows(cuda, M, K, n):
    check(M, K, n, torch.float32, (0, 1))


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("M", [1, 3, 8, 20, 70])
def test_weights_off_a_16_byte_boundary(cuda, dtype, M):
    """No kernel that copies whole pieces may take them."""
    check(M, 64, 130, dtype, ((1, 0),))


# sums travel four rows at a time: quads with one to four rows that exist, groups of four columns that share a bank, eight ranks and one
@pytest.mark.parametrize("M,K,n", [(1, 8, 4), (1, 4096, 512), (2, 2048, 132), (3, 520, 2052), (4, 264, 1024), (7, 1024, 40000), (9, 4096, 128), (61, 136, 256)])
def test_row_quads(cuda, M, K, n):
    check(M, K, n, torch.float16, (0, 1))


# 65 to 128 rows and 6144 k or more: K slices, whose sums the last CTA of a tile adds; a slice that ends in half a step, ragged rows, both epilogues
@pytest.mark.parametrize("M,K,n", [(65, 6144, 300), (100, 11008, 4096), (127, 6152, 130), (128, 8200, 2048)])
def test_k_slices(cuda, M, K, n):
    check(M, K, n, torch.float16, (0, 1))
