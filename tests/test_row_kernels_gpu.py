"""Norms of whole rows in registers, rotation and append by 16-byte pieces, softmax on a cluster and the head of a nucleus, at the edges of
the rules that choose them."""
import numpy as np
import pytest
import torch

from seq2seqsharp_b200 import _native as N
from seq2seqsharp_b200.ops import Ops
from tests.test_fused_gpu import dev, host, stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 2e-5), (torch.float16, 4e-3)])   # 4e-3: two roundings to fp16 of values up to 8
@pytest.mark.parametrize("norm_type", [0, 1])
@pytest.mark.parametrize("M,d", [(1, 768), (3, 4096), (300, 2048), (700, 4096), (2, 4100), (301, 1028), (5, 12288), (4, 130), (2, 33)])
def test_norm_of_rows(cuda, oracle, dtype, tol, norm_type, M, d):
    rng = np.random.default_rng(M + d)
    x = dev((rng.standard_normal((M, d)) * 1.7 + 0.2).astype(np.float32))
    delta = dev((rng.standard_normal((M, d)) * 0.3).astype(np.float32), dtype)
    g, b = dev((1 + 0.1 * rng.standard_normal(d)).astype(np.float32), dtype), dev((0.1 * rng.standard_normal(d)).astype(np.float32), dtype)
    for dl, beta in ((None, b), (delta, None)):
        rows = x.clone()
        h = torch.empty(M, d, device="cuda", dtype=dtype)
        torch.cuda.synchronize()
        N.call("TSB200_NormResidual", 0, N.F16 if dtype == torch.float16 else N.F32, h.data_ptr(), rows.data_ptr(), dl.data_ptr() if dl is not None else None, g.data_ptr(),
               beta.data_ptr() if beta is not None else None, norm_type, 1e-6, M, d, stream())
        want = host(x) + (host(dl) if dl is not None else 0.0)
        np.testing.assert_allclose(host(rows), want, atol=1e-6)
        bh = host(beta) if beta is not None else None
        ref = oracle.layernorm(want, host(g), bh if bh is not None else np.zeros(d, np.float32), 1e-6) if norm_type == 0 else oracle.rmsnorm(want, host(g), bh, 1e-6)
        np.testing.assert_allclose(host(h), ref, atol=tol * max(1.0, float(np.abs(ref).max()) / 4))


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 2e-5), (torch.float16, 4e-3)])   # 4e-3: rounding to fp16 of values up to 5
@pytest.mark.parametrize("hd,shift", [(64, 0), (64, 2), (6, 0), (8, 0), (12, 0)])      # 16-byte pieces; an odd boundary or head size: pairs
def test_rotation_and_append(cuda, dtype, tol, hd, shift):
    B, S, H, Hkv, T0, Tmax = 2, 5, 4, 2, 3, 11
    Nq, dt = (H + 2 * Hkv) * hd, N.F16 if dtype == torch.float16 else N.F32
    rng = np.random.default_rng(hd + shift)
    qkv0 = rng.standard_normal((B, S, Nq)).astype(np.float32)
    raw = torch.zeros(B * S * Nq + shift, device="cuda", dtype=dtype)
    raw[shift:] = dev(qkv0.reshape(-1), dtype)
    qkv = raw[shift:].reshape(B, S, Nq)
    before = host(qkv).astype(np.float64)
    cK, cV = (torch.zeros(B, Hkv, Tmax, hd, device="cuda", dtype=dtype) for _ in range(2))
    es = qkv.element_size()
    torch.cuda.synchronize()
    N.call("TSB200_RopeAppend", 0, dt, qkv.data_ptr(), qkv.data_ptr() + H * hd * es, qkv.data_ptr() + (H + Hkv) * hd * es, Nq, Nq, cK.data_ptr(), cV.data_ptr(), B, S, H,
           Hkv, hd, T0, Tmax, 1, 10000.0, stream())
    x = before.reshape(B, S, H + 2 * Hkv, hd)
    angle = (T0 + np.arange(S))[:, None] * 10000.0 ** (-2.0 * np.arange(hd // 2) / hd)
    c, s = np.cos(angle)[None, :, None], np.sin(angle)[None, :, None]
    turned = np.stack((x[..., 0::2] * c - x[..., 1::2] * s, x[..., 1::2] * c + x[..., 0::2] * s), -1).reshape(x.shape)
    np.testing.assert_allclose(host(qkv).reshape(x.shape)[:, :, :H], turned[:, :, :H], atol=tol)
    np.testing.assert_allclose(host(cK)[:, :, T0:T0 + S], turned[:, :, H:H + Hkv].transpose(0, 2, 1, 3), atol=tol)
    np.testing.assert_array_equal(host(cV)[:, :, T0:T0 + S], x[:, :, H + Hkv:].transpose(0, 2, 1, 3).astype(np.float32))
    assert not host(cK)[:, :, T0 + S:].any() and not host(cV)[:, :, :T0].any()


@pytest.mark.parametrize("B,V", [(1, 4095), (1, 4096), (3, 4099), (2, 32769), (74, 32000), (75, 32000), (1, 65537), (1, 131072), (1, 131073)])
def test_softmax_and_first_maximum(cuda, oracle, B, V):
    rng = np.random.default_rng(V)
    z = (rng.standard_normal((B, V)) * 2).astype(np.float32)
    z[0, [7, V // 2, V - 1]] = z[0].max() + 1.0     # three equal maxima, in different parts of the row: the lowest index
    if B > 1:
        z[-1, 3:V // 3] = -np.inf
    blocked = dev(np.array([0, V - 1], dtype=np.int32))
    for t in (1.0, 0.7):
        ids, probs = torch.empty(B, dtype=torch.int32, device="cuda"), torch.empty(B, V, device="cuda")
        zd = dev(z)
        torch.cuda.synchronize()
        N.call("TSB200_SoftmaxArgmax", 0, ids.data_ptr(), probs.data_ptr(), zd.data_ptr(), B, V, t, blocked.data_ptr(), 2, stream())
        zt = (z / np.float32(t)).astype(np.float64)
        e = np.exp(zt - zt.max(1, keepdims=True))
        p = e / e.sum(1, keepdims=True)
        p[:, [0, V - 1]] -= 1.0
        # an exponent of up to 30 is rounded to 2^-24 of itself, the exponential to a few units in the last place
        np.testing.assert_allclose(host(probs), p, atol=1e-7, rtol=5e-6)
        np.testing.assert_array_equal(ids.cpu().numpy(), oracle.argmax(host(probs)))
        assert ids[0].item() == 7


@pytest.mark.parametrize("rows", [2, 40])      # a cluster per row; one CTA per row
@pytest.mark.parametrize("n", [1, 2, 5, 900, 1025, 2047, 2048, 2049, 3000])
def test_nuclei_around_the_selection_limit(cuda, oracle, rows, n):
    """n equal or nearly equal weights hold 0.96 of the mass: the nucleus of 0.9 is inside them, with ties in the order of their indexes."""
    V = 32000
    rng = np.random.default_rng(n)
    p = np.full((rows, V), 0.04 / (V - n), dtype=np.float32)
    for r in range(rows):
        at = rng.permutation(V)[:n]
        p[r, at] = (0.96 / n) * (1.0 if r % 2 else 1.0 + 0.3 * rng.random(n))
    u = rng.random(rows).astype(np.float32)
    for top in (0.5, 0.9, 0.9595, 2.0):
        out = Ops.TopPSample(torch.from_numpy(p).cuda(), top, 0.0, None, torch.from_numpy(u))
        torch.cuda.synchronize()
        np.testing.assert_array_equal(out.cpu().numpy(), oracle.topp(p, top, 0.0, None, u))
    big = p * np.float32(4.0)      # weights that add up to more than the selection's units hold
    out = Ops.TopPSample(torch.from_numpy(big).cuda(), 2.2, 0.0, None, torch.from_numpy(u))
    torch.cuda.synchronize()
    np.testing.assert_array_equal(out.cpu().numpy(), oracle.topp(big, 2.2, 0.0, None, u))


@pytest.mark.parametrize("B,V", [(1, 6143), (18, 6144), (19, 6144), (18, 7999), (37, 8000), (38, 8000), (38, 19999), (74, 20000), (74, 65536), (37, 65537), (38, 98304), (74, 98305)])
def test_softmax_at_the_limits_of_the_clusters(cuda, oracle, B, V):
    """Rows and widths at both sides of the rule that gives a row eight CTAs or one."""
    test_softmax_and_first_maximum(cuda, oracle, B, V)


def test_rotation_of_many_long_rows_with_a_table(cuda):
    """400 rows of 768 pieces, a CTA each, against 200 at a time, where a row is shared out: the engine's prompt pass, where the table is."""
    from seq2seqsharp_b200.gpt import (ActivateFuncEnums, DecodingOptions, GPT, GPTConfig, MultiHeadAttentionTypeEnums, NormEnums, PositionEmbeddingEnums, synthetic_weights)
    cfg = GPTConfig(L=1, d=2048, H=32, hd=64, F=256, V=515, norm=NormEnums.RMSNorm, act=ActivateFuncEnums.SwiGLU, pe=PositionEmbeddingEnums.RoPE,
                    attn=MultiHeadAttentionTypeEnums.MHA, dtype="float16")
    w = synthetic_weights(cfg, 9, std=0.05)
    prompt = np.random.default_rng(2).integers(1, cfg.V, size=(2, 200)).astype(np.int32)
    opts = DecodingOptions(MaxTgtSentLength=204)
    gpt = GPT(cfg, max_batch=2, max_tokens=206)
    gpt.LoadWeights(w)

    def run(p):
        gpt.Reset()
        gpt.Prefill(p, opts)
        gpt.StepHost(np.full(len(p), 7, np.int32), opts)     # attends over every appended row
        return gpt.Logits(want_probs=False)[0].copy()
    both, each = run(prompt), np.concatenate([run(prompt[i:i + 1]) for i in range(2)])
    assert np.abs(both - each).max() <= 8 * 2.0 ** -11 * np.abs(each).max()      # the linears' sums in another order, rounded to fp16 through one layer
