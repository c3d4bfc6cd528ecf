"""Linears at the edges of the rules that choose their kernels: fp32 rows beyond 16 (clusters over K), deep and shallow rings of the tensor-core
kernel, and the engine's step with rotation and append in the q | k | v epilogue at widths of all kinds."""
import numpy as np
import pytest
import torch

from seq2seqsharp_b200 import _native as N
from tests.test_fused_gpu import dev, host, linear_packed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,K,Nn", [(17, 4, 8), (32, 512, 2048), (33, 2048, 512), (64, 100, 130), (65, 96, 64), (200, 132, 1001), (1000, 512, 1536), (40, 36, 5), (20, 131, 72)])
def test_fp32_rows(cuda, oracle, M, K, Nn):
    rng = np.random.default_rng(M + K + Nn)
    x, W = dev(rng.standard_normal((M, K)).astype(np.float32)), dev((rng.standard_normal((K, Nn)) * 0.05).astype(np.float32))
    b, res = dev((rng.standard_normal((1, Nn)) * 0.1).astype(np.float32)), dev(rng.standard_normal((M, Nn)).astype(np.float32))
    ref = host(x).astype(np.float64) @ host(W).astype(np.float64) + host(b)
    tol = K * 2.0 ** -23 * float(np.abs(host(x)).max() * np.abs(host(W)).max()) + 1e-6     # every one of K roundings at its largest
    got = host(linear_packed(x, W, b, N.ACT_NONE))
    np.testing.assert_allclose(got, ref, atol=tol)
    np.testing.assert_array_equal(host(linear_packed(x, W, b, N.ACT_NONE)), got)
    np.testing.assert_allclose(host(linear_packed(x, W, b, N.ACT_NONE, residual=res, want_f32=True)), ref + host(res), atol=tol)
    np.testing.assert_allclose(host(linear_packed(x, W, b, N.ACT_RELU)), np.maximum(ref, 0), atol=tol)
    if Nn % 2 == 0:
        np.testing.assert_allclose(host(linear_packed(x, W, b, N.ACT_GLU_NOACT)), ref[:, 0::2] * ref[:, 1::2], atol=2 * tol * max(1.0, np.abs(ref).max()))


@pytest.mark.parametrize("M,K,Nn", [(129, 32, 128), (129, 96, 160), (256, 1056, 2048), (257, 256, 1009), (1300, 128, 1920), (1301, 128, 2048), (70, 4096, 512), (2000, 2080, 2592)])
def test_tensor_core_epilogues(cuda, oracle, M, K, Nn):
    """fp16: every activation with whole and broken groups of 32 columns, 16-bit and fp32 outputs, few tiles (deep rings) and many."""
    rng = np.random.default_rng(M + K + Nn)
    x = dev((rng.standard_normal((M, K)) * 0.5).astype(np.float32), torch.float16)
    W, b = dev((rng.standard_normal((K, Nn)) * 0.05).astype(np.float32), torch.float16), dev((rng.standard_normal((1, Nn)) * 0.1).astype(np.float32), torch.float16)
    ref = host(x).astype(np.float64) @ host(W).astype(np.float64) + host(b)
    scale = max(1.0, float(np.abs(ref).max()))
    tol = 2.0 ** -10 * scale       # the output's rounding to fp16, and as much again for the sums
    for act, kind in ((N.ACT_NONE, None), (N.ACT_RELU, 0), (N.ACT_SILU, 1), (N.ACT_LEAKYRELU, 2), (N.ACT_GELU, 5)):
        want = ref if kind is None else oracle.act(ref.astype(np.float32), kind)
        np.testing.assert_allclose(host(linear_packed(x, W, b, act, dtype=torch.float16)), want, atol=tol)
    res = dev(rng.standard_normal((M, Nn)).astype(np.float32))
    np.testing.assert_allclose(host(linear_packed(x, W, b, N.ACT_NONE, residual=res, dtype=torch.float16, want_f32=True)), ref + host(res), atol=tol)
    if Nn % 2 == 0:
        a, g = ref[:, 0::2], ref[:, 1::2]
        np.testing.assert_allclose(host(linear_packed(x, W, b, N.ACT_GLU_NOACT, dtype=torch.float16)), a * g, atol=tol * scale)
        np.testing.assert_allclose(host(linear_packed(x, W, b, N.ACT_SWIGLU, dtype=torch.float16)), oracle.act(a.astype(np.float32), 1) * g, atol=tol * scale)


@pytest.mark.parametrize("d,H,B,norm", [(64, 1, 8, "LayerNorm"), (320, 5, 3, "RMSNorm"), (768, 12, 8, "LayerNorm"), (992, 31, 7, "RMSNorm"), (1056, 33, 8, "LayerNorm"),
                                        (2080, 65, 4, "RMSNorm")])
def test_rotation_and_append_in_the_epilogue_at_any_width(cuda, oracle, monkeypatch, d, H, B, norm):
    """The captured step with rotation and append in the epilogue of q | k | v against the same step with a launch for them; norms, which are
    launches in both, and all else against the oracle."""
    from seq2seqsharp_b200.gpt import (ActivateFuncEnums, DecodingOptions, GPT, GPTConfig, MultiHeadAttentionTypeEnums, NormEnums, PositionEmbeddingEnums, synthetic_weights)
    cfg = GPTConfig(L=2, d=d, H=H, hd=d // H, F=256, V=515, norm=getattr(NormEnums, norm), act=ActivateFuncEnums.GELU, pe=PositionEmbeddingEnums.RoPE,
                    attn=MultiHeadAttentionTypeEnums.MHA, dtype="float16")
    w = synthetic_weights(cfg, 7, std=0.05, bias_std=0.02)
    prompt = np.random.default_rng(d).integers(1, cfg.V, size=(B, 9)).astype(np.int32)
    opts = DecodingOptions(MaxTgtSentLength=20)
    logits, fed = [], [np.arange(B, dtype=np.int32) + 3 + i for i in range(3)]
    for fused in ("1", "0"):
        monkeypatch.setenv("TSB200_FUSED_STEP", fused)
        gpt = GPT(cfg, max_batch=B, max_tokens=24)
        gpt.LoadWeights(w)
        gpt.Prefill(prompt, opts)
        for ids in fed:
            gpt.StepHost(ids, opts)
        logits.append(gpt.Logits()[0].copy())
    # the same kernels sum in the same order, and the value is rounded to fp16 before it is rotated in both
    assert np.abs(logits[0] - logits[1]).max() <= 4 * 2.0 ** -11 * np.abs(logits[1]).max()
    orc = oracle.OracleGPT(cfg, w, max_pos=24, threads=4)
    ref = orc.step(prompt)[0]
    for ids in fed:
        ref = orc.step(ids[:, None])[0]
    for got in logits:      # fp16 weights and activations through two layers: the bound of the token loop's tests
        assert np.abs(got - ref).max() <= 2e-2 * np.abs(ref).max()
