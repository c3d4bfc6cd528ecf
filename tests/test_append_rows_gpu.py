"""Rotation and append of prompts with more rows than twice the SMs (a CTA per row) against the same prompts one by one (rows shared out)."""
import numpy as np
import pytest
import torch

from seq2seqsharp_b200 import _native as N
from seq2seqsharp_b200.gpt import (ActivateFuncEnums, DecodingOptions, GPT, GPTConfig, MultiHeadAttentionTypeEnums, NormEnums, PositionEmbeddingEnums,
                                   synthetic_weights)

pytestmark = pytest.mark.gpu


# rows of 144, 384, 512, 544 (a third pass that is not full), 768 and 960 (four passes) pieces; lengths that differ lie one after the other with cleared positions behind each
@pytest.mark.parametrize("H,Hkv,hd,dtype", [(14, 2, 64, "float16"), (32, 8, 64, "float16"), (24, 4, 128, "float16"), (30, 2, 128, "float16"), (48, 6, 128, "float16"), (32, 8, 128, "float16"), (8, 4, 64, "float32")])
@pytest.mark.parametrize("lens", [(140, 140, 140), (190, 33, 171)])
def test_many_rows_against_few(cuda, H, Hkv, hd, dtype, lens):
    cfg = GPTConfig(L=2, d=H * hd, H=H, Hkv=Hkv, hd=hd, F=256, V=501, norm=NormEnums.RMSNorm, act=ActivateFuncEnums.SwiGLU, pe=PositionEmbeddingEnums.RoPE,
                    attn=MultiHeadAttentionTypeEnums.GQA, dtype=dtype)
    w, rng, opts = synthetic_weights(cfg, 3, std=0.02), np.random.default_rng(hd), DecodingOptions(MaxTgtSentLength=200)
    texts = [rng.integers(1, cfg.V, size=n).astype(np.int32) for n in lens]

    def run(prompts):
        gpt = GPT(cfg, max_batch=len(prompts), max_tokens=200)
        gpt.LoadWeights(w)
        gpt.PrefillRagged(prompts, opts)
        gpt.StepHost(np.full(len(prompts), 7, dtype=np.int32), opts)
        out = gpt.Logits(want_probs=False)[0].copy()
        gpt.close()
        return out
    both = run(texts)
    for b, text in enumerate(texts):
        alone = run([text])
        # the same sums in another order, through two layers of 16-bit (32-bit) activations
        assert np.abs(both[b] - alone[0]).max() <= (8 * 2.0 ** -11 if dtype == "float16" else 1e-5) * np.abs(alone).max()


@pytest.mark.parametrize("S", [148, 149, 700])
def test_append_alone(cuda, S):
    B, H, Hkv, hd, T0 = 2, 16, 4, 64, 5
    g = torch.Generator("cuda")
    g.manual_seed(S)
    qkv = torch.randn(B * S, (H + 2 * Hkv) * hd, device="cuda", generator=g).half()
    before = qkv.clone()
    cK, cV = (torch.zeros(B, Hkv, T0 + S + 3, hd, device="cuda", dtype=torch.float16) for _ in range(2))
    at = lambda head: qkv.data_ptr() + head * hd * 2  # noqa: E731
    torch.cuda.synchronize()
    N.call("TSB200_RopeAppend", 0, N.F16, at(0), at(H), at(H + Hkv), qkv.shape[1], qkv.shape[1], cK.data_ptr(), cV.data_ptr(), B, S, H, Hkv, hd, T0, T0 + S + 3, 0, 10000.0, None)
    N.call("TSB200_Synchronize", 0, None)
    x = before.reshape(B, S, H + 2 * Hkv, hd).transpose(1, 2)
    assert torch.equal(qkv, before)
    for cache, first in ((cK, H), (cV, H + Hkv)):
        assert torch.equal(cache[:, :, T0:T0 + S], x[:, first:first + Hkv])
        assert not cache[:, :, :T0].any() and not cache[:, :, T0 + S:].any()
