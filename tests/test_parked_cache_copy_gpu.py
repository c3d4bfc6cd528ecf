"""Parked caches are copied by one launch for up to 64 parts, 32 KB of a row per CTA: rows of several pieces, and more parts than one launch
takes.  A restored cache must continue bit for bit as the one that was parked, whatever the engine held in between."""
import numpy as np
import pytest

from seq2seqsharp_b200.gpt import (ActivateFuncEnums, DecodingOptions, GPT, GPTConfig, MultiHeadAttentionTypeEnums, NormEnums, PositionEmbeddingEnums,
                                   synthetic_weights)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,hd,S,dtype", [(1, 128, 127, "float16"), (2, 128, 128, "float16"), (1, 64, 700, "float16"), (2, 64, 513, "float32"),   # 1 .. 5 pieces
                                          (33, 64, 40, "float16"), (65, 64, 5, "float16")])                                                      # 66 and 130 parts
def test_a_restored_cache_continues_bit_for_bit(cuda, L, hd, S, dtype):
    cfg = GPTConfig(L=L, d=hd, H=1, hd=hd, F=64, V=211, norm=NormEnums.RMSNorm, act=ActivateFuncEnums.ReLU, pe=PositionEmbeddingEnums.RoPE,
                    attn=MultiHeadAttentionTypeEnums.MHA, dtype=dtype)
    B, n = 3, 4
    opts = DecodingOptions(MaxTgtSentLength=S + n)
    gpt = GPT(cfg, max_batch=B, max_tokens=S + n + 2)
    gpt.LoadWeights(synthetic_weights(cfg, 5, std=0.05))
    rng = np.random.default_rng(S)
    prompt, other = (rng.integers(1, cfg.V, size=(B, S)).astype(np.int32) for _ in range(2))
    fed = [np.arange(B, dtype=np.int32) + 3 * i + 1 for i in range(n)]

    def go_on():
        out = []
        for ids in fed:
            gpt.StepHost(ids, opts)
            out.append(gpt.Logits(want_probs=False)[0].copy())
        return out
    gpt.Prefill(prompt, opts)
    snap = gpt.CacheSnapshot()
    want = go_on()
    gpt.Reset()
    gpt.Prefill(other, opts)       # other rows everywhere
    gpt.CacheRestore(snap)
    for a, b in zip(want, go_on()):
        np.testing.assert_array_equal(a, b)
    gpt.close()
