"""What a captured step reads before the launch in front of it has ended: cached rows of earlier positions and the step state."""
import numpy as np
import pytest

from seq2seqsharp_b200.gpt import (ActivateFuncEnums, DecodingOptions, GPT, GPTConfig, MultiHeadAttentionTypeEnums, NormEnums, PositionEmbeddingEnums,
                                   synthetic_weights)

pytestmark = pytest.mark.gpu


# the row of the new position opens a stage of 64 (fp16) or a lane group's next token (fp32), closes one, or lies in the middle; one split and several
@pytest.mark.parametrize("hd,dtype,lens", [(64, "float16", (1, 62, 63, 64, 65, 127, 128, 319, 576)), (128, "float16", (63, 64, 129)),
                                           (64, "float32", (1, 7, 8, 9, 31, 32, 33, 63, 64, 100)), (32, "float32", (15, 16, 17, 65))])
def test_cached_rows_around_the_new_position(cuda, hd, dtype, lens):
    cfg = GPTConfig(L=2, d=4 * hd, H=4, Hkv=2, hd=hd, F=256, V=501, norm=NormEnums.RMSNorm, act=ActivateFuncEnums.SwiGLU, pe=PositionEmbeddingEnums.RoPE,
                    attn=MultiHeadAttentionTypeEnums.GQA, dtype=dtype)
    opts = DecodingOptions(MaxTgtSentLength=max(lens) + 8)
    gpt = GPT(cfg, max_batch=3, max_tokens=max(lens) + 8)
    gpt.LoadWeights(synthetic_weights(cfg, 5, std=0.05))
    for T in lens:
        text = np.random.default_rng(T).integers(1, cfg.V, size=(3, T + 3)).astype(np.int32)
        gpt.Reset()
        gpt.Prefill(text[:, :T], opts)
        for i in range(3):
            gpt.StepHost(text[:, T + i], opts)
        stepped = gpt.Logits(want_probs=False)[0].copy()
        gpt.Reset()
        gpt.Prefill(text, opts)
        whole = gpt.Logits(want_probs=False)[0]
        # the same sums in another order, through two layers of 16-bit (32-bit) activations
        assert np.abs(stepped - whole).max() <= (8 * 2.0 ** -11 if dtype == "float16" else 1e-5) * np.abs(whole).max()
