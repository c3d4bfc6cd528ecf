"""What a captured step reads before the launch in front of it has ended (cached rows of earlier positions, the step state) and what a linear does
before its products (the norm of fp32 rows): against engines that do neither."""
import numpy as np
import pytest

from seq2seqsharp_b200.gpt import (ActivateFuncEnums, DecodingOptions, DecodingStrategyEnums, GPT, GPTConfig, MultiHeadAttentionTypeEnums, NormEnums, PositionEmbeddingEnums,
                                   synthetic_weights)
from tests import gunuvik_models as GM, layered_models as LM, test_gunuvik_gpu as GG, test_layered_gpu as LG

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


# 64 to 1024: normed by the linears (a lane's registers full at 1024), 5 rows and more only below 512; 1056: by a launch
@pytest.mark.parametrize("d,H,B,norm", [(64, 1, 1, "LayerNorm"), (64, 1, 8, "RMSNorm"), (416, 13, 2, "LayerNorm"), (512, 8, 1, "LayerNorm"), (448, 7, 8, "LayerNorm"), (512, 8, 5, "RMSNorm"), (1024, 16, 4, "RMSNorm"),
                                        (1024, 16, 8, "LayerNorm"), (1056, 33, 3, "LayerNorm")])
def test_fp32_rows_normed_by_the_linear(cuda, oracle, monkeypatch, d, H, B, norm):
    cfg = GPTConfig(L=2, d=d, H=H, hd=d // H, F=192, V=515, norm=getattr(NormEnums, norm), act=ActivateFuncEnums.ReLU, pe=PositionEmbeddingEnums.RoPE,
                    attn=MultiHeadAttentionTypeEnums.MHA, dtype="float32")
    w = synthetic_weights(cfg, 7, std=0.05, bias_std=0.02)
    prompt = np.random.default_rng(d).integers(1, cfg.V, size=(B, 9)).astype(np.int32)
    opts, logits = DecodingOptions(MaxTgtSentLength=20), []
    fed = [np.arange(B, dtype=np.int32) + 3 + i for i in range(3)]
    for fused in ("1", "0"):
        monkeypatch.setenv("TSB200_FUSED_STEP", fused)
        gpt = GPT(cfg, max_batch=B, max_tokens=24)
        gpt.LoadWeights(w)
        gpt.Prefill(prompt, opts)
        for ids in fed:
            gpt.StepHost(ids, opts)
        logits.append(gpt.Logits()[0].copy())
    assert np.abs(logits[0] - logits[1]).max() <= 1e-5 * np.abs(logits[1]).max()      # fp32 sums of the rows in another order
    orc = oracle.OracleGPT(cfg, w, max_pos=24, threads=4)
    ref = orc.step(prompt)[0]
    for ids in fed:
        ref = orc.step(ids[:, None])[0]
    assert np.abs(logits[0] - ref).max() <= 1e-3 * np.abs(ref).max()                  # the bound of the token loop's tests


def steps_from(g, ids, at, n):
    """Logits of positions at .. at + n - 1: a prompt of `at` tokens, then n steps."""
    opts, rows = DecodingOptions(DecodingStrategy=DecodingStrategyEnums.GreedySearch), []
    g.Reset()
    g.SlotLogits(0, ids[:at], [])
    for t in ids[at:at + n]:
        g.StepHost([t], opts)
        rows.append(g.Logits(want_probs=False)[0][0])
    return rows


# stages of 32 cached rows: the new position opens one, closes one, or lies in its middle
@pytest.mark.parametrize("at", [1, 31, 32, 33, 63, 64, 65, 95, 96, 127, 128, 129, 191, 192])
def test_the_newest_row_of_the_latent_cache(cuda, at):
    """The token on which the answer hangs is the first that is decoded: its own step reads the row that the launch in front has appended, the next ones read it early."""
    cfg, w, ids = LG._needle(at=at)
    want = LM.oracle(cfg, w).forward(ids)[at:at + 4]
    g = LG.engine(cfg, w, "bfloat16")
    assert LM.rel(steps_from(g, ids, at, 4), want) < LM.TOL["bfloat16"]
    g.close()


# stages of 64; windows that have not begun to leave rows out, do so at this step, and did before; first rows that are kept in front of them
@pytest.mark.parametrize("window,keep", [(16, 4), (64, 0), (65, 17), (130, 1), (5, 70)])
def test_the_newest_row_of_grouped_attention(cuda, window, keep):
    n = 210
    for at in sorted({1, 15, 16, 63, 64, 65, 127, 128, 129, window - 1, window, window + 1, keep, keep + 1, 192} - {0}):
        cfg, w, ids = GM.needle(at, n, window, keep, layers=2)
        want = GM.Expected(cfg, w, ids, "bfloat16")
        g = GG.engine(cfg, w, "bfloat16")
        assert want.worst(steps_from(g, ids, at, 4), slice(at, at + 4)) < 1, at
        g.close()
