"""Decode attention whose splits meet in a cluster (two to eight of them) or through records: against float64, for every kernel that does it,
and in an engine whose short sequence leaves splits without keys."""
import numpy as np
import pytest
import torch

from seq2seqsharp_b200 import _native as N
from seq2seqsharp_b200.gpt import (ActivateFuncEnums, DecodingOptions, GPT, GPTConfig, MultiHeadAttentionTypeEnums, NormEnums, PositionEmbeddingEnums,
                                   synthetic_weights)

pytestmark = pytest.mark.gpu


# keys: 2, 3, 5, 7, 8 and more than eight splits of one or two KV heads (fp16 of 64 / 128: 256 keys per split, else 32)
CASES = [(torch.float16, hd, T) for hd in (64, 128) for T in (257, 700, 1281, 1700, 2048, 4000)] + \
        [(t, hd, T) for t, hd in ((torch.float16, 32), (torch.float32, 64), (torch.float32, 32)) for T in (33, 90, 150, 220, 256, 700)]


@pytest.mark.parametrize("G", [1, 2, 4, 8])
@pytest.mark.parametrize("dtype,hd,T", CASES)
def test_splits_against_float64(cuda, dtype, hd, T, G):
    B, Hkv, Tmax = 2, 1, T + 5
    H = G * Hkv
    g = torch.Generator("cuda")
    g.manual_seed(T + hd + G)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).to(dtype)  # noqa: E731
    q, k, v = rnd(B, H * hd), torch.full((B, Hkv, Tmax, hd), float("nan"), device="cuda", dtype=dtype), torch.full((B, Hkv, Tmax, hd), float("nan"), device="cuda", dtype=dtype)
    k[:, :, :T], v[:, :, :T] = rnd(B, Hkv, T, hd), rnd(B, Hkv, T, hd)
    o = torch.empty_like(q)
    ws = torch.empty(N.lib().TSB200_FlashDecodeWorkspaceBytes(B, H, hd, T), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    call = lambda: N.call("TSB200_FlashDecode", 0, N.F16 if dtype == torch.float16 else N.F32, o.data_ptr(), q.data_ptr(), H * hd, k.data_ptr(), v.data_ptr(), B, H, Hkv,  # noqa: E731
                          hd, T, Tmax, ws.data_ptr(), ws.numel(), None)
    call()
    N.call("TSB200_Synchronize", 0, None)
    z = torch.einsum("bkgd,bktd->bkgt", q.double().reshape(B, Hkv, G, hd), k[:, :, :T].double()) * hd ** -0.5
    ref = torch.einsum("bkgt,bktd->bkgd", z.softmax(-1), v[:, :, :T].double()).reshape(B, H * hd)
    # fp16: weights and outputs of at most 5 are rounded to 2^-11 of themselves; fp32: exponents of up to 30 to 2^-24, the exponential to 2^-21
    tol = 2 * 5 * 2.0 ** -11 if dtype == torch.float16 else 5 * 2.0 ** -18
    assert (o.double() - ref).abs().max().item() <= tol
    first = o.clone()
    call()
    N.call("TSB200_Synchronize", 0, None)
    assert torch.equal(first, o)


@pytest.mark.parametrize("hd,dtype", [(64, "float16"), (128, "float16"), (64, "float32")])
def test_a_short_sequence_leaves_splits_without_keys(cuda, hd, dtype):
    cfg = GPTConfig(L=2, d=2 * hd, H=2, Hkv=1, hd=hd, F=256, V=501, norm=NormEnums.RMSNorm, act=ActivateFuncEnums.SwiGLU, pe=PositionEmbeddingEnums.RoPE,
                    attn=MultiHeadAttentionTypeEnums.GQA, dtype=dtype)
    w = synthetic_weights(cfg, 3, std=0.05)
    opts = DecodingOptions(MaxTgtSentLength=1200)
    rng = np.random.default_rng(hd)
    texts = [rng.integers(1, cfg.V, size=n).astype(np.int32) for n in (1100, 3)]      # splits for 2048 keys; three keys
    feed = np.array([5, 9], dtype=np.int32)

    def run(prompts, ids):
        gpt = GPT(cfg, max_batch=len(prompts), max_tokens=1200)
        gpt.LoadWeights(w)
        gpt.PrefillRagged(prompts, opts)
        for i in range(2):
            gpt.StepHost(ids + i, opts)
        out = gpt.Logits(want_probs=False)[0]
        gpt.close()
        return out
    both = run(texts, feed)
    for b in range(2):
        alone = run(texts[b:b + 1], feed[b:b + 1])
        # the same sums in another order, through two layers of 16-bit (32-bit) activations
        assert np.abs(both[b] - alone[0]).max() <= (8 * 2.0 ** -11 if dtype == "float16" else 1e-5) * np.abs(alone).max()
