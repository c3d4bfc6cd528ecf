"""Causal prompt attention on tcgen05 against float64, at the edges of its tiles: 128 rows of (query, head) pairs and 128 keys, one or two
row tiles per CTA, prompts on top of cached tokens, and cache rows beyond the prompt that hold NaN."""
import numpy as np
import pytest
import torch

from seq2seqsharp_b200 import _native as N
from tests.test_fused_gpu import stream

pytestmark = pytest.mark.gpu

# Weights and outputs are rounded to fp16 (2^-11 each, relative); values are N(0, 1), so an output is at most about 5.
TOL = 2 * 5 * 2.0 ** -11


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("H,Hkv", [(4, 4), (4, 2), (8, 2), (8, 1)])
@pytest.mark.parametrize("S,T0", [(16, 0), (31, 100), (64, 64), (65, 63), (127, 1), (129, 0), (257, 128)])
def test_against_float64(cuda, hd, H, Hkv, S, T0):
    B, Tmax = 2, T0 + S + 3
    g = torch.Generator("cuda")
    g.manual_seed(S * 31 + H)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).half()  # noqa: E731
    Nq = (H + 2 * Hkv) * hd
    q = rnd(B, S, Nq)
    cK = torch.full((B, Hkv, Tmax, hd), float("nan"), device="cuda", dtype=torch.float16)
    cV = cK.clone()
    cK[:, :, :T0 + S], cV[:, :, :T0 + S] = rnd(B, Hkv, T0 + S, hd), rnd(B, Hkv, T0 + S, hd)
    k, v = (c[:, :, :T0 + S].double().repeat_interleave(H // Hkv, 1) for c in (cK, cV))
    z = q[:, :, :H * hd].reshape(B, S, H, hd).transpose(1, 2).double() @ k.transpose(2, 3) * hd ** -0.5
    seen = torch.arange(T0 + S, device="cuda")[None] <= T0 + torch.arange(S, device="cuda")[:, None]
    ref = (z.masked_fill(~seen, float("-inf")).softmax(-1) @ v).transpose(1, 2)
    for shift in (0, 2):    # an output on a 16-byte boundary, and on one of 4 bytes
        raw = torch.zeros(B * S * H * hd + 8, device="cuda", dtype=torch.float16)
        out = raw[shift:shift + B * S * H * hd]
        torch.cuda.synchronize()
        N.call("TSB200_PrefillAttention", 0, N.F16, out.data_ptr(), q.data_ptr(), Nq, cK.data_ptr(), cV.data_ptr(), B, S, H, Hkv, hd, T0, Tmax, stream())
        torch.cuda.synchronize()
        np.testing.assert_allclose(out.reshape(B, S, H, hd).double().cpu().numpy(), ref.cpu().numpy(), atol=TOL)
        assert raw[:shift].abs().sum() == 0 and raw[shift + B * S * H * hd:].abs().sum() == 0


@pytest.mark.parametrize("hd,H,Hkv,S,T0", [(64, 4, 4, 16, 48), (64, 4, 4, 16, 49), (64, 8, 1, 64, 64), (64, 8, 2, 65, 64), (64, 12, 12, 128, 0), (128, 8, 2, 64, 0), (128, 8, 2, 100, 28),
                                            (128, 8, 4, 65, 0), (128, 8, 8, 64, 0), (128, 8, 8, 65, 0), (128, 8, 1, 129, 0)])
def test_at_the_limits_of_short_prompts(cuda, hd, H, Hkv, S, T0):
    """Keys and heads at both sides of the rule that chooses between mma.sync and tcgen05."""
    test_against_float64(cuda, hd, H, Hkv, S, T0)


@pytest.mark.parametrize("B", [37, 75])      # 16 rows on top of 130 keys, 8 KV heads: within and beyond two waves of whole SMs
def test_many_short_prompts_on_a_cache(cuda, B):
    H, Hkv, hd, S, T0 = 8, 8, 64, 16, 130
    q = torch.randn(B, S, H * hd, device="cuda").half()
    k, v = (torch.randn(B, Hkv, T0 + S, hd, device="cuda").half() for _ in range(2))
    o = torch.empty_like(q)
    torch.cuda.synchronize()
    N.call("TSB200_PrefillAttention", 0, N.F16, o.data_ptr(), q.data_ptr(), H * hd, k.data_ptr(), v.data_ptr(), B, S, H, Hkv, hd, T0, T0 + S, None)
    N.call("TSB200_Synchronize", 0, None)
    z = q.reshape(B, S, H, hd).transpose(1, 2).double() @ k.double().transpose(2, 3) * hd ** -0.5
    seen = torch.arange(T0 + S, device="cuda")[None] <= T0 + torch.arange(S, device="cuda")[:, None]
    ref = (z.masked_fill(~seen, float("-inf")).softmax(-1) @ v.double()).transpose(1, 2).reshape(B, S, H * hd)
    assert (o.double() - ref).abs().max().item() <= TOL
