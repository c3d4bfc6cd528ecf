"""Prompts whose rows each take a CTA (fp32, and fp16 head sizes or groups that no tensor-core kernel takes) against float64: groups of every width, keys around
the tokens that four warps of lane groups see at a time, cached tokens in front, NaN behind."""
import numpy as np
import pytest
import torch

from seq2seqsharp_b200 import _native as N
from tests.test_fused_gpu import stream

pytestmark = pytest.mark.gpu


# hd 64 fp32: 8 tokens at a time; 16 fp16: 64; 256 fp16: 4; 16 / 1 heads: a group of 16 in two CTAs
@pytest.mark.parametrize("dtype,H,Hkv,hd", [("float32", 3, 3, 64), ("float32", 4, 2, 64), ("float32", 4, 1, 128), ("float32", 16, 2, 32), ("float16", 3, 3, 16), ("float16", 4, 2, 32),
                                            ("float16", 4, 1, 256), ("float16", 16, 1, 64)])
@pytest.mark.parametrize("S,T0", [(2, 0), (7, 1), (9, 7), (17, 8), (33, 31), (65, 64), (130, 3)])
def test_against_float64(cuda, dtype, H, Hkv, hd, S, T0):
    B, Tmax, t = 2, T0 + S + 3, getattr(torch, dtype)
    g = torch.Generator("cuda")
    g.manual_seed(S * 31 + H)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).to(t)  # noqa: E731
    q, out = rnd(B, S, H * hd), torch.zeros(B, S, H, hd, device="cuda", dtype=t)
    cK, cV = (torch.full((B, Hkv, Tmax, hd), float("nan"), device="cuda", dtype=t) for _ in range(2))
    cK[:, :, :T0 + S], cV[:, :, :T0 + S] = rnd(B, Hkv, T0 + S, hd), rnd(B, Hkv, T0 + S, hd)
    k, v = (c[:, :, :T0 + S].double().repeat_interleave(H // Hkv, 1) for c in (cK, cV))
    z = q.reshape(B, S, H, hd).transpose(1, 2).double() @ k.transpose(2, 3) * hd ** -0.5
    seen = torch.arange(T0 + S, device="cuda")[None] <= T0 + torch.arange(S, device="cuda")[:, None]
    ref = (z.masked_fill(~seen, float("-inf")).softmax(-1) @ v).transpose(1, 2)
    torch.cuda.synchronize()
    N.call("TSB200_PrefillAttention", 0, N.F16 if dtype == "float16" else N.F32, out.data_ptr(), q.data_ptr(), H * hd, cK.data_ptr(), cV.data_ptr(), B, S, H, Hkv, hd, T0, Tmax, stream())
    torch.cuda.synchronize()
    # scores up to 30 with hd + 4 fp32 roundings, exponentials and T0 + S sums on top; values are at most 6; a 16-bit output is rounded once
    tol = 6 * (30 * (hd + 4) + T0 + S + 8) * 2.0 ** -24 + (6 * 2.0 ** -11 if dtype == "float16" else 0.0)
    np.testing.assert_allclose(out.double().cpu().numpy(), ref.cpu().numpy(), atol=tol)
