"""Calls at both sides of a rule that chooses a kernel: the smaller one must not cost clearly more than its neighbour.  Times are the smallest
of several replays of a captured row of calls, both sides in turn; the limits leave room for noise, not for the wrong kernel."""
import pytest
import torch

from seq2seqsharp_b200 import _native as N

pytestmark = pytest.mark.gpu


def times(*calls, n=10):
    """us per call of each of `calls` (functions of a stream)."""
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    graphs, best = [], [1e9] * len(calls)
    with torch.cuda.stream(s):
        for f in calls:
            f(s.cuda_stream)
            s.synchronize()
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=s):
                for _ in range(n):
                    f(torch.cuda.current_stream().cuda_stream)
            graphs.append(g)
        for _ in range(8):
            for i, g in enumerate(graphs):
                a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
                a.record(s)
                g.replay()
                b.record(s)
                s.synchronize()
                best[i] = min(best[i], a.elapsed_time(b) * 1000.0 / n)
    return best


def prompt_attention(B, S, H, Hkv, hd):
    q = torch.randn(B, S, (H + 2 * Hkv) * hd, device="cuda", dtype=torch.float16)
    k, v = (torch.randn(B, Hkv, S, hd, device="cuda", dtype=torch.float16) for _ in range(2))
    o = torch.empty(B, S, H * hd, device="cuda", dtype=torch.float16)
    return lambda st: N.call("TSB200_PrefillAttention", 0, N.F16, o.data_ptr(), q.data_ptr(), q.shape[2], k.data_ptr(), v.data_ptr(), B, S, H, Hkv, hd, 0, S, st)


@pytest.mark.parametrize("B,H,Hkv,hd", [(64, 12, 12, 64), (64, 32, 8, 64), (64, 32, 32, 128), (64, 32, 8, 128)])
def test_short_prompts_cost_less_than_long_ones(cuda, B, H, Hkv, hd):
    short, long_ = times(prompt_attention(B, 16, H, Hkv, hd), prompt_attention(B, 128, H, Hkv, hd))
    assert short < 0.3 * long_, (short, long_)      # an eighth of the tokens; with whole tiles of 256 rows 0.33 to 0.87 of the time


@pytest.mark.parametrize("V", [4096, 8000])
def test_softmax_of_many_short_rows(cuda, V):
    def call(B):
        z, p, ids = torch.randn(B, V, device="cuda"), torch.empty(B, V, device="cuda"), torch.empty(B, dtype=torch.int32, device="cuda")
        return lambda st: N.call("TSB200_SoftmaxArgmax", 0, ids.data_ptr(), p.data_ptr(), z.data_ptr(), B, V, 1.0, None, 0, st)
    fewer, more = times(call(74), call(75))
    assert fewer < 1.3 * more, (fewer, more)        # eight CTAs for each of 74 rows: 1.8 to 2.5


def test_append_of_one_row_without_a_table(cuda):
    def call(H, Hkv, hd):
        q, k = torch.randn(1, 1, (H + 2 * Hkv) * hd, device="cuda", dtype=torch.float16), torch.zeros(1, Hkv, 2, hd, device="cuda", dtype=torch.float16)
        v = torch.zeros_like(k)
        at = [q.data_ptr() + i * hd * 2 for i in (0, H, H + Hkv)]
        return lambda st: N.call("TSB200_RopeAppend", 0, N.F16, *at, q.shape[2], q.shape[2], k.data_ptr(), v.data_ptr(), 1, 1, H, Hkv, hd, 1, 2, 1, 10000.0, st)
    wide, narrow = times(call(32, 8, 128), call(4, 2, 8))
    assert wide < 2.0 * narrow, (wide, narrow)      # one CTA for the row and four pairs per thread: 4.3


@pytest.mark.parametrize("B,launches", [(8, 1), (16, 2)])
def test_splits_are_a_cluster_only_while_all_are_resident(cuda, B, launches):
    """8 KV heads of 128, 530 keys: three splits.  192 CTAs fit at two per SM; 384 do not, and run as single CTAs before a launch that merges."""
    H, Hkv, hd, T = 32, 8, 128, 530
    k, v = (torch.randn(B, Hkv, T, hd, device="cuda", dtype=torch.float16) for _ in range(2))
    q = torch.randn(B, H * hd, device="cuda", dtype=torch.float16)
    o, ws = torch.empty_like(q), torch.empty(N.lib().TSB200_FlashDecodeWorkspaceBytes(B, H, hd, T), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    n = [N.C.c_int64(), N.C.c_int64()]
    N.call("TSB200_LaunchCount", 0, N.C.byref(n[0]))
    N.call("TSB200_FlashDecode", 0, N.F16, o.data_ptr(), q.data_ptr(), H * hd, k.data_ptr(), v.data_ptr(), B, H, Hkv, hd, T, T, ws.data_ptr(), ws.numel(), None)
    N.call("TSB200_LaunchCount", 0, N.C.byref(n[1]))
    assert n[1].value - n[0].value == launches
    N.call("TSB200_Synchronize", 0, None)
    g = H // Hkv
    z = torch.einsum("bhgd,bhtd->bhgt", q.double().reshape(B, Hkv, g, hd), k.double()) * hd ** -0.5
    ref = torch.einsum("bhgt,bhtd->bhgd", z.softmax(-1), v.double()).reshape(B, H * hd)
    assert (o.double() - ref).abs().max().item() <= 2.0 ** -10     # outputs of N(0, 1/23): weights and outputs rounded to fp16


def linear(M, K, n, dtype):
    code = N.F16 if dtype == torch.float16 else N.F32
    W = (torch.randn(K, n, device="cuda") * 0.05).to(dtype)
    Wp = torch.empty(N.lib().TSB200_PackedWeightBytes(code, K, n), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    N.call("TSB200_PackWeight", 0, code, Wp.data_ptr(), W.data_ptr(), code, K, n, None)
    N.call("TSB200_Synchronize", 0, None)
    x, y = torch.randn(M, K, device="cuda").to(dtype), torch.empty(M, n, device="cuda", dtype=dtype)
    ws = torch.empty(N.lib().TSB200_LinearPackedWorkspaceBytes(code, M, K, n), dtype=torch.uint8, device="cuda")
    keep = (Wp, x, y, ws)
    return lambda st, keep=keep: N.call("TSB200_LinearPacked", 0, code, y.data_ptr(), None, x.data_ptr(), None, None, None, -1, 0.0, Wp.data_ptr(), None, None, M, K, n, -1,
                                        ws.data_ptr(), ws.numel(), st)


def test_linear_of_64_short_rows(cuda):
    many, few = times(linear(64, 64, 64, torch.float16), linear(5, 64, 64, torch.float16))
    assert many < 2.5 * few, (many, few)        # 10.6 against 5.5 us; with a division per pushed sum 19.5 against 6.2


@pytest.mark.parametrize("K,n", [(4096, 4096), (2048, 3072)])
def test_linear_of_one_row_tile_against_two(cuda, K, n):
    one, two = times(linear(100, K, n, torch.float16), linear(160, K, n, torch.float16))
    assert one < 1.3 * two, (one, two)          # with K slices for the single row tile 1.7 to 2.3


def test_top_p_of_flat_rows_against_the_full_sort(cuda):
    """topP = 2.6 leaves no choice but the sort; on a flat row the look at the largest weights must cost next to nothing beside it."""
    B, V = 32, 50257
    p = torch.full((B, V), 1.0 / V, device="cuda")
    u, ids = torch.rand(B, device="cuda"), torch.empty(B, dtype=torch.int32, device="cuda")
    ws = torch.empty(N.lib().TSB200_TopPWorkspaceBytes(B, V), dtype=torch.uint8, device="cuda")
    call = lambda top: lambda st: N.call("TSB200_TopPSample", 0, ids.data_ptr(), p.data_ptr(), B, V, top, 0.0, None, None, 0, u.data_ptr(), ws.data_ptr(), ws.numel(), st)  # noqa: E731
    look, sort = times(call(0.95), call(2.6))
    assert look < 1.07 * sort, (look, sort)     # 1.00; with one shared counter for all keys of a bin 1.11
