"""The give-up path of the persistent decode-step kernel, exercised without any fault: the host lowers the bound of the
kernel's dependency polls to one, so the first CTA that looks at a counter before its producers have finished gives
up.  The kernel must return (every CTA walks through the rest of its program without waiting), the call must fail with
a message, the engine must stay usable, and with the default bound restored the same prompt must give the same ids as
an engine that never failed.  Nothing here traps, faults or waits without a limit."""
import numpy as np
import pytest

from seq2seqsharp_b200 import _native as N
from seq2seqsharp_b200.gpt import DecodingOptions, GPT, synthetic_weights
from seq2seqsharp_b200.synthetic import prompt_ids
from tests.test_gpt_gpu import ARCHS

pytestmark = pytest.mark.gpu


@pytest.mark.timeout(300)
@pytest.mark.parametrize("cfg", [ARCHS[1], ARCHS[0]], ids=["fp16_tensor_core_consumers", "fp32_cuda_core_consumers"])
@pytest.mark.parametrize("call", ["decode", "step_host"])
def test_a_wait_that_runs_out_fails_the_call_and_leaves_the_engine_usable(cuda, cfg, call, monkeypatch):
    monkeypatch.setenv("TSB200_OWNER_MAXB", "1")    # one sequence on a persistent kernel (one-GPU fp16 engines default to one
    monkeypatch.setenv("TSB200_STACK_MAXB", "1")    # launch per operation): the kernels whose cross-CTA waits are bounded
    w = synthetic_weights(cfg, 21, std=0.04)
    prompt = prompt_ids(9, 1, 24, cfg.V)
    opts = DecodingOptions(MaxTgtSentLength=64, BlockedTokens=[0])
    gpt = GPT(cfg, max_batch=1, max_tokens=64)
    gpt.LoadWeights(w)
    first = gpt.Prefill(prompt, opts)
    good = gpt.Decode(6, opts)
    assert gpt.ProfileDecode(1, opts)["decode_stack"][1] == 1      # one sequence decodes through the persistent kernel
    # --- the wait runs out
    gpt.Reset()
    np.testing.assert_array_equal(gpt.Prefill(prompt, opts), first)
    gpt.SetWaitLimit(1)
    T_before = gpt.CacheLength()
    with pytest.raises(N.TSB200Error, match="gave up waiting"):
        if call == "decode":
            gpt.Decode(3, opts)
        else:
            gpt.StepHost(first, opts)
    assert gpt.CacheLength() == T_before       # the failed call committed nothing on the host side
    # --- and the engine is still good for ordinary calls
    gpt.SetWaitLimit(0)
    gpt.Reset()
    np.testing.assert_array_equal(gpt.Prefill(prompt, opts), first)
    np.testing.assert_array_equal(gpt.Decode(6, opts), good)
    gpt.close()


def test_a_wait_that_runs_out_in_a_stand_alone_call_is_reported_where_the_host_waits(cuda):
    """One poll per wait (an environment variable, hence a process of its own): the prompt attention gives up before its first tile has
    arrived, waits for its copies and products in flight, and returns; the synchronisation fails, and only the first one."""
    import os
    import subprocess
    import sys
    code = """
import torch
from seq2seqsharp_b200 import _native as N
q = torch.randn(2, 300, 3 * 64, device="cuda", dtype=torch.float16)
k, v = (torch.randn(2, 1, 300, 64, device="cuda", dtype=torch.float16) for _ in range(2))
o = torch.empty(2, 300, 64, device="cuda", dtype=torch.float16)
torch.cuda.synchronize()
N.call("TSB200_PrefillAttention", 0, N.F16, o.data_ptr(), q.data_ptr(), 192, k.data_ptr(), v.data_ptr(), 2, 300, 1, 1, 64, 0, 300, None)
try:
    N.call("TSB200_Synchronize", 0, None)
    print("silent")
except N.TSB200Error as e:
    print(e)
N.call("TSB200_Synchronize", 0, None)
print("usable", float(torch.ones(4, device="cuda").sum()))
"""
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=120, env=dict(os.environ, TSB200_WAIT_LIMIT="1"),
                       cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    assert r.returncode == 0, r.stderr
    assert "gave up waiting" in r.stdout and "usable 4.0" in r.stdout, r.stdout


@pytest.mark.parametrize("rows,dtype", [(1, "16"), (64, "16"), (100, "16"), (300, "16"), (3, "32")])
def test_linears_end_in_order_when_a_wait_runs_out(cuda, rows, dtype):
    """The same for the linears: one fp16 row and 64 on clusters, 100 on tiles of one CTA with K slices, 300 on pairs of CTAs, fp32 rows on clusters.  Every warp gives up in its
    own place; copies and products in flight end before a CTA leaves its shared memory and TMEM, so the calls behind it are sound."""
    import os
    import subprocess
    import sys
    code = """
import torch
from seq2seqsharp_b200 import _native as N
M, K, n, code = %d, 11008, 8192, N.F%s
t = torch.float16 if code == N.F16 else torch.float32
W = torch.randn(K, n, device="cuda", dtype=t)
Wp = torch.empty(N.lib().TSB200_PackedWeightBytes(code, K, n), device="cuda", dtype=torch.uint8)
x, y = torch.randn(M, K, device="cuda", dtype=t), torch.empty(M, n, device="cuda", dtype=t)
ws = torch.empty(N.lib().TSB200_LinearPackedWorkspaceBytes(code, M, K, n), device="cuda", dtype=torch.uint8)
torch.cuda.synchronize()
N.call("TSB200_PackWeight", 0, code, Wp.data_ptr(), W.data_ptr(), code, K, n, None)
N.call("TSB200_Synchronize", 0, None)
for i in range(8):
    N.call("TSB200_LinearPacked", 0, code, y.data_ptr(), None, x.data_ptr(), None, None, None, -1, 0.0, Wp.data_ptr(), None, None, M, K, n, N.ACT_NONE, ws.data_ptr(), ws.numel(), None)
try:
    N.call("TSB200_Synchronize", 0, None)
    print("silent")
except N.TSB200Error as e:
    print(e)
N.call("TSB200_Synchronize", 0, None)
print("usable", torch.equal(W.flip(1).flip(1), W), float(torch.ones(4, device="cuda").sum()))
""" % (rows, dtype)
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=120, cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                       env=dict(os.environ, TSB200_WAIT_LIMIT="1", TSB200_GEMV_MAXROWS="0"))
    assert r.returncode == 0, r.stderr
    assert "gave up waiting" in r.stdout and "usable True 4.0" in r.stdout, r.stdout
