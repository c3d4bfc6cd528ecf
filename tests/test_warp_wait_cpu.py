"""The bounded wait of the tensor-core kernels' warps, from its source, on 32 host threads: lanes that see the phase end at different polls, or not at all,
have to leave with one answer."""
import os
import re
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HARNESS = r"""
#include <atomic>
#include <barrier>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <thread>
#include <vector>
#define __device__
#define __forceinline__
constexpr unsigned kTcSpin = 1u << 22;
static int g_ready[32];                     // poll at which a lane sees the phase end; -1: never
static thread_local int t_lane, t_poll, t_vote;
static std::barrier<> g_meet(32);
static std::atomic<unsigned> g_votes[4096];
static bool tc_try_wait(uint32_t, unsigned) { const int i = t_poll++; return g_ready[t_lane] >= 0 && i >= g_ready[t_lane]; }
static unsigned ballot(bool p) {
  std::atomic<unsigned>& votes = g_votes[t_vote++];
  votes += p ? 1u : 0u;
  g_meet.arrive_and_wait();
  return votes;
}
static bool __all_sync(unsigned, bool p) { return ballot(p) == 32u; }
static bool __any_sync(unsigned, bool p) { return ballot(p) != 0u; }
%s
int main(int argc, char** argv) {
  for (int i = 0; i < 32; ++i) g_ready[i] = atoi(argv[2 + i]);
  static volatile int err = 0;
  std::vector<int> out(32);
  std::vector<std::thread> lanes;
  for (int i = 0; i < 32; ++i) lanes.emplace_back([&, i] { t_lane = i; out[i] = tc_wait_or(0, 0, &err, (unsigned)atoi(argv[1])); });
  for (auto& l : lanes) l.join();
  for (int v : out) printf("%%d", v);
  printf(" %%d\n", (int)err);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    with open(os.path.join(ROOT, "seq2seqsharp_b200", "csrc", "tc_common.cuh")) as f:
        wait = re.search(r"^__device__ __forceinline__ bool tc_wait_or\(.*?^}", f.read(), re.S | re.M).group(0)
    at = tmp_path_factory.mktemp("wait")
    (at / "wait.cpp").write_text(HARNESS % wait)
    subprocess.run(["g++", "-O1", "-std=c++20", "-pthread", str(at / "wait.cpp"), "-o", str(at / "wait")], check=True)
    return str(at / "wait")


@pytest.mark.parametrize("limit,ready,answer", [
    (1, [0] * 32, 1), (1, [0] * 31 + [1], 0), (100, list(range(32)), 1), (100, [99] * 32, 1), (100, [0] * 16 + [100] * 16, 0), (100, [-1] + [0] * 31, 0),
    (500, [0] * 31 + [-1], 0), (500, [-1] * 32, 0)])
def test_one_answer_for_all_lanes(program, limit, ready, answer):
    r = subprocess.run([program, str(limit), *map(str, ready)], capture_output=True, text=True, timeout=60, check=True)
    assert r.stdout.split() == [str(answer) * 32, str(1 - answer)]
