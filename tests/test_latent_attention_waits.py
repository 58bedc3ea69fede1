"""The two warps that share 32 rows of `latent_attention_tc_kernel` meet at a named barrier several times a key tile. Their
waits on the copy engine and the tensor cores are bounded and may end differently in the two; a warp that left while its
partner stands at the barrier would leave it there for good. Shown on the CPU: the control flow of the kernel's softmax branch
(its waits, meetings and ways out, as they stand in the source) is compiled for the host and walked by two threads for
every outcome of their waits."""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

SOURCE = Path(__file__).resolve().parent.parent / "cuca_b200" / "csrc" / "latent_attention_tc.cu"

HARNESS = r"""
#include <condition_variable>
#include <cstdio>
#include <mutex>
#include <thread>
struct Pair {  // a barrier of two that also sees when it can never be met
  std::mutex m;
  std::condition_variable cv;
  int here = 0, turn = 0, left = 0;
  bool all = true, result = true, stuck = false;
  bool meet(bool ok) {
    std::unique_lock<std::mutex> l(m);
    all = all && ok;
    if (++here == 2) { result = all; all = true; here = 0; ++turn; cv.notify_all(); return result; }
    const int t = turn;
    cv.wait(l, [&] { return turn != t || left; });
    if (turn == t) { stuck = true; return false; }
    return result;
  }
  void leave() { std::lock_guard<std::mutex> l(m); ++left; cv.notify_all(); }
};
struct Stuck {};
static void walk(Pair& pair, unsigned outcomes, int n_tiles, int& stored) {
  auto wait_ends = [&] { const bool r = outcomes & 1; outcomes >>= 1; return r; };
  auto pair_sync = [&] { pair.meet(true); if (pair.stuck) throw Stuck(); };
  auto pair_vote = [&](bool ok) { const bool r = pair.meet(ok); if (pair.stuck) throw Stuck(); return r; };
  try {
//BODY
  } catch (Stuck&) {}
  pair.leave();
}
int main() {
  for (int n = 1; n <= 2; ++n) {
    const int waits = 2 * n;  // the scores of every tile and the contraction behind every tile
    for (unsigned a = 0; a < 1u << waits; ++a)
      for (unsigned b = 0; b < 1u << waits; ++b) {
        Pair pair;
        int stored[2] = {0, 0};
        std::thread other(walk, std::ref(pair), b, n, std::ref(stored[1]));
        walk(pair, a, n, stored[0]);
        other.join();
        const bool good = a == (1u << waits) - 1 && b == a;
        if (pair.stuck) { printf("stuck: %d tiles, waits %x and %x\n", n, a, b); return 1; }
        if (stored[0] != good || stored[1] != good) { printf("stored %d %d: %d tiles, waits %x and %x\n", stored[0], stored[1], n, a, b); return 2; }
      }
  }
  return 0;
}
"""


def _control_flow(source: str) -> str:
    """The softmax branch from its loop to its end, of each line only what decides where the warp goes."""
    begin = source.index("float m = -INFINITY, l = 0.f;")
    depth, end = 0, begin
    while depth >= 0:  # (to the brace that closes the branch)
        depth += {"{": 1, "}": -1}.get(source[end], 0)
        end += 1
    kept = []
    for line in source[begin:end - 1].splitlines():
        line = line.split("//")[0]
        line = re.sub(r"warp_wait\((?:[^()]|\([^()]*\))*\)", "wait_ends()", line)
        line = line.replace("soft_sync(quarter)", "pair_sync()").replace("soft_vote(quarter, ", "pair_vote(")
        if re.search(r"wait_ends|pair_|\bok\b|for \(int j|if \(j > 0\)|\bbreak\b|\bcontinue\b|\breturn\b", line):
            kept.append(line)
        else:
            kept.append(re.sub(r"[^{};]", "", line) if re.search(r"[{}]", line) else "")
            if "p.out + " in line:
                kept.append("stored = 1;")
    return "\n".join(kept)


def test_a_warp_never_leaves_its_partner_at_the_barrier(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("no host compiler")
    flow = _control_flow(SOURCE.read_text())
    assert flow.count("wait_ends()") == 3 and "stored" in flow
    src, exe = tmp_path / "walk.cpp", tmp_path / "walk"
    src.write_text(HARNESS.replace("//BODY", flow))
    made = subprocess.run(["g++", "-std=c++17", "-pthread", "-w", "-o", str(exe), str(src)], capture_output=True, text=True)
    assert made.returncode == 0, made.stderr + flow
    ran = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert ran.returncode == 0, ran.stdout
