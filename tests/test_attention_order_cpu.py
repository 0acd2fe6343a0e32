"""The MMA issuer of csrc/attention_infer.cu, replayed on the host: its source is compiled with stand-ins for the instructions, which
record what it issues and waits for.

P of a block lies over the logits it was made from, so the product P V that reads it and the S product two blocks later write and read
the same columns.  Products with different accumulators and shapes have no order of their own: the second may only be issued after a
wait that the first one's completion ended.

A wait that runs out ends the kernel: the waits after it, one or more for every block that is left, must be short."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

SOURCE = os.path.join(ROOT, "fastfold_b200", "csrc", "attention_infer.cu")

# Barriers are numbers.  `commits[bar]` holds how many products had been issued at each commit on it, `seen[bar]` how many of its phases
# this warp knows to be over; a wait for a parity is only sure to end at the first phase of that parity after those, which has to have a
# commit.  The softmax warps answer an S product with P at once; Q, K, V and bias tiles are always there.
HARNESS = r"""
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <vector>
#define __device__
#define __forceinline__
using std::min;
typedef uint16_t bf16;
%(constants)s
%(args)s
%(smem)s
%(round)s
struct Keys { uint32_t lo, hi; };
struct KeyMask { uint16_t a, b; };
static KeyMask load_keys(const bf16*, int, int, int) { return {1, 1}; }
static Keys key_bits(KeyMask) { return {~0u, ~0u}; }
enum { ST_TIMEOUT_TMA = 1, ST_TIMEOUT_MMA, ST_TIMEOUT_EPI };
#define FFB_LOCAL_WAIT_NS 2000000000ull
static void fail(const char* what, int a, int b) { std::printf("%%s (%%d, %%d)\n", what, a, b); std::exit(1); }

constexpr uint32_t base = 0, q_full = 1000, q_empty = 1100, kv_full = 1200, kv_empty = 1300, bias_full = 1400, bias_empty = 1500, s_full = 1600,
                   p_full = 1700, o_done = 1800;
struct Replay {
  std::map<uint32_t, std::vector<int>> commits;
  std::map<uint32_t, int> seen;
  int issued = 0, done = 0, s = 0, pv = 0, g, releases = 0;
  int reader[2] = {0, 0};                       // last product that reads the P in either buffer
  int waits = 0, lost = 1 << 30;                // waits so far, and the first that nothing ends (as after a copy that never lands)
  int reports = 0, tries_after = 0, flag = 0;   // reports of a wait that ran out, tries made since then
  uint64_t clock = 0;
  void wait(uint32_t bar, uint32_t parity) {
    const uint32_t group = bar / 100 * 100;
    if (group == q_full || group == kv_full || group == bias_full) return;
    int n = seen[bar];
    while ((uint32_t)(n & 1) == (parity & 1)) ++n;          // phases over when a wait for this parity ends
    const std::vector<int>& c = commits[group == p_full ? bar - p_full + s_full : bar];
    if (n > (int)c.size()) fail("a wait that nothing ends", (int)group, n);
    seen[bar] = n;
    if (n > 0) done = std::max(done, c[n - 1]);
  }
};

template <int D, bool BIAS>
static Replay issuer(const AttnInferArgs& a, int g0, int r_begin, int r_end, int lost) {
  constexpr uint32_t LAYOUT = D == 32 ? 4 : 6, GROUP = 8 * D * 2;
  Replay x;
  x.g = g0;
  x.lost = lost;
  const int warp = g0 + 1, lane = 0;
  const uint32_t tmem = 0;
  std::vector<uint8_t> memory(AttnInferSmem::TOTAL);
  uint8_t* sm = memory.data();
  const Round rd0(a, r_begin);
  auto elect_one = []() { return 1u; };
  auto make_idesc_bf16 = [](int, int, int, int) constexpr { return 0u; };
  auto make_desc = [](uint32_t, uint32_t, uint32_t, uint32_t) { return (uint64_t)0; };
  auto tc_fence_after = []() {};
  volatile int* abort_flag = &x.flag;
  auto globaltimer_ns = [&]() { return x.clock += 700000000ull; };
  auto report = [&](int, int) { ++x.reports; };
  auto mbar_try_wait = [&](uint32_t bar, uint32_t parity) {
    if (x.waits < x.lost) {
      ++x.waits;
      x.wait(bar, parity);
      return true;
    }
    x.tries_after += x.flag;
    return false;
  };
  %(wait)s
  auto mbar_arrive = [&](uint32_t bar) { x.releases += bar / 100 * 100 == bias_empty; };
  auto umma_commit_by = [&](uint32_t, uint32_t bar) { x.commits[bar].push_back(x.issued); };
  auto umma_bf16_by = [&](uint32_t, uint32_t d, uint64_t, uint64_t, uint32_t, uint32_t acc) {
    const int buf = (int)(d - g0 * AF_TM_GROUP) / AF_BK;
    if (!x.flag && x.reader[buf] > x.done) fail("S product over a P that may still be read: S product, products known to be over", x.s, x.done);
    ++x.issued;
    x.s += !acc;
  };
  auto umma_bf16_ts_by = [&](uint32_t, uint32_t, uint32_t p, uint64_t, uint32_t, uint32_t) {
    const uint32_t col = p - g0 * AF_TM_GROUP, buf = col / AF_BK;
    ++x.issued;
    x.reader[buf] = x.issued;
    x.pv += col %% AF_BK == 0;
  };
  %(issuer)s
  return x;
}

int main() {
  std::srand(1);
  for (int run = 0; run < 4000; ++run) {
    AttnInferArgs a = {};
    a.B = 1 + std::rand() %% 9;
    a.H = 1 + std::rand() %% 3;
    a.n_qt = 1 + std::rand() %% 3;
    a.n_kb = 1 + std::rand() %% 9;
    a.n_k = a.n_kb * 64;
    const int c = 1 + std::rand() %% AF_GROUPS;
    a.rounds = (a.B + c - 1) / c;
    a.few = a.B / a.rounds;
    a.rest = a.B - a.few * a.rounds;
    const bool bias = run & 1;
    a.bias_resident = bias && a.n_kb <= AF_BSLOTS;
    const int all = a.H * a.n_qt * a.rounds, begin = std::rand() %% all, end = begin + 1 + std::rand() %% (all - begin), g = run %% AF_GROUPS;
    int blocks = 0, tiles = 0;
    for (Round r(a, begin); r.i < end; r.next(a)) {
      if (g < r.cnt) blocks += a.n_kb;
      if (bias && (!a.bias_resident || r.i + 1 == end || r.last(a))) tiles += a.n_kb;
    }
    const Replay x = bias ? issuer<32, true>(a, g, begin, end, 1 << 30) : issuer<16, false>(a, g, begin, end, 1 << 30);
    if (x.s != blocks || x.pv != blocks) fail("blocks issued and due", x.pv, blocks);
    if (x.releases != tiles) fail("bias tiles released and due", x.releases, tiles);
  }
  // a wait that runs out early: at most nine tries (of 4 us each) for each of those after it, at most five waits a block
  for (int lost = 0; lost < 20; ++lost) {
    AttnInferArgs a = {};
    a.H = 4;
    a.n_qt = 8;
    a.n_kb = 6;
    a.n_k = a.n_kb * 64;
    a.rounds = 100;
    a.few = 3;
    a.B = 300;
    const int rounds = a.H * a.n_qt * a.rounds;
    const Replay x = issuer<32, true>(a, 0, 0, rounds, lost);
    if (x.reports != 1 || x.tries_after > 9 * 5 * rounds * a.n_kb) fail("reports, tries after a wait that ran out", x.reports, x.tries_after);
  }
  std::printf("ok\n");
}
"""


def _between(text, first, last, head=True, tail=True):
    """What lies from ``first`` to ``last``, with or without these two."""
    i = text.index(first)
    j = text.index(last, i)
    return text[i if head else i + len(first):j + len(last) if tail else j]


def _program():
    with open(SOURCE) as f:
        text = f.read()
    body = _between(text, "// ---------------- MMA issuer of one group ----------------", "  } else {\n    // ---------------- softmax / output", head=False, tail=False)
    return HARNESS % {
        "constants": "\n".join(line for line in text.splitlines() if line.startswith("constexpr") and " AF_" in line),
        "args": _between(text, "struct AttnInferArgs {", "\n};"),
        "smem": _between(text, "struct AttnInferSmem {", "\n};"),
        "round": _between(text, "struct Round {", "\n};"),
        "wait": _between(text, "  auto wait = [&](uint32_t bar", "  // The producer and the issuers", tail=False),
        "issuer": body,
    }


@pytest.mark.skipif(shutil.which("g++") is None, reason="no C++ compiler")
def test_issuer_waits_for_readers_and_ends_after_a_lost_wait(tmp_path):
    src = tmp_path / "issuer.cpp"
    src.write_text(_program())
    exe = str(tmp_path / "issuer")
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-w", str(src), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[:3000]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout
