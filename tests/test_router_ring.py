"""The order of waits of the router GEMM's normalising warps, run on the host against an emulated ring: copies land in any
order, every thread of control runs at its own pace, and barriers answer a parity wait as an mbarrier does."""

import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

EMULATOR = r"""
#include <cstdio>
#include <random>
#include <vector>
#include "router_ring.h"

struct Barrier {
  int count, pending, tx = 0;
  uint32_t phase = 0;
  explicit Barrier(int n) : count(n), pending(n) {}
  bool passed(uint32_t parity) const { return (phase & 1u) != parity; }  // the phase of that parity before the present one is over
  void settle() {
    if (pending == 0 && tx == 0) {
      ++phase;
      pending = count;
    }
  }
  void arrive() { --pending; settle(); }
  void expect() { tx += 1; arrive(); }
  void landed() { tx -= 1; settle(); }
};

// one pass over `blocks` k-blocks; what went wrong, or null
template <int kStages, int kGroups, int kWarps, bool kRule>
const char* pass(int blocks, std::mt19937& gen) {
  using Waits = fmoe::NormaliseWaits<kStages, kGroups>;
  std::vector<Barrier> full(kStages, Barrier(1)), ready(kStages, Barrier(kWarps)), empty(kStages, Barrier(1));
  std::vector<int> holds(kStages, -1), done(kStages, 0);  // the k-block whose tile a stage holds, the warps that normalised it
  std::vector<int> flying;
  int produced = 0, multiplied = 0;
  std::vector<int> at(kGroups * kWarps), step(kGroups * kWarps, 0);
  for (int i = 0; i < kGroups * kWarps; ++i) at[i] = i / kWarps;
  std::vector<double> pace(kGroups * kWarps + 2);
  for (double& p : pace) p = 0.05 + 0.95 * std::generate_canonical<double, 32>(gen);
  const double landing = 0.02 + 0.5 * std::generate_canonical<double, 32>(gen);
  auto lucky = [&](double p) { return std::generate_canonical<double, 32>(gen) < p; };
  for (long turn = 0; multiplied < blocks; ++turn) {
    if (turn > 2000000) return "no progress";
    if (!flying.empty() && lucky(landing)) {
      const int i = static_cast<int>(gen() % flying.size()), kb = flying[i], s = kb % kStages;
      flying.erase(flying.begin() + i);
      holds[s] = kb;
      done[s] = 0;
      full[s].landed();
    }
    if (produced < blocks && lucky(pace[0])) {
      const int s = produced % kStages;
      if (empty[s].passed((produced / kStages + 1) & 1u)) {
        full[s].expect();
        flying.push_back(produced++);
      }
    }
    for (int i = 0; i < kGroups * kWarps; ++i) {
      const int kb = at[i], s = kb % kStages;
      if (kb >= blocks || !lucky(pace[2 + i])) continue;
      if (step[i] == 0 && kRule && Waits::behind_empty(kb) && !empty[s].passed(Waits::empty_parity(kb))) continue;
      step[i] = 1;
      if (!full[s].passed(Waits::full_parity(kb))) continue;
      if (holds[s] != kb) return "a warp normalised a tile that has not landed";
      ++done[s];
      ready[s].arrive();
      at[i] += kGroups;
      step[i] = 0;
    }
    if (lucky(pace[1])) {
      const int s = multiplied % kStages;
      if (ready[s].passed((multiplied / kStages) & 1u)) {
        if (holds[s] != multiplied || done[s] != kWarps) return "a product read a tile that is not normalised";
        empty[s].arrive();
        ++multiplied;
      }
    }
  }
  return flying.empty() ? nullptr : "a copy outlasts the pass";
}

template <int kStages, int kGroups, bool kRule>
int passes(int n) {
  std::mt19937 gen(kStages * 100 + kGroups);
  int wrong = 0;
  for (int i = 0; i < n; ++i)
    if (pass<kStages, kGroups, 4, kRule>(1 + static_cast<int>(gen() % 48), gen) != nullptr) ++wrong;
  return wrong;
}

int main() {
  std::printf("%d %d %d %d\n", passes<8, 4, true>(2000), passes<4, 4, true>(2000), passes<6, 4, true>(2000), passes<6, 4, false>(2000));
}
"""


@pytest.fixture(scope="module")
def wrong_passes(tmp_path_factory):
    d = tmp_path_factory.mktemp("ring")
    source, program = d / "ring.cpp", d / "ring"
    source.write_text(EMULATOR)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", os.path.join(ROOT, "flash_moe_b200", "csrc"), "-o", str(program), str(source)],
                   check=True)
    out = subprocess.run([str(program)], check=True, capture_output=True, text=True, timeout=300).stdout
    return [int(v) for v in out.split()]


def test_normalising_warps_wait_for_their_own_tile(wrong_passes):
    """Ring depths of the three tile shapes: 8, 4 and 6 stages with four groups of warps."""
    assert wrong_passes[:3] == [0, 0, 0]


def test_the_emulated_ring_shows_a_missing_wait(wrong_passes):
    """With `full` alone, six stages and four groups: the wait for a phase passes while the one before it is still open."""
    assert wrong_passes[3] > 0


def test_the_kernel_waits_by_the_rule():
    with open(os.path.join(ROOT, "flash_moe_b200", "csrc", "gemm_router_bn.cu")) as f:
        text = f.read()
    assert "Waits::behind_empty(kb)" in text and "Waits::full_parity(kb)" in text
    assert text.count("mbar_wait_bounded(full_bar(s)") == 1
