"""CPU: the producer warps' turns on a ring of stages (csrc/ring.cuh), stepped against a model of the barriers under random interleavings.

A slot's "empty" barrier is waited for by parity, so a warp more than one round ahead of the consumer is let into a slot whose operands have not
been read.  The model flags that; four warps stepping by four on a ring of two or three slots (a planted mistake) must be caught by it."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
MODEL = r"""
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>
#include "ring.cuh"

struct Warp { uint32_t i, step, s, ph; bool on; };

// 0: every stage was filled once and read once; 1: a stage was overwritten before it was read; 2: slot, parity or progress wrong
int run(uint32_t n, uint32_t stages, uint32_t seed, bool planted) {
  std::mt19937 rng(seed);
  std::vector<fovi::RingTurn> turn;
  std::vector<Warp> w;
  for (uint32_t i = 0; i < (uint32_t)fovi::PRODUCER_WARPS; ++i) {
    turn.emplace_back(i, n);
    w.push_back({i, planted ? (uint32_t)fovi::PRODUCER_WARPS : turn[i].step, i % n, (i / n) & 1u, planted || !turn[i].idle});
    if (!planted && w[i].on && turn[i].step > n) return 2;
  }
  std::vector<long> holds(n, -1);
  std::vector<uint32_t> read(n, 0);
  uint32_t next = 0;
  for (uint64_t spin = 0; next < stages && spin < 400ull * stages; ++spin) {
    const uint32_t pick = rng() % (fovi::PRODUCER_WARPS + 1);
    if (pick == (uint32_t)fovi::PRODUCER_WARPS) {                       // the consumer reads the next stage once it is there
      const uint32_t s = next % n;
      if (holds[s] != (long)next) continue;
      holds[s] = -1; ++read[s]; ++next;
      continue;
    }
    Warp& p = w[pick];
    if (!p.on || p.i >= stages) continue;
    if (!planted && (turn[pick].s != p.s || turn[pick].ph != p.ph)) return 2;
    if ((read[p.s] & 1u) == (p.ph ^ 1u)) continue;                      // try_wait.parity: the phase of that parity has not completed
    if (holds[p.s] != -1) return 1;
    holds[p.s] = p.i;
    p.i += p.step; p.s = p.i % n; p.ph = (p.i / n) & 1u;
    if (!planted) turn[pick].next();
  }
  return next == stages ? 0 : 2;
}

int main(int argc, char** argv) {
  const uint32_t n = (uint32_t)atoi(argv[1]);
  const bool planted = atoi(argv[2]) != 0;
  int seen = 0;
  for (uint32_t seed = 0; seed < 200; ++seed) seen |= 1 << run(n, 300, seed, planted);
  printf("%d\n", seen);
  return 0;
}
"""


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    d = tmp_path_factory.mktemp("ring")
    src, exe = d / "model.cpp", d / "model"
    src.write_text(MODEL)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I", os.path.join(ROOT, "fovi_b200", "csrc"), str(src), "-o", str(exe)], check=True)
    return lambda n, planted: int(subprocess.run([str(exe), str(n), str(int(planted))], check=True, capture_output=True, text=True).stdout)


@pytest.mark.parametrize("nstage", range(1, 9))
def test_turns_never_overwrite_an_unread_stage(model, nstage):
    assert model(nstage, False) == 1 << 0


@pytest.mark.parametrize("nstage", (2, 3))
def test_the_model_catches_more_warps_than_slots(model, nstage):
    assert model(nstage, True) & (1 << 1)
