"""The way out of the tcgen05 kernels after an abort (csrc/ring.h), played through without a GPU: producer warps, copies, a consumer and
mbarriers as a random interleaving of small steps, with the abort flag raised anywhere in it."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "haste_b200", "csrc")

MODEL = r"""
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>
#include "ring.h"

#define CHECK(x) do { if (!(x)) { std::printf("NXS=%d NPW=%d NSH=%d seed=%d: %s\n", NXS, NPW, NSH, seed, #x); std::exit(1); } } while (0)

struct Barrier {                                  // an mbarrier: a phase ends when all arrivals are in and all announced bytes have landed
  int count, pending, tx = 0, phase = 0;
  bool underflow = false;
  explicit Barrier(int n) : count(n), pending(n) {}
  void settle() { if (pending == 0 && tx == 0) { pending = count; ++phase; } }
  void arrive(int bytes) { if (pending == 0) underflow = true; --pending; tx += bytes; settle(); }
  void land(int bytes) { tx -= bytes; settle(); }
  bool done(int parity) const { return (phase & 1) != parity; }
};

template <int NXS, int NPW, int NSH>
int play(int seed) {
  std::mt19937 rng(seed);
  constexpr int STEP = NPW / NSH;
  const int n_items = 1 + rng() % 40;
  std::vector<Barrier> full(NXS, Barrier(NSH)), empty(NXS, Barrier(1));
  struct Producer { int it, last = -1; bool sure = false, out = false; };
  struct Copy { int item; };
  std::vector<Producer> prod(NPW);
  std::vector<Copy> flying;
  for (int p = 0; p < NPW; ++p) prod[p].it = p / NSH;
  int consumed = 0;
  bool abort = false;
  const int abort_at = rng() % 400;
  const int slow = rng() % NPW;                   // a warp that hardly gets to run
  for (int step = 0; step < 100000; ++step) {
    if (step >= abort_at) abort = true;
    bool all_out = true;
    for (auto& w : prod) all_out = all_out && w.out;
    if (all_out) break;
    const int who = rng() % (NPW + 2);
    if (who < NPW) {
      Producer& w = prod[who];
      if (who == slow && rng() % 8) continue;
      if (w.out) continue;
      if (w.it >= n_items) { w.out = true; continue; }
      const int s = w.it % NXS;
      if (w.sure) {                               // the announcement follows the look at the flag at any distance
        full[s].arrive(1);
        flying.push_back({w.it});
        w.last = w.it; w.it += STEP; w.sure = false;
      } else if (abort) {
        w.out = true;
      } else if (empty[s].done(((w.it / NXS) & 1) ^ 1)) {
        w.sure = true;
      }
    } else if (who == NPW) {
      if (!flying.empty() && rng() % 2) {
        const int i = rng() % flying.size();
        full[flying[i].item % NXS].land(1);
        flying.erase(flying.begin() + i);
      }
    } else if (!abort && consumed < n_items && full[consumed % NXS].done((consumed / NXS) & 1)) {
      empty[consumed % NXS].arrive(0);
      ++consumed;
    }
  }
  int short_of = 0;
  auto last = [&](int p) { return prod[p].last; };
  std::vector<int> waited(NXS, -1);
  for (int s = 0; s < NXS; ++s) {
    const haste::RingDrain d = haste::ring_drain<NXS, NPW, NSH>(s, last);
    waited[s] = d.item;
    if (d.item < 0) continue;
    short_of += d.missing;
    if (d.missing > 0) CHECK(!full[s].done((d.item / NXS) & 1));             // without them the wait would never end
    for (int i = 0; i < d.missing; ++i) full[s].arrive(0);
  }
  for (const Copy& c : flying) CHECK(waited[c.item % NXS] == c.item);       // nothing is in flight that is not waited for
  for (int s = 0; s < NXS; ++s) {
    if (waited[s] < 0) continue;
    bool in_flight = false;
    for (const Copy& c : flying) in_flight = in_flight || c.item % NXS == s;
    CHECK(full[s].done((waited[s] / NXS) & 1) == !in_flight);                // the wait ends when the copies have landed, not before
  }
  for (const Copy& c : flying) full[c.item % NXS].land(1);
  for (int s = 0; s < NXS; ++s) {
    CHECK(!full[s].underflow);
    if (waited[s] >= 0) CHECK(full[s].done((waited[s] / NXS) & 1));
  }
  return short_of;
}

template <int NXS, int NPW, int NSH>
void all() {
  static_assert(NPW / NSH <= NXS, "as the kernels assert");
  int short_of = 0;
  for (int seed = 0; seed < 4000; ++seed) short_of += play<NXS, NPW, NSH>(seed);
  const int seed = -1;
  if (NSH > 1) CHECK(short_of > 100);             // the interesting case is among them
}

int main() {
  all<4, 4, 2>(); all<3, 4, 2>(); all<4, 4, 4>(); all<5, 4, 2>(); all<4, 8, 2>(); all<5, 8, 2>(); all<6, 8, 2>(); all<2, 2, 1>(); all<3, 3, 1>();
  return 0;
}
"""


def test_copies_in_flight_at_an_abort_are_waited_for(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no C++ compiler")
    src = tmp_path / "model.cpp"
    src.write_text(MODEL)
    subprocess.run([gxx, "-std=c++17", "-O1", "-Wall", "-Werror", "-I", CSRC, str(src), "-o", str(tmp_path / "model")], check=True)
    r = subprocess.run([str(tmp_path / "model")], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
