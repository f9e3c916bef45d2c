"""The load walk of the tensor-core combination kernel (csrc/block_ring.h) with
a model of its copies and barriers, compiled for the host.

The model is the hardware's rule: a barrier's phase completes when its arrivals
are in and every announced byte has landed; copies land in any order, some only
when the walk waits for them.  Bars, for walks that run to the end and for ones
whose wait for a free slot gives up at any step: no copy is on its way when the
walk returns, no barrier has an arrival too many or a phase that cannot
complete, no slot is overwritten before the K steps that read it are cut.
"""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "quantum_package_gb300", "csrc")

MODEL = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>
#include "block_ring.h"

struct Copy { int tile, slot; long bytes; };
struct Model {
  int nb, nsd, nks, ks, nslots, ntile, give_up;  // the give_up-th wait fails (-1: none)
  bool eager;               // copies land at once, or only when waited for
  long bytes_of_block;
  int waits = 0, bad = 0;
  int phase[2] = {0, 0}, pending[2] = {1, 1};
  long tx[2] = {0, 0};
  std::vector<Copy> flight;
  std::vector<int> slot_tile, slot_block;
  int cut_steps = 0;        // K steps cut so far
  int ahead = 0, rnd = 1, finished = 0;
  void complete(int i) {
    if (pending[i] == 0 && tx[i] == 0) { ++phase[i]; pending[i] = 1; }
  }
  void land(size_t k) {
    const Copy c = flight[k];
    flight.erase(flight.begin() + k);
    tx[c.tile & 1] -= c.bytes;
    complete(c.tile & 1);
  }
  void land_tile(int t) {
    for (size_t k = flight.size(); k-- > 0;)
      if (flight[k].tile == t) land(k);
  }
  // the consumers: a tile's steps are cut in order once its phase is complete
  int cut(int step) {
    if (waits++ == give_up) return 0;
    while (cut_steps <= step || ahead > 0) {  // up to `ahead` steps more, as far as the tiles have been started
      if (cut_steps > step && ahead-- <= 0) break;
      const int t = cut_steps / nks;
      if (t >= ntile || (cut_steps > step && t >= finished)) break;
      land_tile(t);
      if (phase[t & 1] <= t / 2) { bad |= 1; return 0; }  // would wait for ever
      ++cut_steps;
    }
    ahead = rnd = (rnd * 5 + 3) % 8;
    return cut_steps;
  }
  int begun = -1;
  void begin(int t) {
    if (t != begun + 1) bad |= 128;
    begun = t;
  }
  void copy(int t, int b, int n, int slot) {
    if (t != begun) bad |= 128;
    if (n < 1 || b + n > nb) { bad |= 64; return; }
    for (int i = 0; i < n; ++i) copy1(t, b + i, slot + i);
  }
  void copy1(int t, int b, int slot) {
    if (slot < 0 || slot >= nslots) { bad |= 2; return; }
    if (slot_tile[slot] >= 0) {
      const int last = slot_tile[slot] * nks + ((slot_block[slot] + 1) * nsd - 1) / ks;
      if (cut_steps <= last) bad |= 4;
    }
    slot_tile[slot] = t;
    slot_block[slot] = b;
    if (phase[t & 1] != t / 2) bad |= 8;  // announced on another tile's phase
    tx[t & 1] += bytes_of_block;
    flight.push_back({t, slot, bytes_of_block});
    if (eager) land(flight.size() - 1);
  }
  void finish(int t) {
    if (phase[t & 1] != t / 2 || pending[t & 1] == 0) { bad |= 16; return; }
    pending[t & 1] = 0;
    finished = t + 1;
    complete(t & 1);
  }
  void drain(int t) {
    land_tile(t);
    if (phase[t & 1] <= t / 2) bad |= 32;  // a phase that cannot complete: the drain runs out
  }
};

int main() {
  long runs = 0;
  for (int nsd : {1, 2, 3, 4, 5, 7, 8, 11, 15, 16})
    for (int nb : {1, 2, 3, 7, 8, 17, 40})
      for (int nslots = nb; nslots <= 2 * nb; nslots += nb > 8 ? 5 : 1)
        for (int ntile : {0, 1, 2, 3, 5})
          for (int eager : {0, 1})
            for (int give_up = -1; give_up <= ntile * nb; ++give_up) {
              Model m;
              m.nb = nb; m.nsd = nsd; m.ks = 16; m.nks = (nb * nsd + 15) / 16;
              m.nslots = nslots; m.ntile = ntile; m.give_up = give_up; m.eager = eager != 0;
              m.bytes_of_block = 128L * nsd * 8;
              m.slot_tile.assign(nslots, -1);
              m.slot_block.assign(nslots, -1);
              const bool ok = block_ring_load<16>(m, ntile, nb, nslots, nsd, m.nks);
              const bool gave_up = give_up >= 0 && m.waits > give_up;
              ++runs;
              if (m.bad || !m.flight.empty() || ok == gave_up) {
                std::printf("nsd %d nb %d nslots %d ntile %d eager %d give_up %d: bad %d, in flight %zu, ok %d\n", nsd,
                            nb, nslots, ntile, eager, give_up, m.bad, m.flight.size(), (int)ok);
                return 1;
              }
            }
  std::printf("%ld runs\n", runs);
  return 0;
}
"""


def test_nothing_in_flight_when_the_walk_returns(tmp_path):
    src, exe = tmp_path / "model.cpp", tmp_path / "model"
    src.write_text(MODEL)
    subprocess.run(["g++", "-O1", "-std=c++17", "-Wall", "-Werror", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
