"""Tiles whose copies a mover warp of the symmetry-adapted stage has in flight
when a bounded wait runs out (csrc/dglm_ring.h), against a walk over the ring
that keeps the set itself: for every ring of the compiled variants, several
lengths and every wait that can run out."""
import subprocess

from exadglm_b200 import build as _build

WALK = r"""
#include <cstdio>
#include <set>
#include "dglm_ring.h"

template <int NB, int NM>
int walk(int total, int mw, int expire) {
  std::set<int> flying;   // loaded, not known to have landed
  for (int it = mw; it < total + NB; it += NM) {
    if (it >= NB && it - NB < total) {
      if (it == expire) {
        std::set<int> got;
        dglm::mover_in_flight<NB, NM>(it, total, [&](int q) { got.insert(q); });
        return got == flying ? 0 : 1;
      }
      flying.erase(it - NB);   // done: its copies landed before the compute warps had it
    }
    if (it < total) flying.insert(it);
  }
  return 0;
}

template <int NB, int NM>
int check() {
  int bad = 0;
  for (int total = 1; total <= 4 * NB + 1; total++)
    for (int mw = 0; mw < NM; mw++)
      for (int expire = NB; expire < total + NB; expire++) bad += walk<NB, NM>(total, mw, expire);
  return bad;
}

int main() {
  const int bad = check<8, 2>() + check<6, 2>() + check<3, 1>() + check<2, 2>();
  printf("%d\n", bad);
  return bad != 0;
}
"""


def test_expired_wait_settles_every_copy_in_flight(tmp_path):
    src, exe = tmp_path / "walk.cpp", tmp_path / "walk"
    src.write_text(WALK)
    subprocess.run(["g++", "-std=c++17", "-I", _build.CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], stdout=subprocess.PIPE, text=True)
    assert r.returncode == 0, f"{r.stdout.strip()} walks leave copies in flight"
