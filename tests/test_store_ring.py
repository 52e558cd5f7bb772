"""The pieces that a product's results leave through (csrc/store_ring.h), compiled and run on the host against a queue that reads as
late as its waits allow: no piece is filled while a request may still be reading it, also where some pieces send nothing."""
import shutil
import subprocess

import pytest

PROGRAM = r"""
#include "store_ring.h"
#include <cstdio>
#include <vector>

struct Thread {                           // a thread's requests in groups; a group is read only when a wait says so
  std::vector<std::vector<unsigned>> groups;
  std::vector<unsigned> open;
  size_t read = 0;
  bool reading(unsigned place) const {
    for (size_t g = read; g < groups.size(); ++g)
      for (unsigned p : groups[g]) if (p == place) return true;
    for (unsigned p : open) if (p == place) return true;
    return false;
  }
};
struct Queue {
  Thread* t;
  void commit() const { t->groups.push_back(t->open); t->open.clear(); }
  template <int N> void wait_read() const { if (t->groups.size() > N + t->read) t->read = t->groups.size() - N; }
};

template <int PIECES>
int overwritten(unsigned pattern, int pieces) {
  Thread t;
  StoreRing<PIECES> ring;
  int bad = 0;
  for (int i = 0; i < pieces; ++i) {
    ring.reuse(true, Queue{&t});
    const unsigned place = ring.place();
    bad += t.reading(place);
    ring.post(true, pattern >> i & 1, Queue{&t}, [&] { t.open.push_back(place); });
  }
  return bad;
}

int main() {
  int bad = 0, most = 0;
  for (unsigned pattern = 0; pattern < 1u << 12; ++pattern) {
    bad += overwritten<2>(pattern, 12) + overwritten<3>(pattern, 12);
    Thread t;                             // ... and no wait is longer than it has to be: two pieces are in flight
    StoreRing<2> ring;
    for (int i = 0; i < 12; ++i) {
      ring.reuse(true, Queue{&t});
      ring.post(true, pattern >> i & 1, Queue{&t}, [&] { t.open.push_back(ring.place()); });
      if ((int)(t.groups.size() - t.read) > most) most = (int)(t.groups.size() - t.read);
    }
  }
  std::printf("%d %d\n", bad, most);
}
"""


def test_no_piece_is_filled_while_it_may_be_read(tmp_path):
    from gemmars_b200.csrc import build
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no C++ compiler")
    (tmp_path / "ring.cc").write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-Wall", "-Werror", "-I", build.HERE, str(tmp_path / "ring.cc"), "-o", str(tmp_path / "ring")], check=True)
    out = subprocess.run([str(tmp_path / "ring")], check=True, capture_output=True, text=True).stdout.split()
    assert out == ["0", "2"]
