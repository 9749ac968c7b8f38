"""The shelf of idle stream sets kept between calls (idle_shelf.h), driven on the host with counted
objects in place of streams."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "dogpup_b200" / "csrc"

PROGRAM = r"""
#include <cstdio>
#include "idle_shelf.h"
static int made = 0, destroyed = 0, abandoned = 0;
struct Set {
  bool handles = true;
  Set() { ++made; }
  void abandon() { handles = false; ++abandoned; }
  ~Set() { destroyed += handles; }
};
using Shelf = dgp::IdleShelf<Set>;
static void call(Shelf &s, int dev, unsigned long long ctx) {
  auto t = s.take(dev, ctx);
  if (!t) t = std::make_unique<Set>();
  s.put(dev, ctx, std::move(t));
}
#define CHECK(c) if (!(c)) { std::printf("line %d: made %d destroyed %d abandoned %d\n", __LINE__, made, destroyed, abandoned); return 1; }
int main() {
  {
    Shelf s;
    // six devices in turn, many times: one set each, none lost, none made twice
    for (int r = 0; r < 10; ++r)
      for (int d = 0; d < 6; ++d) call(s, d, 100 + d);
    CHECK(made == 6 && destroyed == 0 && abandoned == 0);
    // device 2's context is reset: its set's handles are forgotten, the others stay
    call(s, 2, 200);
    CHECK(made == 7 && destroyed == 0 && abandoned == 1);
    for (int d = 0; d < 6; ++d) call(s, d, d == 2 ? 200 : 100 + d);
    CHECK(made == 7 && abandoned == 1);
    // seven calls at once on one device: what does not fit is destroyed, not forgotten
    std::unique_ptr<Set> t[7];
    for (auto &x : t)
      if (!(x = s.take(0, 100))) x = std::make_unique<Set>();
    for (auto &x : t) s.put(0, 100, std::move(x));
    CHECK(made == 13 && destroyed == 7 - (int)Shelf::MAX && abandoned == 1);
  }
  CHECK(made == destroyed + abandoned);
  return 0;
}
"""


def test_sets_of_live_contexts_are_never_lost(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no g++")
    (tmp_path / "shelf.cpp").write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-Wall", f"-I{CSRC}", str(tmp_path / "shelf.cpp"), "-o", str(tmp_path / "shelf")],
                   check=True)
    p = subprocess.run([tmp_path / "shelf"], text=True, capture_output=True)
    assert p.returncode == 0, p.stdout
