"""How the clusters of a grid are handed out (csrc/tile_draw.cuh), compiled for the host against a grid that is a counter:
every tile published once, one request at a time, none after an empty answer; and when a wait is abandoned at any point, no
answer is left on its way and no cluster is left to start."""
import subprocess

from .conftest import PKG_ROOT

SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "tile_draw.cuh"
using namespace moe::tc;

#define CHECK(c) do { if (!(c)) { std::printf("line %d: %s (clusters %d, total %d, event %d, broken %d)\n", __LINE__, #c, \
                                              clusters, total, fail_at, broken); std::exit(1); } } while (0)

int clusters, total, fail_at, broken;  // fail_at: which wait is abandoned; broken: answers stop coming from there on

struct Port {
  int next = 1;       // first cluster that has not started
  int waits = 0;
  bool pending = false, seen_empty = false, arrived = false;
  bool bad() { return waits++ == fail_at; }
  void request() { CHECK(!pending); CHECK(!seen_empty); pending = true; arrived = false; }
  bool wait() { CHECK(pending); if (bad()) return false; arrived = true; return true; }
  bool wait_through() { CHECK(pending); if (broken) return false; arrived = true; return true; }
  int answer() {
    CHECK(pending && arrived);
    pending = false;
    if (next >= clusters) { seen_empty = true; return -1; }
    return 2 * next++;
  }
};

void pair_form() {
  Port port;
  std::vector<int> got;
  hand_out_tiles<2>(port, total, 0, [&](int tile) { if (port.bad()) return false; got.push_back(tile); return true; });
  const bool abandoned = port.waits > fail_at;
  if (!abandoned) {
    CHECK((int)got.size() == total + 1 && got.back() == -1);
    for (int i = 0; i < total; ++i) CHECK(got[i] == i);
  }
  if (!broken) CHECK(!port.pending && port.next == clusters && port.seen_empty);
}

// a thread with work of its own between the request and its answer, as the producer of the single-CTA weight gradient
void own_work_form() {
  Port port;
  ClusterDraw<Port> draw(port);
  int next = 0, done = 0;
  bool ok = true;
  while (ok) {
    const int item = next;
    if (port.bad()) break;  // publish
    if (item >= 0) draw.ask();
    if (item < 0) break;
    for (int i = 0; i < 2 && ok; ++i) ok = !port.bad();
    if (!ok) break;
    ++done;
    const int cta = draw.collect();
    if (cta == ClusterDraw<Port>::ABANDONED) break;
    next = cta < 0 ? -1 : cta / 2;
  }
  draw.leave();
  if (port.waits <= fail_at) CHECK(done == clusters);
  if (!broken) CHECK(!port.pending && port.next == clusters && port.seen_empty);
}

int main() {
  for (clusters = 1; clusters <= 9; ++clusters)
    for (total = 0; total <= clusters; ++total)
      for (fail_at = 0; fail_at <= 6 * clusters + 4; ++fail_at)
        for (broken = 0; broken < 2; ++broken) { pair_form(); own_work_form(); }
  return 0;
}
"""


def test_handing_out_ends_with_nothing_left(tmp_path):
    src = tmp_path / "draw.cpp"
    src.write_text(SOURCE)
    exe = tmp_path / "draw"
    subprocess.run(["g++", "-std=c++17", "-Wall", "-I", str(PKG_ROOT / "csrc"), str(src), "-o", str(exe)], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert res.returncode == 0, res.stdout
