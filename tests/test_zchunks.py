"""The automatic z chunk (csrc/zchunks.h, host-compiled): a model on its own
fills the GPU with short chunks; models advanced together are not cut shorter
than the work items of all of them need, however small each is."""
import os
import subprocess

from conftest import PKG

CODE = r'''
#include "zchunks.h"
#include <cstdio>
using namespace sgfd;
constexpr int kSms = 148;
#define CHECK(c) do { if (!(c)) { std::printf("%s: edge %d, %d models\n", #c, edge, n); return 1; } } while (0)
static int tiles_of(int computed) { return ((computed + 31) / 32) * ((computed + 7) / 8); }
int main() {
  // one model: both sides of each line of the rule (tiles, planes, chunk)
  const int solo[][3] = {{1, 12, 1}, {14, 54, 2}, {27, 70, 5}, {14, 390, 13}, {31, 196, 14}, {32, 196, 8},
                         {90, 140, 8}, {240, 90, 12}, {341, 256, 16}, {576, 384, 30}, {1024, 512, 48}, {3969, 14, 14}};
  for (auto &c : solo)
    if (solo_chunk(c[0], c[1], kSms) != c[2]) {
      std::printf("solo %d x %d: %d, not %d\n", c[0], c[1], solo_chunk(c[0], c[1], kSms), c[2]);
      return 1;
    }
  // 64 x 8 tiles (FP32, 16 bits): one wave of two CTAs per SM, then as above, or chunks of 16 planes
  const int pairs[][4] = {{20, 80, 6, 6}, {30, 120, 14, 14}, {51, 130, 8, 8}, {66, 170, 8, 16},
                          {123, 81, 8, 14}, {72, 190, 8, 16}, {592, 20, 8, 8}, {592, 46, 16, 16},
                          {144, 256, 16, 16}, {9, 390, 13, 13}};
  for (auto &c : pairs)
    for (int half = 0; half < 2; ++half)
      if (solo_chunk(c[0], c[1], kSms, true, half) != c[2 + half]) {
        std::printf("64 x 8, %d x %d, half %d: %d\n", c[0], c[1], half, solo_chunk(c[0], c[1], kSms, true, half));
        return 1;
      }
  for (int edge = 20; edge <= 400; ++edge) {
    const int nz = edge - 10, t = tiles_of(nz), own = solo_chunk(t, nz, kSms);
    for (int n : {1, 2, 3, 4, 8, 12, 16, 32, 64, 200}) {
      const int64_t all = (int64_t)n * t;
      for (int even = 0; even < 2; ++even) {
        const int zc = graph_batch_chunk(own, all, nz, 3 * kSms, even != 0);
        CHECK(zc >= own && zc <= nz && (zc <= (even ? 8 : 16) || zc == own));
        CHECK(zc == own || zc == nz || !even || zc % 2 == 0);
        if (even && own >= 6) { CHECK(zc == own); continue; }
        // longer than the model's own only while the batch still makes two waves and a half
        CHECK(zc == own || even || zc == 1 || all * ((nz + zc - 2) / (zc - 1)) * 2 >= 5 * 3 * kSms);
        // and never so short that the batch makes more than twice that, unless chunks of 16 planes do
        CHECK(zc >= (even ? 8 : 16) || zc == own || all * ((nz + zc - 1) / zc) <= 5 * 3 * kSms + all);
      }
      const int ctas = 2 * kSms, zc = persistent_chunk(own, all, nz, ctas);
      const int64_t items = all * ((nz + zc - 1) / zc);
      CHECK(zc >= 1 && zc <= nz && (zc <= 16 || zc == own));
      CHECK(own > 16 || zc == 16 || zc == nz || items <= 2 * ctas);
    }
  }
  // batches of many small models: several planes, where each alone takes one or two
  struct { int edge, models, graph, pers; } small[] = {{40, 64, 6, 15}, {64, 12, 8, 16}, {64, 32, 16, 16}, {28, 64, 3, 6}};
  for (auto &c : small) {
    const int edge = c.edge, n = c.models, nz = edge - 10, t = tiles_of(nz), own = solo_chunk(t, nz, kSms);
    CHECK(own <= 2);
    CHECK(graph_batch_chunk(own, (int64_t)n * t, nz, 3 * kSms, false) == c.graph);
    CHECK(persistent_chunk(own, (int64_t)n * t, nz, 2 * kSms) == c.pers);
  }
  std::puts("ok");
  return 0;
}
'''


def test_chunk_rules(tmp_path):
    src = tmp_path / "z.cpp"
    src.write_text(CODE)
    exe = tmp_path / "z"
    inc = os.path.join(PKG, "csrc")
    r = subprocess.run(["g++", "-std=c++17", "-O1", f"-I{inc}", str(src), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout
