"""The growing scratch block of a context (csrc/scratch.h): a block that a recorded launch sequence points at survives growth, one that
none points at is given back, and what is kept stays bounded.  Plain C++: compiled and run here without a GPU."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r'''
#include <cstdio>
#include <cstdlib>
#include <map>
#include "scratch.h"
std::map<void*, uint64_t> live;
uint64_t room = ~0ull;
int take(void** p, uint64_t n) { uint64_t t = n; for (auto& b : live) t += b.second; if (t > room) return 2; *p = malloc(1); live[*p] = n; return 0; }
void give(void* p) { if (!live.erase(p)) exit(9); free(p); }
uint64_t total() { uint64_t t = 0; for (auto& b : live) t += b.second; return t; }
int main() {
  const uint64_t MB = 1ull << 20;
  {   // no recording: one block at a time, the size asked for
    p0p::Scratch s;
    if (s.grow(100, take, give) || s.bytes != 8 * MB) return 1;
    if (s.grow(9 * MB + 1, take, give) || s.bytes != 10 * MB || live.size() != 1) return 2;
    s.clear(give); if (!live.empty()) return 3;
  }
  {   // recorded: the block stays until the context closes; many recordings and growths stay bounded
    p0p::Scratch s;
    s.grow(100, take, give); void* first = s.ptr; s.recorded = true;
    if (s.grow(9 * MB, take, give) || !live.count(first) || s.ptr == first || s.bytes != 12 * MB || s.recorded) return 4;
    for (int i = 0; i < 200; i++) {
      s.recorded = true; void* old = s.ptr;
      if (s.grow(s.bytes + MB / 2, take, give) || !live.count(old)) return 5;
      if (total() > 3 * s.bytes) return 6;
      if (s.bytes > (1ull << 40)) break;
    }
    s.clear(give); if (!live.empty()) return 7;
  }
  {   // no room for the larger size: the size asked for; no room at all: the kept block stays in use
    p0p::Scratch s;
    s.grow(100 * MB, take, give); s.recorded = true; room = 210 * MB;
    if (s.grow(105 * MB, take, give) || s.bytes != 105 * MB || live.size() != 2) return 8;
    s.recorded = true; void* cur = s.ptr;
    if (s.grow(120 * MB, take, give) != 2 || s.ptr != cur || s.bytes != 105 * MB || !s.recorded) return 10;
    s.clear(give); if (!live.empty()) return 11;
    if (s.grow(300 * MB, take, give) != 2 || s.ptr || s.bytes) return 12;
  }
  std::puts("ok");
  return 0;
}
'''


def test_scratch_blocks(tmp_path):
    src = tmp_path / "scratch.cpp"; exe = tmp_path / "scratch"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "p0pc0rn_kernels_b200", "csrc"), str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", (r.returncode, r.stdout, r.stderr)
