"""Growth policy of a context's device scratch (csrc/arena.h) against an allocator that refuses: memory that a
call must have, memory that only makes it faster (FrodoKEM's operand tiles), stream captures, reserved arenas."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include <map>
#include "arena.h"
using namespace dpkem;

struct Fake final : ArenaMem {
  size_t limit, used = 0, peak = 0;
  int calls = 0, drains = 0;
  std::map<void *, size_t> live;
  explicit Fake(size_t l) : limit(l) {}
  void *alloc(size_t n) override {
    calls++;
    if (used + n > limit) return nullptr;
    void *p = std::malloc(1);
    live[p] = n;
    used += n;
    peak = std::max(peak, used);
    return p;
  }
  void release(void *p) override {
    calls++;
    used -= live.at(p);
    live.erase(p);
    std::free(p);
  }
  void drain() override { drains++; }
};
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)

int main() {
  {  // memory that a call needs: geometric growth within the budget, the exact size where the device has no more
    Fake m(1000);
    Arena a;
    CHECK(a.need(100, 800, m) && a.bytes == 100 && m.drains == 0);
    CHECK(a.need(110, 800, m) && a.bytes == 150 && m.drains == 1);
    CHECK(a.need(700, 800, m) && a.bytes == 700 && !a.need(801, 800, m) && a.bytes == 700);
    Fake t(130);
    Arena b;
    CHECK(b.need(100, 800, t) && b.need(120, 800, t) && b.bytes == 120);
    CHECK(!b.need(131, 800, t) && b.need(120, 800, t));
    a.free_all(m);
    b.free_all(t);
    CHECK(m.used == 0 && t.used == 0 && a.base == nullptr);
  }
  {  // a refused optional size leaves the arena alone and is not asked for again
    Fake m(1000);
    Arena a;
    CHECK(a.need(200, 4000, m));
    void *base = a.base;
    CHECK(!a.want(2000, 4000, m) && a.base == base && a.bytes == 200 && m.drains == 0 && m.live.size() == 1);
    const int calls = m.calls;
    for (int k = 0; k < 3; k++) CHECK(!a.want(2000, 4000, m) && !a.want(2500, 4000, m) && a.need(200, 4000, m));
    CHECK(m.calls == calls && a.base == base);
    CHECK(a.want(300, 4000, m) && a.bytes >= 300 && m.peak <= 1000);
    a.free_all(m);
    CHECK(m.used == 0);
  }
  {  // old and new memory together stay within the budget, else the old goes first and comes back on a refusal
    Fake m(10000);
    Arena a;
    CHECK(a.need(600, 1000, m) && a.want(900, 1000, m) && a.bytes >= 900 && m.peak <= 1000);
    a.free_all(m);
    Fake t(800);
    Arena b;
    CHECK(b.need(600, 1000, t) && !b.want(900, 1000, t) && b.bytes == 600 && t.live.size() == 1);
    const int calls = t.calls;
    CHECK(!b.want(900, 1000, t) && t.calls == calls);
    b.free_all(t);
  }
  {  // a fixed arena serves what it holds and grows for needs only
    Fake m(10000);
    Arena a;
    CHECK(a.need(500, 5000, m));
    a.fix();
    const int calls = m.calls;
    CHECK(a.want(500, 5000, m) && !a.want(501, 5000, m) && m.calls == calls);
    CHECK(a.need(600, 5000, m) && a.bytes == 750);
    a.free_all(m);
  }
  {  // captured memory outlives growth, counts against the budget of optional memory, goes at the end
    Fake m(10000);
    Arena a;
    CHECK(a.need(500, 2000, m));
    void *graph = a.base;
    a.captured();
    CHECK(a.need(1000, 2000, m) && a.base != graph && m.live.count(graph) && m.drains == 0);
    CHECK(!a.want(1600, 2000, m) && a.bytes == 1000 && m.live.count(graph));
    CHECK(a.want(1500, 2000, m) && a.bytes == 1500 && m.live.size() == 2 && m.live.count(graph));
    a.captured();
    CHECK(!a.want(1501, 2000, m) && a.need(1600, 2000, m) && m.live.size() == 3);
    a.free_all(m);
    CHECK(m.used == 0 && m.live.empty());
  }
  std::puts("ok");
  return 0;
}
"""


def test_arena_policy(tmp_path):
    src, exe = tmp_path / "arena.cc", tmp_path / "arena"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", os.path.join(ROOT, "dpcrypto_b200", "csrc"), str(src),
                    "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout
