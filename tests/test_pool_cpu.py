"""The scratch that contexts keep (ed_pool.h), with a host allocator of limited
room: kept and reused, given back to an allocation that does not fit, never
while in use, and sound with several threads."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include "ed_pool.h"
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <thread>
static const size_t ROOM = 1000;
static std::mutex m;
static std::map<void*, size_t> held;
static size_t used = 0;
struct Mem {
  static int get(void** p, size_t n) {
    std::lock_guard<std::mutex> lk(m);
    *p = nullptr;
    if (n == 666) return 7;  // a failure that is not about room
    if (used + n > ROOM) return 2;
    *p = malloc(n ? n : 1);
    held[*p] = n;
    used += n;
    return 0;
  }
  static bool full(int rc) { return rc == 2; }
  static void put(void* p) {
    std::lock_guard<std::mutex> lk(m);
    if (!held.count(p)) { printf("freed twice\n"); exit(1); }
    used -= held[p];
    held.erase(p);
    free(p);
  }
};
#define CHECK(c) do { if (!(c)) { printf("line %d: %s\n", __LINE__, #c); return 1; } } while (0)
int main() {
  ed_scratch_pool<Mem> pool;
  ed_scratch_slot a, b, other;
  other.device = 1;
  pool.add(&a); pool.add(&b); pool.add(&other);
  bool own, own2;
  void* p = pool.take(&a, 300, 500, &own);
  CHECK(p && !own && used == 300);
  void* q = pool.take(&a, 100, 500, &own2);  // in use: the call's own
  CHECK(q && own2 && q != p && used == 400);
  pool.give(&a, q, own2);
  CHECK(used == 300);
  void* x = nullptr;
  CHECK(pool.alloc(&x, 800, 0) == 2 && !x && a.ptr == p);  // busy: stays
  pool.give(&a, p, own);
  CHECK(used == 300 && pool.take(&a, 200, 500, &own) == p && !own);  // kept
  pool.give(&a, p, own);
  p = pool.take(&other, 100, 500, &own);
  pool.give(&other, p, own);
  p = pool.take(&b, 200, 500, &own);
  pool.give(&b, p, own);
  CHECK(used == 600);
  CHECK(pool.alloc(&x, 666, 0) == 7 && used == 600);  // nothing given back for it
  CHECK(pool.alloc(&x, 800, 0) == 0 && x && !a.ptr && !b.ptr && other.ptr && used == 900);
  Mem::put(x);
  CHECK(pool.take(&a, 950, 2000, &own) == nullptr && !a.busy && used == 100);  // the other device's slot stays
  pool.trim(&other);
  CHECK(used == 0);
  p = pool.take(&a, 400, 500, &own);
  pool.trim(&a);  // in use: stays
  CHECK(used == 400);
  pool.give(&a, p, own);
  p = pool.take(&b, 700, 500, &own);  // too large to keep: a's room is given back for it
  CHECK(p && own && !a.ptr && used == 700);
  pool.give(&b, p, own);
  CHECK(used == 0);
  p = pool.take(&a, 50, 500, &own);
  pool.give(&a, p, own);
  pool.remove(&a);
  CHECK(used == 0);
  pool.remove(&b); pool.remove(&other);
  std::atomic<int> bad{0};
  std::vector<std::thread> t;
  for (int k = 0; k < 8; ++k)
    t.emplace_back([&, k] {
      ed_scratch_slot s;
      pool.add(&s);
      for (int i = 0; i < 4000; ++i) {
        bool o;
        const size_t n = 40 + (size_t)((i * 7 + k * 13) % 60);
        char* c = (char*)pool.take(&s, n, 80, &o);
        if (!c) { bad++; continue; }  // eight of at most 99 fit
        c[0] = c[n - 1] = (char)k;
        void* y = nullptr;
        if (i % 5 == 0 && pool.alloc(&y, 150, 0) == 0) Mem::put(y);
        if (c[0] != (char)k || c[n - 1] != (char)k) bad += 1000;
        pool.give(&s, c, o);
        if (i % 11 == 0) pool.trim(&s);
      }
      pool.remove(&s);
    });
  for (auto& th : t) th.join();
  CHECK(bad < 1000);
  CHECK(used == 0 && held.empty());
  return 0;
}
"""


def test_scratch_pool(tmp_path):
    f = tmp_path / 'pool.cpp'
    f.write_text(SRC)
    exe = tmp_path / 'pool'
    r = subprocess.run(['g++', '-std=c++17', '-O1', '-g', '-Wall', '-Wextra', '-pthread',
                        '-I' + os.path.join(ROOT, 'lsquantumed_gb300', 'csrc'), str(f), '-o', str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
