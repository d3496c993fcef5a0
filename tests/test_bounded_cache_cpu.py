"""Eviction of the cache behind the tensor maps (ops/csrc/bounded_cache.h), compiled for the host with a small limit."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "create_llm_by_cupy_b200" / "ops" / "csrc"

PROGRAM = r"""
#include <cassert>
#include <thread>
#include <vector>
#include "bounded_cache.h"

struct Value { long a[16]; };                          // as large as a tensor map
using Cache = b200::BoundedCache<long, Value, std::hash<long>>;

static bool make(long k, Value* v) {
  for (long& x : v->a) x = 3 * k;
  return true;
}
static bool holds(const Value& v, long k) {
  for (long x : v.a) if (x != 3 * k) return false;
  return true;
}

int main() {
  {  // what one launch looked up stays whole when its later lookups drop every entry
    Cache c(2);
    Value v[5];
    for (long k = 0; k < 5; ++k) assert(c.get(k, &v[k], [&](Value* o) { return make(k, o); }));
    for (long k = 0; k < 5; ++k) assert(holds(v[k], k));
    assert(c.size() <= 2);
  }
  {  // a kept value is not made again; one that could not be made is not kept
    Cache c(4);
    Value v;
    int made = 0;
    for (int i = 0; i < 3; ++i) assert(c.get(7, &v, [&](Value* o) { ++made; return make(7, o); }));
    assert(made == 1 && holds(v, 7));
    assert(!c.get(8, &v, [&](Value*) { ++made; return false; }) && c.size() == 1);
    assert(c.get(8, &v, [&](Value* o) { ++made; return make(8, o); }) && holds(v, 8) && made == 3);
  }
  {  // threads that drop one another's entries all the time
    Cache c(3);
    std::vector<std::thread> ts;
    for (long t = 0; t < 4; ++t)
      ts.emplace_back([&c, t] {
        for (long i = 0; i < 20000; ++i) {
          Value a, b;
          const long ka = (i * 7 + t) % 11, kb = (i * 5 + t) % 13;
          assert(c.get(ka, &a, [&](Value* o) { return make(ka, o); }));
          assert(c.get(kb, &b, [&](Value* o) { return make(kb, o); }));
          assert(holds(a, ka) && holds(b, kb));
        }
      });
    for (auto& t : ts) t.join();
    assert(c.size() <= 3);
  }
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_values_outlive_the_entries_they_came_from(tmp_path):
    src, exe = tmp_path / "cache.cpp", tmp_path / "cache"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-UNDEBUG", "-pthread", "-I", str(CSRC), str(src), "-o", str(exe)], check=True)
    subprocess.run([str(exe)], check=True, timeout=60)
