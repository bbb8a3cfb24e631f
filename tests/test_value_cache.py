"""The table that the launchers keep their tensor maps in (csrc/value_cache.h), compiled for the host."""
import os
import subprocess

from conftest import ROOT

PROGRAM = r"""
#include "value_cache.h"

#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <thread>
#include <vector>

struct Value { unsigned long long word[16]; };
static std::atomic<int> made{0};
static int make(int key, Value *v) {
  if (key < 0) return 7;
  ++made;
  for (auto &w : v->word) w = (unsigned long long)key;
  return 0;
}
static bool is(const Value &v, int key) {
  for (auto w : v.word)
    if (w != (unsigned long long)key) return false;
  return true;
}
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)

int main() {
  orion::ValueCache<int, Value> cache(2);
  auto get = [&](int key, Value *v) { return cache.get(key, v, [&](Value *o) { return make(key, o); }); };
  // a launch's three values in a table for two
  Value a, b, c;
  CHECK(!get(1, &a) && !get(2, &b) && !get(3, &c));
  CHECK(is(a, 1) && is(b, 2) && is(c, 3) && made == 3);
  // only the oldest made room
  CHECK(!get(2, &b) && !get(3, &c) && made == 3);
  CHECK(!get(1, &a) && is(a, 1) && made == 4);
  // a status is handed on, and what could not be made is not kept
  CHECK(get(-1, &a) == 7 && get(-1, &a) == 7 && !get(3, &c) && is(c, 3) && made == 4);
  // threads that take each other's room
  std::atomic<int> wrong{0};
  std::vector<std::thread> threads;
  for (int t = 0; t < 8; ++t)
    threads.emplace_back([&, t] {
      for (int i = 0; i < 20000; ++i) {
        Value v[3];
        for (int k = 0; k < 3; ++k)
          if (get(t + i + k, &v[k])) ++wrong;
        for (int k = 0; k < 3; ++k)
          if (!is(v[k], t + i + k)) ++wrong;
      }
    });
  for (auto &t : threads) t.join();
  CHECK(wrong == 0);
  return 0;
}
"""


def test_values_outlive_their_place_in_the_table(tmp_path):
    source, program = tmp_path / "cache.cpp", tmp_path / "cache"
    source.write_text(PROGRAM)
    csrc = os.path.join(ROOT, "orionserve-rs_b200", "csrc")
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-fsanitize=address", "-pthread", "-I", csrc, str(source), "-o", str(program)], check=True)
    r = subprocess.run([str(program)], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=120)
    assert r.returncode == 0, r.stdout[-2000:]
