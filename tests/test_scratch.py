"""The buffers a context keeps between calls (lw_scratch.h), on a fake device:
what a captured call has used is never freed before the context closes, and
what is set aside stays smaller than what is in use."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "brams_gb300", "csrc")

FAKE = r"""
#include <cstdio>
#include <cstdlib>
#include <map>
#include "lw_scratch.h"
static std::map<void*, size_t> live;          // what is allocated
static size_t limit = ~size_t(0);             // of the fake device, bytes
static int gets = 0, puts_ = 0;
static size_t used() { size_t n = 0; for (auto& e : live) n += e.second; return n; }
static void* get(size_t n) {
  ++gets;
  if (used() + n > limit) return nullptr;
  void* p = std::malloc(1);
  live[p] = n;
  return p;
}
static void put(void* p) {
  ++puts_;
  if (!live.erase(p)) { std::printf("freed twice\n"); std::exit(1); }
  std::free(p);
}
static const GbAlloc A = {get, put};
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)
int main() {
BODY
  return 0;
}
"""


def _run(tmp_path, body):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no host C++ compiler")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(FAKE.replace("BODY", body))
    subprocess.run([gxx, "-std=c++17", "-Wall", "-I", CSRC, "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def test_a_captured_buffer_outlives_larger_calls(tmp_path):
    _run(tmp_path, """
  GbScratch s;
  CHECK(s.ensure(100, 10, false, A));
  CHECK(s.ensure(80, 10, true, A));           // captured at this address
  void* held = s.p;
  CHECK(s.ensure(1000, 10, false, A) && s.bytes >= 1000 && s.p != held);
  CHECK(live.count(held));                    // a replay may still write there
  CHECK(s.ensure(5000, 10, false, A));        // outgrown without a capture: freed
  CHECK(live.size() == 2 && live.count(held));
  s.close(A);
  CHECK(live.empty() && s.p == nullptr);
""")


def test_capture_keeps_a_smaller_buffer(tmp_path):
    _run(tmp_path, """
  GbScratch s;
  CHECK(s.ensure(100, 10, false, A));
  void* p = s.p;
  const int g = gets;
  CHECK(s.ensure(1000, 60, true, A));         // more passes: nothing is allocated or freed
  CHECK(s.p == p && s.bytes == 100 && gets == g && puts_ == 0);
  CHECK(s.ensure(1000, 200, true, A));        // too small to run with: a new one, the old one stays
  CHECK(live.count(p) && puts_ == 0 && s.bytes >= 1000);
  s.close(A);
  CHECK(live.empty());
""")


def test_what_is_set_aside_is_bounded(tmp_path):
    _run(tmp_path, """
  GbScratch s;
  for (size_t want = 1000; want < 100000; want += 37) {
    CHECK(s.ensure(want, want < 50000 ? want / 20 : want, false, A));
    CHECK(s.ensure(want / 2, want / 20, true, A));
    CHECK(used() <= 2 * s.bytes);             // set aside: less than in use
    CHECK(s.bytes <= 4 * want);
  }
  s.close(A);
  CHECK(live.empty());
""")


def test_less_is_taken_where_less_is_free(tmp_path):
    _run(tmp_path, """
  limit = 300;
  GbScratch s;
  CHECK(s.ensure(1000, 100, false, A) && s.bytes >= 100 && s.bytes <= 300);
  GbScratch t;
  CHECK(!t.ensure(1000, 500, false, A) && t.p == nullptr);
  s.close(A);
""")


def test_a_size_that_did_not_fit_is_not_asked_for_again(tmp_path):
    _run(tmp_path, """
  limit = 300;
  GbScratch s;
  CHECK(s.ensure(1000, 100, false, A));       // 250 of it
  void* p = s.p;
  const size_t n = s.bytes;
  const int g = gets, f = puts_;
  for (int k = 0; k < 5; ++k) {
    CHECK(s.ensure(1000, 100, false, A));
    CHECK(s.ensure(4000, 200, false, A));
    CHECK(s.ensure(90, 10, false, A));
  }
  CHECK(s.p == p && s.bytes == n && gets == g && puts_ == f);
  limit = 1000;                               // a smaller size is still tried
  CHECK(s.ensure(600, 100, false, A) && s.bytes == 600 && live.size() == 1);
  CHECK(s.ensure(1000, 100, false, A) && s.bytes == 600);
  CHECK(!s.ensure(1001, 1001, false, A));     // too little to run with, nothing larger
  limit = 5000;
  CHECK(s.ensure(2000, 2000, false, A) && s.bytes == 2000 && live.size() == 1);
  s.close(A);
  CHECK(live.empty());
""")


def test_a_buffer_that_does_is_not_given_up_for_a_larger_one(tmp_path):
    _run(tmp_path, """
  GbScratch s;
  CHECK(s.ensure(300, 100, false, A));
  void* p = s.p;
  limit = 400;                                // no room for a larger one beside it
  CHECK(s.ensure(5000, 100, false, A) && s.p == p && live.count(p));
  CHECK(s.ensure(5000, 100, false, A) && s.p == p && puts_ == 0);
  CHECK(s.ensure(350, 350, false, A) && s.bytes == 350 && live.size() == 1);  // needed: the old one makes room
  s.close(A);
  CHECK(live.empty());
""")


def test_nothing_is_freed_under_capture(tmp_path):
    _run(tmp_path, """
  GbScratch s;
  CHECK(s.ensure(300, 100, false, A));
  void* p = s.p;
  limit = 300;
  CHECK(!s.ensure(1000, 500, true, A));       // the call fails, the buffer stays
  CHECK(live.count(p) && puts_ == 0 && s.p == p && s.bytes == 300);
  limit = 2000;
  CHECK(s.ensure(1000, 500, false, A) && s.bytes == 1000);  // and the size is tried again afterwards
  s.close(A);
""")
