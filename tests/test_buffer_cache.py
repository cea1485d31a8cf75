"""Bookkeeping of the device buffers kept between solves (buffer_cache.h), on
the CPU with a fake allocator and two context ids: each context keeps at most
its own 2 GiB, evicts and gives up its own buffers only, and every buffer that
leaves the cache without being handed out is freed exactly once, while its
context is current."""
import os
import subprocess

import pytest

from libpt_b200 import build

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <map>
#include <vector>
#include "buffer_cache.h"
using namespace ptb;

static std::map<void *, uint64_t> owner;   // live buffers and their context
static std::map<void *, size_t> bytes_of;
static uint64_t current;
static int bad;
#define CHECK(x) do { if (!(x)) { ++bad; std::printf("%d: %s\n", __LINE__, #x); } } while (0)

static void fake_free(void *p) {
  CHECK(owner.count(p) && owner[p] == current);
  owner.erase(p);
  bytes_of.erase(p);
}
static void *fake_malloc(size_t n) {
  static uintptr_t next = 4096;
  void *p = (void *)(next += 4096);
  owner[p] = current;
  bytes_of[p] = n;
  return p;
}
static size_t live(uint64_t ctx) {
  size_t s = 0;
  for (auto &o : owner) if (o.second == ctx) s += bytes_of[o.first];
  return s;
}

int main() {
  BufferCache c(fake_free);
  const size_t M = (size_t)1 << 20;
  size_t n = 0;
  // a solve's buffers in either context in turn, past the bound of both
  std::srand(1);
  for (int r = 0; r < 200; ++r) {
    current = 1 + r % 2;
    std::vector<std::pair<void *, size_t>> held;
    for (int b = 0; b < 20; ++b) {
      const size_t want = BufferCache::rounded(M * (1 + std::rand() % 300));
      void *p = c.take(current, want, &n);
      if (!p) p = fake_malloc(n = want);
      CHECK(owner.count(p) && owner[p] == current);
      CHECK(n >= want && n == bytes_of[p]);
      held.push_back({p, n});
    }
    for (auto &h : held) c.give(current, h.first, h.second);
    // nothing is lost: what is live is what the cache keeps, within its bound
    CHECK(live(1) <= KEEP_BYTES && live(2) <= KEEP_BYTES);
    if (r > 1) CHECK(live(3 - current) > KEEP_BYTES / 2);
  }
  // a buffer of the other context is not handed out
  current = 1;
  CHECK(c.give_up(1) > 0 && live(1) == 0 && live(2) > 0);
  CHECK(c.take(1, M, &n) == nullptr && c.give_up(1) == 0);
  CHECK(c.take(7, M, &n) == nullptr && c.give_up(7) == 0);
  // too large to be kept
  c.give(1, fake_malloc(KEEP_BUFFER + 1), KEEP_BUFFER + 1);
  CHECK(live(1) == 0);
  // the smallest that fits, and not one much larger than asked for
  void *a = fake_malloc(8 * M), *b = fake_malloc(64 * M);
  c.give(1, a, 8 * M);
  c.give(1, b, 64 * M);
  CHECK(c.take(1, 30 * M, &n) == nullptr);
  CHECK(c.take(1, 8 * M, &n) == a && n == 8 * M);
  CHECK(c.take(1, 60 * M, &n) == b && n == 64 * M);
  current = 2;
  const size_t all = live(2);
  CHECK(c.give_up(2) == all && live(2) == 0);
  if (!bad) std::printf("ok\n");
  return bad != 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("cache")
    src = d / "cache.cpp"
    src.write_text(PROGRAM)
    subprocess.run([build.HOST_CXX, "-std=c++17", "-Wall", "-Werror",
                    "-I" + build.CSRC, str(src), "-o", str(d / "cache")],
                   check=True)
    return os.path.join(d, "cache")


def test_contexts_do_not_lose_each_others_buffers(program):
    r = subprocess.run([program], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout
