"""The books of the device blocks kept between allocations (kept_blocks.hpp),
with a pool of the host's own: who gets a kept block, the limits, and an
allocation that finds the pool full while other streams keep blocks."""
import os
import subprocess

from conftest import ROOT

PROGRAM = r"""
#include "kept_blocks.hpp"
#include <cstdio>
#include <cstdlib>
#include <set>
using namespace osh;
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); std::exit(1); } } while (0)

// a pool of `room` bytes; a block is free to any stream once it is waited for
struct Pool {
  bool full = false;
  size_t room;
  std::map<void*, size_t> out;
  std::map<void*, size_t> pending;   // freed on a stream: bytes until it is waited for
  char* next = (char*)0x1000;
  void* alloc(size_t bytes, void*)
  {
    if (bytes > room) { full = true; return nullptr; }
    room -= bytes;
    void* p = next;
    next += 16;
    out[p] = bytes;
    return p;
  }
  void free(void* p, void* s)
  {
    CHECK(out.count(p));
    pending[s] += out[p];
    out.erase(p);
  }
  void wait(void* s) { room += pending[s]; pending.erase(s); }
};

void* S(int k) { return (void*)(uintptr_t)(k * 64); }

void* get(BlockTable& t, Pool& pool, size_t bytes, void* s)
{
  size_t rounded = bytes;
  u_int32_t cls = 0;
  bool const small = bytes <= BLOCK_MAX;
  if (small) {
    cls = block_class(bytes, &rounded);
    if (void* p = t.take(0, s, cls)) return p;
  }
  void* p = alloc_or_drop(t, pool, 0, rounded, s);
  if (p) { if (small) t.made(p, 0, cls); else t.not_a_block(p); }
  return p;
}
void put(BlockTable& t, Pool& pool, void* p, void* s)
{
  if (!t.keep(p, s, true)) { pool.free(p, s); pool.wait(s); }
}

int main()
{
  for (size_t b = 1; b <= BLOCK_MAX; b = b < 4096 ? b + 1 : b * 33 / 32 + 1) {
    size_t r = 0;
    u_int32_t const c = block_class(b, &r);
    CHECK(c < BLOCK_CLASSES && r >= b && r == class_bytes(c) && (b <= 512 || r <= b + b / 4 + 1));
  }
  {  // a kept block goes to its own stream, class and device alone
    BlockTable t;
    Pool pool{false, (size_t)1 << 30};
    void* p = get(t, pool, 3000, S(1));
    put(t, pool, p, S(1));
    CHECK(t.kept_bytes(0) == 3072);
    CHECK(!t.take(0, S(2), block_class(3000, new size_t)));
    CHECK(!t.take(1, S(1), block_class(3000, new size_t)));
    CHECK(!t.take(0, S(1), block_class(4000, new size_t)));
    CHECK(get(t, pool, 2900, S(1)) == p && t.kept_bytes(0) == 0);
  }
  {  // the limits: of a stream, and of the device
    BlockTable t;
    Pool pool{false, (size_t)64 << 30};
    size_t const per_stream = KEEP_MAX / BLOCK_MAX, most = KEEP_DEVICE / KEEP_MAX;
    for (size_t s = 1; s <= most + 2; ++s) {
      std::vector<void*> v;
      for (size_t k = 0; k < per_stream + 3; ++k) v.push_back(get(t, pool, BLOCK_MAX, S(s)));
      for (void* p : v) put(t, pool, p, S(s));
      CHECK(t.kept_bytes(0) == (s < most ? s : most) * KEEP_MAX);
    }
    CHECK(t.drop(0, S(1)).size() == per_stream);
    CHECK(t.kept_bytes(0) == (most - 1) * KEEP_MAX);
    CHECK(t.drop(0, S(1)).empty());
  }
  {  // a full pool: the blocks that other streams keep are given back to it
    BlockTable t;
    Pool pool{false, (size_t)100 << 20};
    for (int s = 1; s <= 4; ++s) {
      std::vector<void*> v;
      for (int k = 0; k < 5; ++k) v.push_back(get(t, pool, BLOCK_MAX, S(s)));
      for (void* p : v) put(t, pool, p, S(s));
    }
    CHECK(t.kept_bytes(0) == (size_t)80 << 20 && pool.room == (size_t)20 << 20);
    void* large = get(t, pool, (size_t)90 << 20, S(9));
    CHECK(large);
    CHECK(t.kept_bytes(0) == 0);
    CHECK(!get(t, pool, (size_t)90 << 20, S(9)));  // out of memory for good
    put(t, pool, large, S(9));
    CHECK(pool.room == (size_t)100 << 20);
  }
  std::printf("ok\n");
}
"""


def test_books(tmp_path):
    src, exe = tmp_path / "books.cpp", tmp_path / "books"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-o", str(exe), str(src),
                    "-I", os.path.join(ROOT, "omega_h_v1_b200", "csrc")], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout + r.stderr
