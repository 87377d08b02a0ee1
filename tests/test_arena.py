"""Device memory of the engines (csrc/arena.cu, host code) over a stand-in for
cudaMalloc with little memory: what freed blocks an arena keeps, and that
nothing it keeps makes another allocation fail."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "graph500-bfs_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include "engine.h"
using namespace b200bfs;

static size_t g_room = 0, g_used = 0;
static std::map<void*, size_t> g_blocks;
extern "C" cudaError_t cudaMalloc(void** p, size_t n) {
  if (g_used + n > g_room) return cudaErrorMemoryAllocation;
  *p = malloc(1);
  g_blocks[*p] = n;
  g_used += n;
  return cudaSuccess;
}
extern "C" cudaError_t cudaFree(void* p) {
  if (!g_blocks.count(p)) abort();
  g_used -= g_blocks[p];
  g_blocks.erase(p);
  free(p);
  return cudaSuccess;
}
extern "C" cudaError_t cudaGetLastError() { return cudaSuccess; }

constexpr size_t M = 1 << 20;
#define CHECK(x) do { if (!(x)) { printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)

static bool fails(DeviceArena& a, size_t n) {
  try {
    a.free(a.alloc(n, "test"));
    return false;
  } catch (const Error& e) {
    return e.code == B200BFS_ERR_OOM;
  }
}

// a block that one engine keeps is another's when the device is full
static int others() {
  g_room = 100 * M;
  DeviceArena a, b, c;
  a.open(0);
  b.open(0);
  c.open(1);  // (the stand-in has one memory; only a and b are on one device)
  a.settle(64 * M);
  c.settle(64 * M);
  a.free(a.alloc(60 * M, "kept"));
  CHECK(g_used == 60 * M);
  void* p = b.alloc(60 * M, "second engine");
  CHECK(g_used == 60 * M);
  b.free(p);
  void* q = c.alloc(60 * M, "other device");
  c.free(q);
  CHECK(g_used == 60 * M && fails(b, 60 * M));  // not taken from there
  c.settle(0);
  CHECK(!fails(b, 60 * M) && fails(b, 101 * M));
  return 0;
}

// an arena's own blocks are used again, or make room for it
static int own() {
  g_room = 100 * M;
  DeviceArena a;
  a.open(0);
  a.hold(90 * M);
  void* p = a.alloc(60 * M, "x");
  a.free(p);
  CHECK(a.alloc(55 * M, "reused") == p && a.in_use() == 55 * M);
  a.free(p);
  p = a.alloc(80 * M, "larger");
  CHECK(g_used == 80 * M);
  a.free(p);
  a.settle(0);
  CHECK(g_used == 0 && a.in_use() == 0);
  return 0;
}

// what is kept stays within the limit, oldest out first
static int limit() {
  g_room = 1000 * M;
  DeviceArena a;
  a.open(0);
  a.hold(30 * M);
  void* x[5];
  for (int i = 0; i < 5; ++i) x[i] = a.alloc((10 + 3 * i) * M, "x");
  for (int i = 0; i < 5; ++i) {
    a.free(x[i]);
    CHECK(g_used - a.in_use() <= 30 * M);
  }
  CHECK(g_used == 22 * M);
  a.free(a.alloc(31 * M, "beyond the limit"));
  CHECK(g_used == 22 * M);
  a.settle(0);
  return 0;
}

// with a budget nothing is kept
static int budget() {
  g_room = 1000 * M;
  SharedBudget sb;
  DeviceArena a(50 * M), b;
  a.open(0);
  a.hold(~0ull);
  b.open(0);
  b.set_shared(&sb);
  b.hold(~0ull);
  for (DeviceArena* x : {&a, &b}) {
    void* p = x->alloc(40 * M, "x");
    CHECK(x != &a || fails(a, 11 * M));
    x->free(p);
    CHECK(g_used == 0 && x->in_use() == 0 && sb.used == 0);
  }
  return 0;
}

// buffers that the owner can do without give way to an allocation that fails,
// for want of budget or of memory
static int spare() {
  g_room = 100 * M;
  DeviceArena a(50 * M), b;
  b.open(0);
  b.settle(64 * M);
  for (DeviceArena* x : {&a, &b}) {
    void* p = x->alloc(30 * M, "spare");
    int asked = 0;
    x->on_full([&] {
      ++asked;
      if (!p) return false;
      x->free(p);
      p = nullptr;
      return true;
    });
    CHECK(!fails(*x, 20 * M) && asked == 0);
    CHECK(!fails(*x, x == &a ? 50 * M : 100 * M) && asked == 1);
    CHECK(fails(*x, 101 * M) && asked == 2);
    x->settle(0);
  }
  return 0;
}

int main(int, char** argv) {
  const char* names[] = {"others", "own", "limit", "budget", "spare"};
  int (*tests[])() = {others, own, limit, budget, spare};
  for (int i = 0; i < 5; ++i)
    if (!strcmp(argv[1], names[i])) return tests[i]();
  return 2;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("arena")
    src = d / "arena_test.cc"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, "-I/usr/local/cuda/include", "-o",
                    str(d / "arena"), str(src), "-x", "c++", os.path.join(CSRC, "arena.cu")],
                   check=True)
    return str(d / "arena")


@pytest.mark.parametrize("name", ["others", "own", "limit", "budget", "spare"])
def test_arena(program, name):
    p = subprocess.run([program, name], capture_output=True, text=True)
    assert p.returncode == 0, p.stdout
