"""The slabs that small device blocks are cut from (csrc/slab_arena.cuh), on the host:
random takes and gives against a model (no overlap, alignment, sizes at most twice
or a quarter beyond what is asked for, reuse, the limits), slabs given back by trim()
and at the end, no allocation by give(), and an upstream without memory."""

import shutil
import subprocess
from pathlib import Path

import pytest

SOURCE = r'''
#include "%s"

#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <new>
#include <random>
#include <utility>

static bool forbidden = false;
void* operator new(std::size_t n)
{
  if (forbidden) {
    std::puts("give() allocated");
    std::exit(1);
  }
  if (void* p = std::malloc(n)) return p;
  throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }

#define CHECK(c)                                       \
  do {                                                 \
    if (!(c)) {                                        \
      std::printf("line %%d: %%s\n", __LINE__, #c);      \
      std::exit(1);                                    \
    }                                                  \
  } while (0)

struct State {
  std::map<char*, std::size_t> out;
  std::size_t bytes = 0, calls = 0, limit = SIZE_MAX;
};
struct Up {
  State* s;
  void* allocate(std::size_t n)
  {
    ++s->calls;
    if (s->bytes + n > s->limit) return nullptr;
    char* const p = static_cast<char*>(std::aligned_alloc(256, n));
    s->out[p]     = n;
    s->bytes += n;
    return p;
  }
  void deallocate(void* p, std::size_t n)
  {
    CHECK(s->out.count(static_cast<char*>(p)) && s->out[static_cast<char*>(p)] == n);
    s->out.erase(static_cast<char*>(p));
    s->bytes -= n;
    std::free(p);
  }
};
using Arena = cspt::SlabArena<Up>;

static void walk(unsigned seed, std::size_t first, std::size_t most, std::size_t limit,
                 bool fine)
{
  State st;
  st.limit = limit;
  std::mt19937 rng(seed);
  {
    Arena a(Up{&st}, first, most, fine);
    std::map<char*, std::pair<std::size_t, std::size_t>> live;  // asked, room up to the next block
    for (int step = 0; step < 4000; ++step) {
      bool const shrink = (step / 500) %% 2;
      if (live.empty() || rng() %% 8 >= (shrink ? 6u : 3u)) {
        std::size_t n = std::size_t{1} << (rng() %% 23);
        n += rng() %% n;
        char* const p = static_cast<char*>(a.take(n));
        if (n > Arena::kMaxBlock) CHECK(!p);
        if (!p) continue;
        CHECK(a.owns(p) && reinterpret_cast<std::uintptr_t>(p) %% 256 == 0);
        auto next = live.lower_bound(p);
        CHECK(next == live.end() || p + n <= next->first);
        if (next != live.begin()) {
          auto before = std::prev(next);
          CHECK(before->first + before->second.first <= p);
        }
        bool inside = false;
        for (auto const& s : st.out) inside |= p >= s.first && p + n <= s.first + s.second;
        CHECK(inside);
        live[p] = {n, 0};
      } else {
        auto it = live.begin();
        std::advance(it, rng() %% live.size());
        char* const p       = it->first;
        std::size_t const n = it->second.first;
        live.erase(it);
        forbidden = true;
        CHECK(a.give(p, n));
        forbidden = false;
        if (n %% 3 == 0) {  // reused by size
          void* const again = a.take(n);
          CHECK(again == p);
          CHECK(a.give(again, n));
        }
      }
      CHECK(st.bytes <= most && st.bytes == a.slab_bytes());
      if (step %% 700 == 699) {
        a.trim();
        for (auto const& b : live) CHECK(a.owns(b.first));
        if (live.empty()) CHECK(st.bytes == 0);
      }
    }
    for (auto const& b : live) CHECK(a.give(b.first, b.second.first));
    a.trim();
    CHECK(st.bytes == 0 && st.out.empty());
    char here;
    CHECK(!a.give(&here, 1) && !a.owns(&here));
    void* const p = limit > first ? a.take(1000) : nullptr;  // usable after a trim
    if (limit > first) CHECK(p && a.owns(p));
  }
  CHECK(st.out.empty());
}

int main()
{
  for (unsigned s = 0; s < 6; ++s) {
    walk(s, std::size_t{2} << 20, std::size_t{158} << 20, SIZE_MAX, false);
    walk(s, std::size_t{1} << 20, std::size_t{31} << 20, SIZE_MAX, true);
    walk(s, std::size_t{2} << 20, std::size_t{158} << 20, std::size_t{7} << 20, s %% 2 == 0);
    walk(s, std::size_t{2} << 20, std::size_t{158} << 20, 0, true);
  }
  // the size of a block: what two of them of one slab lie apart
  for (bool fine : {false, true}) {
    State st;
    Arena a(Up{&st}, std::size_t{32} << 20, std::size_t{32} << 20, fine);
    for (std::size_t n = 1; n <= Arena::kMaxBlock / 4; n += 1 + n / 7) {
      char* const p = static_cast<char*>(a.take(n));
      char* const q = static_cast<char*>(a.take(n));
      if (!p || !q) break;
      std::size_t const size = q - p;
      CHECK(size >= n && size %% 256 == 0 &&
            (size <= (fine ? n + n / 4 : 2 * n) || size < n + 256));
    }
  }
  std::puts("ok");
}
'''


def test_slab_arena(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    header = Path(__file__).resolve().parent.parent / "cuspatial_gb300" / "csrc" / "slab_arena.cuh"
    src, exe = tmp_path / "arena.cpp", tmp_path / "arena"
    src.write_text(SOURCE % header)
    subprocess.run([gxx, "-O1", "-std=c++17", str(src), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
