"""The engine's buffers after an allocation that fails (on the host, with a stand-in for the CUDA
allocator: no GPU).

Every group of buffers is grown with each of its allocations failing in turn.  Afterwards the engine
holds no pointer that was freed, and a later request, of any size, ends with every buffer of the
group there and large enough; nothing is freed twice and nothing is left over at the end.
"""

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "blackhole_nebula_simulator_b200", "csrc")

ALLOCATOR = r"""
#include <cstddef>
#include <cstdint>
#include <map>

std::map<void*, size_t> live;  // what the stand-in handed out, with its size
long fail_at = -1, made = 0, bad_frees = 0;
static size_t next_address = 1 << 20;

static int give(void** p, size_t bytes) {
  if (made++ == fail_at) return 2;  // cudaErrorMemoryAllocation
  *p = (void*)next_address;
  next_address += (bytes + 511) / 256 * 256;
  live[*p] = bytes;
  return 0;
}
static int take(void* p) {
  if (p && !live.erase(p)) bad_frees += 1;
  return 0;
}
extern "C" {
int cudaMalloc(void** p, size_t b) { return give(p, b); }
int cudaMallocHost(void** p, size_t b) { return give(p, b); }
int cudaFree(void* p) { return take(p); }
int cudaFreeHost(void* p) { return take(p); }
int cudaMemset(void*, int, size_t) { return 0; }
int cudaGetLastError() { return 0; }
const char* cudaGetErrorName(int) { return "out of memory"; }
const char* cudaGetErrorString(int) { return "out of memory"; }
int cudaEventCreate(void** e) { return give(e, 1); }
int cudaEventDestroy(void* e) { return take(e); }
int cudaEventRecord(void*, void*) { return 0; }
int cudaEventSynchronize(void*) { return 0; }
int cudaEventElapsedTime(float*, void*, void*) { return 0; }
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
}
"""

HARNESS = r"""
#include <cstdlib>
#include <map>
#include <vector>
#include "engine.cuh"

extern std::map<void*, size_t> live;
extern long fail_at, made, bad_frees;

namespace nbk {
size_t cub_bytes_needed(int64_t n, int64_t m) { return 64 * n + 8 * m; }
size_t workspace_cub_bytes(int64_t n) { return 80 * n; }
size_t deposit_cub_bytes(int64_t n) { return 72 * n; }
}  // namespace nbk
using namespace nbk;

struct Need {
  const char* name;
  void* p;
  size_t bytes;
};
struct Group {
  const char* name;
  int (*ensure)(Engine&, int64_t);
  std::vector<Need> (*needs)(Engine&, int64_t);
};
#define N(f, b) {#f, (void*)E.f, (size_t)(b)}
static const std::vector<Group> groups = {
    {"n", [](Engine& E, int64_t n) { return E.ensure_n(n); },
     [](Engine& E, int64_t n) -> std::vector<Need> {
       return {N(d_err, 16), N(h_err, 16), N(bbox, 64), N(h_red, 512), N(d_rowmax, 128), N(h_build, 32),
               N(bbox_part, 1), N(keys_a, 8 * n), N(keys_b, 8 * n), N(vals_a, 4 * n), N(counts, 8 * (n + 1)),
               N(red, 1), N(lists.perm, 4 * n), N(lists.inv_perm, 4 * n), N(lists.spos, 32 * n),
               N(lists.off, 8 * (n + 1)), N(cub_tmp, cub_bytes_needed(n, 0))};
     }},
    {"nodes", [](Engine& E, int64_t n) { return E.ensure_nodes(n); },
     [](Engine& E, int64_t n) -> std::vector<Need> {
       return {N(node_lo, 32 * n), N(node_hi, 32 * n), N(node_q, 32 * n)};
     }},
    {"sub", [](Engine& E, int64_t n) { return E.ensure_sub(n); },
     [](Engine& E, int64_t n) -> std::vector<Need> {
       return {N(sub_lo, 32 * n), N(sub_hi, 32 * n), N(sub_q, 32 * n)};
     }},
    {"list", [](Engine& E, int64_t n) { return E.ensure_list_capacity(n); },
     [](Engine& E, int64_t n) -> std::vector<Need> { return {N(lists.idx, 4 * n)}; }},
    {"tight", [](Engine& E, int64_t n) { return E.ensure_tight(n); },
     [](Engine& E, int64_t n) -> std::vector<Need> { return {N(tidx, 4 * n)}; }},
    {"leaves", [](Engine& E, int64_t n) { return E.ensure_leaves(n); },
     [](Engine& E, int64_t n) -> std::vector<Need> {
       return {N(leaf_cbase, 8 * n), N(leaf_bbase, 8 * n), N(leaf_ibase, 8 * n), N(leaf_ncand, 4 * n)};
     }},
    {"tiles", [](Engine& E, int64_t n) { return E.ensure_tiles(n, n / 4 + 1, n / 8 + 1); },
     [](Engine& E, int64_t n) -> std::vector<Need> {
       return {N(cands, 4 * n), N(masks, 128 * (n / 4 + 1)), N(items, 8 * (n / 8 + 1)),
               N(part_count, 128 * (n / 8 + 1))};
     }},
    {"deposit", [](Engine& E, int64_t n) { return E.ensure_deposit(n); },
     [](Engine& E, int64_t n) -> std::vector<Need> {
       return {N(dep_k0, 8 * n), N(dep_k1, 8 * n), N(dep_i0, 4 * n), N(dep_i1, 4 * n), N(dep_buf, 96 * n),
               N(cub_tmp, deposit_cub_bytes(n))};
     }},
    {"shells", [](Engine& E, int64_t n) { return E.ensure_shells(n); },
     [](Engine& E, int64_t n) -> std::vector<Need> { return {N(dep_shells, 16 * n)}; }},
    {"bricks", [](Engine& E, int64_t n) { return E.ensure_bricks(n); },
     [](Engine& E, int64_t n) -> std::vector<Need> {
       return {N(dep_count, 32), N(brick_count, 8 * n), N(brick_cursor, 4 * n), N(brick_off, 8 * (n + 1))};
     }},
    {"brick_lists", [](Engine& E, int64_t n) { return E.ensure_brick_lists(n, n / 2 + 1); },
     [](Engine& E, int64_t n) -> std::vector<Need> {
       return {N(brick_pairs, 4 * n), N(brick_tasks, 8 * (n / 2 + 1))};
     }},
    {"sort_keys", [](Engine& E, int64_t n) { return E.ensure_sort_keys(n); },
     [](Engine& E, int64_t n) -> std::vector<Need> {
       return {N(sort_keys, 8 * n), N(cub_tmp, cub_bytes_needed(0, n))};
     }},
    {"workspace", [](Engine& E, int64_t n) { return E.ws.ensure(E, n); },
     [](Engine& E, int64_t n) -> std::vector<Need> {
       return {N(ws.d_a, 8 * n), N(ws.d_uh, 8 * n), N(ws.v_flow, 24 * n), N(ws.v_tmp, 24 * n), N(ws.pk0, 32 * n),
               N(ws.pk3, 32 * n), N(ws.pk32, 32 * n), N(ws.pf1, 32 * n), N(ws.pf2, 16 * n), N(ws.pf3, 16 * n),
               N(ws.rows, 8 * n), N(ws.i_tmp2, 8 * n), N(ws.m_rows, n), N(ws.m_smark, n), N(ws.i32a, 4 * n),
               N(ws.i32b, 4 * n), N(ws.dk_b, 8 * n), N(ws.tk_key0, 8), N(ws.tk_idx1, 4), N(ws.d_int, 64),
               N(ws.d_i64, 128), N(ws.h_int, 64), N(ws.h_i64, 128), N(ws.h_dbl, 640), N(ws.d_scal_i, 128),
               N(ws.h_scal, 128), N(ws.cache.x_ref, 24 * n), N(ws.cache.hs, 8 * n),
               N(cub_tmp, workspace_cub_bytes(n))};
     }},
    {"grad", [](Engine& E, int64_t n) { return E.ws.ensure_grad(E, n); },
     [](Engine& E, int64_t n) -> std::vector<Need> {
       return {N(ws.pk4, 32 * n), N(ws.gvel, 72 * n), N(ws.gvel32, 36 * n)};
     }},
    {"prof", [](Engine& E, int64_t) { return E.prof.ensure(); },
     [](Engine& E, int64_t) -> std::vector<Need> {
       return {N(prof.ev[0], 1), N(prof.ev[2 * Prof::POOL - 1], 1), N(prof.d_pairs, 8 * PROF_NCAT)};
     }},
};

static int wrong = 0;
static void holds(const Group& g, Engine& E, int64_t n, long k, const char* when) {
  for (const Need& w : g.needs(E, n)) {
    auto it = live.find(w.p);
    if (it != live.end() && it->second >= w.bytes) continue;
    std::printf("%s, allocation %ld failed, %s: %s %s\n", g.name, k, when, w.name,
                !w.p ? "missing" : it == live.end() ? "freed" : "too small");
    wrong += 1;
  }
}

int main() {
  for (const Group& g : groups)
    for (int64_t after : {900, 5000, 70000})  // less than before, between, more than asked for
      for (int first = 0; first < 2; ++first)
        for (long k = 0;; ++k) {
          live.clear();
          Engine E;
          fail_at = -1;
          const int64_t old = 2000, want = 60000;
          if (first && (E.ensure_n(old) || E.ws.ensure(E, old) || g.ensure(E, old))) return 2;
          E.lists.n = old;
          E.ws.cache.valid = first;
          made = 0;
          fail_at = k;
          const int r = g.ensure(E, want);
          const bool failed = made > k;
          fail_at = -1;
          if (failed != (r != 0)) {
            std::printf("%s, allocation %ld: returned %d\n", g.name, k, r);
            wrong += 1;
          }
          if (failed) {
            // the cached lists of a run count as lost, or their buffers are all there
            if (first && E.ws.cache.valid && E.lists.n == old) {
              holds(groups[0], E, old, k, "cached lists");
              if (!std::strcmp(g.name, "list")) holds(g, E, old, k, "cached lists");
              if (!E.ws.cache.x_ref || !live.count(E.ws.cache.x_ref) || !live.count(E.ws.cache.hs)) {
                std::printf("%s, allocation %ld failed: cache without its buffers\n", g.name, k);
                wrong += 1;
              }
            }
            if (g.ensure(E, after) != 0) return 3;
            holds(g, E, after, k, "next call");
            // the groups that every other call starts with
            if (E.ensure_n(old) || E.ws.ensure(E, old)) return 4;
            holds(groups[0], E, old, k, "then lists");
            for (const Group& w : groups)
              if (!std::strcmp(w.name, "workspace")) holds(w, E, old, k, "then workspace");
          }
          E.release();
          if (bad_frees || !live.empty()) {
            std::printf("%s, allocation %ld: %ld frees of nothing, %zu left\n", g.name, k, bad_frees, live.size());
            wrong += 1;
            bad_frees = 0;
          }
          if (!failed) break;
        }
  std::printf("%d wrong\n", wrong);
  return wrong ? 1 : 0;
}
"""


def test_failed_allocations_leave_nothing_that_looks_valid(tmp_path):
    from blackhole_nebula_simulator_b200 import build

    try:
        nvcc = build.nvcc()
    except RuntimeError:
        pytest.skip("needs nvcc")
    assert shutil.which("g++")
    src, alloc, exe = tmp_path / "harness.cu", tmp_path / "allocator.cpp", tmp_path / "harness"
    src.write_text(HARNESS)
    alloc.write_text(ALLOCATOR)
    subprocess.run([nvcc, "-std=c++17", "-O1", *build.ARCH, "--expt-relaxed-constexpr", "-cudart", "none",
                    "-I", CSRC, str(src), str(alloc), os.path.join(CSRC, "scratch.cu"), "-o", str(exe)],
                   check=True)  # fmt: skip
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout[-4000:]
