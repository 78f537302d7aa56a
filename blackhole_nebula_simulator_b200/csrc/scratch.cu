// Device and pinned host buffers of the engine and of its step runtime, grown on demand.
//
// Buffers that grow together are one group with one capacity.  A group that grows counts as having no
// room until its last buffer is there, and a freed pointer is null, so after an allocation that fails
// the next call allocates the whole group again instead of using what is missing or gone.
#include <initializer_list>

#include "engine.cuh"

namespace nbk {

struct Buffer {
  void** p;
  size_t element;  // bytes per element
};

template <typename T>
static Buffer buf(T*& p, size_t elements = 1) {
  return Buffer{(void**)&p, sizeof(T) * elements};
}

// *p stays null if the allocation fails; the failure is this call's, not a later check's
static int give(Engine& E, void** p, size_t bytes, bool pinned = false) {
  void* got = nullptr;
  const cudaError_t e = pinned ? cudaMallocHost(&got, bytes) : cudaMalloc(&got, bytes);
  if (e != cudaSuccess) cudaGetLastError();
  NB_CUDA(e);
  *p = got;
  return 0;
}

static void take(void** p) {
  if (*p) cudaFree(*p);
  *p = nullptr;
}

static bool all_there(std::initializer_list<Buffer> group) {
  for (const Buffer& b : group)
    if (!*b.p) return false;
  return true;
}

// Every buffer of the group with room for c elements (and one more: offset arrays have n + 1).
static int allocate(Engine& E, int64_t& cap, int64_t c, std::initializer_list<Buffer> group) {
  cap = 0;
  for (const Buffer& b : group) take(b.p);
  for (const Buffer& b : group) NB_TRY(give(E, b.p, b.element * (size_t)(c + 1)));
  cap = c;
  return 0;
}

// Room for `want` elements in every buffer of the group; what grows gets a quarter more, `least` at
// least.
static int grow(Engine& E, int64_t& cap, int64_t want, int64_t least,
                std::initializer_list<Buffer> group) {
  if (want <= cap && all_there(group)) return 0;
  return allocate(E, cap, std::max<int64_t>(want + want / 4, least), group);
}

// Temporary storage of the library's sorts and scans.  Every call takes it for large enough after its
// own group is, so without it those groups count as having no room, and a run's lists as lost.
int Engine::ensure_cub(size_t bytes) {
  Engine& E = *this;
  if (bytes <= cub_bytes && cub_tmp) return 0;
  const size_t b = bytes + bytes / 4 + 4096;
  cub_bytes = 0;
  take(&cub_tmp);
  const int r = give(E, &cub_tmp, b);
  if (r != 0) {
    cap_n = ws.cap = 0;
    lists.n = 0;
    return r;
  }
  cub_bytes = b;
  return 0;
}

int Engine::ensure_n(int64_t n) {
  Engine& E = *this;
  if (!d_err) {
    int* word = nullptr;
    NB_TRY(give(E, (void**)&word, sizeof(int) * 4));
    d_err = word;
    NB_CUDA(cudaMemset(d_err, 0, sizeof(int) * 4));
  }
  if (!h_err) NB_TRY(give(E, (void**)&h_err, sizeof(int) * 4, true));
  if (!bbox) NB_TRY(give(E, (void**)&bbox, sizeof(double) * 8));
  if (!h_red) NB_TRY(give(E, (void**)&h_red, sizeof(double) * 64, true));
  if (!d_rowmax) NB_TRY(give(E, (void**)&d_rowmax, 16 * sizeof(unsigned long long)));
  if (!h_build) NB_TRY(give(E, (void**)&h_build, sizeof(int64_t) * 4, true));
  if (!bbox_part) NB_TRY(give(E, (void**)&bbox_part, sizeof(double) * 6 * 1184));
  if (!red) NB_TRY(give(E, (void**)&red, sizeof(double) * 16 * 1184));
  if (n <= cap_n && cap_n > 0) return 0;
  lists.n = 0;
  NB_TRY(grow(E, cap_n, n, 1024, {buf(keys_a), buf(keys_b), buf(vals_a), buf(counts), buf(lists.perm),
                                  buf(lists.inv_perm), buf(lists.spos), buf(lists.off)}));
  return ensure_cub(cub_bytes_needed(cap_n, 0));
}

int Prof::ensure() {
  if (d_pairs) return 0;  // the last of them
  for (int k = 0; k < 2 * POOL; ++k)
    if (!ev[k] && cudaEventCreate(&ev[k]) != cudaSuccess) return ev[k] = nullptr, -2;
  unsigned long long* counts = nullptr;
  if (cudaMalloc((void**)&counts, sizeof(unsigned long long) * PROF_NCAT) != cudaSuccess) return -2;
  if (cudaMemset(counts, 0, sizeof(unsigned long long) * PROF_NCAT) != cudaSuccess) {
    cudaFree(counts);
    return -2;
  }
  d_pairs = counts;
  return 0;
}

// boxes of the tree's nodes and of the sub-leaves: two double4 and a 32-byte record each
int Engine::ensure_nodes(int64_t m) {
  return grow(*this, cap_nodes, m, 256, {buf(node_lo), buf(node_hi), Buffer{&node_q, 32}});
}

int Engine::ensure_sub(int64_t m) {
  return grow(*this, cap_sub, m, 256, {buf(sub_lo), buf(sub_hi), Buffer{&sub_q, 32}});
}

int Engine::ensure_list_capacity(int64_t m) {
  if (m > cap_list || !lists.idx) lists.n = 0;
  return grow(*this, cap_list, std::max<int64_t>(m, 1), 1024, {buf(lists.idx)});
}

int Engine::ensure_tight(int64_t m) {
  return grow(*this, cap_tidx, std::max<int64_t>(m, 1), 1024, {buf(tidx)});
}

int Engine::ensure_leaves(int64_t m) {
  return grow(*this, cap_leaf, m, 1024,
              {buf(leaf_cbase), buf(leaf_bbase), buf(leaf_ibase), buf(leaf_ncand)});
}

int Engine::ensure_tiles(int64_t ncand, int64_t nbatch, int64_t nitem) {
  Engine& E = *this;
  NB_TRY(grow(E, cap_cands, std::max<int64_t>(ncand, 1), 1024, {buf(cands)}));
  NB_TRY(grow(E, cap_masks, std::max<int64_t>(nbatch * 32, 32), 1024, {buf(masks)}));
  return grow(E, cap_items, nitem, 1024, {buf(items), buf(part_count, 32)});
}

int Engine::ensure_deposit(int64_t n) {
  NB_TRY(grow(*this, dep_cap, n, 1024,
              {buf(dep_k0), buf(dep_k1), buf(dep_i0), buf(dep_i1), buf(dep_buf, 12)}));
  return ensure_cub(deposit_cub_bytes(dep_cap));
}

int Engine::ensure_shells(int64_t m) {
  if (m <= cap_shells && dep_shells) return 0;
  return allocate(*this, cap_shells, m, {Buffer{&dep_shells, 2 * sizeof(double)}});
}

int Engine::ensure_bricks(int64_t nbricks) {
  Engine& E = *this;
  if (!dep_count) NB_TRY(give(E, (void**)&dep_count, 4 * sizeof(int64_t)));
  if (nbricks <= cap_bricks && cap_bricks > 0) return 0;
  return allocate(E, cap_bricks, nbricks, {buf(brick_count), buf(brick_cursor), buf(brick_off)});
}

int Engine::ensure_brick_lists(int64_t pairs, int64_t tasks) {
  Engine& E = *this;
  NB_TRY(grow(E, cap_brick_pairs, pairs, 1024, {buf(brick_pairs)}));
  return grow(E, cap_brick_tasks, tasks, 1024, {buf(brick_tasks)});
}

int Engine::ensure_sort_keys(int64_t m) {
  NB_TRY(grow(*this, cap_sort, m, 1024, {buf(sort_keys)}));
  return ensure_cub(cub_bytes_needed(cap_n, m));
}

void Engine::release() {
  void* ps[] = {dep_k0, dep_k1, dep_i0, dep_i1, dep_buf, d_err, bbox, bbox_part, keys_a, keys_b, vals_a, counts, node_lo, node_hi, sub_lo, sub_hi, node_q, sub_q,
                cub_tmp, sort_keys, red, lists.perm, lists.inv_perm, lists.spos, lists.off,
                lists.idx, d_rowmax, tidx, leaf_cbase, leaf_bbase, leaf_ibase, leaf_ncand, cands, masks, items, part_count,
                dep_shells, dep_count, brick_count, brick_cursor, brick_off, brick_pairs, brick_tasks,
                ws.cache.x_ref, ws.cache.hs};
  for (void* p : ps)
    if (p) cudaFree(p);
  if (h_err) cudaFreeHost(h_err);
  if (h_build) cudaFreeHost(h_build);
  prof.release();
  if (h_red) cudaFreeHost(h_red);
  ws.release();
}

// Room for n particles.  The capacity is set last: until then the next call starts again.
int Workspace::ensure(Engine& E, int64_t n) {
  if (n <= cap && cap > 0) return 0;
  release();
  const int64_t c = std::max<int64_t>(n + n / 4, 1024);
  const int64_t tk = (c / TOPK_CHUNK + 2) * TOPK;
  for (const Buffer& b :
       {buf(d_a), buf(d_b), buf(d_c), buf(d_hg), buf(d_hs), buf(d_heff), buf(d_hlim), buf(d_disp),
        buf(d_P), buf(d_cs), buf(d_vsig), buf(d_ddudt), buf(d_dm), buf(d_tmp), buf(d_uh),
        buf(v_flow, 3), buf(v_pred, 3), buf(v_eval, 3), buf(v_dacc, 3), buf(v_tmp, 3), buf(pk0),
        buf(pk1), buf(pk2), buf(pk3), buf(pk32, 2), buf(pf1, 2), buf(pf2), buf(pf3), buf(rows),
        buf(rows_s), buf(rows2), buf(iters), buf(flags), buf(need), buf(i_tmp), buf(pairs),
        buf(i_lvl), buf(i_tmp2), buf(m_rows), buf(m_done), buf(m_need), buf(m_tmp), buf(m_x),
        buf(m_sorted), buf(m_smark), buf(i32a), buf(i32b), buf(dk_b)})
    NB_TRY(give(E, b.p, b.element * (size_t)(c + 1)));
  for (const Buffer& b : {buf(tk_key0, tk), buf(tk_key1, tk), buf(tk_idx0, tk), buf(tk_idx1, tk),
                          buf(d_int, 16), buf(d_i64, 16), buf(d_scal_i, 16)})
    NB_TRY(give(E, b.p, b.element));
  for (const Buffer& b : {buf(h_int, 16), buf(h_i64, 16), buf(h_dbl, 80), buf(h_scal, 16)})
    NB_TRY(give(E, b.p, b.element, true));
  d_scal = reinterpret_cast<double*>(d_scal_i + 8);
  if (cache.cap < c) {
    cache.valid = false;
    NB_TRY(allocate(E, cache.cap, c, {buf(cache.x_ref, 3), buf(cache.hs)}));
  }
  NB_TRY(E.ensure_cub(workspace_cub_bytes(c)));
  cap = c;
  return 0;
}

int Workspace::ensure_grad(Engine& E, int64_t n) {
  if (n <= gcap && gcap > 0) return 0;
  return allocate(E, gcap, std::max<int64_t>(cap, n), {buf(pk4), buf(gvel, 9), buf(gvel32, 9)});
}

void Workspace::release() {
  void* ps[] = {pk4, gvel, gvel32, d_a, d_b, d_c, d_hg, d_hs, d_heff, d_hlim, d_disp, d_P, d_cs, d_vsig, d_ddudt,
                d_dm, d_tmp, d_uh, v_flow, v_pred, v_eval, v_dacc, v_tmp, pk0, pk1, pk2, pk3, pk32,
                pf1, pf2, pf3, m_x, m_sorted, m_smark,
                rows, rows_s, rows2, iters, flags, need, i_tmp, pairs, i_lvl, i_tmp2, m_rows, m_done, m_need,
                m_tmp, i32a, i32b, dk_b, d_int, d_i64, tk_key0, tk_key1, tk_idx0, tk_idx1, d_scal_i};
  for (void* p : ps)
    if (p) cudaFree(p);
  if (h_int) cudaFreeHost(h_int);
  if (h_i64) cudaFreeHost(h_i64);
  if (h_dbl) cudaFreeHost(h_dbl);
  if (h_scal) cudaFreeHost(h_scal);
  *this = Workspace{cache};
}

}  // namespace nbk
