// Neighbour lists on the GPU: particles sorted along a Hilbert curve, an implicit 8-ary tree of boxes over
// leaves of 32 consecutive sorted particles, and a warp-per-leaf traversal that writes exact
// symmetric lists.
//
// The set is the reference's (sim/neighbours.py:240-281, find_neighbours_numba):
//     N(i) = { j : r_ij^2 < (2 h_i)^2  or  r_ij^2 < (2 h_j)^2 },  i itself included,
// with r_ij^2 = dx*dx + dy*dy + dz*dz, dx = x_j - x_i, evaluated in double with the reference's
// rounding (no fused multiply-add), so the lists are identical bit for bit.  The tree only
// prunes: a node is skipped when the distance between its box and the query leaf's box is at
// least 2 max(h_query_max, h_node_max) (with a 1e-12 relative margin on the safe side), which
// can never drop a pair the test above accepts.
//
// Rows come out in sorted (curve) order with each row's entries in ascending sorted index.
#include <cub/cub.cuh>
#include <thrust/iterator/counting_iterator.h>

#include "common.cuh"
#include "engine.cuh"

namespace nbk {

static constexpr int LEAF = 32;
static constexpr int SUB = 8;  // sub-leaf: the unit of the candidate queue (4 per staged batch)
static constexpr int FAN = 8;
static constexpr int STACK = 96;

// ---------------------------------------------------------------- bounding box
__global__ void k_bbox_partial(int64_t n, const double* __restrict__ pos, double* __restrict__ part) {
  __shared__ double s[6][NB_THREADS];
  double mn[3] = {1e308, 1e308, 1e308}, mx[3] = {-1e308, -1e308, -1e308};
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    for (int c = 0; c < 3; ++c) {
      double v = pos[3 * i + c];
      mn[c] = fmin(mn[c], v);
      mx[c] = fmax(mx[c], v);
    }
  }
  for (int c = 0; c < 3; ++c) {
    s[c][threadIdx.x] = mn[c];
    s[3 + c][threadIdx.x] = mx[c];
  }
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w)
      for (int c = 0; c < 3; ++c) {
        s[c][threadIdx.x] = fmin(s[c][threadIdx.x], s[c][threadIdx.x + w]);
        s[3 + c][threadIdx.x] = fmax(s[3 + c][threadIdx.x], s[3 + c][threadIdx.x + w]);
      }
    __syncthreads();
  }
  if (threadIdx.x == 0)
    for (int c = 0; c < 6; ++c) part[6 * blockIdx.x + c] = s[c][0];
}

__global__ void k_bbox_final(int nb, const double* __restrict__ part, double* __restrict__ box6) {
  __shared__ double s[6][NB_THREADS];
  double r[6] = {1e308, 1e308, 1e308, -1e308, -1e308, -1e308};
  for (int b = threadIdx.x; b < nb; b += blockDim.x)
    for (int c = 0; c < 3; ++c) {
      r[c] = fmin(r[c], part[6 * b + c]);
      r[3 + c] = fmax(r[3 + c], part[6 * b + 3 + c]);
    }
  for (int c = 0; c < 6; ++c) s[c][threadIdx.x] = r[c];
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w)
      for (int c = 0; c < 3; ++c) {
        s[c][threadIdx.x] = fmin(s[c][threadIdx.x], s[c][threadIdx.x + w]);
        s[3 + c][threadIdx.x] = fmax(s[3 + c][threadIdx.x], s[3 + c][threadIdx.x + w]);
      }
    __syncthreads();
  }
  if (threadIdx.x == 0)
    for (int c = 0; c < 6; ++c) box6[c] = s[c][0];
}

// ---------------------------------------------------------------- curve keys
__device__ __forceinline__ uint64_t spread21(uint64_t v) {
  v &= 0x1fffffull;
  v = (v | (v << 32)) & 0x1f00000000ffffull;
  v = (v | (v << 16)) & 0x1f0000ff0000ffull;
  v = (v | (v << 8)) & 0x100f00f00f00f00full;
  v = (v | (v << 4)) & 0x10c30c30c30c30c3ull;
  v = (v | (v << 2)) & 0x1249249249249249ull;
  return v;
}

// Hilbert index of a point on the 2^21 grid over the bounding box: J. Skilling's transform
// ("Programming the Hilbert curve", AIP Conf. Proc. 707, 2004) from axes to the transposed
// index, then the three coordinates' bits interleaved (first axis most significant).  Runs of
// consecutive particles along the Hilbert curve have tighter boxes than Morton runs (fewer jumps
// between distant octants), so leaves and sub-leaves prune better.
__device__ __forceinline__ uint64_t hilbert_key(uint32_t x0, uint32_t x1, uint32_t x2) {
  uint32_t X[3] = {x0, x1, x2};
  const uint32_t M = 1u << 20;
  for (uint32_t Q = M; Q > 1; Q >>= 1) {
    const uint32_t P = Q - 1;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      if (X[i] & Q) {
        X[0] ^= P;  // invert the low bits of the first axis
      } else {
        uint32_t t = (X[0] ^ X[i]) & P;  // exchange the low bits of axes 0 and i
        X[0] ^= t;
        X[i] ^= t;
      }
    }
  }
  X[1] ^= X[0];  // Gray encode
  X[2] ^= X[1];
  uint32_t t = 0;
  for (uint32_t Q = M; Q > 1; Q >>= 1)
    if (X[2] & Q) t ^= Q - 1;
  X[0] ^= t;
  X[1] ^= t;
  X[2] ^= t;
  return (spread21(X[0]) << 2) | (spread21(X[1]) << 1) | spread21(X[2]);
}

__global__ void k_curve_keys(int64_t n, const double* __restrict__ pos,
                             const double* __restrict__ box6, uint64_t* __restrict__ keys,
                             int32_t* __restrict__ vals) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  double span = fmax(fmax(box6[3] - box6[0], box6[4] - box6[1]), box6[5] - box6[2]);
  double scale = span > 0 ? 2097151.0 / span : 0.0;
  uint32_t q[3];
  for (int c = 0; c < 3; ++c) {
    double t = (pos[3 * i + c] - box6[c]) * scale;
    t = fmin(fmax(t, 0.0), 2097151.0);
    q[c] = (uint32_t)t;
  }
  keys[i] = hilbert_key(q[0], q[1], q[2]);
  vals[i] = (int32_t)i;
}

__global__ void k_gather_sorted(int64_t n, const int32_t* __restrict__ perm,
                                const double* __restrict__ pos, const double* __restrict__ hs,
                                double4* __restrict__ spos, int32_t* __restrict__ inv_perm) {
  int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k >= n) return;
  int32_t i = perm[k];
  spos[k] = make_double4(pos[3 * (int64_t)i], pos[3 * (int64_t)i + 1], pos[3 * (int64_t)i + 2], hs[i]);
  inv_perm[i] = (int32_t)k;
}

// ---------------------------------------------------------------- tree of boxes
// A box as the candidate walk reads it, one 32-byte record: its corners on a 2^32 grid over the
// particles' bounding box, rounded outward, and twice its largest h in units of that grid, rounded
// up with 1e-6 to spare, so that a test on the records can only keep more than the exact one.
struct Box32 {
  uint32_t lx, ly, lz;
  float reach;
  uint32_t hx, hy, hz, pad;
};

// grid cells per unit length; 0 where the bounding box has no extent or is not finite
__device__ __forceinline__ double box_scale(const double* __restrict__ box6) {
  const double span = fmax(fmax(box6[3] - box6[0], box6[4] - box6[1]), box6[5] - box6[2]);
  return span > 0.0 && isfinite(span) ? 4294967040.0 / span : 0.0;
}

__device__ __forceinline__ Box32 box32(const double4& lo, const double4& hi,
                                       const double* __restrict__ box6) {
  const double s = box_scale(box6);
  Box32 b;
  b.lx = __double2uint_rd(__dmul_rd(__dsub_rd(lo.x, box6[0]), s));
  b.ly = __double2uint_rd(__dmul_rd(__dsub_rd(lo.y, box6[1]), s));
  b.lz = __double2uint_rd(__dmul_rd(__dsub_rd(lo.z, box6[2]), s));
  b.hx = __double2uint_ru(__dmul_ru(__dsub_ru(hi.x, box6[0]), s));
  b.hy = __double2uint_ru(__dmul_ru(__dsub_ru(hi.y, box6[1]), s));
  b.hz = __double2uint_ru(__dmul_ru(__dsub_ru(hi.z, box6[2]), s));
  b.reach = __double2float_ru(2.0 * lo.w * s * (1.0 + 1e-6));
  b.pad = 0;
  return b;
}

__device__ __forceinline__ Box32 ld_box(const Box32* p) {
  Box32 b;
  asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(b.lx), "=r"(b.ly), "=r"(b.lz), "=f"(b.reach), "=r"(b.hx), "=r"(b.hy), "=r"(b.hz),
        "=r"(b.pad)
      : "l"(p));
  return b;
}

// whether two boxes may hold a pair within reach (every rounding on the keeping side)
__device__ __forceinline__ bool box_near(const Box32& a, const Box32& b) {
  const float gx = __uint2float_rd((max(b.lx, a.hx) - a.hx) + (max(a.lx, b.hx) - b.hx));
  const float gy = __uint2float_rd((max(b.ly, a.hy) - a.hy) + (max(a.ly, b.hy) - b.hy));
  const float gz = __uint2float_rd((max(b.lz, a.hz) - a.hz) + (max(a.lz, b.hz) - b.hz));
  const float r = fmaxf(a.reach, b.reach);
  return __fmaf_rd(gz, gz, __fmaf_rd(gy, gy, __fmul_rd(gx, gx))) <= __fmul_ru(r, r);
}

__global__ void k_leaf_boxes(int64_t n, int64_t nleaf, const double4* __restrict__ spos,
                             const double* __restrict__ box6, double4* __restrict__ lo,
                             double4* __restrict__ hi, Box32* __restrict__ q) {
  int64_t l = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (l >= nleaf) return;
  int64_t a = l * LEAF, b = min(a + LEAF, n);
  double4 mn = make_double4(1e308, 1e308, 1e308, 0.0), mx = make_double4(-1e308, -1e308, -1e308, 0.0);
  for (int64_t k = a; k < b; ++k) {
    double4 p = spos[k];
    mn.x = fmin(mn.x, p.x);
    mn.y = fmin(mn.y, p.y);
    mn.z = fmin(mn.z, p.z);
    mx.x = fmax(mx.x, p.x);
    mx.y = fmax(mx.y, p.y);
    mx.z = fmax(mx.z, p.z);
    mn.w = fmax(mn.w, p.w);  // lo.w carries the largest h of the node
  }
  lo[l] = mn;
  hi[l] = mx;
  q[l] = box32(mn, mx, box6);
}

// Boxes (and largest h) of the sub-leaves of SUB consecutive sorted particles.
__global__ void k_sub_boxes(int64_t n, int64_t nsub, const double4* __restrict__ spos,
                            const double* __restrict__ box6, double4* __restrict__ lo,
                            double4* __restrict__ hi, Box32* __restrict__ q) {
  int64_t l = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (l >= nsub) return;
  int64_t a = l * SUB, b = min(a + SUB, n);
  double4 mn = make_double4(1e308, 1e308, 1e308, 0.0), mx = make_double4(-1e308, -1e308, -1e308, 0.0);
  for (int64_t k = a; k < b; ++k) {
    double4 p = spos[k];
    mn.x = fmin(mn.x, p.x);
    mn.y = fmin(mn.y, p.y);
    mn.z = fmin(mn.z, p.z);
    mx.x = fmax(mx.x, p.x);
    mx.y = fmax(mx.y, p.y);
    mx.z = fmax(mx.z, p.z);
    mn.w = fmax(mn.w, p.w);
  }
  lo[l] = mn;
  hi[l] = mx;
  q[l] = box32(mn, mx, box6);
}

__global__ void k_level_up(int64_t nchild, int64_t nparent, const double4* __restrict__ clo,
                           const double4* __restrict__ chi, const double* __restrict__ box6,
                           double4* __restrict__ plo, double4* __restrict__ phi,
                           Box32* __restrict__ q) {
  int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (p >= nparent) return;
  double4 mn = make_double4(1e308, 1e308, 1e308, 0.0), mx = make_double4(-1e308, -1e308, -1e308, 0.0);
  for (int64_t c = p * FAN; c < min((p + 1) * FAN, nchild); ++c) {
    double4 a = clo[c], b = chi[c];
    mn.x = fmin(mn.x, a.x);
    mn.y = fmin(mn.y, a.y);
    mn.z = fmin(mn.z, a.z);
    mn.w = fmax(mn.w, a.w);
    mx.x = fmax(mx.x, b.x);
    mx.y = fmax(mx.y, b.y);
    mx.z = fmax(mx.z, b.z);
  }
  plo[p] = mn;
  phi[p] = mx;
  q[p] = box32(mn, mx, box6);
}

struct TreeView {
  const double4* lo;
  const double4* hi;
  const Box32* q;  // the same boxes as the walk's records
  int64_t level_off[MAX_LEVELS + 1];
  int64_t level_size[MAX_LEVELS];
  int nlevels;
};

__device__ __forceinline__ double box_gap2(double4 alo, double4 ahi, double4 blo, double4 bhi) {
  double gx = fmax(fmax(blo.x - ahi.x, alo.x - bhi.x), 0.0);
  double gy = fmax(fmax(blo.y - ahi.y, alo.y - bhi.y), 0.0);
  double gz = fmax(fmax(blo.z - ahi.z, alo.z - bhi.z), 0.0);
  return gx * gx + gy * gy + gz * gz;
}

// The rows of one query leaf of LEAF consecutive sorted particles, one lane per particle, tested
// tile by tile.  The leaf's candidates are the sub-leaves whose boxes lie within its reach, in
// ascending order.  Every 4 of them (32 candidates) are staged in shared memory, one candidate per
// lane with coalesced loads, as float offsets from the query leaf's centre, and every lane tests its
// own particle against all 32: the whole warp stays busy on the same candidates, with no per-lane
// queues.
//
// The test is the reference's FP64 r^2 < (2 h_i)^2 or r^2 < (2 h_j)^2 decided in FP32 with a
// rigorous band.  With D the largest offset component of the query lanes and the staged batch
// and u = 2^-24, the offsets round with error <= u D, their differences with error <= 4 u D,
// and the float r^2 of a pair (three rounded squares and sums of terms <= 12 D^2) differs from
// the exact one by at most 84 u D^2; the float thresholds and their subtractions add at most
// 36 u D^2 for every threshold that can matter (r^2 <= 12 D^2).  With B = 192 u D^2 and the
// float threshold T lowered by B, q = fl(r^2 - (T - B)) < 0 is a certain hit (the sign of a
// rounded difference is exact, and r^2 + 84 u D^2 < T - B + 36 u D^2 < T) and q >= 2 B a
// certain miss (r^2 >= T - B + 2 B (1 - u) - 120 u D^2 > T); pairs in between are decided by
// the exact FP64 test (no fused multiply-add) from the double positions.  So the lists are the
// reference's bit for bit.
//
// Three passes: k_lists_cand finds the candidates of each query leaf, level by level through the tree
// of boxes (k_lists_wide for the leaves whose frontiers outgrow a warp's buffer, and in it a
// depth-first walk for those that outgrow a block's), each in its own slice of the candidate and mask
// buffers; k_lists_test runs the tests once, storing each lane's 32-bit hit mask per batch and its
// row's entry count; k_lists_expand turns the masks into the CSR entries at the rows' offsets, each
// row ascending (batches come in ascending candidate order, a mask's bits from the lowest slot up).

constexpr float BAND_U = 192.0f / 16777216.0f;  // 192 u, u = 2^-24

// The query leaf's box, centre and largest search radius.
struct QueryLeaf {
  double4 lo, hi;
  double cx, cy, cz;
};

__device__ __forceinline__ QueryLeaf query_leaf(const TreeView& tv, int64_t leaf) {
  QueryLeaf q;
  q.lo = tv.lo[leaf];
  q.hi = tv.hi[leaf];
  q.cx = 0.5 * (q.lo.x + q.hi.x);
  q.cy = 0.5 * (q.lo.y + q.hi.y);
  q.cz = 0.5 * (q.lo.z + q.hi.z);
  return q;
}

// Depth-first walk of the tree for one query leaf by one warp, with a stack in shared memory (entries
// (level << 40) | index, children pushed highest first); on_subs(s0, mask) is called warp-uniformly for every
// candidate leaf with its first sub-leaf s0 and the ballot of its sub-leaves within reach of the
// query leaf's box (bit c: sub-leaf s0 + c), in ascending order.  Returns false if the stack
// overflowed.
template <typename F>
__device__ __forceinline__ bool walk_candidates(int64_t n, const TreeView& tv, const QueryLeaf& q,
                                                const double4* __restrict__ slo,
                                                const double4* __restrict__ shi,
                                                int64_t* stack, int lane, F&& on_subs) {
  const unsigned FULL = 0xffffffffu;
  const int64_t nsub = (n + SUB - 1) / SUB;
  const double qh = q.lo.w;
  int sp = 0;
  __syncwarp();
  if (lane == 0) stack[0] = ((int64_t)(tv.nlevels - 1) << 40);
  sp = 1;
  __syncwarp();
  while (sp > 0) {
    const int64_t e = stack[sp - 1];
    __syncwarp();
    sp -= 1;
    const int lvl = (int)(e >> 40);
    const int64_t node = e & ((1ll << 40) - 1);
    if (lvl == 0) {
      const int64_t s0 = node * (LEAF / SUB);
      const int64_t s1 = min(s0 + LEAF / SUB, nsub);
      bool near = false;
      if (lane < s1 - s0) {
        const double4 blo = slo[s0 + lane], bhi = shi[s0 + lane];
        const double reach = 2.0 * fmax(qh, blo.w);
        near = box_gap2(q.lo, q.hi, blo, bhi) < reach * reach * (1.0 + 1e-12);
      }
      const unsigned mk = __ballot_sync(FULL, near);
      if (mk) on_subs(s0, mk);
      continue;
    }
    const int64_t c0 = node * FAN;
    const int64_t csize = tv.level_size[lvl - 1];
    const int64_t child = c0 + lane;
    bool hit = false;
    if (lane < FAN && child < csize) {
      const int64_t g = tv.level_off[lvl - 1] + child;
      const double4 blo = tv.lo[g], bhi = tv.hi[g];
      const double reach = 2.0 * fmax(qh, blo.w);
      hit = box_gap2(q.lo, q.hi, blo, bhi) < reach * reach * (1.0 + 1e-12);
    }
    const unsigned mask = __ballot_sync(FULL, hit);
    const int nh = __popc(mask);
    if (sp + nh > STACK) return false;
    if (hit) {
      const int above = __popc(mask & ~((2u << lane) - 1u));
      stack[sp + above] = ((int64_t)(lvl - 1) << 40) | child;
    }
    __syncwarp();
    sp += nh;
  }
  return true;
}

// Where each query leaf's candidates, batches and work items lie, and the cursors that place them.
// A work item is a stretch of at most `chunk` batches of one leaf, so that a leaf in reach of much
// more than the others (a large h beside a dense region) is shared by as many warps as it needs.
struct ListSlices {
  int64_t *cbase, *bbase, *ibase;  // per leaf: first candidate, batch and item
  int32_t* ncand;                  // per leaf: candidate sub-leaves
  uint64_t* items;                 // (part << 32) | leaf
  unsigned long long* cursor;      // candidates, batches, items taken so far
  int64_t cap_cands, cap_batches, cap_items;
  int chunk;
};

// One thread takes a leaf's slices with three atomic adds (so slices of different leaves lie in
// any order).  Returns the first candidate, or -1 if a slice would pass its buffer's capacity:
// nothing is written then; the host grows the buffers from the cursors' final values and runs
// the pass again.
__device__ __forceinline__ int64_t take_slices(const ListSlices& ls, int64_t leaf, int64_t count) {
  const int64_t nbat = (count + 3) / 4;
  const int64_t nit = nbat > ls.chunk ? (nbat + ls.chunk - 1) / ls.chunk : 1;
  const int64_t cb = (int64_t)atomicAdd(ls.cursor, (unsigned long long)count);
  const int64_t bb = (int64_t)atomicAdd(ls.cursor + 1, (unsigned long long)nbat);
  const int64_t ib = (int64_t)atomicAdd(ls.cursor + 2, (unsigned long long)nit);
  ls.cbase[leaf] = cb;
  ls.bbase[leaf] = bb;
  ls.ibase[leaf] = ib;
  ls.ncand[leaf] = (int32_t)count;
  if (cb + count > ls.cap_cands || bb + nbat > ls.cap_batches || ib + nit > ls.cap_items) return -1;
  for (int64_t p = 0; p < nit; ++p) ls.items[ib + p] = ((uint64_t)p << 32) | (uint64_t)leaf;
  return cb;
}

// whether child `c` of a level (its boxes at clo, chi, cq) is within reach of the query leaf
__device__ __forceinline__ bool child_near(bool records, const QueryLeaf& q, const Box32& qb,
                                           const double4* clo, const double4* chi,
                                           const Box32* cq, int64_t c) {
  if (records) return box_near(qb, ld_box(cq + c));
  const double4 blo = clo[c], bhi = chi[c];
  const double reach = 2.0 * fmax(q.lo.w, blo.w);
  return box_gap2(q.lo, q.hi, blo, bhi) < reach * reach * (1.0 + 1e-12);
}

// Pass 1: the candidate sub-leaves of each query leaf, in ascending order, into its own slice of
// the candidate buffer.  The walk goes level by level: the nodes within reach of the query box at
// one level (a frontier in shared memory, ascending) give the next level's nodes to test, 32 at
// a time, one per lane; the leaves within reach give the sub-leaves to test the same way, and the
// sub-leaves within reach are the leaf's candidate list (ascending, since every frontier is).  A
// leaf whose frontier outgrows its buffer goes to the list `wide`, for k_lists_wide.  A sub-leaf is
// within reach if one of the leaf's own sub-leaves is: 32 particles along the curve rarely fill
// their box, so this costs 0.04 ms here and saves 0.16 + 0.06 ms of passes 2 and 3 (1M torus).
// Latency bound (a dependent chain of box loads per level): 0.18 ms on the 1M torus,
// 0.04 on the 262,144-particle cloud.  With 64-byte boxes in double, and the few leaves
// with large frontiers walked node by node by their warps, twice, 1.34, 2.3 and 0.04 ms.
constexpr int CAND_WARPS = 4;
#ifndef CAND_SMEM
#define CAND_SMEM 1024  // entries of a frontier buffer
#endif

__global__ void __launch_bounds__(CAND_WARPS * 32) k_lists_cand(
    int64_t n, int64_t nwork, const uint64_t* __restrict__ order,
    unsigned long long* __restrict__ next, TreeView tv, const double4* __restrict__ slo,
    const double4* __restrict__ shi, const Box32* __restrict__ sq, const double* __restrict__ box6,
    ListSlices ls, int32_t* __restrict__ cands, int32_t* __restrict__ wide,
    unsigned long long* __restrict__ nwide) {
  __shared__ int32_t fronts[CAND_WARPS][2][CAND_SMEM];
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  int32_t(*front)[CAND_SMEM] = fronts[threadIdx.x >> 5];
  const int64_t nsub = (n + SUB - 1) / SUB;
  // records where the grid resolves anything, else (a bounding box that is not finite) the doubles
  const bool records = box_scale(box6) > 0.0;
  while (true) {
    unsigned long long t = 0;
    if (lane == 0) t = atomicAdd(next, 1ull);
    t = __shfl_sync(FULL, t, 0);
    if (t >= (unsigned long long)nwork) break;  // warp-uniform
    const int64_t leaf = (int64_t)(order[t] & 0xffffffffull);
    const QueryLeaf q = query_leaf(tv, leaf);
    const Box32 qb = ld_box(tv.q + leaf);
    Box32 own[LEAF / SUB];
#pragma unroll
    for (int i = 0; i < LEAF / SUB; ++i)
      own[i] = ld_box(sq + min(leaf * (LEAF / SUB) + i, nsub - 1));
    // level by level from the root; `cur` holds the frontier (ascending node indices)
    int cur = 0, fn = 1;
    bool over = false;
    __syncwarp();
    if (lane == 0) front[0][0] = 0;
    __syncwarp();
    for (int lvl = tv.nlevels - 1; lvl >= 0 && !over; --lvl) {
      // children of the frontier: nodes of level lvl - 1, or at the leaves their sub-leaves
      const int fan = lvl > 0 ? FAN : LEAF / SUB;
      const int64_t csize = lvl > 0 ? tv.level_size[lvl - 1] : nsub;
      const int64_t coff = lvl > 0 ? tv.level_off[lvl - 1] : 0;
      const double4* clo = lvl > 0 ? tv.lo : slo;
      const double4* chi = lvl > 0 ? tv.hi : shi;
      const Box32* cq = lvl > 0 ? tv.q : sq;
      const int total = fn * fan;
      int nn = 0;
      for (int c0 = 0; c0 < total; c0 += 32) {
        const int c = c0 + lane;
        bool hit = false;
        int32_t child = 0;
        if (c < total) {
          child = front[cur][c / fan] * fan + c % fan;
          if (lvl == 0 && records) {
            // the leaf's box holds more than its own sub-leaves do
            hit = false;
            if (child < csize) {
              const Box32 cb = ld_box(sq + child);
#pragma unroll
              for (int i = 0; i < LEAF / SUB; ++i) hit = hit || box_near(own[i], cb);
            }
          } else {
            hit = child < csize && child_near(records, q, qb, clo, chi, cq, coff + child);
          }
        }
        const unsigned mk = __ballot_sync(FULL, hit);
        if (nn + __popc(mk) > CAND_SMEM) {
          over = true;
          break;
        }
        if (hit) front[cur ^ 1][nn + __popc(mk & below)] = child;
        nn += __popc(mk);
      }
      __syncwarp();
      cur ^= 1;
      fn = nn;
    }
    if (over) {
      if (lane == 0) wide[atomicAdd(nwide, 1ull)] = (int32_t)leaf;
      continue;
    }
    int64_t cb = 0;
    if (lane == 0) cb = take_slices(ls, leaf, fn);
    cb = __shfl_sync(FULL, cb, 0);
    if (cb >= 0)
      for (int c = lane; c < fn; c += 32) cands[cb + c] = front[cur][c];
    __syncwarp();
  }
}

// Pass 1 for the leaves with large frontiers: a block per leaf tests WIDE_THREADS children at a
// time, with the leaf-level frontier (up to WIDE_CAP leaves) in shared memory; its sub-leaves are
// counted and then written in two sweeps over it.  A frontier beyond that is left to a depth-first
// walk by one warp.
constexpr int WIDE_THREADS = 512;
constexpr int WIDE_CAP = 12288;

__global__ void __launch_bounds__(WIDE_THREADS) k_lists_wide(
    int64_t n, const int32_t* __restrict__ wide, const unsigned long long* __restrict__ nwide,
    TreeView tv, const double4* __restrict__ slo, const double4* __restrict__ shi,
    const Box32* __restrict__ sq, const double* __restrict__ box6, ListSlices ls,
    int32_t* __restrict__ cands, int* err) {
  extern __shared__ int32_t wide_front[];  // two frontiers of WIDE_CAP
  __shared__ int64_t stack[STACK];
  __shared__ int hits_s[WIDE_THREADS / 32];
  __shared__ int64_t base_s, count_s;
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned below = (1u << lane) - 1u;
  const int64_t nsub = (n + SUB - 1) / SUB;
  const bool records = box_scale(box6) > 0.0;
  const int64_t all = (int64_t)*nwide;
  for (int64_t w = blockIdx.x; w < all; w += gridDim.x) {
    const int64_t leaf = wide[w];
    const QueryLeaf q = query_leaf(tv, leaf);
    const Box32 qb = ld_box(tv.q + leaf);
    int32_t* cur = wide_front;
    int32_t* nxt = wide_front + WIDE_CAP;
    int fn = 1;
    bool over = false;
    __syncthreads();
    if (threadIdx.x == 0) cur[0] = 0;
    __syncthreads();
    // children of the frontier's nodes, WIDE_THREADS at a time; f(child, its rank) for the near
    // ones, ranks ascending.  Returns their number.
    auto sweep = [&](int lvl, auto&& f) {
      const int fan = lvl > 0 ? FAN : LEAF / SUB;
      const int64_t csize = lvl > 0 ? tv.level_size[lvl - 1] : nsub;
      const int64_t coff = lvl > 0 ? tv.level_off[lvl - 1] : 0;
      const double4* clo = lvl > 0 ? tv.lo : slo;
      const double4* chi = lvl > 0 ? tv.hi : shi;
      const Box32* cq = lvl > 0 ? tv.q : sq;
      const int total = fn * fan;
      int64_t nn = 0;
      for (int c0 = 0; c0 < total; c0 += WIDE_THREADS) {
        const int c = c0 + (int)threadIdx.x;
        bool hit = false;
        int32_t child = 0;
        if (c < total) {
          child = cur[c / fan] * fan + c % fan;
          hit = child < csize && child_near(records, q, qb, clo, chi, cq, coff + child);
        }
        const unsigned mk = __ballot_sync(FULL, hit);
        if (lane == 0) hits_s[warp] = __popc(mk);
        __syncthreads();
        int before = 0, sum = 0;
#pragma unroll
        for (int v = 0; v < WIDE_THREADS / 32; ++v) {
          before += v < warp ? hits_s[v] : 0;
          sum += hits_s[v];
        }
        if (hit) f(child, nn + before + __popc(mk & below));
        nn += sum;
        __syncthreads();
      }
      return nn;
    };
    for (int lvl = tv.nlevels - 1; lvl > 0 && !over; --lvl) {
      const int64_t nn = sweep(lvl, [&](int32_t child, int64_t at) {
        if (at < WIDE_CAP) nxt[at] = child;
      });
      over = nn > WIDE_CAP;  // block-uniform
      fn = (int)min(nn, (int64_t)WIDE_CAP);
      int32_t* swap = cur;
      cur = nxt;
      nxt = swap;
      __syncthreads();
    }
    if (!over) {
      const int64_t count = sweep(0, [](int32_t, int64_t) {});
      if (threadIdx.x == 0) base_s = take_slices(ls, leaf, count);
      __syncthreads();
      const int64_t cb = base_s;
      if (cb >= 0) sweep(0, [&](int32_t child, int64_t at) { cands[cb + at] = child; });
    } else if (warp == 0) {
      int64_t count = 0;
      if (!walk_candidates(n, tv, q, slo, shi, stack, lane,
                           [&](int64_t, unsigned mk) { count += __popc(mk); }))
        set_error(err, ERR_TRAVERSAL_STACK);
      if (lane == 0) {
        base_s = take_slices(ls, leaf, count);
        count_s = count;
      }
      __syncwarp();
      const int64_t cb = base_s;
      if (cb >= 0) {
        int64_t c2 = 0;
        walk_candidates(n, tv, q, slo, shi, stack, lane, [&](int64_t s0, unsigned mk) {
          const int pos = __popc(mk & below);
          if (((mk >> lane) & 1u) && c2 + pos < count_s) cands[cb + c2 + pos] = (int32_t)(s0 + lane);
          c2 += __popc(mk);
        });
      }
    }
  }
}

// Two floats in one register pair: the packed operations of sm_100 (each half rounds to nearest as
// the scalar operation does).
__device__ __forceinline__ uint64_t pack2(float a, float b) {
  return (uint64_t)__float_as_uint(a) | ((uint64_t)__float_as_uint(b) << 32);
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

// Pass 2: the tests, on each work item's batches of candidates.  Each batch's final hit masks go
// to masks[(batch base + b) * 32 + lane], the item's entries per row to part_count and, added up,
// to counts (zeroed before).  Bound by issue (60 % active, cold, at two blocks of 120 registers an SM;
// four rows by eight candidates a lane, with a quarter of the shared loads, gain 1 %): 0.83 ms on the
// 1M torus.  Two candidates per packed instruction, the whole batch unrolled (three blocks spill);
// with scalar tests, a warp alone on its leaf whatever the leaf's number of batches and candidates by
// the leaf's box alone, 1.30 ms.
#ifndef TEST_BLOCKS_PER_SM
#define TEST_BLOCKS_PER_SM 2
#endif
__global__ void __launch_bounds__(NB_THREADS, TEST_BLOCKS_PER_SM) k_lists_test(
    int64_t n, unsigned long long* __restrict__ next, TreeView tv,
    const double4* __restrict__ spos, const int32_t* __restrict__ cands, ListSlices ls,
    uint32_t* __restrict__ masks, uint32_t* __restrict__ part_count,
    int64_t* __restrict__ counts) {
  // the staged candidates' offsets and negated thresholds, four arrays of 32 per warp
  __shared__ __align__(16) float cand_s[NB_THREADS / 32][4][32];
  __shared__ int32_t cidx_s[NB_THREADS / 32][32];
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  float(*cand)[32] = cand_s[threadIdx.x >> 5];
  int32_t* cidx = cidx_s[threadIdx.x >> 5];
  const unsigned long long nitems = ls.cursor[2];
  while (true) {
    unsigned long long t = 0;
    if (lane == 0) t = atomicAdd(next, 1ull);
    t = __shfl_sync(FULL, t, 0);
    if (t >= nitems) break;  // warp-uniform
    const uint64_t item = ls.items[t];
    const int64_t leaf = (int64_t)(item & 0xffffffffull), part = (int64_t)(item >> 32);
    const QueryLeaf q = query_leaf(tv, leaf);
    const int64_t cbase = ls.cbase[leaf], bbase = ls.bbase[leaf];
    const int64_t ncand = ls.ncand[leaf], nbat = (ncand + 3) / 4;
    const int64_t b_end = min(nbat, (part + 1) * ls.chunk);
    const int64_t k = leaf * LEAF + lane;
    const bool valid = k < n;
    const double4 me = valid ? spos[k] : make_double4(0, 0, 0, 0);
    float mx = 1e30f, my = 1e30f, mz = 1e30f, Dl = 0.0f, r2i_f = -1.0f;
    const double ri = 2.0 * me.w;
    const double r2i = __dmul_rn(ri, ri);
    if (valid) {
      mx = (float)(me.x - q.cx);
      my = (float)(me.y - q.cy);
      mz = (float)(me.z - q.cz);
      Dl = fmaxf(fmaxf(fabsf(mx), fabsf(my)), fabsf(mz));
      r2i_f = (float)r2i;
    }
    // non-negative floats order like their bits
    const float Dq = __uint_as_float(__reduce_max_sync(FULL, __float_as_uint(Dl)));
    int64_t m = 0;
    for (int64_t b = part * ls.chunk; b < b_end; ++b) {
      // stage: slot = lane, candidate sub-leaf 4 b + lane / 8, particle lane % 8 of it
      const int64_t c = 4 * b + (lane >> 3);
      const int32_t sb = c < ncand ? cands[cbase + c] : -1;
      const int64_t j = (int64_t)sb * SUB + (lane & 7);
      float4 cc = make_float4(1e30f, 1e30f, 1e30f, 0.0f);
      float Dj = 0.0f;
      int32_t jj = -1;
      if (sb >= 0 && j < n) {
        const double4 p = spos[j];
        cc.x = (float)(p.x - q.cx);
        cc.y = (float)(p.y - q.cy);
        cc.z = (float)(p.z - q.cz);
        const double rj = 2.0 * p.w;
        cc.w = (float)(rj * rj);
        Dj = fmaxf(fmaxf(fabsf(cc.x), fabsf(cc.y)), fabsf(cc.z));
        jj = (int32_t)j;
      }
      const float D = fmaxf(Dq, __uint_as_float(__reduce_max_sync(FULL, __float_as_uint(Dj))));
      // offsets beyond float's comfortable range (never in code units): every pair exactly
      const bool wide = !(D < 1e15f);
      const float B = wide ? 0.0f : BAND_U * D * D;
      cand[0][lane] = cc.x;
      cand[1][lane] = cc.y;
      cand[2][lane] = cc.z;
      cand[3][lane] = -(cc.w - B);
      cidx[lane] = jj;
      __syncwarp();
      const float nri = -(r2i_f - B), twoB = 2.0f * B;
      // q = r^2 - (threshold - B) of each candidate: its sign bit is a certain hit, shifted into
      // the mask (candidate 31 first, so bit tt is candidate tt); the smallest non-negative q
      // (signed floats' bits sort above every non-negative float's) tells whether any lies in
      // the band 0 <= q < 2B.  Two candidates per packed instruction, each lane of which rounds
      // as the scalar one.
      const uint64_t nmx = pack2(-mx, -mx), nmy = pack2(-my, -my), nmz = pack2(-mz, -mz);
      unsigned hit = 0u, closest = 0xffffffffu;
#pragma unroll
      for (int t4 = 7; t4 >= 0; --t4) {
        const ulonglong2 X = reinterpret_cast<const ulonglong2*>(cand[0])[t4];
        const ulonglong2 Y = reinterpret_cast<const ulonglong2*>(cand[1])[t4];
        const ulonglong2 Z = reinterpret_cast<const ulonglong2*>(cand[2])[t4];
        const float4 W = reinterpret_cast<const float4*>(cand[3])[t4];
        uint64_t q2[2];
#pragma unroll
        for (int p = 0; p < 2; ++p) {
          const uint64_t dx = add2(p ? X.y : X.x, nmx), dy = add2(p ? Y.y : Y.x, nmy),
                         dz = add2(p ? Z.y : Z.x, nmz);
          const uint64_t r2 = fma2(dz, dz, fma2(dy, dy, mul2(dx, dx)));
          q2[p] = add2(r2, pack2(fminf(p ? W.z : W.x, nri), fminf(p ? W.w : W.y, nri)));
        }
        const unsigned a = (unsigned)q2[0], b = (unsigned)(q2[0] >> 32), c = (unsigned)q2[1],
                       d = (unsigned)(q2[1] >> 32);
        hit = __funnelshift_l(d, hit, 1);
        hit = __funnelshift_l(c, hit, 1);
        hit = __funnelshift_l(b, hit, 1);
        hit = __funnelshift_l(a, hit, 1);
        closest = __vimin3_u32(closest, a, b);
        closest = __vimin3_u32(closest, c, d);
      }
      unsigned amb = 0u;
      if (wide) {
        hit = 0u;
        amb = __ballot_sync(FULL, jj >= 0);
      } else if (__any_sync(FULL, valid && closest < __float_as_uint(twoB))) {
        for (int tt = 0; tt < 32; ++tt) {
          const float dx = cand[0][tt] - mx, dy = cand[1][tt] - my, dz = cand[2][tt] - mz;
          const float q = fmaf(dz, dz, fmaf(dy, dy, dx * dx)) + fminf(cand[3][tt], nri);
          amb |= q >= 0.0f && q < twoB ? 1u << tt : 0u;
        }
      }
      if (!valid) hit = amb = 0u;
      if (__any_sync(FULL, amb != 0u)) {
        // the band: the reference's exact FP64 test from the double positions
        while (amb) {
          const int tt = __ffs(amb) - 1;
          amb &= amb - 1u;
          const double4 pj = spos[cidx[tt]];
          const double d2 = d2_exact(pj.x - me.x, pj.y - me.y, pj.z - me.z);
          const double rj = 2.0 * pj.w;
          if (d2 < r2i || d2 < __dmul_rn(rj, rj)) hit |= 1u << tt;
        }
      }
      masks[(bbase + b) * 32 + lane] = hit;
      m += __popc(hit);
      __syncwarp();  // the next batch overwrites the staged candidates
    }
    part_count[t * 32 + lane] = (uint32_t)m;
    if (valid) {
      if (nbat <= ls.chunk)
        counts[k] = m;
      else
        atomicAdd(reinterpret_cast<unsigned long long*>(counts + k), (unsigned long long)m);
    }
  }
}

// Pass 3: masks -> CSR entries.  One warp per work item, EXPAND_BATCHES batches at a time, in order:
// lane c holds candidate c of each batch, and for every row with a hit in them the lanes whose bit
// is set in the row's mask store their candidates at the row's next positions (a bit's rank in
// the mask), so a row's entries come ascending.
// Bound by issue (73 % active, about ten instructions per row and batch): 0.59 ms on the 1M torus
// (160M entries), 0.51 on a 400,000-particle Wendland torus, 12 us on a 4,096-particle cloud.  Rings in
// shared memory that the warp empties in aligned stretches of 32 (fewer stores, but a loop over the
// longest of 32 masks) took 0.78, 0.75 ms and 22 us; batches at a time 2 / 4 / 8: 0.65 / 0.65 / 0.68 ms,
// before the candidates were culled by sub-leaf.
constexpr int EXPAND_WARPS = 4;
constexpr int EXPAND_BATCHES = 4;

__global__ void __launch_bounds__(EXPAND_WARPS * 32) k_lists_expand(
    int64_t n, int64_t nitems, const int32_t* __restrict__ cands, ListSlices ls,
    const uint32_t* __restrict__ masks, const uint32_t* __restrict__ part_count,
    const int64_t* __restrict__ off, int32_t* __restrict__ idx, int* err) {
  __shared__ __align__(16) uint32_t mask_s[EXPAND_WARPS][EXPAND_BATCHES * 32];
  const unsigned FULL = 0xffffffffu;
  const int64_t t = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (t >= nitems) return;  // warp-uniform
  const int64_t leaf = (int64_t)(ls.items[t] & 0xffffffffull), part = (int64_t)(ls.items[t] >> 32);
  uint32_t* ms = mask_s[threadIdx.x >> 5];
  const int32_t* cand = cands + ls.cbase[leaf];
  const uint32_t* mask = masks + ls.bbase[leaf] * 32 + lane;
  const int64_t ncand = ls.ncand[leaf], nbat = (ncand + 3) / 4;
  const int64_t b_beg = part * ls.chunk, b_end = min(nbat, b_beg + ls.chunk);
  const int64_t k0 = leaf * LEAF;
  const int rows = (int)(n - k0 < LEAF ? n - k0 : LEAF);
  const int64_t base = off[k0];  // positions are relative to the leaf's first one
  if (off[k0 + rows] - base > 0x7fffffc0ll) {  // beyond 32-bit positions within one leaf
    if (lane == 0) set_error(err, ERR_LIST_OVERFLOW);
    return;
  }
  int32_t* out = idx + base;
  int w = lane < rows ? (int)(off[k0 + lane] - base) : 0;  // next position of the row
  for (int64_t p = part; p > 0; --p) w += (int)part_count[(t - p) * 32 + lane];  // earlier items
  const unsigned below = (1u << lane) - 1u;
  for (int64_t b0 = b_beg; b0 < b_end; b0 += EXPAND_BATCHES) {
    uint32_t some = 0u;
    int32_t id[EXPAND_BATCHES];
#pragma unroll
    for (int u = 0; u < EXPAND_BATCHES; ++u) {
      const bool in = b0 + u < b_end;
      const int64_t c = 4 * (b0 + u) + (lane >> 3);
      const uint32_t m = in ? __ldcs(mask + (b0 + u) * 32) : 0u;
      id[u] = in && c < ncand ? cand[c] * SUB + (lane & 7) : 0;
      ms[lane * EXPAND_BATCHES + u] = m;
      some |= m;
    }
    __syncwarp();
    for (unsigned left = __ballot_sync(FULL, some != 0u); left; left &= left - 1) {
      const int r = __ffs(left) - 1;
      int at = __shfl_sync(FULL, w, r);
#pragma unroll
      for (int u = 0; u < EXPAND_BATCHES; ++u) {
        const uint32_t m = ms[r * EXPAND_BATCHES + u];
        if (m >> lane & 1u) out[at + __popc(m & below)] = id[u];
        at += __popc(m);
      }
      if (lane == r) w = at;
    }
    __syncwarp();
  }
  if (b_end == nbat && lane < rows && w != (int)(off[k0 + lane + 1] - base))
    set_error(err, ERR_LIST_OVERFLOW);
}

// The longest row.
__global__ void __launch_bounds__(NB_THREADS) k_row_max(int64_t n, const int64_t* __restrict__ counts,
                                                        unsigned long long* __restrict__ rowmax) {
  unsigned m = 0;
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n;
       k += (int64_t)gridDim.x * blockDim.x)
    m = max(m, (unsigned)counts[k]);
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0) atomicMax(rowmax, (unsigned long long)m);
}

// Order key of each query leaf: its cost class (the binary exponent of the linear size of the
// region its traversal covers, box extent plus twice the largest search diameter), heaviest
// first, then the leaf's curve position.
__global__ void k_leaf_cost(int64_t nleaf, const double4* __restrict__ lo,
                            const double4* __restrict__ hi, uint64_t* __restrict__ key) {
  int64_t l = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (l >= nleaf) return;
  double4 a = lo[l], b = hi[l];
  double ext = fmax(fmax(b.x - a.x, b.y - a.y), b.z - a.z);
  float c = (float)(ext + 4.0 * a.w);
  const uint64_t cls = 255u - ((__float_as_uint(c) >> 23) & 255u);
  key[l] = (cls << 32) | (uint64_t)l;
}

// ---------------------------------------------------------------- export to original order
__global__ void k_export_counts(int64_t n, const int32_t* __restrict__ inv_perm,
                                const int64_t* __restrict__ off_s, int64_t* __restrict__ cnt_o) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  int32_t k = inv_perm[i];
  cnt_o[i] = off_s[k + 1] - off_s[k];
}

// Ascending sort of 32 K keys held by one warp, K per lane (element lane K + r in v[r]): a bitonic
// network whose merges start with the mirrored comparison (element e against e ^ (size - 1)), so
// that every comparison is ascending.  Strides below K stay within a lane, the others are
// shuffles.
template <int K>
__device__ __forceinline__ void warp_sort(int32_t (&v)[K], int lane) {
  const unsigned FULL = 0xffffffffu;
#pragma unroll
  for (int size = 2; size <= 32 * K; size *= 2) {
    if (size <= K) {
#pragma unroll
      for (int r = 0; r < K; ++r) {
        const int o = r ^ (size - 1);
        if (o > r) {
          const int32_t a = v[r], b = v[o];
          v[r] = min(a, b);
          v[o] = max(a, b);
        }
      }
    } else {
      const int m = size / K - 1;
      const bool low = lane < (lane ^ m);
      int32_t w[K];
#pragma unroll
      for (int r = 0; r < K; ++r) w[r] = __shfl_xor_sync(FULL, v[K - 1 - r], m);
#pragma unroll
      for (int r = 0; r < K; ++r) v[r] = low ? min(v[r], w[r]) : max(v[r], w[r]);
    }
#pragma unroll
    for (int stride = size / 4; stride > 0; stride /= 2) {
      if (stride < K) {
#pragma unroll
        for (int r = 0; r < K; ++r)
          if ((r & stride) == 0) {
            const int32_t a = v[r], b = v[r | stride];
            v[r] = min(a, b);
            v[r | stride] = max(a, b);
          }
      } else {
        const int m = stride / K;
        const bool low = (lane & m) == 0;
#pragma unroll
        for (int r = 0; r < K; ++r) {
          const int32_t o = __shfl_xor_sync(FULL, v[r], m);
          v[r] = low ? min(v[r], o) : max(v[r], o);
        }
      }
    }
  }
}

// One row of at most 32 K entries: sorted positions to caller indices, sorted, written 32
// consecutive entries a store through `stage` (33 words of 32, so both sides are conflict-free).
template <int K>
__device__ __forceinline__ void export_row(const int32_t* __restrict__ src, int len,
                                           const int32_t* __restrict__ perm, int32_t* stage,
                                           int64_t* __restrict__ dst, int lane) {
  int32_t v[K];
#pragma unroll
  for (int r = 0; r < K; ++r) v[r] = 32 * r + lane < len ? ld_stream(src + 32 * r + lane) : -1;
#pragma unroll
  for (int r = 0; r < K; ++r) v[r] = v[r] >= 0 ? perm[v[r]] : INT32_MAX;
  warp_sort<K>(v, lane);
#pragma unroll
  for (int r = 0; r < K; ++r) {
    const int e = lane * K + r;
    stage[e + (e >> 5)] = v[r];
  }
  __syncwarp();
  for (int t = lane; t < len; t += 32) dst[t] = stage[t + (t >> 5)];
  __syncwarp();
}

// Rows in the caller's order and numbering, each ascending: one warp per row, sorted in registers.
// Bound by the network's shuffles and minima; the entries are read and written once: 1.03 ms on the 1M
// torus (160M entries).  With rows filled by one thread each and sorted as 64-bit keys by a segmented
// device sort, building and exporting those lists took 76.5 ms, of a 4,096-particle cloud 0.90 ms;
// with this kernel in its place, on the list build of then, 5.56 and 0.52 ms (3.19 and 0.33 now).  The network is chosen by the row's length; a row over
// EXPORT_MAX entries (the registers of the largest network) goes unsorted to `keys` and into the
// segment list, for the device sort.
constexpr int EXPORT_MAX = 1024;
constexpr int EXPORT_WARPS = 8;

__global__ void __launch_bounds__(EXPORT_WARPS * 32) k_export_rows(
    int64_t n, const int32_t* __restrict__ perm, const int64_t* __restrict__ off_s,
    const int32_t* __restrict__ idx_s, const int64_t* __restrict__ off_o,
    int64_t* __restrict__ idx_o, int64_t* __restrict__ keys, int64_t* __restrict__ seg_beg,
    int64_t* __restrict__ seg_end, unsigned long long* __restrict__ nseg) {
  __shared__ int32_t stage_s[EXPORT_WARPS][EXPORT_MAX + EXPORT_MAX / 32];
  const int64_t k = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (k >= n) return;  // warp-uniform
  int32_t* stage = stage_s[threadIdx.x >> 5];
  const int64_t e0 = off_s[k];
  const int64_t len = off_s[k + 1] - e0;
  const int64_t at = off_o[perm[k]];
  const int32_t* src = idx_s + e0;
  int64_t* dst = idx_o + at;
  if (len <= 128)
    export_row<4>(src, (int)len, perm, stage, dst, lane);
  else if (len <= 256)
    export_row<8>(src, (int)len, perm, stage, dst, lane);
  else if (len <= 512)
    export_row<16>(src, (int)len, perm, stage, dst, lane);
  else if (len <= EXPORT_MAX)
    export_row<32>(src, (int)len, perm, stage, dst, lane);
  else {
    for (int64_t t = lane; t < len; t += 32) keys[at + t] = perm[src[t]];
    if (lane == 0) {
      const unsigned long long s = atomicAdd(nseg, 1ull);
      seg_beg[s] = at;
      seg_end[s] = at + len;
    }
  }
}

// ---------------------------------------------------------------- host orchestration
// Synchronise the stream after a pass whose size the host needs next, and stop on a device
// error the pass raised (so no buffer is sized from a failed pass).
static int pending_check(Engine& E, cudaStream_t st) {
  NB_CUDA(cudaMemcpyAsync(E.h_err, E.d_err, sizeof(int), cudaMemcpyDeviceToHost, st));
  NB_CUDA(host_sync(st));
  if (E.h_err[0] != 0) return check_device_error(E, st);
  return 0;
}

// Resident blocks of the persistent list kernels over the whole device (fewest of the two).
static int list_kernel_slots(Engine& E) {
  if (E.list_slots > 0) return 0;
  int sms = 0, b0 = 0, b1 = 0;
  NB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, E.device));
  NB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b0, k_lists_cand, CAND_WARPS * 32, 0));
  NB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b1, k_lists_test, NB_THREADS, 0));
  // resident warps of each pass over the whole device
  E.list_slots = (int64_t)sms * std::max(1, b1) * (NB_THREADS / 32);
  E.wide_slots = sms;
  E.cand_slots = (int64_t)sms * std::max(1, b0) * CAND_WARPS;
  NB_CUDA(cudaFuncSetAttribute(k_lists_wide, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               2 * WIDE_CAP * (int)sizeof(int32_t)));
  return 0;
}
int build_lists(Engine& E, int64_t n, const double* pos, const double* hs, cudaStream_t st) {
  NB_TRY(E.ensure_n(n));
  if (n == 0) {
    E.lists.n = 0;
    E.lists.total = 0;
    E.lists.longest = 0;
    NB_CUDA(cudaMemsetAsync(E.lists.off, 0, sizeof(int64_t), st));
    return 0;
  }
  Lists& L = E.lists;
  L.gen += 1;
  L.n = 0;  // no lists until these are whole
  E.prof.begin(st);
  // bounding box and Hilbert keys
  int nbb = (int)std::min<int64_t>(grid_for(n), 1184);
  count_launch(), k_bbox_partial<<<nbb, NB_THREADS, 0, st>>>(n, pos, E.bbox_part);
  count_launch(), k_bbox_final<<<1, NB_THREADS, 0, st>>>(nbb, E.bbox_part, E.bbox);
  count_launch(), k_curve_keys<<<grid_for(n), NB_THREADS, 0, st>>>(n, pos, E.bbox, E.keys_a, E.vals_a);
  // the top 48 of the 63 key bits (2^16 cells per axis over the box; within a cell the caller's
  // order): six radix passes instead of eight, and the leaves stay as compact
  size_t tmp = E.cub_bytes;
  NB_CUDA(cub::DeviceRadixSort::SortPairs(E.cub_tmp, tmp, E.keys_a, E.keys_b, E.vals_a, L.perm,
                                          (int)n, 15, 63, st));
  count_launch(), k_gather_sorted<<<grid_for(n), NB_THREADS, 0, st>>>(n, L.perm, pos, hs, L.spos, L.inv_perm);
  // tree
  int64_t nleaf = (n + LEAF - 1) / LEAF;
  TreeView tv;
  int64_t size = nleaf, offs = 0;
  int nl = 0;
  while (true) {
    tv.level_off[nl] = offs;
    tv.level_size[nl] = size;
    offs += size;
    nl += 1;
    if (size == 1 || nl == MAX_LEVELS) break;
    size = (size + FAN - 1) / FAN;
  }
  tv.level_off[nl] = offs;
  tv.nlevels = nl;
  if (tv.level_size[nl - 1] != 1) return set_host_error(E, "tree deeper than MAX_LEVELS");
  NB_TRY(E.ensure_nodes(offs));
  Box32* node_q = static_cast<Box32*>(E.node_q);
  count_launch(), k_leaf_boxes<<<grid_for(nleaf), NB_THREADS, 0, st>>>(
      n, nleaf, L.spos, E.bbox, E.node_lo, E.node_hi, node_q);
  for (int l = 1; l < nl; ++l)
    count_launch(), k_level_up<<<grid_for(tv.level_size[l]), NB_THREADS, 0, st>>>(
        tv.level_size[l - 1], tv.level_size[l], E.node_lo + tv.level_off[l - 1],
        E.node_hi + tv.level_off[l - 1], E.bbox, E.node_lo + tv.level_off[l],
        E.node_hi + tv.level_off[l], node_q + tv.level_off[l]);
  tv.lo = E.node_lo;
  tv.hi = E.node_hi;
  tv.q = node_q;
  int64_t nsub = (n + SUB - 1) / SUB;
  NB_TRY(E.ensure_sub(nsub));
  count_launch(), k_sub_boxes<<<grid_for(nsub), NB_THREADS, 0, st>>>(
      n, nsub, L.spos, E.bbox, E.sub_lo, E.sub_hi, static_cast<Box32*>(E.sub_q));
  // query leaves by cost class, heaviest first, each class in curve order
  uint64_t* cost = E.keys_a;
  uint64_t* order = E.keys_b;
  count_launch(), k_leaf_cost<<<grid_for(nleaf), NB_THREADS, 0, st>>>(nleaf, E.node_lo, E.node_hi, cost);
  tmp = 0;
  NB_CUDA(cub::DeviceRadixSort::SortKeys(nullptr, tmp, cost, order, (int)nleaf, 0, 40, st));
  NB_TRY(E.ensure_cub(tmp));
  tmp = E.cub_bytes;
  NB_CUDA(cub::DeviceRadixSort::SortKeys(E.cub_tmp, tmp, cost, order, (int)nleaf, 0, 40, st));
  NB_TRY(list_kernel_slots(E));
  const unsigned cand_grid = (unsigned)std::max<int64_t>(
      1, std::min<int64_t>(nleaf, E.cand_slots) / CAND_WARPS);
  // candidate lists of the query leaves, each in its own slice of the buffers (sized from the
  // last build's totals; a pass that outgrows them is run again with buffers of its size)
  NB_TRY(E.ensure_leaves(nleaf));
  // batches per work item: 64, less where the leaves are too few to fill the GPU with a warp each
  ListSlices ls{};
  ls.chunk = (int)std::max<int64_t>(4, std::min<int64_t>(64, 64 * nleaf / E.list_slots));
  ls.cbase = E.leaf_cbase;
  ls.bbase = E.leaf_bbase;
  ls.ibase = E.leaf_ibase;
  ls.ncand = E.leaf_ncand;
  ls.cursor = E.d_rowmax + 4;
  int64_t want_cands = E.last_cands > 0 ? E.last_cands + E.last_cands / 4 : nleaf * 512;
  int64_t want_batches = E.last_batches > 0 ? E.last_batches + E.last_batches / 4 : nleaf * 128;
  int64_t nitems = 0;
  for (int attempt = 0;; ++attempt) {
    NB_TRY(E.ensure_tiles(want_cands, want_batches, want_batches / ls.chunk + nleaf));
    ls.items = E.items;
    ls.cap_cands = E.cap_cands;
    ls.cap_batches = E.cap_masks / 32;
    ls.cap_items = E.cap_items;
    NB_CUDA(cudaMemsetAsync(E.d_rowmax, 0, 16 * sizeof(unsigned long long), st));
    count_launch(), k_lists_cand<<<cand_grid, CAND_WARPS * 32, 0, st>>>(
        n, nleaf, order, E.d_rowmax + 2, tv, E.sub_lo, E.sub_hi,
        static_cast<const Box32*>(E.sub_q), E.bbox, ls, E.cands, E.vals_a, E.d_rowmax + 8);
    count_launch(), k_lists_wide<<<(unsigned)std::min<int64_t>(nleaf, E.wide_slots), WIDE_THREADS,
                                   2 * WIDE_CAP * sizeof(int32_t), st>>>(
        n, E.vals_a, E.d_rowmax + 8, tv, E.sub_lo, E.sub_hi, static_cast<const Box32*>(E.sub_q),
        E.bbox, ls, E.cands, E.d_err);
    NB_CUDA(cudaMemcpyAsync(E.h_build, E.d_rowmax + 4, 3 * sizeof(int64_t), cudaMemcpyDeviceToHost, st));
    NB_TRY(pending_check(E, st));
    const int64_t ncand = E.h_build[0], nbatch = E.h_build[1];
    nitems = E.h_build[2];
    E.last_cands = ncand;
    E.last_batches = nbatch;
    if (ncand <= ls.cap_cands && nbatch <= ls.cap_batches && nitems <= ls.cap_items) break;
    if (attempt > 0) return set_host_error(E, "list build: candidate buffers outgrown twice");
    want_cands = ncand + ncand / 4;
    want_batches = nbatch + nbatch / 4;
  }
  // the tests, once: hit masks per batch and lane, entries per row
  NB_CUDA(cudaMemsetAsync(E.counts, 0, sizeof(int64_t) * n, st));
  const unsigned grid = (unsigned)std::max<int64_t>(
      1, std::min<int64_t>(nitems, E.list_slots) / (NB_THREADS / 32));
  count_launch(), k_lists_test<<<grid, NB_THREADS, 0, st>>>(
      n, E.d_rowmax + 3, tv, L.spos, E.cands, ls, E.masks, E.part_count, E.counts);
  count_launch(), k_row_max<<<std::min(grid_for(n), 592u), NB_THREADS, 0, st>>>(n, E.counts, E.d_rowmax);
  NB_CUDA(cudaMemsetAsync(L.off, 0, sizeof(int64_t), st));
  tmp = E.cub_bytes;
  NB_CUDA(cub::DeviceScan::InclusiveSum(E.cub_tmp, tmp, E.counts, L.off + 1, (int)n, st));
  NB_CUDA(cudaMemcpyAsync(E.h_build, L.off + n, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
  NB_CUDA(cudaMemcpyAsync(E.h_build + 1, E.d_rowmax, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
  NB_TRY(pending_check(E, st));
  const int64_t total = E.h_build[0], longest = E.h_build[1];
  NB_TRY(E.ensure_list_capacity(total));
  // masks -> entries at the rows' offsets (the store of a row's stretch stays inside the row: the
  // counts are the masks' own)
  count_launch(), k_lists_expand<<<grid_for(nitems * 32, EXPAND_WARPS * 32), EXPAND_WARPS * 32, 0, st>>>(
      n, nitems, E.cands, ls, E.masks, E.part_count, L.off, L.idx, E.d_err);
  E.prof.end(PROF_LISTS, st, (double)n, (double)total);
  L.n = n;
  L.total = total;
  L.longest = longest;
  return check_device_error(E, st);
}

// Offsets (n + 1) of the last build's lists in the caller's order.
int export_lists_offsets(Engine& E, int64_t* off_out, cudaStream_t st) {
  Lists& L = E.lists;
  int64_t n = L.n;
  NB_CUDA(cudaMemsetAsync(off_out, 0, sizeof(int64_t), st));
  if (n == 0) return 0;
  count_launch(), k_export_counts<<<grid_for(n), NB_THREADS, 0, st>>>(n, L.inv_perm, L.off, E.counts);
  size_t tmp = E.cub_bytes;
  NB_CUDA(cub::DeviceScan::InclusiveSum(E.cub_tmp, tmp, E.counts, off_out + 1, (int)n, st));
  return check_device_error(E, st);
}

// Entries of the last build's lists in the caller's order and numbering, each row ascending;
// off_out must hold the offsets from export_lists_offsets.
int export_lists(Engine& E, int64_t* off_out, int64_t* idx_out, cudaStream_t st) {
  Lists& L = E.lists;
  int64_t n = L.n;
  if (n == 0) return 0;
  const bool long_rows = L.longest > EXPORT_MAX;
  unsigned long long* nseg = E.d_rowmax + 9;
  int64_t* seg_beg = E.counts;  // scratch of at least n entries each, free between builds
  int64_t* seg_end = reinterpret_cast<int64_t*>(E.keys_b);
  if (long_rows) {
    NB_TRY(E.ensure_sort_keys(L.total));
    NB_CUDA(cudaMemsetAsync(nseg, 0, sizeof(unsigned long long), st));
  }
  count_launch(), k_export_rows<<<grid_for(n * 32, EXPORT_WARPS * 32), EXPORT_WARPS * 32, 0, st>>>(
      n, L.perm, L.off, L.idx, off_out, idx_out, E.sort_keys, seg_beg, seg_end, nseg);
  if (long_rows) {
    NB_CUDA(cudaMemcpyAsync(E.h_build, nseg, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
    NB_CUDA(host_sync(st));
    size_t tmp = E.cub_bytes;
    NB_CUDA(cub::DeviceSegmentedSort::SortKeys(E.cub_tmp, tmp, E.sort_keys, idx_out, L.total,
                                                (int)E.h_build[0], seg_beg, seg_end, st));
  }
  return check_device_error(E, st);
}

// ---------------------------------------------------------------- the reference's cell grid
// sim/neighbours.py:95-126 (_cell_of, _build_grid): per axis k = floor((x - lo) * inv_cell),
// clamped to [0, ncell - 1], cell = (cx * ny + cy) * nz + cz, and a stable counting sort of the
// particles by cell (start: ncell + 1 offsets, order: particles by cell, ascending index within a
// cell).  The subtraction and product round as the reference's (no fused multiply-add), so the
// assignment is the same bit for bit.  The lists above do not need these cells (their tree
// prunes with exact tests); this is the reference's cell assignment on its own, for callers and
// for the parity tests.
__global__ void k_cell_index(int64_t n, const double* __restrict__ pos, double lo0, double lo1,
                             double lo2, double ic0, double ic1, double ic2, int64_t n0,
                             int64_t n1, int64_t n2, uint32_t* __restrict__ cell,
                             int32_t* __restrict__ iota,
                             unsigned long long* __restrict__ per_cell) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double lo[3] = {lo0, lo1, lo2}, ic[3] = {ic0, ic1, ic2};
  const int64_t nc[3] = {n0, n1, n2};
  int64_t k[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    double t = __dmul_rn(__dsub_rn(pos[3 * i + c], lo[c]), ic[c]);
    int64_t v = (int64_t)floor(t);
    k[c] = v < 0 ? 0 : (v >= nc[c] ? nc[c] - 1 : v);
  }
  const int64_t id = (k[0] * n1 + k[1]) * n2 + k[2];
  cell[i] = (uint32_t)id;
  iota[i] = (int32_t)i;
  atomicAdd(per_cell + id, 1ull);
}

__global__ void k_widen_order(int64_t n, const int32_t* __restrict__ src, int64_t* __restrict__ dst) {
  int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k < n) dst[k] = src[k];
}

int build_cells(Engine& E, int64_t n, const double* pos, const double* lo, const double* inv_cell,
                const int64_t* ncell, int64_t* start, int64_t* order, cudaStream_t st) {
  const int64_t total = ncell[0] * ncell[1] * ncell[2];
  if (ncell[0] < 1 || ncell[1] < 1 || ncell[2] < 1 || total > (int64_t)INT32_MAX)
    return set_host_error(E, "cell counts must be positive and hold at most 2^31 cells");
  NB_TRY(E.ensure_n(std::max<int64_t>(n, 1)));
  NB_TRY(E.ensure_sort_keys(total));
  unsigned long long* per_cell = reinterpret_cast<unsigned long long*>(E.sort_keys);
  NB_CUDA(cudaMemsetAsync(per_cell, 0, sizeof(int64_t) * total, st));
  NB_CUDA(cudaMemsetAsync(start, 0, sizeof(int64_t), st));
  if (n > 0) {
    uint32_t* cell = reinterpret_cast<uint32_t*>(E.keys_a);
    uint32_t* cell_sorted = reinterpret_cast<uint32_t*>(E.keys_b);
    int32_t* by_cell = reinterpret_cast<int32_t*>(E.keys_b) + E.cap_n;  // second half of keys_b
    count_launch(), k_cell_index<<<grid_for(n), NB_THREADS, 0, st>>>(
        n, pos, lo[0], lo[1], lo[2], inv_cell[0], inv_cell[1], inv_cell[2], ncell[0], ncell[1],
        ncell[2], cell, E.vals_a, per_cell);
    int end_bit = 1;
    while (end_bit < 32 && (int64_t(1) << end_bit) < total) ++end_bit;
    size_t tmp = 0;
    NB_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tmp, cell, cell_sorted, E.vals_a, by_cell,
                                            (int)n, 0, end_bit, st));
    NB_TRY(E.ensure_cub(tmp));
    tmp = E.cub_bytes;
    // radix sort is stable: within a cell the particles keep ascending index, as the reference's
    // counting sort leaves them
    NB_CUDA(cub::DeviceRadixSort::SortPairs(E.cub_tmp, tmp, cell, cell_sorted, E.vals_a, by_cell,
                                            (int)n, 0, end_bit, st));
    count_launch(), k_widen_order<<<grid_for(n), NB_THREADS, 0, st>>>(n, by_cell, order);
  }
  size_t tmp = 0;
  const int64_t* counts = reinterpret_cast<const int64_t*>(per_cell);
  NB_CUDA(cub::DeviceScan::InclusiveSum(nullptr, tmp, counts, start + 1, (int)total, st));
  NB_TRY(E.ensure_cub(tmp));
  tmp = E.cub_bytes;
  NB_CUDA(cub::DeviceScan::InclusiveSum(E.cub_tmp, tmp, counts, start + 1, (int)total, st));
  return check_device_error(E, st);
}

// sim/neighbours.py:250-265 (find_neighbours_numba, no periodic box): lo = the smallest
// coordinates, cell = max(R_KERN * median(h) / 2, max(span) / 160, 1e-300), ncell = floor(span /
// cell) + 1 per axis, inv_cell = 1 / cell (host outputs; the call synchronises its stream).
int cell_geometry(Engine& E, int64_t n, const double* pos, const double* h, double* lo,
                  double* inv_cell, int64_t* ncell, cudaStream_t st) {
  if (n <= 0) return set_host_error(E, "the cell grid needs at least one particle");
  NB_TRY(E.ensure_n(n));
  int nbb = (int)std::min<int64_t>(grid_for(n), 1184);
  double* span6 = E.red;  // not E.bbox: the FP32 records of a run on its cached lists are in that box
  count_launch(), k_bbox_partial<<<nbb, NB_THREADS, 0, st>>>(n, pos, E.bbox_part);
  count_launch(), k_bbox_final<<<1, NB_THREADS, 0, st>>>(nbb, E.bbox_part, span6);
  double* h_sorted = reinterpret_cast<double*>(E.keys_b);
  size_t tmp = 0;
  NB_CUDA(cub::DeviceRadixSort::SortKeys(nullptr, tmp, h, h_sorted, (int)n, 0, 64, st));
  NB_TRY(E.ensure_cub(tmp));
  tmp = E.cub_bytes;
  NB_CUDA(cub::DeviceRadixSort::SortKeys(E.cub_tmp, tmp, h, h_sorted, (int)n, 0, 64, st));
  double box[6], mid[2];
  NB_CUDA(cudaMemcpyAsync(box, span6, sizeof(box), cudaMemcpyDeviceToHost, st));
  NB_CUDA(cudaMemcpyAsync(mid, h_sorted + (n - 1) / 2, sizeof(double) * (n % 2 ? 1 : 2),
                          cudaMemcpyDeviceToHost, st));
  NB_CUDA(host_sync(st));
  // numpy's median: the middle value, or the mean of the two middle values for even n
  const double median = n % 2 ? mid[0] : (mid[0] + mid[1]) / 2.0;
  double span[3], smax = 0.0;
  for (int c = 0; c < 3; ++c) {
    lo[c] = box[c];
    span[c] = box[3 + c] - box[c];
    smax = std::max(smax, span[c]);
  }
  const double cell = std::max(std::max(0.5 * 2.0 * median, smax / 160.0), 1e-300);
  for (int c = 0; c < 3; ++c) {
    ncell[c] = std::max<int64_t>((int64_t)std::floor(span[c] / cell) + 1, 1);
    inv_cell[c] = 1.0 / cell;
  }
  return check_device_error(E, st);
}

size_t cub_bytes_needed(int64_t n, int64_t m) {
  size_t a = 0, b = 0, c = 0, d = 0;
  cub::DeviceRadixSort::SortPairs((void*)nullptr, a, (uint64_t*)nullptr, (uint64_t*)nullptr,
                                  (int32_t*)nullptr, (int32_t*)nullptr, (int)n, 0, 63);
  cub::DeviceScan::InclusiveSum((void*)nullptr, b, (int64_t*)nullptr, (int64_t*)nullptr, (int)n);
  if (m > 0)
    cub::DeviceSegmentedSort::SortKeys((void*)nullptr, c, (int64_t*)nullptr, (int64_t*)nullptr,
                                       m, (int)n, (int64_t*)nullptr, (int64_t*)nullptr);
  cub::DeviceSelect::Flagged((void*)nullptr, d, (int64_t*)nullptr, (const uint8_t*)nullptr,
                             (int64_t*)nullptr, (int64_t*)nullptr, (int)n);
  size_t e = 0;
  cub::DeviceSelect::Flagged((void*)nullptr, e, thrust::counting_iterator<int64_t>(0),
                             (const uint8_t*)nullptr, (int64_t*)nullptr, (int64_t*)nullptr, (int)n);
  return std::max(std::max(std::max(a, b), std::max(c, d)), e) + 256;
}

}  // namespace nbk
