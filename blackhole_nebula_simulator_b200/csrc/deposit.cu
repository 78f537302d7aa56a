// Particle -> grid deposition for the renderer (render/gasgrid.py:316-597 of the reference):
// each particle's fields (m, m T, m T^4, m v) go to the cells whose centres lie inside its
// support (q < 2), weighted by f(q) V_c and normalised; fewer than 8 such centres: trilinear
// weights in index space over the 8 nearest centres.  Weight beyond the grid goes to the
// `outside` total.  On the log grid a thread (a warp for wide supports) walks a particle's candidate
// centres twice (sum of weights, then the atomic adds); the box is gathered brick by brick; the
// cell sums are FP64.  Which centres count towards the choice of weights is the reference's own
// arithmetic (compiled without contraction); the weights themselves are within rounding of it, and the
// order of the additions is not its order.
#include <cub/cub.cuh>

#include "common.cuh"
#include "deposit.cuh"
#include "engine.cuh"

namespace nbk {

constexpr int DEP_MIN_CELLS = 8;
constexpr int DEP_INNER_VIRTUAL = 64;  // virtual log shells below r_min (render/gasgrid.py:49)

// the azimuth in [0, 2 pi): Python's atan2(y, x) % (2 pi)
__device__ __forceinline__ double azimuth(double y, double x) {
  const double a = atan2(y, x);
  return a < 0.0 ? a + 2.0 * 3.141592653589793 : a;
}
__device__ __forceinline__ int py_imod(int a, int b) { return ((a % b) + b) % b; }

__device__ __forceinline__ void particle_vals(int64_t p, const double* m, const double* t,
                                              const double* v, double* vals) {
  const double mp = m[p], tp = t[p];
  vals[0] = mp;
  vals[1] = mp * tp;
  const double t2 = tp * tp;
  vals[2] = mp * (t2 * t2);
  vals[3] = mp * v[3 * p];
  vals[4] = mp * v[3 * p + 1];
  vals[5] = mp * v[3 * p + 2];
}

__device__ __forceinline__ void add_cell(double* acc, int64_t cell, double w, const double* vals) {
  double* c = acc + cell * DEP_FIELDS;
#pragma unroll
  for (int f = 0; f < DEP_FIELDS; ++f) atomicAdd(c + f, w * vals[f]);
}

// ---------------------------------------------------------------- log-spherical grid
// Shell i of a log grid, from -DEP_INNER_VIRTUAL: radius of its centres and (r2^3 - r1^3) / 3.
__device__ __forceinline__ double2 log_shell(const LogGeom& g, int i) {
  const double rc = g.r_min * exp((i + 0.5) * g.dlnr);
  const double r1 = g.r_min * exp(i * g.dlnr);
  const double r2 = r1 * exp(g.dlnr);
  return make_double2(rc, (r2 * r2 * r2 - r1 * r1 * r1) / 3.0);
}

__global__ void k_log_shells(LogGeom g, double2* __restrict__ shells) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < g.nr + DEP_INNER_VIRTUAL) shells[i] = log_shell(g, i - DEP_INNER_VIRTUAL);
}

// The tables of a grid in the order sth, cth, dcth (nth each), cph, sph (nph each), cell volumes
// (nr, nth) (render/gasgrid.py:125-129, 688-692).
__global__ void k_log_tables(LogGeom g, double* __restrict__ out) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  double* vol = out + 3 * g.nth + 2 * g.nph;
  if (e < g.nth) {
    const double th = (e + 0.5) * g.dth;
    out[e] = sin(th);
    out[g.nth + e] = cos(th);
    out[2 * g.nth + e] = cos(e * g.dth) - cos((e + 1) * g.dth);
  }
  if (e < g.nph) {
    const double ph = (e + 0.5) * g.dph;
    out[3 * g.nth + e] = cos(ph);
    out[3 * g.nth + g.nph + e] = sin(ph);
  }
  if (e < g.nr * g.nth) {
    const int i = e / g.nth, j = e % g.nth;
    const double r1 = g.r_min * exp(i * g.dlnr), r2 = r1 * exp(g.dlnr);
    vol[e] = (r2 * r2 * r2 - r1 * r1 * r1) / 3.0 *
             (cos(j * g.dth) - cos((j + 1) * g.dth)) * g.dph;
  }
}

// One particle's candidate centres: a block of shells, theta rows and phi columns that holds every
// centre inside its support, from the support's angular radius asin(2h / r) and the widest
// azimuth asin(2h / (r sin theta)) of that cap, both wider than acos and asin round (1.5e-8 at worst).
struct LogParticle {
  double x, y, z, h, rr, th, ph;
  int i_lo, i_hi, j0, nj, k0, nk;
};

__device__ __forceinline__ LogParticle log_particle(const LogGeom& g, int64_t p,
                                                    const double* __restrict__ x,
                                                    const double* __restrict__ h) {
  LogParticle q;
  q.x = x[3 * p];
  q.y = x[3 * p + 1];
  q.z = x[3 * p + 2];
  q.h = h[p];
  const double big = 2.0 * q.h;
  q.rr = sqrt(q.x * q.x + q.y * q.y + q.z * q.z);
  q.th = acos(fmin(1.0, fmax(-1.0, q.z / q.rr)));
  q.ph = azimuth(q.y, q.x);
  const double s = big / q.rr;
  const int i_max = (int)fmin(720.0 / g.dlnr, 1e9);  // beyond, radii overflow
  q.j0 = q.k0 = 0;
  q.nj = g.nth;
  q.nk = g.nph;
  if (s < 1.0) {
    // log(1 + s) <= s, log(1 - s) >= -s / (1 - s)
    const double fr = log(q.rr / g.r_min) / g.dlnr;
    q.i_hi = (int)floor(fmin(fr + s / g.dlnr - 0.5 + 1e-6, (double)i_max));
    q.i_lo = (int)ceil(fmax(fr - s / ((1.0 - s) * g.dlnr) - 0.5 - 1e-6, -(double)DEP_INNER_VIRTUAL));
    const double a = asin(s) + 1e-7, st = sqrt(q.x * q.x + q.y * q.y) / q.rr;
    q.j0 = max(0, (int)ceil((q.th - a) / g.dth - 0.5));
    q.nj = max(0, min(g.nth - 1, (int)floor((q.th + a) / g.dth - 0.5)) - q.j0 + 1);
    if (s < st * (1.0 - 1e-6)) {
      const double d = asin(s / st) + 1e-7;
      const int k0 = (int)ceil((q.ph - d) / g.dph - 0.5), k1 = (int)floor((q.ph + d) / g.dph - 0.5);
      if (k1 < k0) {
        q.nj = 0;
      } else if (k1 - k0 + 1 < g.nph) {
        q.k0 = k0;
        q.nk = k1 - k0 + 1;
      }
    }
  } else {
    q.i_hi = (int)fmin(floor((log(q.rr + big) - log(g.r_min)) / g.dlnr), (double)i_max);
    q.i_lo = -DEP_INNER_VIRTUAL;
  }
  q.i_lo = max(q.i_lo, -DEP_INNER_VIRTUAL);
  if (!(big > 0.0) || isnan(s) || isinf(q.rr)) q.nj = 0;  // no centre is inside
  return q;
}

// render/gasgrid.py:316-412 (_nb_log_kernel_pass) over those candidates, dealt to `size` threads:
// MODE 0 sums f V and counts the centres inside the support, MODE 1 adds the normalised weights
// and the mass beyond the grid.  d^2 is a few fused operations from (rc sin th) cos ph - x and its
// like, as the reference forms them: within 12 u |d| (r + |d|), u = 2^-53.  A centre ten times that
// close to (2h)^2 is decided by the reference's own arithmetic, which counts it for the kernel's or
// the trilinear weights; the weights take q = sqrt(d^2) (1 / h), within rounding of its quotient.
template <int MODE>
__device__ __forceinline__ void log_pass(const LogGeom& g, const double2* __restrict__ shells,
                                         const LogParticle& q, int rank, int size, int kid,
                                         double inv, const double* vals, double* acc,
                                         double& wsum, int& n_in, double& outside) {
  const double big = 2.0 * q.h, big2 = big * big;
  const double edge = 1e-12 * big2 + 1.4e-14 * big * q.rr, in2 = big2 - edge, out2 = big2 + edge;
  const double ih = 1.0 / q.h;
  const int dj = size / q.nk, dk = size % q.nk;
  int j = q.j0 + rank / q.nk, c = rank % q.nk;
  for (int e = rank; e < q.nj * q.nk; e += size) {
    int k = q.k0 + c;
    if (k < 0 || k >= g.nph) k = py_imod(k, g.nph);
    const double sth = g.sth[j], cth = g.cth[j], cph = g.cph[k], sph = g.sph[k];
    const double ux = sth * cph, uy = sth * sph;
    // the nearest point of the ray through this column's centres
    const double along = q.x * ux + q.y * uy + q.z * cth;
    const double off2 = along > 0.0 ? q.rr * q.rr - along * along : q.rr * q.rr;
    if (off2 < out2 + 1e-9 * q.rr * q.rr) {
      const double dvol = g.dcth[j] * g.dph;
      for (int i = q.i_lo; i <= q.i_hi; ++i) {
        const double2 sh = i < g.nr ? shells[i + DEP_INNER_VIRTUAL] : log_shell(g, i);
        const double dxc = fma(sh.x, ux, -q.x), dyc = fma(sh.x, uy, -q.y), dzc = fma(sh.x, cth, -q.z);
        const double dd = fma(dzc, dzc, fma(dyc, dyc, dxc * dxc));
        if (dd >= out2) continue;
        if (dd >= in2) {
          const double rst = sh.x * sth;
          const double ex = rst * cph - q.x, ey = rst * sph - q.y, ez = sh.x * cth - q.z;
          if (!(sqrt(d2_exact(ex, ey, ez)) / q.h < 2.0)) continue;
        }
        const double f = kernel_f<double>(sqrt(dd) * ih, kid) * (sh.y * dvol);
        if (MODE == 0) {
          n_in += 1;
          wsum += f;
        } else {
          const double w = f * inv;
          if (0 <= i && i < g.nr)
            add_cell(acc, ((int64_t)i * g.nth + j) * g.nph + k, w, vals);
          else
            outside += w * vals[0];
        }
      }
    }
    j += dj;
    c += dk;
    if (c >= q.nk) {
      c -= q.nk;
      j += 1;
    }
  }
}

// render/gasgrid.py:217-237: trilinear weights in index space over the eight nearest centres
__device__ __forceinline__ void log_trilinear(const LogGeom& g, const LogParticle& q,
                                              const double* vals, double* acc, double& out) {
  const double fr = log(q.rr / g.r_min) / g.dlnr - 0.5;
  const double fth = q.th / g.dth - 0.5;
  const double fph = q.ph / g.dph - 0.5;
  const int i0 = (int)floor(fr);
  int j0 = (int)floor(fth);
  const int k0 = (int)floor(fph);
  const double ti = fr - i0, tk = fph - k0;
  double tj = fth - j0;
  if (j0 < 0) {
    j0 = 0;
    tj = 0.0;
  }
  if (j0 > g.nth - 2) {
    j0 = g.nth - 2;
    tj = 1.0;
  }
  for (int di = 0; di < 2; ++di) {
    const double wi = di == 1 ? ti : 1.0 - ti;
    for (int dj = 0; dj < 2; ++dj) {
      const double wj = dj == 1 ? tj : 1.0 - tj;
      for (int dk = 0; dk < 2; ++dk) {
        const double wk = dk == 1 ? tk : 1.0 - tk;
        const double w = wi * wj * wk;
        const int64_t i = (int64_t)i0 + di;
        if (0 <= i && i < g.nr)
          add_cell(acc, (i * g.nth + j0 + dj) * g.nph + py_imod(k0 + dk, g.nph), w, vals);
        else
          out += w * vals[0];
      }
    }
  }
}

struct LogTarget {
  LogGeom g;
  const double2* shells;
  double* acc;
  double* outside;
  unsigned long long* n_tri;
};

// render/gasgrid.py:415-531 (_nb_log_deposit_chunk) for one particle, by one thread or by a warp;
// returns (a part of) the mass beyond the grid
template <int SIZE>
__device__ __forceinline__ double log_one(const LogTarget& T, const LogParticle& q, int64_t p,
                                          int rank, const double* __restrict__ m,
                                          const double* __restrict__ t,
                                          const double* __restrict__ v, int kid, bool& tri) {
  double vals[DEP_FIELDS];
  particle_vals(p, m, t, v, vals);
  double wsum = 0.0, out = 0.0;
  int n_in = 0;
  log_pass<0>(T.g, T.shells, q, rank, SIZE, kid, 0.0, vals, T.acc, wsum, n_in, out);
  if (SIZE > 1) {
    n_in = __reduce_add_sync(0xffffffffu, n_in);
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) wsum += __shfl_xor_sync(0xffffffffu, wsum, d);
  }
  // (where every centre is a rounding from the edge none has a weight: trilinear too, not counted)
  if (n_in >= DEP_MIN_CELLS && wsum > 0.0) {
    log_pass<1>(T.g, T.shells, q, rank, SIZE, kid, 1.0 / wsum, vals, T.acc, wsum, n_in, out);
  } else if (rank == 0) {
    tri = n_in < DEP_MIN_CELLS;
    log_trilinear(T.g, q, vals, T.acc, out);
  }
  return out;
}

// A thread per particle, those with more than LOG_WIDE candidates listed for a warp each in a second
// launch: a serial walk of thousands of centres would be a tail of its own, and a small input with
// wide supports would leave the chip idle.  Bound by L2's FP64 adds (eight a centre) and the walk's
// FP64 arithmetic.  The whole call for the disc sampled by 1,000,003 particles (cubic) 0.90 ms; 2.08
// with a thread for every particle over the reference's wider windows, one grid after the other.  20,000 / 150,000 / 2,000,000 particles 1.1 / 0.73 / 1.35 ms (8.1 / 3.87 / 2.38).
// LOG_WIDE 64 / 128 / 256 differ by 2 % but for 50,000 Wendland particles: 1.56 / 1.60 / 1.71 ms.  Blocks
// an SM of the first launch, 4 / 5 / 6: 0.905 / 0.894 / 0.926 ms at 1,000,003.
// Particles from n_narrow on are the second grid's (the coarser one of very wide particles).
constexpr int LOG_WIDE = 128;
constexpr int LOG_B = 4;  // blocks an SM of the second launch
__global__ void __launch_bounds__(128, 5) k_deposit_log(
    int64_t n, const unsigned long long* __restrict__ n_wide, const double* __restrict__ x,
    const double* __restrict__ h, const double* __restrict__ m, const double* __restrict__ t,
    const double* __restrict__ v, LogTarget fine, LogTarget coarse, int kid,
    int32_t* __restrict__ list, unsigned long long* __restrict__ nlist) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t n_narrow = n_wide ? n - (int64_t)*n_wide : n;
  double out = 0.0;
  bool heavy = false, tri = false;
  if (p < n) {
    const LogTarget& T = p < n_narrow ? fine : coarse;
    const LogParticle q = log_particle(T.g, p, x, h);
    heavy = (int64_t)(q.i_hi - q.i_lo + 1) * q.nj * q.nk > LOG_WIDE;
    if (!heavy) {
      const double o = log_one<1>(T, q, p, 0, m, t, v, kid, tri);
      if (p < n_narrow)
        out = o;
      else if (o != 0.0)
        atomicAdd(coarse.outside, o);
    }
  }
  const unsigned hm = __ballot_sync(FULL, heavy);
  if (hm) {
    unsigned long long at = 0;
    if (lane == 0) at = atomicAdd(nlist, (unsigned long long)__popc(hm));
    at = __shfl_sync(FULL, at, 0);
    if (heavy) list[at + __popc(hm & ((1u << lane) - 1u))] = (int32_t)p;
  }
  // one count per warp and grid: an atomic per particle on one address would bound the small supports
  const unsigned tf = __ballot_sync(FULL, tri && p < n_narrow), tc = __ballot_sync(FULL, tri && p >= n_narrow);
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) out += __shfl_xor_sync(FULL, out, d);
  if (lane == 0) {
    if (out != 0.0) atomicAdd(fine.outside, out);
    if (tf) atomicAdd(fine.n_tri, (unsigned long long)__popc(tf));
    if (tc) atomicAdd(coarse.n_tri, (unsigned long long)__popc(tc));
  }
}

__global__ void __launch_bounds__(128, LOG_B) k_deposit_log_heavy(
    int64_t n, const unsigned long long* __restrict__ n_wide, const double* __restrict__ x,
    const double* __restrict__ h, const double* __restrict__ m, const double* __restrict__ t,
    const double* __restrict__ v, LogTarget fine, LogTarget coarse, int kid,
    const int32_t* __restrict__ list, const unsigned long long* __restrict__ nlist) {
  const int lane = threadIdx.x & 31;
  const int64_t n_narrow = n_wide ? n - (int64_t)*n_wide : n;
  const int64_t all = (int64_t)*nlist;
  for (int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; w < all;
       w += ((int64_t)gridDim.x * blockDim.x) >> 5) {
    const int64_t p = list[w];
    const LogTarget& T = p < n_narrow ? fine : coarse;
    bool tri = false;
    const double o = log_one<32>(T, log_particle(T.g, p, x, h), p, lane, m, t, v, kid, tri);
    if (tri) atomicAdd(T.n_tri, 1ull);
    if (o != 0.0) atomicAdd(T.outside, o);
  }
}

// ---------------------------------------------------------------- Cartesian box
// render/gasgrid.py:534-597 (_nb_box_deposit_chunk), as a gather.  A particle's weights need the
// sum of its kernel values over every centre of its support first; then each cell adds up the
// particles that reach it:
//   k_box_classify  a thread per particle: particles wholly beyond the box only add their mass to
//                   `outside`; the others go to a work list, those with wide supports from its end
//   k_box_weights   a warp (a block for the wide ones) per listed particle: the kernel sum, the
//                   part of it outside the box, the trilinear fallback below 8 centres; the
//                   record of the particle and the number of particles per brick of 8^3 cells
//   k_box_lists     the bricks' particle lists, BOX_PAIRS entries at a time
//   k_box_bricks    a block per brick and stretch of its list, a warp per 2 x 4 x 4 cells, a cell
//                   per lane, the six sums in registers: no atomic add per (particle, cell)
// Bound by the FP64 pipe (a kernel value per lane of every sub-brick a support reaches, about a
// third to a half of the lanes inside).  The 1,048,576-particle torus into 160^3 cells takes
// 3.73 ms (bricks 1.40, weights 1.37 + 0.66 for the wide particles); one thread per particle
// walking its support with six atomic adds per cell kept 5 of 32 lanes busy, sent 1.8e9
// reductions to L2 and took 61 ms.  A particle of BOX_WIDE candidate cells (25.4^3) or more takes a
// block, so that none keeps a warp alone for a millisecond.
constexpr int BRICK = 8;            // cells per brick edge
constexpr int BRICK_WARPS = 16;     // sub-bricks of 2 x 4 x 4 cells
constexpr int BRICK_STAGE = 128;    // records staged in shared memory at a time
constexpr int BRICK_CHUNK = 512;    // records of one block's stretch of a brick's list
constexpr int BOX_REC = 12;         // doubles per record: x, y, z, h, 1/h, -, six weighted fields
constexpr int BOX_WIDE = 16384;     // candidate cells from which a block takes the particle

// Entries of the bricks' lists held at once (1 GiB): twice what a frame of ten million particles
// of twenty-odd bricks each needs, so only supports far wider than a brick are taken in parts.
constexpr int64_t BOX_PAIRS = int64_t(1) << 28;

struct BoxGeom {
  double x0, y0, z0, dx;
  int nb, bricks;  // cells and bricks per axis
};

// (int)floor of the reference's index expressions; a NaN gives the lowest int (the conversion of a
// double does), a cell beyond the box
__device__ __forceinline__ int cell_of(double v, double lo, double dx) {
  return (int)floor((v - lo) / dx);
}

// d^2 of a centre, in one arithmetic for the weights' sum and for the bricks: only so do a particle's
// weights add up to one where its centres all lie close to the support's edge
__device__ __forceinline__ double box_yz2(double dy, double dz) { return fma(dz, dz, dy * dy); }
__device__ __forceinline__ double box_d2(double dx, double yz2) { return fma(dx, dx, yz2); }

struct BoxRange {
  int a0, a1, b0, b1, c0, c1;
};
__device__ __forceinline__ BoxRange box_range(const BoxGeom& g, double x, double y, double z,
                                              double big) {
  BoxRange r;
  r.a0 = cell_of(x - big, g.x0, g.dx), r.a1 = cell_of(x + big, g.x0, g.dx);
  r.b0 = cell_of(y - big, g.y0, g.dx), r.b1 = cell_of(y + big, g.y0, g.dx);
  r.c0 = cell_of(z - big, g.z0, g.dx), r.c1 = cell_of(z + big, g.z0, g.dx);
  return r;
}
__device__ __forceinline__ bool box_beyond(const BoxRange& r, int nb) {
  return r.a1 < 0 || r.a0 >= nb || r.b1 < 0 || r.b0 >= nb || r.c1 < 0 || r.c0 >= nb;
}
// Any point lies within sqrt(3) cells of the eight centres around it, so a support of that
// radius holds at least eight centres; false for NaN and infinite positions, which hold none.
__device__ __forceinline__ bool box_holds_eight(double x, double y, double z, double big, double dx) {
  return big >= 1.7320508075688774 * (1.0 + 1e-9) * dx && isfinite(x) && isfinite(y) && isfinite(z);
}

__global__ void __launch_bounds__(NB_THREADS) k_box_classify(
    int64_t n, const double* __restrict__ x, const double* __restrict__ h,
    const double* __restrict__ m, BoxGeom g, int32_t* __restrict__ list,
    unsigned long long* __restrict__ nlist, double* outside_sum) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  bool small = false, wide = false;
  double out = 0.0;
  if (p < n) {
    const double xp = x[3 * p], yp = x[3 * p + 1], zp = x[3 * p + 2];
    const double big = 2.0 * h[p];
    const BoxRange r = box_range(g, xp, yp, zp, big);
    if (box_beyond(r, g.nb) && box_holds_eight(xp, yp, zp, big, g.dx)) {
      out = m[p];
    } else {
      const double cells = ((double)r.a1 - r.a0 + 1.0) * ((double)r.b1 - r.b0 + 1.0) *
                           ((double)r.c1 - r.c0 + 1.0);
      wide = cells >= (double)BOX_WIDE;
      small = !wide;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) out += __shfl_xor_sync(FULL, out, o);
  if (lane == 0 && out != 0.0) atomicAdd(outside_sum, out);
  // a warp takes its places in the list with one add per end
  const unsigned ms = __ballot_sync(FULL, small), mw = __ballot_sync(FULL, wide);
  unsigned long long bs = 0, bw = 0;
  if (lane == 0) {
    if (ms) bs = atomicAdd(nlist, (unsigned long long)__popc(ms));
    if (mw) bw = atomicAdd(nlist + 1, (unsigned long long)__popc(mw));
  }
  bs = __shfl_sync(FULL, bs, 0);
  bw = __shfl_sync(FULL, bw, 0);
  const unsigned below = (1u << lane) - 1u;
  if (small) list[bs + __popc(ms & below)] = (int32_t)p;
  if (wide) list[n - 1 - (int64_t)(bw + __popc(mw & below))] = (int32_t)p;
}

// calls f(brick) for the bricks that the support reaches, dealt to the threads of a group
template <typename F>
__device__ __forceinline__ void for_bricks(const BoxGeom& g, double x, double y, double z,
                                           double big, int rank, int size, F&& f) {
  const BoxRange r = box_range(g, x, y, z, big);
  if (box_beyond(r, g.nb)) return;
  const int a0 = max(r.a0, 0) / BRICK, a1 = min(r.a1, g.nb - 1) / BRICK;
  const int b0 = max(r.b0, 0) / BRICK, b1 = min(r.b1, g.nb - 1) / BRICK;
  const int c0 = max(r.c0, 0) / BRICK, c1 = min(r.c1, g.nb - 1) / BRICK;
  const int nb = b1 - b0 + 1, nc = c1 - c0 + 1;
  const int64_t all = (int64_t)(a1 - a0 + 1) * nb * nc;
  const double reach2 = big * big * (1.0 + 1e-9);
  const double edge = BRICK * g.dx;
  for (int64_t e = rank; e < all; e += size) {
    const int a = a0 + (int)(e / ((int64_t)nb * nc)), b = b0 + (int)(e / nc % nb), c = c0 + (int)(e % nc);
    // the distance to the brick's box, a hair wider than its centres' box
    const double lx = g.x0 + a * edge, ly = g.y0 + b * edge, lz = g.z0 + c * edge;
    const double gx = fmax(fmax(lx - x, x - (lx + edge)), 0.0);
    const double gy = fmax(fmax(ly - y, y - (ly + edge)), 0.0);
    const double gz = fmax(fmax(lz - z, z - (lz + edge)), 0.0);
    if (gx * gx + gy * gy + gz * gz < reach2) f(((int64_t)a * g.bricks + b) * g.bricks + c);
  }
}

// sums over the threads of a group (a warp or the block), the same on every thread
template <int GROUP>
__device__ __forceinline__ double group_sum(double v, double* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if constexpr (GROUP > 32) {
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    v = 0.0;
#pragma unroll
    for (int w = 0; w < GROUP / 32; ++w) v += red[w];
  }
  return v;
}

template <int GROUP>
__global__ void __launch_bounds__(NB_THREADS) k_box_weights(
    int64_t n, const double* __restrict__ x, const double* __restrict__ h,
    const double* __restrict__ m, const double* __restrict__ t, const double* __restrict__ v,
    BoxGeom g, int kid, const int32_t* __restrict__ list,
    const unsigned long long* __restrict__ nlist, double* __restrict__ rec,
    unsigned long long* __restrict__ brick_count, double* __restrict__ acc, double* outside_sum,
    unsigned long long* n_tri) {
  __shared__ double red[NB_THREADS / 32];
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, rank = threadIdx.x % GROUP;
  const int64_t groups = (int64_t)gridDim.x * (NB_THREADS / GROUP);
  const int64_t count = (int64_t)nlist[GROUP > 32 ? 1 : 0];
  const double dx = g.dx;
  double out_all = 0.0;
  for (int64_t item = blockIdx.x * (int64_t)(NB_THREADS / GROUP) + threadIdx.x / GROUP;
       item < count; item += groups) {
    const int64_t slot = GROUP > 32 ? n - 1 - item : item;
    const int64_t p = list[slot];
    const double xp = x[3 * p], yp = x[3 * p + 1], zp = x[3 * p + 2];
    const double hp = h[p], big = 2.0 * hp, big2 = big * big, ih = 1.0 / hp;
    const BoxRange r = box_range(g, xp, yp, zp, big);
    const int64_t nbb = (int64_t)r.b1 - r.b0 + 1, ncc = (int64_t)r.c1 - r.c0 + 1;
    const int64_t plane = nbb > 0 && ncc > 0 ? nbb * ncc : 0;
    double w_in = 0.0, w_out = 0.0;
    bool eight = box_holds_eight(xp, yp, zp, big, dx);
    if (eight) {
      // columns of the support along x, one (b, c) per thread; lane l of a warp keeps the x
      // distance of plane a + l, so a centre costs one fused operation before its weight
      for (int64_t e0 = rank - lane; e0 < plane; e0 += GROUP) {
        const int64_t e = e0 + lane;
        // (a warp's support has less than BOX_WIDE cells: 32-bit quotients)
        const int64_t eb = GROUP > 32 ? e / ncc : (int64_t)((unsigned)e / (unsigned)ncc);
        const int b = (int)(r.b0 + eb), c = (int)(r.c0 + (e - eb * ncc));
        const double dy = g.y0 + (b + 0.5) * dx - yp, dz = g.z0 + (c + 0.5) * dx - zp;
        const double yz2 = e < plane ? box_yz2(dy, dz) : INFINITY;
        const bool in_bc = b >= 0 && b < g.nb && c >= 0 && c < g.nb;
        if (!__any_sync(FULL, yz2 < big2)) continue;
        double s_in = 0.0, s_all = 0.0;
        for (int64_t a32 = r.a0; a32 <= r.a1; a32 += 32) {
          const double da = g.x0 + ((double)(a32 + lane) + 0.5) * dx - xp;
          const int na = (int)min((int64_t)32, (int64_t)r.a1 - a32 + 1);
          for (int k = 0; k < na; ++k) {
            const double dd = box_d2(__shfl_sync(FULL, da, k), yz2);
            if (dd < big2) {
              const double f = kernel_f<double>(sqrt(dd) * ih, kid);
              s_all += f;
              if (a32 + k >= 0 && a32 + k < g.nb) s_in += f;
            }
          }
        }
        if (in_bc) {
          w_in += s_in;
          w_out += s_all - s_in;
        } else {
          w_out += s_all;
        }
      }
    } else {
      // a support of a few cells: the reference's own test decides each centre, since their
      // number chooses between the kernel's weights and the trilinear ones
      const double in2 = big2 * (1.0 - 1e-12), out2 = big2 * (1.0 + 1e-12);
      double n_in = 0.0;
      for (int64_t a = r.a0; a <= r.a1; ++a) {
        const double dxc = g.x0 + (a + 0.5) * dx - xp;
        for (int64_t e = rank; e < plane; e += GROUP) {
          const int b = r.b0 + (int)(e / ncc), c = r.c0 + (int)(e % ncc);
          const double dyc = g.y0 + (b + 0.5) * dx - yp, dzc = g.z0 + (c + 0.5) * dx - zp;
          const double dd = dxc * dxc + dyc * dyc + dzc * dzc;
          if (dd < in2 || (dd < out2 && sqrt(dd) / hp < 2.0)) n_in += 1.0;
          const double df = box_d2(dxc, box_yz2(dyc, dzc));
          if (!(df < big2)) continue;
          const double f = kernel_f<double>(sqrt(df) * ih, kid);
          if (a >= 0 && a < g.nb && b >= 0 && b < g.nb && c >= 0 && c < g.nb)
            w_in += f;
          else
            w_out += f;
        }
      }
      eight = group_sum<GROUP>(n_in, red) >= (double)DEP_MIN_CELLS;
    }
    w_in = group_sum<GROUP>(w_in, red);
    w_out = group_sum<GROUP>(w_out, red);
    double vals[DEP_FIELDS];
    particle_vals(p, m, t, v, vals);
    if (!eight || !(w_in + w_out > 0.0)) {
      // trilinear weights over the eight nearest centres, one per lane (also, uncounted, where every
      // centre is a rounding from the edge and has no weight)
      if (rank == 0 && !eight) atomicAdd(n_tri, 1ull);
      const double fa = (xp - g.x0) / dx - 0.5, fb = (yp - g.y0) / dx - 0.5,
                   fc = (zp - g.z0) / dx - 0.5;
      const int ia = (int)floor(fa), ib = (int)floor(fb), ic = (int)floor(fc);
      const double ta = fa - ia, tb = fb - ib, tc = fc - ic;
      if (rank < 8) {
        const int da = rank >> 2, db = (rank >> 1) & 1, dc = rank & 1;
        const double w = (da ? ta : 1.0 - ta) * (db ? tb : 1.0 - tb) * (dc ? tc : 1.0 - tc);
        const int64_t a = (int64_t)ia + da, b = (int64_t)ib + db, c = (int64_t)ic + dc;
        if (0 <= a && a < g.nb && 0 <= b && b < g.nb && 0 <= c && c < g.nb)
          add_cell(acc, (a * g.nb + b) * g.nb + c, w, vals);
        else
          out_all += w * vals[0];
      }
      if (rank == 0) rec[BOX_REC * slot + 3] = -1.0;  // nothing for the bricks
      continue;
    }
    const double inv = 1.0 / (w_in + w_out);
    if (rank == 0 && w_out != 0.0) out_all += w_out * inv * vals[0];
    if (rank < BOX_REC) {
      const double head[6] = {xp, yp, zp, hp, ih, 0.0};
      double val = 0.0;
#pragma unroll
      for (int f = 0; f < 6; ++f) {
        if (rank == f) val = head[f];
        if (rank == 6 + f) val = vals[f] * inv;
      }
      rec[BOX_REC * slot + rank] = val;
    }
    for_bricks(g, xp, yp, zp, big, rank, GROUP,
               [&](int64_t brick) { atomicAdd(brick_count + brick, 1ull); });
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) out_all += __shfl_xor_sync(FULL, out_all, o);
  if (lane == 0 && out_all != 0.0) atomicAdd(outside_sum, out_all);
}

// the bricks' stretches of BRICK_CHUNK list entries, as (brick, first entry) tasks
__global__ void k_box_tasks(int64_t nbricks, const unsigned long long* __restrict__ count,
                            unsigned* __restrict__ cursor, int2* __restrict__ tasks,
                            unsigned long long* __restrict__ ntasks) {
  const int64_t b = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (b >= nbricks) return;
  cursor[b] = 0;
  const unsigned c = (unsigned)count[b];  // at most one entry per particle
  if (c == 0) return;
  const unsigned nt = (c + BRICK_CHUNK - 1) / BRICK_CHUNK;
  const unsigned long long at = atomicAdd(ntasks, (unsigned long long)nt);
  for (unsigned k = 0; k < nt; ++k) tasks[at + k] = make_int2((int)b, (int)k);
}

// the work list's entries [w0, w1): counted per brick (a part of the list), or put in its list
template <bool FILL>
__global__ void __launch_bounds__(NB_THREADS) k_box_lists(
    int64_t n, BoxGeom g, int64_t w0, int64_t w1, const unsigned long long* __restrict__ nlist,
    const double* __restrict__ rec, unsigned long long* __restrict__ count,
    const int64_t* __restrict__ brick_off, unsigned* __restrict__ cursor, int32_t* __restrict__ pairs) {
  const int lane = threadIdx.x & 31;
  const int64_t small = (int64_t)nlist[0], all = min(small + (int64_t)nlist[1], w1);
  for (int64_t w = w0 + ((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5); w < all;
       w += ((int64_t)gridDim.x * blockDim.x) >> 5) {
    const int64_t slot = w < small ? w : n - 1 - (w - small);
    const double* r = rec + BOX_REC * slot;
    if (r[3] < 0.0) continue;  // trilinear
    for_bricks(g, r[0], r[1], r[2], 2.0 * r[3], lane, 32, [&](int64_t brick) {
      if (FILL)
        pairs[brick_off[brick] + atomicAdd(cursor + brick, 1u)] = (int32_t)slot;
      else
        atomicAdd(count + brick, 1ull);
    });
  }
}

__global__ void __launch_bounds__(BRICK_WARPS * 32, 2) k_box_bricks(
    BoxGeom g, int kid, const double* __restrict__ rec, const unsigned long long* __restrict__ count,
    const int64_t* __restrict__ brick_off, const int32_t* __restrict__ pairs,
    const int2* __restrict__ tasks, const unsigned long long* __restrict__ ntasks,
    double* __restrict__ acc) {
  __shared__ __align__(16) double stage[BRICK_STAGE][BOX_REC];
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // sub-brick of the warp: 4 x 2 x 2 of them, each of 2 x 4 x 4 cells
  const int sa = (warp >> 2) * 2, sb = ((warp >> 1) & 1) * 4, sc = (warp & 1) * 4;
  const int64_t total = (int64_t)*ntasks;
  for (int64_t task = blockIdx.x; task < total; task += gridDim.x) {
    const int2 tk = tasks[task];
    const int64_t brick = tk.x;
    const int ba = (int)(brick / ((int64_t)g.bricks * g.bricks)) * BRICK;
    const int bb = (int)(brick / g.bricks % g.bricks) * BRICK;
    const int bc = (int)(brick % g.bricks) * BRICK;
    const unsigned cnt = (unsigned)count[brick];
    const unsigned first = (unsigned)tk.y * BRICK_CHUNK;
    const unsigned last = min(cnt, first + BRICK_CHUNK);
    const int32_t* list = pairs + brick_off[brick];
    // the lane's cell and the box of the warp's centres
    const int a = ba + sa + (lane >> 4), b = bb + sb + ((lane >> 2) & 3), c = bc + sc + (lane & 3);
    const double cx = g.x0 + (a + 0.5) * g.dx, cy = g.y0 + (b + 0.5) * g.dx,
                 cz = g.z0 + (c + 0.5) * g.dx;
    const double lx = g.x0 + (ba + sa + 0.5) * g.dx, ly = g.y0 + (bb + sb + 0.5) * g.dx,
                 lz = g.z0 + (bc + sc + 0.5) * g.dx;
    const double hx = lx + g.dx, hy = ly + 3.0 * g.dx, hz = lz + 3.0 * g.dx;
    double s[DEP_FIELDS] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    for (unsigned at = first; at < last; at += BRICK_STAGE) {
      const int nst = (int)min(last - at, (unsigned)BRICK_STAGE);
      __syncthreads();
      for (int e = threadIdx.x; e < nst * (BOX_REC / 2); e += BRICK_WARPS * 32) {
        const int k = e / (BOX_REC / 2), f = e % (BOX_REC / 2);
        reinterpret_cast<double2*>(stage[k])[f] =
            reinterpret_cast<const double2*>(rec + BOX_REC * (int64_t)list[at + k])[f];
      }
      __syncthreads();
      for (int k0 = 0; k0 < nst; k0 += 32) {
        // the records whose supports reach the warp's centres, one record per lane
        bool reach = false;
        if (k0 + lane < nst) {
          const double* q = stage[k0 + lane];
          const double gx = fmax(fmax(lx - q[0], q[0] - hx), 0.0);
          const double gy = fmax(fmax(ly - q[1], q[1] - hy), 0.0);
          const double gz = fmax(fmax(lz - q[2], q[2] - hz), 0.0);
          const double big = 2.0 * q[3];
          reach = gx * gx + gy * gy + gz * gz < big * big * (1.0 + 1e-9);
        }
        for (unsigned mk = __ballot_sync(FULL, reach); mk; mk &= mk - 1) {
          const double* q = stage[k0 + __ffs(mk) - 1];
          const double ddx = cx - q[0], ddy = cy - q[1], ddz = cz - q[2];
          const double dd = box_d2(ddx, box_yz2(ddy, ddz));
          const double big = 2.0 * q[3];
          if (dd < big * big) {
            const double w = kernel_f<double>(sqrt(dd) * q[4], kid);
#pragma unroll
            for (int f = 0; f < DEP_FIELDS; ++f) s[f] = fma(w, q[6 + f], s[f]);
          }
        }
      }
    }
    if (a < g.nb && b < g.nb && c < g.nb) {
      double* o = acc + (((int64_t)a * g.nb + b) * g.nb + c) * DEP_FIELDS;
#pragma unroll
      for (int f = 0; f < DEP_FIELDS; ++f)
        if (s[f] != 0.0) atomicAdd(o + f, s[f]);
    }
  }
}

// the bricks' counts; the four work counters, the mass outside and the trilinear count with the first
__global__ void k_box_zero(int64_t nbricks, unsigned long long* __restrict__ count,
                           int64_t* __restrict__ brick_off, unsigned long long* __restrict__ counters,
                           double* __restrict__ outside, unsigned long long* __restrict__ n_tri) {
  const int64_t b = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (b < nbricks) count[b] = 0;
  if (b == 0) {
    brick_off[0] = 0;
    if (outside) {
      for (int k = 0; k < 4; ++k) counters[k] = 0;
      *outside = 0.0;
      *n_tri = 0;
    }
  }
}

// acc is zeroed by the caller; the mass outside and the number of trilinear particles come back with
// the lists' length, so a call whose particles reach no cell by the kernel waits once (a thousand
// supports of 0.2 cells into 32^3: 0.146 ms, 0.163 with a wait of their own and four clears).
// The context's buffers are free again on return.
int deposit_box(Engine& E, int64_t n, const double* x, const double* h, const double* m,
                const double* t, const double* v, double x0, double y0, double z0, double dx,
                int nb, int kid, double* acc, double* outside_out, int64_t* n_tri_out,
                cudaStream_t st) {
  *outside_out = 0.0;
  *n_tri_out = 0;
  if (n <= 0) return 0;
  BoxGeom g{x0, y0, z0, dx, nb, (nb + BRICK - 1) / BRICK};
  const int64_t nbricks = (int64_t)g.bricks * g.bricks * g.bricks;
  Workspace& W = E.ws;
  NB_TRY(W.ensure(E, std::max<int64_t>(W.cap, 1024)));
  NB_TRY(E.ensure_deposit(n));
  NB_TRY(E.ensure_bricks(nbricks));
  int sms = 0;
  NB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, E.device));
  double* outside = W.d_scal;
  unsigned long long* n_tri = reinterpret_cast<unsigned long long*>(W.d_i64);
  // small and wide particles listed, and the tasks
  unsigned long long* counters = reinterpret_cast<unsigned long long*>(E.dep_count);
  unsigned long long* bcount = E.brick_count;
  count_launch(), k_box_zero<<<grid_for(nbricks), NB_THREADS, 0, st>>>(nbricks, bcount, E.brick_off, counters, outside, n_tri);
  count_launch(), k_box_classify<<<grid_for(n), NB_THREADS, 0, st>>>(n, x, h, m, g, E.dep_i0, counters, outside);
  const unsigned warps = (unsigned)std::min<int64_t>(grid_for(n * 32), (int64_t)sms * 8);
  count_launch(), k_box_weights<32><<<warps, NB_THREADS, 0, st>>>(
      n, x, h, m, t, v, g, kid, E.dep_i0, counters, E.dep_buf, bcount, acc, outside, n_tri);
  count_launch(), k_box_weights<NB_THREADS><<<(unsigned)std::min<int64_t>(n, (int64_t)sms * 4), NB_THREADS, 0, st>>>(
      n, x, h, m, t, v, g, kid, E.dep_i0, counters, E.dep_buf, bcount, acc, outside, n_tri);
  NB_CUDA(cudaMemcpyAsync(W.h_dbl, outside, sizeof(double), cudaMemcpyDeviceToHost, st));
  NB_CUDA(cudaMemcpyAsync(W.h_i64, n_tri, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
  size_t tmp = 0;
  NB_CUDA(cub::DeviceScan::InclusiveSum(nullptr, tmp, reinterpret_cast<int64_t*>(bcount),
                                        E.brick_off + 1, (int)nbricks, st));
  NB_TRY(E.ensure_cub(tmp));
  // the bricks' offsets from their counts, and the number of pairs on the host
  auto offsets = [&](int64_t* pairs) -> int {
    tmp = E.cub_bytes;
    NB_CUDA(cub::DeviceScan::InclusiveSum(E.cub_tmp, tmp, reinterpret_cast<int64_t*>(bcount),
                                          E.brick_off + 1, (int)nbricks, st));
    NB_CUDA(cudaMemcpyAsync(E.h_build, E.brick_off + nbricks, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
    NB_CUDA(host_sync(st));
    *pairs = E.h_build[0];
    return 0;
  };
  // the lists of the entries [w0, w1) and their bricks' sums
  auto gather = [&](int64_t pairs, int64_t w0, int64_t w1) -> int {
    if (pairs == 0) return 0;
    NB_TRY(E.ensure_brick_lists(pairs, pairs / BRICK_CHUNK + nbricks));
    count_launch(), k_box_tasks<<<grid_for(nbricks), NB_THREADS, 0, st>>>(nbricks, bcount, E.brick_cursor,
                                                                           E.brick_tasks, counters + 2);
    count_launch(), k_box_lists<true><<<warps, NB_THREADS, 0, st>>>(
        n, g, w0, w1, counters, E.dep_buf, bcount, E.brick_off, E.brick_cursor, E.brick_pairs);
    count_launch(), k_box_bricks<<<(unsigned)(sms * 2), BRICK_WARPS * 32, 0, st>>>(
        g, kid, E.dep_buf, bcount, E.brick_off, E.brick_pairs, E.brick_tasks, counters + 2, acc);
    return 0;
  };
  int64_t pairs = 0;
  NB_TRY(offsets(&pairs));
  *outside_out = W.h_dbl[0];
  *n_tri_out = W.h_i64[0];
  if (pairs == 0) return 0;
  if (pairs <= BOX_PAIRS) {
    NB_TRY(gather(pairs, 0, n));
    NB_CUDA(host_sync(st));
    return 0;
  }
  // Wide supports reach so many bricks that their lists would take gigabytes: part of the work list
  // at a time, of twice the mean's room; one that still does not fit is halved, down to the length
  // that fits whatever it holds.
  NB_CUDA(cudaMemcpyAsync(E.h_build, counters, 2 * sizeof(int64_t), cudaMemcpyDeviceToHost, st));
  NB_CUDA(host_sync(st));
  const int64_t all = E.h_build[0] + E.h_build[1];
  const int64_t least = std::max<int64_t>(BOX_PAIRS / nbricks, 1);
  int64_t part = std::max<int64_t>(least, (int64_t)((double)all * BOX_PAIRS / (2.0 * pairs)));
  for (int64_t w = 0; w < all;) {
    const int64_t end = std::min(all, w + part);
    count_launch(), k_box_zero<<<grid_for(nbricks), NB_THREADS, 0, st>>>(nbricks, bcount, E.brick_off, nullptr, nullptr, nullptr);
    count_launch(), k_box_lists<false><<<warps, NB_THREADS, 0, st>>>(
        n, g, w, end, counters, E.dep_buf, bcount, E.brick_off, E.brick_cursor, nullptr);
    NB_TRY(offsets(&pairs));
    if (pairs > BOX_PAIRS && part > least) {
      part = std::max(least, part / 2);
      continue;
    }
    NB_CUDA(cudaMemsetAsync(counters + 2, 0, sizeof(unsigned long long), st));
    NB_TRY(gather(pairs, w, end));
    w = end;
  }
  NB_CUDA(host_sync(st));
  return 0;
}

// render/gasgrid.py:293-313 (_finish): mass, rho = M / V, mass-weighted T, (sum m T^4 /
// sum m)^(1/4), mass-weighted v; empty cells 0.  vol[cell / per] is the cell's volume.
__global__ void k_grid_finish(int64_t ncell, const double* __restrict__ acc,
                              const double* __restrict__ vol, int64_t per, double* mass,
                              float* rho, float* t_mass, float* t_em, float* vel) {
  const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (c >= ncell) return;
  const double* a = acc + c * DEP_FIELDS;
  const double mc = a[0];
  const bool has = mc > 0.0;
  const double safe = has ? mc : 1.0;
  mass[c] = mc;
  rho[c] = (float)(mc / vol[c / per]);
  t_mass[c] = (float)(has ? a[1] / safe : 0.0);
  const double t4 = a[2] / safe;
  t_em[c] = (float)(has ? sqrt(sqrt(t4 > 0.0 ? t4 : 0.0)) : 0.0);
#pragma unroll
  for (int d = 0; d < 3; ++d) vel[3 * c + d] = (float)(has ? a[3 + d] / safe : 0.0);
}

// render/gasgrid.py:757-788 (refine_sums): fine sums from the coarse sums' densities,
// trilinear in index space (theta and r clamped, phi periodic), times the fine volume
__device__ __forceinline__ void refine_axis(int i, int c, int nc, bool periodic, int& i0,
                                            int& i1, double& w) {
  double f = (i + 0.5) / c - 0.5;
  if (periodic) {
    const int b = (int)floor(f);
    i0 = py_imod(b, nc);
    i1 = py_imod(b + 1, nc);
    w = f - b;
    return;
  }
  f = fmin(fmax(f, 0.0), nc - 1.0);
  int b = 0;
  if (nc > 1) b = min((int)floor(f), nc - 2);
  i0 = b;
  i1 = min(b + 1, nc - 1);
  w = f - b;
}

__global__ void k_refine(const double* __restrict__ acc_c, const double* __restrict__ vc,
                         int nrc, int nthc, int nphc, const double* __restrict__ vf, int nr,
                         int nth, int nph, int cr, int ct, int cp, double* __restrict__ out) {
  const int64_t cell = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (cell >= (int64_t)nr * nth * nph) return;
  const int k = (int)(cell % nph);
  const int j = (int)((cell / nph) % nth);
  const int i = (int)(cell / ((int64_t)nph * nth));
  int ri[2], ti[2], pi[2];
  double rw, tw, pw;
  refine_axis(i, cr, nrc, false, ri[0], ri[1], rw);
  refine_axis(j, ct, nthc, false, ti[0], ti[1], tw);
  refine_axis(k, cp, nphc, true, pi[0], pi[1], pw);
  const double wr[2] = {1.0 - rw, rw}, wt[2] = {1.0 - tw, tw}, wp[2] = {1.0 - pw, pw};
  double s[DEP_FIELDS] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  for (int a = 0; a < 2; ++a)
    for (int b = 0; b < 2; ++b)
      for (int c = 0; c < 2; ++c) {
        const double w = wr[a] * wt[b] * wp[c];
        const int64_t cc = ((int64_t)ri[a] * nthc + ti[b]) * nphc + pi[c];
        const double vcc = vc[(int64_t)ri[a] * nthc + ti[b]];
#pragma unroll
        for (int f = 0; f < DEP_FIELDS; ++f) s[f] += w * (acc_c[cc * DEP_FIELDS + f] / vcc);
      }
  const double vfc = vf[(int64_t)i * nth + j];
#pragma unroll
  for (int f = 0; f < DEP_FIELDS; ++f) out[cell * DEP_FIELDS + f] = s[f] * vfc;
}

// the sum of the first field (mass), one add per warp of a grid-stride pass
__global__ void k_field_sum(int64_t ncell, const double* __restrict__ acc, double* sum) {
  double v = 0.0;
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < ncell;
       c += (int64_t)gridDim.x * blockDim.x)
    v += acc[c * DEP_FIELDS];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(sum, v);
}

__global__ void k_refine_scale(int64_t nval, const double* __restrict__ sums, double* out) {
  const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (e >= nval) return;
  const double fine = sums[0], coarse = sums[1];
  if (fine > 0.0) out[e] *= coarse / fine;
}

// ---------------------------------------------------------------- spatial order
// The particles are dealt to the deposition threads in the order of the cell holding their
// centre, so neighbouring threads add to neighbouring cells while those lines sit in L2 (in the
// caller's order each atomic add of a large grid travels to DRAM).  Keys: the grid's own linear
// cell index, with the out-of-grid cells clamped to one layer beyond each face.
// With wide_cells > 0 the particles whose support spans that many fine angular cells or more
// (render/gasgrid.py:751-754) come last, and are counted.
__global__ void k_dep_keys_log(int64_t n, const double* __restrict__ x,
                               const double* __restrict__ h, LogGeom g, double wide_cells,
                               unsigned long long* keys, int32_t* idx,
                               unsigned long long* __restrict__ n_wide) {
  const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  bool wide = false;
  if (p < n) {
    const double xp = x[3 * p], yp = x[3 * p + 1], zp = x[3 * p + 2];
    const double rr = sqrt(xp * xp + yp * yp + zp * zp);
    const int i = min(max((int)floor(log(rr / g.r_min) / g.dlnr), -1), g.nr) + 1;
    const int j = min(max((int)floor(acos(fmin(1.0, fmax(-1.0, zp / rr))) / g.dth), 0), g.nth - 1);
    const int k = min(max((int)floor(azimuth(yp, xp) / g.dph), 0), g.nph - 1);
    wide = wide_cells > 0.0 && 2.0 * h[p] >= wide_cells * fmax(rr, g.r_min) * g.dth;
    const unsigned long long cells = (unsigned long long)(g.nr + 2) * g.nth * g.nph;
    keys[p] = wide ? cells : ((unsigned long long)i * g.nth + j) * g.nph + k;
    idx[p] = (int32_t)p;
  }
  const unsigned w = __ballot_sync(0xffffffffu, wide);
  if (w && (threadIdx.x & 31) == 0) atomicAdd(n_wide, (unsigned long long)__popc(w));
}

__global__ void k_dep_gather(int64_t n, const int32_t* __restrict__ idx,
                             const double* __restrict__ x, const double* __restrict__ h,
                             const double* __restrict__ m, const double* __restrict__ t,
                             const double* __restrict__ v, double* __restrict__ out) {
  const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (q >= n) return;
  const int64_t p = idx[q];
  double* xs = out;
  double* hs = out + 3 * n;
  double* ms = hs + n;
  double* ts = ms + n;
  double* vs = ts + n;
  for (int c = 0; c < 3; ++c) {
    xs[3 * q + c] = x[3 * p + c];
    vs[3 * q + c] = v[3 * p + c];
  }
  hs[q] = h[p];
  ms[q] = m[p];
  ts[q] = t[p];
}

// Inputs of this size on, and those split over two grids, are deposited in the spatial order of
// their centres' cells (sorted keys, gathered copies of the particle data).
constexpr int64_t DEPOSIT_SORT_MIN = 1 << 16;

size_t deposit_cub_bytes(int64_t n) {
  size_t b = 0;
  cub::DeviceRadixSort::SortPairs((void*)nullptr, b, (unsigned long long*)nullptr,
                                  (unsigned long long*)nullptr, (int32_t*)nullptr,
                                  (int32_t*)nullptr, (int)n);
  return b;
}

void launch_log_tables(const LogGeom& g, double* out, cudaStream_t st) {
  const int64_t most = std::max<int64_t>(std::max<int64_t>(g.nph, g.nth), (int64_t)g.nr * g.nth);
  count_launch(), k_log_tables<<<grid_for(most), NB_THREADS, 0, st>>>(g, out);
}

// scal: device doubles, the mass outside of each grid; ints: device words, the trilinear counts of
// each grid, the number of wide particles and one for the walk; all and the sums zeroed by the caller
int deposit_log(Engine& E, int64_t n, const double* x, const double* h, const double* m,
                const double* t, const double* v, const LogGeom& fine, const LogGeom* coarse,
                double wide_cells, int kid, double* acc, double* acc_c, double* scal,
                unsigned long long* ints, cudaStream_t st) {
  if (n <= 0) return 0;
  NB_TRY(E.ensure_deposit(n));
  const int nsh = fine.nr + DEP_INNER_VIRTUAL, nsh_c = coarse ? coarse->nr + DEP_INNER_VIRTUAL : 0;
  NB_TRY(E.ensure_shells(nsh + nsh_c));
  double2* shells = static_cast<double2*>(E.dep_shells);
  count_launch(), k_log_shells<<<grid_for(nsh), NB_THREADS, 0, st>>>(fine, shells);
  if (coarse) count_launch(), k_log_shells<<<grid_for(nsh_c), NB_THREADS, 0, st>>>(*coarse, shells + nsh);
  if (coarse || n >= DEPOSIT_SORT_MIN) {
    count_launch(), k_dep_keys_log<<<grid_for(n), NB_THREADS, 0, st>>>(
        n, x, h, fine, coarse ? wide_cells : 0.0, E.dep_k0, E.dep_i0, ints + 2);
    const unsigned long long max_key = (unsigned long long)(fine.nr + 2) * fine.nth * fine.nph;
    int bits = 1;
    while (bits < 64 && (1ull << bits) <= max_key) ++bits;
    cub::DoubleBuffer<unsigned long long> kb(E.dep_k0, E.dep_k1);
    cub::DoubleBuffer<int32_t> vb(E.dep_i0, E.dep_i1);
    size_t tmp = E.cub_bytes;
    NB_CUDA(cub::DeviceRadixSort::SortPairs(E.cub_tmp, tmp, kb, vb, (int)n, 0, bits, st));
    count_launch(), k_dep_gather<<<grid_for(n), NB_THREADS, 0, st>>>(n, vb.Current(), x, h, m, t, v, E.dep_buf);
    x = E.dep_buf;
    h = E.dep_buf + 3 * n;
    m = h + n;
    t = m + n;
    v = t + n;
  }
  const LogTarget a{fine, shells, acc, scal, ints};
  const LogTarget b = coarse ? LogTarget{*coarse, shells + nsh, acc_c, scal + 1, ints + 1} : a;
  int sms = 0;
  NB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, E.device));
  const unsigned long long* n_wide = coarse ? ints + 2 : nullptr;
  unsigned long long* nlist = ints + 3;
  int32_t* list = reinterpret_cast<int32_t*>(E.dep_k0);  // the sort's keys are done with
  count_launch(), k_deposit_log<<<grid_for(n, 128), 128, 0, st>>>(n, n_wide, x, h, m, t, v, a, b,
                                                                    kid, list, nlist);
  const unsigned gb = (unsigned)std::min<int64_t>(grid_for(n * 32, 128), (int64_t)sms * LOG_B);
  count_launch(), k_deposit_log_heavy<<<gb, 128, 0, st>>>(n, n_wide, x, h, m, t, v, a, b, kid, list,
                                                          nlist);
  return 0;
}

// ---------------------------------------------------------------- launchers
void launch_grid_finish(int64_t ncell, const double* acc, const double* vol, int64_t per,
                        double* mass, float* rho, float* t_mass, float* t_em, float* vel,
                        cudaStream_t st) {
  if (ncell > 0)
    count_launch(), k_grid_finish<<<grid_for(ncell), NB_THREADS, 0, st>>>(
        ncell, acc, vol, per, mass, rho, t_mass, t_em, vel);
}

void launch_refine_sums(const double* acc_c, const double* vol_c, int nrc, int nthc, int nphc,
                        const double* vol_f, int nr, int nth, int nph, int cr, int ct, int cp,
                        double* out, double* sums2, cudaStream_t st) {
  const int64_t nf = (int64_t)nr * nth * nph, nc = (int64_t)nrc * nthc * nphc;
  count_launch(), k_refine<<<grid_for(nf), NB_THREADS, 0, st>>>(
      acc_c, vol_c, nrc, nthc, nphc, vol_f, nr, nth, nph, cr, ct, cp, out);
  count_launch(), k_field_sum<<<std::min(grid_for(nf), 1184u), NB_THREADS, 0, st>>>(nf, out, sums2);
  count_launch(), k_field_sum<<<std::min(grid_for(nc), 1184u), NB_THREADS, 0, st>>>(nc, acc_c, sums2 + 1);
  count_launch(), k_refine_scale<<<grid_for(nf * DEP_FIELDS), NB_THREADS, 0, st>>>(
      nf * DEP_FIELDS, sums2, out);
}

}  // namespace nbk
