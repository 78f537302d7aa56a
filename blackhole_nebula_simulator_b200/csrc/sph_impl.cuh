// SPH pair passes on neighbour lists (implementation, included by sph64.cu and sph32.cu): the h-rho Newton solve and the fused pressure + artificial
// viscosity (+ conductivity, + disc viscosity) force and du/dt pass.
//
// The density solve runs 8 lanes per row (FP64: 8 or 32, see launch_density64) with a shared-memory
// cache of the inner entries; the force pass eight lanes per row.  Both walk CSR lists.  They are
// templated on the list index type so the same code serves the caller-order int64 lists of the
// operator API and the engine's sorted int32 lists.  The FP64 kernels form every pair term in double;
// the FP32 ones take positions as float offsets from cell centres, float pair terms and
// Kahan-compensated sums, with the Newton update and all per-particle state in double.
#pragma once
#include "common.cuh"
#include "engine.cuh"
#include "sph.cuh"

namespace nbk {

// ---------------------------------------------------------------- position differences
// FP64 density: packed (x, y, z, mass) doubles.
struct Pos64 {
  const double4* p;
  struct Own {
    double4 a;
  };
  __device__ __forceinline__ Own own(int64_t i) const { return Own{p[i]}; }
  // the difference x_j - x_i and particle j's mass (the record's w)
  __device__ __forceinline__ void diff_m(const Own& o, int64_t j, double& dx, double& dy,
                                         double& dz, double& m) const {
    const double4 b = ld_rec(p + j);
    dx = b.x - o.a.x;
    dy = b.y - o.a.y;
    dz = b.z - o.a.z;
    m = b.w;
  }
};

// FP32: per particle the cell of a uniform grid of edge `cell` (at most 1024 per axis) and the
// float offset from that cell's centre, packed as two float4: (offset x, y, z, mass) and (cell
// x, y, z as exact small floats, h: the smoothing length where the force pass needs it).  dx = (c_j - c_i) cell + (o_j - o_i): the cell difference
// is an exact float, and one fused multiply-add rounds the sum once, so the difference keeps full
// float precision at any distance from the origin.
struct Pos32 {
  const float4* p;
  float cell;
  const double* box6 = nullptr;  // grid corner and far corner; the edge is derived on the device
  struct Own {
    float4 a, c;
  };
  // edge of the grid cells: the largest side of the box over 1000, as the packing kernel uses
  __device__ __forceinline__ void ready() {
    if (box6) {
      double span = fmax(fmax(box6[3] - box6[0], box6[4] - box6[1]), box6[5] - box6[2]);
      cell = (float)fmax(span / 1000.0, 1e-30);
    }
  }
  __device__ __forceinline__ Own own(int64_t i) const { return Own{p[2 * i], p[2 * i + 1]}; }
  // the difference and particle j's mass, in one load
  __device__ __forceinline__ void diff_m(const Own& o, int64_t j, float& dx, float& dy, float& dz,
                                         float& m) const {
    float4 b, cb;
    ld_rec(p + 2 * j, b, cb);
    dx = fmaf(cb.x - o.c.x, cell, b.x - o.a.x);
    dy = fmaf(cb.y - o.c.y, cell, b.y - o.a.y);
    dz = fmaf(cb.z - o.c.z, cell, b.z - o.a.z);
    m = b.w;
  }
  __device__ __forceinline__ void diff(const Own& o, int64_t j, float& dx, float& dy,
                                       float& dz) const {
    const float4 b = p[2 * j], cb = p[2 * j + 1];
    dx = fmaf(cb.x - o.c.x, cell, b.x - o.a.x);
    dy = fmaf(cb.y - o.c.y, cell, b.y - o.a.y);
    dz = fmaf(cb.z - o.c.z, cell, b.z - o.a.z);
  }
  __device__ __forceinline__ void diff(int64_t i, int64_t j, float& dx, float& dy,
                                       float& dz) const {
    diff(own(i), j, dx, dy, dz);
  }
  // the difference and particle j's smoothing length, from the same record
  __device__ __forceinline__ void diff_h(const Own& o, int64_t j, float& dx, float& dy, float& dz,
                                         float& hj) const {
    float4 b, cb;
    ld_rec(p + 2 * j, b, cb);
    dx = fmaf(cb.x - o.c.x, cell, b.x - o.a.x);
    dy = fmaf(cb.y - o.c.y, cell, b.y - o.a.y);
    dz = fmaf(cb.z - o.c.z, cell, b.z - o.a.z);
    hj = cb.w;
  }
};

__device__ __forceinline__ double sqdist(double dx, double dy, double dz) { return d2_exact(dx, dy, dz); }
__device__ __forceinline__ float sqdist(float dx, float dy, float dz) {
  return fmaf(dz, dz, fmaf(dy, dy, dx * dx));
}

// ---------------------------------------------------------------- density
// Reference sim/sph.py:215-297 (_sums, _distances, _density_kernel): Newton-Raphson on
// f(h) = sum_j m_j W(r_ij, h) - m_i (eta/h)^3 inside a bisection bracket, tol * h0, at most 50
// iterations; the cap test near the search limit; Omega = 1 + h/(3 rho) sum m dW/dh (1 at h_max).

// Sums over the L lanes of a row group (lanes L g .. L g + L - 1 of a warp).  Every lane of the
// group ends with the same value (each butterfly step adds the same two operands on both lanes).
// FP64: plain sums.  FP32: each lane's Kahan partial (s, -c) is combined pairwise with an exact
// two-sum, the rounding errors and the lanes' compensations carried in a second float.
template <int L = 8>
__device__ __forceinline__ double group_total(double v) {
#pragma unroll
  for (int o = L / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double group_total(const Kahan& a) {
  float s = a.s, k = -a.c;
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) {
    float s2 = __shfl_xor_sync(0xffffffffu, s, o);
    float k2 = __shfl_xor_sync(0xffffffffu, k, o);
    float t = __fadd_rn(s, s2);
    float bp = __fsub_rn(t, s);
    float e = __fadd_rn(__fsub_rn(s, __fsub_rn(t, bp)), __fsub_rn(s2, bp));
    s = t;
    k = __fadd_rn(__fadd_rn(k, k2), e);
  }
  return (double)s + (double)k;
}

constexpr int DENSITY_THREADS = 128;  // 16 rows per block
// FP32: entries inside r_in a row keeps in shared memory: 16 rows x 128 x 8 B = 16 KiB per block, so
// 8 resident blocks (the register limit) leave most of the SM's L1 to the gathered records
constexpr int DENSITY_CAP = 128;
// rounds of 8 entries loaded at once by the first walk and by a walk within a sum, and resident
// blocks.  Measured on the 4M torus (launches of the first evaluation, from a guess of h that is
// far off, and of a step's 2.7M rows): 4, 2, 9: 35.8 and 4.05 ms; 4, 2, 8: 38.5 and 4.10; 4, 4, 8:
// 34.7 and 4.59; 3, 3, 8: 40.2 and 4.31; 2, 2, 10: 35.1 and 4.39
constexpr int DENSITY_UNROLL = 4, DENSITY_WALK = 2, DENSITY_BLOCKS = 9;

// FP32 form.  Eight lanes per row, four rows per warp.  The lanes of a row split its list (entry e to
// lane e mod 8, coalesced index loads) and store the squared distance and mass of every entry
// inside r_in = 2.1 h_start (the Newton iterates stay near the start h) in shared memory, in list
// order; each Newton iteration then sums the kernel terms over that cache and reduces across the
// eight lanes, so the lanes of a row take the same Newton steps.  The first sum turns the squares
// into distances.  A sum at an h whose support reaches past r_in adds the entries beyond it from
// the list (the same distances, recomputed); rows with more entries inside r_in than the cache
// holds re-walk their list in every sum.  (The compensated float sums depend on the order of
// their terms in the eighth digit: which lane adds which entry when is part of the result, and so
// are the fused operations of a term, written out below where a rearrangement changed them.)
// Bound by issue (74 % active, about 820 warp instructions per row of a 1M torus step, at half the
// warp slots).  With a square root per list entry, three loads per record, divergent kernel branches
// and conflicting cache rows the two launches above took 51.5 and 5.49 ms.
template <int KID, typename I>
__global__ void __launch_bounds__(DENSITY_THREADS, DENSITY_BLOCKS)
    k_density32(int64_t nrows, const int64_t* __restrict__ rows, Pos32 geo,
              const double* __restrict__ mass, const double* __restrict__ h_start,
              const double* __restrict__ h_search, const int64_t* __restrict__ off,
              const I* __restrict__ idx, DensityParams prm, const int32_t* __restrict__ out_map,
              double* __restrict__ h_out, double* __restrict__ rho, double* __restrict__ omega,
              int64_t* __restrict__ iters, int64_t* __restrict__ flags, int64_t* __restrict__ work) {
  geo.ready();
  // (rows half the banks apart: the four rows of a warp read in two wavefronts)
  __shared__ float2 cache_s[DENSITY_THREADS / 8][DENSITY_CAP + 8];
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, gl = lane & 7, g = lane >> 3;
  const int64_t q = ((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5) * 4 + g;
  const bool live = q < nrows;
  if (!__any_sync(FULL, live)) return;  // warp-uniform
  float2* cache = cache_s[threadIdx.x >> 3];
  int64_t i = 0, e0 = 0;
  unsigned len = 0;
  double m_i = 1.0, hs = 1.0, h = 1.0;
  if (live) {
    i = rows ? rows[q] : q;
    m_i = mass[i];
    hs = fmin(h_search[i], prm.h_max);
    h = fmin(h_start[i], hs);
    e0 = off[i];
    len = (unsigned)(off[i + 1] - e0);
  }
  const I* list = idx + e0;
  const Pos32::Own me_rec = geo.own(i);  // the row's own record, loaded once
  const float r2max = (float)(2.0 * hs * (2.0 * hs));
  const float cn = (float)prm.cnorm;
  // entries inside r_in = 2.1 h are cached, and a sum at h adds the others only when r_in / h < 2
  // (else every one of them has q >= 2, a zero term).  sqrt(d2) < r_in holds for the floats d2
  // below the square of the midpoint of r_in and the float before it (exact in double)
  const float r_in = (float)(2.1 * h);
  const double mid = 0.5 * ((double)r_in + (double)__uint_as_float(__float_as_uint(r_in) - 1u));
  const float d2_in = r_in > 0.0f ? fminf(__double2float_ru(mid * mid), r2max) : 0.0f;
  const unsigned maxlen = __reduce_max_sync(FULL, len);
  int cnt = 0;
  // DENSITY_UNROLL rounds of 8 entries per pass: their index and record loads are issued together
  // (the walk is bound by the latency of those dependent gathers), then the rounds are appended
  // to the cache one after the other
  constexpr int U = DENSITY_UNROLL;
  for (unsigned b = 0; b < maxlen; b += 8 * U) {
    int jj[U];
    float d2[U], mm[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const unsigned e = b + 8 * u + gl;
      jj[u] = e < len ? (int)ld_stream(list + e) : -1;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      d2[u] = INFINITY;
      mm[u] = 0.0f;
      if (jj[u] >= 0) {
        float dx, dy, dz;
        geo.diff_m(me_rec, jj[u], dx, dy, dz, mm[u]);
        d2[u] = sqdist(dx, dy, dz);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const bool inner = d2[u] < d2_in;
      const unsigned seg = (__ballot_sync(FULL, inner) >> (8 * g)) & 0xffu;
      const int pos = cnt + __popc(seg & ((1u << gl) - 1u));
      if (inner && pos < DENSITY_CAP)  // overflow: the walk below instead
        cache[pos] = make_float2(d2[u], mm[u]);
      cnt += __popc(seg);
    }
  }
  __syncwarp();
  const bool cached = cnt <= DENSITY_CAP;
  bool squared = true;
  int evals = 0;
  // kernel sums at h of the rows whose `active` is set; every lane takes part in the reductions
  auto sums = [&](float h, bool active, double& rs_out, double& dws_out) {
    Kahan rs, dws;
    if (active) {
      float inv_h = 1.0f / h;
      float ih2 = inv_h * inv_h;
      float ih3 = ih2 * inv_h;
      float ih4 = ih2 * ih2;
      auto term = [&](float rj, float mj) {
        float qq = rj * inv_h;
        if (qq < 2.0f) {
          evals += 1;
          float fq, df;
          if (KID == 0) {
            // both pieces of the spline, then the one that holds: no divergent branch
            const float t = 2.0f - qq;
            const float f1 = 1.0f - 1.5f * qq * qq + 0.75f * qq * qq * qq;
            const float d1 = fmaf(2.25f * qq, qq, __fmul_rn(-3.0f, qq));
            const float f2 = 0.25f * t * t * t, d2 = -0.75f * t * t;
            fq = qq < 1.0f ? f1 : f2;
            df = qq < 1.0f ? d1 : d2;
          } else {
            fq = kernel_f<float>(qq, 1);
            df = kernel_df<float>(qq, 1);
          }
          rs.add(mj * cn * ih3 * fq);
          dws.add(mj * (-cn * ih4 * fmaf(3.0f, fq, __fmul_rn(qq, df))));
        }
      };
      const bool beyond = cached && !(r_in * inv_h >= 2.0f);
      if (cached) {
        for (int t = gl; t < cnt; t += 8) {
          float2 v = cache[t];
          if (squared) {
            v.x = sqrtf(v.x);
            cache[t].x = v.x;  // only this lane reads it
          }
          term(v.x, v.y);
        }
        squared = false;
      }
      if (!cached || beyond) {
        // the list, or its entries beyond r_in, DENSITY_WALK rounds' loads in flight at once; an
        // entry well outside 2 h (no term) costs no square root
        constexpr int W = DENSITY_WALK;
        const float d2_far = (2.001f * h) * (2.001f * h);
        for (unsigned b = gl; b < len; b += 8 * W) {
          int jj[W];
          float d2[W], mm[W];
#pragma unroll
          for (int u = 0; u < W; ++u) jj[u] = b + 8 * u < len ? (int)list[b + 8 * u] : -1;
#pragma unroll
          for (int u = 0; u < W; ++u) {
            d2[u] = INFINITY;
            mm[u] = 0.0f;
            if (jj[u] >= 0) {
              float dx, dy, dz;
              geo.diff_m(me_rec, jj[u], dx, dy, dz, mm[u]);
              d2[u] = sqdist(dx, dy, dz);
            }
          }
#pragma unroll
          for (int u = 0; u < W; ++u)
            if (d2[u] < r2max && !(d2[u] > d2_far) && !(beyond && d2[u] < d2_in))
              term(sqrtf(d2[u]), mm[u]);
        }
      }
    }
    rs_out = group_total(rs);
    dws_out = group_total(dws);
  };
  double lo = 0.0, hi = hs;
  const double h0 = h;
  int flag = 3, it = 0;
  bool done = !live;
  const double eta = prm.eta, e3 = eta * eta * eta;
  while (__any_sync(FULL, !done)) {
    double rs, dws;
    sums((float)h, !done, rs, dws);
    if (!done) {
      it += 1;
      double t = eta / h;
      double f = rs - m_i * (t * t * t);
      double h2 = h * h;
      double df = dws + 3.0 * m_i * e3 / (h2 * h2);
      if (f > 0)
        hi = h;
      else
        lo = h;
      double h_new = df > 0 ? h - f / df : 0.5 * (lo + hi);
      if (!(lo <= h_new && h_new <= hi)) h_new = 0.5 * (lo + hi);
      if (fabs(h_new - h) < prm.tol * h0) {
        flag = 0;
        done = true;
      } else if (it >= 50) {
        done = true;
      }
      h = h_new;
    }
  }
  const bool cap_test = live && h >= hs * (1 - 1e-3);
  if (__any_sync(FULL, cap_test)) {
    double rs_lim, dummy;
    sums((float)hs, cap_test, rs_lim, dummy);
    double t = eta / hs;
    if (cap_test && rs_lim - m_i * (t * t * t) < 0) {
      h = hs;
      flag = hs >= prm.h_max ? 1 : 2;
    }
  }
  double rs, dws;
  sums((float)h, live, rs, dws);
  if (work) {
#pragma unroll
    for (int of = 4; of > 0; of >>= 1) evals += __shfl_xor_sync(FULL, evals, of);
  }
  if (live && gl == 0) {
    const int64_t o = out_map ? (int64_t)out_map[i] : q;
    h_out[o] = h;
    rho[o] = rs;
    omega[o] = flag == 1 ? 1.0 : 1.0 + h / (3.0 * rs) * dws;
    if (iters) iters[o] = it;
    if (flags) flags[o] = flag;
    if (work) work[o] = evals;
  }
}

// Terms of one entry (r, m) at 1/h, FP64: m f and m (3 f + q f') with the powers of 1/h factored
// out of the sums.
template <int KID>
struct DensityTerm {
  double inv_h, cn;
  __device__ __forceinline__ DensityTerm(double h, double cn_) : inv_h(1.0 / h), cn(cn_) {}
  __device__ __forceinline__ int add(double r, double m, double& rs, double& dws) const {
    const double q = r * inv_h;
    if (!(q < 2.0)) return 0;
    double f, g;  // f(q) and 3 f + q f'
    if (KID == 0) {
      if (q < 1.0) {
        const double q2 = q * q;
        f = fma(q2, fma(0.75, q, -1.5), 1.0);
        g = fma(q2, fma(4.5, q, -7.5), 3.0);
      } else {
        const double t = 2.0 - q, t2 = t * t;
        f = 0.25 * t2 * t;
        g = 1.5 * t2 * (1.0 - q);
      }
    } else {
      const double x = fma(-0.5, q, 1.0), x2 = x * x, x5 = x2 * x2 * x;
      f = x5 * x * fma(fma(35.0 / 12.0, q, 3.0), q, 1.0);
      g = fma(3.0, f, (-7.0 / 3.0) * (q * q) * x5 * fma(5.0, q, 2.0));
    }
    rs = fma(m, f, rs);
    dws = fma(m, g, dws);
    return 1;
  }
  __device__ __forceinline__ double rho(double s) const { return cn * (inv_h * inv_h * inv_h) * s; }
  __device__ __forceinline__ double drho(double s) const {
    const double i2 = inv_h * inv_h;
    return -cn * (i2 * i2) * s;
  }
};

// FP64 form.  L lanes per row.  The lanes of a row split its list (entry e to lane e mod L,
// coalesced index loads) and keep the squared distance and the index of every entry inside r_in =
// 2.1 h in shared memory, in list order; the Newton sums run over that cache and reduce across
// the lanes, so the lanes of a row take the same Newton steps.  The first sum over a filled cache
// turns the squares into distances (two thirds of the entries are not worth a square root); a
// cached entry's mass is the row's own where all of them are equal, else gathered again.  The
// iterates stay near the start h where it is the last step's; where h leaves the cached range
// (2 h > r_in), or has shrunk enough that the entries of a row too long for the cache may fit, the
// cache is filled again at the present h.  A row with more entries inside 2.1 h than the cache
// holds walks its list in every sum.
// Bound by issue and by the gathers' latency (8 lanes, 262,144 cloud rows: 55 % issue active, L1 66 %,
// FP64 pipe 36 %, 35 % of the warp slots; 920 warp instructions per row).  With one thread per row,
// the list read uncoalesced and walked again in every sum, that call took 1.69 ms; 0.45 ms now.
// Entries kept: about 67 lie inside 2.1 h with the cubic kernel, 159 with Wendland C4.
template <int KID>
constexpr int D64_CAP = KID == 0 ? 128 : 224;
// 8 lanes share the Newton arithmetic among four rows of a warp, 32 give a row all the loads in
// flight at once: see launch_density64 for where each is the faster.
constexpr int D64_UNROLL = 3;  // rounds loaded at once (2, 4, 5 measured up to 10 % slower)

template <int KID, int L, typename I>
__global__ void __launch_bounds__(DENSITY_THREADS, 6)
    k_density64(int64_t nrows, const int64_t* __restrict__ rows, Pos64 geo,
              const double* __restrict__ mass, const double* __restrict__ h_start,
              const double* __restrict__ h_search, const int64_t* __restrict__ off,
              const I* __restrict__ idx, DensityParams prm,
              const int32_t* __restrict__ out_map, double* __restrict__ h_out,
              double* __restrict__ rho, double* __restrict__ omega, int64_t* __restrict__ iters,
              int64_t* __restrict__ flags, int64_t* __restrict__ work) {
  constexpr int CAP = D64_CAP<KID>;
  __shared__ double cache_r[DENSITY_THREADS / L][CAP];
  __shared__ int32_t cache_j[DENSITY_THREADS / L][CAP];
  const unsigned FULL = 0xffffffffu;
  const unsigned GROUP = (unsigned)((1ull << L) - 1ull);
  const int lane = threadIdx.x & 31, gl = lane & (L - 1), g = lane / L;
  const int64_t q = ((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5) * (32 / L) + g;
  const bool live = q < nrows;
  if (!__any_sync(FULL, live)) return;  // warp-uniform
  double* cr = cache_r[threadIdx.x / L];
  int32_t* cj = cache_j[threadIdx.x / L];
  int64_t i = 0, o = 0, e0 = 0;
  unsigned len = 0;
  double m_i = 1.0, hs = 1.0;
  if (live) {
    i = rows ? rows[q] : q;
    o = out_map ? (int64_t)out_map[i] : q;
    m_i = mass[i];
    hs = fmin(h_search[i], prm.h_max);
    e0 = off[i];
    len = (unsigned)(off[i + 1] - e0);
  }
  const I* list = idx + e0;
  const Pos64::Own me_rec = geo.own(i);  // the row's own record, loaded once
  const double r_max = 2.0 * hs;
  const double r2max = r_max * r_max;
  double r_in = 0.0;  // radius of the cached entries
  int cnt = 0;
  bool cached = false, squared = false, uniform = false;
  int evals = 0;
  // The entries inside rin of the rows whose `need` is set, appended in list order.  D64_UNROLL
  // rounds of L entries per pass: their index and record loads are issued together (the walk is
  // bound by the latency of those dependent gathers), then the rounds are appended one after the
  // other.
  constexpr int U = D64_UNROLL;
  auto fill = [&](bool need, double rin) {
    const unsigned mylen = need ? len : 0u;
    const unsigned maxlen = __reduce_max_sync(FULL, mylen);
    const double r2in = fmin(rin * rin, r2max);
    int c = 0;
    bool same = true;
    __syncwarp();
    for (unsigned b = 0; b < maxlen; b += L * U) {
      int jj[U];
      double d2[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const unsigned e = b + L * u + gl;
        jj[u] = e < mylen ? (int)ld_stream(list + e) : -1;
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        d2[u] = INFINITY;
        if (jj[u] >= 0) {
          double dx, dy, dz, m;
          geo.diff_m(me_rec, jj[u], dx, dy, dz, m);
          d2[u] = sqdist(dx, dy, dz);
          if (d2[u] < r2in && m != m_i) same = false;
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const bool inner = d2[u] < r2in;
        const unsigned seg = (__ballot_sync(FULL, inner) >> (L * g)) & GROUP;
        const int pos = c + __popc(seg & ((1u << gl) - 1u));
        if (inner && pos < CAP) {  // overflow: the walk in `sums` instead
          cr[pos] = d2[u];
          cj[pos] = jj[u];
        }
        c += __popc(seg);
      }
    }
    const unsigned differ = (__ballot_sync(FULL, !same) >> (L * g)) & GROUP;
    __syncwarp();
    if (need) {
      r_in = rin;
      cnt = c;
      cached = c <= CAP;
      squared = true;
      uniform = differ == 0;
    }
  };
  // kernel sums at h of the rows whose `active` is set; every lane takes part in the reductions
  auto sums = [&](double h, bool active, double& rs_out, double& dws_out) {
    const DensityTerm<KID> term(h, prm.cnorm);
    const bool outgrown = !(r_in * term.inv_h >= 2.0);
    const bool need = active && (cached ? outgrown : r_in == 0.0 || 2.1 * h < 0.85 * r_in);
    if (__any_sync(FULL, need)) fill(need, 2.1 * h);
    double rs = 0.0, dws = 0.0;
    if (active) {
      if (cached) {
        for (int t = gl; t < cnt; t += L) {
          double r = cr[t];
          if (squared) {
            r = sqrt(r);
            cr[t] = r;  // only this lane reads it
          }
          evals += term.add(r, uniform ? m_i : geo.p[cj[t]].w, rs, dws);
        }
        squared = false;
      } else {
        for (unsigned e = gl; e < len; e += L) {
          double dx, dy, dz, m;
          geo.diff_m(me_rec, (int)list[e], dx, dy, dz, m);
          const double d2 = sqdist(dx, dy, dz);
          if (d2 < r2max) evals += term.add(sqrt(d2), m, rs, dws);
        }
      }
    }
    rs_out = term.rho(group_total<L>(rs));
    dws_out = term.drho(group_total<L>(dws));
  };
  double lo = 0.0, hi = hs;
  double h = live ? fmin(h_start[i], hi) : 1.0;
  double h0 = h;
  int flag = 3, it = 0;
  bool done = !live;
  const double eta = prm.eta, e3 = eta * eta * eta;
  while (__any_sync(FULL, !done)) {
    double rs, dws;
    sums(h, !done, rs, dws);
    if (!done) {
      it += 1;
      double t = eta / h;
      double f = rs - m_i * (t * t * t);
      double h2 = h * h;
      double df = dws + 3.0 * m_i * e3 / (h2 * h2);
      if (f > 0)
        hi = h;
      else
        lo = h;
      double h_new = df > 0 ? h - f / df : 0.5 * (lo + hi);
      if (!(lo <= h_new && h_new <= hi)) h_new = 0.5 * (lo + hi);
      if (fabs(h_new - h) < prm.tol * h0) {
        flag = 0;
        done = true;
      } else if (it >= 50) {
        done = true;
      }
      h = h_new;
    }
  }
  const bool cap_test = live && h >= hs * (1 - 1e-3);
  if (__any_sync(FULL, cap_test)) {
    double rs_lim, dummy;
    sums(cap_test ? hs : h, cap_test, rs_lim, dummy);
    double t = eta / hs;
    if (cap_test && rs_lim - m_i * (t * t * t) < 0) {
      h = hs;
      flag = hs >= prm.h_max ? 1 : 2;
    }
  }
  double rs, dws;
  sums(h, live, rs, dws);
  if (work) {
#pragma unroll
    for (int of = L / 2; of > 0; of >>= 1) evals += __shfl_xor_sync(FULL, evals, of);
  }
  if (live && gl == 0) {
    h_out[o] = h;
    rho[o] = rs;
    omega[o] = flag == 1 ? 1.0 : 1.0 + h / (3.0 * rs) * dws;
    if (iters) iters[o] = it;
    if (flags) flags[o] = flag;
    if (work) work[o] = evals;
  }
}

// ---------------------------------------------------------------- forces
// Reference sim/sph.py:519-652 (_forces_kernel, no reconstruction) and sim/sph.py:1084-1117
// (_disc_kernel).  r_ab = x_a - x_b; F(h) = dW/dr; pair terms antisymmetric.
constexpr int FORCE_QUEUE = 64;  // interacting entries a row queues before its lanes drain them
constexpr int FORCE_UNROLL = 4;  // rounds of eight entries a walk issues at once

// The FP32 pass without the reconstruction runs as two launches: k_walk32 tests the rows' lists and
// writes their interacting entries, with few registers and so many resident warps to hide the
// dependent loads; k_pairs32 then reads those entries, every lane busy on pair terms, with no walk
// state alive beside the accumulators.
//
// k_walk32: every row's interacting entries (r < 2 max(h_a, h_b), self included, list order) to
// prm.tidx (the lists' layout) and their number to prm.tcnt.  With prm.pos64 the level limiter reads
// them too: entries within 1e-5 of the boundary are decided by the reference's FP64 test.
// Bound by the gathers; 2.35M rows of the 4M torus: 2.33 ms (3.01 with the record in two loads and
// the row's own read again per entry; 8 blocks per SM 2.28 for these rows but 3.86 against 3.80
// for all, 5 blocks 2.58).
template <typename I>
__global__ void __launch_bounds__(NB_THREADS, 6)
    k_walk32(int64_t nrows, const int64_t* __restrict__ rows, Pos32 geo,
             const int64_t* __restrict__ off, const I* __restrict__ idx, ForceParams prm) {
  geo.ready();
  const unsigned FULL = 0xffffffffu;
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t q = t >> 3;
  const int gl = (int)(t & 7), g = (threadIdx.x & 31) >> 3;
  const bool live = q < nrows;
  if (!__any_sync(FULL, live)) return;  // warp-uniform
  const int a = live ? (int)(rows ? rows[q] : q) : 0;
  const Pos32::Own me = geo.own(a);
  const float h_a = me.c.w;
  const int64_t e_beg = live ? off[a] : 0;
  const unsigned len = live ? (unsigned)(off[a + 1] - e_beg) : 0u;
  const unsigned maxlen = __reduce_max_sync(FULL, len);
  const I* list = idx + e_beg;
  int32_t* out = prm.tidx + e_beg;
  int m_tot = 0;
  constexpr int U = FORCE_UNROLL;
  for (unsigned base = 0; base < maxlen; base += 8 * U) {
    int bb[U];
    bool tight[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const unsigned e = base + 8 * u + gl;
      bb[u] = e < len ? (int)ld_stream(list + e) : -1;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      tight[u] = bb[u] == a;  // self: listed for the limiter, not a pair
      if (bb[u] >= 0 && bb[u] != a) {
        float dx, dy, dz, h_b;
        geo.diff_h(me, bb[u], dx, dy, dz, h_b);
        const float rr = 2.0f * (h_a > h_b ? h_a : h_b);
        const float d2 = sqdist(dx, dy, dz), r2 = rr * rr;
        bool tk = d2 < r2;
        if (prm.pos64 && d2 > r2 * (float)(1.0 - 1e-5) && d2 < r2 * (float)(1.0 + 1e-5)) {
          const double4 pa = prm.pos64[a], pb = prm.pos64[bb[u]];
          const double e2 = d2_exact(pb.x - pa.x, pb.y - pa.y, pb.z - pa.z);
          const double er = 2.0 * fmax(pa.w, pb.w);
          tk = e2 < er * er;
        }
        tight[u] = tk;
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const unsigned seg = (__ballot_sync(FULL, tight[u]) >> (8 * g)) & 0xffu;
      if (tight[u]) out[m_tot + __popc(seg & ((1u << gl) - 1u))] = bb[u];
      m_tot += __popc(seg);
    }
  }
  if (live && gl == 0) prm.tcnt[q] = m_tot;
}

// k_pairs32: the pair terms of the rows' interacting entries.  One reciprocal square root per pair,
// and reciprocals of the per-particle denominators that come with the records: pk (offset, m)
// (cell, h); pv (v, m) (1/h, rho, 1/(Omega rho^2), P); aux (u, c_s, alpha, Omega).
// Bound by issue and the gathers' latency; the same rows, 58 pairs each: 3.71 ms (4.55 with two
// reciprocals per pair and five loads; 3 blocks per SM 3.85, 5 blocks 4.76).  The flags are looked
// at per pair on purpose: a variant compiled for one of them fuses other operations, which changes
// the float sums in their eighth digit.
static __global__ void __launch_bounds__(NB_THREADS, 4)
    k_pairs32(int64_t nrows, const int64_t* __restrict__ rows, Pos32 geo,
              const float4* __restrict__ pv, const float4* __restrict__ aux,
              const int64_t* __restrict__ off, ForceParams prm,
              const int32_t* __restrict__ out_map, ForceOut out) {
  geo.ready();
  using R = float;
  const unsigned FULL = 0xffffffffu;
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t q = t >> 3;
  const int gl = (int)(t & 7);
  const bool live = q < nrows;
  if (!__any_sync(FULL, live)) return;  // warp-uniform
  const int a = live ? (int)(rows ? rows[q] : q) : 0;
  const Pos32::Own me = geo.own(a);
  const float4 va = pv[2 * (int64_t)a], ha = pv[2 * (int64_t)a + 1], xa = aux[a];
  const R h_a = me.c.w, rho_a = ha.y, P_a = ha.w;
  const R inv_or_a = R(1) / (xa.w * rho_a), inv_orr_a = ha.z;
  const R cs_a = xa.y, al_a = xa.z, u_a = xa.x;
  const R beta = (R)prm.beta, alpha_u = (R)prm.alpha_u, aav = (R)prm.disc_alpha_av;
  const R cn = (R)prm.cnorm;
  const int kid = prm.kid;
  const R ih_a = ha.x;
  const R cn4_a = cn * (ih_a * ih_a) * (ih_a * ih_a);
  Kahan ax, ay, az, work, heat, vheat, cheat, dax, day, daz, dheat;
  R vmax = prm.use_visc ? cs_a : R(0);
  int npairs = 0;
  auto pair = [&](int b) {
    R ddx, ddy, ddz, h_b;
    geo.diff_h(me, b, ddx, ddy, ddz, h_b);  // x_b - x_a
    float4 vb, hb4;
    ld_rec(pv + 2 * (int64_t)b, vb, hb4);
    const float4 xb = aux[b];
    const R d2 = sqdist(ddx, ddy, ddz);
    npairs += 1;
    const R rho_b = hb4.y, P_b = hb4.w;
    const R m_b = vb.w;
    const R inv_r = rsqrtf(d2);
    const R r = d2 * inv_r;
    const R rx = -ddx * inv_r, ry = -ddy * inv_r, rz = -ddz * inv_r;  // r_hat of x_a - x_b
    const R ih_b = hb4.x;
    const R fa = cn4_a * kernel_df<R>(r * ih_a, kid);
    const R fb = cn * (ih_b * ih_b) * (ih_b * ih_b) * kernel_df<R>(r * ih_b, kid);
    const R dvx = va.x - vb.x, dvy = va.y - vb.y, dvz = va.z - vb.z;
    const R vdotr = dvx * rx + dvy * ry + dvz * rz;
    R num_a = P_a, num_b = P_b;
    const R inv_orr_b = hb4.z;
    if (prm.use_visc) {
      R vsig_a = al_a * cs_a + beta * fabs(vdotr);
      R vsig_b = xb.z * xb.y + beta * fabs(vdotr);
      if (vsig_a > vmax) vmax = vsig_a;
      if (vdotr < R(0)) {
        num_a += R(-0.5) * rho_a * vsig_a * vdotr;
        num_b += R(-0.5) * rho_b * vsig_b * vdotr;
        R dh = m_b * vsig_a * R(0.5) * vdotr * vdotr * fa * inv_or_a;
        heat.add(-dh);
        vheat.add(-dh);
      }
      if (prm.use_cond) {
        R vu;
        if (prm.cond_signal == 0)
          vu = sqrt(fabs(P_a - P_b) * __frcp_rn(R(0.5) * (rho_a + rho_b)));
        else
          vu = fabs(vdotr);
        R dc = m_b * alpha_u * vu * (u_a - xb.x) * R(0.5) *
               (fa * inv_or_a + fb * inv_orr_b * rho_b);
        heat.add(dc);
        cheat.add(dc);
      }
    }
    R f = m_b * (num_a * inv_orr_a * fa + num_b * inv_orr_b * fb);
    ax.add(-f * rx);
    ay.add(-f * ry);
    az.add(-f * rz);
    work.add(m_b * vdotr * fa);
    if (prm.use_disc) {
      const R vdr = vdotr;  // v_ab . (x_a - x_b) / r
      R qa = -rho_a * h_a * R(0.5) * inv_r * aav * cs_a * vdr * inv_orr_a;
      R qb = -rho_b * h_b * R(0.5) * inv_r * aav * xb.y * vdr * inv_orr_b;
      R f = m_b * (qa * fa + qb * fb);
      dax.add(-(f * rx));
      day.add(-(f * ry));
      daz.add(-(f * rz));
      dheat.add(m_b * qa * vdr * fa);
    }
  };
  const int cnt = live ? prm.tcnt[q] : 0;
  const int32_t* list = prm.tidx + (live ? off[a] : 0);
  int next = gl < cnt ? ld_stream(list + gl) : a;
  for (int k = gl; k < cnt; k += 8) {
    const int b = next;
    next = k + 8 < cnt ? ld_stream(list + k + 8) : a;
    if (b != a) pair(b);
  }
  double s_ax = group_total(ax), s_ay = group_total(ay), s_az = group_total(az);
  double s_work = group_total(work), s_heat = group_total(heat);
  double s_vheat = group_total(vheat), s_cheat = group_total(cheat);
  double s_dax = 0, s_day = 0, s_daz = 0, s_dheat = 0;
  if (prm.use_disc) {
    s_dax = group_total(dax);
    s_day = group_total(day);
    s_daz = group_total(daz);
    s_dheat = group_total(dheat);
  }
#pragma unroll
  for (int of = 4; of > 0; of >>= 1) {
    R vo = __shfl_xor_sync(FULL, vmax, of);
    vmax = vo > vmax ? vo : vmax;
    npairs += __shfl_xor_sync(FULL, npairs, of);
  }
  if (!live || gl != 0) return;
  const int64_t o = out_map ? (int64_t)out_map[a] : q;
  if (out.acc) {
    out.acc[3 * o + 0] = s_ax;
    out.acc[3 * o + 1] = s_ay;
    out.acc[3 * o + 2] = s_az;
  }
  if (out.dudt) out.dudt[o] = (double)P_a * (double)inv_or_a / (double)rho_a * s_work + s_heat;
  if (out.vsig) out.vsig[o] = (double)vmax;
  if (out.vheat) out.vheat[o] = s_vheat;
  if (out.cheat) out.cheat[o] = s_cheat;
  if (prm.use_disc) {
    if (out.dacc) {
      out.dacc[3 * o + 0] = s_dax;
      out.dacc[3 * o + 1] = s_day;
      out.dacc[3 * o + 2] = s_daz;
    }
    if (out.ddudt) out.ddudt[o] = s_dheat;
  }
  if (out.pairs) out.pairs[o] = npairs;
}

// FP32 with the reconstruction: pressure + artificial viscosity (+ conductivity) + P dV (+ disc
// viscosity) in one launch, eight lanes per row (lanes 8g .. 8g+7 of a warp); the walk queues the
// interacting entries in shared memory and drains them into the pair terms as it goes.  Two
// blocks per SM: with two 3x3 gradients per pair more would spill.
template <typename I>
__global__ void __launch_bounds__(NB_THREADS, 2)
    k_forces_recon32(int64_t nrows, const int64_t* __restrict__ rows, Pos32 geo,
             const float4* __restrict__ vm,    // (vx, vy, vz, mass)
             const float4* __restrict__ hydro, // (h, rho, omega, P)
             const float4* __restrict__ aux,   // (u, c_s, alpha, unused)
             const int64_t* __restrict__ off, const I* __restrict__ idx, ForceParams prm,
             const int32_t* __restrict__ out_map, ForceOut out) {
  using R = float;
  geo.ready();
  const unsigned FULL = 0xffffffffu;
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t q = t >> 3;
  const int gl = (int)(t & 7);
  const bool live = q < nrows;
  if (!__any_sync(FULL, live)) return;  // warp-uniform
  int64_t a = 0, o = 0;
  if (live) {
    a = rows ? rows[q] : q;
    o = out_map ? (int64_t)out_map[a] : q;
  }
  const float4 va = vm[a], ha = hydro[a], xa = aux[a];
  const R h_a = (R)ha.x, rho_a = (R)ha.y, om_a = (R)ha.z, P_a = (R)ha.w;
  const R inv_or_a = R(1) / (om_a * rho_a);
  const R inv_orr_a = R(1) / (om_a * rho_a * rho_a);
  const R cs_a = (R)xa.y, al_a = (R)xa.z;
  const R beta = (R)prm.beta, alpha_u = (R)prm.alpha_u, aav = (R)prm.disc_alpha_av;
  const R cn = (R)prm.cnorm;
  const int kid = prm.kid;
  Kahan ax, ay, az, work, heat, vheat, cheat, dax, day, daz, dheat;
  R vmax = prm.use_visc ? cs_a : R(0);
  int64_t npairs = 0;
  // the row's list in rounds of eight entries: lanes test their entry, the interacting ones are
  // queued in shared memory in list order, and full queues are drained with all eight lanes
  // busy on pair terms
  __shared__ int32_t queue_s[NB_THREADS / 8][FORCE_QUEUE + 8 * FORCE_UNROLL];
  int32_t* pq = queue_s[threadIdx.x >> 3];
  const int g = (threadIdx.x & 31) >> 3;
  const int64_t e_beg = live ? off[a] : 0, e_end = live ? off[a + 1] : 0;
  const unsigned len = (unsigned)(e_end - e_beg);
  const unsigned maxlen = __reduce_max_sync(FULL, len);
  int pc = 0;
  // velocity reconstruction (sim/sph.py:568-609; physics/viscosity.py:116-158): the jump that
  // drives q is the velocity difference extrapolated to the pair midpoint with each side's
  // gradient, limited by the van Leer limiter of their projections and by the closeness factor;
  // the shock heating keeps the actual v_ab . r_hat
  R Ga[9];
#pragma unroll
  for (int e = 0; e < 9; ++e) {
    Ga[e] = prm.gv32[9 * a + e];
  }
  const R eta_crit = (R)prm.eta_crit, eta_fold = (R)prm.eta_fold;
  auto recon_visc = [&](int64_t b, R dx0, R dx1, R dx2, R r, R rx, R ry, R rz, R h_b, R vdotr,
                        const float4& vb, const float4& xb, R rho_b, R m_b, R fa, R& num_a, R& num_b) {
    R Gb[9];
#pragma unroll
    for (int e = 0; e < 9; ++e) Gb[e] = prm.gv32[9 * b + e];
    const R ga0 = Ga[0] * dx0 + Ga[1] * dx1 + Ga[2] * dx2;
    const R ga1 = Ga[3] * dx0 + Ga[4] * dx1 + Ga[5] * dx2;
    const R ga2 = Ga[6] * dx0 + Ga[7] * dx1 + Ga[8] * dx2;
    const R gb0 = Gb[0] * dx0 + Gb[1] * dx1 + Gb[2] * dx2;
    const R gb1 = Gb[3] * dx0 + Gb[4] * dx1 + Gb[5] * dx2;
    const R gb2 = Gb[6] * dx0 + Gb[7] * dx1 + Gb[8] * dx2;
    const R pa = dx0 * ga0 + dx1 * ga1 + dx2 * ga2;
    const R pb = dx0 * gb0 + dx1 * gb1 + dx2 * gb2;
    R phi = R(0);
    if (pb != R(0)) {
      const R ratio = pa / pb;
      if (ratio > R(0)) {
        const R t = R(4) * ratio / ((R(1) + ratio) * (R(1) + ratio));
        phi = t < R(1) ? t : R(1);
      }
    }
    if (prm.closeness) {
      const R e_a = r / h_a, e_b = r / h_b;
      const R eta_ab = e_b < e_a ? e_b : e_a;
      if (eta_ab < eta_crit) {
        const R t = (eta_ab - eta_crit) / eta_fold;
        phi *= exp(-t * t);
      }
    }
    const R hp = R(0.5) * phi;
    R vdr = (((R)va.x - hp * ga0) - ((R)vb.x + hp * gb0)) * rx +
            (((R)va.y - hp * ga1) - ((R)vb.y + hp * gb1)) * ry +
            (((R)va.z - hp * ga2) - ((R)vb.z + hp * gb2)) * rz;
    bool on = vdr < R(0) && vdotr < R(0);
    if (prm.gate == 1)
      on = vdr < R(0);
    else if (prm.gate == 2 && vdotr > vdr)
      vdr = vdotr;
    const R vsig_a = al_a * cs_a + beta * fabs(vdr);
    const R vsig_b = (R)xb.z * (R)xb.y + beta * fabs(vdr);
    const R vsig_cfl = al_a * cs_a + beta * fabs(vdotr);
    if (vsig_cfl > vmax) vmax = vsig_cfl;
    if (on) {
      num_a += R(-0.5) * rho_a * vsig_a * vdr;
      num_b += R(-0.5) * rho_b * vsig_b * vdr;
      R dh = m_b * vsig_a * R(0.5) * vdr * vdotr * fa * inv_or_a;
      heat.add(-dh);
      vheat.add(-dh);
    }
  };
  // FP32 form: the same terms with one reciprocal square root per pair and reciprocals of the
  // per-particle denominators instead of divisions (rounding differs from the FP64 form by a few
  // float ulps, far inside the FP32 tolerances)
  const R ih_a = R(1) / h_a;
  const R cn4_a = cn * (ih_a * ih_a) * (ih_a * ih_a);
  auto pair_fast = [&](int64_t b) {
    R ddx, ddy, ddz;
    geo.diff(a, b, ddx, ddy, ddz);  // x_b - x_a
    const float4 hb4 = hydro[b];
    const R h_b = (R)hb4.x;
    const R d2 = sqdist(ddx, ddy, ddz);
    npairs += 1;
    const float4 vb = vm[b];
    const R rho_b = (R)hb4.y, om_b = (R)hb4.z, P_b = (R)hb4.w;
    const R m_b = (R)vb.w;
    const R inv_r = rsqrtf(d2);
    const R r = d2 * inv_r;
    const R rx = -ddx * inv_r, ry = -ddy * inv_r, rz = -ddz * inv_r;  // r_hat of x_a - x_b
    const R ih_b = __frcp_rn(h_b);
    const R fa = cn4_a * kernel_df<R>(r * ih_a, kid);
    const R fb = cn * (ih_b * ih_b) * (ih_b * ih_b) * kernel_df<R>(r * ih_b, kid);
    const R dvx = (R)(va.x - vb.x), dvy = (R)(va.y - vb.y), dvz = (R)(va.z - vb.z);
    const R vdotr = dvx * rx + dvy * ry + dvz * rz;
    R num_a = P_a, num_b = P_b;
    const R inv_orr_b = __frcp_rn(om_b * rho_b * rho_b);
    if (prm.use_visc) {
      const float4 xb = aux[b];
      recon_visc(b, -ddx, -ddy, -ddz, r, rx, ry, rz, h_b, vdotr, vb, xb, rho_b, m_b, fa, num_a,
                 num_b);
      if (prm.use_cond) {
        R vu;
        if (prm.cond_signal == 0)
          vu = sqrt(fabs(P_a - P_b) * __frcp_rn(R(0.5) * (rho_a + rho_b)));
        else
          vu = fabs(vdotr);
        R dc = m_b * alpha_u * vu * (R)(xa.x - xb.x) * R(0.5) *
               (fa * inv_or_a + fb * inv_orr_b * rho_b);
        heat.add(dc);
        cheat.add(dc);
      }
    }
    R f = m_b * (num_a * inv_orr_a * fa + num_b * inv_orr_b * fb);
    ax.add(-f * rx);
    ay.add(-f * ry);
    az.add(-f * rz);
    work.add(m_b * vdotr * fa);
    if (prm.use_disc) {
      const float4 xb = aux[b];
      const R vdr = vdotr;  // v_ab . (x_a - x_b) / r
      R qa = -rho_a * h_a * R(0.5) * inv_r * aav * cs_a * vdr * inv_orr_a;
      R qb = -rho_b * h_b * R(0.5) * inv_r * aav * (R)xb.y * vdr * inv_orr_b;
      R f = m_b * (qa * fa + qb * fb);
      dax.add(-(f * rx));
      day.add(-(f * ry));
      daz.add(-(f * rz));
      dheat.add(m_b * qa * vdr * fa);
    }
  };
  auto drain = [&]() {
    for (int k2 = gl; k2 < pc; k2 += 8) {
      pair_fast((int64_t)pq[k2]);
    }
    __syncwarp();
    pc = 0;
  };
  // with prm.tidx the row's interacting entries (self included), in list order, are also
  // written out for the level limiter: exactly the reference's FP64 test, which the FP32 form
  // takes from prm.pos64 where its float test falls within 1e-5 of the boundary
  int m_tot = 0;
  // FORCE_UNROLL rounds of eight entries at a time: their index and position loads are issued
  // together, then the rounds are queued one after the other in list order
  constexpr int FU = FORCE_UNROLL;
  for (unsigned base = 0; base < maxlen; base += 8 * FU) {
    int64_t bb[FU];
    bool take[FU], tight[FU];
#pragma unroll
    for (int u = 0; u < FU; ++u) {
      const unsigned e = base + 8 * u + gl;
      bb[u] = e < len ? (int64_t)ld_stream(idx + e_beg + e) : -1;
    }
#pragma unroll
    for (int u = 0; u < FU; ++u) {
      const int64_t b = bb[u];
      take[u] = false;
      tight[u] = false;
      if (b >= 0) {
        if (b != a) {
          R ddx, ddy, ddz, h_b;
          geo.diff_h(geo.own(a), b, ddx, ddy, ddz, h_b);
          R rr = R(2) * (h_a > h_b ? h_a : h_b);
          const R d2 = sqdist(ddx, ddy, ddz), r2 = rr * rr;
          bool tk = d2 < r2;
          if (prm.pos64 && d2 > r2 * R(1.0 - 1e-5) && d2 < r2 * R(1.0 + 1e-5)) {
            const double4 pa = prm.pos64[a], pb = prm.pos64[b];
            const double e2 = d2_exact(pb.x - pa.x, pb.y - pa.y, pb.z - pa.z);
            const double er = 2.0 * fmax(pa.w, pb.w);
            tk = e2 < er * er;
          }
          take[u] = tk;
          tight[u] = tk;
        } else {
          tight[u] = true;  // self: listed for the limiter, not a pair
        }
      }
    }
#pragma unroll
    for (int u = 0; u < FU; ++u) {
      unsigned seg = (__ballot_sync(FULL, take[u]) >> (8 * g)) & 0xffu;
      if (take[u]) pq[pc + __popc(seg & ((1u << gl) - 1u))] = (int32_t)bb[u];
      pc += __popc(seg);
      if (prm.tidx) {
        const unsigned tseg = (__ballot_sync(FULL, tight[u]) >> (8 * g)) & 0xffu;
        if (tight[u])
          prm.tidx[e_beg + m_tot + __popc(tseg & ((1u << gl) - 1u))] = (int32_t)bb[u];
        m_tot += __popc(tseg);
      }
    }
    if (__any_sync(FULL, pc > FORCE_QUEUE - 8)) drain();
  }
  drain();
  if (prm.tcnt && live && gl == 0) prm.tcnt[q] = m_tot;
  // sums over the row's eight lanes (uniform flags: every lane takes part in every reduction)
  double s_dax = 0, s_day = 0, s_daz = 0, s_dheat = 0;
  const double s_ax = group_total(ax), s_ay = group_total(ay), s_az = group_total(az);
  const double s_work = group_total(work), s_heat = group_total(heat);
  const double s_vheat = group_total(vheat), s_cheat = group_total(cheat);
  if (prm.use_disc) {
    s_dax = group_total(dax);
    s_day = group_total(day);
    s_daz = group_total(daz);
    s_dheat = group_total(dheat);
  }
#pragma unroll
  for (int of = 4; of > 0; of >>= 1) {
    R vo = __shfl_xor_sync(FULL, vmax, of);
    vmax = vo > vmax ? vo : vmax;
    npairs += __shfl_xor_sync(FULL, npairs, of);
  }
  if (!live || gl != 0) return;
  const double du = (double)P_a * (double)inv_or_a / (double)rho_a * s_work + s_heat;
  if (out.acc) {
    out.acc[3 * o + 0] = s_ax;
    out.acc[3 * o + 1] = s_ay;
    out.acc[3 * o + 2] = s_az;
  }
  if (out.dudt) out.dudt[o] = du;
  if (out.vsig) out.vsig[o] = (double)vmax;
  if (out.vheat) out.vheat[o] = s_vheat;
  if (out.cheat) out.cheat[o] = s_cheat;
  if (prm.use_disc) {
    if (out.dacc) {
      out.dacc[3 * o + 0] = s_dax;
      out.dacc[3 * o + 1] = s_day;
      out.dacc[3 * o + 2] = s_daz;
    }
    if (out.ddudt) out.ddudt[o] = s_dheat;
  }
  if (out.pairs) out.pairs[o] = npairs;
}

// ---------------------------------------------------------------- forces, FP64
// The same pass in double (sim/sph.py:519-652, 568-609, 1084-1117).  What a division would give per
// pair is precomputed per particle: the records are (x, y, z, h), (v, m), (1/h, rho, 1/(Omega
// rho^2), P), (u, c_s, alpha, -) and, with the reconstruction, the symmetric part of the velocity
// gradient (xx, yy, zz, xy, xz, yz, -, -), each fetched in one 32-byte load; a pair needs one
// reciprocal square root, and one division more with the reconstruction.
//   SPH   pressure, viscosity, conductivity, P dV;  DISC  disc viscosity
//   RECON velocity reconstruction (the jump only enters through its projections on the pair
//         axis: with pa = dx.Ga dx and pb = dx.Gb dx the jump is v_ab . r_hat - phi/2 (pa + pb) / r,
//         and the limiter 4 x / (1 + x)^2 of x = pa / pb is 4 pa pb / (pa + pb)^2)
//   TIGHT the list holds entries beyond 2 max(h_a, h_b): the walk tests them, queues the
//         interacting ones in shared memory and drains full queues with all lanes busy; without
//         it every entry is a pair and the lanes take them straight from the list
// Bound by the FP64 pipe and the gathers' latency at 12 to 24 resident warps (128 B per pair).
// 148,000 torus rows of 58 pairs: 207 us with viscosity and conductivity, 165 us disc viscosity
// (about 385 each with a division per term); 100,000 rows of 137 pairs with the reconstruction:
// 423 us (898 with 3x3 gradients and 210 registers).
constexpr int F64_THREADS = 128;

template <bool SPH, bool DISC, bool RECON>
struct F64Blocks {
  // 4 and 5 blocks with the reconstruction spill (5: 1.40 ms against 1.08 for its case), 6 and 8
  // without it gain nothing more
  static constexpr int value = RECON ? 3 : !SPH ? 6 : DISC ? 4 : 5;
};

template <bool SPH, bool DISC, bool RECON, bool TIGHT, typename I>
__global__ void __launch_bounds__(F64_THREADS, (F64Blocks<SPH, DISC, RECON>::value))
    k_forces64(int64_t nrows, const int64_t* __restrict__ rows, const double4* __restrict__ pos,
               const double4* __restrict__ vm, const double4* __restrict__ hyd,
               const double4* __restrict__ aux, const double4* __restrict__ sym,
               const int64_t* __restrict__ off, const I* __restrict__ idx, ForceParams prm,
               const int32_t* __restrict__ out_map, ForceOut out) {
  const unsigned FULL = 0xffffffffu;
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t q = t >> 3;
  const int gl = (int)(t & 7), g = (threadIdx.x & 31) >> 3;
  const bool live = q < nrows;
  if (!__any_sync(FULL, live)) return;  // warp-uniform
  const int64_t a = live ? (rows ? rows[q] : q) : 0;
  const double4 xa = pos[a], va = vm[a], ha = hyd[a], ua = aux[a];
  const double ih_a = ha.x, rho_a = ha.y, iorr_a = ha.z, P_a = ha.w, cs_a = ua.y, al_a = ua.z;
  const double cn4_a = prm.cnorm * (ih_a * ih_a) * (ih_a * ih_a);
  const double ior_a = iorr_a * rho_a;  // 1 / (Omega rho)
  const double beta = prm.beta;
  // disc viscosity: q_a = k_a (v . r_hat) / r, with the pair's side b alike
  const double disc_a = -0.5 * rho_a * xa.w * prm.disc_alpha_av * cs_a * iorr_a;
  double4 sa0 = make_double4(0, 0, 0, 0), sa1 = sa0;
  if constexpr (RECON) {
    sa0 = sym[2 * a];
    sa1 = sym[2 * a + 1];
  }
  double ax = 0, ay = 0, az = 0, work = 0, vheat = 0, cheat = 0;
  double dax = 0, day = 0, daz = 0, dheat = 0;
  double vmax = SPH && prm.use_visc ? cs_a : 0.0;
  int npairs = 0;
  auto pair = [&](int b) {
    const double4 xb = ld_rec(pos + b), vb = ld_rec(vm + b), hb = ld_rec(hyd + b);
    double4 ub = make_double4(0, 0, 0, 0);
    if (DISC || prm.use_visc) ub = ld_rec(aux + b);
    npairs += 1;
    const double dx = xa.x - xb.x, dy = xa.y - xb.y, dz = xa.z - xb.z;
    const double d2 = fma(dz, dz, fma(dy, dy, dx * dx));
    const double ir = rsqrt(d2);
    double r = d2 * ir;
    if (!(r > 0.0)) r = d2;  // 0 and infinity, as a square root gives them
    const double rx = dx * ir, ry = dy * ir, rz = dz * ir;
    const double ih_b = hb.x, ih2 = ih_b * ih_b;
    const double fa = cn4_a * kernel_df<double>(r * ih_a, prm.kid);
    const double fb = prm.cnorm * (ih2 * ih2) * kernel_df<double>(r * ih_b, prm.kid);
    const double m = vb.w;
    const double vr = fma(va.z - vb.z, rz, fma(va.y - vb.y, ry, (va.x - vb.x) * rx));
    if constexpr (SPH) {
      double na = P_a, nb = hb.w;
      if (prm.use_visc) {
        double jump = vr;  // drives the viscosity
        bool on = vr < 0.0;
        if constexpr (RECON) {
          const double4 sb0 = ld_rec(sym + 2 * (int64_t)b), sb1 = ld_rec(sym + 2 * (int64_t)b + 1);
          const double xx = dx * dx, yy = dy * dy, zz = dz * dz;
          const double xy = 2.0 * dx * dy, xz = 2.0 * dx * dz, yz = 2.0 * dy * dz;
          const double pa = fma(sa1.y, yz, fma(sa1.x, xz, fma(sa0.w, xy, fma(sa0.z, zz, fma(sa0.y, yy, sa0.x * xx)))));
          const double pb = fma(sb1.y, yz, fma(sb1.x, xz, fma(sb0.w, xy, fma(sb0.z, zz, fma(sb0.y, yy, sb0.x * xx)))));
          double phi = 0.0;
          const double pp = pa * pb;
          if (pp > 0.0) {
            const double s = pa + pb;
            phi = fmin(4.0 * pp / (s * s), 1.0);
            if (prm.closeness) {
              const double eta_ab = r * fmin(ih_a, ih_b);
              if (eta_ab < prm.eta_crit) {
                const double c = (eta_ab - prm.eta_crit) / prm.eta_fold;
                phi *= exp(-c * c);
              }
            }
          }
          jump = fma(-0.5 * phi * (pa + pb), ir, vr);
          on = jump < 0.0 && vr < 0.0;
          if (prm.gate == 1)
            on = jump < 0.0;
          else if (prm.gate == 2 && vr > jump)
            jump = vr;
        }
        const double aj = fabs(jump);
        const double vs_a = fma(beta, aj, al_a * cs_a), vs_b = fma(beta, aj, ub.z * ub.y);
        const double cfl = RECON ? fma(beta, fabs(vr), al_a * cs_a) : vs_a;
        if (cfl > vmax) vmax = cfl;
        if (on) {
          const double hj = -0.5 * jump;
          na = fma(rho_a * vs_a, hj, na);
          nb = fma(hb.y * vs_b, hj, nb);
          vheat = fma(m * vs_a * hj * vr, fa * ior_a, vheat);
        }
        if (prm.use_cond) {
          const double vu = prm.cond_signal == 0
                                ? sqrt(fabs(P_a - hb.w) / (0.5 * (rho_a + hb.y)))
                                : fabs(vr);
          cheat = fma(m * prm.alpha_u * vu * (ua.x - ub.x) * 0.5,
                      fma(fb, hb.z * hb.y, fa * ior_a), cheat);
        }
      }
      const double f = -m * fma(nb * hb.z, fb, na * iorr_a * fa);
      ax = fma(f, rx, ax);
      ay = fma(f, ry, ay);
      az = fma(f, rz, az);
      work = fma(m * vr, fa, work);
    }
    if constexpr (DISC) {
      const double s = vr * ir;
      const double qa = disc_a * s;
      const double qb = -0.5 * hb.y * xb.w * prm.disc_alpha_av * ub.y * hb.z * s;
      const double f = -m * fma(qb, fb, qa * fa);
      dax = fma(f, rx, dax);
      day = fma(f, ry, day);
      daz = fma(f, rz, daz);
      dheat = fma(m * qa * vr, fa, dheat);
    }
  };
  const int64_t e0 = live ? off[a] : 0;
  const unsigned len = live ? (unsigned)(off[a + 1] - e0) : 0u;
  const I* list = idx + e0;
  if constexpr (!TIGHT) {
    int next = gl < len ? (int)ld_stream(list + gl) : -1;
    for (unsigned e = gl; e < len; e += 8) {
      const int b = next;
      next = e + 8 < len ? (int)ld_stream(list + e + 8) : -1;
      if (b != (int)a) pair(b);
    }
  } else {
    // rounds of eight entries, FORCE_UNROLL of them with their loads issued together; with
    // prm.tidx the interacting entries (self included, list order) are also written out for the
    // level limiter
    constexpr int U = FORCE_UNROLL;
    __shared__ int32_t queue_s[F64_THREADS / 8][FORCE_QUEUE + 8 * U];
    int32_t* pq = queue_s[threadIdx.x >> 3];
    int pc = 0, m_tot = 0;
    auto drain = [&]() {
      __syncwarp();
      for (int k = gl; k < pc; k += 8) pair(pq[k]);
      __syncwarp();
      pc = 0;
    };
    const unsigned maxlen = __reduce_max_sync(FULL, len);
    for (unsigned base = 0; base < maxlen; base += 8 * U) {
      int bb[U];
      bool near[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const unsigned e = base + 8 * u + gl;
        bb[u] = e < len ? (int)ld_stream(list + e) : -1;
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        near[u] = false;
        if (bb[u] >= 0) {
          const double4 o = ld_rec(pos + bb[u]);
          const double d2 = d2_exact(o.x - xa.x, o.y - xa.y, o.z - xa.z);
          const double rr = 2.0 * (xa.w > o.w ? xa.w : o.w);
          near[u] = bb[u] == (int)a || d2 < rr * rr;
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const bool take = near[u] && bb[u] != (int)a;
        const unsigned below = (1u << gl) - 1u;
        const unsigned seg = (__ballot_sync(FULL, take) >> (8 * g)) & 0xffu;
        if (take) pq[pc + __popc(seg & below)] = bb[u];
        pc += __popc(seg);
        if (prm.tidx) {
          const unsigned tseg = (__ballot_sync(FULL, near[u]) >> (8 * g)) & 0xffu;
          if (near[u]) prm.tidx[e0 + m_tot + __popc(tseg & below)] = bb[u];
          m_tot += __popc(tseg);
        }
      }
      if (__any_sync(FULL, pc > FORCE_QUEUE - 8)) drain();
    }
    drain();
    if (prm.tcnt && live && gl == 0) prm.tcnt[q] = m_tot;
  }
  if constexpr (SPH) {
    ax = group_total(ax);
    ay = group_total(ay);
    az = group_total(az);
    work = group_total(work);
    vheat = group_total(vheat);
    cheat = group_total(cheat);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
      const double vo = __shfl_xor_sync(FULL, vmax, o);
      vmax = vo > vmax ? vo : vmax;
    }
  }
  if constexpr (DISC) {
    dax = group_total(dax);
    day = group_total(day);
    daz = group_total(daz);
    dheat = group_total(dheat);
  }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) npairs += __shfl_xor_sync(FULL, npairs, o);
  if (!live || gl != 0) return;
  const int64_t o = out_map ? (int64_t)out_map[a] : q;
  if constexpr (SPH) {
    if (out.acc) {
      out.acc[3 * o + 0] = ax;
      out.acc[3 * o + 1] = ay;
      out.acc[3 * o + 2] = az;
    }
    if (out.dudt) out.dudt[o] = fma(P_a * iorr_a, work, vheat + cheat);
    if (out.vsig) out.vsig[o] = vmax;
    if (out.vheat) out.vheat[o] = vheat;
    if (out.cheat) out.cheat[o] = cheat;
  }
  if constexpr (DISC) {
    if (out.dacc) {
      out.dacc[3 * o + 0] = dax;
      out.dacc[3 * o + 1] = day;
      out.dacc[3 * o + 2] = daz;
    }
    if (out.ddudt) out.ddudt[o] = dheat;
  }
  if (out.pairs) out.pairs[o] = npairs;
}

// ---------------------------------------------------------------- corrected gradients
// Reference sim/sph.py:693-902 (_near_singular, _velocity_gradient_kernel, _gradients_kernel):
//     R_lj = sum_b m_b (x_b - x_a)^l dW_ab(h_a)/dx_a^j,  G_kj = sum_b m_b (v_b - v_a)^k dW/dx_a^j,
//     dv/dx = G R^-1 (the same with accelerations for d(div v)/dt),
// with dW_ab(h_a)/dx_a = (x_a - x_b) F(r, h_a) / r.  Fewer than 4 list entries (self excluded),
// tr R <= 0 or |det R| < 1e-6 (tr R / 3)^3: G / (tr R / 3) instead (0 when tr R <= 0).  R^-1 is
// the adjugate over the determinant.  Eight lanes per row, FP64 only (the FP32 form converts).
constexpr double SINGULAR_TOL = 1e-6;

// R is symmetric, (xx, yy, zz, xy, xz, yz); g <- g R^-1 (or the fallback) for the 3x3 row-major
// gradient sums g
template <int NG>
__device__ __forceinline__ void corrected_gradients(const double* rm, int64_t cnt, double (*g)[9]) {
  const double scale = (rm[0] + rm[1] + rm[2]) / 3.0;
  const double c00 = rm[1] * rm[2] - rm[5] * rm[5], c01 = rm[5] * rm[4] - rm[3] * rm[2],
               c02 = rm[3] * rm[5] - rm[1] * rm[4];
  const double det = rm[0] * c00 + rm[3] * c01 + rm[4] * c02;
  const bool singular =
      cnt < 4 || !(scale > 0.0) || !(fabs(det) >= SINGULAR_TOL * scale * scale * scale);
  if (singular) {
    const double inv_s = scale > 0.0 ? 1.0 / scale : 0.0;
#pragma unroll
    for (int k = 0; k < NG; ++k)
#pragma unroll
      for (int e = 0; e < 9; ++e) g[k][e] = g[k][e] * inv_s;
    return;
  }
  double ri[9];
  ri[0] = c00 / det;
  ri[1] = ri[3] = c01 / det;
  ri[2] = ri[6] = c02 / det;
  ri[4] = (rm[0] * rm[2] - rm[4] * rm[4]) / det;
  ri[5] = ri[7] = (rm[4] * rm[3] - rm[0] * rm[5]) / det;
  ri[8] = (rm[0] * rm[1] - rm[3] * rm[3]) / det;
#pragma unroll
  for (int k = 0; k < NG; ++k) {
    double o[9];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j)
        o[3 * i + j] = g[k][3 * i + 0] * ri[j] + g[k][3 * i + 1] * ri[3 + j] +
                       g[k][3 * i + 2] * ri[6 + j];
#pragma unroll
    for (int e = 0; e < 9; ++e) g[k][e] = o[e];
  }
}

// 100,000 rows of 137 entries: 197 us for the velocity gradients, 226 us with the accelerations
// (299 and 333 with a square root and divisions per entry and all nine sums of R).
// The sums R (symmetric) and G of one row (and of the accelerations, with ACC) over the entries of
// a pass, each one rsqrt and fused adds: F(r, h_a) / r = cn4 f'(r / h_a) / r.
// SKIP: entries with F(r, h_a) = 0 are passed over (the step's untightened lists hold many); without
// it they add their zeros, as the operators' reference does.
template <bool ACC, bool SKIP>
struct GradSums {
  double rm[6] = {0, 0, 0, 0, 0, 0}, gv[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0},
         ga[ACC ? 9 : 1] = {0};
  // (dx, dy, dz) = x_a - x_b
  __device__ __forceinline__ void add(double dx, double dy, double dz, double d2, double ih_a,
                                      double cn4, int kid, const double4& va,
                                      const double4* __restrict__ vm, const double4& aa,
                                      const double4* __restrict__ acc, int64_t b, bool use_acc) {
    const double ir = rsqrt(d2);
    double r = d2 * ir;
    if (!(r > 0.0)) r = d2;  // 0 and infinity, as a square root gives them
    const double q = r * ih_a;
    if (SKIP && !(q < 2.0)) return;
    const double4 vb = ld_rec(vm + b);
    const double mf = vb.w * (cn4 * kernel_df<double>(q, kid) * ir);
    const double gx = mf * dx, gy = mf * dy, gz = mf * dz;
    rm[0] = fma(-dx, gx, rm[0]);
    rm[1] = fma(-dy, gy, rm[1]);
    rm[2] = fma(-dz, gz, rm[2]);
    rm[3] = fma(-dx, gy, rm[3]);
    rm[4] = fma(-dx, gz, rm[4]);
    rm[5] = fma(-dy, gz, rm[5]);
    const double dv[3] = {vb.x - va.x, vb.y - va.y, vb.z - va.z};
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      gv[3 * i] = fma(dv[i], gx, gv[3 * i]);
      gv[3 * i + 1] = fma(dv[i], gy, gv[3 * i + 1]);
      gv[3 * i + 2] = fma(dv[i], gz, gv[3 * i + 2]);
    }
    if constexpr (ACC) {
      if (use_acc) {
        const double4 ab = ld_rec(acc + b);
        const double da[3] = {ab.x - aa.x, ab.y - aa.y, ab.z - aa.z};
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          ga[3 * i] = fma(da[i], gx, ga[3 * i]);
          ga[3 * i + 1] = fma(da[i], gy, ga[3 * i + 1]);
          ga[3 * i + 2] = fma(da[i], gz, ga[3 * i + 2]);
        }
      }
    }
  }
  // sums over the row's eight lanes
  __device__ __forceinline__ void total() {
#pragma unroll
    for (int e = 0; e < 6; ++e) rm[e] = group_total(rm[e]);
#pragma unroll
    for (int e = 0; e < 9; ++e) {
      gv[e] = group_total(gv[e]);
      if (ACC) ga[ACC ? e : 0] = group_total(ga[ACC ? e : 0]);
    }
  }
};

// the symmetric part of a velocity gradient as the force pass reads it (8 doubles)
__device__ __forceinline__ void store_sym(double4* out, const double* g) {
  out[0] = make_double4(g[0], g[4], g[8], 0.5 * (g[1] + g[3]));
  out[1] = make_double4(0.5 * (g[2] + g[6]), 0.5 * (g[5] + g[7]), 0.0, 0.0);
}

// physics/viscosity.py:83-113: xi (Balsara), alpha_loc, decay time, then the jump to alpha_loc
// or the backward-Euler decay toward it, for the particle at output index o
__device__ __forceinline__ void switch_update(const GradOut& out, int64_t o, double div,
                                              double curl, double ddiv) {
  // physics/viscosity.py:83-113: xi (Balsara), alpha_loc, decay time, the jump or the decay
  const double d2 = div * div, cc2 = curl * curl;
  const double xi = d2 + cc2 > 0.0 ? d2 / (d2 + cc2) : 0.0;
  const double mdd = -ddiv < 0.0 ? 0.0 : -ddiv;  // max(-d(div v)/dt, 0); NaN stays NaN
  const double h = out.h[o], cs = out.cs[o];
  const double al = 10.0 * h * h * (xi * mdd) / (cs * cs);
  const double a_loc = al > 1.0 ? 1.0 : al;  // min(alpha_loc, alpha_max = 1)
  const double dt =
      out.n_beg ? 2.0 * (0.5 * (double)(out.n_end[o] - out.n_beg[o]) * out.tick) : out.dt;
  const double tau = h / (0.1 * cs);
  const double alpha = out.alpha[o];
  const double decayed = (alpha + a_loc * dt / tau) / (1.0 + dt / tau);
  out.alpha[o] = a_loc > alpha ? a_loc : decayed;
}

// div v, |curl v| and d(div v)/dt from the gradients of v and of the acceleration
__device__ __forceinline__ void switch_scalars(const double (*g)[9], double& div, double& curl,
                                               double& ddiv) {
  const double* v = g[0];
  div = v[0] + v[4] + v[8];
  const double c0 = v[7] - v[5], c1 = v[2] - v[6], c2 = v[3] - v[1];
  curl = sqrt(c0 * c0 + c1 * c1 + c2 * c2);
  double sdd = 0.0;
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) sdd += v[3 * i + j] * v[3 * j + i];
  ddiv = g[1][0] + g[1][4] + g[1][8] - sdd;
}

template <typename I, bool ACC>
__global__ void __launch_bounds__(NB_THREADS, 2)
    k_gradients(int64_t nrows, const int64_t* __restrict__ rows, const double4* __restrict__ pos,
                const double4* __restrict__ vm,   // (vx, vy, vz, mass); pos: (x, y, z, h)
                const double4* __restrict__ acc,  // (ax, ay, az, -), with ACC
                const int64_t* __restrict__ off, const I* __restrict__ idx, int kid, double cnorm,
                GradOut out) {
  const unsigned FULL = 0xffffffffu;
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t q = t >> 3;
  const int gl = (int)(t & 7);
  const bool live = q < nrows;
  if (!__any_sync(FULL, live)) return;  // warp-uniform
  const int64_t a = live ? (rows ? rows[q] : q) : 0;
  const double4 xa = pos[a], va = vm[a];
  const double4 aa = ACC ? acc[a] : make_double4(0.0, 0.0, 0.0, 0.0);
  const double ih_a = 1.0 / xa.w, cn4 = cnorm * (ih_a * ih_a) * (ih_a * ih_a);
  GradSums<ACC, false> s;
  int cnt = 0;
  // eight lanes per row, each taking every eighth list entry (the next one's index is on its way
  // while an entry is summed); the sums are then added over the row's lanes
  const int64_t e0 = live ? off[a] : 0, e1 = live ? off[a + 1] : 0;
  int64_t next = e0 + gl < e1 ? (int64_t)ld_stream(idx + e0 + gl) : -1;
  for (int64_t k = e0 + gl; k < e1; k += 8) {
    const int64_t b = next;
    next = k + 8 < e1 ? (int64_t)ld_stream(idx + k + 8) : -1;
    if (b == a) continue;
    cnt += 1;
    const double4 xb = ld_rec(pos + b);
    const double dx = xa.x - xb.x, dy = xa.y - xb.y, dz = xa.z - xb.z;
    const double d2 = fma(dz, dz, fma(dy, dy, dx * dx));
    s.add(dx, dy, dz, d2, ih_a, cn4, kid, va, vm, aa, acc, b, true);
  }
  s.total();
#pragma unroll
  for (int of = 4; of > 0; of >>= 1) cnt += __shfl_xor_sync(FULL, cnt, of);
  if (!live || gl != 0) return;
  double g[ACC ? 2 : 1][9];
#pragma unroll
  for (int e = 0; e < 9; ++e) {
    g[0][e] = s.gv[e];
    if (ACC) g[ACC ? 1 : 0][e] = s.ga[ACC ? e : 0];
  }
  corrected_gradients<ACC ? 2 : 1>(s.rm, cnt, g);
  if (out.gv) {
#pragma unroll
    for (int e = 0; e < 9; ++e) out.gv[9 * a + e] = g[0][e];
  }
  if constexpr (ACC) {
    double div, curl, ddiv;
    switch_scalars(g, div, curl, ddiv);
    if (out.div) out.div[q] = div;
    if (out.curl) out.curl[q] = curl;
    if (out.ddiv) out.ddiv[q] = ddiv;
  }
}

// The switch and the reconstruction's gradients of a step in one walk of the cached lists
// (sorted order).  A list entry adds to R, G (and the acceleration sum) only where
// F(r, h_a) != 0, i.e. r / h_a < 2, and such an entry always passes the tightening test
// (r < 2 h_a <= 2 max(h_a, h_b)); the other entries add exact zeros.  So the sums over a row's
// tightened list (the switch, and the reconstruction of shared steps) and over its untightened
// list (the reconstruction of block steps) are the same sums over the same nonzero terms in
// the same order, and only the entry counts of the singular-matrix test differ: both are kept.
//   live: particles whose gradient the reconstruction needs (mask, caller order; null = all),
//         or none without it; rows: the switch's rows (sorted mask; null = no switch)
//   pos: (x, y, z, h) records; out.gs (8 doubles per particle, for the FP64 force pass) or out.gv
template <typename I, bool SW>
__global__ void __launch_bounds__(NB_THREADS)
    k_shock_grad(int64_t n, const double4* __restrict__ pos, const double4* __restrict__ vm,
                 const double4* __restrict__ acc, const int64_t* __restrict__ off,
                 const I* __restrict__ idx, int kid, double cnorm, int recon, int recon_full,
                 const uint8_t* __restrict__ live_mask, const uint8_t* __restrict__ row_sorted,
                 const int32_t* __restrict__ perm, GradOut out) {
  const unsigned FULL = 0xffffffffu;
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t a = t >> 3;
  const int gl = (int)(t & 7);
  bool need_g = false, is_row = false;
  int64_t o = 0;
  if (a < n) {
    o = perm[a];
    need_g = recon && (!live_mask || live_mask[o]);
    is_row = SW && row_sorted[a];
  }
  const bool live = need_g || is_row;
  if (!__any_sync(FULL, live)) return;  // warp-uniform
  const double4 xa = pos[live ? a : 0], va = vm[live ? a : 0];
  double4 aa = make_double4(0.0, 0.0, 0.0, 0.0);
  if (SW && is_row) aa = acc[a];
  const double h_a = xa.w, ih_a = 1.0 / h_a, cn4 = cnorm * (ih_a * ih_a) * (ih_a * ih_a);
  GradSums<SW, true> s;
  int cnt_f = 0, cnt_t = 0;
  const int64_t e0 = live ? off[a] : 0, e1 = live ? off[a + 1] : 0;
  int64_t next = e0 + gl < e1 ? (int64_t)ld_stream(idx + e0 + gl) : -1;
  for (int64_t k = e0 + gl; k < e1; k += 8) {
    const int64_t b = next;
    next = k + 8 < e1 ? (int64_t)ld_stream(idx + k + 8) : -1;
    if (b == a) continue;
    cnt_f += 1;
    const double4 xb = ld_rec(pos + b);
    const double dx = xa.x - xb.x, dy = xa.y - xb.y, dz = xa.z - xb.z;
    const double d2 = d2_exact(dx, dy, dz);
    const double rr = 2.0 * (h_a > xb.w ? h_a : xb.w);
    if (d2 < rr * rr) cnt_t += 1;
    s.add(dx, dy, dz, d2, ih_a, cn4, kid, va, vm, aa, acc, b, is_row);
  }
  s.total();
#pragma unroll
  for (int of = 4; of > 0; of >>= 1) {
    cnt_f += __shfl_xor_sync(FULL, cnt_f, of);
    cnt_t += __shfl_xor_sync(FULL, cnt_t, of);
  }
  if (!live || gl != 0) return;
  if (need_g) {
    double g1[1][9];
#pragma unroll
    for (int e = 0; e < 9; ++e) g1[0][e] = s.gv[e];
    corrected_gradients<1>(s.rm, recon_full ? cnt_f : cnt_t, g1);
    if (out.gs)
      store_sym(out.gs + 2 * a, g1[0]);
    else {
#pragma unroll
      for (int e = 0; e < 9; ++e) out.gv[9 * a + e] = g1[0][e];
    }
  }
  if (SW && is_row) {
    double g2[2][9];
#pragma unroll
    for (int e = 0; e < 9; ++e) {
      g2[0][e] = s.gv[e];
      g2[1][e] = s.ga[SW ? e : 0];
    }
    corrected_gradients<2>(s.rm, cnt_t, g2);
    double div, curl, ddiv;
    switch_scalars(g2, div, curl, ddiv);
    switch_update(out, o, div, curl, ddiv);
  }
}

}  // namespace nbk
