// FP64 instantiations of the pair passes.  Compiled without contraction, so that an operation is fused
// only where an fma is written: the list tests round like the reference, the sums' terms do not.
#include <type_traits>

#include "sph_impl.cuh"

namespace nbk {

template <typename I>
void launch_density64(int64_t nrows, const int64_t* rows, const double4* pos, const double* mass,
                      const double* h_start, const double* h_search, const int64_t* off,
                      const I* idx, DensityParams prm, const int32_t* out_map, double* h_out,
                      double* rho, double* omega, int64_t* iters, int64_t* flags, int64_t* work,
                      cudaStream_t st) {
  if (nrows <= 0) return;
  Pos64 geo{pos};
  auto run = [&](auto kid, auto lanes) {
    constexpr int KID = decltype(kid)::value, L = decltype(lanes)::value;
    count_launch(), k_density64<KID, L, I><<<grid_for(nrows * L, DENSITY_THREADS), DENSITY_THREADS, 0, st>>>(
        nrows, rows, geo, mass, h_start, h_search, off, idx, prm, out_map, h_out, rho, omega,
        iters, flags, work);
  };
  using std::integral_constant;
  // Cubic: 8 lanes per row once the rows fill the GPU, 32 for fewer, whose rows are then in flight
  // together.  Where the two meet depends on the gas and the guess; from the last step's h, call
  // times in us with 8 / 32 lanes: a cloud of 10,000 rows 93 / 94, 30,000 130 / 142, 60,000 169 / 203,
  // 262,144 458 / 649; a torus of 30,000 210 / 156, 60,000 268 / 229, 100,000 314 / 306, 200,000
  // 465 / 516.  The line lies between the two gases.  (From a guess far off, 32 lanes stay ahead
  // on a torus: 200,000 rows 3,367 / 2,104.)  Wendland C4: 32 lanes at any size, whose block keeps 4
  // rows' caches (11 KB) instead of 16 rows' (43 KB) out of L1 (200,001 torus rows 0.98 ms
  // against 1.24 with 16 lanes and 1.94 with 8).
  if (prm.kid != 0)
    run(integral_constant<int, 1>{}, integral_constant<int, 32>{});
  else if (nrows >= 65536)
    run(integral_constant<int, 0>{}, integral_constant<int, 8>{});
  else
    run(integral_constant<int, 0>{}, integral_constant<int, 32>{});
}

template <typename I>
void launch_forces64(int64_t nrows, const int64_t* rows, const double4* pos, const double4* vm,
                     const double4* hydro, const double4* aux, const int64_t* off, const I* idx,
                     ForceParams prm, const int32_t* out_map, ForceOut out, cudaStream_t st) {
  if (nrows <= 0) return;
  auto run = [&](auto sph, auto disc, auto recon) {
    constexpr bool S = decltype(sph)::value, D = decltype(disc)::value, R = decltype(recon)::value;
    // the operators' int64 lists are taken as they are, every entry a pair, as their reference does;
    // the engine's int32 lists hold the search radius' entries, which the walk tests
    constexpr bool T = sizeof(I) == 4;
    count_launch(), k_forces64<S, D, R, T, I><<<grid_for(nrows * 8, F64_THREADS), F64_THREADS, 0, st>>>(
        nrows, rows, pos, vm, hydro, aux, prm.gs64, off, idx, prm, out_map, out);
  };
  const std::true_type yes;
  const std::false_type no;
  const bool recon = prm.use_recon && prm.use_visc;
  if (!prm.use_sph)
    run(no, yes, no);
  else if (recon && prm.use_disc)
    run(yes, yes, yes);
  else if (recon)
    run(yes, no, yes);
  else if (prm.use_disc)
    run(yes, yes, no);
  else
    run(yes, no, no);
}

void launch_gradients(int64_t nrows, const int64_t* rows, const double4* pos, const double4* vm,
                      const double4* acc, const int64_t* off, const int64_t* idx, int kid,
                      double cnorm, GradOut out, cudaStream_t st) {
  if (nrows <= 0) return;
  if (acc)
    count_launch(), k_gradients<int64_t, true><<<grid_for(nrows * 8), NB_THREADS, 0, st>>>(
        nrows, rows, pos, vm, acc, off, idx, kid, cnorm, out);
  else
    count_launch(), k_gradients<int64_t, false><<<grid_for(nrows * 8), NB_THREADS, 0, st>>>(
        nrows, rows, pos, vm, acc, off, idx, kid, cnorm, out);
}

void launch_shock_gradients(int64_t n, const double4* pos, const double4* vm, const double4* acc,
                            const int64_t* off, const int32_t* idx, int kid, double cnorm,
                            int recon, int recon_full, const uint8_t* live_mask,
                            const uint8_t* row_sorted, const int32_t* perm, GradOut out,
                            cudaStream_t st) {
  if (n <= 0) return;
  if (row_sorted)
    count_launch(), k_shock_grad<int32_t, true><<<grid_for(n * 8), NB_THREADS, 0, st>>>(
        n, pos, vm, acc, off, idx, kid, cnorm, recon, recon_full, live_mask, row_sorted, perm, out);
  else
    count_launch(), k_shock_grad<int32_t, false><<<grid_for(n * 8), NB_THREADS, 0, st>>>(
        n, pos, vm, acc, off, idx, kid, cnorm, recon, recon_full, live_mask, row_sorted, perm, out);
}

template void launch_density64<int64_t>(int64_t, const int64_t*, const double4*, const double*,
                                        const double*, const double*, const int64_t*,
                                        const int64_t*, DensityParams, const int32_t*, double*,
                                        double*, double*, int64_t*, int64_t*, int64_t*,
                                        cudaStream_t);
template void launch_density64<int32_t>(int64_t, const int64_t*, const double4*, const double*,
                                        const double*, const double*, const int64_t*,
                                        const int32_t*, DensityParams, const int32_t*, double*,
                                        double*, double*, int64_t*, int64_t*, int64_t*,
                                        cudaStream_t);
template void launch_forces64<int64_t>(int64_t, const int64_t*, const double4*, const double4*,
                                       const double4*, const double4*, const int64_t*,
                                       const int64_t*, ForceParams, const int32_t*, ForceOut,
                                       cudaStream_t);
template void launch_forces64<int32_t>(int64_t, const int64_t*, const double4*, const double4*,
                                       const double4*, const double4*, const int64_t*,
                                       const int32_t*, ForceParams, const int32_t*, ForceOut,
                                       cudaStream_t);

// ---------------------------------------------------------------- packing (caller order)
__global__ void k_pack_pos(int64_t n, const double* __restrict__ pos, const double* __restrict__ w,
                           double4* __restrict__ out) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  out[i] = make_double4(pos[3 * i], pos[3 * i + 1], pos[3 * i + 2], w ? w[i] : 0.0);
}

__global__ void k_pack_forces64(int64_t n, const double* __restrict__ pos,
                                const double* __restrict__ vel, const double* __restrict__ m,
                                const double* __restrict__ h, const double* __restrict__ rho,
                                const double* __restrict__ omega, const double* __restrict__ P,
                                const double* __restrict__ u, const double* __restrict__ cs,
                                const double* __restrict__ alpha, double4* __restrict__ pk0,
                                double4* __restrict__ pk1, double4* __restrict__ pk2,
                                double4* __restrict__ pk3) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double hi = h[i], ri = rho[i];
  pk0[i] = make_double4(pos[3 * i], pos[3 * i + 1], pos[3 * i + 2], hi);
  pk1[i] = make_double4(vel[3 * i], vel[3 * i + 1], vel[3 * i + 2], m[i]);
  pk2[i] = make_double4(1.0 / hi, ri, 1.0 / (omega[i] * ri * ri), P ? P[i] : 0.0);
  pk3[i] = make_double4(u ? u[i] : 0.0, cs ? cs[i] : 0.0, alpha ? alpha[i] : 0.0, 0.0);
}

__global__ void k_pack_sym(int64_t n, const double* __restrict__ gv, double4* __restrict__ out) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) store_sym(out + 2 * i, gv + 9 * i);
}

__global__ void k_pack_vm(int64_t n, const double* __restrict__ vel, const double* __restrict__ m,
                          double4* __restrict__ out) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  out[i] = make_double4(vel[3 * i], vel[3 * i + 1], vel[3 * i + 2], m[i]);
}


void pack_pos(int64_t n, const double* pos, const double* w, double4* out, cudaStream_t st) {
  if (n > 0) count_launch(), k_pack_pos<<<grid_for(n), NB_THREADS, 0, st>>>(n, pos, w, out);
}
void pack_forces64(int64_t n, const double* pos, const double* vel, const double* mass,
                   const double* h, const double* rho, const double* omega, const double* P,
                   const double* u, const double* cs, const double* alpha, double4* pk0,
                   double4* pk1, double4* pk2, double4* pk3, cudaStream_t st) {
  if (n > 0)
    count_launch(), k_pack_forces64<<<grid_for(n), NB_THREADS, 0, st>>>(
        n, pos, vel, mass, h, rho, omega, P, u, cs, alpha, pk0, pk1, pk2, pk3);
}
void pack_sym(int64_t n, const double* gv, double4* out, cudaStream_t st) {
  if (n > 0) count_launch(), k_pack_sym<<<grid_for(n), NB_THREADS, 0, st>>>(n, gv, out);
}
void pack_vm(int64_t n, const double* vel, const double* m, double4* out, cudaStream_t st) {
  if (n > 0) count_launch(), k_pack_vm<<<grid_for(n), NB_THREADS, 0, st>>>(n, vel, m, out);
}

}  // namespace nbk
