// FP64 O(N^2) direct summation on the GPU, the judge of every FMM result
// and the drop-in for NaiveUpdate::update (naive_update.cpp:9-35).
// Targets are split over blocks and sources over a second grid dimension;
// partial sums meet through FP64 atomics.
#include <algorithm>

#include "direct.cuh"

namespace fmm {

static constexpr int DS_THREADS = 256;

// One pair: f = the factor of -d in the force, pw = the potential term.
//
// Bound by the FP64 pipe (two issue cycles per warp instruction), so the
// divisions and square roots count: NaiveUpdate's m / ((r^2 + 1e-4) r) is one
// reciprocal square root, of r^2 (r^2 + 1e-4)^2, while that product stays
// well inside the FP64 range (r^2 in [2^-300, 2^300), tested on the exponent
// bits; outside, the two divisions and the square root), and nothing is
// computed for a potential that is not asked for.  The mass is the last
// factor of both, so that a force that leaves the range does not take a
// potential with it that is still inside.
template <int DIM, int SOFT, bool POT>
__device__ __forceinline__ void direct_pair(double r2, double w, double eps2, double &f, double &pw) {
  if (DIM == 3) {
    if (SOFT == FMM_SOFT_NAIVE_REF) {
      const double s = r2 + 1.0e-4;
      const unsigned ex = (unsigned)__double2hiint(r2) >> 20;
      if (ex - 723u < 600u) {
        const double g = rsqrt(r2 * s * s);
        f = w * g;
        if (POT) pw = w * (g * s);
      } else {
        const double r = sqrt(r2);
        f = w / (s * r);
        if (POT) pw = w / r;
      }
    } else {
      const double ir = rsqrt(r2 + eps2);
      pw = w * ir;
      f = pw * ir * ir;
    }
  } else {
    const double rr = SOFT == FMM_SOFT_NAIVE_REF ? r2 + 1.0e-4 : r2 + eps2;
    f = w / rr;
    if (POT) pw = -0.5 * w * log(rr);
  }
}

// A thread sums one target over the block's share of the sources, staged
// DS_THREADS at a time, four pairs unrolled to fill the FP64 pipe's latency.
// (Two targets per thread, two pairs unrolled: all pairs of 20,011 particles
// 0.70 against 0.60 ms with NaiveUpdate's softening and 0.62 against 0.56 with
// Plummer's, 4096 targets of 2^20 6.4 against 6.0 ms, and idle threads in every
// call whose targets are no multiple of 512: 256 of 2^20 0.74 against 0.40.)
// The test for j == i runs only in the stages that hold one of the warp's own
// targets; a warp without targets only stages.
template <int DIM, int SOFT, bool POT>
__global__ void __launch_bounds__(DS_THREADS) k_direct(const double *pos, const double *mass, int64_t n,
                                                       const int64_t *targets, int64_t nt, double eps2, int64_t chunk,
                                                       double G, double *acc, double *pot) {
  __shared__ double4 sp[DS_THREADS];
  const int64_t ti = (int64_t)blockIdx.x * DS_THREADS + threadIdx.x;
  const int64_t me = ti < nt ? (targets ? targets[ti] : ti) : -1;
  double x[3], a[3], ph = 0.0;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    x[k] = me >= 0 && k < DIM ? pos[me * DIM + k] : 0.0;
    a[k] = 0.0;
  }
  const bool busy = __any_sync(0xffffffffu, me >= 0);
  const int64_t j0 = (int64_t)blockIdx.y * chunk, j1 = min(n, j0 + chunk);
  auto sum = [&](int cnt, int64_t jb, bool own) {
#pragma unroll 4
    for (int k = 0; k < cnt; ++k) {
      const double4 q = sp[k];
      if (own && jb + k == me) continue;
      const double dx = x[0] - q.x, dy = x[1] - q.y, dz = DIM == 3 ? x[2] - q.z : 0.0;
      const double r2 = DIM == 3 ? dx * dx + dy * dy + dz * dz : dx * dx + dy * dy;
      double f, pw = 0.0;
      direct_pair<DIM, SOFT, POT>(r2, q.w, eps2, f, pw);
      a[0] -= f * dx;
      a[1] -= f * dy;
      if (DIM == 3) a[2] -= f * dz;
      if (POT) ph += pw;
    }
  };
  for (int64_t jb = j0; jb < j1; jb += DS_THREADS) {
    const int64_t j = jb + threadIdx.x;
    if (j < j1)
      sp[threadIdx.x] = make_double4(pos[j * DIM], pos[j * DIM + 1], DIM == 3 ? pos[j * DIM + 2] : 0.0, mass[j]);
    __syncthreads();
    const int cnt = (int)min((int64_t)DS_THREADS, j1 - jb);
    if (__any_sync(0xffffffffu, me >= jb && me < jb + DS_THREADS)) sum(cnt, jb, true);
    else if (busy) sum(cnt, jb, false);
    __syncthreads();
  }
  if (ti >= nt) return;
#pragma unroll
  for (int k = 0; k < DIM; ++k) {
    if (gridDim.y == 1) acc[ti * DIM + k] = G * a[k];
    else atomicAdd(&acc[ti * DIM + k], G * a[k]);
  }
  if (POT) {
    if (gridDim.y == 1) pot[ti] = G * ph;
    else atomicAdd(&pot[ti], G * ph);
  }
}

int direct_sum(const double *d_pos, const double *d_mass, int64_t n, const int64_t *d_targets, int64_t nt, int dim,
               double eps2, int soft_mode, double G, double *d_acc, double *d_pot, cudaStream_t st, int64_t &launches) {
  if (nt <= 0 || n <= 0) return FMM_OK;
  const int64_t bx = (nt + DS_THREADS - 1) / DS_THREADS;
  // source shares for about 16 blocks per SM, of at least two stages (shorter shares also round less)
  const int64_t by = std::max<int64_t>(
      1, std::min<int64_t>({(148 * 16 + bx - 1) / bx, (n + 2 * DS_THREADS - 1) / (2 * DS_THREADS), 65535}));
  const int64_t chunk = (n + by - 1) / by;
  if (by > 1) {
    cudaMemsetAsync(d_acc, 0, sizeof(double) * nt * dim, st);
    if (d_pot) cudaMemsetAsync(d_pot, 0, sizeof(double) * nt, st);
  }
  const dim3 grid((unsigned)bx, (unsigned)by);
  auto run = [&](auto kern) {
    kern<<<grid, DS_THREADS, 0, st>>>(d_pos, d_mass, n, d_targets, nt, eps2, chunk, G, d_acc, d_pot);
  };
  const bool naive = soft_mode == FMM_SOFT_NAIVE_REF;
  constexpr int P = FMM_SOFT_PLUMMER, N = FMM_SOFT_NAIVE_REF;
  if (dim == 3) {
    if (d_pot) naive ? run(k_direct<3, N, true>) : run(k_direct<3, P, true>);
    else naive ? run(k_direct<3, N, false>) : run(k_direct<3, P, false>);
  } else {
    if (d_pot) naive ? run(k_direct<2, N, true>) : run(k_direct<2, P, true>);
    else naive ? run(k_direct<2, N, false>) : run(k_direct<2, P, false>);
  }
  launches += 1;
  return cudaGetLastError() == cudaSuccess ? FMM_OK : FMM_ERR_CUDA;
}

// ---------------------------------------------------------- integrators
// SyplecticEuler::integrate (symplectic_euler.cpp:10-14): v += dt a; x += dt v.
__global__ void k_se_update(double *x, double *v, const double *a, int64_t nd, double dt) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nd) return;
  double vv = v[i] + dt * a[i];
  v[i] = vv;
  x[i] += dt * vv;
}

// Classical RK4 for x' = v, v' = a(x).  From stage s (position x_s,
// velocity v_s, acceleration a_s = a(x_s); x_1 = x0, v_1 = v0):
//   v_{s+1} = v0 + c_s dt a_s,   x_{s+1} = x0 + c_s dt v_s,   c = 1/2, 1/2, 1
// and finally
//   v += dt/6 (a1 + 2a2 + 2a3 + a4),  x += dt/6 (v1 + 2v2 + 2v3 + v4),
// which is what runge_kutta_4.cpp:10-93 sets out to compute.  `cdt` is
// c_s * dt and `wprev` the weight of stage s in the final sums.
__global__ void k_rk4_stage(const double *x0, const double *v0, const double *a_prev, double *xs, double *vs,
                            double *asum, double *vsum, int64_t nd, double cdt, double wprev, int first) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nd) return;
  double vprev = first ? v0[i] : vs[i];
  double as = first ? 0.0 : asum[i], vsm = first ? 0.0 : vsum[i];
  asum[i] = as + wprev * a_prev[i];
  vsum[i] = vsm + wprev * vprev;
  vs[i] = v0[i] + cdt * a_prev[i];
  xs[i] = x0[i] + cdt * vprev;
}

__global__ void k_rk4_final(double *x, double *v, const double *a4, const double *v4, const double *asum,
                            const double *vsum, int64_t nd, double dt) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nd) return;
  double as = asum[i] + a4[i], vsm = vsum[i] + v4[i];
  v[i] += dt / 6.0 * as;
  x[i] += dt / 6.0 * vsm;
}

void se_update(double *x, double *v, const double *a, int64_t nd, double dt, cudaStream_t st, int64_t &launches) {
  k_se_update<<<(int)((nd + 255) / 256), 256, 0, st>>>(x, v, a, nd, dt);
  launches += 1;
}

void rk4_stage(const double *x0, const double *v0, const double *a_prev, double *xs, double *vs, double *asum,
               double *vsum, int64_t nd, double c, double wprev, int first, cudaStream_t st, int64_t &launches) {
  k_rk4_stage<<<(int)((nd + 255) / 256), 256, 0, st>>>(x0, v0, a_prev, xs, vs, asum, vsum, nd, c, wprev, first);
  launches += 1;
}

void rk4_final(double *x, double *v, const double *a4, const double *v4, const double *asum, const double *vsum,
               int64_t nd, double dt, cudaStream_t st, int64_t &launches) {
  k_rk4_final<<<(int)((nd + 255) / 256), 256, 0, st>>>(x, v, a4, v4, asum, vsum, nd, dt);
  launches += 1;
}

}  // namespace fmm
