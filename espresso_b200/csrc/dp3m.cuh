// Dipolar P3M kernels (magnetostatics/dp3m.cpp, p3m/influence_function_dipolar.hpp).
//
// The three dipole-moment components are assigned to three meshes with the
// charge-assignment kernels (three charges in one particle record) and
// transformed forward with the z and y passes of the
// charge path.  This file adds what is specific to point dipoles:
//  * the dipolar influence functions G_energy (S = 2) and G_force (S = 3)
//    on the r2c half mesh, and the aliasing sum of the energy correction;
//  * a forward x pass that forms mu(k) . d_op(k) once per point from two
//    transforms and accumulates the k-space energy, and a backward one that
//    emits the five spectra from which the y and z passes form the three
//    torque fields and the six entries of the symmetric force-field tensor;
//  * the per-particle combination of the interpolated fields into forces
//    and torques, and the real-space pair kernel over the Verlet lists.
#pragma once

#include "fft.cuh"
#include "p3m_kernels.cuh"
#include "pair.cuh"

namespace p3mx {

// Resident blocks per SM of the pair kernels (Engine::pair_lanes): FP32, FP32 with
// energies, FP64.
constexpr int kDpPairBlocks32 = 3, kDpPairBlocks32Ev = 2, kDpPairBlocks64 = 2;

// calc_meshift (p3m/common.hpp:248-264): index shift of the influence
// function (M/2 -> -M/2) and of the differential operator (M/2 -> 0).
__host__ __device__ inline int dp_shift(int i, int m) { return (i < m / 2) ? i : i - m; }
__host__ __device__ inline int dp_dop(int i, int m) { return (i == m / 2) ? 0 : dp_shift(i, m); }

// G_opt_dipolar<S> for m = 0 aliasing at mesh index (x, y, z) of a cubic
// mesh M, box L (influence_function_dipolar.hpp:62-130): numerator
// U^2 exp(-pi^2 |n|^2 / alpha_L^2) / |n|^2 (d_op . n)^S, denominator
// |d_op|^(2S) (U^2)^2, zero at the points whose indices are all multiples
// of M/2, scaled by 2 M^3 / L^2.  Both S = 2 (energy) and S = 3 (force).
__device__ inline void dp3m_g(int x, int y, int z, int M, double L, double alpha, int cao,
                              double &g2, double &g3) {
  g2 = g3 = 0.0;
  int const h = M / 2;
  if (x % h == 0 && y % h == 0 && z % h == 0)
    return;
  int const sx = dp_shift(x, M), sy = dp_shift(y, M), sz = dp_shift(z, M);
  int const dx = dp_dop(x, M), dy = dp_dop(y, M), dz = dp_dop(z, M);
  double const mi = 1.0 / M;
  double const u = sinc_d(sx * mi) * sinc_d(sy * mi) * sinc_d(sz * mi);
  double const u2 = pow(u, 2.0 * cao);
  double const n2 = static_cast<double>(sx * sx + sy * sy + sz * sz);
  double const pa = kPi / (alpha * L);
  double const ex = pa * pa * n2;
  if (!(ex < 30.0))
    return;
  double const dn = static_cast<double>(dx * sx + dy * sy + dz * sz);
  double const dd = static_cast<double>(dx * dx + dy * dy + dz * dz);
  double const base = u2 * exp(-ex) / n2;
  double const fac = 2.0 * static_cast<double>(M) * M * M / (L * L);
  g2 = fac * (base * dn * dn) / (dd * dd * u2 * u2);
  g3 = fac * (base * dn * dn * dn) / (dd * dd * dd * u2 * u2);
}

// Both influence functions on the r2c half mesh (same point layout and
// block table as k_influence); computed in FP64, stored in Real.
template <typename Real>
__global__ void k_dp3m_influence(const RepGeom *__restrict__ reps, const int2 *__restrict__ blk,
                                 Real *__restrict__ g_e, Real *__restrict__ g_f) {
  int2 const bk = blk[blockIdx.x];
  RepGeom const &G = reps[bk.x];
  int const M = G.mesh[0];
  long long const local = static_cast<long long>(bk.y) * blockDim.x + threadIdx.x;
  long long const csize = static_cast<long long>(M) * M * G.hp;
  if (local >= csize)
    return;
  int const kz = static_cast<int>(local % G.hp);
  int const y = static_cast<int>((local / G.hp) % M);
  int const x = static_cast<int>(local / (static_cast<long long>(M) * G.hp));
  double g2 = 0.0, g3 = 0.0;
  if (kz <= M / 2)
    dp3m_g(x, y, kz, M, G.box[0], G.alpha, G.cao, g2, g3);
  g_e[G.km_off + local] = static_cast<Real>(g2);
  g_f[G.km_off + local] = static_cast<Real>(g3);
}

// Per-block partials of sum G_energy U2s |d_op|^2 over the full mesh, the
// mesh sum of calc_average_self_energy_k_space (dp3m.cpp:320-360): U2s the
// product of sinc(shift/M + m M)^(2 cao) summed over m in [-1, 1]^3 (the
// reference's aliasing loop steps the sinc argument by whole meshes).  A
// fixed grid-stride assignment of points to threads and fixed reductions:
// deterministic.
__global__ void k_dp3m_self_sum(int M, double L, double alpha, int cao,
                                double *__restrict__ partials) {
  long long const total = static_cast<long long>(M) * M * M;
  double acc = 0.0;
  for (long long p = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; p < total;
       p += static_cast<long long>(gridDim.x) * blockDim.x) {
    int const z = static_cast<int>(p % M), y = static_cast<int>((p / M) % M),
              x = static_cast<int>(p / (static_cast<long long>(M) * M));
    double g2, g3;
    dp3m_g(x, y, z, M, L, alpha, cao, g2, g3);
    if (g2 == 0.0)
      continue;
    double const mi = 1.0 / M;
    int const s[3] = {dp_shift(x, M), dp_shift(y, M), dp_shift(z, M)};
    double sn[3][3];
#pragma unroll
    for (int d = 0; d < 3; ++d)
#pragma unroll
      for (int m = -1; m <= 1; ++m)
        sn[d][m + 1] = sinc_d(s[d] * mi + m * M);
    double u2s = 0.0;
    for (int m0 = 0; m0 < 3; ++m0)
      for (int m1 = 0; m1 < 3; ++m1)
        for (int m2 = 0; m2 < 3; ++m2)
          u2s += pow(sn[0][m0] * sn[1][m1] * sn[2][m2], 2.0 * cao);
    int const dx = dp_dop(x, M), dy = dp_dop(y, M), dz = dp_dop(z, M);
    acc += g2 * u2s * static_cast<double>(dx * dx + dy * dy + dz * dz);
  }
  __shared__ double red[32];
  int const lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int o = 16; o > 0; o >>= 1)
    acc += __shfl_down_sync(0xffffffffu, acc, o);
  if (lane == 0)
    red[wid] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < (blockDim.x >> 5); ++w)
      s += red[w];
    partials[blockIdx.x] = s;
  }
}

// Per-block partials of the dipolar k-space error sum of the tuner
// (dp3m_k_space_error and dp3m_tune_aliasing_sums, dp3m.cpp:680-740, with
// the m = 0 aliasing term): over n in [-M/2, M/2)^3 without n = 0,
//   d = ex^2 |n|^2 - (U2 ex |n|^4 / cs)^2 / |n|^6,  ex = exp(-(pi/alpha_L)^2 |n|^2),
// cs the product of the analytic cotangent sums, added where d > 0 and
// |d / (ex^2 |n|^2)| > 1e-14.  Fixed grid-stride assignment and reductions.
__global__ void k_dp3m_ks_error(int M, int cao, double alpha_L, double *__restrict__ partials) {
  long long const total = static_cast<long long>(M) * M * M;
  double const mi = 1.0 / M;
  double const f1 = (kPi / alpha_L) * (kPi / alpha_L);
  double acc = 0.0;
  for (long long t = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; t < total;
       t += static_cast<long long>(gridDim.x) * blockDim.x) {
    int const nz = static_cast<int>(t % M) - M / 2;
    int const ny = static_cast<int>((t / M) % M) - M / 2;
    int const nx = static_cast<int>(t / (static_cast<long long>(M) * M)) - M / 2;
    if (nx == 0 && ny == 0 && nz == 0)
      continue;
    double const n2 = double(nx) * nx + double(ny) * ny + double(nz) * nz;
    double const cs = cot_sum(cao, nx, mi) * cot_sum(cao, ny, mi) * cot_sum(cao, nz, mi);
    double const ex = exp(-f1 * n2);
    double const u2 = pow(sinc_d(nx * mi) * sinc_d(ny * mi) * sinc_d(nz * mi), 2.0 * cao);
    double const a1 = ex * ex * n2;
    double const a2 = u2 * ex * (n2 * n2 * n2) / n2;
    double const d = a1 - (a2 / cs) * (a2 / cs) / (n2 * n2 * n2);
    if (d > 0.0 && fabs(d / a1) > 1e-14)
      acc += d;
  }
  __shared__ double red[32];
  for (int o = 16; o > 0; o >>= 1)
    acc += __shfl_down_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0)
    red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < (blockDim.x >> 5); ++w)
      s += red[w];
    partials[blockIdx.x] = s;
  }
}

// Dipole moments (AoS, 3 per particle) -> the list selector
// sel = 1 for a particle with a non-zero moment (0 otherwise: it has no
// real-space partners), a flag set when a selector changed since the last
// call, and per-block partials {n_dipoles, sum mu^2, M_x, M_y, M_z}.
__global__ void k_dp3m_prepare(long long n, const double *__restrict__ mu,
                               double *__restrict__ sel,
                               int *__restrict__ sel_changed, double *__restrict__ partials) {
  double acc[5] = {0, 0, 0, 0, 0};
  long long const i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < n) {
    double const m0 = mu[3 * i], m1 = mu[3 * i + 1], m2 = mu[3 * i + 2];
    double const m2s = m0 * m0 + m1 * m1 + m2 * m2;
    double const s = (m2s != 0.0) ? 1.0 : 0.0;
    if (sel[i] != s) {
      sel[i] = s;
      atomicOr(sel_changed, 1);
    }
    if (m2s != 0.0) {
      acc[0] = 1.0;
      acc[1] = m2s;
      acc[2] = m0;
      acc[3] = m1;
      acc[4] = m2;
    }
  }
  __shared__ double red[5][8];
  int const lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    double v = acc[k];
    for (int o = 16; o > 0; o >>= 1)
      v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0)
      red[k][wid] = v;
  }
  __syncthreads();
  if (threadIdx.x < 5) {
    double s = 0.0;
    for (int w = 0; w < (blockDim.x >> 5); ++w)
      s += red[threadIdx.x][w];
    partials[static_cast<long long>(blockIdx.x) * 5 + threadIdx.x] = s;
  }
}

// Fixed-order sum of nblk rows of `width` partials: one warp per column
// (launched with 32 * width threads), lane l summing rows l, l + 32, ...,
// then a fixed shuffle tree (deterministic; the loads of a lane are
// independent, not one serial chain per column).
__global__ void k_dp3m_sum_rows(const double *__restrict__ partials, int nblk, int width,
                                double *__restrict__ out) {
  int const k = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (k >= width)
    return;
  double s = 0.0;
  for (int b = lane; b < nblk; b += 32)
    s += partials[static_cast<long long>(b) * width + k];
  for (int o = 16; o > 0; o >>= 1)
    s += __shfl_down_sync(0xffffffffu, s, o);
  if (lane == 0)
    out[k] = s;
}

// ---- x passes of the dipolar k-space operator -----------------------------
// Forward (per block: one ky, a tile of kz, the block table of the charge x
// pass): mk = sum_d d_op_d F_d in x-transformed space from the three
// components F_d.  d_op_y and d_op_z are constant along x, so
//   mk = d_op_x FFT_x(F_x) + FFT_x(d_op_y F_y + d_op_z F_z):
// two transforms; mk replaces component x in place (each block rewrites only
// the lines it read).
// EV: per-block partial of the k-space energy sum G_energy |mk|^2 with the
// Hermitian weights of the half mesh (1 at kz = 0 and M/2, else 2).
// Shared memory: 2 x tile staged lines of line_ld(M) (3 x for KIND 0: a
// scratch buffer), twiddles (M): the charge x pass's layout.
template <typename Real, bool EV, int KIND>
__global__ void __launch_bounds__(256, sizeof(Real) == 4 && KIND ? 3 : 2)
k_fft_x_dp3m(const RepGeom *__restrict__ reps, const Blk *__restrict__ blks,
             typename CplxOf<Real>::type *__restrict__ comp_hat, long long fstride,
             const Real *__restrict__ g_e, int tile, double *__restrict__ partials,
             const typename CplxOf<Real>::type *__restrict__ twtab) {
  using C = typename CplxOf<Real>::type;
  pdl_enter();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Blk const bk = blks[blockIdx.x];
  RepGeom const &G = reps[bk.rep];
  int const M0 = G.mesh[0], M1 = G.mesh[1], M2 = G.mesh[2];
  int const y = bk.a, kz0 = bk.b;
  int const T = bk.w;
  int const ld = line_ld(M0);
  int const L = tile * ld;
  C *a = reinterpret_cast<C *>(smem_raw);
  C *b = a + L;
  C *c = KIND ? nullptr : b + L;
  C *tw = a + (KIND ? 2 : 3) * L;
  load_twiddles(tw, twtab, G.plan[0]);
  long long const stride_x = static_cast<long long>(M1) * G.hp;
  int const tq = threadIdx.x & 15, xq = threadIdx.x >> 4;
  bool const col = tq < T;
  int const kz = kz0 + tq;
  long long const base = G.km_off + static_cast<long long>(y) * G.hp + kz;
  Real const dop_y = static_cast<Real>(dp_dop(y, M1)), dop_z = static_cast<Real>(dp_dop(kz, M2));
  // 4 rows of the three components in flight, unconditional as in the y pass
  int const rows = col ? (M0 - xq + 15) >> 4 : 0;
  const C *src = comp_hat + base - tq + min(tq, T - 1);
  for (int u0 = 0; u0 < rows; u0 += 4) {
    C v[3][4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const C *p = src + min(xq + 16 * (u0 + u), M0 - 1) * stride_x;
#pragma unroll
      for (int d = 0; d < 3; ++d)
        v[d][u] = p[d * fstride];
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (u0 + u < rows) {
        int const at = tq * ld + xq + 17 * (u0 + u);
        a[at] = v[0][u];
        b[at] = C{dop_y * v[1][u].x + dop_z * v[2][u].x, dop_y * v[1][u].y + dop_z * v[2][u].y};
      }
  }
  __syncthreads();
  C *ra = fft_lines<KIND, true>(a, c, T, ld, G.plan[0], tw);
  // with KIND 0: the buffer that the first transform left free
  C *rb = fft_lines<KIND, true>(b, ra == a ? c : a, T, ld, G.plan[0], tw);
  double acc = 0.0;
  double const wgt = (kz == 0 || kz == M2 / 2) ? 1.0 : 2.0;
  for (int x = xq; col && x < M0; x += 16) {
    Real const op = static_cast<Real>(dp_dop(x, M0));
    C const u = ra[tq * ld + pix(x)], v = rb[tq * ld + pix(x)];
    C const m = C{op * u.x + v.x, op * u.y + v.y};
    long long const at = base + x * stride_x;
    comp_hat[at] = m;
    if constexpr (EV)
      acc += wgt * static_cast<double>(g_e[at]) *
             (static_cast<double>(m.x) * m.x + static_cast<double>(m.y) * m.y);
  }
  if constexpr (EV) {
    __shared__ double red[8];
    int const lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int o = 16; o > 0; o >>= 1)
      acc += __shfl_down_sync(0xffffffffu, acc, o);
    if (lane == 0)
      red[wid] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
      double s = 0.0;
      for (int w = 0; w < (blockDim.x >> 5); ++w)
        s += red[w];
      partials[blockIdx.x] = s;
    }
  }
}

// Backward: block 5 k + o forms spectrum o of tile k from mk and transforms it
// along x:
//   o = 0, 1:    d_op_x^p G_energy mk,     p = 1, 0  (torques, AssignTorques,
//                dp3m.cpp:372-395)
//   o = 2, 3, 4: -i d_op_x^p G_force mk,   p = 2, 1, 0  (forces, AssignForces,
//                dp3m.cpp:396-430)
// d_op along y and z commutes with the x transform: the y and z passes apply
// its powers (dp_y_pass, dp_z_pass), so 5 backward x transforms serve the
// three torque fields and the six entries of the symmetric force-field tensor.
// Shared memory: the forward pass's.
template <typename Real, int KIND>
__global__ void __launch_bounds__(256, sizeof(Real) == 4 && KIND ? 3 : 2)
k_fft_x_dp3m_inv(const RepGeom *__restrict__ reps, const Blk *__restrict__ blks,
                 const typename CplxOf<Real>::type *__restrict__ mk_hat, long long fstride,
                 const Real *__restrict__ g_e, const Real *__restrict__ g_f,
                 typename CplxOf<Real>::type *__restrict__ field0, int tile,
                 const typename CplxOf<Real>::type *__restrict__ twtab) {
  using C = typename CplxOf<Real>::type;
  pdl_enter();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  int const blk = blockIdx.x / 5, o = blockIdx.x - 5 * blk;
  Blk const bk = blks[blk];
  RepGeom const &G = reps[bk.rep];
  int const M0 = G.mesh[0], M1 = G.mesh[1];
  int const T = bk.w;
  int const ld = line_ld(M0);
  C *a = reinterpret_cast<C *>(smem_raw);
  C *b = KIND ? nullptr : a + tile * ld;
  C *tw = a + (KIND ? 2 : 3) * tile * ld;
  load_twiddles(tw, twtab, G.plan[0]);
  long long const stride_x = static_cast<long long>(M1) * G.hp;
  int const tq = threadIdx.x & 15, xq = threadIdx.x >> 4;
  bool const col = tq < T;
  long long const base = G.km_off + static_cast<long long>(bk.a) * G.hp + bk.b + tq;
  bool const tor = o < 2;
  int const p = tor ? 1 - o : 4 - o; // power of d_op_x
  const Real *g = tor ? g_e : g_f;
  // 8 rows in flight, unconditional as in the y pass
  int const rows = col ? (M0 - xq + 15) >> 4 : 0;
  long long const first = base - tq + min(tq, T - 1);
  for (int u0 = 0; u0 < rows; u0 += 8) {
    C v[8];
    Real gv[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      long long const at = first + min(xq + 16 * (u0 + u), M0 - 1) * stride_x;
      v[u] = mk_hat[at];
      gv[u] = g[at];
    }
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (u0 + u < rows) {
        int const dx = dp_dop(xq + 16 * (u0 + u), M0);
        Real const c = static_cast<Real>(p == 0 ? 1 : (p == 1 ? dx : dx * dx)) * gv[u];
        // c mk, or -i c mk; real and imaginary parts swapped (backward)
        a[tq * ld + xq + 17 * (u0 + u)] = tor ? C{c * v[u].y, c * v[u].x} : C{-c * v[u].x, c * v[u].y};
      }
  }
  __syncthreads();
  C const *res = fft_lines<KIND, true>(a, b, T, ld, G.plan[0], tw) + tq * ld + xq;
  C *q = field0 + fstride * o + base + xq * stride_x;
#pragma unroll 4
  for (int u = 0; u < rows; ++u)
    q[u * 16 * stride_x] = cswap(res[17 * u]);
}

// Backward y pass over the x pass's five arrays: nine fields (E_x, E_y, E_z in
// arrays 0, 5, 6; the tensor's xx, xy, xz, yy, yz, zz in 2, 7, 8, 9, 10, 11);
// and their backward z pass, sets (E_x, E_y, E_z), (xx, xy, xz), (yy, yz, zz).
constexpr int kDipoleSpectra = 12;
inline YPass dp_y_pass() {
  return YPass{9, {0, 1, 1, 2, 3, 3, 4, 4, 4}, {0, 5, 6, 2, 7, 8, 9, 10, 11},
               {0, 1, 0, 0, 1, 0, 2, 1, 0}};
}
// (of the sets from `set` on)
inline ZPass dp_z_pass(int set) {
  constexpr signed char arr[9] = {0, 5, 6, 2, 7, 8, 9, 10, 11}, pw[9] = {0, 0, 1, 0, 0, 1, 0, 1, 2};
  ZPass z{};
  for (int k = 3 * set; k < 9; ++k) {
    z.arr[k - 3 * set] = arr[k];
    z.pw[k - 3 * set] = pw[k];
  }
  return z;
}

// Forces and torques from the interpolated fields (AoS, 3 per particle):
//   tau = -pt mu x E_t                        (dp3m.cpp:380-395)
//   F_d = pf sum_c mu_c E_f(d, c)             (dp3m.cpp:410-430)
// with et = E_t, efa = (E_xx, E_xy, E_xz), efb = (E_yy, E_yz, E_zz); for a
// non-metallic boundary (ps != 0) the surface-term torque
// tau -= ps mu x M, M = the total moment at sums[2..4] (calc_surface_term,
// dp3m.cpp:452-510).
__global__ void k_dp3m_combine(long long n, const double *__restrict__ mu,
                               const double *__restrict__ et, const double *__restrict__ efa,
                               const double *__restrict__ efb, double pt, double pf, double ps,
                               const double *__restrict__ sums, double *__restrict__ f,
                               double *__restrict__ tq, int overwrite) {
  long long const i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n)
    return;
  double const m0 = mu[3 * i], m1 = mu[3 * i + 1], m2 = mu[3 * i + 2];
  double e0 = pt * et[3 * i], e1 = pt * et[3 * i + 1], e2 = pt * et[3 * i + 2];
  if (ps != 0.0) {
    e0 += ps * sums[2];
    e1 += ps * sums[3];
    e2 += ps * sums[4];
  }
  double const t0 = -(m1 * e2 - m2 * e1);
  double const t1 = -(m2 * e0 - m0 * e2);
  double const t2 = -(m0 * e1 - m1 * e0);
  double const xx = efa[3 * i], xy = efa[3 * i + 1], xz = efa[3 * i + 2];
  double const yy = efb[3 * i], yz = efb[3 * i + 1], zz = efb[3 * i + 2];
  double const f0 = pf * (m0 * xx + m1 * xy + m2 * xz);
  double const f1 = pf * (m0 * xy + m1 * yy + m2 * yz);
  double const f2 = pf * (m0 * xz + m1 * yz + m2 * zz);
  if (overwrite) {
    f[3 * i] = f0;
    f[3 * i + 1] = f1;
    f[3 * i + 2] = f2;
    tq[3 * i] = t0;
    tq[3 * i + 1] = t1;
    tq[3 * i + 2] = t2;
  } else {
    f[3 * i] += f0;
    f[3 * i + 1] += f1;
    f[3 * i + 2] += f2;
    tq[3 * i] += t0;
    tq[3 * i + 1] += t1;
    tq[3 * i + 2] += t2;
  }
}

// Dipole moments in cell-sorted order (the pair kernel's partner reads):
// FP64 records, or FP32 records in the same buffer for k_dp3m_pairs_rel.
__global__ void k_dp3m_sort_mu(long long n, const int *__restrict__ perm,
                               const double *__restrict__ mu, double4 *__restrict__ smu,
                               int fp32) {
  long long const s = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (s >= n)
    return;
  int const i = perm[s];
  if (fp32)
    reinterpret_cast<float4 *>(smu)[s] =
        make_float4(static_cast<float>(mu[3 * i]), static_cast<float>(mu[3 * i + 1]),
                    static_cast<float>(mu[3 * i + 2]), 0.f);
  else
    smu[s] = make_double4(mu[3 * i], mu[3 * i + 1], mu[3 * i + 2], 0.0);
}

// Real-space dipole-dipole energy, force and torque over the Verlet lists
// (dp3m.hpp:142-232, pair_force / pair_energy): with d = x_i - x_j and
//   B = (erfc(a r) / r + 2a/sqrt(pi) exp(-a^2 r^2)) / r^2
//   C = (3 B + 2 a^2 (2a/sqrt(pi)) exp(-a^2 r^2)) / r^2
//   D = (5 C + 4 a^4 (2a/sqrt(pi)) exp(-a^2 r^2)) / r^2
//   E   = mu_i.mu_j B - (mu_i.d)(mu_j.d) C
//   F_i = (mu_i.mu_j) C d + (mu_j.d) C mu_i + (mu_i.d) C mu_j - (mu_i.d)(mu_j.d) D d
//   T_i = -mu_i x mu_j B + (mu_i x d)(mu_j.d) C
// for r < r_cut; erfc(a r) exp(a^2 r^2) by Abramowitz & Stegun 7.1.26 when
// the target accuracy is above 5e-6, else erfc itself.  The lists hold both
// directions of every pair, so each particle sums its own force and torque
// (no atomics, a fixed order: deterministic); the energy takes half of
// every ordered pair.  LPP lanes share a cell-sorted particle (whole groups
// of 8 entries each, as k_pair_forces_rel): 16 384 dipoles fill the GPU only
// with 8 lanes each.

// The particle's own moment leaves the sums:
//   F = sum (cd d + q mu_j) + mu_i sum s,  T = mu_i x sum (s d - B mu_j)
// with cd = (mu_i.mu_j) C - (mu_i.d)(mu_j.d) D, s = (mu_j.d) C, q = (mu_i.d) C:
// seven sums, nine operations per pair fewer than six sums of whole terms.
// Sums w of the LPP lanes of a particle (force part, torque part, sum s), its
// outputs (times pref; f may be nullptr) and the block's energy partial.
template <bool EV, int LPP>
__device__ inline void dp_pairs_finish(double (&w)[7], double mx, double my, double mz,
                                       double energy, double pref, bool active,
                                       long long a, const int *__restrict__ perm,
                                       double *__restrict__ f, double *__restrict__ tq,
                                       int overwrite, double *__restrict__ partials) {
#pragma unroll
  for (int o = 1; o < LPP; o <<= 1)
#pragma unroll
    for (int k = 0; k < 7; ++k)
      w[k] += __shfl_xor_sync(0xffffffffu, w[k], o);
  double const v[6] = {w[0] + mx * w[6], w[1] + my * w[6], w[2] + mz * w[6],
                       my * w[5] - mz * w[4], mz * w[3] - mx * w[5], mx * w[4] - my * w[3]};
  if (f && active && threadIdx.x % LPP == 0) {
    int const i = perm[a];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      if (overwrite) {
        f[3 * i + k] = pref * v[k];
        tq[3 * i + k] = pref * v[3 + k];
      } else {
        f[3 * i + k] += pref * v[k];
        tq[3 * i + k] += pref * v[3 + k];
      }
    }
  }
  if constexpr (EV) {
    double const e[1] = {pref * energy};
    block_halves<1>(e, 1, [](int) { return 0; }, partials);
  }
}

template <bool EV, int LPP>
__global__ void __launch_bounds__(256, kDpPairBlocks64)
k_dp3m_pairs(const RepGeom *__restrict__ reps, const int2 *__restrict__ blk,
             const double4 *__restrict__ spq, const double4 *__restrict__ smu,
             const int *__restrict__ perm, const int *__restrict__ nb,
             const int *__restrict__ nb_cnt, double pref, int exact_erfc,
             double *__restrict__ f, double *__restrict__ tq, int overwrite,
             double *__restrict__ partials) {
  int2 const bk = blk[blockIdx.x / LPP];
  RepGeom const &G = reps[bk.x];
  int const sub = threadIdx.x % LPP;
  long long const la = static_cast<long long>(bk.y) * 256 + (blockIdx.x % LPP) * (256 / LPP) +
                       threadIdx.x / LPP;
  bool const active = la < G.np;
  long long const a = G.p0 + la;
  double energy = 0.0;
  double s7[7] = {0, 0, 0, 0, 0, 0, 0};
  double4 const ma = active ? smu[a] : make_double4(0.0, 0.0, 0.0, 0.0);
  if (active) {
    double4 const pa = spq[a];
    double const alpha = G.alpha, rc = G.r_cut;
    double const coeff = 2.0 * alpha / sqrt(kPi);
    double const a2 = alpha * alpha;
    int const cw = nb_cnt[a];
    int const ga = (nb_count_a(cw) + 7) >> 3, gt = ga + ((nb_count_b(cw) + 7) >> 3);
    const int *nbp = nb + nb_base(G.nb_off, G.max_nb, la);
    int const ngroups = G.max_nb >> 3;
    const double4 *pos = spq + G.p0, *mom = smu + G.p0;
    auto group = [&](int v) {
      int const grp = v < ga ? v : ngroups - 1 - (v - ga);
      return nbp + (static_cast<long long>(grp) << 8);
    };
    // the next partner's records are loaded while the current pair is
    // evaluated (two dependent gathers per entry otherwise serialise)
    const int *gp = (sub < gt) ? group(sub) : nbp;
    unsigned b = (sub < gt) ? nb_index(static_cast<unsigned>(gp[0])) : 0u;
    double4 p_next = (sub < gt) ? pos[b] : pa, m_next = (sub < gt) ? mom[b] : ma;
    for (int v = sub; v < gt; v += LPP) {
      const int *gn = (v + LPP < gt) ? group(v + LPP) : gp;
      for (int u = 0; u < 8; ++u) {
        double4 const pb = p_next;
        double4 const mb = m_next;
        b = nb_index(static_cast<unsigned>(u < 7 ? gp[u + 1] : gn[0]));
        p_next = pos[b];
        m_next = mom[b];
        double const d0 = mi_d(pa.x - pb.x, G.box[0], G.box_i[0]);
        double const d1 = mi_d(pa.y - pb.y, G.box[1], G.box_i[1]);
        double const d2 = mi_d(pa.z - pb.z, G.box[2], G.box_i[2]);
        double const r2 = d0 * d0 + d1 * d1 + d2 * d2;
        if (!(r2 > 0.0))
          continue;
        double const inv_r = rsqrt(r2), r = r2 * inv_r;
        if (!(r < rc))
          continue;
        double const inv_r2 = inv_r * inv_r;
        double const ad = alpha * r;
        double const exa = exp(-ad * ad);
        double B;
        if (exact_erfc) {
          B = (erfc(ad) * inv_r + coeff * exa) * inv_r2;
        } else {
          double const t = rcp_newton(fma(0.3275911, ad, 1.0));
          double const asp =
              t * (0.254829592 + t * (-0.284496736 + t * (1.421413741 + t * (-1.453152027 +
                                                                           t * 1.061405429))));
          B = (asp * inv_r + coeff) * exa * inv_r2;
        }
        double const common = a2 * coeff * exa;
        double const Cc = (3.0 * B + 2.0 * common) * inv_r2;
        double const Dd = (5.0 * Cc + 4.0 * common * a2) * inv_r2;
        double const mimj = ma.x * mb.x + ma.y * mb.y + ma.z * mb.z;
        double const mir = ma.x * d0 + ma.y * d1 + ma.z * d2;
        double const mjr = mb.x * d0 + mb.y * d1 + mb.z * d2;
        if constexpr (EV)
          energy += mimj * B - mir * mjr * Cc;
        double const cd = mimj * Cc - mir * mjr * Dd;
        double const s = mjr * Cc, q = mir * Cc;
        s7[0] += cd * d0 + q * mb.x;
        s7[1] += cd * d1 + q * mb.y;
        s7[2] += cd * d2 + q * mb.z;
        s7[3] += s * d0 - B * mb.x;
        s7[4] += s * d1 - B * mb.y;
        s7[5] += s * d2 - B * mb.z;
        s7[6] += s;
      }
      gp = gn;
    }
  }
  dp_pairs_finish<EV, LPP>(s7, ma.x, ma.y, ma.z, energy, pref, active, a, perm, f, tq, overwrite,
                           partials);
}

// The same pair terms for the FP32-mesh mode, in FP32 from the cell-relative
// offsets (as k_pair_forces_rel: d = (off_a - off_b) - dc cs with dc from
// the entry's offset code, no minimum-image arithmetic): hardware reciprocal
// square root, reciprocal and 2^x, A&S 7.1.26 or erfcf; the pairs' force and
// torque terms and energies summed in FP64.  Bound by instruction issue: at
// 131 072 dipoles 207 us for a cutoff of 4.7 (215 us with the six sums in pairs of
// FP32 values, whose two-sums take more issue slots than the conversions and FP64
// additions and hold 48 bits), 268 us for 5.2; at 30 000 64 (69).
template <bool EV, int LPP>
__global__ void __launch_bounds__(256, EV ? kDpPairBlocks32Ev : kDpPairBlocks32)
k_dp3m_pairs_rel(const RepGeom *__restrict__ reps, const int2 *__restrict__ blk,
                 const float4 *__restrict__ spf, const float4 *__restrict__ smu,
                 const int *__restrict__ perm, const int *__restrict__ nb,
                 const int *__restrict__ nb_cnt, double pref, int exact_erfc,
                 double *__restrict__ f, double *__restrict__ tq, int overwrite,
                 double *__restrict__ partials) {
  int2 const bk = blk[blockIdx.x / LPP];
  RepGeom const &G = reps[bk.x];
  int const sub = threadIdx.x % LPP;
  long long const la = static_cast<long long>(bk.y) * 256 + (blockIdx.x % LPP) * (256 / LPP) +
                       threadIdx.x / LPP;
  bool const active = la < G.np;
  long long const a = G.p0 + la;
  double energy = 0.0;
  double s7[7] = {0, 0, 0, 0, 0, 0, 0};
  float4 const ma = active ? smu[a] : make_float4(0.f, 0.f, 0.f, 0.f);
  if (active) {
    float4 const pa = spf[a];
    float const alpha = static_cast<float>(G.alpha);
    float const rc2 = static_cast<float>(G.r_cut * G.r_cut);
    float const coeff = static_cast<float>(2.0 * G.alpha / sqrt(kPi));
    float const a2 = static_cast<float>(G.alpha * G.alpha);
    // exp(-(alpha r)^2) = 2^(c_exp r^2)
    float const c_exp = static_cast<float>(-G.alpha * G.alpha * 1.4426950408889634);
    float const ncs_x = -static_cast<float>(G.box[0] / G.cg[0]);
    float const ncs_y = -0.25f * static_cast<float>(G.box[1] / G.cg[1]);
    float const ncs_z = -0.0625f * static_cast<float>(G.box[2] / G.cg[2]);
    int const cw = nb_cnt[a];
    int const ga = (nb_count_a(cw) + 7) >> 3, gt = ga + ((nb_count_b(cw) + 7) >> 3);
    const int *nbp = nb + nb_base(G.nb_off, G.max_nb, la);
    int const ngroups = G.max_nb >> 3;
    const float4 *pos = spf + G.p0, *mom = smu + G.p0;
    for (int v = sub; v < gt; v += LPP) {
      int const grp = v < ga ? v : ngroups - 1 - (v - ga);
      const int4 *gp = reinterpret_cast<const int4 *>(nbp + (static_cast<long long>(grp) << 8));
      int4 const g0 = gp[0], g1 = gp[1];
      unsigned const ent[8] = {static_cast<unsigned>(g0.x), static_cast<unsigned>(g0.y),
                               static_cast<unsigned>(g0.z), static_cast<unsigned>(g0.w),
                               static_cast<unsigned>(g1.x), static_cast<unsigned>(g1.y),
                               static_cast<unsigned>(g1.z), static_cast<unsigned>(g1.w)};
#pragma unroll
      for (int h = 0; h < 8; h += 2) {
        float4 pv[2], mv[2]; // four gathers in flight
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          pv[u] = pos[nb_index(ent[h + u])];
          mv[u] = mom[nb_index(ent[h + u])];
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          unsigned const e = ent[h + u];
          float4 const pb = pv[u], mb = mv[u];
          float const d0 = fmaf(code_axis(e, 0), ncs_x, pa.x - pb.x);
          float const d1 = fmaf(code_axis(e, 1), ncs_y, pa.y - pb.y);
          float const d2 = fmaf(code_axis(e, 2), ncs_z, pa.z - pb.z);
          float const r2 = d0 * d0 + d1 * d1 + d2 * d2;
          if (!(r2 < rc2) || !(r2 > 0.f))
            continue;
          float const inv_r = rsqrt_approx(r2);
          float const inv_r2 = inv_r * inv_r;
          float const ad = alpha * (r2 * inv_r);
          float const exa = ex2_approx(c_exp * r2);
          float B;
          if (exact_erfc) {
            B = (erfcf(ad) * inv_r + coeff * exa) * inv_r2;
          } else {
            float const t = rcp_r(1.f + 0.3275911f * ad);
            float const asp =
                t * (0.254829592f + t * (-0.284496736f + t * (1.421413741f + t * (-1.453152027f +
                                                                               t * 1.061405429f))));
            B = (asp * inv_r + coeff) * exa * inv_r2;
          }
          float const common = a2 * coeff * exa;
          float const Cc = (3.f * B + 2.f * common) * inv_r2;
          float const Dd = (5.f * Cc + 4.f * common * a2) * inv_r2;
          float const mimj = ma.x * mb.x + ma.y * mb.y + ma.z * mb.z;
          float const mir = ma.x * d0 + ma.y * d1 + ma.z * d2;
          float const mjr = mb.x * d0 + mb.y * d1 + mb.z * d2;
          if constexpr (EV)
            energy += static_cast<double>(mimj * B - mir * mjr * Cc);
          float const cd = mimj * Cc - mir * mjr * Dd;
          float const s = mjr * Cc, q = mir * Cc;
          s7[0] += static_cast<double>(cd * d0 + q * mb.x);
          s7[1] += static_cast<double>(cd * d1 + q * mb.y);
          s7[2] += static_cast<double>(cd * d2 + q * mb.z);
          s7[3] += static_cast<double>(s * d0 - B * mb.x);
          s7[4] += static_cast<double>(s * d1 - B * mb.y);
          s7[5] += static_cast<double>(s * d2 - B * mb.z);
          s7[6] += static_cast<double>(s);
        }
      }
    }
  }
  dp_pairs_finish<EV, LPP>(s7, ma.x, ma.y, ma.z, energy, pref, active, a, perm, f, tq, overwrite,
                           partials);
}

} // namespace p3mx
