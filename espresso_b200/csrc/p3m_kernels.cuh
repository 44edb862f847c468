// P3M particle <-> mesh kernels (sm_100a): corner binning and brick-sorted
// particle records, B-spline weights, deterministic charge assignment by
// super-bricks, force back-interpolation, influence function, charge census and
// the k-space error sum.
#pragma once

#include "common.cuh"
#include "sort.cuh"

#include <algorithm>
#include <vector>

namespace p3mx {

// Fold into [0, L) like algorithm/periodic_fold.hpp:72-89 (repeated shifts);
// far-away coordinates are first brought close by whole periods.
__device__ inline double fold_coord(double x, double L) {
  if (x < -2.0 * L || x >= 3.0 * L)
    x -= floor(x / L) * L;
  int guard = 0;
  while (x < 0.0 && guard++ < 8)
    x += L;
  while (x >= L && guard++ < 16)
    x -= L;
  return x;
}

// Cardinal B-spline weights of order P at the P points around a particle
// (x = distance to the nearest mesh point, [-0.5, 0.5]): w[i] = M_P(x + 1/2 +
// P-1-i), the values tabulated in utils/math/bspline.hpp:30-177.  Weight i is
// one polynomial in x; its coefficients follow from
//   M_P(t) = sum_l (-1)^l binom(P, l) max(t - l, 0)^(P-1) / (P-1)!
// (every term a dyadic fraction, exact in FP64 before the division).
struct SplineTable {
  double c[8][8][8]; // [order][weight][power of x]
};
constexpr SplineTable spline_table() {
  SplineTable t{};
  for (int P = 1; P <= 7; ++P) {
    double binom_p[8] = {1}, binom_n[8] = {1}, fact = 1.0;
    for (int k = 1; k <= P; ++k)
      binom_p[k] = binom_p[k - 1] * (P - k + 1) / k;
    for (int k = 1; k < P; ++k) {
      binom_n[k] = binom_n[k - 1] * (P - k) / k;
      fact *= k;
    }
    for (int i = 0; i < P; ++i)
      for (int m = 0; m < P; ++m) {
        int const j = P - 1 - i;
        double sum = 0.0;
        for (int l = 0; l <= j; ++l) {
          double pw = 1.0;
          for (int e = 0; e < P - 1 - m; ++e)
            pw *= 0.5 + j - l;
          sum += ((l & 1) ? -1.0 : 1.0) * binom_p[l] * pw;
        }
        t.c[P][i][m] = binom_n[m] * sum / fact;
      }
  }
  return t;
}
__constant__ SplineTable kSpline = spline_table();
// Weight i of order P at x, coefficients c[0 .. P-1].
template <int P, typename Real> __device__ inline Real spline_eval(const Real *c, Real x) {
  Real w = c[P - 1];
#pragma unroll
  for (int m = P - 2; m >= 0; --m)
    w = w * x + c[m];
  return w;
}
template <int P, typename Real> __device__ inline void spline_coef(int i, Real *c) {
#pragma unroll
  for (int m = 0; m < P; ++m)
    c[m] = static_cast<Real>(kSpline.c[P][i][m]);
}

// Record of a particle in brick-sorted order: the distances to its nearest
// mesh point, up to three charges (a charge, or the moment components), the
// corner key inside the replica and the particle index -- one 32-byte sector
// in FP32.  The assignment and the interpolation compute the 3 P stencil
// weights from it in shared memory (8 lanes per particle, one weight of each
// axis per lane): the weight records they replace were 112 bytes, written by
// a gathering kernel and read twice.  At 2^20 ions on 256^3, order 7, the records
// save that kernel (79 us) and cost the interpolation 311 -> 325 us (20 bytes of
// spill stores at 96 registers, from evaluating the weights) and the assignment
// 241 -> 257 us.
template <typename Real> struct PRec;
template <> struct __align__(32) PRec<float> {
  float d[3], q[3];
  int key, idx;
};
template <> struct __align__(64) PRec<double> {
  double d[3], q[3];
  int key, idx;
  double pad;
};

// Per particle: nearest-mesh-point corner and the distance to it, following
// p3m_calculate_interpolation_weights (p3m/interpolation.hpp:138-178) with
// the single-rank CA-mesh origin of P3MLocalMesh (p3m/common.cpp:34-106).
// key = corner, brick-major: brick*B^3 + (lx*B + ly)*B + lz with
// brick = (bx*nby + by)*nbz + bz and (lx, ly, lz) the corner inside it; the
// sort key is brk_off + brick, so the particles of one brick form one
// contiguous range of the sorted order.  rep_of: nullptr for one replica.
template <typename Real>
__device__ inline void bin_particle(RepGeom const &G, long long i, double const (&x)[3],
                                    int *__restrict__ key, int *__restrict__ slot,
                                    int *__restrict__ cnt, Real *__restrict__ dist) {
  int g[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    double const xf = fold_coord(x[d], G.box[d]);
    double const p = ((xf - G.ld_pos[d]) * G.ai[d]) - G.pos_shift;
    int const nmp = static_cast<int>(p);
    double const ds = (p - nmp) - 0.5;
    int c = (G.ld_ind[d] + nmp) % G.mesh[d];
    if (c < 0)
      c += G.mesh[d];
    g[d] = c;
    dist[3 * i + d] = static_cast<Real>(ds);
  }
  int const B = G.brick;
  int const brick = ((g[0] / B) * G.nby + g[1] / B) * G.nbz + g[2] / B;
  key[i] = brick * B * B * B + ((g[0] % B) * B + g[1] % B) * B + g[2] % B;
  slot[i] = atomicAdd(&cnt[static_cast<int>(G.brk_off) + brick], 1);
}
// zero: nzero words cleared (the |q| maxima that the placing kernel raises next).
template <typename Real>
__global__ void __launch_bounds__(256)
k_p3m_bin(const RepGeom *__restrict__ reps, const int *__restrict__ rep_of,
          const double *__restrict__ pos, long long n, int *__restrict__ key,
          int *__restrict__ slot, int *__restrict__ cnt, Real *__restrict__ dist,
          unsigned *__restrict__ zero, int nzero) {
  pdl_enter();
  long long const i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  for (long long k = i; k < nzero; k += static_cast<long long>(gridDim.x) * blockDim.x)
    zero[k] = 0u;
  if (i >= n)
    return;
  double const x[3] = {pos[3 * i], pos[3 * i + 1], pos[3 * i + 2]};
  bin_particle(reps[rep_of ? rep_of[i] : 0], i, x, key, slot, cnt, dist);
}

// Every particle's record to its sorted place (start of its brick plus the
// slot from the counting atomics), and each replica's largest |q| per charge
// (FP32 bits rounded up, atomic maximum: order-independent; set c at
// qmax_bits + c * n_rep) for the fixed-point scale of the charge assignment.
// NC charges per particle, q[NC i + c].  The brick counts `cnt` are cleared for
// the next sort (without SCAN, where `start` already holds their scan).  A
// particle is one full 32-byte sector (FP32) written at random: the gathering
// weight kernel it replaces read five random sectors and wrote 112 bytes.
// SCAN (small systems, up to kPlaceScan bricks): `start` is not given but made,
// every block scanning all counts for itself (16 KB from L2 at most) and block 0 storing the
// result; the assignment, behind this kernel, clears the counts (a last block that
// does so here needs a ticket between two fences: 4.2 -> 5.1 us at 2000 ions).
// A small system's pass is bound by the number of dependent launches, and this
// is one less.
constexpr int kPlaceScan = 4096;
template <typename Real, int NC, bool SCAN>
__global__ void __launch_bounds__(256)
k_p3m_place(const RepGeom *__restrict__ reps, const int *__restrict__ rep_of, int n_rep,
            const int *__restrict__ key, const int *__restrict__ slot,
            int *__restrict__ start, const Real *__restrict__ dist,
            const double *__restrict__ q, long long n, PRec<Real> *__restrict__ rec,
            unsigned *__restrict__ qmax_bits, int *__restrict__ cnt, int nkeys) {
  __shared__ int s_start[SCAN ? kPlaceScan : 1];
  pdl_enter();
  long long const i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if constexpr (SCAN) {
    constexpr int PER = kPlaceScan / 256;
    int v[PER], sum = 0, total;
    int const k0 = threadIdx.x * PER;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      v[k] = k0 + k < nkeys ? cnt[k0 + k] : 0;
      sum += v[k];
    }
    int run = block_excl_scan(sum, total);
#pragma unroll
    for (int k = 0; k < PER; ++k)
      if (k0 + k < nkeys) {
        s_start[k0 + k] = run;
        if (blockIdx.x == 0)
          start[k0 + k] = run;
        run += v[k];
      }
    if (blockIdx.x == 0 && threadIdx.x == 0)
      start[nkeys] = total;
    __syncthreads();
  } else {
    for (long long k = i; k <= nkeys; k += static_cast<long long>(gridDim.x) * blockDim.x)
      cnt[k] = 0;
  }
  if (i >= n)
    return;
  int const rep = rep_of ? rep_of[i] : 0;
  RepGeom const &G = reps[rep];
  PRec<Real> r;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    r.d[d] = dist[3 * i + d];
    r.q[d] = Real(0);
  }
  r.key = key[i];
  r.idx = static_cast<int>(i);
  unsigned const act = __activemask();
  unsigned const grp = __match_any_sync(act, rep);
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    double const qi = q[NC * i + c];
    r.q[c] = static_cast<Real>(qi);
    // one atomic per group of lanes of the same replica, and only where the
    // maximum seen so far is smaller
    unsigned const mx =
        __reduce_max_sync(grp, __float_as_uint(__double2float_ru(fabs(qi))));
    unsigned *const w = qmax_bits + c * n_rep + rep;
    if (static_cast<int>(threadIdx.x & 31) == __ffs(grp) - 1 &&
        mx > *reinterpret_cast<volatile unsigned *>(w))
      atomicMax(w, mx);
  }
  int const lb = G.brick == 4 ? 6 : 9; // log2 of the corners per brick
  int const b = static_cast<int>(G.brk_off) + (r.key >> lb);
  rec[(SCAN ? s_start[b] : start[b]) + slot[i]] = r;
}

// Edge (mesh points) of the sort bricks that bin the particles by stencil
// corner for order P (the interpolation stages one brick's field tile of
// (B + P - 1)^3 points; owner blocks of the assignment are whole numbers
// of bricks).
template <int P> __host__ __device__ constexpr int brick_edge() { return (P <= 5) ? 4 : 8; }

struct TileStrides {
  int sy, sx;
};

// ---------------------------------------------------------------------------
// Charge assignment by super-bricks (AssignCharges, p3m.cpp:225-265;
// charge_assign, p3m.cpp:283-330).  One CTA takes the particles whose
// stencil corners lie in a super-brick of E^3 corner positions (whole
// sort bricks: a few contiguous ranges of the brick-major order), so every
// particle is visited once.  For each particle one warp covers its P^2
// (x, y) stencil rows (one row per lane, the P z points of a row unrolled)
// and adds q wx wy wz into a shared-memory tile of (E + P - 1)^3
// points, in fixed point.  E = 16, or 8
// when the 16^3 super-bricks would not give every SM two blocks (small
// meshes: more, smaller tiles with a larger halo share).  Tiles of
// neighbouring super-bricks overlap by P - 1 points.  Every block stores its
// whole tile, halo included, to its own place in HBM, and the forward z pass
// sums the tiles that cover a mesh point while it loads its lines
// (TileMap): all super-bricks run in one launch, no mesh is zeroed and none
// is read back and rewritten, and the sum over the (up to 8, in wrap corners
// 27) tiles has a fixed order, so the mesh is bitwise reproducible.  The
// tiles hold ((16 + P - 1) / 16)^3 = 2.6 mesh sizes at P = 7.  The kernel is
// bound by the shared-memory atomics and loads of the stencil terms: 2^20 ions on
// 256^3 at order 7 257 us against 241 us in eight coloured launches that added
// to the mesh, which also needed 79 us of weight records; 131 072 ions on 128^3
// 47 against 64 + 17 us, 23 457 ions 10 against 55 + 9 us.
//
// Fixed point: a term v = q wx wy wz becomes t = rint(v S) by one FP64 FMA
// with the magic constant 1.5 * 2^52 (the bits of the sum are those of the
// constant plus t while |t| < 2^51) and is added with one integer atomic:
// FP32-mixed path, the low 32 bits (the constant's low word is zero, so the
// word is t modulo 2^32, and a tile point's sum is exact modulo 2^32); FP64
// path, the 64-bit t.  S is a power of two with n qmax wmax^3 S < 2^31
// (FP32-mixed) or < 2^62 and qmax wmax^3 S < 2^51 (FP64), n the particles of
// the super-brick, qmax the replica's largest |q|, wmax the largest B-spline
// weight of order P: no term leaves the exact range and no tile point's
// final sum overflows (wrap-around of intermediate two's complement sums
// cancels).  Integer sums do not depend on the order of the atomics; the
// quantum 1/S is about 2^-25 of a charge at 2^20 ions on a 256^3 mesh
// (FP32-mixed) and 2^-56 in FP64, and each tile point is rounded once to
// the working precision before it is stored.
constexpr int kSbEdge = 16;   // corner positions per dimension of a super-brick (multiple of 4 and 8)
constexpr int kSbEdgeSmall = 8; // the edge for meshes with too few 16^3 super-bricks to fill the GPU
constexpr int kSbWarps = 8;   // warps per super-brick block
constexpr int kSbChunk = 64;  // particles whose records are staged at a time

// Largest cardinal B-spline weight of order P over dist in [-1/2, 1/2],
// rounded up (1, 1, 3/4, 2/3, 115/192, 11/20, 0.51102...).
template <int P> __host__ __device__ constexpr double bspline_wmax() {
  return P <= 2 ? 1.0 : P == 3 ? 0.7501 : P == 4 ? 0.6668 : P == 5 ? 0.5991 : P == 6 ? 0.5501 : 0.5112;
}

template <typename Real> struct SbWord;
template <> struct SbWord<float> {
  using type = unsigned;
  static constexpr int sum_bits = 31;
};
template <> struct SbWord<double> {
  using type = unsigned long long;
  static constexpr int sum_bits = 62;
};
constexpr int kSbTermBits = 51;
// t = rint(a b) for |a b| < 2^51, added modulo 2^32 (low word of the FMA
// with the magic constant) or as a 64-bit integer
__device__ inline void sb_add(unsigned *p, double a, double b) {
  double const r = fma(a, b, 6755399441055744.0); // 1.5 * 2^52
  atomicAdd(p, static_cast<unsigned>(__double2loint(r)));
}
// FP64 path: the 64-bit t added as two 32-bit words (the low word's atomic
// returns its old value, whose wrap-around gives the carry into the high
// word), so the sum is exact modulo 2^64 with native 32-bit shared-memory
// atomics only
__device__ inline void sb_add(unsigned long long *p, double a, double b) {
  double const r = fma(a, b, 6755399441055744.0);
  unsigned long long const t =
      static_cast<unsigned long long>(__double_as_longlong(r)) - 0x4338000000000000ull;
  unsigned *w = reinterpret_cast<unsigned *>(p); // little endian: w[0] low, w[1] high
  unsigned const lo = static_cast<unsigned>(t);
  unsigned const old = atomicAdd(w, lo);
  unsigned const hi = static_cast<unsigned>(t >> 32) + ((old + lo < old) ? 1u : 0u);
  if (hi != 0u)
    atomicAdd(w + 1, hi);
}
__device__ inline float sb_value(unsigned v, float inv_s) {
  return static_cast<float>(static_cast<int>(v)) * inv_s;
}
__device__ inline double sb_value(unsigned long long v, double inv_s) {
  return static_cast<double>(static_cast<long long>(v)) * inv_s;
}

// Tile edge of a super-brick of edge E for order P.
template <int P, int E> __host__ __device__ constexpr int sb_tile_edge() { return E + P - 1; }
// Strides of the tile [x][y][z] (z contiguous, words of WB bytes): the
// smallest y stride >= the tile edge and x stride >= edge * (y stride) for
// which the lanes of one shared-memory wavefront (128 bytes: 32 lanes of
// 4-byte words, 16 of 8-byte words), one (x, y) stencil row each (row
// r = lane + 32 q, x = r / P, y = r % P), hit distinct banks.
template <int P, int WB, int E> __host__ __device__ constexpr TileStrides sb_strides() {
  constexpr int TE = sb_tile_edge<P, E>();
  constexpr int L = 128 / WB;
  for (int sy = TE; sy < TE + L; ++sy)
    for (int sx = TE * sy; sx < TE * sy + 2 * L; ++sx) {
      bool ok = true;
      for (int r0 = 0; r0 < P * P && ok; r0 += L) {
        unsigned long long used = 0;
        for (int r = r0; r < r0 + L && r < P * P; ++r) {
          unsigned long long const bit = 1ull << (((r / P) * sx + (r % P) * sy) % L);
          if (used & bit) {
            ok = false;
            break;
          }
          used |= bit;
        }
      }
      if (ok)
        return TileStrides{sy, sx};
    }
  return TileStrides{TE, TE * TE};
}
template <typename Real, int P, int E> __host__ __device__ constexpr size_t sb_tile_bytes() {
  using W = typename SbWord<Real>::type;
  return (sizeof(W) * sb_tile_edge<P, E>() * static_cast<size_t>(sb_strides<P, sizeof(W), E>().sx) +
          63) / 64 * 64;
}
// shared memory: tile, staged records, per staged particle its z weights
// times S in FP64, its x weights times the charge and its y weights (8 slots
// each), and its tile offset
template <typename Real, int P, int E> __host__ __device__ constexpr size_t sb_smem() {
  return sb_tile_bytes<Real, P, E>() + (sizeof(PRec<Real>) + 8 * sizeof(double) +
                                        16 * sizeof(Real) + sizeof(int)) * kSbChunk;
}
// The stored tiles of a replica, TE = E + P - 1 points per edge, z rows
// padded to TZ values (a multiple of 4): value (lx, ly, lz) of super-brick
// (bx, by, bz) at ((bx TE + lx) (n1 TE) + by TE + ly) (n2 TZ) + bz TZ + lz,
// n1, n2 the super-bricks along y and z -- the rows of a mesh line's tiles
// along z are one contiguous range.
__host__ __device__ constexpr int sb_tile_z(int te) { return (te + 3) / 4 * 4; }
// sort-brick runs of a super-brick: (kSbEdge / B)^2 brick columns, one
// contiguous z run each
constexpr int kSbMaxRuns = (kSbEdge / 4) * (kSbEdge / 4);

template <typename Real, int P, int E, bool MC>
__global__ void __launch_bounds__(32 * kSbWarps, sizeof(Real) == 4 ? 4 : 1)
k_p3m_assign_sb(const RepGeom *__restrict__ reps, const int2 *__restrict__ sbs, int nsb,
                const int *__restrict__ start, const PRec<Real> *__restrict__ recs,
                const unsigned *__restrict__ qmax_bits, Real *__restrict__ tiles,
                int *__restrict__ err, long long comp_tile, int comp_q, int *__restrict__ clear,
                int nclear) {
  // clear: nclear words set to zero (the brick counts that the placing kernel
  // before this one has scanned).
  // MC: blockIdx.y picks one of several charge sets assigned by one launch
  // (the dipole components): its tiles and |q| maxima lie comp_tile / comp_q
  // elements after the previous set's. The single-set instance leaves the
  // pointers as kernel parameters: the offset copies cost registers at the
  // FP32 instances' 64-register bound.
  if constexpr (MC) {
    tiles += blockIdx.y * comp_tile;
    qmax_bits += blockIdx.y * comp_q;
  }
  using Word = typename SbWord<Real>::type;
  constexpr int P2 = P * P;
  constexpr int NQ = (P2 + 31) / 32;
  constexpr int NT = 32 * kSbWarps;
  constexpr int TE = sb_tile_edge<P, E>();
  constexpr int B = brick_edge<P>(), B3 = B * B * B, NBS = E / B;
  constexpr int LB = (B == 4) ? 2 : 3;
  constexpr TileStrides TS = sb_strides<P, sizeof(Word), E>();
  constexpr int SY = TS.sy, SX = TS.sx;
  constexpr int TW = static_cast<int>(sb_tile_bytes<Real, P, E>() / sizeof(Word));
  static_assert(E % B == 0 && E <= kSbEdge, "super-brick edge: a multiple of the sort brick");
  constexpr int CH = kSbChunk;
  static_assert(NBS * NBS <= kSbMaxRuns, "run table too small");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ __align__(8) unsigned long long bar;
  __shared__ int s_r0[kSbMaxRuns], s_pre[kSbMaxRuns + 1];
  __shared__ Real s_cf[8 * 8];
  pdl_enter();
  for (int k = blockIdx.x * NT + threadIdx.x; k < nclear; k += gridDim.x * NT)
    clear[k] = 0;
  if (static_cast<int>(blockIdx.x) >= nsb)
    return; // whole block
  Word *tile = reinterpret_cast<Word *>(smem_raw);
  PRec<Real> *rec = reinterpret_cast<PRec<Real> *>(smem_raw + sb_tile_bytes<Real, P, E>());
  double *wzd = reinterpret_cast<double *>(rec + CH);
  Real *wxs = reinterpret_cast<Real *>(wzd + 8 * CH), *wys = wxs + 8 * CH;
  int *toff = reinterpret_cast<int *>(wys + 8 * CH);
  int const tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  int2 const sb = sbs[blockIdx.x];
  RepGeom const &G = reps[sb.x];
  int const M0 = G.mesh[0], M1 = G.mesh[1], M2 = G.mesh[2];
  int const no1 = (M1 + E - 1) / E, no2 = (M2 + E - 1) / E;
  int const o0 = (sb.y / (no1 * no2)) * E, o1 = ((sb.y / no2) % no1) * E, o2 = (sb.y % no2) * E;
  // the super-brick's sort bricks (fewer at the high end of a mesh that is
  // not a multiple of E)
  int const bx0 = o0 / B, by0 = o1 / B, bz0 = o2 / B;
  int const nbx = min(NBS, G.nbx - bx0), nby = min(NBS, G.nby - by0), nbz = min(NBS, G.nbz - bz0);
  int const ncol = nbx * nby;
  if (warp == 0) {
    // the runs' first particles and the prefix of their counts
    int r0 = 0, c = 0;
    if (lane < ncol) {
      const int *st = start + G.brk_off;
      int const col = ((bx0 + lane / nby) * G.nby + (by0 + lane % nby)) * G.nbz + bz0;
      r0 = st[col];
      c = st[col + nbz] - r0;
    }
    int incl = c;
#pragma unroll
    for (int o = 1; o < kSbMaxRuns; o <<= 1) {
      int const t = __shfl_up_sync(0xffffffffu, incl, o);
      incl += lane >= o ? t : 0;
    }
    if (lane < ncol) {
      s_r0[lane] = r0;
      s_pre[lane + 1] = incl;
    }
    if (lane == 0)
      s_pre[0] = 0;
  }
  if (tid < 64 && (tid & 7) < P && (tid >> 3) < P)
    s_cf[tid] = static_cast<Real>(kSpline.c[P][tid >> 3][tid & 7]);
  // zero the tile; initialise the staging barrier
  for (int t = tid; t < TW; t += NT)
    tile[t] = Word(0);
  if (tid == 0)
    mbar_init(&bar, 1);
  __syncthreads();
  int const count = s_pre[ncol];
  float const qmax = __uint_as_float(qmax_bits[sb.x]);
  // store the tile, value(x, y, z) (lanes along z: conflict-free shared
  // reads, row segments stored whole; the row padding is zero)
  auto store_tile = [&](auto const &value) {
    constexpr int TZ = sb_tile_z(TE);
    int const rz = no2 * TZ;
    long long const rx = static_cast<long long>(no1) * TE * rz;
    Real *const out = tiles + G.tl_off + (o0 / E) * TE * rx +
                      static_cast<long long>(o1 / E) * TE * rz + (o2 / E) * TZ;
    for (int t = tid; t < TE * TE * TZ; t += NT) {
      int const row = t / TZ, z = t - row * TZ;
      int const x = row / TE, y = row - x * TE;
      out[x * rx + y * rz + z] = (z < TE) ? value(x, y, z) : Real(0);
    }
  };
  if (count == 0 || !(qmax > 0.0f)) {
    store_tile([](int, int, int) { return Real(0); });
    return;
  }
  int es;
  {
    double const unit = static_cast<double>(qmax) * bspline_wmax<P>() * bspline_wmax<P>() *
                        bspline_wmax<P>();
    int ea, eb;
    frexp(unit, &ea);
    frexp(unit * static_cast<double>(count), &eb);
    es = min(kSbTermBits - ea, SbWord<Real>::sum_bits - eb);
    es = max(min(es, 1000), -1000);
  }
  double const S = ldexp(1.0, es);
  // per-lane (x, y) stencil row of each round and its tile offset
  int qx[NQ], qy[NQ], qoff[NQ];
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    int const r = lane + 32 * q;
    int const rr = (r < P2) ? r : 0;
    qx[q] = rr / P;
    qy[q] = rr % P;
    qoff[q] = qx[q] * SX + qy[q] * SY;
  }
  unsigned parity = 0;
  // chunks of particles across the runs (a chunk per run would end in a short
  // one for every other run)
  for (int c0 = 0; c0 < count; c0 += CH) {
    {
      int const cn = min(CH, count - c0);
      __syncthreads(); // the previous chunk is consumed
      if (warp == 0) {
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        if (lane == 0) {
          mbar_arrive_expect_tx(&bar, static_cast<unsigned>(cn * sizeof(PRec<Real>)));
        }
        __syncwarp();
        if (lane < ncol) {
          int const lo = max(c0, s_pre[lane]), hi = min(c0 + cn, s_pre[lane + 1]);
          if (lo < hi)
            bulk_g2s(rec + (lo - c0), recs + (s_r0[lane] + lo - s_pre[lane]),
                     static_cast<unsigned>((hi - lo) * sizeof(PRec<Real>)), &bar);
        }
      }
      bool const got = mbar_wait(&bar, parity);
      parity ^= 1u;
      if (__syncthreads_or(!got)) {
        if (tid == 0) {
          atomicExch(err, 1);
          mbar_wait(&bar, parity ^ 1u); // bounded wait for the copy in flight
        }
        return;
      }
      // weights of the staged particles: lane k of a particle's 8 the weight k
      // of each axis (z in FP64, times S), lane 7 the tile offset
      {
        int const k = tid & 7;
        Real cf[P];
#pragma unroll
        for (int m = 0; m < P; ++m)
          cf[m] = s_cf[8 * min(k, P - 1) + m];
        for (int j = tid >> 3; j < cn; j += NT / 8) {
          PRec<Real> const &r = rec[j];
          if (k < P) {
            wxs[8 * j + k] = r.q[MC ? blockIdx.y : 0] * spline_eval<P>(cf, r.d[0]);
            wys[8 * j + k] = spline_eval<P>(cf, r.d[1]);
            wzd[8 * j + k] = static_cast<double>(spline_eval<P>(cf, r.d[2])) * S;
          } else if (k == 7) {
            // corner offset inside the super-brick, [0, E)^3
            int const sk = r.key;
            int run = 0;
            while (c0 + j >= s_pre[run + 1])
              ++run;
            int const bx = bx0 + run / nby, by = by0 + run % nby;
            int const bz = (sk >> (3 * LB)) - (bx * G.nby + by) * G.nbz;
            int const l = sk & (B3 - 1);
            int const dx = bx * B + (l >> (2 * LB)) - o0, dy = by * B + ((l >> LB) & (B - 1)) - o1,
                      dz = bz * B + (l & (B - 1)) - o2;
            toff[j] = dx * SX + dy * SY + dz;
          }
        }
      }
      __syncthreads();
      for (int j = warp; j < cn; j += kSbWarps) {
        int const base = toff[j];
        double wz[8];
#pragma unroll
        for (int k = 0; k < P; k += 2) {
          double2 const w = reinterpret_cast<const double2 *>(wzd)[4 * j + k / 2];
          wz[k] = w.x;
          wz[k + 1] = w.y;
        }
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
          if (lane + 32 * q < P2) {
            double const wxy = static_cast<double>(wxs[8 * j + qx[q]] * wys[8 * j + qy[q]]);
            Word *pt = tile + base + qoff[q];
#pragma unroll
            for (int k = 0; k < P; ++k)
              sb_add(pt + k, wxy, wz[k]);
          }
        }
      }
    }
  }
  __syncthreads();
  Real const inv_S = static_cast<Real>(ldexp(1.0, -es));
  store_tile([&](int x, int y, int z) { return sb_value(tile[x * SX + y * SY + z], inv_S); });
}

// Cover table of an axis of M mesh points in super-bricks of edge E, order P:
// entry j (j < 3) of point i names the j-th super-brick b whose tile holds
// the point (offset l: b E + l = i modulo M) as (b << 8) | l, or -1; the
// point's own super-brick comes first.  A point lies in its own super-brick's
// tile and maybe in the halo of the one before; the first P - 1 points of an
// axis whose last super-brick is shorter than P - 1 also in that of the one
// before the last.  Entry j of point i is at cov[cov_off + j M + i].
inline void cover_table(int M, int E, int P, std::vector<int> &cov) {
  size_t const at = cov.size();
  cov.resize(at + 3 * static_cast<size_t>(M), -1);
  std::vector<int> n(M, 0);
  int const nb = (M + E - 1) / E;
  for (int halo = 0; halo < 2; ++halo)
    for (int b = 0; b < nb; ++b) {
      int const len = std::min(E, M - b * E);
      for (int l = halo ? len : 0; l < (halo ? len + P - 1 : len); ++l) {
        int const i = (b * E + l) % M;
        if (n[i] == 3)
          throw Error(3, "assignment tiles: more than three covers of a mesh point");
        cov[at + static_cast<size_t>(n[i]++) * M + i] = (b << 8) | l;
      }
    }
}

// Per-axis offset contributions of cover entries in the stored tiles (-1 for
// no entry).
struct TileMap {
  long long sx;
  int te, sy, tz;
  __device__ explicit TileMap(RepGeom const &G, int E)
      : te(E + G.cao - 1), tz(sb_tile_z(te)) {
    sy = G.sbn[2] * tz;
    sx = static_cast<long long>(G.sbn[1]) * te * sy;
  }
  __device__ long long x(int c) const {
    return c < 0 ? -1 : ((c >> 8) * te + (c & 255)) * sx;
  }
  __device__ int y(int c) const { return c < 0 ? -1 : ((c >> 8) * te + (c & 255)) * sy; }
  __device__ int z(int c) const { return c < 0 ? -1 : (c >> 8) * tz + (c & 255); }
};

__device__ inline float tile_add(float a, float b) { return a + b; }
__device__ inline double tile_add(double a, double b) { return a + b; }
template <typename V> __device__ inline V tile_add(V a, V b) {
  a.x += b.x;
  a.y += b.y;
  a.z += b.z;
  a.w += b.w;
  return a;
}
// Sum over the (x, y) covers of a line (offset contributions bx, by: entry 0
// always there, 1 and 2 may be -1) of the value V (one or four points along
// z) at z offset z.  The up to 4 loads of the first two entries are issued
// together; a third entry occurs in wrap corners only.
template <typename V, typename Real>
__device__ inline V tile_rows(const Real *__restrict__ t, const long long *bx, const int *by,
                              int z) {
  V v[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    long long const x = bx[c >> 1];
    int const y = by[c & 1];
    v[c] = (c == 0 || (x >= 0 && y >= 0)) ? *reinterpret_cast<const V *>(t + (x + y + z)) : V{};
  }
  V s = tile_add(tile_add(v[0], v[1]), tile_add(v[2], v[3]));
  if (bx[2] >= 0 || by[2] >= 0)
    for (int i = 0; i < 3; ++i)
      for (int j = 0; j < 3; ++j)
        if ((i == 2 || j == 2) && bx[i] >= 0 && by[j] >= 0)
          s = tile_add(s, *reinterpret_cast<const V *>(t + (bx[i] + by[j] + z)));
  return s;
}

// The charge mesh from the stored tiles (mesh copies for parity checks; the
// path itself sums the tiles inside the forward z pass).
template <typename Real>
__global__ void k_tiles_to_mesh(const RepGeom *__restrict__ reps, int r,
                                const Real *__restrict__ tiles, const int *__restrict__ cov, int E,
                                Real *__restrict__ rho) {
  RepGeom const &G = reps[r];
  int const M0 = G.mesh[0], M1 = G.mesh[1], M2 = G.mesh[2];
  long long const local = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (local >= static_cast<long long>(M0) * M1 * M2)
    return;
  int const z = static_cast<int>(local % M2), y = static_cast<int>((local / M2) % M1),
            x = static_cast<int>(local / (static_cast<long long>(M1) * M2));
  TileMap const tm(G, E);
  long long bx[3];
  int by[3], bz[3];
  for (int j = 0; j < 3; ++j) {
    bx[j] = tm.x(cov[G.cov_off[0] + j * M0 + x]);
    by[j] = tm.y(cov[G.cov_off[1] + j * M1 + y]);
    bz[j] = tm.z(cov[G.cov_off[2] + j * M2 + z]);
  }
  Real s = tile_rows<Real>(tiles + G.tl_off, bx, by, bz[0]);
  if (bz[1] >= 0) {
    Real h = tile_rows<Real>(tiles + G.tl_off, bx, by, bz[1]);
    if (bz[2] >= 0)
      h += tile_rows<Real>(tiles + G.tl_off, bx, by, bz[2]);
    s += h;
  }
  rho[local] = s;
}

// Force back-interpolation (AssignForces, electrostatics/p3m.cpp:344-373) as
// a warp-specialised pipeline over bricks.  Each block takes the bricks
// blockIdx.x, blockIdx.x + gridDim.x, ... (a persistent grid); its warp 0
// (the producer) fills kInterpStages shared-memory stages ahead of the
// kInterpWarps consumer warps.  A stage holds one brick's field tile --
// (B+P-1)^3 packed (Ex, Ey, Ez, 0) records from the brick origin, one 3-d
// tensor copy (TMA engine) from the replica's ghost-padded field mesh, whose
// high-side ghost layers hold the periodic images -- and the weight records,
// sort keys and source indices of up to kInterpCap of the brick's particles
// (contiguous in the brick-major order: one bulk copy each).  A full barrier
// per stage counts the producer lanes' arrivals and the copied bytes; an
// empty barrier per stage counts the consumer warps that finished with it.
// Consumers read shared memory only (particles past the cap of a dense brick
// read their records from global memory) and store the forces.
//
// Eight lanes serve one particle: lane kz owns the stencil z offset kz and
// walks the P^2 (x, y) rows; lane sums are FP32 (FP64 for the FP64 path),
// the group reduction is FP64 in a fixed shuffle order (deterministic).
// F -= prefactor/V * sum (q wx wy wz) E, plus the dipole term for
// epsilon != 0 (p3m.cpp:540-547).  Writes (or adds) f[3*i] of the original
// particle index.  Every barrier wait is bounded: on a timeout the kernel
// sets *err, the producer waits (bounded) for its copies in flight, and the
// block returns.
constexpr int kInterpStages = 2;
constexpr int kInterpWarps = 8; // consumer warps
constexpr int kInterpCap = 64;  // particles per stage with staged records

template <typename Real, int P> struct InterpStage {
  using R4 = typename Real4Of<Real>::type;
  static constexpr int Ed = brick_edge<P>() + P - 1;
  static constexpr size_t tile = sizeof(R4) * Ed * Ed * Ed;
  static constexpr size_t rec_at = (tile + 63) / 64 * 64;
  static constexpr size_t rec = sizeof(PRec<Real>) * kInterpCap;
  // stages start on 128-byte boundaries (tensor copy destinations)
  static constexpr size_t bytes = (rec_at + rec + 127) / 128 * 128;
};
// (stages, then per consumer warp the x and y weights of its four particles;
// + 128: the kernel rounds the dynamic shared-memory base up to 128 bytes)
template <typename Real, int P> __host__ __device__ constexpr size_t interp_smem() {
  return kInterpStages * InterpStage<Real, P>::bytes + kInterpWarps * 4 * 16 * sizeof(Real) + 128;
}

struct InterpInfo {
  int rep, brick, s0, s1; // rep < 0: no more bricks
  double pref, cdip;
};

__device__ inline void mbar_arrive(unsigned long long *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

template <typename Real, int P>
__global__ void __launch_bounds__(32 * (1 + kInterpWarps), sizeof(Real) == 4 ? 2 : 1)
k_p3m_interp(const RepGeom *__restrict__ reps, const int2 *__restrict__ bricks, int nbricks,
             const int *__restrict__ start, const PRec<Real> *__restrict__ recs, int unit,
             const CUtensorMap *__restrict__ tmaps, int map_stride,
             const double *__restrict__ q, const double *__restrict__ dipole,
             double *__restrict__ f, long long f_stride, int overwrite, int *__restrict__ err) {
  // blockIdx.y: field set (tensor maps and outputs map_stride / f_stride
  // apart); unit: charges of one instead of the records'
  tmaps += blockIdx.y * map_stride;
  f += blockIdx.y * f_stride;
  static_assert(P <= 8, "one lane per stencil z offset");
  constexpr int S = kInterpStages, CW = kInterpWarps, CAP = kInterpCap;
  using L = InterpStage<Real, P>;
  using R4 = typename L::R4;
  constexpr int B = brick_edge<P>(), B3 = B * B * B, Ed = L::Ed, E2 = Ed * Ed;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ __align__(8) unsigned long long full[S], empty[S];
  __shared__ InterpInfo s_info[S];
  pdl_enter();
  int const tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
#pragma unroll
    for (int k = 0; k < S; ++k) {
      mbar_init(&full[k], 32);  // the producer's lanes
      mbar_init(&empty[k], CW); // one arrival per consumer warp
    }
  }
  __syncthreads();
  unsigned char *const smem_base = smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u);
  auto stage_ptr = [&](int k) { return smem_base + static_cast<size_t>(k) * L::bytes; };

  if (warp == 0) {
    // ---------------- producer ----------------
    // the next brick's table entry and particle range are fetched one brick
    // ahead, so their load latency overlaps the copies of the current one
    int it = 0, last_rep = -1;
    bool ok = true;
    int n = blockIdx.x;
    int2 bk = make_int2(0, 0);
    int s0 = 0, s1 = 0;
    if (n < nbricks) {
      bk = bricks[n];
      const int *st = start + reps[bk.x].brk_off;
      s0 = st[bk.y];
      s1 = st[bk.y + 1];
    }
    for (; n < nbricks; n += gridDim.x) {
      int const nn = n + gridDim.x;
      int2 const bkn = (nn < nbricks) ? bricks[nn] : make_int2(0, 0);
      if (s0 != s1) {
        RepGeom const &G = reps[bk.x];
        int const k = it % S;
        bool const got = mbar_wait(&empty[k], ((it / S) & 1) ^ 1u);
        if (!__all_sync(0xffffffffu, got)) {
          ok = false;
          break;
        }
        unsigned char *sp = stage_ptr(k);
        R4 *tile = reinterpret_cast<R4 *>(sp);
        PRec<Real> *rec = reinterpret_cast<PRec<Real> *>(sp + L::rec_at);
        int const cn = min(s1 - s0, CAP);
        if (lane == 0) {
          InterpInfo inf;
          inf.rep = bk.x;
          inf.brick = bk.y;
          inf.s0 = s0;
          inf.s1 = s1;
          inf.pref = G.prefactor / G.V;
          inf.cdip = (G.epsilon != 0.0)
                         ? G.prefactor * 4.0 * kPi / G.V / (2.0 * G.epsilon + 1.0)
                         : 0.0;
          s_info[k] = inf;
        }
        // the consumers' reads of the stage were generic-proxy accesses:
        // order them before the asynchronous-proxy writes that refill it
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        int const bz = bk.y % G.nbz, by = (bk.y / G.nbz) % G.nby, bx = bk.y / (G.nbz * G.nby);
        // lane 0: the tile; lane 1: the particle records
        unsigned bytes = 0;
        if (lane == 0)
          bytes = static_cast<unsigned>(E2 * Ed * sizeof(R4));
        else if (lane == 1)
          bytes = static_cast<unsigned>(cn * sizeof(PRec<Real>));
        mbar_arrive_expect_tx(&full[k], bytes);
        if (lane == 0) {
          if (bk.x != last_rep) {
            tensormap_acquire(&tmaps[bk.x]);
            last_rep = bk.x;
          }
          tma_load_3d(tile, &tmaps[bk.x], 4 * bz * B, by * B, bx * B, &full[k]);
        } else if (lane == 1) {
          bulk_g2s(rec, recs + s0, bytes, &full[k]);
        }
        ++it;
      }
      int s0n = 0, s1n = 0;
      if (nn < nbricks) {
        const int *st = start + reps[bkn.x].brk_off;
        s0n = st[bkn.y];
        s1n = st[bkn.y + 1];
      }
      bk = bkn;
      s0 = s0n;
      s1 = s1n;
    }
    // end marker for the consumers
    if (ok) {
      int const k = it % S;
      bool const got = mbar_wait(&empty[k], ((it / S) & 1) ^ 1u);
      if (__all_sync(0xffffffffu, got)) {
        if (lane == 0)
          s_info[k].rep = -1;
        mbar_arrive(&full[k]);
      } else {
        ok = false;
      }
    }
    if (!ok) {
      if (lane == 0)
        atomicExch(err, 1);
      // bounded wait for the fills that may still be in flight
      for (int j = max(0, it - S); j < it; ++j)
        mbar_wait(&full[j % S], (j / S) & 1);
    }
    return;
  }

  // ---------------- consumers ----------------
  int const cw = warp - 1, g = lane >> 3, kz = lane & 7;
  // weight kz of an axis is this lane's polynomial; x and y weights meet in
  // the warp's slots
  Real cf[P];
  spline_coef<P>(min(kz, P - 1), cf);
  Real *const wsl = reinterpret_cast<Real *>(smem_base + S * L::bytes) + (4 * cw + g) * 16;
  for (int it = 0;; ++it) {
    int const k = it % S;
    bool const got = mbar_wait(&full[k], (it / S) & 1);
    if (!__all_sync(0xffffffffu, got)) {
      if (lane == 0)
        atomicExch(err, 1);
      return;
    }
    InterpInfo const inf = s_info[k];
    if (inf.rep < 0)
      return;
    unsigned char *sp = stage_ptr(k);
    const R4 *tile = reinterpret_cast<const R4 *>(sp);
    const PRec<Real> *rec = reinterpret_cast<const PRec<Real> *>(sp + L::rec_at);
    int const s0 = inf.s0, s1 = inf.s1;
    // four particles per warp (one per 8-lane group), warps interleaved
    for (int sb = s0 + 4 * cw; sb < s1; sb += 4 * CW) {
      int const s = sb + g, j = s - s0;
      bool const live = s < s1;
      Real ax = Real(0), ay = Real(0), az = Real(0), wzk = Real(0);
      int l = 0, idx = 0;
      if (live) {
        PRec<Real> r;
        if (j < CAP)
          r = rec[j];
        else
          r = recs[s];
        l = r.key - inf.brick * B3;
        idx = r.idx;
        wsl[kz] = (unit ? Real(1) : r.q[0]) * spline_eval<P>(cf, r.d[0]);
        wsl[8 + kz] = spline_eval<P>(cf, r.d[1]);
        wzk = spline_eval<P>(cf, r.d[2]);
      }
      __syncwarp();
      if (live && kz < P) {
        int const lb = __ffs(B) - 1; // B is a power of two
        int const lx = l >> (2 * lb), ly = (l >> lb) & (B - 1), lz = l & (B - 1);
        Real wx[8], wy[8];
#pragma unroll
        for (int h = 0; h < P; h += 4) {
          R4 const u = reinterpret_cast<const R4 *>(wsl)[h / 4];
          R4 const v = reinterpret_cast<const R4 *>(wsl)[2 + h / 4];
          wx[h] = u.x, wx[h + 1] = u.y, wx[h + 2] = u.z, wx[h + 3] = u.w;
          wy[h] = v.x, wy[h + 1] = v.y, wy[h + 2] = v.z, wy[h + 3] = v.w;
        }
        const R4 *tp = tile + (lx * Ed + ly) * Ed + lz + kz;
#pragma unroll
        for (int kx = 0; kx < P; ++kx) {
          Real const wxz = wx[kx] * wzk;
#pragma unroll
          for (int ky = 0; ky < P; ++ky) {
            R4 const e = tp[(kx * Ed + ky) * Ed];
            Real const wt = wxz * wy[ky];
            ax += wt * e.x;
            ay += wt * e.y;
            az += wt * e.z;
          }
        }
      }
      __syncwarp(); // the slots are refilled for the next four particles
      double fx = static_cast<double>(ax), fy = static_cast<double>(ay),
             fz = static_cast<double>(az);
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) {
        fx += __shfl_xor_sync(0xffffffffu, fx, o);
        fy += __shfl_xor_sync(0xffffffffu, fy, o);
        fz += __shfl_xor_sync(0xffffffffu, fz, o);
      }
      if (live && kz == 0) {
        int const i = idx;
        double ox = -inf.pref * fx, oy = -inf.pref * fy, oz = -inf.pref * fz;
        if (inf.cdip != 0.0) {
          double const qi = q[i];
          ox -= qi * inf.cdip * dipole[3 * inf.rep + 0];
          oy -= qi * inf.cdip * dipole[3 * inf.rep + 1];
          oz -= qi * inf.cdip * dipole[3 * inf.rep + 2];
        }
        if (overwrite) {
          f[3 * i + 0] = ox;
          f[3 * i + 1] = oy;
          f[3 * i + 2] = oz;
        } else {
          f[3 * i + 0] += ox;
          f[3 * i + 1] += oy;
          f[3 * i + 2] += oz;
        }
      }
    }
    __syncwarp();
    if (lane == 0)
      mbar_arrive(&empty[k]);
  }
}

// sinc with the Taylor branch of p3m/math.hpp:53-81.
__device__ inline double sinc_d(double x) {
  double const pix = kPi * x;
  if (fabs(x) > 0.1)
    return sin(pix) / pix;
  double const p2 = pix * pix;
  return 1.0 + p2 * (-1.0 / 6.0 + p2 * (1.0 / 120.0 + p2 * (-1.0 / 5040.0 + p2 * (1.0 / 362880.0))));
}

// Optimal influence function on the r2c half mesh for m = 0 aliasing
// (G_opt<S,0>, p3m/influence_function.hpp:53-150): computed in FP64,
// stored in the working precision.  With m = 0 the force (S=1) and energy
// (S=0) functions are identical, so one array serves both.
template <typename Real>
__global__ void k_influence(const RepGeom *__restrict__ reps, const int2 *__restrict__ blk,
                            Real *__restrict__ ginf) {
  int2 const bk = blk[blockIdx.x];
  RepGeom const &G = reps[bk.x];
  int const M0 = G.mesh[0], M1 = G.mesh[1], M2 = G.mesh[2];
  long long const local = static_cast<long long>(bk.y) * blockDim.x + threadIdx.x;
  long long const csize = static_cast<long long>(M0) * M1 * G.hp;
  if (local >= csize)
    return;
  int const kz = static_cast<int>(local % G.hp);
  int const y = static_cast<int>((local / G.hp) % M1);
  int const x = static_cast<int>(local / (static_cast<long long>(M1) * G.hp));
  double val = 0.0;
  if (kz <= M2 / 2) {
    bool const all_half = (x % (M0 / 2) == 0) && (y % (M1 / 2) == 0) && (kz % (M2 / 2) == 0);
    if (!all_half) {
      auto shift = [](int i, int m) { return (i < m / 2) ? i : i - m; }; // M/2 -> -M/2
      int const sh[3] = {shift(x, M0), shift(y, M1), shift(kz, M2)};
      double k[3], fnm[3];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        k[d] = sh[d] * ((2.0 * kPi) * G.box_i[d]);
        double const h = G.box[d] / G.mesh[d];
        double const wvi = 1.0 / ((2.0 * kPi) / h);
        fnm[d] = sinc_d(k[d] * wvi);
      }
      double const k2 = k[0] * k[0] + k[1] * k[1] + k[2] * k[2];
      if (k2 != 0.0) {
        double const U2 = pow(fnm[0] * fnm[1] * fnm[2], 2.0 * G.cao);
        double const ex = (1.0 / (2.0 * G.alpha)) * (1.0 / (2.0 * G.alpha)) * k2;
        double num = 0.0;
        if (ex < 30.0)
          num = U2 * (exp(-ex) * (4.0 * kPi / k2));
        val = num / (U2 * U2);
      }
    }
  }
  ginf[G.km_off + local] = static_cast<Real>(val);
}

// Per-block FP64 partial sums over particles of one replica:
// {n_charged, sum q, sum q^2, Mx, My, Mz} (p3m.cpp:98-115, 376-386).
__global__ void k_census(const int2 *__restrict__ blk, const RepGeom *__restrict__ reps,
                         const double *__restrict__ pos, const double *__restrict__ q,
                         double *__restrict__ partials) {
  int2 const bk = blk[blockIdx.x];
  RepGeom const &G = reps[bk.x];
  long long const i0 = G.p0 + static_cast<long long>(bk.y) * 2048;
  long long const i1 = min(G.p0 + G.np, i0 + 2048);
  double acc[6] = {0, 0, 0, 0, 0, 0};
  for (long long i = i0 + threadIdx.x; i < i1; i += blockDim.x) {
    double const qi = q[i];
    if (qi != 0.0) {
      acc[0] += 1.0;
      acc[1] += qi;
      acc[2] += qi * qi;
      acc[3] += qi * pos[3 * i + 0];
      acc[4] += qi * pos[3 * i + 1];
      acc[5] += qi * pos[3 * i + 2];
    }
  }
  __shared__ double red[6][32];
  int const lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    double v = acc[k];
    for (int o = 16; o > 0; o >>= 1)
      v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0)
      red[k][wid] = v;
  }
  __syncthreads();
  if (threadIdx.x < 6) {
    double s = 0.0;
    for (int w = 0; w < (blockDim.x >> 5); ++w)
      s += red[threadIdx.x][w];
    partials[static_cast<long long>(blockIdx.x) * 6 + threadIdx.x] = s;
  }
}

// Sum per-block partials of replica blockIdx.x, column blockIdx.y (width
// columns; `per` rows per table block): thread t adds rows t, t + 256, ..., then
// a fixed shuffle tree and the warps in order (deterministic; one thread per
// replica walking all rows and columns took 70 us for 235 rows of 20).
__global__ void __launch_bounds__(256)
k_reduce_partials(const double *__restrict__ partials, int width,
                  const int *__restrict__ blk_start, int per, double *__restrict__ out) {
  int const r = blockIdx.x, k = blockIdx.y;
  int const b0 = blk_start[r] * per, b1 = blk_start[r + 1] * per;
  double s = 0.0;
  for (int b = b0 + static_cast<int>(threadIdx.x); b < b1; b += 256)
    s += partials[static_cast<long long>(b) * width + k];
  for (int o = 16; o > 0; o >>= 1)
    s += __shfl_down_sync(0xffffffffu, s, o);
  __shared__ double red[8];
  if ((threadIdx.x & 31) == 0)
    red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < 8; ++w)
      t += red[w];
    out[static_cast<long long>(r) * width + k] = t;
  }
}

// Closed-form aliasing sum sum_m sinc^(2P)(n/M + m) (Hockney & Eastwood
// eq. 7-66, p3m/math.hpp:92-149).
__device__ inline double cot_sum(int cao, int n, double mesh_i) {
  double const th = static_cast<double>(n) * mesh_i * kPi;
  double const c = cos(th) * cos(th);
  switch (cao) {
  case 1: return 1.0;
  case 2: return (1. + c * 2.) / 3.;
  case 3: return (2. + c * (11. + c * 2.)) / 15.;
  case 4: return (17. + c * (180. + c * (114. + c * 4.))) / 315.;
  case 5: return (62. + c * (1072. + c * (1452. + c * (247. + c * 2.)))) / 2835.;
  case 6:
    return (1382. + c * (35396. + c * (83021. + c * (34096. + c * (2026. + c * 4.))))) / 155925.;
  default:
    return (21844. + c * (776661. + c * (2801040. + c * (2123860. + c * (349500. + c * (8166. + c * 4.)))))) /
           6081075.;
  }
}

// Hockney-Eastwood k-space error sum in FP64 (p3m_k_space_error with
// p3m_tune_aliasing_sums, p3m.cpp:146-243; the GPU version of
// p3m_gpu_error_cuda.cu:47-143), per-block partials, fixed-order reduce.
__global__ void k_ks_error(int M0, int M1, int M2, int cao, double alpha_L,
                           double *__restrict__ partials) {
  long long const total = static_cast<long long>(M0) * M1 * M2;
  double const mi0 = 1.0 / M0, mi1 = 1.0 / M1, mi2 = 1.0 / M2;
  double const f1 = (kPi / alpha_L) * (kPi / alpha_L);
  double acc = 0.0;
  for (long long t = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; t < total;
       t += static_cast<long long>(gridDim.x) * blockDim.x) {
    int const nz = static_cast<int>(t % M2) - M2 / 2;
    int const ny = static_cast<int>((t / M2) % M1) - M1 / 2;
    int const nx = static_cast<int>(t / (static_cast<long long>(M1) * M2)) - M0 / 2;
    if (nx == 0 && ny == 0 && nz == 0)
      continue;
    double const n2 = double(nx) * nx + double(ny) * ny + double(nz) * nz;
    double const cs = cot_sum(cao, nx, mi0) * cot_sum(cao, ny, mi1) * cot_sum(cao, nz, mi2);
    double const ex = exp(-f1 * n2);
    double const en = pow(sinc_d(nx * mi0) * sinc_d(ny * mi1) * sinc_d(nz * mi2), 2.0 * cao);
    double const a1 = ex * ex / n2;
    double const a2 = en * ex * n2 / n2;
    double const d = a1 - (a2 / cs) * (a2 / cs) / n2;
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

} // namespace p3mx
