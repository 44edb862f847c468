// Short-range path (sm_100a): regular-decomposition cell binning, Verlet
// list build, and the real-space erfc-Coulomb + LJ/WCA pair kernel.
#pragma once

#include "common.cuh"
#include "p3m_kernels.cuh"

#include <type_traits>

namespace p3mx {

// LJ/WCA parameters of a type pair, device copy (lj.hpp, wca.hpp).
struct PairIA {
  double lj_eps, lj_sig, lj_cut, lj_shift, lj_offset, lj_min;
  double wca_eps, wca_sig, wca_cut;
  double ia_cut; // max of active cutoffs, -1 when inactive
};

// FP32 offset of a particle from the corner of cell `loc` (cell index inside
// the replica) that it was binned into at the last list build: the folded
// build-time position minus the corner, plus the minimum-image displacement
// since the build (below skin/2 by the Verlet rebuild rule), so the offset
// stays continuous when the particle leaves its cell or crosses the box
// boundary, for any cell grid.  At build time xref = x.
__device__ inline float4 cell_offset(RepGeom const &G, int loc, const double *xref,
                                     const double *x, double q) {
  int const c[3] = {loc % G.cg[0], (loc / G.cg[0]) % G.cg[1], loc / (G.cg[0] * G.cg[1])};
  float o[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    double const cs = G.box[d] / G.cg[d];
    double const v = fold_coord(xref[d], G.box[d]) - c[d] * cs;
    double dd = x[d] - xref[d];
    dd -= G.box[d] * rint(dd * G.box_i[d]);
    o[d] = static_cast<float>(v + dd);
  }
  return make_float4(o[0], o[1], o[2], static_cast<float>(q));
}

// Cell of a folded position, position_to_cell_index
// (RegularDecomposition.cpp:51-80) on a single rank: floor(x/cell)+1,
// clamped to the grid for x < L.  Returns interior coordinates 0..cg-1.
__device__ inline void cell_coords(RepGeom const &G, const double *xf, int *c) {
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    int cp = static_cast<int>(floor(xf[d] * G.inv_cs[d])) + 1;
    if (cp < 1)
      cp = 1;
    else if (cp > G.cg[d])
      cp = G.cg[d];
    c[d] = cp - 1;
  }
}

// Cell key (column-major over the interior grid, x fastest, as the
// reference orders cells) and counting-sort slot of every particle; also
// the folded position (double4 with charge in w) for the pair kernels.  The
// sort runs on G.oct_mult keys per cell (8 when any replica sorts by
// octant, else 1): cell * oct_mult + the octant of the cell the particle
// lies in (each axis halved) where the replica sorts by octant (G.oct_on:
// crowded cells, whose far octants the list build skips), else
// cell * oct_mult; bkey keeps the sort key.
__global__ void k_cell_bin(const RepGeom *__restrict__ reps, const int *__restrict__ rep_of,
                           const double *__restrict__ pos, const double *__restrict__ q,
                           long long n, int *__restrict__ key, int *__restrict__ bkey,
                           int *__restrict__ slot, int *__restrict__ cnt,
                           double4 *__restrict__ pq, int *__restrict__ ghost_index,
                           const int *__restrict__ cond, const int *__restrict__ rflag) {
  if (cond && !*cond)
    return;
  long long const i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n)
    return;
  RepGeom const &G = reps[rep_of[i]];
  double xf[3];
#pragma unroll
  for (int d = 0; d < 3; ++d)
    xf[d] = fold_coord(pos[3 * i + d], G.box[d]);
  int c[3];
  cell_coords(G, xf, c);
  int kb;
  if (rflag && !rflag[rep_of[i]]) {
    // replica keeps its lists: same cells, hence the same sorted order
    kb = bkey[i];
  } else {
    int const k = static_cast<int>(G.cell_off) + c[0] + G.cg[0] * (c[1] + G.cg[1] * c[2]);
    int oct = 0;
    if (G.oct_on) {
#pragma unroll
      for (int d = 0; d < 3; ++d)
        oct |= (xf[d] * G.inv_cs[d] - c[d] >= 0.5) ? (1 << d) : 0;
    }
    kb = G.oct_mult * k + oct;
    key[i] = k;
    bkey[i] = kb;
  }
  slot[i] = atomicAdd(&cnt[kb], 1);
  pq[i] = make_double4(xf[0], xf[1], xf[2], q[i]);
  if (ghost_index) {
    int const g0 = G.cg[0] + 2, g1 = G.cg[1] + 2;
    ghost_index[i] = (c[0] + 1) + g0 * ((c[1] + 1) + g1 * (c[2] + 1));
  }
}

// Gather particle data into cell-sorted order (and the inverse permutation).
__global__ void k_cell_gather(const RepGeom *__restrict__ reps, const int *__restrict__ rep_of,
                              const int *__restrict__ perm, const double4 *__restrict__ pq,
                              const int *__restrict__ type, const int *__restrict__ key,
                              long long n, double4 *__restrict__ spq, float4 *__restrict__ spf,
                              int *__restrict__ stype, int *__restrict__ scell,
                              int *__restrict__ inv, const int *__restrict__ cond) {
  if (cond && !*cond)
    return;
  long long const s = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (s >= n)
    return;
  int const i = perm[s];
  inv[i] = static_cast<int>(s); // sorted slot of particle i
  double4 const v = pq[i];
  spq[s] = v;
  stype[s] = type ? type[i] : 0;
  scell[s] = key[i];
  RepGeom const &G = reps[rep_of[i]];
  double const xv[3] = {v.x, v.y, v.z};
  spf[s] = cell_offset(G, key[i] - static_cast<int>(G.cell_off), xv, xv, v.w);
}

__device__ inline double mi_d(double dx, double L, double Li) {
  // get_mi_coord (BoxGeometry.hpp:47-60)
  if (fabs(dx) > 0.5 * L)
    return dx - rint(dx * Li) * L;
  return dx;
}

// Verlet list layout: per warp tile of 32 consecutive particles of a replica,
// each particle's entries in groups of 8 (one 32-byte sector), the groups of
// the 32 particles interleaved: entry k of local particle la at
//   nb_off + ((la/32) * (cap/8) + k/8) * 256 + (la%32) * 8 + k%8
// (cap, the per-replica capacity, a multiple of 8).  The build writes whole
// groups with vector stores and the pair kernels read whole groups with
// vector loads.  An entry packs the partner's index inside the replica
// (upper 26 bits) and its cell offset code (cell_offset_code, lower 6 bits:
// one mask-and-or turns a field into an FP32 value).  The entries behind the
// last of a group's are the particle itself with dc = 0.
constexpr int kNbIndexBits = 26;
constexpr int kNbCodeBits = 6;
__host__ __device__ constexpr unsigned nb_index(unsigned e) { return e >> kNbCodeBits; }
__host__ __device__ constexpr unsigned nb_pack(unsigned index, int code) {
  return (index << kNbCodeBits) | static_cast<unsigned>(code);
}
// Cell offset code of an entry: the partner image's cell offset dc (each
// axis -1, 0 or +1) as three 2-bit fields dc + 1 (x lowest).
__host__ __device__ constexpr int cell_offset_code(int dx, int dy, int dz) {
  return (dx + 1) | ((dy + 1) << 2) | ((dz + 1) << 4);
}
// 4^d dc of axis d from an entry, as an FP32 value (exact: 2^23 + field,
// minus 2^23 + 4^d)
__device__ inline float code_axis(unsigned e, int d) {
  return __uint_as_float(0x4B000000u | (e & (3u << (2 * d)))) -
         (8388608.0f + static_cast<float>(1 << (2 * d)));
}
// First entry (group 0) of local particle la; group g at + g * 256.
__host__ __device__ inline long long nb_base(long long nb_off, int cap, long long la) {
  return nb_off + (((la >> 5) * (cap >> 3)) << 8) + ((la & 31) << 3);
}
__host__ __device__ inline long long nb_entry(long long base, int k) {
  return base + (static_cast<long long>(k >> 3) << 8) + (k & 7);
}
// Two classes of entries share a particle's capacity: class A (the pair's
// LJ / WCA range plus the skin at build time: all terms) fills groups from
// the first one up, class B (beyond it: the pair stays outside the LJ / WCA
// cutoff until the next rebuild, as no particle moves more than skin/2, so
// only Coulomb can act) fills groups from the last one down.  nb_cnt packs
// nA (low 16 bits) and nB (high 16 bits).
__host__ __device__ inline int nb_count_a(int c) { return c & 0xFFFF; }
__host__ __device__ inline int nb_count_b(int c) { return static_cast<int>(static_cast<unsigned>(c) >> 16); }
__host__ __device__ inline int nb_count(int c) { return nb_count_a(c) + nb_count_b(c); }
// Group g of class B (g = 0 the first).
__host__ __device__ inline long long nb_group_b(long long base, int cap, int g) {
  return base + (static_cast<long long>((cap >> 3) - 1 - g) << 8);
}
// Entry k of the logical list [class A entries, class B entries].
__host__ __device__ inline long long nb_logical(long long base, int cap, int na, int k) {
  if (k < na)
    return nb_entry(base, k);
  int const kk = k - na;
  return nb_group_b(base, cap, kk >> 3) + (kk & 7);
}

// Copy one group of 8 entries (32 bytes, 16-byte aligned on both sides).
__device__ inline void store_group(int *p, const int *g) {
  reinterpret_cast<int4 *>(p)[0] = reinterpret_cast<const int4 *>(g)[0];
  reinterpret_cast<int4 *>(p)[1] = reinterpret_cast<const int4 *>(g)[1];
}

// Verlet list (full, both directions) of every cell-sorted particle a:
// partners b != a in the 27 (unique) neighbour cells with the
// VerletCriterion (VerletCriterion.hpp:68-97): d^2 <= (max_cut+skin)^2 and
// (both charged and d^2 <= (r_cut+skin)^2, or the type pair is active and
// d^2 <= (ia_cut+skin)^2).  Stored in the warp-tiled layout above
// (per-replica capacity G.max_nb), class A entries (type pair active and
// d^2 <= (ia_cut+skin)^2) from the first group up, class B from the last
// group down; a replica whose capacity is exceeded reports the capacity it
// needs in overflow[replica] (nothing more is stored for that particle and
// its counts are those of the entries stored).
// Verlet list of one cell-sorted particle a (k_verlet_build); gbuf / gbuf_b
// are the lane's shared-memory buffers of the class A / B group being
// filled, s_icut the ia_cut table of the type pairs in shared memory.
template <bool OCT>
__device__ inline void verlet_build_one(long long a, const RepGeom *__restrict__ reps,
                                        const int *__restrict__ rep_of_sorted,
                                        const double4 *__restrict__ spq,
                                        const float4 *__restrict__ spf,
                                        const int *__restrict__ stype,
                                        const int *__restrict__ scell,
                                        const int *__restrict__ cstart,
                                        const PairIA *__restrict__ ia, int ntypes,
                                        int *__restrict__ nb, int *__restrict__ nb_cnt,
                                        int *__restrict__ overflow,
                                        const int *__restrict__ rflag, const float *s_icut,
                                        int *gbuf, int *gbuf_b) {
  int const rep = rep_of_sorted[a];
  if (rflag && !rflag[rep])
    return; // this replica keeps its list
  RepGeom const &G = reps[rep];
  int const max_nb = G.max_nb;
  int *nbp = nb + nb_base(G.nb_off, max_nb, a - G.p0);
  int const ngroups = max_nb >> 3;
  double4 const pa = spq[a];
  double const cs[3] = {G.box[0] / G.cg[0], G.box[1] / G.cg[1], G.box[2] / G.cg[2]};
  double const ics[3] = {G.cg[0] * G.box_i[0], G.cg[1] * G.box_i[1], G.cg[2] * G.box_i[2]};
  bool const small_grid = (G.cg[0] < 3) || (G.cg[1] < 3) || (G.cg[2] < 3);
  // FP32 geometry on the cell-relative offsets (error ~1e-6 of the cell
  // size): a candidate whose FP32 distance lies within a relative band of
  // 1e-4 around one of its thresholds is decided by the FP64 minimum-image
  // test (the reference's criterion); all others are decided in FP32, which
  // cannot differ from FP64 outside the band, so the pair set is the FP64 one
  float4 const pfa = spf[a];
  float const csf[3] = {static_cast<float>(cs[0]), static_cast<float>(cs[1]),
                        static_cast<float>(cs[2])};
  int const ta = stype[a];
  int const loc = scell[a] - static_cast<int>(G.cell_off);
  int const c0 = loc % G.cg[0];
  int const c1 = (loc / G.cg[0]) % G.cg[1];
  int const c2 = loc / (G.cg[0] * G.cg[1]);
  double const emax2 = (G.max_cut + G.skin) * (G.max_cut + G.skin);
  float const emax2_pre = static_cast<float>(emax2 * (1.0 + 1e-4));
  double const ecoul2 = (G.coulomb_cut > 0.0) ? (G.coulomb_cut + G.skin) * (G.coulomb_cut + G.skin) : -1.0;
  // Coulomb threshold band in FP32 (no Coulomb pairs when a is uncharged)
  bool const coul_a = ecoul2 >= 0.0 && pa.w != 0.0;
  float const ec_lo = static_cast<float>(ecoul2 * (1.0 - 1e-4));
  float const ec_hi = static_cast<float>(ecoul2 * (1.0 + 1e-4));
  float const skin_f = static_cast<float>(G.skin);
  double const Li[3] = {G.box_i[0], G.box_i[1], G.box_i[2]};
  int na = 0, nb_b = 0; // entries stored per class
  int need_a = 0, need_b = 0; // entries found per class
  // store one taken entry of class A (LJ / WCA range) or B
  auto put = [&](int b, bool cls_a, int code) {
    // room for the entry: class A groups [0, ceil(na'/8)) and class B
    // groups [ngroups - ceil(nb'/8), ngroups) disjoint
    bool const room = (need_a == na) && (need_b == nb_b) &&
                      ((cls_a ? (na & 7) : (nb_b & 7)) != 0 ||
                       ((na + 7) >> 3) + ((nb_b + 7) >> 3) + 1 <= ngroups);
    if (room) {
      int const ent = static_cast<int>(nb_pack(static_cast<unsigned>(b - G.p0), code));
      if (cls_a) {
        int const slot = na & 7;
        gbuf[slot] = ent;
        if (slot == 7)
          store_group(nbp + (static_cast<long long>(na >> 3) << 8), gbuf);
        ++na;
      } else {
        int const slot = nb_b & 7;
        gbuf_b[slot] = ent;
        if (slot == 7)
          store_group(nbp + (static_cast<long long>(ngroups - 1 - (nb_b >> 3)) << 8), gbuf_b);
        ++nb_b;
      }
    }
    if (cls_a)
      ++need_a;
    else
      ++need_b;
  };
  // offsets per axis without duplicates for grids of size 1 or 2
  int lo[3], hi[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    lo[d] = (G.cg[d] >= 3) ? -1 : 0;
    hi[d] = (G.cg[d] >= 2) ? 1 : 0;
  }
  for (int dz = lo[2]; dz <= hi[2]; ++dz) {
    int z = c2 + dz;
    z = (z < 0) ? z + G.cg[2] : (z >= G.cg[2] ? z - G.cg[2] : z);
    for (int dy = lo[1]; dy <= hi[1]; ++dy) {
      int y = c1 + dy;
      y = (y < 0) ? y + G.cg[1] : (y >= G.cg[1] ? y - G.cg[1] : y);
      for (int dx = lo[0]; dx <= hi[0]; ++dx) {
        int x = c0 + dx;
        x = (x < 0) ? x + G.cg[0] : (x >= G.cg[0] ? x - G.cg[0] : x);
        int const cell = static_cast<int>(G.cell_off) + x + G.cg[0] * (y + G.cg[1] * z);
        if (!small_grid) {
          // skip a neighbour cell lying wholly beyond the list range: distance
          // from the particle (cell-relative offset) to the cell's box
          float const ax = (dx == 0) ? 0.f : (dx > 0 ? csf[0] - pfa.x : pfa.x);
          float const ay = (dy == 0) ? 0.f : (dy > 0 ? csf[1] - pfa.y : pfa.y);
          float const az = (dz == 0) ? 0.f : (dz > 0 ? csf[2] - pfa.z : pfa.z);
          float const bx = fmaxf(ax, 0.f), by = fmaxf(ay, 0.f), bz = fmaxf(az, 0.f);
          if (bx * bx + by * by + bz * bz > emax2_pre)
            continue;
        }
        float const shx = -dx * csf[0], shy = -dy * csf[1], shz = -dz * csf[2];
        // exact (FP64 minimum-image) test and store of one candidate
        auto consider = [&](int b) {
            double4 const pb = spq[b];
            double const d0 = mi_d(pa.x - pb.x, G.box[0], Li[0]);
            double const d1 = mi_d(pa.y - pb.y, G.box[1], Li[1]);
            double const d2v = mi_d(pa.z - pb.z, G.box[2], Li[2]);
            double const d2 = d0 * d0 + d1 * d1 + d2v * d2v;
            if (d2 > emax2)
              return;
            double const ic = ia[ta * ntypes + stype[b]].ia_cut;
            bool const cls_a = (ic != -1.0) && d2 <= (ic + G.skin) * (ic + G.skin);
            bool const take =
                cls_a || (ecoul2 >= 0.0 && d2 <= ecoul2 && pa.w != 0.0 && pb.w != 0.0);
            if (take) {
              // cell offset dc of the partner's image: x_b' - x_a = dc cs +
              // (off_b - off_a), an exact multiple of the cell size; with
              // cells >= the list range, dc is -1, 0 or +1 per axis.  With
              // 3 or more cells along an axis the minimum image is the image
              // in the visited neighbour cell, so dc is the loop offset;
              // with 1 or 2 cells it follows from the minimum-image vector.
              int dcv[3] = {dx, dy, dz};
              if (small_grid) {
                int const lb = scell[b] - static_cast<int>(G.cell_off);
                int const cb[3] = {lb % G.cg[0], (lb / G.cg[0]) % G.cg[1],
                                   lb / (G.cg[0] * G.cg[1])};
                int const ca[3] = {c0, c1, c2};
                double const xa[3] = {pa.x, pa.y, pa.z}, xb[3] = {pb.x, pb.y, pb.z};
                double const dmi[3] = {-d0, -d1, -d2v};
#pragma unroll
                for (int d = 0; d < 3; ++d)
                  if (G.cg[d] < 3) {
                    double const oa = xa[d] - ca[d] * cs[d], ob = xb[d] - cb[d] * cs[d];
                    dcv[d] = static_cast<int>(rint((dmi[d] - (ob - oa)) * ics[d]));
                  }
              }
              put(b, cls_a, cell_offset_code(dcv[0], dcv[1], dcv[2]));
            }
        };
        if (small_grid) {
          int const om = G.oct_mult;
          int const b_lo = cstart[om * cell], b_hi = cstart[om * cell + om];
          for (int b = b_lo; b < b_hi; ++b)
            if (b != a)
              consider(b);
        } else {
          int const code = cell_offset_code(dx, dy, dz);
          // with octant-sorted cells, the octants of the neighbour cell
          // wholly beyond the list range are skipped (the particle relative
          // to the neighbour cell's corner against each half-cell box)
          float const qx = pfa.x + shx, qy = pfa.y + shy, qz = pfa.z + shz;
          float const hx = 0.5f * csf[0], hy = 0.5f * csf[1], hz = 0.5f * csf[2];
          int const noct = (OCT && G.oct_on) ? 8 : 1;
          for (int oct = 0; oct < noct; ++oct) {
          int b_lo = cstart[G.oct_mult * cell], b_hi = cstart[G.oct_mult * (cell + 1)];
          if (OCT && G.oct_on) {
            float const lx = (oct & 1) ? hx : 0.f, ly = (oct & 2) ? hy : 0.f,
                        lz = (oct & 4) ? hz : 0.f;
            float const ex = fmaxf(fmaxf(lx - qx, qx - (lx + hx)), 0.f);
            float const ey = fmaxf(fmaxf(ly - qy, qy - (ly + hy)), 0.f);
            float const ez = fmaxf(fmaxf(lz - qz, qz - (lz + hz)), 0.f);
            if (ex * ex + ey * ey + ez * ez > emax2_pre)
              continue;
            b_lo = cstart[G.oct_mult * cell + oct];
            b_hi = cstart[G.oct_mult * cell + oct + 1];
          }
          // kPre candidates per round (loads issued together): an FP32
          // pre-check, then for the candidates near or inside the list
          // range the FP32 decision, or the FP64 test inside the bands
          constexpr int kPre = 8;
          for (int b0 = b_lo; b0 < b_hi; b0 += kPre) {
            float4 pf[kPre];
#pragma unroll
            for (int u = 0; u < kPre; ++u)
              pf[u] = (b0 + u < b_hi) ? spf[b0 + u] : pfa;
            unsigned keep = 0;
            float r2v[kPre];
#pragma unroll
            for (int u = 0; u < kPre; ++u) {
              float const e0 = (pfa.x - pf[u].x) + shx, e1 = (pfa.y - pf[u].y) + shy,
                          e2 = (pfa.z - pf[u].z) + shz;
              r2v[u] = e0 * e0 + e1 * e1 + e2 * e2;
              bool const in = (b0 + u < b_hi) && (b0 + u != a) && (r2v[u] <= emax2_pre);
              keep |= (in ? 1u : 0u) << u;
            }
            while (keep) {
              int const u = __ffs(keep) - 1;
              keep &= keep - 1;
              int const b = b0 + u;
              float r2 = r2v[0];
              float qb = pf[0].w;
#pragma unroll
              for (int w = 1; w < kPre; ++w) {
                r2 = (u == w) ? r2v[w] : r2;
                qb = (u == w) ? pf[w].w : qb;
              }
              float const icf = (ntypes == 1) ? s_icut[0] : s_icut[ta * ntypes + stype[b]];
              float const it = icf + skin_f;
              float const it2 = it * it;
              bool const ia_on = icf != -1.f;
              bool const a_lo = ia_on && r2 < it2 * (1.f - 1e-4f);
              bool const a_band = ia_on && !a_lo && r2 <= it2 * (1.f + 1e-4f);
              // Coulomb: both charged (an FP32 zero charge is checked in FP64)
              bool const c_lo = coul_a && qb != 0.f && r2 < ec_lo;
              bool const c_band = coul_a && r2 <= ec_hi && !c_lo;
              if (a_band || c_band)
                consider(b);
              else if (a_lo || c_lo)
                put(b, a_lo, code);
            }
          }
          }
        }
      }
    }
  }
  // last partial groups, filled up with the particle itself (zero distance:
  // no term of a pair kernel passes its range test)
  int const self = static_cast<int>(
      nb_pack(static_cast<unsigned>(a - G.p0), cell_offset_code(0, 0, 0)));
  for (int k = na & 7; k != 0 && k < 8; ++k)
    gbuf[k] = self;
  for (int k = nb_b & 7; k != 0 && k < 8; ++k)
    gbuf_b[k] = self;
  if (na & 7)
    store_group(nbp + (static_cast<long long>(na >> 3) << 8), gbuf);
  if (nb_b & 7)
    store_group(nbp + (static_cast<long long>(ngroups - 1 - (nb_b >> 3)) << 8), gbuf_b);
  nb_cnt[a] = na | (nb_b << 16);
  int const need = 8 * (((need_a + 7) >> 3) + ((need_b + 7) >> 3));
  if (need > max_nb)
    atomicMax(&overflow[rep], need);
}

// Verlet lists, one thread per cell-sorted particle (the 32 lanes of a warp
// are consecutive particles: the same or adjacent cells).
template <bool OCT>
__global__ void __launch_bounds__(256, 2)
k_verlet_build(const RepGeom *__restrict__ reps, const int *__restrict__ rep_of_sorted,
               const double4 *__restrict__ spq, const float4 *__restrict__ spf,
               const int *__restrict__ stype, const int *__restrict__ scell,
               const int *__restrict__ cstart, const PairIA *__restrict__ ia, int ntypes,
               long long n, int *__restrict__ nb, int *__restrict__ nb_cnt,
               int *__restrict__ overflow, const int *__restrict__ cond,
               const int *__restrict__ rflag) {
  if (cond && !*cond)
    return;
  __shared__ __align__(16) int s_group[256 * 8], s_group_b[256 * 8];
  // ia_cut of every type pair (-1: inactive) in shared memory (the skin,
  // per replica, is added per candidate)
  extern __shared__ float s_icut[];
  for (int k = threadIdx.x; k < ntypes * ntypes; k += blockDim.x)
    s_icut[k] = static_cast<float>(ia[k].ia_cut);
  __syncthreads();
  long long const a = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (a >= n)
    return;
  verlet_build_one<OCT>(a, reps, rep_of_sorted, spq, spf, stype, scell, cstart, ia, ntypes, nb,
                   nb_cnt, overflow, rflag, s_icut, s_group + threadIdx.x * 8,
                   s_group_b + threadIdx.x * 8);
}

// FP32 exp(x) over the real-space kernels' range (x = -(alpha r)^2 in [-88, 0]), the
// accurate form that p3mx_exp_check sets beside the kernels' single ex2:
// e^x = 2^y with y = x log2(e) split error-free into y_hi + y_lo (the FMA
// residual of the product, Dekker's TwoProduct, plus the low part of the
// constant), then 2^y = 2^y_hi (hardware ex2.approx, ~2 ulp) * (1 + y_lo ln 2).
// Relative error ~2^-21 over the range, against ~2^-24 * |y| for a plain
// ex2(x * log2 e).
__device__ inline float exp_fast(float x) {
  float const l2e_hi = 1.44269502162933349609375f;    // log2(e) rounded to FP32
  float const l2e_lo = 1.9259629911266175e-8f;        // log2(e) - l2e_hi
  float const y_hi = x * l2e_hi;
  float const y_lo = fmaf(x, l2e_hi, -y_hi) + x * l2e_lo;
  float e;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(y_hi));
  return fmaf(e, y_lo * 0.693147180559945309f, e);
}

// Reciprocal in the working precision: FP32 uses the hardware approximation
// (~1 ulp; the FP32-mixed path tolerates ulp-level differences); FP64 keeps the
// IEEE division.
template <typename Real> __device__ inline Real rcp_r(Real x);
template <> __device__ inline float rcp_r<float>(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
template <> __device__ inline double rcp_r<double>(double x) { return 1.0 / x; }

// LJ/WCA parameters of one type pair in the working precision.
template <typename Real> struct PairR {
  Real lcut, lmin, loff, lsig, leps, lshift, wcut, wsig, weps;
  bool active;
  __device__ explicit PairR(PairIA const &p)
      : lcut(static_cast<Real>(p.lj_cut + p.lj_offset)),
        lmin(static_cast<Real>(p.lj_min + p.lj_offset)), loff(static_cast<Real>(p.lj_offset)),
        lsig(static_cast<Real>(p.lj_sig)), leps(static_cast<Real>(p.lj_eps)),
        lshift(static_cast<Real>(p.lj_shift)), wcut(static_cast<Real>(p.wca_cut)),
        wsig(static_cast<Real>(p.wca_sig)), weps(static_cast<Real>(p.wca_eps)),
        active(p.ia_cut != -1.0) {}
};

// LJ + WCA force factor and energy of one pair (lj.hpp:41-60, wca.hpp:39-55).
template <typename Real>
__device__ inline void lj_wca(PairR<Real> const &p, Real dist, Real inv_d, Real &fn, Real &en) {
  if (dist < p.lcut && dist > p.lmin) {
    Real const r_off = dist - p.loff;
    Real const inv_off = rcp_r(r_off);
    Real const s = p.lsig * inv_off;
    Real const s2 = s * s;
    Real const f6 = s2 * s2 * s2;
    fn += Real(48) * p.leps * f6 * (f6 - Real(0.5)) * (inv_off * inv_d);
    en += Real(4) * p.leps * (f6 * f6 - f6 + p.lshift);
  }
  if (dist < p.wcut) {
    Real const s = p.wsig * inv_d;
    Real const s2 = s * s;
    Real const f6 = s2 * s2 * s2;
    fn += Real(48) * p.weps * f6 * (f6 - Real(0.5)) * (inv_d * inv_d);
    en += Real(4) * p.weps * (f6 * f6 - f6 + Real(0.25));
  }
}

// Branch-free form of lj_wca for the FP32 kernel: every term is evaluated
// and selected by its range test (the lanes of a warp, different particles,
// would otherwise diverge on the tests); WCA only when the pair has it.
__device__ inline void lj_wca_sel(PairR<float> const &p, float dist, float inv_d, float &fn,
                                  float &en) {
  {
    float const r_off = dist - p.loff;
    float const inv_off = rcp_r(r_off);
    float const s = p.lsig * inv_off;
    float const s2 = s * s;
    float const f6 = s2 * s2 * s2;
    bool const in = dist < p.lcut && dist > p.lmin;
    fn += in ? 48.f * p.leps * f6 * (f6 - 0.5f) * (inv_off * inv_d) : 0.f;
    en += in ? 4.f * p.leps * (f6 * f6 - f6 + p.lshift) : 0.f;
  }
  if (p.wcut > 0.f) {
    float const s = p.wsig * inv_d;
    float const s2 = s * s;
    float const f6 = s2 * s2 * s2;
    bool const in = dist < p.wcut;
    fn += in ? 48.f * p.weps * f6 * (f6 - 0.5f) * (inv_d * inv_d) : 0.f;
    en += in ? 4.f * p.weps * (f6 * f6 - f6 + 0.25f) : 0.f;
  }
}

// 2^x, hardware approximation (ex2.approx, relative error ~2^-22).
__device__ inline float ex2_approx(float x) {
  float e;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(x));
  return e;
}

// The FP32 exponentials of the real-space kernels on n values, for their
// accuracy test: out[k] = exp_fast(x), out[n + k] = one ex2.approx of
// x log2(e) rounded to FP32 (the form of the force-only kernel, which folds
// log2(e) into its coefficient), out[2n + k] = CUDA's expf(x).
__global__ void k_exp_check(long long n, const float *__restrict__ x, float *__restrict__ out) {
  long long const k = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k >= n)
    return;
  float const v = x[k];
  out[k] = exp_fast(v);
  out[n + k] = ex2_approx(v * 1.44269504088896341f);
  out[2 * n + k] = expf(v);
}

__device__ inline float rsqrt_approx(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Two FP32 values in one register pair and their packed arithmetic (one
// instruction for both, each half rounded as the scalar operation).
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pk2(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 up2(f32x2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) {
  return fma2(b, pk2(-1.0f, -1.0f), a); // exact product: one rounding
}

// Reciprocal in FP64 from the FP32 approximation by one step of the third-order
// iteration y' = y + y (e + e^2), e = 1 - x y (Householder, The Numerical
// Treatment of a Single Nonlinear Equation, 1970; the truncated geometric series
// of 1 / (1 - e)).  |e| < 2^-21, so the step leaves a relative error of e^3 <
// 2^-63 beside the last FMA's rounding: below 2^-53 (1 + 2^-8), within 2^-8 of
// the correctly rounded quotient's bound; x of FP32's normal range (1 + p alpha r
// here).
__device__ inline double rcp_newton(double x) {
  double const y = static_cast<double>(rcp_r<float>(static_cast<float>(x)));
  double const e = fma(-x, y, 1.0);
  return fma(y, fma(e, e, e), y);
}

// The FP64 reciprocal and CUDA's rsqrt of the FP64 pair kernels on n values, for
// their accuracy test: out[k] = rcp_newton(x), out[n + k] = rsqrt(x).
__global__ void k_rcp_check(long long n, const double *__restrict__ x, double *__restrict__ out) {
  long long const k = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k >= n)
    return;
  out[k] = rcp_newton(x[k]);
  out[n + k] = rsqrt(x[k]);
}

// LJ / WCA parameters of a type pair for the FP32 force kernel; ranges of an
// inactive pair are empty (-1).
struct __align__(16) PairF {
  float lcut, lmin, lsig, le48, wcut, wsig, we48, loff;
};
__device__ inline PairF pair_f(PairIA const &p) {
  bool const on = p.ia_cut != -1.0;
  PairF r;
  r.lcut = on ? static_cast<float>(p.lj_cut + p.lj_offset) : -1.f;
  r.lmin = static_cast<float>(p.lj_min + p.lj_offset);
  r.lsig = static_cast<float>(p.lj_sig);
  r.le48 = 48.f * static_cast<float>(p.lj_eps);
  r.wcut = on ? static_cast<float>(p.wca_cut) : -1.f;
  r.wsig = static_cast<float>(p.wca_sig);
  r.we48 = 48.f * static_cast<float>(p.wca_eps);
  r.loff = static_cast<float>(p.lj_offset);
  return r;
}
// Parameter modes of the FP32 force kernel: one type without LJ offset
// (parameters in registers, the LJ powers from the Coulomb term's 1/r^2),
// several types without offsets, LJ offsets.
constexpr int kPairOneType = 0, kPairTypes = 1, kPairOffset = 2;
// Resident blocks per SM (Engine::pair_lanes) of the force kernels, FP32 and FP64,
// and of the FP64 kernel with energies and virials (174 registers).
constexpr int kPairBlocks32 = 4, kPairBlocks64 = 2, kPairBlocks64Ev = 1;
// Tenths of waves up to which two lanes per particle replace one
// (Engine::pair_lanes): one particle type and FP64; several types and dipoles.
constexpr int kPairTail = 15, kPairTailLong = 18;

// Force kernel of the FP32-mixed path over the Verlet list: real-space Coulomb
// (CoulombP3M::pair_force, p3m.hpp:146-180) plus LJ and WCA (lj.hpp:41-60,
// wca.hpp:39-55).  Positions are FP32 offsets from each particle's build-time
// cell corner (cell_offset), the list stores every partner's cell offset
// code, so
//   d = x_a - x_b' = (off_a - off_b) - dc * cs
// is formed in FP32 from small numbers (no minimum-image arithmetic, 16-byte
// gathers); the geometry error is about one ulp of the cell size.
// LPP lanes share a particle (lane `sub` takes the list groups sub, sub + LPP,
// ...); no atomics: each particle owns its force (full list), lane sums meet
// in a fixed shuffle order.  Per-particle sums are FP32 over the 8 entries of
// a group and FP64 across groups.
// Bound by instruction issue (about 45 scalar instructions per entry and
// three MUFU operations): the range-independent arithmetic runs on two
// entries at a time in packed FP32, with the scalar code's roundings.  The kernel
// alone at density 0.5, cutoff 3.5: 2^20 ions 294 -> 271 us, 131 072 ions 49 -> 42 us.
template <int MODE, int LPP>
__global__ void __launch_bounds__(256, kPairBlocks32)
k_pair_forces_rel(const RepGeom *__restrict__ reps, const int2 *__restrict__ blk,
                  const float4 *__restrict__ spf, const int *__restrict__ stype,
                  const int *__restrict__ perm, const PairIA *__restrict__ ia_g, int ntypes,
                  const int *__restrict__ nb, const int *__restrict__ nb_cnt,
                  double *__restrict__ f, int overwrite, double *__restrict__) {
  pdl_enter();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  PairF *ia = reinterpret_cast<PairF *>(smem_raw);
  for (int k = threadIdx.x; k < ntypes * ntypes; k += blockDim.x)
    ia[k] = pair_f(ia_g[k]);
  int2 const bk = blk[blockIdx.x / LPP];
  RepGeom const &G = reps[bk.x];
  float const cs_x = static_cast<float>(G.box[0] / G.cg[0]);
  float const cs_y = static_cast<float>(G.box[1] / G.cg[1]);
  float const cs_z = static_cast<float>(G.box[2] / G.cg[2]);
  __syncthreads();
  int const sub = threadIdx.x % LPP;
  long long const la = static_cast<long long>(bk.y) * 256 + (blockIdx.x % LPP) * (256 / LPP) +
                       threadIdx.x / LPP;
  bool const active = la < G.np;
  long long const a = G.p0 + la;
  // groups of 8 entries: class A first (all terms), then class B (Coulomb
  // only); the loop runs to the warp's largest group count so that the vote on
  // LJ stays warp-wide
  int na = 0, nbb = 0;
  if (active) {
    int const c = nb_cnt[a];
    na = nb_count_a(c);
    nbb = nb_count_b(c);
  }
  int const ga = (na + 7) >> 3, gt = ga + ((nbb + 7) >> 3);
  int const gmax = __reduce_max_sync(0xffffffffu, gt);
  float4 const pa = active ? spf[a] : make_float4(0.f, 0.f, 0.f, 0.f);
  int const ta = (MODE != kPairOneType && active) ? stype[a] * ntypes : 0;
  float const rc2 = static_cast<float>(G.r_cut * G.r_cut);
  float const two_a = static_cast<float>(2.0 * G.alpha / sqrt(kPi));
  float const pref_qa = static_cast<float>(G.prefactor) * pa.w;
  // exp(-(alpha r)^2) = 2^(c_exp r^2); A&S t = 1 / (1 + p alpha r)
  float const c_exp = static_cast<float>(-G.alpha * G.alpha * 1.4426950408889634);
  float const p_alpha = static_cast<float>(0.3275911 * G.alpha);
  PairF const p0 = ia[0];
  double fx = 0.0, fy = 0.0, fz = 0.0;
  const int *nbp = nb + nb_base(G.nb_off, G.max_nb, active ? la : 0);
  int const ngroups = G.max_nb >> 3;
  const float4 *pos = spf + G.p0;
  const int *typ = stype + G.p0;
  f32x2 const pa_xy = pk2(pa.x, pa.y), ncs_xy = pk2(-cs_x, -0.25f * cs_y);
  float const ncs_z = -0.0625f * cs_z;
  // two entries: Coulomb always, LJ / WCA when the group may hold class A
  auto two = [&](auto lj, unsigned const *e, float4 const *pb, float &sx, float &sy, float &sz) {
    float dx[2], dy[2], dz[2], r2[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      // d = (x_a - x_b) - dc cs (dc in {-1, 0, 1}: the product is exact); the
      // y and z fields carry factors 4 and 16 that the cell sizes undo
      f32x2 const dc = pk2(code_axis(e[u], 0), code_axis(e[u], 1));
      float2 const xy = up2(fma2(dc, ncs_xy, sub2(pa_xy, pk2(pb[u].x, pb[u].y))));
      dx[u] = xy.x;
      dy[u] = xy.y;
      dz[u] = fmaf(code_axis(e[u], 2), ncs_z, pa.z - pb[u].z);
      r2[u] = dx[u] * dx[u] + dy[u] * dy[u] + dz[u] * dz[u];
    }
    f32x2 const d2 = pk2(r2[0], r2[1]);
    f32x2 const inv = pk2(rsqrt_approx(r2[0]), rsqrt_approx(r2[1]));
    f32x2 const dist = mul2(d2, inv);
    float2 const ea = up2(mul2(pk2(c_exp, c_exp), d2));
    f32x2 const ex = pk2(ex2_approx(ea.x), ex2_approx(ea.y));
    float2 const td = up2(fma2(pk2(p_alpha, p_alpha), dist, pk2(1.f, 1.f)));
    f32x2 const t = pk2(rcp_r(td.x), rcp_r(td.y));
    f32x2 poly = fma2(t, pk2(1.061405429f, 1.061405429f), pk2(-1.453152027f, -1.453152027f));
    poly = fma2(t, poly, pk2(1.421413741f, 1.421413741f));
    poly = fma2(t, poly, pk2(-0.284496736f, -0.284496736f));
    poly = fma2(t, poly, pk2(0.254829592f, 0.254829592f));
    f32x2 const er = mul2(mul2(t, poly), inv);
    f32x2 const pq = mul2(pk2(pref_qa, pref_qa), pk2(pb[0].w, pb[1].w));
    f32x2 const i2 = mul2(inv, inv);
    float2 const fc = up2(mul2(mul2(mul2(pq, ex), add2(er, pk2(two_a, two_a))), i2));
    float fcv[2] = {fc.x, fc.y};
    float fnv[2] = {0.f, 0.f};
    if constexpr (decltype(lj)::value) {
      float2 const dv = up2(dist), iv = up2(inv);
      float const dd[2] = {dv.x, dv.y}, ii[2] = {iv.x, iv.y};
      if constexpr (MODE == kPairOneType) {
        if (p0.le48 != 0.f) {
          f32x2 const s2 = mul2(pk2(p0.lsig * p0.lsig, p0.lsig * p0.lsig), i2);
          f32x2 const f6 = mul2(mul2(s2, s2), s2);
          float2 const v = up2(mul2(mul2(mul2(pk2(p0.le48, p0.le48), f6),
                                         add2(f6, pk2(-0.5f, -0.5f))), i2));
          fnv[0] = (dd[0] < p0.lcut && dd[0] > p0.lmin) ? v.x : 0.f;
          fnv[1] = (dd[1] < p0.lcut && dd[1] > p0.lmin) ? v.y : 0.f;
        }
        if (p0.wcut > 0.f) {
          f32x2 const s2 = mul2(pk2(p0.wsig * p0.wsig, p0.wsig * p0.wsig), i2);
          f32x2 const f6 = mul2(mul2(s2, s2), s2);
          float2 const v = up2(mul2(mul2(mul2(pk2(p0.we48, p0.we48), f6),
                                         add2(f6, pk2(-0.5f, -0.5f))), i2));
          fnv[0] += dd[0] < p0.wcut ? v.x : 0.f;
          fnv[1] += dd[1] < p0.wcut ? v.y : 0.f;
        }
      } else {
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          PairF const p = ia[ta + typ[nb_index(e[u])]];
          float const inv_d = ii[u], inv_d2 = inv_d * inv_d;
          {
            float const inv_off = MODE == kPairOffset ? rcp_r(dd[u] - p.loff) : inv_d;
            float const s = p.lsig * inv_off, s2 = s * s, f6 = s2 * s2 * s2;
            bool const in = dd[u] < p.lcut && dd[u] > p.lmin;
            fnv[u] += in ? p.le48 * f6 * (f6 - 0.5f) * (inv_off * inv_d) : 0.f;
          }
          {
            float const s = p.wsig * inv_d, s2 = s * s, f6 = s2 * s2 * s2;
            fnv[u] += dd[u] < p.wcut ? p.we48 * f6 * (f6 - 0.5f) * inv_d2 : 0.f;
          }
        }
      }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      bool const on = r2[u] > 0.f;
      float ft = (on && r2[u] < rc2) ? fcv[u] : 0.f;
      if constexpr (decltype(lj)::value)
        ft += on ? fnv[u] : 0.f;
      sx += ft * dx[u];
      sy += ft * dy[u];
      sz += ft * dz[u];
    }
  };
  auto group = [&](auto lj, int v) {
    // the lane's group v: class A group v, or class B group v - ga
    int const grp = v < ga ? v : ngroups - 1 - (v - ga);
    const int4 *gp = reinterpret_cast<const int4 *>(nbp + (static_cast<long long>(grp) << 8));
    int4 const g0 = gp[0], g1 = gp[1];
    unsigned const ent[8] = {static_cast<unsigned>(g0.x), static_cast<unsigned>(g0.y),
                             static_cast<unsigned>(g0.z), static_cast<unsigned>(g0.w),
                             static_cast<unsigned>(g1.x), static_cast<unsigned>(g1.y),
                             static_cast<unsigned>(g1.z), static_cast<unsigned>(g1.w)};
    float sx = 0.f, sy = 0.f, sz = 0.f;
#pragma unroll
    for (int h = 0; h < 8; h += 4) {
      float4 pb[4]; // four gathers in flight
#pragma unroll
      for (int u = 0; u < 4; ++u)
        pb[u] = pos[nb_index(ent[h + u])];
      two(lj, ent + h, pb, sx, sy, sz);
      two(lj, ent + h + 2, pb + 2, sx, sy, sz);
    }
    // FP32 sums of this group into the FP64 accumulators
    fx += static_cast<double>(sx);
    fy += static_cast<double>(sy);
    fz += static_cast<double>(sz);
  };
  for (int v0 = 0; v0 < gmax; v0 += LPP) {
    int const v = v0 + sub;
    bool const any_a = __any_sync(0xffffffffu, v < ga);
    if (v < gt) {
      if (any_a)
        group(std::true_type{}, v);
      else
        group(std::false_type{}, v);
    }
  }
#pragma unroll
  for (int o = 1; o < LPP; o <<= 1) {
    fx += __shfl_xor_sync(0xffffffffu, fx, o);
    fy += __shfl_xor_sync(0xffffffffu, fy, o);
    fz += __shfl_xor_sync(0xffffffffu, fz, o);
  }
  if (active && sub == 0) {
    int const i = perm[a];
    if (overwrite) {
      f[3 * i + 0] = fx;
      f[3 * i + 1] = fy;
      f[3 * i + 2] = fz;
    } else {
      f[3 * i + 0] += fx;
      f[3 * i + 1] += fy;
      f[3 * i + 2] += fz;
    }
  }
}

// Block sums of N per-thread values (FP64, fixed order) into the columns of
// partials[blockIdx.x * width + ...]: value k goes to every column c with
// map(c) == k, times 1/2 (each pair is seen from both ends).
template <int N, typename Map>
__device__ inline void block_halves(double const *ev, int width, Map const &map,
                                    double *__restrict__ partials) {
  __shared__ double red[N][8];
  int const lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < N; ++k) {
    double v = ev[k];
    for (int o = 16; o > 0; o >>= 1)
      v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0)
      red[k][wid] = v;
  }
  __syncthreads();
  if (static_cast<int>(threadIdx.x) < width) {
    int const k = map(threadIdx.x);
    double s = 0.0;
    for (int w = 0; w < 8; ++w)
      s += red[k][w];
    partials[static_cast<long long>(blockIdx.x) * width + threadIdx.x] = 0.5 * s;
  }
}
// Columns {E_coul, E_nb, Vc[9], Vn[9]} (width 20) from {E_coul, E_nb, the six
// entries xx xy xz yy yz zz of Vc, of Vn}.
__device__ inline int ev_column(int c) {
  if (c < 2)
    return c;
  int const t = (c - 2) / 9, m = (c - 2) % 9, i = min(m / 3, m % 3), j = max(m / 3, m % 3);
  return 2 + 6 * t + (i == 0 ? j : i + j + 1);
}
// Energy / virial sums of one pair into ev[14] (factors fc, fn of the two
// forces, d the pair vector).
__device__ inline void ev_add(double *ev, double ec, double en, double fc, double fn, double d0,
                              double d1, double d2) {
  ev[0] += ec;
  ev[1] += en;
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    double const g = t ? fn : fc;
    double const x = g * d0, y = g * d1, z = g * d2;
    double *v = ev + 2 + 6 * t;
    v[0] += x * d0;
    v[1] += x * d1;
    v[2] += x * d2;
    v[3] += y * d1;
    v[4] += y * d2;
    v[5] += z * d2;
  }
}

// The FP32-mixed pair kernel with energies and virials in FP32 arithmetic
// (P3MX_MIXED_OBSERVABLES, the energies of the batch): one thread per particle,
// whole groups of entries with four gathers in flight, LJ / WCA for class A
// groups, sums in FP64.
__global__ void __launch_bounds__(256)
k_pair_forces_rel_ev(const RepGeom *__restrict__ reps, const int2 *__restrict__ blk,
                     const float4 *__restrict__ spf, const int *__restrict__ stype,
                     const int *__restrict__ perm, const PairIA *__restrict__ ia_g, int ntypes,
                     const int *__restrict__ nb, const int *__restrict__ nb_cnt,
                     double *__restrict__ f, int overwrite, double *__restrict__ partials) {
  pdl_enter();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  PairIA *ia = reinterpret_cast<PairIA *>(smem_raw);
  for (int k = threadIdx.x; k < ntypes * ntypes; k += blockDim.x)
    ia[k] = ia_g[k];
  int2 const bk = blk[blockIdx.x];
  RepGeom const &G = reps[bk.x];
  float const cs_x = static_cast<float>(G.box[0] / G.cg[0]);
  float const cs_y = static_cast<float>(G.box[1] / G.cg[1]);
  float const cs_z = static_cast<float>(G.box[2] / G.cg[2]);
  __syncthreads();
  long long const a = G.p0 + static_cast<long long>(bk.y) * blockDim.x + threadIdx.x;
  double ev[14];
#pragma unroll
  for (int k = 0; k < 14; ++k)
    ev[k] = 0.0;
  if (a < G.p0 + G.np) {
    int const c = nb_cnt[a];
    int const ga = (nb_count_a(c) + 7) >> 3, gt = ga + ((nb_count_b(c) + 7) >> 3);
    float4 const pa = spf[a];
    int const ta = stype[a] * ntypes;
    float const rc2 = static_cast<float>(G.r_cut * G.r_cut);
    float const two_a = static_cast<float>(2.0 * G.alpha / sqrt(kPi));
    float const pref_qa = static_cast<float>(G.prefactor) * pa.w;
    float const c_exp = static_cast<float>(-G.alpha * G.alpha * 1.4426950408889634);
    float const p_alpha = static_cast<float>(0.3275911 * G.alpha);
    double fx = 0.0, fy = 0.0, fz = 0.0;
    const int *nbp = nb + nb_base(G.nb_off, G.max_nb, a - G.p0);
    int const ngroups = G.max_nb >> 3;
    const float4 *pos = spf + G.p0;
    const int *typ = stype + G.p0;
    for (int v = 0; v < gt; ++v) {
      bool const cls_a = v < ga;
      int const grp = cls_a ? v : ngroups - 1 - (v - ga);
      const int4 *gp = reinterpret_cast<const int4 *>(nbp + (static_cast<long long>(grp) << 8));
#pragma unroll 1
      for (int h = 0; h < 2; ++h) {
        int4 const g = gp[h];
        unsigned const ent[4] = {static_cast<unsigned>(g.x), static_cast<unsigned>(g.y),
                                 static_cast<unsigned>(g.z), static_cast<unsigned>(g.w)};
        float4 pb[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          pb[u] = pos[nb_index(ent[u])];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          float const d0 = fmaf(code_axis(ent[u], 0), -cs_x, pa.x - pb[u].x);
          float const d1 = fmaf(code_axis(ent[u], 1), -0.25f * cs_y, pa.y - pb[u].y);
          float const d2 = fmaf(code_axis(ent[u], 2), -0.0625f * cs_z, pa.z - pb[u].z);
          float const r2 = d0 * d0 + d1 * d1 + d2 * d2;
          // zero distance (the list's filling): no term
          bool const on = r2 > 0.f, in_c = on && r2 < rc2;
          float const inv_d = rsqrt_approx(r2);
          float const dist = r2 * inv_d;
          float const ex = ex2_approx(c_exp * r2);
          float const t = rcp_r(fmaf(p_alpha, dist, 1.f));
          float const asp =
              t * (0.254829592f +
                   t * (-0.284496736f + t * (1.421413741f + t * (-1.453152027f + t * 1.061405429f))));
          float const er = asp * inv_d;
          float const pq = pref_qa * pb[u].w;
          float const fc = in_c ? (pq * ex) * (er + two_a) * (inv_d * inv_d) : 0.f;
          float const ec = in_c ? pq * er * ex : 0.f;
          float fn = 0.f, en = 0.f;
          if (cls_a && on) {
            PairR<float> const p(ia[ta + (ntypes == 1 ? 0 : typ[nb_index(ent[u])])]);
            if (p.active)
              lj_wca_sel(p, dist, inv_d, fn, en);
          }
          float const ft = fc + fn;
          fx += static_cast<double>(ft * d0);
          fy += static_cast<double>(ft * d1);
          fz += static_cast<double>(ft * d2);
          ev_add(ev, ec, en, fc, fn, d0, d1, d2);
        }
      }
    }
    int const i = perm[a];
    if (overwrite) {
      f[3 * i + 0] = fx;
      f[3 * i + 1] = fy;
      f[3 * i + 2] = fz;
    } else {
      f[3 * i + 0] += fx;
      f[3 * i + 1] += fy;
      f[3 * i + 2] += fz;
    }
  }
  block_halves<14>(ev, 20, [](int c) { return ev_column(c); }, partials);
}

// FP64 pair kernel: minimum-image differences of the folded positions, pair
// arithmetic and sums in FP64; the same lists, lanes and classes as
// k_pair_forces_rel (LJ / WCA for class A groups only).  EV adds energies and
// virials: per-block FP64 partials {E_coul, E_nb, Vc[9], Vn[9]} (width 20).
// Blocks map to replicas through the block table so partials never straddle
// replicas.  Bound by latency and the FP64 pipe: the inverse distance is one rsqrt
// (over squared distances of 0.05 to 30 its largest error is 0.51 ulp, that of 1 /
// sqrt 1.49), the A&S reciprocal rcp_newton; two pairs at a time, since
// a pair's chain (rsqrt, exp, polynomial) is long and two blocks per SM do not
// hide it (131 072 ions 234 -> 187 us).
template <bool EV, int LPP>
__global__ void __launch_bounds__(256, EV ? kPairBlocks64Ev : kPairBlocks64)
k_pair_forces(const RepGeom *__restrict__ reps, const int2 *__restrict__ blk,
              const double4 *__restrict__ spq, const int *__restrict__ stype,
              const int *__restrict__ perm, const PairIA *__restrict__ ia_g, int ntypes,
              const int *__restrict__ nb, const int *__restrict__ nb_cnt, double *__restrict__ f,
              int overwrite, double *__restrict__ partials) {
  pdl_enter();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  PairIA *ia = reinterpret_cast<PairIA *>(smem_raw);
  for (int k = threadIdx.x; k < ntypes * ntypes; k += blockDim.x)
    ia[k] = ia_g[k];
  __syncthreads();
  int2 const bk = blk[blockIdx.x / LPP];
  RepGeom const &G = reps[bk.x];
  int const sub = threadIdx.x % LPP;
  long long const la = static_cast<long long>(bk.y) * 256 + (blockIdx.x % LPP) * (256 / LPP) +
                       threadIdx.x / LPP;
  bool const active = la < G.np;
  long long const a = G.p0 + la;
  double ev[EV ? 14 : 1];
#pragma unroll
  for (int k = 0; k < (EV ? 14 : 1); ++k)
    ev[k] = 0.0;
  double fx = 0.0, fy = 0.0, fz = 0.0;
  if (active) {
    double4 const pa = spq[a];
    int const ta = stype[a] * ntypes;
    double const L0 = G.box[0], L1 = G.box[1], L2 = G.box[2];
    double const Li0 = G.box_i[0], Li1 = G.box_i[1], Li2 = G.box_i[2];
    double const alpha = G.alpha, r_cut = G.r_cut;
    double const two_a = 2.0 * G.alpha / sqrt(kPi);
    double const pref_qa = G.prefactor * pa.w;
    int const cw = nb_cnt[a];
    int const ga = (nb_count_a(cw) + 7) >> 3, gt = ga + ((nb_count_b(cw) + 7) >> 3);
    const int *nbp = nb + nb_base(G.nb_off, G.max_nb, la);
    int const ngroups = G.max_nb >> 3;
    const double4 *pos = spq + G.p0;
    const int *typ = stype + G.p0;
    for (int v = sub; v < gt; v += LPP) {
      bool const cls_a = v < ga;
      int const grp = cls_a ? v : ngroups - 1 - (v - ga);
      const int4 *gp = reinterpret_cast<const int4 *>(nbp + (static_cast<long long>(grp) << 8));
      // the next half group's positions are loaded ahead of the pairs
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        int4 const g = gp[h];
        unsigned const idx[4] = {nb_index(g.x), nb_index(g.y), nb_index(g.z), nb_index(g.w)};
        double4 pv[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          pv[u] = pos[idx[u]];
        // two pairs at a time, selected instead of branched around: their
        // dependent chains (rsqrt, exp, polynomial) overlap
#pragma unroll
        for (int w = 0; w < 4; w += 2) {
          double d0[2], d1[2], d2[2], dist2[2], inv[2], dist[2], fc[2], ec[2];
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            double4 const pb = pv[w + u];
            d0[u] = mi_d(pa.x - pb.x, L0, Li0);
            d1[u] = mi_d(pa.y - pb.y, L1, Li1);
            d2[u] = mi_d(pa.z - pb.z, L2, Li2);
            dist2[u] = d0[u] * d0[u] + d1[u] * d1[u] + d2[u] * d2[u];
          }
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            // zero distance (the list's filling): no term
            inv[u] = rsqrt(dist2[u] > 0.0 ? dist2[u] : 1.0);
            dist[u] = dist2[u] > 0.0 ? dist2[u] * inv[u] : 2.0 * r_cut;
            double const adist = alpha * dist[u];
            double const ex = exp(-adist * adist);
            double const t = rcp_newton(fma(0.3275911, adist, 1.0));
            double const asp =
                t * (0.254829592 +
                     t * (-0.284496736 +
                          t * (1.421413741 + t * (-1.453152027 + t * 1.061405429))));
            double const er = asp * inv[u];
            double const pq = pref_qa * pv[w + u].w;
            bool const in = dist[u] < r_cut;
            fc[u] = in ? pq * (ex * (er + two_a) * (inv[u] * inv[u])) : 0.0;
            if constexpr (EV)
              ec[u] = in ? pq * er * ex : 0.0;
          }
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            double fn = 0.0, en = 0.0;
            if (cls_a && dist2[u] > 0.0) {
              PairR<double> const p(ia[ta + typ[idx[w + u]]]);
              if (p.active)
                lj_wca(p, dist[u], inv[u], fn, en);
            }
            double const ft = fc[u] + fn;
            fx += ft * d0[u];
            fy += ft * d1[u];
            fz += ft * d2[u];
            if constexpr (EV)
              ev_add(ev, ec[u], en, fc[u], fn, d0[u], d1[u], d2[u]);
          }
        }
      }
    }
  }
#pragma unroll
  for (int o = 1; o < LPP; o <<= 1) {
    fx += __shfl_xor_sync(0xffffffffu, fx, o);
    fy += __shfl_xor_sync(0xffffffffu, fy, o);
    fz += __shfl_xor_sync(0xffffffffu, fz, o);
  }
  if (active && sub == 0) {
    int const i = perm[a];
    if (overwrite) {
      f[3 * i + 0] = fx;
      f[3 * i + 1] = fy;
      f[3 * i + 2] = fz;
    } else {
      f[3 * i + 0] += fx;
      f[3 * i + 1] += fy;
      f[3 * i + 2] += fz;
    }
  }
  if constexpr (EV)
    block_halves<14>(ev, 20, [](int c) { return ev_column(c); }, partials);
}

// Largest squared displacement since the last list build, as a flag:
// set when any particle moved more than skin/2 (check_resort_required,
// CellStructure.hpp:393-401).
// A particle whose type differs from its type at the last build, or that
// became charged or neutral, also triggers the rebuild: the lists hold
// per-type-pair cutoffs, the sorted types and the Coulomb pairs of charged
// particles (as the reference resorts on a particle change).
__device__ inline int list_kind(int type, double q) { return 2 * type + (q != 0.0 ? 1 : 0); }
__global__ void k_displacement_check(const RepGeom *__restrict__ reps, const int *__restrict__ rep_of,
                                     const double *__restrict__ pos, const double *__restrict__ pos_ref,
                                     const int *__restrict__ type, const double *__restrict__ q,
                                     const int *__restrict__ type_ref, long long n,
                                     int *__restrict__ flag, int *__restrict__ rflag) {
  long long const i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n)
    return;
  int const r = rep_of[i];
  RepGeom const &G = reps[r];
  double d2 = 0.0;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    double const dx = pos[3 * i + d] - pos_ref[3 * i + d];
    d2 += dx * dx;
  }
  double const lim = 0.5 * G.skin;
  if (d2 > lim * lim || list_kind(type[i], q[i]) != type_ref[i]) {
    atomicOr(flag, 1);
    if (rflag) // per-replica decision: only this replica rebuilds
      atomicOr(&rflag[r], 1);
  }
}

// Reference positions and kinds (list_kind) of the replicas that rebuilt
// (all when rflag is null).
__global__ void k_copy_pos_ref(double *__restrict__ pos_ref, const double *__restrict__ pos,
                               int *__restrict__ type_ref, const int *__restrict__ type,
                               const double *__restrict__ q, const int *__restrict__ rep_of, const int *__restrict__ rflag,
                               long long n, const int *__restrict__ cond) {
  if (cond && !*cond)
    return;
  long long const i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n || (rflag && !rflag[rep_of[i]]))
    return;
#pragma unroll
  for (int d = 0; d < 3; ++d)
    pos_ref[3 * i + d] = pos[3 * i + d];
  type_ref[i] = list_kind(type[i], q[i]);
}

} // namespace p3mx
