// Sums over all pairs and slices of the path: ShortRangeClass::d_dBeta
// (ShortRangeClass.cc:316-355) and, in the same pass, ShortRangePotClass::V
// (ShortRangePotClass.cc:28-47), for the energy estimator.
//
// Design.  A unit of work is one pair walked along consecutive links of the
// path.  Slice s + 1 of one link is slice s of the next, so a walk forms each
// slice's minimum-image displacement, its length and its one-slice table
// values once and hands them on; only what depends on both slices (off-diagonal
// terms, the tricubic spline, the Coulomb 1/q) is left per link.  DistDisp's
// second displacement takes the image that follows the first; it is the
// slice's own minimum image whenever the two are less than half a box apart
// in every dimension, which one comparison of s^2 establishes; otherwise the
// walk forms it as the reference does.
// Blocks take (tile of particles) x (tile of particles) x (chunk of links).
// For a 1-D table that ends well inside the box, and enough pairs (see
// launch_pair_path), a block first lists the pairs of its tiles whose bounding
// spheres over the chunk come within the table's range; all others contribute
// the table's end value on every link.
// Sums are taken in a fixed order, so results are bitwise reproducible.
//
// Measured as pimc_energy, against one thread per (pair, link) that decoded its
// indices with 64-bit divisions and evaluated both ends of every link, and a
// second such pass for V: N = 4096, M = 256, range 0.11 of the box 73.7 -> 0.52
// ms; N = 512, M = 128, tricubic 1042 -> 625 us; N = 128, M = 64, Coulomb
// (both passes) 34 -> 22 us.  FP64 operations and their latencies bound it.
#include <cuda_runtime.h>

#include <algorithm>

#include "action_kernels.cuh"
#include "device_math.cuh"

namespace pimc {

namespace {

constexpr int kMaxTile = 64;
// With lists a block takes one i tile against up to kGroup j tiles: their pairs
// gather in one list, so the walks fill the block although few of a tile's pairs
// survive (the energy of N = 4096, M = 256, a range of 0.11 box sides: 560 us
// with a list a tile pair, 513 in groups).
constexpr int kGroup = 8;
constexpr int kListMax = kMaxTile * kMaxTile + 1024;  // walked when past 1024: the next tile fits
// Threads a block.  Tricubic, 128 against 256 threads (pimc_energy, us): M = 128, N = 16
// 30.5 / 28, 37 36.5 / 38, 64 46.6 / 46.2, 128 75.7 / 77, 192 140 / 134, 256 196 / 202, 384 440 / 399,
// 512 660 / 638; M = 32, N = 64 32.8 / 35, 256 75.9 / 76, 512 191 / 193: neither is the better one
// throughout, and no size tells them apart before 384.
template <int KIND>
constexpr int kThreadsOf = KIND == PA_TRICUBIC ? 128 : 256;

struct PairPathArgs {
  const double *path;
  DevSystem sys;
  DevPA pa;
  int slice1, skip, nlinks, level;
  int tile_log2, chunk;      // particles per tile (log2), links per chunk
  long long ntp, items;      // tile pairs (with lists: tile x group pairs); those x chunks
  const float4 *bounds;      // [chunk][N] {centre, radius} or null (every pair is taken)
  double near2;              // (0.49 smallest box side)^2
};

// Values of one pair at one slice: f enters the link terms of d_dBeta
// (DavidPA: V + dU_00; tricubic: V; Coulomb: dUlong of the level), v is V of
// the potential estimator.
struct SliceVal {
  double f, v;
};

// (y, y'', dU, dU'') rows of the estimator table: two 32-byte loads a point pair.
__device__ __forceinline__ void est_row(const double *p, double r[4]) {
  asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(r[0]), "=d"(r[1]), "=d"(r[2]), "=d"(r[3]) : "l"(p));
}

template <bool DO_V>
__device__ __forceinline__ SliceVal david_slice(const DDavid<double> &d, const double *est, const double *est0,
                                                double r) {
  const SplineCell<double> c = spline_cell(d.grid, r);
  double lo[4], hi[4];
  est_row(est + (size_t)c.low * 4, lo);
  est_row(est + (size_t)c.hi * 4, hi);
  SliceVal s;
  s.v = spline_apply(c, lo[0], hi[0], lo[1], hi[1]);
  s.f = spline_apply(c, lo[2], hi[2], lo[3], hi[3]) + s.v;
  if (DO_V && est0 != est) {  // DavidPAClass::V reads the first tau's table
    est_row(est0 + (size_t)c.low * 4, lo);
    est_row(est0 + (size_t)c.hi * 4, hi);
    s.v = spline_apply(c, lo[0], hi[0], lo[1], hi[1]);
  }
  return s;
}

// What a thread keeps of the tables for the whole launch.
template <int KIND>
struct Tables {
  const double *est, *est0;  // DavidPA: rows of this level and of tau table 0
  SliceVal end;              // DavidPA: the values at and beyond the grid's end
  const double *F;           // tricubic: dU nodes of this level
  const double *dul;         // Coulomb: dUlong of this level
};

template <int KIND, bool DO_V>
__device__ __forceinline__ SliceVal slice_value(const DevPA &pa, const Tables<KIND> &t, double r) {
  if (KIND == PA_DAVID) {
    const DDavid<double> &d = pa.d64;
    // a length that overflowed is not "beyond the table": the spline makes it NaN, which is reported
    if (r >= d.grid.end && __double2hiint(r) != 0x7ff00000) return t.end;
    return david_slice<DO_V>(d, t.est, t.est0, r < d.grid.start ? d.grid.start : r);
  }
  SliceVal s;
  if (KIND == PA_TRICUBIC) {
    s.f = s.v = pot_V_pairs(pa.t64.pot_grid, reinterpret_cast<const double2 *>(pa.t64.pot_pairs), r);
    return s;
  }
  const DCoulomb<double> &c = pa.c64;
  s.f = c.long_range ? quintic_at(c, t.dul, r) : 0.0;
  s.v = 0.0;
  if (DO_V) s.v = c.z1z2 / r - (t.dul == c.dulong ? s.f : c.long_range ? quintic_at(c, c.dulong, r) : 0.0);
  return s;
}

// Displacement b - a in the minimum image (PathClass::DistDisp): raw and boxed.
__device__ __forceinline__ void displacement(const double *a, const double *b, const DevSystem &s, double raw[3],
                                             double d[3]) {
#pragma unroll
  for (int i = 0; i < 3; i++) {
    raw[i] = __ldg(b + i) - __ldg(a + i);
    const double n = -round_even_magic(rmul(raw[i], s.boxinv[i]));
    d[i] = radd(raw[i], rmul(n, s.box[i]));
  }
}

// One in-fit tricubic term listed for the warp's lane teams: its in-cell
// coordinates and its cell.  (With the Hermite bases in the list, 112 bytes a
// term, the team's lanes save work but the L1 left for the node table misses:
// no gain; a third more blocks an SM: 842 us against 648.)
struct __align__(16) PathTerm {
  double u[3];
  int cell;
};

// One lane's part of a listed term: components 4 (pt & 1) .. + 3 of node
// iz + (pt >> 1) of the cell's four (x, y) node pairs (as tricubic_team_part,
// with the sums over y taken first).
__device__ __forceinline__ double team_part(const double *F, const DTricubic<double> &t, const PathTerm &P, int pt) {
  const size_t sy = (size_t)t.nt * 8, sx = (size_t)t.ny * sy;
  const int nz = pt >> 1, hi = pt & 1;
  const double *p = F + (size_t)P.cell * 8 + nz * 8 + hi * 4;
  double v[4][4];
#pragma unroll
  for (int k = 0; k < 4; k++) ld4_nc(p + (k >> 1) * sx + (k & 1) * sy, v[k]);
  double a[4], b[4], c[4];
  hermite4(P.u[0], t.qg.delta, a);
  hermite4(P.u[1], t.yg.delta, b);
  hermite4(P.u[2], t.tg.delta, c);
  // (F, Fx, Fy, Fz) weigh (A0 B0 Cv, A1 B0 Cv, A0 B1 Cv, A0 B0 Cd), (Fxy, Fxz,
  // Fyz, Fxyz) weigh (A1 B1 Cv, A1 B0 Cd, A0 B1 Cd, A1 B1 Cd)
  const double Cv = nz ? c[1] : c[0], Cd = nz ? c[3] : c[2], Ce = hi ? Cd : Cv;
  double s = 0.0, e = 0.0;
#pragma unroll
  for (int dx = 0; dx < 2; dx++) {
    double x = 0.0, y = 0.0, z = 0.0;
#pragma unroll
    for (int dy = 0; dy < 2; dy++) {
      const double *w = v[2 * dx + dy];
      x += (hi ? b[2 + dy] : b[dy]) * (Cv * w[0] + Cd * w[3]);
      y += b[dy] * w[1];
      z += b[2 + dy] * w[2];
    }
    s += (hi ? a[2 + dx] : a[dx]) * x;
    e += a[2 + dx] * y + a[dx] * z;
  }
  return s + Ce * e;
}

// KIND's d_dBeta over links and, with DO_V, V over slices 0 .. nlinks (weight
// 1/2 at both ends; slice1 = 0 and skip = 1 then).  out[0] = d_dBeta, out[1] = V.
template <int KIND, bool DO_V>
__global__ void __launch_bounds__(kThreadsOf<KIND>, KIND == PA_TRICUBIC ? 4 : 3)
    pair_path_kernel(const __grid_constant__ PairPathArgs a, double2 *partials, unsigned int *counter, double *out) {
  constexpr int kThreads = kThreadsOf<KIND>, kWarps = kThreads / 32;
  constexpr int kStep = KIND == PA_TRICUBIC ? 4 : 1;  // links between two gathers: their terms fill the teams' rounds
  __shared__ float4 s_bi[kMaxTile], s_bj[kMaxTile];
  __shared__ unsigned short s_list[kListMax];  // i << 9 | j in the group
  __shared__ int s_cnt[kWarps + 1];
  __shared__ PathTerm s_terms[KIND == PA_TRICUBIC ? kWarps * 32 * kStep : 1];
  PathTerm *const E = s_terms + (KIND == PA_TRICUBIC ? (threadIdx.x >> 5) * 32 * kStep : 0);
  __shared__ double sh[2][kWarps];
  __shared__ int s_last;
  const DevSystem &sys = a.sys;
  const int N = sys.N, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int T = 1 << a.tile_log2;
  Tables<KIND> tb;
  if (KIND == PA_DAVID) {
    const DDavid<double> &d = a.pa.d64;
    tb.est0 = d.est;
    tb.est = d.est + (size_t)(a.level + d.tau_pos) * d.grid.n * 4;
    tb.end = david_slice<DO_V>(d, tb.est, tb.est0, d.grid.end);
  } else if (KIND == PA_TRICUBIC) {
    const DTricubic<double> &t = a.pa.t64;
    tb.F = t.dU + (size_t)a.level * t.nq * t.ny * t.nt * 8;
  } else {
    tb.dul = a.pa.c64.dulong + (size_t)a.level * a.pa.c64.np * 6;
  }
  double du = 0.0, vs = 0.0;
  for (long long item = blockIdx.x; item < a.items; item += gridDim.x) {
    const int c = (int)(item / a.ntp);
    const bool lists = KIND == PA_DAVID && a.bounds;
    int ti, tj, tj1;  // j tiles [tj, tj1)
    if (lists) {
      // groups of tile row ti: 0 .. ti / kGroup; rows [kGroup b, kGroup (b + 1)) have b + 1 each
      const long long k = item - c * a.ntp;
      int b, r;
      tri_decode(k / kGroup, b, r);
      const int rem = (int)(k - (long long)kGroup * b * (b + 1) / 2);
      ti = kGroup * b + rem / (b + 1);
      tj = kGroup * (rem % (b + 1));
      tj1 = min(tj + kGroup, ti + 1);
      if (ti << a.tile_log2 >= N) continue;  // the last row block's empty rows
    } else {
      tri_decode(item - c * a.ntp, ti, tj);
      tj1 = tj + 1;
    }
    const int i0 = ti << a.tile_log2, j0 = tj << a.tile_log2;
    const int ni = min(T, N - i0);
    const int lbeg = c * a.chunk, lend = min(a.nlinks, lbeg + a.chunk);
    int n = T << a.tile_log2;  // units' pairs: all (i, j) of the tiles, or the list
    if (lists) n = 0;
    for (int tc = tj; tc < tj1; tc++) {
      const int jc = tc << a.tile_log2, nj = min(T, N - jc);
      if (KIND == PA_DAVID && a.bounds) {
        const float4 *bc = a.bounds + (size_t)c * N;
        __syncthreads();  // the previous readers are done
        if (tc == tj && tid < ni) s_bi[tid] = bc[i0 + tid];
        if (tid >= kMaxTile && tid - kMaxTile < nj) s_bj[tid - kMaxTile] = bc[jc + tid - kMaxTile];
        __syncthreads();
        // Warp w tests rows w, w + 8, ...: two lanes' worth of columns each; the
        // ballots stay in registers until the warps' counts give the places.
        const float Lx = (float)sys.box[0], Ly = (float)sys.box[1], Lz = (float)sys.box[2];
        const float ix = (float)sys.boxinv[0], iy = (float)sys.boxinv[1], iz = (float)sys.boxinv[2];
        // FP32 slack: centres, box sides and the image arithmetic round at 2^-24 of a box side each
        const float lim0 = (float)a.pa.d64.grid.end * 1.000001f + 4e-6f * fmaxf(Lx, fmaxf(Ly, Lz));
        unsigned m[kMaxTile / kWarps][2];
        int cnt = 0;
#pragma unroll
        for (int k = 0; k < kMaxTile / kWarps; k++) {
          const int i = warp + k * kWarps;
          const float4 p = s_bi[i];
#pragma unroll
          for (int h = 0; h < 2; h++) {
            const int j = lane + 32 * h;
            const float4 q = s_bj[j];
            float dx = q.x - p.x, dy = q.y - p.y, dz = q.z - p.z;
            dx -= round_even_magic(dx * ix) * Lx;
            dy -= round_even_magic(dy * iy) * Ly;
            dz -= round_even_magic(dz * iz) * Lz;
            const float lim = lim0 + p.w + q.w;
            const bool take = i < ni && j < (ti == tc ? min(i, nj) : nj) &&
                              !(dx * dx + dy * dy + dz * dz > lim * lim);  // a NaN is taken: the sum reports it
            m[k][h] = __ballot_sync(0xffffffffu, take);
            cnt += __popc(m[k][h]);
          }
        }
        if (lane == 0) s_cnt[warp] = cnt;
        __syncthreads();
        int at = n, found = 0;
        for (int w = 0; w < kWarps; w++) {
          if (w == warp) at += found;
          found += s_cnt[w];
        }
        const unsigned below = (1u << lane) - 1u;
        const int jg = (tc - tj) << a.tile_log2;
#pragma unroll
        for (int k = 0; k < kMaxTile / kWarps; k++)
#pragma unroll
          for (int h = 0; h < 2; h++) {
            if (m[k][h] >> lane & 1u)
              s_list[at + __popc(m[k][h] & below)] =
                  (unsigned short)((warp + k * kWarps) << 9 | (jg + lane + 32 * h));
            at += __popc(m[k][h]);
          }
        n += found;
        if (tid == 0) {  // the pairs left out: the end value on every link
          const int out_of_range = (ti == tc ? ni * (ni - 1) / 2 : ni * nj) - found;
          du += (double)out_of_range * (double)(lend - lbeg) * tb.end.f;
          if (DO_V) {
            double w = (double)(lend - lbeg);
            if (lbeg == 0) w -= 0.5;
            if (lend == a.nlinks) w += 0.5;
            vs += (double)out_of_range * w * tb.end.v;
          }
        }
        if (n <= kListMax - kMaxTile * kMaxTile && tc + 1 < tj1) continue;  // room for the next tile
        __syncthreads();
      }
      if (n == 0) continue;
      // Few pairs: their walks are cut so that about two units come to a thread
      int nsub = 1;
      const int links = lend - lbeg;
      if (KIND == PA_DAVID && a.bounds)
        while (n * nsub < 2 * kThreads && 4 * nsub < links) nsub *= 2;
      const int len = (links + nsub - 1) / nsub;
      const int units = n * nsub;
      for (int u0 = 0; u0 < units; u0 += kThreads) {
        const int u = u0 + tid;
        const int sub = u / n, e = u - sub * n;
        int i, j;
        bool live = u < units;
        if (KIND == PA_DAVID && a.bounds) {
          const int code = live ? s_list[e] : 0;
          i = code >> 9;
          j = code & 511;
        } else {
          i = e >> a.tile_log2;
          j = e & (T - 1);
          live = live && i < ni && j < nj && (ti != tj || j < i);
        }
        const int l0 = lbeg + sub * len, l1 = min(lend, l0 + len);
        live = live && l0 < l1;
        if (KIND != PA_TRICUBIC && !live) continue;  // the tricubic teams need whole warps
        const size_t row = (size_t)a.skip * N * 3;
        const double *pi = a.path + ((size_t)(a.slice1 + (live ? l0 : lbeg) * a.skip) * N + i0 + (live ? i : 0)) * 3;
        const double *pj = a.path + ((size_t)(a.slice1 + (live ? l0 : lbeg) * a.skip) * N + j0 + (live ? j : 0)) * 3;
        // ShortRangeClass.cc:333-336 / DistDisp(slice, slice + skip, p1, p2): p1 = i, p2 = j
        double raw[3], dA[3], dB[3];
        displacement(pi, pj, sys, raw, dA);
        double ra = sqrt(dA[0] * dA[0] + dA[1] * dA[1] + dA[2] * dA[2]);
        SliceVal va = {0.0, 0.0}, vb = {0.0, 0.0};
        if (live && (KIND != PA_TRICUBIC || DO_V)) va = slice_value<KIND, DO_V>(a.pa, tb, ra);
        for (int l = l0; l < l0 + len; l += kStep) {
          int listed = 0;
#pragma unroll 1
          for (int k = 0; k < kStep; k++) {
            bool in = false;
            PathTerm tt;
            if (live && l + k < l1) {
              pi += row;
              pj += row;
              displacement(pi, pj, sys, raw, dB);
              double rb = sqrt(dB[0] * dB[0] + dB[1] * dB[1] + dB[2] * dB[2]);
              if (KIND != PA_TRICUBIC || DO_V) vb = slice_value<KIND, DO_V>(a.pa, tb, rb);
              const double e0 = dA[0] - dB[0], e1 = dA[1] - dB[1], e2 = dA[2] - dB[2];
              double s2 = e0 * e0 + e1 * e1 + e2 * e2;
              double rl = rb, fl = vb.f;  // the link's second length and value
              if (!(s2 < a.near2)) {      // the image at the second slice that follows the first (PathClass.h:720-735)
                double dl[3];
#pragma unroll
                for (int x = 0; x < 3; x++)
                  dl[x] = radd(raw[x], rmul(rint(rmul(rsub(dA[x], raw[x]), sys.boxinv[x])), sys.box[x]));
                const double g0 = dA[0] - dl[0], g1 = dA[1] - dl[1], g2 = dA[2] - dl[2];
                s2 = g0 * g0 + g1 * g1 + g2 * g2;
                rl = sqrt(dl[0] * dl[0] + dl[1] * dl[1] + dl[2] * dl[2]);
                if (KIND != PA_TRICUBIC || DO_V) fl = slice_value<KIND, false>(a.pa, tb, rl).f;
              }
              if (KIND == PA_DAVID) {
                du += 0.5 * (va.f + fl);
                const DDavid<double> &d = a.pa.d64;
                if (d.num_terms > 0) {
                  const double q = 0.5 * (ra + rl);
                  if (s2 > 0.0 && q < d.grid.end) {
                    const size_t o = (size_t)(a.level + d.tau_pos) * d.grid.n * d.ncols;
                    du += david_offdiag_add<double>(d.grid, d.duy + o, d.dud2 + o, d.ncols, d.num_terms, 0.0, s2, q,
                                                    ra - rl);
                  }
                }
              } else if (KIND == PA_COULOMB) {
                du += a.pa.c64.z1z2 / (0.5 * (ra + rl)) - 0.5 * (va.f + fl);
              } else {
                const TriPrep<double> pr = tricubic_prep<double>(a.pa.t64, 0.5 * (ra + rl), ra - rl, s2);
                in = pr.inside;
                if (pr.inside) {
                  for (int x = 0; x < 3; x++) tt.u[x] = pr.u[x];
                  tt.cell = pr.cell;
                } else if (DO_V) {
                  du += 0.5 * (va.f + fl);
                } else {
                  du += 0.5 * (slice_value<KIND, false>(a.pa, tb, ra).f + slice_value<KIND, false>(a.pa, tb, rl).f);
                }
              }
              if (DO_V) vs += (l + k == 0 ? 0.5 : 1.0) * va.v;
#pragma unroll
              for (int x = 0; x < 3; x++) dA[x] = dB[x];
              ra = rb;
              va = vb;
            }
            if (KIND == PA_TRICUBIC) {
              const unsigned m = __ballot_sync(0xffffffffu, in);
              if (in) E[listed + __popc(m & ((1u << lane) - 1u))] = tt;
              listed += __popc(m);
            }
          }
          if (KIND == PA_TRICUBIC) {
            // The in-fit terms of the warp's step, gathered by teams of four
            // lanes: a cell's node pair is one 128-byte line a team, against a line
            // a lane.
            __syncwarp();
            for (int x = lane >> 2; x < listed; x += 8) du += team_part(tb.F, a.pa.t64, E[x], lane & 3);
            __syncwarp();
          }
        }
        if (DO_V && live && l1 == a.nlinks) vs += 0.5 * va.v;
      }
      if (lists) n = 0;  // walked
    }
  }
  // this block's sums, then the last block adds every block's in block order
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    du += __shfl_xor_sync(0xffffffffu, du, o);
    if (DO_V) vs += __shfl_xor_sync(0xffffffffu, vs, o);
  }
  if (lane == 0) {
    sh[0][warp] = du;
    sh[1][warp] = vs;
  }
  __syncthreads();
  if (tid == 0) {
    double x = 0.0, y = 0.0;
    for (int w = 0; w < kWarps; w++) {
      x += sh[0][w];
      y += sh[1][w];
    }
    partials[blockIdx.x] = make_double2(x, y);
    __threadfence();
    s_last = atomicAdd(counter, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  du = vs = 0.0;
  for (int i = tid; i < (int)gridDim.x; i += kThreads) {
    const double2 p = __ldcg(&partials[i]);
    du += p.x;
    vs += p.y;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    du += __shfl_xor_sync(0xffffffffu, du, o);
    vs += __shfl_xor_sync(0xffffffffu, vs, o);
  }
  __syncthreads();
  if (lane == 0) {
    sh[0][warp] = du;
    sh[1][warp] = vs;
  }
  __syncthreads();
  if (tid == 0) {
    double x = 0.0, y = 0.0;
    for (int w = 0; w < kWarps; w++) {
      x += sh[0][w];
      y += sh[1][w];
    }
    out[0] = x;
    if (DO_V) out[1] = y;
    *counter = 0u;
  }
}

// Bounding sphere of every particle over every chunk's slices: centre = its
// position at the chunk's middle slice (boxed), radius = the largest
// minimum-image distance from it, rounded up.
__global__ void __launch_bounds__(128) path_bounds_kernel(const double *__restrict__ path, DevSystem sys, int slice1,
                                                          int skip, int nlinks, int chunk, float4 *bounds) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x, c = blockIdx.y;
  if (p >= sys.N) return;
  const int beg = c * chunk, end = min(nlinks, beg + chunk), mid = (beg + end) >> 1;
  const double *q = path + ((size_t)(slice1 + mid * skip) * sys.N + p) * 3;
  double ctr[3] = {q[0], q[1], q[2]};
  put_in_box(ctr, sys);
  double r2 = 0.0, far = 0.0;  // far: the largest coordinate, whose rounding the boxed distances carry
  const double *x = path + ((size_t)(slice1 + beg * skip) * sys.N + p) * 3;
#pragma unroll 4
  for (int l = beg; l <= end; l++, x += (size_t)skip * sys.N * 3) {
    double d2 = 0.0;
#pragma unroll
    for (int i = 0; i < 3; i++) {
      double d = x[i] - ctr[i];
      far = fmax(far, fabs(x[i]));
      d -= round_even_magic(d * sys.boxinv[i]) * sys.box[i];
      d2 += d * d;
    }
    r2 = d2 > r2 || d2 != d2 ? d2 : r2;  // a NaN stays: its pairs are taken
  }
  bounds[(size_t)c * sys.N + p] = make_float4((float)ctr[0], (float)ctr[1], (float)ctr[2],
                                              (float)sqrt(r2) * 1.000001f + (float)(far * 1e-15));
}

}  // namespace

size_t pair_path_bounds_bytes(int N, int S) {
  return (size_t)((S - 1 + kBoundsChunk - 1) / kBoundsChunk) * N * sizeof(float4);
}

cudaError_t launch_pair_path(const ReduceTarget &t, const double *path, const DevSystem &sys, const DevPA &pa,
                             int slice1, int skip, int nlinks, int level, bool do_v, float4 *bounds, int sm_count) {
  PairPathArgs a;
  a.path = path;
  a.sys = sys;
  a.pa = pa;
  a.slice1 = slice1;
  a.skip = skip;
  a.nlinks = nlinks;
  a.level = level;
  const double side = std::min(sys.box[0], std::min(sys.box[1], sys.box[2]));
  a.near2 = 0.49 * side * 0.49 * side;
  // Lists take long chunks and few items, so they cost a latency of their own and
  // pay from a number of (pair, link)s on, the sooner the shorter the range: the
  // times cross at about 5e7 range / side.  pimc_energy with / without, us, at 0.1,
  // 0.2 and 0.3 sides:
  //   N = 256, M = 16 (5e5):    68 / 40    95 / 42   123 / 40
  //   N = 400, M = 64 (5e6):    87 / 84   130 / 100  190 / 108
  //   N = 512, M = 64 (8e6):    93 / 109  147 / 127  200 / 136
  //   N = 2048, M = 4 (8e6):    94 / 122  110 / 126  134 / 134
  //   N = 512, M = 128 (17e6):  91 / 174  138 / 203  200 / 222
  //   N = 4096, M = 2 (17e6):  104 / 225  135 / 244  187 / 261
  //   N = 800, M = 64 (20e6):  104 / 235  164 / 278  250 / 309
  //   N = 1200, M = 128 (92e6): 173 / 706  280 / 801  438 / 890
  // (Beyond 0.3 sides they would gain 10-30 % from 3e7 on.  Below 256 particles, at
  // 0.15 / 0.3 sides: N = 192, M = 256 74 / 128 with, 93 / 107 without; N = 128
  // 75 / 133 and 60 / 64.)
  const double end = pa.d64.grid.end, pair_links = 0.5 * sys.N * (sys.N - 1.0) * nlinks;
  const bool cull = pa.kind == PA_DAVID && sys.N >= 256 && end <= 0.3 * side && pair_links * side >= 5e7 * end;
  a.bounds = cull ? bounds : nullptr;
  a.chunk = cull ? kBoundsChunk : 8;
  a.tile_log2 = 6;
  auto count = [&]() {
    const long long nt = (sys.N + (1 << a.tile_log2) - 1) >> a.tile_log2, nb = (nt + kGroup - 1) / kGroup;
    a.ntp = cull ? kGroup * nb * (nb + 1) / 2 : nt * (nt + 1) / 2;
    return a.ntp * ((nlinks + a.chunk - 1) / a.chunk);
  };
  while (count() < 4 * sm_count && a.tile_log2 > 4) a.tile_log2--;
  while (!cull && count() < 2 * sm_count && a.chunk > 1) a.chunk >>= 1;
  a.items = count();
  const int blocks = (int)std::min(a.items, (long long)std::min(kPartialSlots / 2, 16 * sm_count));
  if (cull) {
    const dim3 grid((sys.N + 127) / 128, (nlinks + a.chunk - 1) / a.chunk);
    path_bounds_kernel<<<grid, 128, 0, t.stream>>>(path, sys, slice1, skip, nlinks, a.chunk, bounds);
  }
  double2 *partials = reinterpret_cast<double2 *>(t.partials);
#define PIMC_PAIR_PATH(KIND)                                                                                        \
  do {                                                                                                              \
    if (do_v)                                                                                                       \
      pair_path_kernel<KIND, true><<<blocks, kThreadsOf<KIND>, 0, t.stream>>>(a, partials, t.counter, t.out);              \
    else                                                                                                            \
      pair_path_kernel<KIND, false><<<blocks, kThreadsOf<KIND>, 0, t.stream>>>(a, partials, t.counter, t.out);             \
  } while (0)
  if (pa.kind == PA_DAVID)
    PIMC_PAIR_PATH(PA_DAVID);
  else if (pa.kind == PA_COULOMB)
    PIMC_PAIR_PATH(PA_COULOMB);
  else
    PIMC_PAIR_PATH(PA_TRICUBIC);
#undef PIMC_PAIR_PATH
  return cudaGetLastError();
}

}  // namespace pimc
