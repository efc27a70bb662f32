// Action-level kernels behind the ActionBaseClass drop-in entry points:
// SingleAction and d_dBeta of ShortRangeClass and KineticClass, and the
// PathClass accept/reject copies.  One launch per call; each reduces its
// terms in a fixed order (warp shuffle tree, block tree, then the last block
// over the per-block partials), so results are bitwise reproducible.
#include <cuda_runtime.h>

#include <algorithm>

#include "action_kernels.cuh"
#include "device_math.cuh"
#include "gofr_shape.h"

namespace pimc {

// Threads per block of the reductions.  Most calls are one window of one
// particle: a few hundred to a few thousand terms, each a serial chain of FP64
// operations and dependent loads, so small blocks spread the terms over SMs.
constexpr int kReduceThreads = 128;

// Block-wide sum; the result is valid in thread 0.  `sh` holds a double per warp.
__device__ __forceinline__ double block_sum(double v, double *sh) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) sh[w] = v;
  __syncthreads();
  double r = 0.0;
  if (threadIdx.x == 0)
#pragma unroll
    for (int i = 0; i < kReduceThreads / 32; i++) r += sh[i];
  return r;
}

// Writes this block's partial and lets the last block to finish add all
// partials in block order into *out.  A single block writes its sum itself.
__device__ __forceinline__ void finish_sum(double partial, double *partials, unsigned int *counter, double *out,
                                           double *sh) {
  __shared__ int s_last;
  if (gridDim.x == 1) {
    if (threadIdx.x == 0) *out = partial;
    return;
  }
  if (threadIdx.x == 0) {
    partials[blockIdx.x] = partial;
    __threadfence();
    unsigned int t = atomicAdd(counter, 1u);
    s_last = (t == gridDim.x - 1);
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  double v = 0.0;
  for (int i = threadIdx.x; i < (int)gridDim.x; i += blockDim.x) v += __ldcg(&partials[i]);
  double total = block_sum(v, sh);
  if (threadIdx.x == 0) {
    *out = total;
    *counter = 0u;
  }
}

__device__ __forceinline__ void load3(const double *__restrict__ p, double v[3]) {
  v[0] = __ldg(p);
  v[1] = __ldg(p + 1);
  v[2] = __ldg(p + 2);
}

// ShortRangeClass::SingleAction (ShortRangeClass.cc:191-236).  Item order:
// active particle, link, partner (partner fastest, for coalesced path reads).
template <int KIND, typename R>
__global__ void __launch_bounds__(kReduceThreads) sr_single_kernel(const double *__restrict__ path, DevSystem sys, DevPA pa,
                                                        ActiveList act, int slice1, int skip, int nlinks, int level,
                                                        double *partials, unsigned int *counter, double *out) {
  __shared__ double sh[kReduceThreads / 32];
  typedef typename Pair2<R>::T P2;
  const P2 *diag = nullptr;
  if (KIND == PA_DAVID) {
    const DDavid<R> &d = david_of<R>(pa);
    diag = reinterpret_cast<const P2 *>(d.diag) + (size_t)(level + d.tau_pos) * d.diag_stride;
  }
  const int N = sys.N;
  const long long per_active = (long long)N * nlinks;
  const long long total = per_active * act.n;
  double acc = 0.0;
  const bool small = total <= 0x7fffffffll;  // 32-bit divisions: the 64-bit ones are a call each
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    int pi, link, p2;
    if (small) {
      const unsigned i = (unsigned)idx, pa1 = (unsigned)per_active;
      pi = act.n == 1 ? 0 : (int)(i / pa1);
      const unsigned rem = i - (unsigned)pi * pa1;
      link = (int)(rem / (unsigned)N);
      p2 = (int)(rem - (unsigned)link * (unsigned)N);
    } else {
      pi = (int)(idx / per_active);
      const long long rem = idx - pi * per_active;
      link = (int)(rem / N);
      p2 = (int)(rem - (long long)link * N);
    }
    const int p1 = act.p[pi];
    bool visited = false;  // Path.DoPtcl: moved particles count once
    for (int k = 0; k <= pi; k++) visited |= (act.p[k] == p2);
    if (visited) continue;
    const int slice = slice1 + link * skip;
    double a1[3], a2[3], b1[3], b2[3], dA[3], dB[3];
    load3(path + ((size_t)slice * N + p1) * 3, a1);
    load3(path + ((size_t)slice * N + p2) * 3, a2);
    load3(path + ((size_t)(slice + skip) * N + p1) * 3, b1);
    load3(path + ((size_t)(slice + skip) * N + p2) * 3, b2);
    dist_disp(a1, a2, b1, b2, sys, dA, dB);
    LinkGeom<R> g = link_geom<R>(dA, dB);
    acc += (double)pa_U<R, KIND>(pa, diag, g, level);
  }
  double r = block_sum(acc, sh);
  finish_sum(r, partials, counter, out, sh);
}

// ---- observables: PairCorrelationClass::Accumulate ----
// PathClass::DistDisp one-slice form (PathClass.h:637-660): minimum image by
// nearbyint(disp / L), then |disp|.
__device__ __forceinline__ double dist_one_slice(const double a[3], const double b[3], const DevSystem &s) {
  double d2 = 0.0;
#pragma unroll
  for (int i = 0; i < 3; i++) {
    double d = b[i] - a[i];
    const double n = rint(rmul(d, s.boxinv[i]));
    d = rsub(d, rmul(n, s.box[i]));
    d2 = radd(d2, rmul(d, d));
  }
  return sqrt(d2);
}

// The g(r) histogram: slices [0, S-2] x pairs p2 < p1 of the OLD path, pair
// distances below the grid end in bin (int)nearbyint((r - start) * deltainv -
// 0.5) (ObservableCorrelation.cc:191-207, Grid.h:81-84); bins counted per block
// in shared memory, then added to the 64-bit histogram.
// A block takes (tile of particles) x (tile) x slice items: the tiles'
// positions are boxed in FP64 and staged as 32-bit fractions of the box, so a
// difference wraps to the minimum image by itself; a pair's distance, in bins,
// and its place on the grid are formed from it in FP32.  The place carries an
// error below `err` bins (see launch_gofr); a pair nearer than that to a bin's
// edge, and every pair of two tiles with a position that the fractions cannot
// hold, is binned from its FP64 distance, so the counts are the FP64
// evaluation's.  Bound by instruction issue (75 %, 42 instructions a pair).
// N = 512, M = 128, 100 bins (ncu): 138 us with FP64 distances and 64-bit index
// arithmetic for every pair, 44 with FP32 coordinates and the image by rounding,
// 40 with the fractions, 34 with the open pairs noted and binned after the rows
// instead of a branch at each.  Tiles of 128: 52, too few items to share out evenly.
template <int JPL>  // j particles per lane: tiles of 32 JPL particles
__global__ void __launch_bounds__(256, 4) gofr_kernel(const double *__restrict__ path, DevSystem sys, GofrGrid gg,
                                                      long long items, float half, unsigned long long *hist) {
  constexpr int T = 32 * JPL;
  extern __shared__ unsigned int s_hist[];
  __shared__ int4 s_pos[2 * T];  // the i tile, then the j tile
  const int N = sys.N, S1 = sys.S - 1, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < gg.nbins; i += blockDim.x) s_hist[i] = 0u;
  // squares of the bins in a 2^32nd of each box side; the grid start and half a bin, in bins
  const double ux = 0x1p-32 * sys.box[0] * gg.deltainv, uy = 0x1p-32 * sys.box[1] * gg.deltainv,
               uz = 0x1p-32 * sys.box[2] * gg.deltainv;
  const float sx = (float)(ux * ux), sy = (float)(uy * uy), sz = (float)(uz * uz);
  const float t0 = (float)(gg.start * gg.deltainv + 0.5);
  // A block takes consecutive items, slice fastest, so it divides once.
  const long long beg = gofr_first(items, gridDim.x, blockIdx.x), end = gofr_first(items, gridDim.x, blockIdx.x + 1ll);
  int ti, tj, slice = (int)(beg % S1);
  tri_decode(beg / S1, ti, tj);
  for (long long item = beg; item < end; item++) {
    const int i0 = ti * T, j0 = tj * T;
    const int ni = min(T, N - i0), nj = min(T, N - j0);
    const double *row = path + (size_t)slice * N * 3;
    __syncthreads();  // the previous item's readers are done
    bool far = false;
    if (tid < 2 * T) {
      const int p = tid < T ? i0 + tid : j0 + tid - T;
      if (p < N) {
        int v[3];
#pragma unroll
        for (int d = 0; d < 3; d++) {
          const double f = row[(size_t)p * 3 + d] * sys.boxinv[d];
          far |= !(fabs(f) <= 1e6);
          v[d] = (int)(unsigned)__double2ll_rn((f - round_even_magic(f)) * 0x1p32);  // both halves: -2^31
        }
        s_pos[tid] = make_int4(v[0], v[1], v[2], 0);
      }
    }
    const float lim = __syncthreads_or(far) ? -1.0f : half;
    int4 q[JPL];
#pragma unroll
    for (int h = 0; h < JPL; h++) q[h] = s_pos[T + lane + 32 * h];
    unsigned edges = 0u;  // this lane's pairs that FP32 leaves open, binned below: no branch in the loop
#pragma unroll
    for (int r = 0; r < T / 8; r++) {
      const int i = warp + 8 * r;
      const int4 p = s_pos[i];
      const int jend = i < ni ? (ti == tj ? i : nj) : 0;
#pragma unroll
      for (int h = 0; h < JPL; h++) {
        const float dx = (float)(int)((unsigned)q[h].x - (unsigned)p.x), dy = (float)(int)((unsigned)q[h].y - (unsigned)p.y),
                    dz = (float)(int)((unsigned)q[h].z - (unsigned)p.z);
        float dist;
        asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(dist) : "f"(dx * dx * sx + dy * dy * sy + dz * dz * sz));
        const float t = dist - t0, m = __fadd_rn(t, 12582912.0f);  // t's integer, as in round_even_magic
        const unsigned bin = __float_as_uint(m) - 0x4B400000u;
        const bool in = lane + 32 * h < jend, sure = fabsf(t - __fadd_rn(m, -12582912.0f)) < lim;
        if (in && !sure) edges |= 1u << (r * JPL + h);
        if (in && sure && bin < (unsigned)gg.nbins) atomicAdd(&s_hist[bin], 1u);
      }
    }
    while (edges) {
      const int k = __ffs(edges) - 1, i = warp + 8 * (k / JPL), j = lane + 32 * (k % JPL);
      edges &= edges - 1u;
      double a[3], b[3];
      load3(row + (size_t)(i0 + i) * 3, a);
      load3(row + (size_t)(j0 + j) * 3, b);
      const double d64 = dist_one_slice(a, b, sys);
      const int bin = d64 < gg.end ? (int)rint(rsub(rmul(rsub(d64, gg.start), gg.deltainv), 0.5)) : -1;
      if ((unsigned)bin < (unsigned)gg.nbins) atomicAdd(&s_hist[bin], 1u);
    }
    if (++slice == S1) {
      slice = 0;
      if (++tj > ti) {
        ti++;
        tj = 0;
      }
    }
  }
  __syncthreads();
  for (int i = tid; i < gg.nbins; i += blockDim.x)
    if (s_hist[i]) atomicAdd(&hist[i], (unsigned long long)s_hist[i]);
}

__device__ __forceinline__ void velocity(const double *__restrict__ path, int N, int sa, int sb, int p,
                                         const DevSystem &sys, double v[3]) {
  double a[3], b[3];
  load3(path + ((size_t)sa * N + p) * 3, a);
  load3(path + ((size_t)sb * N + p) * 3, b);
  for (int i = 0; i < 3; i++) v[i] = b[i] - a[i];
  put_in_box(v, sys);
}

// KineticClass::SingleAction (KineticClass.cc:33-90)
__global__ void __launch_bounds__(kReduceThreads) kin_single_kernel(const double *__restrict__ path, DevSystem sys,
                                                         ActiveList act, int slice1, int skip, int nlinks, int level,
                                                         double *partials, unsigned int *counter, double *out) {
  __shared__ double sh[kReduceThreads / 32];
  const double levelTau = sys.tau * (1 << level);
  const double F = 1.0 / (4.0 * sys.lambda * levelTau);
  const int total = act.n * nlinks;
  double acc = 0.0;
  if (sys.lambda != 0.0)
    for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += gridDim.x * blockDim.x) {
      const int pi = idx / nlinks, link = idx - pi * nlinks;
      const int slice = slice1 + link * skip;
      double vel[3];
      velocity(path, sys.N, slice, slice + skip, act.p[pi], sys, vel);
      acc += kinetic_link(vel, F, sys.num_images, sys);
    }
  double r = block_sum(acc, sh);
  finish_sum(r, partials, counter, out, sh);
}

// KineticClass::d_dBeta (KineticClass.cc:187-256)
__global__ void __launch_bounds__(kReduceThreads) kin_dbeta_kernel(const double *__restrict__ path, DevSystem sys, int slice1,
                                                        int skip, int nlinks, int level, double *partials,
                                                        unsigned int *counter, double *out) {
  __shared__ double sh[kReduceThreads / 32];
  const double levelTau = ldexp(sys.tau, level);
  const double F = 1.0 / (4.0 * sys.lambda * levelTau);
  const int total = sys.N * nlinks;
  double acc = 0.0;
  if (sys.lambda != 0.0)
    for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += gridDim.x * blockDim.x) {
      const int link = idx / sys.N, p = idx - link * sys.N;
      const int slice = slice1 + link * skip;
      double vel[3];
      velocity(path, sys.N, slice, slice + skip, p, sys, vel);
      double spring = (0.5 * 3) / levelTau;
      double Z = 1.0, GaussSum[3] = {0, 0, 0}, numSum[3] = {0, 0, 0};
      for (int dim = 0; dim < 3; dim++) {
        for (int image = -sys.num_images; image <= sys.num_images; image++) {
          double dist = vel[dim] + (double)image * sys.box[dim];
          double d2overFLT = dist * dist * F;
          double expPart = exp(-d2overFLT);
          GaussSum[dim] += expPart;
          numSum[dim] += -d2overFLT / levelTau * expPart;
        }
        Z *= GaussSum[dim];
      }
      double scalarnumSum = 0.0;
      for (int dim = 0; dim < 3; dim++) {
        double numProd = 1.0;
        for (int dim2 = 0; dim2 < 3; dim2++) numProd *= (dim2 != dim) ? GaussSum[dim2] : numSum[dim2];
        scalarnumSum += numProd;
      }
      acc += spring + scalarnumSum / Z;
    }
  double r = block_sum(acc, sh);
  finish_sum(r, partials, counter, out, sh);
}

// PathClass::AcceptCopy (PathClass.cc:797-863): PutInBoxFast on NEW, NEW -> OLD.
__global__ void accept_kernel(double *path_old, double *path_new, DevSystem sys, ActiveList act, int slice1,
                              int nslices) {
  int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= act.n * nslices) return;
  int pi = idx / nslices, slice = slice1 + (idx - pi * nslices);
  size_t o = ((size_t)slice * sys.N + act.p[pi]) * 3;
  double v[3] = {path_new[o], path_new[o + 1], path_new[o + 2]};
  put_in_box_fast(v, sys);
  for (int i = 0; i < 3; i++) {
    path_new[o + i] = v[i];
    path_old[o + i] = v[i];
  }
}

// PathClass::RejectCopy (PathClass.cc:865-899): OLD -> NEW.
__global__ void reject_kernel(const double *path_old, double *path_new, DevSystem sys, ActiveList act, int slice1,
                              int nslices) {
  int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= act.n * nslices) return;
  int pi = idx / nslices, slice = slice1 + (idx - pi * nslices);
  size_t o = ((size_t)slice * sys.N + act.p[pi]) * 3;
  for (int i = 0; i < 3; i++) path_new[o + i] = path_old[o + i];
}

// ---------------------------------------------------------------------------
// Host launchers
// ---------------------------------------------------------------------------
static int grid_for(long long items, int sm_count) {
  long long b = (items + kReduceThreads - 1) / kReduceThreads;
  b = std::min(b, std::min((long long)sm_count * 16, (long long)kPartialSlots));
  return (int)std::max(b, 1ll);
}

cudaError_t launch_sr_single(const ReduceTarget &t, const double *path, const DevSystem &sys, const DevPA &pa,
                             const ActiveList &act, int slice1, int skip, int nlinks, int level, int precision,
                             int sm_count) {
  long long items = (long long)act.n * sys.N * nlinks;
  int blocks = grid_for(items, sm_count);
  if (pa.kind == PA_DAVID) {
    if (precision == PIMC_MIXED)
      sr_single_kernel<PA_DAVID, float><<<blocks, kReduceThreads, 0, t.stream>>>(path, sys, pa, act, slice1, skip, nlinks, level,
                                                                       t.partials, t.counter, t.out);
    else
      sr_single_kernel<PA_DAVID, double><<<blocks, kReduceThreads, 0, t.stream>>>(path, sys, pa, act, slice1, skip, nlinks, level,
                                                                        t.partials, t.counter, t.out);
  } else if (pa.kind == PA_COULOMB) {
    if (precision == PIMC_MIXED)
      sr_single_kernel<PA_COULOMB, float><<<blocks, kReduceThreads, 0, t.stream>>>(path, sys, pa, act, slice1, skip, nlinks,
                                                                         level, t.partials, t.counter, t.out);
    else
      sr_single_kernel<PA_COULOMB, double><<<blocks, kReduceThreads, 0, t.stream>>>(path, sys, pa, act, slice1, skip, nlinks,
                                                                          level, t.partials, t.counter, t.out);
  } else {
    if (precision == PIMC_MIXED)
      sr_single_kernel<PA_TRICUBIC, float><<<blocks, kReduceThreads, 0, t.stream>>>(path, sys, pa, act, slice1, skip, nlinks,
                                                                          level, t.partials, t.counter, t.out);
    else
      sr_single_kernel<PA_TRICUBIC, double><<<blocks, kReduceThreads, 0, t.stream>>>(path, sys, pa, act, slice1, skip, nlinks,
                                                                           level, t.partials, t.counter, t.out);
  }
  return cudaGetLastError();
}

cudaError_t launch_kin_single(const ReduceTarget &t, const double *path, const DevSystem &sys, const ActiveList &act,
                              int slice1, int skip, int nlinks, int level, int sm_count) {
  int blocks = grid_for((long long)act.n * nlinks, sm_count);
  kin_single_kernel<<<blocks, kReduceThreads, 0, t.stream>>>(path, sys, act, slice1, skip, nlinks, level, t.partials, t.counter,
                                                  t.out);
  return cudaGetLastError();
}

cudaError_t launch_kin_dbeta(const ReduceTarget &t, const double *path, const DevSystem &sys, int slice1, int skip,
                             int nlinks, int level, int sm_count) {
  int blocks = grid_for((long long)sys.N * nlinks, sm_count);
  kin_dbeta_kernel<<<blocks, kReduceThreads, 0, t.stream>>>(path, sys, slice1, skip, nlinks, level, t.partials, t.counter,
                                                 t.out);
  return cudaGetLastError();
}

// err, in bins, with u = 2^-24.  A coordinate's fraction: 2^-33 for the integer
// and 1e6 2^-52 for boxing; the FP64 distance's own rounding at such a coordinate
// is as large: below 2^-29 of the side for a difference, twice that where the two
// choose different images at half a box, sqrt(3) times that for the distance:
// 2^-27 L.  The conversion, the squares, the scales and the sum round by 7 u of
// the square, the root by 4 u: 7.5 u of a distance, the start and the place by
// 2 u of themselves, at most nbins + 1 bins beyond the start where it counts.
// From 1/2 on every pair takes the FP64 path, as for boxes of less than 1e-6 or
// more than 1e6 bins, which the FP32 squares and the rounding do not hold.
cudaError_t launch_gofr(cudaStream_t st, const double *path, const DevSystem &sys, const GofrGrid &gg,
                        unsigned long long *hist, int sm_count) {
  double err = 0.0;
  for (double L : sys.box) {
    const double bins = L * gg.deltainv;
    err = fmax(err, bins > 1e-6 && bins < 1e6 ? bins * 0x1p-27 : HUGE_VAL);
  }
  err += 16.0 * (gg.nbins + 2 + fabs(gg.start * gg.deltainv)) * 0x1p-24;
  const float half = fmax(0.5 - err, -1.0);  // a place nearer than this to its bin's centre is sure
  const GofrShape shape = gofr_shape(sys.N, sys.S - 1, sm_count);
  const size_t dyn = (size_t)gg.nbins * sizeof(unsigned int);
  auto kfn = shape.tile == 64 ? gofr_kernel<2> : gofr_kernel<1>;
  const cudaError_t e = cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             12288 * (int)sizeof(unsigned int));  // beside the static tiles
  if (e != cudaSuccess) return e;
  kfn<<<shape.blocks, 256, dyn, st>>>(path, sys, gg, shape.items, half, hist);
  return cudaGetLastError();
}

cudaError_t launch_accept(cudaStream_t st, double *path_old, double *path_new, const DevSystem &sys,
                          const ActiveList &act, int slice1, int slice2) {
  int nslices = slice2 - slice1 + 1;
  int items = act.n * nslices;
  accept_kernel<<<(items + 127) / 128, 128, 0, st>>>(path_old, path_new, sys, act, slice1, nslices);
  return cudaGetLastError();
}

cudaError_t launch_reject(cudaStream_t st, const double *path_old, double *path_new, const DevSystem &sys,
                          const ActiveList &act, int slice1, int slice2) {
  int nslices = slice2 - slice1 + 1;
  int items = act.n * nslices;
  reject_kernel<<<(items + 127) / 128, 128, 0, st>>>(path_old, path_new, sys, act, slice1, nslices);
  return cudaGetLastError();
}

}  // namespace pimc
