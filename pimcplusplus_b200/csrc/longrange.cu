// Long-range (Ewald breakup) k-space pieces on the device:
//   PathClass::SetupkVecs3D       (PathClass.cc:534-586)  — host, in capi
//   PathClass::CalcRho_ks_Fast    (PathClass.cc:616-647)  — rhok_full_kernel
//   PathClass::UpdateRho_ks       (PathClass.cc:649-707)  — rhok_update_kernel
//   LongRangeClass::SingleAction  (LongRangeClass.cc:273-371) and
//   LongRangeClass::d_dBeta       (LongRangeClass.cc:374-442) — lr_sum_kernel
//   DavidLongRangeClassYk::SingleAction / d_dBeta / V
//                                 (DavidLongRangeClassYk.cc:230-389) — lr_sum_kernel
//
// rho_k is stored [slice][k] as double2 (re, im), one species.  The phase
// factors follow the reference exactly: per particle and dimension,
// C_d(n) = e^{i n kBox_d x_d} is built by repeated multiplication from
// C_d(1) = (cos, sin)(kBox_d x_d), C_d(-n) = conj(C_d(n)), and a k-vector's
// term is (C_0(kx) C_1(ky)) C_2(kz).  The tables of the particles a block
// handles are built cooperatively in shared memory.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "action_kernels.cuh"
#include "device_math.cuh"
#include "longrange.cuh"

namespace cg = cooperative_groups;

namespace pimc {

namespace {

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// Fills C[d][n + kmax_d] for one coordinate x of dimension d into shared
// memory (one thread per dimension).
__device__ __forceinline__ void fill_phase_table(double x, int d, const LRDesc &lr, double2 *C) {
  const int m = lr.kmax[d];
  const double phi = x * lr.kbox[d];
  double s, c;
  sincos(phi, &s, &c);
  const double2 t = make_double2(c, s);
  double2 *Cd = C + lr.coff[d];
  double2 w = make_double2(1.0, 0.0);  // the running power stays in registers: a shared-memory round trip a step costs more
  Cd[m] = w;
  for (int n = 1; n <= m; n++) {
    w = cmul(t, w);
    Cd[m + n] = w;
    Cd[m - n] = make_double2(w.x, -w.y);
  }
}

__device__ __forceinline__ double2 k_term(const double2 *C, const LRDesc &lr, int3 ki) {
  const double2 a = C[lr.coff[0] + ki.x], b = C[lr.coff[1] + ki.y], c = C[lr.coff[2] + ki.z];
  return cmul(cmul(a, b), c);
}

constexpr int kMaxPhase = 3 * (2 * 64 + 1);  // kmax <= 64 per dimension

// rho_k(slice) = sum over particles of the k terms: one cluster of CL blocks
// per slice, each block a contiguous share of the particles.  A block builds
// the phase tables of up to `batch` particles at once (thread t: particle
// t / 3, dimension t % 3), then every thread adds its k-vectors' terms of the
// whole batch; at the end the cluster's partial sums are added in rank order
// through distributed shared memory, so the result is reproducible.
// What bounds it: the shared-memory reads of the phases (three 16-byte reads
// per k-vector and particle against 10 FP64 operations; neighbouring threads
// share kx and ky, so most are broadcasts) and, at few particles per block, the
// latency of sincos and of the recurrence.  Measured against one block per
// slice that builds one particle's table at a time between two barriers
// (pimc_calc_rhok): N = 128, 65 slices, 510 k-vectors 142 -> 26 us (the kernel
// 139 -> 15), N = 1024, 65 slices, 787 k-vectors 1397 -> 104 us, N = 4000, 3
// slices, 230 k-vectors 3347 -> 48 us.
__global__ void __launch_bounds__(256) rhok_full_kernel(const double *__restrict__ path, int N, LRDesc lr, int batch,
                                                        double2 *rhok) {
  extern __shared__ double2 sh2[];  // phase tables [batch][tab], then the partial sums [nk]
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), CL = (int)cluster.num_blocks();
  const int slice = (int)blockIdx.x / CL;
  const int tab = lr.coff[2] + 2 * lr.kmax[2] + 1;
  const int per = (N + CL - 1) / CL, beg = min(N, rank * per), end = min(N, beg + per);
  double2 acc[4];
  int o0[4], o1[4], o2[4];  // this thread's k-vectors (nk <= 1024): offsets into a phase table
#pragma unroll
  for (int j = 0; j < 4; j++) {
    acc[j] = make_double2(0.0, 0.0);
    const int k = threadIdx.x + j * blockDim.x;
    const int3 ki = k < lr.nk ? lr.kidx[k] : make_int3(0, 0, 0);
    o0[j] = lr.coff[0] + ki.x;
    o1[j] = lr.coff[1] + ki.y;
    o2[j] = lr.coff[2] + ki.z;
  }
  for (int p0 = beg; p0 < end; p0 += batch) {
    const int np = min(batch, end - p0);
    for (int t = threadIdx.x; t < 3 * np; t += blockDim.x) {
      const int p = t / 3, d = t - 3 * p;
      fill_phase_table(path[((size_t)slice * N + p0 + p) * 3 + d], d, lr, sh2 + (size_t)p * tab);
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 4; j++) {
      if ((int)threadIdx.x + j * (int)blockDim.x >= lr.nk) break;
#pragma unroll 2
      for (int p = 0; p < np; p++) {
        const double2 *C = sh2 + (size_t)p * tab;
        const double2 t = cmul(cmul(C[o0[j]], C[o1[j]]), C[o2[j]]);
        acc[j].x += t.x;
        acc[j].y += t.y;
      }
    }
    __syncthreads();
  }
  if (CL == 1) {
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int k = threadIdx.x + j * blockDim.x;
      if (k < lr.nk) rhok[(size_t)slice * lr.nk + k] = acc[j];
    }
    return;
  }
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const int k = threadIdx.x + j * blockDim.x;
    if (k < lr.nk) sh2[k] = acc[j];
  }
  cluster.sync();
  for (int k = rank * (int)blockDim.x + (int)threadIdx.x; k < lr.nk; k += CL * (int)blockDim.x) {
    double2 v = make_double2(0.0, 0.0);
    for (int r = 0; r < CL; r++) {
      const double2 w = cluster.map_shared_rank(sh2, r)[k];
      v.x += w.x;
      v.y += w.y;
    }
    rhok[(size_t)slice * lr.nk + k] = v;
  }
  cluster.sync();  // no block leaves while a peer reads its sums
}

__device__ __forceinline__ double lr_block_sum(double v, double *sh) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) sh[w] = v;
  __syncthreads();
  double r = 0.0;
  if (threadIdx.x == 0)
    for (int i = 0; i < (int)(blockDim.x >> 5); i++) r += sh[i];
  return r;
}

// This block's partial, and the last block's sum of all partials in block order.
__device__ __forceinline__ void lr_finish(double acc, double *partials, unsigned int *counter, double *out) {
  __shared__ double sh[32];
  __shared__ int s_last;
  const double v = lr_block_sum(acc, sh);
  if (threadIdx.x == 0) {
    partials[blockIdx.x] = v;
    __threadfence();
    s_last = (atomicAdd(counter, 1u) == gridDim.x - 1);
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  double w = 0.0;
  for (int i = threadIdx.x; i < (int)gridDim.x; i += blockDim.x) w += __ldcg(&partials[i]);
  const double tot = lr_block_sum(w, sh);
  if (threadIdx.x == 0) {
    *out = tot;
    *counter = 0u;
  }
}

// One block per updated slice (slice1 + b*skip): NEW = OLD, then per active
// particle NEW += C(r_new), NEW -= C(r_old), in the reference's order.  SUM: the
// k sum of lr_sum_kernel over the updated slices in the same launch, from the
// values in registers (LongRangeClass::SingleAction on the NEW copy).
template <bool SUM>
__global__ void __launch_bounds__(256) rhok_update_kernel(const double *__restrict__ path_old,
                                                          const double *__restrict__ path_new, int N, LRDesc lr,
                                                          ActiveList act, int slice1, int skip,
                                                          const double2 *__restrict__ rho_old, double2 *rho_new,
                                                          const double *__restrict__ uk, int slice2,
                                                          double end_weight, double *partials,
                                                          unsigned int *counter, double *out) {
  __shared__ double2 Cn[kMaxPhase], Co[kMaxPhase];
  const int slice = slice1 + blockIdx.x * skip;
  double2 acc[4];  // this thread's k-vectors (nk <= 1024)
  int3 ki[4];
  double u[4];
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const int k = threadIdx.x + j * blockDim.x;
    if (k >= lr.nk) break;
    acc[j] = rho_old[(size_t)slice * lr.nk + k];
    ki[j] = lr.kidx[k];
    u[j] = SUM ? uk[k] : 0.0;
  }
  for (int pi = 0; pi < act.n; pi++) {
    __syncthreads();
    const int p = act.p[pi];
    if (threadIdx.x < 3) {
      fill_phase_table(path_new[((size_t)slice * N + p) * 3 + threadIdx.x], threadIdx.x, lr, Cn);
    } else if (threadIdx.x >= 32 && threadIdx.x < 35) {
      fill_phase_table(path_old[((size_t)slice * N + p) * 3 + threadIdx.x - 32], threadIdx.x - 32, lr, Co);
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 4; j++) {
      if ((int)threadIdx.x + j * (int)blockDim.x >= lr.nk) break;
      const double2 tn = k_term(Cn, lr, ki[j]);
      acc[j].x += tn.x;
      acc[j].y += tn.y;
      const double2 to = k_term(Co, lr, ki[j]);
      acc[j].x -= to.x;
      acc[j].y -= to.y;
    }
  }
  double sum = 0.0;
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const int k = threadIdx.x + j * blockDim.x;
    if (k >= lr.nk) break;
    rho_new[(size_t)slice * lr.nk + k] = acc[j];
    if (SUM) sum += (acc[j].x * acc[j].x + acc[j].y * acc[j].y) * u[j];
  }
  if (SUM) lr_finish(slice == slice1 || slice == slice2 ? sum * end_weight : sum, partials, counter, out);
}

// sum over slices [slice1, slice2] step skip of factor * sum_k |rho_k|^2 u_k
// (the homologous k-space term); factor 1/2 at the two ends.
__global__ void __launch_bounds__(256) lr_sum_kernel(const double2 *__restrict__ rhok, LRDesc lr,
                                                     const double *__restrict__ uk, int slice1, int slice2, int skip,
                                                     double end_weight, double *partials, unsigned int *counter,
                                                     double *out) {
  const int nsl = (slice2 - slice1) / skip + 1;
  const long long total = (long long)nsl * lr.nk;
  double acc = 0.0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int b = (int)(i / lr.nk), k = (int)(i - (long long)b * lr.nk);
    const int slice = slice1 + b * skip;
    const double factor = (slice == slice1 || slice == slice2) ? end_weight : 1.0;
    const double2 r = rhok[(size_t)slice * lr.nk + k];
    const double rhok2 = r.x * r.x + r.y * r.y;
    acc += factor * 0.5 * 2.0 * rhok2 * uk[k];
  }
  lr_finish(acc, partials, counter, out);
}

__global__ void rhok_copy_kernel(const double2 *__restrict__ src, double2 *dst, int nk, int slice1, int nslices) {
  const long long total = (long long)nslices * nk;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const size_t o = (size_t)slice1 * nk + (size_t)i;
    dst[o] = src[o];
  }
}

}  // namespace

// Blocks per slice: doubled until about four blocks come to every SM (their
// sincos and table latencies overlap), while each keeps eight particles or
// more; one block per slice where the slices alone do that.
cudaError_t launch_rhok_full(cudaStream_t st, const double *path, int N, int S, const LRDesc &lr, int sm_count,
                             double2 *rhok) {
  int cl = 1;
  while (cl < 8 && S * cl < 4 * sm_count && N >= 16 * cl) cl *= 2;
  const int tab = lr.coff[2] + 2 * lr.kmax[2] + 1;
  const int share = (N + cl - 1) / cl;
  // tables of as many particles as 45 KB hold (kmax <= 64: 7 or more), 85 at most (a thread per particle and dimension)
  const int batch = std::min(share, std::max(1, std::min(85, 45 * 1024 / (tab * (int)sizeof(double2)))));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(S * cl, 1, 1);
  cfg.blockDim = dim3(256, 1, 1);
  cfg.dynamicSmemBytes = (size_t)std::max(batch * tab, lr.nk) * sizeof(double2);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cl;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, rhok_full_kernel, path, N, lr, batch, rhok);
}

cudaError_t launch_rhok_update(cudaStream_t st, const double *path_old, const double *path_new, int N,
                               const LRDesc &lr, const ActiveList &act, int slice1, int slice2, int skip,
                               const double2 *rho_old, double2 *rho_new) {
  const int nsl = (slice2 - slice1) / skip + 1;
  rhok_update_kernel<false><<<nsl, 256, 0, st>>>(path_old, path_new, N, lr, act, slice1, skip, rho_old, rho_new,
                                                 nullptr, 0, 0.0, nullptr, nullptr, nullptr);
  return cudaGetLastError();
}

cudaError_t launch_rhok_update_sum(const ReduceTarget &t, const double *path_old, const double *path_new, int N,
                                   const LRDesc &lr, const ActiveList &act, int slice1, int slice2, int skip,
                                   const double2 *rho_old, double2 *rho_new, const double *uk, int sm_count,
                                   double end_weight) {
  const int nsl = (slice2 - slice1) / skip + 1;
  if (nsl > kPartialSlots) {  // a partial a slice
    const cudaError_t e = launch_rhok_update(t.stream, path_old, path_new, N, lr, act, slice1, slice2, skip, rho_old,
                                             rho_new);
    return e != cudaSuccess ? e : launch_lr_sum(t, rho_new, lr, uk, slice1, slice2, skip, sm_count, end_weight);
  }
  rhok_update_kernel<true><<<nsl, 256, 0, t.stream>>>(path_old, path_new, N, lr, act, slice1, skip, rho_old, rho_new,
                                                      uk, slice2, end_weight, t.partials, t.counter, t.out);
  return cudaGetLastError();
}

cudaError_t launch_lr_sum(const ReduceTarget &t, const double2 *rhok, const LRDesc &lr, const double *uk, int slice1,
                          int slice2, int skip, int sm_count, double end_weight) {
  const int nsl = (slice2 - slice1) / skip + 1;
  long long items = (long long)nsl * lr.nk;
  long long blocks = (items + 255) / 256;
  if (blocks > sm_count * 4) blocks = sm_count * 4;
  if (blocks > kPartialSlots) blocks = kPartialSlots;
  if (blocks < 1) blocks = 1;
  lr_sum_kernel<<<(int)blocks, 256, 0, t.stream>>>(rhok, lr, uk, slice1, slice2, skip, end_weight, t.partials,
                                                   t.counter, t.out);
  return cudaGetLastError();
}

cudaError_t launch_rhok_copy(cudaStream_t st, const double2 *src, double2 *dst, int nk, int slice1, int slice2) {
  const int nsl = slice2 - slice1 + 1;
  const long long items = (long long)nsl * nk;
  rhok_copy_kernel<<<(int)((items + 255) / 256), 256, 0, st>>>(src, dst, nk, slice1, nsl);
  return cudaGetLastError();
}

}  // namespace pimc
