// Small utility kernels of the numeric path: zeroing a level's fronts and
// the FP64 residual / backward-error / update kernels of iterative
// refinement.  The residual uses the matrix in pivot order as a full CSR
// whose values are read through the user's value array (no copy), so a
// same-pattern refactorisation needs no symbolic work.  The backward error is
// the scaled residual of tests/ssids/ssids.f90:1762-1810:
//   max_i |b - A x|_i / (||A||_inf ||x||_inf + ||b||_inf).
#include "ssids_gpu.cuh"

namespace ssids300 {

namespace {

// zero n elements from p (16-byte aligned) with 16-byte stores
template <typename T>
__device__ __forceinline__ void zero_range(T* p, int64_t n, int64_t i0, int64_t stride) {
  constexpr int V = 16 / sizeof(T);
  const int64_t nv = n / V;
  int4* q = reinterpret_cast<int4*>(p);
  for (int64_t i = i0; i < nv; i += stride) q[i] = make_int4(0, 0, 0, 0);
  for (int64_t i = nv * V + i0; i < n; i += stride) p[i] = T(0);
}

// Zero a level's fronts: L (ld x n, contiguous) and D.  Fronts start
// 256-byte aligned, so the stores are 16 bytes wide.  The contribution
// blocks are zeroed column by column by the extend-add, which owns them.
template <typename T>
__global__ void k_zero_fronts(FrontDesc<T>* fds, const int* fronts) {
  const FrontDesc<T> fd = fds[fronts[blockIdx.y]];
  const int64_t nl = (int64_t)fd.ld * fd.n;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t i0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  zero_range(fd.L, nl, i0, stride);
  zero_range(fd.D, 2 * (int64_t)fd.n, i0, stride);
}

// Maxima of magnitudes as integers: non-negative doubles order like their bit
// patterns, and an FP64 maximum issues some 30 times slower than an integer
// one on GB300.
typedef unsigned long long u64;
__device__ __forceinline__ u64 mag_bits(double v) {  // a NaN is above every number
  return (u64)__double_as_longlong(v) & 0x7fffffffffffffffULL;
}
__device__ __forceinline__ u64 warp_max(u64 k) {
  const unsigned hi = (unsigned)(k >> 32), lo = (unsigned)k;
  const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
  const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
  return ((u64)mh << 32) | ml;
}
__device__ __forceinline__ void atomic_max_pos(double* a, u64 bits) {
  atomicMax(reinterpret_cast<u64*>(a), bits);
}

// r = b - A x and the maxima of the scaled backward error in one pass.  Each
// non-zero is applied to kResQC right-hand sides at once (chunk blockIdx.y),
// so the row's index and value loads are shared by the chunk.  work: [0]
// ||A||_inf, then per rhs (||x||, ||b||, ||r||) at 1 + 3q (maxima,
// order-independent).
//
// Bound by FP64 issue (about 75 cycles a warp instruction): a non-zero costs
// one multiply-add per right-hand side and, in the first chunk, one addition
// for the row sum.  One lane per row needs the fewest (no partial sums to add
// over lanes), but a warp waits for its longest row: a row of more than
// kResShort non-zeros is read by four lanes.  Each row goes by its own length,
// so its residual has the same bits whatever rows and matrices are beside it.
// A warp takes RPW rows: 32, or 8 where rows average more than kResShort
// non-zeros and most are read by four lanes (the order of a row's sum does not
// depend on it).  320 stacked 2D Laplacians (n = 0.93M, one right-hand side):
// 751 -> 123 us, 48^3 Laplacian with 8 right-hand sides 127 -> 62 us, with the
// maxima in integers.
constexpr int kResQC = 4;
constexpr int kResShort = 12;
// the non-zeros k0, k0 + step, ... < k1 of a row
__device__ __forceinline__ void resid_row(const int* acol, const int64_t* asrc, const double* aval,
                                          const double* x, int ld, int q0, int nq, bool norm,
                                          int64_t k0, int64_t k1, int step, double (&s)[kResQC],
                                          double& ra) {
  for (int64_t k = k0; k < k1; k += step) {
    const double a = aval[asrc[k]];
    const int64_t c = acol[k];
    if (norm) ra += fabs(a);
#pragma unroll
    for (int q = 0; q < kResQC; ++q)
      if (q < nq) s[q] = fma(a, x[(int64_t)(q0 + q) * ld + c], s[q]);
  }
}
// With row groups (row_group != nullptr: the group of each row, e.g. the
// matrix of a batch it belongs to) the maxima are kept per group, at
// work[g * kResStride ...], so the backward error can be judged per group.
template <int RPW>
__global__ void __launch_bounds__(256) k_resid_norms(const int64_t* aptr, const int* acol,
                                                     const int64_t* asrc, const double* aval,
                                                     int n, const double* x, const double* b,
                                                     double* r, int nrhs, int ld, double* work,
                                                     const int* row_group) {
  constexpr int QC = kResQC, NV = 1 + 3 * QC;
  const int lane = threadIdx.x & 31;
  const int q0 = blockIdx.y * QC;
  const int nq = min(QC, nrhs - q0);
  const bool norm = blockIdx.y == 0;  // this chunk forms ||A||
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarp = ((int64_t)gridDim.x * blockDim.x) >> 5;
  u64 m[NV];  // ||A||, then (x, b, r) per right-hand side
#pragma unroll
  for (int v = 0; v < NV; ++v) m[v] = 0;
  for (int64_t base = warp * RPW; base < n; base += nwarp * RPW) {
    const int64_t i = base + lane;  // this lane's row
    const bool ok = lane < RPW && i < n;
    const int64_t k0 = ok ? aptr[i] : 0, k1 = ok ? aptr[i + 1] : 0;
    const bool wide = k1 - k0 > kResShort;
    double s[QC], ra = 0.0;
#pragma unroll
    for (int q = 0; q < QC; ++q) s[q] = 0.0;
    if (!wide) resid_row(acol, asrc, aval, x, ld, q0, nq, norm, k0, k1, 1, s, ra);
    const unsigned wides = __ballot_sync(0xffffffffu, wide);
    if (wides) {
#pragma unroll 1
      for (int j = 0; j < RPW / 8; ++j) {  // eight rows, four lanes each
        if (!((wides >> (8 * j)) & 0xffu)) continue;
        const int w = 8 * j + (lane >> 2);  // the row's own lane
        const int64_t j0 = __shfl_sync(0xffffffffu, k0, w), j1 = __shfl_sync(0xffffffffu, k1, w);
        double t[QC], ta = 0.0;
#pragma unroll
        for (int q = 0; q < QC; ++q) t[q] = 0.0;
        if ((wides >> w) & 1u)
          resid_row(acol, asrc, aval, x, ld, q0, nq, norm, j0 + (lane & 3), j1, 4, t, ta);
        const bool back = wide && (lane >> 3) == j;
        const int from = 4 * (lane & 7);
#pragma unroll
        for (int q = -1; q < QC; ++q) {
          if (q < 0 ? !norm : q >= nq) continue;
          double v = q < 0 ? ta : t[q < 0 ? 0 : q];
          v += __shfl_xor_sync(0xffffffffu, v, 2);
          v += __shfl_xor_sync(0xffffffffu, v, 1);
          v = __shfl_sync(0xffffffffu, v, from);
          if (back) {
            if (q < 0) ra = v;
            else s[q < 0 ? 0 : q] = v;
          }
        }
      }
    }
    if (row_group) {
#pragma unroll
      for (int v = 0; v < NV; ++v) m[v] = 0;
    }
    if (ok) {
      m[0] = max(m[0], mag_bits(ra));
#pragma unroll
      for (int q = 0; q < QC; ++q) {
        if (q < nq) {
          const int64_t e = (int64_t)(q0 + q) * ld + i;
          const double bi = b[e], ri = bi - s[q];
          r[e] = ri;
          m[1 + 3 * q] = max(m[1 + 3 * q], mag_bits(x[e]));
          m[2 + 3 * q] = max(m[2 + 3 * q], mag_bits(bi));
          m[3 + 3 * q] = max(m[3 + 3 * q], mag_bits(ri));
        }
      }
    }
    if (!row_group) continue;
    // grouped maxima: a warp whose rows share one group reduces them and
    // makes one atomic per value; otherwise each row makes its own
    const int g = ok ? row_group[i] : -1;
    const int g0 = __shfl_sync(0xffffffffu, g, 0);
    if (__all_sync(0xffffffffu, g == g0 || g < 0)) {
      double* w = work + (int64_t)g0 * kResStride;  // g0 >= 0: the warp's first row exists
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        if (v == 0 ? !norm : (v - 1) / 3 >= nq) continue;
        const u64 k = warp_max(m[v]);
        if (lane == 0) atomic_max_pos(&w[v == 0 ? 0 : 3 * q0 + v], k);
      }
    } else if (ok) {
      double* w = work + (int64_t)g * kResStride;
#pragma unroll
      for (int v = 0; v < NV; ++v)
        if (v == 0 ? norm : (v - 1) / 3 < nq) atomic_max_pos(&w[v == 0 ? 0 : 3 * q0 + v], m[v]);
    }
  }
  if (row_group) return;
  // warp maxima -> block maxima in shared memory -> one atomic per value
  // and block (same-address atomics from every warp would serialise)
  __shared__ u64 red[256 / 32][NV];
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const u64 k = warp_max(m[v]);
    if (lane == 0) red[threadIdx.x >> 5][v] = k;
  }
  __syncthreads();
  if (threadIdx.x < NV) {
    const int v = threadIdx.x;
    u64 k = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) k = max(k, red[w][v]);
    if (v == 0 ? norm : (v - 1) / 3 < nq) atomic_max_pos(&work[v == 0 ? 0 : 3 * q0 + v], k);
  }
}

// out[q] = the largest scaled backward error of right-hand side q over the
// groups (one group when rows are not grouped), out[nrhs + q] = 0, or the
// groups' bwd_ratio flags where a NaN or Inf leaves a group without an error
__global__ void k_bwd_finish(const double* work, int nrhs, int ngroups, double* out) {
  __shared__ double red[256];
  for (int q = 0; q < nrhs; ++q) {
    double m = 0.0;
    int bad = 0;
    for (int g = threadIdx.x; g < ngroups; g += blockDim.x) {
      const double* w = work + (int64_t)g * kResStride;
      m = fmax(m, bwd_ratio(w[0], w[1 + 3 * q], w[2 + 3 * q], w[3 + 3 * q], bad));
    }
    red[threadIdx.x] = m;
    bad = (__syncthreads_or(bad & 1) ? 1 : 0) | (__syncthreads_or(bad & 2) ? 2 : 0);
    for (int h = blockDim.x / 2; h > 0; h >>= 1) {
      if ((int)threadIdx.x < h) red[threadIdx.x] = fmax(red[threadIdx.x], red[threadIdx.x + h]);
      __syncthreads();
    }
    if (threadIdx.x == 0) {
      out[q] = red[0];
      out[nrhs + q] = bad;
    }
    __syncthreads();
  }
}

__global__ void k_axpy(int64_t total, int n, int ld, double* x, const double* d,
                       const int* row_group, const unsigned char* active) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * blockDim.x) {
    int64_t q = e / n, i = e % n;
    if (active && !active[row_group[i]]) continue;
    x[q * ld + i] += d[q * ld + i];
  }
}

}  // namespace

template <typename T>
void launch_zero_fronts(FrontDesc<T>* fd, const int* fronts, int nf, int max_elems,
                        cudaStream_t s) {
  if (nf <= 0) return;
  // 16-byte stores: one thread per 8 elements (FP32) or 4 (FP64) per round
  const int per = 256 * (16 / (int)sizeof(T)) * 4;
  int gx = std::max(1, std::min((max_elems + per - 1) / per, 4 * 152));
  { k_zero_fronts<T><<<dim3(gx, nf), 256, 0, s>>>(fd, fronts); note_launches(1); }
}
template void launch_zero_fronts<double>(FrontDesc<double>*, const int*, int, int, cudaStream_t);
template void launch_zero_fronts<float>(FrontDesc<float>*, const int*, int, int, cudaStream_t);

// r = b - A x and the scaled backward error of each right-hand side, the
// largest over the row groups when row_group is given (work must hold
// 2 nrhs + max(ngroups, 1) * kResStride doubles; the result per rhs, see k_bwd_finish, is written to
// work[0 .. 2 nrhs), the groups' maxima follow).  nnz: entries of the full CSR.
void launch_resid_bwd_err(const int64_t* aptr, const int* acol, const int64_t* asrc,
                          const double* aval, int n, int64_t nnz, const double* x,
                          const double* b, double* r, int nrhs, int ld, double* work,
                          const int* row_group, int ngroups,
                          cudaStream_t s) {
  double* acc = work + 2 * nrhs;
  const int ng = row_group ? std::max(ngroups, 1) : 1;
  cudaMemsetAsync(acc, 0, (size_t)ng * kResStride * sizeof(double), s);
  const bool small = nnz <= (int64_t)kResShort * n;
  const int rows_per_block = small ? 256 : 64;
  const int bx = std::max(1, std::min((n + rows_per_block - 1) / rows_per_block, 4 * 152));
  const dim3 grid(bx, (nrhs + kResQC - 1) / kResQC);
  if (small)
    k_resid_norms<32><<<grid, 256, 0, s>>>(aptr, acol, asrc, aval, n, x, b, r, nrhs, ld, acc,
                                           row_group);
  else
    k_resid_norms<8><<<grid, 256, 0, s>>>(aptr, acol, asrc, aval, n, x, b, r, nrhs, ld, acc,
                                          row_group);
  note_launches(1);
  { k_bwd_finish<<<1, 256, 0, s>>>(acc, nrhs, ng, work); note_launches(1); }
}

// x += d; with a mask (active != nullptr) only on the rows whose group is
// active (the others' d was not solved for)
void launch_axpy(int n, int nrhs, int ld, double* x, const double* d, cudaStream_t s,
                 const int* row_group, const unsigned char* active) {
  int64_t total = (int64_t)n * nrhs;
  int blocks = (int)std::max<int64_t>(1, std::min<int64_t>((total + 255) / 256, 4096));
  { k_axpy<<<blocks, 256, 0, s>>>(total, n, ld, x, d, row_group, active); note_launches(1); }
}

}  // namespace ssids300

// FP64 FMA throughput probe: independent DFMA chains per thread, no memory
// traffic; used to state the FP64 roofline of the FP64 path (the driver's
// measured peaks cover HBM and bf16 tensor only).
namespace ssids300 {
namespace {
__global__ void k_dfma_probe(double* out, int iters, double seed) {
  double a0 = seed + threadIdx.x, a1 = a0 + 1, a2 = a0 + 2, a3 = a0 + 3;
  double a4 = a0 + 4, a5 = a0 + 5, a6 = a0 + 6, a7 = a0 + 7;
  const double m = 0.999999, c = 1e-7;
  for (int i = 0; i < iters; ++i) {
    a0 = fma(a0, m, c); a1 = fma(a1, m, c); a2 = fma(a2, m, c); a3 = fma(a3, m, c);
    a4 = fma(a4, m, c); a5 = fma(a5, m, c); a6 = fma(a6, m, c); a7 = fma(a7, m, c);
  }
  double s = a0 + a1 + a2 + a3 + a4 + a5 + a6 + a7;
  if (s == 12345.678) out[0] = s;  // keep the chains live
}
}  // namespace

double fp64_peak_tflops(int device) {
  cudaSetDevice(device);
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  double* out = nullptr;
  cudaMalloc(&out, sizeof(double));
  const int blocks = sms * 8, threads = 256, iters = 4096;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  k_dfma_probe<<<blocks, threads>>>(out, 64, 1.0);
  cudaEventRecord(e0);
  k_dfma_probe<<<blocks, threads>>>(out, iters, 1.0);
  cudaEventRecord(e1);
  cudaEventSynchronize(e1);
  float ms = 0;
  cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(out);
  double flops = 2.0 * 8.0 * (double)iters * blocks * threads;
  return ms > 0 ? flops / (ms * 1e-3) / 1e12 : 0.0;
}
}  // namespace ssids300
