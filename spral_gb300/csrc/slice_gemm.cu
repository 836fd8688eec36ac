// FP64 trailing updates on the tensor cores, by error-free slicing.
//
//   C(r, c) -= sum_k A(r, k) B(c, k),   r >= c,   everything FP64
//
// with A = L21 and B = L21 D of a front (the contribution block).  GB300 issues
// about 1.06 TF/s of FP64 multiply-adds, and 1900 TF/s of FP16 on the tensor
// cores; the update is therefore formed from exact FP16 products (the
// splitting of Ozaki, Ogita, Oishi and Rump, "Error-free transformations of
// matrix multiplication", Numer. Algorithms 59, 2012, in the form with a
// common exponent per row that Mukunoki, Ozaki, Ogita and Imamura, "DGEMM
// using tensor cores", ISC 2020, use on FP16 tensor cores):
//
//   * every row of A and of B is scaled by a power of two so that its
//     largest entry lies in [1/2, 1), truncated to a 62-bit integer and cut
//     into kSlices = 8 balanced base-256 digits in [-128, 128], each exact in
//     FP16.  Entries within a factor 2^9 of the row's largest keep all 53
//     bits, smaller ones what is left of the 62;
//   * the digit products of equal weight (levels l = 0..7 of the two digits'
//     indices) are summed by tcgen05.mma in FP32 accumulators in TMEM.  A
//     product is at most 2^14 and a level has at most 8 of them per column,
//     so the sums over 128 columns stay within 2^24: every accumulation is
//     exact, whatever its order;
//   * every chunk is added to 64-bit integers, and the total becomes one FP64
//     number, rounded once, that is subtracted from C.
//
// What is lost are the bits past the 62nd and the products below level 7,
// about 2^-62 sqrt(K) of (row maximum of A) x (row maximum of B) in all; an
// FP64 accumulation over K columns loses about 2^-54 sqrt(K) of the size of
// its partial sums.  (Seven digits, 2^-55, were up to three times less exact
// than FP64 on rows whose entries spread over e^6.)  Columns are balanced before
// that: column k of A is multiplied by 2^h and column k of B divided by it, 2^h
// ~ sqrt|D_k| (slice_balance), so both rows are those of L sqrt|D| and the loss
// follows a diagonal scaling of the matrix, exactly for 1x1 pivots; the two
// columns of a 2x2 pivot without diagonal entries share a scale.  The loss
// goes by the size of two rows of L sqrt|D|, as the error bound of a
// factorisation does, and lies below that bound; a C(r, c) far smaller than
// both keeps fewer bits than multiply-adds would leave it.  The result of an
// entry depends on nothing but its two rows, so a front gives the same bits
// alone and in a batch.
//
// Bound: 36 FP16 products of 16 columns per tile (128 x 64, so that the eight
// level accumulators fit the 512 TMEM columns) at 6 KiB of shared-memory
// operands per 32 cycles of the tensor pipe, then the integer drain of the
// accumulators.  A block of 3000 rows and 1024 columns: 8.24 ms (1.12 TF/s)
// with multiply-adds, 0.44 ms (20.8 TF/s) in slices; 48^3 Laplacian, all
// contribution blocks of a factorisation: 50.8 -> 3.9 ms.
#include <cstdint>
#include <algorithm>
#include <climits>
#include <cstring>
#include <new>
#include <vector>

#include "spral_ssids_gpu.h"
#include "slices.cuh"
#include "ssids_gpu.cuh"
#include "tcgen05.cuh"

namespace ssids300 {

namespace {

constexpr int SL_M = 128, SL_N = 64, SL_K = 32;  // tile rows, columns, columns per stage
constexpr int SL_CHUNK = 4;                      // stages per exact FP32 accumulation (128 columns)
static_assert(kSlices * SL_CHUNK * SL_K <= 1024, "a level's sum of products must stay within 2^24");
static_assert(SL_M == 2 * SL_N, "tiles of a trapezoid");
constexpr int SL_A_SLICE = SL_M * SL_K * 2;      // 8 KiB
constexpr int SL_B_SLICE = SL_N * SL_K * 2;      // 4 KiB
constexpr int SL_A_BYTES = kSlices * SL_A_SLICE;  // 64 KiB per stage
constexpr int SL_B_BYTES = kSlices * SL_B_SLICE;  // 32 KiB per stage
constexpr int SL_STAGES = 2;
constexpr int SL_EPI_THREADS = 512;
constexpr int SL_THREADS = 64 + SL_EPI_THREADS;
constexpr int SL_PART = SL_N / 4;                // columns of a tile per epilogue warp
static_assert(kSlices * SL_N <= 512 && SL_PART == 16, "TMEM columns");

__host__ __device__ constexpr int pad_to(int x, int p) { return (x + p - 1) / p * p; }

}  // namespace

// ---------------------------------------------------------------------------
// The geometry of every job, from the fronts' states in device memory (the
// elimination counts are known only there), and the first
// tile of each job.  One CTA.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(1024) k_slice_plan(SliceJob* jobs, int njobs, int* tile0,
                                                     const FrontDesc<double>* fds,
                                                     const FrontState* sts) {
  __shared__ int wsum[32];
  __shared__ int base;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) base = 0;
  __syncthreads();
  for (int j0 = 0; j0 < njobs; j0 += blockDim.x) {
    const int i = j0 + threadIdx.x;
    int tiles = 0;
    if (i < njobs) {
      SliceJob j = jobs[i];
      if (j.kind != kSliceGiven) {
        const FrontDesc<double> fd = fds[j.front];
        const FrontState st = sts[j.front];
        j.D = fd.D;
        j.lda = fd.ld;
        j.dlast = st.nelim;
        j.K = max(0, min(st.nelim - j.k0, j.kcap));
        j.A = fd.L + (int64_t)j.k0 * fd.ld + fd.n;
        j.B = fd.LD + (int64_t)j.k0 * fd.cm;
        j.ldb = fd.cm;
        j.C = fd.C;
        j.ldc = fd.ldc;
        j.M = j.N = fd.cm;
        // the buffers were sized for at most mcap rows and ncap columns
        if (j.M > j.mcap || j.N > j.ncap || j.M <= 0 || j.N <= 0) j.K = 0;
        jobs[i] = j;
      }
      tiles = j.K > 0 ? trapezoid_tiles<SL_N>(j.M, j.N) : 0;
    }
    int incl = tiles;
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    if (warp == 0) {
      int w = wsum[lane];
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += v;
      }
      wsum[lane] = w;
    }
    __syncthreads();
    const int before = base + (warp ? wsum[warp - 1] : 0) + incl - tiles;
    if (i < njobs) tile0[i] = before;
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) base = before + tiles;
    __syncthreads();
  }
  if (threadIdx.x == 0) tile0[njobs] = base;
}

// ---------------------------------------------------------------------------
// Slices of the operands: one CTA per 32 rows of A (blockIdx.y = 0) or of B
// (1) of a job.  A first pass over the rows finds their largest exponents, a
// second (from L2) writes the digits.  Layout, per block of 128 (A) or 64 (B)
// rows and 32-column stage one contiguous piece, which the GEMM loads with
// one bulk copy: [slice][8-column group][row][8 columns], i.e. 128-byte core
// matrices of 8 rows x 16 bytes, rows adjacent.  Rows and columns past the
// operand are zero.  Integer instructions only: an FP64 instruction issues
// some 70 times slower.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_slice(const SliceJob* jobs) {
  const SliceJob& j = jobs[blockIdx.z];
  const bool isb = blockIdx.y != 0;
  const int K = j.K;
  if (K <= 0) return;
  const int rows = isb ? j.N : j.M, pad = isb ? SL_N : SL_M;
  const int row0 = blockIdx.x * 32;
  if (row0 >= pad_to(rows, pad)) return;
  const double* src = isb ? j.B : j.A;
  const int ld = isb ? j.ldb : j.lda;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __shared__ short hs[kSliceMaxK];
  __shared__ int emax[8][32];
  for (int k = threadIdx.x; k < K; k += 256) {
    const int h = j.D ? slice_balance(j.D, j.k0 + k, j.dlast) : 0;
    hs[k] = (short)(isb ? -h : h);
  }
  __syncthreads();
  const int r = row0 + lane;
  const bool valid = r < rows;
  const double* col = src + (valid ? r : 0);
  int em = INT_MIN;
  constexpr int U = 8;
  for (int k0 = warp; k0 < K; k0 += 8 * U) {
    unsigned long long b[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = k0 + 8 * u;
      b[u] = (valid && k < K) ? (unsigned long long)__double_as_longlong(col[(int64_t)k * ld]) : 0ULL;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = k0 + 8 * u;
      if ((b[u] << 1) != 0ULL) em = max(em, slice_exponent(b[u], hs[k]));
    }
  }
  emax[warp][lane] = em;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < 8; ++w) em = max(em, emax[w][lane]);
  if (em == INT_MIN) em = 0;
  if (warp == 0) (isb ? j.eB : j.eA)[r] = em;
  const int nkt = (K + SL_K - 1) / SL_K;
  const int64_t piece = isb ? SL_B_BYTES : SL_A_BYTES;
  char* dst = (isb ? j.sB : j.sA) + (int64_t)(row0 / pad) * nkt * piece +
              (row0 % pad + lane) * 16;
  for (int o = warp; o < 4 * nkt; o += 8) {
    const int k0 = 8 * o;
    unsigned long long b[8];
#pragma unroll
    for (int q = 0; q < 8; ++q)
      b[q] = (valid && k0 + q < K)
                 ? (unsigned long long)__double_as_longlong(col[(int64_t)(k0 + q) * ld])
                 : 0ULL;
    int e[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) e[q] = slice_exponent(b[q], k0 + q < K ? hs[k0 + q] : 0);
    slice_store(b, e, em, dst + (int64_t)(o >> 2) * piece + (o & 3) * (pad * 16),
                pad * SL_K * 2);
  }
}

namespace {

// contiguous global -> shared copy (16-byte aligned, multiple of 16 bytes)
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes,
                                          uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
          "r"(smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

// shared-memory matrix descriptor, K-major without swizzle: core matrices
// of 8 rows x 16 bytes, `lead` bytes apart along K, 128 along the rows
__device__ __forceinline__ uint64_t smem_desc_plain(uint32_t saddr, uint32_t lead) {
  return (uint64_t)((saddr >> 4) & 0x3FFF) | ((uint64_t)(lead >> 4) << 16) |
         ((uint64_t)(128 >> 4) << 32) | ((uint64_t)1 << 46);
}

// D = F32, A = B = F16, both K-major, N = SL_N, M = SL_M
constexpr uint32_t kIdescF16 = (1u << 4) | ((uint32_t)(SL_N >> 3) << 17) | ((uint32_t)(SL_M >> 4) << 24);

}  // namespace

// ---------------------------------------------------------------------------
// Persistent kernel, one CTA per SM:
//   warp 0 lane 0   bulk copies of the tile's stages (8 slices of A, 8 of B)
//                   into a ring of two
//   warp 1 lane 0   tcgen05.mma: 36 slice products per stage, summed by level
//                   into eight TMEM accumulators
//   warps 2..17     every chunk, the eight accumulators into 64-bit integers
//                   (levels 0..3 and 4..7), after the last one C
// The next tile's products run while this tile's C is updated.  The drain is
// bound by the latency of the TMEM loads: sixteen warps of 16 columns each
// (eight of 32: 10,000 cycles a chunk beside 17,000 of products).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(SL_THREADS, 1)
    k_slice_gemm(const SliceJob* jobs, const int* tile0, int njobs, int* status) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  unsigned char* sA = smem;
  unsigned char* sB = smem + SL_STAGES * SL_A_BYTES;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + SL_STAGES * (SL_A_BYTES + SL_B_BYTES));
  uint64_t* empty = full + SL_STAGES;
  uint64_t* accf = empty + SL_STAGES;  // the accumulators hold a finished chunk
  uint64_t* acce = accf + 1;           // they have been read
  uint64_t* drain = acce + 1;          // all MMAs of this CTA have completed
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
  int* s_abort = reinterpret_cast<int*>(tmem_slot + 1);
  int* s_issued = s_abort + 1;

  const int ntiles = tile0[njobs];
  if ((int)blockIdx.x >= ntiles) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < SL_STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    mbar_init(accf, 1);
    mbar_init(acce, SL_EPI_THREADS);
    mbar_init(drain, 1);
    *s_abort = 0;
    *s_issued = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(512u));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = *tmem_slot;
  volatile int* abort_flag = s_abort;
  // the job of tile t: the last one that starts at or before it and is not empty
  auto job_of = [&](int t) {
    int lo = 0, hi = njobs;  // tile0[lo] <= t < tile0[hi]
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (tile0[mid] <= t) lo = mid;
      else hi = mid;
    }
    return lo;
  };

  if (warp == 0) {
    if (lane == 0) {
      // ---- producer ----
      uint32_t it = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x) {
        const int ji = job_of(t);
        const SliceJob& j = jobs[ji];
        int ti, tj;
        trapezoid_tile<SL_N>(t - tile0[ji], j.N, ti, tj);
        const int nkt = (j.K + SL_K - 1) / SL_K;
        const char* a = j.sA + (int64_t)ti * nkt * SL_A_BYTES;
        const char* b = j.sB + (int64_t)tj * nkt * SL_B_BYTES;
        for (int kt = 0; kt < nkt; ++kt, ++it) {
          const uint32_t s = it % SL_STAGES;
          if (it >= (uint32_t)SL_STAGES &&
              !mbar_wait(&empty[s], ((it / SL_STAGES) - 1) & 1, abort_flag)) {
            ok = false;
            break;
          }
          mbar_expect_tx(&full[s], SL_A_BYTES + SL_B_BYTES);
          bulk_load(sA + s * SL_A_BYTES, a + (int64_t)kt * SL_A_BYTES, SL_A_BYTES, &full[s]);
          bulk_load(sB + s * SL_B_BYTES, b + (int64_t)kt * SL_B_BYTES, SL_B_BYTES, &full[s]);
        }
      }
      *s_issued = (int)it;
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // ---- MMA issuer ----
      uint32_t it = 0, ch = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x) {
        const int nkt = (jobs[job_of(t)].K + SL_K - 1) / SL_K;
        for (int k0 = 0; k0 < nkt && ok; k0 += SL_CHUNK, ++ch) {
          if (ch >= 1 && !mbar_wait(acce, (ch - 1) & 1, abort_flag)) { ok = false; break; }
          asm volatile("tcgen05.fence::after_thread_sync;");
          const int k1 = min(nkt, k0 + SL_CHUNK);
          for (int kt = k0; kt < k1; ++kt, ++it) {
            const uint32_t s = it % SL_STAGES;
            if (!mbar_wait(&full[s], (it / SL_STAGES) & 1, abort_flag)) { ok = false; break; }
            asm volatile("tcgen05.fence::after_thread_sync;");
            const uint32_t a0 = smem_u32(sA + s * SL_A_BYTES), b0 = smem_u32(sB + s * SL_B_BYTES);
#pragma unroll
            for (int l = 0; l < kSlices; ++l) {
#pragma unroll
              for (int i = 0; i <= l; ++i) {
#pragma unroll
                for (int kk = 0; kk < SL_K / 16; ++kk) {
                  const uint64_t ad =
                      smem_desc_plain(a0 + i * SL_A_SLICE + kk * 2 * (SL_M * 16), SL_M * 16);
                  const uint64_t bd =
                      smem_desc_plain(b0 + (l - i) * SL_B_SLICE + kk * 2 * (SL_N * 16), SL_N * 16);
                  const uint32_t acc = (kt > k0 || i > 0 || kk > 0) ? 1u : 0u;
                  asm volatile(
                      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(
                          tmem + l * SL_N),
                      "l"(ad), "l"(bd), "r"(kIdescF16), "r"(acc));
                }
              }
            }
            mma_commit(&empty[s]);
          }
          if (ok) mma_commit(accf);
        }
      }
      // every MMA issued above has completed once `drain` flips
      mma_commit(drain);
      (void)mbar_wait_plain(drain, 0);
    }
  } else {
    // ---- drain and C ----
    // warp w reads TMEM lane quarter w % 4 and owns the column quarter
    // (w - 2) / 4: one row and 16 columns of the tile per thread
    const int q = warp & 3;
    const int part = (warp - 2) >> 2;
    uint32_t ch = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x) {
      const int ji = job_of(t);
      const SliceJob& j = jobs[ji];
      int ti, tj;
      trapezoid_tile<SL_N>(t - tile0[ji], j.N, ti, tj);
      const int nkt = (j.K + SL_K - 1) / SL_K;
      long long H[SL_PART], L[SL_PART];
#pragma unroll
      for (int c = 0; c < SL_PART; ++c) H[c] = L[c] = 0;
      for (int k0 = 0; k0 < nkt; k0 += SL_CHUNK, ++ch) {
        // the TMEM loads below are warp-collective: decide as a warp
        const bool got = mbar_wait(accf, ch & 1, abort_flag);
        if (!__all_sync(0xffffffffu, got)) { *abort_flag = 1; ok = false; break; }
        asm volatile("tcgen05.fence::after_thread_sync;");
        const uint32_t tbase = tmem + ((uint32_t)(q * 32) << 16) + part * SL_PART;
#pragma unroll
        for (int l = 0; l < kSlices; ++l) {
          const int w = 1 << (8 * (3 - l % 4));
          uint32_t v[16];
          tmem_ld16(tbase + (uint32_t)(l * SL_N), v);
#pragma unroll
          for (int c = 0; c < SL_PART; ++c) {
            const long long p = (long long)__float2int_rn(__uint_as_float(v[c])) * w;
            if (l < 4) H[c] += p;
            else L[c] += p;
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;");
        mbar_arrive(acce);
      }
      if (!ok) break;
      const int r = ti * SL_M + q * 32 + lane;
      if (r >= j.M) continue;
      const int col0 = tj * SL_N + part * SL_PART;
      const int er = j.eA[r];
      const int* eb = j.eB + col0;
      const int64_t ldc = j.ldc;
      double* crow = j.C + r + col0 * ldc;
      const int N = j.N;
      // 4 columns at a time: all loads in flight before the stores
#pragma unroll
      for (int cb = 0; cb < SL_PART; cb += 4) {
        double cv[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const int cc = col0 + cb + c;
          cv[c] = (cc < N && r >= cc) ? crow[(cb + c) * ldc] : 0.0;
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const int cc = col0 + cb + c;
          if (cc < N && r >= cc) {
            const int ec = eb[cb + c];
            double p = fixed_to_double(H[cb + c], L[cb + c], slice_product_exponent(er, ec));
            if (max(er, ec) >= kSliceNonFinite / 2) p = __longlong_as_double(0x7ff8000000000000LL);
            crow[(cb + c) * ldc] = cv[c] - p;
          }
        }
      }
    }
  }
  __syncthreads();
  if (*abort_flag) {
    if (threadIdx.x == 0) {
      atomicExch(status, kDevBadState);
      // let the copies still in flight land before shared memory is released
      const int issued = *s_issued;
      for (int it = max(0, issued - SL_STAGES); it < issued; ++it)
        (void)mbar_wait_plain(&full[it % SL_STAGES], (it / SL_STAGES) & 1);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
static size_t up256(size_t b) { return (b + 255) & ~size_t(255); }

size_t slice_job_bytes(int mcap, int ncap, int kcap) {
  const size_t nkt = (kcap + SL_K - 1) / SL_K;
  const size_t ra = pad_to(mcap, SL_M), rb = pad_to(ncap, SL_N);
  return up256(ra * nkt * SL_K * 2 * kSlices) + up256(rb * nkt * SL_K * 2 * kSlices) +
         up256(ra * sizeof(int)) + up256(rb * sizeof(int));
}

void slice_job_place(SliceJob& j, char* base) {
  const size_t nkt = (j.kcap + SL_K - 1) / SL_K;
  const size_t ra = pad_to(j.mcap, SL_M), rb = pad_to(j.ncap, SL_N);
  j.sA = base;
  j.sB = j.sA + up256(ra * nkt * SL_K * 2 * kSlices);
  j.eA = reinterpret_cast<int*>(j.sB + up256(rb * nkt * SL_K * 2 * kSlices));
  j.eB = reinterpret_cast<int*>(reinterpret_cast<char*>(j.eA) + up256(ra * sizeof(int)));
}

size_t slice_table_bytes(int njobs) {
  return up256((size_t)njobs * sizeof(SliceJob)) + up256((size_t)(njobs + 1) * sizeof(int));
}

constexpr size_t kSliceSmem =
    1024 + (size_t)SL_STAGES * (SL_A_BYTES + SL_B_BYTES) + (2 * SL_STAGES + 3) * 8 + 16;

int launch_slice_gemm(void* table, const std::vector<SliceJob>& jobs, size_t first, size_t count,
                      const FrontDesc<double>* fds, const FrontState* sts, int* status,
                      cudaStream_t s) {
  if (count == 0) return 0;
  SliceJob* dj = static_cast<SliceJob*>(table);
  int* tile0 = reinterpret_cast<int*>(static_cast<char*>(table) + up256(count * sizeof(SliceJob)));
  int rows = 0;
  long long tiles = 0;
  for (size_t i = first; i < first + count; ++i) {
    rows = std::max(rows, std::max(pad_to(jobs[i].mcap, SL_M), pad_to(jobs[i].ncap, SL_N)));
    tiles += trapezoid_tiles<SL_N>(jobs[i].mcap, jobs[i].ncap);
  }
  int dev = 0, nsm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return -3;
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  if (cudaFuncSetAttribute(k_slice_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)kSliceSmem) != cudaSuccess)
    return -3;
  k_slice_plan<<<1, 1024, 0, s>>>(dj, (int)count, tile0, fds, sts);
  k_slice<<<dim3(rows / 32, 2, (unsigned)count), 256, 0, s>>>(dj);
  const int grid = (int)std::min<long long>(tiles, std::max(nsm, 1));
  k_slice_gemm<<<grid, SL_THREADS, kSliceSmem, s>>>(dj, tile0, (int)count, status);
  note_launches(3);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

}  // namespace ssids300

// ---------------------------------------------------------------------------
// Stand-alone entry point: C -= A B^T on the lower trapezoid (r >= c), device
// pointers, column-major FP64.
// ---------------------------------------------------------------------------
extern "C" int spral_ssids_gpu_slice_gemm_f64(int M, int N, int K, const double* A, int lda,
                                              const double* B, int ldb, double* C, int ldc,
                                              int reps, void* stream) try {
  using namespace ssids300;
  if (M < 0 || N < 0 || K < 0 || N > M || lda < M || ldb < N || ldc < M || reps < 1) return -1;
  if (M == 0 || N == 0 || K == 0) return 0;
  if (!A || !B || !C) return -1;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int kc = std::min(K, kSliceMaxK);
  std::vector<SliceJob> jobs;
  for (int k0 = 0; k0 < K; k0 += kc) {
    SliceJob j{};
    j.kind = kSliceGiven;
    j.mcap = j.M = M;
    j.ncap = j.N = N;
    j.kcap = kc;
    j.K = std::min(kc, K - k0);
    j.A = A + (int64_t)k0 * lda;
    j.B = B + (int64_t)k0 * ldb;
    j.C = C;
    j.lda = lda; j.ldb = ldb; j.ldc = ldc;
    jobs.push_back(j);
  }
  const size_t tb = slice_table_bytes(1), sb = slice_job_bytes(M, N, kc);
  char* base = nullptr;
  if (cudaMalloc(&base, jobs.size() * tb + sb + 256) != cudaSuccess) {
    cudaGetLastError();
    return -50;
  }
  int* status = reinterpret_cast<int*>(base);
  char* tab = base + 256;
  int rc = 0, hs = 0;
  if (cudaMemsetAsync(status, 0, sizeof(int), s) != cudaSuccess) rc = -51;
  for (size_t i = 0; i < jobs.size() && rc == 0; ++i) {
    slice_job_place(jobs[i], tab + jobs.size() * tb);
    if (cudaMemcpyAsync(tab + i * tb, &jobs[i], sizeof(SliceJob), cudaMemcpyHostToDevice, s) !=
        cudaSuccess)
      rc = -51;
  }
  for (int r = 0; r < reps && rc == 0; ++r)
    for (size_t i = 0; i < jobs.size() && rc == 0; ++i)
      if (launch_slice_gemm(tab + i * tb, jobs, i, 1, nullptr, nullptr, status, s) != 0) rc = -51;
  if (cudaMemcpyAsync(&hs, status, sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess) {
    cudaGetLastError();
    rc = -51;
  }
  if (rc == 0 && hs != 0) rc = -52;
  cudaFree(base);
  return rc;
} catch (std::bad_alloc const&) {
  return -50;
}
