// FP64 kernels of the CISS subspace steps on n x m complex128 blocks.
//
// The reference performs these on the host in complex64 with numpy/scipy
// (src/aospectrum/ciss.py:296-372): S @ probes, the moment axpys, the Gram
// matrix M^H S M, the basis transform, B^H H B, B^H S B and the residual
// norms.  Here they run on the device in FP64 so that the projected
// problems and the reported residuals carry FP64 accuracy.
#include "common.cuh"
#include "dmma.cuh"
#include "timing.h"

#include <algorithm>
#include <mutex>
#include <vector>

namespace aosb {
namespace {

// y = A x: one warp per row, lanes over 32 columns at a time.
__global__ void spmm_kernel(int64_t n, int ncols, const int64_t* __restrict__ indptr,
                            const int32_t* __restrict__ indices, const float2* __restrict__ vals,
                            const double2* __restrict__ x, int64_t ldx, double2* __restrict__ y,
                            int64_t ldy) {
  const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= n) return;
  const int64_t e0 = indptr[row], e1 = indptr[row + 1];
  for (int c0 = 0; c0 < ncols; c0 += 32) {
    const int c = c0 + lane;
    if (c >= ncols) break;
    double sr = 0.0, si = 0.0;
    for (int64_t e = e0; e < e1; ++e) {
      const float2 a = vals[e];
      const double2 v = x[(size_t)indices[e] * ldx + c];
      sr += (double)a.x * v.x - (double)a.y * v.y;
      si += (double)a.x * v.y + (double)a.y * v.x;
    }
    y[(size_t)row * ldy + c] = make_double2(sr, si);
  }
}

__global__ void moments_kernel(int64_t n, int L, int M, const double2* __restrict__ x,
                               const double2* __restrict__ coef, double2* __restrict__ mom) {
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= n * L) return;
  const int64_t j = idx / L;
  const int c = (int)(idx - j * L);
  const double2 v = x[idx];
  double2* row = mom + (size_t)j * L * M;
  for (int m = 0; m < M; ++m) {
    const double2 w = coef[m];
    double2 o = row[m * L + c];
    o.x += w.x * v.x - w.y * v.y;
    o.y += w.x * v.y + w.y * v.x;
    row[m * L + c] = o;
  }
}

// Partial Gram blocks: scratch[chunk][p][q] = sum over rows in chunk of
// conj(x[j][a]) y[j][b].  grid = (ceil(p / TILE), ceil(q / TILE), chunks).
//
// FP64 matrix instructions on fragments loaded straight from global memory
// (the eight columns of a fragment are one 128-byte line of a row; neighbouring
// warps share lines in L1).  TILE 32: a CTA's four warps own 16 x 16 blocks
// each over all rows of the chunk.  TILE 16, for grids that would leave SMs
// idle: the warps split the chunk's rows and add up in shared memory.  The
// SIMT form it replaces read five shared-memory words per four products: n =
// 13000, 128 x 128: 436 us, now 66 (floor 46 at 37 TFLOP/s); n = 1715, 96 x
// 96: 172, now 10.
constexpr int kGramRows = 512;

template <int TILE>
__global__ void __launch_bounds__(128) gram_partial_kernel(int64_t n, int p, int q,
                                                           const double2* __restrict__ x,
                                                           int64_t ldx,
                                                           const double2* __restrict__ y,
                                                           int64_t ldy,
                                                           double2* __restrict__ part) {
  constexpr bool kSplit = TILE == 16;  // warps split the rows
  __shared__ double2 sums[kSplit ? 4 : 1][16][17];
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int a0 = blockIdx.x * TILE + (kSplit ? 0 : warp / 2 * 16);
  const int b0 = blockIdx.y * TILE + (kSplit ? 0 : warp % 2 * 16);
  constexpr int kWarpRows = kSplit ? kGramRows / 4 : kGramRows;
  const int64_t r0 = (int64_t)blockIdx.z * kGramRows + (kSplit ? warp * kWarpRows : 0);
  const int64_t r1 = min(n, r0 + kWarpRows);
  const int col = lane / 4, row = lane % 4;
  const double2 zero = make_double2(0.0, 0.0);
  DBlock acc[2][2] = {};
  const bool va[2] = {a0 + col < p, a0 + 8 + col < p};
  const bool vb[2] = {b0 + col < q, b0 + 8 + col < q};
  constexpr int U = 4;  // steps of four rows in flight
  double2 fa[U][2], fb[U][2];
  auto load = [&](int u, int64_t r) {
    const bool in = r + row < r1;
    const double2* xr = x + (size_t)(r + row) * ldx + a0 + col;
    const double2* yr = y + (size_t)(r + row) * ldy + b0 + col;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      fa[u][h] = in && va[h] ? xr[8 * h] : zero;
      fb[u][h] = in && vb[h] ? yr[8 * h] : zero;
    }
  };
#pragma unroll
  for (int u = 0; u < U; ++u) load(u, r0 + 4 * u);
  for (int64_t r = r0; r < r1; r += 4 * U) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const double2 c = make_double2(fa[u][h].x, -fa[u][h].y);  // conj(x)
        zmma(acc[h][0], c, fb[u][0]);
        zmma(acc[h][1], c, fb[u][1]);
      }
      load(u, r + 4 * (U + u));
    }
  }
  double2* out = part + (size_t)blockIdx.z * p * q;
  const int orow = lane / 4, ocol = 2 * (lane % 4);
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int a = 8 * i + orow, b = 8 * j + ocol + e;
        const double2 v = make_double2(acc[i][j].re[e], acc[i][j].im[e]);
        if (kSplit)
          sums[warp][a][b] = v;
        else if (a0 + a < p && b0 + b < q)
          out[(size_t)(a0 + a) * q + b0 + b] = v;
      }
  if (!kSplit) return;
  __syncthreads();
  for (int e = threadIdx.x; e < 256; e += 128) {
    const int a = e / 16, b = e % 16;
    if (a0 + a >= p || b0 + b >= q) continue;
    double2 v = sums[0][a][b];
#pragma unroll
    for (int w = 1; w < (kSplit ? 4 : 1); ++w) {
      v.x += sums[w][a][b].x;
      v.y += sums[w][a][b].y;
    }
    out[(size_t)(a0 + a) * q + b0 + b] = v;
  }
}

// TILE 32 needs two CTAs a SM to fill it; below that the finer tiles do.
void launch_gram_partial(int64_t n, int p, int q, const double2* x, int64_t ldx, const double2* y,
                         int64_t ldy, double2* part, int chunks, cudaStream_t st) {
  const int64_t coarse = (int64_t)ceil_div(p, 32) * ceil_div(q, 32) * chunks;
  if (coarse >= 2 * 148) {
    dim3 grid(ceil_div(p, 32), ceil_div(q, 32), chunks);
    gram_partial_kernel<32><<<grid, 128, 0, st>>>(n, p, q, x, ldx, y, ldy, part);
  } else {
    dim3 grid(ceil_div(p, 16), ceil_div(q, 16), chunks);
    gram_partial_kernel<16><<<grid, 128, 0, st>>>(n, p, q, x, ldx, y, ldy, part);
  }
}

__global__ void gram_reduce_kernel(int chunks, int64_t pq, const double2* __restrict__ part,
                                   double2* __restrict__ g) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= pq) return;
  double sr = 0.0, si = 0.0;
  for (int c = 0; c < chunks; ++c) {
    const double2 v = part[(size_t)c * pq + i];
    sr += v.x;
    si += v.y;
  }
  g[i] = make_double2(sr, si);
}

// y (n x r) = x (n x p) t (p x r): a warp owns 16 rows x 32 columns, a CTA 64
// rows, on FP64 matrix instructions with fragments straight from global memory
// (t stays in L1 and L2).  n = 13000, p = 128, r = 104: 100 us with the former
// shared-memory form, now 59 (floor 37 at 37 TFLOP/s).  A launch takes the
// columns from `first` on, as many as the grid's y extent covers.
constexpr int kDenseColumns = 32;
__global__ void __launch_bounds__(128) dense_mul_kernel(int64_t n, int p, int r, int first,
                                                        const double2* __restrict__ x,
                                                        int64_t ldx,
                                                        const double2* __restrict__ t,
                                                        double2* __restrict__ y, int64_t ldy) {
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int64_t r0 = (int64_t)blockIdx.x * 64 + warp * 16;
  const int c0 = first + blockIdx.y * kDenseColumns;
  if (r0 >= n) return;
  const int hi = lane / 4, lo = lane % 4;
  const double2 zero = make_double2(0.0, 0.0);
  DBlock acc[2][4] = {};
  const bool vr[2] = {r0 + hi < n, r0 + 8 + hi < n};
  const double2* xr = x + (size_t)(r0 + hi) * ldx + lo;
  const double2* tr = t + (size_t)lo * r + c0 + hi;
  double2 fa[2][2], fb[2][4];
  auto load = [&](int buf, int k) {
    const bool in = k + lo < p;
#pragma unroll
    for (int i = 0; i < 2; ++i) fa[buf][i] = in && vr[i] ? xr[(size_t)8 * i * ldx + k] : zero;
#pragma unroll
    for (int j = 0; j < 4; ++j)
      fb[buf][j] = in && c0 + 8 * j + hi < r ? tr[(size_t)k * r + 8 * j] : zero;
  };
  load(0, 0);
  for (int k = 0; k < p; k += 8) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      load(h ^ 1, k + 4 * (h + 1));
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) zmma(acc[i][j], fa[h][i], fb[h][j]);
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    if (!vr[i]) continue;
    double2* out = y + (size_t)(r0 + 8 * i + hi) * ldy + c0;
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int c = 8 * j + 2 * lo + e;
        if (c0 + c < r) out[c] = make_double2(acc[i][j].re[e], acc[i][j].im[e]);
      }
  }
}

// out[j] = || a[:, j] - e[j] b[:, j] ||.  A cluster of kNormCtas CTAs takes
// eight columns (one 128-byte line of a row) and splits the rows; its first CTA
// adds the others' sums in rank order from their shared memory, so that the
// result does not depend on timing and needs no scratch.  One CTA per 32
// columns, as before, left all but a few SMs idle: n = 13000, 104 columns: 470
// us, now 35 (floor 7, 43 MB).
constexpr int kNormCtas = 8, kNormThreads = 256;

__global__ void __cluster_dims__(kNormCtas, 1, 1) __launch_bounds__(kNormThreads)
    column_norms_kernel(int64_t n, int m, const double2* __restrict__ a,
                        const double2* __restrict__ b, int64_t ld, const double* __restrict__ e,
                        double* __restrict__ out) {
  __shared__ double part[kNormThreads / 8][9];
  __shared__ double sum[8];
  const int rank = (int)blockIdx.x % kNormCtas;
  const int c = threadIdx.x % 8, rl = threadIdx.x / 8;
  const int j = (int)(blockIdx.x / kNormCtas) * 8 + c;
  double s = 0.0;
  if (j < m) {
    const double ej = e[j];
#pragma unroll 4
    for (int64_t i = (int64_t)rank * (kNormThreads / 8) + rl; i < n;
         i += kNormCtas * (kNormThreads / 8)) {
      const double2 av = a[(size_t)i * ld + j], bv = b[(size_t)i * ld + j];
      const double dr = av.x - ej * bv.x, di = av.y - ej * bv.y;
      s += dr * dr + di * di;
    }
  }
  part[rl][c] = s;
  __syncthreads();
  if (threadIdx.x < 8) {
    double t = 0.0;
    for (int q = 0; q < kNormThreads / 8; ++q) t += part[q][threadIdx.x];
    sum[threadIdx.x] = t;
  }
  __syncwarp();  // the aligned barrier wants the whole warp together
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::
                   : "memory");
  if (rank == 0 && threadIdx.x < 8 && j < m) {
    const uint32_t mine = (uint32_t)__cvta_generic_to_shared(&sum[threadIdx.x]);
    double t = 0.0;
    for (int q = 0; q < kNormCtas; ++q) {
      uint32_t peer;
      double v;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(mine), "r"(q));
      asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(peer) : "memory");
      t += v;
    }
    out[j] = sqrt(t);
  }
  // no CTA leaves while the first may still read its sums
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::
                   : "memory");
}

}  // namespace
}  // namespace aosb

extern "C" {

int aosb_spmm(int64_t n, int32_t ncols, const int64_t* indptr, const int32_t* indices,
              const aosb_complex64* values, const aosb_complex128* x, int64_t ldx,
              aosb_complex128* y, int64_t ldy, void* stream, char* err, size_t cap) {
  if (indptr == nullptr || indices == nullptr || values == nullptr || x == nullptr || y == nullptr)
    return aosb::set_error(err, cap, AOSB_ERR_NULL, "null argument");
  if (n <= 0 || ncols <= 0 || ldx < ncols || ldy < ncols)
    return aosb::set_error(err, cap, AOSB_ERR_ARGUMENT, "invalid spmm shape");
  cudaEvent_t ev[2];
  const bool timed = aosb::timing_begin((cudaStream_t)stream, ev);
  aosb::spmm_kernel<<<aosb::ceil_div(n, 8), 256, 0, (cudaStream_t)stream>>>(
      n, ncols, indptr, indices, (const float2*)values, (const double2*)x, ldx, (double2*)y, ldy);
  aosb::count_launches(1);
  if (timed) {
    // nnz of a pattern, read once per indptr array (timing runs only)
    static std::mutex mu;
    static std::vector<std::pair<const int64_t*, int64_t>> seen;
    int64_t nnz = -1;
    {
      std::lock_guard<std::mutex> lock(mu);
      for (auto& e : seen)
        if (e.first == indptr + n) nnz = e.second;
    }
    if (nnz < 0) {
      cudaMemcpy(&nnz, indptr + n, sizeof(int64_t), cudaMemcpyDeviceToHost);
      std::lock_guard<std::mutex> lock(mu);
      seen.emplace_back(indptr + n, nnz);
    }
    aosb::timing_end(aosb::kTimedSpmm, (cudaStream_t)stream, ev, 8.0 * nnz * ncols,
                     12.0 * nnz + (double)n * ncols * 32.0);
  }
  return aosb::launch_check(err, cap, "spmm");
}

int aosb_moments_accumulate(int64_t n, int32_t L, int32_t M, const aosb_complex128* x,
                            const aosb_complex128* coef, aosb_complex128* mom, void* stream,
                            char* err, size_t cap) {
  if (x == nullptr || coef == nullptr || mom == nullptr)
    return aosb::set_error(err, cap, AOSB_ERR_NULL, "null argument");
  if (n <= 0 || L <= 0 || M <= 0)
    return aosb::set_error(err, cap, AOSB_ERR_ARGUMENT, "invalid moment shape");
  aosb::moments_kernel<<<aosb::ceil_div(n * L, 256), 256, 0, (cudaStream_t)stream>>>(
      n, L, M, (const double2*)x, (const double2*)coef, (double2*)mom);
  aosb::count_launches(1);
  return aosb::launch_check(err, cap, "moments");
}

size_t aosb_gram_scratch_bytes(int64_t n, int32_t p, int32_t q) {
  if (n <= 0 || p <= 0 || q <= 0) return 0;
  const int64_t chunks = (n + aosb::kGramRows - 1) / aosb::kGramRows;
  return (size_t)chunks * (size_t)p * (size_t)q * sizeof(double2);
}

namespace aosb {
// The partial-sum grid is (ceil(p/32), ceil(q/32), ceil(n/512)); its y and z
// extents are limited to 65535, so n above 33,553,920 rows (or q above
// 2,097,120 columns) is rejected before anything is launched.
static int gram_grid_check(int64_t n, int32_t q, char* err, size_t cap) {
  const int64_t chunks = (n + kGramRows - 1) / kGramRows;
  if (chunks > 65535 || ceil_div((int64_t)q, 32) > 65535)
    return set_error(err, cap, AOSB_ERR_SIZE,
                     "gram: n=%lld rows in %lld chunks of %d (or q=%d) exceeds the launch grid "
                     "limit of 65535 chunks", (long long)n, (long long)chunks, kGramRows, q);
  return 0;
}
}  // namespace aosb

int aosb_gram(int64_t n, int32_t p, int32_t q, const aosb_complex128* x, int64_t ldx,
              const aosb_complex128* y, int64_t ldy, aosb_complex128* g, void* scratch,
              void* stream, char* err, size_t cap) {
  if (x == nullptr || y == nullptr || g == nullptr || scratch == nullptr)
    return aosb::set_error(err, cap, AOSB_ERR_NULL, "null argument");
  if (n <= 0 || p <= 0 || q <= 0 || ldx < p || ldy < q)
    return aosb::set_error(err, cap, AOSB_ERR_ARGUMENT, "invalid gram shape");
  if (int rc = aosb::gram_grid_check(n, q, err, cap)) return rc;
  const int chunks = (int)((n + aosb::kGramRows - 1) / aosb::kGramRows);
  cudaStream_t st = (cudaStream_t)stream;
  aosb::launch_gram_partial(n, p, q, (const double2*)x, ldx, (const double2*)y, ldy,
                            (double2*)scratch, chunks, st);
  const int64_t pq = (int64_t)p * q;
  aosb::gram_reduce_kernel<<<aosb::ceil_div(pq, 256), 256, 0, st>>>(
      chunks, pq, (const double2*)scratch, (double2*)g);
  aosb::count_launches(2);
  return aosb::launch_check(err, cap, "gram");
}

int aosb_dense_mul(int64_t n, int32_t p, int32_t r, const aosb_complex128* x, int64_t ldx,
                   const aosb_complex128* t, aosb_complex128* y, int64_t ldy, void* stream,
                   char* err, size_t cap) {
  if (x == nullptr || t == nullptr || y == nullptr)
    return aosb::set_error(err, cap, AOSB_ERR_NULL, "null argument");
  if (n <= 0 || p <= 0 || r <= 0 || ldx < p || ldy < r)
    return aosb::set_error(err, cap, AOSB_ERR_ARGUMENT, "invalid dense_mul shape");
  constexpr int kMost = 65535 * aosb::kDenseColumns;  // columns of a launch: the grid's y limit
  for (int64_t first = 0; first < r; first += kMost) {
    dim3 grid(aosb::ceil_div(n, 64),
              aosb::ceil_div(std::min<int64_t>(r - first, kMost), aosb::kDenseColumns));
    aosb::dense_mul_kernel<<<grid, 128, 0, (cudaStream_t)stream>>>(
        n, p, r, (int)first, (const double2*)x, ldx, (const double2*)t, (double2*)y, ldy);
    aosb::count_launches(1);
  }
  return aosb::launch_check(err, cap, "dense_mul");
}

int aosb_column_norms(int64_t n, int32_t m, const aosb_complex128* a, const aosb_complex128* b,
                      int64_t ld, const double* e, double* out, void* stream, char* err,
                      size_t cap) {
  if (a == nullptr || b == nullptr || e == nullptr || out == nullptr)
    return aosb::set_error(err, cap, AOSB_ERR_NULL, "null argument");
  if (n <= 0 || m <= 0 || ld < m)
    return aosb::set_error(err, cap, AOSB_ERR_ARGUMENT, "invalid norm shape");
  aosb::column_norms_kernel<<<aosb::kNormCtas * aosb::ceil_div(m, 8), aosb::kNormThreads, 0,
                              (cudaStream_t)stream>>>(
      n, m, (const double2*)a, (const double2*)b, ld, e, out);
  aosb::count_launches(1);
  return aosb::launch_check(err, cap, "column_norms");
}

// ---------------------------------------------------------------------------
// Gram product without any allocation, for callers that cannot allocate
// device memory at the point of the call: code running inside another
// framework's stream-ordered memory pool or under a memory cap that forbids
// new cudaMalloc, real-time or callback contexts where an allocation could
// block or deadlock, and embedders that must not grow the device heap after
// start-up.  The partial sums live in one file-scope device array of
// kNoAllocGramBytes (16 MiB); every GPU that loads this library's device
// code holds it until the process exits.
constexpr size_t kNoAllocGramBytes = (size_t)16 << 20;
static __device__ __align__(256) unsigned char g_noalloc_gram_scratch[kNoAllocGramBytes];

namespace {
constexpr int kMaxDevices = 64;
std::mutex g_noalloc_mu;
void* g_noalloc_ptr[kMaxDevices] = {};
}  // namespace

}  // namespace aosb

extern "C" int aosb_gram_noalloc(int64_t n, int32_t p, int32_t q, const aosb_complex128* x,
                                 int64_t ldx, const aosb_complex128* y, int64_t ldy,
                                 aosb_complex128* g, void* stream, char* err, size_t cap) {
  using namespace aosb;
  if (x == nullptr || y == nullptr || g == nullptr)
    return set_error(err, cap, AOSB_ERR_NULL, "null argument");
  if (n <= 0 || p <= 0 || q <= 0 || ldx < p || ldy < q)
    return set_error(err, cap, AOSB_ERR_ARGUMENT, "invalid gram shape");
  if (int rc = gram_grid_check(n, q, err, cap)) return rc;
  const size_t need = aosb_gram_scratch_bytes(n, p, q);
  if (need > kNoAllocGramBytes)
    return set_error(err, cap, AOSB_ERR_SIZE,
                     "aosb_gram_noalloc: n=%lld, p=%d, q=%d needs %zu bytes of partial sums, "
                     "more than its fixed %zu-byte scratch (ceil(n/512)*p*q*16 must not exceed "
                     "it); use aosb_gram with caller-provided scratch",
                     (long long)n, p, q, need, kNoAllocGramBytes);
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess)
    return set_error(err, cap, AOSB_ERR_CUDA, "cudaGetDevice failed: %s", cudaGetErrorString(e));
  if (dev < 0 || dev >= kMaxDevices)
    return set_error(err, cap, AOSB_ERR_UNSUPPORTED, "device index %d not supported", dev);
  void* scratch = nullptr;
  {
    // First call on a device: resolve the array's device address once, with
    // that device current (a synchronous runtime call; make this first call
    // before any stream capture).
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (g_noalloc_ptr[dev] == nullptr) {
      void* ptr = nullptr;
      e = cudaGetSymbolAddress(&ptr, g_noalloc_gram_scratch);
      if (e != cudaSuccess || ptr == nullptr)
        return set_error(err, cap, AOSB_ERR_CUDA, "cudaGetSymbolAddress failed: %s",
                         cudaGetErrorString(e));
      g_noalloc_ptr[dev] = ptr;
    }
    scratch = g_noalloc_ptr[dev];
  }
  // Nothing in the scratch needs clearing: the partial kernel writes every
  // element that the reduction then reads.
  const int chunks = (int)((n + kGramRows - 1) / kGramRows);
  cudaStream_t st = (cudaStream_t)stream;
  launch_gram_partial(n, p, q, (const double2*)x, ldx, (const double2*)y, ldy, (double2*)scratch,
                      chunks, st);
  const int64_t pq = (int64_t)p * q;
  gram_reduce_kernel<<<ceil_div(pq, 256), 256, 0, st>>>(chunks, pq, (const double2*)scratch,
                                                        (double2*)g);
  count_launches(2);
  return launch_check(err, cap, "gram_noalloc");
}
