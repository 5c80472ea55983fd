// Numeric tile LU of shifted pencils A_p = H(k_p) - z_p S(k_p) (plain FP32).
//
// Storage: factor[p][slot][2][T][T] floats, real plane then imaginary
// plane, each row-major.  Right-looking over tile steps k:
//   1. diag_lu: LU of tile (k,k) with partial pivoting inside the tile,
//      then in-place inversion of both triangles; the slot keeps inv(L_kk)
//      strictly below the diagonal and inv(U_kk) on and above it.
//   2. panel:   L_ik = A_ik inv(U_kk)        (i > k, CTA owns row strips)
//               U_kj = inv(L_kk) P_k A_kj    (j > k, CTA owns column strips)
//   3. schur:   A_ij -= L_ik U_kj            for every (i, j) target.
// All kernels batch over pencils (grid.y / grid.x).
#include <atomic>
#include "plan.h"
#include "cgemm.cuh"
#include "diag_lu.cuh"
#include "factor.h"
#include "side_stream.h"

namespace aosb {
namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ size_t tile_base(int64_t p, int64_t n_slots, int64_t slot, int T) {
  return ((size_t)p * (size_t)n_slots + (size_t)slot) * (size_t)(2 * T * T);
}

// ---------------------------------------------------------------------------
// Assembly of H - z S into the tile storage (factor must be zeroed first).
__global__ void assemble_kernel(int64_t n, int64_t nnz, const int64_t* __restrict__ indptr,
                                const int32_t* __restrict__ indices,
                                const float2* __restrict__ hv, const float2* __restrict__ sv,
                                const int32_t* __restrict__ pencil_k,
                                const double2* __restrict__ shifts,
                                const int32_t* __restrict__ pinv, const int32_t* __restrict__ slot,
                                int64_t nb, int64_t n_slots, int T, float* __restrict__ factor) {
  const int64_t warp = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const int p = blockIdx.y;
  if (warp >= n) return;
  const int64_t r = warp;
  const int64_t kp = pencil_k[p];
  const double2 zd = shifts[p];
  const float2 z = make_float2((float)zd.x, (float)zd.y);
  const float2* h = hv + kp * nnz;
  const float2* s = sv != nullptr ? sv + kp * nnz : nullptr;
  const int pr = pinv[r];
  const int I = pr / T, rr = pr - I * T;
  for (int64_t e = indptr[r] + lane; e < indptr[r + 1]; e += 32) {
    const int pc = pinv[indices[e]];
    const int J = pc / T, cc = pc - J * T;
    const int sl = slot[(int64_t)I * nb + J];
    const float2 hval = h[e];
    const float2 sval = s != nullptr ? s[e] : make_float2(0.f, 0.f);
    const float re = hval.x - (z.x * sval.x - z.y * sval.y);
    const float im = hval.y - (z.x * sval.y + z.y * sval.x);
    const size_t b = tile_base(p, n_slots, sl, T) + (size_t)rr * T + cc;
    factor[b] = re;
    factor[b + (size_t)T * T] = im;
  }
}

// Padding rows and columns carry an identity diagonal.
__global__ void pad_identity_kernel(int64_t n_pad, const int32_t* __restrict__ perm,
                                    const int32_t* __restrict__ diag_slot, int64_t n_slots, int T,
                                    float* __restrict__ factor) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int p = blockIdx.y;
  if (i >= n_pad || perm[i] >= 0) return;
  const int k = (int)(i / T), r = (int)(i - (int64_t)k * T);
  factor[tile_base(p, n_slots, diag_slot[k], T) + (size_t)r * T + r] = 1.0f;
}

// ---------------------------------------------------------------------------
// Panel updates.  blockIdx.x enumerates (tile, strip); blockIdx.y = pencil.
// L strips are 32 rows x T columns, U strips are T rows x 32 columns.
template <int T>
struct PanelCfg {
  static constexpr int kStrip = 32;
  static constexpr int kStrips = T / kStrip;
  // micro tiles so that (rows / TM) * (cols / TN) == 256
  static constexpr int LTM = T == 128 ? 4 : 2, LTN = T == 32 ? 2 : 4;   // 32 x T
  static constexpr int UTM = T == 32 ? 2 : (T == 64 ? 2 : 4), UTN = T == 32 ? 2 : 4;  // T x 32
  static_assert((32 / LTM) * (T / LTN) == 256, "L panel layout");
  static_assert((T / UTM) * (32 / UTN) == 256, "U panel layout");
};

// REAL: the factor's imaginary planes are zero and stay so (real pencils).
template <int T, bool REAL>
__global__ void __launch_bounds__(kThreads) panel_kernel(int k, int nL, int nU,
                                                         const int32_t* __restrict__ lslot,
                                                         const int32_t* __restrict__ uslot,
                                                         const int32_t* __restrict__ diag_slot,
                                                         int64_t n_slots, int64_t n_pad,
                                                         float* __restrict__ factor,
                                                         const int32_t* __restrict__ pivots) {
  using C = PanelCfg<T>;
  constexpr int S = C::kStrip;
  constexpr size_t kRaw = 2 * (sizeof(CgemmSmem<S, T>) > sizeof(CgemmSmem<T, S>)
                                   ? sizeof(CgemmSmem<S, T>) : sizeof(CgemmSmem<T, S>));
  __shared__ __align__(16) unsigned char raw[kRaw];
  const int p = blockIdx.y;
  const int item = blockIdx.x / C::kStrips, strip = blockIdx.x % C::kStrips;
  const float* D = factor + tile_base(p, n_slots, diag_slot[k], T);
  if (item < nL) {
    // rows [strip*S, +S) of A_ik times inv(U_kk) (upper incl. diagonal)
    constexpr int TM = C::LTM, TN = C::LTN;
    auto& sm = *reinterpret_cast<CgemmSmem<S, T>(*)[2]>(raw);
    float* A = factor + tile_base(p, n_slots, lslot[item], T);
    float accr[TM][TN] = {}, acci[TM][TN] = {};
    const int r0 = strip * S;
    auto la = [&](int m, int q) {
      const size_t o = (size_t)(r0 + m) * T + q;
      return make_float2(A[o], REAL ? 0.f : A[o + T * T]);
    };
    auto lb = [&](int q, int c) {
      if (q > c) return make_float2(0.f, 0.f);
      const size_t o = (size_t)q * T + c;
      return make_float2(D[o], REAL ? 0.f : D[o + T * T]);
    };
    cgemm_cta<S, T, TM, TN, false, REAL>(accr, acci, T, sm, la, lb);
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const size_t o = (size_t)(r0 + cg_row<S, T, TM, TN>(i)) * T + cg_col<S, T, TM, TN>(j);
        A[o] = accr[i][j];
        if (!REAL) A[o + T * T] = acci[i][j];
      }
  } else if (item < nL + nU) {
    // columns [strip*S, +S) of inv(L_kk) (P_k A_kj)
    constexpr int TM = C::UTM, TN = C::UTN;
    auto& sm = *reinterpret_cast<CgemmSmem<T, S>(*)[2]>(raw);
    float* A = factor + tile_base(p, n_slots, uslot[item - nL], T);
    const int32_t* pv = pivots + (size_t)p * n_pad + (size_t)k * T;
    float accr[TM][TN] = {}, acci[TM][TN] = {};
    const int c0 = strip * S;
    auto la = [&](int r, int q) {
      if (q > r) return make_float2(0.f, 0.f);
      if (q == r) return make_float2(1.f, 0.f);
      const size_t o = (size_t)r * T + q;
      return make_float2(D[o], REAL ? 0.f : D[o + T * T]);
    };
    auto lb = [&](int q, int c) {
      const size_t o = (size_t)pv[q] * T + c0 + c;
      return make_float2(A[o], REAL ? 0.f : A[o + T * T]);
    };
    cgemm_cta<T, S, TM, TN, false, REAL>(accr, acci, T, sm, la, lb);
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const size_t o = (size_t)cg_row<T, S, TM, TN>(i) * T + c0 + cg_col<T, S, TM, TN>(j);
        A[o] = accr[i][j];
        if (!REAL) A[o + T * T] = acci[i][j];
      }
  }
}

// ---------------------------------------------------------------------------
// Schur update, word by word: blockIdx.x = (pair, sub-block), blockIdx.y =
// pencil.  For 32-wide tiles, and for factor storage that does not start on a
// 16-byte boundary.
template <int T>
struct SchurCfg {
  static constexpr int BM = T >= 64 ? 64 : 32;
  static constexpr int BN = T >= 64 ? 64 : 32;
  static constexpr int TM = T >= 64 ? 4 : 2;
  static constexpr int TN = T >= 64 ? 4 : 2;
  static constexpr int kSub = (T / BM) * (T / BN);
};

template <int T>
__global__ void __launch_bounds__(kThreads) schur_words_kernel(
    int nU, int first, const int32_t* __restrict__ lslot, const int32_t* __restrict__ uslot,
    const int32_t* __restrict__ tslot, int64_t n_slots, float* __restrict__ factor) {
  using C = SchurCfg<T>;
  constexpr int BM = C::BM, BN = C::BN, TM = C::TM, TN = C::TN;
  __shared__ CgemmSmem<BM, BN> sm[2];
  const int p = blockIdx.y;
  const int pair = first + blockIdx.x / C::kSub, sub = blockIdx.x % C::kSub;
  const int a = pair / nU, b = pair % nU;
  const int m0 = (sub / (T / BN)) * BM, n0 = (sub % (T / BN)) * BN;
  const float* L = factor + tile_base(p, n_slots, lslot[a], T);
  const float* U = factor + tile_base(p, n_slots, uslot[b], T);
  float* Cc = factor + tile_base(p, n_slots, tslot[pair], T);
  float accr[TM][TN] = {}, acci[TM][TN] = {};
  auto la = [&](int m, int q) {
    const size_t o = (size_t)(m0 + m) * T + q;
    return make_float2(L[o], L[o + T * T]);
  };
  auto lb = [&](int q, int c) {
    const size_t o = (size_t)q * T + n0 + c;
    return make_float2(U[o], U[o + T * T]);
  };
  cgemm_cta<BM, BN, TM, TN>(accr, acci, T, sm, la, lb);
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const size_t o = (size_t)(m0 + cg_row<BM, BN, TM, TN>(i)) * T + n0 + cg_col<BM, BN, TM, TN>(j);
      Cc[o] -= accr[i][j];
      Cc[o + T * T] -= acci[i][j];
    }
}

// Schur update of 64- and 128-wide tiles: blockIdx.x = (pair, 64 x 64 part),
// blockIdx.y = pencil.  128 threads own 8 x 4 complex elements each (rows 8
// apart), so a K step of four reads 24 16-byte words of shared memory for 512
// FMAs and issue is the bound (2304 CTAs: 2.9 instructions a cycle, FMA pipe
// 66 %); the operands come as they lie in the tiles by cp.async, two K slices of
// 16 deep, and four CTAs fit an SM.  The former 4 x 4 form with scalar words and slices staged through registers ran
// at a third of the FP32 rate: 8 pencils of the 343-atom cube (5 orbitals) 88
// us a step, now 72; 70 tiles of 64, one pencil: 71 us, now 59.
// Real pencils (the imaginary planes are zero and stay so) take a quarter of
// the FMAs on half the data, in slices of 32 deep, with the same results to the
// bit: 70 tiles of 64, one pencil, 19 us a step instead of 59.
constexpr int kSchurThreads = 128;
template <bool REAL>
struct SchurSlice {
  static constexpr int kPlanes = REAL ? 1 : 2, kDepth = REAL ? 32 : 16;
  float a[kPlanes][64][kDepth + 4];  // planes of L rows
  float b[kPlanes][kDepth][64];      // planes of U rows
};

__device__ __forceinline__ void copy16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}

template <int T, bool REAL>
__global__ void __launch_bounds__(kSchurThreads, 4) schur_kernel(
    int nU, int first, const int32_t* __restrict__ lslot, const int32_t* __restrict__ uslot,
    const int32_t* __restrict__ tslot, int64_t n_slots, float* __restrict__ factor) {
  using Slice = SchurSlice<REAL>;
  constexpr int kParts = T / 64, kDepth = Slice::kDepth, I = Slice::kPlanes - 1;
  __shared__ __align__(16) Slice sm[2];
  const int p = blockIdx.y;
  const int pair = first + blockIdx.x / (kParts * kParts), part = blockIdx.x % (kParts * kParts);
  const int m0 = part / kParts * 64, n0 = part % kParts * 64;
  const float* L = factor + tile_base(p, n_slots, lslot[pair / nU], T) + (size_t)m0 * T;
  const float* U = factor + tile_base(p, n_slots, uslot[pair % nU], T) + n0;
  const int tid = threadIdx.x, tr = tid / 16, tc = tid % 16 * 4;
  auto fetch = [&](int buf, int k0) {
#pragma unroll
    for (int plane = 0; plane < Slice::kPlanes; ++plane) {
#pragma unroll
      for (int e = tid; e < 64 * (kDepth / 4); e += kSchurThreads) {
        const int m = e / (kDepth / 4), k = e % (kDepth / 4) * 4;
        copy16(&sm[buf].a[plane][m][k], L + plane * T * T + m * T + k0 + k);
      }
#pragma unroll
      for (int e = tid; e < kDepth * 16; e += kSchurThreads) {
        const int k = e / 16, n = e % 16 * 4;
        copy16(&sm[buf].b[plane][k][n], U + plane * T * T + (k0 + k) * T + n);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float2 acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = make_float2(0.f, 0.f);
  fetch(0, 0);
  for (int k0 = 0; k0 < T; k0 += kDepth) {
    const int buf = k0 / kDepth & 1;
    if (k0 + kDepth < T) {
      fetch(buf ^ 1, k0 + kDepth);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    const Slice& s = sm[buf];
#pragma unroll
    for (int k = 0; k < kDepth; k += 4) {
      float4 br[4], bi[4];
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        br[h] = *reinterpret_cast<const float4*>(&s.b[0][k + h][tc]);
        if (!REAL) bi[h] = *reinterpret_cast<const float4*>(&s.b[I][k + h][tc]);
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float4 ar = *reinterpret_cast<const float4*>(&s.a[0][tr + 8 * i][k]);
        float4 ai;
        if (!REAL) ai = *reinterpret_cast<const float4*>(&s.a[I][tr + 8 * i][k]);
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          const float re = h == 0 ? ar.x : h == 1 ? ar.y : h == 2 ? ar.z : ar.w;
          const float xr[4] = {br[h].x, br[h].y, br[h].z, br[h].w};
          if (REAL) {
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j].x = fmaf(re, xr[j], acc[i][j].x);
            continue;
          }
          const float im = h == 0 ? ai.x : h == 1 ? ai.y : h == 2 ? ai.z : ai.w;
          const float xi[4] = {bi[h].x, bi[h].y, bi[h].z, bi[h].w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            acc[i][j].x = fmaf(re, xr[j], acc[i][j].x);
            acc[i][j].y = fmaf(re, xi[j], acc[i][j].y);
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            acc[i][j].x = fmaf(-im, xi[j], acc[i][j].x);
            acc[i][j].y = fmaf(im, xr[j], acc[i][j].y);
          }
        }
      }
    }
    __syncthreads();
  }
  float* C = factor + tile_base(p, n_slots, tslot[pair], T) + (size_t)m0 * T + n0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    float4* re = reinterpret_cast<float4*>(C + (tr + 8 * i) * T + tc);
    float4 r = *re;
    r.x -= acc[i][0].x; r.y -= acc[i][1].x; r.z -= acc[i][2].x; r.w -= acc[i][3].x;
    *re = r;
    if (REAL) continue;
    float4* im = re + T * T / 4;
    float4 m = *im;
    m.x -= acc[i][0].y; m.y -= acc[i][1].y; m.z -= acc[i][2].y; m.w -= acc[i][3].y;
    *im = m;
  }
}

// The targets first .. first + n - 1 of step k.
template <int T>
int launch_schur(const aosb_plan* P, const aosb_factor_args_v1* a, int64_t k, int nU, int64_t first,
                 int64_t n, bool real, char* err, size_t cap) {
  constexpr int parts = SchurCfg<T>::kSub;
  const int64_t blocks = n * parts;
  if (n == 0) return 0;
  if (blocks > INT32_MAX) return set_error(err, cap, AOSB_ERR_SIZE, "schur grid too large");
  const dim3 grid((unsigned)blocks, a->n_pencils);
  const int32_t *l = P->d_lb_slot + P->lb_off[k], *u = P->d_ur_slot + P->ur_off[k];
  const int32_t* t = P->d_sc_slot + P->sc_off[k];
  cudaStream_t st = (cudaStream_t)a->stream;
  count_launches(1);
  if constexpr (T >= 64) {
    if (((uintptr_t)a->factor & 15) == 0) {
      const auto kernel = real ? schur_kernel<T, true> : schur_kernel<T, false>;
      kernel<<<grid, kSchurThreads, 0, st>>>(nU, (int)first, l, u, t, P->n_slots, a->factor);
      return 0;
    }
  }
  schur_words_kernel<T><<<grid, kThreads, 0, st>>>(nU, (int)first, l, u, t, P->n_slots, a->factor);
  return 0;
}

template <int T>
int ensure_diag_attr(char* err, size_t cap) {
  // kernel attributes belong to each device's context: set once per device
  // (devices past 63 set it on every call)
  static std::atomic<uint64_t> attr_devices{0};
  int device = 0;
  cudaGetDevice(&device);
  const uint64_t dev_bit = device < 64 ? (uint64_t)1 << device : 0;
  if (dev_bit != 0 && (attr_devices.load() & dev_bit) != 0) return 0;
  const size_t diag_smem = diag_smem_bytes<T>();
  cudaError_t e = cudaFuncSetAttribute(
      diag_lu_kernel<T, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)diag_smem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(diag_lu_kernel<T, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)diag_smem);
  if (e != cudaSuccess)
    return set_error(err, cap, AOSB_ERR_CUDA, "diag_lu smem attribute: %s", cudaGetErrorString(e));
  attr_devices.fetch_or(dev_bit);
  return 0;
}

// Diagonal LU of step k (FP32 SIMT) on stream st.
template <int T>
void step_diag(const aosb_plan* P, const aosb_factor_args_v1* a, int64_t k, cudaStream_t st,
               bool real = false, float* diag_tiles = nullptr) {
  const auto kernel = real ? diag_lu_kernel<T, true> : diag_lu_kernel<T, false>;
  kernel<<<a->n_pencils, DiagShape<T>::kThreads, diag_smem_bytes<T>(), st>>>(
      (int)k, P->d_diag_slot, P->n_slots, P->n_pad, a->factor, a->pivots, a->status, diag_tiles);
  count_launches(1);
}

// Panel updates of step k (FP32 SIMT).
template <int T>
void step_panels(const aosb_plan* P, const aosb_factor_args_v1* a, int64_t k, bool real = false) {
  const int nL = P->lb_off[k + 1] - P->lb_off[k];
  const int nU = P->ur_off[k + 1] - P->ur_off[k];
  if (nL + nU == 0) return;
  dim3 grid((unsigned)((nL + nU) * PanelCfg<T>::kStrips), a->n_pencils);
  const auto kernel = real ? panel_kernel<T, true> : panel_kernel<T, false>;
  kernel<<<grid, kThreads, 0, (cudaStream_t)a->stream>>>(
      (int)k, nL, nU, P->d_lb_slot + P->lb_off[k], P->d_ur_slot + P->ur_off[k], P->d_diag_slot,
      P->n_slots, P->n_pad, a->factor, a->pivots);
  count_launches(1);
}

// The diagonal LU of step k + 1, one CTA per pencil and a chain of T pivots,
// needs only one target of step k: with lookahead that target comes first, and
// the LU runs on a high-priority side stream beside the other targets.  ms a
// factorization in line / beside: 70 tiles of 64, one real pencil 4.75 / 4.10;
// 27 tiles, 8 pencils 3.31 / 3.10, 64: 16.9 both; 44 tiles, 2 pencils 4.49 / 4.20.
// Updates of fewer than about two blocks an SM end before the events are through
// (10 tiles, one pencil 0.567 / 0.598; 13 tiles 0.734 / 0.785).
constexpr int64_t kLookaheadBlocks = 300;
template <int T>
int run_plain(const aosb_plan* P, const aosb_factor_args_v1* a, char* err, size_t cap, bool real,
              float* diag_tiles) {
  if (int rc = ensure_diag_attr<T>(err, cap)) return rc;
  cudaStream_t st = (cudaStream_t)a->stream;
  SideWork work;
  step_diag<T>(P, a, 0, st, real, diag_tiles);
  for (int64_t k = 0; k < P->nb; ++k) {
    step_panels<T>(P, a, k, real);
    const int nL = P->lb_off[k + 1] - P->lb_off[k];
    const int nU = P->ur_off[k + 1] - P->ur_off[k];
    const int64_t targets = (int64_t)nL * nU;
    const bool next = k + 1 < P->nb;
    if (!next || targets * SchurCfg<T>::kSub * a->n_pencils < kLookaheadBlocks) {
      if (int rc = launch_schur<T>(P, a, k, nU, 0, targets, real, err, cap)) return rc;
      if (next) step_diag<T>(P, a, k + 1, st, real, diag_tiles);
      continue;
    }
    if (work.stream == nullptr)
      if (int rc = work.open(st, kSideFactor, err, cap)) return rc;
    // the lists are in tile order, so tile (k + 1, k + 1) is the first target
    const bool leads = P->lb_tile[P->lb_off[k]] == k + 1 && P->ur_tile[P->ur_off[k]] == k + 1;
    const int64_t head = leads ? 1 : 0;
    if (int rc = launch_schur<T>(P, a, k, nU, 0, head, real, err, cap)) return rc;
    if (int rc = work.fork(err, cap)) return rc;
    step_diag<T>(P, a, k + 1, work.stream, real, diag_tiles);
    if (int rc = launch_schur<T>(P, a, k, nU, head, targets - head, real, err, cap)) return rc;
    if (int rc = work.join(err, cap)) return rc;
  }
  return launch_check(err, cap, "plain factorization");
}

// Diagonal LU and panel updates of step k.
template <int T>
int diag_and_panels(const aosb_plan* P, const aosb_factor_args_v1* a, int64_t k, char* err,
                    size_t cap) {
  if (int rc = ensure_diag_attr<T>(err, cap)) return rc;
  step_diag<T>(P, a, k, (cudaStream_t)a->stream);
  step_panels<T>(P, a, k);
  return 0;
}

}  // namespace

int factor_assemble(const aosb_plan* P, const aosb_factor_args_v1* a, char* err, size_t cap) {
  cudaStream_t st = (cudaStream_t)a->stream;
  const int np = a->n_pencils;
  const size_t bytes = (size_t)np * P->n_slots * 2 * P->T * P->T * sizeof(float);
  AOSB_CUDA_TRY(cudaMemsetAsync(a->factor, 0, bytes, st), err, cap);
  dim3 g1(ceil_div(P->n, 8), np);
  assemble_kernel<<<g1, 256, 0, st>>>(P->n, P->nnz, P->d_indptr, P->d_indices,
                                      (const float2*)a->h_values, (const float2*)a->s_values,
                                      a->pencil_k, (const double2*)a->shifts, P->d_pinv, P->d_slot,
                                      P->nb, P->n_slots, (int)P->T, a->factor);
  dim3 g2(ceil_div(P->n_pad, 256), np);
  pad_identity_kernel<<<g2, 256, 0, st>>>(P->n_pad, P->d_perm, P->d_diag_slot, P->n_slots,
                                          (int)P->T, a->factor);
  count_launches(2);
  return launch_check(err, cap, "assemble");
}

int factor_step_panels(const aosb_plan* P, const aosb_factor_args_v1* a, int k, char* err,
                       size_t cap) {
  switch (P->T) {
    case 32: return diag_and_panels<32>(P, a, k, err, cap);
    case 64: return diag_and_panels<64>(P, a, k, err, cap);
    case 128: return diag_and_panels<128>(P, a, k, err, cap);
  }
  return set_error(err, cap, AOSB_ERR_UNSUPPORTED, "unsupported tile size");
}

int factor_step_diag(const aosb_plan* P, const aosb_factor_args_v1* a, int k, cudaStream_t st,
                     char* err, size_t cap) {
  if (P->T != 128) return set_error(err, cap, AOSB_ERR_UNSUPPORTED, "diagonal step needs tile 128");
  if (int rc = ensure_diag_attr<128>(err, cap)) return rc;
  diag_lu_kernel<128, false><<<a->n_pencils, DiagShape<128>::kThreads, diag_smem_bytes<128>(), st>>>(
      k, P->d_diag_slot, P->n_slots, P->n_pad, a->factor, a->pivots, a->status, nullptr);
  count_launches(1);
  return 0;
}

int factor_plain(const aosb_plan* P, const aosb_factor_args_v1* a, char* err, size_t cap, bool real,
                 float* diag_tiles) {
  switch (P->T) {
    case 32: return run_plain<32>(P, a, err, cap, real, diag_tiles);
    case 64: return run_plain<64>(P, a, err, cap, real, diag_tiles);
    case 128: return run_plain<128>(P, a, err, cap, real, diag_tiles);
  }
  return set_error(err, cap, AOSB_ERR_UNSUPPORTED, "unsupported tile size");
}

}  // namespace aosb

extern "C" {

size_t aosb_factor_bytes(const aosb_plan_t* p, int32_t n_pencils) {
  if (p == nullptr || n_pencils <= 0) return 0;
  return (size_t)n_pencils * (size_t)p->n_slots * (size_t)(2 * p->T * p->T) * sizeof(float);
}

int aosb_factor(const aosb_plan_t* plan, const aosb_factor_args_v1* a, char* err, size_t cap) {
  using aosb::set_error;
  if (plan == nullptr || a == nullptr) return set_error(err, cap, AOSB_ERR_NULL, "null argument");
  if (a->abi_version != AOSPECTRUM_B200_ABI_VERSION || a->struct_size != sizeof(*a))
    return set_error(err, cap, AOSB_ERR_ABI, "factor args ABI mismatch");
  if (a->n_pencils <= 0 || a->n_pencils > 65535)
    return set_error(err, cap, AOSB_ERR_BATCH, "n_pencils must be in 1..65535");
  if (a->h_values == nullptr || a->pencil_k == nullptr ||
      a->shifts == nullptr || a->factor == nullptr || a->pivots == nullptr || a->status == nullptr)
    return set_error(err, cap, AOSB_ERR_NULL, "required pointer is null");
  if (!plan->uploaded)
    return set_error(err, cap, AOSB_ERR_ARGUMENT, "call aosb_plan_upload first");
  int rc = aosb::factor_assemble(plan, a, err, cap);
  if (rc) return rc;
  if (a->precision == AOSB_PRECISION_PLAIN) return aosb::factor_plain(plan, a, err, cap);
  if (a->precision == AOSB_PRECISION_BF16X3 || a->precision == AOSB_PRECISION_BF16X3_FP32_PANELS ||
      a->precision == AOSB_PRECISION_BF16X3_ONE_STEP)
    return aosb::factor_tc(plan, a, err, cap);
  return set_error(err, cap, AOSB_ERR_ARGUMENT, "unknown precision %d", a->precision);
}

}  // extern "C"
