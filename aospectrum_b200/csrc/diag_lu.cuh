// LU of one diagonal tile with partial pivoting inside the tile, and the
// inverses of both triangles, in place: the tile ends with inv(L) strictly
// below the diagonal and inv(U) on and above it (L unit lower).
//
// One CTA per pencil, so the kernel is a latency chain (128 pivots); the tile
// is held in registers and the pivots are taken off that chain:
//
//  * "data" warp w owns rows 8w .. 8w+7, lane l the columns l, l + 32, ...
//    Each 8-column block step b (columns k0 .. k0+7) is one sweep over the
//    whole tile that eliminates below the block and, in the rows above it,
//    back-substitutes: with L, U the factors of the pivoted block column and
//    Q = inv(L_bb) A_b (the block's rows),
//      rows below:  A_i -= L_ib Q        (all columns: right of the block this
//                                         is the trailing update, left of it
//                                         the rows of inv(L) in the making)
//      rows above:  A_i -= A_ib S        (columns right of the block, with
//                                         S = inv(U_bb) Q: these rows hold
//                                         inv(U_11) U_12 until their column's
//                                         turn comes)
//      the block:   Q left of it, S right of it
//      its columns: -A_ib inv(U_bb) above, -L_ib inv(L_bb) below, and
//                   inv(L_bb), inv(U_bb) in the block's own rows.
//    After the last block no further pass is needed for the inverses.
//  * T / 32 "panel" warps, one thread per row, work one block column ahead:
//    they bring the next block column up to date themselves, factor it while
//    the data warps apply the current block to the whole tile, and form Q
//    and S.  Rows are not interchanged while a block column is factored: a
//    row that was a pivot is only retired, and its place is taken when the
//    block is handed over.
//
// The chain that is left is 350-450 cycles a pivot (search, broadcast, one
// update; more beside busy data warps) and the hand-overs; at T = 128 the FP32 pipe in the update is about
// as long.  The former kernel kept the tile in shared memory (four loads per
// four FMAs in the inverses) with the panel in line: 283 us at T = 128, 88 us
// at T = 64 for up to one pencil per SM, against 100 us and 34 us here.
#pragma once

#include "common.cuh"

namespace aosb {

constexpr int kDiagBlock = 8;  // columns per block step, rows per data warp

template <int T>
struct DiagShape {
  static constexpr int kWarps = T / kDiagBlock;  // data warps
  static constexpr int kChunks = T / 32;         // columns per lane
  static constexpr int kPanel = T / 32;          // panel warps
  static constexpr int kThreads = (kWarps + kPanel) * 32;
};

template <int T>
struct DiagShared {
  // block column b in coef[b & 1]: above the block the back-substituted
  // columns, from the block down the pivoted L and U
  alignas(16) float2 coef[2][T][kDiagBlock];
  alignas(16) float2 q[kDiagBlock][T];    // the block's rows, then Q
  alignas(16) float2 s[kDiagBlock][T];    // S
  alignas(16) float2 old[kDiagBlock][T];  // rows that left the block
  alignas(16) float2 fin[T][kDiagBlock];  // final block columns
  // each panel warp's candidate row (then 1 / its pivot) and its key, by
  // column parity
  alignas(16) float2 row[2][DiagShape<T>::kPanel][kDiagBlock + 2];
  alignas(16) unsigned key[2][4];
  alignas(16) int tag[T];   // row whose content moves to this row in this block step
  alignas(16) int dest[T];  // the inverse map
  float2 dinv[2][kDiagBlock];  // 1 / u_jj
  int pivot[kDiagBlock];       // pivot rows of the block column
  int perm[T];                 // original row of each row
};

template <int T>
constexpr size_t diag_smem_bytes() {
  return sizeof(DiagShared<T>);
}

__device__ __forceinline__ void diag_bar_sync(int id, int threads) {
  __syncwarp();
  asm volatile("barrier.cta.sync.aligned %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void diag_bar_arrive(int id, int threads) {
  __syncwarp();
  asm volatile("barrier.cta.arrive.aligned %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// x -= a b.  REAL, here and below: the imaginary parts are zero and are neither
// computed nor read from or written to the factor (the same results to the bit;
// T = 64, beside the updates, 27 us against 32).
template <bool REAL>
__device__ __forceinline__ void csub(float2& x, float2 a, float2 b) {
  x.x = fmaf(-a.x, b.x, x.x);
  if (REAL) return;
  x.x = fmaf(a.y, b.y, x.x);
  x.y = fmaf(-a.x, b.y, x.y);
  x.y = fmaf(-a.y, b.x, x.y);
}

// 1 / a by scaling with a power of two to |a| about 1, so that |a|^2 neither
// overflows nor underflows, and one Newton step on the reciprocal of |a|^2.
// `m` = |re| + |im| > 0 and finite.  No branch, so it overlaps the search.
template <bool REAL>
__device__ __forceinline__ float2 crecip(float2 a, float m) {
  const unsigned e = min(max(__float_as_uint(m) >> 23, 1u), 253u);
  const float s = __uint_as_float((254u - e) << 23);
  const float x = a.x * s, y = REAL ? 0.0f : a.y * s;
  const float d = REAL ? x * x : fmaf(x, x, y * y);
  float r = __fdividef(1.0f, d);
  r = fmaf(r, fmaf(-d, r, 1.0f), r);
  return make_float2(x * r * s, REAL ? 0.0f : -y * r * s);
}
template <bool REAL>
__device__ __forceinline__ float2 times(float2 a, float2 b) {
  return REAL ? make_float2(a.x * b.x, 0.0f) : cmul(a, b);
}

// Panel warps, thread = row `row` holding x, its part of block column b:
// partial pivoting LU of the rows k0 .. T-1.  Returns a device status code of
// this row's pivot (0 = fine).
template <int T, bool REAL>
__device__ __forceinline__ int diag_panel(DiagShared<T>& sh, int b, int row,
                                          float2 (&x)[kDiagBlock], int barrier) {
  constexpr int NB = kDiagBlock, PW = DiagShape<T>::kPanel;
  const int k0 = b * NB, wi = row / 32, lane = row % 32;
  const int old_perm = sh.perm[row];
  bool active = row >= k0;
  int dest = row, bad = 0;
#pragma unroll
  for (int q = 0; q < NB; ++q) {
    const int buf = q & 1;
    // largest |re| + |im| of the column to 18 bits, lowest row among equals
    // (the low five bits of the key hold the lane); NaNs never win
    const float m = REAL ? fabsf(x[q].x) : fabsf(x[q].x) + fabsf(x[q].y);
    unsigned key = m >= 0.0f ? (__float_as_uint(m) & ~31u) + 32u : 32u;
    key = active ? key | (31 - lane) : 31 - lane;
    const unsigned best = __reduce_max_sync(0xffffffffu, key);
    // every thread inverts its own candidate while the search runs
    const float d = REAL ? x[q].x * x[q].x : x[q].x * x[q].x + x[q].y * x[q].y;
    const bool usable = d > 0.0f && d <= 3.402823466e38f;
    const float2 own = usable ? crecip<REAL>(x[q], m) : make_float2(1.0f, 0.0f);
    const bool mine = key == best;
    if (mine) {
      float2* to = sh.row[buf][wi];
#pragma unroll
      for (int c = 0; c < NB; c += 2)
        if (c + 1 > q)
          *reinterpret_cast<float4*>(&to[c]) = make_float4(x[c].x, x[c].y, x[c + 1].x, x[c + 1].y);
      to[NB] = own;
      sh.key[buf][wi] = best;
    }
    int win = 0;
    if (PW > 1) {
      diag_bar_sync(barrier, PW * 32);
      unsigned top = sh.key[buf][0] >> 5;
#pragma unroll
      for (int w = 1; w < PW; ++w) {
        const unsigned other = sh.key[buf][w] >> 5;
        if (other > top) { top = other; win = w; }
      }
    } else {
      __syncwarp();
    }
    const float2* from = sh.row[buf][win];
    const float2 inv = from[NB];
    float2 u[NB];
#pragma unroll
    for (int c = 0; c < NB; c += 2) {
      if (c + 1 <= q) continue;
      const float4 v = *reinterpret_cast<const float4*>(&from[c]);
      u[c] = make_float2(v.x, v.y);
      u[c + 1] = make_float2(v.z, v.w);
    }
    const bool pivot = mine && win == wi;
    active = active && !pivot;
    const float2 l = active ? times<REAL>(x[q], inv) : make_float2(0.0f, 0.0f);
#pragma unroll
    for (int c = q + 1; c < NB; ++c) csub<REAL>(x[c], l, u[c]);
    if (active) x[q] = l;
    if (pivot) {
      if (!usable) {
        bad = isfinite(d) ? kDevZeroPivot : kDevNonFinite;
        x[q] = make_float2(1.0f, 0.0f);
      }
      dest = k0 + q;
      sh.pivot[q] = row;
      sh.dinv[b & 1][q] = inv;
    }
  }
  // the block's rows that were no pivots take the places of the outside rows
  // that were
  if (PW > 1) diag_bar_sync(barrier, PW * 32);
  else __syncwarp();
  const bool displaced = active && row < k0 + NB;
  const unsigned who = __ballot_sync(0xffffffffu, displaced);
  if (displaced) {
    int rank = __popc(who & ((1u << lane) - 1));
#pragma unroll
    for (int q = 0; q < NB; ++q) {
      const int from = sh.pivot[q];
      if (from >= k0 + NB && rank-- == 0) dest = from;
    }
  }
#pragma unroll
  for (int c = 0; c < NB; c += 2)
    *reinterpret_cast<float4*>(&sh.coef[b & 1][dest][c]) =
        make_float4(x[c].x, x[c].y, x[c + 1].x, x[c + 1].y);
  sh.tag[dest] = row;
  sh.dest[row] = dest;
  sh.perm[dest] = old_perm;
  return bad;
}

// Panel warps, thread = row: its part of block column b + 1, which the data
// warps wrote into coef before the update of block b, brought up to date.
template <int T, bool REAL>
__device__ __forceinline__ void diag_next(DiagShared<T>& sh, int b, int row,
                                          float2 (&x)[kDiagBlock]) {
  constexpr int NB = kDiagBlock;
  const int k0 = b * NB, next = k0 + NB;
  const bool inside = row >= k0 && row < next;
  const float2(*src)[T] = row < next ? sh.s : sh.q;
  const float2* at = inside ? &sh.s[row - k0][next] : sh.coef[(b + 1) & 1][row];
#pragma unroll
  for (int c = 0; c < NB; c += 2) {
    const float4 v = *reinterpret_cast<const float4*>(&at[c]);
    x[c] = make_float2(v.x, v.y);
    x[c + 1] = make_float2(v.z, v.w);
  }
#pragma unroll
  for (int q = 0; q < NB; ++q) {
    float2 l = sh.coef[b & 1][row][q];
    if (inside) l = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int c = 0; c < NB; c += 2) {
      const float4 v = *reinterpret_cast<const float4*>(&src[q][next + c]);
      csub<REAL>(x[c], l, make_float2(v.x, v.y));
      csub<REAL>(x[c + 1], l, make_float2(v.z, v.w));
    }
  }
}

// Column c of the block's rows: Q = inv(L_bb) A_b in place, S = inv(U_bb) Q
// right of the block; both zero in the block's own columns.
template <int T, bool REAL>
__device__ __forceinline__ void diag_column(DiagShared<T>& sh, int b, int c) {
  constexpr int NB = kDiagBlock;
  const int k0 = b * NB;
  const float2(*lu)[NB] = &sh.coef[b & 1][k0];
  const float2 zero = make_float2(0.0f, 0.0f);
  float2 v[NB];
  if (c >= k0 && c < k0 + NB) {
#pragma unroll
    for (int j = 0; j < NB; ++j) sh.q[j][c] = sh.s[j][c] = zero;
    return;
  }
#pragma unroll
  for (int j = 0; j < NB; ++j) v[j] = sh.q[j][c];
#pragma unroll
  for (int q = 0; q < NB; ++q)
#pragma unroll
    for (int j = q + 1; j < NB; ++j) csub<REAL>(v[j], lu[j][q], v[q]);
#pragma unroll
  for (int j = 0; j < NB; ++j) sh.q[j][c] = v[j];
  if (c < k0) {
#pragma unroll
    for (int j = 0; j < NB; ++j) sh.s[j][c] = zero;
    return;
  }
#pragma unroll
  for (int q = NB - 1; q >= 0; --q) {
    v[q] = times<REAL>(v[q], sh.dinv[b & 1][q]);
#pragma unroll
    for (int j = 0; j < q; ++j) csub<REAL>(v[j], lu[j][q], v[q]);
  }
#pragma unroll
  for (int j = 0; j < NB; ++j) sh.s[j][c] = v[j];
}

// Row r of the block's final columns: -A_rb inv(U_bb) above the block,
// -L_rb inv(L_bb) below it, and in it the rows of inv(L_bb) and inv(U_bb).
template <int T, bool REAL>
__device__ __forceinline__ void diag_row(DiagShared<T>& sh, int b, int r) {
  constexpr int NB = kDiagBlock;
  const int k0 = b * NB, in = r - k0;  // 0 .. NB-1 inside the block
  const float2(*lu)[NB] = &sh.coef[b & 1][k0];
  const float2(*row) = sh.coef[b & 1][r];
  const bool inside = in >= 0 && in < NB;
  float2 v[NB];
  auto start = [&]() {
#pragma unroll
    for (int j = 0; j < NB; ++j)
      v[j] = inside ? make_float2(j == in ? 1.0f : 0.0f, 0.0f) : make_float2(-row[j].x, -row[j].y);
  };
  if (in < NB) {
    start();
#pragma unroll
    for (int q = 0; q < NB; ++q) {
      v[q] = times<REAL>(v[q], sh.dinv[b & 1][q]);
#pragma unroll
      for (int j = q + 1; j < NB; ++j) csub<REAL>(v[j], v[q], lu[q][j]);
    }
#pragma unroll
    for (int j = 0; j < NB; ++j) sh.fin[r][j] = v[j];
  }
  if (in >= 0) {
    start();
#pragma unroll
    for (int q = NB - 1; q > 0; --q)
#pragma unroll
      for (int j = 0; j < q; ++j) csub<REAL>(v[j], v[q], lu[q][j]);
#pragma unroll
    for (int j = 0; j < NB; ++j)
      if (j < in) sh.fin[r][j] = v[j];  // in the block: strictly left of the diagonal
  }
}

// Rank-8 update of the column chunks in MASK of a data warp's rows: the
// chunks of one call share the loads of the coefficients, which every lane
// needs (these loads and the FMAs are then about even).
template <int T, bool REAL, int MASK>
__device__ __forceinline__ void diag_rank8(float2 (&x)[kDiagBlock][T / 32],
                                           const float2 (*__restrict__ cf)[kDiagBlock],
                                           const float2 (*__restrict__ src)[T], int lane) {
  constexpr int NB = kDiagBlock, CH = T / 32;
#pragma unroll 1
  for (int q = 0; q < NB; q += 2) {
    float2 v[2][CH];
#pragma unroll
    for (int j = 0; j < CH; ++j)
      if (MASK >> j & 1) {
        v[0][j] = src[q][lane + 32 * j];
        v[1][j] = src[q + 1][lane + 32 * j];
      }
    // eight independent accumulators between the two uses of each one
    constexpr int G = CH == 4 ? 1 : CH == 2 ? 2 : 4;
#pragma unroll
    for (int r0 = 0; r0 < NB; r0 += G) {
      float4 a[G];
#pragma unroll
      for (int r = 0; r < G; ++r) a[r] = *reinterpret_cast<const float4*>(&cf[r0 + r][q]);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
#pragma unroll
        for (int r = 0; r < G; ++r)
#pragma unroll
          for (int j = 0; j < CH; ++j)
            if (MASK >> j & 1) {
              const float ar = h ? a[r].z : a[r].x;
              x[r0 + r][j].x = fmaf(-ar, v[h][j].x, x[r0 + r][j].x);
              if (REAL) continue;
              x[r0 + r][j].y = fmaf(-ar, v[h][j].y, x[r0 + r][j].y);
            }
#pragma unroll
        for (int r = 0; r < G; ++r)
#pragma unroll
          for (int j = 0; j < CH; ++j)
            if (!REAL && (MASK >> j & 1)) {
              const float ai = h ? a[r].w : a[r].y;
              x[r0 + r][j].x = fmaf(ai, v[h][j].y, x[r0 + r][j].x);
              x[r0 + r][j].y = fmaf(-ai, v[h][j].x, x[r0 + r][j].y);
            }
      }
    }
  }
}

// The masks a block step asks for: all chunks, or the last few.
template <int T, bool REAL>
__device__ __forceinline__ void diag_update(float2 (&x)[kDiagBlock][T / 32], int mask,
                                            const float2 (*cf)[kDiagBlock],
                                            const float2 (*src)[T], int lane) {
  switch (mask) {
    case 1: if (T == 32) diag_rank8<T, REAL, 1>(x, cf, src, lane); break;
    case 2: if (T == 64) diag_rank8<T, REAL, 2>(x, cf, src, lane); break;
    case 3: if (T == 64) diag_rank8<T, REAL, 3>(x, cf, src, lane); break;
    case 8: if (T == 128) diag_rank8<T, REAL, 8>(x, cf, src, lane); break;
    case 12: if (T == 128) diag_rank8<T, REAL, 12>(x, cf, src, lane); break;
    case 14: if (T == 128) diag_rank8<T, REAL, 14>(x, cf, src, lane); break;
    case 15: if (T == 128) diag_rank8<T, REAL, 15>(x, cf, src, lane); break;
  }
}

// `saved`, if given, keeps the real plane of pencil 0's tile as it was found:
// the Schur complement of everything eliminated before it (tile k at k T^2).
template <int T, bool REAL>
__global__ void __launch_bounds__(DiagShape<T>::kThreads, 1)
    diag_lu_kernel(int k, const int32_t* __restrict__ diag_slot, int64_t n_slots, int64_t n_pad,
                   float* __restrict__ factor, int32_t* __restrict__ pivots,
                   int32_t* __restrict__ status, float* __restrict__ saved) {
  constexpr int NB = kDiagBlock, W = DiagShape<T>::kWarps, CH = DiagShape<T>::kChunks;
  constexpr int kAll = DiagShape<T>::kThreads, kData = W * 32;
  // named barriers, in the order of a block step: block column factored, moved
  // rows written, next block column written, Q and S written, final columns
  // written (data warps); panel warps among themselves.  Between two arrivals
  // of one side at a barrier it waits for the other side, so no arrival can
  // count twice.
  constexpr int kBarFactored = 1, kBarMoved = 2, kBarColumn = 3, kBarRows = 4, kBarFinal = 5,
                kBarPanel = 6;
  extern __shared__ __align__(16) unsigned char diag_smem[];
  DiagShared<T>& sh = *reinterpret_cast<DiagShared<T>*>(diag_smem);
  const int p = blockIdx.x, warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  float* g = factor + ((size_t)p * (size_t)n_slots + (size_t)diag_slot[k]) * (size_t)(2 * T * T);
  if (warp >= W) {
    const int row = threadIdx.x - kData;
    float2 x[NB];
#pragma unroll
    for (int c = 0; c < NB; ++c) x[c] = make_float2(g[row * T + c], REAL ? 0.0f : g[row * T + c + T * T]);
    sh.perm[row] = row;
    int bad = 0;
    for (int b = 0; b < W; ++b) {
      const int found = diag_panel<T, REAL>(sh, b, row, x, kBarPanel);
      if (found != 0) bad = found;
      diag_bar_arrive(kBarFactored, kAll);
      diag_bar_sync(kBarMoved, kAll);
      diag_column<T, REAL>(sh, b, row);
      diag_bar_arrive(kBarRows, kAll);
      diag_bar_sync(kBarColumn, kAll);
      if (b + 1 < W) diag_next<T, REAL>(sh, b, row, x);
    }
    pivots[(size_t)p * n_pad + (size_t)k * T + row] = sh.perm[row];
    if (bad != 0) atomicCAS(&status[p], 0, bad);
    return;
  }
  const int row0 = warp * NB;
  float2 x[NB][CH];  // rows row0 + r, columns lane + 32 j
#pragma unroll
  for (int r = 0; r < NB; ++r)
#pragma unroll
    for (int j = 0; j < CH; ++j) {
      const int e = (row0 + r) * T + lane + 32 * j;
      x[r][j] = make_float2(g[e], REAL ? 0.0f : g[e + T * T]);
    }
  if (saved != nullptr && p == 0) {
#pragma unroll
    for (int r = 0; r < NB; ++r)
#pragma unroll
      for (int j = 0; j < CH; ++j)
        saved[(size_t)k * (T * T) + (row0 + r) * T + lane + 32 * j] = x[r][j].x;
  }
  for (int b = 0; b < W; ++b) {
    const int k0 = b * NB, next = k0 + NB;
    diag_bar_sync(kBarFactored, kAll);
    // the rows that the interchanges move, through shared memory
    if (warp >= b) {
      int to[NB];
      *reinterpret_cast<int4*>(to) = *reinterpret_cast<const int4*>(&sh.dest[row0]);
      *reinterpret_cast<int4*>(to + 4) = *reinterpret_cast<const int4*>(&sh.dest[row0 + 4]);
#pragma unroll
      for (int r = 0; r < NB; ++r) {
        const bool into = to[r] < next;
        if (into || warp == b) {
          float2* dst = into ? sh.q[to[r] - k0] : sh.old[r];
#pragma unroll
          for (int j = 0; j < CH; ++j) dst[lane + 32 * j] = x[r][j];
        }
      }
    }
    diag_bar_sync(kBarMoved, kAll);
    if (warp > b) {
      int from[NB];
      *reinterpret_cast<int4*>(from) = *reinterpret_cast<const int4*>(&sh.tag[row0]);
      *reinterpret_cast<int4*>(from + 4) = *reinterpret_cast<const int4*>(&sh.tag[row0 + 4]);
#pragma unroll
      for (int r = 0; r < NB; ++r) {
        if (from[r] < next) {
#pragma unroll
          for (int j = 0; j < CH; ++j) x[r][j] = sh.old[from[r] - k0][lane + 32 * j];
        }
      }
    }
#pragma unroll
    for (int j = 0; j < CH; ++j) {
      const int c = lane + 32 * j - next;
      if (c >= 0 && c < NB) {
#pragma unroll
        for (int r = 0; r < NB; ++r) sh.coef[(b + 1) & 1][row0 + r][c] = x[r][j];
      }
    }
    diag_bar_arrive(kBarColumn, kAll);
    diag_bar_sync(kBarRows, kAll);
    if (warp == b) {
#pragma unroll
      for (int j = 0; j < CH; ++j) {
        const int c = lane + 32 * j;
#pragma unroll
        for (int r = 0; r < NB; ++r) x[r][j] = c < k0 ? sh.q[r][c] : sh.s[r][c];
      }
    } else {
      // rows above the block change only right of it
      const int all = (1 << CH) - 1;
      diag_update<T, REAL>(x, warp > b ? all : all & ~((1 << (next / 32)) - 1), &sh.coef[b & 1][row0],
                     warp > b ? sh.q : sh.s, lane);
    }
    if (warp < CH) diag_row<T, REAL>(sh, b, threadIdx.x);
    diag_bar_sync(kBarFinal, kData);
#pragma unroll
    for (int j = 0; j < CH; ++j) {
      const int c = lane + 32 * j - k0;
      if (c >= 0 && c < NB) {
#pragma unroll
        for (int r = 0; r < NB; ++r) x[r][j] = sh.fin[row0 + r][c];
      }
    }
  }
#pragma unroll
  for (int r = 0; r < NB; ++r)
#pragma unroll
    for (int j = 0; j < CH; ++j) {
      const int e = (row0 + r) * T + lane + 32 * j;
      g[e] = x[r][j].x;
      if (!REAL) g[e + T * T] = x[r][j].y;
    }
}

}  // namespace aosb
