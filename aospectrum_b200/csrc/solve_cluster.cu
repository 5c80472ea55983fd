// Block-RHS triangular solves (tile 128, tensor cores), one launch for a whole
// solve: a cluster of C CTAs takes one unit of work -- one pencil and one strip
// of up to 32 right-hand sides -- through all steps of both sweeps.
//
// With one launch per diagonal step and one per update a solve is bound by the
// chain of 4 nb launches (8-20 us each: launch, TMEM and barrier set-up, a few
// dependent slabs, drain), not by the factor it reads.  Here the units never
// wait for one another, a cluster's CTAs meet twice a step through mbarriers
// in each other's shared memory, and the factor streams through a TMA ring that
// runs ahead of the steps.
//
// Step k (forward, then backward over the steps; op = the sweep's triangle or
// its conjugate transpose):
//   1. every CTA reads X_k (all rows) and forms its 128 / C rows of
//      Y = op(D_kk) X_k in FP32, D_kk the stored triangle inverse;
//   2. the rows go to every CTA of the cluster as the B operand of the update,
//      split in BF16 (x = hi + lo) and written into the peers' shared memory in
//      fragment order: 16 bytes hold two rows of one column;
//   3. X_k = Y, and X_i -= op(F) Y for the step's tiles, cut into units of 32
//      rows dealt out over the CTAs.  Four warps take a 32 KB unit (16 rows and
//      half of K each; the halves are added through shared memory): A fragments
//      of mma.sync.m16n8k16 are read from the FP32 tile and split in registers,
//      three products per real product (hi hi + hi lo + lo hi), FP32
//      accumulation; -acc is added to X in L2 (one red.add per element and
//      step, so the result does not depend on timing).
// The legacy tensor path suits this: with 32 columns a tile needs 3.2 us of it
// per SM and 3.0 us of the SM's share of HBM, and its operands need no pass
// through shared memory in the tensor core's layout.  A warp owns all columns
// of its rows so that the split of A, the larger part of the other
// instructions, is done once.  What bounds the update is the latency of these
// instructions (a scheduler with two such warps issues every third cycle), so
// twelve warps share the work, as many as 128 registers allow: 64 pencils of
// 102 tile steps, 32 columns, take 119 us a step against 128 with eight warps
// that hold all of K, 8 pencils 30.3 against 32.0.  Sixteen warps at 96
// registers spill (122 to 167), a split by columns repeats the split of A (140),
// and a deeper ring (five units), an earlier release of its slots or slots of
// 8 KB gain nothing (124, 126, 137).
//
// All waits are bounded: a wait that gives up sets AOSB_ERR_TIMEOUT for the
// pencil, the CTA leaves its loops, waits for its own copies in flight and
// meets the cluster at its end.
#include "plan.h"
#include "solve_cluster.h"
#include "tc_common.cuh"

#include <algorithm>
#include <atomic>
#include <mutex>

namespace aosb {
namespace {

using namespace tc;

constexpr int kT = 128;
constexpr int kStrip = 32;                             // right-hand sides per cluster
constexpr int kUnitRows = 32;                          // X rows of an update unit
constexpr int kParts = kT / kUnitRows;                 // units of a tile
constexpr int kUnitPlane = kUnitRows * kT * 4;         // bytes of one plane of a unit
constexpr uint32_t kUnitBytes = 2 * kUnitPlane;        // 32 KB
constexpr int kBox = 32 * 32 * 4;                      // one TMA box
constexpr int kGroups = 3;                             // groups of four warps
constexpr int kWarps = 4 * kGroups, kConsumers = kWarps * 32;
constexpr int kDiagWarps = 8;                          // warps of the diagonal product
constexpr int kThreads = kConsumers + 32;              // + the producer warp: 13, four a scheduler
// Units in the ring.  Entry g of the ring lies in slot g % kStages but counts
// on full barrier g % kFull: a group waits only for its own entries, and with
// 16 barriers it can never be a phase behind or ahead of one.
constexpr int kStages = 4, kFull = 16;
// Pitch of a row pair of Y (32 columns of 16 bytes): the four pairs of a
// fragment then start 32 bytes apart modulo 128, so eight lanes' 16-byte loads
// cover all banks once.
constexpr int kYPitch = kStrip * 16 + 32;

struct Sweep {
  const int32_t* off;   // [nb + 1]
  const int32_t* tile;  // X tile of each list entry
  const int32_t* slot;  // its factor tile
};

struct Args {
  Sweep forward, backward;
  const int32_t* diag_slot;
  int nb, nrhs, strips;
  int64_t n_pad, n_slots;
  int cluster;  // CTAs per cluster
  const float* factor;
  const int32_t* pivots;
  float2* work;
  int32_t* status;
  int wide;  // X rows can be read and added to 16 bytes at a time
  long long limit;
};

// The first D CTAs of a cluster share the diagonal product.
template <int D>
struct Shape {
  static constexpr int kRows = kT / D;               // rows of Y per CTA
  static constexpr int kTR = kRows >= 16 ? 4 : 2;    // rows per thread in the diagonal product
  static constexpr int kRowGroups = kRows / (4 * kTR);
  static constexpr int kSlices = kDiagWarps / kRowGroups;  // warps that share K
  // ring entries that hold the CTA's rows of D: 32 rows each
  static constexpr int kDUnits = kRows > kUnitRows ? kRows / kUnitRows : 1;
};

struct Shared {
  alignas(1024) unsigned char ring[kStages][kUnitBytes];
  alignas(128) unsigned char y[kT / 2 * kYPitch];
  // X_k, then the partial products of the diagonal step [slice][row][column]
  alignas(128) float2 x[kT][kStrip];
  int order[kT];       // row interchanges of the step (conjugate backward sweep)
  int tile[kFull];     // X tile of a ring entry
  uint64_t full[kFull], empty[kStages];
  uint64_t bar_y, bar_x;  // every CTA of the cluster has written Y / updated X
  int failed;
};
constexpr size_t kSmem = sizeof(Shared) + 1024;
static_assert(kSmem <= 232448, "shared memory budget");
static_assert(Shape<16>::kSlices * Shape<16>::kRows <= kT, "partials fit X_k");

__device__ __forceinline__ uint32_t peer_address(uint32_t addr, int cta) {
  uint32_t out;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(out) : "r"(addr), "r"(cta));
  return out;
}
__device__ __forceinline__ void peer_store16(uint32_t addr, uint32_t a, uint32_t b, uint32_t c,
                                             uint32_t d) {
  asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b),
               "r"(c), "r"(d)
               : "memory");
}
// All of this thread block's writes (ordered before by a barrier) are visible
// to whoever acquires the peer's barrier.
__device__ __forceinline__ void peer_arrive(uint32_t addr) {
  asm volatile(
      "fence.acq_rel.cluster;\n\t"
      "mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(addr)
      : "memory");
}
__device__ __forceinline__ bool cluster_wait(uint64_t* bar, uint32_t parity, long long limit) {
  const uint32_t addr = smem_u32(bar);
  for (long long it = 0; it < limit; ++it) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(addr), "r"(parity)
        : "memory");
    if (done) return true;
    if (it > 4096) __nanosleep(64);
  }
  return false;
}
__device__ __forceinline__ void cluster_meet() {
  __syncwarp();  // the aligned forms want the whole warp together
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::
                   : "memory");
}
// Barrier of the consumer warps; true when any of them passes true.
__device__ __forceinline__ bool consumers_any(bool v) {
  int out;
  __syncwarp();
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %1, 0;\n\t"
      "barrier.cta.red.or.pred.aligned q, 1, %2, p;\n\t"
      "selp.b32 %0, 1, 0, q;\n\t}"
      : "=r"(out)
      : "r"((int)v), "n"(kConsumers)
      : "memory");
  return out != 0;
}

__device__ __forceinline__ void pair_sync(int id) {
  __syncwarp();
  asm volatile("barrier.cta.sync.aligned %0, 64;" ::"r"(id) : "memory");
}

// Two floats as BF16 pairs, x = hi + lo.
__device__ __forceinline__ void split2(float x0, float x1, uint32_t& hi, uint32_t& lo) {
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(hi) : "f"(x1), "f"(x0));
  const float r0 = x0 - __uint_as_float(hi << 16), r1 = x1 - __uint_as_float(hi & 0xffff0000u);
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(lo) : "f"(r1), "f"(r0));
}

__device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0,
                                    uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// acc = op(F) Y for the 16 rows m16 .. m16 + 15 of a unit, one half of K and NB
// blocks of eight columns.  `order` (conjugate backward sweep): row r of Y
// belongs to row order[r] of F.
template <bool ADJ, bool ORDER, int NB>
__device__ __forceinline__ void unit_product(const unsigned char* slab, const unsigned char* y,
                                             const int* order, int m16, int khalf, int lane,
                                             float (&re)[4][4], float (&im)[4][4]) {
  const int fg = lane / 4, ft = lane % 4;  // fragment row (column of B), k pair
#pragma unroll 2
  for (int kb = khalf * (kT / 32); kb < (khalf + 1) * (kT / 32); ++kb) {
    uint32_t arh[4], arl[4], aih[4], ail[4];
#pragma unroll
    for (int f = 0; f < 4; ++f) {
      // fragment f: rows fg (+ 8 for odd f), k = 2 ft (+ 8 for f >= 2)
      const int m = m16 + fg + 8 * (f & 1), k = kb * 16 + 2 * ft + 8 * (f >> 1);
      float r0, r1, i0, i1;
      if (!ADJ) {
        const unsigned char* b =
            slab + (k >> 5) * kBox + m * 128 + ((((k & 31) >> 2) ^ (m & 7)) << 4) + (k & 3) * 4;
        const float2 vr = *reinterpret_cast<const float2*>(b);
        const float2 vi = *reinterpret_cast<const float2*>(b + kUnitPlane);
        r0 = vr.x; r1 = vr.y; i0 = vi.x; i1 = vi.y;
      } else {
        const int k0 = ORDER ? order[k] : k, k1 = ORDER ? order[k + 1] : k + 1;
        const unsigned char* b = slab + (m & 3) * 4;
        const unsigned char* b0 = b + k0 * 128 + (((m >> 2) ^ (k0 & 7)) << 4);
        const unsigned char* b1 = b + k1 * 128 + (((m >> 2) ^ (k1 & 7)) << 4);
        r0 = *reinterpret_cast<const float*>(b0);
        r1 = *reinterpret_cast<const float*>(b1);
        i0 = *reinterpret_cast<const float*>(b0 + kUnitPlane);
        i1 = *reinterpret_cast<const float*>(b1 + kUnitPlane);
      }
      split2(r0, r1, arh[f], arl[f]);
      split2(i0, i1, aih[f], ail[f]);
    }
    // plain: re -= Fi Yi, im += Fi Yr; conjugate: re += Fi Yi, im -= Fi Yr
    uint32_t nih[4], nil[4];
#pragma unroll
    for (int f = 0; f < 4; ++f) {
      nih[f] = aih[f] ^ 0x80008000u;
      nil[f] = ail[f] ^ 0x80008000u;
    }
    // two blocks of columns at a time: four accumulators in turn
#pragma unroll
    for (int b = 0; b < NB; b += 2) {
      const bool two = b + 1 < NB;
      const int c = two ? b + 1 : b;
      uint4 y0[2], y1[2];  // (re_hi, re_lo, im_hi, im_lo) of k pairs ft and ft + 4
#pragma unroll
      for (int h = 0; h < 2; ++h)
        if (h == 0 || two) {
          const unsigned char* at = y + (kb * 8 + ft) * kYPitch + ((b + h) * 8 + fg) * 16;
          y0[h] = *reinterpret_cast<const uint4*>(at);
          y1[h] = *reinterpret_cast<const uint4*>(at + 4 * kYPitch);
        }
      auto word = [](const uint4& v, int w) {
        return w == 0 ? v.x : w == 1 ? v.y : w == 2 ? v.z : v.w;
      };
      // re += ar (word r of Y), im += ai (word i of Y)
      auto both = [&](const uint32_t(&ar)[4], int r, const uint32_t(&ai)[4], int i) {
        mma(re[b], ar, word(y0[0], r), word(y1[0], r));
        mma(im[b], ai, word(y0[0], i), word(y1[0], i));
        if (two) {
          mma(re[c], ar, word(y0[1], r), word(y1[1], r));
          mma(im[c], ai, word(y0[1], i), word(y1[1], i));
        }
      };
      both(arh, 0, arh, 2);
      both(arh, 1, arh, 3);
      both(arl, 0, arl, 2);
      if (ADJ) {
        both(aih, 2, nih, 0);
        both(aih, 3, nih, 1);
        both(ail, 2, nil, 0);
      } else {
        both(nih, 2, aih, 0);
        both(nih, 3, aih, 1);
        both(nil, 2, ail, 0);
      }
    }
  }
}

// X row elements (re, im) of two neighbouring columns: X -= v.
__device__ __forceinline__ void subtract(float2* x, float re0, float im0, float re1, float im1,
                                         bool wide, bool second) {
  if (wide) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(x), "f"(-re0), "f"(-im0),
                 "f"(-re1), "f"(-im1)
                 : "memory");
  } else {
    asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(x), "f"(-re0), "f"(-im0) : "memory");
    if (second)
      asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(x + 1), "f"(-re1), "f"(-im1)
                   : "memory");
  }
}

template <bool ADJ, int D>
__global__ void __launch_bounds__(kThreads, 1)
    solve_cluster_kernel(const Args a, const __grid_constant__ CUtensorMap fmap) {
  using S = Shape<D>;
  constexpr int R = S::kRows, TR = S::kTR;
  extern __shared__ unsigned char dyn[];
  Shared& sh = *reinterpret_cast<Shared*>(
      (reinterpret_cast<uintptr_t>(dyn) + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int C = a.cluster;
  const int rank = (int)blockIdx.x % C, unit = (int)blockIdx.x / C;
  const bool diagonal = rank < D;
  const int p = unit / a.strips, c0 = (unit % a.strips) * kStrip;
  const int ncols = min(kStrip, a.nrhs - c0);
  const int steps = 2 * a.nb;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kFull; ++s) mbar_init(&sh.full[s], 1);
    for (int s = 0; s < kStages; ++s) mbar_init(&sh.empty[s], 4);
    mbar_init(&sh.bar_y, D);
    mbar_init(&sh.bar_x, C);
    sh.failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  cluster_meet();
  volatile int* failed = &sh.failed;
  auto fail = [&]() {
    *failed = 1;
    atomicCAS(&a.status[p], 0, (int)AOSB_ERR_TIMEOUT);
  };
  int issued = 0;  // producer: ring entries filled

  if (warp == kConsumers / 32) {
    if (lane == 0) {
      int g = 0;
      const int64_t base = (int64_t)p * a.n_slots;
      // one ring entry: 32 rows (ADJ: columns) from `part` on of a factor tile
      auto fill = [&](int slot, int part, int tile) {
        const int st = g % kStages;
        if (!mbar_wait(&sh.empty[st], ((uint32_t)(g / kStages) & 1u) ^ 1u, a.limit)) {
          fail();
          return false;
        }
        uint64_t* bar = &sh.full[g % kFull];
        sh.tile[g % kFull] = tile;
        mbar_expect_tx(bar, kUnitBytes);
        const int row0 = (int)((base + slot) * (2 * kT));
#pragma unroll
        for (int plane = 0; plane < 2; ++plane)
#pragma unroll
          for (int j = 0; j < kT / 32; ++j)
            tma_load_2d(sh.ring[st] + plane * kUnitPlane + j * kBox, &fmap, ADJ ? part : 32 * j,
                        row0 + plane * kT + (ADJ ? 32 * j : part), bar);
        issued = ++g;
        return true;
      };
      bool ok = true;
      for (int s = 0; s < steps && ok && !*failed; ++s) {
        const Sweep& sw = s < a.nb ? a.forward : a.backward;
        const int k = s < a.nb ? s : steps - 1 - s;
        const int o0 = sw.off[k], units = (sw.off[k + 1] - o0) * kParts;
        // the CTA's rows of D lie in the 32-row parts that hold them
        for (int d = 0; d < S::kDUnits && ok && diagonal; ++d)
          ok = fill(a.diag_slot[k], (rank * R) / kUnitRows * kUnitRows + d * kUnitRows, 0);
        for (int u = rank; u < units && ok; u += C)
          ok = fill(sw.slot[o0 + u / kParts], u % kParts * kUnitRows, sw.tile[o0 + u / kParts] * kT +
                                                                         u % kParts * kUnitRows);
      }
    }
  } else {
    const int tid = threadIdx.x;
    const int32_t* pivots = a.pivots + (size_t)p * a.n_pad;
    float2* X = a.work + (size_t)p * a.n_pad * a.nrhs + c0;
    int g = 0;  // ring entry
    const int group = warp / 4, m16 = (warp & 1) * 16, khalf = warp / 2 & 1;
    const uint32_t y_local = smem_u32(sh.y);
    auto entry_ready = [&](int e) {
      return mbar_wait(&sh.full[e % kFull], (uint32_t)(e / kFull) & 1u, a.limit);
    };
    for (int s = 0; s < steps; ++s) {
      const bool fwd = s < a.nb;
      const int k = fwd ? s : steps - 1 - s;
      const Sweep& sw = fwd ? a.forward : a.backward;
      const uint32_t phase = (uint32_t)s & 1u;
      const int32_t* pv = pivots + (size_t)k * kT;
      const int units = (sw.off[k + 1] - sw.off[k]) * kParts;
      const bool gather = !ADJ && fwd, scatter = ADJ && !fwd;
      bool ok = true;
      constexpr int kPairs = (R / 2 + kWarps - 1) / kWarps;  // row pairs per warp
      float2 y[kPairs][2];
      if (scatter && tid < kT) sh.order[tid] = pv[tid];
      if (diagonal) {
        // rows of X_k this thread stages, through the row interchanges
        constexpr int kStaged = (kT + kConsumers / 16 - 1) / (kConsumers / 16);
        int from[kStaged];
#pragma unroll
        for (int t = 0; t < kStaged; ++t) {
          const int r = tid / 16 + kConsumers / 16 * t;
          from[t] = gather && r < kT ? pv[r] : r;
        }
        ok = s == 0 || cluster_wait(&sh.bar_x, phase ^ 1u, a.limit);
        const float2* Xk = X + (size_t)k * kT * a.nrhs;
        {
          const int c = 2 * (tid % 16);
          float4 v[kStaged];
#pragma unroll
          for (int t = 0; t < kStaged; ++t) {
            const float2* src = Xk + (size_t)from[t] * a.nrhs + c;
            v[t] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (tid / 16 + kConsumers / 16 * t >= kT) break;
            if (a.wide) {
              if (c < ncols) v[t] = __ldcg(reinterpret_cast<const float4*>(src));
            } else {
              if (c < ncols) {
                const float2 e = __ldcg(src);
                v[t].x = e.x;
                v[t].y = e.y;
              }
              if (c + 1 < ncols) {
                const float2 e = __ldcg(src + 1);
                v[t].z = e.x;
                v[t].w = e.y;
              }
            }
          }
#pragma unroll
          for (int t = 0; t < kStaged; ++t)
            if (tid / 16 + kConsumers / 16 * t < kT)
              *reinterpret_cast<float4*>(&sh.x[tid / 16 + kConsumers / 16 * t][c]) = v[t];
        }
#pragma unroll
        for (int d = 0; d < S::kDUnits; ++d) ok = ok && entry_ready(g + d);
        if (consumers_any(!ok)) {
          if (tid == 0) fail();
          break;
        }
        // Y rows of this CTA: thread tile TR rows x 4 columns, warps split K
        {
          const int rg = warp % S::kRowGroups * (4 * TR) + lane / 8 * TR;
          const int slice = warp / S::kRowGroups, cg = 2 * (lane % 8);
          // ring slot and row (ADJ: column) in it of this thread's first row
          const unsigned char* slab = sh.ring[(g + (R > kUnitRows ? rg / kUnitRows : 0)) % kStages];
          const int in = (rank * R + rg) % kUnitRows, row = rank * R + rg;
          // the rows use inv(L) (unit diagonal) or inv(U)
          const bool unit_lower = fwd != ADJ, lower = fwd;
          constexpr int KS = kT / S::kSlices;
          float2 acc[TR][4];
#pragma unroll
          for (int i = 0; i < TR; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = make_float2(0.f, 0.f);
#pragma unroll 1
          for (int q = slice * KS; q < (slice + 1) * KS && warp < kDiagWarps; q += 4) {
            if (lower ? q > row + TR - 1 : q + 3 < row) continue;  // outside the triangle
            float dr[4][TR], di[4][TR];  // [k][row]
            if (!ADJ) {
#pragma unroll
              for (int i = 0; i < TR; ++i) {
                const unsigned char* b = slab + (q >> 5) * kBox + (in + i) * 128 +
                                         ((((q & 31) >> 2) ^ ((in + i) & 7)) << 4);
                const float4 vr = *reinterpret_cast<const float4*>(b);
                const float4 vi = *reinterpret_cast<const float4*>(b + kUnitPlane);
                dr[0][i] = vr.x; dr[1][i] = vr.y; dr[2][i] = vr.z; dr[3][i] = vr.w;
                di[0][i] = vi.x; di[1][i] = vi.y; di[2][i] = vi.z; di[3][i] = vi.w;
              }
            } else {
#pragma unroll
              for (int h = 0; h < 4; ++h) {
                const unsigned char* b =
                    slab + (q + h) * 128 + (((in >> 2) ^ ((q + h) & 7)) << 4) + (in & 3) * 4;
#pragma unroll
                for (int i = 0; i < TR; ++i) {
                  dr[h][i] = *reinterpret_cast<const float*>(b + 4 * i);
                  di[h][i] = -*reinterpret_cast<const float*>(b + 4 * i + kUnitPlane);
                }
              }
            }
#pragma unroll
            for (int h = 0; h < 4; ++h)
#pragma unroll
              for (int i = 0; i < TR; ++i) {
                const int off = q + h - (row + i);  // column minus row
                const bool take = lower ? off < 0 : off > 0;
                if (!take) {
                  const bool diag = off == 0;
                  dr[h][i] = diag ? (unit_lower ? 1.0f : dr[h][i]) : 0.0f;
                  di[h][i] = diag && !unit_lower ? di[h][i] : 0.0f;
                }
              }
#pragma unroll
            for (int h = 0; h < 4; ++h) {
              const float4 x0 = *reinterpret_cast<const float4*>(&sh.x[q + h][cg]);
              const float4 x1 = *reinterpret_cast<const float4*>(&sh.x[q + h][16 + cg]);
              const float2 xv[4] = {make_float2(x0.x, x0.y), make_float2(x0.z, x0.w),
                                    make_float2(x1.x, x1.y), make_float2(x1.z, x1.w)};
#pragma unroll
              for (int i = 0; i < TR; ++i) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  acc[i][j].x = fmaf(dr[h][i], xv[j].x, acc[i][j].x);
                  acc[i][j].y = fmaf(dr[h][i], xv[j].y, acc[i][j].y);
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  acc[i][j].x = fmaf(-di[h][i], xv[j].y, acc[i][j].x);
                  acc[i][j].y = fmaf(di[h][i], xv[j].x, acc[i][j].y);
                }
              }
            }
          }
          consumers_any(false);  // X_k and D are read: their space is free
          if (warp < 4 && lane == 0)
#pragma unroll
            for (int d = 0; d < S::kDUnits; ++d) mbar_arrive(&sh.empty[(g + d) % kStages]);
          float2(*part)[kStrip] = sh.x;  // [slice * R + row]
#pragma unroll
          for (int i = 0; i < TR && warp < kDiagWarps; ++i) {
            float2* to = part[slice * R + rg + i];
            *reinterpret_cast<float4*>(&to[cg]) =
                make_float4(acc[i][0].x, acc[i][0].y, acc[i][1].x, acc[i][1].y);
            *reinterpret_cast<float4*>(&to[16 + cg]) =
                make_float4(acc[i][2].x, acc[i][2].y, acc[i][3].x, acc[i][3].y);
          }
        }
        g += S::kDUnits;
        consumers_any(false);
        // sums of the partials for two rows of one column, to every peer
#pragma unroll
        for (int o = 0; o < kPairs; ++o) {
          const int i = 2 * (warp + kWarps * o);
          if (i >= R) break;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            float2 v = sh.x[i + h][lane];
#pragma unroll
            for (int sl = 1; sl < S::kSlices; ++sl) {
              const float2 w = sh.x[sl * R + i + h][lane];
              v.x += w.x;
              v.y += w.y;
            }
            y[o][h] = v;
          }
          uint32_t rh, rl, ih, il;
          split2(y[o][0].x, y[o][1].x, rh, rl);
          split2(y[o][0].y, y[o][1].y, ih, il);
          const uint32_t dst = y_local + (rank * R + i) / 2 * kYPitch + lane * 16;
          for (int c = 0; c < C; ++c) peer_store16(peer_address(dst, c), rh, rl, ih, il);
        }
        consumers_any(false);
        if (tid < C) peer_arrive(peer_address(smem_u32(&sh.bar_y), tid));
      } else {
        consumers_any(false);  // order[] is written
      }
      ok = cluster_wait(&sh.bar_y, phase, a.limit);
#pragma unroll
      for (int o = 0; o < kPairs; ++o) {
        const int i = 2 * (warp + kWarps * o);
        if (!diagonal || i >= R || lane >= ncols) break;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int r = rank * R + i + h;
          X[((size_t)k * kT + (scatter ? sh.order[r] : r)) * a.nrhs + lane] = y[o][h];
        }
      }
      // update units of this CTA, in turn to the groups of warps
      for (int u = rank, j = 0; u < units; u += C, ++g, ++j) {
        if (j % kGroups != group) continue;
        // Each lane polls for itself, so a wait may run out in some lanes of a
        // warp only: all of them vote, those that gave up above among them.
        ok = __all_sync(0xffffffffu, ok && entry_ready(g) ? 1 : 0);
        // after a failure both warps of a pair still meet
        if (!ok) {
          pair_sync(2 + group * 2 + (warp & 1));
          pair_sync(2 + group * 2 + (warp & 1));
          continue;
        }
        const int row = sh.tile[g % kFull] + m16 + lane / 4;
        const unsigned char* slab = sh.ring[g % kStages];
        float re[4][4], im[4][4];
#pragma unroll
        for (int b = 0; b < 4; ++b)
#pragma unroll
          for (int e = 0; e < 4; ++e) re[b][e] = im[b][e] = 0.0f;
        if (ncols <= 8)
          scatter ? unit_product<ADJ, ADJ, 1>(slab, sh.y, sh.order, m16, khalf, lane, re, im)
                  : unit_product<ADJ, false, 1>(slab, sh.y, nullptr, m16, khalf, lane, re, im);
        else if (ncols <= 16)
          scatter ? unit_product<ADJ, ADJ, 2>(slab, sh.y, sh.order, m16, khalf, lane, re, im)
                  : unit_product<ADJ, false, 2>(slab, sh.y, nullptr, m16, khalf, lane, re, im);
        else if (ncols <= 24)
          scatter ? unit_product<ADJ, ADJ, 3>(slab, sh.y, sh.order, m16, khalf, lane, re, im)
                  : unit_product<ADJ, false, 3>(slab, sh.y, nullptr, m16, khalf, lane, re, im);
        else
          scatter ? unit_product<ADJ, ADJ, 4>(slab, sh.y, sh.order, m16, khalf, lane, re, im)
                  : unit_product<ADJ, false, 4>(slab, sh.y, nullptr, m16, khalf, lane, re, im);
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh.empty[g % kStages]);
        // The two warps of a row half add up: each hands over the blocks that
        // the other one subtracts from X (the first half of K the low ones).
        const int blocks = (ncols + 7) / 8, low = (blocks + 1) / 2;
        float4* out = reinterpret_cast<float4*>(&sh.x[0][0]) + warp * 128 + lane;
        const float4* in = reinterpret_cast<float4*>(&sh.x[0][0]) + (warp ^ 2) * 128 + lane;
        pair_sync(2 + group * 2 + (warp & 1));  // the peer has read its last ones
#pragma unroll
        for (int b = 0; b < 4; ++b)
          if (b < blocks && (b < low) == (khalf == 1)) {
            const int to = b < low ? b : b - low;
            out[to * 64] = make_float4(re[b][0], re[b][1], re[b][2], re[b][3]);
            out[to * 64 + 32] = make_float4(im[b][0], im[b][1], im[b][2], im[b][3]);
          }
        pair_sync(2 + group * 2 + (warp & 1));
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          const int c = b * 8 + 2 * (lane % 4);
          if (b >= blocks || (b < low) != (khalf == 0)) continue;
          const int at = b < low ? b : b - low;
          const float4 r = in[at * 64], m = in[at * 64 + 32];
          if (c >= ncols) continue;
          float2* to = X + (size_t)row * a.nrhs + c;
          subtract(to, re[b][0] + r.x, im[b][0] + m.x, re[b][1] + r.y, im[b][1] + m.y, a.wide,
                   c + 1 < ncols);
          subtract(to + (size_t)8 * a.nrhs, re[b][2] + r.z, im[b][2] + m.z, re[b][3] + r.w,
                   im[b][3] + m.w, a.wide, c + 1 < ncols);
        }
      }
      if (consumers_any(!ok)) {
        if (tid == 0) fail();
        break;
      }
      if (tid < C) peer_arrive(peer_address(smem_u32(&sh.bar_x), tid));
    }
  }
  // After a failure the producer waits (bounded) until the ring entries in
  // flight have received their bytes; peers may write into this CTA's shared
  // memory until the cluster has met.
  __syncthreads();
  if (sh.failed && warp == kConsumers / 32 && lane == 0)
    for (int e = max(issued - kStages, 0); e < issued; ++e)
      mbar_wait(&sh.full[e % kFull], (uint32_t)(e / kFull) & 1u);
  __syncthreads();
  cluster_meet();
}

// Cluster sizes and the CTAs of each that share the diagonal product.  Sizes
// between the powers of two are there because a cluster lives in one GPC (16
// to 20 SMs): 15 clusters of 8 or 9 fit the chip, 11 of 10, 22 of 6, 33 of 4.
struct Form {
  int cluster, diagonal;
};
constexpr Form kForms[] = {{16, 16}, {10, 8}, {9, 8}, {6, 4}, {5, 4}, {4, 4}, {3, 2}, {2, 2}};
constexpr int kFormCount = sizeof(kForms) / sizeof(kForms[0]);

using Kernel = void (*)(const Args, const CUtensorMap);
template <bool ADJ>
Kernel kernel_of(int diagonal) {
  switch (diagonal) {
    case 16: return solve_cluster_kernel<ADJ, 16>;
    case 8: return solve_cluster_kernel<ADJ, 8>;
    case 4: return solve_cluster_kernel<ADJ, 4>;
    default: return solve_cluster_kernel<ADJ, 2>;
  }
}

cudaLaunchConfig_t launch_config(int cluster, int units, cudaStream_t st,
                                 cudaLaunchAttribute* attr) {
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)cluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)units * cluster);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

// Clusters of each form that run at the same time on a device (0: none), with
// the kernels' attributes set; found once per device.
struct Residency {
  int clusters[kFormCount];
};
Residency residency(int device) {
  static std::mutex mu;
  static Residency known[64];
  static uint64_t have = 0;
  std::lock_guard<std::mutex> lock(mu);
  if (device < 64 && (have >> device & 1)) return known[device];
  Residency r{};
  for (int f = 0; f < kFormCount; ++f) {
    r.clusters[f] = 1 << 30;
    for (Kernel fn : {kernel_of<false>(kForms[f].diagonal), kernel_of<true>(kForms[f].diagonal)}) {
      int n = 0;
      cudaLaunchAttribute attr[1];
      const cudaLaunchConfig_t cfg = launch_config(kForms[f].cluster, 1, nullptr, attr);
      if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem) !=
              cudaSuccess ||
          cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) !=
              cudaSuccess ||
          cudaOccupancyMaxActiveClusters(&n, fn, &cfg) != cudaSuccess) {
        cudaGetLastError();
        n = 0;
      }
      r.clusters[f] = std::min(r.clusters[f], n);
    }
  }
  if (device < 64) {
    known[device] = r;
    have |= (uint64_t)1 << device;
  }
  return r;
}

// Microseconds of one step of `units` units in a form: the chain of a step,
// the diagonal product over its CTAs, the update units of the busiest CTA, all
// times the waves of clusters.  Fitted to whole solves of plans of 7 to 114
// steps with 16 to 600 units; us a step, 32 columns, this kernel / one launch
// per step: 1000-atom bundle (102 steps) 8 pencils 30 / 41, 16: 47 / 56, 32: 63
// / 84, 64: 119 / 142; 64 atoms (7 steps), 5 pencils 10 / 32, 16: 16 / 42, 300:
// 133 / 347.  The waves are what loses: past one wave of the smallest clusters
// the separate launches, which share all units out over all SMs, are as fast or
// faster where the last wave is short and a step has some thirty tiles (102
// steps, 99 pencils: 189 / 206, 108: 235 / 221, 127: 248 / 257; 75 steps, 108
// pencils: 203 / 189).
double step_cost(const Form& f, int resident, int units, double tiles, int columns) {
  if (resident <= 0) return 1e30;
  const double waves = (units + resident - 1) / resident;
  const double rows = kT / f.diagonal;
  const double unit = 0.45 + 0.24 * ((columns + 7) / 8);
  return 1.05 * waves * (6.5 + 0.15 * rows + unit * kParts * tiles / f.cluster);
}

// The same for one launch per diagonal step and one per update, where the
// columns hardly matter (102 steps, 96 pencils: 200 us with 32, 191 with 8).
// With these two costs the form taken was at most 2 % behind the better one in
// 140 batches on nine plans of up to 416 steps; with 0.85 + 0.027 tiles, and a factor of 1 for the
// clusters, it was up to 7 % behind (108 pencils above).
double launch_cost(int units, double tiles) { return 27.0 + units * (0.35 + 0.042 * tiles); }

}  // namespace

bool solve_cluster(const aosb_plan* P, const aosb_solve_args_v1* s, int32_t* status, int* rc,
                   char* err, size_t cap) {
  const int strips = (s->n_rhs + kStrip - 1) / kStrip, units = s->n_pencils * strips;
  const double tiles = (double)P->lb_tile.size() / (double)P->nb;
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess) return false;
  const Residency res = residency(device);
  int best = -1;
  double least = launch_cost(units, tiles);
  for (int f = 0; f < kFormCount; ++f) {
    const double c = step_cost(kForms[f], res.clusters[f], units, tiles, std::min(s->n_rhs, kStrip));
    if (c < least) {
      least = c;
      best = f;
    }
  }
  if (best < 0) return false;
  CUtensorMap map;
  *rc = encode_f32_2d((void*)s->factor, kT, (uint64_t)s->n_pencils * P->n_slots * 2 * kT, 32, 32,
                      true, &map, err, cap);
  if (*rc) return true;
  Args a{};
  a.nb = (int)P->nb;
  a.nrhs = s->n_rhs;
  a.strips = strips;
  a.n_pad = P->n_pad;
  a.n_slots = P->n_slots;
  a.diag_slot = P->d_diag_slot;
  a.cluster = kForms[best].cluster;
  a.factor = s->factor;
  a.pivots = s->pivots;
  a.work = (float2*)s->work;
  a.status = status;
  a.wide = s->n_rhs % 2 == 0 && ((uintptr_t)s->work & 15) == 0;
  a.limit = tc_wait_limit();
  if (!s->adjoint) {
    a.forward = {P->d_lb_off, P->d_lb_tile, P->d_lb_slot};
    a.backward = {P->d_ua_off, P->d_ua_tile, P->d_ua_slot};
  } else {
    a.forward = {P->d_ur_off, P->d_ur_tile, P->d_ur_slot};
    a.backward = {P->d_ll_off, P->d_ll_tile, P->d_ll_slot};
  }
  cudaLaunchAttribute attr[1];
  const cudaLaunchConfig_t cfg =
      launch_config(a.cluster, units, (cudaStream_t)s->stream, attr);
  const Kernel fn = s->adjoint ? kernel_of<true>(kForms[best].diagonal)
                               : kernel_of<false>(kForms[best].diagonal);
  const cudaError_t e = cudaLaunchKernelEx(&cfg, fn, a, map);
  if (e != cudaSuccess)
    *rc = set_error(err, cap, AOSB_ERR_CUDA, "cluster solve launch failed: %s",
                    cudaGetErrorString(e));
  else
    count_launches(1);
  return true;
}

}  // namespace aosb
