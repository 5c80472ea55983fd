// Bloch pattern (host, once per bundle) and Bloch sum (device, per k).
//
// The reference expands every block entry into (row, col, source, phase)
// tuples and argsorts them (src/aospectrum/sparse.py:64-140), then per k
// gathers, multiplies and segment-sums them (sparse.py:181-245).  Here the
// pattern is built at block granularity: blocks with the same atom pair
// (i, j) form one "group" whose entries land in the same 2D window of the
// CSR arrays, because every row of atom i has the same column structure.
// Entry (a, c) of group (i, j) sits at dst_base + a * rowlen_i + c.
//
// Two device kernels sum the member blocks of (i, j) and of its mirror (j, i) in
// block order (the order the reference's stable sort leaves them in) and apply
// the Hermitian projection of sparse.py:25-36: one gives a CTA a strip of up to
// eight neighbouring windows of one row atom and writes it row by row, the other
// gives a warp a window (which one when: strips_pay).  With
// real block values the products v * phase are exact, so the output is
// bit-identical to the reference's numpy path.
#include "common.cuh"
#include "timing.h"

#include <algorithm>
#include <numeric>
#include <vector>

// The windows in strips, the mean windows, columns and values of a strip, and the
// mean of its largest window's values over its mean window's.
struct StripShape {
  double windows = 0, per_strip = 0, columns = 0, values = 0, uneven = 0;
};

struct aosb_bloch {
  int64_t n = 0, n_atoms = 0, n_blocks = 0, nnz = 0;
  std::vector<int64_t> indptr;
  std::vector<int32_t> indices;
  std::vector<int32_t> shifts;       // n_shifts * 3
  std::vector<int32_t> block_shift;  // n_blocks
  // device tables
  int64_t n_groups = 0, n_members = 0;
  int64_t* d_indptr = nullptr;
  int32_t* d_indices = nullptr;
  int4* d_group = nullptr;        // (nr, nc, rowlen, mirror)
  int64_t* d_group_dst = nullptr;  // dst base
  int2* d_group_members = nullptr; // [begin, end) into members
  int64_t* d_member_off = nullptr; // value offset of each member block
  int32_t* d_member_shift = nullptr;
  int2* d_strips = nullptr;        // [first, last) groups of each strip
  int32_t* d_others = nullptr;     // groups in no strip
  // host copies of the device tables (uploaded by aosb_bloch_upload)
  std::vector<int4> g_info;
  std::vector<int64_t> g_dst;
  std::vector<int2> g_mem;
  std::vector<int64_t> m_off;
  std::vector<int32_t> m_shift;
  std::vector<int2> strips;
  std::vector<int32_t> others;
  StripShape shape;
  int64_t n_values = 0;  // stored block values (sum of block sizes), set at upload
  bool uploaded = false;
};

namespace {

template <typename T>
int upload(T** dst, const std::vector<T>& src, char* err, size_t cap) {
  size_t bytes = std::max<size_t>(src.size(), 1) * sizeof(T);
  cudaError_t e = cudaMalloc((void**)dst, bytes);
  if (e != cudaSuccess)
    return aosb::set_error(err, cap, AOSB_ERR_MEMORY, "cudaMalloc(%zu) failed: %s", bytes,
                           cudaGetErrorString(e));
  if (!src.empty()) {
    e = cudaMemcpy(*dst, src.data(), src.size() * sizeof(T), cudaMemcpyHostToDevice);
    if (e != cudaSuccess)
      return aosb::set_error(err, cap, AOSB_ERR_CUDA, "cudaMemcpy failed: %s",
                             cudaGetErrorString(e));
  }
  return 0;
}

template <typename V>
__device__ __forceinline__ float2 load_value(const V* v, int64_t i);
template <>
__device__ __forceinline__ float2 load_value<float>(const float* v, int64_t i) {
  return make_float2(v[i], 0.0f);
}
template <>
__device__ __forceinline__ float2 load_value<float2>(const float2* v, int64_t i) {
  return v[i];
}

// Complex product without FMA contraction, matching a plain
// (ac - bd, ad + bc) evaluation in float32.
__device__ __forceinline__ float2 cmul_rn(float2 a, float2 b) {
  return make_float2(__fsub_rn(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)),
                     __fadd_rn(__fmul_rn(a.x, b.y), __fmul_rn(a.y, b.x)));
}

// k points whose phases a thread holds at a time
constexpr int kBlochKChunk = 4;

// Sums of one element over the member blocks [range.x, range.y) of a group
// for the k points k0 .. k0+nk-1 (nk <= kBlochKChunk): each member value is
// loaded once and multiplied by the phase of its lattice shift at every k.
// Members are added in block order, first product first, for every k.
template <typename V>
__device__ __forceinline__ void group_sums(const V* vals, const int64_t* moff, const int32_t* msh,
                                           const float2* ph0, int64_t n_shifts, int nk,
                                           int2 range, int64_t elem,
                                           float2 (&s)[kBlochKChunk]) {
#pragma unroll
  for (int q = 0; q < kBlochKChunk; ++q) s[q] = make_float2(0.0f, 0.0f);
  for (int m = range.x; m < range.y; ++m) {
    const float2 v = load_value<V>(vals, moff[m] + elem);
    const float2* ph = ph0 + msh[m];
#pragma unroll
    for (int q = 0; q < kBlochKChunk; ++q) {
      if (q < nk) {
        const float2 p = cmul_rn(v, ph[q * n_shifts]);
        if (m == range.x) {
          s[q] = p;
        } else {
          s[q].x = __fadd_rn(s[q].x, p.x);
          s[q].y = __fadd_rn(s[q].y, p.y);
        }
      }
    }
  }
}

__device__ __forceinline__ float2 hermitian_mean(float2 x, float2 y) {
  return make_float2(__fmul_rn(__fadd_rn(x.x, y.x), 0.5f), __fmul_rn(__fsub_rn(x.y, y.y), 0.5f));
}

// Strips: neighbouring windows (i, j) of one row atom, whose segments of each
// CSR row are contiguous; at most kStripWindows of them, kStripColumns columns
// and kStripValues elements, and one member block each way in every window (a
// single lattice image).  Windows that do not fit belong to no strip.
constexpr int kStripWindows = 8, kStripColumns = 128, kStripValues = 1376;
constexpr int kStripThreads = 256;

// Element (a, c) of window (i, j) and element (c, a) of its mirror (j, i) hold
// the Hermitian mean of the pair and its conjugate: the upper window (i < j)
// writes mean(x_ij(a, c), x_ji(c, a)), the lower window writes the conjugate of
// its upper mirror's mean formed the same way; in a diagonal window the
// elements above and below the diagonal do so, and the diagonal keeps its real
// part.

// One warp, one window: any number of member blocks, any size.
template <typename V>
__device__ __forceinline__ void window_sums(
    int g, int lane, int k0, int n_k, const int4* __restrict__ group,
    const int64_t* __restrict__ gdst, const int2* __restrict__ gmem,
    const int64_t* __restrict__ moff, const int32_t* __restrict__ msh, const V* __restrict__ hv,
    const V* __restrict__ sv, const float2* __restrict__ phases, int64_t n_shifts, int64_t nnz,
    float2* __restrict__ hout, float2* __restrict__ sout) {
  const int nk = min(n_k - k0, kBlochKChunk);
  const float2* ph0 = phases + (int64_t)k0 * n_shifts;
  const int64_t out0 = (int64_t)k0 * nnz;
  const int4 gi = group[g];  // nr, nc, rowlen, mirror
  const int nr = gi.x, nc = gi.y, rl = gi.z, gm = gi.w;
  const int ne = nr * nc;
  const int64_t base = gdst[g];
  const int2 rg = gmem[g];
  float2 x[kBlochKChunk], y[kBlochKChunk];
  if (gm == g) {
    // diagonal window: t runs over [matrix H|S][row-major element]; the mean
    // of the pair (lo, hi) is formed the same way for both of its entries
    for (int t = lane; t < 2 * ne; t += 32) {
      const int which = t >= ne;
      const int e = t - which * ne;
      const int a = e / nc, c = e - (e / nc) * nc;
      const V* vals = which == 0 ? hv : sv;
      float2* out = (which == 0 ? hout : sout) + out0 + base + (int64_t)a * rl + c;
      const int lo = min(a, c), hi = max(a, c);
      group_sums<V>(vals, moff, msh, ph0, n_shifts, nk, rg, lo * nc + hi, x);
      if (a != c) group_sums<V>(vals, moff, msh, ph0, n_shifts, nk, rg, hi * nc + lo, y);
#pragma unroll
      for (int q = 0; q < kBlochKChunk; ++q) {
        if (q < nk) {
          float2 v;
          if (a == c) {
            v = make_float2(x[q].x, 0.0f);
          } else {
            const float2 mean = hermitian_mean(x[q], y[q]);
            v = a < c ? mean : make_float2(mean.x, -mean.y);
          }
          out[q * nnz] = v;
        }
      }
    }
    return;
  }
  const bool lower = gm < g;
  const int2 mr = gmem[gm];
  // the mean's first operand comes from the upper group of the pair
  const int2 r1 = lower ? mr : rg, r2 = lower ? rg : mr;
  if (r1.y - r1.x == 1 && r2.y - r2.x == 1) {
    // One member block each way (a single lattice image, the common case):
    // value offsets and phases are warp-uniform and loaded once; each lane
    // keeps two elements' value loads in flight.
    const int64_t o1 = moff[r1.x], o2 = moff[r2.x];
    const float2* ph1 = ph0 + msh[r1.x];
    const float2* ph2 = ph0 + msh[r2.x];
    float2 p1[kBlochKChunk], p2[kBlochKChunk];
#pragma unroll
    for (int q = 0; q < kBlochKChunk; ++q) {
      p1[q] = q < nk ? ph1[q * n_shifts] : make_float2(0.0f, 0.0f);
      p2[q] = q < nk ? ph2[q * n_shifts] : make_float2(0.0f, 0.0f);
    }
    for (int t0 = lane; t0 < 2 * ne; t0 += 64) {
      float2 v1[2], v2[2];
      float2* out[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int t = t0 + 32 * u;
        out[u] = nullptr;
        v1[u] = v2[u] = make_float2(0.0f, 0.0f);
        if (t < 2 * ne) {
          const int which = t >= ne;
          const int e = t - which * ne;
          const int a = e / nc, c = e - a * nc;
          const int eg = a * nc + c, em = c * nr + a;
          const V* vals = which == 0 ? hv : sv;
          out[u] = (which == 0 ? hout : sout) + out0 + base + (int64_t)a * rl + c;
          v1[u] = load_value<V>(vals, o1 + (lower ? em : eg));
          v2[u] = load_value<V>(vals, o2 + (lower ? eg : em));
        }
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        if (out[u] == nullptr) continue;
#pragma unroll
        for (int q = 0; q < kBlochKChunk; ++q) {
          if (q < nk) {
            const float2 mean = hermitian_mean(cmul_rn(v1[u], p1[q]), cmul_rn(v2[u], p2[q]));
            out[u][q * nnz] = lower ? make_float2(mean.x, -mean.y) : mean;
          }
        }
      }
    }
    return;
  }
  // general: t runs over [matrix H|S][row-major element]
  for (int t = lane; t < 2 * ne; t += 32) {
    const int which = t >= ne;
    const int e = t - which * ne;
    const int a = e / nc, c = e - a * nc;
    const int eg = a * nc + c, em = c * nr + a;
    const V* vals = which == 0 ? hv : sv;
    float2* out = (which == 0 ? hout : sout) + out0 + base + (int64_t)a * rl + c;
    group_sums<V>(vals, moff, msh, ph0, n_shifts, nk, r1, lower ? em : eg, x);
    group_sums<V>(vals, moff, msh, ph0, n_shifts, nk, r2, lower ? eg : em, y);
#pragma unroll
    for (int q = 0; q < kBlochKChunk; ++q) {
      if (q < nk) {
        const float2 mean = hermitian_mean(x[q], y[q]);
        out[q * nnz] = lower ? make_float2(mean.x, -mean.y) : mean;
      }
    }
  }
}

// A warp per window and chunk of k points.  Neighbouring warps write
// neighbouring windows of the same CSR rows at the same time, so that the 32-byte
// sectors they share are completed in L2.
constexpr int kWindowWarps = 8;
template <typename V>
__global__ void __launch_bounds__(kWindowWarps * 32, 4) bloch_windows_kernel(
    int64_t n_groups, const int4* __restrict__ group, const int64_t* __restrict__ gdst,
    const int2* __restrict__ gmem, const int64_t* __restrict__ moff,
    const int32_t* __restrict__ msh, const V* __restrict__ hv, const V* __restrict__ sv,
    const float2* __restrict__ phases, int64_t n_shifts, int64_t nnz, int n_k,
    float2* __restrict__ hout, float2* __restrict__ sout) {
  const int64_t g = (int64_t)blockIdx.x * kWindowWarps + threadIdx.x / 32;
  if (g < n_groups)
    window_sums<V>((int)g, threadIdx.x % 32, blockIdx.y * kBlochKChunk, n_k, group, gdst, gmem,
                   moff, msh, hv, sv, phases, n_shifts, nnz, hout, sout);
}

// One CTA per strip (x) and share of the k chunks (y), after `lead` CTAs with a
// warp for each window outside strips and each chunk.  The strip's blocks are
// copied to shared memory, contiguous as they are stored, with all copies in
// flight at once; then a thread keeps one column of the strip, its window's
// phases in registers, and walks the rows: a warp writes 256 contiguous bytes of
// a CSR row, and the blocks are read once for all k.  A warp per window gathers
// single values in rounds of two per lane and is bound by their latency (43 % of
// the copy bandwidth).  4096 atoms, 13 orbitals, 4 k points (4.6 GB): 1.60 ms
// with it, 1.08 here (0.70 at the copy bandwidth; streaming stores and other
// register limits were slower); 64 atoms, 1 k point: 9.8 and 5.8 us.
template <typename V>
__global__ void __launch_bounds__(kStripThreads) bloch_strips_kernel(
    const int2* __restrict__ strips, int lead, int n_others, const int32_t* __restrict__ others,
    const int4* __restrict__ group, const int64_t* __restrict__ gdst, const int2* __restrict__ gmem,
    const int64_t* __restrict__ moff, const int32_t* __restrict__ msh, const V* __restrict__ hv,
    const V* __restrict__ sv, const float2* __restrict__ phases, int64_t n_shifts, int64_t nnz,
    int n_k, float2* __restrict__ hout, float2* __restrict__ sout) {
  // [own, mirror block][H, S][values of the strip's windows in turn]
  __shared__ V vals[2][2][kStripValues];
  __shared__ int first_value[kStripWindows], first_column[kStripWindows + 1], widths[kStripWindows];
  __shared__ int mirrors[kStripWindows], own_shift[kStripWindows], mirror_shift[kStripWindows];
  __shared__ int64_t own_offset[kStripWindows], mirror_offset[kStripWindows];
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int chunks = (n_k + kBlochKChunk - 1) / kBlochKChunk;
  if ((int)blockIdx.x < lead) {
    const int item = (int)blockIdx.x * (kStripThreads / 32) + warp;
    if (blockIdx.y == 0 && item < n_others * chunks)
      window_sums<V>(others[item / chunks], lane, item % chunks * kBlochKChunk, n_k, group, gdst,
                     gmem, moff, msh, hv, sv, phases, n_shifts, nnz, hout, sout);
    return;
  }
  const int2 st = strips[blockIdx.x - lead];
  const int nw = st.y - st.x;
  if (warp == 0) {
    // window tables: one lane per window, prefix sums by shuffles
    int4 gi = make_int4(0, 0, 0, 0);
    if (lane < nw) gi = group[st.x + lane];
    int cols = gi.y, values = gi.x * gi.y;
#pragma unroll
    for (int o = 1; o < kStripWindows; o *= 2) {
      const int c = __shfl_up_sync(0xffffffffu, cols, o), v = __shfl_up_sync(0xffffffffu, values, o);
      if (lane >= o) {
        cols += c;
        values += v;
      }
    }
    if (lane < nw) {
      first_column[lane] = cols - gi.y;
      first_value[lane] = values - gi.x * gi.y;
      widths[lane] = gi.y;
      mirrors[lane] = gi.w;
      const int own = gmem[st.x + lane].x, mir = gmem[gi.w].x;
      own_shift[lane] = msh[own];
      mirror_shift[lane] = msh[mir];
      own_offset[lane] = moff[own];
      mirror_offset[lane] = moff[mir];
      if (lane == nw - 1) first_column[nw] = cols;
    }
  }
  __syncthreads();
  const int4 g0 = group[st.x];
  const int nr = g0.x, rl = g0.z;
  if (warp < nw) {
    const int ne = nr * widths[warp], v0 = first_value[warp];
    const int64_t own = own_offset[warp], mir = mirror_offset[warp];
    for (int e = lane; e < ne; e += 32) {
      const V* src[4] = {hv + own + e, sv + own + e, hv + mir + e, sv + mir + e};
#pragma unroll
      for (int t = 0; t < 4; ++t)
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(
                         (uint32_t)__cvta_generic_to_shared(&vals[t / 2][t % 2][v0 + e])),
                     "l"(src[t]), "n"(sizeof(V))
                     : "memory");
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  // this thread's column: window, column in it, its value arrays
  constexpr int kRowLanes = kStripThreads / kStripColumns;
  const int col = threadIdx.x % kStripColumns, a0 = threadIdx.x / kStripColumns;
  if (col >= first_column[nw]) return;
  int w = 0;
  while (col >= first_column[w + 1]) ++w;
  const int c = col - first_column[w], nc = widths[w], g = st.x + w, gm = mirrors[w];
  const V* own = &vals[0][0][first_value[w]];
  const V* mir = &vals[1][0][first_value[w]];
  const int64_t at0 = gdst[st.x] + col;
  for (int chunk = blockIdx.y; chunk < chunks; chunk += gridDim.y) {
    const int k0 = chunk * kBlochKChunk, nk = min(n_k - k0, kBlochKChunk);
    const float2* ph0 = phases + (int64_t)k0 * n_shifts;
    float2 po[kBlochKChunk], pm[kBlochKChunk];
#pragma unroll
    for (int q = 0; q < kBlochKChunk; ++q) {
      po[q] = q < nk ? ph0[q * n_shifts + own_shift[w]] : make_float2(0.0f, 0.0f);
      pm[q] = q < nk ? ph0[q * n_shifts + mirror_shift[w]] : make_float2(0.0f, 0.0f);
    }
    for (int a = a0; a < nr; a += kRowLanes) {
      const bool lower = gm < g || (gm == g && a > c);
      const int64_t at = (int64_t)k0 * nnz + at0 + (int64_t)a * rl;
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const float2 vo = load_value<V>(own + m * kStripValues, a * nc + c);
        const float2 vm = load_value<V>(mir + m * kStripValues, c * nr + a);
        float2* out = (m == 0 ? hout : sout) + at;
#pragma unroll
        for (int q = 0; q < kBlochKChunk; ++q) {
          if (q < nk) {
            const float2 xo = cmul_rn(vo, po[q]), xm = cmul_rn(vm, pm[q]);
            const float2 mean = lower ? hermitian_mean(xm, xo) : hermitian_mean(xo, xm);
            float2 v = lower ? make_float2(mean.x, -mean.y) : mean;
            if (gm == g && a == c) v = make_float2(xo.x, 0.0f);
            out[q * nnz] = v;
          }
        }
      }
    }
  }
}

// Whether the strips of a bundle take the strip kernel for n_k points (the
// windows outside strips never do).  Strips cost a CTA with two barriers each
// and use as many of 128 column threads as they are wide, but read their blocks
// once and write whole rows.  They win where they are wide (13 orbitals: 8
// windows, 104 columns); with few windows on the chip, where a warp per window
// is bound by its own chain; where windows of one strip differ in size, which
// leaves warps idle; and with many k points, the more so the fewer values there
// are to load (complex blocks load twice as many).  us, a warp per window /
// strips, 1728 atoms, real: 5 orbitals, 4 k 130 / 200, 16 k 504 / 420; 10
// orbitals, 4 k 398 / 366; 512 atoms: 13 orbitals, 4 k 214 / 140; 20 orbitals,
// 4 k 474 / 445, complex 492 / 502; 36 atoms (252 neighbours): 20 orbitals, 4 k 22
// / 12; 216 atoms of 5, 14 and 25 orbitals, 4 k 154 / 95.  Over 1600 measured
// pairs of bundle and n_k the kernel taken is 1.3 % slower than the better one
// on average; strips for all of them were 8 %, windows 23 %.
bool strips_pay(const StripShape& s, bool complex_values, int n_k) {
  if (s.columns >= 88) return true;
  const bool uneven = s.uneven >= 1.5, several = s.per_strip >= 1.5;
  if (uneven && s.values >= 900) return true;
  if (s.windows <= 4000) {
    if (n_k <= 4) return s.values >= 500;
    if (n_k <= 16) return s.values >= (s.windows <= 1500 || uneven ? 500 : 1150);
    return n_k <= 32 && s.values >= 1150 && several;
  }
  if (n_k <= 4) return !complex_values && several && s.values >= (uneven ? 500 : 900);
  if (complex_values && n_k <= 8) return several && s.values >= (uneven ? 500 : 600);
  return s.values >= 350 || s.values <= 16 || (n_k >= 32 && !complex_values);
}

template <typename V>
void launch_sums(const aosb_bloch* b, const void* h_values, const void* s_values,
                 const void* phases, int n_k, void* h_out, void* s_out, cudaStream_t st) {
  const auto *hv = (const V*)h_values, *sv = (const V*)s_values;
  const auto* ph = (const float2*)phases;
  auto *ho = (float2*)h_out, *so = (float2*)s_out;
  const int64_t nsh = (int64_t)(b->shifts.size() / 3), strips = (int64_t)b->strips.size();
  const int64_t chunks = aosb::ceil_div(n_k, kBlochKChunk), others = (int64_t)b->others.size();
  aosb::count_launches(1);
  // The windows outside strips run beside them while they are a few (one in
  // fifty): a warp takes longer over one than a CTA over a strip.
  if (others * 50 <= b->n_groups && others * chunks < INT32_MAX / 2 &&
      strips_pay(b->shape, sizeof(V) == sizeof(float2), n_k)) {
    // A CTA goes through all k chunks with its blocks loaded once, unless the
    // strips alone leave SMs without eight CTAs.
    const int64_t share = std::min<int64_t>(chunks, std::max<int64_t>(1, 148 * 8 / strips));
    const int lead = (int)aosb::ceil_div(others * chunks, kStripThreads / 32);
    bloch_strips_kernel<V><<<dim3((unsigned)(lead + strips), (unsigned)share), kStripThreads, 0,
                             st>>>(b->d_strips, lead, (int)others, b->d_others, b->d_group,
                                   b->d_group_dst, b->d_group_members, b->d_member_off,
                                   b->d_member_shift, hv, sv, ph, nsh, b->nnz, n_k, ho, so);
    return;
  }
  const dim3 grid(aosb::ceil_div(b->n_groups, kWindowWarps), (unsigned)chunks);
  bloch_windows_kernel<V><<<grid, kWindowWarps * 32, 0, st>>>(
      b->n_groups, b->d_group, b->d_group_dst, b->d_group_members, b->d_member_off,
      b->d_member_shift, hv, sv, ph, nsh, b->nnz, n_k, ho, so);
}

}  // namespace

extern "C" {

int aosb_bloch_create(int64_t n_orbitals, int64_t n_atoms, const int64_t* atom_offsets,
                      int64_t n_blocks, const int32_t* row_atom, const int32_t* col_atom,
                      const int32_t* lattice_shift, const int64_t* block_offsets,
                      aosb_bloch_t** out, char* err, size_t cap) {
  if (out == nullptr || atom_offsets == nullptr || row_atom == nullptr || col_atom == nullptr ||
      lattice_shift == nullptr || block_offsets == nullptr)
    return aosb::set_error(err, cap, AOSB_ERR_NULL, "required pointer is null");
  *out = nullptr;
  if (n_orbitals <= 0 || n_atoms <= 0 || n_blocks <= 0 || atom_offsets[n_atoms] != n_orbitals)
    return aosb::set_error(err, cap, AOSB_ERR_DIMS, "invalid bundle dimensions");
  for (int64_t b = 0; b < n_blocks; ++b) {
    if (row_atom[b] < 0 || row_atom[b] >= n_atoms || col_atom[b] < 0 || col_atom[b] >= n_atoms)
      return aosb::set_error(err, cap, AOSB_ERR_ARGUMENT, "block %lld references an unknown atom",
                             (long long)b);
    const int64_t nr = atom_offsets[row_atom[b] + 1] - atom_offsets[row_atom[b]];
    const int64_t nc = atom_offsets[col_atom[b] + 1] - atom_offsets[col_atom[b]];
    if (block_offsets[b + 1] - block_offsets[b] != nr * nc)
      return aosb::set_error(err, cap, AOSB_ERR_ARGUMENT, "block %lld size mismatch", (long long)b);
  }
  auto* B = new aosb_bloch();
  B->n = n_orbitals;
  B->n_atoms = n_atoms;
  B->n_blocks = n_blocks;

  // Distinct lattice shifts, lexicographic (the order numpy.unique(axis=0) gives).
  std::vector<int64_t> sidx(n_blocks);
  std::iota(sidx.begin(), sidx.end(), 0);
  auto shift_less = [&](int64_t a, int64_t b) {
    for (int d = 0; d < 3; ++d) {
      int32_t x = lattice_shift[a * 3 + d], y = lattice_shift[b * 3 + d];
      if (x != y) return x < y;
    }
    return false;
  };
  std::stable_sort(sidx.begin(), sidx.end(), shift_less);
  B->block_shift.assign(n_blocks, 0);
  int32_t ns = -1;
  for (int64_t t = 0; t < n_blocks; ++t) {
    if (t == 0 || shift_less(sidx[t - 1], sidx[t])) {
      ++ns;
      for (int d = 0; d < 3; ++d) B->shifts.push_back(lattice_shift[sidx[t] * 3 + d]);
    }
    B->block_shift[sidx[t]] = ns;
  }

  // Groups: blocks sorted by (row atom, col atom), block order kept inside.
  std::vector<int64_t> order(n_blocks);
  std::iota(order.begin(), order.end(), 0);
  std::stable_sort(order.begin(), order.end(), [&](int64_t a, int64_t b) {
    if (row_atom[a] != row_atom[b]) return row_atom[a] < row_atom[b];
    return col_atom[a] < col_atom[b];
  });
  std::vector<int32_t> g_row, g_col;
  std::vector<int2> g_mem;
  std::vector<int64_t> m_off;
  std::vector<int32_t> m_shift;
  for (int64_t t = 0; t < n_blocks; ++t) {
    const int64_t b = order[t];
    if (t == 0 || row_atom[b] != row_atom[order[t - 1]] || col_atom[b] != col_atom[order[t - 1]]) {
      g_row.push_back(row_atom[b]);
      g_col.push_back(col_atom[b]);
      g_mem.push_back(make_int2((int)m_off.size(), (int)m_off.size()));
    }
    m_off.push_back(block_offsets[b]);
    m_shift.push_back(B->block_shift[b]);
    g_mem.back().y = (int)m_off.size();
  }
  const int64_t ng = (int64_t)g_row.size();
  B->n_groups = ng;
  // Row structure per atom.
  std::vector<int64_t> rowlen(n_atoms, 0), first_group(n_atoms + 1, ng);
  std::vector<int64_t> colpos(ng, 0);
  for (int64_t g = ng - 1; g >= 0; --g) first_group[g_row[g]] = g;
  for (int64_t a = n_atoms - 1; a >= 0; --a)
    if (first_group[a] == ng) first_group[a] = first_group[a + 1];
  for (int64_t g = 0; g < ng; ++g) {
    const int32_t i = g_row[g], j = g_col[g];
    colpos[g] = rowlen[i];
    rowlen[i] += atom_offsets[j + 1] - atom_offsets[j];
  }
  B->indptr.assign(n_orbitals + 1, 0);
  for (int64_t a = 0; a < n_atoms; ++a)
    for (int64_t r = atom_offsets[a]; r < atom_offsets[a + 1]; ++r)
      B->indptr[r + 1] = B->indptr[r] + rowlen[a];
  B->nnz = B->indptr[n_orbitals];
  if (B->nnz == 0) {
    delete B;
    return aosb::set_error(err, cap, AOSB_ERR_DIMS, "empty pattern");
  }
  B->indices.resize(B->nnz);
  for (int64_t g = 0; g < ng; ++g) {
    const int32_t i = g_row[g], j = g_col[g];
    for (int64_t r = atom_offsets[i]; r < atom_offsets[i + 1]; ++r) {
      int64_t p = B->indptr[r] + colpos[g];
      for (int64_t c = atom_offsets[j]; c < atom_offsets[j + 1]; ++c) B->indices[p++] = (int32_t)c;
    }
  }
  for (int64_t r = 0; r < n_orbitals; ++r)
    if (B->indptr[r + 1] == B->indptr[r]) {
      // Rows without entries are allowed by the reference pattern builder;
      // the solver rejects them later (missing diagonal).
    }
  // Mirror groups (Hermitian topology).
  std::vector<int4> g_info(ng);
  std::vector<int64_t> g_dst(ng);
  for (int64_t g = 0; g < ng; ++g) {
    const int32_t i = g_row[g], j = g_col[g];
    int64_t lo = first_group[j], hi = first_group[j + 1];
    int64_t m = -1;
    while (lo < hi) {
      int64_t mid = (lo + hi) / 2;
      if (g_col[mid] < i) lo = mid + 1; else hi = mid;
    }
    if (lo < first_group[j + 1] && g_col[lo] == i) m = lo;
    if (m < 0) {
      delete B;
      return aosb::set_error(err, cap, AOSB_ERR_TOPOLOGY, "operator topology is not Hermitian");
    }
    const int nr = (int)(atom_offsets[i + 1] - atom_offsets[i]);
    const int nc = (int)(atom_offsets[j + 1] - atom_offsets[j]);
    g_info[g] = make_int4(nr, nc, (int)rowlen[i], (int)m);
    g_dst[g] = B->indptr[atom_offsets[i]] + colpos[g];
  }
  B->n_members = (int64_t)m_off.size();
  // Strips of each row atom, of about equal window counts.
  StripShape& shape = B->shape;
  for (int64_t a = 0; a < n_atoms; ++a) {
    const int64_t lo = first_group[a], hi = first_group[a + 1];
    const int64_t most = std::max<int64_t>(1, (hi - lo + kStripWindows - 1) / kStripWindows);
    const int64_t even = (hi - lo + most - 1) / most;
    for (int64_t g = lo; g < hi;) {
      int64_t e = g, cols = 0, values = 0, largest = 0;
      while (e < hi && e - g < even) {
        const int4 w = g_info[e];
        const int64_t c = cols + w.y, v = values + (int64_t)w.x * w.y;
        const bool single = g_mem[e].y - g_mem[e].x == 1 && g_mem[w.w].y - g_mem[w.w].x == 1;
        if (!single || c > kStripColumns || v > kStripValues) break;
        largest = std::max<int64_t>(largest, v - values);
        cols = c;
        values = v;
        ++e;
      }
      if (e == g) {
        B->others.push_back((int32_t)g++);
        continue;
      }
      B->strips.push_back(make_int2((int)g, (int)e));
      shape.windows += (double)(e - g);
      shape.columns += (double)cols;
      shape.values += (double)values;
      if (values > 0) shape.uneven += (double)largest * (double)(e - g) / (double)values;
      g = e;
    }
  }
  if (!B->strips.empty()) {
    const double n = (double)B->strips.size();
    shape.per_strip = shape.windows / n;
    shape.columns /= n;
    shape.values /= n;
    shape.uneven /= n;
  }
  B->g_info = std::move(g_info);
  B->g_dst = std::move(g_dst);
  B->g_mem = std::move(g_mem);
  B->m_off = std::move(m_off);
  B->m_shift = std::move(m_shift);
  *out = B;
  return 0;
}

int aosb_bloch_upload(aosb_bloch_t* B, char* err, size_t cap) {
  if (B == nullptr) return aosb::set_error(err, cap, AOSB_ERR_NULL, "null handle");
  if (B->uploaded) return 0;
  int rc = 0;
  if ((rc = upload(&B->d_indptr, B->indptr, err, cap)) ||
      (rc = upload(&B->d_indices, B->indices, err, cap)) ||
      (rc = upload(&B->d_group, B->g_info, err, cap)) ||
      (rc = upload(&B->d_group_dst, B->g_dst, err, cap)) ||
      (rc = upload(&B->d_group_members, B->g_mem, err, cap)) ||
      (rc = upload(&B->d_member_off, B->m_off, err, cap)) ||
      (rc = upload(&B->d_member_shift, B->m_shift, err, cap)) ||
      (rc = upload(&B->d_strips, B->strips, err, cap)) ||
      (rc = upload(&B->d_others, B->others, err, cap)))
    return rc;
  int64_t values = 0;
  for (size_t g = 0; g < B->g_info.size(); ++g)
    values += (int64_t)B->g_info[g].x * B->g_info[g].y * (B->g_mem[g].y - B->g_mem[g].x);
  B->n_values = values;
  B->uploaded = true;
  return 0;
}

int aosb_bloch_info(const aosb_bloch_t* b, int64_t* nnz, int64_t* n_shifts) {
  if (b == nullptr) return AOSB_ERR_NULL;
  if (nnz) *nnz = b->nnz;
  if (n_shifts) *n_shifts = (int64_t)(b->shifts.size() / 3);
  return 0;
}

int aosb_bloch_export(const aosb_bloch_t* b, int64_t* indptr, int32_t* indices, int32_t* shifts,
                      int32_t* block_shift) {
  if (b == nullptr) return AOSB_ERR_NULL;
  if (indptr) std::copy(b->indptr.begin(), b->indptr.end(), indptr);
  if (indices) std::copy(b->indices.begin(), b->indices.end(), indices);
  if (shifts) std::copy(b->shifts.begin(), b->shifts.end(), shifts);
  if (block_shift) std::copy(b->block_shift.begin(), b->block_shift.end(), block_shift);
  return 0;
}

int aosb_bloch_export_groups(const aosb_bloch_t* b, int64_t* n_groups, int64_t* n_members,
                             int32_t* group_info, int64_t* group_dst, int32_t* group_members,
                             int64_t* member_off, int32_t* member_shift) {
  if (b == nullptr) return AOSB_ERR_NULL;
  if (n_groups) *n_groups = (int64_t)b->g_info.size();
  if (n_members) *n_members = (int64_t)b->m_off.size();
  for (size_t g = 0; g < b->g_info.size(); ++g) {
    if (group_info) {
      group_info[4 * g] = b->g_info[g].x;
      group_info[4 * g + 1] = b->g_info[g].y;
      group_info[4 * g + 2] = b->g_info[g].z;
      group_info[4 * g + 3] = b->g_info[g].w;
    }
    if (group_dst) group_dst[g] = b->g_dst[g];
    if (group_members) {
      group_members[2 * g] = b->g_mem[g].x;
      group_members[2 * g + 1] = b->g_mem[g].y;
    }
  }
  if (member_off) std::copy(b->m_off.begin(), b->m_off.end(), member_off);
  if (member_shift) std::copy(b->m_shift.begin(), b->m_shift.end(), member_shift);
  return 0;
}

int aosb_bloch_device_pattern(const aosb_bloch_t* b, const int64_t** indptr,
                              const int32_t** indices) {
  if (b == nullptr) return AOSB_ERR_NULL;
  if (!b->uploaded) return AOSB_ERR_ARGUMENT;
  if (indptr) *indptr = b->d_indptr;
  if (indices) *indices = b->d_indices;
  return 0;
}

int aosb_bloch_apply(const aosb_bloch_t* b, int32_t value_kind, const void* h_values,
                     const void* s_values, const aosb_complex64* phases, int32_t n_k,
                     aosb_complex64* h_out, aosb_complex64* s_out, void* stream, char* err,
                     size_t cap) {
  if (b == nullptr || h_values == nullptr || s_values == nullptr || phases == nullptr ||
      h_out == nullptr || s_out == nullptr)
    return aosb::set_error(err, cap, AOSB_ERR_NULL, "required pointer is null");
  if (!b->uploaded)
    return aosb::set_error(err, cap, AOSB_ERR_ARGUMENT, "call aosb_bloch_upload first");
  if (n_k <= 0 || n_k > 65535)
    return aosb::set_error(err, cap, AOSB_ERR_ARGUMENT, "n_k must be in 1..65535");
  if (value_kind != 0 && value_kind != 1)
    return aosb::set_error(err, cap, AOSB_ERR_ARGUMENT, "value_kind must be 0 or 1");
  cudaStream_t st = (cudaStream_t)stream;
  cudaEvent_t ev[2];
  const bool timed = aosb::timing_begin(st, ev);
  if (value_kind == 0)
    launch_sums<float>(b, h_values, s_values, phases, n_k, h_out, s_out, st);
  else
    launch_sums<float2>(b, h_values, s_values, phases, n_k, h_out, s_out, st);
  // algorithmic bytes: the stored H and S block values read once per launch,
  // the complex64 H(k) and S(k) CSR values written once per k point
  if (timed)
    aosb::timing_end(aosb::kTimedBloch, st, ev, 0.0,
                     (double)b->n_values * 2.0 * (value_kind ? 8.0 : 4.0) +
                         (double)n_k * (double)b->nnz * 2.0 * 8.0);
  return aosb::launch_check(err, cap, "bloch sums");
}

void aosb_bloch_destroy(aosb_bloch_t* b) {
  if (b == nullptr) return;
  cudaFree(b->d_indptr);
  cudaFree(b->d_indices);
  cudaFree(b->d_group);
  cudaFree(b->d_group_dst);
  cudaFree(b->d_group_members);
  cudaFree(b->d_member_off);
  cudaFree(b->d_member_shift);
  cudaFree(b->d_strips);
  cudaFree(b->d_others);
  delete b;
}

}  // extern "C"
