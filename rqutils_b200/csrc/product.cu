// Product-subspace layout of the cached matvec (cache_strategy (1, 2)).
//
// SQD subspaces are usually the Cartesian product of strings on the high half of the qubits
// (beta) and strings on the low half (alpha).  Sorted, row r = h * nl + l holds H[h] | L[l].
// The stored pairs of a row come in three classes (k_gpre_flags, operator.cu;
// lists of the halves' partners: connect.cu):
//   H: x on the high half only, source (h', l) with H[h'] = H[h] ^ x.  Every row of slab h has
//      the same H sources in the same order;
//   L: the diagonal group and x on the low half only, source (h, l') with L[l'] = L[l] ^ x.
//      Every row with low string l has the same L sources in the same order;
//   M: the rest (both halves change).
// An H or L source is implied by (slab, position), so the elements of those pairs are laid out
// again as dense slabs and the matvec streams them with coalesced loads and gathers v (or its
// transpose vT[l][h]) with coalesced loads too, instead of one scattered gather and one index
// per pair.  One matvec is five launches:
//   1. vT = transpose(v)                                (32 x 32 tiles through shared memory)
//   2. t2[l][h] = sum_e VL(lo[l] + e, h) vT[l'_e][h]     (L part; FP64 partial)
//   3. t2' = transpose(t2) into the vT buffer           (now [h][l])
//   4. t3[r] = sum of the row's M pairs                  (FP64 partial; see below)
//   5. out[h][l] = t2'[h][l] + t3[r] + sum_k VH(ho[h] + k, l) v[h'_k][l]
// Steps 2 and 5 are one kernel (k_slab) over an A x B grid of outputs (A slabs of B rows each,
// A = nh for H, A = nl for L): a warp owns one slab a and 32 consecutive b (one "panel"), a
// block 8 slabs of the same panel, and blocks run panel-major, so the 32-wide panel of the
// gathered vector stays in L2 while all slabs pass over it.  The elements are stored in the
// same panel-major order, VH(k, l) at ((l / 32) * KH + k) * 32 + l % 32 (KH = entries of all
// slabs), so the element stream of a panel pass is one contiguous sweep.  Source indices are
// kept premultiplied (h' * nl, l' * nh).  At 48 qubits the FP64 passes stream their elements
// at ~5 TB/s while L2 serves one amplitude per entry (~19 TB/s).  The FP32 copies of the slabs
// of even-sized halves use 64-wide panels, read by k_slab2 with two adjacent positions per
// lane (paired 16-byte amplitude loads).
// Step 4: SQD_LAYOUT_PRODUCT reads the M pairs in panels (k_tail_panels: no source per pair, the
// gathered row of v in shared memory) when most combinations of the halves' partners exist;
// otherwise, and under SQD_LAYOUT_PRODUCT_CSR, the CSR kernel runs over the row tails, gathering
// from global memory: from a contiguous copy of the tails (row offsets, elements, source rows)
// when they average at most kCompactTailMax pairs per row, else inside the rows' pair lists.
// FP32 vectors keep the compensated accumulation in every part and pass partials in FP64, so
// the result is rounded once.  The elements are the same numbers as in the CSR arrays; only
// the summation order of a row changes (L and M pairs before H pairs).
#include <cstdlib>
#include <algorithm>
#include <climits>
#include <type_traits>
#include <vector>

#include "internal.cuh"
#include "dispatch.cuh"
#include "accum.cuh"

namespace sqd {
namespace {

// Source offsets of the slabs from the halves' partner lists: hsrc[k] = h' * nl over the H lists,
// lsrc[e] = l' * nh over the L lists, each low string's diagonal entry (d) first; lo with those
// diagonal entries counted.
__global__ void k_slab_sources(PlanView c, int64_t th, uint32_t* hsrc, int64_t* lo,
                               uint32_t* lsrc) {
  const int64_t t0 = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  const int64_t step = int64_t(gridDim.x) * blockDim.x;
  for (int64_t k = t0; k < th; k += step) hsrc[k] = static_cast<uint32_t>(c.part[k] * c.nl);
  const int64_t l0 = c.loff[0];
  for (int64_t l = t0; l <= c.nl; l += step) {
    int64_t e = c.loff[l] - l0 + c.d * l;
    lo[l] = e;
    if (l == c.nl) continue;
    if (c.d) lsrc[e++] = static_cast<uint32_t>(l * c.nh);
    for (int64_t i = c.loff[l]; i < c.loff[l + 1]; ++i)
      lsrc[e++] = static_cast<uint32_t>(c.part[i] * c.nh);
  }
}

__global__ void k_to_float32(const double* __restrict__ in, float* __restrict__ out, int64_t n) {
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x)
    out[i] = static_cast<float>(in[i]);
}

// A vector element as it is copied.
template <typename R, int NC>
struct RawOf {
  using type = std::conditional_t<sizeof(R) == 8, double2, float2>;
};
template <typename R>
struct RawOf<R, 1> {
  using type = R;
};
struct __align__(16) Double4 {
  double2 a, b;
};
template <typename R>
struct RawOf<R, 4> {
  using type = Double4;
};
template <typename R, int NC>
using Raw = typename RawOf<R, NC>::type;

// out[c][r] = in[r][c] for an rows x cols matrix of elements E (32 x 32 tiles, 256 threads).
template <typename E>
__global__ void __launch_bounds__(256)
k_transpose(const E* __restrict__ in, E* __restrict__ out, int64_t rows, int64_t cols) {
  __shared__ E tile[32][33];
  const int64_t tr = (rows + 31) / 32, tc = (cols + 31) / 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (int64_t t = blockIdx.x; t < tr * tc; t += gridDim.x) {
    const int64_t r0 = (t / tc) * 32, c0 = (t % tc) * 32;
    for (int i = ty; i < 32; i += 8) {
      const int64_t r = r0 + i, c = c0 + tx;
      if (r < rows && c < cols) tile[i][tx] = in[r * cols + c];
    }
    __syncthreads();
    for (int i = ty; i < 32; i += 8) {
      const int64_t c = c0 + i, r = r0 + tx;
      if (c < cols && r < rows) out[c * rows + r] = tile[tx][i];
    }
    __syncthreads();
  }
}

// One slab pass over an A x B grid: element (a, b) accumulates VS(k, b) * x[src[k] + b] over
// k in [off[a], off[a + 1]) (VS panel-major over total_k entries, src premultiplied).  Warp =
// one slab a and a 32-wide panel of b; block = 8 slabs of one panel; blocks panel-major.
//   FINAL = false: store the FP64 partial at out_part[a * B + b];
//   FINAL = true:  start from part_t[a * B + b] (+ part_m[a * B + b] when HAS_M) and store the
//                  result at out[a * B + b].
// Eight entries per step keep eight independent index -> amplitude chains in flight.
template <typename R, int NCV, int NCA, bool FINAL, bool HAS_M>
__device__ __forceinline__ void
slab_block(int64_t blk, int64_t A, int64_t B, int64_t total_k, int64_t a_tiles,
           const int64_t* __restrict__ off, const uint32_t* __restrict__ src,
           const R* __restrict__ V, const R* __restrict__ x, const double* __restrict__ part_t,
           const double* __restrict__ part_m, R* __restrict__ out, double* __restrict__ out_part,
           int prefetch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // A step's elements are one contiguous chunk of 8 x 32 entries (2 or 4 KB).  The chunk about
  // 2 KB ahead is prefetched into L2, one 128-byte line per lane, so the element loads wait on
  // L2 rather than on DRAM (measured: C3 FP64 matvec 5.9 -> 5.1 ms, C2 0.370 -> 0.324 ms; 4 KB
  // ahead was slightly slower, 8 KB no better than none).
  constexpr int U = NCV == 4 ? 4 : 8;   // entries per step; four when an amplitude is 32 bytes
  constexpr int kChunkLines = U * 32 * NCA * static_cast<int>(sizeof(R)) / 128;
  constexpr int pv = kChunkLines >= 16 ? 1 : 16 / kChunkLines;   // steps ahead
  const int64_t p = blk / a_tiles;
  const int64_t a = (blk - p * a_tiles) * 8 + warp;
  const int64_t b = p * 32 + lane;
  if (a < A && b < B) {
    CAcc<R, NCV, NCA> acc;
    if constexpr (FINAL) {
      acc.add_partial(part_t, a * B + b);
      if constexpr (HAS_M) acc.add_partial(part_m, a * B + b);
    }
    const int64_t k1 = __ldg(off + a + 1);
    int64_t k = __ldg(off + a);
    const R* vp = V + ((p * total_k + k) * 32 + lane) * NCA;
    for (; k + U - 1 < k1; k += U) {
      // prefetch: the next step's source offsets (one 32-byte sector) into L1 ahead of use
      if (prefetch && k + 2 * U - 1 < k1)
        asm volatile("prefetch.global.L1 [%0];" ::"l"(src + k + U));
      if (lane < kChunkLines && k + U * pv + U - 1 < k1)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(
            reinterpret_cast<const char*>(vp - lane * NCA + U * 32 * NCA * pv) + lane * 128));
      uint32_t si[U];
#pragma unroll
      for (int u = 0; u < U; ++u) si[u] = __ldg(src + k + u);
      Cx<R> m[U];
      Elem<R, NCV> xv[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        m[u] = ld_elem<R, NCA>(vp, 32 * u);
        xv[u] = ld_elem<R, NCV>(x, int64_t(si[u]) + b);
      }
#pragma unroll
      for (int u = 0; u < U; u += 4) acc.add4(m + u, xv + u);
      vp += U * 32 * NCA;
    }
    // remainder: one entry at a time (a predicated eight-entry step measured 5-11 % slower
    // for FP64 at 32 and 48 qubits)
    for (; k < k1; ++k) {
      acc.add(ld_elem<R, NCA>(vp, 0), ld_elem<R, NCV>(x, int64_t(__ldg(src + k)) + b));
      vp += 32 * NCA;
    }
    if constexpr (FINAL) acc.store(out, a * B + b);
    else acc.store_partial(out_part, a * B + b);
  }
}

// Blocks per SM that the register counts have to leave room for: the passes wait on their loads, and
// one block less costs about 10 % (3072 x 2816 strings: complex64 final pass 461 -> 515 us at 50
// instead of 48 registers).
template <typename R, int NCV, int NCA, bool FINAL, bool HAS_M>
__global__ void __launch_bounds__(256, NCV == 4 || NCA == 2 ? 4 : 6)
k_slab(int64_t A, int64_t B, int64_t total_k, int64_t a_tiles, const int64_t* __restrict__ off,
       const uint32_t* __restrict__ src, const R* __restrict__ V, const R* __restrict__ x,
       const double* __restrict__ part_t, const double* __restrict__ part_m, R* __restrict__ out,
       double* __restrict__ out_part, int prefetch) {
  slab_block<R, NCV, NCA, FINAL, HAS_M>(blockIdx.x, A, B, total_k, a_tiles, off, src, V, x, part_t,
                                        part_m, out, out_part, prefetch);
}

// FP32 slabs in 64-wide panels: a lane owns two adjacent positions b, b + 1, so one 16-byte
// (complex64) or 8-byte (float) load reads both amplitudes and one 8- or 16-byte load both
// elements; four entries per step.  Same sums per position as k_slab (FMA chains of four
// products into the compensated sums).  VEC: x and out allow the paired vector accesses
// (source offsets and B even, pointers aligned), else each position is read on its own.
template <typename R, int NCA>
__device__ __forceinline__ void pair_elem(const R* p, Cx<R>& e0, Cx<R>& e1) {
  if constexpr (NCA == 2) {
    const float4 v = __ldg(reinterpret_cast<const float4*>(p));
    e0 = cx_make<R>(v.x, v.y);
    e1 = cx_make<R>(v.z, v.w);
  } else {
    const float2 v = __ldg(reinterpret_cast<const float2*>(p));
    e0 = cx_make<R>(v.x, R(0));
    e1 = cx_make<R>(v.y, R(0));
  }
}

template <typename R, int NCV, bool VEC>
__device__ __forceinline__ void pair_vec(const R* x, int64_t i, Cx<R>& v0, Cx<R>& v1) {
  if constexpr (VEC && NCV == 2) {
    const float4 v = __ldg(reinterpret_cast<const float4*>(x + 2 * i));
    v0 = cx_make<R>(v.x, v.y);
    v1 = cx_make<R>(v.z, v.w);
  } else if constexpr (VEC) {
    const float2 v = __ldg(reinterpret_cast<const float2*>(x + i));
    v0 = cx_make<R>(v.x, R(0));
    v1 = cx_make<R>(v.y, R(0));
  } else {
    v0 = ld_elem<R, NCV>(x, i);
    v1 = ld_elem<R, NCV>(x, i + 1);
  }
}

template <typename R, int NCV, int NCA, bool FINAL, bool HAS_M, bool VEC>
__device__ __forceinline__ void
slab2_block(int64_t blk, int64_t A, int64_t B, int64_t total_k, int64_t a_tiles,
            const int64_t* __restrict__ off, const uint32_t* __restrict__ src,
            const R* __restrict__ V, const R* __restrict__ x, const double* __restrict__ part_t,
            const double* __restrict__ part_m, R* __restrict__ out,
            double* __restrict__ out_part) {
  static_assert(sizeof(R) == 4, "two positions per lane: FP32 slabs");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // element chunk of a step (4 x 64 entries, 1 or 2 KB) prefetched into L2 about 2 KB ahead,
  // as in k_slab (C3 FP32 matvec 3.32 -> 2.78 ms, C2 0.234 -> 0.210 ms; 1 KB ahead: 2.95 ms);
  // in the first pass only: the final pass, which also reads both FP64 partials, measured
  // slower with it (c3_small 90.5 -> 104.9 us, C3 1171 -> 1295 us)
  constexpr int kChunkLines = FINAL ? 0 : 4 * 64 * NCA * static_cast<int>(sizeof(R)) / 128;
  constexpr int pv = kChunkLines >= 16 ? 1 : kChunkLines > 0 ? 16 / kChunkLines : 1;
  const int64_t p = blk / a_tiles;
  const int64_t a = (blk - p * a_tiles) * 8 + warp;
  const int64_t b = p * 64 + 2 * lane;  // positions b and b + 1 (B is even)
  if (a < A && b < B) {
    CAcc<R, NCV, NCA> acc0, acc1;
    if constexpr (FINAL) {
      acc0.add_partial(part_t, a * B + b);
      acc1.add_partial(part_t, a * B + b + 1);
      if constexpr (HAS_M) {
        acc0.add_partial(part_m, a * B + b);
        acc1.add_partial(part_m, a * B + b + 1);
      }
    }
    const int64_t k1 = __ldg(off + a + 1);
    int64_t k = __ldg(off + a);
    const R* vp = V + ((p * total_k + k) * 64 + 2 * lane) * NCA;
    for (; k + 3 < k1; k += 4) {
      if (lane < kChunkLines && k + 4 * pv + 3 < k1)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(
            reinterpret_cast<const char*>(vp - 2 * lane * NCA + 4 * 64 * NCA * pv) + lane * 128));
      uint32_t si[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) si[u] = __ldg(src + k + u);
      Cx<R> m0[4], m1[4], x0[4], x1[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        pair_elem<R, NCA>(vp + 64 * NCA * u, m0[u], m1[u]);
        pair_vec<R, NCV, VEC>(x, int64_t(si[u]) + b, x0[u], x1[u]);
      }
      acc0.add4(m0, x0);
      acc1.add4(m1, x1);
      vp += 4 * 64 * NCA;
    }
    // remainder (fewer than four entries): one predicated step
    if (k < k1) {
      uint32_t si[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) si[u] = (k + u < k1) ? __ldg(src + k + u) : 0u;
      Cx<R> m0[4], m1[4], x0[4], x1[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (k + u < k1) {
          pair_elem<R, NCA>(vp + 64 * NCA * u, m0[u], m1[u]);
          pair_vec<R, NCV, VEC>(x, int64_t(si[u]) + b, x0[u], x1[u]);
        } else {
          m0[u] = m1[u] = x0[u] = x1[u] = cx_make<R>(R(0), R(0));
        }
      }
      acc0.add4(m0, x0);
      acc1.add4(m1, x1);
    }
    if constexpr (FINAL) {
      if constexpr (VEC && NCV == 2) {
        reinterpret_cast<float4*>(out)[(a * B + b) >> 1] =
            make_float4(acc0.re.value(), acc0.im.value(), acc1.re.value(), acc1.im.value());
      } else if constexpr (VEC) {
        reinterpret_cast<float2*>(out)[(a * B + b) >> 1] =
            make_float2(acc0.re.value(), acc1.re.value());
      } else {
        st_elem<R, NCV>(out, a * B + b, cx_make<R>(acc0.re.value(), acc0.im.value()));
        st_elem<R, NCV>(out, a * B + b + 1, cx_make<R>(acc1.re.value(), acc1.im.value()));
      }
    } else {
      acc0.store_partial(out_part, a * B + b);
      acc1.store_partial(out_part, a * B + b + 1);
    }
  }
}

template <typename R, int NCV, int NCA, bool FINAL, bool HAS_M, bool VEC>
__global__ void __launch_bounds__(256, NCA == 2 ? 4 : NCV == 2 ? 5 : 6)
k_slab2(int64_t A, int64_t B, int64_t total_k, int64_t a_tiles, const int64_t* __restrict__ off,
        const uint32_t* __restrict__ src, const R* __restrict__ V, const R* __restrict__ x,
        const double* __restrict__ part_t, const double* __restrict__ part_m, R* __restrict__ out,
        double* __restrict__ out_part) {
  slab2_block<R, NCV, NCA, FINAL, HAS_M, VEC>(blockIdx.x, A, B, total_k, a_tiles, off, src, V, x,
                                              part_t, part_m, out, out_part);
}

// M pairs of every row, FP64 partial per row.  Same schedule as the CSR matvec: LPR lanes per
// row, interleaved or chunked rows.  The pairs are the row's CSR tail after its H and L entries
// (row_ptr, cols, vals: the operator's arrays; ho, lo give the H and L counts) or, COMPACT, the
// contiguous copy of the tails (row_ptr = mptr, cols = mcol, vals = mval; ho, lo unused).
template <typename R, int NCV, int NCA, int LPR, bool COMPACT>
__global__ void __launch_bounds__(256)
k_mv_mixed(const int64_t* __restrict__ row_ptr, const uint32_t* __restrict__ cols,
           const R* __restrict__ vals, const R* __restrict__ v, const int64_t* __restrict__ ho,
           const int64_t* __restrict__ lo, int64_t nl, double* __restrict__ part,
           int64_t n_rows, int64_t chunk) {
  constexpr int RPW = 32 / LPR;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int sub = lane % LPR, slot = lane / LPR;
  auto one_step = [&](int64_t rb, int64_t lim) {
    const int64_t row = rb + slot;
    CAcc<R, NCV, NCA> acc;
    if (row < lim) {
      int64_t b = __ldg(row_ptr + row);
      const int64_t e = __ldg(row_ptr + row + 1);
      if constexpr (!COMPACT) {
        const int64_t h = row / nl, l = row - h * nl;
        b += (__ldg(ho + h + 1) - __ldg(ho + h)) + (__ldg(lo + l + 1) - __ldg(lo + l));
      }
      csr_row_dot<R, NCV, NCA, LPR>(cols, vals, v, b + sub, e, acc);
    }
    acc.merge(LPR);
    if (sub == 0 && row < lim) acc.store_partial(part, row);
  };
  if (chunk <= 0) {
    const int64_t w0 = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5;
    const int64_t nw = (int64_t(gridDim.x) * blockDim.x) >> 5;
    for (int64_t rb = w0 * RPW; rb < n_rows; rb += nw * RPW) one_step(rb, n_rows);
  } else {
    const int nwb = blockDim.x >> 5;
    for (int64_t c0 = int64_t(blockIdx.x) * chunk; c0 < n_rows; c0 += int64_t(gridDim.x) * chunk) {
      const int64_t lim = min(c0 + chunk, n_rows);
      for (int64_t rb = c0 + int64_t(warp) * RPW; rb < lim; rb += int64_t(nwb) * RPW)
        one_step(rb, lim);
    }
  }
}

// ---- M pairs in panels -------------------------------------------------------------------
// A row's two-half sources are A(h) x B(l) (connect.cu): h' from the high string alone, l' from
// the low string alone.  So no source is stored per pair: for a fixed A entry (h, h') the sources
// lie in one row of v, nl amplitudes that a block stages in shared memory, at positions that are
// the same for every A entry (panel_src, kept in L1).  A lane owns one low string and keeps its
// sum over all A entries, and the elements of 32 low strings are one 256-byte line per step.
// Low strings are sorted by the length of their lists, so the lanes of a panel end together; high
// strings run longest A list first, so that the last blocks are short.
// Bound by the element stream (DRAM) and the shared-memory gathers, about 10 wavefronts per 32
// complex128 amplitudes.  32 qubits, 512 x 512 strings, 49.6 M pairs: 117 us complex128, 79 us
// complex64 (285 us with all source slabs of a high string in shared memory and 32 lanes per row,
// about 170 us at its best with 16 lanes from the pair list); 48 qubits, 3072 x 2816, 48 M
// pairs, complex64: 0.20 ms (1.87 ms with 32 lanes per row).
constexpr unsigned kAbsent64 = 0x7ff8deadu;   // high word of an absent element (a NaN)
constexpr unsigned kAbsent32 = 0x7fc0deadu;
constexpr int kPanelMaxWarps = 32, kPanelMaxPerWarp = 4;
constexpr size_t kPanelSmem = 200 * 1024;

__device__ __forceinline__ bool is_absent(double re) {
  return static_cast<unsigned>(__double2hiint(re)) == kAbsent64;
}
__device__ __forceinline__ bool is_absent(float re) { return __float_as_uint(re) == kAbsent32; }

__device__ __forceinline__ int64_t tail_begin(const int64_t* row_ptr, const int64_t* ho,
                                              const int64_t* lo, int64_t r, int64_t nl) {
  const int64_t h = r / nl, l = r - h * nl;
  return row_ptr[r] + (ho[h + 1] - ho[h]) + (lo[l + 1] - lo[l]);
}

// Source positions of the panels' steps (B entry t of the lane's low string, nl in the padding).
__global__ void k_panel_src(PlanView c, const int32_t* __restrict__ at,
                            const uint32_t* __restrict__ perm, int64_t panels, uint16_t* src) {
  const int lane = threadIdx.x & 31;
  const int64_t w0 = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5;
  const int64_t nw = (int64_t(gridDim.x) * blockDim.x) >> 5;
  for (int64_t p = w0; p < panels; p += nw) {
    const uint32_t l = perm[p * 32 + lane];
    const int64_t b0 = l < c.nl ? c.boff[l] : 0, b1 = l < c.nl ? c.boff[l + 1] : 0;
    for (int32_t t = 0; t < at[p + 1] - at[p]; ++t)
      src[(int64_t(at[p]) + t) * 32 + lane] =
          static_cast<uint16_t>(b0 + t < b1 ? c.part[b0 + t] : static_cast<uint32_t>(c.nl));
  }
}

// Elements from the pair list: a warp is one high string and one panel; every lane walks its
// row's tail, whose order is A(h) x B(l) without the absent groups.
template <int NCA>
__global__ void __launch_bounds__(256)
k_panel_fill(PlanView c, const int64_t* __restrict__ row_ptr, const double* __restrict__ vals,
             const int64_t* __restrict__ ho, const int64_t* __restrict__ lo,
             const int32_t* __restrict__ at, const uint32_t* __restrict__ perm, int64_t panels,
             int64_t steps, int full, double* vm, float* vm32) {
  const int lane = threadIdx.x & 31;
  const int64_t w0 = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5;
  const int64_t nw = (int64_t(gridDim.x) * blockDim.x) >> 5;
  const int64_t a_first = c.aoff[0];
  const double gone = __hiloint2double(static_cast<int>(kAbsent64), 0);
  for (int64_t w = w0; w < c.nh * panels; w += nw) {
    const int64_t h = w / panels, p = w - h * panels;
    const uint32_t l = perm[p * 32 + lane];
    const bool live = l < c.nl;
    const int64_t b0 = live ? c.boff[l] : 0, b1 = live ? c.boff[l + 1] : 0;
    int64_t i = live ? tail_begin(row_ptr, ho, lo, h * c.nl + l, c.nl) : 0;
    const int32_t t0 = at[p], len = at[p + 1] - t0;
    for (int64_t k = c.aoff[h]; k < c.aoff[h + 1]; ++k) {
      const uint32_t a = __ldg(c.key + k);
      for (int32_t t = 0; t < len; ++t) {
        const bool there = b0 + t < b1 && plan_group(c, a, __ldg(c.key + b0 + t)) >= 0;
        const int64_t q = ((k - a_first) * steps + t0 + t) * 32 + lane;
        double re = full ? 0.0 : gone, im = 0.0;   // full: only the padding, a zero
        if (there) {
          const Cx<double> el = ld_elem<double, NCA>(vals, i++);
          re = el.re;
          im = el.im;
        }
        if (vm) {
          if constexpr (NCA == 2) reinterpret_cast<double2*>(vm)[q] = make_double2(re, im);
          else vm[q] = re;
        }
        if (vm32) {
          const float fr = there || full ? static_cast<float>(re) : __uint_as_float(kAbsent32);
          if constexpr (NCA == 2)
            reinterpret_cast<float2*>(vm32)[q] = make_float2(fr, static_cast<float>(im));
          else
            vm32[q] = fr;
        }
      }
    }
  }
}

// Bytes of a staged row of nl elements and the zero behind it.
__host__ __device__ __forceinline__ int64_t panel_row(int64_t nl, int element_bytes) {
  return ((nl + 1) * element_bytes + 15) / 16 * 16;
}

template <int BYTES>
__device__ __forceinline__ void copy_async(void* smem, const void* global) {
  const unsigned dst = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(global));
  else if constexpr (BYTES == 8)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(global));
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(global));
}

template <typename R, int NC>
__device__ __forceinline__ Elem<R, NC> sm_elem(const R* p, int64_t i) {
  if constexpr (NC == 4) {
    return Cx2<R>{sm_elem<R, 2>(p, 2 * i), sm_elem<R, 2>(p, 2 * i + 1)};
  } else if constexpr (NC == 2) {
    if constexpr (sizeof(R) == 8) {
      const double2 d = reinterpret_cast<const double2*>(p)[i];
      return cx_make<R>(d.x, d.y);
    } else {
      const float2 d = reinterpret_cast<const float2*>(p)[i];
      return cx_make<R>(d.x, d.y);
    }
  } else {
    return cx_make<R>(p[i], R(0));
  }
}

// M pairs of one high string, chunk `blockIdx % chunks` of its panels: FP64 partials.  Up to four
// A entries at a time: their rows of v are staged together (STAGED; rows too long for shared
// memory are gathered from global memory), then every step of a panel loads its source position
// once and one element per A entry, four independent 256-byte lines, and one barrier pair serves
// four entries (one entry at a time spent a third of its time at barriers and in the chain
// position -> amplitude: 202 us at 512 x 512 strings, 32 qubits, complex128).  Each step's lines
// are prefetched into L2 six steps ahead (900 x 800 strings: 890 -> 739 us).  Six blocks per SM for
// the narrow forms cap the registers at 42.
constexpr int kPanelGroup = 4;
constexpr int kPanelAhead = 6;

struct PanelArgs {
  const int32_t* at;
  const uint32_t* perm;
  const uint16_t* src;
  const uint32_t* horder;
  int panels, steps, chunks, group;
};

template <typename R, int NCV, int NCA, int P, bool STAGED, bool FULL>
__device__ __forceinline__ void
panel_block(int blk, const PlanView& c, const PanelArgs& q, const R* __restrict__ vm,
            const R* __restrict__ v, double* __restrict__ part) {
  const int32_t* __restrict__ at = q.at;
  const uint32_t* __restrict__ perm = q.perm;
  const uint16_t* __restrict__ src = q.src;
  const uint32_t* __restrict__ horder = q.horder;
  const int panels = q.panels, steps = q.steps, chunks = q.chunks, group = q.group;
  extern __shared__ __align__(16) unsigned char panel_raw[];
  constexpr int EB = static_cast<int>(sizeof(R)) * NCV;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, W = blockDim.x >> 5;
  const int at_h = blk / chunks, chunk = blk - at_h * chunks;
  const int h = __ldg(horder + at_h);
  const int nl = static_cast<int>(c.nl);
  const int64_t a_first = __ldg(c.aoff);
  const int64_t k0 = __ldg(c.aoff + h);
  const int nk = static_cast<int>(__ldg(c.aoff + h + 1) - k0);
  const uint32_t* part_h = c.part + k0;
  const int row = panel_row(nl, EB) / static_cast<int>(sizeof(R));          // staged row, in R
  R* rows = reinterpret_cast<R*>(panel_raw);
  const int64_t stride = int64_t(steps) * 32 * NCA;                         // one A entry of vm
  CAcc<R, NCV, NCA> acc[P];
  for (int kb = 0; kb < nk; kb += group) {
    const int kn = min(group, nk - kb);
    if constexpr (STAGED) {
      if (kb) __syncthreads();   // the previous rows are consumed
      for (int u = 0; u < kn; ++u) {
        const char* from = reinterpret_cast<const char*>(v) +
                           int64_t(__ldg(part_h + kb + u)) * c.nl * EB;
        char* to = reinterpret_cast<char*>(rows + u * row);
        constexpr int CB = EB < 16 ? EB : 16;
        for (int i = threadIdx.x; i < nl * (EB / CB); i += blockDim.x)
          copy_async<CB>(to + i * CB, from + int64_t(i) * CB);
        if (threadIdx.x < NCV) rows[u * row + nl * NCV + threadIdx.x] = R(0);   // padding's source
      }
      asm volatile("cp.async.commit_group;");
      asm volatile("cp.async.wait_group 0;");
      __syncthreads();
    }
    const R* x[kPanelGroup];
#pragma unroll
    for (int u = 0; u < kPanelGroup; ++u) {
      if constexpr (STAGED) x[u] = rows + u * row;
      else x[u] = v + (u < kn ? int64_t(__ldg(part_h + kb + u)) * c.nl * NCV : 0);
    }
    const R* vk = vm + (k0 - a_first + kb) * stride;
#pragma unroll
    for (int i = 0; i < P; ++i) {
      // the panels of a chunk in zigzag order over the warps (their lengths descend)
      const int p = (i * W + (i & 1 ? W - 1 - warp : warp)) * chunks + chunk;
      if (p >= panels) continue;
      const int t0 = __ldg(at + p), len = __ldg(at + p + 1) - t0;
      const R* vp = vk + (int64_t(t0) * 32 + lane) * NCA;
      const uint16_t* sp = src + int64_t(t0) * 32 + lane;
      // KN entries, no branches inside.  FULL: padding multiplies zero by the zero behind the
      // staged row.  Otherwise absent elements and their amplitudes are replaced by zeros (a
      // product with an amplitude that does not belong there could be a NaN).
      auto steps_of = [&](auto kn_t) {
        constexpr int KN = decltype(kn_t)::value;
        // a step's lines of one entry, and the entry whose line this lane prefetches
        constexpr int kLines = 32 * NCA * static_cast<int>(sizeof(R)) / 128;
        const R* ahead = vp - lane * NCA + (lane / kLines) * stride +
                         (lane % kLines) * (128 / static_cast<int>(sizeof(R)));
#pragma unroll 2
        for (int t = 0; t < len; ++t) {
          if (lane < KN * kLines && t + kPanelAhead < len)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(ahead + (t + kPanelAhead) * 32 * NCA));
          int s = __ldg(sp + t * 32);
          if constexpr (!STAGED) s = min(s, nl - 1);
          Cx<R> el[kPanelGroup];
          Elem<R, NCV> xv[kPanelGroup];
#pragma unroll
          for (int u = 0; u < KN; ++u) el[u] = ld_elem<R, NCA>(vp + u * stride, t * 32);
#pragma unroll
          for (int u = 0; u < KN; ++u)
            xv[u] = STAGED ? sm_elem<R, NCV>(x[u], s) : ld_elem<R, NCV>(x[u], s);
#pragma unroll
          for (int u = 0; u < KN; ++u) {
            if constexpr (FULL) break;
            const bool gone = is_absent(el[u].re);
            el[u].re = gone ? R(0) : el[u].re;
            xv[u] = elem_unless<R, NCV>(gone, xv[u]);
          }
#pragma unroll
          for (int u = KN; u < kPanelGroup; ++u) {
            el[u] = cx_make<R>(R(0), R(0));
            xv[u] = zero_elem<R, NCV>();
          }
          acc[i].add4(el, xv);
        }
      };
      if (kn == 4) steps_of(IntTag<4>{});
      else if (kn == 3) steps_of(IntTag<3>{});
      else if (kn == 2) steps_of(IntTag<2>{});
      else steps_of(IntTag<1>{});
    }
  }
#pragma unroll
  for (int i = 0; i < P; ++i) {
    const int p = (i * W + (i & 1 ? W - 1 - warp : warp)) * chunks + chunk;
    if (p >= panels) continue;
    const uint32_t l = __ldg(perm + p * 32 + lane);
    if (l < c.nl) acc[i].store_partial(part, h * c.nl + l);
  }
}

template <typename R, int NCV, int NCA, int P, bool STAGED, bool FULL>
__global__ void __launch_bounds__(P < kPanelMaxPerWarp ? 256 : 1024,
                                  P == kPanelMaxPerWarp ? 1 : NCV == 4 ? 4 : 6)
k_tail_panels(PlanView c, PanelArgs q, const R* __restrict__ vm, const R* __restrict__ v,
              double* __restrict__ part) {
  panel_block<R, NCV, NCA, P, STAGED, FULL>(blockIdx.x, c, q, vm, v, part);
}

// ---- small grids: the three parts in one launch --------------------------------------------
// The H, L and M parts depend only on v and its transpose.  On subspaces whose slab grids are
// under two waves each pass waits on its own chains with most of the chip idle, so one launch
// runs the blocks of all three (M first, whose blocks are the longest) into FP64 partials and
// k_combine adds them: three launches instead of five.  M parts: eight warps, P panels each.
template <typename R>
struct SlabArgs {
  int64_t A, B, total_k, a_tiles, blocks;
  const int64_t* off;
  const uint32_t* src;
  const R* V;
  const R* x;
  double* part;
  int vec;                   // FP32 pairs of positions: x allows the paired accesses
};

template <typename R, int NCV, int NCA, int P, bool FULL, bool WIDE>
__global__ void __launch_bounds__(256, NCV == 4 ? 3 : P > 1 ? 4 : 5)
k_parts(PlanView c, PanelArgs q, int64_t m_blocks, const R* __restrict__ vm,
        const R* __restrict__ v, double* __restrict__ part_m, SlabArgs<R> L, SlabArgs<R> H) {
  int64_t blk = blockIdx.x;
  if (blk < m_blocks) {
    panel_block<R, NCV, NCA, P, true, FULL>(static_cast<int>(blk), c, q, vm, v, part_m);
    return;
  }
  blk -= m_blocks;
  const bool low = blk < L.blocks;
  const SlabArgs<R>& S = low ? L : H;
  if (!low) blk -= L.blocks;
  if constexpr (WIDE) {
    if (S.vec)
      slab2_block<R, NCV, NCA, false, false, true>(blk, S.A, S.B, S.total_k, S.a_tiles, S.off,
                                                   S.src, S.V, S.x, nullptr, nullptr, nullptr,
                                                   S.part);
    else
      slab2_block<R, NCV, NCA, false, false, false>(blk, S.A, S.B, S.total_k, S.a_tiles, S.off,
                                                    S.src, S.V, S.x, nullptr, nullptr, nullptr,
                                                    S.part);
  } else {
    slab_block<R, NCV, NCA, false, false>(blk, S.A, S.B, S.total_k, S.a_tiles, S.off, S.src, S.V,
                                          S.x, nullptr, nullptr, nullptr, S.part, 1);
  }
}

// out[h][l] = tL[l][h] + tH[h][l] (+ tM[h][l]), rounded once (32 x 32 tiles).
template <typename R, int NCV, bool HAS_M>
__global__ void __launch_bounds__(256)
k_combine(const double* __restrict__ pl, const double* __restrict__ ph,
          const double* __restrict__ pm, int64_t nh, int64_t nl, R* __restrict__ out) {
  __shared__ double tile[NCV][32][33];
  const int64_t th = (nh + 31) / 32, tl = (nl + 31) / 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (int64_t t = blockIdx.x; t < th * tl; t += gridDim.x) {
    const int64_t h0 = (t / tl) * 32, l0 = (t % tl) * 32;
    for (int i = ty; i < 32; i += 8) {
      const int64_t l = l0 + i, h = h0 + tx;
      if (l < nl && h < nh) {
#pragma unroll
        for (int q = 0; q < NCV; ++q) tile[q][i][tx] = pl[(l * nh + h) * NCV + q];
      }
    }
    __syncthreads();
    for (int i = ty; i < 32; i += 8) {
      const int64_t h = h0 + i, l = l0 + tx;
      if (h < nh && l < nl) {
        const int64_t r = (h * nl + l) * NCV;
#pragma unroll
        for (int q = 0; q < NCV; ++q) {
          double s = tile[q][tx][i];
          if constexpr (HAS_M) s += pm[r + q];
          out[r + q] = static_cast<R>(s + ph[r + q]);
        }
      }
    }
    __syncthreads();
  }
}

// ---- short row tails ----------------------------------------------------------------------
__global__ void k_tail_lengths(const int64_t* __restrict__ row_ptr, const int64_t* __restrict__ ho,
                               const int64_t* __restrict__ lo, int64_t n, int64_t nl,
                               int64_t* len) {
  for (int64_t r = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; r < n;
       r += int64_t(gridDim.x) * blockDim.x)
    len[r] = row_ptr[r + 1] - tail_begin(row_ptr, ho, lo, r, nl);
}

// Contiguous copy of the row tails: elements and (mcol, when given) source rows.
template <int NCA>
__global__ void k_tail_fill(const int64_t* __restrict__ row_ptr, const uint32_t* __restrict__ cols,
                            const double* __restrict__ vals, const int64_t* __restrict__ ho,
                            const int64_t* __restrict__ lo, int64_t n, int64_t nl,
                            const int64_t* __restrict__ mptr, double* mval, uint32_t* mcol) {
  for (int64_t r = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; r < n;
       r += int64_t(gridDim.x) * blockDim.x) {
    const int64_t b = tail_begin(row_ptr, ho, lo, r, nl), e = row_ptr[r + 1];
    int64_t j = mptr[r];
    for (int64_t i = b; i < e; ++i, ++j) {
#pragma unroll
      for (int t = 0; t < NCA; ++t) mval[NCA * j + t] = vals[NCA * i + t];
      if (mcol != nullptr) mcol[j] = cols[i];
    }
  }
}

// One block per tile: at most n / 256 + n / 32 of them for n < 2^31 rows.
unsigned tile_grid(int64_t blocks) {
  SQD_REQUIRE(blocks <= INT_MAX, "grid too large");
  return static_cast<unsigned>(std::max<int64_t>(1, blocks));
}

// wide: FP32 slabs in 64-wide panels (k_slab2); vec: x and out allow its paired accesses.
template <typename R, int NCV, int NCA, bool FINAL, bool HAS_M>
void launch_slab(int64_t A, int64_t B, int64_t total_k, const int64_t* off, const uint32_t* src,
                 const R* V, const R* x, const double* part_t, const double* part_m, R* out,
                 double* out_part, cudaStream_t st, bool wide = false, bool vec = false) {
  if (A == 0 || B == 0) return;
  if constexpr (sizeof(R) == 4) {
    if (wide) {
      const int64_t a_tiles = (A + 7) / 8, panels = (B + 63) / 64;
      if (vec)
        k_slab2<R, NCV, NCA, FINAL, HAS_M, true><<<tile_grid(a_tiles * panels), 256, 0, st>>>(
            A, B, total_k, a_tiles, off, src, V, x, part_t, part_m, out, out_part);
      else
        k_slab2<R, NCV, NCA, FINAL, HAS_M, false><<<tile_grid(a_tiles * panels), 256, 0, st>>>(
            A, B, total_k, a_tiles, off, src, V, x, part_t, part_m, out, out_part);
      SQD_CHECK_LAUNCH();
      return;
    }
  }
  const int64_t a_tiles = (A + 7) / 8, panels = (B + 31) / 32;
  // With at most two waves of warps (64 per SM) too few warps hide the latency of each step's
  // source-offset load, which the gathers wait on, so it is prefetched one step ahead (C2:
  // 8,192 warps, FP64 matvec 0.348 -> 0.320 ms); on larger grids the other warps hide it and
  // the extra requests cost 2-4 % (C3, 524,288 warps).
  const int prefetch = A * panels <= 2 * 64 * int64_t(num_sms()) ? 1 : 0;
  k_slab<R, NCV, NCA, FINAL, HAS_M><<<tile_grid(a_tiles * panels), 256, 0, st>>>(
      A, B, total_k, a_tiles, off, src, V, x, part_t, part_m, out, out_part, prefetch);
  SQD_CHECK_LAUNCH();
}

template <typename E>
void launch_transpose(const void* in, void* out, int64_t rows, int64_t cols, cudaStream_t st) {
  const unsigned G = tile_grid(
      std::min<int64_t>(((rows + 31) / 32) * ((cols + 31) / 32), int64_t(num_sms()) * 32));
  k_transpose<E><<<G, 256, 0, st>>>(static_cast<const E*>(in), static_cast<E*>(out), rows, cols);
  SQD_CHECK_LAUNCH();
}

unsigned mixed_grid(int64_t rows, int lpr) {
  const int64_t warps = (rows * lpr + 31) / 32;
  const int64_t blocks = (warps + 7) / 8;
  const int64_t cap = static_cast<int64_t>(num_sms()) * 16;
  return static_cast<unsigned>(std::max<int64_t>(1, std::min(blocks, cap)));
}

void to_float(const DevBuf<double>& in, DevBuf<float>& out, cudaStream_t st) {
  out.alloc(in.count, st);
  k_to_float32<<<grid_for(static_cast<int64_t>(in.count), 256, 16384), 256, 0, st>>>(
      in.ptr, out.ptr, static_cast<int64_t>(in.count));
  SQD_CHECK_LAUNCH();
}

// Slabs (f64) and their FP32 copies (f32) from the elements in the pair list.
void fill_slabs(sqd_op_s* op, bool f64, bool f32, cudaStream_t st) {
  ProductLayout& L = op->prod;
  ElementOut out{};
  out.values = op->values.ptr;
  if (f64) {
    out.vh = L.vh.ptr;
    out.vl = L.vl.ptr;
  }
  if (f32) {
    out.vh32 = L.vh32.ptr;
    out.vl32 = L.vl32.ptr;
  }
  out.wide32 = L.wide32;
  op_slab_elements(op, out, st);
}

void alloc_slabs32(sqd_op_s* op, cudaStream_t st) {
  ProductLayout& L = op->prod;
  const int nca = op->value_complex ? 2 : 1;
  const int64_t w = L.wide32 ? 64 : 32;
  DevBuf<float> vh, vl;   // both or none: a failed allocation leaves the layout as it was
  vh.alloc(static_cast<size_t>(std::max<int64_t>((L.nl + w - 1) / w * L.th * w, 1)) * nca, st);
  vl.alloc(static_cast<size_t>(std::max<int64_t>((L.nh + w - 1) / w * L.tl * w, 1)) * nca, st);
  L.vh32 = std::move(vh);
  L.vl32 = std::move(vl);
}

// A row tail read in place is a short segment of the row's long pair list (48-qubit subspaces:
// ~11 M pairs among ~160), so its element and source loads use few bytes of the sectors they
// fetch.  Tails up to this many pairs per row on average are also copied contiguously.
constexpr int64_t kCompactTailMax = 32;

void fill_panels(sqd_op_s* op, bool f64, bool f32, cudaStream_t st) {
  ProductLayout& L = op->prod;
  const unsigned G = grid_for(L.nh * L.panels * 32, 256, num_sms() * 64);
  auto run = [&](auto nca) {
    k_panel_fill<decltype(nca)::value><<<G, 256, 0, st>>>(
        plan_view(*op->plan), op->row_ptr.ptr, op->values.ptr, L.ho.ptr, L.lo.ptr, L.panel_at.ptr,
        L.perm.ptr, L.panels, L.steps, L.panel_full, f64 ? L.vm.ptr : nullptr,
        f32 ? L.vm32.ptr : nullptr);
    SQD_CHECK_LAUNCH();
  };
  if (op->value_complex) run(IntTag<2>{});
  else run(IntTag<1>{});
}

// Panel form of the M pairs.  It applies when most of A(h) x B(l) exists (the panels hold every
// combination; up to 1.6 elements per stored pair) and 16 bits reach a row of v.  Matvec in us,
// panels / pair-list tails, complex128 and complex64, by elements per pair: 32 qubits, 512 x 512
// strings with a share of the two-half groups left out, 1.0 223/327 144/255, 1.5 213/290 137/229,
// 2.1 211/249 136/177, 2.6 212/233 137/169; 300 x 300 1.6 62/81 50/83; 48 qubits, 2000 x 1800, 1.3
// 516/575 355/375, 2.6 515/559 355/369.  Sums whose parts hardly ever meet (random Paulis): 5.8 64/27
// 59/25, 10 492/95 412/85, 25 183/45 156/35.  The limit stays on the safe side of the two.
void build_panels(sqd_op_s* op, cudaStream_t st) {
  ProductLayout& L = op->prod;
  const ProductPlan& q = *op->plan;
  L.panel_state = -1;
  if (L.pairs_m <= 0 || q.ta == 0 || q.tb == 0 || L.nl > 65535) return;
  std::vector<int64_t> boff(static_cast<size_t>(L.nl) + 1);
  copy_to_host(boff.data(), plan_view(q).boff, boff.size(), st);
  std::vector<uint32_t> perm(static_cast<size_t>((L.nl + 31) / 32 * 32), 0xffffffffu);
  for (int64_t l = 0; l < L.nl; ++l) perm[static_cast<size_t>(l)] = static_cast<uint32_t>(l);
  auto len = [&](uint32_t l) { return boff[l + 1] - boff[l]; };
  std::stable_sort(perm.begin(), perm.begin() + L.nl,
                   [&](uint32_t a, uint32_t b) { return len(a) > len(b); });
  std::vector<int64_t> aoff(static_cast<size_t>(L.nh) + 1);
  copy_to_host(aoff.data(), plan_view(q).aoff, aoff.size(), st);
  std::vector<uint32_t> horder(static_cast<size_t>(L.nh));
  for (int64_t h = 0; h < L.nh; ++h) horder[static_cast<size_t>(h)] = static_cast<uint32_t>(h);
  std::stable_sort(horder.begin(), horder.end(), [&](uint32_t a, uint32_t b) {
    return aoff[a + 1] - aoff[a] > aoff[b + 1] - aoff[b];
  });
  // Rows too long to stage have no zero behind them for the padding.
  L.panel_full = L.pairs_m == q.ta * q.tb &&
                 panel_row(L.nl, 32) <= static_cast<int64_t>(kPanelSmem);
  const int64_t panels = (L.nl + 31) / 32;
  std::vector<int32_t> at(static_cast<size_t>(panels) + 1, 0);
  int64_t steps = 0;
  for (int64_t p = 0; p < panels; ++p) {
    at[static_cast<size_t>(p)] = static_cast<int32_t>(steps);
    steps += len(perm[static_cast<size_t>(p * 32)]);
  }
  at[static_cast<size_t>(panels)] = static_cast<int32_t>(steps);
  const double total = double(q.ta) * double(steps) * 32.0;
  if (steps > INT_MAX / 64 || total > 1.6 * double(L.pairs_m)) return;
  const int nca = op->value_complex ? 2 : 1;
  try {
    L.panel_at.alloc(at.size(), st);
    L.perm.alloc(perm.size(), st);
    L.horder.alloc(horder.size(), st);
    L.panel_src.alloc(static_cast<size_t>(steps) * 32, st);
    L.vm.alloc(static_cast<size_t>(q.ta * steps * 32) * nca, st);
  } catch (const Error& e) {   // no memory: the tails are read as CSR rows
    if (e.status != SQD_ERR_MEMORY) throw;
    (void)cudaGetLastError();
    L.panel_at = DevBuf<int32_t>();
    L.perm = DevBuf<uint32_t>();
    L.horder = DevBuf<uint32_t>();
    L.panel_src = DevBuf<uint16_t>();
    L.vm = DevBuf<double>();
    return;
  }
  SQD_CUDA(cudaMemcpyAsync(L.panel_at.ptr, at.data(), L.panel_at.bytes(), cudaMemcpyHostToDevice,
                           st));
  SQD_CUDA(cudaMemcpyAsync(L.perm.ptr, perm.data(), L.perm.bytes(), cudaMemcpyHostToDevice, st));
  SQD_CUDA(cudaMemcpyAsync(L.horder.ptr, horder.data(), L.horder.bytes(), cudaMemcpyHostToDevice,
                           st));
  L.panels = panels;
  L.steps = steps;
  k_panel_src<<<grid_for(panels * 32, 256, 4096), 256, 0, st>>>(
      plan_view(q), L.panel_at.ptr, L.perm.ptr, panels, L.panel_src.ptr);
  SQD_CHECK_LAUNCH();
  fill_panels(op, true, false, st);
  SQD_CUDA(cudaStreamSynchronize(st));   // the host vectors above go out of scope
  L.panel_state = 1;
}

void fill_tail(sqd_op_s* op, bool sources, cudaStream_t st) {
  ProductLayout& L = op->prod;
  const int64_t n = L.nh * L.nl;
  const unsigned G = grid_for(n, 256, 16384);
  auto run = [&](auto nca) {
    k_tail_fill<decltype(nca)::value><<<G, 256, 0, st>>>(
        op->row_ptr.ptr, op->cols.ptr, op->values.ptr, L.ho.ptr, L.lo.ptr, n, L.nl, L.mptr.ptr,
        L.mval.ptr, sources ? L.mcol.ptr : nullptr);
    SQD_CHECK_LAUNCH();
  };
  if (op->value_complex) run(IntTag<2>{});
  else run(IntTag<1>{});
}

// Contiguous copy of short row tails; longer ones, or without memory for it, are read in place.
void build_tail(sqd_op_s* op, cudaStream_t st) {
  ProductLayout& L = op->prod;
  const int64_t n = L.nh * L.nl;
  L.tail_state = -1;
  if (L.pairs_m <= 0 || L.pairs_m > kCompactTailMax * n) return;
  DevBuf<int64_t> len;
  const int nca = op->value_complex ? 2 : 1;
  try {
    len.alloc(n, st);
    L.mptr.alloc(n + 1, st);
    L.mval.alloc(static_cast<size_t>(L.pairs_m) * nca, st);
    L.mcol.alloc(static_cast<size_t>(L.pairs_m), st);
  } catch (const Error& e) {
    if (e.status != SQD_ERR_MEMORY) throw;
    (void)cudaGetLastError();  // the failed pool allocation
    L.mptr = DevBuf<int64_t>();
    L.mval = DevBuf<double>();
    L.mcol = DevBuf<uint32_t>();
    return;
  }
  k_tail_lengths<<<grid_for(n, 256, 16384), 256, 0, st>>>(op->row_ptr.ptr, L.ho.ptr, L.lo.ptr, n,
                                                          L.nl, len.ptr);
  SQD_CHECK_LAUNCH();
  exclusive_scan_i64(len.ptr, L.mptr.ptr, n, true, st);
  fill_tail(op, true, st);
  L.tail_state = 1;
}

// The form of the M pairs that a layout reads, on its first use.
void build_mixed(sqd_op_s* op, int layout, cudaStream_t st) {
  ProductLayout& L = op->prod;
  if (layout == SQD_LAYOUT_PRODUCT && L.panel_state == 0) build_panels(op, st);
  if ((layout == SQD_LAYOUT_PRODUCT_CSR || L.panel_state < 0) && L.tail_state == 0)
    build_tail(op, st);
}

// FP32 copies of whatever exists in FP64 and has none yet.
void ensure_floats(sqd_op_s* op, cudaStream_t st) {
  ProductLayout& L = op->prod;
  if (!L.vh32.ptr || !L.vl32.ptr) {
    alloc_slabs32(op, st);
    fill_slabs(op, false, true, st);
  }
  if (L.panel_state == 1 && !L.vm32.ptr && L.panel32_state == 0) {
    try {
      L.vm32.alloc(L.vm.count, st);
      fill_panels(op, false, true, st);
    } catch (const Error& e) {   // no memory: FP32 tails are read from the pair list
      if (e.status != SQD_ERR_MEMORY) throw;
      (void)cudaGetLastError();
      L.panel32_state = -1;
    }
  }
  if (L.tail_state == 1 && !L.mval32.ptr) to_float(L.mval, L.mval32, st);
}

// How k_tail_panels runs: rows staged together, panels per block (chunks), per warp.
struct PanelShape {
  PanelArgs args;
  bool staged;
  size_t dyn;
  int64_t per, warps, blocks;
};

// max_dyn: shared memory for the staged rows; max_warps: of a block.
PanelShape panel_shape(const ProductLayout& L, int element_bytes, double line, size_t max_dyn,
                       int64_t max_warps) {
  PanelShape s{};
  // Rows staged together: four, or what fits, at least one.
  const size_t row = static_cast<size_t>(panel_row(L.nl, element_bytes));
  s.staged = row <= kPanelSmem;
  const int group =
      s.staged ? static_cast<int>(std::max<size_t>(1, std::min<size_t>(kPanelGroup, max_dyn / row)))
               : kPanelGroup;
  s.dyn = s.staged ? group * row : 0;
  // Panels per block: one per warp, eight warps, unless the staged row is more than their elements
  // (short B lists: 48 qubits, 2.3 steps a panel) or there are fewer than six blocks per SM.
  int64_t mine = std::max<int64_t>(8, static_cast<int64_t>(double(row) / std::max(line, 1.0)));
  mine = std::min(std::min(mine, max_warps * kPanelMaxPerWarp), L.panels);
  while (mine > 4 && L.nh * ((L.panels + mine - 1) / mine) < 6 * int64_t(num_sms())) --mine;
  const int64_t chunks = (L.panels + mine - 1) / mine;
  mine = (L.panels + chunks - 1) / chunks;
  s.per = std::max((mine + max_warps - 1) / max_warps,
                   std::min<int64_t>(kPanelMaxPerWarp, (mine + 7) / 8));
  s.warps = (mine + s.per - 1) / s.per;
  s.blocks = L.nh * chunks;
  s.args = PanelArgs{L.panel_at.ptr, L.perm.ptr, L.panel_src.ptr, L.horder.ptr,
                     static_cast<int>(L.panels), static_cast<int>(L.steps),
                     static_cast<int>(chunks), group};
  return s;
}

template <typename R>
const R* panel_elements(const ProductLayout& L) {
  if (L.panel_state != 1) return nullptr;
  if constexpr (sizeof(R) == 8) return L.vm.ptr;
  else return L.vm32.ptr;
}
// Bytes of a panel's elements per A entry, on average.
template <typename R, int NCA>
double panel_line(const ProductLayout& L) {
  return 32.0 * sizeof(R) * NCA * double(L.steps) / double(L.panels);
}

void allow_smem(const void* kern, size_t dyn) {
  if (dyn > 48 * 1024)
    SQD_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  static_cast<int>(kPanelSmem)));
}

template <typename R, int NCV, int NCA>
bool launch_panels(sqd_op_s* op, const R* vin, double* part, cudaStream_t st) {
  ProductLayout& L = op->prod;
  const R* vm = panel_elements<R>(L);
  if (vm == nullptr) return false;
  // two blocks per SM at least
  const PanelShape s = panel_shape(L, static_cast<int>(sizeof(R)) * NCV, panel_line<R, NCA>(L),
                                   kPanelSmem / 2, kPanelMaxWarps);
  SQD_REQUIRE(s.blocks <= INT_MAX, "too many high strings");
  auto go = [&](auto kern) {
    allow_smem(reinterpret_cast<const void*>(kern), s.dyn);
    kern<<<static_cast<unsigned>(s.blocks), static_cast<unsigned>(s.warps * 32), s.dyn, st>>>(
        plan_view(*op->plan), s.args, vm, vin, part);
    SQD_CHECK_LAUNCH();
  };
  auto pick = [&](auto p) {
    constexpr int P = decltype(p)::value;
    if (!s.staged) go(k_tail_panels<R, NCV, NCA, P, false, false>);
    else if (L.panel_full) go(k_tail_panels<R, NCV, NCA, P, true, true>);
    else go(k_tail_panels<R, NCV, NCA, P, true, false>);
  };
  switch (s.per) {
    case 1: pick(IntTag<1>{}); break;
    case 2: pick(IntTag<2>{}); break;
    case 3: pick(IntTag<3>{}); break;
    default: pick(IntTag<4>{}); break;
  }
  return true;
}

// Slab grids of at most two waves of warps (64 per SM) run the three parts in one launch: 512 x 512
// strings at 32 qubits (0.9 waves) complex128 273 -> 212 us, complex64 172 -> 146, 130 x 100 36 -> 21.
// Beyond, one launch and five are within 15 % either way (900 x 800, 2.4 waves: complex128 1082 /
// 1225 us, float64 1023 / 917; 48 qubits, 1100 x 1000, 3.7 waves: complex64 88 / 104, float64 119 /
// 117) and the additional partial vector costs memory.
bool small_grid(const ProductLayout& L) {
  const int64_t warps = std::max(L.nh * ((L.nl + 31) / 32), L.nl * ((L.nh + 31) / 32));
  return warps <= 2 * 64 * int64_t(num_sms());
}
constexpr size_t kPartsSmem = 40 * 1024;

template <typename R>
SlabArgs<R> slab_args(int64_t A, int64_t B, int64_t total_k, const int64_t* off,
                      const uint32_t* src, const R* V, const R* x, double* part, bool wide,
                      bool vec) {
  SlabArgs<R> s{};
  s.A = A;
  s.B = B;
  s.total_k = total_k;
  s.a_tiles = (A + 7) / 8;
  s.blocks = s.a_tiles * (wide ? (B + 63) / 64 : (B + 31) / 32);
  s.off = off;
  s.src = src;
  s.V = V;
  s.x = x;
  s.part = part;
  s.vec = vec ? 1 : 0;
  return s;
}

// Launches k_parts and k_combine; false where the M part does not fit beside the slabs (rows of v
// over kPartsSmem) or is not in panels.
template <typename R, int NCV, int NCA>
bool launch_parts(sqd_op_s* op, const R* vin, R* vout, const SlabArgs<R>& low,
                  const SlabArgs<R>& high, bool wide, double* part_m, cudaStream_t st) {
  ProductLayout& L = op->prod;
  PanelShape s{};
  const R* vm = nullptr;
  if (L.pairs_m > 0) {
    vm = panel_elements<R>(L);
    if (vm == nullptr) return false;
    s = panel_shape(L, static_cast<int>(sizeof(R)) * NCV, panel_line<R, NCA>(L), kPartsSmem, 8);
    if (!s.staged || s.dyn > kPartsSmem) return false;
  }
  const int64_t blocks = s.blocks + low.blocks + high.blocks;
  if (blocks == 0 || blocks > INT_MAX) return false;
  auto go = [&](auto kern) {
    kern<<<static_cast<unsigned>(blocks), 256, s.dyn, st>>>(
        plan_view(*op->plan), s.args, s.blocks, vm, vin, part_m, low, high);
    SQD_CHECK_LAUNCH();
  };
  auto pick = [&](auto p) {
    constexpr int P = decltype(p)::value;
    if constexpr (sizeof(R) == 4) {
      if (wide) {
        if (L.panel_full) go(k_parts<R, NCV, NCA, P, true, true>);
        else go(k_parts<R, NCV, NCA, P, false, true>);
        return;
      }
    }
    if (L.panel_full) go(k_parts<R, NCV, NCA, P, true, false>);
    else go(k_parts<R, NCV, NCA, P, false, false>);
  };
  if (s.per <= 1) pick(IntTag<1>{});
  else pick(IntTag<4>{});
  const int64_t tiles = ((L.nh + 31) / 32) * ((L.nl + 31) / 32);
  const unsigned G = static_cast<unsigned>(std::min<int64_t>(tiles, int64_t(num_sms()) * 16));
  if (L.pairs_m > 0)
    k_combine<R, NCV, true><<<G, 256, 0, st>>>(low.part, high.part, part_m, L.nh, L.nl, vout);
  else
    k_combine<R, NCV, false><<<G, 256, 0, st>>>(low.part, high.part, nullptr, L.nh, L.nl, vout);
  SQD_CHECK_LAUNCH();
  return true;
}

}  // namespace

void op_product_build(sqd_op_s* op, int layout, cudaStream_t st) {
  if (op->prod.built) {
    build_mixed(op, layout, st);
    return;
  }
  SQD_REQUIRE(op->x_cache == 1 && op->z_cache == 2,
              "the product layout needs cache_strategy (1, 2)");
  SQD_REQUIRE(op->nnz == 0 || op->grps.ptr != nullptr,
              "the operator released its group indices; create a new operator");
  if (!op_plan(op, st))
    throw Error(SQD_ERR_UNSUPPORTED,
                "the subspace is not a product of high-half and low-half strings without "
                "fill-in slots; the product layout does not apply");
  const ProductPlan& q = *op->plan;
  const int64_t nh = q.nh, nl = q.nl, n = nh * nl;
  ProductLayout L;
  L.nh = nh;
  L.nl = nl;
  L.wide32 = (nh % 2 == 0 && nl % 2 == 0) ? 1 : 0;
  L.th = q.th;
  L.tl = q.tl + q.d * nl;
  L.pairs_h = L.th * nl;
  L.pairs_l = L.tl * nh;
  L.pairs_m = op->nnz - L.pairs_h - L.pairs_l;
  if (L.pairs_m < 0)
    throw Error(SQD_ERR_DEVICE, "stored pairs do not follow the product structure");
  L.ho.alloc(nh + 1, st);
  L.lo.alloc(nl + 1, st);
  L.hsrc.alloc(std::max<int64_t>(L.th, 1), st);
  L.lsrc.alloc(std::max<int64_t>(L.tl, 1), st);
  SQD_CUDA(cudaMemcpyAsync(L.ho.ptr, q.offs.ptr, (nh + 1) * sizeof(int64_t),
                           cudaMemcpyDeviceToDevice, st));
  k_slab_sources<<<grid_for(std::max(L.th, nl + 1), 256, 4096), 256, 0, st>>>(
      plan_view(q), L.th, L.hsrc.ptr, L.lo.ptr, L.lsrc.ptr);
  SQD_CHECK_LAUNCH();
  const int nca = op->value_complex ? 2 : 1;
  // Panel-major slabs, each panel padded to 32 positions (the padding is never read).
  L.vh.alloc(static_cast<size_t>(std::max<int64_t>(L.th * ((nl + 31) / 32) * 32, 1)) * nca, st);
  L.vl.alloc(static_cast<size_t>(std::max<int64_t>(L.tl * ((nh + 31) / 32) * 32, 1)) * nca, st);
  L.vt.alloc(static_cast<size_t>(n) * 2, st);
  L.tt.alloc(static_cast<size_t>(n) * 2, st);
  L.t.alloc(L.pairs_m > 0 ? static_cast<size_t>(n) * 2 : 1, st);
  if (small_grid(L)) L.t2.alloc(static_cast<size_t>(n) * 2, st);
  op->prod = std::move(L);
  try {
    fill_slabs(op, true, false, st);
    build_mixed(op, layout, st);
    SQD_CUDA(cudaStreamSynchronize(st));
  } catch (...) {
    op->prod = ProductLayout();
    throw;
  }
  op->prod.built = 1;
}

// A coefficient update (sources unchanged): the slabs are filled beside the pair list, the tails
// from it.
void op_product_targets(sqd_op_s* op, ElementOut* out) {
  ProductLayout& L = op->prod;
  if (!L.built) return;
  out->vh = L.vh.ptr;
  out->vl = L.vl.ptr;
  out->vh32 = L.vh32.ptr;
  out->vl32 = L.vl32.ptr;
  out->wide32 = L.wide32;
}

void op_product_refresh(sqd_op_s* op, cudaStream_t st) {
  ProductLayout& L = op->prod;
  if (!L.built) return;
  if (L.panel_state == 1) fill_panels(op, true, L.vm32.ptr != nullptr, st);
  if (L.tail_state == 1) fill_tail(op, false, st);
  if (L.mval32.ptr) to_float(L.mval, L.mval32, st);
}

void op_product_values32(sqd_op_s* op, cudaStream_t st) {
  if (op->prod.built) ensure_floats(op, st);
}

namespace {

// Scratch of one product matvec: FP64 values per row and vector component.
// th: only for small grids (small_grid), else NULL.
struct ProductScratch {
  double *vt, *tt, *t, *th;
};

template <typename R, int NCV, int NCA>
void product_matvec(sqd_op_s* op, const R* vin, R* vout, const ProductScratch& w,
                    cudaStream_t st) {
  ProductLayout& L = op->prod;
  const int64_t nh = L.nh, nl = L.nl, n = nh * nl;
  const int prec = sizeof(R) == 8 ? 0 : 1;
  using E = Raw<R, NCV>;
  using ED = Raw<double, NCV>;
  const R* VH;
  const R* VL;
  const R* VC;
  if constexpr (sizeof(R) == 8) {
    VH = L.vh.ptr;
    VL = L.vl.ptr;
    VC = op->values.ptr;
  } else {
    VH = L.vh32.ptr;
    VL = L.vl32.ptr;
    VC = op->values32.ptr;
  }
  R* vt = reinterpret_cast<R*>(w.vt);
  // FP32 slabs in 64-wide panels (both halves even): paired accesses to the library's own
  // buffers always, to v and Hv when their addresses allow
  const bool wide = sizeof(R) == 4 && L.wide32;
  const uintptr_t pair_bytes = 2 * NCV * sizeof(R);
  const bool vec_io = reinterpret_cast<uintptr_t>(vin) % pair_bytes == 0 &&
                      reinterpret_cast<uintptr_t>(vout) % pair_bytes == 0;
  // 1. vT[l][h] = v[h][l]
  launch_transpose<E>(vin, vt, nh, nl, st);
  if (small_grid(L) && op->layout[prec] == SQD_LAYOUT_PRODUCT && w.th != nullptr) {
    const SlabArgs<R> low = slab_args<R>(nl, nh, L.tl, L.lo.ptr, L.lsrc.ptr, VL, vt, w.tt, wide,
                                         true);
    const SlabArgs<R> high = slab_args<R>(nh, nl, L.th, L.ho.ptr, L.hsrc.ptr, VH, vin, w.th, wide,
                                          vec_io);
    if (launch_parts<R, NCV, NCA>(op, vin, vout, low, high, wide, w.t, st)) return;
  }
  // 2. L part: t2[l][h]
  launch_slab<R, NCV, NCA, false, false>(nl, nh, L.tl, L.lo.ptr, L.lsrc.ptr, VL, vt, nullptr,
                                         nullptr, nullptr, w.tt, st, wide, true);
  // 3. t2 back in row order, into the vT buffer
  launch_transpose<ED>(w.tt, w.vt, nl, nh, st);
  // 4. M part: t3[r]
  if (L.pairs_m > 0) {
    if (op->layout[prec] == SQD_LAYOUT_PRODUCT_CSR ||
        !launch_panels<R, NCV, NCA>(op, vin, w.t, st)) {
      const R* MV = nullptr;  // the short-tail copy's elements, when it exists
      if (L.tail_state == 1) {
        if constexpr (sizeof(R) == 8) MV = L.mval.ptr;
        else MV = L.mval32.ptr;
      }
      // lanes from the mean tail length unless the caller chose them (48 qubits, 3072 x 2816
      // strings: 5.6 pairs a tail, 1.87 ms with the whole row's 32 lanes)
      const int lanes = op->lanes_chosen[prec] ? op->lanes_per_row[prec]
                                               : lanes_for(double(L.pairs_m) / double(n));
      dispatch_lpr(lanes, [&](auto lpr_t) {
        constexpr int LPR = decltype(lpr_t)::value;
        if (MV != nullptr)
          k_mv_mixed<R, NCV, NCA, LPR, true><<<mixed_grid(n, LPR), 256, 0, st>>>(
              L.mptr.ptr, L.mcol.ptr, MV, vin, nullptr, nullptr, nl, w.t, n,
              op->chunk_rows[prec]);
        else
          k_mv_mixed<R, NCV, NCA, LPR, false><<<mixed_grid(n, LPR), 256, 0, st>>>(
              op->row_ptr.ptr, op->cols.ptr, VC, vin, L.ho.ptr, L.lo.ptr, nl, w.t, n,
              op->chunk_rows[prec]);
        SQD_CHECK_LAUNCH();
      });
    }
    // 5. H part plus both partials
    launch_slab<R, NCV, NCA, true, true>(nh, nl, L.th, L.ho.ptr, L.hsrc.ptr, VH, vin, w.vt, w.t,
                                         vout, nullptr, st, wide, vec_io);
  } else {
    launch_slab<R, NCV, NCA, true, false>(nh, nl, L.th, L.ho.ptr, L.hsrc.ptr, VH, vin, w.vt,
                                          nullptr, vout, nullptr, st, wide, vec_io);
  }
}

}  // namespace

void op_product_matvec(sqd_op_s* op, const void* v, void* out, int dtype, cudaStream_t st) {
  ProductLayout& L = op->prod;
  SQD_REQUIRE(dtype_is_double(dtype) || (L.vh32.ptr != nullptr && L.vl32.ptr != nullptr),
              "FP32 product-layout elements were not prepared");
  const ProductScratch w{L.vt.ptr, L.tt.ptr, L.t.ptr, L.t2.ptr};
  dispatch_vec(dtype, op->value_complex, [&](auto rt, auto ncv_t, auto nca_t) {
    using R = typename decltype(rt)::type;
    product_matvec<R, decltype(ncv_t)::value, decltype(nca_t)::value>(
        op, static_cast<const R*>(v), static_cast<R*>(out), w, st);
  });
}

void op_product_matvec_pair(sqd_op_s* op, const double* v, double* out, double* scratch,
                            cudaStream_t st) {
  const int64_t n = op->prod.nh * op->prod.nl;
  const ProductScratch w{scratch, scratch + 4 * n, scratch + 8 * n, scratch + 12 * n};
  if (op->value_complex) product_matvec<double, 4, 2>(op, v, out, w, st);
  else product_matvec<double, 4, 1>(op, v, out, w, st);
}

}  // namespace sqd

using namespace sqd;

extern "C" int sqd_op_set_layout(sqd_op_t op, int precision, int layout, void* stream) {
  return guarded([&] {
    SQD_REQUIRE(op != nullptr, "NULL operator");
    SQD_REQUIRE(precision == 0 || precision == 1, "precision must be 0 (FP64) or 1 (FP32)");
    SQD_REQUIRE(layout == SQD_LAYOUT_CSR || layout == SQD_LAYOUT_PRODUCT ||
                    layout == SQD_LAYOUT_PRODUCT_CSR,
                "unknown layout");
    if (layout != SQD_LAYOUT_CSR) {
      cudaStream_t st = as_stream(stream);
      op_product_build(op, layout, st);
      if (precision == 1) {
        const int prev = op->layout[1];
        op->layout[1] = layout;
        try {
          op_ensure_values32(op, st);
          SQD_CUDA(cudaStreamSynchronize(st));
        } catch (...) {
          op->layout[1] = prev;
          throw;
        }
      }
    }
    op->layout[precision] = layout;
    ++op->schedule_version;
  });
}

extern "C" int sqd_op_get_layout(sqd_op_t op, int precision, int* layout) {
  return guarded([&] {
    SQD_REQUIRE(op != nullptr && layout != nullptr, "NULL argument");
    SQD_REQUIRE(precision == 0 || precision == 1, "precision must be 0 (FP64) or 1 (FP32)");
    *layout = op->layout[precision];
  });
}

extern "C" int sqd_op_product_info(sqd_op_t op, void* stream, int64_t* n_high, int64_t* n_low,
                                   int64_t* pairs_high, int64_t* pairs_low,
                                   int64_t* pairs_mixed) {
  return guarded([&] {
    SQD_REQUIRE(op != nullptr, "NULL operator");
    int64_t nh = 0, nl = 0, ph = -1, pl = -1, pm = -1;
    if (op->prod.built) {
      nh = op->prod.nh;
      nl = op->prod.nl;
      ph = op->prod.pairs_h;
      pl = op->prod.pairs_l;
      pm = op->prod.pairs_m;
    } else if (op->x_cache == 1 && op->z_cache == 2) {
      op_product_detect(op, as_stream(stream), &nh, &nl);
    }
    if (n_high) *n_high = nh;
    if (n_low) *n_low = nl;
    if (pairs_high) *pairs_high = ph;
    if (pairs_low) *pairs_low = pl;
    if (pairs_mixed) *pairs_mixed = pm;
  });
}
