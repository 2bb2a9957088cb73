// Hv on the subspace: (Hv)_i = sum_j C^(j)_i v[src_j(i)]  (sqd.py:65-68, apply_h* :643-743).
//
// Row-oriented gather, no atomics.  A warp serves 32 / LPR rows at a time, LPR lanes per row
// stride over the row's stored pairs (coalesced loads of the pair arrays), gather the source
// amplitudes with 128-bit (c128) / 64-bit (c64) loads, and reduce with warp shuffles.
//
//  * k_mv_csr  (cache_strategy (1, 2)): matrix elements cached per stored pair.
//  * k_mv_xc   (cache_strategy (1, 0) / (1, 1)): sources cached, composed diagonal recomputed
//               from popcount(s & z) per pair (the reference's default, apply_h_x_cached).
//               The diagonal group (x = 0, K_0 terms, the largest group) is split over the LPR
//               lanes of the row.
//  * sweep APPLY (cache_strategy (0, *)): sources searched inside the matvec (apply_h).
//  * k_mv_plan (both of the above on product subspaces where op_plan_pays, unless a hash or binary
//               search was asked for): pairs enumerated from the halves' partner lists, elements
//               composed.
// FP32 vectors accumulate with error-free transformations (TwoProduct via fma, TwoSum), i.e.
// the compensated dot product of Ogita, Rump and Oishi (SIAM J. Sci. Comput. 26, 2005), so the
// FP32 result is as accurate as if accumulated in twice the working precision.
#include "internal.cuh"
#include "dispatch.cuh"
#include "accum.cuh"
#include "sweep.cuh"

namespace sqd {
namespace {

template <typename R, int NCV, int NCA, int LPR>
__global__ void __launch_bounds__(256)
k_mv_csr(const int64_t* __restrict__ row_ptr, const uint32_t* __restrict__ cols,
         const R* __restrict__ vals, const R* __restrict__ v, R* __restrict__ out,
         int64_t n_rows, int64_t chunk) {
  constexpr int RPW = 32 / LPR;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int sub = lane % LPR, slot = lane / LPR;
  auto one_step = [&](int64_t rb, int64_t lim) {
    const int64_t row = rb + slot;
    CAcc<R, NCV, NCA> acc;
    if (row < lim) {
      const int64_t b = __ldg(row_ptr + row), e = __ldg(row_ptr + row + 1);
      csr_row_dot<R, NCV, NCA, LPR>(cols, vals, v, b + sub, e, acc);
    }
    acc.merge(LPR);
    if (sub == 0 && row < lim) acc.store(out, row);
  };
  if (chunk <= 0) {
    // Interleaved: consecutive warps of the grid take consecutive row groups.
    const int64_t w0 = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5;
    const int64_t nw = (int64_t(gridDim.x) * blockDim.x) >> 5;
    for (int64_t rb = w0 * RPW; rb < n_rows; rb += nw * RPW) one_step(rb, n_rows);
  } else {
    // Chunked: a block owns `chunk` consecutive rows at a time, so the source amplitudes its
    // rows share (same high-sector block, neighbouring rows) are reused from its L1.
    const int nwb = blockDim.x >> 5;
    for (int64_t c0 = int64_t(blockIdx.x) * chunk; c0 < n_rows; c0 += int64_t(gridDim.x) * chunk) {
      const int64_t lim = min(c0 + chunk, n_rows);
      for (int64_t rb = c0 + int64_t(warp) * RPW; rb < lim; rb += int64_t(nwb) * RPW)
        one_step(rb, lim);
    }
  }
}

template <typename R, int NCV, int NCA, int LPR>
__global__ void __launch_bounds__(256)
k_mv_xc(const int64_t* __restrict__ row_ptr, const uint32_t* __restrict__ cols,
        const uint32_t* __restrict__ grps, const uint64_t* __restrict__ states, int64_t n_unique,
        uint64_t fill_state, int has_diag, TermTable T, const R* __restrict__ v,
        R* __restrict__ out, int64_t n_rows) {
  constexpr int RPW = 32 / LPR;
  const int lane = threadIdx.x & 31;
  const int sub = lane % LPR, slot = lane / LPR;
  const int64_t w0 = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5;
  const int64_t nw = (int64_t(gridDim.x) * blockDim.x) >> 5;
  for (int64_t rb = w0 * RPW; rb < n_rows; rb += nw * RPW) {
    const int64_t row = rb + slot;
    const bool live = row < n_rows;
    CAcc<R, NCV, NCA> acc;
    int64_t b = 0, e = 0;
    uint64_t s = 0;
    if (live) {
      b = __ldg(row_ptr + row);
      e = __ldg(row_ptr + row + 1);
      s = row < n_unique ? __ldg(states + row) : fill_state;
    }
    // Diagonal group, lanes of the row split its terms.
    const bool diag = live && has_diag && e > b;
    Cx<double> d = cx_make<double>(0.0, 0.0);
    if (diag) d = compose<NCA, LPR>(T, __ldg(T.span), s, sub);
    for (int o = LPR >> 1; o > 0; o >>= 1) {
      d.re += __shfl_xor_sync(kFullMask, d.re, o);
      if constexpr (NCA == 2) d.im += __shfl_xor_sync(kFullMask, d.im, o);
    }
    if (diag && sub == 0)
      acc.add(cx_make<R>(R(d.re), R(d.im)), ld_elem<R, NCV>(v, __ldg(cols + b)));
    if (live) {
      for (int64_t i = b + (diag ? 1 : 0) + sub; i < e; i += LPR) {
        const Cx<R> x = ld_elem<R, NCV>(v, __ldg(cols + i));
        const Cx<double> el = compose<NCA>(T, __ldg(T.span + __ldg(grps + i)), s);
        acc.add(cx_make<R>(R(el.re), R(el.im)), x);
      }
    }
    acc.merge(LPR);
    if (sub == 0 && live) st_elem<R, NCV>(out, row, cx_make<R>(acc.re.value(), acc.im.value()));
  }
}

// Hv on a product subspace with elements composed on the fly, from the halves' partner lists
// alone (cache_strategy (1, 0), (1, 1) and (0, *) where the lists exist).  A block owns a tile of
// 32 high x 32 low strings.  A warp takes one high string for the tile's 32 low strings: its H
// pairs share their group across the lanes, so the table loads are one address a warp, and the
// amplitudes v[h'][l ..] one segment.  The L pairs share their group across the high strings
// instead: a warp takes one low string for 32 high strings and hands its sums over through shared
// memory (FP64).  The two-half pairs run lane by lane over A(h) x B(l), whose groups' terms lie
// together (ascending masks, high part first) and stay in L1.  No scratch vector: calls on
// several streams are independent.
// Bound by the L1 accesses of the two-half pairs' table entries, then by the terms' popcounts.
// 32 qubits, complex128: 320 x 288 strings 0.42 ms (28.6 ms when every (row, group) was tested
// against the subspace), 509 x 512 strings 1.44 ms (3.45 ms with stored sources and a lane per pair);
// L1TEX 88-90 % busy in the SMs that work.
constexpr int kTileStrings = 32;

template <typename R, int NCV, int NCA>
__global__ void __launch_bounds__(1024, 1)
k_mv_plan(PlanView c, TermTable T, const uint64_t* __restrict__ states, const R* __restrict__ v,
          R* __restrict__ out) {
  __shared__ double part[NCV][kTileStrings][kTileStrings + 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t th = (c.nh + kTileStrings - 1) / kTileStrings;
  const int64_t tl = (c.nl + kTileStrings - 1) / kTileStrings;
  for (int64_t t = blockIdx.x; t < th * tl; t += gridDim.x) {
    const int64_t h0 = (t / tl) * kTileStrings, l0 = (t % tl) * kTileStrings;
    // L pairs: low string l0 + warp, high strings h0 + lane.
    {
      const int64_t h = h0 + lane, l = l0 + warp;
      CAcc<R, NCV, NCA> acc;
      if (l < c.nl) {                      // the same for the whole warp
        const int64_t row0 = (h < c.nh ? h : c.nh - 1) * c.nl;
        const uint64_t s = __ldg(states + row0 + l);
        auto add = [&](uint2 span, int64_t src) {
          const Cx<R> x = ld_elem<R, NCV>(v, row0 + src);
          const Cx<double> el = compose<NCA>(T, span, s);
          acc.add(cx_make<R>(R(el.re), R(el.im)), x);
        };
        if (c.d) add(__ldg(T.span), l);
        const int64_t e = __ldg(c.loff + l + 1);
        for (int64_t i = __ldg(c.loff + l); i < e; ++i)
          add(__ldg(T.span + __ldg(c.key + i)), __ldg(c.part + i));
      }
      part[0][warp][lane] = acc.re.value_d();
      if constexpr (NCV == 2) part[1][warp][lane] = acc.im.value_d();
    }
    __syncthreads();
    // H and two-half pairs: high string h0 + warp, low strings l0 + lane.
    const int64_t h = h0 + warp, l = l0 + lane;
    if (h < c.nh) {
      const bool live = l < c.nl;
      const int64_t lc = live ? l : c.nl - 1;
      CAcc<R, NCV, NCA> acc;
      acc.re.add_d(part[0][lane][warp]);
      if constexpr (NCV == 2) acc.im.add_d(part[1][lane][warp]);
      const uint64_t s = __ldg(states + h * c.nl + lc);
      const int64_t e = __ldg(c.hoff + h + 1);
      for (int64_t i = __ldg(c.hoff + h); i < e; ++i) {
        const Cx<R> x = ld_elem<R, NCV>(v, int64_t(__ldg(c.part + i)) * c.nl + lc);
        const Cx<double> el = compose<NCA>(T, __ldg(T.span + __ldg(c.key + i)), s);
        acc.add(cx_make<R>(R(el.re), R(el.im)), x);
      }
      const int64_t b0 = __ldg(c.boff + lc), b1 = live ? __ldg(c.boff + lc + 1) : b0;
      const int64_t a1 = __ldg(c.aoff + h + 1);
      for (int64_t i = __ldg(c.aoff + h); i < a1; ++i) {
        const uint32_t a = __ldg(c.key + i);
        const int64_t base = int64_t(__ldg(c.part + i)) * c.nl;
        for (int64_t j = b0; j < b1; ++j) {
          const int32_t g = plan_group(c, a, __ldg(c.key + j));
          if (g < 0) continue;
          const Cx<R> x = ld_elem<R, NCV>(v, base + __ldg(c.part + j));
          const Cx<double> el = compose<NCA>(T, __ldg(T.span + g), s);
          acc.add(cx_make<R>(R(el.re), R(el.im)), x);
        }
      }
      if (live)
        st_elem<R, NCV>(out, h * c.nl + l, cx_make<R>(acc.re.value(), acc.im.value()));
    }
    __syncthreads();
  }
}

template <typename R, int NCV>
__global__ void k_zero_tail(R* out, int64_t from, int64_t to) {
  for (int64_t i = from + blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < to;
       i += int64_t(gridDim.x) * blockDim.x)
    st_elem<R, NCV>(out, i, cx_make<R>(0, 0));
}

// Fill-in slots under the uncached matvec: only the last slot connects (to the first fill-in
// slot, through the diagonal group evaluated at the all-ones state).
template <typename R, int NCV, int NCA>
__global__ void k_fill_tail(const R* v, R* out, int64_t n_unique, int64_t size,
                            uint64_t fill_state, const int64_t* gs, const int32_t* ge,
                            const uint64_t* tz, const double* tc) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  const int64_t b = gs[0];
  const int32_t K = ge[0];
  double dr = 0.0, di = 0.0;
  for (int32_t t = 0; t < K; ++t) {
    const bool neg = parity64(fill_state & tz[b + t]);
    dr += neg ? -tc[2 * (b + t)] : tc[2 * (b + t)];
    if constexpr (NCA == 2) di += neg ? -tc[2 * (b + t) + 1] : tc[2 * (b + t) + 1];
  }
  const Cx<R> x = ld_elem_rw<R, NCV>(v, n_unique);
  Cx<R> o;
  o.re = R(dr) * x.re - R(di) * x.im;
  o.im = R(dr) * x.im + R(di) * x.re;
  st_elem<R, NCV>(out, size - 1, o);
}

// Two vectors into one of interleaved elements (E: a real or complex element), and back.
template <typename E>
__global__ void k_interleave(const E* __restrict__ a, const E* __restrict__ b, E* __restrict__ out,
                             int64_t n) {
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x) {
    out[2 * i] = a[i];
    out[2 * i + 1] = b[i];
  }
}
template <typename E>
__global__ void k_deinterleave(const E* __restrict__ in, E* __restrict__ a, E* __restrict__ b,
                               int64_t n) {
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x) {
    a[i] = in[2 * i];
    b[i] = in[2 * i + 1];
  }
}

// From where the pair list is read for two vectors at once (op_pair_scratch).  FP64 iteration in us,
// pair / two matvecs, float64 and complex128 with real elements:
//   rows      16 a row          24               33               64
//   16,384                                                        65/65   71/71
//   32,768    64/63   69/68     68/67   74/73    68/68   76/76    78/81   87/87
//   65,536    78/77   86/85     83/85   93/93    86/87   95/98    100/107 118/120
//   131,072   105/106 120/118   113/117 132/132  119/122 142/141
//   262,144   164/164 203/193   188/194 231/234  204/210 252/259
//   1,048,576 326/348 464/460   402/440 563/592
// 16,384 rows of 129: 71/75 81/79, 30,600 of 108: 83/87 100/99; complex elements at 262,144 rows of
// 24: 256/284.
constexpr int64_t kPairMinRows[2] = {16384, 32768};   // real, complex vectors
constexpr int64_t kPairMinPerRow = 24, kPairMinPairs = int64_t(3) << 19;

unsigned mv_grid(int64_t rows, int lpr) {
  const int64_t warps = (rows * lpr + 31) / 32;
  const int64_t blocks = (warps + 7) / 8;
  const int64_t cap = static_cast<int64_t>(num_sms()) * 16;
  return static_cast<unsigned>(std::max<int64_t>(1, std::min(blocks, cap)));
}

}  // namespace

// Whether the composing matvec runs over the halves' lists (k_mv_plan) or, without them, over the
// stored pairs (k_mv_xc) or by searching (k_sweep).  Times at complex128 in us, lists / other.
//
// The lists' kernel looks up a group for every combination of A(h) x B(l), about 4.2 ps each on a
// full chip, found or not.  Without stored pairs the sweep costs 4.6 ps a (row, group) test and
// about 80 ps a pair; a share f of the tests of two-half groups finds one, f being that of the
// parts' partners that exist, so the lists are the better way while
//     combinations <= tests (1 + 19 f),   f = combinations / (rows na nb).
// All states of 16 qubits, strings of random Paulis on every qubit: 300 of them 8588 / 1722, 1000
// 14876 / 5632, 3000 15998 / 16468, 10000 19007 / 52520; molecular and local sums are far on the
// lists' side (320 x 288 strings at 32 qubits 420 / 28600).
//
// With stored pairs a pair costs k_mv_xc about 4 ps per term more than it costs the lists' kernel
// (terms of a group on one lane each against all lanes on the same group), which has to pay for the
// combinations: 16 qubits, all states, 1000 terms 707 / 416 (7 combinations and 1.1 terms a pair),
// 8000 2458 / 2770, 20000 3706 / 5933 (5.2 and 8).  And its blocks are few and long: 32 qubits, 64 x
// 64 strings 104 / 31, 128 x 128 179 / 80, 200 x 200 297 / 223, 220 x 200 (5.9 M pairs) 274 / 250, 230
// x 220 (7.2 M) 265 / 300, 64 x 800 (12 M) 370 / 531; 48 qubits, 250 x 250 (0.6 M) 119 / 90, 320 x 300
// (1.2 M) 127 / 129, 500 x 500 266 / 371; Ising chain of 16 qubits 15 / 12, of 18 29 / 43.  Fewer
// strings than half a tile in one half leave most lanes idle: 16 x 1820 (13 M pairs) 538 / 625, 12 x
// 1000 (3 M) 326 / 160, 3 x 1800 519 / 113.
bool op_plan_pays(const sqd_op_s* op) {
  const ProductPlan& q = *op->plan;
  const double rows = double(q.nh) * double(q.nl);
  const double combinations = double(q.ta) * double(q.tb);
  if (op->x_cache == 0) {
    const double parts = std::max(double(q.na) * double(q.nb), 1.0);
    return combinations * (1.0 - 19.0 * double(q.nm) / parts) <= rows * double(op->n_gpre);
  }
  const double terms = double(op->p->num_terms) / double(op->p->num_groups);
  if (combinations > terms * double(op->nnz) || std::min(q.nh, q.nl) < kTileStrings / 2)
    return false;
  return rows >= 90 * 1024 || op->nnz >= 6.5 * 1024 * 1024;
}

void op_matvec(sqd_op_s* op, const void* v, void* out, int dtype, cudaStream_t st) {
  sqd_paulis_s* p = op->p;
  sqd_space_s* sp = op->s;
  const int64_t size = sp->states_size;
  if (op->x_cache == 1 && op->z_cache == 2 && !dtype_is_double(dtype)) op_ensure_values32(op, st);
  if (op->x_cache == 1 && op->z_cache == 2 && op->prod.built &&
      op->layout[dtype_is_double(dtype) ? 0 : 1] != SQD_LAYOUT_CSR) {
    op_product_matvec(op, v, out, dtype, st);
    return;
  }
  dispatch_vec(dtype, op->value_complex, [&](auto rt, auto ncv_t, auto nca_t) {
    using R = typename decltype(rt)::type;
    constexpr int NCV = decltype(ncv_t)::value;
    constexpr int NCA = decltype(nca_t)::value;
    const R* vin = static_cast<const R*>(v);
    R* vout = static_cast<R*>(out);
    if (op->z_cache != 2 && op->plan && op_plan_pays(op)) {
      const int64_t tiles = ((op->plan->nh + kTileStrings - 1) / kTileStrings) *
                            ((op->plan->nl + kTileStrings - 1) / kTileStrings);
      k_mv_plan<R, NCV, NCA><<<static_cast<unsigned>(tiles), 1024, 0, st>>>(
          plan_view(*op->plan), term_table(p), sp->states.ptr, vin, vout);
      SQD_CHECK_LAUNCH();
      return;
    }
    if (op->x_cache == 1) {
      dispatch_lpr(op->lanes_per_row[sizeof(R) == 8 ? 0 : 1], [&](auto lpr_t) {
        constexpr int LPR = decltype(lpr_t)::value;
        const unsigned G = mv_grid(size, LPR);
        if (op->z_cache == 2) {
          const R* vals;
          if constexpr (sizeof(R) == 8) vals = op->values.ptr;
          else vals = op->values32.ptr;
          const int64_t chunk = op->chunk_rows[sizeof(R) == 8 ? 0 : 1];
          k_mv_csr<R, NCV, NCA, LPR><<<G, 256, 0, st>>>(op->row_ptr.ptr, op->cols.ptr, vals,
                                                        vin, vout, size, chunk);
        } else {
          k_mv_xc<R, NCV, NCA, LPR><<<G, 256, 0, st>>>(
              op->row_ptr.ptr, op->cols.ptr, op->grps.ptr, sp->states.ptr, sp->n_unique,
              sp->fill_state, op->has_diag_group, term_table(p), vin, vout, size);
        }
        SQD_CHECK_LAUNCH();
      });
      return;
    }
    // Uncached: sources searched in the matvec.
    SweepParams P = sweep_params(op);
    P.vin = v;
    P.vout = out;
    P.has_diag = op->has_diag_group;
    constexpr int kRows = 512;
    const size_t dyn = sweep_shared(P);
    auto kern = k_sweep<SWEEP_APPLY, R, NCV, NCA, kRows, 1>;
    SQD_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  static_cast<int>(dyn)));
    if (sp->n_unique > 0) {
      kern<<<grid_for(sp->n_unique, kRows), kRows, dyn, st>>>(P);
      SQD_CHECK_LAUNCH();
    }
    if (size > sp->n_unique) {
      k_zero_tail<R, NCV><<<grid_for(size - sp->n_unique, 256, 1024), 256, 0, st>>>(
          vout, sp->n_unique, size);
      SQD_CHECK_LAUNCH();
      if (op->has_diag_group) {
        k_fill_tail<R, NCV, NCA><<<1, 32, 0, st>>>(vin, vout, sp->n_unique, size, sp->fill_state,
                                                  p->group_start.ptr, p->group_eff.ptr,
                                                  p->term_z.ptr, p->term_c.ptr);
        SQD_CHECK_LAUNCH();
      }
    }
  });
}

// Two FP64 vectors share one pass over the elements.  Interleaving them costs four reads and
// writes of each vector, so it pays where a row has many more pairs than that.  Real vectors
// become one complex vector over the same (real) elements.  On the pair list every component is
// summed as it is alone, bit for bit; on the product layouts the twice as long elements may take
// another number of high-string partners at a time, or leave the one-launch form, which adds the
// same products in another order.
size_t op_pair_scratch(const sqd_op_s* op, int nc) {
  if (op->x_cache != 1 || op->z_cache != 2) return 0;
  const int64_t n = op->s->states_size;
  // The product layouts' five launches per matvec make the pair the better way at every size
  // (100 x 98 strings 120 / 136 us an iteration).
  const bool product = op->prod.built && op->layout[0] != SQD_LAYOUT_CSR;
  if (!product && (n < kPairMinRows[nc - 1] || op->nnz < kPairMinPairs ||
                   op->nnz < kPairMinPerRow * n))
    return 0;
  return static_cast<size_t>(n) * nc * 4 + (product && nc == 2 ? static_cast<size_t>(n) * 16 : 0);
}

void op_matvec_pair(sqd_op_s* op, const void* v0, void* out0, const void* v1, void* out1, int nc,
                    double* scratch, cudaStream_t st) {
  const int64_t n = op->s->states_size;
  double* in = scratch;
  double* out = scratch + n * nc * 2;
  double* rest = scratch + n * nc * 4;
  const unsigned G = grid_for(n, 256, num_sms() * 16);
  if (nc == 1)
    k_interleave<double><<<G, 256, 0, st>>>(static_cast<const double*>(v0),
                                            static_cast<const double*>(v1), in, n);
  else
    k_interleave<double2><<<G, 256, 0, st>>>(static_cast<const double2*>(v0),
                                             static_cast<const double2*>(v1),
                                             reinterpret_cast<double2*>(in), n);
  SQD_CHECK_LAUNCH();
  if (nc == 1) {
    op_matvec(op, in, out, SQD_C128, st);
  } else if (op->prod.built && op->layout[0] != SQD_LAYOUT_CSR) {
    op_product_matvec_pair(op, in, out, rest, st);
  } else {
    dispatch_lpr(op->lanes_per_row[0], [&](auto lpr_t) {
      constexpr int LPR = decltype(lpr_t)::value;
      const unsigned GM = mv_grid(n, LPR);
      if (op->value_complex)
        k_mv_csr<double, 4, 2, LPR><<<GM, 256, 0, st>>>(op->row_ptr.ptr, op->cols.ptr,
                                                        op->values.ptr, in, out, n,
                                                        op->chunk_rows[0]);
      else
        k_mv_csr<double, 4, 1, LPR><<<GM, 256, 0, st>>>(op->row_ptr.ptr, op->cols.ptr,
                                                        op->values.ptr, in, out, n,
                                                        op->chunk_rows[0]);
      SQD_CHECK_LAUNCH();
    });
  }
  if (nc == 1)
    k_deinterleave<double><<<G, 256, 0, st>>>(out, static_cast<double*>(out0),
                                              static_cast<double*>(out1), n);
  else
    k_deinterleave<double2><<<G, 256, 0, st>>>(reinterpret_cast<const double2*>(out),
                                               static_cast<double2*>(out0),
                                               static_cast<double2*>(out1), n);
  SQD_CHECK_LAUNCH();
}

}  // namespace sqd

using namespace sqd;

extern "C" int sqd_matvec(sqd_op_t op, const void* v, void* out, int dtype, void* stream) {
  return guarded([&] {
    SQD_REQUIRE(op != nullptr && v != nullptr && out != nullptr, "NULL argument");
    SQD_REQUIRE(v != out, "sqd_matvec cannot work in place");
    op_matvec(op, v, out, dtype, as_stream(stream));
  });
}
