// Matrix elements of the stored pairs: the composed diagonals C^(j)_i (sqd.py:95-98), summed term
// by term in the reference's order (get_diagonal, sqd.py:603-628; compose() in internal.cuh).
//
// A term costs a 16-byte table load, a 64-bit AND, one popcount and one FP64 add, so a full warp
// on uniform loads is popcount-bound (16 a clock and SM).  What keeps a kernel away from that is
// the table access (a warp whose lanes hold different groups takes one L1 line per lane and
// waits for its longest group) and the diagonal, whose hundreds of terms are one pair of a row
// (one lane of the warp that serves the row).  So:
//  * the diagonal is a kernel of its own, a thread per row, every lane on the same term;
//  * in a large product subspace (ProductPlan) the H pairs are computed with a warp on 32 rows of
//    one slab and the L pairs with a warp on 32 rows of one low string: the lanes share the group;
//  * the other pairs take a lane each; groups of more than kLongGroup terms wait in a queue in
//    shared memory until 32 of them run together.
// 48 qubits, 1152 x 1000 strings, 46 M pairs: 1.55 ms (L with the 1,129-term diagonals 1.04, H 0.34,
// the rest 0.16) against 22.6 ms as one lane per pair, diagonal included; 131,072 random states of
// 40 qubits with a 2,400-term diagonal: 0.14 against 2.02 ms.
#include "internal.cuh"

namespace sqd {
namespace {

template <int NCA>
__device__ __forceinline__ void put(double* out, int64_t i, Cx<double> v, bool out_complex) {
  if (NCA == 2 || out_complex) {
    reinterpret_cast<double2*>(out)[i] = make_double2(v.re, v.im);
  } else {
    out[i] = v.re;
  }
}

// First entry of every row that starts with the diagonal group: real rows, and the last fill-in
// slot (at the all-ones state).
template <int NCA>
__global__ void __launch_bounds__(128)
k_diag_elements(TermTable T, const int64_t* __restrict__ row_ptr,
                const uint64_t* __restrict__ states, int64_t n_unique, uint64_t fill_state,
                int64_t size, double* out, int out_complex) {
  const uint2 sp = __ldg(T.span);
  for (int64_t r = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; r < size;
       r += int64_t(gridDim.x) * blockDim.x) {
    const bool real = r < n_unique;
    if (!real && r != size - 1) continue;
    const uint64_t s = real ? __ldg(states + r) : fill_state;
    put<NCA>(out, row_ptr[r], compose<NCA>(T, sp, s), out_complex);
  }
}

constexpr unsigned kLongGroup = 24;
constexpr int kQueue = 64;   // per warp; at most 31 wait when a row's 32 lanes add theirs

struct LongPair {
  uint64_t state;
  int64_t at;
  uint2 span;
};

// Pairs of row r from row_ptr[r] + skip (PLAN: after the row's diagonal, H and L entries).
template <int NCA, bool PLAN>
__global__ void __launch_bounds__(256)
k_pair_elements(TermTable T, const int64_t* __restrict__ row_ptr,
                const uint32_t* __restrict__ grps, const uint64_t* __restrict__ states,
                int64_t n_rows, int skip, PlanView plan, double* out, int out_complex) {
  __shared__ LongPair queue[8][kQueue];
  LongPair* mine = queue[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const int64_t w0 = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5;
  const int64_t nw = (int64_t(gridDim.x) * blockDim.x) >> 5;
  int waiting = 0;
  auto run_long = [&](int count) {   // the last `count` entries
    __syncwarp();
    if (lane < count) {
      const LongPair e = mine[waiting - count + lane];
      put<NCA>(out, e.at, compose<NCA>(T, e.span, e.state), out_complex);
    }
    waiting -= count;
    __syncwarp();
  };
  for (int64_t r = w0; r < n_rows; r += nw) {
    const uint64_t s = __ldg(states + r);
    int64_t b = __ldg(row_ptr + r) + skip;
    const int64_t e = __ldg(row_ptr + r + 1);
    if constexpr (PLAN) {
      const int64_t h = r / plan.nl, l = r - h * plan.nl;
      b += (__ldg(plan.hoff + h + 1) - __ldg(plan.hoff + h)) +
           (__ldg(plan.loff + l + 1) - __ldg(plan.loff + l));
    }
    for (int64_t i0 = b; i0 < e; i0 += 32) {
      const int64_t i = i0 + lane;
      uint2 sp = make_uint2(0, 0);
      if (i < e) sp = __ldg(T.span + __ldg(grps + i));
      const bool later = i < e && sp.y > kLongGroup;
      const unsigned b_later = __ballot_sync(kFullMask, later);
      if (later) {
        LongPair q;
        q.state = s;
        q.at = i;
        q.span = sp;
        mine[waiting + __popc(b_later & lt)] = q;
      }
      waiting += __popc(b_later);
      if (i < e && !later) put<NCA>(out, i, compose<NCA>(T, sp, s), out_complex);
      if (waiting >= 32) run_long(32);
    }
  }
  if (waiting) run_long(waiting);
}

// Slab position of entry k at position b (product.cu): 32-wide panels, and for FP32 copies of
// even-sized halves 64-wide ones.
__device__ __forceinline__ int64_t slab_at(int64_t k, int64_t b, int64_t total, int shift) {
  return (((b >> shift) * total + k) << shift) + (b & ((int64_t(1) << shift) - 1));
}

template <int NCA>
__device__ __forceinline__ void put_slab(double* v, float* v32, int64_t k, int64_t b,
                                         int64_t total, int wide, Cx<double> el) {
  if (v) put<NCA>(v, slab_at(k, b, total, 5), el, false);
  if (v32) {
    const int64_t i = slab_at(k, b, total, wide ? 6 : 5);
    if constexpr (NCA == 2)
      reinterpret_cast<float2*>(v32)[i] =
          make_float2(static_cast<float>(el.re), static_cast<float>(el.im));
    else
      v32[i] = static_cast<float>(el.re);
  }
}

template <int NCA>
__device__ __forceinline__ Cx<double> get(const double* v, int64_t i) {
  return ld_elem<double, NCA>(v, i);
}

// One warp: the entries of list string a (HIGH: high string a, L: low string a, its diagonal
// entry first) for 32 strings b of the other half.  All lanes are on the same group.  COPY: the
// elements are read back from the pair list (values) instead of composed.
template <int NCA, bool HIGH, bool COPY>
__global__ void __launch_bounds__(256)
k_half_elements(TermTable T, PlanView c, const int64_t* __restrict__ row_ptr,
                const uint64_t* __restrict__ states, double* values, int out_complex, double* slab,
                float* slab32, int wide, int64_t total) {
  const int lane = threadIdx.x & 31;
  const int64_t A = HIGH ? c.nh : c.nl, B = HIGH ? c.nl : c.nh;
  const int64_t panels = (B + 31) >> 5;
  const int64_t w0 = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5;
  const int64_t nw = (int64_t(gridDim.x) * blockDim.x) >> 5;
  const int64_t* off = HIGH ? c.hoff : c.loff;
  const int64_t first = __ldg(off);
  for (int64_t w = w0; w < A * panels; w += nw) {
    const int64_t a = w / panels;   // a block's warps share the string's groups
    const int64_t b = (w - a * panels) * 32 + lane;
    const bool live = b < B;
    const int64_t r = live ? (HIGH ? a * c.nl + b : b * c.nl + a) : 0;
    const uint64_t s = __ldg(states + r);
    const int64_t k0 = __ldg(off + a), k1 = __ldg(off + a + 1);
    const int d = c.d;
    int64_t at = 0;
    if (values) {
      at = __ldg(row_ptr + r) + d;
      if constexpr (!HIGH) at += live ? __ldg(c.hoff + b + 1) - __ldg(c.hoff + b) : 0;
    }
    int64_t k = k0 - first + (HIGH ? 0 : d * a);   // entry index over all strings
    if constexpr (!HIGH) {
      if (d) {
        const Cx<double> el = COPY ? get<NCA>(values, __ldg(row_ptr + r))
                                   : compose<NCA>(T, __ldg(T.span), s);
        if (live) {
          if (!COPY && values) put<NCA>(values, __ldg(row_ptr + r), el, out_complex);
          put_slab<NCA>(slab, slab32, k, b, total, wide, el);
        }
        ++k;
      }
    }
    for (int64_t i = k0; i < k1; ++i, ++k) {
      const Cx<double> el = COPY ? get<NCA>(values, at + (i - k0))
                                 : compose<NCA>(T, __ldg(T.span + __ldg(c.key + i)), s);
      if (live) {
        if (!COPY && values) put<NCA>(values, at + (i - k0), el, out_complex);
        put_slab<NCA>(slab, slab32, k, b, total, wide, el);
      }
    }
  }
}

// H and L elements into o (copy: read from the pair list o.values).
template <int NCA, bool COPY>
void half_elements(sqd_op_s* op, const ElementOut& o, cudaStream_t st) {
  const ProductPlan& q = *op->plan;
  const PlanView c = plan_view(q);
  const TermTable T = term_table(op->p);
  const uint64_t* states = op->s->states.ptr;
  const int64_t total_l = q.tl + q.d * q.nl;
  if (q.th > 0) {
    k_half_elements<NCA, true, COPY>
        <<<grid_for(q.nh * ((q.nl + 31) / 32) * 32, 256, num_sms() * 64), 256, 0, st>>>(
            T, c, op->row_ptr.ptr, states, o.values, o.out_complex, o.vh, o.vh32, o.wide32, q.th);
    SQD_CHECK_LAUNCH();
  }
  if (total_l > 0) {
    k_half_elements<NCA, false, COPY>
        <<<grid_for(q.nl * ((q.nh + 31) / 32) * 32, 256, num_sms() * 64), 256, 0, st>>>(
            T, c, op->row_ptr.ptr, states, o.values, o.out_complex, o.vl, o.vl32, o.wide32,
            total_l);
    SQD_CHECK_LAUNCH();
  }
}

// Whether the halves' kernels compute the elements of a product subspace.  A warp of theirs sums a
// string's whole list, the diagonal's hundreds of terms with it, so they need strings enough to
// fill the chip and both halves wide enough to fill the lanes.  Refresh in us, halves / rows: 32
// qubits, 64 x 64 strings 104 / 45, 128 x 128 157 / 83, 180 x 170 204 / 135, 256 x 240 315 / 300, 400 x
// 360 712 / 1030, 32 x 1800 627 / 700, 64 x 800 353 / 348, 12 x 1000 318 / 121, 1 x 1820 486 / 68; 48
// qubits, 100 x 100 94 / 78, 300 x 300 131 / 153.
bool halves_pay(const ProductPlan& q) {
  return q.nh * q.nl >= 56 * 1024 && std::min(q.nh, q.nl) >= 32;
}

template <int NCA>
void pair_elements(sqd_op_s* op, const ElementOut& o, cudaStream_t st) {
  sqd_space_s* sp = op->s;
  const TermTable T = term_table(op->p);
  const int64_t size = sp->states_size, nu = sp->n_unique;
  if (op->plan && halves_pay(*op->plan)) {
    half_elements<NCA, false>(op, o, st);
    if (op->plan->ta > 0 && op->plan->tb > 0) {
      k_pair_elements<NCA, true><<<grid_for(nu * 32, 256, num_sms() * 64), 256, 0, st>>>(
          T, op->row_ptr.ptr, op->grps.ptr, sp->states.ptr, nu, op->has_diag_group,
          plan_view(*op->plan), o.values, o.out_complex);
      SQD_CHECK_LAUNCH();
    }
    return;
  }
  if (op->has_diag_group) {
    k_diag_elements<NCA><<<grid_for(size, 128), 128, 0, st>>>(
        T, op->row_ptr.ptr, sp->states.ptr, nu, sp->fill_state, size, o.values, o.out_complex);
    SQD_CHECK_LAUNCH();
  }
  k_pair_elements<NCA, false><<<grid_for(nu * 32, 256, num_sms() * 64), 256, 0, st>>>(
      T, op->row_ptr.ptr, op->grps.ptr, sp->states.ptr, nu, op->has_diag_group, PlanView{},
      o.values, o.out_complex);
  SQD_CHECK_LAUNCH();
  if (o.vh || o.vh32) half_elements<NCA, true>(op, o, st);
}

}  // namespace

void op_pair_elements(sqd_op_s* op, const ElementOut& out, cudaStream_t st) {
  if (op->value_complex) pair_elements<2>(op, out, st);
  else pair_elements<1>(op, out, st);
}

void op_slab_elements(sqd_op_s* op, const ElementOut& out, cudaStream_t st) {
  if (op->value_complex) half_elements<2, true>(op, out, st);
  else half_elements<1, true>(op, out, st);
}

}  // namespace sqd
