// Hellmann-Feynman per-term reduction  g_t = Re sum_i conj(u_i) ph_t (-1)^{|s_i & z_t|} v_src(i),
// ph_t = (-i)^{|x & z_t|}, for every merged term t.
//
//  * Product subspaces (ProductPlan): a block or warp owns a group, so its terms' sums stay in
//    registers and are stored once.  Long groups (a few masks on many states, as in lattice models)
//    have several owners, each adding its sums once.  An H group x joins the pairs (h, h') of high
//    strings with every low string, an L group the other way round, a two-half group the pairs of
//    its high part with the pairs of its low part; the pairs per group come from the halves' lists
//    sorted by key.
//  * Other subspaces: a lane per stored pair and one atomic addition per term.
//  * The diagonal group: blocks of 1,024 rows by up to 64 terms, a warp per term.
// Bound by the terms' popcounts and adds.  32 qubits, 256 x 240 strings, complex128: H 0.14, L 0.17,
// two-half groups 0.07 ms (1.1 ms together with an atomic per pair and term); the diagonal under
// 0.03 ms (0.29 ms with one block per row tile taking the terms one after the other).  All states of
// 20 qubits, float64: an Ising chain 0.54 ms (one owner per group 15.1, an atomic per pair and term
// 3.8), a Heisenberg chain 0.57 (28.8, 13.4).
#include "internal.cuh"
#include "dispatch.cuh"

namespace sqd {
namespace {

// w = conj(u) v
template <int NCV>
__device__ __forceinline__ double2 overlap(Cx<double> a, Cx<double> b) {
  if constexpr (NCV == 1) return make_double2(a.re * b.re, 0.0);
  return make_double2(a.re * b.re + a.im * b.im, a.re * b.im - a.im * b.re);
}

// Re((-i)^ph (-1)^{|s & z|} w)
__device__ __forceinline__ double signed_part(double wr, double wi, int ph, uint64_t s,
                                              uint64_t z) {
  const double v = (ph & 1) ? wi : wr;
  const uint64_t m = s & z;
  const uint64_t flip = static_cast<uint64_t>(
      __popc(static_cast<unsigned>(m) ^ static_cast<unsigned>(m >> 32)) + (ph >> 1)) << 63;
  return __longlong_as_double(__double_as_longlong(v) ^ static_cast<long long>(flip));
}

// Diagonal group (x = 0, src = i, phase 1); a block takes every gridDim.y-th batch of terms.
constexpr int GR_TILE = 1024, GR_TERMS = 64;

template <int NCV>
__global__ void __launch_bounds__(256)
k_grad_diag(const uint64_t* __restrict__ states, int64_t n_unique, TermTable T,
            const double* __restrict__ u, const double* __restrict__ v, double* g) {
  __shared__ uint64_t s_st[GR_TILE];
  __shared__ double s_w[GR_TILE];
  const uint2 sp = __ldg(T.span);
  if (blockIdx.y * GR_TERMS >= sp.y) return;
  const int64_t r0 = static_cast<int64_t>(blockIdx.x) * GR_TILE;
  for (int k = threadIdx.x; k < GR_TILE; k += blockDim.x) {
    const int64_t r = r0 + k;
    const bool live = r < n_unique;
    s_st[k] = live ? __ldg(states + r) : 0;
    s_w[k] = live ? overlap<NCV>(ld_elem<double, NCV>(u, r), ld_elem<double, NCV>(v, r)).x : 0.0;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (unsigned t0 = blockIdx.y * GR_TERMS; t0 < sp.y; t0 += gridDim.y * GR_TERMS) {
    for (unsigned t = t0 + warp; t < min(t0 + GR_TERMS, sp.y); t += 8) {
      const uint64_t z = __ldg(T.rec + sp.x + t).x;
      double a = 0.0;
#pragma unroll 4
      for (int k = lane; k < GR_TILE; k += 32) a += signed_part(s_w[k], 0.0, 0, s_st[k], z);
      a = warp_sum(a);
      if (lane == 0) atomicAdd(g + sp.x + t, a);
    }
  }
}

// Off-diagonal stored pairs: per pair, loop over the group's terms and atomically add.
template <int NCV>
__global__ void k_grad_offdiag(const int64_t* row_ptr, const uint32_t* cols,
                               const uint32_t* grps, const uint64_t* states, int64_t n_unique,
                               int has_diag, TermTable T, const uint64_t* gx, const double* u,
                               const double* v, double* g) {
  const int lane = threadIdx.x & 31;
  const int64_t w0 = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5;
  const int64_t nw = (int64_t(gridDim.x) * blockDim.x) >> 5;
  for (int64_t r = w0; r < n_unique; r += nw) {
    const uint64_t s = states[r];
    const Cx<double> a = ld_elem<double, NCV>(u, r);
    const int64_t b = row_ptr[r] + has_diag, e = row_ptr[r + 1];
    for (int64_t i = b + lane; i < e; i += 32) {
      const uint32_t j = __ldg(grps + i);
      const double2 w = overlap<NCV>(a, ld_elem<double, NCV>(v, __ldg(cols + i)));
      const uint64_t x = __ldg(gx + j);
      const uint2 sp = __ldg(T.span + j);
      for (uint32_t t = sp.x; t < sp.x + sp.y; ++t) {
        const uint64_t z = __ldg(T.rec + t).x;
        atomicAdd(g + t, signed_part(w.x, w.y, __popcll(x & z) & 3, s, z));
      }
    }
  }
}

// ---- product subspaces ----------------------------------------------------------------------
// The halves' list entries sorted by (class, key): the string and its partner.
__global__ void k_entry_keys(PlanView c, int64_t th, int64_t tl, int64_t ta, int64_t tb,
                             uint64_t* keys, uint32_t* index) {
  const int64_t n = th + tl + ta + tb;
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x) {
    const uint64_t cls = i < th ? 0 : i < th + tl ? 1 : i < th + tl + ta ? 2 : 3;
    keys[i] = (cls << 32) | c.key[i];
    index[i] = static_cast<uint32_t>(i);
  }
}

__global__ void k_entry_pairs(PlanView c, const uint64_t* __restrict__ keys,
                              const uint32_t* __restrict__ index, int64_t n, uint32_t* key,
                              uint2* pair) {
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x) {
    const int cls = static_cast<int>(keys[i] >> 32);
    const int64_t e = index[i];
    const int64_t* off = cls == 0 ? c.hoff : cls == 1 ? c.loff : cls == 2 ? c.aoff : c.boff;
    int64_t lo = 0, hi = cls % 2 == 0 ? c.nh : c.nl;   // the last string that starts at or before e
    while (hi - lo > 1) {
      const int64_t mid = (lo + hi) >> 1;
      if (off[mid] <= e) lo = mid; else hi = mid;
    }
    key[i] = static_cast<uint32_t>(keys[i]);
    pair[i] = make_uint2(static_cast<uint32_t>(lo), c.part[e]);
  }
}

__device__ __forceinline__ int64_t first_of(const uint32_t* __restrict__ key, int64_t n,
                                            uint32_t want) {
  int64_t lo = 0, hi = n;
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if (__ldg(key + mid) < want) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// The longest run of one key in each class.
__global__ void k_longest_runs(const uint32_t* __restrict__ key, int64_t th, int64_t tl,
                               int64_t ta, int64_t tb, unsigned long long* longest) {
  const int64_t n = th + tl + ta + tb;
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x) {
    const int cls = i < th ? 0 : i < th + tl ? 1 : i < th + tl + ta ? 2 : 3;
    const int64_t first = cls == 0 ? 0 : cls == 1 ? th : cls == 2 ? th + tl : th + tl + ta;
    const int64_t count = cls == 0 ? th : cls == 1 ? tl : cls == 2 ? ta : tb;
    if (i > first && key[i] == key[i - 1]) continue;
    atomicMax(longest + cls, static_cast<unsigned long long>(
                                 first_of(key + first, count, key[i] + 1) - (i - first)));
  }
}

// Owners of a group (blocks of k_grad_half, warps of k_grad_mixed): one, unless the longest group
// has more than `most` pairs or there are too few groups to fill the chip (`room` owners), then
// shares of at least `least` pairs.  At most kOwners over all groups.
constexpr int64_t kOwners = 1 << 16;
constexpr int64_t kHalfLeast = 1024, kHalfMost = 16384, kMixedLeast = 256, kMixedMost = 4096;
unsigned owners(int64_t longest, int64_t groups, int64_t least, int64_t most, int64_t room) {
  groups = std::max<int64_t>(groups, 1);
  const int64_t split = std::min((longest + most - 1) / most, kOwners / groups);
  const int64_t fill = std::min((longest + least - 1) / least, (room + groups - 1) / groups);
  return static_cast<unsigned>(std::min<int64_t>(std::max({split, fill, int64_t(1)}), 65535));
}

// One block per H (HIGH) or L group and share of its pairs: 256 pairs at a time in shared memory,
// each warp sums up to eight of 64 terms over them.
template <int NCV, bool HIGH, bool SPLIT>
__global__ void __launch_bounds__(256)
k_grad_half(PlanView c, TermTable T, const GroupPre* __restrict__ groups,
            const uint32_t* __restrict__ key, const uint2* __restrict__ pair, int64_t count,
            const uint64_t* __restrict__ states, const double* __restrict__ u,
            const double* __restrict__ v, double* g) {
  __shared__ uint64_t s_st[256];
  __shared__ double s_wr[256], s_wi[NCV == 2 ? 256 : 1];
  __shared__ int64_t range[2];
  const GroupPre grp = groups[blockIdx.x];
  const uint32_t j = static_cast<uint32_t>(grp.group);
  const uint2 sp = __ldg(T.span + j);
  if (threadIdx.x < 2) range[threadIdx.x] = first_of(key, count, j + threadIdx.x);
  __syncthreads();
  const int64_t first = range[0];
  const int64_t ni = range[1] - first;
  if (ni == 0) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t total = ni * (HIGH ? c.nl : c.nh);
  int64_t begin = 0, end = total;
  if constexpr (SPLIT) {
    const int64_t even = (total + gridDim.y - 1) / gridDim.y;
    const int64_t share = max(kHalfLeast, (even + 255) / 256 * 256);
    begin = blockIdx.y * share;
    end = min(total, begin + share);
    if (begin >= total) return;
  }
  for (unsigned t0 = 0; t0 < sp.y; t0 += 64) {
    const unsigned left = sp.y - t0;
    const int mine = left > static_cast<unsigned>(warp) ? min(8u, (left - warp + 7) / 8) : 0;
    double acc[8];
    uint64_t z[8];
    int ph[8];
#pragma unroll
    for (int m = 0; m < 8; ++m) {
      acc[m] = 0.0;
      z[m] = m < mine ? __ldg(T.rec + sp.x + t0 + warp + 8 * m).x : 0;
      ph[m] = __popcll(grp.x & z[m]) & 3;
    }
    for (int64_t q0 = begin; q0 < end; q0 += 256) {
      const int64_t q = q0 + threadIdx.x;
      uint64_t s = 0;
      double2 w = make_double2(0.0, 0.0);
      if (q < end) {
        int64_t r, src;
        if constexpr (HIGH) {
          const int64_t i = q / c.nl, l = q - i * c.nl;
          const uint2 p = __ldg(pair + first + i);
          r = p.x * c.nl + l;
          src = p.y * c.nl + l;
        } else {
          const int64_t h = q / ni;
          const uint2 p = __ldg(pair + first + (q - h * ni));
          r = h * c.nl + p.x;
          src = h * c.nl + p.y;
        }
        s = __ldg(states + r);
        w = overlap<NCV>(ld_elem<double, NCV>(u, r), ld_elem<double, NCV>(v, src));
      }
      __syncthreads();
      s_st[threadIdx.x] = s;
      s_wr[threadIdx.x] = w.x;
      if constexpr (NCV == 2) s_wi[threadIdx.x] = w.y;
      __syncthreads();
      for (int e = lane; e < 256; e += 32) {
        const uint64_t se = s_st[e];
        const double wr = s_wr[e], wi = NCV == 2 ? s_wi[e] : 0.0;
#pragma unroll
        for (int m = 0; m < 8; ++m)
          if (m < mine) acc[m] += signed_part(wr, wi, ph[m], se, z[m]);
      }
    }
#pragma unroll
    for (int m = 0; m < 8; ++m) {
      if (m < mine) {
        const double a = warp_sum(acc[m]);
        if (lane == 0) {
          double* at = g + sp.x + t0 + warp + 8 * m;
          if (SPLIT && end - begin < total) atomicAdd(at, a);
          else *at = a;
        }
      }
    }
  }
}

// One warp per two-half group and share of its pairs, eight terms at a time.
template <int NCV, bool SPLIT>
__global__ void __launch_bounds__(256)
k_grad_mixed(PlanView c, TermTable T, const GroupPre* __restrict__ groups, int64_t n_groups,
             uint64_t mlo, uint64_t mhi, int64_t na, const uint32_t* __restrict__ akey,
             const uint2* __restrict__ apair, int64_t ta, const uint32_t* __restrict__ bkey,
             const uint2* __restrict__ bpair, int64_t tb, const uint64_t* __restrict__ states,
             const double* __restrict__ u, const double* __restrict__ v, double* g) {
  const int lane = threadIdx.x & 31;
  const int64_t w0 = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5;
  const int64_t nw = (int64_t(gridDim.x) * blockDim.x) >> 5;
  for (int64_t k = w0; k < n_groups; k += nw) {
    const GroupPre grp = groups[k];
    const uint2 sp = __ldg(T.span + grp.group);
    const uint32_t a = static_cast<uint32_t>(sorted_find(c.xa, na, grp.x & mhi));
    const uint32_t b = static_cast<uint32_t>(sorted_find(c.xb, c.nb, grp.x & mlo));
    const int64_t a0 = first_of(akey, ta, a), b0 = first_of(bkey, tb, b);
    const unsigned nA = static_cast<unsigned>(first_of(akey, ta, a + 1) - a0);
    const unsigned nB = static_cast<unsigned>(first_of(bkey, tb, b + 1) - b0);
    const unsigned total = nA * nB;       // at most nh * nl
    const unsigned share = max(static_cast<unsigned>(kMixedLeast),
                               (total + gridDim.y - 1) / gridDim.y);
    const unsigned begin = SPLIT ? min(total, blockIdx.y * share) : 0;   // total < 2^31
    const unsigned end = SPLIT ? min(total, begin + share) : total;
    if (begin == end) continue;
    for (unsigned t0 = 0; t0 < sp.y; t0 += 8) {
      const int mine = min(8u, sp.y - t0);
      double acc[8];
      uint64_t z[8];
      int ph[8];
#pragma unroll
      for (int m = 0; m < 8; ++m) {
        acc[m] = 0.0;
        z[m] = m < mine ? __ldg(T.rec + sp.x + t0 + m).x : 0;
        ph[m] = __popcll(grp.x & z[m]) & 3;
      }
      for (unsigned q = begin + lane; q < end; q += 32) {
        const unsigned i = q / nB;
        const uint2 ph_ = __ldg(apair + a0 + i), pl = __ldg(bpair + b0 + (q - i * nB));
        const int64_t r = ph_.x * c.nl + pl.x, src = ph_.y * c.nl + pl.y;
        const uint64_t s = __ldg(states + r);
        const double2 w = overlap<NCV>(ld_elem<double, NCV>(u, r), ld_elem<double, NCV>(v, src));
#pragma unroll
        for (int m = 0; m < 8; ++m)
          if (m < mine) acc[m] += signed_part(w.x, w.y, ph[m], s, z[m]);
      }
#pragma unroll
      for (int m = 0; m < 8; ++m) {
        if (m < mine) {
          const double s = warp_sum(acc[m]);
          if constexpr (SPLIT) {
            if (lane == 0) atomicAdd(g + sp.x + t0 + m, s);
          } else {
            if (lane == 0) g[sp.x + t0 + m] = s;
          }
        }
      }
    }
  }
}

// The sorted lists, on the first gradient (kept with the plan).  Not during a stream capture,
// whose allocations would belong to the graph.
bool plan_groups(sqd_op_s* op, cudaStream_t st) {
  if (!op->plan) return false;
  ProductPlan& q = *op->plan;
  std::lock_guard<std::mutex> lock(q.gmutex);
  if (q.gkey.ptr) return true;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  SQD_CUDA(cudaStreamIsCapturing(st, &cap));
  if (cap != cudaStreamCaptureStatusNone) return false;
  const int64_t n = q.th + q.tl + q.ta + q.tb;
  if (n >= (int64_t(1) << 31)) return false;   // more than the sort takes: a lane per stored pair
  DevBuf<uint64_t> keys;
  DevBuf<uint32_t> index, gkey;
  DevBuf<uint2> gpair;
  DevBuf<unsigned long long> longest;
  unsigned long long runs[4] = {0, 0, 0, 0};
  try {
    longest.alloc(4, st);
    keys.alloc(std::max<int64_t>(n, 1), st);
    index.alloc(std::max<int64_t>(n, 1), st);
    gkey.alloc(std::max<int64_t>(n, 1), st);
    gpair.alloc(std::max<int64_t>(n, 1), st);
    if (n > 0) {
      const unsigned G = grid_for(n, 256, 4096);
      k_entry_keys<<<G, 256, 0, st>>>(plan_view(q), q.th, q.tl, q.ta, q.tb, keys.ptr, index.ptr);
      SQD_CHECK_LAUNCH();
      radix_sort_u64(keys.ptr, index.ptr, n, 34, st);
      k_entry_pairs<<<G, 256, 0, st>>>(plan_view(q), keys.ptr, index.ptr, n, gkey.ptr, gpair.ptr);
      SQD_CHECK_LAUNCH();
      SQD_CUDA(cudaMemsetAsync(longest.ptr, 0, longest.bytes(), st));
      k_longest_runs<<<G, 256, 0, st>>>(gkey.ptr, q.th, q.tl, q.ta, q.tb, longest.ptr);
      SQD_CHECK_LAUNCH();
      SQD_CUDA(cudaMemcpyAsync(runs, longest.ptr, longest.bytes(), cudaMemcpyDeviceToHost, st));
    }
  } catch (const Error& e) {   // no memory: a lane per stored pair
    if (e.status != SQD_ERR_MEMORY) throw;
    (void)cudaGetLastError();
    return false;
  }
  SQD_CUDA(cudaStreamSynchronize(st));   // later calls may come on other streams
  for (int c = 0; c < 4; ++c) q.longest[c] = static_cast<int64_t>(runs[c]);
  q.gkey = std::move(gkey);
  q.gpair = std::move(gpair);
  return true;
}

template <int NCV>
void grad_terms(sqd_op_s* op, const double* u, const double* v, double* g, cudaStream_t st) {
  sqd_paulis_s* p = op->p;
  sqd_space_s* sp = op->s;
  const TermTable T = term_table(p);
  if (op->has_diag_group && sp->n_unique > 0) {
    const unsigned chunks = static_cast<unsigned>(
        std::min<int64_t>((p->max_k + GR_TERMS - 1) / GR_TERMS, 65535));
    k_grad_diag<NCV><<<dim3(grid_for(sp->n_unique, GR_TILE), chunks), 256, 0, st>>>(
        sp->states.ptr, sp->n_unique, T, u, v, g);
    SQD_CHECK_LAUNCH();
  }
  if (plan_groups(op, st)) {
    const ProductPlan& q = *op->plan;
    const PlanView c = plan_view(q);
    const uint32_t* key = q.gkey.ptr;
    const uint2* pair = q.gpair.ptr;
    const int64_t n0 = op->n_gpre_cls[0], n1 = op->n_gpre_cls[1], n2 = op->n_gpre_cls[2];
    // SPLIT: G.y owners per group
    const int64_t room = 8 * num_sms();
    auto half = [&](auto high, const GroupPre* groups, int64_t n, int64_t first, int64_t count,
                    int64_t longest) {
      constexpr bool HIGH = decltype(high)::value != 0;
      const dim3 G(static_cast<unsigned>(n), owners(longest, n, kHalfLeast, kHalfMost, room));
      auto kern = G.y > 1 ? k_grad_half<NCV, HIGH, true> : k_grad_half<NCV, HIGH, false>;
      kern<<<G, 256, 0, st>>>(c, T, groups, key + first, pair + first, count, sp->states.ptr, u,
                              v, g);
      SQD_CHECK_LAUNCH();
    };
    if (q.th > 0) half(IntTag<1>{}, op->gpre.ptr, n0, 0, q.th, q.longest[0] * c.nl);
    if (q.tl > 0) half(IntTag<0>{}, op->gpre.ptr + n0, n1, q.th, q.tl, q.longest[1] * c.nh);
    if (q.ta > 0 && q.tb > 0) {
      const uint64_t mlo = half_mask_low(sp->num_qubits), mhi = sp->fill_state & ~mlo;
      const int64_t oa = q.th + q.tl, ob = oa + q.ta;
      const dim3 G(grid_for(n2 * 32, 256, num_sms() * 64),
                   owners(q.longest[2] * q.longest[3], n2, kMixedLeast, kMixedMost, 8 * room));
      auto kern = G.y > 1 ? k_grad_mixed<NCV, true> : k_grad_mixed<NCV, false>;
      kern<<<G, 256, 0, st>>>(c, T, op->gpre.ptr + n0 + n1, n2, mlo, mhi, q.na, key + oa,
                              pair + oa, q.ta, key + ob, pair + ob, q.tb, sp->states.ptr, u, v, g);
      SQD_CHECK_LAUNCH();
    }
    return;
  }
  k_grad_offdiag<NCV><<<grid_for(sp->n_unique * 32, 256, 16384), 256, 0, st>>>(
      op->row_ptr.ptr, op->cols.ptr, op->grps.ptr, sp->states.ptr, sp->n_unique,
      op->has_diag_group, T, p->group_x.ptr, u, v, g);
  SQD_CHECK_LAUNCH();
}

}  // namespace
}  // namespace sqd

using namespace sqd;

extern "C" int sqd_grad_terms(sqd_op_t op, const void* u, const void* v, int dtype,
                              double* out_terms, void* stream) {
  return guarded([&] {
    SQD_REQUIRE(op != nullptr && u && v && out_terms, "NULL argument");
    SQD_REQUIRE(op->x_cache == 1, "the coefficient gradient needs cache_strategy x = 1");
    SQD_REQUIRE(op->nnz == 0 || op->grps.ptr != nullptr,
                "the operator released its group indices; create a new operator");
    SQD_REQUIRE(dtype == SQD_F64 || dtype == SQD_C128, "gradient dtype must be F64 or C128");
    SQD_REQUIRE(dtype == SQD_C128 || !op->value_complex, "complex Hamiltonian needs C128");
    cudaStream_t st = as_stream(stream);
    SQD_CUDA(cudaMemsetAsync(out_terms, 0, op->p->num_terms * sizeof(double), st));
    const double* ud = static_cast<const double*>(u);
    const double* vd = static_cast<const double*>(v);
    if (dtype == SQD_C128) grad_terms<2>(op, ud, vd, out_terms, st);
    else grad_terms<1>(op, ud, vd, out_terms, st);
  });
}
