// Connectivity of a product subspace from its half strings (SQD_LOOKUP_PRODUCT).
//
// The (row, group) sweep tests every group against every row.  In a product of high-half and
// low-half strings a group acting on one half connects a row iff the row's string of that half
// has a partner, so the partners are searched once per string of the half, and a two-half group
// connects (h, l) iff both halves have partners.  The lists of partners (ProductPlan) are a few
// hundred entries per string; the stored pairs of every row, when they are kept, are assembled
// from them in the sweep's order: diagonal, H groups, L groups, M groups, each class in ascending
// group index (= ascending x: for M groups, ascending high part, then low part).
#include "internal.cuh"

namespace sqd {
namespace {

__device__ __forceinline__ void warp_count_add(unsigned long long c, unsigned long long* dst) {
  for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(kFullMask, c, o);
  if ((threadIdx.x & 31) == 0 && c) atomicAdd(dst, c);
}

// Number of distinct high strings (rows whose high half differs from the previous row's).
__global__ void k_count_slabs(const uint64_t* __restrict__ s, int64_t n, uint64_t mhi,
                              unsigned long long* cnt) {
  unsigned long long c = 0;
  for (int64_t r = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; r < n;
       r += int64_t(gridDim.x) * blockDim.x)
    if (r == 0 || ((s[r] ^ s[r - 1]) & mhi) != 0) ++c;
  warp_count_add(c, cnt);
}

// Rows that are not H[r / nl] | L[r % nl].
__global__ void k_check_product(const uint64_t* __restrict__ s, int64_t n, int64_t nl,
                                uint64_t mlo, uint64_t mhi, unsigned long long* bad) {
  unsigned long long c = 0;
  for (int64_t r = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; r < n;
       r += int64_t(gridDim.x) * blockDim.x) {
    const int64_t l = r % nl;
    const uint64_t v = s[r];
    if (((v ^ s[l]) & mlo) != 0 || ((v ^ s[r - l]) & mhi) != 0) ++c;
  }
  warp_count_add(c, bad);
}

__global__ void k_half_strings(const uint64_t* __restrict__ s, int64_t count, int64_t stride,
                               uint64_t mask, uint64_t* out) {
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < count;
       i += int64_t(gridDim.x) * blockDim.x)
    out[i] = s[i * stride] & mask;
}

// Masks and groups of one class as arrays; with mask, that part of the masks only.
__global__ void k_split_groups(const GroupPre* __restrict__ g, int64_t n, uint64_t mask,
                               uint64_t* x, int32_t* group) {
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x) {
    x[i] = g[i].x & mask;
    if (group) group[i] = g[i].group;
  }
}

__global__ void k_run_heads(const uint64_t* __restrict__ x, int64_t n, int64_t* head) {
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x)
    head[i] = (i == 0 || x[i] != x[i - 1]) ? 1 : 0;
}

__global__ void k_run_values(const uint64_t* __restrict__ x, const int64_t* __restrict__ head,
                             const int64_t* __restrict__ pos, int64_t n, uint64_t* out) {
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x)
    if (head[i]) out[pos[i]] = x[i];
}

__global__ void k_mtable(const uint64_t* __restrict__ xm, const int32_t* __restrict__ gm, int64_t n,
                         uint64_t mlo, uint64_t mhi, const uint64_t* __restrict__ xa, int64_t na,
                         const uint64_t* __restrict__ xb, int64_t nb, int32_t* table) {
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x)
    table[sorted_find(xa, na, xm[i] & mhi) * nb + sorted_find(xb, nb, xm[i] & mlo)] = gm[i];
}

// Partner lists of all four classes in one launch: one block per (class, string), its warps
// take consecutive stretches of the class's masks and ballots keep the mask order.  COUNT writes
// the entries per (string, warp), whose scan gives every warp its place for FILL.  With the
// halves' weights conserved (weighed), a mask can only have a partner when it moves as many bits
// up as down, one popcount instead of a search (48 qubits: 22 % of the masks pass; both passes
// take 0.47 ms for 1152 x 1000 strings, one warp per string and a search per mask took 1.4 ms).
// Beyond kListStrings strings they are enough for one warp each, which keeps the counts small.
constexpr int kListWarps = 8;
constexpr int64_t kListStrings = 1 << 16;
constexpr int64_t kListBlocks = 1 << 20;   // grid; beyond, a block takes several strings
struct ListSearch {
  const uint64_t* strs[4];
  int64_t first[5];           // first block of each class; [4] = all blocks
  const uint64_t* xs[4];
  const int32_t* ids[4];      // key of mask k, NULL = k itself
  int64_t nx[4], nstr[4];
  int weighed, warps;
};

template <bool FILL>
__global__ void __launch_bounds__(kListWarps * 32)
k_partner_lists(ListSearch q, int64_t* counts, const int64_t* __restrict__ place, uint32_t* key,
                uint32_t* part) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  for (int64_t blk = blockIdx.x; blk < q.first[4]; blk += gridDim.x) {
    int c = 0;
    while (c < 3 && blk >= q.first[c + 1]) ++c;
    const uint64_t* __restrict__ strs = q.strs[c];
    const uint64_t* __restrict__ xs = q.xs[c];
    const int64_t nstr = q.nstr[c], nx = q.nx[c];
    const uint64_t base = __ldg(strs + (blk - q.first[c]));
    const int64_t seg = (nx + q.warps - 1) / q.warps;
    const int64_t k0 = warp * seg, k1 = min(nx, k0 + seg);
    const int64_t slot = blk * q.warps + warp;
    int64_t pos = FILL ? place[slot] : 0;
    for (int64_t kb = k0; kb < k1; kb += 32) {
      const int64_t k = kb + lane;
      int64_t found = -1;
      if (k < k1) {
        const uint64_t x = __ldg(xs + k);
        if (!q.weighed || 2 * __popcll(base & x) == __popcll(x))
          found = sorted_find(strs, nstr, base ^ x);
      }
      const unsigned b = __ballot_sync(kFullMask, found >= 0);
      if (FILL && found >= 0) {
        const int64_t i = pos + __popc(b & lt);
        key[i] = q.ids[c] ? static_cast<uint32_t>(__ldg(q.ids[c] + k)) : static_cast<uint32_t>(k);
        part[i] = static_cast<uint32_t>(found);
      }
      pos += __popc(b);
    }
    if (!FILL && lane == 0) counts[slot] = pos;
  }
}

__global__ void k_every(const int64_t* __restrict__ in, int64_t n, int stride, int64_t* out) {
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x)
    out[i] = in[i * stride];
}

__global__ void k_row_counts(PlanView c, int64_t* counts) {
  const int64_t n = c.nh * c.nl;
  for (int64_t r = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; r < n;
       r += int64_t(gridDim.x) * blockDim.x) {
    const int64_t h = r / c.nl, l = r - h * c.nl;
    const int64_t a0 = c.aoff[h], a1 = c.aoff[h + 1], b0 = c.boff[l], b1 = c.boff[l + 1];
    int64_t m = 0;
    for (int64_t i = a0; i < a1; ++i)
      for (int64_t j = b0; j < b1; ++j) m += plan_group(c, c.key[i], c.key[j]) >= 0;
    counts[r] = c.d + (c.hoff[h + 1] - c.hoff[h]) + (c.loff[l + 1] - c.loff[l]) + m;
  }
}

// One warp per row, lanes over the row's entries, so the pair lists are written in whole lines
// (0.30 ms for 46 M pairs; a thread per row wrote every entry to a line of its own: 0.82 ms).
__global__ void __launch_bounds__(256)
k_row_pairs(PlanView c, const int64_t* __restrict__ row_ptr, uint32_t* __restrict__ cols,
            uint32_t* __restrict__ grps) {
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const int64_t n = c.nh * c.nl;
  const int64_t w0 = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5;
  const int64_t nw = (int64_t(gridDim.x) * blockDim.x) >> 5;
  for (int64_t r = w0; r < n; r += nw) {
    const int64_t h = r / c.nl, l = r - h * c.nl;
    const int64_t h0 = __ldg(c.hoff + h), l0 = __ldg(c.loff + l);
    const int nkh = static_cast<int>(__ldg(c.hoff + h + 1) - h0);
    const int nkl = static_cast<int>(__ldg(c.loff + l + 1) - l0);
    int64_t p = row_ptr[r];
    if (c.d) {
      if (lane == 0) {
        cols[p] = static_cast<uint32_t>(r);
        grps[p] = 0;
      }
      ++p;
    }
    for (int i = lane; i < nkh; i += 32) {
      cols[p + i] = static_cast<uint32_t>(int64_t(__ldg(c.part + h0 + i)) * c.nl + l);
      grps[p + i] = __ldg(c.key + h0 + i);
    }
    p += nkh;
    for (int i = lane; i < nkl; i += 32) {
      cols[p + i] = static_cast<uint32_t>(h * c.nl + __ldg(c.part + l0 + i));
      grps[p + i] = __ldg(c.key + l0 + i);
    }
    p += nkl;
    const int64_t a0 = __ldg(c.aoff + h), b0 = __ldg(c.boff + l);
    const unsigned nA = static_cast<unsigned>(__ldg(c.aoff + h + 1) - a0);
    const unsigned nB = static_cast<unsigned>(__ldg(c.boff + l + 1) - b0);
    const unsigned total = nA * nB;   // at most nh * nl < 2^31 (distinct masks, distinct partners)
    for (unsigned q0 = 0; q0 < total; q0 += 32) {
      const unsigned q = q0 + lane;
      int32_t g = -1;
      uint32_t col = 0;
      if (q < total) {
        const unsigned i = q / nB, j = q - i * nB;
        g = plan_group(c, __ldg(c.key + a0 + i), __ldg(c.key + b0 + j));
        col = static_cast<uint32_t>(int64_t(__ldg(c.part + a0 + i)) * c.nl + __ldg(c.part + b0 + j));
      }
      const unsigned b = __ballot_sync(kFullMask, g >= 0);
      if (g >= 0) {
        cols[p + __popc(b & lt)] = col;
        grps[p + __popc(b & lt)] = static_cast<uint32_t>(g);
      }
      p += __popc(b);
    }
  }
}

// Distinct values of a sorted array; returns their number.
int64_t distinct(const uint64_t* x, int64_t n, DevBuf<uint64_t>& out, cudaStream_t st) {
  if (n == 0) {
    out.alloc(1, st);
    return 0;
  }
  DevBuf<int64_t> head, pos;
  head.alloc(n, st);
  pos.alloc(n + 1, st);
  const unsigned G = grid_for(n, 256, 4096);
  k_run_heads<<<G, 256, 0, st>>>(x, n, head.ptr);
  SQD_CHECK_LAUNCH();
  exclusive_scan_i64(head.ptr, pos.ptr, n, true, st);
  int64_t count = 0;
  copy_to_host(&count, pos.ptr + n, 1, st);
  out.alloc(count, st);
  k_run_values<<<G, 256, 0, st>>>(x, head.ptr, pos.ptr, n, out.ptr);
  SQD_CHECK_LAUNCH();
  return count;
}

}  // namespace

bool op_product_detect(sqd_op_s* op, cudaStream_t st, int64_t* nh_out, int64_t* nl_out) {
  sqd_space_s* sp = op->s;
  const int64_t n = sp->n_unique;
  *nh_out = *nl_out = 0;
  if (n == 0 || sp->states_size != n || sp->num_qubits < 2) return false;
  const uint64_t mlo = half_mask_low(sp->num_qubits), mhi = sp->fill_state & ~mlo;
  DevBuf<unsigned long long> cnt;
  cnt.alloc(2, st);
  SQD_CUDA(cudaMemsetAsync(cnt.ptr, 0, 2 * sizeof(unsigned long long), st));
  const unsigned G = grid_for(n, 256, 4096);
  k_count_slabs<<<G, 256, 0, st>>>(sp->states.ptr, n, mhi, cnt.ptr);
  SQD_CHECK_LAUNCH();
  unsigned long long nh = 0;
  copy_to_host(&nh, cnt.ptr, 1, st);
  if (nh == 0 || n % static_cast<int64_t>(nh) != 0) return false;
  const int64_t nl = n / static_cast<int64_t>(nh);
  k_check_product<<<G, 256, 0, st>>>(sp->states.ptr, n, nl, mlo, mhi, cnt.ptr + 1);
  SQD_CHECK_LAUNCH();
  unsigned long long bad = 0;
  copy_to_host(&bad, cnt.ptr + 1, 1, st);
  if (bad) return false;
  *nh_out = static_cast<int64_t>(nh);
  *nl_out = nl;
  return true;
}

bool op_plan(sqd_op_s* op, cudaStream_t st, int64_t most) {
  if (op->plan) return true;
  auto plan = std::make_unique<ProductPlan>();
  ProductPlan& q = *plan;
  if (!op_product_detect(op, st, &q.nh, &q.nl)) return false;
  sqd_space_s* sp = op->s;
  const uint64_t mlo = half_mask_low(sp->num_qubits), mhi = sp->fill_state & ~mlo;
  q.d = op->has_diag_group;
  // Masks of each class (op->gpre: H, L, M in that order, ascending group index in each).
  const int64_t n0 = op->n_gpre_cls[0], n1 = op->n_gpre_cls[1], nm = op->n_gpre_cls[2];
  q.nm = nm;
  DevBuf<uint64_t> hstr, lstr, xh, xl;
  DevBuf<int32_t> gh, gl;
  hstr.alloc(q.nh, st);
  lstr.alloc(q.nl, st);
  k_half_strings<<<grid_for(q.nh, 256, 4096), 256, 0, st>>>(sp->states.ptr, q.nh, q.nl, mhi,
                                                            hstr.ptr);
  k_half_strings<<<grid_for(q.nl, 256, 4096), 256, 0, st>>>(sp->states.ptr, q.nl, 1, mlo,
                                                            lstr.ptr);
  SQD_CHECK_LAUNCH();
  auto split = [&](int64_t first, int64_t n, uint64_t mask, DevBuf<uint64_t>& x,
                   DevBuf<int32_t>* g) {
    x.alloc(std::max<int64_t>(n, 1), st);
    if (g) g->alloc(std::max<int64_t>(n, 1), st);
    if (n == 0) return;
    k_split_groups<<<grid_for(n, 256, 4096), 256, 0, st>>>(op->gpre.ptr + first, n, mask, x.ptr,
                                                           g ? g->ptr : nullptr);
    SQD_CHECK_LAUNCH();
  };
  split(0, n0, ~0ull, xh, &gh);
  split(n0, n1, ~0ull, xl, &gl);
  split(n0 + n1, nm, ~0ull, q.xm, &q.gm);
  // Distinct high parts (M masks ascend, so equal high parts are neighbours) and low parts.
  {
    DevBuf<uint64_t> part;
    split(n0 + n1, nm, mhi, part, nullptr);
    q.na = distinct(part.ptr, nm, q.xa, st);
    split(n0 + n1, nm, mlo, part, nullptr);
    radix_sort_u64(part.ptr, nullptr, nm, sp->num_qubits / 2, st);
    q.nb = distinct(part.ptr, nm, q.xb, st);
  }
  if (nm > 0 && double(q.na) * double(q.nb) <= double(1 << 24)) {
    q.mtable.alloc(static_cast<size_t>(q.na * q.nb), st);
    SQD_CUDA(cudaMemsetAsync(q.mtable.ptr, 0xff, q.mtable.bytes(), st));
    k_mtable<<<grid_for(nm, 256, 4096), 256, 0, st>>>(q.xm.ptr, q.gm.ptr, nm, mlo, mhi, q.xa.ptr,
                                                      q.na, q.xb.ptr, q.nb, q.mtable.ptr);
    SQD_CHECK_LAUNCH();
  }
  ListSearch f{};
  const int64_t nstr[4] = {q.nh, q.nl, q.nh, q.nl};
  const int64_t nx[4] = {n0, n1, q.na, q.nb};
  const uint64_t* xs[4] = {xh.ptr, xl.ptr, q.xa.ptr, q.xb.ptr};
  int64_t blocks = 0;
  for (int c = 0; c < 4; ++c) {
    f.strs[c] = c % 2 == 0 ? hstr.ptr : lstr.ptr;
    f.xs[c] = xs[c];
    f.nx[c] = nx[c];
    f.nstr[c] = nstr[c];
    f.first[c] = blocks;
    blocks += nstr[c];
  }
  f.first[4] = blocks;
  f.ids[0] = gh.ptr;
  f.ids[1] = gl.ptr;
  f.weighed = sp->num_sectors == 2 ? 1 : 0;
  f.warps = blocks <= kListStrings ? kListWarps : 1;
  const unsigned G = static_cast<unsigned>(std::min(blocks, kListBlocks));
  DevBuf<int64_t> counts, place;
  counts.alloc(blocks * f.warps, st);
  place.alloc(blocks * f.warps + 1, st);
  k_partner_lists<false><<<G, static_cast<unsigned>(f.warps * 32), 0, st>>>(
      f, counts.ptr, nullptr, nullptr, nullptr);
  SQD_CHECK_LAUNCH();
  exclusive_scan_i64(counts.ptr, place.ptr, blocks * f.warps, true, st);
  q.offs.alloc(blocks + 1, st);
  k_every<<<grid_for(blocks + 1, 256, 4096), 256, 0, st>>>(place.ptr, blocks + 1, f.warps,
                                                           q.offs.ptr);
  SQD_CHECK_LAUNCH();
  int64_t end[4];
  for (int c = 0; c < 4; ++c)
    SQD_CUDA(cudaMemcpyAsync(end + c, q.offs.ptr + f.first[c + 1], sizeof(int64_t),
                             cudaMemcpyDeviceToHost, st));
  SQD_CUDA(cudaStreamSynchronize(st));
  q.th = end[0];
  q.tl = end[1] - end[0];
  q.ta = end[2] - end[1];
  q.tb = end[3] - end[2];
  if (end[3] > most) return false;
  q.key.alloc(std::max<int64_t>(end[3], 1), st);
  q.part.alloc(std::max<int64_t>(end[3], 1), st);
  k_partner_lists<true><<<G, static_cast<unsigned>(f.warps * 32), 0, st>>>(
      f, nullptr, place.ptr, q.key.ptr, q.part.ptr);
  SQD_CHECK_LAUNCH();
  op->plan = std::move(plan);
  return true;
}

bool op_connect_product(sqd_op_s* op, cudaStream_t st) {
  if (!op_plan(op, st)) return false;
  const PlanView c = plan_view(*op->plan);
  const int64_t n = c.nh * c.nl;
  DevBuf<int64_t> counts;
  counts.alloc(n, st);
  k_row_counts<<<grid_for(n, 256, 16384), 256, 0, st>>>(c, counts.ptr);
  SQD_CHECK_LAUNCH();
  op->row_ptr.alloc(n + 1, st);
  exclusive_scan_i64(counts.ptr, op->row_ptr.ptr, n, true, st);
  copy_to_host(&op->nnz, op->row_ptr.ptr + n, 1, st);
  counts.release();
  op->cols.alloc(op->nnz > 0 ? op->nnz : 1, st);
  op->grps.alloc(op->nnz > 0 ? op->nnz : 1, st);
  k_row_pairs<<<grid_for(n * 32, 256, num_sms() * 64), 256, 0, st>>>(c, op->row_ptr.ptr, op->cols.ptr,
                                                               op->grps.ptr);
  SQD_CHECK_LAUNCH();
  op->product_built = 1;
  return true;
}

}  // namespace sqd
