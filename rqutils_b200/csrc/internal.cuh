// Internal handle layouts shared by the library's translation units.
#pragma once

#include <mutex>

#include "common.cuh"

// Grouped Pauli table (device CSR).  Mirrors PauliSumXZ (paulis/symplectic.py:41-48): groups
// ascending in x, terms ascending in z inside a group, coefficients already multiplied by
// (-i)^{popcount(x & z)}.
struct sqd_paulis_s {
  int num_qubits = 0;
  int64_t num_raw = 0;
  int64_t num_terms = 0;   // M (merged)
  int64_t num_groups = 0;  // J
  int64_t max_k = 0;       // largest group
  int is_complex = 0;      // any phased coefficient with a nonzero imaginary part
  sqd::DevBuf<uint64_t> group_x;      // [J]
  sqd::DevBuf<int64_t> group_start;   // [J+1]
  sqd::DevBuf<int32_t> group_eff;     // [J] terms used by the diagonal (stop at first zero)
  sqd::DevBuf<uint64_t> term_z;       // [M]
  sqd::DevBuf<double> term_c;         // [2M] interleaved (re, im)
  sqd::DevBuf<int32_t> term_group;    // [M]
  // The same table packed for the kernels that compose elements: one 8-byte load gives a
  // group's terms, one 16-byte load a term's mask and real coefficient.
  sqd::DevBuf<uint2> group_span;      // [J] (first term, group_eff)
  sqd::DevBuf<ulonglong2> term_rec;   // [M] (z, bits of Re c)
  uint64_t version = 0;               // bumped by sqd_paulis_set_coeffs
  sqd::DevBuf<int32_t> raw_to_term;   // [num_raw]
  // term -> raw terms merged into it, in input order (for coefficient updates)
  int64_t num_kept = 0;
  uint32_t flags = 0;
  sqd::DevBuf<int64_t> term_raw_start;  // [M + 1] into term_raw
  sqd::DevBuf<uint32_t> term_raw;       // [num_kept] raw indices
  sqd::DevBuf<uint64_t> term_x;         // [M]
};

// Sorted unique subspace plus lookup structures.
struct sqd_space_s {
  int num_qubits = 0;
  int64_t n_unique = 0;
  int64_t states_size = 0;
  uint64_t fill_state = 0;            // all-ones over the qubit bits (the 255 rows' diagonal)
  sqd::DevBuf<uint64_t> states;       // [n_unique]
  // Open-addressing hash table (linear probing, load <= 1/2): key -> row index.
  sqd::DevBuf<uint64_t> hkeys;
  sqd::DevBuf<uint32_t> hvals;
  uint64_t hmask = 0;
  // Conserved-weight sectors: popcount(s & sector_mask[l]) == sector_weight[l] for every state.
  int num_sectors = 0;
  uint64_t sector_mask[2] = {0, 0};
  int sector_weight[2] = {0, 0};
  // Membership filter of the sweep: 2^filter_log2 bits, bit filter_bit(s) set for every state s,
  // at least eight bits per state up to kFilterMax.
  sqd::DevBuf<uint32_t> filter;
  int filter_log2 = 0;
};

constexpr int kFilterMin = 10, kFilterMax = 28;
constexpr int kFilterShared = 20;     // largest filter that the sweep keeps in shared memory

namespace sqd {
// Low half of the qubits (bits 0 .. n/2 - 1): the low sector of the conserved-weight sectors and
// of the product layout.
inline uint64_t half_mask_low(int num_qubits) {
  const int h = num_qubits / 2;
  return h == 0 ? 0ull : ((1ull << h) - 1ull);
}
}  // namespace sqd

// Per-group data for the connectivity sweep.
struct GroupPre {
  uint64_t x;
  int32_t group;     // group index j
  int32_t cx;        // popcount(x & sector_mask[l]) packed as bytes (l = 0, 1)
};

// Product-subspace layout of the cached matvec (product.cu).  Rows r = h * nl + l.  H entries
// of slab h: k in [ho[h], ho[h+1]), source offset hsrc[k] = h' * nl, elements vh at
// panel-major ((l / 32) * th + k) * 32 + l % 32; L entries of low string l: e in
// [lo[l], lo[l+1]), source offset lsrc[e] = l' * nh (into the transposed vector), elements vl
// at ((h / 32) * tl + e) * 32 + h % 32.  The rest of a row (M pairs) stays in the CSR arrays
// after the first (ho[h+1] - ho[h]) + (lo[l+1] - lo[l]) pairs.
struct ProductLayout {
  int built = 0;
  int64_t nh = 0, nl = 0;
  int64_t th = 0, tl = 0;            // H and L entries over all slabs
  int64_t pairs_h = 0, pairs_l = 0, pairs_m = 0;
  sqd::DevBuf<int64_t> ho, lo;       // [nh + 1], [nl + 1]
  sqd::DevBuf<uint32_t> hsrc, lsrc;  // [th], [tl]
  sqd::DevBuf<double> vh, vl;        // FP64 elements (x2 interleaved when complex)
  sqd::DevBuf<float> vh32, vl32;     // FP32 copies (64-wide panels when wide32)
  int wide32 = 0;                    // both halves even: FP32 slabs read two positions per lane
  sqd::DevBuf<double> vt, tt, t;     // per-matvec scratch: transposed input, L and M partials
  sqd::DevBuf<double> t2;            // H partial (small grids only)
  // Two-half (M) pairs.  Panel form (SQD_LAYOUT_PRODUCT, product.cu k_tail_panels): the low
  // strings sorted by the length of their B list (perm, 0xffffffff in the padding) in panels of
  // 32, panel p with panel_at[p + 1] - panel_at[p] steps; element of A entry k, step t, lane at
  // ((k * steps + panel_at[p] + t) * 32 + lane); source l' of a step at
  // panel_src[(panel_at[p] + t) * 32 + lane], nl in the padding.  horder: high strings by the
  // length of their A list, longest first.  panel_full: every combination's group exists;
  // otherwise absent elements are marked (kAbsent*).
  int panel_state = 0;               // 0 not tried, 1 built, -1 does not apply
  int64_t panels = 0, steps = 0;
  sqd::DevBuf<int32_t> panel_at;     // [panels + 1]
  sqd::DevBuf<uint32_t> perm;        // [panels * 32]
  sqd::DevBuf<uint16_t> panel_src;   // [steps * 32]
  sqd::DevBuf<uint32_t> horder;      // [nh]
  int panel_full = 0;
  int panel32_state = 0;             // -1: no memory for the FP32 copy
  sqd::DevBuf<double> vm;            // [ta * steps * 32] (x2 interleaved when complex)
  sqd::DevBuf<float> vm32;
  // Otherwise the CSR kernel runs over the row tails: in place, or over a contiguous copy when
  // they are short (row offsets, elements, source rows).
  int tail_state = 0;                // 0 not tried, 1 copied, -1 read in place
  sqd::DevBuf<int64_t> mptr;         // [n + 1]
  sqd::DevBuf<uint32_t> mcol;        // [pairs_m]
  sqd::DevBuf<double> mval;          // [pairs_m] (x2 interleaved when complex)
  sqd::DevBuf<float> mval32;
};

// Connectivity of a product subspace by half strings (connect.cu): rows r = h * nl + l.  Four
// lists of (key, partner) entries, each string's entries in ascending mask order:
//   H: X masks on the high half only,  key = group, partner h' (H[h'] = H[h] ^ x);
//   L: X masks on the low half only,   key = group, partner l';
//   A: distinct high parts of the two-half masks, key = index a, partner h';
//   B: distinct low parts of the two-half masks,  key = index b, partner l'.
// A two-half group connects (h, l) for every (a in A(h), b in B(l)) whose group exists.  The
// lists take a few hundred entries per string, so an operator without cached sources keeps
// them too, unless they are long or its matvec has no use for them (op_plan_pays).
struct ProductPlan {
  int64_t nh = 0, nl = 0;
  int d = 0;                          // the diagonal group exists
  int64_t th = 0, tl = 0, ta = 0, tb = 0;   // entries per list
  sqd::DevBuf<int64_t> offs;          // [2 nh + 2 nl + 1]: H, L, A, B offsets into key / part
  sqd::DevBuf<uint32_t> key, part;
  int64_t na = 0, nb = 0, nm = 0;
  sqd::DevBuf<int32_t> mtable;        // [na * nb] group of (a, b) or -1 (dense form)
  sqd::DevBuf<uint64_t> xa, xb, xm;   // distinct parts; two-half masks, ascending (sparse form)
  sqd::DevBuf<int32_t> gm;            // [nm] groups of xm
  // The lists' entries by (class, key), for sums per group (grad.cu, on first use): key and
  // (string, partner); classes H, L, A, B one after the other.
  sqd::DevBuf<uint32_t> gkey;
  sqd::DevBuf<uint2> gpair;
  int64_t longest[4] = {0, 0, 0, 0};  // entries of one key at most, per class
  std::mutex gmutex;                  // gradients of one operator from several threads
};

// Solver objects an operator keeps between LOCG solves (locg.cu): work vectors and the
// instantiated CUDA graphs of the iteration, rebuilt when the matvec schedule changes.
struct LocgCacheBase {
  virtual ~LocgCacheBase() = default;
};

constexpr uint64_t kUnsettled = ~0ull;   // values_version after a refresh

struct sqd_op_s {
  sqd_paulis_s* p = nullptr;   // borrowed: must outlive the operator
  sqd_space_s* s = nullptr;    // borrowed
  int x_cache = 1, z_cache = 0, lookup = SQD_LOOKUP_HASH;
  int has_diag_group = 0;      // group 0 has x == 0
  int value_complex = 0;
  int64_t nnz = 0;
  int lanes_per_row[2] = {32, 32};  // [0]: FP64 vectors, [1]: FP32 vectors
  int lanes_chosen[2] = {0, 0};     // set by the caller: also for the tails' CSR kernel
  int64_t chunk_rows[2] = {0, 0};   // rows a block owns at a time (0 = interleaved rows)
  sqd::DevBuf<int64_t> row_ptr;   // [states_size + 1]
  sqd::DevBuf<uint32_t> cols;     // [nnz] source index of each stored pair
  sqd::DevBuf<uint32_t> grps;     // [nnz] group index of each stored pair
  sqd::DevBuf<double> values;     // [nnz] or [2 nnz]: composed diagonal per stored pair
  sqd::DevBuf<float> values32;    // FP32 copy for the mixed-precision matvec
  sqd::DevBuf<GroupPre> gpre;     // groups that can connect (x != 0, even sector counts)
  int64_t n_gpre = 0;
  int64_t n_gpre_cls[3] = {0, 0, 0};  // gpre entries per class (H, L, M), in that order
  int product_built = 0;          // connectivity assembled from the two halves' lists
  std::unique_ptr<ProductPlan> plan;  // product subspaces: the halves' lists
  uint64_t values_version = 0;    // p->version of elements whose computation has been waited for
  int layout[2] = {0, 0};         // SQD_LAYOUT_* per precision
  ProductLayout prod;
  // Bumped whenever the kernels or buffers a matvec launches may change (lanes, chunk,
  // layout, coefficient refresh): cached solver graphs captured before are then stale.
  uint64_t schedule_version = 0;
  std::unique_ptr<LocgCacheBase> locg_cache;
};

namespace sqd {

// Lanes that share a row of the CSR kernels, from the mean number of pairs per row.
inline int lanes_for(double avg) {
  return avg >= 96 ? 32 : avg >= 40 ? 16 : avg >= 16 ? 8 : avg >= 6 ? 4 : 2;
}

// The packed Pauli table as the kernels read it.
struct TermTable {
  const uint2* span;
  const ulonglong2* rec;
  const double* c;
};
inline TermTable term_table(const sqd_paulis_s* p) {
  return TermTable{p->group_span.ptr, p->term_rec.ptr, p->term_c.ptr};
}

// Composed diagonal of a group (its span) at state s, term by term in the reference's order
// (get_diagonal, sqd.py:603-628): sums of c or -c by the parity of s & z.  STEP > 1: every
// STEP-th term from `first` on, one lane's share of the sum.
template <int NCA, int STEP = 1>
__device__ __forceinline__ Cx<double> compose(const TermTable& T, uint2 sp, uint64_t s,
                                              int first = 0) {
  double dr = 0.0, di = 0.0;
#pragma unroll 4
  for (uint32_t t = sp.x + first; t < sp.x + sp.y; t += STEP) {
    const ulonglong2 r = __ldg(T.rec + t);
    const uint64_t v = s & r.x;
    const uint64_t flip =
        static_cast<uint64_t>(__popc(static_cast<unsigned>(v) ^ static_cast<unsigned>(v >> 32)))
        << 63;
    dr += __longlong_as_double(static_cast<long long>(r.y ^ flip));
    if constexpr (NCA == 2)
      di += __longlong_as_double(__double_as_longlong(__ldg(T.c + 2 * int64_t(t) + 1)) ^
                                 static_cast<long long>(flip));
  }
  return cx_make<double>(dr, di);
}

// Device view of a ProductPlan.
struct PlanView {
  int64_t nh, nl;
  int d;
  const int64_t *hoff, *loff, *aoff, *boff;   // [nh + 1], [nl + 1], [nh + 1], [nl + 1]
  const uint32_t *key, *part;
  const int32_t* table;
  int64_t nb;
  const uint64_t *xa, *xb, *xm;
  const int32_t* gm;
  int64_t nm;
};
inline PlanView plan_view(const ProductPlan& q) {
  PlanView v{};
  v.nh = q.nh;
  v.nl = q.nl;
  v.d = q.d;
  v.hoff = q.offs.ptr;
  v.loff = v.hoff + q.nh;
  v.aoff = v.loff + q.nl;
  v.boff = v.aoff + q.nh;
  v.key = q.key.ptr;
  v.part = q.part.ptr;
  v.table = q.mtable.ptr;
  v.nb = q.nb;
  v.xa = q.xa.ptr;
  v.xb = q.xb.ptr;
  v.xm = q.xm.ptr;
  v.gm = q.gm.ptr;
  v.nm = q.nm;
  return v;
}

__device__ __forceinline__ int64_t sorted_find(const uint64_t* __restrict__ a, int64_t n,
                                               uint64_t key) {
  int64_t lo = 0, hi = n;
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if (__ldg(a + mid) < key) lo = mid + 1; else hi = mid;
  }
  return (lo < n && __ldg(a + lo) == key) ? lo : -1;
}

// Group of the two-half mask with parts a and b, or -1.
__device__ __forceinline__ int32_t plan_group(const PlanView& c, uint32_t a, uint32_t b) {
  if (c.table) return __ldg(c.table + int64_t(a) * c.nb + b);
  const int64_t i = sorted_find(c.xm, c.nm, __ldg(c.xa + a) | __ldg(c.xb + b));
  return i >= 0 ? __ldg(c.gm + i) : -1;
}

// Lookup of key in the space: index or -1.
__device__ __forceinline__ int64_t hash_lookup(const uint64_t* __restrict__ keys,
                                               const uint32_t* __restrict__ vals, uint64_t mask,
                                               uint64_t key) {
  uint64_t slot = mix64(key) & mask;
  for (uint64_t probe = 0; probe <= mask; ++probe) {
    const uint64_t k = __ldg(keys + slot);
    if (k == key) return static_cast<int64_t>(__ldg(vals + slot));
    if (k == kEmptyKey) return -1;
    slot = (slot + 1) & mask;
  }
  return -1;
}

__device__ __forceinline__ int64_t bsearch_lookup(const uint64_t* __restrict__ states, int64_t n,
                                                  uint64_t key) {
  int64_t lo = 0, hi = n;
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if (__ldg(states + mid) < key) lo = mid + 1; else hi = mid;
  }
  return (lo < n && __ldg(states + lo) == key) ? lo : -1;
}

// Multiplicative hashing of both halves (the 32-bit primes of xxHash, Y. Collet), one mixing
// step, top bits.
__device__ __forceinline__ uint32_t filter_bit(uint64_t key, int log2) {
  uint32_t h = static_cast<uint32_t>(key) * 0x9E3779B1u +
               static_cast<uint32_t>(key >> 32) * 0x85EBCA77u;
  h ^= h >> 15;
  return (h * 0xC2B2AE3Du) >> (32 - log2);
}

// Build helpers implemented in operator.cu and matvec.cu.
void op_build(sqd_op_s* op, cudaStream_t st);
// With op->plan: the matvec that composes its elements reads the lists.
bool op_plan_pays(const sqd_op_s* op);
void op_matvec(sqd_op_s* op, const void* v, void* out, int dtype, cudaStream_t st);
// Hv of two FP64 vectors (nc = 1: real, 2: complex) in one pass over the cached elements; scratch
// of op_pair_scratch() doubles, 0 where two matvecs are the better way.
size_t op_pair_scratch(const sqd_op_s* op, int nc);
void op_matvec_pair(sqd_op_s* op, const void* v0, void* out0, const void* v1, void* out1, int nc,
                    double* scratch, cudaStream_t st);
void op_product_matvec_pair(sqd_op_s* op, const double* v, double* out, double* scratch,
                            cudaStream_t st);
void op_ensure_values32(sqd_op_s* op, cudaStream_t st);
// Product layout (product.cu).
bool op_product_detect(sqd_op_s* op, cudaStream_t st, int64_t* nh, int64_t* nl);
void op_product_build(sqd_op_s* op, int layout, cudaStream_t st);
void op_product_refresh(sqd_op_s* op, cudaStream_t st);
void op_product_values32(sqd_op_s* op, cudaStream_t st);
void op_product_matvec(sqd_op_s* op, const void* v, void* out, int dtype, cudaStream_t st);
// Product subspaces (connect.cu): builds op->plan unless it exists (false when the subspace is
// not such a product, or its lists have more than `most` entries), and the connectivity (row_ptr,
// cols, grps, nnz) from it.
bool op_plan(sqd_op_s* op, cudaStream_t st, int64_t most = INT64_MAX);
bool op_connect_product(sqd_op_s* op, cudaStream_t st);
// Where the elements of the stored pairs go (elements.cu): the pair list (values: NCA doubles per
// pair, or complex128 with out_complex) and, for the H and L pairs of a product subspace, the
// slabs and their FP32 copies (NULL = not wanted).
struct ElementOut {
  double* values;
  int out_complex;
  double *vh, *vl;
  float *vh32, *vl32;
  int wide32;
};
void op_pair_elements(sqd_op_s* op, const ElementOut& out, cudaStream_t st);
// Slabs from the elements in the pair list (op->plan exists).
void op_slab_elements(sqd_op_s* op, const ElementOut& out, cudaStream_t st);
// The slab buffers of op->prod that a refresh has to fill.
void op_product_targets(sqd_op_s* op, ElementOut* out);
// Copies the packed Pauli table from the current coefficients (paulis.cu).
void paulis_pack(sqd_paulis_s* p, cudaStream_t st);

}  // namespace sqd
