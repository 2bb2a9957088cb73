// The (row, X-group) sweep: for every real row s and every group x that can connect, test
// whether s ^ x is in the subspace.  This is get_xsource (sqd.py:485-548) for all groups at
// once, restricted to the pairs whose source can exist:
//   1. sector filter: a state of the subspace has popcount(s & m_l) == w_l in every conserved
//      sector l, so s ^ x can only be a state if 2 * popcount(s & x & m_l) == popcount(x & m_l);
//   2. the subspace's state filter (one hashed bit per state, eight or more bits of table per
//      state, so at most one absent key in eight passes), in shared memory up to kFilterShared
//      bits and read through L1/L2 above;
//   3. exact lookup (hash table or binary search) of s ^ x.
// Candidates surviving 1-2 are pushed into a per-warp FIFO in shared memory and looked up 32 at
// a time, so the expensive step runs on full warps.  Candidates of one row enter the FIFO in
// the order of the group list, so every row's pairs follow that order (the high-sector-only
// groups first, see k_gpre_flags).
//
// Modes: COUNT (pairs per row and group chunk, and each pair with its rank in its (row, chunk)
// into a buffer while it has room), FILL (write (col, group) at the row's CSR slots; only when
// the buffer overflowed), APPLY (accumulate diag_j(s) * v[src] per row: the uncached matvec,
// cache_strategy (0, *)).
//
// COUNT and FILL split the groups into chunks, a block per (row tile, chunk), so that a few
// hundred thousand rows fill the chip.  131,072 random states of 40 qubits against 20,000 groups:
// 0.74 ms, bound by issue (popcounts and hashing); two sweeps of one block per 1,024 rows that
// looked up every weight-conserving candidate took 17.1 ms.
#pragma once
#include "internal.cuh"

namespace sqd {

constexpr int SW_CHUNK = 256;     // groups staged in shared memory at a time
constexpr int SW_QCAP = 64;
constexpr int kSweepMaxChunks = 128;

enum SweepMode { SWEEP_COUNT = 0, SWEEP_FILL = 1, SWEEP_APPLY = 2 };

// A pair found by COUNT: rank among its row's pairs of its chunk, in group order.
struct alignas(16) SweepHit {
  uint32_t row, col, group;
  uint32_t chunk_rank;      // chunk in the top 7 bits
};

struct SweepParams {
  const uint64_t* states;
  int64_t n_unique;
  const GroupPre* gpre;
  int64_t n_gpre;
  int chunks;               // COUNT, FILL: group chunks of chunk_groups groups
  int64_t chunk_groups;
  const uint64_t* hkeys;
  const uint32_t* hvals;
  uint64_t hmask;
  int lookup;
  int nsec;
  uint64_t m0, m1;
  const uint32_t* filter;
  int filter_log2;
  // COUNT
  int64_t* counts;          // [row * chunks + chunk]
  SweepHit* hits;
  unsigned long long* n_hits;
  unsigned long long max_hits;
  // FILL
  const int64_t* place;     // [row * chunks + chunk] first slot
  uint32_t* cols;
  uint32_t* grps;
  int diag_first;
  // APPLY
  TermTable terms;
  const void* vin;
  void* vout;
  int has_diag;
};

// The parts that every mode needs.
inline SweepParams sweep_params(const sqd_op_s* op) {
  const sqd_space_s* sp = op->s;
  SweepParams P{};
  P.states = sp->states.ptr;
  P.n_unique = sp->n_unique;
  P.gpre = op->gpre.ptr;
  P.n_gpre = op->n_gpre;
  P.chunks = 1;
  P.chunk_groups = op->n_gpre;
  P.hkeys = sp->hkeys.ptr;
  P.hvals = sp->hvals.ptr;
  P.hmask = sp->hmask;
  P.lookup = op->lookup == SQD_LOOKUP_BSEARCH ? SQD_LOOKUP_BSEARCH : SQD_LOOKUP_HASH;
  P.nsec = sp->num_sectors;
  P.m0 = sp->sector_mask[0];
  P.m1 = sp->sector_mask[1];
  P.filter = sp->filter.ptr;
  P.filter_log2 = sp->filter_log2;
  P.terms = term_table(op->p);
  return P;
}
inline size_t sweep_shared(const SweepParams& P) {
  return P.filter_log2 <= kFilterShared ? (size_t(1) << P.filter_log2) / 8 : 0;
}

struct QEntry {
  uint64_t key;
  uint32_t group;
  uint32_t lrow;
};

template <typename R, int NCA>
__device__ __forceinline__ Cx<R> group_diag(const SweepParams& P, int64_t j, uint64_t s) {
  const Cx<double> d = compose<NCA>(P.terms, __ldg(P.terms.span + j), s);
  return cx_make<R>(R(d.re), R(d.im));
}

// THREADS threads with RPT rows each.
template <int MODE, typename R, int NCV, int NCA, int THREADS, int RPT>
__global__ void __launch_bounds__(THREADS)
k_sweep(SweepParams P) {
  constexpr int TILE = THREADS * RPT;
  extern __shared__ uint32_t sm_filter[];
  __shared__ GroupPre sm_groups[SW_CHUNK];
  __shared__ QEntry sm_queue[THREADS / 32][SW_QCAP];
  __shared__ int32_t sm_cnt[MODE == SWEEP_APPLY ? 1 : TILE];
  __shared__ Cx<R> sm_acc[MODE == SWEEP_APPLY ? TILE : 1];

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned lt_mask = (1u << lane) - 1u;
  const int64_t tile_base = static_cast<int64_t>(blockIdx.x / P.chunks) * TILE;
  const int chunk = static_cast<int>(blockIdx.x % P.chunks);
  const int64_t g_first = chunk * P.chunk_groups;
  const int64_t g_last = min(P.n_gpre, g_first + P.chunk_groups);
  const bool shared_filter = P.filter_log2 <= kFilterShared;

  if (shared_filter) {
    const int words = 1 << (P.filter_log2 - 5);
    for (int w = tid; w < words; w += THREADS) sm_filter[w] = __ldg(P.filter + w);
  }

  uint64_t srow[RPT];
  bool valid[RPT];
#pragma unroll
  for (int k = 0; k < RPT; ++k) {
    const int lr = k * THREADS + tid;
    const int64_t r = tile_base + lr;
    valid[k] = r < P.n_unique;
    srow[k] = valid[k] ? __ldg(P.states + r) : 0ull;
    if constexpr (MODE == SWEEP_APPLY) {
      Cx<R> a = cx_make<R>(0, 0);
      if (valid[k] && P.has_diag) {
        const Cx<R> d = group_diag<R, NCA>(P, 0, srow[k]);
        const Cx<R> x = ld_elem<R, NCV>(static_cast<const R*>(P.vin), r);
        a.re = d.re * x.re - d.im * x.im;
        a.im = d.re * x.im + d.im * x.re;
      }
      sm_acc[lr] = a;
    } else {
      sm_cnt[lr] = 0;
    }
  }

  int head = 0, tail = 0;  // warp-uniform FIFO cursors

  auto process = [&](int count) {
    QEntry e;
    int64_t found = -1;
    if (lane < count) {
      e = sm_queue[warp][(head + lane) & (SW_QCAP - 1)];
      found = (P.lookup == SQD_LOOKUP_BSEARCH) ? bsearch_lookup(P.states, P.n_unique, e.key)
                                               : hash_lookup(P.hkeys, P.hvals, P.hmask, e.key);
    }
    const bool hit = found >= 0;
    const unsigned all = __ballot_sync(kFullMask, hit);
    if (!all) return;
    if constexpr (MODE != SWEEP_APPLY) {
      const unsigned key = hit ? e.lrow : (0x10000u + lane);
      const unsigned peers = __match_any_sync(kFullMask, key);
      int rank = 0;
      if (hit) rank = sm_cnt[e.lrow] + __popc(peers & lt_mask);
      __syncwarp();
      if (hit && (peers >> lane) == 1u) sm_cnt[e.lrow] = rank + 1;   // the row's last hit
      __syncwarp();
      if constexpr (MODE == SWEEP_COUNT) {
        unsigned long long at = 0;
        if (lane == 0) at = atomicAdd(P.n_hits, static_cast<unsigned long long>(__popc(all)));
        at = __shfl_sync(kFullMask, at, 0) + __popc(all & lt_mask);
        if (hit && at < P.max_hits) {
          SweepHit h;
          h.row = static_cast<uint32_t>(tile_base + e.lrow);
          h.col = static_cast<uint32_t>(found);
          h.group = e.group;
          h.chunk_rank = (static_cast<uint32_t>(chunk) << 25) | static_cast<uint32_t>(rank);
          P.hits[at] = h;
        }
      } else if (hit) {
        const int64_t row = tile_base + e.lrow;
        const int64_t slot = P.place[row * P.chunks + chunk] + (chunk == 0 ? P.diag_first : 0) +
                             rank;
        P.cols[slot] = static_cast<uint32_t>(found);
        P.grps[slot] = e.group;
      }
    } else {
      // APPLY: contributions added to the row accumulator in FIFO (= group) order.
      Cx<R> c = cx_make<R>(0, 0);
      if (hit) {
        const int64_t row = tile_base + e.lrow;
        const uint64_t srow_state = __ldg(P.states + row);
        const Cx<R> d = group_diag<R, NCA>(P, e.group, srow_state);
        const Cx<R> x = ld_elem<R, NCV>(static_cast<const R*>(P.vin), found);
        c.re = d.re * x.re - d.im * x.im;
        c.im = d.re * x.im + d.im * x.re;
      }
      unsigned hits = all;
      while (hits) {
        const int src = __ffs(hits) - 1;
        hits &= hits - 1;
        const unsigned lr = __shfl_sync(kFullMask, e.lrow, src);
        const R cr = __shfl_sync(kFullMask, c.re, src);
        const R ci = __shfl_sync(kFullMask, c.im, src);
        if (lane == 0) {
          sm_acc[lr].re += cr;
          sm_acc[lr].im += ci;
        }
        __syncwarp();
      }
    }
  };

  for (int64_t c0 = g_first; c0 < g_last; c0 += SW_CHUNK) {
    const int64_t left = g_last - c0;
    const int clen = left < SW_CHUNK ? static_cast<int>(left) : SW_CHUNK;
    __syncthreads();
    for (int g = tid; g < clen; g += THREADS) sm_groups[g] = P.gpre[c0 + g];
    __syncthreads();
    for (int g = 0; g < clen; ++g) {
      const GroupPre gp = sm_groups[g];
      const int cx0 = gp.cx & 0xff, cx1 = (gp.cx >> 8) & 0xff;
#pragma unroll
      for (int k = 0; k < RPT; ++k) {
        const uint64_t cand = srow[k] ^ gp.x;
        bool pass = valid[k];
        if (P.nsec > 0) {
          pass = pass && (2 * __popcll(srow[k] & gp.x & P.m0) == cx0);
          if (P.nsec > 1) pass = pass && (2 * __popcll(srow[k] & gp.x & P.m1) == cx1);
        }
        if (pass) {
          const uint32_t b = filter_bit(cand, P.filter_log2);
          const uint32_t w = shared_filter ? sm_filter[b >> 5] : __ldg(P.filter + (b >> 5));
          pass = (w >> (b & 31)) & 1u;
        }
        const unsigned ballot = __ballot_sync(kFullMask, pass);
        if (ballot) {
          if (pass) {
            QEntry q;
            q.key = cand;
            q.group = static_cast<uint32_t>(gp.group);
            q.lrow = static_cast<uint32_t>(k * THREADS + tid);
            sm_queue[warp][(tail + __popc(ballot & lt_mask)) & (SW_QCAP - 1)] = q;
          }
          tail += __popc(ballot);
          __syncwarp();
          if (tail - head >= 32) {
            process(32);
            head += 32;
          }
        }
      }
    }
  }
  while (tail - head > 0) {
    const int cnt = min(32, tail - head);
    __syncwarp();
    process(cnt);
    head += cnt;
  }
  __syncwarp();
  __syncthreads();
  if constexpr (MODE != SWEEP_FILL) {
#pragma unroll
    for (int k = 0; k < RPT; ++k) {
      const int lr = k * THREADS + tid;
      const int64_t r = tile_base + lr;
      if (!valid[k]) continue;
      if constexpr (MODE == SWEEP_COUNT) {
        P.counts[r * P.chunks + chunk] = sm_cnt[lr] + (chunk == 0 ? P.diag_first : 0);
      } else {
        st_elem<R, NCV>(static_cast<R*>(P.vout), r, sm_acc[lr]);
      }
    }
  }
}

}  // namespace sqd
