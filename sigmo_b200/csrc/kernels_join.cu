// Join kernels (isomorphism::join::joinCandidates, isomorphism.hpp:270-381).
//
// k_join_literal restates the reference's DFS step by step: one block per
// data graph, thread lid takes GMCR slots lid, lid+wg, ...; each pair runs the
// explicit-stack DFS in identity query order with the range-masked candidate
// count / k-th candidate (candidates.hpp:86-162), the uint8-indexed `visited`
// bitset (utils.hpp:64-96) and the induced adjacency check
// (isomorphism.hpp:150-168).  mapping[] starts zeroed per thread and is
// carried across the pairs the thread handles, as in the reference.  Under
// REF_PTX the visited bitset is inert for any data graph whose first vertex is
// >= 256; the literal search therefore runs only for the few graphs below that
// (k_join_literal_sets), for REF_X86, and for graphs over 256 vertices.
//
// The other kernels count the same matches with graph-local bit sets.  For the
// pairs they handle, the reference's count is order independent:
//   REF_PTX (visited inert): #{(d_0..d_{n-1}) in prod C_i : for all i<j,
//       adjQ(i,j) == adjD(d_i,d_j)}  (non-adjacent query vertices may share a
//       data vertex);
//   EXACT: the same with d injective.
// so each level's candidates are one AND over the earlier levels' adjacency
// rows, the last level is a popcount, and query vertices are placed in a
// connectivity order.  Find-first stops at the first match.
#include <cuda_runtime.h>

#include <algorithm>

#include "internal.hpp"

namespace sigmo_b200 {
namespace {

// Step budget (JoinLimit): a lane counts the DFS levels it leaves; past the
// budget it raises the status word and stops.  Lanes check the word before
// taking more work, so a spent budget ends the launch soon after.
__device__ __forceinline__ bool budget_spent(const JoinLimit& lim, uint64_t& steps) {
  if (lim.budget && ++steps > lim.budget) {
    atomicOr(lim.status, kJoinStatusBudget);
    return true;
  }
  return false;
}
__device__ __forceinline__ bool join_stopped(const JoinLimit& lim) {
  return lim.budget && *reinterpret_cast<volatile const unsigned int*>(lim.status) != 0u;
}

// getCandidatesCount(src, s, e) on one bitset row.
__device__ __forceinline__ uint32_t cand_count(const uint32_t* __restrict__ row, uint32_t s, uint32_t e, int prof) {
  const uint32_t i0 = s >> 5, i1 = (e + 31u) >> 5;
  uint32_t c = 0;
  for (uint32_t i = i0; i < i1; ++i) c += __popc(row[i] & range_mask(i, s, e, prof));
  return c;
}

// getCandidateAt(src, idx, s, e): global id of the idx-th masked candidate.
__device__ __forceinline__ uint32_t cand_at(const uint32_t* __restrict__ row, uint32_t idx, uint32_t s, uint32_t e, int prof) {
  const uint32_t i0 = s >> 5, i1 = (e + 31u) >> 5;
  uint32_t c = 0;
  for (uint32_t i = i0; i < i1; ++i) {
    uint32_t blk = row[i] & range_mask(i, s, e, prof);
    const uint32_t bc = __popc(blk);
    if (c + bc > idx) {
      while (blk) {
        const uint32_t t = __ffs(blk) - 1;
        if (c == idx) return (i << 5) + t;
        blk &= blk - 1;
        ++c;
      }
    } else {
      c += bc;
    }
  }
  return 0xFFFFFFFFu;
}

// DeviceBatchedCSRGraph::isNeighbor (graph.hpp:72-77) for two vertices of
// data graph [s, e): via the local adjacency rows when the graph fits them.
__device__ __forceinline__ bool data_neighbor(uint32_t a, uint32_t b, uint32_t s, uint32_t ng, const uint64_t* __restrict__ adj,
                                              uint32_t AW, const uint32_t* __restrict__ roff, const uint32_t* __restrict__ col) {
  if (ng <= 64u * AW) {
    const uint32_t t = b - s;
    return (adj[static_cast<uint64_t>(a) * AW + (t >> 6)] >> (t & 63u)) & 1ull;
  }
  for (uint32_t i = roff[a]; i < roff[a + 1]; ++i)
    if (col[i] == b) return true;
  return false;
}

// Graph-local candidate set of one bitset row for data graph [s, e): bit t =
// global candidate s + t, after the profile's range masks.
template <int AW>
__device__ __forceinline__ void extract_local(const uint32_t* __restrict__ row, uint32_t s, uint32_t e, int prof, uint64_t* out) {
#pragma unroll
  for (int k = 0; k < AW; ++k) out[k] = 0;
  const uint32_t i0 = s >> 5, i1 = (e + 31u) >> 5;
  for (uint32_t i = i0; i < i1; ++i) {
    uint32_t wv = row[i] & range_mask(i, s, e, prof);
    if (!wv) continue;
    int32_t off = static_cast<int32_t>(i << 5) - static_cast<int32_t>(s);
    if (off < 0) {
      wv >>= static_cast<uint32_t>(-off);
      off = 0;
    }
    const uint32_t k = static_cast<uint32_t>(off) >> 6, sh = static_cast<uint32_t>(off) & 63u;
#pragma unroll
    for (int kk = 0; kk < AW; ++kk) {
      if (static_cast<uint32_t>(kk) == k) out[kk] |= static_cast<uint64_t>(wv) << sh;
      if (sh > 32u && static_cast<uint32_t>(kk) == k + 1) out[kk] |= static_cast<uint64_t>(wv) >> (64u - sh);
    }
  }
}

// Candidate set of query vertex v (global id) in data graph g = [s, e) from
// either source.  AW words are written; dAW is the planes' words per set.
template <int AW>
__device__ __forceinline__ void source_mask(const MaskSource& src, uint32_t dAW, uint32_t v, uint32_t g, uint32_t s, uint32_t e,
                                            uint64_t* out) {
  if (!src.planes) {
    extract_local<AW>(src.bits + static_cast<uint64_t>(v) * src.Wp, s, e, src.prof, out);
    return;
  }
  const uint64_t* base = src.planes + (src.tiled ? static_cast<uint64_t>(g >> 5) * src.K * dAW * 32 + (g & 31u)
                                                 : static_cast<uint64_t>(g) * src.K * dAW);
  const uint32_t step = src.tiled ? 32u : 1u;
#pragma unroll
  for (int w = 0; w < AW; ++w) out[w] = ~0ull;
  const uint32_t c = src.cls[v], e1 = src.prog_off[c + 1];
  for (uint32_t i = src.prog_off[c]; i < e1; ++i) {
    const uint64_t ids = src.prog[i];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint64_t* row = base + static_cast<uint32_t>((ids >> (16 * j)) & 0xFFFFu) * (dAW * step);
#pragma unroll
      for (int w = 0; w < AW; ++w) out[w] &= row[step * w];
    }
  }
}

struct Frame {
  uint32_t depth;
  uint32_t idx;
};

// Per-pair cache of the range-masked candidate words of every query vertex
// (a data graph of <= 64 vertices spans at most 3 bitset words), so the DFS's
// repeated getCandidatesCount / getCandidateAt read registers/L1 instead of
// the bitset.  Values are exactly those of candidates.hpp:86-162.
struct PairCands {
  uint32_t w[kMaxQueryNodes][3];
  uint32_t cnt[kMaxQueryNodes];
  uint32_t i0, nw;
  __device__ __forceinline__ void load(const uint32_t* __restrict__ bits, uint64_t Wp, uint32_t qoff, uint32_t n, uint32_t s,
                                       uint32_t e, int prof) {
    i0 = s >> 5;
    nw = ((e + 31u) >> 5) - i0;
    for (uint32_t j = 0; j < n; ++j) {
      const uint32_t* row = bits + static_cast<uint64_t>(qoff + j) * Wp;
      uint32_t c = 0;
      for (uint32_t k = 0; k < 3; ++k) {
        const uint32_t v = k < nw ? (row[i0 + k] & range_mask(i0 + k, s, e, prof)) : 0u;
        w[j][k] = v;
        c += __popc(v);
      }
      cnt[j] = c;
    }
  }
  __device__ __forceinline__ uint32_t at(uint32_t j, uint32_t idx) const {
    uint32_t c = 0;
    for (uint32_t k = 0; k < nw; ++k) {
      uint32_t blk = w[j][k];
      const uint32_t bc = __popc(blk);
      if (c + bc > idx) {
        while (blk) {
          const uint32_t t = __ffs(blk) - 1;
          if (c == idx) return ((i0 + k) << 5) + t;
          blk &= blk - 1;
          ++c;
        }
      } else {
        c += bc;
      }
    }
    return 0xFFFFFFFFu;
  }
};

__global__ void k_join_literal(const uint32_t* __restrict__ bits, uint64_t Wp, int prof,
                               const uint32_t* __restrict__ qgoff, const uint64_t* __restrict__ qadj,
                               const uint32_t* __restrict__ dgoff, const uint64_t* __restrict__ dadj, uint32_t dAW,
                               const uint32_t* __restrict__ droff, const uint32_t* __restrict__ dcol,
                               const uint32_t* __restrict__ offsets, const uint32_t* __restrict__ indices, uint32_t g0,
                               uint32_t g1, uint32_t q_begin, uint32_t q_end, int find_first, uint64_t* __restrict__ counts,
                               unsigned long long* __restrict__ d_total, JoinLimit lim) {
  const uint32_t wg = blockDim.x, lid = threadIdx.x;
  uint64_t my_total = 0;
  uint64_t steps = 0;
  bool stop = false;
  PairCands pc;
  uint64_t rowc[kMaxQueryNodes];   // adjacency row of mapping[i] (graphs <= 64 vertices)
  uint64_t vmask[kMaxQueryNodes];  // candidates passing isValidMapping at depth d (graphs <= 64 vertices)
  for (uint32_t g = g0 + blockIdx.x; g < g1; g += gridDim.x) {
    const uint32_t s = dgoff[g], e = dgoff[g + 1], ng = e - s;
    const bool small = ng <= 64u;
    // the segment's slots whose query graph is in [q_begin, q_end) (segments
    // are sorted by query graph, so they are contiguous)
    uint32_t seg0 = offsets[g], seg1 = offsets[g + 1];
    if (q_begin != 0 || q_end != 0xFFFFFFFFu) {
      uint32_t lo = seg0, hi = seg1;
      while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (indices[mid] < q_begin) lo = mid + 1;
        else hi = mid;
      }
      uint32_t lo2 = lo, hi2 = seg1;
      while (lo2 < hi2) {
        const uint32_t mid = (lo2 + hi2) >> 1;
        if (indices[mid] < q_end) lo2 = mid + 1;
        else hi2 = mid;
      }
      seg0 = lo;
      seg1 = lo2;
    }
    const uint32_t seglen = seg1 - seg0;
    uint32_t mapping[kMaxQueryNodes + 1];
#pragma unroll 1
    for (uint32_t k = 0; k <= kMaxQueryNodes; ++k) mapping[k] = 0;
    for (uint32_t it = lid; it < seglen; it += wg) {
      if (join_stopped(lim)) {
        stop = true;
        break;
      }
      const uint32_t qg = indices[seg0 + it];
      const uint32_t qoff = qgoff[qg], n = qgoff[qg + 1] - qoff;
      if (small) pc.load(bits, Wp, qoff, n, s, e, prof);
      auto count_of = [&](uint32_t qn) -> uint32_t {
        return small ? pc.cnt[qn] : cand_count(bits + static_cast<uint64_t>(qoff + qn) * Wp, s, e, prof);
      };
      auto cand_of = [&](uint32_t qn, uint32_t idx) -> uint32_t {
        return small ? pc.at(qn, idx) : cand_at(bits + static_cast<uint64_t>(qoff + qn) * Wp, idx, s, e, prof);
      };
      // isValidMapping (isomorphism.hpp:150-168).  Its result depends only on
      // mapping[0..qn-1], which stay fixed while the frame at depth qn runs, so
      // for graphs of <= 64 vertices it is evaluated once per push as the bit
      // set vmask[qn] and each candidate is then one bit test.
      auto valid = [&](uint32_t qn, uint32_t cand) -> bool {
        if (small) return (vmask[qn] >> (cand - s)) & 1ull;
        const uint64_t qrow_bit = 1ull << qn;
        for (uint32_t i = 0; i < qn; ++i) {
          const bool qa = (qadj[qoff + i] & qrow_bit) != 0;
          if (qa != data_neighbor(mapping[i], cand, s, ng, dadj, dAW, droff, dcol)) return false;
        }
        return true;
      };
      // vmask[d] from rowc[0..d-1]: local t is valid iff for every i < d,
      // (d in query row i) == (t in data row of mapping[i]).
      auto push_mask = [&](uint32_t d) {
        if (!small || d >= n) return;
        uint64_t vm = ~0ull;
        const uint64_t qbit = 1ull << d;
        for (uint32_t i = 0; i < d; ++i) vm &= ((qadj[qoff + i] & qbit) ? rowc[i] : ~rowc[i]);
        vmask[d] = vm;
      };
      if (small) vmask[0] = ~0ull;
      uint64_t found = 0;
      Frame stack[kMaxQueryNodes + 2];
      uint32_t top = 0;
      stack[top++] = {0u, 0u};
      {
        uint64_t visited = 0;  // Bitset<uint64_t>{offset = s}
        while (top > 0) {
          const Frame fr = stack[top - 1];
          const uint32_t qn = fr.depth;
          if (qn == n) {
            ++found;
            --top;
            if (find_first) break;
            continue;
          }
          if (small && qn + 1 == n && fr.idx == 0) {
            // The last level in one step (graphs of <= 64 vertices).  Its
            // candidates are distinct local bits, so placing one never hides a
            // later one, and valid() does not read `visited`: the frame finds
            // popc(candidates & valid & ~visited), sets the bits of those below
            // vertex 256 (refbit gives none above), leaves mapping[n - 1] at the
            // last one placed (the first under find-first, which stops there),
            // then is used up -- what the candidate-by-candidate loop does.
            const uint32_t sh = s & 31u;
            const uint64_t lo = static_cast<uint64_t>(pc.w[qn][0]) | (static_cast<uint64_t>(pc.w[qn][1]) << 32);
            const uint64_t cm = (lo >> sh) | (sh ? (static_cast<uint64_t>(pc.w[qn][2]) << (64u - sh)) : 0ull);
            // REF_X86: every local bit is live (a <= 64-vertex graph's set is exact)
            const uint64_t low = prof == kProfileX86 ? ~0ull
                                 : (s >= 256u ? 0ull : (256u - s >= 64u ? ~0ull : ((1ull << (256u - s)) - 1ull)));
            uint64_t place = cm & vmask[qn] & ~visited;
            if (place) {
              if (find_first) place &= 0ull - place;
              found += __popcll(place);
              visited |= place & low;
              mapping[qn] = s + 63u - static_cast<uint32_t>(__clzll(static_cast<long long>(place)));
              if (find_first) break;
            }
            --top;
            visited &= ~refbit_prof(mapping[qn], s, prof);
            if (top == 1) visited = 0;
            if (budget_spent(lim, steps)) {
              stop = true;
              break;
            }
            continue;
          }
          if (fr.idx >= count_of(qn)) {
            --top;
            visited &= ~refbit_prof(mapping[qn], s, prof);
            if (top == 1) visited = 0;
            if (budget_spent(lim, steps)) {
              stop = true;
              break;
            }
            continue;
          }
          const uint32_t cand = cand_of(qn, fr.idx);
          stack[top - 1].idx++;
          if (visited & refbit_prof(cand, s, prof)) continue;
          if (valid(qn, cand)) {
            mapping[qn] = cand;
            if (small) rowc[qn] = dadj[static_cast<uint64_t>(cand) * dAW];
            visited |= refbit_prof(cand, s, prof);
            stack[top++] = {qn + 1, 0u};
            push_mask(qn + 1);
          }
        }
      }
      if (stop) break;
      counts[seg0 + it] = found;
      my_total += found;
    }
    if (stop) break;
  }
  // block reduction, one atomic per block
  for (int o = 16; o; o >>= 1) my_total += __shfl_xor_sync(0xFFFFFFFFu, my_total, o);
  __shared__ uint64_t part[32];
  if ((lid & 31u) == 0) part[lid >> 5] = my_total;
  __syncthreads();
  if (lid < 32) {
    uint64_t v = lid < ((wg + 31u) >> 5) ? part[lid] : 0ull;
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    if (lid == 0 && v) atomicAdd(d_total, static_cast<unsigned long long>(v));
  }
}

// k_join_literal for graphs of at most 64 * AW vertices (and, under REF_X86, of
// at most 64).  The same DFS, step for step, on graph-local sets, with the
// per-level state of each thread in shared memory ([level][thread]) for AW = 1
// and queries of at most kLitLevels vertices (SMEM), else in local memory:
//   cm[j]   the pair's range-masked candidates of query vertex j as graph-local
//           bits (candidates.hpp:86-162), from the candidate bitset or from the
//           batched form's planes (the same sets);
//   rem[j]  the candidates the frame at depth j has still to try, taken in
//           ascending order like getCandidateAt(idx) for idx = 0, 1, ...
//           Only those passing isValidMapping are kept (its result depends on
//           mapping[0..j-1], fixed while the frame runs, so it is one AND
//           when the frame is pushed); the others are skipped by the
//           reference with no effect, so the placements are the same;
//           As in k_join_dfs, the test is the rows of the earlier neighbours
//           and a count: p0[j], p1[j] are the bit planes (to 3) of the number
//           of rows of mapping[0..j-1] that hold a vertex;
//   map[j]  mapping[j] as a local id, carried across the thread's pairs of a
//           data graph like the reference's private array (isomorphism.hpp:309);
//           a fresh work-item's mapping[] holds global vertex 0, which is
//           local 0 of a graph starting at vertex 0 and kLitOutside (a local
//           id that never has a bit in the visited set) otherwise.
// The reference's `visited` bookkeeping (utils.hpp:64-96,
// isomorphism.hpp:346-369) is kept: a frame that runs out unsets only
// mapping[depth] (perhaps stale), and the set is cleared when the DFS is back
// at depth 0.  Its 64 bits hold local ids below 64 (REF_PTX: whose global id is
// below 256).  The last query vertex is placed in one step, as in
// k_join_literal.
//
// A serial chain per pair (and per work-item), and few of them: bound by the
// latency of a step.  So the sets are taken from the planes where the caller
// has them (writing them as bitset words first took seven more launches, 130 us
// before the join of a batch of any size), the graph's rows are staged in
// shared memory, a round's masks are built by the whole block, and the
// work-items of a graph are spread over blocks of kLitItems: a warp steps through
// its lanes' different moves in turn, so four lanes take less time than 32, and
// blocks of up to 4 KB fit beside the persistent join's.  (One block of 128
// work-items per graph, walking the earlier rows at each step: 1.02 ms for the
// first ten molecules of 100,000 x 600 pairs, 112 us of 1,000 x 20; this form
// 190 and 74 us.)  Launches over many graphs (REF_X86) take kLitItemsMany
// work-items per block, whose state (33 bytes per work-item and level of the
// batch's longest query) leaves room for many blocks: 1,000 x 20 and 5,000 x 100
// pairs take 420 / 1,467 us with 4, 263 / 758 with 16, 279 / 778 with 32 and 263 /
// 2,571 with the 128 of one block per graph.  Molecules over 64 atoms and queries
// over 32 vertices used to take k_join_literal's candidate-by-candidate form: 3.7
// ms for the first ten molecules of 60,000 x 500 uneven pairs.
constexpr uint32_t kLitLevels = 32;
constexpr uint8_t kLitOutside = 0xFFu;
constexpr uint32_t kLitItems = 4, kLitItemsMany = 16;
constexpr size_t kLitBytesPerLevel = 4 * sizeof(uint64_t) + 1;  // of a thread

// wg: work-items of a graph (the reference's work-group size); bt of them per
// block, one thread each.  With SMEM the block may have more threads, which only
// help to build the level masks.
template <int AW, bool SMEM>
__global__ void k_join_literal_sets(MaskSource src, int prof, const uint32_t* __restrict__ qgoff, const uint64_t* __restrict__ qsel_id,
                                    const uint32_t* __restrict__ dgoff, const uint64_t* __restrict__ dadj, uint32_t dAW,
                                    const uint32_t* __restrict__ offsets, const uint32_t* __restrict__ indices, uint32_t g0,
                                    uint32_t g1, uint32_t wg, uint32_t bt, uint32_t levels, uint32_t q_begin, uint32_t q_end,
                                    int find_first, uint64_t* __restrict__ counts,
                                    unsigned long long* __restrict__ d_total, JoinLimit lim) {
  extern __shared__ uint64_t lit_sm[];
  __shared__ uint64_t s_row[SMEM ? 64 : 1];  // the graph's adjacency rows (word 0)
  const uint32_t tid = threadIdx.x;
  uint64_t* cm_s = lit_sm + tid;  // the threads past bt - 1 do not search
  uint64_t* rem_s = lit_sm + levels * bt + tid;
  uint64_t* p0_s = lit_sm + 2 * levels * bt + tid;
  uint64_t* p1_s = lit_sm + 3 * levels * bt + tid;
  uint8_t* map_s = reinterpret_cast<uint8_t*>(lit_sm + 4 * levels * bt) + tid;
  constexpr uint32_t kLocal = SMEM ? 1 : kMaxQueryNodes;
  uint64_t cm_l[kLocal * AW], rem_l[kLocal * AW], p0_l[kLocal * AW], p1_l[kLocal * AW];
  uint8_t map_l[kLocal];
#define CM(j, w) (SMEM ? cm_s[(j) * bt] : cm_l[(j) * AW + (w)])
#define REM(j, w) (SMEM ? rem_s[(j) * bt] : rem_l[(j) * AW + (w)])
#define P0(j, w) (SMEM ? p0_s[(j) * bt] : p0_l[(j) * AW + (w)])
#define P1(j, w) (SMEM ? p1_s[(j) * bt] : p1_l[(j) * AW + (w)])
#define MAP(j) (SMEM ? map_s[(j) * bt] : map_l[(j)])
  const uint32_t parts = (wg + bt - 1u) / bt;  // blocks per graph
  const uint64_t blocks = static_cast<uint64_t>(g1 - g0) * parts;
  uint64_t my_total = 0, steps = 0;
  bool stop = false;
#pragma unroll
  for (int w = 0; w < AW; ++w)
    if (tid < bt) P0(0, w) = P1(0, w) = 0;
  for (uint64_t blk = blockIdx.x; blk < blocks; blk += gridDim.x) {
    const uint32_t g = g0 + static_cast<uint32_t>(blk / parts), lid = static_cast<uint32_t>(blk % parts) * bt + tid;
    const uint32_t s = dgoff[g], e = dgoff[g + 1];
    if (SMEM) {
      __syncthreads();  // the previous graph's rows are no longer read
      for (uint32_t i = tid; i < e - s; i += blockDim.x) s_row[i] = dadj[static_cast<uint64_t>(s + i) * dAW];
      __syncthreads();
    }
    const bool searches = tid < bt && lid < wg;
    auto row_of = [&](uint32_t t, int w) -> uint64_t { return SMEM ? s_row[t] : dadj[static_cast<uint64_t>(s + t) * dAW + w]; };
    uint32_t seg0 = offsets[g], seg1 = offsets[g + 1];
    if (q_begin != 0 || q_end != 0xFFFFFFFFu) {  // the segment's slots with query graph in [q_begin, q_end)
      uint32_t lo = seg0, hi = seg1;
      while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (indices[mid] < q_begin) lo = mid + 1;
        else hi = mid;
      }
      uint32_t lo2 = lo, hi2 = seg1;
      while (lo2 < hi2) {
        const uint32_t mid = (lo2 + hi2) >> 1;
        if (indices[mid] < q_end) lo2 = mid + 1;
        else hi2 = mid;
      }
      seg0 = lo;
      seg1 = lo2;
    }
    const uint8_t map0 = s == 0 ? 0 : kLitOutside;
#pragma unroll 1
    for (uint32_t k = 0; searches && k < levels; ++k) MAP(k) = map0;  // mapping[] of a fresh work-item
    // graph-local bits the reference's uint8-indexed visited set can hold:
    // under REF_PTX those whose global id is below 256; under REF_X86 all
    // (the count modulo 64 is the local id).  A fresh work-item's mapping[]
    // (global vertex 0) names under REF_X86 the bit (0 - s) mod 64.
    const uint64_t low = prof == kProfileX86 ? ~0ull
                         : (s >= 256u ? 0ull : (256u - s >= 64u ? ~0ull : ((1ull << (256u - s)) - 1ull)));
    const uint64_t outside_bit = prof == kProfileX86 ? (1ull << ((0u - s) & 63u)) : 0ull;
    const uint32_t lid0 = lid - tid;  // the block's first work-item
    for (uint32_t it = lid; lid0 < wg && it - tid < seg1 - seg0; it += wg) {
      if (SMEM) {  // the masks of the round's pairs, (work-item, level) per thread
        __syncthreads();  // the round before is done
        for (uint32_t x = tid; x < bt * levels; x += blockDim.x) {
          const uint32_t i = x % bt, j = x / bt, slot = it - tid + i;
          if (lid0 + i >= wg || slot >= seg1 - seg0) continue;
          const uint32_t q0 = qgoff[indices[seg0 + slot]];
          if (q0 + j < qgoff[indices[seg0 + slot] + 1]) source_mask<AW>(src, dAW, q0 + j, g, s, e, lit_sm + j * bt + i);
        }
        __syncthreads();
      }
      if (stop || !searches || it >= seg1 - seg0) continue;
      if (join_stopped(lim)) {
        stop = true;
        continue;
      }
      const uint32_t qg = indices[seg0 + it];
      const uint32_t qoff = qgoff[qg], n = qgoff[qg + 1] - qoff;
      for (uint32_t j = 0; !SMEM && j < n; ++j) {
        uint64_t m[AW];
        source_mask<AW>(src, dAW, qoff + j, g, s, e, m);
#pragma unroll
        for (int w = 0; w < AW; ++w) CM(j, w) = m[w];
      }
      uint64_t found = 0, visited = 0;
      uint32_t top = 1;  // frames at depths 0 .. top-1
#pragma unroll
      for (int w = 0; w < AW; ++w) REM(0, w) = CM(0, w);
      while (top > 0) {
        const uint32_t qn = top - 1;
        if (qn + 1 == n) {
          // the last query vertex in one step: the frame was just pushed
          uint32_t placed = 0, first = 0, final = 0;
#pragma unroll
          for (int w = 0; w < AW; ++w) {
            const uint64_t p = REM(qn, w) & (w ? ~0ull : ~visited);
            if (!p) continue;
            if (!placed) first = 64u * w + __ffsll(static_cast<long long>(p)) - 1u;
            placed += __popcll(p);
            final = 64u * w + 63u - __clzll(static_cast<long long>(p));
            if (w == 0 && !find_first) visited |= p & low;
          }
          if (placed) {
            if (find_first) {
              found = 1;
              MAP(qn) = static_cast<uint8_t>(first);
              break;
            }
            found += placed;
            MAP(qn) = static_cast<uint8_t>(final);
          }
        } else {
          uint32_t t = 0xFFFFFFFFu;
#pragma unroll
          for (int w = 0; w < AW; ++w) {
            const uint64_t r = REM(qn, w);
            if (t == 0xFFFFFFFFu && r) {
              t = 64u * w + __ffsll(static_cast<long long>(r)) - 1u;
              REM(qn, w) = r & (r - 1);
            }
          }
          if (t != 0xFFFFFFFFu) {
            const uint64_t bit = t < 64u ? (1ull << t) & low : 0ull;
            if (visited & bit) continue;
            // place t at depth qn and push the frame of depth qn + 1
            MAP(qn) = static_cast<uint8_t>(t);
            visited |= bit;
            // isValidMapping for depth d = qn + 1 against mapping[0..qn]: a
            // candidate is in the rows of d's earlier neighbours and no other
            const uint32_t d = qn + 1;
            const uint64_t sel = qsel_id[qoff + d];  // bit i: query vertex i < d has d in its row
            const uint32_t cn = __popcll(sel);
            const uint32_t i1 = cn ? __ffsll(static_cast<long long>(sel)) - 1u : 0u, i2 = cn ? 63u - __clzll(static_cast<long long>(sel)) : 0u;
            const uint32_t t1 = i1 == qn ? t : MAP(i1), t2 = i2 == qn ? t : MAP(i2);
            const uint64_t e0 = cn == 1u ? ~0ull : 0ull, e1 = cn == 2u ? ~0ull : 0ull;
#pragma unroll
            for (int w = 0; w < AW; ++w) {
              const uint64_t r = row_of(t, w), b0 = P0(qn, w), b1 = P1(qn, w);
              const uint64_t n0 = (b0 ^ r) | (b1 & b0), n1 = b1 | (b0 & r);
              uint64_t vm = CM(d, w);
              if (cn <= 2u) {
                if (cn) vm &= row_of(t1, w) & row_of(t2, w);
                vm &= ~((n0 ^ e0) | (n1 ^ e1));
              } else {
                for (uint32_t i = 0; i <= qn; ++i)
                  vm &= ~(row_of(i == qn ? t : MAP(i), w) ^ (0ull - ((sel >> i) & 1ull)));
              }
              REM(d, w) = vm;
              P0(d, w) = n0;
              P1(d, w) = n1;
            }
            ++top;
            continue;
          }
        }
        // the frame at depth qn is used up
        --top;
        const uint32_t mq = MAP(qn);  // mapping[qn], perhaps stale
        visited &= ~(mq < 64u ? ((1ull << mq) & low) : (mq == kLitOutside ? outside_bit : 0ull));
        if (top == 1) visited = 0;
        if (budget_spent(lim, steps)) {
          stop = true;
          break;
        }
      }
      if (stop) continue;
      counts[seg0 + it] = found;
      my_total += found;
    }
  }
#undef CM
#undef REM
#undef P0
#undef P1
#undef MAP
  __shared__ unsigned long long s_total;
  if (tid == 0) s_total = 0;
  __syncthreads();
  if (my_total) atomicAdd(&s_total, static_cast<unsigned long long>(my_total));
  __syncthreads();
  if (tid == 0 && s_total) atomicAdd(d_total, s_total);
}

// getEdgeLabel (graph.hpp:88-93): label of the CSR entry a -> b, or 255.
__device__ __forceinline__ uint8_t csr_edge_label(uint32_t a, uint32_t b, const uint32_t* __restrict__ roff,
                                                  const uint32_t* __restrict__ col, const uint8_t* __restrict__ el) {
  for (uint32_t i = roff[a]; i < roff[a + 1]; ++i)
    if (col[i] == b) return el[i];
  return 0xFFu;
}

// joinWildcardCandidates (isomorphism.hpp:435-560) with defineMatchingOrder
// (:383-408) and the bond-label isValidMapping (:410-433).  A block is the
// reference's work-group of join_work_group_size items, one data graph at a
// time; warp w is sub-group w and takes GMCR segment slots w, w + warps, ...
// For a slot the warp picks the root (the query vertex among the first 32
// with the most candidates, highest id on ties: two warp max-reductions), and
// lane l runs one DFS per starting candidate l, l + 32, ... of the root, with
// the driver join's `visited` bitset (cleared and re-seeded with the root when
// the DFS is back at depth 1).  find_first ends a lane's DFS at its first match.  mapping[]
// (per query vertex) starts zeroed per lane and carries over between its DFS
// runs, as the reference's private array does.  Like the driver's join, the
// count depends on these steps only where the visited set is live.  This kernel
// takes batches with graphs over 256 vertices; in the others
// k_join_wildcard_sets takes the graphs starting below vertex 256 (REF_PTX) and
// k_join_wide<.., BONDS> the rest.
__global__ void k_join_wildcard(const uint32_t* __restrict__ bits, uint64_t Wp, int prof, const uint32_t* __restrict__ qgoff,
                                const uint64_t* __restrict__ qadj, const uint32_t* __restrict__ qroff,
                                const uint32_t* __restrict__ qcol, const uint8_t* __restrict__ qel,
                                const uint32_t* __restrict__ dgoff, const uint64_t* __restrict__ dadj, uint32_t dAW,
                                const uint32_t* __restrict__ droff, const uint32_t* __restrict__ dcol,
                                const uint8_t* __restrict__ del, const uint32_t* __restrict__ offsets,
                                const uint32_t* __restrict__ indices, uint32_t G, int find_first,
                                uint64_t* __restrict__ counts, unsigned long long* __restrict__ d_total) {
  const unsigned lane = threadIdx.x & 31u, sg = threadIdx.x >> 5, nsg = blockDim.x >> 5;
  uint64_t my_total = 0;
  PairCands pc;
  uint32_t mapping[kMaxQueryNodes];
#pragma unroll 1
  for (uint32_t k = 0; k < kMaxQueryNodes; ++k) mapping[k] = 0;
  uint8_t order[kMaxQueryNodes];
  for (uint32_t g = blockIdx.x; g < G; g += gridDim.x) {
    const uint32_t s = dgoff[g], e = dgoff[g + 1], ng = e - s;
    const bool small = ng <= 64u;
    const uint32_t seg0 = offsets[g], seglen = offsets[g + 1] - seg0;
    for (uint32_t it = sg; it < seglen; it += nsg) {
      const uint32_t qg = indices[seg0 + it];
      const uint32_t qoff = qgoff[qg], n = qgoff[qg + 1] - qoff;
      if (small) pc.load(bits, Wp, qoff, n, s, e, prof);
      auto count_of = [&](uint32_t qn) -> uint32_t {
        return small ? pc.cnt[qn] : cand_count(bits + static_cast<uint64_t>(qoff + qn) * Wp, s, e, prof);
      };
      auto cand_of = [&](uint32_t qn, uint32_t idx) -> uint32_t {
        return small ? pc.at(qn, idx) : cand_at(bits + static_cast<uint64_t>(qoff + qn) * Wp, idx, s, e, prof);
      };
      // defineMatchingOrder: lane i holds query vertex i (< 32)
      const uint32_t mine = lane < n ? count_of(lane) : 0u;
      const uint32_t max_c = __reduce_max_sync(0xFFFFFFFFu, mine);
      const int root = __reduce_max_sync(0xFFFFFFFFu, (lane < n && mine == max_c) ? static_cast<int>(lane) : -1);
      order[0] = static_cast<uint8_t>(root);
#pragma unroll 1
      for (uint32_t i = 0, j = 1; i < n; ++i)
        if (static_cast<int>(i) != root) order[j++] = static_cast<uint8_t>(i);
      auto valid = [&](uint32_t cand, uint32_t depth) -> bool {
        const uint32_t qd = order[depth];
        for (uint32_t i = 0; i < depth; ++i) {
          const uint32_t qi = order[i];
          const bool qa = (qadj[qoff + qi] >> qd) & 1ull;
          if (qa != data_neighbor(mapping[qi], cand, s, ng, dadj, dAW, droff, dcol)) return false;
          if (qa && csr_edge_label(mapping[qi], cand, droff, dcol, del) != csr_edge_label(qoff + qi, qoff + qd, qroff, qcol, qel))
            return false;
        }
        return true;
      };
      uint64_t found = 0;
      for (uint32_t sc = lane; sc < max_c; sc += 32u) {
        Frame stack[kMaxQueryNodes + 2];
        uint32_t top = 0;
        const uint32_t r = order[0];
        mapping[r] = cand_of(r, sc);
        stack[top++] = {1u, 0u};
        uint64_t visited = refbit(mapping[r], s);  // Bitset<uint64_t>{offset = s}
        while (top > 0) {
          const Frame fr = stack[top - 1];
          if (fr.depth == n) {
            ++found;
            --top;
            if (find_first) break;
            continue;
          }
          const uint32_t qn = order[fr.depth];
          if (fr.idx >= count_of(qn)) {
            --top;
            visited &= ~refbit(mapping[qn], s);
            if (top == 1) visited = refbit(mapping[r], s);
            continue;
          }
          const uint32_t cand = cand_of(qn, fr.idx);
          stack[top - 1].idx++;
          if (visited & refbit(cand, s)) continue;
          if (valid(cand, fr.depth)) {
            mapping[qn] = cand;
            visited |= refbit(cand, s);
            stack[top++] = {fr.depth + 1, 0u};
          }
        }
      }
      my_total += found;
      uint64_t slot_total = found;
      for (int o = 16; o; o >>= 1) slot_total += __shfl_xor_sync(0xFFFFFFFFu, slot_total, o);
      if (lane == 0 && counts) counts[seg0 + it] = slot_total;
    }
  }
  for (int o = 16; o; o >>= 1) my_total += __shfl_xor_sync(0xFFFFFFFFu, my_total, o);
  if (lane == 0 && my_total) atomicAdd(d_total, static_cast<unsigned long long>(my_total));
}

// Position of the r-th (0-based) set bit of m; m has more than r set bits.
__device__ __forceinline__ uint32_t nth_set32(uint32_t m, uint32_t r) {
  uint32_t pos = 0, c = __popc(m & 0xFFFFu);
  if (r >= c) { r -= c; pos += 16; m >>= 16; }
  c = __popc(m & 0xFFu);
  if (r >= c) { r -= c; pos += 8; m >>= 8; }
  c = __popc(m & 0xFu);
  if (r >= c) { r -= c; pos += 4; m >>= 4; }
  c = __popc(m & 0x3u);
  if (r >= c) { r -= c; pos += 2; m >>= 2; }
  if (r >= (m & 1u)) pos += 1;
  return pos;
}
__device__ __forceinline__ uint32_t nth_set64(uint64_t m, uint32_t r) {
  const uint32_t lo = static_cast<uint32_t>(m), c = __popc(lo);
  const bool up = r >= c;
  return (up ? 32u : 0u) + nth_set32(up ? static_cast<uint32_t>(m >> 32) : lo, up ? r - c : r);
}

// The set's members whose rank is `share` modulo 1 << log2n.
__device__ __forceinline__ uint64_t share_of(uint64_t set, uint32_t share, uint32_t log2n) {
  if (!log2n) return set;
  uint64_t keep = 0;
  for (uint32_t r = 0; set; ++r, set &= set - 1)
    if ((r & ((1u << log2n) - 1u)) == share) keep |= set & (0ull - set);
  return keep;
}

// The join of the pairs listed by k_pair_masks as too large for the two-phase
// join: queries of up to kMaxQueryNodes vertices, molecules of up to 64 * AW
// atoms.  A warp takes a batch of up to `batch` pairs, builds their level masks
// in shared memory with all lanes busy (an item per (pair, level), as in
// k_pair_masks), and then its lanes run k_join_dfs's turns, each lane on one
// root candidate of one pair at a time (or, where a pair has few, on a share of one
// candidate's searches, by the next level's candidates), so a heavy pair is spread
// over the warp.  (A star of four in a star of 100 atoms: 2.25 ms by one lane, 0.20
// so; the first turn of a share is taken with the item, so the turns are as before.)
// The per-level state is in local memory (the pairs are few).  The
// one-lane-per-part form that this replaced rebuilt every mask in every part:
// 1.43 ms for the 0.4 % of 6.86 M pairs with queries over 16 vertices.
constexpr uint32_t kWideWarps = 4;
constexpr uint32_t kWideBatch = 8;
constexpr size_t kWideMaskBytes = 8192;  // level masks of one warp's batch, at most
struct WideEntry {
  uint64_t cnt;
  uint32_t qoff, n, s, slot;  // qoff: identity-order flag in bit 31
  uint32_t root;              // BONDS: the query vertex placed first
  uint32_t items, log2n;      // root candidates x shares of the next level's candidates (2^log2n)
  uint32_t next;              // items taken
};
// [batch] entries, [batch][AW] root candidates, [batch][stride] masks per warp
inline size_t wide_smem(uint32_t batch, uint32_t aw, uint32_t stride) {
  return kWideWarps * batch * (sizeof(WideEntry) + 8ull * aw + 8ull * stride);
}

//
// BONDS: joinWildcardCandidates for every slot of the data graphs from
// `first_graph` on (no list): the root is the query vertex (of the first 32)
// with the most candidates, highest id on ties, the others follow in id order,
// an earlier neighbour's row holds only the bonds with the query edge's label,
// and with find_first every root candidate that extends to a match counts 1.
// (k_join_wildcard on all slots: 5.09 ms for 22,323 pairs of 2,003 molecules x
// 40 queries, one lane per root candidate and a walk over the earlier levels
// and CSR rows for every candidate.)
struct BondGraphs {
  const uint64_t* qadj = nullptr;
  const uint32_t *qroff = nullptr, *qcol = nullptr, *droff = nullptr, *dcol = nullptr, *doffsets = nullptr;
  const uint8_t *qel = nullptr, *del = nullptr;
  uint32_t first_graph = 0;
  uint64_t total_slots = 0;
};

// Neighbours of data vertex a (graph [s, s + 64 AW)) over bonds of label l; the
// first CSR entry of a neighbour gives its label (graph.hpp:88-93).
template <int AW>
__device__ __forceinline__ void bond_row(const BondGraphs& bg, uint32_t a, uint32_t s, uint8_t l, uint64_t* out) {
  uint64_t seen[AW];
#pragma unroll
  for (int w = 0; w < AW; ++w) seen[w] = out[w] = 0;
  const uint32_t i1 = bg.droff[a + 1];
  for (uint32_t i = bg.droff[a]; i < i1; ++i) {
    const uint32_t t = bg.dcol[i] - s;
    const bool same = bg.del[i] == l;
#pragma unroll
    for (int w = 0; w < AW; ++w) {
      const uint64_t bit = (t >> 6) == static_cast<uint32_t>(w) ? 1ull << (t & 63u) : 0ull;
      if (same) out[w] |= bit & ~seen[w];
      seen[w] |= bit;
    }
  }
}

// k_join_wildcard (REF_PTX) for graphs of at most 64 * AW vertices, on
// graph-local sets: the same searches in the same order, a warp per sub-group
// of a graph (sub-group sg of nsg takes the segment's slots sg, sg + nsg, ...),
// its slot's masks built once by all lanes, and per lane and level the
// candidates left and the neighbour counts in shared memory, as in
// k_join_literal_sets.  With the walk over the earlier levels and CSR rows per
// candidate: 1.53 ms for the first ten molecules of 2,003 x 40 pairs, this
// 0.21 ms.
inline size_t wildcard_smem(uint32_t aw, uint32_t levels) {
  return 32ull * levels * (24ull * aw + 1u) + 8ull * levels * aw;
}

template <int AW>
__global__ void __launch_bounds__(32) k_join_wildcard_sets(MaskSource src, BondGraphs bg, const uint32_t* __restrict__ qgoff,
                                                           const uint64_t* __restrict__ qsel_id,
                                                           const uint32_t* __restrict__ dgoff,
                                                           const uint64_t* __restrict__ dadj,
                                                           const uint32_t* __restrict__ indices, uint32_t graphs, uint32_t nsg,
                                                           uint32_t levels, int find_first, uint64_t* __restrict__ counts,
                                                           unsigned long long* __restrict__ d_total) {
  extern __shared__ uint64_t wild_sm[];
  constexpr unsigned kAll = 0xFFFFFFFFu;
  const uint32_t lane = threadIdx.x, L = levels;
  uint64_t* M = wild_sm;                          // [vertex][AW]
  uint64_t* rem = wild_sm + L * AW + lane;        // [level][AW][32]
  uint64_t* p0 = rem + 32u * L * AW;
  uint64_t* p1 = p0 + 32u * L * AW;
  uint8_t* map = reinterpret_cast<uint8_t*>(wild_sm + L * AW + 96u * L * AW) + lane;  // [vertex][32] local ids
#define LVL(arr, d, w) arr[((d) * AW + (w)) * 32u]
  uint64_t my_total = 0;
  for (uint32_t blk = blockIdx.x; blk < graphs * nsg; blk += gridDim.x) {
    const uint32_t g = blk / nsg, sg = blk % nsg;
    const uint32_t s = dgoff[g], e = dgoff[g + 1];
    const uint32_t seg0 = bg.doffsets[g], seglen = bg.doffsets[g + 1] - seg0;
    const uint64_t low = s >= 256u ? 0ull : (256u - s >= 64u ? ~0ull : ((1ull << (256u - s)) - 1ull));
    auto bit_of = [&](uint32_t t) -> uint64_t { return t < 64u ? (1ull << t) & low : 0ull; };
    // mapping[] of a fresh work-item: global vertex 0
#pragma unroll 1
    for (uint32_t k = 0; k < L; ++k) map[k * 32u] = s == 0 ? 0 : kLitOutside;
    for (uint32_t it = sg; it < seglen; it += nsg) {
      const uint32_t qg = indices[seg0 + it];
      const uint32_t v0 = qgoff[qg], n = qgoff[qg + 1] - v0;
      __syncwarp();
      for (uint32_t j = lane; j < n; j += 32u) source_mask<AW>(src, AW, v0 + j, g, s, e, M + j * AW);
      __syncwarp();
      uint32_t mine = 0;
      if (lane < n)
#pragma unroll
        for (int w = 0; w < AW; ++w) mine += __popcll(M[lane * AW + w]);
      const uint32_t max_c = __reduce_max_sync(kAll, mine);
      const uint32_t root = __reduce_max_sync(kAll, lane < n && mine == max_c ? lane : 0u);
      const uint64_t below = (1ull << root) - 1ull;
      uint64_t found = 0;
      for (uint32_t sc = lane; sc < max_c; sc += 32u) {
        uint32_t t0 = 0, skip = sc;  // the sc-th candidate of the root
#pragma unroll
        for (int w = 0; w < AW; ++w) {
          uint64_t m = M[root * AW + w];
          const uint32_t c = __popcll(m);
          if (skip < c) {
            for (; skip; --skip) m &= m - 1;
            t0 = 64u * w + __ffsll(static_cast<long long>(m)) - 1u;
            skip = 0xFFFFFFFFu;
          } else if (skip != 0xFFFFFFFFu) {
            skip -= c;
          }
        }
        map[root * 32u] = static_cast<uint8_t>(t0);
        uint64_t visited = bit_of(t0);
        uint32_t d = 0, t = t0;  // t was placed at level d: find the candidates of level d + 1
        for (bool placed = true;;) {
          if (placed) {
            const uint32_t v = d + 1u <= root ? d : d + 1u;
            uint64_t sel = qsel_id[v0 + v];
            sel = ((bg.qadj[v0 + root] >> v) & 1ull) | ((sel & below) << 1) | (sel & ~((below << 1) | 1ull));
            const uint32_t cn = __popcll(sel);
            uint64_t n0[AW], n1[AW], f[AW];
#pragma unroll
            for (int w = 0; w < AW; ++w) {
              const uint64_t r = dadj[static_cast<uint64_t>(s + t) * AW + w];
              const uint64_t b0 = d ? LVL(p0, d, w) : 0ull, b1 = d ? LVL(p1, d, w) : 0ull;
              n0[w] = (b0 ^ r) | (b1 & b0);
              n1[w] = b1 | (b0 & r);
              f[w] = M[v * AW + w];
            }
            for (uint64_t m = sel; m; m &= m - 1) {
              const uint32_t i = __ffsll(static_cast<long long>(m)) - 1;
              const uint32_t u = i == 0 ? root : (i <= root ? i - 1u : i);
              uint64_t row[AW];
              bond_row<AW>(bg, s + map[u * 32u], s, csr_edge_label(v0 + u, v0 + v, bg.qroff, bg.qcol, bg.qel), row);
#pragma unroll
              for (int w = 0; w < AW; ++w) f[w] &= row[w];
            }
            if (cn <= 2u) {
              const uint64_t e0 = cn == 1u ? ~0ull : 0ull, e1 = cn == 2u ? ~0ull : 0ull;
#pragma unroll
              for (int w = 0; w < AW; ++w) f[w] &= ~((n0[w] ^ e0) | (n1[w] ^ e1));
            } else {
              for (uint32_t i = 0; i <= d; ++i) {
                const uint32_t u = i == 0 ? root : (i <= root ? i - 1u : i);
                const uint64_t* row = dadj + static_cast<uint64_t>(s + map[u * 32u]) * AW;
                const uint64_t want = 0ull - ((sel >> i) & 1ull);
#pragma unroll
                for (int w = 0; w < AW; ++w) f[w] &= ~(row[w] ^ want);
              }
            }
            ++d;
#pragma unroll
            for (int w = 0; w < AW; ++w) {
              LVL(rem, d, w) = f[w];
              LVL(p0, d, w) = n0[w];
              LVL(p1, d, w) = n1[w];
            }
            placed = false;
          }
          const uint32_t v = d <= root ? d - 1u : d;  // the frame's query vertex
          if (d + 1u == n) {  // the last one in one step, as in k_join_literal_sets
            uint32_t c = 0, first = 0, final = 0;
#pragma unroll
            for (int w = 0; w < AW; ++w) {
              const uint64_t p = LVL(rem, d, w) & (w ? ~0ull : ~visited);
              if (!p) continue;
              if (!c) first = 64u * w + __ffsll(static_cast<long long>(p)) - 1u;
              c += __popcll(p);
              final = 64u * w + 63u - __clzll(static_cast<long long>(p));
              if (w == 0 && !find_first) visited |= p & low;
            }
            if (c) {
              map[v * 32u] = static_cast<uint8_t>(find_first ? first : final);
              found += find_first ? 1u : c;
              if (find_first) break;
            }
          } else {
            t = 0xFFFFFFFFu;
#pragma unroll
            for (int w = 0; w < AW; ++w) {
              const uint64_t r = LVL(rem, d, w);
              if (t == 0xFFFFFFFFu && r) {
                t = 64u * w + __ffsll(static_cast<long long>(r)) - 1u;
                LVL(rem, d, w) = r & (r - 1);
              }
            }
            if (t != 0xFFFFFFFFu) {
              if (!(visited & bit_of(t))) {
                map[v * 32u] = static_cast<uint8_t>(t);
                visited |= bit_of(t);
                placed = true;
              }
              continue;
            }
          }
          // the frame is used up
          visited &= ~bit_of(map[v * 32u]);  // mapping[], perhaps stale
          if (--d == 0) break;
          if (d == 1u) visited = bit_of(t0);  // back at the first frame: the root alone
        }
      }
      my_total += found;
      uint64_t slot_total = found;
      for (int o = 16; o; o >>= 1) slot_total += __shfl_xor_sync(kAll, slot_total, o);
      if (lane == 0) counts[seg0 + it] = slot_total;
    }
  }
#undef LVL
  for (int o = 16; o; o >>= 1) my_total += __shfl_xor_sync(kAll, my_total, o);
  if (lane == 0 && my_total) atomicAdd(d_total, static_cast<unsigned long long>(my_total));
}

template <int AW, bool EXACT, bool BONDS>
__global__ void __launch_bounds__(kWideWarps * 32) k_join_wide(
    MaskSource src, BondGraphs bg, const uint32_t* __restrict__ qgoff, const uint8_t* __restrict__ qorder, const uint64_t* __restrict__ qsel,
    const uint64_t* __restrict__ qsel_id, const uint8_t* __restrict__ qsym, const uint32_t* __restrict__ dgoff,
    const uint64_t* __restrict__ dadj, const uint8_t* __restrict__ dsym, const uint32_t* __restrict__ indices,
    const uint32_t* __restrict__ pair_graph, const uint32_t* __restrict__ list, const unsigned long long* __restrict__ list_len,
    uint32_t batch, uint32_t stride, int find_first, unsigned long long* __restrict__ cursor, uint64_t* __restrict__ counts,
    unsigned long long* __restrict__ d_total, JoinLimit lim) {
  extern __shared__ __align__(16) unsigned char wide_raw[];
  constexpr unsigned kAll = 0xFFFFFFFFu;
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  unsigned char* base = wide_raw + static_cast<size_t>(warp) * batch * (sizeof(WideEntry) + 8u * AW + 8ull * stride);
  WideEntry* ent = reinterpret_cast<WideEntry*>(base);
  unsigned long long* roots = reinterpret_cast<unsigned long long*>(ent + batch);
  uint64_t* masks = reinterpret_cast<uint64_t*>(roots + batch * AW);
  uint64_t rest[kMaxQueryNodes][AW], p0[kMaxQueryNodes][AW], p1[kMaxQueryNodes][AW];
  uint8_t pick[kMaxQueryNodes];
#pragma unroll
  for (int w = 0; w < AW; ++w) p0[0][w] = p1[0][w] = 0;
  const uint64_t first = BONDS ? bg.doffsets[bg.first_graph] : 0;
  const uint64_t total = BONDS ? bg.total_slots - first : *list_len;
  uint64_t my_total = 0, steps = 0;
  for (;;) {
    unsigned long long b = total;
    if (lane == 0 && !join_stopped(lim)) b = atomicAdd(cursor, static_cast<unsigned long long>(batch));
    b = __shfl_sync(kAll, b, 0);
    if (b >= total) break;
    const uint32_t ne = static_cast<uint32_t>(total - b < batch ? total - b : batch);
    // the batch's pairs, one lane each
    uint32_t n = 0, qoff = 0, g = 0, s = 0, e = 0;
    bool ident = true;
    if (lane < ne) {
      const uint32_t slot = BONDS ? static_cast<uint32_t>(first + b + lane) : list[b + lane];
      const uint32_t qg = indices[slot];
      qoff = qgoff[qg];
      n = qgoff[qg + 1] - qoff;
      g = pair_graph[slot];
      s = dgoff[g];
      e = dgoff[g + 1];
      ident = BONDS || !(qsym[qg] && dsym[g]);
      ent[lane] = WideEntry{0, qoff | (ident ? 0x80000000u : 0u), n, s, slot, 0, 0, 0, 0};
    }
    uint32_t incl = n;
#pragma unroll
    for (unsigned o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(kAll, incl, o);
      if (lane >= o) incl += v;
    }
    const uint32_t excl = incl - n, items = __shfl_sync(kAll, incl, 31);
    for (uint32_t i0 = 0; i0 < items; i0 += 32) {
      const uint32_t it = i0 + lane;
      uint32_t pos = 0;  // the last pair whose first item is <= it
      for (uint32_t k = 1; k < ne; ++k)
        if (__shfl_sync(kAll, excl, k) <= it) pos = k;
      const uint32_t j = it - __shfl_sync(kAll, excl, pos), oq = __shfl_sync(kAll, qoff, pos), og = __shfl_sync(kAll, g, pos);
      const uint32_t os = __shfl_sync(kAll, s, pos), oe = __shfl_sync(kAll, e, pos);
      const bool oi = __shfl_sync(kAll, static_cast<unsigned>(ident), pos) != 0u;
      if (it < items) source_mask<AW>(src, AW, oq + (oi ? j : qorder[oq + j]), og, os, oe, masks + pos * stride + j * AW);
    }
    __syncwarp();
    if (BONDS) {  // the root of each pair (defineMatchingOrder, isomorphism.hpp:383-408)
      for (uint32_t c = 0; c < ne; ++c) {
        const uint32_t m = ent[c].n < 32u ? ent[c].n : 32u;
        uint32_t mine = 0;
        if (lane < m)
#pragma unroll
          for (int w = 0; w < AW; ++w) mine += __popcll(masks[c * stride + lane * AW + w]);
        const uint32_t most = __reduce_max_sync(kAll, mine);
        const uint32_t root = __reduce_max_sync(kAll, lane < m && mine == most ? lane : 0u);
        if (lane == 0) ent[c].root = root;
      }
      __syncwarp();
    }
    for (uint32_t i = lane; i < ne * AW; i += 32)
      roots[i] = masks[(i / AW) * stride + (BONDS ? ent[i / AW].root * AW : 0u) + i % AW];
    __syncwarp();
    // an item is a root candidate, or a share of its searches (by the next
    // level's candidates) where a pair has fewer of them than its part of the
    // warp's lanes (BONDS: the root has the most candidates of all)
    if (lane < ne) {
      WideEntry& en = ent[lane];
      uint32_t c0 = 0, c1 = 0;
#pragma unroll
      for (int w = 0; w < AW; ++w) {
        c0 += __popcll(roots[lane * AW + w]);
        c1 += __popcll(masks[lane * stride + AW + w]);
      }
      uint32_t log2n = 0;
      while (!BONDS && ((c0 * ne) << log2n) < 32u && (2u << log2n) <= c1) ++log2n;
      en.log2n = log2n;
      en.items = c0 << log2n;
    }
    __syncwarp();
    // the lanes' searches
    uint64_t alive = 0, cnt = 0;  // alive: levels with untried candidates
    uint32_t my = 0;              // this lane's pair within the batch
    const uint64_t* selp = qsel;
    const uint64_t* M = masks;
    const uint64_t* arow = dadj;
    uint32_t root = 0, v0 = 0;    // BONDS: the root, and the query's first vertex
    bool dry = false;  // no item left for this lane
    auto flush = [&]() {
      auto* at = reinterpret_cast<unsigned long long*>(&ent[my].cnt);
      if (find_first && !BONDS) atomicExch(at, 1ull);
      else atomicAdd(at, static_cast<unsigned long long>(find_first ? 1ull : cnt));
      cnt = 0;
    };
    for (;;) {
      if (!alive && cnt) flush();
      while (!alive && !dry) {
        dry = true;
        uint32_t item = 0;
        for (uint32_t i = 0; i < ne && dry; ++i) {
          const uint32_t c = (lane + i) % ne, items = ent[c].items;
          if (find_first && !BONDS && *reinterpret_cast<volatile uint64_t*>(&ent[c].cnt)) continue;
          if (*reinterpret_cast<volatile uint32_t*>(&ent[c].next) >= items) continue;
          item = atomicAdd(&ent[c].next, 1u);
          if (item < items) {
            dry = false;
            my = c;
          }
        }
        if (dry) break;
        const WideEntry& en = ent[my];
        n = en.n;
        selp = ((en.qoff >> 31) ? qsel_id : qsel) + (en.qoff & 0x7FFFFFFFu);
        arow = dadj + static_cast<uint64_t>(en.s) * AW;
        M = masks + my * stride;
        root = en.root;
        v0 = en.qoff & 0x7FFFFFFFu;
        s = en.s;
        // the item's root candidate
        uint32_t skip = item >> en.log2n, t = 0;
        bool found = false;
#pragma unroll
        for (int w = 0; w < AW; ++w) {
          const uint64_t v = roots[my * AW + w];
          const uint32_t c = __popcll(v);
          const bool here = !found && skip < c;
          if (here) t = 64u * w + nth_set64(v, skip);
          found |= here;
          skip -= found ? 0u : c;
        }
        if (BONDS || !en.log2n) {
#pragma unroll
          for (int w = 0; w < AW; ++w) rest[0][w] = (t >> 6) == static_cast<uint32_t>(w) ? 1ull << (t & 63u) : 0ull;
          alive = 1;
          continue;
        }
        // a share: its first turn here, with the share of level 1's candidates
        const uint32_t mod = (1u << en.log2n) - 1u;
        const uint64_t next_to = 0ull - (selp[1] & 1ull);
        pick[0] = static_cast<uint8_t>(t);
        uint32_t rank = 0, c = 0;
        for (uint32_t w = 0; w < AW; ++w) {
          uint64_t keep = 0;
          for (uint64_t x = M[AW + w]; x; x &= x - 1, ++rank)
            if ((rank & mod) == (item & mod)) keep |= x & (0ull - x);
          const uint64_t r = arow[t * AW + w];
          const uint64_t bit = EXACT && (t >> 6) == w ? 1ull << (t & 63u) : 0ull;
          keep &= ~(r ^ next_to) & ~bit;
          rest[1][w] = keep;
          p0[1][w] = r | bit;
          p1[1][w] = bit;
          c += __popcll(keep);
        }
        if (n > 2u) {
          alive = c ? 2u : 0u;
        } else if (c) {  // level 1 is the last
          cnt = c;
          flush();
        }
      }
      if (!__any_sync(kAll, alive != 0)) break;
      if (!alive) continue;
      if (find_first && !BONDS && *reinterpret_cast<volatile uint64_t*>(&ent[my].cnt)) {
        alive = 0;
        continue;
      }
      // one turn of k_join_dfs on AW-word sets
      const uint32_t k = 63u - __clzll(static_cast<long long>(alive));
      uint32_t t = 0;
      uint64_t left = 0;
#pragma unroll
      for (int w = 0; w < AW; ++w)
        if (rest[k][w]) t = 64u * w + 63u - __clzll(static_cast<long long>(rest[k][w]));
#pragma unroll
      for (int w = 0; w < AW; ++w) {
        if ((t >> 6) == static_cast<uint32_t>(w)) rest[k][w] ^= 1ull << (t & 63u);
        left |= rest[k][w];
      }
      if (!left) alive ^= 1ull << k;
      pick[k] = static_cast<uint8_t>(t);
      // the next level's query vertex and its earlier neighbours (by level)
      const uint32_t v = !BONDS ? k + 1u : (k + 1u <= root ? k : k + 1u);
      uint64_t sel = selp[v];
      if (BONDS) {
        const uint64_t below = (1ull << root) - 1ull;
        const uint64_t to_root = (bg.qadj[v0 + root] >> v) & 1ull;
        sel = to_root | ((sel & below) << 1) | (sel & ~((below << 1) | 1ull));
      }
      const uint32_t cn = __popcll(sel);
      uint64_t n0[AW], n1[AW], f[AW];
#pragma unroll
      for (int w = 0; w < AW; ++w) {
        const uint64_t r = arow[t * AW + w], b0 = p0[k][w], b1 = p1[k][w];
        const uint64_t bit = EXACT && (t >> 6) == static_cast<uint32_t>(w) ? 1ull << (t & 63u) : 0ull;
        n0[w] = (b0 ^ r) | (b1 & b0) | bit;
        n1[w] = b1 | (b0 & r) | bit;
        f[w] = M[v * AW + w];
      }
      if (BONDS) {  // bond labels of the earlier neighbours
        for (uint64_t m = sel; m; m &= m - 1) {
          const uint32_t i = __ffsll(static_cast<long long>(m)) - 1;
          const uint32_t u = i == 0 ? root : (i <= root ? i - 1u : i);
          uint64_t row[AW];
          bond_row<AW>(bg, s + pick[i], s, csr_edge_label(v0 + u, v0 + v, bg.qroff, bg.qcol, bg.qel), row);
#pragma unroll
          for (int w = 0; w < AW; ++w) f[w] &= row[w];
        }
      }
      if (cn <= 2u) {
        for (uint64_t m = BONDS ? 0ull : sel; m; m &= m - 1) {
          const uint64_t* row = arow + static_cast<uint32_t>(pick[__ffsll(static_cast<long long>(m)) - 1]) * AW;
#pragma unroll
          for (int w = 0; w < AW; ++w) f[w] &= row[w];
        }
        const uint64_t e0 = cn == 1u ? ~0ull : 0ull, e1 = cn == 2u ? ~0ull : 0ull;
#pragma unroll
        for (int w = 0; w < AW; ++w) f[w] &= ~((n0[w] ^ e0) | (n1[w] ^ e1));
      } else {
        for (uint32_t i = 0; i <= k; ++i) {
          const uint64_t* row = arow + static_cast<uint32_t>(pick[i]) * AW;
          const uint64_t want = 0ull - ((sel >> i) & 1ull);
#pragma unroll
          for (int w = 0; w < AW; ++w) {
            f[w] &= ~(row[w] ^ want);
            if (EXACT && (pick[i] >> 6) == w) f[w] &= ~(1ull << (pick[i] & 63u));
          }
        }
      }
      uint32_t c = 0;
#pragma unroll
      for (int w = 0; w < AW; ++w) c += __popcll(f[w]);
      if (c) {
        if (k + 2u == n) {  // the last level: every candidate is a match
          cnt += c;
          if (find_first) alive = 0;
        } else {
#pragma unroll
          for (int w = 0; w < AW; ++w) {
            rest[k + 1][w] = f[w];
            p0[k + 1][w] = n0[w];
            p1[k + 1][w] = n1[w];
          }
          alive |= 2ull << k;
        }
      }
      if (!left && budget_spent(lim, steps)) {
        alive = 0;
        dry = true;
      }
    }
    __syncwarp();
    if (lane < ne) {
      const uint64_t c = ent[lane].cnt;
      counts[ent[lane].slot] = c;
      my_total += c;
    }
    __syncwarp();
  }
  for (int o = 16; o; o >>= 1) my_total += __shfl_xor_sync(kAll, my_total, o);
  if (lane == 0 && my_total) atomicAdd(d_total, static_cast<unsigned long long>(my_total));
}

// Two-phase join for pairs whose query has <= kPhaseLevels vertices.
// Phase A (k_pair_masks): per slot of a chunk and per level j, the candidate
// set of the query vertex placed at level j = AND of its class's plane program
// for the slot's data graph, stored [slot-in-chunk][level] (coalesced: one
// 128-byte line per slot, so a pair's later levels hit in cache).
// Phase B: the DFS on those masks, k_join_dfs by default (k_join_masks and
// k_join_frontier for callers that set sigmo_tuning.join_kernel).
constexpr uint32_t kPhaseLevels = 16;
constexpr uint32_t kDfsLevels = 10;  // most vertices of a query in k_join_dfs's short form
constexpr uint32_t kPhaseThreads = 256;

// Bound by the L1 wavefronts of its gathers (a lane's class program and its
// plane words are its own), so a program is read four plane ids at a time
// (0.65 -> 0.52 ms for 6.86 M pairs against an id per load).
// Work layout: a warp takes 32 consecutive slots per round, one lane per slot
// for the slot's metadata and setup record, then the round's sum of query
// sizes (slot, level) items with every lane busy; an item finds its slot by a
// binary search over the lanes' exclusive prefix sums (warp shuffles).
template <bool FROM_PLANES>
__global__ void __launch_bounds__(256) k_pair_masks(
    MaskSource src, uint32_t AW, const uint32_t* __restrict__ qgoff, const uint8_t* __restrict__ qorder,
    const uint8_t* __restrict__ qsym, const uint32_t* __restrict__ dgoff, const uint8_t* __restrict__ dsym,
    const uint32_t* __restrict__ indices, const uint32_t* __restrict__ pair_graph, uint64_t slot0, uint64_t count,
    uint64_t* __restrict__ masks, uint4* __restrict__ rec, uint32_t skip_below, uint32_t* __restrict__ overflow,
    unsigned long long* __restrict__ overflow_len, uint32_t* __restrict__ longs, unsigned long long* __restrict__ longs_len,
    uint64_t* __restrict__ counts, int zero_counts) {
  const unsigned lane = threadIdx.x & 31u;
  const uint64_t warp = (static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = (static_cast<uint64_t>(gridDim.x) * blockDim.x) >> 5;
  for (uint64_t s0 = warp * 32; s0 < count; s0 += nwarps * 32) {
    const uint64_t local = s0 + lane;
    uint32_t n = 0, qoff = 0, g = 0, items = 0, ds = 0, de = 0;
    bool ident = true;
    if (local < count) {
      const uint64_t slot = slot0 + local;
      const uint32_t qg = indices[slot];
      qoff = qgoff[qg];
      n = qgoff[qg + 1] - qoff;
      g = pair_graph[slot];
      ident = !(qsym[qg] && dsym[g]);
      ds = dgoff[g];
      de = dgoff[g + 1];
      // queries over kPhaseLevels vertices and molecules over 64 atoms (a
      // vertex set wider than one word) go to k_join_wide
      const bool generic = n > kPhaseLevels || de - ds > 64u;
      // the pair's setup record: first data vertex, query size | flags (0x100
      // identity order, 0x200 generic, 0x400 long, 0x800 the literal join's),
      // query offset, query graph
      const bool lng = !generic && n > kDfsLevels;
      rec[local] = make_uint4(ds, n | (ident ? 0x100u : 0u) | (generic ? 0x200u : 0u) | (lng ? 0x400u : 0u) |
                                      (g < skip_below ? 0x800u : 0u), qoff, qg);
      if (longs && lng && g >= skip_below) {  // joined by k_join_dfs's long form, in parts
        longs[atomicAdd(longs_len, 1ull)] = static_cast<uint32_t>(slot);
        counts[slot] = 0;
      }
      if (generic && g >= skip_below) {
        overflow[atomicAdd(overflow_len, 1ull)] = static_cast<uint32_t>(slot);
      }
      if (zero_counts && g >= skip_below) counts[slot] = 0;  // the join adds up a pair's parts
      items = generic ? 0u : n;
    }
    uint32_t incl = items;
#pragma unroll
    for (unsigned o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
      if (lane >= o) incl += v;
    }
    const uint32_t excl = incl - items;
    const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
    for (uint32_t base = 0; base < total; base += 32) {
      const uint32_t it = base + lane;
      // owner: the last lane whose exclusive prefix is <= it
      uint32_t pos = 0;
#pragma unroll
      for (uint32_t step = 16; step; step >>= 1) {
        const uint32_t cand = pos + step;
        const uint32_t e = __shfl_sync(0xFFFFFFFFu, excl, cand & 31u);
        if (cand < 32u && e <= it) pos = cand;
      }
      const uint32_t o_excl = __shfl_sync(0xFFFFFFFFu, excl, pos);
      const uint32_t o_qoff = __shfl_sync(0xFFFFFFFFu, qoff, pos);
      const uint32_t o_g = __shfl_sync(0xFFFFFFFFu, g, pos);
      const bool o_ident = __shfl_sync(0xFFFFFFFFu, static_cast<unsigned>(ident), pos) != 0u;
      uint32_t o_s = 0, o_e = 0;
      if (!FROM_PLANES) {
        o_s = __shfl_sync(0xFFFFFFFFu, ds, pos);
        o_e = __shfl_sync(0xFFFFFFFFu, de, pos);
      }
      if (it >= total) continue;
      const uint32_t j = it - o_excl;
      const uint32_t v = o_qoff + (o_ident ? j : qorder[o_qoff + j]);
      // one word: the graph's vertex set fits it (word 0 of each plane)
      uint64_t m = ~0ull;
      if (FROM_PLANES) {
        const uint64_t* pb = src.planes + (src.tiled ? static_cast<uint64_t>(o_g >> 5) * src.K * AW * 32 + (o_g & 31u)
                                                     : static_cast<uint64_t>(o_g) * src.K * AW);
        const uint32_t step = src.tiled ? AW * 32u : AW;
        const uint32_t c = src.cls[v], e1 = src.prog_off[c + 1];
        for (uint32_t e = src.prog_off[c]; e < e1; ++e) {
          const uint64_t ids = src.prog[e];
          const uint32_t lo = static_cast<uint32_t>(ids), hi = static_cast<uint32_t>(ids >> 32);
          m &= (pb[(lo & 0xFFFFu) * step] & pb[(lo >> 16) * step]) & (pb[(hi & 0xFFFFu) * step] & pb[(hi >> 16) * step]);
        }
      } else {
        extract_local<1>(src.bits + static_cast<uint64_t>(v) * src.Wp, o_s, o_e, src.prof, &m);
      }
      masks[(s0 + pos) * kPhaseLevels + j] = m;
    }
  }
}

// Phase B with sigmo_tuning.join_kernel = 0: the DFS as a flat per-lane state
// machine whose pair setup is just the load of the masks (issued one pair ahead,
// so the DRAM latency of a refill overlaps the current pair's DFS), with the
// per-level state in shared memory ([level][thread]).  Trying a candidate t at
// level k is O(1): next = base[k+1] & (row(t) or ~row(t)) [& ~used]; base[k+2] is
// computed once per descent.
// DAW: words per adjacency row of the data batch (the pairs here use word 0).
template <bool EXACT, uint32_t DAW>
__global__ void __launch_bounds__(kPhaseThreads) k_join_masks(
    const uint64_t* __restrict__ masks, const uint4* __restrict__ rec, uint64_t slot0, uint64_t count,
    const uint64_t* __restrict__ qsel, const uint64_t* __restrict__ qsel_id, const uint64_t* __restrict__ dadj,
    int find_first, uint32_t kChunk, unsigned long long* __restrict__ cursor,
    uint64_t* __restrict__ counts, unsigned long long* __restrict__ d_total, JoinLimit lim) {
  extern __shared__ uint64_t sm[];
  uint64_t steps = 0;
  const unsigned tid = threadIdx.x, lane = tid & 31u;
  uint64_t* cand = sm;
  uint64_t* base = sm + kPhaseLevels * kPhaseThreads;
  uint8_t* pk = reinterpret_cast<uint8_t*>(sm + 2 * kPhaseLevels * kPhaseThreads);
#define AT(arr, lvl) arr[(lvl) * kPhaseThreads + tid]
  uint64_t my_total = 0;
  uint64_t next = 0, end = 0, local = 0, cnt = 0;
  uint32_t n = 0, s = 0;
  const uint64_t* selp = nullptr;
  uint64_t used = 0;
  int k = -1;
  bool have = false;
  // the next slot's record and first two level masks, loaded one pair ahead
  uint4 pr = make_uint4(0, 0, 0, 0);
  uint64_t pm0 = 0, pm1 = 0, plocal = 0;
  bool pre = false;
  auto fetch = [&]() {
    pre = false;
    if (next >= end) {
      if (join_stopped(lim)) return;
      const unsigned am = __activemask();
      const unsigned leader = __ffs(am) - 1;
      const unsigned rank = __popc(am & ((1u << lane) - 1u));
      unsigned long long b = 0;
      if (lane == leader) b = atomicAdd(cursor, static_cast<unsigned long long>(__popc(am)) * kChunk);
      b = __shfl_sync(am, b, leader);
      next = b + static_cast<uint64_t>(rank) * kChunk;
      end = next + kChunk < count ? next + kChunk : count;
      if (next >= count) return;
    }
    plocal = next++;
    pr = rec[plocal];
    pm0 = masks[plocal * kPhaseLevels];
    pm1 = masks[plocal * kPhaseLevels + 1];
    pre = true;
  };
  fetch();
  for (;;) {
    if (k < 0) {
      if (have) {
        if (find_first && cnt) cnt = 1;
        counts[slot0 + local] = cnt;
        my_total += cnt;
        have = false;
      }
      if (!pre) break;
      local = plocal;
      const uint4 r = pr;  // first data vertex, query size | flags, query offset, query graph
      const uint64_t m0 = pm0, m1 = pm1;
      fetch();
      if (r.y & 0xA00u) continue;  // the literal join's, or in the overflow list
      n = r.y & 0xFFu;
      s = r.x;
      selp = ((r.y & 0x100u) ? qsel_id : qsel) + r.z;
      AT(cand, 0) = m0;
      AT(base, 1) = m1;
      used = 0;
      cnt = 0;
      k = 0;
      have = true;
      continue;
    }
    const uint64_t ck = AT(cand, k);
    if (!ck) {
      --k;
      if (EXACT && k >= 0) used &= ~(1ull << AT(pk, k));
      if (budget_spent(lim, steps)) break;
      continue;
    }
    const uint32_t t = __ffsll(static_cast<long long>(ck)) - 1;
    AT(cand, k) = ck & (ck - 1);
    const uint64_t rw = dadj[static_cast<uint64_t>(s + t) * DAW];
    const uint64_t keep = 0ull - ((selp[k + 1] >> k) & 1ull);
    uint64_t nx = AT(base, k + 1) & ~(rw ^ keep);
    if (EXACT) nx &= ~(used | (1ull << t));
    if (static_cast<uint32_t>(k + 1) == n - 1) {
      cnt += __popcll(nx);
      if (find_first && cnt) k = -1;
      continue;
    }
    if (!nx) continue;
    AT(pk, k) = static_cast<uint8_t>(t);
    if (EXACT) used |= 1ull << t;
    AT(cand, k + 1) = nx;
    const uint64_t sl2 = selp[k + 2];
    uint64_t b2 = masks[local * kPhaseLevels + k + 2] & ~(rw ^ (0ull - ((sl2 >> k) & 1ull)));
    for (int i = 0; i < k; ++i) b2 &= ~(dadj[static_cast<uint64_t>(s + AT(pk, i)) * DAW] ^ (0ull - ((sl2 >> i) & 1ull)));
    AT(base, k + 2) = b2;
    ++k;
  }
#undef AT
  for (int o = 16; o; o >>= 1) my_total += __shfl_xor_sync(0xFFFFFFFFu, my_total, o);
  if (lane == 0 && my_total) atomicAdd(d_total, static_cast<unsigned long long>(my_total));
}

// Join phase B, default form (sigmo_tuning.join_kernel = 2): a per-lane DFS in
// which every turn is one candidate tried, by the same straight-line code, so
// the 32 lanes of a warp stay together whatever their pairs are doing.
//
// What makes turns differ is the test of a level against all earlier picks
// (one adjacency row per earlier level).  Here a lane keeps, for every vertex x
// of its molecule, the number of placed levels whose row holds x, counted to 3
// in two bit planes (b1 b0).  Level j with earlier neighbours S may take x
// exactly when x is in the rows of S and in no other, i.e. in the rows of S and
// counted |S| times; |S| is 1 or 2 at nearly every level of a molecular pattern
// (otherwise the rows are walked):
//     candidates = M[j] & row(S1) & row(S2) & (count == |S|)
// Each level keeps its untried candidates, the planes before its pick and its
// pick's row in shared memory, and a bit per level says where candidates are
// left, so a turn starts at the deepest such level whatever the turn before
// did: there are no separate moves back.  The last level is a popcount.
// Trying candidates from the highest vertex down needs no bit reversal.
//
// Bound by the latency of the chain level -> candidate -> row -> candidates of
// the next level at 15 warps per SM (ncu, 60,000 molecules x 600 queries, 4.0 M
// pairs: 56 % of the issue slots, 53 % of the integer pipe, 23 of 32 lanes per
// instruction); the state is kept per level in shared memory rather than
// recomputed because those loads use a pipe that is idle otherwise.  The form
// before this one walked the earlier rows and went back level by level: 7 of 32
// lanes per instruction, 6.2 ms for the pairs of 100,000 molecules x 600 queries
// where the short form takes 2.4 and the long one 0.6 beside it; the join stage of
// 10,007 ring systems x 100 automorphic queries went from 14.8 to 3.8 ms.
//
// A lane that ends its pair waits until `refill` lanes of its warp are idle, so
// the (divergent) setup of new pairs is shared by several lanes.  Work: each
// CTA first takes items from its own contiguous region of the chunk, so its
// lanes join neighbouring molecules whose adjacency rows stay in L1, then from
// a tail pool shared by all CTAs (pool16 sixteenths of the chunk).  An item is
// one of the 1 << lparts parts of a pair (every 2^lparts-th root candidate, and
// where the pair has fewer of them, of each a share of the next level's
// candidates): pairs are split when there are fewer of them than lanes.  (A star of
// five vertices in a star of 64, one root candidate: 73.7 ms by one lane, 4.8 so.)
//
// LV: most vertices of a query (LV - 1 levels of state per lane).  Pairs of
// longer queries are flagged and listed by k_pair_masks; with a list, the
// items are its entries.  Queries of up to kDfsLevels vertices are 93 % of the
// pairs and 97 % of the turns of the mixed query set, so the short form's
// lanes carry 402 B instead of 654.  Its CTAs have 160 threads so that three
// leave 60 KB of an SM to L1: with 192 (28 KB of L1) the rows fall out of it (an
// early state of this form: 5.9 instead of 4.8 ms).
// Loads of data that is read once, kept out of L1 (which holds the adjacency
// rows), and a hint that brings a later pair's data to L2.
__device__ __forceinline__ uint4 load_once(const uint4* p) {
  uint4 v;
  asm volatile("ld.global.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
struct Masks4 {
  uint64_t m[4];
};
__device__ __forceinline__ Masks4 load_once(const Masks4* p) {  // 32-byte aligned
  Masks4 v;
  asm volatile("ld.global.L1::no_allocate.v4.u64 {%0, %1, %2, %3}, [%4];" : "=l"(v.m[0]), "=l"(v.m[1]), "=l"(v.m[2]), "=l"(v.m[3]) : "l"(p));
  return v;
}
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

template <uint32_t LV>
constexpr uint32_t dfs_threads() { return LV <= kDfsLevels ? 160u : 96u; }
template <uint32_t LV>
constexpr size_t dfs_smem() { return dfs_threads<LV>() * (LV * 3 * 8 + (LV - 1) * (2 * 8 + 2)); }
constexpr uint32_t kDfsAhead = 256;  // slots ahead of the one taken that are brought to L2
constexpr uint32_t kRefillAll = 12, kRefillFirst = 20;

template <uint32_t LV, bool EXACT, uint32_t DAW>
__global__ void __launch_bounds__(dfs_threads<LV>()) k_join_dfs(
    const uint64_t* __restrict__ masks, const uint4* __restrict__ rec, uint64_t slot0, uint64_t count,
    const uint32_t* __restrict__ list, const unsigned long long* __restrict__ list_len, uint32_t lparts,
    const uint16_t* __restrict__ qmeta, const uint16_t* __restrict__ qmeta_id, const uint64_t* __restrict__ qsel,
    const uint64_t* __restrict__ qsel_id, const uint64_t* __restrict__ dadj, int find_first,
    uint32_t pool16, uint32_t refill, unsigned long long* __restrict__ cursor, uint64_t* __restrict__ counts,
    unsigned long long* __restrict__ d_total, JoinLimit lim) {
  extern __shared__ uint64_t sm[];
  __shared__ unsigned long long s_taken;  // items of this CTA's region handed out so far
  constexpr unsigned kAll = 0xFFFFFFFFu, T = dfs_threads<LV>(), D = LV - 1;
  const unsigned tid = threadIdx.x, lane = tid & 31u;
  uint64_t* rest = sm + tid;                        // [LV][T] untried candidates of each level
  uint64_t* p0 = sm + LV * T + tid;                 // [LV][T] planes before each level's pick (level 0: zero)
  uint64_t* p1 = sm + 2 * LV * T + tid;
  uint64_t* rows = sm + 3 * LV * T + tid;           // [LV - 1][T] row of each level's pick
  uint64_t* nextm = sm + (3 * LV + D) * T + tid;    // [LV - 1][T] mask of the level after
  uint16_t* meta = reinterpret_cast<uint16_t*>(sm + (3 * LV + 2 * D) * T) + tid;  // [LV - 1][T] query side of the level after
  if (list) count = *list_len;
  const uint64_t items = count << lparts;
  const uint64_t shared_items = items / 16u * (pool16 < 16u ? pool16 : 16u);
  const uint64_t rlen = (items - shared_items) / gridDim.x;
  const uint64_t pool0 = rlen * gridDim.x;
  const uint64_t r0 = static_cast<uint64_t>(blockIdx.x) * rlen;
  if (tid == 0) s_taken = 0;
  p0[0] = p1[0] = 0;
  __syncthreads();
  uint64_t steps = 0, my_total = 0, slot = 0, cnt = 0;
  uint32_t n = 0, qoff = 0;     // query size; query offset | identity-order flag << 31
  uint32_t alive = 0;           // levels with untried candidates
  const uint64_t* arow = dadj;  // adjacency rows of the lane's molecule
  const bool limited = lim.budget != 0;
  bool have = false, more = items != 0;  // more: the same for every lane of the warp
  for (;;) {
    const unsigned idle = __ballot_sync(kAll, alive == 0);
    const unsigned nidle = __popc(idle);
    if (nidle == 32u || (more && nidle >= refill)) {
      if (alive == 0 && have) {
        if (find_first && cnt) cnt = 1;
        if (lparts == 0) {
          counts[slot] = cnt;
          my_total += cnt;
        } else if (cnt) {  // counts[] zeroed by k_pair_masks
          auto* at = reinterpret_cast<unsigned long long*>(counts + slot);
          if (!find_first) atomicAdd(at, static_cast<unsigned long long>(cnt));
          if (!find_first || atomicExch(at, 1ull) == 0ull) my_total += cnt;
        }
        have = false;
      }
      if (more && __shfl_sync(kAll, join_stopped(lim) ? 1u : 0u, 0)) more = false;
      if (!more) {
        if (nidle == 32u) break;
      } else {
        unsigned long long rb = 0, pb = 0;
        if (lane == 0) {
          rb = atomicAdd(&s_taken, static_cast<unsigned long long>(nidle));
          const uint64_t in_region = rb < rlen ? (rlen - rb < nidle ? rlen - rb : nidle) : 0ull;
          if (nidle > in_region) pb = atomicAdd(cursor, static_cast<unsigned long long>(nidle - in_region));
        }
        rb = __shfl_sync(kAll, rb, 0);
        pb = __shfl_sync(kAll, pb, 0);
        const uint64_t in_region = rb < rlen ? (rlen - rb < nidle ? rlen - rb : nidle) : 0ull;
        if (nidle > in_region && pool0 + pb + (nidle - in_region) >= items) more = false;
        const unsigned rank = __popc(idle & ((1u << lane) - 1u));
        const uint64_t item = rank < in_region ? r0 + rb + rank : pool0 + pb + (rank - in_region);
        if (alive == 0 && item < items) {
          uint64_t local = item >> lparts;
          if (list) local = list[local] - slot0;
          const uint64_t ahead = local + kDfsAhead;
          if (!list && ahead < count) {
            prefetch_l2(masks + ahead * kPhaseLevels);
            prefetch_l2(rec + ahead);
          }
          const uint4 r = load_once(rec + local);  // first data vertex, query size | flags, query offset, query
          // else the literal join's, or another list's
          if (!(r.y & (0x800u | 0x200u)) && (LV > kDfsLevels || !(r.y & 0x400u))) {
            n = r.y & 0xFFu;
            slot = slot0 + local;
            const bool ident = (r.y & 0x100u) != 0u;
            qoff = r.z | (ident ? 0x80000000u : 0u);
            arow = dadj + static_cast<uint64_t>(r.x) * DAW;
            // all loads first, then the stores
            const Masks4* mp = reinterpret_cast<const Masks4*>(masks + local * kPhaseLevels);
            const uint4* qp = reinterpret_cast<const uint4*>((ident ? qmeta_id : qmeta) + static_cast<uint64_t>(r.w) * kPhaseLevels);
            constexpr uint32_t kQuads = (LV + 3) / 4;
            Masks4 mm[kQuads];
            uint32_t qm[8];  // two levels each
#pragma unroll
            for (uint32_t j = 0; j < kQuads; ++j)
              if (4 * j < n) mm[j] = load_once(mp + j);
            const uint4 qa = load_once(qp);
            uint4 qb = make_uint4(0, 0, 0, 0);
            if (n > 8) qb = load_once(qp + 1);
            qm[0] = qa.x, qm[1] = qa.y, qm[2] = qa.z, qm[3] = qa.w, qm[4] = qb.x, qm[5] = qb.y, qm[6] = qb.z, qm[7] = qb.w;
            uint64_t root = mm[0].m[0];
#pragma unroll
            for (uint32_t j = 1; j < LV; ++j)
              if (j < n) {
                nextm[(j - 1) * T] = mm[j / 4].m[j % 4];
                meta[(j - 1) * T] = static_cast<uint16_t>(qm[j / 2] >> (16u * (j % 2)));
              }
            if (lparts) {  // this part's root candidates, and where they are fewer than the parts its share of the next level's
              const uint32_t part = static_cast<uint32_t>(item) & ((1u << lparts) - 1u), c0 = __popcll(root);
              const uint32_t by_root = c0 > 1u ? min(lparts, 32u - __clz(c0 - 1u)) : 0u;  // log2
              root = share_of(root, part & ((1u << by_root) - 1u), by_root);
              if (by_root < lparts) nextm[0] = share_of(mm[0].m[1], part >> by_root, lparts - by_root);
            }
            rest[0] = root;
            alive = root ? 1u : 0u;
            cnt = 0;
            have = true;
          }
        }
      }
    }
    if (alive == 0) continue;
    // try the highest untried candidate t of the deepest level k that has one
    const uint32_t k = 31u - __clz(alive);
    uint64_t rem = rest[k * T];
    const uint32_t hi = static_cast<uint32_t>(rem >> 32);
    const uint32_t t = (31u - __clz(hi ? hi : static_cast<uint32_t>(rem))) + (hi ? 32u : 0u);
    const uint64_t r = arow[t * DAW];
    const uint64_t bit = 1ull << t;
    rem ^= bit;
    rest[k * T] = rem;
    const uint64_t b0 = p0[k * T], b1 = p1[k * T];
    uint64_t f = nextm[k * T];
    const uint32_t q = meta[k * T];  // level k + 1's earlier neighbours i1, i2 (4 bits each), bit 8: two of them, bit 9: none or more than two
    if (EXACT) meta[k * T] = static_cast<uint16_t>((q & 0x3FFu) | (t << 10));
    uint64_t n0 = (b0 ^ r) | (b1 & b0), n1 = b1 | (b0 & r);  // count + 1 where r holds the vertex, at most 3
    if (EXACT) {  // a placed vertex is never a candidate again
      n0 |= bit;
      n1 |= bit;
    }
    rows[k * T] = r;
    if (!(q & 0x200u)) {
      const uint64_t two = 0ull - static_cast<uint64_t>((q >> 8) & 1u);
      f &= rows[(q & 15u) * T] & rows[((q >> 4) & 15u) * T];
      f &= (n0 ^ two) & ~(n1 ^ two);
    } else {
      const uint64_t sel = ((qoff >> 31) ? qsel_id : qsel)[(qoff & 0x7FFFFFFFu) + k + 1u];
      if (sel == 0) {
        f &= ~(n0 | n1);
      } else {
        for (uint32_t i = 0; i <= k; ++i) {
          f &= ~(rows[i * T] ^ (0ull - ((sel >> i) & 1ull)));
          if (EXACT) f &= ~(1ull << (meta[i * T] >> 10));
        }
      }
    }
    const bool last = k + 2u == n;
    // level k + 1's state, used when it has candidates (of the last level: never)
    rest[(k + 1u) * T] = f;
    p0[(k + 1u) * T] = n0;
    p1[(k + 1u) * T] = n1;
    alive ^= (rem ? 0u : 1u << k) | (f && !last ? 2u << k : 0u);
    const uint32_t found = last ? __popcll(f) : 0u;  // every candidate of the last level is a match
    cnt += found;
    if (find_first && found) alive = 0;
    if (limited && !rem && budget_spent(lim, steps)) {
      have = false;  // the count is incomplete
      alive = 0;
    }
  }
  for (int o = 16; o; o >>= 1) my_total += __shfl_xor_sync(kAll, my_total, o);
  if (lane == 0 && my_total) atomicAdd(d_total, static_cast<unsigned long long>(my_total));
}

// Phase B, warp-cooperative form (k_join_frontier).  A warp keeps up to 32
// pairs in flight (slot p: its root candidates, count and live-entry count).
// A partial embedding of depth L >= 1 is an entry {candidates left at level
// L; meta = pair | vertex placed at level L-1 << 5 | parent entry << 11} in a
// per-warp pool where each level's entries form one region, stacked in level
// order.  A round takes the next 32 (entry, candidate) items of the current
// level L, one per lane: the lane rebuilds the level-(L+1) constraint by
// walking the parent chain, tries its candidate (the same test as the
// per-lane machine) and appends the child entry at level L+1, or adds the
// popcount when L+1 is the last level.  The warp goes one level deeper once
// the next level holds a full round (levels above kFrontDeep: any entry), and
// back up when the current level is used up, so a level holds at most 63
// entries (31 above kFrontDeep) and the pool is bounded by kFrontPool.
// Counts are order-independent sums, so they equal the per-lane machine's.
constexpr uint32_t kFrontPairs = 32;
constexpr uint32_t kFrontDeep = 4;
constexpr uint32_t kFrontPool = kFrontDeep * 63u + (kPhaseLevels - 2u - kFrontDeep) * 32u;
constexpr uint32_t kFrontWarps = 8;
constexpr uint32_t kFrontFree = 0xFFFFFFFFu;
struct FrontWarp {
  unsigned long long pcnt[kFrontPairs];  // embeddings found per pair slot
  uint64_t pcand[kFrontPairs];           // level-0 candidates not yet taken
  uint64_t ecand[kFrontPool];
  uint32_t emeta[kFrontPool];
  // per pair slot: first data vertex of the graph, query offset | identity-order
  // flag << 31, chunk-local slot (kFrontFree when the slot is free), query size
  uint4 pinfo[kFrontPairs];
  uint32_t pref[kFrontPairs];  // live entries (root included)
  uint16_t head[kPhaseLevels + 1], tail[kPhaseLevels + 1];
};

template <bool EXACT, uint32_t DAW>
__global__ void __launch_bounds__(kFrontWarps * 32, 3) k_join_frontier(
    const uint64_t* __restrict__ masks, const uint4* __restrict__ rec, uint64_t slot0, uint64_t count,
    const uint64_t* __restrict__ qsel, const uint64_t* __restrict__ qsel_id, const uint64_t* __restrict__ dadj,
    int find_first, uint32_t kChunk, unsigned long long* __restrict__ cursor,
    uint64_t* __restrict__ counts, unsigned long long* __restrict__ d_total, JoinLimit lim) {
  extern __shared__ __align__(16) unsigned char front_raw[];
  uint64_t rounds = 0;
  FrontWarp& w = reinterpret_cast<FrontWarp*>(front_raw)[threadIdx.x >> 5];
  const unsigned lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
  constexpr unsigned kAll = 0xFFFFFFFFu;
  w.pinfo[lane].z = kFrontFree;
  w.pcand[lane] = 0;
  w.pref[lane] = 0;
  if (lane <= kPhaseLevels) w.head[lane] = w.tail[lane] = 0;
  __syncwarp();
  uint64_t next = 0, end = 0;  // warp-uniform range of chunk-local slots
  bool more = true;
  uint64_t my_total = 0;
  uint32_t L = 0;
  for (;;) {
    // the budget counts this warp's rounds (warp-uniform)
    if (lim.budget && ++rounds > lim.budget) {
      if (lane == 0) atomicOr(lim.status, kJoinStatusBudget);
      break;
    }
    if (L == 0 && more) {
      // fill the free pair slots (lane i owns slot i) from the work range
      bool fr = w.pinfo[lane].z == kFrontFree;
      unsigned F = __ballot_sync(kAll, fr);
      while (F && more) {
        if (next >= end) {
          if (__shfl_sync(kAll, join_stopped(lim) ? 1u : 0u, 0)) {
            more = false;
            break;
          }
          unsigned long long b = 0;
          if (lane == 0) b = atomicAdd(cursor, 32ull * kChunk);
          b = __shfl_sync(kAll, b, 0);
          next = b;
          end = b + 32ull * kChunk < count ? b + 32ull * kChunk : count;
          if (next >= count) {
            more = false;
            break;
          }
        }
        const uint32_t avail = static_cast<uint32_t>(end - next < 32 ? end - next : 32);
        const uint32_t take = min(static_cast<uint32_t>(__popc(F)), avail);
        const uint32_t rank = __popc(F & lt);
        if (fr && rank < take) {
          const uint64_t local = next + rank;
          const uint4 r = rec[local];  // first data vertex, query size | flags, query offset, query graph
          if (!(r.y & 0xA00u)) {
            const uint64_t c0 = masks[local * kPhaseLevels];
            if (c0) {
              w.pinfo[lane] = make_uint4(r.x, r.z | ((r.y & 0x100u) ? 0x80000000u : 0u), static_cast<uint32_t>(local), r.y & 0xFFu);
              w.pcand[lane] = c0;
              w.pcnt[lane] = 0;
              w.pref[lane] = 1;
              fr = false;
            } else {
              counts[slot0 + local] = 0;  // no candidate for the first query vertex
            }
          }
        }
        next += take;
        F = __ballot_sync(kAll, fr);
      }
      __syncwarp();
    }
    // ---- one round at level L: this lane's source entry (L = 0: pair slot)
    const uint32_t head = w.head[L], tail = w.tail[L];
    uint64_t cand;
    if (L == 0) cand = w.pcand[lane];
    else cand = head + lane < tail ? w.ecand[head + lane] : 0ull;
    const uint32_t c = __popcll(cand);
    uint32_t incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(kAll, incl, o);
      if (lane >= static_cast<unsigned>(o)) incl += y;
    }
    const uint32_t excl = incl - c;
    const uint32_t total = __shfl_sync(kAll, incl, 31);
    if (total) {
      const uint32_t nitems = total < 32u ? total : 32u;
      // the owner of item `lane`: the first source lane whose inclusive
      // count exceeds it (binary search over the non-decreasing counts)
      uint32_t o = 0;
#pragma unroll
      for (uint32_t step = 16; step; step >>= 1) {
        const uint32_t v = __shfl_sync(kAll, incl, o + step - 1u);
        if (v <= lane) o += step;
      }
      o = o < 31u ? o : 31u;
      const uint32_t oexcl = __shfl_sync(kAll, excl, o), oincl = __shfl_sync(kAll, incl, o);
      const uint64_t ocand = __shfl_sync(kAll, cand, o);
      const bool item = lane < nitems;
      bool child = false, exhausted = false;
      uint64_t nx = 0;
      uint32_t p = 0, t = 0;
      if (item) {
        t = nth_set64(ocand, lane - oexcl);
        const bool last_of_owner = lane + 1u == (oincl < nitems ? oincl : nitems);
        uint32_t meta = 0;
        if (L == 0) {
          p = o;
        } else {
          meta = w.emeta[head + o];
          p = meta & 31u;
        }
        if (last_of_owner) {  // the owner's candidates up to t are taken
          const uint64_t left = ocand & ~((2ull << t) - 1ull);
          if (L == 0) w.pcand[o] = left;
          else w.ecand[head + o] = left;
          exhausted = left == 0;
        }
        const uint4 pi = w.pinfo[p];
        const uint32_t s = pi.x, sv = pi.y, local = pi.z, n = pi.w;
        const uint64_t* selp = ((sv >> 31) ? qsel_id : qsel) + (sv & 0x7FFFFFFFu);
        const uint64_t sl = selp[L + 1];
        uint64_t b = masks[static_cast<uint64_t>(local) * kPhaseLevels + L + 1u];
        uint64_t used = 0;
        if (L) {  // constraints of the vertices placed at levels L-1 .. 0
          uint32_t m = meta;
          for (int i = static_cast<int>(L) - 1;; --i) {
            const uint32_t ti = (m >> 5) & 63u;
            b &= ~(dadj[static_cast<uint64_t>(s + ti) * DAW] ^ (0ull - ((sl >> i) & 1ull)));
            if (EXACT) used |= 1ull << ti;
            if (i == 0) break;
            m = w.emeta[m >> 11];
          }
        }
        const uint64_t rw = dadj[static_cast<uint64_t>(s + t) * DAW];
        nx = b & ~(rw ^ (0ull - ((sl >> L) & 1ull)));
        if (EXACT) nx &= ~(used | (1ull << t));
        if (!(find_first && w.pcnt[p])) {
          if (L + 1u == n - 1u) {
            if (nx) atomicAdd(&w.pcnt[p], static_cast<unsigned long long>(__popcll(nx)));
          } else {
            child = nx != 0;
          }
        }
      }
      // children at level L + 1, in lane order
      const unsigned cb = __ballot_sync(kAll, child);
      const uint32_t at = w.tail[L + 1];
      if (child) {
        const uint32_t pos = at + __popc(cb & lt);
        if (pos < kFrontPool) {  // always true: the level bounds above sum to kFrontPool
          w.ecand[pos] = nx;
          w.emeta[pos] = p | (t << 5) | ((L ? head + o : 0u) << 11);
          atomicAdd(&w.pref[p], 1u);
        }
      }
      __syncwarp();
      if (lane == 0 && cb) {
        const uint32_t nt = min(at + static_cast<uint32_t>(__popc(cb)), kFrontPool);
        w.tail[L + 1] = static_cast<uint16_t>(nt);
        w.head[L + 2] = w.tail[L + 2] = static_cast<uint16_t>(nt);  // level L+2 is empty
      }
      // entries used up in this round release their pair; the last one ends it
      if (exhausted && atomicSub(&w.pref[p], 1u) == 1u) {
        unsigned long long cn = w.pcnt[p];
        if (find_first && cn) cn = 1;
        counts[slot0 + w.pinfo[p].z] = cn;
        my_total += cn;
        w.pinfo[p].z = kFrontFree;
      }
      if (L) {  // the used-up entries are a prefix of the level
        const unsigned gone = __ballot_sync(kAll, incl <= 32u);
        const uint32_t lead = gone == kAll ? 32u : static_cast<uint32_t>(__ffs(~gone) - 1);
        if (lane == 0) w.head[L] = static_cast<uint16_t>(head + lead < tail ? head + lead : tail);
      }
      __syncwarp();
    }
    // ---- next level (warp-uniform)
    const bool left = L ? w.head[L] < w.tail[L] : __any_sync(kAll, w.pcand[lane] != 0);
    const uint32_t waiting = w.tail[L + 1] - w.head[L + 1];
    const uint32_t thr = L + 1u <= kFrontDeep ? 32u : 1u;
    if (waiting && (waiting >= thr || !left)) {
      ++L;
      continue;
    }
    if (!left) {
      if (L) {
        const uint16_t start = L == 1 ? 0 : w.tail[L - 1];
        __syncwarp();
        if (lane == 0) w.head[L] = w.tail[L] = w.head[L + 1] = w.tail[L + 1] = start;
        __syncwarp();
        --L;
      } else if (!more) {
        break;  // no pair in flight and no work left
      }
    }
  }
  for (int o = 16; o; o >>= 1) my_total += __shfl_xor_sync(0xFFFFFFFFu, my_total, o);
  if (lane == 0 && my_total) atomicAdd(d_total, static_cast<unsigned long long>(my_total));
}

}  // namespace

int launch_join_literal(Queue* q, const Graph* query, const Graph* data, const MaskSource& src, Gmcr* m, int find_first,
                        uint32_t graph_begin, uint32_t graph_end, uint64_t* d_total, uint32_t q_begin, uint32_t q_end) {
  if (graph_end <= graph_begin) return SIGMO_OK;
  if (query->max_nodes > kMaxQueryNodes)
    return fail(SIGMO_ERR_DOMAIN, "query graphs of up to %u vertices are supported (largest: %u)", kMaxQueryNodes, query->max_nodes);
  if (q->opts.profile == kProfileExact)
    return fail(SIGMO_ERR_DOMAIN, "exact profile supports data graphs of at most %u vertices", 64u * kMaxAdjWords);
  const uint32_t wg = q->opts.join_work_group_size ? q->opts.join_work_group_size : 128u;
  if (wg > 1024u || (wg & 31u)) return fail(SIGMO_ERR_INVALID, "join work-group size %u must be a multiple of 32 <= 1024", wg);
  SIGMO_TRY(launch_query_order(const_cast<Graph*>(query)));
  const uint32_t graphs = graph_end - graph_begin;
  auto* tot = reinterpret_cast<unsigned long long*>(d_total);
  uint32_t range_max = data->max_nodes;
  if (range_max > 64u) {
    range_max = 0;
    for (uint32_t g = graph_begin; g < graph_end; ++g)
      range_max = std::max(range_max, data->host_graph_offsets[g + 1] - data->host_graph_offsets[g]);
  }
  // one word per set where the range's graphs allow it; its state is in shared
  // memory up to kLitLevels levels
  const bool one = range_max <= 64u;
  const uint32_t levels = query->max_nodes;
  const bool smem_fits = one && levels <= kLitLevels;
  // few graphs (those below vertex 256): the smallest blocks; else small ones where
  // a block's threads share the masks, and a block per graph where they do not
  const uint32_t block = graphs <= kLowOffsetLimit ? kLitItems : smem_fits ? kLitItemsMany : wg;
  const uint64_t want = static_cast<uint64_t>(graphs) * ((wg + block - 1u) / block);
  if (one || (q->opts.profile == kProfilePtx && range_max <= 64u * kMaxAdjWords)) {
    const size_t smem = smem_fits ? kLitBytesPerLevel * levels * block : 0;
    auto kern = smem_fits ? k_join_literal_sets<1, true>
                : one     ? k_join_literal_sets<1, false>
                : data->adj_words == 2 ? k_join_literal_sets<2, false>
                                       : k_join_literal_sets<4, false>;
    if (smem) SIGMO_TRY(allow_max_dynamic_smem(reinterpret_cast<const void*>(kern), q->device));
    kern<<<grid_for(want, 1, 148u * 64u), smem_fits ? std::max(block, 32u) : block, smem, q->stream>>>(
        src, q->opts.profile, query->graph_offsets, query->qsel_id, data->graph_offsets, data->adj, data->adj_words, m->offsets,
        m->indices, graph_begin, graph_end, wg, block, levels, q_begin, q_end, find_first, m->counts, tot, join_limit(q));
    return check_launch(q, "k_join_literal_sets");
  }
  if (!src.bits) return fail(SIGMO_ERR_INVALID, "internal: the literal join of graphs over %u vertices reads the bitset", 64u * kMaxAdjWords);
  k_join_literal<<<std::min<uint32_t>(graphs, 148u * 64u), wg, 0, q->stream>>>(src.bits, src.Wp, q->opts.profile, query->graph_offsets, query->adj,
                                             data->graph_offsets, data->adj, data->adj_words, data->row_offsets,
                                             data->column_indices, m->offsets, m->indices, graph_begin, graph_end, q_begin,
                                             q_end, find_first, m->counts, tot, join_limit(q));
  return check_launch(q, "k_join_literal");
}

int launch_join_wildcard(Queue* q, const Graph* query, const Graph* data, const Candidates* c, Gmcr* m, int find_first,
                         uint64_t* d_total) {
  if (query->max_nodes > kMaxQueryNodes)
    return fail(SIGMO_ERR_DOMAIN, "query graphs of up to %u vertices are supported (largest: %u)", kMaxQueryNodes, query->max_nodes);
  const bool exact = q->opts.profile == kProfileExact;
  if (exact && data->max_nodes > 64u * kMaxAdjWords)
    return fail(SIGMO_ERR_DOMAIN, "exact profile supports data graphs of at most %u vertices", 64u * kMaxAdjWords);
  const uint32_t wg = q->opts.join_work_group_size ? q->opts.join_work_group_size : 128u;
  if (wg > 1024u || (wg & 31u)) return fail(SIGMO_ERR_INVALID, "join work-group size %u must be a multiple of 32 <= 1024", wg);
  const uint32_t G = data->num_graphs;
  if (!G || !m->total) return SIGMO_OK;
  auto* tot = reinterpret_cast<unsigned long long*>(d_total);
  MaskSource src;
  src.bits = c->bits;
  src.Wp = c->Wp;
  src.prof = q->opts.profile;
  BondGraphs bg;
  bg.qadj = query->adj;
  bg.qroff = query->row_offsets;
  bg.qcol = query->column_indices;
  bg.qel = query->edge_labels;
  bg.droff = data->row_offsets;
  bg.dcol = data->column_indices;
  bg.del = data->edge_labels;
  bg.doffsets = m->offsets;
  bg.total_slots = m->total;
  // graphs [0, literal): step by step, on the side stream; the others in any order
  uint32_t literal = G;
  const bool sets = data->max_nodes <= 64u * kMaxAdjWords;
  if (sets) {
    SIGMO_TRY(launch_query_order(const_cast<Graph*>(query)));  // before the fork: both streams read it
    literal = 0;
    while (!exact && literal < G && data->host_graph_offsets[literal] < kLowOffsetLimit) ++literal;
  }
  if (literal) {
    if (cudaEventRecord(q->ev_fork, q->stream) != cudaSuccess || cudaStreamWaitEvent(q->side, q->ev_fork, 0) != cudaSuccess)
      return fail(SIGMO_ERR_CUDA, "stream fork failed");
    const unsigned grid = std::min<uint32_t>(literal, 148u * 64u);
    const size_t smem = wildcard_smem(data->adj_words, query->max_nodes);
    if (sets) {
      auto kern = data->adj_words == 1 ? k_join_wildcard_sets<1> : data->adj_words == 2 ? k_join_wildcard_sets<2> : k_join_wildcard_sets<4>;
      SIGMO_TRY(allow_max_dynamic_smem(reinterpret_cast<const void*>(kern), q->device));
      kern<<<grid_for(static_cast<uint64_t>(literal) * (wg / 32u), 1, 148u * 64u), 32, smem, q->side>>>(
          src, bg, query->graph_offsets, query->qsel_id, data->graph_offsets, data->adj, m->indices, literal, wg / 32u,
          query->max_nodes, find_first, m->counts, tot);
    } else {
      k_join_wildcard<<<grid, wg, 0, q->side>>>(c->bits, c->Wp, q->opts.profile, query->graph_offsets, query->adj, query->row_offsets,
                                   query->column_indices, query->edge_labels, data->graph_offsets, data->adj, data->adj_words,
                                   data->row_offsets, data->column_indices, data->edge_labels, m->offsets, m->indices, literal,
                                   find_first, m->counts, tot);
    }
    SIGMO_TRY(check_launch(q, "k_join_wildcard"));
  }
  int rc = SIGMO_OK;
  if (literal < G) {
    void* cursor = nullptr;
    rc = tmp_alloc(q, &cursor, 8);
    if (!rc && cudaMemsetAsync(cursor, 0, 8, q->stream) != cudaSuccess) rc = fail(SIGMO_ERR_CUDA, "memset failed");
    bg.first_graph = literal;
    const uint32_t aw = data->adj_words, stride = query->max_nodes * aw;
    const uint32_t batch = std::max(1u, std::min<uint32_t>(kWideBatch, static_cast<uint32_t>(kWideMaskBytes / (8ull * stride))));
    const size_t smem = wide_smem(batch, aw, stride);
    auto kern = aw == 1   ? (exact ? k_join_wide<1, true, true> : k_join_wide<1, false, true>)
                : aw == 2 ? (exact ? k_join_wide<2, true, true> : k_join_wide<2, false, true>)
                          : (exact ? k_join_wide<4, true, true> : k_join_wide<4, false, true>);
    if (!rc) rc = allow_max_dynamic_smem(reinterpret_cast<const void*>(kern), q->device);
    if (!rc) {
      kern<<<grid_for(m->total, kWideWarps * batch, q->tune.overflow_blocks), kWideWarps * 32, smem, q->stream>>>(
          src, bg, query->graph_offsets, query->qorder, query->qsel_id, query->qsel_id, query->sym, data->graph_offsets, data->adj,
          data->sym, m->indices, m->pair_graph, nullptr, nullptr, batch, stride, find_first,
          static_cast<unsigned long long*>(cursor), m->counts, tot, JoinLimit{0, q->d_status});
      rc = check_launch(q, "k_join_wide<bonds>");
    }
    dev_free(q, cursor);
  }
  if (literal && (cudaEventRecord(q->ev_join, q->side) != cudaSuccess || cudaStreamWaitEvent(q->stream, q->ev_join, 0) != cudaSuccess))
    rc = rc ? rc : fail(SIGMO_ERR_CUDA, "stream join failed");
  return rc;
}

namespace {

// Device memory of the pair join for `slots` slots.
struct PairScratch {
  void *buf = nullptr, *mbuf[2] = {nullptr, nullptr};
  uint64_t chunk = 0;  // slots per mask buffer
  bool two = false;    // several chunks: two mask buffers
  bool has_long = false, has_overflow = false;
  size_t lists = 0;    // counters, overflow list, long-pair lists
  size_t masks = 0;    // one mask buffer
};
PairScratch pair_scratch(const sigmo_tuning& tn, uint32_t query_nodes, uint32_t data_nodes, uint64_t slots) {
  PairScratch p;
  p.chunk = std::min<uint64_t>(slots, static_cast<uint64_t>(tn.mask_chunk_slots) << 20);
  p.two = slots > p.chunk;
  p.has_long = tn.join_kernel == 2 && query_nodes > kDfsLevels;
  p.has_overflow = query_nodes > kPhaseLevels || data_nodes > 64u;
  p.lists = 256 + (p.has_overflow ? 4ull * slots : 0) + (p.has_long ? 4ull * p.chunk * (p.two ? 2 : 1) : 0);
  p.masks = 8ull * kPhaseLevels * p.chunk + 16ull * p.chunk;
  return p;
}

int alloc_scratch(Queue* q, PairScratch* p) {
  int rc = tmp_alloc(q, &p->buf, p->lists);
  if (!rc) rc = tmp_alloc(q, &p->mbuf[0], p->masks);
  if (!rc && p->two) rc = tmp_alloc(q, &p->mbuf[1], p->masks);
  if (rc) {
    dev_free(q, p->mbuf[0]);
    dev_free(q, p->buf);
  }
  return rc;
}

// The pairs in slots [first, first + slots); frees the scratch.
int join_slots(Queue* q, const Graph* query, const Graph* data, const MaskSource& src, Gmcr* m, int find_first, uint32_t skip,
               uint64_t* d_total, uint64_t first, uint64_t slots, const PairScratch& sc) {
  const bool exact = q->opts.profile == kProfileExact;
  const sigmo_tuning& tn = q->tune;
  void *buf = sc.buf, *mbuf[2] = {sc.mbuf[0], sc.mbuf[1]};
  const uint64_t chunk = sc.chunk;
  // several chunks: even ones on the main stream, odd ones on the aux stream,
  // each stream with its own mask buffer and work cursor, so one chunk's level
  // masks run beside the previous chunk's persistent join
  const bool two = sc.two, has_long = sc.has_long, has_overflow = sc.has_overflow;
  // [0] work cursor of the even chunks, [1] generic-join cursor, [2] overflow
  // length, [3] odd chunks' cursor; then per chunk parity the long pairs'
  // list length [4 + 2 i] and cursor [5 + 2 i]
  auto* ctr = static_cast<unsigned long long*>(buf);
  uint32_t* overflow = reinterpret_cast<uint32_t*>(static_cast<char*>(buf) + 256);
  uint32_t* longs = has_long ? overflow + (has_overflow ? slots : 0) : nullptr;  // [two ? 2 : 1][chunk]
  int rc = cudaMemsetAsync(ctr, 0, 256, q->stream) == cudaSuccess ? SIGMO_OK : fail(SIGMO_ERR_CUDA, "memset failed");
  auto* tot = reinterpret_cast<unsigned long long*>(d_total);
  // two-phase join, in chunks of slots, for the pairs of queries of <= 16
  // vertices and molecules of <= 64 atoms; the rest go to the overflow list
  const bool frontier = tn.join_kernel == 1, dfs = tn.join_kernel == 2;
  // the long pairs run beside the short ones
  const cudaStream_t long_stream = two ? q->side : q->aux;
  {
    const cudaStream_t streams[2] = {q->stream, q->aux};
    if (!rc && two &&
        (cudaEventRecord(q->ev_aux_fork, q->stream) != cudaSuccess || cudaStreamWaitEvent(q->aux, q->ev_aux_fork, 0) != cudaSuccess))
      rc = fail(SIGMO_ERR_CUDA, "stream fork failed");
    // the kernels for this batch's adjacency-row width and profile
    const size_t smem = frontier ? sizeof(FrontWarp) * kFrontWarps
                        : dfs    ? dfs_smem<kDfsLevels>()
                                 : static_cast<size_t>(kPhaseLevels) * kPhaseThreads * (2 * 8 + 1);
    const unsigned block = frontier ? kFrontWarps * 32u : dfs ? dfs_threads<kDfsLevels>() : kPhaseThreads;
    void (*join_kernel)(const uint64_t*, const uint4*, uint64_t, uint64_t, const uint64_t*, const uint64_t*, const uint64_t*,
                        int, uint32_t, unsigned long long*, uint64_t*, unsigned long long*, JoinLimit) = nullptr;
    using DfsKernel = void (*)(const uint64_t*, const uint4*, uint64_t, uint64_t, const uint32_t*, const unsigned long long*,
                               uint32_t, const uint16_t*, const uint16_t*, const uint64_t*, const uint64_t*, const uint64_t*,
                               int, uint32_t, uint32_t, unsigned long long*, uint64_t*, unsigned long long*, JoinLimit);
    DfsKernel dfs_short = nullptr, dfs_long = nullptr;
#define SIGMO_PICK_JOIN(AWV)                                                                                     \
  dfs_short = exact ? k_join_dfs<kDfsLevels, true, AWV> : k_join_dfs<kDfsLevels, false, AWV>;                    \
  dfs_long = exact ? k_join_dfs<kPhaseLevels, true, AWV> : k_join_dfs<kPhaseLevels, false, AWV>;                 \
  join_kernel = frontier ? (exact ? k_join_frontier<true, AWV> : k_join_frontier<false, AWV>)                   \
                         : (exact ? k_join_masks<true, AWV> : k_join_masks<false, AWV>)
    switch (data->adj_words) {
      case 1: SIGMO_PICK_JOIN(1); break;
      case 2: SIGMO_PICK_JOIN(2); break;
      default: SIGMO_PICK_JOIN(4); break;
    }
#undef SIGMO_PICK_JOIN
    if (!rc)
      rc = allow_max_dynamic_smem(dfs ? reinterpret_cast<const void*>(dfs_short) : reinterpret_cast<const void*>(join_kernel), q->device);
    if (!rc && has_long) rc = allow_max_dynamic_smem(reinterpret_cast<const void*>(dfs_long), q->device);
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, q->device);
    // persistent CTAs; every join kernel keeps at most three resident (a fourth
    // of k_join_dfs would start its region only when another CTA has ended)
    const unsigned grid = static_cast<unsigned>(sms) * (dfs ? std::min(tn.join_blocks_per_sm, 3u) : tn.join_blocks_per_sm);
    // fewer pairs than lanes: every pair in up to 16 parts by root candidate
    uint32_t lparts = 0;
    while (dfs && lparts < 4 && (slots << (lparts + 1)) <= static_cast<uint64_t>(grid) * block) ++lparts;
    const uint32_t long_parts = find_first ? lparts : std::max(lparts, 1u);
    uint64_t c = 0;
    for (uint64_t slot0 = first; slot0 < first + slots && !rc; slot0 += chunk, ++c) {
      const uint64_t cnt = std::min<uint64_t>(chunk, first + slots - slot0);
      const uint32_t par = c & 1;
      const cudaStream_t st = streams[par];
      auto* masks = static_cast<uint64_t*>(mbuf[par]);
      auto* recs = reinterpret_cast<uint4*>(masks + kPhaseLevels * chunk);
      unsigned long long* cursor = ctr + (par ? 3 : 0);
      unsigned long long* lctr = ctr + 4 + 2 * par;
      uint32_t* llist = has_long ? longs + par * chunk : nullptr;
      if (c >= 2 && (cudaMemsetAsync(cursor, 0, 8, st) != cudaSuccess || cudaMemsetAsync(lctr, 0, 16, st) != cudaSuccess))
        rc = fail(SIGMO_ERR_CUDA, "memset failed");
      if (rc) break;
      (src.planes ? k_pair_masks<true> : k_pair_masks<false>)<<<grid_for(cnt, 256, 148u * 16u), 256, 0, st>>>(
          src, data->adj_words, query->graph_offsets, query->qorder, query->sym,
          data->graph_offsets, data->sym, m->indices, m->pair_graph, slot0, cnt, masks, recs, skip, overflow, ctr + 2, llist,
          lctr, m->counts, lparts != 0);
      rc = check_launch(q, "k_pair_masks");
      if (!rc && cudaEventRecord(q->ev_masks[par], st) != cudaSuccess) rc = fail(SIGMO_ERR_CUDA, "event record failed");
      if (!rc) {
        if (dfs)
          dfs_short<<<grid, block, smem, st>>>(masks, recs, slot0, cnt, nullptr, nullptr, lparts, query->qmeta, query->qmeta_id,
                                               query->qsel, query->qsel_id, data->adj, find_first, tn.join_pool,
                                               find_first ? kRefillFirst : kRefillAll, cursor, m->counts, tot, join_limit(q));
        else  // join_chunk slots per grab
          join_kernel<<<grid, block, smem, st>>>(masks, recs, slot0, cnt, query->qsel, query->qsel_id, data->adj, find_first,
                                                 tn.join_chunk, cursor, m->counts, tot, join_limit(q));
        rc = check_launch(q, frontier ? "k_join_frontier" : dfs ? "k_join_dfs" : "k_join_masks");
      }
      // the long pairs after the short ones: their CTAs take the room that the
      // persistent CTAs of the short form leave as they end
      if (!rc && has_long) {
        const unsigned lblock = dfs_threads<kPhaseLevels>();
        if (cudaStreamWaitEvent(long_stream, q->ev_masks[par], 0) != cudaSuccess) rc = fail(SIGMO_ERR_CUDA, "stream fork failed");
        if (!rc) {
          dfs_long<<<3u * static_cast<unsigned>(sms), lblock, dfs_smem<kPhaseLevels>(), long_stream>>>(
              masks, recs, slot0, cnt, llist, lctr, long_parts, query->qmeta, query->qmeta_id, query->qsel,
              query->qsel_id, data->adj, find_first, 8u, find_first ? kRefillFirst : kRefillAll, lctr + 1, m->counts, tot, join_limit(q));
          rc = check_launch(q, "k_join_dfs<long>");
        }
        if (!rc && cudaEventRecord(q->ev_long[par], long_stream) != cudaSuccess) rc = fail(SIGMO_ERR_CUDA, "event record failed");
      }
      // the chunk's buffers are free again once its long pairs are joined too
      if (has_long && cudaStreamWaitEvent(st, q->ev_long[par], 0) != cudaSuccess) rc = rc ? rc : fail(SIGMO_ERR_CUDA, "stream join failed");
    }
    // the aux stream joins the main one before its buffer is released
    if (two && (cudaEventRecord(q->ev_aux_join, q->aux) != cudaSuccess ||
                cudaStreamWaitEvent(q->stream, q->ev_aux_join, 0) != cudaSuccess))
      rc = rc ? rc : fail(SIGMO_ERR_CUDA, "stream join failed");
    dev_free(q, mbuf[0]);
    dev_free(q, mbuf[1]);
  }
  const cudaStream_t main_stream = q->stream;
  const bool side = has_overflow && !q->tune.overflow_serial;
  if (!rc && side) {
    // the overflow list is complete after the last Phase A of each stream: its
    // pairs run on the side stream, overlapping Phase B
    if (cudaStreamWaitEvent(q->side, q->ev_masks[0], 0) != cudaSuccess ||
        (two && cudaStreamWaitEvent(q->side, q->ev_masks[1], 0) != cudaSuccess))
      rc = fail(SIGMO_ERR_CUDA, "stream fork failed");
    q->stream = q->side;
  }
  if (!rc && has_overflow) {
    // the overflow list; a warp's batch is as large as its masks' shared memory allows
    const uint32_t aw = data->adj_words, stride = query->max_nodes * aw;
    const uint32_t batch = std::max(1u, std::min<uint32_t>(kWideBatch, static_cast<uint32_t>(kWideMaskBytes / (8ull * stride))));
    const size_t smem = wide_smem(batch, aw, stride);
    auto kern = aw == 1   ? (exact ? k_join_wide<1, true, false> : k_join_wide<1, false, false>)
                : aw == 2 ? (exact ? k_join_wide<2, true, false> : k_join_wide<2, false, false>)
                          : (exact ? k_join_wide<4, true, false> : k_join_wide<4, false, false>);
    rc = allow_max_dynamic_smem(reinterpret_cast<const void*>(kern), q->device);
    if (!rc) {
      kern<<<q->tune.overflow_blocks, kWideWarps * 32, smem, q->stream>>>(
          src, BondGraphs{}, query->graph_offsets, query->qorder, query->qsel, query->qsel_id, query->sym, data->graph_offsets,
          data->adj, data->sym, m->indices, m->pair_graph, overflow, ctr + 2, batch, stride, find_first, ctr + 1, m->counts, tot,
          join_limit(q));
      rc = check_launch(q, "k_join_wide");
    }
  }
  q->stream = main_stream;
  if (side && cudaEventRecord(q->ev_join, q->side) == cudaSuccess) cudaStreamWaitEvent(q->stream, q->ev_join, 0);
  dev_free(q, buf);
  return rc;
}

// Smallest number of slots that the pair join is cut down to: 0.6 MB of masks.
constexpr uint64_t kMinJoinSlots = 4096;

}  // namespace

uint64_t join_pairs_bytes(const Queue* q, const Graph* query, const Graph* data, uint64_t slots) {
  const PairScratch sc = pair_scratch(q->tune, query->max_nodes, data->max_nodes, slots);
  return sc.lists + sc.masks * (sc.two ? 2 : 1);
}

// All slots at once; where the device memory does not allow that, runs of half
// as many one after the other, and so on.
int launch_join_pairs(Queue* q, const Graph* query, const Graph* data, const MaskSource& src, Gmcr* m, int find_first, uint32_t skip,
                      uint64_t* d_total) {
  if (!m->total) return SIGMO_OK;
  if (query->max_nodes > kMaxQueryNodes)
    return fail(SIGMO_ERR_DOMAIN, "query graphs of up to %u vertices are supported (largest: %u)", kMaxQueryNodes, query->max_nodes);
  SIGMO_TRY(launch_query_order(const_cast<Graph*>(query)));
  uint64_t run = m->total;
  for (uint64_t first = 0; first < m->total;) {
    const uint64_t slots = std::min(run, m->total - first);
    PairScratch sc = pair_scratch(q->tune, query->max_nodes, data->max_nodes, slots);
    const int rc = alloc_scratch(q, &sc);
    if (rc == SIGMO_ERR_OOM && slots > kMinJoinSlots) {
      run = std::max((slots + 1) / 2, kMinJoinSlots);
      continue;
    }
    SIGMO_TRY(rc);
    SIGMO_TRY(join_slots(q, query, data, src, m, find_first, skip, d_total, first, slots, sc));
    first += slots;
  }
  return SIGMO_OK;
}

int launch_join(Queue* q, const Graph* query, const Graph* data, const MaskSource& src, Gmcr* m, int find_first, uint32_t literal,
                uint64_t* d_total, const uint32_t* ranges, uint32_t nranges) {
  if (!m->total) return SIGMO_OK;
  SIGMO_TRY(launch_query_order(const_cast<Graph*>(query)));  // before the fork: both streams read it
  int rc = SIGMO_OK;
  if (literal) {
    if (cudaEventRecord(q->ev_fork, q->stream) != cudaSuccess || cudaStreamWaitEvent(q->side, q->ev_fork, 0) != cudaSuccess)
      return fail(SIGMO_ERR_CUDA, "stream fork failed");
    const cudaStream_t main_stream = q->stream;
    q->stream = q->side;
    if (!ranges || nranges == 0)
      rc = launch_join_literal(q, query, data, src, m, find_first, 0, literal, d_total, 0, 0xFFFFFFFFu);
    for (uint32_t r = 0; ranges && r < nranges && !rc; ++r)
      rc = launch_join_literal(q, query, data, src, m, find_first, 0, literal, d_total, ranges[r], ranges[r + 1]);
    q->stream = main_stream;
  }
  if (!rc && literal < data->num_graphs) rc = launch_join_pairs(q, query, data, src, m, find_first, literal, d_total);
  // join the side stream back (only when this call forked it: a CUDA-graph
  // capture may wait only on events of streams that joined the capture)
  if (literal && (cudaEventRecord(q->ev_join, q->side) != cudaSuccess || cudaStreamWaitEvent(q->stream, q->ev_join, 0) != cudaSuccess))
    rc = rc ? rc : fail(SIGMO_ERR_CUDA, "stream join failed");
  return rc;
}

}  // namespace sigmo_b200
