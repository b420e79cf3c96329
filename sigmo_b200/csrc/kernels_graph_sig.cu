// Graph-derived device structures and the signature kernels.
//
// Signatures follow Signature<PowerGraph,4> (library/include/signature.hpp):
// generateCSRSignatures (:125-152) and refineCSRSignatures<PowerGraph>
// (:336-390).  The refinement is a bounded BFS per vertex; here each graph's
// local adjacency is kept as one bit row per vertex (u64 words, local ids), so
// a BFS level is an OR of rows selected by the frontier's bits.
#include <cuda_runtime.h>

#include "bulk.cuh"
#include "internal.hpp"

namespace sigmo_b200 {
namespace {

// What is derived of a batch at its creation, a thread per vertex, in one launch:
//   node_graph  the vertex's graph,
//   adj         its local adjacency row: bit t of row v = (prev + t) appears in
//               v's CSR row, for local ids t < 64 * AW (prev = first vertex of
//               v's graph),
//   sym         (ones before the launch) cleared when a row is not mirrored, or
//               the graph has more than 64 * AW vertices.
// A block takes 256 consecutive vertices: one warp finds the graph of the first
// (32 probes per step), their graphs' offsets go to shared memory, and a vertex
// finds its own there.  An edge's reverse is looked up in the neighbour's CSR
// row, so nothing waits for the adjacency rows.  (Three kernels before, the
// graph-per-thread ones with a serial chain per graph: 121 us for 100,000
// molecules, 45 us for the two uploads of a small search; this one 67 and 11.)
//
// Looking an edge's reverse up costs the neighbour's degree, so a block with a
// vertex of more than kDeriveDegree entries tests bits instead: it stages the
// rows of all graphs that its vertices belong to (those of the first and the last
// one that lie outside its range are built a second time) and a vertex looks its
// own bit up in each neighbour's row.  Creation of 2,000 complete graphs of 256
// vertices 8.4 -> 1.0 ms, 10,000 of 64 0.85 -> 0.16, 50,000 of 16 0.20 -> 0.14,
// of 80,000 of 10 vertices 0.19 and 0.18 ms; molecules have no such vertex.
constexpr uint32_t kDeriveRange = 256, kDeriveDegree = 8;

// The local adjacency row of a vertex, CSR entries [i0, i1), of the graph
// [prev, prev + n), into shared memory.
template <int AW>
__device__ __forceinline__ void stage_row(uint32_t i0, uint32_t i1, uint32_t prev, uint32_t n, const uint32_t* __restrict__ col,
                                          uint64_t* row) {
#pragma unroll
  for (int k = 0; k < AW; ++k) row[k] = 0;
  if (n > 64u * AW) n = 64u * AW;
  for (uint32_t i = i0; i < i1; ++i) {
    const uint32_t t = col[i] - prev;  // neighbours outside the graph set no bit
    if (t < n) row[t >> 6] |= 1ull << (t & 63u);
  }
}

template <int AW>
__global__ void __launch_bounds__(kDeriveRange) k_graph_derive(uint64_t N, uint32_t G, const uint32_t* __restrict__ goff,
                                                               const uint32_t* __restrict__ roff,
                                                               const uint32_t* __restrict__ col,
                                                               uint32_t* __restrict__ node_graph, uint64_t* __restrict__ adj,
                                                               uint8_t* __restrict__ sym) {
  constexpr uint32_t kMax = 64u * AW;  // vertices of a graph whose rows are complete
  __shared__ uint32_t s_off[kDeriveRange + 1];
  __shared__ uint32_t s_first;
  __shared__ uint32_t s_lo, s_hi, s_last;  // staged vertices [s_lo, s_hi); first vertex of the last one's graph
  __shared__ uint64_t s_rows[kDeriveRange + 2 * kMax][AW];
  for (uint64_t v0 = static_cast<uint64_t>(blockIdx.x) * kDeriveRange; v0 < N; v0 += static_cast<uint64_t>(gridDim.x) * kDeriveRange) {
    if (threadIdx.x < 32) {  // the last graph that starts at or before v0: in [lo, hi)
      uint32_t lo = 0, hi = G;
      while (hi - lo > 1) {
        const uint32_t step = (hi - lo + 31u) / 32u;
        const uint64_t probe = lo + static_cast<uint64_t>(threadIdx.x) * step;
        const bool le = probe < hi && goff[probe] <= v0;  // monotone over the lanes; lane 0 holds lo
        const uint32_t last = 31u - __clz(__ballot_sync(0xFFFFFFFFu, le) | 1u);
        lo += last * step;
        hi = lo + step < hi ? lo + step : hi;
      }
      if (threadIdx.x == 0) s_first = lo;
    }
    __syncthreads();
    const uint32_t first = s_first, have = G - first < kDeriveRange ? G - first : kDeriveRange;  // graphs staged
    for (uint32_t i = threadIdx.x; i <= have; i += blockDim.x) s_off[i] = goff[first + i];
    __syncthreads();
    const uint64_t v = v0 + threadIdx.x, v1 = v0 + kDeriveRange < N ? v0 + kDeriveRange : N;
    uint32_t g = 0, prev = 0, end = 0, i0 = 0, i1 = 0;
    if (v < N) {
      if (s_off[have] > v) {
        uint32_t lo = 0, hi = have;  // the last staged graph that starts at or before v
        while (hi - lo > 1) {
          const uint32_t mid = (lo + hi) >> 1;
          if (s_off[mid] <= v) lo = mid;
          else hi = mid;
        }
        g = first + lo;
        prev = s_off[lo];
        end = s_off[lo + 1];
      } else {  // past the staged graphs (many empty ones)
        uint32_t lo = first + have, hi = G;
        while (hi - lo > 1) {
          const uint32_t mid = lo + (hi - lo) / 2;
          if (goff[mid] <= v) lo = mid;
          else hi = mid;
        }
        g = lo;
        prev = goff[g];
        end = goff[g + 1];
      }
      i0 = roff[v];
      i1 = roff[v + 1];
    }
    const uint32_t n = end - prev;
    bool mirrored = n <= kMax && static_cast<uint32_t>(v) - prev < n && end <= N;
    if (__syncthreads_or(i1 - i0 > kDeriveDegree)) {
      if (v == v0) s_lo = mirrored ? prev : static_cast<uint32_t>(v0);
      if (v + 1 == v1) {
        s_hi = mirrored ? end : static_cast<uint32_t>(v1);
        s_last = prev;
      }
      __syncthreads();
      const uint32_t lo = s_lo, before = static_cast<uint32_t>(v0) - lo, after = s_hi - static_cast<uint32_t>(v1);
      uint64_t* mine = s_rows[before + threadIdx.x];
      if (v < N) stage_row<AW>(i0, i1, prev, n, col, mine);
      // the vertices outside the range: of its first graph and of its last one
      // (bits past a graph's end are not read)
      for (uint32_t i = threadIdx.x; i < before + after; i += blockDim.x) {
        const uint32_t u = i < before ? lo + i : static_cast<uint32_t>(v1) + (i - before);
        stage_row<AW>(roff[u], roff[u + 1], i < before ? lo : s_last, kMax, col, s_rows[u - lo]);
      }
      __syncthreads();
      if (v < N) {
#pragma unroll
        for (int k = 0; k < AW; ++k) {
          const uint64_t bits = mine[k];
          adj[v * AW + k] = bits;
          for (uint64_t m = bits; m && mirrored; m &= m - 1) {
            const uint32_t at = prev + 64u * k + __ffsll(static_cast<long long>(m)) - 1u - lo, me = static_cast<uint32_t>(v) - prev;
            mirrored = at < s_hi - lo && ((s_rows[at][me >> 6] >> (me & 63u)) & 1ull);
          }
        }
      }
    } else if (v < N) {
      uint64_t row[AW];
#pragma unroll
      for (int k = 0; k < AW; ++k) row[k] = 0;
      for (uint32_t i = i0; i < i1; ++i) {
        const uint32_t t = col[i] - prev;  // neighbours outside the graph set no bit
        if (t >= n || t >= kMax) continue;
        const uint64_t bit = 1ull << (t & 63u);
#pragma unroll
        for (int k = 0; k < AW; ++k) row[k] |= (t >> 6) == static_cast<uint32_t>(k) ? bit : 0ull;
        if (mirrored) {
          const uint32_t j1 = roff[prev + t + 1];
          bool back = false;
          for (uint32_t j = roff[prev + t]; j < j1 && !back; ++j) back = col[j] == v;
          mirrored = back;
        }
      }
#pragma unroll
      for (int k = 0; k < AW; ++k) adj[v * AW + k] = row[k];
    }
    if (v < N) {
      node_graph[v] = g;
      if (!mirrored) sym[g] = 0;
    }
    __syncthreads();  // the offsets are no longer read
  }
}

// generateCSRSignatures (signature.hpp:136-146): +1 per neighbour label, on
// top of the current value.
__global__ void k_sig_generate(uint64_t N, const uint32_t* __restrict__ roff, const uint32_t* __restrict__ col,
                               const uint8_t* __restrict__ lab, uint64_t* __restrict__ sig) {
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < N; v += (uint64_t)gridDim.x * blockDim.x) {
    uint64_t s = sig[v];
    for (uint32_t i = roff[v]; i < roff[v + 1]; ++i) s = sig_inc(s, lab[col[i]]);
    sig[v] = s;
  }
}

// REF_PTX BFS for graphs of more than 256 vertices: the reference's bitset
// truncates local ids to uint8_t, so vertex t occupies bit (t & 255) when that
// is < 64 and no bit otherwise; bit b is expanded through vertex prev + b.
__device__ uint64_t ptx_wide_ball(uint32_t v, uint32_t prev, uint32_t view, const uint32_t* __restrict__ roff,
                                  const uint32_t* __restrict__ col, uint64_t* self_bit) {
  const uint64_t self = refbit(v - prev, 0);
  uint64_t F = self, R = self;
  for (uint32_t it = 0; it < view && F; ++it) {
    uint64_t nx = 0, m = F;
    while (m) {
      const uint32_t b = __ffsll(static_cast<long long>(m)) - 1;
      m &= m - 1;
      const uint32_t u = prev + b;
      for (uint32_t i = roff[u]; i < roff[u + 1]; ++i) nx |= refbit(col[i] - prev, 0);
    }
    nx &= ~R;
    R |= nx;
    F = nx;
  }
  *self_bit = self;
  return R;
}

// refineCSRSignatures<PowerGraph> (signature.hpp:348-386), REF_PTX profile:
// sphere = ball_view(v) \ {v} \ old(v); sig = label histogram of the sphere;
// old |= sphere.  Local ids >= 64 have no bit (graph sizes <= 256).
// X86 (REF_X86, graphs of <= 256 vertices): the 64-bit sets take local id
// mod 64 (Bitset<uint64_t> with the shift count modulo 64), so a vertex's
// neighbours land on their ids mod 64 (its adjacency words ORed together),
// and the frontier's bit b expands vertex b of the graph.
template <bool X86>
__global__ void k_sig_refine_ptx(uint64_t N, const uint32_t* __restrict__ goff, const uint32_t* __restrict__ node_graph,
                                 const uint64_t* __restrict__ adj, uint32_t AW, const uint32_t* __restrict__ roff,
                                 const uint32_t* __restrict__ col, const uint8_t* __restrict__ lab, uint32_t view,
                                 uint64_t* __restrict__ sig, uint64_t* __restrict__ reach) {
  for (uint64_t vv = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; vv < N; vv += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t v = static_cast<uint32_t>(vv);
    const uint32_t g = node_graph[v];
    const uint32_t prev = goff[g], n = goff[g + 1] - prev;
    uint64_t self, R;
    if (!X86 && n > 256u) {
      R = ptx_wide_ball(v, prev, view, roff, col, &self);
    } else {
      const uint32_t lv = v - prev;
      self = X86 ? (1ull << (lv & 63u)) : (lv < 64u ? (1ull << lv) : 0ull);
      uint64_t F = self;
      R = self;
      for (uint32_t it = 0; it < view && F; ++it) {
        uint64_t nx = 0, m = F;
        while (m) {
          const uint32_t b = __ffsll(static_cast<long long>(m)) - 1;
          m &= m - 1;
          const uint64_t* row = adj + static_cast<uint64_t>(prev + b) * AW;
          if (X86) {
            for (uint32_t k = 0; k < AW; ++k) nx |= row[k];
          } else {
            nx |= row[0];
          }
        }
        nx &= ~R;
        R |= nx;
        F = nx;
      }
    }
    R &= ~self;
    const uint64_t old = reach[v];
    uint64_t sphere = R & ~old;
    const uint64_t keep = sphere;
    uint64_t s = 0;
    while (sphere) {
      const uint32_t b = __ffsll(static_cast<long long>(sphere)) - 1;
      sphere &= sphere - 1;
      s = sig_inc(s, lab[prev + b]);
    }
    sig[v] = s;
    reach[v] = keep | old;
  }
}

// EXACT profile: true local sets of up to 64*AW vertices.
template <int AW>
__global__ void k_sig_refine_exact(uint64_t N, const uint32_t* __restrict__ goff, const uint32_t* __restrict__ node_graph,
                                   const uint64_t* __restrict__ adj, const uint8_t* __restrict__ lab, uint32_t view,
                                   uint64_t* __restrict__ sig, uint64_t* __restrict__ reach) {
  for (uint64_t vv = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; vv < N; vv += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t v = static_cast<uint32_t>(vv);
    const uint32_t prev = goff[node_graph[v]];
    const uint32_t lv = v - prev;
    uint64_t F[AW], R[AW];
#pragma unroll
    for (int k = 0; k < AW; ++k) F[k] = R[k] = ((lv >> 6) == (uint32_t)k) ? (1ull << (lv & 63u)) : 0ull;
    for (uint32_t it = 0; it < view; ++it) {
      bool any = false;
#pragma unroll
      for (int k = 0; k < AW; ++k) any |= F[k] != 0;
      if (!any) break;
      uint64_t nx[AW];
#pragma unroll
      for (int k = 0; k < AW; ++k) nx[k] = 0;
#pragma unroll
      for (int w = 0; w < AW; ++w) {
        uint64_t m = F[w];
        while (m) {
          const uint32_t b = __ffsll(static_cast<long long>(m)) - 1 + 64u * w;
          m &= m - 1;
          const uint64_t* row = adj + static_cast<uint64_t>(prev + b) * AW;
#pragma unroll
          for (int k = 0; k < AW; ++k) nx[k] |= row[k];
        }
      }
#pragma unroll
      for (int k = 0; k < AW; ++k) {
        nx[k] &= ~R[k];
        R[k] |= nx[k];
        F[k] = nx[k];
      }
    }
    uint64_t s = 0;
#pragma unroll
    for (int k = 0; k < AW; ++k) {
      if ((lv >> 6) == (uint32_t)k) R[k] &= ~(1ull << (lv & 63u));
      uint64_t* old = reach + static_cast<uint64_t>(v) * kMaxAdjWords + k;
      uint64_t sphere = R[k] & ~*old;
      *old |= R[k];
      while (sphere) {
        const uint32_t b = __ffsll(static_cast<long long>(sphere)) - 1;
        sphere &= sphere - 1;
        s = sig_inc(s, lab[prev + 64u * k + b]);
      }
    }
    sig[v] = s;
  }
}

// All refinement iterations 1..R at once (batched form): starting from empty
// reachables, iteration r's sphere is exactly BFS level r, so one BFS to
// depth R emits every iteration's signature.  sig_all is [R][N].
//
// Each CTA's graphs are staged on chip.  A CTA takes 256 consecutive
// vertices; they belong to a run of whole graphs whose adjacency rows
// [row_lo, row_hi) (at most 256 + 128 * AW rows for graphs of up to 64 * AW
// vertices) arrive in shared memory by one bulk asynchronous copy (the TMA
// engine, cp.async.bulk, completion counted on an mbarrier), and whose labels
// arrive by plain loads meanwhile; every vertex's BFS then reads shared memory
// only.  The copy starts on a 16-byte boundary of the adjacency array, is a
// multiple of 16 bytes and ends inside the array (a last 8-byte row past the
// final 16-byte boundary is loaded by a thread).  A range whose graphs do not
// fit (wide graphs) reads global memory instead.  The mbarrier
// wait is bounded; past the bound the range is computed from global memory
// (results are the same either way) and the CTA stops staging.
constexpr uint32_t kSigRange = 256;
template <int AW, bool EXACT>
__global__ void __launch_bounds__(kSigRange) k_sig_all_staged(uint64_t N, const uint32_t* __restrict__ goff,
                                                              const uint32_t* __restrict__ node_graph,
                                                              const uint64_t* __restrict__ adj,
                                                              const uint32_t* __restrict__ roff,
                                                              const uint32_t* __restrict__ col,
                                                              const uint8_t* __restrict__ lab, uint32_t Rn,
                                                              uint64_t* __restrict__ sig_all) {
  constexpr uint32_t kCap = kSigRange + 128u * AW;         // rows of one range's graphs, at most
  __shared__ __align__(16) uint64_t s_rows[kCap * AW + 2];  // + 16 bytes: the copy may start one row early
  __shared__ uint8_t s_lab[kCap];
  __shared__ __align__(8) uint64_t s_bar;
  __shared__ int s_ok;  // the CTA still stages (no wait has run out)
  const uint64_t adj_bytes = N * AW * 8ull;
  if (threadIdx.x == 0) {
    mbar_init(&s_bar, 1);
    s_ok = 1;
  }
  __syncthreads();
  uint32_t parity = 0;
  for (uint64_t v0 = static_cast<uint64_t>(blockIdx.x) * kSigRange; v0 < N; v0 += static_cast<uint64_t>(gridDim.x) * kSigRange) {
    const uint64_t v1 = v0 + kSigRange < N ? v0 + kSigRange : N;
    const uint32_t row_lo = goff[node_graph[v0]], row_hi = goff[node_graph[v1 - 1] + 1];
    const bool stage = s_ok && row_hi - row_lo <= kCap;  // the same for every thread
    __syncthreads();  // the previous range's rows and labels are no longer read
    uint32_t extra = 0;  // words copied before row_lo (the copy starts on a 16-byte boundary)
    if (stage) {
      const uint64_t b_lo = static_cast<uint64_t>(row_lo) * AW * 8, b_hi = static_cast<uint64_t>(row_hi) * AW * 8;
      const uint64_t a_lo = b_lo & ~15ull;
      const uint64_t a_hi = (b_hi + 15) & ~15ull;
      const uint64_t c_hi = a_hi <= adj_bytes ? a_hi : (b_hi & ~15ull);  // the copy ends inside the array
      extra = static_cast<uint32_t>((b_lo - a_lo) / 8);
      if (threadIdx.x == 0) {
        if (c_hi > a_lo) {
          mbar_expect_tx(&s_bar, static_cast<uint32_t>(c_hi - a_lo));
          bulk_copy_g2s(s_rows, reinterpret_cast<const char*>(adj) + a_lo, static_cast<uint32_t>(c_hi - a_lo), &s_bar);
        } else {
          mbar_expect_tx(&s_bar, 0);  // completes the phase with nothing in flight
        }
      }
      if (threadIdx.x == 32 && c_hi < b_hi) {  // the last 8-byte row past the final 16-byte boundary
        s_rows[(c_hi - a_lo) / 8] = adj[(c_hi) / 8];
        // order this generic store before any later bulk copy into the buffer
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
      }
      for (uint32_t i = threadIdx.x; i < row_hi - row_lo; i += blockDim.x) s_lab[i] = lab[row_lo + i];
      if (!mbar_wait(&s_bar, parity)) s_ok = 0;
      parity ^= 1u;
    }
    __syncthreads();  // labels and the tail row are in; s_ok is settled
    const bool use_smem = stage && s_ok;
    const uint64_t vv = v0 + threadIdx.x;
    if (vv >= v1) continue;
    const uint32_t v = static_cast<uint32_t>(vv);
    const uint32_t prev = goff[node_graph[v]];
    const uint32_t n = goff[node_graph[v] + 1] - prev;
    const uint32_t lv = v - prev;
    // rows and labels of this vertex's graph: shared memory or global memory
    const uint64_t* grow = use_smem ? s_rows + extra + static_cast<uint64_t>(prev - row_lo) * AW : adj + static_cast<uint64_t>(prev) * AW;
    const uint8_t* glab = use_smem ? s_lab + (prev - row_lo) : lab + prev;
    uint64_t F[AW], R[AW];
    const bool wide = !EXACT && n > 256u;
#pragma unroll
    for (int k = 0; k < AW; ++k) F[k] = 0;
    if (EXACT) {
#pragma unroll
      for (int k = 0; k < AW; ++k) F[k] = ((lv >> 6) == (uint32_t)k) ? (1ull << (lv & 63u)) : 0ull;
    } else {
      F[0] = wide ? refbit(lv, 0) : (lv < 64u ? (1ull << lv) : 0ull);
    }
#pragma unroll
    for (int k = 0; k < AW; ++k) R[k] = F[k];
    // One walk over a level's vertices expands it and counts its labels (its
    // signature is written then); the last level is only counted.  Issue-bound:
    // a walk each for expanding and counting took 0.36 ms for 100,000 molecules
    // of 10-60 atoms and six levels, this 0.29 ms.
    for (uint32_t r = 0; r <= Rn; ++r) {
      uint64_t nx[AW];
#pragma unroll
      for (int k = 0; k < AW; ++k) nx[k] = 0;
      uint64_t sg = 0;
      const bool expand = r < Rn;
      if (EXACT) {
#pragma unroll
        for (int w = 0; w < AW; ++w) {
          uint64_t m = F[w];
          while (m) {
            const uint32_t b = __ffsll(static_cast<long long>(m)) - 1 + 64u * w;
            m &= m - 1;
            sg = sig_inc(sg, glab[b]);
            if (expand) {
              const uint64_t* row = grow + static_cast<uint64_t>(b) * AW;
#pragma unroll
              for (int k = 0; k < AW; ++k) nx[k] |= row[k];
            }
          }
        }
      } else {
        uint64_t m = F[0];
        while (m) {
          const uint32_t b = __ffsll(static_cast<long long>(m)) - 1;
          m &= m - 1;
          sg = sig_inc(sg, glab[b]);
          if (wide) {
            const uint32_t u = prev + b;
            for (uint32_t i = roff[u]; expand && i < roff[u + 1]; ++i) nx[0] |= refbit(col[i] - prev, 0);
          } else if (expand) {
            nx[0] |= grow[static_cast<uint64_t>(b) * AW];
          }
        }
      }
      if (r) sig_all[static_cast<uint64_t>(r - 1) * N + v] = sg;  // level 0 is the vertex itself
#pragma unroll
      for (int k = 0; k < AW; ++k) {
        nx[k] &= ~R[k];
        R[k] |= nx[k];
        F[k] = nx[k];
        if (!EXACT) break;
      }
    }
  }
  // a copy whose wait ran out may still be in flight: wait again (bounded)
  // before the CTA's shared memory is released
  __syncthreads();
  if (!s_ok) mbar_wait(&s_bar, parity ^ 1u);
}

// Matching order per query graph (batched join): start at the vertex of
// highest degree, then repeatedly take the vertex with the most neighbours
// already placed (ties: higher degree, lower id).  qorder[off + k] = local id
// placed at level k; qsel[off + k] = levels i < k adjacent to level k in that
// order; qsel_id[off + k] = the same for the identity order (used when a graph
// has an asymmetric adjacency, which only self-loops produce).  sym[g] = 1 if
// every adjacency row of graph g is mirrored.
//
// A warp per query: lane l holds the rows of vertices l and l + 32, a level's
// vertex is one warp maximum over (placed neighbours, degree, lower id), and
// the level sets are built from the rows of the placed vertices by shuffles,
// level k by lane k.  (One thread per query took 93 us for 600 queries of up
// to 30 vertices, a serial walk over global memory; this takes
// 7 us.)
__device__ __forceinline__ uint64_t shfl_row(uint64_t lo, uint64_t hi, uint32_t u) {
  const uint64_t a = __shfl_sync(0xFFFFFFFFu, lo, u & 31u), b = __shfl_sync(0xFFFFFFFFu, hi, u & 31u);
  return u < 32u ? a : b;
}

// A level's set in the packed form of Graph::qmeta.
__device__ __forceinline__ uint16_t pack_level(uint64_t sel) {
  const uint32_t s = static_cast<uint32_t>(sel), cnt = __popc(s);
  const uint32_t a = s ? __ffs(s) - 1 : 0u, rest = s & (s - 1), b = rest ? __ffs(rest) - 1 : a;
  return static_cast<uint16_t>(a | (b << 4) | (cnt == 2u ? 0x100u : 0u) | (cnt == 0u || cnt > 2u ? 0x200u : 0u));
}

__global__ void k_query_order(uint32_t QG, const uint32_t* __restrict__ goff, const uint64_t* __restrict__ adj,
                              uint8_t* __restrict__ qorder, uint64_t* __restrict__ qsel, uint64_t* __restrict__ qsel_id,
                              uint16_t* __restrict__ qmeta, uint16_t* __restrict__ qmeta_id) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t warp = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), nwarps = gridDim.x * (blockDim.x >> 5);
  for (uint32_t q = warp; q < QG; q += nwarps) {
    const uint32_t off = goff[q], n = goff[q + 1] - off;
    if (n > kMaxQueryNodes) continue;
    const uint64_t r0 = lane < n ? adj[off + lane] : 0ull, r1 = lane + 32u < n ? adj[off + lane + 32u] : 0ull;
    uint64_t placed = 0;
    uint32_t ord0 = 0, ord1 = 0;  // vertices placed at levels lane and lane + 32
    for (uint32_t k = 0; k < n; ++k) {
      uint32_t best = 0;  // conn : 8, degree : 8, 63 - id : 8 bits, + 1
      if (lane < n && !((placed >> lane) & 1ull))
        best = ((static_cast<uint32_t>(__popcll(r0 & placed)) << 16) | (static_cast<uint32_t>(__popcll(r0)) << 8) | (63u - lane)) + 1u;
      if (lane + 32u < n && !((placed >> (lane + 32u)) & 1ull)) {
        const uint32_t x = ((static_cast<uint32_t>(__popcll(r1 & placed)) << 16) | (static_cast<uint32_t>(__popcll(r1)) << 8) | (31u - lane)) + 1u;
        best = x > best ? x : best;
      }
      const uint32_t v = 63u - ((__reduce_max_sync(0xFFFFFFFFu, best) - 1u) & 0xFFu);
      if (lane == (k & 31u)) (k < 32u ? ord0 : ord1) = v;
      placed |= 1ull << v;
    }
    uint64_t sel0 = 0, sel1 = 0, id0 = 0, id1 = 0;  // levels lane and lane + 32
    for (uint32_t i = 0; i < n; ++i) {
      const uint32_t a = __shfl_sync(0xFFFFFFFFu, ord0, i & 31u), b = __shfl_sync(0xFFFFFFFFu, ord1, i & 31u);
      const uint64_t row = shfl_row(r0, r1, i < 32u ? a : b), row_id = shfl_row(r0, r1, i);
      if (i < lane) {
        sel0 |= ((row >> ord0) & 1ull) << i;
        id0 |= ((row_id >> lane) & 1ull) << i;
      }
      if (i < lane + 32u) {
        sel1 |= ((row >> ord1) & 1ull) << i;
        id1 |= ((row_id >> (lane + 32u)) & 1ull) << i;
      }
    }
    if (lane < n) {
      qorder[off + lane] = static_cast<uint8_t>(ord0);
      qsel[off + lane] = sel0;
      qsel_id[off + lane] = id0;
    }
    if (lane + 32u < n) {
      qorder[off + lane + 32u] = static_cast<uint8_t>(ord1);
      qsel[off + lane + 32u] = sel1;
      qsel_id[off + lane + 32u] = id1;
    }
    if (n <= 16u && lane < 16u) {
      qmeta[16ull * q + lane] = pack_level(sel0);
      qmeta_id[16ull * q + lane] = pack_level(id0);
    }
  }
}

}  // namespace

int launch_graph_derive(Graph* g) {
  Queue* q = g->q;
  // words per local adjacency row: 1, 2 or 4 (the kernels are instantiated
  // for those widths; a batch whose largest graph has 129-192 vertices gets 4)
  const uint32_t mx = g->max_nodes;
  uint32_t aw = 1;
  while (aw < kMaxAdjWords && aw * 64u < mx) aw *= 2;
  g->adj_words = aw;
  const uint64_t adj_elems = g->total_nodes * aw;
  if (g->total_nodes) SIGMO_TRY(dev_alloc(q, reinterpret_cast<void**>(&g->node_graph), sizeof(uint32_t) * g->total_nodes));
  SIGMO_TRY(dev_alloc(q, reinterpret_cast<void**>(&g->adj), sizeof(uint64_t) * (adj_elems ? adj_elems : 1)));
  SIGMO_TRY(dev_alloc(q, reinterpret_cast<void**>(&g->sym), g->num_graphs ? g->num_graphs : 1));
  if (g->num_graphs) SIGMO_CUDA_TRY(cudaMemsetAsync(g->sym, 1, g->num_graphs, q->stream));
  if (g->total_nodes) {
    auto kern = aw == 1 ? k_graph_derive<1> : aw == 2 ? k_graph_derive<2> : k_graph_derive<4>;
    kern<<<grid_for(g->total_nodes, kDeriveRange, 148u * 32u), kDeriveRange, 0, q->stream>>>(
        g->total_nodes, g->num_graphs, g->graph_offsets, g->row_offsets, g->column_indices, g->node_graph, g->adj, g->sym);
    SIGMO_TRY(check_launch(q, "k_graph_derive"));
  }
  return SIGMO_OK;
}

int launch_query_order(Graph* g) {
  Queue* q = g->q;
  if (g->qorder) return SIGMO_OK;
  // the graph takes the arrays once all of them are there and filled: a call
  // that ran short of memory is made again as if it had not been made
  const uint64_t N = g->total_nodes ? g->total_nodes : 1, G = g->num_graphs ? g->num_graphs : 1;
  void* p[5] = {nullptr, nullptr, nullptr, nullptr, nullptr};  // qorder, qsel, qsel_id, qmeta, qmeta_id
  const uint64_t bytes[5] = {N, 8 * N, 8 * N, 32 * G, 32 * G};
  int rc = SIGMO_OK;
  for (int i = 0; i < 5 && !rc; ++i) rc = dev_alloc(q, &p[i], bytes[i]);
  if (!rc && g->num_graphs && g->adj_words == 1) {
    k_query_order<<<grid_for(32ull * g->num_graphs, 128, 4096u), 128, 0, q->stream>>>(
        g->num_graphs, g->graph_offsets, g->adj, static_cast<uint8_t*>(p[0]), static_cast<uint64_t*>(p[1]),
        static_cast<uint64_t*>(p[2]), static_cast<uint16_t*>(p[3]), static_cast<uint16_t*>(p[4]));
    rc = check_launch(q, "k_query_order");
  }
  if (rc) {
    for (void* x : p) dev_free(q, x);
    return rc;
  }
  g->qorder = static_cast<uint8_t*>(p[0]);
  g->qsel = static_cast<uint64_t*>(p[1]);
  g->qsel_id = static_cast<uint64_t*>(p[2]);
  g->qmeta = static_cast<uint16_t*>(p[3]);
  g->qmeta_id = static_cast<uint16_t*>(p[4]);
  return SIGMO_OK;
}

int launch_sig_generate(Queue* q, const Graph* g, uint64_t* sig) {
  if (!g->total_nodes) return SIGMO_OK;
  k_sig_generate<<<grid_for(g->total_nodes, 256, 148u * 32u), 256, 0, q->stream>>>(g->total_nodes, g->row_offsets,
                                                                                   g->column_indices, g->node_labels, sig);
  return check_launch(q, "k_sig_generate");
}

int launch_sig_refine(Queue* q, const Graph* g, uint32_t view, uint64_t* sig, uint64_t* reach, uint32_t reach_words) {
  if (!g->total_nodes) return SIGMO_OK;
  const unsigned grid = grid_for(g->total_nodes, 256, 148u * 32u);
  if (q->opts.profile == kProfileExact) {
    if (g->max_nodes > 64u * kMaxAdjWords)
      return fail(SIGMO_ERR_DOMAIN, "exact profile supports graphs of at most %u vertices (largest: %u)", 64u * kMaxAdjWords, g->max_nodes);
    if (reach_words != kMaxAdjWords) return fail(SIGMO_ERR_INVALID, "exact profile needs %u reachable words", kMaxAdjWords);
    switch (g->adj_words) {
      case 1: k_sig_refine_exact<1><<<grid, 256, 0, q->stream>>>(g->total_nodes, g->graph_offsets, g->node_graph, g->adj, g->node_labels, view, sig, reach); break;
      case 2: k_sig_refine_exact<2><<<grid, 256, 0, q->stream>>>(g->total_nodes, g->graph_offsets, g->node_graph, g->adj, g->node_labels, view, sig, reach); break;
      default: k_sig_refine_exact<4><<<grid, 256, 0, q->stream>>>(g->total_nodes, g->graph_offsets, g->node_graph, g->adj, g->node_labels, view, sig, reach); break;
    }
    return check_launch(q, "k_sig_refine_exact");
  }
  if (q->opts.profile == kProfileX86) {
    if (g->max_nodes > 64u * kMaxAdjWords)
      return fail(SIGMO_ERR_DOMAIN, "REF_X86 profile supports graphs of at most %u vertices (largest: %u)", 64u * kMaxAdjWords,
                  g->max_nodes);
    k_sig_refine_ptx<true><<<grid, 256, 0, q->stream>>>(g->total_nodes, g->graph_offsets, g->node_graph, g->adj, g->adj_words,
                                                        g->row_offsets, g->column_indices, g->node_labels, view, sig, reach);
    return check_launch(q, "k_sig_refine_x86");
  }
  k_sig_refine_ptx<false><<<grid, 256, 0, q->stream>>>(g->total_nodes, g->graph_offsets, g->node_graph, g->adj, g->adj_words,
                                                       g->row_offsets, g->column_indices, g->node_labels, view, sig, reach);
  return check_launch(q, "k_sig_refine_ptx");
}

int launch_sig_all(Queue* q, const Graph* g, uint32_t R, uint64_t* sig_all) {
  if (!g->total_nodes || !R) return SIGMO_OK;
  const unsigned grid = grid_for(g->total_nodes, 256, 148u * 32u);
  if (q->opts.profile == kProfileExact) {
    if (g->max_nodes > 64u * kMaxAdjWords)
      return fail(SIGMO_ERR_DOMAIN, "exact profile supports graphs of at most %u vertices (largest: %u)", 64u * kMaxAdjWords, g->max_nodes);
    switch (g->adj_words) {
      case 1: k_sig_all_staged<1, true><<<grid, kSigRange, 0, q->stream>>>(g->total_nodes, g->graph_offsets, g->node_graph, g->adj, g->row_offsets, g->column_indices, g->node_labels, R, sig_all); break;
      case 2: k_sig_all_staged<2, true><<<grid, kSigRange, 0, q->stream>>>(g->total_nodes, g->graph_offsets, g->node_graph, g->adj, g->row_offsets, g->column_indices, g->node_labels, R, sig_all); break;
      default: k_sig_all_staged<4, true><<<grid, kSigRange, 0, q->stream>>>(g->total_nodes, g->graph_offsets, g->node_graph, g->adj, g->row_offsets, g->column_indices, g->node_labels, R, sig_all); break;
    }
    return check_launch(q, "k_sig_all<exact>");
  }
  switch (g->adj_words) {
    case 1: k_sig_all_staged<1, false><<<grid, kSigRange, 0, q->stream>>>(g->total_nodes, g->graph_offsets, g->node_graph, g->adj, g->row_offsets, g->column_indices, g->node_labels, R, sig_all); break;
    case 2: k_sig_all_staged<2, false><<<grid, kSigRange, 0, q->stream>>>(g->total_nodes, g->graph_offsets, g->node_graph, g->adj, g->row_offsets, g->column_indices, g->node_labels, R, sig_all); break;
    default: k_sig_all_staged<4, false><<<grid, kSigRange, 0, q->stream>>>(g->total_nodes, g->graph_offsets, g->node_graph, g->adj, g->row_offsets, g->column_indices, g->node_labels, R, sig_all); break;
  }
  return check_launch(q, "k_sig_all<ptx>");
}

}  // namespace sigmo_b200
