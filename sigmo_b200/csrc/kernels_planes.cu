// Batched form: per-graph candidate planes.
//
// The reference's candidate test for query vertex j and data vertex d after
// R refinements is (isomorphism.hpp:48-55, 103-111)
//     label(j) == label(d) (or label(j) is the wildcard)
//     and, for every iteration r and label l, count_l(sig_r(j)) <= count_l(sig_r(d)).
// For a fixed query batch the set of thresholds that appear is small, so each
// data graph gets one u64 mask ("plane") per distinct query label and per
// distinct (r, l, c) threshold: bit t = local vertex t passes.  The candidate
// set of query vertex j in data graph g is then the AND of the planes in j's
// program; graph-local range visibility (the REF_PTX last-word rule of
// candidates.hpp:98) is folded into the label planes.  Identical query
// vertices share one program ("class").
//
// Plane layouts in memory (u64 words): a batch's planes are graph-major,
// planes[g][k][AW], so the join's level masks of one molecule read one run of
// K words (k_pair_masks, whose lanes hold levels of a few molecules: 0.85 ->
// 0.67 ms for 6.86 M pairs against tile-major rows); the serving loop's resident
// planes are tile-major, planes[g / 32][k][AW][g % 32], so that the rows of a
// tile that a batch uses are gathered in 256-byte runs.  In shared memory a
// tile is [k][AW][32], read with lane = graph, conflict-free.
#include <cuda_runtime.h>

#include <algorithm>

#include "internal.hpp"

namespace sigmo_b200 {
namespace {

// spec[k]: bit 31 set = label plane (bits 0..7 = label value, 255 = any);
// otherwise r = bits 16..23, l = bits 8..15, c = bits 0..7 (count >= c).
// Label planes come first, then thresholds in (r, l, c) order.

// One graph's planes into column `col` of a shared-memory tile whose rows are
// `row_words` words apart, by one warp.  With `out`, the words also go to
// out[k][AW] (row row_of[k] when given).
//
// Label planes: the lanes hold vertices lane + 32 p, a plane is a ballot per
// 32-vertex chunk.  Threshold planes: the lanes hold 32 planes (consecutive
// planes share an iteration, so a load of a vertex's counters is a broadcast of
// two or three words) and walk the vertices from the last to the first, shifting
// each comparison's carry into the lane's word: a load, a shift and two
// additions per vertex for 32 planes, where a ballot per plane took a
// load, the extraction, a vote and a select for 32 vertices of molecules with
// 35 (k_planes_admit 1.36 -> 1.09 ms on 100,000 molecules x 600 queries, 0.93 ->
// 0.51 ms on 60,013 x 500 with sets of two words).
//
// plane_test: what a plane compares.  Labels: {value, -}.  Thresholds:
// {2^32 - (c << 28), left shift that brings the counter's four bits to the top
// of its 32-bit half | 0x100 for the high half | iteration << 16}: count >= c
// exactly when the shifted half >= c << 28 (the bits below the counter only add
// to it), i.e. when adding 2^32 - (c << 28) carries out.
__device__ __forceinline__ uint2 plane_test(uint32_t sp) {
  if (sp & 0x80000000u) return make_uint2(sp & 0xFFu, 0u);
  const uint32_t l = (sp >> 8) & 0xFFu;
  return make_uint2(0u - ((sp & 0xFFu) << 28), (28u - 4u * (l & 7u)) | (l >= 8u ? 0x100u : 0u) | (sp & 0xFF0000u));
}

// 2 * acc + the carry of x + y
__device__ __forceinline__ uint32_t shift_in_carry(uint32_t acc, uint32_t x, uint32_t y) {
  uint32_t r;
  asm("{\n .reg .u32 t;\n add.cc.u32 t, %2, %3;\n addc.u32 %0, %1, %1;\n}\n" : "=r"(r) : "r"(acc), "r"(x), "r"(y));
  return r;
}

template <int AW>
__device__ __forceinline__ void build_graph_planes(uint64_t* col, uint32_t row_words, uint32_t s, uint32_t e, unsigned lane,
                                                   const uint8_t* __restrict__ lab, const uint64_t* __restrict__ sig_all,
                                                   uint64_t N, uint32_t K, uint32_t nlab, const uint2* tests, int prof,
                                                   uint32_t base, uint64_t* __restrict__ out,
                                                   const uint32_t* __restrict__ row_of) {
  constexpr int P = 2 * AW;  // 32-vertex chunks per graph
  const uint32_t n = e - s;
  {
    uint8_t lb[P];
    bool vis[P];
#pragma unroll
    for (int p = 0; p < P; ++p) {
      const uint32_t t = lane + 32u * p;
      const bool in = t < n;
      const uint32_t v = s + t;
      lb[p] = in ? lab[v] : 0;
      // visibility follows global ids (base + local id): the range-mask rule
      // depends on where the graph ends relative to 32-vertex words
      const uint32_t gv = base + v;
      vis[p] = in && ((range_mask(gv >> 5, base + s, base + e, prof) >> (gv & 31u)) & 1u);
    }
    for (uint32_t k = 0; k < nlab; ++k) {
      const uint32_t val = tests[k].x;
      uint32_t chunk[P];
#pragma unroll
      for (int p = 0; p < P; ++p) chunk[p] = __ballot_sync(0xFFFFFFFFu, vis[p] && (val == kWildcard || lb[p] == val));
#pragma unroll
      for (int w = 0; w < AW; ++w)
        if (lane == static_cast<unsigned>(w)) {
          const uint64_t word = static_cast<uint64_t>(chunk[2 * w]) | (static_cast<uint64_t>(chunk[2 * w + 1]) << 32);
          col[k * row_words + w * 32] = word;
          if (out) out[static_cast<uint64_t>(row_of ? row_of[k] : k) * AW + w] = word;
        }
    }
  }
  for (uint32_t k0 = nlab; k0 < K; k0 += 32) {
    const uint32_t k = k0 + lane;
    const uint2 ts = tests[k < K ? k : K - 1u];
    const uint32_t sh = ts.y & 31u, bound = ts.x;
    const uint32_t* sg = reinterpret_cast<const uint32_t*>(sig_all + static_cast<uint64_t>((ts.y >> 16) & 0xFFu) * N + s) + ((ts.y >> 8) & 1u);
    uint64_t word[AW];
#pragma unroll
    for (int w = 0; w < AW; ++w) {
      uint32_t acc[2] = {0, 0};
#pragma unroll
      for (int h = 1; h >= 0; --h) {
        const uint32_t v0 = 64u * w + 32u * h;
        if (n <= v0) continue;
        uint32_t v = n - v0 < 32u ? n : v0 + 32u;
        for (; (v & 7u) && v > v0; --v) acc[h] = shift_in_carry(acc[h], __ldg(sg + 2 * (v - 1)) << sh, bound);
        for (; v > v0; v -= 8) {  // eight loads in flight
          uint32_t x[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) x[i] = __ldg(sg + 2 * (v - 1 - i));
#pragma unroll
          for (int i = 0; i < 8; ++i) acc[h] = shift_in_carry(acc[h], x[i] << sh, bound);
        }
      }
      word[w] = static_cast<uint64_t>(acc[0]) | (static_cast<uint64_t>(acc[1]) << 32);
    }
    if (k < K) {
      const uint64_t row = row_of && out ? row_of[k] : k;
#pragma unroll
      for (int w = 0; w < AW; ++w) {
        col[k * row_words + w * 32] = word[w];
        if (out) out[row * AW + w] = word[w];
      }
    }
  }
}

// Per tile of 32 * H graphs (one CTA per tile, grid-stride): build the tile's
// planes in shared memory from the data signatures (and write them out; the
// join reads them), then decide the GMCR admission of every query graph for
// the tile's graphs (gmcr.hpp:33-128: every query vertex has a candidate in
// the graph):
//     admit[q][tile] = AND over q's classes c of NE(c),
//     NE(c) = ballot over the tile's graphs of "AND of c's program planes != 0".
// Warps take query graphs; a query's classes are visited in the order the
// host chose (rarest label first, longer programs first), so most queries
// are rejected for all graphs after one or two classes and stop there.  A
// class's AND chain starts with the graphs the classes before it left and
// stops once it is zero in all of them (at every four planes: one 8-byte load
// gives four plane ids).  NE(c) is evaluated for each query that reaches it:
// classes are rarely shared between queries.  The per-graph admitted counts
// (the GMCR segment lengths) are summed in shared memory.  Queries of one
// vertex are never admitted (the reference's mapping skips them, gmcr.hpp:100):
// their class lists are empty.
//
// Bound by instruction issue (60,000 molecules x 600 queries: 63 % of the slots,
// 66 % of the integer pipe, 56 % of the shared-memory wavefronts).  H = 2: a lane carries two graphs through the
// chain, so the program, its addresses and the votes are paid once for 64
// graphs instead of twice (a model of 1,024 molecules x 600 queries: 4.1
// classes of 6.5 planes per 32-graph tile and query; 1.35 -> 1.09 ms on 100,000
// x 600, 0.533 -> 0.512 ms on 200,000 x 60); it needs twice the shared memory,
// so it is taken where two CTAs of 512 threads still fit an SM, and enough tiles
// for the CTAs that one graph per lane would keep on the chip (four per SM): the
// filter stage of 37,000 / 30,000 / 25,000 / 20,000 / 10,000 molecules x 300
// takes 0.314 / 0.253 / 0.222 / 0.189 / 0.119 ms with one, 0.283 / 0.238 / 0.197
// / 0.189 / 0.148 with two.  A tile whose graphs all have at most 64
// atoms works on word 0 alone in a batch of wider sets.
constexpr uint32_t kAdmitWarps = 16;

// 16-byte asynchronous global -> shared copies (no registers in between).
__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gmem_src) {
  const unsigned dst = static_cast<unsigned>(__cvta_generic_to_shared(smem_dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// Resident rows s_map[k] of the 32-graph tiles gw * H .. into dst
// [K][H][AW * 32], as 16-byte asynchronous copies spread over the block (tiles
// past the last one: zeros).
template <int AW, int H>
__device__ __forceinline__ void gather_tile_async(uint64_t* dst, const uint64_t* __restrict__ rplanes, uint32_t rrows,
                                                  uint32_t gw, uint32_t GW, uint32_t K, const uint32_t* s_map) {
  constexpr uint32_t kRow = AW * 32u, kChunks = AW * 16u * H;  // 16-byte chunks per row of the tile
  for (uint32_t i = threadIdx.x; i < K * kChunks; i += blockDim.x) {
    const uint32_t k = i / kChunks, c = i % kChunks, h = c / (AW * 16u), tile = gw * H + h;
    uint64_t* at = dst + static_cast<size_t>(k) * (H * kRow) + 2 * c;
    if (tile < GW) {
      cp_async16(at, rplanes + (static_cast<uint64_t>(tile) * rrows + s_map[k]) * kRow + 2 * (c % (AW * 16u)));
    } else {
      at[0] = at[1] = 0;
    }
  }
  cp_async_commit();
}

// Shared-memory layout of k_planes_admit: tile buffer [K][H][AW * 32] u64, the
// planes' tests [K] (uint2) or, for a gathered tile, their resident rows [K]
// (u32), then the queries' programs when they fit: prog[n_quads] (u64: four
// plane ids), q_off[QG + 1] (u32).
struct AdmitSmem {
  size_t specs, lists, total;
};
__host__ __device__ inline AdmitSmem admit_smem_layout(uint32_t K, uint32_t AW, uint32_t H, bool gather, size_t list_bytes) {
  AdmitSmem l{};
  size_t off = static_cast<size_t>(K) * H * AW * 32 * 8;
  l.specs = off;
  off += (gather ? 4ull : 8ull) * K;
  off = (off + 15) & ~static_cast<size_t>(15);
  l.lists = off;
  off += list_bytes;
  l.total = off;
  return l;
}

// The admission words of every query graph for one tile, on W of the AW words.
// A query's program is one run of quads, prog[q_off[qg], q_off[qg + 1]): its
// classes one after the other, bit 15 of a quad's last id marking a class's
// end.
template <int AW, int H, int W>
__device__ __forceinline__ void admit_tile(const uint64_t* tile, uint32_t QG, const uint32_t* q_off, const uint2* prog,
                                           const uint32_t (&valid)[H], uint32_t tile0, uint32_t GW,
                                           uint32_t* __restrict__ admit, uint32_t (&my_cnt)[H]) {
  constexpr uint32_t kRow = H * AW * 32u;
  const unsigned lane = threadIdx.x & 31u, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const uint64_t* tl = tile + lane;
  uint32_t i0 = wid < QG ? q_off[wid] : 0u;
  for (uint32_t qg = wid; qg < QG; qg += nw) {
    const uint32_t i1 = q_off[qg + 1];
    uint64_t m[H][W];
    bool left = i1 > i0;  // an empty program: a query of at most one vertex
#pragma unroll
    for (int h = 0; h < H; ++h)
#pragma unroll
      for (int w = 0; w < W; ++w) m[h][w] = left && ((valid[h] >> lane) & 1u) ? ~0ull : 0ull;
    uint2 ids = left ? prog[i0] : make_uint2(0, 0);
    for (uint32_t i = i0; i < i1;) {
      const uint2 cur = ids;
      if (++i < i1) ids = prog[i];  // one entry ahead
      const uint64_t* a = tl + (cur.x & 0xFFFFu) * kRow;
      const uint64_t* b = tl + (cur.x >> 16) * kRow;
      const uint64_t* c = tl + (cur.y & 0xFFFFu) * kRow;
      const uint64_t* d = tl + ((cur.y >> 16) & 0x7FFFu) * kRow;
      uint64_t some = 0;
#pragma unroll
      for (int h = 0; h < H; ++h)
#pragma unroll
        for (int w = 0; w < W; ++w) {
          const int o = (h * AW + w) * 32;
          m[h][w] &= (a[o] & b[o]) & (c[o] & d[o]);
          some |= m[h][w];
        }
      if (!__any_sync(0xFFFFFFFFu, some != 0)) {  // no graph has a candidate: the query is out
        left = false;
        break;
      }
      if (cur.y & 0x80000000u) {  // the class's end: the next one starts with the graphs that are left
#pragma unroll
        for (int h = 0; h < H; ++h) {
          uint64_t x = 0;
#pragma unroll
          for (int w = 0; w < W; ++w) x |= m[h][w];
#pragma unroll
          for (int w = 0; w < W; ++w) m[h][w] = x ? ~0ull : 0ull;
        }
      }
    }
    if (qg + nw < QG) i0 = q_off[qg + nw];
#pragma unroll
    for (int h = 0; h < H; ++h) {
      const uint32_t alive = __ballot_sync(0xFFFFFFFFu, left && m[h][0] != 0);
      if (lane == 0 && tile0 + h < GW) admit[static_cast<uint64_t>(qg) * GW + tile0 + h] = alive;
      my_cnt[h] += (alive >> lane) & 1u;
    }
  }
}

template <int AW, bool GATHER, int H>
__global__ void __launch_bounds__(kAdmitWarps * 32, AW == 1 ? (H == 1 ? 4 : 3) : 2) k_planes_admit(
    uint32_t G, const uint32_t* __restrict__ goff, const uint8_t* __restrict__ lab, const uint64_t* __restrict__ sig_all,
    uint64_t N, uint32_t K, uint32_t nlab, const uint32_t* __restrict__ spec, int prof, uint32_t base,
    const uint64_t* __restrict__ rplanes, uint32_t rrows, const uint32_t* __restrict__ row_map,
    uint32_t QG, const uint2* __restrict__ g_prog, const uint32_t* __restrict__ g_q_off, uint32_t n_quads, int stage_lists, const uint32_t* __restrict__ row_of, uint32_t out_rows, int accumulate,
    uint64_t* __restrict__ planes, uint32_t* __restrict__ admit, uint32_t* __restrict__ counts) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ uint32_t tile_cnt[32 * H];
  constexpr uint32_t kRow = H * AW * 32u;
  const unsigned lane = threadIdx.x & 31u, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const uint32_t GW = (G + 31u) / 32u, tiles = (GW + H - 1u) / H;
  const size_t list_bytes = stage_lists ? 8ull * n_quads + 4ull * (QG + 1) : 0;
  const AdmitSmem L = admit_smem_layout(K, AW, H, GATHER, list_bytes);
  uint64_t* tile = reinterpret_cast<uint64_t*>(smem_raw);
  uint32_t* s_map = reinterpret_cast<uint32_t*>(smem_raw + L.specs);
  uint2* s_test = reinterpret_cast<uint2*>(smem_raw + L.specs);
  // per-batch constants: the row map or the planes' tests, and (when they fit) the programs
  const uint32_t* q_off = g_q_off;
  const uint2* prog = g_prog;
  for (uint32_t i = threadIdx.x; i < K; i += blockDim.x) {
    if (GATHER) s_map[i] = row_map[i];
    else s_test[i] = plane_test(spec[i]);
  }
  if (stage_lists) {
    uint2* pp = reinterpret_cast<uint2*>(smem_raw + L.lists);
    for (uint32_t i = threadIdx.x; i < n_quads; i += blockDim.x) pp[i] = g_prog[i];
    uint32_t* p = reinterpret_cast<uint32_t*>(pp + n_quads);
    for (uint32_t i = threadIdx.x; i <= QG; i += blockDim.x) p[i] = g_q_off[i];
    prog = pp;
    q_off = p;
  }
  __syncthreads();
  for (uint32_t gw = blockIdx.x; gw < tiles; gw += gridDim.x) {
    __syncthreads();  // the previous tile is no longer read
    // every graph of the tile has at most 64 vertices (uniform: all threads vote)
    bool narrow = AW == 1;
    if (AW > 1) {
      bool wide = false;
      for (uint32_t i = threadIdx.x; i < 32u * H; i += blockDim.x) {
        const uint32_t g = gw * (32u * H) + i;
        if (g < G) wide |= goff[g + 1] - goff[g] > 64u;
      }
      narrow = !__syncthreads_or(wide);
    }
    if (GATHER) {
      // one tile buffer (not two, double-buffered): more CTAs share an SM and
      // hide each other's gathers
      gather_tile_async<AW, H>(tile, rplanes, rrows, gw, GW, K, s_map);
      cp_async_wait_all();  // this thread's copies; the barrier below covers the others'
    } else {
      for (uint32_t gl = wid; gl < 32u * H; gl += nw) {
        const uint32_t g = gw * (32u * H) + gl;
        uint64_t* col = tile + (gl >> 5) * (AW * 32u) + (gl & 31u);
        if (g < G) {
          build_graph_planes<AW>(col, kRow, goff[g], goff[g + 1], lane, lab, sig_all, N, K, nlab, s_test, prof, base,
                                 planes + static_cast<uint64_t>(g) * out_rows * AW, row_of);
        } else {
          for (uint32_t i = lane; i < K * AW; i += 32) col[(i / AW) * kRow + (i % AW) * 32] = 0;
        }
      }
    }
    if (threadIdx.x < 32u * H) tile_cnt[threadIdx.x] = 0;
    __syncthreads();
    uint32_t valid[H], my_cnt[H];
#pragma unroll
    for (int h = 0; h < H; ++h) {
      const uint32_t g0 = (gw * H + h) * 32u, in = g0 < G ? G - g0 : 0u;
      valid[h] = in >= 32u ? 0xFFFFFFFFu : ((1u << in) - 1u);
      my_cnt[h] = 0;
    }
    if (AW > 1 && narrow) admit_tile<AW, H, 1>(tile, QG, q_off, prog, valid, gw * H, GW, admit, my_cnt);
    else admit_tile<AW, H, AW>(tile, QG, q_off, prog, valid, gw * H, GW, admit, my_cnt);
#pragma unroll
    for (int h = 0; h < H; ++h) atomicAdd(&tile_cnt[32 * h + lane], my_cnt[h]);
    __syncthreads();
    const uint32_t g = gw * (32u * H) + threadIdx.x;
    if (threadIdx.x < 32u * H && g < G) {
      if (accumulate) atomicAdd(&counts[g], tile_cnt[threadIdx.x]);
      else counts[g] = tile_cnt[threadIdx.x];
    }
  }
  if (GATHER) cp_async_wait_all();
}

// Planes of a fixed spec for every graph, into out[tile][out_rows][AW][32]
// (rows K .. out_rows - 1 zeroed): the resident planes of the serving loop.
template <int AW>
__global__ void __launch_bounds__(kAdmitWarps * 32) k_build_planes(
    uint32_t G, const uint32_t* __restrict__ goff, const uint8_t* __restrict__ lab, const uint64_t* __restrict__ sig_all,
    uint64_t N, uint32_t K, uint32_t nlab, const uint32_t* __restrict__ spec, int prof, uint32_t base, uint32_t out_rows,
    uint64_t* __restrict__ out) {
  extern __shared__ uint64_t tile[];  // [K * AW][32], then the planes' tests [K]
  const uint32_t GW = (G + 31u) / 32u;
  uint2* tests = reinterpret_cast<uint2*>(tile + static_cast<size_t>(K) * AW * 32);
  for (uint32_t i = threadIdx.x; i < K; i += blockDim.x) tests[i] = plane_test(spec[i]);
  for (uint32_t gw = blockIdx.x; gw < GW; gw += gridDim.x) {
    __syncthreads();
    for (uint32_t gl = threadIdx.x >> 5; gl < 32; gl += blockDim.x >> 5) {
      const uint32_t g = gw * 32u + gl, lane = threadIdx.x & 31u;
      if (g < G) {
        build_graph_planes<AW>(tile + gl, AW * 32u, goff[g], goff[g + 1], lane, lab, sig_all, N, K, nlab, tests, prof, base,
                               nullptr, nullptr);
      } else {
        for (uint32_t i = lane; i < K * AW; i += 32) tile[i * 32 + gl] = 0;
      }
    }
    __syncthreads();
    uint4* dst = reinterpret_cast<uint4*>(out + static_cast<uint64_t>(gw) * out_rows * AW * 32);
    const uint4* src = reinterpret_cast<const uint4*>(tile);
    const uint32_t have = K * AW * 16, all = out_rows * AW * 16;
    for (uint32_t i = threadIdx.x; i < all; i += blockDim.x) dst[i] = i < have ? src[i] : make_uint4(0, 0, 0, 0);
  }
}

// Largest count of label l at iteration r over all vertices: cmax[r * 16 + l].
__global__ void k_sig_cmax(const uint64_t* __restrict__ sig_all, uint64_t N, uint32_t R, unsigned int* __restrict__ cmax) {
  for (uint32_t r = 0; r < R; ++r) {
    uint32_t mx[16];
#pragma unroll
    for (int l = 0; l < 16; ++l) mx[l] = 0;
    for (uint64_t v = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; v < N;
         v += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
      const uint64_t sv = sig_all[static_cast<uint64_t>(r) * N + v];
#pragma unroll
      for (int l = 0; l < 16; ++l) mx[l] = max(mx[l], static_cast<uint32_t>((sv >> (4 * l)) & 0xFull));
    }
#pragma unroll
    for (int l = 0; l < 16; ++l) {
      const uint32_t m = __reduce_max_sync(0xFFFFFFFFu, mx[l]);
      if ((threadIdx.x & 31u) == 0 && m) atomicMax(&cmax[r * 16 + l], m);
    }
  }
}

// Vertices per label value (shared-memory bins, one atomic per bin per block).
__global__ void k_label_hist(const uint8_t* __restrict__ lab, uint64_t n, unsigned long long* __restrict__ hist) {
  __shared__ unsigned int bins[256];
  for (uint32_t i = threadIdx.x; i < 256; i += blockDim.x) bins[i] = 0;
  __syncthreads();
  for (uint64_t v = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; v < n;
       v += static_cast<uint64_t>(gridDim.x) * blockDim.x)
    atomicAdd(&bins[lab[v]], 1u);
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < 256; i += blockDim.x)
    if (bins[i]) atomicAdd(&hist[i], static_cast<unsigned long long>(bins[i]));
}

}  // namespace

int ensure_label_hist(Queue* q, Graph* g) {
  if (g->label_hist.size() == 256) return SIGMO_OK;
  void* buf = nullptr;
  SIGMO_TRY(tmp_alloc(q, &buf, 256 * 8));
  int rc = SIGMO_OK;
  if (cudaMemsetAsync(buf, 0, 256 * 8, q->stream) != cudaSuccess) rc = fail(SIGMO_ERR_CUDA, "memset failed");
  if (!rc && g->total_nodes) {
    k_label_hist<<<grid_for(g->total_nodes, 256, 148u * 4u), 256, 0, q->stream>>>(g->node_labels, g->total_nodes,
                                                                                 static_cast<unsigned long long*>(buf));
    rc = check_launch(q, "k_label_hist");
  }
  std::vector<uint64_t> h(256, 0);
  if (!rc && (cudaMemcpyAsync(h.data(), buf, 256 * 8, cudaMemcpyDeviceToHost, q->stream) != cudaSuccess ||
              cudaStreamSynchronize(q->stream) != cudaSuccess))
    rc = fail(SIGMO_ERR_CUDA, "label histogram read-back failed");
  dev_free(q, buf);
  if (!rc) g->label_hist = std::move(h);
  return rc;
}

size_t planes_admit_smem(uint32_t K, uint32_t AW) {
  return static_cast<size_t>(K) * AW * 32 * 8;
}

namespace {

// What one admission launch needs of a program: the whole batch's, or one
// group's (local ids; planes scattered to row_of).
struct AdmitView {
  uint32_t K, nlab, QG;
  const uint32_t* spec;
  const uint32_t* q_off;   // [QG + 1] entries of prog per query graph
  const uint32_t* row_of;  // group launches: local plane row -> row of the batch's plane array
  const uint64_t* prog;    // four plane ids per entry
  size_t n_quads;
  uint32_t out_rows;
  int accumulate;
};

template <int AW, bool GATHER, int H>
int admit_launch_h(Queue* q, const Graph* data, const uint64_t* sig_all, const AdmitView& v, const uint64_t* rplanes,
                   uint32_t rrows, const uint32_t* row_map, uint64_t* planes, uint32_t* admit, uint32_t* counts, unsigned sms) {
  const uint32_t G = data->num_graphs, GW = (G + 31u) / 32u, QG = v.QG;
  const uint32_t n_quads = static_cast<uint32_t>(v.n_quads);
  const size_t list_bytes = 8ull * n_quads + 4ull * (QG + 1);
  const size_t base = admit_smem_layout(v.K, AW, H, GATHER, 0).total;
  // stage the programs when the block still fits three to an SM
  const int stage = base + list_bytes <= 72u * 1024u ? 1 : 0;
  const size_t smem = admit_smem_layout(v.K, AW, H, GATHER, stage ? list_bytes : 0).total;
  if (smem > 220u * 1024u) return fail(SIGMO_ERR_DOMAIN, "k_planes_admit needs %zu bytes of shared memory", smem);
  const unsigned block = 32u * kAdmitWarps;
  int per_sm = 0;
  SIGMO_TRY(allow_max_dynamic_smem(reinterpret_cast<const void*>(k_planes_admit<AW, GATHER, H>), q->device));
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_planes_admit<AW, GATHER, H>, block, smem);
  if (e != cudaSuccess) return fail(SIGMO_ERR_CUDA, "k_planes_admit shared-memory setup failed: %s", cudaGetErrorString(e));
  const uint64_t grid = std::min<uint64_t>((GW + H - 1u) / H, static_cast<uint64_t>(std::max(per_sm, 1)) * sms);
  k_planes_admit<AW, GATHER, H><<<grid, block, smem, q->stream>>>(
      G, data->graph_offsets, data->node_labels, sig_all, data->total_nodes, v.K, v.nlab, v.spec, q->opts.profile,
      data->vertex_base, rplanes, rrows, row_map, QG, reinterpret_cast<const uint2*>(v.prog), v.q_off, n_quads,
      stage, v.row_of, v.out_rows, v.accumulate, planes, admit, counts);
  return check_launch(q, "k_planes_admit");
}

template <int AW, bool GATHER>
int admit_launch(Queue* q, const Graph* data, const uint64_t* sig_all, const AdmitView& v, const uint64_t* rplanes,
                 uint32_t rrows, const uint32_t* row_map, uint64_t* planes, uint32_t* admit, uint32_t* counts) {
  int sms = 0;
  SIGMO_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, q->device));
  // two graphs per lane: see k_planes_admit
  const uint32_t GW = (data->num_graphs + 31u) / 32u;
  if constexpr (AW == 1)
    if (admit_smem_layout(v.K, AW, 2, GATHER, 0).total <= 110u * 1024u && GW >= 4u * static_cast<unsigned>(sms))
      return admit_launch_h<AW, GATHER, 2>(q, data, sig_all, v, rplanes, rrows, row_map, planes, admit, counts, sms);
  return admit_launch_h<AW, GATHER, 1>(q, data, sig_all, v, rplanes, rrows, row_map, planes, admit, counts, sms);
}

AdmitView whole_batch(const Graph* query, const PlaneProgram& pp) {
  return AdmitView{pp.K, pp.nlab, query->num_graphs, pp.spec, pp.q_off, nullptr, pp.quads, pp.n_quads, pp.K, 0};
}

}  // namespace

int launch_planes_admit(Queue* q, const Graph* query, const Graph* data, const uint64_t* sig_all, const PlaneProgram& pp,
                        uint64_t* planes, uint32_t* admit, uint32_t* counts) {
  if (!data->num_graphs) return SIGMO_OK;
  const AdmitView v = whole_batch(query, pp);
  switch (data->adj_words) {
    case 1: return admit_launch<1, false>(q, data, sig_all, v, nullptr, 0, nullptr, planes, admit, counts);
    case 2: return admit_launch<2, false>(q, data, sig_all, v, nullptr, 0, nullptr, planes, admit, counts);
    default: return admit_launch<4, false>(q, data, sig_all, v, nullptr, 0, nullptr, planes, admit, counts);
  }
}

int launch_planes_admit_group(Queue* q, const Graph* query, const Graph* data, const uint64_t* sig_all, const PlaneGroup& grp,
                              uint32_t K_total, uint64_t* planes, uint32_t* admit, uint32_t* counts) {
  if (!data->num_graphs || grp.q1 <= grp.q0) return SIGMO_OK;
  const uint32_t GW = (data->num_graphs + 31u) / 32u;
  const AdmitView v{grp.K,      grp.nlab, grp.q1 - grp.q0, grp.spec, grp.q_off, grp.row_of, grp.quads, grp.n_quads,
                    K_total, 1};
  uint32_t* adm = admit + static_cast<uint64_t>(grp.q0) * GW;
  switch (data->adj_words) {
    case 1: return admit_launch<1, false>(q, data, sig_all, v, nullptr, 0, nullptr, planes, adm, counts);
    case 2: return admit_launch<2, false>(q, data, sig_all, v, nullptr, 0, nullptr, planes, adm, counts);
    default: return admit_launch<4, false>(q, data, sig_all, v, nullptr, 0, nullptr, planes, adm, counts);
  }
}

int launch_planes_admit_resident(Queue* q, const Graph* query, const Graph* data, const ResidentPlanes& rp, uint32_t K,
                                 const uint64_t* quads, size_t n_quads, const uint32_t* q_off, const uint32_t* row_map,
                                 uint32_t* admit, uint32_t* counts) {
  if (!data->num_graphs) return SIGMO_OK;
  const AdmitView v{K, 0, query->num_graphs, nullptr, q_off, nullptr, quads, n_quads, 0, 0};
  switch (data->adj_words) {
    case 1: return admit_launch<1, true>(q, data, nullptr, v, rp.planes, rp.rows, row_map, nullptr, admit, counts);
    case 2: return admit_launch<2, true>(q, data, nullptr, v, rp.planes, rp.rows, row_map, nullptr, admit, counts);
    default: return admit_launch<4, true>(q, data, nullptr, v, rp.planes, rp.rows, row_map, nullptr, admit, counts);
  }
}

// Resident planes of every (label) and (iteration, label, count) that occurs
// in the database: label planes for each label present and the wildcard,
// thresholds c = 1..cmax(r, l), then one zero row.
int build_resident_planes(Queue* q, Graph* data, const uint64_t* sig_all, uint32_t R, ResidentPlanes* out) {
  SIGMO_TRY(ensure_label_hist(q, data));
  const uint64_t N = data->total_nodes;
  const uint32_t G = data->num_graphs, GW = (G + 31u) / 32u, AW = data->adj_words;
  std::vector<unsigned int> cmax(16ull * (R ? R : 1), 0);
  if (R && N) {
    void* d = nullptr;
    SIGMO_TRY(dev_alloc(q, &d, 4ull * 16 * R));
    int rc = cudaMemsetAsync(d, 0, 4ull * 16 * R, q->stream) == cudaSuccess ? SIGMO_OK : fail(SIGMO_ERR_CUDA, "memset failed");
    if (!rc) {
      k_sig_cmax<<<grid_for(N, 256, 148u * 8u), 256, 0, q->stream>>>(sig_all, N, R, static_cast<unsigned int*>(d));
      rc = check_launch(q, "k_sig_cmax");
    }
    if (!rc && (cudaMemcpyAsync(cmax.data(), d, 4ull * 16 * R, cudaMemcpyDeviceToHost, q->stream) != cudaSuccess ||
                cudaStreamSynchronize(q->stream) != cudaSuccess))
      rc = fail(SIGMO_ERR_CUDA, "cmax read-back failed");
    dev_free(q, d);
    SIGMO_TRY(rc);
  }
  std::vector<uint32_t> spec;
  out->label_row.assign(256, 0);
  for (uint32_t l = 0; l < 256; ++l)
    if (data->label_hist[l] || l == kWildcard) {
      out->label_row[l] = static_cast<uint32_t>(spec.size());
      spec.push_back(0x80000000u | l);
    }
  const uint32_t nlab = static_cast<uint32_t>(spec.size());
  out->base_row.assign(16ull * R, 0);
  out->cmax.assign(16ull * R, 0);
  for (uint32_t r = 0; r < R; ++r) {
    for (uint32_t l = 0; l < 16; ++l) {
      const uint32_t cm = cmax[r * 16 + l];
      out->cmax[r * 16 + l] = static_cast<uint8_t>(cm);
      out->base_row[r * 16 + l] = static_cast<uint32_t>(spec.size());
      for (uint32_t c = 1; c <= cm; ++c) spec.push_back((r << 16) | (l << 8) | c);
    }
  }
  const uint32_t K = static_cast<uint32_t>(spec.size());
  out->zero_row = K;
  for (uint32_t l = 0; l < 256; ++l)
    if (!data->label_hist[l] && l != kWildcard) out->label_row[l] = K;
  out->rows = K + 1;
  out->R = R;
  const size_t smem = static_cast<size_t>(K) * (AW * 32 * 8 + 8);
  if (planes_admit_smem(K, AW) > kTileSmemLimit) return fail(SIGMO_ERR_DOMAIN, "the database needs %u resident planes (too many for one tile)", K);
  void* dspec = nullptr;
  SIGMO_TRY(dev_alloc(q, &dspec, 4ull * K));
  int rc = SIGMO_OK;
  if (cudaMemcpyAsync(dspec, spec.data(), 4ull * K, cudaMemcpyHostToDevice, q->stream) != cudaSuccess)
    rc = fail(SIGMO_ERR_CUDA, "H2D copy failed");
  if (!rc) rc = dev_alloc(q, reinterpret_cast<void**>(&out->planes), 8ull * GW * out->rows * AW * 32 + 8);
  if (!rc && GW) {
    int per_sm = 0, sms = 0;
    cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, q->device);
    const unsigned block = 32u * kAdmitWarps;
#define SIGMO_BUILD(AWV)                                                                                             \
  if (e == cudaSuccess &&                                                                                             \
      allow_max_dynamic_smem(reinterpret_cast<const void*>(k_build_planes<AWV>), q->device) != SIGMO_OK)               \
    e = cudaErrorInvalidValue;                                                                                         \
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_build_planes<AWV>, block, smem);  \
  if (e == cudaSuccess)                                                                                              \
    k_build_planes<AWV><<<std::min<uint64_t>(GW, static_cast<uint64_t>(std::max(per_sm, 1)) * sms), block, smem,      \
                          q->stream>>>(G, data->graph_offsets, data->node_labels, sig_all, N, K, nlab,               \
                                       static_cast<const uint32_t*>(dspec), q->opts.profile, data->vertex_base, out->rows, out->planes)
    switch (AW) {
      case 1: SIGMO_BUILD(1); break;
      case 2: SIGMO_BUILD(2); break;
      default: SIGMO_BUILD(4); break;
    }
#undef SIGMO_BUILD
    if (e != cudaSuccess) rc = fail(SIGMO_ERR_CUDA, "k_build_planes setup failed: %s", cudaGetErrorString(e));
    if (!rc) rc = check_launch(q, "k_build_planes");
  }
  if (!rc && cudaStreamSynchronize(q->stream) != cudaSuccess) rc = fail(SIGMO_ERR_CUDA, "resident plane build failed");
  dev_free(q, dspec);
  return rc;
}

}  // namespace sigmo_b200
