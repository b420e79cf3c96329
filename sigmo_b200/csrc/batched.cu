// The batched form (sigmo_match_batched): signatures for all iterations in
// one BFS, per-graph candidate planes, GMCR from the plane AND-programs, and
// the persistent join, with one host synchronisation (the admitted-pair
// total, as in gmcr.hpp:80) between the launches.  Results are identical to
// the stage-per-launch calls (library/src/sigmo.cpp:98-160).
#include <cuda_runtime.h>

#include <algorithm>
#include <thread>
#include <cstring>
#include <vector>

#include "internal.hpp"

namespace sigmo_b200 {
namespace {

void free_groups(PlaneProgram* pp) {
  pp->groups.clear();
  pp->groups_aw = 0;
}

void free_program(Queue* q, PlaneProgram* pp) {
  dev_free(q, pp->qsig_all);
  *pp = PlaneProgram{};
}

// Threads for host loops over n items: one per 1,024 items, at most 8 and at
// most the machine's hardware threads.
unsigned host_threads(uint64_t n) {
  const unsigned hw = std::max(1u, std::thread::hardware_concurrency());
  return static_cast<unsigned>(std::max<uint64_t>(1, std::min<uint64_t>({n / 1024, 8, hw})));
}
// f(part, begin, end) over `parts` contiguous ranges of [0, n), part 0 on the
// calling thread; parts <= 1 runs inline.
template <class F>
void parallel_ranges(uint64_t n, unsigned parts, F&& f) {
  if (parts <= 1) {
    f(0, 0, n);
    return;
  }
  std::vector<std::thread> th;
  th.reserve(parts - 1);
  for (unsigned p = 1; p < parts; ++p) th.emplace_back([&, p] { f(p, n * p / parts, n * (p + 1) / parts); });
  f(0, 0, n / parts);
  for (auto& t : th) t.join();
}

// A class program (plane ids below 2^15) appended to `quads`, four ids per
// entry, its last id repeated to fill the last entry, whose bit 63 is set.
template <class F>
void append_quads(size_t n, F&& id, std::vector<uint64_t>* quads) {
  for (size_t i = 0; i < n; i += 4) {
    uint64_t x = 0;
    for (size_t j = 0; j < 4; ++j) x |= static_cast<uint64_t>(id(std::min(i + j, n - 1))) << (16 * j);
    quads->push_back(x);
  }
  quads->back() |= 1ull << 63;
}

// The queue's pinned staging buffer, at least `bytes` large and free to write.
int stage_buffer(Queue* q, size_t bytes, void** p) {
  SIGMO_CUDA_TRY(cudaEventSynchronize(q->ev_stage));  // the last copy from it is done
  if (bytes > q->stage_bytes) {
    if (q->stage) cudaFreeHost(q->stage);
    q->stage = nullptr;
    q->stage_bytes = 0;
    const size_t want = std::max<size_t>(2 * bytes, 1 << 18);
    SIGMO_CUDA_TRY(cudaMallocHost(&q->stage, want));
    q->stage_bytes = want;
  }
  *p = q->stage;
  return SIGMO_OK;
}

// Host arrays packed into the staging buffer and copied to one device block:
// add() them all, then send().  at(i): the device address of array i.
struct Blob {
  std::vector<std::pair<const void*, size_t>> parts;
  std::vector<size_t> offs;
  size_t bytes = 0;
  char* dev = nullptr;
  template <class T>
  size_t add(const std::vector<T>& v) {
    offs.push_back(bytes);
    parts.emplace_back(v.data(), v.size() * sizeof(T));
    bytes += (v.size() * sizeof(T) + 255) & ~static_cast<size_t>(255);
    return parts.size() - 1;
  }
  // On q->stream; ev_stage is recorded after the copy.
  int send(Queue* q, std::shared_ptr<DeviceBlock>* block) {
    void* host = nullptr;
    SIGMO_TRY(stage_buffer(q, bytes, &host));
    for (size_t i = 0; i < parts.size(); ++i)
      if (parts[i].second) std::memcpy(static_cast<char*>(host) + offs[i], parts[i].first, parts[i].second);
    void* p = nullptr;
    SIGMO_TRY(dev_alloc(q, &p, bytes + 256));
    *block = std::make_shared<DeviceBlock>(q, p);
    dev = static_cast<char*>(p);
    SIGMO_CUDA_TRY(cudaMemcpyAsync(dev, host, bytes, cudaMemcpyHostToDevice, q->stream));
    SIGMO_CUDA_TRY(cudaEventRecord(q->ev_stage, q->stream));
    return SIGMO_OK;
  }
  template <class T>
  const T* at(size_t i) const {
    return reinterpret_cast<const T*>(dev + offs[i]);
  }
};

}  // namespace

// Builds (or reuses) the plane program of a query batch for R iterations:
// query signatures of iterations 1..R on the device, then on the host the
// distinct labels and (r, l, c) thresholds (the planes), the classes of
// identical (label, signature_1..R) vertices, each class's program (label plane
// first, then its thresholds), and per query graph its distinct classes in the
// order the admission kernel evaluates them: rarest label first (by the query
// batch's own vertices, whose labels are distributed like the molecules': a
// model of 1,024 molecules x 600 queries evaluates 4.04 classes per tile and
// query in this order, 4.09 by the molecules' histogram, which took a kernel and
// a read-back per data graph), then longer programs first, so a query that a
// graph cannot admit is usually rejected by its first class.
//
// One pass over the vertices with a hash table of classes, everything sent in
// one copy that the device waits for by an event: the sorted, threaded form
// with an upload and a wait per array took 0.9 ms of a call with 300 new
// queries, this one 0.5.
int build_plane_program(Queue* q, Graph* query, uint32_t R) {
  PlaneProgram& pp = query->pp;
  if (pp.valid && pp.R == R && pp.profile == q->opts.profile) return SIGMO_OK;
  free_program(q, &pp);
  // The program's device work runs on the side stream after the query
  // graph's own creation work only, so a data graph upload queued on the main
  // stream meanwhile overlaps the host work below.
  struct OnSide {
    Queue* q;
    cudaStream_t main;
    ~OnSide() { q->stream = main; }
  } on_side{q, q->stream};
  if (query->ready) SIGMO_CUDA_TRY(cudaStreamWaitEvent(q->side, query->ready, 0));
  q->stream = q->side;
  const uint64_t Qn = query->total_nodes;
  const uint32_t QG = query->num_graphs;
  SIGMO_TRY(dev_alloc(q, reinterpret_cast<void**>(&pp.qsig_all), 8ull * (R ? R : 1) * (Qn ? Qn : 1)));
  SIGMO_TRY(launch_sig_all(q, query, R, pp.qsig_all));
  std::vector<uint64_t> sig(static_cast<size_t>(R) * Qn);  // [vertex][R]
  std::vector<uint8_t> lab(Qn);
  if (Qn) {
    void* host = nullptr;
    SIGMO_TRY(stage_buffer(q, 8ull * R * Qn + Qn, &host));
    auto* h_sig = static_cast<uint64_t*>(host);
    auto* h_lab = reinterpret_cast<uint8_t*>(h_sig + static_cast<size_t>(R) * Qn);
    if (R) SIGMO_CUDA_TRY(cudaMemcpyAsync(h_sig, pp.qsig_all, 8ull * R * Qn, cudaMemcpyDeviceToHost, q->stream));
    SIGMO_CUDA_TRY(cudaMemcpyAsync(h_lab, query->node_labels, Qn, cudaMemcpyDeviceToHost, q->stream));
    SIGMO_CUDA_TRY(cudaStreamSynchronize(q->stream));
    for (uint32_t r = 0; r < R; ++r)
      for (uint64_t v = 0; v < Qn; ++v) sig[v * R + r] = h_sig[static_cast<size_t>(r) * Qn + v];
    std::memcpy(lab.data(), h_lab, Qn);
  }

  // classes, in order of their first vertex: an open-addressing table of first
  // vertices, compared exactly (hashed by the multiply and xor-shift step of
  // MurmurHash3's 64-bit finaliser)
  std::vector<uint32_t> cls(Qn), first;
  std::vector<uint64_t> label_count(256, 0);
  // a class's thresholds as raw codes r << 8 | l << 4 | c, back to back, and
  // which codes occur
  std::vector<uint16_t> raw(Qn * 16);
  std::vector<uint32_t> raw_off{0};
  std::vector<uint8_t> occurs(static_cast<size_t>(R) * 256, 0);
  size_t raw_n = 0;
  first.reserve(Qn);
  raw_off.reserve(Qn + 1);
  {
    size_t size = 16;
    while (size < 2 * Qn) size *= 2;
    std::vector<uint32_t> table(size, 0);  // class + 1, 0: free
    for (uint64_t v = 0; v < Qn; ++v) {
      const uint64_t* sv = sig.data() + v * R;
      ++label_count[lab[v]];
      uint64_t h = 0x9E3779B97F4A7C15ull * (lab[v] + 1u);
      for (uint32_t r = 0; r < R; ++r) {
        h ^= sv[r];
        h *= 0xFF51AFD7ED558CCDull;
        h ^= h >> 32;
      }
      size_t at = h & (size - 1);
      for (;; at = (at + 1) & (size - 1)) {
        const uint32_t c = table[at];
        if (!c) {
          table[at] = static_cast<uint32_t>(first.size() + 1);
          cls[v] = static_cast<uint32_t>(first.size());
          first.push_back(static_cast<uint32_t>(v));
          if (raw.size() < raw_n + 16ull * R) raw.resize(2 * raw.size() + 16ull * R);
          for (uint32_t r = 0; r < R; ++r)
            for (uint64_t x = sv[r]; x;) {
              const uint32_t l = static_cast<uint32_t>(__builtin_ctzll(x)) >> 2;
              const uint32_t code = (r << 8) | (l << 4) | static_cast<uint32_t>((x >> (4 * l)) & 0xFu);
              raw[raw_n++] = static_cast<uint16_t>(code);
              occurs[code] = 1;
              x &= ~(0xFull << (4 * l));
            }
          raw_off.push_back(static_cast<uint32_t>(raw_n));
          break;
        }
        const uint64_t f = first[c - 1];
        if (lab[f] == lab[v] && std::equal(sv, sv + R, sig.data() + f * R)) {
          cls[v] = c - 1;
          break;
        }
      }
    }
  }
  const uint32_t C = static_cast<uint32_t>(first.size());
  // planes: label values used by queries (ascending), then the thresholds
  // (r, l, c) that occur, in (r, l, c) order
  std::vector<uint32_t> spec;
  std::vector<uint32_t> label_idx(256, 0), thr_idx(static_cast<size_t>(R) * 256, 0);
  for (uint32_t l = 0; l < 256; ++l)
    if (label_count[l]) {
      label_idx[l] = static_cast<uint32_t>(spec.size());
      spec.push_back(0x80000000u | l);
    }
  const uint32_t nlab = static_cast<uint32_t>(spec.size());
  for (uint32_t code = 0; code < R * 256u; ++code)
    if (occurs[code]) {
      thr_idx[code] = static_cast<uint32_t>(spec.size());
      spec.push_back(((code >> 8) << 16) | (((code >> 4) & 0xFu) << 8) | (code & 0xFu));
    }
  if (spec.size() >= 65535) return fail(SIGMO_ERR_DOMAIN, "query batch needs %zu candidate planes (limit 65535)", spec.size());
  // the classes' programs, and their place in the evaluation order
  std::vector<uint32_t> prog_off(C + 1, 0);
  std::vector<uint16_t> prog(raw_n + C);
  std::vector<uint64_t> rank(C);  // vertices with the label, then longer programs first
  size_t n_prog = 0;
  for (uint32_t c = 0; c < C; ++c) {
    const uint8_t l = lab[first[c]];
    prog[n_prog++] = static_cast<uint16_t>(label_idx[l]);
    for (uint32_t i = raw_off[c]; i < raw_off[c + 1]; ++i) prog[n_prog++] = static_cast<uint16_t>(thr_idx[raw[i]]);
    prog_off[c + 1] = static_cast<uint32_t>(n_prog);
    rank[c] = ((l == kWildcard ? Qn : label_count[l]) << 16) | (0xFFFFu - (prog_off[c + 1] - prog_off[c]));
  }
  std::vector<uint64_t> cquads;  // the classes' programs, four ids per entry
  std::vector<uint32_t> cquad_off(C + 1, 0);
  cquads.reserve(n_prog / 4 + C);
  for (uint32_t c = 0; c < C; ++c) {
    const uint32_t b = prog_off[c], n = prog_off[c + 1] - b;
    for (uint32_t i = 0; i < n; i += 4) {
      uint64_t x = 0;
      for (uint32_t j = 0; j < 4; ++j) x |= static_cast<uint64_t>(prog[b + std::min(i + j, n - 1)]) << (16 * j);
      cquads.push_back(x);
    }
    cquad_off[c + 1] = static_cast<uint32_t>(cquads.size());
  }
  // query graphs in parallel ranges, each range's lists on their own, then
  // concatenated in query order
  const std::vector<uint32_t>& qgoff = query->host_graph_offsets;
  const unsigned nt = host_threads(Qn / 8);
  struct Part {
    std::vector<uint32_t> order, order_n, quads_n;
    std::vector<uint64_t> quads;
  };
  std::vector<Part> parts(nt);
  const bool with_quads = spec.size() < 32768u;
  parallel_ranges(QG, nt, [&](unsigned t, uint64_t q0, uint64_t q1) {
    Part& p = parts[t];
    std::vector<std::pair<uint64_t, uint32_t>> list;
    for (uint64_t qg = q0; qg < q1; ++qg) {
      list.clear();
      // queries of one vertex are never admitted (gmcr.hpp:100): an empty list
      // tells the kernel so
      if (qgoff[qg + 1] - qgoff[qg] > 1)
        for (uint32_t v = qgoff[qg]; v < qgoff[qg + 1]; ++v) list.emplace_back(rank[cls[v]], cls[v]);
      std::sort(list.begin(), list.end());
      list.erase(std::unique(list.begin(), list.end()), list.end());
      const size_t before = p.quads.size();
      for (const auto& x : list) {
        p.order.push_back(x.second);
        if (!with_quads) continue;
        p.quads.insert(p.quads.end(), cquads.begin() + cquad_off[x.second], cquads.begin() + cquad_off[x.second + 1]);
        p.quads.back() |= 1ull << 63;
      }
      p.order_n.push_back(static_cast<uint32_t>(list.size()));
      p.quads_n.push_back(static_cast<uint32_t>(p.quads.size() - before));
    }
  });
  std::vector<uint32_t> q_off{0};
  std::vector<uint64_t> quads;
  pp.order.clear();
  pp.order_off.assign(1, 0);
  for (const Part& p : parts) {
    pp.order.insert(pp.order.end(), p.order.begin(), p.order.end());
    quads.insert(quads.end(), p.quads.begin(), p.quads.end());
    for (uint32_t n : p.order_n) pp.order_off.push_back(pp.order_off.back() + n);
    for (uint32_t n : p.quads_n) q_off.push_back(q_off.back() + n);
  }
  Blob blob;
  const size_t i_spec = blob.add(spec), i_off = blob.add(cquad_off), i_prog = blob.add(cquads), i_cls = blob.add(cls),
               i_qoff = blob.add(q_off), i_quads = blob.add(quads);
  SIGMO_TRY(blob.send(q, &pp.blob));
  SIGMO_CUDA_TRY(cudaStreamWaitEvent(on_side.main, q->ev_stage, 0));
  pp.spec = blob.at<uint32_t>(i_spec);
  pp.prog_off = blob.at<uint32_t>(i_off);
  pp.prog = blob.at<uint64_t>(i_prog);
  pp.cls = blob.at<uint32_t>(i_cls);
  pp.q_off = blob.at<uint32_t>(i_qoff);
  pp.quads = blob.at<uint64_t>(i_quads);
  pp.n_quads = quads.size();
  pp.K = static_cast<uint32_t>(spec.size());
  pp.C = C;
  pp.nlab = nlab;
  pp.h_spec = std::move(spec);
  pp.h_prog = std::move(prog);
  pp.h_quads = std::move(cquads);
  pp.h_prog_off = std::move(prog_off);
  pp.R = R;
  pp.profile = q->opts.profile;
  pp.valid = true;
  return SIGMO_OK;
}

// Splits the query graphs into contiguous groups whose planes fit
// one admission tile (kGroupSmemBudget), greedily in query order, and uploads
// each group's program in local plane ids.  Planned once per set width AW;
// SIGMO_ERR_DOMAIN when a query graph alone does not fit a tile.
int plan_groups(Queue* q, Graph* query, uint32_t AW) {
  PlaneProgram& pp = query->pp;
  if (pp.groups_aw == AW) return SIGMO_OK;
  free_groups(&pp);
  if (planes_admit_smem(pp.K, AW) <= kGroupSmemBudget) {
    pp.groups_aw = AW;
    return SIGMO_OK;
  }
  const std::vector<uint32_t>&off = pp.order_off, &list = pp.order;
  const uint32_t QG = query->num_graphs, K = pp.K, C = pp.C;
  std::vector<uint32_t> plane_mark(K, 0), class_mark(C, 0);  // stamp = group number + 1
  uint32_t stamp = 0, Kg = 0, q0 = 0;
  std::vector<std::pair<uint32_t, uint32_t>> ranges;
  auto query_adds = [&](uint32_t qg, uint32_t* dk) {  // planes query qg adds to the group
    *dk = 0;
    std::vector<uint32_t> seen_planes;
    for (uint32_t e = off[qg]; e < off[qg + 1]; ++e) {
      const uint32_t c = list[e];
      if (class_mark[c] == stamp) continue;
      for (uint32_t i = pp.h_prog_off[c]; i < pp.h_prog_off[c + 1]; ++i) {
        const uint32_t k = pp.h_prog[i];
        if (plane_mark[k] != stamp && std::find(seen_planes.begin(), seen_planes.end(), k) == seen_planes.end()) {
          seen_planes.push_back(k);
          ++*dk;
        }
      }
    }
  };
  auto take = [&](uint32_t qg) {
    for (uint32_t e = off[qg]; e < off[qg + 1]; ++e) {
      const uint32_t c = list[e];
      if (class_mark[c] == stamp) continue;
      class_mark[c] = stamp;
      for (uint32_t i = pp.h_prog_off[c]; i < pp.h_prog_off[c + 1]; ++i)
        if (plane_mark[pp.h_prog[i]] != stamp) {
          plane_mark[pp.h_prog[i]] = stamp;
          ++Kg;
        }
    }
  };
  stamp = 1;
  for (uint32_t qg = 0; qg < QG; ++qg) {
    uint32_t dk;
    query_adds(qg, &dk);
    if (qg > q0 && planes_admit_smem(Kg + dk, AW) > kGroupSmemBudget) {
      ranges.emplace_back(q0, qg);
      ++stamp;
      Kg = 0;
      q0 = qg;
    }
    take(qg);
    if (planes_admit_smem(Kg, AW) > kTileSmemLimit)
      return fail(SIGMO_ERR_DOMAIN, "query graph %u alone needs more than one admission tile of shared memory", qg);
  }
  ranges.emplace_back(q0, QG);
  // each group's arrays, in local ids (planes in global order, so label
  // planes come first and thresholds stay grouped by iteration)
  for (size_t gi = 0; gi < ranges.size(); ++gi) {
    PlaneGroup grp;
    grp.q0 = ranges[gi].first;
    grp.q1 = ranges[gi].second;
    // this group's planes: those of its own queries' classes (marks from the
    // planning pass may have been overwritten by a later group sharing a plane)
    std::vector<uint8_t> in_group(K, 0);
    for (uint32_t qg = grp.q0; qg < grp.q1; ++qg)
      for (uint32_t e = off[qg]; e < off[qg + 1]; ++e)
        for (uint32_t i = pp.h_prog_off[list[e]]; i < pp.h_prog_off[list[e] + 1]; ++i) in_group[pp.h_prog[i]] = 1;
    std::vector<uint32_t> loc_plane(K, 0xFFFFFFFFu), spec, row_of;
    for (uint32_t k = 0; k < K; ++k)
      if (in_group[k]) {
        loc_plane[k] = static_cast<uint32_t>(spec.size());
        spec.push_back(pp.h_spec[k]);
        row_of.push_back(k);
      }
    uint32_t nlab = 0;
    for (uint32_t x : spec) nlab += (x & 0x80000000u) != 0;
    // the queries' programs in local ids
    std::vector<uint32_t> q_off{0};
    std::vector<uint64_t> quads;
    if (spec.size() >= 32768u) return fail(SIGMO_ERR_DOMAIN, "group %zu needs %zu planes (limit 32767)", gi, spec.size());
    for (uint32_t qg = grp.q0; qg < grp.q1; ++qg) {
      for (uint32_t e = off[qg]; e < off[qg + 1]; ++e) {
        const uint32_t b = pp.h_prog_off[list[e]], n = pp.h_prog_off[list[e] + 1] - b;
        // every local id the kernel will index with must be inside its array
        for (uint32_t i = 0; i < n; ++i)
          if (loc_plane[pp.h_prog[b + i]] >= spec.size())
            return fail(SIGMO_ERR_INVALID, "internal: group %zu plane %u outside its %zu planes", gi, loc_plane[pp.h_prog[b + i]], spec.size());
        append_quads(n, [&](size_t i) { return loc_plane[pp.h_prog[b + i]]; }, &quads);
      }
      q_off.push_back(static_cast<uint32_t>(quads.size()));
    }
    grp.K = static_cast<uint32_t>(spec.size());
    if (planes_admit_smem(grp.K, AW) > kTileSmemLimit)
      return fail(SIGMO_ERR_DOMAIN, "group %zu needs more than one admission tile of shared memory", gi);
    grp.nlab = nlab;
    grp.n_quads = quads.size();
    Blob blob;
    const size_t i_spec = blob.add(spec), i_row = blob.add(row_of), i_quads = blob.add(quads), i_off = blob.add(q_off);
    SIGMO_TRY(blob.send(q, &grp.blob));
    grp.spec = blob.at<uint32_t>(i_spec);
    grp.row_of = blob.at<uint32_t>(i_row);
    grp.quads = blob.at<uint64_t>(i_quads);
    grp.q_off = blob.at<uint32_t>(i_off);
    pp.groups.push_back(grp);
  }
  pp.groups_aw = AW;
  return SIGMO_OK;
}

void release_plane_program(Graph* g) {
  if (g->pp.valid || g->pp.qsig_all) free_program(g->q, &g->pp);
}

}  // namespace sigmo_b200

using namespace sigmo_b200;

namespace {

// The bitset route: fused filter writes the final bitset (all words), GMCR
// and the join read it.  Used when the caller asks for the bitset, or when a
// batch does not fit the plane route.
int batched_bitset(Queue* q, Graph* query, Graph* data, uint32_t R, int find_first, Candidates* c, Gmcr* m,
                   uint64_t* d_total, const BatchedRun& run) {
  PlaneProgram& pp = query->pp;
  const uint64_t N = data->total_nodes;
  void* buf = nullptr;
  const uint64_t b_dsig = run.dsig ? 0 : 8ull * R * N, b_planes = 16ull * 16 * R * c->Wp;
  auto al = [](uint64_t x) { return (x + 255) & ~255ull; };
  SIGMO_TRY(tmp_alloc(q, &buf, al(b_dsig) + al(b_planes) + 256));
  uint64_t* dsig = run.dsig ? const_cast<uint64_t*>(run.dsig) : static_cast<uint64_t*>(buf);
  uint32_t* planes = reinterpret_cast<uint32_t*>(static_cast<char*>(buf) + al(b_dsig));
  int rc = run.dsig ? SIGMO_OK : launch_sig_all(q, data, R, dsig);
  for (uint32_t r = 0; r < R && !rc; ++r)
    rc = launch_sig_planes(q, dsig + static_cast<uint64_t>(r) * N, N, c->Wp, planes + static_cast<uint64_t>(r) * 16 * 4 * c->Wp);
  if (!rc && cudaEventRecord(q->ev_match[1], q->stream) != cudaSuccess) rc = fail(SIGMO_ERR_CUDA, "event record failed");
  if (!rc) rc = launch_fused_filter(q, query, data, R, pp.qsig_all, planes, c);
  if (!rc && cudaEventRecord(q->ev_match[2], q->stream) != cudaSuccess) rc = fail(SIGMO_ERR_CUDA, "event record failed");
  if (!rc) rc = launch_gmcr(q, query, data, c, m, true, 0);
  if (!rc && cudaEventRecord(q->ev_match[3], q->stream) != cudaSuccess) rc = fail(SIGMO_ERR_CUDA, "event record failed");
  const bool exact = q->opts.profile == kProfileExact;
  MaskSource src;
  src.bits = c->bits;
  src.Wp = c->Wp;
  src.prof = q->opts.profile;
  if (!rc)
    rc = launch_join(q, query, data, src, m, find_first, exact ? 0u : std::min(data->low_offset_graphs, data->num_graphs), d_total,
                     run.query_ranges, run.nranges);
  dev_free(q, buf);
  return rc;
}

// The plane route (no full bitset in HBM).
int batched_planes(Queue* q, Graph* query, Graph* data, uint32_t R, int find_first, Gmcr* m, uint64_t* d_total,
                   const BatchedRun& run) {
  // stage events are not recorded while the work is captured into a graph
  auto mark = [&](int i) -> int {
    if (run.capture) return SIGMO_OK;
    return cudaEventRecord(q->ev_match[i], q->stream) == cudaSuccess ? SIGMO_OK : fail(SIGMO_ERR_CUDA, "event record failed");
  };
  PlaneProgram& pp = query->pp;
  const uint64_t N = data->total_nodes;
  const uint32_t G = data->num_graphs, GW = (G + 31u) / 32u, AW = data->adj_words;
  const bool exact = q->opts.profile == kProfileExact;
  const uint32_t L = exact ? 0u : std::min(data->low_offset_graphs, G);
  auto al = [](uint64_t x) { return (x + 255) & ~255ull; };
  const ResidentPlanes* rp = run.resident;
  const uint64_t b_dsig = run.dsig ? 0 : 8ull * R * N, b_planes = rp ? 0 : 8ull * G * pp.K * AW,
                 b_ne = 4ull * query->num_graphs * GW + 4ull * G;
  // resident planes: the batch's plane k is resident row row_map[k], and the
  // class programs are rewritten as resident rows for the join.  Where the
  // batch's planes exceed a tile, those with the same row (thresholds and labels
  // that the database does not reach all have the zero row) become one plane of
  // the tile, and the query programs follow: a tile then holds at most the
  // database's rows, which were built to fit one.
  std::vector<uint32_t> row_map, rq_off;
  std::vector<uint64_t> rprog, rquads;
  if (rp) {
    if (rp->R != R) return fail(SIGMO_ERR_INVALID, "resident planes hold %u iterations, the batch asks for %u", rp->R, R);
    row_map.resize(pp.K);
    for (uint32_t k = 0; k < pp.K; ++k) {
      const uint32_t sp = pp.h_spec[k];
      if (sp & 0x80000000u) {
        row_map[k] = rp->label_row[sp & 0xFFu];
      } else {
        const uint32_t r = (sp >> 16) & 0xFFu, l = (sp >> 8) & 0xFFu, c = sp & 0xFFu;
        row_map[k] = c <= rp->cmax[r * 16 + l] ? rp->base_row[r * 16 + l] + c - 1 : rp->zero_row;
      }
    }
    rprog.resize(pp.h_quads.size());
    for (size_t i = 0; i < rprog.size(); ++i) {
      const uint64_t x = pp.h_quads[i];
      for (int j = 0; j < 4; ++j) rprog[i] |= static_cast<uint64_t>(row_map[(x >> (16 * j)) & 0xFFFFu] & 0xFFFFu) << (16 * j);
    }
    if (planes_admit_smem(pp.K, AW) > kTileSmemLimit) {
      std::vector<uint32_t> tile_of(rp->rows, 0xFFFFFFFFu), rows;
      for (uint32_t row : row_map)
        if (tile_of[row] == 0xFFFFFFFFu) {
          tile_of[row] = static_cast<uint32_t>(rows.size());
          rows.push_back(row);
        }
      rq_off.push_back(0);
      for (uint32_t qg = 0; qg < query->num_graphs; ++qg) {
        for (uint32_t e = pp.order_off[qg]; e < pp.order_off[qg + 1]; ++e) {
          const uint32_t b = pp.h_prog_off[pp.order[e]], n = pp.h_prog_off[pp.order[e] + 1] - b;
          append_quads(n, [&](size_t i) { return tile_of[row_map[pp.h_prog[b + i]]]; }, &rquads);
        }
        rq_off.push_back(static_cast<uint32_t>(rquads.size()));
      }
      row_map = std::move(rows);
    }
    pp.gathered = static_cast<uint32_t>(row_map.size());
  }
  const uint64_t b_rows = al(4ull * row_map.size()), b_rprog = al(8ull * rprog.size()), b_rquads = al(8ull * rquads.size());
  const uint64_t b_map = b_rows + b_rprog + b_rquads + 4ull * rq_off.size();
  void* buf = nullptr;
  SIGMO_TRY(tmp_alloc(q, &buf, al(b_dsig) + al(b_planes) + al(b_ne) + al(b_map) + 256));
  char* p = static_cast<char*>(buf);
  uint64_t* dsig = run.dsig ? const_cast<uint64_t*>(run.dsig) : reinterpret_cast<uint64_t*>(p);
  p += al(b_dsig);
  uint64_t* planes = reinterpret_cast<uint64_t*>(p);
  p += al(b_planes);
  uint32_t* admit = reinterpret_cast<uint32_t*>(p);  // [query graphs][GW], then per-graph counts [G]
  uint32_t* adm_counts = admit + static_cast<uint64_t>(query->num_graphs) * GW;
  p += al(b_ne);
  uint32_t* d_row_map = reinterpret_cast<uint32_t*>(p);
  uint64_t* d_rprog = reinterpret_cast<uint64_t*>(p + b_rows);
  uint64_t* d_rquads = reinterpret_cast<uint64_t*>(p + b_rows + b_rprog);
  uint32_t* d_rq_off = reinterpret_cast<uint32_t*>(p + b_rows + b_rprog + b_rquads);
  int rc = run.dsig ? SIGMO_OK : launch_sig_all(q, data, R, dsig);
  if (!rc && rp) {
    if (cudaMemcpyAsync(d_row_map, row_map.data(), 4ull * row_map.size(), cudaMemcpyHostToDevice, q->stream) != cudaSuccess ||
        cudaMemcpyAsync(d_rprog, rprog.data(), 8ull * rprog.size(), cudaMemcpyHostToDevice, q->stream) != cudaSuccess)
      rc = fail(SIGMO_ERR_CUDA, "H2D copy failed");
    if (!rc && !rq_off.empty() &&
        (cudaMemcpyAsync(d_rquads, rquads.data(), 8ull * rquads.size(), cudaMemcpyHostToDevice, q->stream) != cudaSuccess ||
         cudaMemcpyAsync(d_rq_off, rq_off.data(), 4ull * rq_off.size(), cudaMemcpyHostToDevice, q->stream) != cudaSuccess))
      rc = fail(SIGMO_ERR_CUDA, "H2D copy failed");
  }
  if (!rc) rc = mark(1);
  if (!rc && !rp && !pp.groups.empty()) {
    // a batch too large for one tile: group by group into the batch's planes
    if (cudaMemsetAsync(adm_counts, 0, 4ull * G, q->stream) != cudaSuccess) rc = fail(SIGMO_ERR_CUDA, "memset failed");
    for (size_t gi = 0; gi < pp.groups.size() && !rc; ++gi)
      rc = launch_planes_admit_group(q, query, data, dsig, pp.groups[gi], pp.K, planes, admit, adm_counts);
  } else if (!rc) {
    rc = !rp              ? launch_planes_admit(q, query, data, dsig, pp, planes, admit, adm_counts)
         : rq_off.empty() ? launch_planes_admit_resident(q, query, data, *rp, pp.gathered, pp.quads, pp.n_quads, pp.q_off,
                                                         d_row_map, admit, adm_counts)
                          : launch_planes_admit_resident(q, query, data, *rp, pp.gathered, d_rquads, rquads.size(), d_rq_off,
                                                         d_row_map, admit, adm_counts);
  }
  if (!rc) rc = mark(2);
  // captured: the admitted total of the run that built the graph sizes the
  // arrays (the replay checks that it did not change)
  if (!rc) rc = launch_gmcr_from_admit(q, query, data, admit, adm_counts, m, !run.capture, run.capture ? m->total : 0);
  if (!rc) rc = mark(3);
  // REF_PTX: graphs starting below vertex 256 keep the reference's live
  // `visited` bitset, so they take the literal join
  MaskSource src;
  src.prof = q->opts.profile;
  src.planes = rp ? rp->planes : planes;
  src.K = rp ? rp->rows : pp.K;
  src.tiled = rp != nullptr;
  src.prog_off = pp.prog_off;
  src.prog = rp ? d_rprog : pp.prog;
  src.cls = pp.cls;
  if (!rc) rc = launch_join(q, query, data, src, m, find_first, L, d_total, run.query_ranges, run.nranges);
  dev_free(q, buf);
  return rc;
}

}  // namespace

namespace sigmo_b200 {

void drop_graph(Gmcr* m) {
  if (m->graph) cudaGraphExecDestroy(m->graph);
  m->graph = nullptr;
  m->graph_reads.clear();
  for (auto& k : m->graph_key) k = 0;
}

namespace {

// Replays the captured batch: the device work of the planes route (no host
// synchronisation inside), then the match total and the GMCR total to the
// queue's pinned buffer.  Returns SIGMO_ERR_INVALID (and drops the graph)
// when the admitted total differs from the one the graph was sized for.
int replay_graph(Queue* q, Graph* query, Graph* data, Gmcr* m, sigmo_match_result* out) {
  const cudaEvent_t e0 = q->ev_match[0], e1 = q->ev_match[1];
  cudaError_t e = cudaEventRecord(e0, q->stream);
  if (e == cudaSuccess) e = cudaGraphLaunch(m->graph, q->stream);
  if (e == cudaSuccess) q->launches += m->graph_launches;
  if (e == cudaSuccess) e = cudaEventRecord(e1, q->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(q->stream);
  float f = 0;
  if (e == cudaSuccess) cudaEventElapsedTime(&f, e0, e1);
  if (e != cudaSuccess) return fail(SIGMO_ERR_CUDA, "graph replay failed: %s", cudaGetErrorString(e));
  SIGMO_TRY(join_status_result(q));  // the graph read the status word back
  const uint64_t* pin = static_cast<const uint64_t*>(q->pinned);
  const uint32_t gtotal = *reinterpret_cast<const uint32_t*>(pin + 1);
  if (gtotal != m->total) {
    drop_graph(m);
    return fail(SIGMO_ERR_INVALID, "the admitted total changed since the graph was captured");
  }
  std::memset(out, 0, sizeof(*out));
  out->total_matches = pin[0];
  out->admitted_pairs = m->total;
  out->pairs = static_cast<uint64_t>(query->num_graphs) * data->num_graphs;
  out->ms_total = f;
  m->counts_valid = true;
  return SIGMO_OK;
}

// Captures the planes route for (query, data) into m->graph, sized by the
// admitted total of the run that just completed.
int capture_graph(Queue* q, Graph* query, Graph* data, uint32_t R, int find_first, Gmcr* m, const BatchedRun& run0) {
  drop_graph(m);
  BatchedRun run = run0;
  run.capture = true;
  const uint64_t launches0 = q->launches;
  SIGMO_CUDA_TRY(cudaStreamBeginCapture(q->stream, cudaStreamCaptureModeThreadLocal));
  uint64_t* d_total = nullptr;
  int rc = join_status_reset(q);
  if (!rc) rc = tmp_alloc(q, reinterpret_cast<void**>(&d_total), 8);
  if (!rc && cudaMemsetAsync(d_total, 0, 8, q->stream) != cudaSuccess) rc = fail(SIGMO_ERR_CUDA, "memset failed");
  if (!rc) rc = batched_planes(q, query, data, R, find_first, m, d_total, run);
  uint64_t* pin = static_cast<uint64_t*>(q->pinned);
  if (!rc && (cudaMemcpyAsync(pin, d_total, 8, cudaMemcpyDeviceToHost, q->stream) != cudaSuccess ||
              cudaMemcpyAsync(pin + 1, m->offsets + data->num_graphs, 4, cudaMemcpyDeviceToHost, q->stream) != cudaSuccess))
    rc = fail(SIGMO_ERR_CUDA, "capture of the read-back failed");
  if (!rc) rc = join_status_fetch(q);
  if (d_total) dev_free(q, d_total);
  cudaGraph_t g = nullptr;
  const cudaError_t ec = cudaStreamEndCapture(q->stream, &g);
  if (!rc && ec != cudaSuccess) rc = fail(SIGMO_ERR_CUDA, "stream capture failed: %s", cudaGetErrorString(ec));
  if (!rc) {
    const cudaError_t ei = cudaGraphInstantiate(&m->graph, g, 0);
    if (ei != cudaSuccess) {
      m->graph = nullptr;
      rc = fail(SIGMO_ERR_CUDA, "graph instantiation failed: %s", cudaGetErrorString(ei));
    }
  }
  if (g) cudaGraphDestroy(g);
  cudaGetLastError();
  if (!rc) {
    m->graph_reads.push_back(query->pp.blob);
    for (const PlaneGroup& grp : query->pp.groups) m->graph_reads.push_back(grp.blob);
  }
  m->graph_launches = q->launches - launches0;
  q->launches = launches0;  // nothing ran during the capture
  m->counts_valid = true;   // the counts of the run before the capture are still in place
  return rc;
}

}  // namespace

int match_batched(Queue* q, Graph* query, Graph* data, uint32_t R, int find_first, bool materialize, Candidates* c, Gmcr* m,
                  sigmo_match_result* out, const BatchedRun& run, bool graph) {
  if (query->max_nodes > kMaxQueryNodes)
    return fail(SIGMO_ERR_DOMAIN, "query graphs of up to %u vertices are supported (largest: %u)", kMaxQueryNodes, query->max_nodes);
  if (data->max_nodes > 64u * kMaxAdjWords)
    return fail(SIGMO_ERR_DOMAIN, "the batched form supports data graphs of up to %u vertices (largest: %u)", 64u * kMaxAdjWords,
                data->max_nodes);
  if (q->opts.profile == kProfileX86)
    return fail(SIGMO_ERR_DOMAIN, "the batched form runs the REF_PTX and EXACT profiles; REF_X86 runs the stage-per-launch calls");
  SIGMO_CUDA_TRY(cudaSetDevice(q->device));
  const sigmo_tuning& tn = q->tune;
  // (overflow_split has no effect on the device work)
  const uint64_t key[7] = {query->stamp, data->stamp, R | (static_cast<uint64_t>(data->vertex_base) << 32),
                           static_cast<uint64_t>(find_first),
                           static_cast<uint64_t>(q->opts.profile) | (static_cast<uint64_t>(tn.overflow_serial) << 8) |
                               (static_cast<uint64_t>(tn.join_kernel) << 24) | (static_cast<uint64_t>(tn.join_pool) << 32),
                           (static_cast<uint64_t>(tn.join_blocks_per_sm) << 48) | (static_cast<uint64_t>(tn.join_chunk) << 40) |
                               (static_cast<uint64_t>(tn.mask_chunk_slots) << 32) | tn.overflow_blocks,
                           q->join_budget};
  if (graph && !materialize && m->graph && std::equal(key, key + 7, m->graph_key)) {
    const int rc = replay_graph(q, query, data, m, out);
    if (rc != SIGMO_ERR_INVALID) return rc;  // else: recapture below
  }
  drop_graph(m);  // this run may replace the arrays a captured batch refers to
  std::memset(out, 0, sizeof(*out));
  SIGMO_TRY(join_status_reset(q));
  SIGMO_CUDA_TRY(cudaEventRecord(q->ev_match[0], q->stream));
  // the data graph's signatures do not depend on the query batch: launched
  // first, they run while the host builds the query batch's plane program
  BatchedRun prun = run;
  uint64_t* dsig_tmp = nullptr;
  if (!run.dsig && !run.capture && R && data->total_nodes) {
    SIGMO_TRY(tmp_alloc(q, reinterpret_cast<void**>(&dsig_tmp), 8ull * R * data->total_nodes));
    const int src = launch_sig_all(q, data, R, dsig_tmp);
    if (src) {
      dev_free(q, dsig_tmp);
      return src;
    }
    prun.dsig = dsig_tmp;
  }
  struct FreeTmp {
    Queue* q;
    uint64_t* p;
    ~FreeTmp() { dev_free(q, p); }
  } free_dsig{q, dsig_tmp};
  SIGMO_TRY(build_plane_program(q, query, R));
  uint64_t* d_total = nullptr;
  SIGMO_TRY(tmp_alloc(q, reinterpret_cast<void**>(&d_total), 8));
  int rc = cudaMemsetAsync(d_total, 0, 8, q->stream) == cudaSuccess ? SIGMO_OK : fail(SIGMO_ERR_CUDA, "memset failed");
  // the planes route takes any batch whose query graphs each fit an admission
  // tile (larger batches are admitted in groups); planes take 8 B per
  // (plane, graph, word) in device memory
  const size_t tile_bytes = planes_admit_smem(query->pp.K, data->adj_words);
  // (resident planes: a tile holds at most the database's rows, whatever the batch)
  const int prc = run.resident ? SIGMO_OK : plan_groups(q, query, data->adj_words);
  // SIGMO_ERR_DOMAIN: a query graph too large for a tile, bitset route
  if (prc && prc != SIGMO_ERR_DOMAIN) rc = prc;
  const bool planes_fit = run.resident || (!prc && (!query->pp.groups.empty() || tile_bytes <= kTileSmemLimit));
  const bool bitset_route = materialize || !planes_fit;
  if (!rc && bitset_route && data->vertex_base)
    rc = fail(SIGMO_ERR_DOMAIN, "a shard (vertex base %u) runs on the planes route only; this batch needs the bitset route",
              data->vertex_base);
  if (!rc) {
    if (bitset_route) {
      sigmo_candidates_t cc = static_cast<sigmo_candidates_t>(c);
      if (!cc) rc = sigmo_candidates_create(static_cast<sigmo_queue_t>(q), query->total_nodes, data->total_nodes, &cc);
      if (!rc) rc = batched_bitset(q, query, data, R, find_first, cc, m, d_total, prun);
      if (cc != c) sigmo_candidates_destroy(cc);
    } else {
      rc = batched_planes(q, query, data, R, find_first, m, d_total, prun);
    }
  }
  if (!rc && cudaEventRecord(q->ev_match[4], q->stream) != cudaSuccess) rc = fail(SIGMO_ERR_CUDA, "event record failed");
  if (!rc) rc = join_status_fetch(q);
  if (!rc) {
    cudaError_t e = cudaMemcpyAsync(q->pinned, d_total, 8, cudaMemcpyDeviceToHost, q->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(q->stream);
    if (e != cudaSuccess) rc = fail(SIGMO_ERR_CUDA, "batched read-back failed: %s", cudaGetErrorString(e));
  }
  if (!rc) rc = join_status_result(q);
  if (!rc) {
    out->total_matches = *static_cast<uint64_t*>(q->pinned);
    out->admitted_pairs = m->total;
    out->pairs = static_cast<uint64_t>(query->num_graphs) * data->num_graphs;
    float f;
    cudaEventElapsedTime(&f, q->ev_match[0], q->ev_match[1]);
    out->ms_signatures = f;
    cudaEventElapsedTime(&f, q->ev_match[1], q->ev_match[2]);
    out->ms_filter = f;
    cudaEventElapsedTime(&f, q->ev_match[2], q->ev_match[3]);
    out->ms_mapping = f;
    cudaEventElapsedTime(&f, q->ev_match[3], q->ev_match[4]);
    out->ms_join = f;
    cudaEventElapsedTime(&f, q->ev_match[0], q->ev_match[4]);
    out->ms_total = f;
    m->counts_valid = true;
  }
  dev_free(q, d_total);
  if (!rc && graph && !bitset_route) {
    // graph mode: capture this batch for the next calls with the same inputs
    rc = capture_graph(q, query, data, R, find_first, m, run);
    if (!rc) std::copy(key, key + 7, m->graph_key);
  }
  return rc;
}

}  // namespace sigmo_b200

extern "C" int sigmo_match_batched(sigmo_queue_t q, sigmo_graph_t query, sigmo_graph_t data, uint32_t R, int find_first,
                                   uint32_t flags, sigmo_candidates_t c, sigmo_gmcr_t m, sigmo_match_result* out) {
  if (!q || !query || !data || !m || !out) return fail(SIGMO_ERR_INVALID, "null argument");
  const bool materialize = (flags & SIGMO_MATCH_MATERIALIZE_BITSET) != 0;
  if (materialize && !c) return fail(SIGMO_ERR_INVALID, "SIGMO_MATCH_MATERIALIZE_BITSET needs a candidates object");
  if (c && (c->rows != query->total_nodes || c->targets != data->total_nodes))
    return fail(SIGMO_ERR_INVALID, "candidate bitset does not match the graphs");
  if (m->q != q || (c && c->q != q) || query->q != q || data->q != q) return fail(SIGMO_ERR_INVALID, "handles belong to another queue");
  return match_batched(q, query, data, R, find_first, materialize, c, m, out, BatchedRun{},
                       (flags & SIGMO_MATCH_CUDA_GRAPH) != 0);
}

// ---- autotuner --------------------------------------------------------------
extern "C" int sigmo_autotune(sigmo_queue_t q, sigmo_graph_t query, sigmo_graph_t data, uint32_t R, int find_first,
                              uint32_t reps, sigmo_tuning* best, double* best_ms, double* default_ms) {
  if (!q || !query || !data || !best) return fail(SIGMO_ERR_INVALID, "null argument");
  if (query->q != q || data->q != q) return fail(SIGMO_ERR_INVALID, "handles belong to another queue");
  if (reps == 0) reps = 3;
  sigmo_gmcr_t m = nullptr;
  SIGMO_TRY(sigmo_gmcr_create(q, &m));
  const sigmo_tuning saved = q->tune;
  auto measure = [&](const sigmo_tuning& t, double* ms, uint64_t* total) -> int {
    q->tune = t;
    std::vector<double> js;
    sigmo_match_result r{};
    for (uint32_t i = 0; i <= reps; ++i) {
      SIGMO_TRY(match_batched(q, query, data, R, find_first, false, nullptr, m, &r, BatchedRun{}));
      if (i) js.push_back(r.ms_join);
    }
    std::sort(js.begin(), js.end());
    *ms = js[js.size() / 2];
    *total = r.total_matches;
    return SIGMO_OK;
  };
  sigmo_tuning cur = Queue{}.tune;  // the library default
  double cur_ms = 0, d_ms = 0;
  uint64_t d_total = 0, total = 0;
  int rc = measure(cur, &d_ms, &d_total);
  cur_ms = d_ms;
  struct Axis {
    uint32_t sigmo_tuning::*field;
    std::vector<uint32_t> values;
  };
  const Axis axes[] = {
      {&sigmo_tuning::join_kernel, {0, 1, 2}},
      {&sigmo_tuning::overflow_serial, {0, 1}},
      {&sigmo_tuning::join_blocks_per_sm, {1, 2, 3, 4}},
      {&sigmo_tuning::join_pool, {1, 2, 4, 8}},
      {&sigmo_tuning::join_chunk, {1, 2, 4, 8, 16}},
      {&sigmo_tuning::overflow_blocks, {148, 296, 592, 1184, 2368}},
      {&sigmo_tuning::mask_chunk_slots, {2, 8, 32}},
  };
  for (const Axis& ax : axes) {
    for (uint32_t v : ax.values) {
      if (rc) break;
      if (cur.*ax.field == v) continue;
      sigmo_tuning t = cur;
      t.*ax.field = v;
      double ms = 0;
      rc = measure(t, &ms, &total);
      if (!rc && total != d_total)
        rc = fail(SIGMO_ERR_INVALID, "autotune: a launch shape changed the result (%llu vs %llu)", (unsigned long long)total,
                  (unsigned long long)d_total);
      if (!rc && ms < cur_ms * 0.98) {
        cur = t;
        cur_ms = ms;
      }
    }
  }
  sigmo_gmcr_destroy(m);
  if (rc) {
    q->tune = saved;
    return rc;
  }
  q->tune = cur;
  *best = cur;
  if (best_ms) *best_ms = cur_ms;
  if (default_ms) *default_ms = d_ms;
  return SIGMO_OK;
}
