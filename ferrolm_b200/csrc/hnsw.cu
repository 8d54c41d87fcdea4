// Hnsw (src/vector/hnsw.rs): batched search on the GPU, a warp per query or, for small batches, a team of warps.
//
// Device layout: data n x pd f32; links0 n x (m0+1) u32 (count, then ids) exactly as the
// reference stores layer 0 (hnsw.rs:50-51, :154-157); the upper layers as one flat u32 array in
// the order of the FLHNSW01 file (per node, per layer: count, ids) with a per-node start offset.
//
// Search of one query (hnsw.rs:323-351): greedy descent on the upper layers, then the best-first beam of search_layer
// (hnsw.rs:179-226), both in hnsw.cuh: the beam as ONE sorted list of ef entries with an "expanded" bit per entry, the
// visited set exact, in global memory (a team's, and a small graph's, in shared memory first).  A query that fills more than
// half of the latter stops with an overflow mark and is re-run by the host with a table four times larger.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdlib>
#include <memory>
#include <mutex>
#include <thread>

#include "hnsw.cuh"

FV_BOUNDS_TU(hnsw)

namespace fv {

struct HnswDev {
  const float* data;
  const uint8_t* bytes;        // fv_hnsw::d_bytes
  float byte_lo;
  const uint32_t* links0;
  const uint32_t* upper_off;   // n + 1 offsets into upper_flat
  const uint32_t* upper_flat;
  int pd, m0, metric, top;
  uint32_t ep;
  size_t n;
};

// Shared memory of one search, in bytes: the query (BYTES: as bytes too), the visited set's first part, the tie list, a run of rows and
// their distances, the team's job, and the beam where it is not in registers.
static constexpr int SEARCH_BLOCKS_PER_SM = 3;  // of 256 threads
template <int R>
__host__ __device__ __forceinline__ size_t search_smem(int pd, bool bytes, int m0, int ef, int sbits, int nw) {
  return size_t(pd) * 4 + (bytes ? row_bytes(pd) : 0) + visit_smem(sbits) + (TIED_CAP + 32 + 32) * 4 + team_smem(nw, m0) +
         (R == 0 ? ((size_t(ef) * 8 + 15) & ~size_t(15)) : 0);
}

// Bound by the latency of a chain: link row, visited set, rows, insertions, about 65 times per query at ef 64, and by the
// longest of a batch's queries (twice the average) at its end.  24 warps of 80 registers per SM hold a lane's 16
// pieces of a row in flight (10,000 queries at 200k x 128, ef 64, in an earlier form 2.02 ms; 32 warps of 64 registers, where
// the loads are issued a few at a time, 2.46; 16 warps of 128 2.28): now 1.52 ms from floats, 1.03 from bytes.
// work: distances, expansions, queries whose tie list overflowed, queries whose visited set overflowed (marked in
// overflow[] and left for a re-run).  NW = 1: one warp per query, blockDim / 32 queries per block; NW > 1: a query
// per block (Team in hnsw.cuh).
template <bool IS_L2, bool BYTES, int R, int NW>
__global__ void __launch_bounds__(team_threads(NW), team_blocks(NW))
    hnsw_search_kernel(HnswDev g, const float* __restrict__ queries, const uint32_t* __restrict__ qids, size_t nq, int k,
                       int ef, int sbits, int log2slots, uint32_t* __restrict__ tables, fv_neighbor* __restrict__ out,
                       uint32_t* __restrict__ counts, uint32_t* __restrict__ overflow,
                       unsigned long long* __restrict__ work, unsigned int* __restrict__ next_query) {
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int searcher = NW == 1 ? w : 0, per_block = NW == 1 ? int(blockDim.x >> 5) : 1;
  unsigned char* mine = dyn_smem() + size_t(searcher) * search_smem<R>(g.pd, BYTES, g.m0, ef, sbits, NW);
  float* sq = reinterpret_cast<float*>(mine);
  uint8_t* q_bytes = reinterpret_cast<uint8_t*>(sq + g.pd);
  uint32_t* small = reinterpret_cast<uint32_t*>(q_bytes + (BYTES ? row_bytes(g.pd) : 0));
  uint32_t* tied = small + visit_smem(sbits) / 4;
  const size_t gw = size_t(blockIdx.x) * per_block + searcher;
  VisitSet seen;
  visit_setup(seen, small, sbits, tables + (gw << log2slots), log2slots, g.n);
  Team<NW, BYTES> team{g.data, g.pd, tied + TIED_CAP, reinterpret_cast<float*>(tied + TIED_CAP + 32),
                reinterpret_cast<TeamJob*>(tied + TIED_CAP + 64), slot_links(g.m0), uint32_t(g.n), seen, 0u, g.bytes, -1};
  u64* list = reinterpret_cast<u64*>(reinterpret_cast<unsigned char*>(team.job) + team_smem(NW, g.m0));
  if (NW > 1 && w > 0) {
    team_serve<IS_L2, NW>(team);
    return;
  }
  unsigned long long n_dist = 0, n_exp = 0, n_tie_lost = 0, n_over = 0;
  auto upper = [&](uint32_t x, int layer) {
    size_t p = g.upper_off[x];
    for (int s = 1; s < layer; ++s) p += 1 + g.upper_flat[p];
    return g.upper_flat + p;
  };
  auto layer0 = [&](uint32_t x) { return g.links0 + size_t(x) * (g.m0 + 1); };

  // Queries are drawn from a counter (zero at launch): a batch gives every resident searcher two or three of them and
  // they differ in length, so a fixed deal leaves the ones that drew three long ones running alone at the end.
  for (;;) {
    size_t qi = 0;
    if (lane == 0) qi = atomicAdd(next_query, 1u);
    qi = __shfl_sync(FV_FULL, qi, 0);
    if (qi >= nq) break;
    const size_t qsrc = qids ? size_t(qids[qi]) : qi;
    const unsigned long long n_dist0 = n_dist, n_exp0 = n_exp;  // a query that overflows its table is re-run: its work counts once
    if (BYTES) {  // the query in bytes too, if it is of the rows' kind
      bool fits = true;
      int norm = 0;
      for (int c = lane; c < row_bytes(g.pd); c += 32) {
        const float x = c < g.pd ? queries[qsrc * size_t(g.pd) + c] : 0.f, v = c < g.pd ? x - g.byte_lo : 0.f;
        if (c < g.pd) sq[c] = x;
        fits = fits && x == rintf(x) && v >= 0.f && v <= 255.f;  // (x itself: the subtraction can round what is not whole, 5e-6 + 128 is 128)
        const int u = fits ? int(v) : 0;
        q_bytes[c] = uint8_t(u);
        norm += u * u;
      }
      norm = __reduce_add_sync(FV_FULL, norm);
      team.q_norm = __all_sync(FV_FULL, fits) ? norm : -1;
    } else {
      for (int c = lane; c < g.pd; c += 32) sq[c] = queries[qsrc * size_t(g.pd) + c];
    }
    visit_clear(seen);

    // entry point and greedy descent (hnsw.rs:329-347)
    uint32_t cur = g.ep;
    if (lane == 0) team.ids[0] = cur;
    team_eval<IS_L2, NW>(team, sq, 1);
    float curd = team.out[0];
    n_dist += 1;
    greedy_descent<IS_L2, NW>(team, g.n, upper, g.m0, sq, g.top, 0, cur, curd, n_dist, n_exp);

    // layer 0 (hnsw.rs:179-226 with ef = max(ef, k))
    Beam<R> best;
    best.init(ef, list);
    best.insert(beam_key(curd, cur));
    visit_warp(seen, lane == 0, cur);
    bool over = false, tie_lost = false;
    beam_search<IS_L2, R, NW>(team, g.n, layer0, g.m0, sq, best, tied, seen, over, tie_lost, n_dist, n_exp, g.links0);
    if (tie_lost && !over) n_tie_lost += 1;
    if (lane == 0) overflow[qi] = over ? 1 : 0;
    if (over) {
      n_over += 1;
      n_dist = n_dist0;
      n_exp = n_exp0;
    } else {
      const int found = min(best.filled(), k);
      fv_neighbor* dst = out + qsrc * size_t(k);
      best.each([&](int e, u64 b) {
        if (e < k) dst[e] = fv_neighbor{beam_id(b), beam_distance(b)};
      });
      for (int e = found + lane; e < k; e += 32) dst[e] = fv_neighbor{0xFFFFFFFFu, INFINITY};
      if (lane == 0 && counts) counts[qsrc] = uint32_t(found);
    }
    __syncwarp();
  }
  team_dismiss(team);
  if (lane == 0) {
    atomicAdd(work, n_dist);
    atomicAdd(work + 1, n_exp);
    if (n_tie_lost) atomicAdd(work + 2, n_tie_lost);
    if (n_over) atomicAdd(work + 3, n_over);
  }
}

// ------------------------------------------------------------------------------------------------
// host side distances for construction (src/kernels.rs:200-231; same chains as the device code)
static inline float h_hsum8(const float* l) {
  return ((l[0] + l[4]) + (l[2] + l[6])) + ((l[1] + l[5]) + (l[3] + l[7]));
}
static inline float h_distance(int metric, const float* a, const float* b, size_t n) {
  float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  if (metric == FV_L2) {
    for (size_t i = 0; i + 8 <= n; i += 8)
      for (int l = 0; l < 8; l++) {
        const float d = a[i + l] - b[i + l];
        acc[l] = __builtin_fmaf(d, d, acc[l]);
      }
    return h_hsum8(acc);
  }
  for (size_t i = 0; i + 8 <= n; i += 8)
    for (int l = 0; l < 8; l++) acc[l] = __builtin_fmaf(a[i + l], b[i + l], acc[l]);
  return -h_hsum8(acc);
}

struct HNb {
  uint32_t id;
  float d;
};
static inline bool h_less(const HNb& a, const HNb& b) {
  const uint32_t ka = order_bits(a.d), kb = order_bits(b.d);
  return ka != kb ? ka < kb : a.id < b.id;
}

}  // namespace fv

namespace fv {

// upper[node] holds `level` blocks of (m + 1) u32: count then ids.
static inline uint32_t* upper_block(fv_hnsw* h, uint32_t id, size_t layer) { return &h->upper[id][(layer - 1) * (h->m + 1)]; }

static void flatten_upper(const fv_hnsw* h, std::vector<uint32_t>& off, std::vector<uint32_t>& flat) {
  const size_t n = h->n();
  off.assign(n + 1, 0);
  flat.clear();
  for (size_t i = 0; i < n; i++) {
    off[i] = uint32_t(flat.size());
    for (size_t l = 0; l < h->levels[i]; l++) {
      const uint32_t* b = &h->upper[i][l * (h->m + 1)];
      flat.push_back(b[0]);
      flat.insert(flat.end(), b + 1, b + 1 + b[0]);
    }
  }
  off[n] = uint32_t(flat.size());
}

// Smallest and largest value (as order bits), whether all are whole.
__global__ void value_range_kernel(const float* __restrict__ x, size_t n, uint32_t* __restrict__ words) {
  uint32_t lo = 0xFFFFFFFFu, hi = 0u;
  bool whole = true;
  for (size_t i = (blockIdx.x * size_t(blockDim.x) + threadIdx.x) * 4; i < n; i += size_t(gridDim.x) * blockDim.x * 4) {  // (n is a multiple of 8)
    const float4 v = *reinterpret_cast<const float4*>(x + i);
    const float f[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      whole = whole && f[j] == rintf(f[j]) && fabsf(f[j]) <= 65536.f;
      lo = min(lo, order_bits(f[j]));
      hi = max(hi, order_bits(f[j]));
    }
  }
  lo = __reduce_min_sync(FV_FULL, lo);
  hi = __reduce_max_sync(FV_FULL, hi);
  whole = __all_sync(FV_FULL, whole);
  if (lane_id() == 0) {
    atomicMin(words, lo);
    atomicMax(words + 1, hi);
    if (!whole) words[2] = 1u;
  }
}
// one warp per row
__global__ void row_bytes_kernel(const float* __restrict__ x, size_t n, int pd, float lo, uint8_t* __restrict__ out) {
  const size_t row = blockIdx.x * size_t(blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= n) return;
  for (int c = lane_id(); c < row_bytes(pd); c += 32)
    out[row * row_bytes(pd) + c] = c < pd ? uint8_t(x[row * size_t(pd) + c] - lo) : uint8_t(0);
}

// The rows as bytes, where they qualify.  (-0 counts as a whole number: it makes the same distances as 0.)
static int make_bytes(fv_hnsw* h) {
  fv_ctx* ctx = h->ctx;
  h->d_bytes.release();
  const size_t n = h->n();
  if (h->metric != FV_L2 || n == 0) return FV_OK;
  DevBuf words;
  if (words.reserve(16) != FV_OK) return FV_OK;  // (no room: the searches do without)
  const uint32_t init[4] = {0xFFFFFFFFu, 0u, 0u, 0u};
  uint32_t got[4];
  FV_CUDA(cudaMemcpyAsync(words.p, init, sizeof(init), cudaMemcpyHostToDevice, ctx->stream));
  value_range_kernel<<<ctx->sm_count * 4, 256, 0, ctx->stream>>>(h->d_data.as<float>(), n * h->pd, words.as<uint32_t>());
  FV_CUDA(cudaGetLastError());
  FV_CUDA(cudaMemcpyAsync(got, words.p, sizeof(got), cudaMemcpyDeviceToHost, ctx->stream));
  FV_CUDA(cudaStreamSynchronize(ctx->stream));
  words.release();
  if (got[2]) return FV_OK;
  const float lo = order_bits_to_float(got[0]), hi = order_bits_to_float(got[1]);
  // queries may lie a little beyond the rows' values: bytes above 0 or -128 where those hold all rows
  h->byte_lo = lo >= 0.f && hi <= 255.f ? 0.f : lo >= -128.f && hi <= 127.f ? -128.f : lo;
  if (!(hi - h->byte_lo <= 255.f) || double(h->pd) * 255.0 * 255.0 >= 16777216.0) return FV_OK;
  if (h->d_bytes.reserve(n * size_t(row_bytes(int(h->pd)))) != FV_OK) return FV_OK;
  row_bytes_kernel<<<unsigned((n + 7) / 8), 256, 0, ctx->stream>>>(h->d_data.as<float>(), n, int(h->pd), h->byte_lo, h->d_bytes.as<uint8_t>());
  FV_CUDA(cudaGetLastError());
  return FV_OK;
}

int upload_graph(fv_hnsw* h, bool with_data) {
  fv_ctx* ctx = h->ctx;
  std::vector<uint32_t> off, flat;
  flatten_upper(h, off, flat);
  if (with_data) FV_TRY(h->d_data.reserve(h->data.size() * 4 + 16));
  FV_TRY(h->d_links0.reserve(h->links0.size() * 4 + 16));
  FV_TRY(h->d_upper_off.reserve(off.size() * 4 + 16));
  FV_TRY(h->d_upper_flat.reserve(flat.size() * 4 + 16));
  if (with_data)
    FV_CUDA(cudaMemcpyAsync(h->d_data.p, h->data.data(), h->data.size() * 4, cudaMemcpyHostToDevice, ctx->stream));
  FV_CUDA(cudaMemcpyAsync(h->d_links0.p, h->links0.data(), h->links0.size() * 4, cudaMemcpyHostToDevice, ctx->stream));
  FV_CUDA(cudaMemcpyAsync(h->d_upper_off.p, off.data(), off.size() * 4, cudaMemcpyHostToDevice, ctx->stream));
  if (!flat.empty())
    FV_CUDA(cudaMemcpyAsync(h->d_upper_flat.p, flat.data(), flat.size() * 4, cudaMemcpyHostToDevice, ctx->stream));
  FV_TRY(make_bytes(h));
  FV_CUDA(cudaStreamSynchronize(ctx->stream));
  return FV_OK;
}

// ---- construction on the host cores (hnsw.rs:85-129, :230-320)
struct Builder {
  fv_hnsw* h;
  std::unique_ptr<std::mutex[]> locks;
  std::mutex entry_lock;
  const float* vec(uint32_t id) const { return &h->data[size_t(id) * h->pd]; }
  float dist(const float* q, uint32_t id) const { return h_distance(h->metric, q, vec(id), h->pd); }

  void neighbors(uint32_t id, size_t layer, bool locked, std::vector<uint32_t>& out) {
    out.clear();
    std::unique_lock<std::mutex> g;
    if (locked) g = std::unique_lock<std::mutex>(locks[id]);
    const uint32_t* b = layer == 0 ? &h->links0[size_t(id) * (h->m0 + 1)] : upper_block(h, id, layer);
    out.assign(b + 1, b + 1 + b[0]);
  }
  void set_neighbors(uint32_t id, size_t layer, const std::vector<uint32_t>& list) {
    uint32_t* b = layer == 0 ? &h->links0[size_t(id) * (h->m0 + 1)] : upper_block(h, id, layer);
    for (size_t i = 0; i < list.size(); i++) b[1 + i] = list[i];
    b[0] = uint32_t(list.size());
  }

  struct Visited {
    std::vector<uint32_t> v;
    uint32_t stamp = 0;
  };

  std::vector<HNb> search_layer(const float* q, const std::vector<HNb>& entry, size_t ef, size_t layer, Visited& vs) {
    if (vs.v.size() < h->n()) {
      vs.v.assign(h->n(), 0);
      vs.stamp = 0;
    }
    if (++vs.stamp == 0) {
      std::fill(vs.v.begin(), vs.v.end(), 0);
      vs.stamp = 1;
    }
    const uint32_t stamp = vs.stamp;
    auto gt = [](const HNb& a, const HNb& b) { return h_less(b, a); };
    std::vector<HNb> cand, best;  // cand: min-heap, best: max-heap
    for (const HNb& e : entry) {
      vs.v[e.id] = stamp;
      cand.push_back(e);
      std::push_heap(cand.begin(), cand.end(), gt);
      best.push_back(e);
      std::push_heap(best.begin(), best.end(), h_less);
    }
    while (best.size() > ef) {
      std::pop_heap(best.begin(), best.end(), h_less);
      best.pop_back();
    }
    std::vector<uint32_t> nb;
    while (!cand.empty()) {
      std::pop_heap(cand.begin(), cand.end(), gt);
      const HNb c = cand.back();
      cand.pop_back();
      if (best.size() >= ef && c.d > best.front().d) break;
      neighbors(c.id, layer, true, nb);
      for (uint32_t x : nb) {
        if (vs.v[x] == stamp) continue;
        vs.v[x] = stamp;
        const float d = dist(q, x);
        if (best.size() < ef || d < best.front().d) {
          const HNb nn{x, d};
          cand.push_back(nn);
          std::push_heap(cand.begin(), cand.end(), gt);
          best.push_back(nn);
          std::push_heap(best.begin(), best.end(), h_less);
          if (best.size() > ef) {
            std::pop_heap(best.begin(), best.end(), h_less);
            best.pop_back();
          }
        }
      }
    }
    std::sort_heap(best.begin(), best.end(), h_less);
    return best;
  }

  std::vector<uint32_t> select(const std::vector<HNb>& cands, size_t mm) const {
    std::vector<uint32_t> out;
    for (const HNb& c : cands) {
      if (out.size() >= mm) break;
      const float* cv = vec(c.id);
      bool keep = true;
      for (uint32_t s : out)
        if (!(h_distance(h->metric, cv, vec(s), h->pd) > c.d)) {
          keep = false;
          break;
        }
      if (keep) out.push_back(c.id);
    }
    return out;
  }

  void add_links(uint32_t id, size_t layer, const std::vector<uint32_t>& nw, size_t cap) {
    std::lock_guard<std::mutex> g(locks[id]);
    std::vector<uint32_t> list;
    neighbors(id, layer, false, list);
    const size_t before = list.size();
    for (uint32_t x : nw)
      if (x != id && std::find(list.begin(), list.end(), x) == list.end()) list.push_back(x);
    if (list.size() == before) return;
    if (list.size() > cap) {
      std::vector<HNb> c;
      for (uint32_t x : list) c.push_back({x, h_distance(h->metric, vec(id), vec(x), h->pd)});
      std::sort(c.begin(), c.end(), h_less);
      list = select(c, cap);
    }
    set_neighbors(id, layer, list);
  }

  void insert(uint32_t id, size_t ef, Visited& vs) {
    std::vector<float> q(vec(id), vec(id) + h->pd);
    const size_t level = h->levels[id];
    uint32_t e0;
    size_t tp;
    {
      std::lock_guard<std::mutex> g(entry_lock);
      e0 = h->ep;
      tp = h->top;
    }
    HNb cur{e0, dist(q.data(), e0)};
    std::vector<uint32_t> nb;
    for (size_t layer = tp; layer > level; layer--) {
      bool changed = true;
      while (changed) {
        changed = false;
        neighbors(cur.id, layer, true, nb);
        for (uint32_t x : nb) {
          const float d = dist(q.data(), x);
          if (d < cur.d) {
            cur = {x, d};
            changed = true;
          }
        }
      }
    }
    std::vector<HNb> entry{cur};
    for (size_t layer = std::min(level, tp) + 1; layer-- > 0;) {
      auto found = search_layer(q.data(), entry, ef, layer, vs);
      const size_t cap = layer == 0 ? h->m0 : h->m;
      const auto chosen = select(found, cap);
      add_links(id, layer, chosen, cap);
      const std::vector<uint32_t> me{id};
      for (uint32_t x : chosen) add_links(x, layer, me, cap);
      entry = std::move(found);
    }
    if (level > tp) {
      std::lock_guard<std::mutex> g(entry_lock);
      if (level > h->top) {
        h->ep = id;
        h->top = level;
      }
    }
  }
};

// ---- launch shape of a search
// A team of TEAM_WARPS warps per query while the batch is small, a warp per query beyond (team_searches_per_sm).  Measured
// (us a batch, team / warp): 100,000 x 128, ef 64: 1 query 186 / 345, 592 queries 372 / 668, 2,368 queries 926 / 967; ef
// 256: 592 queries 1,274 / 1,829, 2,368 queries 3,342 / 2,382; 50,000 x 32, ef 64: 592 queries 320 / 369, 2,368 queries
// 766 / 390.
typedef void (*SearchKernel)(HnswDev, const float*, const uint32_t*, size_t, int, int, int, int, uint32_t*, fv_neighbor*,
                             uint32_t*, uint32_t*, unsigned long long*, unsigned int*);
struct SearchShape {
  SearchKernel kern;
  size_t blocks, searchers, smem;  // searchers per block
  int threads, sbits;
};

template <bool IS_L2, bool BYTES, int NW>
static SearchKernel pick_search_of(int R) {
  switch (R) {
    case 1: return hnsw_search_kernel<IS_L2, BYTES, 1, NW>;
    case 2: return hnsw_search_kernel<IS_L2, BYTES, 2, NW>;
    case 4: return hnsw_search_kernel<IS_L2, BYTES, 4, NW>;
    case 8: return hnsw_search_kernel<IS_L2, BYTES, 8, NW>;
    default:
      if constexpr (NW == SCOUT_WARPS) return nullptr;  // (scouts_pay)
      else return hnsw_search_kernel<IS_L2, BYTES, 0, NW>;
  }
}
template <int NW>
static SearchKernel pick_search(bool is_l2, bool bytes, int R) {
  return bytes ? pick_search_of<true, true, NW>(R) : is_l2 ? pick_search_of<true, false, NW>(R) : pick_search_of<false, false, NW>(R);
}

static int search_shape(fv_ctx* ctx, bool is_l2, bool bytes, size_t n, int pd, int m0, int ef, size_t active, SearchShape* s) {
  const int R = ef <= 32 ? 1 : ef <= 64 ? 2 : ef <= 128 ? 4 : ef <= 256 ? 8 : 0;
  const size_t budget = std::min<size_t>(ctx->smem_optin, 200 * 1024);
  auto bytes_of = [&](int sbits, int nw) { return R == 0 ? search_smem<0>(pd, bytes, m0, ef, sbits, nw) : search_smem<1>(pd, bytes, m0, ef, sbits, nw); };
  const bool team = active <= size_t(ctx->sm_count) * team_searches_per_sm(pd, m0, ef);
  // (rows too long for a scouting team's slots beside the smallest first part of the visited set: a team of eight)
  const bool scouts = team && scouts_pay(ctx->sm_count, pd, m0, ef, active) && bytes_of(7, SCOUT_WARPS) <= ctx->smem_optin;
  s->sbits = team ? visit_sbits(ef) : visit_sbits_single(n, ef);
  size_t per = bytes_of(s->sbits, scouts ? SCOUT_WARPS : team ? TEAM_WARPS : 1);
  int W = 8;
  if (team) {
    s->searchers = 1;
    s->threads = (scouts ? SCOUT_WARPS : TEAM_WARPS) * 32;
    while (s->sbits > 7 && per > budget) {
      per -= size_t(2) << s->sbits;
      s->sbits--;
    }
  } else {
    while (W > 1 && per * W > budget / 2) W >>= 1;
    s->searchers = size_t(W);
    s->threads = W * 32;
  }
  s->smem = per * s->searchers;
  if (s->smem > ctx->smem_optin) return fail(FV_ERR_UNSUPPORTED, "dimension and ef too large for shared memory");
  const size_t by_warps = scouts ? team_blocks(SCOUT_WARPS) : 8 * SEARCH_BLOCKS_PER_SM / (s->threads / 32);
  const size_t per_sm = std::max<size_t>(1, std::min(size_t(227 * 1024) / (s->smem + 1024), by_warps));
  s->blocks = std::min<size_t>((active + s->searchers - 1) / s->searchers, size_t(ctx->sm_count) * per_sm);
  s->kern = scouts ? pick_search<SCOUT_WARPS>(is_l2, bytes, R) : team ? pick_search<TEAM_WARPS>(is_l2, bytes, R) : pick_search<1>(is_l2, bytes, R);
  FV_TRY(allow_smem(ctx, s->kern, s->smem));
  return FV_OK;
}

// scratch slots: 0 padded queries, 1 keys, 5 overflow flags, 6 retry ids, 7 global tables
// `h_out`, `h_counts` (may be null): bring the results out to the host as well (d_counts lies directly behind d_out then)
static int hnsw_search_dev(fv_hnsw* h, const float* d_queries, size_t nq, size_t k, size_t ef_in, fv_neighbor* d_out,
                           uint32_t* d_counts, fv_neighbor* h_out = nullptr, uint32_t* h_counts = nullptr) {
  fv_ctx* ctx = h->ctx;
  FV_TRY(pin_ready(ctx));
  if (k == 0) return fail(FV_ERR_ARG, "k must be at least 1");
  if (nq == 0) return FV_OK;
  ctx->stats = fv_stats{};
  const size_t n = h->n();
  if (n == 0) {  // hnsw.rs:324-326: an empty index finds nothing
    FV_TRY(ctx->scratch[1].reserve(nq * k * sizeof(u64)));
    u64* keys = ctx->scratch[1].as<u64>();
    FV_CUDA(cudaMemsetAsync(keys, 0xFF, nq * k * sizeof(u64), ctx->stream));
    FV_TRY(keys_to_neighbors(ctx, keys, nq, int(k), int(k), d_out, d_counts));
    if (h_out) return fetch_results(ctx, d_out, nq, k, h_out, h_counts);
    FV_CUDA(cudaStreamSynchronize(ctx->stream));
    return FV_OK;
  }
  const size_t ef = std::max(ef_in, k);
  if (ef > 4096) return fail(FV_ERR_UNSUPPORTED, "ef above 4096 is not supported");
  if (n > 0x7FFFFFFFull) return fail(FV_ERR_UNSUPPORTED, "more than 2^31 nodes");
  stage_begin(ctx);
  const int pd = int(h->pd);
  const float* q = d_queries;
  if (h->pd != h->dim) {
    FV_TRY(ctx->scratch[0].reserve(nq * size_t(pd) * sizeof(float)));
    FV_TRY(upload_padded(ctx, d_queries, true, nq, h->dim, h->pd, ctx->scratch[0].as<float>()));
    q = ctx->scratch[0].as<float>();
  }
  FV_TRY(ctx->scratch[5].reserve(nq * sizeof(uint32_t)));
  uint32_t* d_over = ctx->scratch[5].as<uint32_t>();
  // words 16..23: the four counters; word 24: the next query
  unsigned long long* d_work = reinterpret_cast<unsigned long long*>(ctx->d_flags + 16);
  unsigned int* d_next = reinterpret_cast<unsigned int*>(ctx->d_flags + 24);
  HnswDev g{};
  g.data = h->d_data.as<float>();
  g.bytes = h->d_bytes.as<uint8_t>();
  g.byte_lo = h->byte_lo;
  g.links0 = h->d_links0.as<uint32_t>();
  g.upper_off = h->d_upper_off.as<uint32_t>();
  g.upper_flat = h->d_upper_flat.as<uint32_t>();
  g.pd = pd;
  g.m0 = int(h->m0);
  g.metric = h->metric;
  g.top = int(h->top);
  g.ep = h->ep;
  g.n = n;
  // The visited set's part in global memory: 48 slots per entry of the beam to begin with, one per link of a node where
  // that is more and they stay within 8,192, and twice as many (four times with more than 48 links) within 4,096; it may
  // fill to one half.  The overflow path quadruples it for the queries that need more.  A second launch, for however few,
  // takes as long as the search of one query: 1,776 queries of 50,000 x 96, m = 48, ef 10 285 us, 568 with one of them run
  // again.
  int log2slots = 11;
  const size_t want = ef * (h->m0 > 48 && ef * h->m0 <= 8192 ? h->m0 : 48), roomy = want * (h->m0 > 48 ? 4 : 2);
  while ((size_t(1) << log2slots) < (roomy <= 4096 ? roomy : want) && log2slots < 26) log2slots++;
  const uint32_t* d_qids = nullptr;
  size_t active = nq;
  std::vector<uint32_t> h_over, retry;
  const unsigned long long* wk = reinterpret_cast<const unsigned long long*>(ctx->h_pin);
  unsigned long long total[3] = {0, 0, 0};
  // the results follow the counters out at once: nearly always the first attempt is the last
  const bool early = h_out && results_fit_pin(nq, k);
  bool fetched = false;
  for (int attempt = 0; attempt < 8 && active; ++attempt) {
    SearchShape sh{};
    FV_TRY(search_shape(ctx, h->metric == FV_L2, g.bytes != nullptr, n, pd, int(h->m0), int(ef), active, &sh));
    const size_t tables = sh.blocks * sh.searchers;
    FV_TRY(ctx->scratch[7].reserve((tables << log2slots) * 4));
    FV_CUDA(cudaMemsetAsync(d_work, 0, 4 * sizeof(unsigned long long) + sizeof(unsigned int), ctx->stream));
    sh.kern<<<unsigned(sh.blocks), sh.threads, sh.smem, ctx->stream>>>(g, q, d_qids, active, int(k), int(ef), sh.sbits, log2slots,
                                                                       ctx->scratch[7].as<uint32_t>(), d_out, d_counts, d_over,
                                                                       d_work, d_next);
    ctx->stats.launches++;
    FV_CUDA(cudaGetLastError());
    FV_CUDA(cudaMemcpyAsync(ctx->h_pin, d_work, 4 * sizeof(*wk), cudaMemcpyDeviceToHost, ctx->stream));
    if (early)
      FV_CUDA(cudaMemcpyAsync(ctx->h_pin + FV_PIN_RESULTS, d_out, nq * k * sizeof(fv_neighbor) + nq * sizeof(uint32_t),
                              cudaMemcpyDeviceToHost, ctx->stream));
    FV_CUDA(cudaStreamSynchronize(ctx->stream));
    for (int i = 0; i < 3; ++i) total[i] += wk[i];
    if (wk[3] == 0) {
      active = 0;
      fetched = early;
      break;
    }
    h_over.resize(active);
    FV_CUDA(cudaMemcpyAsync(h_over.data(), d_over, active * sizeof(uint32_t), cudaMemcpyDeviceToHost, ctx->stream));
    FV_CUDA(cudaStreamSynchronize(ctx->stream));
    std::vector<uint32_t> next;
    for (size_t i = 0; i < active; i++)
      if (h_over[i]) next.push_back(d_qids ? retry[i] : uint32_t(i));
    ctx->stats.regrown += next.size();
    retry = next;
    active = retry.size();
    FV_TRY(ctx->scratch[6].reserve(active * sizeof(uint32_t) + 4));
    FV_CUDA(cudaMemcpyAsync(ctx->scratch[6].p, retry.data(), active * sizeof(uint32_t), cudaMemcpyHostToDevice,
                            ctx->stream));
    d_qids = ctx->scratch[6].as<uint32_t>();
    log2slots = std::min(log2slots + 2, 27);
  }
  if (active) return fail(FV_ERR_OVERFLOW, "visited table overflow after regrowing");
  stage_mark(ctx);
  ctx->stats.dist_evals = total[0];
  ctx->stats.expansions = total[1];
  ctx->stats.uncertified = total[2];  // queries whose list of tied, pushed-out entries overflowed (see TIED_CAP)
  if (h_out) FV_TRY(fetch_results(ctx, d_out, nq, k, h_out, h_counts, fetched));
  if (ctx->timing) FV_CUDA(cudaStreamSynchronize(ctx->stream));  // the mark was recorded after the last wait
  stage_end(ctx);
  return bounds_report_hnsw();
}

int hnsw_new(fv_ctx* ctx, int metric, uint32_t dim, const float* vectors, size_t n, const fv_hnsw_params* p,
             std::unique_ptr<fv_hnsw>& out) {
  if (!ctx || !p || (!vectors && n) || dim == 0 || (metric != FV_L2 && metric != FV_INNER_PRODUCT))
    return fail(FV_ERR_ARG, "hnsw build: bad argument");
  if (p->m < 2 || p->m > 64) return fail(FV_ERR_UNSUPPORTED, "m must be in 2..64");
  auto h = std::unique_ptr<fv_hnsw>(new fv_hnsw());
  h->ctx = ctx;
  ctx_retain(ctx);
  h->metric = metric;
  h->dim = dim;
  h->pd = uint32_t(padded(dim));
  h->m = p->m;
  h->m0 = 2 * p->m;
  h->data.assign(n * size_t(h->pd), 0.f);
  for (size_t i = 0; i < n; i++) std::memcpy(&h->data[i * h->pd], vectors + i * size_t(dim), size_t(dim) * sizeof(float));
  // levels: hnsw.rs:88-94, drawn in node order from one generator
  const double ml = 1.0 / std::log(double(p->m));
  uint64_t s = (p->seed * 0x9E3779B97F4A7C15ull) | 1ull;
  h->levels.resize(n);
  for (size_t i = 0; i < n; i++) {
    s ^= s >> 12;
    s ^= s << 25;
    s ^= s >> 27;
    const double u = double((s * 0x2545F4914F6CDD1Dull) >> 11) / double(1ull << 53);
    const double v = -std::log(1.0 - u) * ml;
    const size_t lv = (v != v || v <= 0.0) ? 0 : (v >= 1.8e19 ? size_t(-1) : size_t(v));
    h->levels[i] = uint8_t(std::min<size_t>(lv, 15));
  }
  h->upper.resize(n);
  for (size_t i = 0; i < n; i++) h->upper[i].assign(size_t(h->levels[i]) * (h->m + 1), 0);
  h->links0.assign(n * (h->m0 + 1), 0);
  h->ep = 0;
  h->top = n ? h->levels[0] : 0;
  out = std::move(h);
  return FV_OK;
}

}  // namespace fv

extern "C" {

int fv_hnsw_build(fv_ctx* ctx, int metric, uint32_t dim, const float* vectors, size_t n, const fv_hnsw_params* p,
                  int threads, fv_hnsw** out) {
  if (!out) return fv::fail(FV_ERR_ARG, "fv_hnsw_build: bad argument");
  std::unique_ptr<fv_hnsw> h;
  FV_TRY(fv::hnsw_new(ctx, metric, dim, vectors, n, p, h));
  if (n > 1) {
    fv::Builder b;
    b.h = h.get();
    b.locks.reset(new std::mutex[n]);
    std::atomic<size_t> next{1};
    const int nt = std::max(1, threads);
    auto work = [&]() {
      fv::Builder::Visited vs;
      for (;;) {
        const size_t i = next.fetch_add(1, std::memory_order_relaxed);
        if (i >= n) break;
        b.insert(uint32_t(i), p->ef_construction, vs);
      }
    };
    std::vector<std::thread> th;
    for (int t = 1; t < nt; t++) th.emplace_back(work);
    work();
    for (auto& t : th) t.join();
  }
  fv::CtxGuard g(ctx);
  FV_TRY(fv::upload_graph(h.get()));
  *out = h.release();
  return FV_OK;
}

void fv_hnsw_free(fv_hnsw* ix) {
  if (!ix) return;
  fv_ctx* ctx = ix->ctx;
  {
    fv::CtxGuard g(ctx);
    cudaStreamSynchronize(ctx->stream);
    ix->ctx = nullptr;  // the destructor must not drop the reference while the lock is held
    delete ix;
  }
  fv::ctx_release(ctx);  // may destroy the context
}

size_t fv_hnsw_len(const fv_hnsw* ix) { return ix ? ix->n() : 0; }
uint32_t fv_hnsw_dim(const fv_hnsw* ix) { return ix ? ix->dim : 0; }
int fv_hnsw_metric(const fv_hnsw* ix) { return ix ? ix->metric : -1; }

size_t fv_hnsw_reachable(const fv_hnsw* ix) {  // hnsw.rs:367-385
  if (!ix || ix->n() == 0) return 0;
  std::vector<char> seen(ix->n(), 0);
  std::vector<uint32_t> stack{ix->ep};
  seen[ix->ep] = 1;
  size_t count = 0;
  while (!stack.empty()) {
    const uint32_t x = stack.back();
    stack.pop_back();
    count++;
    const uint32_t* b = &ix->links0[size_t(x) * (ix->m0 + 1)];
    for (uint32_t i = 0; i < b[0]; i++) {
      const uint32_t y = b[1 + i];
      if (!seen[y]) {
        seen[y] = 1;
        stack.push_back(y);
      }
    }
  }
  return count;
}

double fv_hnsw_mean_degree(const fv_hnsw* ix) {  // hnsw.rs:388-393
  if (!ix) return 0.0;
  uint64_t total = 0;
  for (size_t i = 0; i < ix->n(); i++) total += ix->links0[i * (ix->m0 + 1)];
  return double(total) / double(std::max<size_t>(ix->n(), 1));
}

int fv_hnsw_search_batch_dev(fv_hnsw* ix, const float* d_queries, size_t nq, size_t k, size_t ef, fv_neighbor* d_out,
                             uint32_t* d_counts) {
  if (!ix || (nq && (!d_queries || !d_out))) return fv::fail(FV_ERR_ARG, "fv_hnsw_search_batch: null argument");
  fv::CtxGuard g(ix->ctx);
  return fv::hnsw_search_dev(ix, d_queries, nq, k, ef, d_out, d_counts);
}

int fv_hnsw_search_batch(fv_hnsw* ix, const float* queries, size_t nq, size_t k, size_t ef, fv_neighbor* out,
                         uint32_t* counts) {
  if (!ix || (nq && (!queries || !out))) return fv::fail(FV_ERR_ARG, "fv_hnsw_search_batch: null argument");
  if (nq == 0) return FV_OK;
  fv_ctx* ctx = ix->ctx;
  fv::CtxGuard g(ctx);
  const size_t qbytes = nq * size_t(ix->dim) * sizeof(float), obytes = nq * k * sizeof(fv_neighbor);
  FV_TRY(ctx->scratch[10].reserve(qbytes));
  FV_TRY(ctx->scratch[11].reserve(obytes + nq * sizeof(uint32_t)));
  float* dq = ctx->scratch[10].as<float>();
  fv_neighbor* dout = ctx->scratch[11].as<fv_neighbor>();
  uint32_t* dc = reinterpret_cast<uint32_t*>(ctx->scratch[11].as<unsigned char>() + obytes);
  FV_CUDA(cudaMemcpyAsync(dq, queries, qbytes, cudaMemcpyHostToDevice, ctx->stream));
  return fv::hnsw_search_dev(ix, dq, nq, k, ef, dout, dc, out, counts);
}

int fv_hnsw_search(fv_hnsw* ix, const float* query, size_t k, size_t ef, fv_neighbor* out, uint32_t* count) {
  return fv_hnsw_search_batch(ix, query, 1, k, ef, out, count);
}

// ---- FLHNSW01 files (hnsw.rs:395-466)
size_t fv_hnsw_save_size(const fv_hnsw* ix) {
  if (!ix) return 0;
  size_t flat = 0;
  for (size_t i = 0; i < ix->n(); i++)
    for (size_t l = 0; l < ix->levels[i]; l++) flat += 1 + ix->upper[i][l * (ix->m + 1)];
  return 8 + 5 * 4 + (8 + ix->levels.size()) + (8 + ix->links0.size() * 4) + (8 + flat * 4) + (8 + ix->data.size() * 4);
}

int fv_hnsw_save(const fv_hnsw* ix, uint8_t* buf, size_t cap, size_t* written) {
  if (!ix || !buf) return fv::fail(FV_ERR_ARG, "fv_hnsw_save: null argument");
  if (cap < fv_hnsw_save_size(ix)) return fv::fail(FV_ERR_ARG, "fv_hnsw_save: buffer too small");
  uint8_t* w = buf;
  auto raw = [&](const void* p, size_t n) {
    if (n) std::memcpy(w, p, n);
    w += n;
  };
  auto u32 = [&](uint32_t v) { raw(&v, 4); };
  auto u64w = [&](uint64_t v) { raw(&v, 8); };
  raw("FLHNSW01", 8);
  u32(uint32_t(ix->metric));
  u32(ix->dim);
  u32(uint32_t(ix->m));
  u32(ix->ep);
  u32(uint32_t(ix->top));
  u64w(ix->levels.size());
  raw(ix->levels.data(), ix->levels.size());
  u64w(ix->links0.size());
  raw(ix->links0.data(), ix->links0.size() * 4);
  std::vector<uint32_t> off, flat;
  fv::flatten_upper(ix, off, flat);
  u64w(flat.size());
  raw(flat.data(), flat.size() * 4);
  u64w(ix->data.size());
  raw(ix->data.data(), ix->data.size() * 4);
  if (written) *written = size_t(w - buf);
  return FV_OK;
}

int fv_hnsw_load(fv_ctx* ctx, const uint8_t* bytes, size_t len, fv_hnsw** out) {
  if (!ctx || !bytes || !out) return fv::fail(FV_ERR_ARG, "fv_hnsw_load: null argument");
  if (len < 8 || std::memcmp(bytes, "FLHNSW01", 8) != 0) return fv::fail(FV_ERR_FILE, "not an HNSW index file");
  size_t i = 8;
  bool ok = true;
  auto take = [&](size_t n) -> const uint8_t* {
    if (!ok || n > len - i) {
      ok = false;
      return nullptr;
    }
    const uint8_t* p = bytes + i;
    i += n;
    return p;
  };
  auto u32 = [&]() {
    uint32_t v = 0;
    if (auto p = take(4)) std::memcpy(&v, p, 4);
    return v;
  };
  auto span = [&](size_t elem, size_t* count) -> const uint8_t* {
    uint64_t n = 0;
    if (auto p = take(8)) std::memcpy(&n, p, 8);
    if (!ok || n > (len - i) / elem) {
      ok = false;
      return nullptr;
    }
    *count = size_t(n);
    return take(size_t(n) * elem);
  };
  const char* trunc = "index file is truncated";
  auto h = std::unique_ptr<fv_hnsw>(new fv_hnsw());
  h->ctx = ctx;
  fv::ctx_retain(ctx);
  const uint32_t mc = u32();
  h->dim = u32();
  h->m = u32();
  h->ep = u32();
  h->top = u32();
  if (!ok) return fv::fail(FV_ERR_FILE, trunc);
  if ((mc & 0xFF) > 1) return fv::fail(FV_ERR_FILE, "bad metric");
  h->metric = int(mc & 0xFF);
  size_t nl = 0, nk = 0, nf = 0, nd = 0;
  const uint8_t* pl = span(1, &nl);
  const uint8_t* pk = span(4, &nk);
  const uint8_t* pf = span(4, &nf);
  const uint8_t* pdat = span(4, &nd);
  if (!ok) return fv::fail(FV_ERR_FILE, trunc);
  h->levels.assign(pl, pl + nl);
  std::vector<uint32_t> flat(nf);
  if (nf) std::memcpy(flat.data(), pf, nf * 4);
  const size_t n = nl;
  h->pd = uint32_t(fv::padded(h->dim));
  h->m0 = 2 * h->m;
  if (h->dim == 0 || h->m == 0) return fv::fail(FV_ERR_FILE, "index file sizes do not match");
  h->upper.resize(n);
  size_t at = 0;
  for (size_t node = 0; node < n; node++) {
    h->upper[node].assign(size_t(h->levels[node]) * (h->m + 1), 0);
    for (size_t l = 0; l < h->levels[node]; l++) {
      if (at >= nf) return fv::fail(FV_ERR_FILE, "truncated links");
      const size_t c = flat[at];
      if (at + 1 + c > nf) return fv::fail(FV_ERR_FILE, "truncated links");
      if (c > h->m) return fv::fail(FV_ERR_FILE, "index file sizes do not match");
      uint32_t* b = &h->upper[node][l * (h->m + 1)];
      b[0] = uint32_t(c);
      for (size_t t = 0; t < c; t++) b[1 + t] = flat[at + 1 + t];
      at += 1 + c;
    }
  }
  if (nk != n * (2 * h->m + 1) || nd != n * size_t(h->pd)) return fv::fail(FV_ERR_FILE, "index file sizes do not match");
  h->links0.resize(nk);
  if (nk) std::memcpy(h->links0.data(), pk, nk * 4);
  h->data.resize(nd);
  if (nd) std::memcpy(h->data.data(), pdat, nd * 4);
  // a damaged file must not send the kernel out of bounds
  if (n && (h->ep >= n || h->top > 15 || h->levels[h->ep] < h->top)) return fv::fail(FV_ERR_FILE, "bad entry point");
  for (size_t node = 0; node < n; node++) {
    const uint32_t* b = &h->links0[node * (h->m0 + 1)];
    if (b[0] > h->m0) return fv::fail(FV_ERR_FILE, "bad link count");
    for (uint32_t t = 0; t < b[0]; t++)
      if (b[1 + t] >= n) return fv::fail(FV_ERR_FILE, "link out of range");
    for (size_t l = 0; l < h->levels[node]; l++) {
      const uint32_t* u = &h->upper[node][l * (h->m + 1)];
      for (uint32_t t = 0; t < u[0]; t++)
        if (u[1 + t] >= n || h->levels[u[1 + t]] < l + 1) return fv::fail(FV_ERR_FILE, "link out of range");
    }
  }
  fv::CtxGuard g(ctx);
  FV_TRY(fv::upload_graph(h.get()));
  *out = h.release();
  return FV_OK;
}

}  // extern "C"
