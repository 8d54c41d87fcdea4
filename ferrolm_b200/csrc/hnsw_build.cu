// Hnsw construction on the GPU (src/vector/hnsw.rs:85-129 build, :244-290 insert, :230-242 select, :294-320
// add_links), batch-synchronous.
//
// The reference hands nodes out in id order to the pool's threads; what each thread's search sees of the others'
// half-made links depends on timing.  Here nodes go in in id order in BATCHES:
//   1. hnsw_insert_kernel, a warp per node of the batch (a team of eight or nine in batches of up to 16 nodes per SM): the
//      greedy descent and the per-layer search_layer of insert() against the graph as it stood when the batch began
//      (no node of the batch is visible to another), then select() over what was found; the node's own lists are
//      written and one edge (target, layer, source) per chosen neighbour is pushed on a chain headed at (target, layer);
//   2. hnsw_link_kernel, one warp per (target, layer) chain: add_links(target, layer, [source]) for the chain's
//      sources in ascending id, that is in the order a single thread would have reached them.
// Between batches the entry point moves as in hnsw.rs:285-289; a node above the current top layer ends its batch
// before it and goes in alone.  The result does not depend on timing: the same input gives the same graph, and with
// batches of one node it is byte for byte the graph of the reference's single-thread build.
//
// A batch holds at most max_batch nodes and at most 1/divisor of the nodes already in, so that the early graph (the
// backbone every later search walks) is built nearly node by node.
#include <algorithm>
#include <cstring>

#include "hnsw.cuh"

FV_BOUNDS_TU(hnsw_build)

namespace fv {

static constexpr uint32_t NIL = 0xFFFFFFFFu;
static constexpr int BUILD_BLOCKS_PER_SM = 3;  // of 256 threads: 24 warps per SM at up to 80 registers
static constexpr int TEAM_INSERTS_PER_SM = 16;  // batches up to this many nodes per SM are inserted by teams
static constexpr int SRC_CAP = 128;  // sources of one chain sorted in shared memory; longer chains are walked again per source

struct Edge {
  uint32_t tgt, src, blk, next;  // blk: the chain's head slot; next: the edge pushed before this one on the same chain
};

struct BuildDev {
  const float* data;
  uint32_t* links0;         // n x (m0 + 1): count, ids
  uint32_t* up;             // upper layers: blocks of (m + 1) words, per node its layers 1..level
  const uint32_t* up_blk;   // n + 1: first block of each node
  const uint8_t* levels;
  int pd, m, m0;
  uint32_t n;
};

__device__ __forceinline__ uint32_t* link_row(const BuildDev& g, uint32_t x, int layer) {
  return layer == 0 ? g.links0 + size_t(x) * (g.m0 + 1) : g.up + (size_t(g.up_blk[x]) + layer - 1) * (g.m + 1);
}
__device__ __forceinline__ uint32_t head_slot(const BuildDev& g, uint32_t x, int layer) {
  return layer == 0 ? x : g.n + g.up_blk[x] + uint32_t(layer - 1);
}

// rows of one run of distances: what a search's beam can hold, up to SELECT_RUN
static constexpr int SELECT_RUN = 512;
__host__ __device__ __forceinline__ int run_rows(int ncand) { return ncand < SELECT_RUN ? (ncand + 31) & ~31 : SELECT_RUN; }

// select (hnsw.rs:230-242): from candidates sorted nearest first (keys: order bits of the distance above, id at
// `id_shift` below), keep those farther from every kept one than from the base, up to cap.  Worked from the kept
// side: the first candidate nobody has ruled out is kept, and its distances to all the ones still standing behind it
// (one run, team_eval) rule out those nearer to it than to the base.  A distance has the same bits from either end, so
// the choice is the reference's.  (Candidate by candidate, as it was, each of up to ef candidates took a load of its
// row and a run of at most 32 distances: 200 dependent steps where there are now as many as links kept.)
// `cand`, `gone` (a bit per candidate) and `sc` (the kept row) are shared memory of the warp; the runs of `t` hold
// run_rows(ncand) rows.
// Returns the number kept (ids in sel[]).
template <bool IS_L2, int NW>
__device__ __forceinline__ int select_links(const BuildDev& g, const Team<NW>& t, const u64* cand, int ncand, int id_shift,
                                            int cap, float* sc, uint32_t* gone, uint32_t* sel) {
  const int lane = lane_id();
  for (int i = lane; i * 32 < ncand; i += 32) gone[i] = ncand - i * 32 >= 32 ? 0u : ~0u << (ncand - i * 32);
  __syncwarp();
  int nsel = 0, word = 0;
  while (nsel < cap) {
    while (word * 32 < ncand && gone[word] == 0xFFFFFFFFu) ++word;  // the same in every lane
    if (word * 32 >= ncand) break;
    const int i = word * 32 + __ffs(~gone[word]) - 1;
    const uint32_t cid = uint32_t((cand[i] & 0xFFFFFFFFull) >> id_shift);
    __syncwarp();
    if (lane == 0) gone[word] |= 1u << (i & 31);
    if (!FV_IDX_OK(cid, g.n, 3)) {
      __syncwarp();
      continue;
    }
    if (lane == 0) sel[nsel] = cid;
    nsel++;
    __syncwarp();
    if (nsel == cap) break;
    for (int c = lane; c < g.pd; c += 32) sc[c] = g.data[size_t(cid) * g.pd + c];
    // the candidates still standing, in order, up to SELECT_RUN places at a time
    for (int w0 = word; w0 * 32 < ncand; w0 += SELECT_RUN / 32) {
      const int w1 = min(w0 + SELECT_RUN / 32, (ncand + 31) / 32);
      int m = 0;
      for (int w = w0; w < w1; ++w) {
        const unsigned left = ~gone[w];
        if ((left >> lane) & 1u) {
          const uint32_t x = uint32_t((cand[w * 32 + lane] & 0xFFFFFFFFull) >> id_shift);
          t.ids[m + __popc(left & ((1u << lane) - 1u))] = x < g.n ? x : cid;
        }
        m += __popc(left);
      }
      if (m == 0) continue;
      team_eval<IS_L2, NW>(t, sc, m);
      m = 0;
      for (int w = w0; w < w1; ++w) {
        const unsigned left = ~gone[w];
        bool out = false;
        if ((left >> lane) & 1u) {
          const float cd = order_bits_to_float(uint32_t(cand[w * 32 + lane] >> 32));
          out = !(t.out[m + __popc(left & ((1u << lane) - 1u))] > cd);
        }
        const unsigned om = __ballot_sync(FV_FULL, out);
        m += __popc(left);
        __syncwarp();
        if (lane == 0) gone[w] |= om;
        __syncwarp();
      }
    }
  }
  __syncwarp();
  return nsel;
}

// Shared memory of one insertion: the node's row and a kept candidate's, the visited set's first part (a team's), the tie
// list, a run of rows and their distances, the chosen links, the bits of select_links, the team's job, the found list.
__host__ __device__ __forceinline__ size_t insert_smem(int pd, int m0, int ef, int sbits, int nw) {
  const size_t run = size_t(run_rows(ef));
  return size_t(pd) * 8 + visit_smem(sbits) + (TIED_CAP + 2 * run + ((m0 + 3) & ~3) + 128) * 4 + team_smem(nw, m0) +
         ((size_t(ef) * 8 + 15) & ~size_t(15));
}

// flags: [0] visited-table overflows, [1] tie lists that overflowed, [2] edges that did not fit
template <bool IS_L2, int R, int NW>
__global__ void __launch_bounds__(team_threads(NW), team_blocks(NW))
    hnsw_insert_kernel(BuildDev g, uint32_t lo, uint32_t hi, uint32_t ep, int top, int ef, int sbits, int log2slots,
                       uint32_t* __restrict__ tables, Edge* __restrict__ edges, uint32_t* __restrict__ edge_cnt,
                       uint32_t* __restrict__ next_node, uint32_t edge_cap, uint32_t* __restrict__ head,
                       unsigned long long* __restrict__ flags) {
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int searcher = NW == 1 ? w : 0, per_block = NW == 1 ? int(blockDim.x >> 5) : 1;
  const int run = run_rows(ef);
  unsigned char* mine = dyn_smem() + size_t(searcher) * insert_smem(g.pd, g.m0, ef, sbits, NW);
  float* sq = reinterpret_cast<float*>(mine);
  float* sc = sq + g.pd;
  uint32_t* small = reinterpret_cast<uint32_t*>(sc + g.pd);
  uint32_t* tied = small + visit_smem(sbits) / 4;
  uint32_t* sel = tied + TIED_CAP + 2 * run;
  uint32_t* gone = sel + ((g.m0 + 3) & ~3);
  const size_t gw = size_t(blockIdx.x) * per_block + searcher;
  VisitSet seen;
  visit_setup(seen, small, sbits, tables + (gw << log2slots), log2slots, g.n);
  Team<NW> team{g.data, g.pd, tied + TIED_CAP, reinterpret_cast<float*>(tied + TIED_CAP + run),
                reinterpret_cast<TeamJob*>(gone + 128), slot_links(g.m0), g.n, seen, 0u};
  u64* list = reinterpret_cast<u64*>(reinterpret_cast<unsigned char*>(team.job) + team_smem(NW, g.m0));
  if (NW > 1 && w > 0) {
    team_serve<IS_L2, NW>(team);
    return;
  }

  // nodes are drawn from a counter: a search takes anything from a few to a few hundred expansions, and which warp
  // inserts which node changes nothing in the result
  for (;;) {
    uint32_t id = 0;
    if (lane == 0) id = lo + atomicAdd(next_node, 1u);
    id = __shfl_sync(FV_FULL, id, 0);
    if (id >= hi) break;
    const int level = g.levels[id];
    __syncwarp();
    for (int c = lane; c < g.pd; c += 32) sq[c] = g.data[size_t(id) * g.pd + c];

    // greedy descent through the layers above the node's own (hnsw.rs:254-268)
    uint32_t cur = ep;
    if (lane == 0) team.ids[0] = cur;
    team_eval<IS_L2, NW>(team, sq, 1);
    float curd = team.out[0];
    unsigned long long n_dist = 0, n_exp = 0;  // (not reported by the build)
    greedy_descent<IS_L2, NW>(team, g.n, [&](uint32_t x, int layer) { return (const uint32_t*)link_row(g, x, layer); }, g.m,
                              sq, top, level, cur, curd, n_dist, n_exp);

    Beam<R> best;
    best.init(ef, list);
    best.insert(beam_key(curd, cur));
    bool tie_lost = false;
    for (int layer = min(level, top); layer >= 0; --layer) {
      // search_layer starts from everything the layer above found (hnsw.rs:181-193), none of it expanded
      visit_clear(seen);
      __syncwarp();
      best.reopen([&](bool on, uint32_t x) { visit_warp(seen, on, x); });
      bool over = false;
      beam_search<IS_L2, R, NW>(team, g.n, [&](uint32_t c) { return (const uint32_t*)link_row(g, c, layer); },
                                layer == 0 ? g.m0 : g.m, sq, best, tied, seen, over, tie_lost, n_dist, n_exp,
                                layer == 0 ? g.links0 : nullptr);
      if (over) {
        if (lane == 0) atomicAdd(flags, 1ull);
        break;
      }
      const int filled = best.filled();
      if (R > 0) best.each([&](int e, u64 b) { list[e] = b; });
      const int cap = layer == 0 ? g.m0 : g.m;
      const int nsel = select_links<IS_L2, NW>(g, team, list, filled, 1, cap, sc, gone, sel);
      // the node's own list: it is new, so add_links(id, layer, chosen) finds it empty (hnsw.rs:277)
      uint32_t* own = link_row(g, id, layer);
      for (int i = lane; i < nsel; i += 32) own[1 + i] = sel[i];
      uint32_t base = 0;
      if (lane == 0) {
        own[0] = uint32_t(nsel);
        base = atomicAdd(edge_cnt, uint32_t(nsel));
      }
      base = __shfl_sync(FV_FULL, base, 0);
      if (base + uint32_t(nsel) > edge_cap) {
        if (lane == 0) atomicAdd(flags + 2, 1ull);
        break;
      }
      for (int i = lane; i < nsel; i += 32) {
        const uint32_t e = base + uint32_t(i), t = sel[i];
        const uint32_t blk = head_slot(g, t, layer);
        Edge ed;
        ed.tgt = t;
        ed.src = id;
        ed.blk = blk;
        ed.next = atomicExch(head + blk, e);
        edges[e] = ed;
      }
      __syncwarp();
    }
    if (tie_lost && lane == 0) atomicAdd(flags + 1, 1ull);
  }
  team_dismiss(team);
}

// Shared memory of one chain: the target's row and a kept candidate's, two arrays of up to m0 + 1 keys, the list, the
// chosen links, the sources as chained and sorted, the bits of select_links, a run of rows and their distances.
__host__ __device__ __forceinline__ size_t link_smem(int pd, int m0) {
  const size_t nc = size_t(m0) + 1, keys_bytes = (nc * 8 + 15) & ~size_t(15);
  return (size_t(pd) * 8 + 2 * keys_bytes + (nc + m0 + 2 * SRC_CAP + 8 + 2 * run_rows(m0 + 1)) * 4 + 15) & ~size_t(15);
}

// add_links(target, layer, [source]) (hnsw.rs:294-320) for every edge of the batch.  The warp whose edge was the
// first pushed on its chain (next == NIL) owns the chain's (target, layer).
template <bool IS_L2>
__global__ void __launch_bounds__(256, BUILD_BLOCKS_PER_SM)
    hnsw_link_kernel(BuildDev g, const Edge* __restrict__ edges, const uint32_t* __restrict__ edge_cnt,
                     uint32_t edge_cap, uint32_t* __restrict__ head) {
  unsigned char* smem_raw = dyn_smem();
  const int W = blockDim.x >> 5, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int cap_max = g.m0, nc = cap_max + 1;
  const size_t keys_bytes = (size_t(nc) * 8 + 15) & ~size_t(15);
  unsigned char* mine = smem_raw + size_t(w) * link_smem(g.pd, g.m0);
  float* sb = reinterpret_cast<float*>(mine);
  float* sc = sb + g.pd;
  u64* keys = reinterpret_cast<u64*>(mine + size_t(g.pd) * 8);
  u64* sorted = reinterpret_cast<u64*>(mine + size_t(g.pd) * 8 + keys_bytes);
  uint32_t* ids = reinterpret_cast<uint32_t*>(mine + size_t(g.pd) * 8 + 2 * keys_bytes);
  uint32_t* sel = ids + nc;
  uint32_t* srcs = sel + cap_max;
  uint32_t* srcs_sorted = srcs + SRC_CAP;
  uint32_t* gone = srcs_sorted + SRC_CAP;
  const Team<1> team{g.data, g.pd, gone + 8, reinterpret_cast<float*>(gone + 8 + run_rows(nc)), nullptr, 0, g.n, VisitSet{}, 0u};
  const uint32_t count = min(*edge_cnt, edge_cap);
  const uint32_t gw = blockIdx.x * W + w, total_warps = gridDim.x * W;

  for (uint32_t e = gw; e < count; e += total_warps) {
    const Edge first = edges[e];
    if (first.next != NIL) continue;
    const uint32_t t = first.tgt;
    if (!FV_IDX_OK(t, g.n, 5)) continue;
    const int layer = first.blk < g.n ? 0 : int(first.blk - g.n - g.up_blk[t]) + 1;
    const int cap = layer == 0 ? g.m0 : g.m;
    uint32_t* row = link_row(g, t, layer);
    __syncwarp();
    // the chain's sources; the walk is bounded by the number of edges
    int k = 0;
    if (lane == 0) {
      uint32_t x = head[first.blk];
      for (uint32_t hop = 0; x != NIL && hop < count; ++hop) {
        if (!FV_IDX_OK(x, count, 6)) break;
        if (k < SRC_CAP) srcs[k] = edges[x].src;
        k++;
        x = edges[x].next;
      }
    }
    k = __shfl_sync(FV_FULL, k, 0);
    __syncwarp();
    if (k <= SRC_CAP) {  // ascending by rank: ids are distinct
      for (int i = lane; i < k; i += 32) {
        const uint32_t v = srcs[i];
        int r = 0;
        for (int j = 0; j < k; ++j) r += srcs[j] < v;
        srcs_sorted[r] = v;
      }
      __syncwarp();
    }
    for (int c = lane; c < g.pd; c += 32) sb[c] = g.data[size_t(t) * g.pd + c];
    // The list is kept in shared memory and every change is written through to the row as set_neighbors does
    // (hnsw.rs:165-175): a shorter list leaves the old ids behind it in the row, and the FLHNSW01 file holds the
    // rows whole, so the words past the count must be the reference's too.
    int cnt = min(int(row[0]), cap);
    for (int i = lane; i < cnt; i += 32) ids[i] = row[1 + i];
    __syncwarp();
    long long last = -1;
    for (int si = 0; si < k; ++si) {
      uint32_t s;
      if (k <= SRC_CAP) {
        s = srcs_sorted[si];
      } else {  // the smallest source above the last one, by another walk
        uint32_t best_s = NIL;
        if (lane == 0) {
          uint32_t x = head[first.blk];
          for (uint32_t hop = 0; x != NIL && hop < count; ++hop) {
            if (!FV_IDX_OK(x, count, 7)) break;
            const uint32_t v = edges[x].src;
            if ((long long)v > last && v < best_s) best_s = v;
            x = edges[x].next;
          }
        }
        s = __shfl_sync(FV_FULL, best_s, 0);
        if (s == NIL) break;
      }
      last = (long long)s;
      // x != id && !list.contains(&x)  (hnsw.rs:299-303)
      bool dup = s == t;
      for (int i0 = 0; i0 < cnt && !dup; i0 += 32) {
        const int i = i0 + lane;
        dup = __any_sync(FV_FULL, i < cnt && ids[i] == s);
      }
      if (dup || !FV_IDX_OK(s, g.n, 8)) continue;
      __syncwarp();
      if (lane == 0) ids[cnt] = s;
      cnt++;
      __syncwarp();
      if (cnt > cap) {
        // distances from the base, sorted by (distance, id), chosen again (hnsw.rs:307-318)
        for (int i = lane; i < cnt; i += 32) team.ids[i] = ids[i];
        team_eval<IS_L2, 1>(team, sb, cnt);
        for (int i = lane; i < cnt; i += 32) keys[i] = make_key(team.out[i], ids[i]);
        __syncwarp();
        for (int i = lane; i < cnt; i += 32) {
          const u64 v = keys[i];
          int r = 0;
          for (int j = 0; j < cnt; ++j) r += keys[j] < v;
          sorted[r] = v;
        }
        __syncwarp();
        const int nsel = select_links<IS_L2, 1>(g, team, sorted, cnt, 0, cap, sc, gone, sel);
        for (int i = lane; i < nsel; i += 32) {
          ids[i] = sel[i];
          row[1 + i] = sel[i];
        }
        cnt = nsel;
        __syncwarp();
      } else if (lane == 0) {
        row[cnt] = s;
      }
    }
    if (lane == 0) {
      row[0] = uint32_t(cnt);
      head[first.blk] = NIL;
    }
    __syncwarp();
  }
}

// The next batch: at most max_batch nodes, at most 1/divisor of those already in, cut before a node whose level is
// above the current top layer (such a node goes in alone).
static size_t next_batch(const std::vector<uint8_t>& levels, size_t inserted, size_t top, size_t max_batch,
                         size_t divisor) {
  const size_t n = levels.size();
  size_t b = std::max<size_t>(1, std::min(max_batch, inserted / std::max<size_t>(1, divisor)));
  b = std::min(b, n - inserted);
  if (levels[inserted] > top) return 1;
  for (size_t j = 1; j < b; j++)
    if (levels[inserted + j] > top) return j;
  return b;
}

typedef void (*InsertKernel)(BuildDev, uint32_t, uint32_t, uint32_t, int, int, int, int, uint32_t*, Edge*, uint32_t*, uint32_t*,
                             uint32_t, uint32_t*, unsigned long long*);
template <int NW>
static InsertKernel pick_insert(bool is_l2, int R) {
  switch (R) {
    case 2: return is_l2 ? hnsw_insert_kernel<true, 2, NW> : hnsw_insert_kernel<false, 2, NW>;
    case 4: return is_l2 ? hnsw_insert_kernel<true, 4, NW> : hnsw_insert_kernel<false, 4, NW>;
    case 8: return is_l2 ? hnsw_insert_kernel<true, 8, NW> : hnsw_insert_kernel<false, 8, NW>;
    default:
      if constexpr (NW == SCOUT_WARPS) return nullptr;  // (scouts_pay)
      else return is_l2 ? hnsw_insert_kernel<true, 0, NW> : hnsw_insert_kernel<false, 0, NW>;
  }
}

static int build_on_device(fv_hnsw* h, size_t ef, size_t max_batch, size_t divisor) {
  fv_ctx* ctx = h->ctx;
  const size_t n = h->n(), m = h->m, m0 = h->m0;
  if (n > 0x7FFFFFFFull) return fail(FV_ERR_UNSUPPORTED, "more than 2^31 nodes");
  if (ef == 0 || ef > 4096) return fail(FV_ERR_UNSUPPORTED, "ef_construction must be in 1..4096");
  const int pd = int(h->pd);
  // block offsets of the upper layers; the batches and the edges the largest can push
  std::vector<uint32_t> up_blk(n + 1, 0);
  for (size_t i = 0; i < n; i++) up_blk[i + 1] = up_blk[i] + h->levels[i];
  const size_t nblk = up_blk[n];
  if (n + nblk >= 0xFFFFFFFFull) return fail(FV_ERR_UNSUPPORTED, "too many link lists for 32-bit chain heads");
  size_t edge_cap = 0, widest = 0;
  {
    size_t inserted = 1, top = h->levels[0];
    while (inserted < n) {
      const size_t b = next_batch(h->levels, inserted, top, max_batch, divisor);
      size_t e = 0;
      for (size_t j = 0; j < b; j++) e += m0 + std::min<size_t>(h->levels[inserted + j], top) * m;
      edge_cap = std::max(edge_cap, e);
      widest = std::max(widest, b);
      if (h->levels[inserted] > top) top = h->levels[inserted];
      inserted += b;
    }
  }
  if (edge_cap >= 0xFFFFFFFFull) return fail(FV_ERR_UNSUPPORTED, "batch too large");

  DevBuf d_up, d_up_blk, d_levels, d_head, d_edges, d_tables, d_words;
  FV_TRY(h->d_data.reserve(h->data.size() * 4 + 16));
  FV_TRY(h->d_links0.reserve(h->links0.size() * 4 + 16));
  FV_TRY(d_up.reserve(nblk * (m + 1) * 4 + 16));
  FV_TRY(d_up_blk.reserve((n + 1) * 4));
  FV_TRY(d_levels.reserve(n + 16));
  FV_TRY(d_head.reserve((n + nblk) * 4 + 16));
  FV_TRY(d_edges.reserve((edge_cap + 1) * sizeof(Edge)));
  FV_TRY(d_words.reserve(64));
  uint32_t* d_edge_cnt = d_words.as<uint32_t>();
  uint32_t* d_next_node = d_edge_cnt + 1;
  unsigned long long* d_flags = reinterpret_cast<unsigned long long*>(d_words.as<unsigned char>() + 16);
  cudaStream_t st = ctx->stream;
  FV_CUDA(cudaMemcpyAsync(h->d_data.p, h->data.data(), h->data.size() * 4, cudaMemcpyHostToDevice, st));
  FV_CUDA(cudaMemcpyAsync(d_up_blk.p, up_blk.data(), (n + 1) * 4, cudaMemcpyHostToDevice, st));
  FV_CUDA(cudaMemcpyAsync(d_levels.p, h->levels.data(), n, cudaMemcpyHostToDevice, st));

  BuildDev g{};
  g.data = h->d_data.as<float>();
  g.links0 = h->d_links0.as<uint32_t>();
  g.up = d_up.as<uint32_t>();
  g.up_blk = d_up_blk.as<uint32_t>();
  g.levels = d_levels.as<uint8_t>();
  g.pd = pd;
  g.m = int(m);
  g.m0 = int(m0);
  g.n = uint32_t(n);

  // launch shapes: shared memory per searcher, searchers per block, resident blocks
  const int R = ef <= 64 ? 2 : ef <= 128 ? 4 : ef <= 256 ? 8 : 0;
  const size_t budget = std::min<size_t>(ctx->smem_optin, 200 * 1024);
  const bool is_l2 = h->metric == FV_L2;
  const size_t link_warp = link_smem(pd, int(m0));
  int sbits = visit_sbits(int(ef)), W = 8, LW = 8;
  const size_t ins_warp = insert_smem(pd, int(m0), int(ef), -1, 1);  // a single warp's visited set is in global memory
  auto team_bytes = [&](int bits, int nw) { return insert_smem(pd, int(m0), int(ef), bits, nw); };
  // (rows too long for a scouting team's slots beside the smallest first part of the visited set: teams of eight)
  const bool scouting = R > 0 && team_bytes(7, SCOUT_WARPS) <= ctx->smem_optin;
  while (W > 1 && ins_warp * W > budget / BUILD_BLOCKS_PER_SM) W >>= 1;
  while (LW > 1 && link_warp * LW > budget / BUILD_BLOCKS_PER_SM) LW >>= 1;
  while (sbits > 7 && team_bytes(sbits, scouting ? SCOUT_WARPS : TEAM_WARPS) > ctx->smem_optin) sbits--;
  if (std::max({ins_warp * W, team_bytes(sbits, TEAM_WARPS), link_warp * LW}) > ctx->smem_optin)
    return fail(FV_ERR_UNSUPPORTED, "dimension and ef_construction too large for shared memory");
  const size_t resident_blocks = size_t(ctx->sm_count) * BUILD_BLOCKS_PER_SM;
  const size_t searchers_max = std::min(resident_blocks * W, std::max<size_t>(widest, 1));  // (a team is one searcher)
  InsertKernel ins = pick_insert<1>(is_l2, R), ins_team = pick_insert<TEAM_WARPS>(is_l2, R),
               ins_scouts = pick_insert<SCOUT_WARPS>(is_l2, R);
  auto lnk = is_l2 ? hnsw_link_kernel<true> : hnsw_link_kernel<false>;
  FV_TRY(allow_smem(ctx, ins, ins_warp * W));
  FV_TRY(allow_smem(ctx, ins_team, team_bytes(sbits, TEAM_WARPS)));
  if (scouting) FV_TRY(allow_smem(ctx, ins_scouts, team_bytes(sbits, SCOUT_WARPS)));
  FV_TRY(allow_smem(ctx, lnk, link_warp * LW));

  int log2slots = 11;
  while ((size_t(1) << log2slots) < ef * 128 && log2slots < 24) log2slots++;
  for (int attempt = 0; attempt < 3; ++attempt, log2slots += 2) {
    FV_TRY(d_tables.reserve((((searchers_max + W - 1) / W * W) << log2slots) * 4 + 16));
    FV_CUDA(cudaMemsetAsync(h->d_links0.p, 0, h->links0.size() * 4, st));
    FV_CUDA(cudaMemsetAsync(d_up.p, 0, nblk * (m + 1) * 4, st));
    FV_CUDA(cudaMemsetAsync(d_head.p, 0xFF, (n + nblk) * 4, st));
    FV_CUDA(cudaMemsetAsync(d_words.p, 0, 64, st));
    size_t inserted = 1, top = h->levels[0];
    uint32_t ep = 0;
    stage_begin(ctx);  // stage 0: uploads and clears; stage 1: the batches
    stage_mark(ctx);
    while (inserted < n) {
      const size_t b = next_batch(h->levels, inserted, top, max_batch, divisor);
      FV_CUDA(cudaMemsetAsync(d_edge_cnt, 0, 8, st));  // and the node counter
      const bool scouts = scouting && scouts_pay(ctx->sm_count, pd, int(m0), int(ef), b);
      const int nw = scouts ? SCOUT_WARPS : TEAM_WARPS;
      if (b <= size_t(ctx->sm_count) * TEAM_INSERTS_PER_SM)
        (scouts ? ins_scouts : ins_team)<<<unsigned(std::min(b, resident_blocks)), nw * 32, team_bytes(sbits, nw), st>>>(
            g, uint32_t(inserted), uint32_t(inserted + b), ep, int(top), int(ef), sbits, log2slots, d_tables.as<uint32_t>(),
            d_edges.as<Edge>(), d_edge_cnt, d_next_node, uint32_t(edge_cap), d_head.as<uint32_t>(), d_flags);
      else
        ins<<<unsigned(std::min(resident_blocks, (b + W - 1) / W)), W * 32, ins_warp * W, st>>>(
            g, uint32_t(inserted), uint32_t(inserted + b), ep, int(top), int(ef), -1, log2slots, d_tables.as<uint32_t>(),
            d_edges.as<Edge>(), d_edge_cnt, d_next_node, uint32_t(edge_cap), d_head.as<uint32_t>(), d_flags);
      FV_CUDA(cudaGetLastError());
      size_t e_max = 0;
      for (size_t j = 0; j < b; j++) e_max += m0 + std::min<size_t>(h->levels[inserted + j], top) * m;
      const size_t lnk_blocks = std::max<size_t>(1, std::min<size_t>(resident_blocks, (e_max + LW - 1) / LW));
      lnk<<<unsigned(lnk_blocks), LW * 32, link_warp * LW, st>>>(g, d_edges.as<Edge>(), d_edge_cnt, uint32_t(edge_cap),
                                                              d_head.as<uint32_t>());
      FV_CUDA(cudaGetLastError());
      ctx->stats.launches += 2;
      if (h->levels[inserted] > top) {  // hnsw.rs:285-289
        top = h->levels[inserted];
        ep = uint32_t(inserted);
      }
      inserted += b;
    }
    stage_mark(ctx);
    unsigned long long flags[3] = {0, 0, 0};
    FV_CUDA(cudaMemcpyAsync(flags, d_flags, sizeof(flags), cudaMemcpyDeviceToHost, st));
    FV_CUDA(cudaStreamSynchronize(st));
    stage_end(ctx);
    FV_TRY(bounds_report_hnsw_build());
    if (flags[2]) return fail(FV_ERR_OVERFLOW, "hnsw build: edge buffer overflow");
    if (flags[0]) {
      ctx->stats.regrown += flags[0];
      continue;  // a visited table filled up: again with tables four times larger
    }
    ctx->stats.uncertified = flags[1];  // searches whose list of tied, pushed-out entries overflowed (see TIED_CAP)
    h->ep = ep;
    h->top = top;
    FV_CUDA(cudaMemcpyAsync(h->links0.data(), h->d_links0.p, h->links0.size() * 4, cudaMemcpyDeviceToHost, st));
    std::vector<uint32_t> flat(nblk * (m + 1));
    if (!flat.empty()) FV_CUDA(cudaMemcpyAsync(flat.data(), d_up.p, flat.size() * 4, cudaMemcpyDeviceToHost, st));
    FV_CUDA(cudaStreamSynchronize(st));
    for (size_t i = 0; i < n; i++)
      if (h->levels[i])
        std::memcpy(h->upper[i].data(), &flat[size_t(up_blk[i]) * (m + 1)], size_t(h->levels[i]) * (m + 1) * 4);
    return FV_OK;
  }
  return fail(FV_ERR_OVERFLOW, "hnsw build: visited table overflow after regrowing");
}

}  // namespace fv

extern "C" int fv_hnsw_build_batched(fv_ctx* ctx, int metric, uint32_t dim, const float* vectors, size_t n,
                                     const fv_hnsw_params* p, size_t max_batch, size_t divisor, fv_hnsw** out) {
  if (!out || max_batch == 0 || divisor == 0) return fv::fail(FV_ERR_ARG, "fv_hnsw_build_batched: bad argument");
  std::unique_ptr<fv_hnsw> h;
  FV_TRY(fv::hnsw_new(ctx, metric, dim, vectors, n, p, h));
  fv::CtxGuard g(ctx);
  ctx->stats = fv_stats{};
  if (n > 1) {
    FV_TRY(fv::build_on_device(h.get(), p->ef_construction, max_batch, divisor));
    FV_TRY(fv::upload_graph(h.get(), false));
  } else {
    FV_TRY(fv::upload_graph(h.get()));
  }
  *out = h.release();
  return FV_OK;
}
