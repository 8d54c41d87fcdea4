// What the Hnsw search (hnsw.cu) and the construction on the GPU (hnsw_build.cu) share: the index object, the
// per-warp visited table and the beam's entry format.
#pragma once

#include <memory>
#include <vector>

#include "internal.h"

struct fv_hnsw {
  fv_ctx* ctx = nullptr;
  ~fv_hnsw() {
    d_data.release(); d_bytes.release(); d_links0.release(); d_upper_off.release(); d_upper_flat.release();
    if (ctx) fv::ctx_release(ctx);
  }
  int metric = 0;
  uint32_t dim = 0, pd = 0;
  size_t m = 0, m0 = 0;
  uint32_t ep = 0;
  size_t top = 0;
  // host copies (the file's content)
  std::vector<float> data;
  std::vector<uint8_t> levels;
  std::vector<uint32_t> links0;
  std::vector<std::vector<uint32_t>> upper;  // per node: concatenated (count, ids...) per layer, fixed stride m+1
  // device copies
  DevBuf d_data, d_links0, d_upper_off, d_upper_flat;
  // L2 over whole numbers that lie within 255 of each other, so few that every sum of the reference's chain is exact: the
  // rows once more as bytes above byte_lo, row_bytes(pd) per row, for the searches; empty otherwise
  DevBuf d_bytes;
  float byte_lo = 0.f;
  size_t n() const { return levels.size(); }
};

namespace fv {

// An index with its rows padded, its levels drawn (hnsw.rs:88-94) and every link list empty; node 0 is the entry.
int hnsw_new(fv_ctx* ctx, int metric, uint32_t dim, const float* vectors, size_t n, const fv_hnsw_params* p,
             std::unique_ptr<fv_hnsw>& out);
__host__ __device__ __forceinline__ int row_bytes(int pd) { return (pd + 15) & ~15; }
// Copies the host graph to the device in the search kernel's layout; the rows too unless they are there already.
int upload_graph(fv_hnsw* h, bool with_data = true);

// The reference keeps two heaps: an entry pushed out of the result heap stays in the candidate heap, and because its
// loop stops only on a STRICTLY larger distance (hnsw.rs:195-197), such an entry is still expanded if its distance
// equals the worst kept distance when its turn comes.  The beam is one list, so the unexpanded entries it pushes out
// while their distance equals the new worst distance are remembered in a side list of this many ids (all share that
// distance) and take their turn in (distance, id) order; the list is dropped as soon as the worst distance goes down.
static constexpr int TIED_CAP = 64;

// Searches of one launch are run by teams of TEAM_WARPS warps up to a number per SM, by single warps beyond.  A team
// shortens the distances of an expansion and leaves the rest of it to one warp, so it pays the longer the longer the rows
// and the shorter the beam.  Where the two cross, in queries per SM (m = 16, 30,000 to 100,000 nodes): rows of 32
// dimensions 6 at ef 10 and 64, 4 to 7 at 100 to 160, 3 at 200 and 256; of 64 and 96 dimensions 12 and 15 at ef 10, 7 to
// 11 at 32 and 64, 6 to 10, 4 to 8; of 128 and more 10 to 20, 11 to 15, 7 to 9 (with m = 24 and 200 dimensions 7 and 5 from
// ef 100 on); with the beam in shared memory (ef 400 and 1,000) 2 to 4 at any dimension.
static constexpr int TEAM_WARPS = 8;
// Up to two searches per SM run by scouting teams: a warp with the beam and eight that work out the links and distances of
// the node that is next in line while the first is still busy with the one before.  80 to 93 % of the expansions find theirs
// done or under way; what is left of one is mostly the first warp's own part (1,900 cycles of 2,200 at 96 dimensions and 200
// entries).  us with teams of eight and with scouts, 20 queries: 5,183 x 384, ef 64 203 and 176, ef 200 526 and 387; 100,000
// x 128 154 and 141, 333 and 268; 20,000 x 200 with m = 24 248 and 161, 659 and 361.  Not with the beam in shared memory (100,000
// x 128, ef 400: 1,090 and 1,216), nor where the rows are so long and the beam so short that working out what turns out not to
// be next takes longer than it saves (4,000 x 2,048, ef 10: 1 query 108 and 116, 20 141 and 165, 296 189 and 207; ef 32 311 and
// 327; ef 64 510 and 517, 20 queries 451 and 425; 5,000 x 768 the same at ef 10 and 32, 240 and 214 at 64).  Construction,
// 20,000 x 96: 122 ms of kernels and 106.
static constexpr int SCOUT_WARPS = 9;
static constexpr int SCOUT_LINKS = 64;  // links of a node, at most
static inline bool scouts_pay(int sm_count, int pd, int m0, int ef, size_t searches) {
  return m0 <= SCOUT_LINKS && ef <= 256 && (pd < 1024 || ef > 32) && searches <= size_t(sm_count) * 2;
}
static inline size_t team_searches_per_sm(int pd, int m0, int ef) {
  static constexpr size_t most[5][3] = {{6, 14, 16}, {6, 10, 16}, {6, 8, 14}, {3, 6, 8}, {2, 2, 2}};
  const size_t line = most[ef <= 16 ? 0 : ef <= 64 ? 1 : ef <= 160 ? 2 : ef <= 256 ? 3 : 4][pd < 64 ? 0 : pd < 128 ? 1 : 2];
  return ef > 64 && ef <= 256 && m0 > 32 && m0 <= 64 ? line * 3 / 4 : line;
}

#ifdef __CUDACC__
__device__ __forceinline__ uint32_t hash_slot(uint32_t x, int log2slots) { return (x * 2654435761u) >> (32 - log2slots); }

// true if x was not in the table (and is now)
__device__ __forceinline__ bool visit(uint32_t* table, int log2slots, uint32_t x) {
  const uint32_t mask = (1u << log2slots) - 1u;
  uint32_t s = hash_slot(x, log2slots);
  for (uint32_t probe = 0; probe <= mask; ++probe) {
    const uint32_t old = atomicCAS(table + s, 0xFFFFFFFFu, x);
    if (old == 0xFFFFFFFFu) return true;
    if (old == x) return false;
    s = (s + 1) & mask;
  }
  return false;  // full table: cannot happen below the half-full limit
}

// list entry: order bits of the distance (32) | id (31) | expanded (1)
__device__ __forceinline__ u64 beam_key(float d, uint32_t id) { return (u64(order_bits(d)) << 32) | (u64(id) << 1); }
__device__ __forceinline__ uint32_t beam_id(u64 key) { return uint32_t(key >> 1) & 0x7FFFFFFFu; }
__device__ __forceinline__ float beam_distance(u64 key) { return order_bits_to_float(uint32_t(key >> 32)); }

// ---- visited set: exact.
// It is an open-addressing table of whole ids in global memory, cleared by the first id it gets.  A team, which has a
// block's shared memory to itself, puts a first part there, and so does a single warp with a beam beyond 64 where that
// part holds every node of the graph (4,096): a small table in shared memory with two 16-bit entries per word.  x -> x * odd (mod 2^b, b bits
// holding every id) is a bijection; the high bits of the image name the home bucket, so an entry needs only the low
// `rb` bits and how many buckets it sits behind its home.  An id that finds all of its `probes` buckets full goes to
// the second part, an open-addressing table of whole ids in global memory that is cleared by the first id it gets.
// Nothing is ever removed, so a bucket that was full when an id passed it is full whenever the id comes back.
// Measured with and without the first part (us): 592 queries by teams, 100,000 x 128, ef 64 372 and 571, ef 256 1,274 and
// 1,731.  Single warps, with the 32 * ef places that 24 of them have room for, so that more and more ids find their
// buckets full: 10,000 queries, ef 64 2,346 and 1,816, ef 128 3,697 and 3,046, ef 256 8,837 and 5,166; on a graph of 3,000
// nodes, which fit, 10,000 x 48 at ef 100 1,028 and 1,138, at ef 256 2,585 and 3,046.
struct VisitSet {
  uint32_t* small;    // shared memory: 2^sbits words
  uint32_t* big;      // global memory: 2^log2slots words
  int sbits, rb, probes, log2slots;  // sbits < 0: no part in shared memory
  uint32_t idmask;
  int in_big;         // ids in `big`, the same in every lane; -1: not cleared yet
};

// Words of a team's shared part for a beam of ef entries: 128 * ef places (rounded up to a power of two, up to 16,384).
// About 12 ids are visited per entry of the beam on the benchmark's graphs, 22 on a graph of 5,183 text-like rows; at 70 %
// full a look-up takes 1,900 cycles of the 6,400 of an expansion.
__host__ __device__ __forceinline__ int visit_sbits(int ef) {
  int s = 7;
  while (s < 13 && (1 << s) < ef * 64) ++s;
  return s;
}

// bytes of the shared part
__host__ __device__ __forceinline__ size_t visit_smem(int sbits) { return sbits < 0 ? 0 : size_t(4) << sbits; }
// a single warp's: one place per node, if those are at most 4,096 and the beam is long enough to visit many of them
static inline int visit_sbits_single(size_t n, int ef) {
  int s = 7;
  while (s < 11 && (size_t(2) << s) < n) ++s;
  return ef <= 64 || (size_t(2) << s) < n ? -1 : s;
}

__device__ __forceinline__ void visit_setup(VisitSet& v, uint32_t* small, int sbits, uint32_t* big, int log2slots,
                                            size_t n) {
  v.big = big;
  v.log2slots = log2slots;
  v.in_big = -1;
  v.sbits = sbits;
  if (sbits < 0) return;
  int b = 1;
  while (b < 32 && (size_t(1) << b) < n) ++b;
  v.small = small;
  v.rb = b > sbits ? b - sbits : 0;
  v.probes = min(32, int(0xFFFFu >> min(v.rb, 16)));  // (the largest displacement must leave 0xFFFF, "empty", unused)
  v.idmask = b == 32 ? 0xFFFFFFFFu : (1u << b) - 1u;
}

// empties the set; called by a whole warp, which the caller lines up afterwards
__device__ __forceinline__ void visit_clear(VisitSet& v) {
  if (v.sbits >= 0)
    for (int i = lane_id() * 4; i < (1 << v.sbits); i += 128) *reinterpret_cast<uint4*>(v.small + i) = make_uint4(~0u, ~0u, ~0u, ~0u);
  v.in_big = -1;
}

// an id into the part in global memory: true in the lanes whose x (on) was not there and is now; called by a whole warp
__device__ __forceinline__ bool visit_big(VisitSet& v, bool on, uint32_t x) {
  if (v.in_big < 0) {
    for (int s = lane_id() * 4; s < (1 << v.log2slots); s += 128) *reinterpret_cast<uint4*>(v.big + s) = make_uint4(~0u, ~0u, ~0u, ~0u);
    v.in_big = 0;
    __syncwarp();
  }
  const bool fresh = on && visit(v.big, v.log2slots, x);
  v.in_big += __popc(__ballot_sync(FV_FULL, fresh));
  return fresh;
}

// called by a whole warp: true in the lanes whose x (on && x < n) was not in the set and is now.
// The usual case -- the home bucket holds x, or has room and no other lane wants it -- is straight-line code: a branch
// costs a warp here about as much as a trip to shared memory.
__device__ __forceinline__ bool visit_warp(VisitSet& v, bool on, uint32_t x) {
  if (v.sbits < 0) return visit_big(v, on, x);
  const uint32_t h = (x * 0x9E3779B1u) & v.idmask;
  const uint32_t bucket = h >> v.rb, rem = h & ((1u << v.rb) - 1u);
  uint32_t* p = v.small + bucket;
  uint32_t w = *reinterpret_cast<volatile uint32_t*>(p);
  const bool lo_free = (w & 0xFFFFu) == 0xFFFFu, hi_free = (w >> 16) == 0xFFFFu;
  const bool seen = (w & 0xFFFFu) == rem || (w >> 16) == rem;
  const bool want = on && !seen && (lo_free || hi_free) && v.probes > 0;
  const uint32_t nw = lo_free ? ((w & 0xFFFF0000u) | rem) : ((w & 0xFFFFu) | (rem << 16));
  uint32_t old = ~w;
  if (want) old = atomicCAS(p, w, nw);
  bool fresh = want && old == w;
  bool open = on && !fresh && (!seen || v.probes <= 0);  // another lane was quicker, or the bucket is full
  if (!__any_sync(FV_FULL, open)) return fresh;
  bool full = open;
  const uint32_t smask = (1u << v.sbits) - 1u;
  for (int d = 0; d < v.probes && full; ++d) {
    const uint32_t val = (uint32_t(d) << v.rb) | rem;
    p = v.small + ((bucket + uint32_t(d)) & smask);
    w = *reinterpret_cast<volatile uint32_t*>(p);
    for (;;) {  // (a word fills up after two insertions: at most three turns)
      const uint32_t lo = w & 0xFFFFu, hi = w >> 16;
      if (lo == val || hi == val) {
        full = false;
        break;
      }
      uint32_t nv;
      if (lo == 0xFFFFu) nv = (w & 0xFFFF0000u) | val;
      else if (hi == 0xFFFFu) nv = (w & 0xFFFFu) | (val << 16);
      else break;
      const uint32_t was = atomicCAS(p, w, nv);
      if (was == w) {
        full = false;
        fresh = true;
        break;
      }
      w = was;
    }
  }
  if (__any_sync(FV_FULL, full)) {
    const bool big_fresh = visit_big(v, full, x);
    fresh = full ? big_fresh : fresh;
  }
  return fresh;
}
// whether x was in its home bucket a moment ago (it stays then); anyone may ask while the set's warp adds to it
__device__ __forceinline__ bool visit_seen(const VisitSet& v, uint32_t x) {
  if (v.sbits < 0 || v.probes <= 0) return false;
  const uint32_t h = (x * 0x9E3779B1u) & v.idmask, rem = h & ((1u << v.rb) - 1u);
  const uint32_t w = *reinterpret_cast<volatile uint32_t*>(v.small + (h >> v.rb));
  return (w & 0xFFFFu) == rem || (w >> 16) == rem;
}
__device__ __forceinline__ bool visit_overflow(const VisitSet& v) { return v.in_big > (1 << (v.log2slots - 1)); }

// ---- the beam: the ef nearest entries seen so far, ascending, each with its "expanded" bit.
// R > 0: in registers, place 32 r + lane in e[r] (ef <= 32 R): an insertion is one compare and one shuffle per 32
// entries, without the shared-memory round trips and barriers of the list below.  The list ends at the last place, so
// that its last entry is found and dropped without knowing ef; the `off` places before it hold a key below every
// other.  That key and FV_EMPTY_KEY, the unused entry, both read "expanded" in their lowest bit.
template <int R>
struct Beam {
  u64 e[R];
  int off;
  __device__ __forceinline__ void init(int ef, u64*) {
    off = 32 * R - ef;
#pragma unroll
    for (int r = 0; r < R; ++r) e[r] = r * 32 + lane_id() < off ? 1ull : FV_EMPTY_KEY;
  }
  __device__ __forceinline__ u64 last() const { return __shfl_sync(FV_FULL, e[R - 1], 31); }
  __device__ __forceinline__ void insert(u64 key) {  // key < last()
#pragma unroll
    for (int r = R - 1; r >= 0; --r) {
      // the entry one place before: lane 31 passes on its entry of the row below, which lane 0 is the one to read
      const u64 own = e[r], below = e[r > 0 ? r - 1 : 0];
      u64 prev = __shfl_sync(FV_FULL, lane_id() == 31 ? below : own, (lane_id() + 31) & 31);
      if (r == 0 && lane_id() == 0) prev = 0;
      if (!(e[r] < key)) e[r] = prev < key ? key : prev;
    }
  }
  // All pending keys at once, by a sort and a merge (bitonic_merge): what the insertions one by one would leave, as long
  // as no entry that falls off the end is as far as the last one kept -- everything up to that distance is then admitted
  // whenever it comes and never pushed out again, and nothing pushed out can tie.  Otherwise nothing is done.
  __device__ __forceinline__ void take(unsigned& pending, u64 key, u64& bound, int& ntied) {
    const u64 c = warp_sort32((pending >> lane_id()) & 1u ? key : FV_EMPTY_KEY);
    const u64 back = __shfl_sync(FV_FULL, c, 31 - lane_id());
    const u64 x = e[R - 1];
    const u64 low = x < back ? x : back;
    const uint32_t drop = __reduce_min_sync(FV_FULL, uint32_t((x < back ? back : x) >> 32));
    uint32_t keep = __reduce_max_sync(FV_FULL, uint32_t(low >> 32));
    if (R > 1) keep = max(keep, uint32_t(__shfl_sync(FV_FULL, e[R > 1 ? R - 2 : 0], 31) >> 32));
    if (drop == keep && keep != 0xFFFFFFFFu) return;
    e[R - 1] = low;
    bitonic_merge<R>(e);
    const u64 now = last();
    if (uint32_t(now >> 32) < uint32_t(bound >> 32)) ntied = 0;
    bound = now;
    pending = 0;
  }
  // the first entry that is not expanded (FV_EMPTY_KEY: none); marking one
  __device__ __forceinline__ u64 first_open() const {
    unsigned pos = 0x7FFFFFFFu;
    u64 v = FV_EMPTY_KEY;
#pragma unroll
    for (int r = R - 1; r >= 0; --r)
      if (!(e[r] & 1ull)) {
        pos = unsigned(r * 32 + lane_id());
        v = e[r];
      }
    return __shfl_sync(FV_FULL, v, int(__reduce_min_sync(FV_FULL, pos) & 31));  // (none: any lane's)
  }
  __device__ __forceinline__ void mark(u64 key) {
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (e[r] == key) e[r] |= 1ull;
  }
  __device__ __forceinline__ int filled() const {
    int c = 0;
#pragma unroll
    for (int r = 0; r < R; ++r) c += __popc(__ballot_sync(FV_FULL, e[r] != FV_EMPTY_KEY));
    return c - off;
  }
  // fn(position, entry) for every entry in use, entries spread over the lanes
  template <class Fn>
  __device__ __forceinline__ void each(Fn fn) {
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (e[r] != FV_EMPTY_KEY && r * 32 + lane_id() >= off) fn(r * 32 + lane_id() - off, e[r]);
  }
  // takes the "expanded" marks off; fn(in use, id) is called by the whole warp, 32 entries at a time
  template <class Fn>
  __device__ __forceinline__ void reopen(Fn fn) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const bool on = e[r] != FV_EMPTY_KEY && r * 32 + lane_id() >= off;
      if (on) e[r] &= ~1ull;
      fn(on, beam_id(e[r]));
    }
  }
};
// R = 0: in shared memory, any ef
template <>
struct Beam<0> {
  u64* e;
  int ef, n, cursor;  // entries in use; the first entry that may be open
  __device__ __forceinline__ void init(int ef_, u64* smem) {
    e = smem;
    ef = ef_;
    n = 0;
    cursor = 0;
    warp_list_init(e, ef);
  }
  __device__ __forceinline__ u64 last() const { return e[ef - 1]; }
  __device__ __forceinline__ void insert(u64 key) {
    int below = 0;
    for (int e0 = 0; e0 < n; e0 += 32) {
      const int i = e0 + lane_id();
      below += __popc(__ballot_sync(FV_FULL, i < n && e[i] < key));
    }
    __syncwarp();
    warp_list_insert(e, ef, key);
    __syncwarp();
    if (n < ef) n++;
    if (below < cursor) cursor = below;
  }
  __device__ __forceinline__ void take(unsigned&, u64, u64&, int&) {}
  __device__ __forceinline__ u64 first_open() {  // (the cursor comes to stand on it)
    for (int e0 = cursor & ~31; e0 < n; e0 += 32) {
      const int i = e0 + lane_id();
      const unsigned mk = __ballot_sync(FV_FULL, i >= cursor && i < n && !(e[i] & 1ull));
      if (mk) {
        cursor = e0 + __ffs(mk) - 1;
        return e[cursor];
      }
    }
    cursor = n;
    return FV_EMPTY_KEY;
  }
  __device__ __forceinline__ void mark(u64) {  // the one first_open has just found
    __syncwarp();
    if (lane_id() == 0) e[cursor] |= 1ull;
    cursor++;
    __syncwarp();
  }
  __device__ __forceinline__ int filled() const { return n; }
  template <class Fn>
  __device__ __forceinline__ void each(Fn fn) {
    __syncwarp();
    for (int i = lane_id(); i < n; i += 32) fn(i, e[i]);
    __syncwarp();
  }
  template <class Fn>
  __device__ __forceinline__ void reopen(Fn fn) {
    __syncwarp();
    for (int e0 = 0; e0 < n; e0 += 32) {
      const int i = e0 + lane_id();
      const bool on = i < n;
      if (on) e[i] &= ~1ull;
      fn(on, on ? beam_id(e[i]) : 0u);
    }
    cursor = 0;
    __syncwarp();
  }
};

// Who computes a run of distances.  NW = 1: the warp itself.  NW > 1: the block's NW warps together; warp 0 runs the
// search and posts jobs, the others wait for them in team_serve.  A single search is a chain of memory trips, and when there
// are fewer searches than warps the rest of the SM can only help by shortening each link.
// A run of rows is a job that warp 0 takes part in (team_eval): all warps meet before and after it.  Scouting teams have a
// second kind, the links of a node with the distances of those that are not visited yet, which the others work out while
// warp 0 goes on (ask in beam_search).  Their jobs are done in the order they are posted; two may be under way; named barriers
// keep them apart.  (Those and their fences cost teams of eight 3 to 6 %: 600 queries of 4,000 x 1,536, ef 200 2,550 us with
// them, 2,400 with __syncthreads.)
struct TeamJob {
  const float* from;    // shared memory: the vector the distances are from
  int count;            // rows of the run, or the most links to read; -1: no more work
  int q_norm;           // Team::q_norm
  // of scouting teams only (TEAM_JOB_BYTES)
  const uint32_t* row;  // a node's link block (count, ids), or null: a run of rows
  const uint32_t* flat; // link blocks of all nodes, count_max + 1 words each, or null
  int slot;             // where a node's links go
  int unused[3];
};
static_assert(sizeof(TeamJob) == 48, "");
static constexpr size_t TEAM_JOB_BYTES = 16;  // what a team of eight has room for
static constexpr int NODE_SLOTS = 4;  // nodes whose links and distances are kept
static constexpr uint32_t NO_LINK = 0xFFFFFFFFu;
__host__ __device__ __forceinline__ int slot_links(int m0) { return (m0 + 31) & ~31; }
// bytes, a multiple of 16: the job of a run of rows; a scouting team's two jobs, the places of new links and the slots (lists of
// more than SCOUT_LINKS have none: a file may hold some of thousands)
__host__ __device__ __forceinline__ size_t team_smem(int nw, int m0) {
  return nw != SCOUT_WARPS ? TEAM_JOB_BYTES
                           : 2 * sizeof(TeamJob) + 2 * (SCOUT_LINKS + 4) * 4 + NODE_SLOTS * (size_t(slot_links(m0)) * 8 + 4);
}
// blocks of 256 threads per SM; those of scouting teams have 288
__host__ __device__ constexpr int team_threads(int nw) { return nw == 1 ? 256 : nw * 32; }
__host__ __device__ constexpr int team_blocks(int nw) { return nw == SCOUT_WARPS ? 2 : 3; }
// BYTES: the index has its rows as bytes too (a parameter, because the registers of the code for them cost searches without
// any 3 to 9 %: 10,000 queries of 20,000 x 128 floats, ef 64 674 us with it, 629 without; and the room for a query's bytes an
// SM's third block where rows are long: 2,000 queries of 4,000 x 4,096, ef 200 16.4 and 10.9 ms).
template <int NW, bool BYTES = false>
struct Team {
  static constexpr bool SCOUTS = NW == SCOUT_WARPS;
  const float* data;
  int pd;
  uint32_t* ids;  // shared memory: the rows of a run ...
  float* out;     // ... and their distances
  TeamJob* job;   // NW > 1, like the rest: one for even and one for odd jobs
  int links;      // slot_links
  uint32_t n;     // nodes
  VisitSet seen;  // as it was set up: for visit_seen
  mutable unsigned posted;  // jobs so far
  // BYTES: the rows' bytes; those of a query lie behind its floats.  q_norm: the sum of the query's squares, -1 where it has
  // no bytes and distances come from the floats
  const uint8_t* bytes = nullptr;
  int q_norm = -1;
  // of an even and an odd job: the places of the new links, their number in front
  __device__ __forceinline__ uint32_t* fresh(unsigned j) const { return reinterpret_cast<uint32_t*>(job + 2) + (j & 1) * (SCOUT_LINKS + 4); }
  __device__ __forceinline__ uint32_t* slot_cnt() const { return reinterpret_cast<uint32_t*>(job + 2) + 2 * (SCOUT_LINKS + 4); }
  __device__ __forceinline__ uint32_t* slot_ids(int s) const { return slot_cnt() + NODE_SLOTS + s * 2 * links; }  // NO_LINK: visited
  __device__ __forceinline__ float* slot_out(int s) const { return reinterpret_cast<float*>(slot_ids(s) + links); }
};
// Named barriers of scouting teams, one for even and one for odd jobs: 1, 2 a job is posted; 3, 4 a node's links are there; 5, 6 it is done;
// 7 the warps of a job among themselves.
__device__ __forceinline__ void team_arrive(int bar, int threads) {
  __syncwarp();
  asm volatile("fence.acq_rel.cta;" ::: "memory");
  asm volatile("bar.arrive %0, %1;" ::"r"(bar), "r"(threads) : "memory");
}
__device__ __forceinline__ void team_sync(int bar, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(threads) : "memory"); }
template <int NW, bool BYTES>
__device__ __forceinline__ unsigned team_post(const Team<NW, BYTES>& t, const TeamJob& job) {  // the job's number
  const unsigned j = t.posted++;
  if (lane_id() == 0) t.job[j & 1] = job;
  team_arrive(1 + int(j & 1), NW * 32);
  return j;
}
// The same distances from bytes (see fv_hnsw::d_bytes): whole numbers below 2^24, so the order of the sums changes nothing and
// the float is the one the reference's chain ends with.  A quarter of the memory, in loads of 16 bytes.
// (10,000 queries of 200,000 x 128, ef 64: 1,524 us from floats, 1,043 from bytes.)
template <int LPR>
__device__ __forceinline__ float byte_distance(const uint4* __restrict__ q, const uint8_t* __restrict__ row, int pd, int q_norm) {
  const uint4* r = reinterpret_cast<const uint4*>(row);
  unsigned bb = 0, qb = 0;
  const int chunks = row_bytes(pd) / 16;
  for (int c0 = lane_id() & (LPR - 1); c0 < chunks; c0 += 2 * LPR) {
    const int c1 = c0 + LPR;
    const uint4 b0 = __ldg(r + c0), b1 = c1 < chunks ? __ldg(r + c1) : make_uint4(0, 0, 0, 0);
    const uint4 q0 = q[c0], q1 = c1 < chunks ? q[c1] : make_uint4(0, 0, 0, 0);
    bb = __dp4a(b0.x, b0.x, __dp4a(b0.y, b0.y, __dp4a(b0.z, b0.z, __dp4a(b0.w, b0.w, bb))));
    qb = __dp4a(q0.x, b0.x, __dp4a(q0.y, b0.y, __dp4a(q0.z, b0.z, __dp4a(q0.w, b0.w, qb))));
    bb = __dp4a(b1.x, b1.x, __dp4a(b1.y, b1.y, __dp4a(b1.z, b1.z, __dp4a(b1.w, b1.w, bb))));
    qb = __dp4a(q1.x, b1.x, __dp4a(q1.y, b1.y, __dp4a(q1.z, b1.z, __dp4a(q1.w, b1.w, qb))));
  }
  int v = int(bb) - 2 * int(qb);
#pragma unroll
  for (int o = 1; o < LPR; o <<= 1) v += __shfl_xor_sync(FV_FULL, v, o);
  return float(v + q_norm);
}

template <bool IS_L2, int LPR, int NW, bool BYTES>
__device__ __forceinline__ void team_rows(const Team<NW, BYTES>& t, const float* from, int q_norm, int count, int first, int step) {
  const int sub = lane_id() & (LPR - 1), g = lane_id() / LPR;
  for (int i0 = first; i0 < count; i0 += step) {
    const int i = i0 + g;
    const size_t x = t.ids[min(i, count - 1)];  // (rows past the end: the last one again)
    const float d = BYTES && q_norm >= 0
                        ? byte_distance<LPR>(reinterpret_cast<const uint4*>(from + t.pd), t.bytes + x * row_bytes(t.pd), t.pd, q_norm)
                        : group_distance<IS_L2, LPR>(from, t.data + x * t.pd, t.pd);
    if (sub == 0 && i < count) t.out[i] = d;
  }
}
template <bool IS_L2, int NW, bool BYTES>
__device__ __forceinline__ void team_eval(const Team<NW, BYTES>& t, const float* from, int count) {
  __syncwarp();
  if (NW == 1) {
    team_rows<IS_L2, 4>(t, from, t.q_norm, count, 0, 8);
    __syncwarp();
  } else if (count <= 4) {  // one step of this warp: not worth the two barriers
    team_rows<IS_L2, 8>(t, from, t.q_norm, count, 0, 4);
    __syncwarp();
  } else if (Team<NW, BYTES>::SCOUTS) {
    const unsigned j = team_post(t, TeamJob{from, count, t.q_norm, nullptr, nullptr, 0});
    team_rows<IS_L2, 8>(t, from, t.q_norm, count, 0, 4 * NW);
    team_sync(5 + int(j & 1), NW * 32);
  } else {
    if (lane_id() == 0) {
      t.job->from = from;
      t.job->count = count;
      if (BYTES) t.job->q_norm = t.q_norm;
    }
    __syncthreads();
    team_rows<IS_L2, 8>(t, from, t.q_norm, count, 0, 4 * NW);
    __syncthreads();
  }
}
template <bool IS_L2, int NW, bool BYTES>
__device__ __forceinline__ void team_serve(const Team<NW, BYTES>& t) {  // warps 1 .. NW - 1
  const int w = int(threadIdx.x >> 5), sub = lane_id() & 7, g = lane_id() >> 3;
  for (unsigned j = 0;; ++j) {
    if (!Team<NW, BYTES>::SCOUTS) {
      __syncthreads();
      const int count = t.job->count;
      if (count < 0) return;
      team_rows<IS_L2, 8>(t, t.job->from, BYTES ? t.job->q_norm : -1, count, 4 * w, 4 * NW);
      __syncthreads();
      continue;
    }
    const int odd = int(j & 1);
    team_sync(1 + odd, NW * 32);
    const TeamJob job = t.job[odd];
    if (job.count < 0) return;
    if (!job.row) {
      team_rows<IS_L2, 8>(t, job.from, job.q_norm, job.count, 4 * w, 4 * NW);
    } else {
      uint32_t* ids = t.slot_ids(job.slot);
      float* out = t.slot_out(job.slot);
      uint32_t* fresh = t.fresh(j);
      if (w == 1) {
        const int lane = lane_id();
        // (rows of the searched graph are not written while a search runs: the non-coherent path is safe)
        const uint32_t x0 = lane < job.count ? __ldg(job.row + 1 + lane) : 0u;  // requested together with the count
        const uint32_t x1 = lane + 32 < job.count ? __ldg(job.row + 33 + lane) : 0u;
        const int cnt = min(int(__ldg(job.row)), job.count);
        const bool on0 = lane < cnt && FV_IDX_OK(x0, t.n, 2) && !visit_seen(t.seen, x0);
        const unsigned mask0 = __ballot_sync(FV_FULL, on0), below = (1u << lane) - 1u;
        int n = __popc(mask0);
        ids[lane] = on0 ? x0 : NO_LINK;
        if (on0) fresh[4 + __popc(mask0 & below)] = uint32_t(lane);
        if (cnt > 32) {
          const bool on1 = lane + 32 < cnt && FV_IDX_OK(x1, t.n, 2) && !visit_seen(t.seen, x1);
          const unsigned mask1 = __ballot_sync(FV_FULL, on1);
          ids[32 + lane] = on1 ? x1 : NO_LINK;
          if (on1) fresh[4 + n + __popc(mask1 & below)] = uint32_t(32 + lane);
          n += __popc(mask1);
        }
        if (lane == 0) {
          t.slot_cnt()[job.slot] = uint32_t(cnt);
          fresh[0] = uint32_t(n);
        }
        team_arrive(3 + odd, 64);
      }
      team_sync(7, (NW - 1) * 32);
      const int n = int(fresh[0]);
      for (int k0 = 4 * (w - 1); k0 < n; k0 += 4 * (NW - 1)) {
        const uint32_t at = fresh[4 + min(k0 + g, n - 1)], y = ids[at];  // (rows past the end: the last one again)
        const float d = BYTES && job.q_norm >= 0
                            ? byte_distance<8>(reinterpret_cast<const uint4*>(job.from + t.pd), t.bytes + size_t(y) * row_bytes(t.pd), t.pd, job.q_norm)
                            : group_distance_ahead<IS_L2>(job.from, t.data + size_t(y) * t.pd, t.pd);
        if (sub == 0) out[at] = d;
        // its own links, should it be expanded, are brought into L1: one word of each 32 bytes
        if (job.flat && sub * 8 <= job.count) {
          uint32_t word;
          asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(word) : "l"(job.flat + size_t(y) * (job.count + 1) + sub * 8));
        }
      }
    }
    team_arrive(5 + odd, NW * 32);
  }
}
template <int NW, bool BYTES>
__device__ __forceinline__ void team_dismiss(const Team<NW, BYTES>& t) {
  if (Team<NW, BYTES>::SCOUTS) {
    team_post(t, TeamJob{nullptr, -1, -1, nullptr, nullptr, 0});
  } else if (NW > 1) {
    __syncwarp();
    if (lane_id() == 0) t.job->count = -1;
    __syncthreads();
  }
}

// The greedy descent through layers top .. bottom + 1 (hnsw.rs:254-268, :334-347).  `rows(c, layer)` is a node's link
// block on a layer (count, then at most `width` ids).
template <bool IS_L2, int NW, bool BYTES, class Rows>
__device__ __forceinline__ void greedy_descent(const Team<NW, BYTES>& t, size_t n, Rows rows, int width, const float* sq, int top,
                                               int bottom, uint32_t& cur, float& curd, unsigned long long& n_dist,
                                               unsigned long long& n_exp) {
  const int lane = lane_id();
  for (int layer = top; layer > bottom; --layer) {
    bool changed = true;
    while (changed) {
      changed = false;
      const uint32_t* row = rows(cur, layer);
      const int cnt = min(int(row[0]), width);
      n_exp += 1;
      for (int c0 = 0; c0 < cnt; c0 += 32) {
        const int i = c0 + lane, m = min(32, cnt - c0);
        uint32_t x = 0;
        bool on = i < cnt;
        if (on) {
          x = row[1 + i];
          on = FV_IDX_OK(x, n, 4);
        }
        __syncwarp();
        if (i < cnt) t.ids[lane] = on ? x : cur;
        team_eval<IS_L2, NW>(t, sq, m);
        const float d = on ? t.out[lane] : INFINITY;
        n_dist += __popc(__ballot_sync(FV_FULL, on));
        // first minimum of the chunk, taken only if strictly below the current distance
        const unsigned better = __ballot_sync(FV_FULL, on && d < curd);
        if (better) {
          float md = d < curd ? d : INFINITY;
          for (int o = 16; o > 0; o >>= 1) md = fminf(md, __shfl_xor_sync(FV_FULL, md, o));
          const unsigned at = __ballot_sync(FV_FULL, on && d == md);
          cur = __shfl_sync(FV_FULL, x, __ffs(at) - 1);
          curd = md;
          changed = true;
        }
      }
    }
  }
}

// search_layer (hnsw.rs:179-226) from the entries of `best`, all of them not expanded and already in `seen`.
// `rows(c)` is the link block of node c on the searched layer (count, then at most `width` ids; width + 1 words are
// readable).  The reference's pair of heaps is ONE sorted list of ef entries with an "expanded" bit each: a candidate
// that has been evicted from `best` can only be popped after every entry of `best` has been expanded, and then it
// trips the stop test (hnsw.rs:203-205) unless its distance ties the current worst exactly -- see TIED_CAP.
// The unvisited neighbours of the expanded node are offered to the list in stored order, so the admission test
// (hnsw.rs:214) sees the same evolving bound as the sequential loop.  A search that fills more than half of the
// visited set's part in global memory stops with `over`.  `flat`: where the link blocks of all nodes lie one behind the other,
// width + 1 words each, if they do.  n_dist and n_exp grow by the distances evaluated and the nodes
// expanded.
template <bool IS_L2, int R, int NW, bool BYTES, class Rows>
__device__ __forceinline__ void beam_search(const Team<NW, BYTES>& t, size_t n, Rows rows, int width, const float* sq, Beam<R>& best,
                                            uint32_t* tied, VisitSet& seen, bool& over, bool& tie_lost,
                                            unsigned long long& n_dist, unsigned long long& n_exp,
                                            const uint32_t* flat = nullptr) {
  const int lane = lane_id();
  int ntied = 0;  // pushed-out entries still tied with the worst kept distance
  over = false;
  // scouting teams: the nodes whose links are in the slots (lane s: slot s); the slots of the jobs under way (the older
  // first, -1: none), whether the links of the older have been waited for, and its number; the next slot to take
  uint32_t kept = NO_LINK;
  int busy0 = -1, busy1 = -1, next_slot = 0;
  bool links_here = false;
  unsigned oldest = t.posted;
  auto links_done = [&]() {  // of the older job
    if (!links_here) team_sync(3 + int(oldest & 1), 64);
    links_here = true;
  };
  auto job_done = [&]() {
    links_done();
    team_sync(5 + int(oldest & 1), NW * 32);
    busy0 = busy1;
    busy1 = -1;
    links_here = false;
    ++oldest;
  };
  auto ask = [&](uint32_t node, int current) {  // returns the slot; one job at most is under way
    while (next_slot == current || next_slot == busy0) next_slot = (next_slot + 1) & (NODE_SLOTS - 1);
    const int slot = next_slot;
    next_slot = (slot + 1) & (NODE_SLOTS - 1);
    if (lane == slot) kept = node;
    team_post(t, TeamJob{sq, width, t.q_norm, rows(node), flat, slot});
    (busy0 < 0 ? busy0 : busy1) = slot;
    return slot;
  };
  u64 bound = best.last();
  constexpr bool CARRY = R > 0 && Team<NW, BYTES>::SCOUTS;  // (the other forms have no registers for it, or a cursor)
  u64 next = best.first_open();  // the nearest entry that is not expanded
  for (;;) {
    const u64 ck = next;
    bool in_beam = ck != FV_EMPTY_KEY;
    uint32_t c = beam_id(ck);
    if (ntied > 0) {
      // the smallest id among the tied entries; it goes first if the beam has nothing open or only a larger key
      uint32_t tmin = 0xFFFFFFFFu;
      for (int i = lane; i < ntied; i += 32) tmin = min(tmin, tied[i]);
      tmin = __reduce_min_sync(FV_FULL, tmin);
      const u64 tkey = (bound & 0xFFFFFFFF00000000ull) | (u64(tmin) << 1);
      if (!in_beam || tkey < ck) {
        __syncwarp();
        for (int i = lane; i < ntied; i += 32)
          if (tied[i] == tmin) tied[i] = tied[ntied - 1];  // ids are unique: one match
        __syncwarp();
        ntied--;
        in_beam = false;
        c = tmin;
      } else {
        in_beam = true;
      }
    } else if (!in_beam) {
      break;
    }
    if (in_beam) {
      best.mark(ck);
      if (ck == bound) bound |= 1ull;
      if (R > 0) next = best.first_open();
    }
    if (!FV_IDX_OK(c, n, 1)) break;
    n_exp += 1;
    const uint32_t* row = rows(c);
    uint32_t x_first = 0;
    int cnt, slot = 0;
    if (Team<NW, BYTES>::SCOUTS) {
      const unsigned known = __ballot_sync(FV_FULL, kept == c);
      if (known) {
        slot = __ffs(known) - 1;
      } else {
        if (busy1 >= 0) job_done();
        slot = ask(c, -1);
      }
      // the entry that is next in line now is expanded next unless a nearer one is found
      if (busy1 < 0 && next != FV_EMPTY_KEY && FV_IDX_OK(beam_id(next), n, 1) && !__any_sync(FV_FULL, kept == beam_id(next)))
        ask(beam_id(next), slot);
      if (busy1 == slot) job_done();
      if (busy0 == slot) links_done();
      cnt = int(t.slot_cnt()[slot]);
    } else {
      // the first 32 links are requested together with the count: one round trip, not two
      // (rows of the searched graph are not written while a search runs: the non-coherent path is safe)
      x_first = lane < width ? __ldg(row + 1 + lane) : 0u;
      cnt = min(int(__ldg(row)), width);
      if (R > 0 && next != FV_EMPTY_KEY) {
        // the entry that is next in line now is expanded next unless a nearer one is found: its links are on their way
        // (with the beam in shared memory finding it costs what this saves, and 1 to 3 % more)
        const uint32_t* nrow = rows(beam_id(next));
        if (lane * 32 <= width) asm volatile("prefetch.global.L1 [%0];" ::"l"(nrow + min(lane * 32, width)));
      }
    }
    for (int c0 = 0; c0 < cnt; c0 += 32) {
      const int i = c0 + lane;
      u64 key = FV_EMPTY_KEY;  // a new link's, in the lane of its place
      if (Team<NW, BYTES>::SCOUTS) {
        const uint32_t x = i < cnt ? t.slot_ids(slot)[i] : NO_LINK;
        const bool fresh = visit_warp(seen, x != NO_LINK, x);
        n_dist += __popc(__ballot_sync(FV_FULL, fresh));
        if (busy0 == slot) job_done();
        if (fresh) key = beam_key(t.slot_out(slot)[i], x);
      } else {
        uint32_t x = 0;
        if (i < cnt) x = c0 == 0 ? x_first : __ldg(row + 1 + i);
        const bool fresh = visit_warp(seen, i < cnt && FV_IDX_OK(x, n, 2), x);
        const unsigned fmask = __ballot_sync(FV_FULL, fresh);
        const int nfresh = __popc(fmask);
        if (nfresh == 0) continue;
        n_dist += nfresh;
        if (fresh) t.ids[__popc(fmask & ((1u << lane) - 1u))] = x;  // stored order
        team_eval<IS_L2, NW>(t, sq, nfresh);
        if (lane < nfresh) key = beam_key(t.out[lane], t.ids[lane]);
        __syncwarp();
      }
      // offered in stored order: admitted while the list is not full, or on a strictly smaller distance
      const uint32_t hi = uint32_t(key >> 32);
      unsigned pending = __ballot_sync(FV_FULL, hi < uint32_t(bound >> 32));
      // the nearest of them is admitted whatever happens to the others, unless the worst kept distance comes down to its own
      u64 nearest = FV_EMPTY_KEY;
      if (CARRY && pending) {
        const uint32_t near = __reduce_min_sync(FV_FULL, hi);
        const uint32_t low = __reduce_min_sync(FV_FULL, hi == near ? uint32_t(key) : 0xFFFFFFFFu);
        nearest = (u64(near) << 32) | low;
      }
      if (R > 0 && __popc(pending) > (R == 1 ? 8 : R == 2 ? 6 : R == 4 ? 5 : 4))
        best.take(pending, key, bound, ntied);  // (leaves them pending if ties at the cut need the order they came in)
      while (pending) {
        const int src = __ffs(pending) - 1;
        const u64 pushed = bound;  // the entry that falls off the end, if the beam is full
        best.insert(__shfl_sync(FV_FULL, key, src));
        bound = best.last();
        pending = __ballot_sync(FV_FULL, lane > src && hi < uint32_t(bound >> 32));
        // once the worst distance has gone down, nothing pushed out so far can tie with it any more
        const bool lower = uint32_t(bound >> 32) < uint32_t(pushed >> 32);
        ntied = lower ? 0 : ntied;
        if (!lower && !(pushed & 1ull)) {  // (an unused entry reads "expanded")
          if (ntied < TIED_CAP) {
            __syncwarp();
            if (lane == 0) tied[ntied] = beam_id(pushed);
            __syncwarp();
            ntied++;
          } else {
            tie_lost = true;
          }
        }
      }
      if (CARRY && nearest != FV_EMPTY_KEY) {
        if (uint32_t(nearest >> 32) == uint32_t(bound >> 32)) next = best.first_open();
        else next = nearest < next ? nearest : next;
      }
    }
    if (visit_overflow(seen)) {
      over = true;
      break;
    }
    if (!CARRY) next = best.first_open();
  }
  if (Team<NW, BYTES>::SCOUTS)
    while (busy0 >= 0) job_done();
  __syncwarp();
}
#endif

}  // namespace fv
