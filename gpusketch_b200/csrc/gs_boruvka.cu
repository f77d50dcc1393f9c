// gs_boruvka.cu - Boruvka emulation on the device (connected components / spanning forests).
//
// Follows CCSketchAlg::boruvka_emulation (src/cc_sketch_alg.cpp:491-540) round by round:
//   round 0   every vertex samples column `round0_col` of its own sketch (run_round_zero,
//             :250-271; the min-cut forests pass the column their stored sample index reached,
//             src/mc_sketch_alg.cpp:307-328);
//   round r   every current component XORs column r and the deterministic bucket of all its
//             members (Sketch::range_merge, src/sketch.cpp:172-195) and samples column r
//             (perform_boruvka_round, :273-407);
//   sampled edges are unioned into a lock-free DSU; a FAIL sample or a successful union marks
//   the round as modified; the loop stops at the first unmodified round, and a round
//   r >= num_samples is the reference's OutOfSamplesException (src/sketch.cpp:111-113,173-177).
//
// All rounds run inside one persistent kernel, so a query is one launch and one read-back instead of
// a host round trip per round.  A graph's blocks meet at a barrier between phases, in one of two scopes:
//   cluster   one thread-block cluster per graph: the barrier is the hardware's, and any number of
//             graphs share a launch without waiting for one another.  One or few graphs take wide
//             clusters (k_boruvka_flat, at the end: a round in two phases), many take narrow ones
//             (k_boruvka);
//   grid      one graph, or the large ones of several, over the whole GPU (k_boruvka, a cooperative
//             launch); the barrier is a counter in global memory, and every wait on it is bounded and
//             reports GS_DEV_ERR_TIMEOUT.
// gs_boruvka_scope chooses, and says with which figures.
//
// A round of k_boruvka after round 0 (barriers between the phases):
//   compress  parent[v] = root(v); in the same pass every component's size, every vertex's rank in
//             its component and the largest component
//   allocate  a root takes a run of the member list and one task per kPiece members
//   place     every vertex writes itself at its component's run, at its rank
//   gather    a warp per task loads its members' column r and deterministic bucket straight into
//             registers, XORs them and - when the task is the whole component - samples the result
//             and unions the sampled edge; pieces of larger components are XORed into their
//             accumulator row
//   big       components of several pieces (and the largest one) are sampled from their rows, which
//             are zeroed once read: rows are all zero between rounds and launches
// Sample (Bucket_Boruvka::is_good, include/bucket.h:65-67; Sketch::sample, src/sketch.cpp:110-132): the
// deterministic bucket is zero / good first, else the first good bucket by depth, one lane per bucket.
//
// Complement (sketch sets that XOR to zero, because every update reached both endpoints): the XOR of
// ALL of a graph's vertex sketches is zero, so its largest component's merged column equals the XOR of
// the columns of every vertex outside it.  The largest component's members are then never listed or
// read, and every gathered piece is folded into the largest component's row as well.
//
// Closed components (the same sketch sets): a component whose deterministic bucket is zero has no edge out,
// its merged columns are zero, and no other component can sample an edge into it; its vertices are marked
// and cost a load per round from then on (isolated vertices are most of a sparse R-MAT graph).
//
// Bound: latency.  A round is a chain of about a dozen dependent loads and five barriers, whatever the
// graph's size, until the graph is large enough for the member columns' bytes to matter: at V = 10^6 the
// rounds in which most vertices are still gathered take 150 to 350 us each, of which reading the columns
// is about 140, and listing the members 110.
// Measured (one query, us): V = 1024 199 -> 62, 16384 345 -> 188, 100003 835 -> 400, 131072 (R-MAT) 1062 ->
// 518, 1000003 4810 -> 1970; 256 graphs of 256 to 16384 vertices 2230 -> 1050.  Before, every phase of every
// graph was a grid phase of 444 blocks, all members were XORed into their component's row by atomics (82 of
// them per vertex and round at V = 10^6), and roots were appended to a list, so that a round had six barriers.
// DSU: CAS hooking of the larger root under the smaller (include/dsu.h:155-167 unions by random
// priority instead), so every component's root is its minimum vertex id and labels are deterministic;
// every walk is bounded by V+64 steps and reports GS_DEV_ERR_DSU_LIMIT.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>

#include "gs_dsu.cuh"
#include "gs_internal.h"

namespace cg = cooperative_groups;

namespace {

constexpr uint32_t kGood = 0, kZero = 1, kFail = 2;
constexpr uint32_t kClosed = 0xffffffffu;         // rank of a vertex whose component has no edge out
// Threads of a block.  Grid scope: one block per SM, so that the barrier has few arrivals.  Narrow
// clusters (many graphs): two blocks per SM, because a small graph's block mostly waits and another's fills
// in (256 graphs of up to 16384 vertices: 1.08 ms against 1.23 with wide ones).  Wide clusters: few graphs.
enum Scope { kGrid = 0, kNarrow = 1, kWide = 2 };
constexpr uint32_t threads_of(int scope, bool many = false) { return scope == kNarrow ? 512u : many ? 768u : 1024u; }
constexpr uint32_t kPiece = 16;                  // members of a component that one warp gathers
constexpr uint32_t kGroup = 4;                   // member rows a warp asks for together
constexpr uint32_t kRing = 2 * kGroup;           // member rows a warp has room for

__device__ __forceinline__ uint32_t lane_id() { return threadIdx.x & 31u; }


// loads of data written by other blocks earlier in the same launch bypass L1
__device__ __forceinline__ GsBucket ld_bucket_cg(const GsBucket* p) {
  const ulonglong2 v = __ldcg(reinterpret_cast<const ulonglong2*>(p));
  return GsBucket{v.x, v.y};
}

__device__ __forceinline__ bool is_good(const GsBucket& b, uint64_t csmix) {
  return gs_hash_tail(gs_key_mix(b.alpha) ^ csmix) == b.gamma;
}

// Sketch::sample on one column: all lanes of the warp call it and get the same answer.  The
// deterministic bucket and the first 32 column buckets are loaded together.
__device__ __forceinline__ void sample_warp(const GsBucket* col, const GsBucket* det, uint32_t bkt, uint64_t csmix,
                                            uint32_t* code, uint64_t* idx) {
  const uint32_t lane = lane_id();
  const GsBucket d = ld_bucket_cg(det);
  GsBucket b = GsBucket{0, 0};
  if (lane < bkt) b = ld_bucket_cg(col + lane);
  if (d.alpha == 0 && d.gamma == 0) { *code = kZero; *idx = 0; return; }
  if (is_good(d, csmix)) { *code = kGood; *idx = d.alpha; return; }
  for (uint32_t j0 = 0; j0 < bkt; j0 += 32) {
    const uint32_t j = j0 + lane;
    if (j0 > 0 && j < bkt) b = ld_bucket_cg(col + j);
    const bool good = j < bkt && is_good(b, csmix);
    const uint32_t m = __ballot_sync(0xffffffffu, good);
    if (m) {
      *code = kGood;
      *idx = __shfl_sync(0xffffffffu, b.alpha, __ffs(m) - 1);
      return;
    }
  }
  *code = kFail;
  *idx = 0;
}

// Sketch::sample of two vertices by an octet of lanes (round 0, where every vertex samples its own
// sketch: eight vertices per warp).  Lane k of the octet checks depths k, k+8, ...; a vertex's answer is
// the lowest good depth among the octet's lanes.  The deterministic buckets and the first eight depths of
// both vertices are loaded together: most vertices are decided by them, and a pass is one DRAM latency.
// The octets of a warp may belong to graphs of different bkt, so the pass count is the warp's largest: every
// lane runs the same passes and reaches every full-warp collective.
__device__ __forceinline__ void sample_octet2(const GsBucket* const col[2], const GsBucket* const det[2],
                                              const uint32_t bkt[2], const uint64_t csmix[2], const bool active[2],
                                              uint32_t code[2], uint64_t idx[2]) {
  const uint32_t lane = lane_id(), sub = lane & 7u, oct = lane >> 3;
  const uint32_t most = __reduce_max_sync(0xffffffffu, max(bkt[0], bkt[1]));
  GsBucket d[2], b[2];
  bool decided[2];
#pragma unroll
  for (int u = 0; u < 2; u++) {
    d[u] = active[u] ? ld_bucket_cg(det[u]) : GsBucket{0, 0};
    b[u] = active[u] && sub < bkt[u] ? ld_bucket_cg(col[u] + sub) : GsBucket{0, 0};
  }
#pragma unroll
  for (int u = 0; u < 2; u++) {
    code[u] = kFail;
    idx[u] = 0;
    decided[u] = !active[u];
    if (active[u]) {
      if (d[u].alpha == 0 && d[u].gamma == 0) { code[u] = kZero; decided[u] = true; }
      else if (is_good(d[u], csmix[u])) { code[u] = kGood; idx[u] = d[u].alpha; decided[u] = true; }
    }
  }
  for (uint32_t j0 = 0; j0 < most; j0 += 8) {
    if (__all_sync(0xffffffffu, decided[0] && decided[1])) break;
    const uint32_t j = j0 + sub;
    if (j0 > 0) {
#pragma unroll
      for (int u = 0; u < 2; u++)
        if (!decided[u] && j < bkt[u]) b[u] = ld_bucket_cg(col[u] + j);
    }
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const uint32_t m = __ballot_sync(0xffffffffu, !decided[u] && j < bkt[u] && is_good(b[u], csmix[u]));
      const uint32_t mine = (m >> (8u * oct)) & 0xffu;
      const uint64_t a = __shfl_sync(0xffffffffu, b[u].alpha, mine ? 8u * oct + (uint32_t)(__ffs(mine) - 1) : lane);
      if (!decided[u] && mine) {
        code[u] = kGood;
        idx[u] = a;
        decided[u] = true;
      }
    }
  }
}

// A parent entry through L1.  Within a phase a cached entry may be behind, but what it names is still an
// ancestor; the barrier that ends a phase makes every block's earlier writes visible to these loads.  The
// entries near a giant component's root are read by nearly every walk, and through L2 alone those reads
// queue on one slice.
__device__ __forceinline__ uint32_t ld_parent(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.global.ca.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// root of x, writing nothing (each parent entry has one writer in the compress phase)
__device__ __forceinline__ uint32_t cached_root(const uint32_t* parent, uint32_t x, uint32_t limit, uint32_t* err) {
  for (uint32_t it = 0; it < limit; it++) {
    const uint32_t p = ld_parent(parent + x);
    if (p == x) return x;
    x = p;
  }
  atomicOr(err, (uint32_t)GS_DEV_ERR_DSU_LIMIT);
  return x;
}

// Union of the components of s and d: the vertex that was hooked (its component's root until then), or ~0
// when they were one component already.  The parents were compressed when the phase began, so the first
// entries read are the roots unless another union hooked them since - then the CAS fails and both walks go
// on, from fresh loads.  A lower root that is out of date does no harm: parents are smaller than their
// children, so the larger root cannot lie above it.
__device__ __forceinline__ uint32_t cached_union(uint32_t* parent, uint32_t s, uint32_t d, uint32_t limit, uint32_t* err) {
  uint32_t a = ld_parent(parent + s), b = ld_parent(parent + d);
  for (uint32_t it = 0; it < limit; it++) {
    if (a == b) return 0xffffffffu;
    if (a < b) { const uint32_t t = a; a = b; b = t; }
    if (atomicCAS(&parent[a], a, b) == a) return a;
    for (; it < limit; it++) {
      const uint32_t pa = ld_volatile(parent + a), pb = ld_volatile(parent + b);
      if (pa == a && pb == b) break;
      a = pa;
      b = pb;
      if (a == b) return 0xffffffffu;
    }
  }
  atomicOr(err, (uint32_t)GS_DEV_ERR_DSU_LIMIT);
  return 0xffffffffu;
}

// 16-byte global -> shared copy that completes asynchronously
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const uint32_t sa = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// What the blocks of one graph share in a round; two sets, used in turn, so that one can be reset
// while the other is still read.
struct BorCounters {
  unsigned long long largest;  // (size << 32) | ~root of the largest component
  unsigned long long alloc;    // (members listed << 32) | tasks
  uint32_t nbig;
  uint32_t modified;           // some sample of the round failed or some union succeeded
};

struct BorArgs {
  const GsBucket* sk;          // sketch base the tenants' sk_off index into
  const GsBorTenant* tenants;  // device table, or nullptr: the single graph t0
  GsBorTenant t0;
  const uint32_t* qlist;       // cluster scope with a table: the tenant of every cluster
  uint32_t tenant;             // grid scope with a table: the tenant
  uint32_t T1;                 // grid scope over several graphs: entries of the tables, else 0
  const uint32_t* vtenant;     //   tenant of every vertex
  uint32_t vlo, vhi;           //   the graphs' vertices lie in [vlo, vhi)
  uint32_t* tmod;              //   [2][T1] the round was modified, zero at launch
  unsigned long long* tlargest;  // [2][T1] (size << 32) | ~root of the largest component, zero at launch
  uint32_t W;                  // accumulator row width, >= bkt_per_col + 1
  uint32_t R;                  // ring row width: the launch's largest bkt_per_col + 1
  uint32_t* parent;            // per vertex: DSU parent (vertex ids of the whole vertex space)
  uint32_t* size;              // per root: members
  uint32_t* rank;              // per vertex: place among its component's members
  uint32_t* off;               // per root: first member in list
  uint32_t* list;              // members grouped by component
  uint32_t* big;               // roots sampled from their accumulator row
  uint4* tasks;                // {root, first list position, members, pieces of the root}
  GsBucket* acc;               // [vertex][W]
  uint64_t* edge;              // per hooked vertex: the edge that joined its component to another; may be null
  uint32_t* status;            // [0] error bits [4] forest edges (with `edge`)
  uint32_t* out;               // one graph: result words in page-locked host memory (gs_boruvka_enqueue); or null
  uint32_t* labels;            // one graph: [V] its labels in page-locked host memory, may be null
  uint32_t* tstate;            // [tenant][4]: done, -, rounds, out of samples
  BorCounters* ctr;            // grid scope: [2], zero at launch
  uint32_t* barrier;           // grid scope: arrivals, zero at launch
  uint64_t wait_ns;            // grid scope: limit of one barrier wait
  uint32_t complement;         // the graph's sketches XOR to zero
};

// Barrier of a co-resident grid: arrivals are counted up and never reset, barrier k is complete at
// k * gridDim.x.  A wait polls (each poll is a round trip to L2, counted as kPollNs) and gives up
// after wait_ns or when another block did; the answer is the same for the whole block.
constexpr uint64_t kPollNs = 250;
__device__ bool grid_barrier(uint32_t* count, uint32_t target, uint32_t* err, uint64_t wait_ns) {
  __shared__ uint32_t s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t ok = 1, n;
    __threadfence();
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
    uint64_t waited = 0;
    for (uint32_t it = 0;; it++) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(n) : "l"(count) : "memory");
      if ((int32_t)(n - target) >= 0) break;
      waited += kPollNs;
      if (waited > wait_ns) {
        atomicOr(err, (uint32_t)GS_DEV_ERR_TIMEOUT);
        ok = 0;
        break;
      }
      if ((it & 63u) == 63u && (ld_volatile(err) & GS_DEV_ERR_TIMEOUT)) { ok = 0; break; }
    }
    __threadfence();
    s_ok = ok && !(ld_volatile(err) & GS_DEV_ERR_TIMEOUT);
  }
  __syncthreads();
  return s_ok != 0;
}

__device__ __forceinline__ uint64_t ld_volatile64(const unsigned long long* p) {
  return *reinterpret_cast<const volatile unsigned long long*>(p);
}

__device__ __forceinline__ void xor_row(GsBucket* row, uint32_t j, uint64_t a, uint64_t g) {
  atomicXor(reinterpret_cast<unsigned long long*>(&row[j].alpha), (unsigned long long)a);
  atomicXor(reinterpret_cast<unsigned long long*>(&row[j].gamma), (unsigned long long)g);
}

// What the kernels know of the graph that a thread works on.
struct Graph {
  uint32_t vlo, span;
  uint32_t* parent;
  uint64_t* edge;
  uint32_t* err;
};

// the edge of a sample, or ~0: anything but a pair of distinct vertices is a checksum collision
__device__ __forceinline__ uint64_t edge_of(const Graph& G, uint64_t idx) {
  const uint32_t s = (uint32_t)(idx >> 32), d = (uint32_t)idx;
  return s < G.span && d < G.span && s != d ? ((uint64_t)(G.vlo + s) << 32) | (G.vlo + d) : ~0ull;
}

// Every lane unions its edge (~0: none), so that up to 32 overlap.  A vertex is hooked once at most: its edge
// is kept at its place, and the hooked vertices' edges are the forest.
__device__ __forceinline__ void unite(const Graph& G, uint64_t e, uint32_t* s_hooked) {
  if (e == ~0ull) return;
  const uint32_t hooked = cached_union(G.parent, (uint32_t)(e >> 32), (uint32_t)e, G.span + 64, G.err);
  if (hooked == 0xffffffffu) return;
  atomicAdd(s_hooked, 1u);
  if (G.edge) G.edge[hooked] = e;
}

// Several graphs in one launch over one vertex range: a flag per graph says that its round was modified.  It
// is read before it is written: thousands of unions of one graph's round would queue on its line otherwise.
__device__ __forceinline__ void mark(uint32_t* flag) {
  if (!ld_volatile(flag)) *reinterpret_cast<volatile uint32_t*>(flag) = 1u;
}
__device__ __forceinline__ void unite_many(const BorArgs& A, const Graph& G, uint64_t e, uint32_t* tmod) {
  if (e == ~0ull) return;
  const uint32_t hooked = cached_union(G.parent, (uint32_t)(e >> 32), (uint32_t)e, G.span + 64, G.err);
  if (hooked != 0xffffffffu) mark(tmod + A.vtenant[hooked]);
}

// Round 0: every vertex samples its own sketch, an octet of lanes for two; the edges of `per` passes are
// collected one per lane and unioned together.
__device__ __forceinline__ void round_zero(const Graph& G, const GsBucket* sk, const GsBorTenant& T, uint32_t* rank,
                                           bool complement, uint32_t gwarp, uint32_t gwarps, uint32_t* s_mod,
                                           uint32_t* s_hooked) {
  const uint32_t lane = lane_id(), span = G.span;
  const uint32_t per = min(4u, max(1u, (span + 8 * gwarps - 1) / (8 * gwarps)));
  for (uint32_t base = gwarp * 8 * per; base < span; base += gwarps * 8 * per) {
    uint64_t mine = ~0ull;
    bool failed = false;
    for (uint32_t i = 0; i < per; i++) {
      const GsBucket *col[2], *det[2];
      bool active[2];
      uint32_t code[2];
      uint64_t idx[2];
      const uint32_t bkt[2] = {T.bkt, T.bkt};
      const uint64_t csmix[2] = {T.csmix, T.csmix};
#pragma unroll
      for (int u = 0; u < 2; u++) {
        const uint32_t k = base + 8 * i + 4 * u + (lane >> 3);
        active[u] = k < span;
        const GsBucket* own = sk + (size_t)(k < span ? k : 0u) * T.nb;
        col[u] = own + (size_t)T.round0_col * T.bkt;
        det[u] = own + (T.nb - 1);
      }
      sample_octet2(col, det, bkt, csmix, active, code, idx);
#pragma unroll
      for (int u = 0; u < 2; u++) {
        failed |= active[u] && code[u] == kFail;
        if (active[u] && (lane & 7u) == 0)
          rank[G.vlo + base + 8 * i + 4 * u + (lane >> 3)] = complement && code[u] == kZero ? kClosed : 0u;
        const uint64_t e = active[u] && code[u] == kGood ? edge_of(G, idx[u]) : ~0ull;
        const uint64_t x = __shfl_sync(0xffffffffu, e, (lane & 3u) * 8u);
        if ((lane >> 2) == 2 * i + u) mine = x;
      }
    }
    if (failed) *s_mod = 1;
    unite(G, mine, s_hooked);
  }
}

// The same for several graphs over one vertex range: octets of different graphs share a warp.
__device__ __forceinline__ void round_zero_many(const BorArgs& A, const Graph& G, const uint8_t* s_state,
                                                uint32_t gwarp, uint32_t gwarps) {
  const uint32_t lane = lane_id(), span = G.span;
  for (uint32_t base = gwarp * 32; base < span; base += gwarps * 32) {
    uint64_t mine = ~0ull;
    for (uint32_t i = 0; i < 4; i++) {
      const GsBucket *col[2], *det[2];
      bool active[2];
      uint32_t code[2], bkt[2], t[2], vbase[2], V[2];
      uint64_t idx[2], csmix[2];
#pragma unroll
      for (int u = 0; u < 2; u++) {
        const uint32_t k = base + 8 * i + 4 * u + (lane >> 3);
        t[u] = k < span ? A.vtenant[G.vlo + k] : 0u;
        active[u] = k < span && s_state[t[u]] == 0;
        const GsBorTenant& T = A.tenants[t[u]];
        const GsBucket* own = A.sk + T.sk_off + (active[u] ? (size_t)(G.vlo + k - T.vbase) * T.nb : (size_t)0);
        bkt[u] = active[u] ? T.bkt : 0u;
        csmix[u] = T.csmix;
        vbase[u] = T.vbase;
        V[u] = T.V;
        col[u] = own + (size_t)T.round0_col * T.bkt;
        det[u] = own + (T.nb - 1);
      }
      sample_octet2(col, det, bkt, csmix, active, code, idx);
#pragma unroll
      for (int u = 0; u < 2; u++) {
        uint64_t e = ~0ull;
        if (active[u] && code[u] == kFail) mark(A.tmod + t[u]);
        if (active[u] && (lane & 7u) == 0)
          A.rank[G.vlo + base + 8 * i + 4 * u + (lane >> 3)] = A.complement && code[u] == kZero ? kClosed : 0u;
        if (active[u] && code[u] == kGood) e = edge_of(Graph{vbase[u], V[u], nullptr, nullptr, nullptr}, idx[u]);
        const uint64_t x = __shfl_sync(0xffffffffu, e, (lane & 3u) * 8u);
        if ((lane >> 2) == 2 * i + u) mine = x;
      }
    }
    unite_many(A, G, mine, A.tmod);
  }
}

// The answer of a query of one graph, written to the host from the kernel: no read-back is queued behind it,
// and no clearing.  `meet` is the graph's barrier.
template <typename Meet>
__device__ __forceinline__ void write_answer(const BorArgs& A, const Graph& G, uint32_t gtid, uint32_t gthreads,
                                             Meet&& meet) {
  uint32_t count = 0;
  for (uint32_t v = G.vlo + gtid; v < G.vlo + G.span; v += gthreads) {
    const uint32_t r = __ldcg(&G.parent[v]);
    if (A.labels) A.labels[v] = r;
    count += r == v;
  }
  count = __reduce_add_sync(0xffffffffu, count);
  if (lane_id() == 0 && count) atomicAdd(&A.status[17], count);
  if (!meet(nullptr)) return;
  if (gtid == 0) {
    for (int i = 0; i < 18; i++) A.out[i] = ld_volatile(&A.status[i]);
    A.status[0] = 0;   // read with this answer: the calls queued behind it start clean
  }
}

// exclusive scan over the block (every thread calls it), and the block's total
template <uint32_t kWarps>
__device__ __forceinline__ unsigned long long block_scan(unsigned long long x, unsigned long long* s_sums,
                                                         unsigned long long* total) {
  const uint32_t lane = lane_id(), w = threadIdx.x >> 5;
  unsigned long long inc = x;
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long y = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= (uint32_t)o) inc += y;
  }
  if (lane == 31) s_sums[w] = inc;
  __syncthreads();
  unsigned long long all = lane < kWarps ? s_sums[lane] : 0ull, before = lane < w ? all : 0ull;
  for (int o = 16; o > 0; o >>= 1) {
    all += __shfl_xor_sync(0xffffffffu, all, o);
    before += __shfl_xor_sync(0xffffffffu, before, o);
  }
  *total = all;
  return before + inc - x;
}

// SLOTS: buckets of a row (bkt_per_col + 1) per lane; at most 64 registers in either scope.  Dynamic shared
// memory: kRing rows of R buckets per warp.
// MANY (grid scope): the launch's graphs are the tenants whose tstate word 0 is zero; their vertices lie among
// others' in one range, their rounds advance together, and a graph whose round was unmodified stops taking
// part, so each one's partition, round count and out-of-samples status equal a query run alone.  Two more
// tables in dynamic shared memory: every tenant's complement component and state.
template <int SCOPE, int SLOTS, bool MANY = false>
__global__ void __launch_bounds__(threads_of(SCOPE, MANY), SCOPE == kNarrow ? 2 : 1) k_boruvka(const BorArgs A) {
  static_assert(!MANY || SCOPE == kGrid, "several graphs share a launch on clusters or on the whole grid");
  constexpr bool CLUSTER = SCOPE != kGrid;
  constexpr uint32_t kThreads = threads_of(SCOPE, MANY), kWarps = kThreads / 32;
  constexpr uint32_t kTable = CLUSTER ? 1024 : 2048;   // slots of a block's table of roots, at most kThreads of them
  extern __shared__ __align__(16) GsBucket s_ring[];
  __shared__ BorCounters s_ctr[2];                 // cluster scope: the first block's are the cluster's
  __shared__ uint32_t s_row[4][SLOTS * 32];        // the block's share of the largest component's row
  __shared__ uint32_t s_key[kTable], s_cnt[kTable];  // roots among a block's vertices, and their members there
  __shared__ unsigned long long s_sums[kWarps], s_best, s_base;
  __shared__ uint32_t s_mod, s_hooked;             // a sample failed, unions of the phase
  const uint32_t lane = lane_id();

  BorCounters* ctr;
  uint32_t t, block, blocks;
  if constexpr (CLUSTER) {
    cg::cluster_group cl = cg::this_cluster();
    block = cl.block_rank();
    blocks = cl.num_blocks();
    ctr = cl.map_shared_rank(s_ctr, 0);
    t = A.qlist ? A.qlist[blockIdx.x / blocks] : 0u;
  } else {
    block = blockIdx.x;
    blocks = gridDim.x;
    ctr = A.ctr;
    t = A.tenant;
  }
  const GsBorTenant T = A.tenants ? A.tenants[t] : A.t0;   // MANY: not used
  const uint32_t vlo = MANY ? A.vlo : T.vbase, vend = MANY ? A.vhi : T.vbase + T.V, span = vend - vlo;
  const uint32_t W = A.W, R = A.R;
  uint32_t bkt = T.bkt;                                    // MANY: of the component at hand
  uint32_t* const s_comp = reinterpret_cast<uint32_t*>(s_ring + (size_t)kWarps * kRing * R);   // MANY: [T1]
  uint8_t* const s_state = reinterpret_cast<uint8_t*>(s_comp + A.T1);   // MANY: [T1] 0 running, 1 done, 2 last round
  const uint32_t gtid = block * kThreads + threadIdx.x, gthreads = blocks * kThreads;
  const uint32_t gwarp = gtid >> 5, gwarps = gthreads >> 5;
  const uint32_t limit = span + 64;
  uint32_t* const err = A.status;
  uint32_t* const list = A.list + vlo;
  uint32_t* const big = A.big + vlo;
  uint4* const tasks = A.tasks + vlo;
  const GsBucket* const sk = A.sk + T.sk_off;
  uint32_t* const ts = A.tstate + 4 * t;
  uint32_t barriers = 0;

  // Everything the block did becomes visible to the graph's other blocks; false: a wait gave up.
  // `flag`, when given, is set to one if a sample of the block failed or one of its unions succeeded.
  auto meet = [&](uint32_t* flag) -> bool {
    if (flag) {
      __syncthreads();
      if (threadIdx.x == 0) {
        if (s_mod | s_hooked) *reinterpret_cast<volatile uint32_t*>(flag) = 1u;
        if (s_hooked && A.edge) atomicAdd(&A.status[4], s_hooked);
        s_mod = 0;
        s_hooked = 0;
      }
    }
    if constexpr (CLUSTER) {
      cg::this_cluster().sync();
      return true;
    } else {
      barriers += blocks;
      return grid_barrier(A.barrier, barriers, err, A.wait_ns);
    }
  };
  const Graph G{vlo, span, A.parent, A.edge, err};

  if (threadIdx.x == 0) { s_mod = 0; s_hooked = 0; s_best = 0; }
  if (CLUSTER && threadIdx.x < 2 * sizeof(BorCounters) / sizeof(uint32_t))
    reinterpret_cast<uint32_t*>(s_ctr)[threadIdx.x] = 0;
  for (uint32_t i = threadIdx.x; i < 4 * SLOTS * 32; i += kThreads) (&s_row[0][0])[i] = 0;
  for (uint32_t v = vlo + gtid; v < vend; v += gthreads) {
    A.parent[v] = v;
    A.size[v] = 0;
  }
  // with `out` the launch owns the status words: the error bits of earlier ingest calls move to word 16
  if (A.out && gtid == 0) {
    A.status[16] = A.status[0];
    A.status[17] = 0;
    for (int i = 0; i < 16; i++) A.status[i] = 0;
  }
  if (!meet(nullptr)) return;
  uint32_t rounds = 0, oos = MANY ? 0 : T.round0_col >= T.ns;   // OutOfSamplesException before the first round
  if constexpr (MANY) {
    for (uint32_t i = threadIdx.x; i < A.T1; i += kThreads) s_state[i] = A.tstate[4 * i] ? 1 : 0;
    __syncthreads();
    round_zero_many(A, G, s_state, gwarp, gwarps);
  } else {
    if (!oos) round_zero(G, sk, T, A.rank, A.complement, gwarp, gwarps, &s_mod, &s_hooked);
  }

  for (uint32_t round = 0; !oos || round;) {
    if constexpr (MANY) {
      if (!meet(nullptr)) return;
      // every block decides the same from the same flags
      bool some = false;
      for (uint32_t i = threadIdx.x; i < A.T1; i += kThreads) {
        if (s_state[i] == 2) s_state[i] = 1;
        if (s_state[i]) continue;
        if (!ld_volatile(&A.tmod[(round & 1) * A.T1 + i])) {
          s_state[i] = 1;
          continue;
        }
        some = true;
        const bool last = round + 1 >= A.tenants[i].ns;   // out of samples: only the labels are still compressed
        if (last) s_state[i] = 2;
        if (block == 0) {
          A.tstate[4 * i + 2] = round + 1;
          A.tstate[4 * i + 3] = last;
        }
      }
      if (!__syncthreads_or(some)) break;
      ++round;
    } else {
      if (!meet(&ctr[round & 1].modified)) return;
      if (!ld_volatile(&ctr[round & 1].modified)) break;
      rounds = ++round;
      oos = rounds >= T.ns;
    }
    BorCounters* const c = ctr + (round & 1);

    // ---- compress, sizes, ranks, largest.  A block counts the members of every root among 1024 vertices
    //      in shared memory and adds each count to the root's size once: atomics on the size of a giant
    //      component's root queue in L2, one per warp took 170 us of a round at V = 10^6 ----
    unsigned long long best = 0;
    for (uint32_t base = block * kThreads; base < span; base += gthreads) {
      for (uint32_t i = threadIdx.x; i < kTable; i += kThreads) {
        s_key[i] = 0xffffffffu;
        s_cnt[i] = 0;
      }
      __syncthreads();
      const uint32_t v = vlo + base + threadIdx.x;
      uint32_t r = 0xffffffffu;
      if (v < vend && (!MANY || s_state[A.vtenant[v]] != 1) && !(A.complement && __ldcg(&A.rank[v]) == kClosed)) {
        r = cached_root(A.parent, v, limit, err);
        A.parent[v] = r;
      }
      const uint32_t peers = __match_any_sync(0xffffffffu, r);
      const uint32_t lead = __ffs(peers) - 1;
      uint32_t h = 0, local = 0;
      if (r != 0xffffffffu && lane == lead) {
        h = __umulhi(r * 0x9E3779B1u, kTable);   
        for (;;) {
          const uint32_t k = atomicCAS(&s_key[h], 0xffffffffu, r);
          if (k == 0xffffffffu || k == r) break;
          h = (h + 1) & (kTable - 1);
        }
        local = atomicAdd(&s_cnt[h], (uint32_t)__popc(peers));
      }
      __syncthreads();
      for (uint32_t i = threadIdx.x; i < kTable; i += kThreads) {
        const uint32_t root = s_key[i];
        if (root == 0xffffffffu) continue;
        const uint32_t n = s_cnt[i], old = atomicAdd(&A.size[root], n);
        s_cnt[i] = old;
        // the last block to add to a component sees its full size
        const unsigned long long key = ((unsigned long long)(old + n) << 32) | (0xffffffffu - root);
        if constexpr (MANY) {
          if (old + n > 1) atomicMax(&A.tlargest[(round & 1) * A.T1 + A.vtenant[root]], key);
        } else {
          best = key > best ? key : best;
        }
      }
      __syncthreads();
      if (r != 0xffffffffu && lane == lead) local += s_cnt[h];
      local = __shfl_sync(0xffffffffu, local, lead);
      if (r != 0xffffffffu) A.rank[v] = local + __popc(peers & ((1u << lane) - 1u));
      __syncthreads();
    }
    if constexpr (!MANY) {
      for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o);
        best = other > best ? other : best;
      }
      if (lane == 0 && best) atomicMax(&s_best, best);
      __syncthreads();
      if (threadIdx.x == 0) {
        if (s_best) atomicMax(&c->largest, s_best);
        s_best = 0;
      }
    }
    if (!meet(nullptr)) return;
    if (oos) break;   // the labels are compressed
    // the component whose column is the XOR of everything outside it, or ~0: none
    uint32_t comp = 0xffffffffu;
    if constexpr (MANY) {
      for (uint32_t i = threadIdx.x; i < A.T1; i += kThreads) {
        const uint64_t top = ld_volatile64(&A.tlargest[(round & 1) * A.T1 + i]);
        s_comp[i] = A.complement && s_state[i] == 0 && (top >> 32) > 1ull ? 0xffffffffu - (uint32_t)top : 0xffffffffu;
      }
      __syncthreads();
    } else {
      const uint64_t top = ld_volatile64(&c->largest);
      if (A.complement && (top >> 32) > 1ull) comp = 0xffffffffu - (uint32_t)top;
    }
    // sizes that count: not those of the complement components, nor of graphs that are out of samples
    const auto listed = [&](uint32_t v, uint32_t size) -> uint32_t {
      if constexpr (MANY) {
        if (!size) return 0u;
        const uint32_t i = A.vtenant[v];
        return s_state[i] == 0 && v != s_comp[i] ? size : 0u;
      } else {
        return v == comp ? 0u : size;
      }
    };

    // ---- allocate: member runs and tasks, one reservation per block; runs and tasks come in one order ----
    {
      const uint32_t share = (span + blocks - 1) / blocks;
      const uint32_t v0 = vlo + min(span, block * share), v1 = vlo + min(span, block * share + share);
      // only roots have a size; the first vertex's stays in its register for the second pass
      const uint32_t first = v0 + threadIdx.x < v1 ? __ldcg(&A.size[v0 + threadIdx.x]) : 0u;
      unsigned long long mine = 0, total;
      for (uint32_t v = v0 + threadIdx.x; v < v1; v += kThreads) {
        const uint32_t n = listed(v, v == v0 + threadIdx.x ? first : __ldcg(&A.size[v]));
        mine += ((unsigned long long)n << 32) | ((n + kPiece - 1) / kPiece);
      }
      unsigned long long at = block_scan<kWarps>(mine, s_sums, &total);
      if (threadIdx.x == 0) s_base = total ? atomicAdd(&c->alloc, total) : 0ull;
      __syncthreads();
      at += s_base;
      for (uint32_t vb = v0 + (threadIdx.x & ~31u); vb < v1; vb += kThreads) {
        const uint32_t v = vb + lane;
        const uint32_t size = v >= v1 ? 0u : v == v0 + threadIdx.x ? first : __ldcg(&A.size[v]);
        const uint32_t n = v < v1 ? listed(v, size) : 0u, pieces = (n + kPiece - 1) / kPiece;
        const uint32_t start = (uint32_t)(at >> 32), task = (uint32_t)at;
        if (n) A.off[v] = start;
        if (pieces == 1) tasks[task] = make_uint4(v, start, n, 1u);
        at += ((unsigned long long)n << 32) | pieces;
        for (uint32_t m = __ballot_sync(0xffffffffu, pieces > 1); m; m &= m - 1) {
          const uint32_t src = __ffs(m) - 1;   // a larger component's tasks are written by the warp
          const uint32_t hn = __shfl_sync(0xffffffffu, n, src), hp = __shfl_sync(0xffffffffu, pieces, src);
          const uint32_t h0 = __shfl_sync(0xffffffffu, start, src), ht = __shfl_sync(0xffffffffu, task, src);
          for (uint32_t p = lane; p < hp; p += 32)
            tasks[ht + p] = make_uint4(vb + src, h0 + p * kPiece, min(kPiece, hn - p * kPiece), hp);
        }
        const bool is_big = pieces > 1 || (size && (MANY ? v == s_comp[A.vtenant[v]] : v == comp));
        const uint32_t bm = __ballot_sync(0xffffffffu, is_big);
        if (bm) {
          uint32_t b = 0;
          if (lane == 0) b = atomicAdd(&c->nbig, (uint32_t)__popc(bm));
          b = __shfl_sync(0xffffffffu, b, 0);
          if (is_big) big[b + __popc(bm & ((1u << lane) - 1u))] = v;
        }
      }
    }
    if (!meet(nullptr)) return;

    // ---- place the members; clear the sizes and the other counter set for the next round ----
    for (uint32_t v = vlo + gtid; v < vend; v += gthreads) {
      uint32_t out_of = comp;
      if constexpr (MANY) {
        const uint32_t i = A.vtenant[v];
        if (s_state[i] == 1) continue;
        if (s_state[i] == 2) {
          A.size[v] = 0;
          continue;
        }
        out_of = s_comp[i];
      }
      const uint32_t r = __ldcg(&A.parent[v]), rank = __ldcg(&A.rank[v]);
      if (A.complement && rank == kClosed) continue;
      if (r != out_of) list[__ldcg(&A.off[r]) + rank] = v;
      if (r == v) A.size[v] = 0;
    }
    if (gtid < sizeof(BorCounters) / sizeof(uint32_t))
      reinterpret_cast<volatile uint32_t*>(ctr + ((round + 1) & 1))[gtid] = 0;
    if constexpr (MANY) {
      for (uint32_t i = gtid; i < A.T1; i += gthreads) {
        A.tmod[((round + 1) & 1) * A.T1 + i] = 0;
        A.tlargest[((round + 1) & 1) * A.T1 + i] = 0;
      }
    }
    if (!meet(nullptr)) return;

    // ---- gather: each warp a run of tasks, whose members are one run of the list.  The members' rows
    //      stream through a ring in shared memory, kRing of them on their way at once ----
    {
      const uint32_t ntasks = (uint32_t)ld_volatile64(&c->alloc);
      const uint32_t per = (ntasks + gwarps - 1) / gwarps;
      const uint32_t t0 = min(ntasks, gwarp * per), t1 = min(ntasks, t0 + per);
      GsBucket* const ring = s_ring + (size_t)(threadIdx.x >> 5) * kRing * R;
      uint64_t ca[SLOTS] = {}, cb[SLOTS] = {};      // the run's share of the largest component's row
      uint64_t ma[SLOTS] = {}, mb[SLOTS] = {};      // pieces of one larger component
      uint32_t mroot = 0xffffffffu, held = 0;
      uint64_t mine = ~0ull;
      // MANY: the graph that ca and cb belong to, its complement component and its row width
      uint32_t ct = 0xffffffffu, crow = 0xffffffffu, cbkt = 0, mbkt = 0;
      auto flush_complement = [&]() {
        if (crow == 0xffffffffu) return;
#pragma unroll
        for (int k = 0; k < SLOTS; k++) {
          const uint32_t j = lane + 32u * k;
          if (j <= cbkt && (ca[k] | cb[k])) xor_row(A.acc + (size_t)crow * W, j, ca[k], cb[k]);
          ca[k] = cb[k] = 0;
        }
      };
      uint32_t* const tmod = MANY ? A.tmod + (round & 1) * A.T1 : nullptr;
      auto join = [&](uint64_t e) {
        if constexpr (MANY) unite_many(A, G, e, tmod);
        else unite(G, e, &s_hooked);
      };
      auto flush_pieces = [&]() {
        if (mroot == 0xffffffffu) return;
#pragma unroll
        for (int k = 0; k < SLOTS; k++) {
          const uint32_t j = lane + 32u * k;
          if (j <= (MANY ? mbkt : bkt) && (ma[k] | mb[k])) xor_row(A.acc + (size_t)mroot * W, j, ma[k], mb[k]);
          ma[k] = mb[k] = 0;
        }
        mroot = 0xffffffffu;
      };
      if (t0 < t1) {
        const uint4 last = __ldcg(&tasks[t1 - 1]);
        const uint32_t m0 = __ldcg(&tasks[t0].y), total = last.y + last.z - m0;
        // lane l holds list entries l of the current and the next 32
        uint32_t now = lane < total ? __ldcg(&list[m0 + lane]) : vlo;
        uint32_t then = 32 + lane < total ? __ldcg(&list[m0 + 32 + lane]) : vlo;
        uint32_t next = 0;   // the member whose row is asked for next
        // MANY: first bucket of lane l's member, and its graph's bkt << 16 | nb
        uint64_t now_at = 0;
        uint32_t now_geo = 0;
        auto look_up = [&]() {
          if constexpr (MANY) {
            const GsBorTenant& M = A.tenants[A.vtenant[now]];
            now_at = M.sk_off + (uint64_t)(now - M.vbase) * M.nb;
            now_geo = (M.bkt << 16) | M.nb;
          }
        };
        look_up();
        auto ask = [&]() {   // kGroup rows, one commit
#pragma unroll
          for (uint32_t u = 0; u < kGroup; u++) {
            const GsBucket* vb;
            uint32_t b = bkt, nb = T.nb;
            if constexpr (MANY) {
              vb = A.sk + __shfl_sync(0xffffffffu, now_at, (next + u) & 31u);
              const uint32_t geo = __shfl_sync(0xffffffffu, now_geo, (next + u) & 31u);
              b = geo >> 16;
              nb = geo & 0xffffu;
            } else {
              vb = sk + (size_t)(__shfl_sync(0xffffffffu, now, (next + u) & 31u) - vlo) * T.nb;
            }
            if (next + u >= total) continue;
            GsBucket* to = ring + ((next + u) % kRing) * R;
#pragma unroll
            for (int k = 0; k < SLOTS; k++) {
              const uint32_t j = lane + 32u * k;
              if (j <= b) cp_async16(to + j, vb + (j < b ? round * b + j : nb - 1));
            }
          }
          cp_async_commit();
          next += kGroup;
          if ((next & 31u) == 0) {
            now = then;
            look_up();
            then = next + 32 + lane < total ? __ldcg(&list[m0 + next + 32 + lane]) : vlo;
          }
        };
        ask();
        ask();
        uint32_t done = 0;
        uint4 batch = make_uint4(0, 0, 0, 0);
        uint32_t batch_t = 0, batch_base = 0, batch_V = 0, batch_bkt = 0;   // MANY: the tasks' graphs
        uint64_t batch_cs = 0, csmix = T.csmix;
        Graph H = G;
        for (uint32_t tk = t0; tk < t1; tk++) {
          if (((tk - t0) & 31u) == 0 && tk + lane < t1) {
            batch = __ldcg(&tasks[tk + lane]);
            if constexpr (MANY) {
              batch_t = A.vtenant[batch.x];
              const GsBorTenant& M = A.tenants[batch_t];
              batch_base = M.vbase;
              batch_V = M.V;
              batch_bkt = M.bkt;
              batch_cs = M.csmix;
            }
          }
          if constexpr (MANY) {
            const uint32_t src = (tk - t0) & 31u, tt = __shfl_sync(0xffffffffu, batch_t, src);
            bkt = __shfl_sync(0xffffffffu, batch_bkt, src);
            csmix = __shfl_sync(0xffffffffu, batch_cs, src);
            H.vlo = __shfl_sync(0xffffffffu, batch_base, src);
            H.span = __shfl_sync(0xffffffffu, batch_V, src);
            if (tt != ct) {
              flush_complement();
              ct = tt;
              crow = s_comp[tt];
              cbkt = bkt;
            }
          }
          const uint32_t root = __shfl_sync(0xffffffffu, batch.x, (tk - t0) & 31u);
          const uint32_t n = __shfl_sync(0xffffffffu, batch.z, (tk - t0) & 31u);
          const uint32_t pieces = __shfl_sync(0xffffffffu, batch.w, (tk - t0) & 31u);
          uint64_t a[SLOTS] = {}, g[SLOTS] = {};
#pragma unroll 1
          for (uint32_t i = 0; i < n; i++) {
            if (done % kGroup == 0) {        // the group before the last one asked for has landed
              cp_async_wait<1>();
              __syncwarp();
            }
            const GsBucket* row = ring + (done % kRing) * R;
#pragma unroll
            for (int k = 0; k < SLOTS; k++) {
              const uint32_t j = lane + 32u * k;
              if (j <= bkt) {
                const GsBucket b = row[j];
                a[k] ^= b.alpha;
                g[k] ^= b.gamma;
              }
            }
            if (++done % kGroup == 0) {      // its rows are read: the next group takes their place
              __syncwarp();
              ask();
            }
          }
          if ((MANY ? crow : comp) != 0xffffffffu) {
#pragma unroll
            for (int k = 0; k < SLOTS; k++) { ca[k] ^= a[k]; cb[k] ^= g[k]; }
          }
          if (pieces > 1) {
            if (root != mroot) {
              flush_pieces();
              mroot = root;
              mbkt = bkt;
            }
#pragma unroll
            for (int k = 0; k < SLOTS; k++) { ma[k] ^= a[k]; mb[k] ^= g[k]; }
            continue;
          }
          // the whole component: sample it from the registers
          uint64_t da = 0, dg = 0;
          uint32_t good[SLOTS], det_good = 0;
#pragma unroll
          for (int k = 0; k < SLOTS; k++) {
            const uint32_t j = lane + 32u * k;
            if (bkt / 32u == (uint32_t)k) {
              da = __shfl_sync(0xffffffffu, a[k], bkt & 31u);
              dg = __shfl_sync(0xffffffffu, g[k], bkt & 31u);
            }
            good[k] = __ballot_sync(0xffffffffu, j <= bkt && is_good(GsBucket{a[k], g[k]}, csmix));
            if (bkt / 32u == (uint32_t)k) det_good = (good[k] >> (bkt & 31u)) & 1u;
          }
          uint64_t e = ~0ull;
          if ((da | dg) == 0ull) {
            // no edge out, now or later: its members are not looked at again
            if (A.complement && lane < n) A.rank[__ldcg(&list[m0 + done - n + lane])] = kClosed;
          } else {
            uint32_t at = 0xffffffffu;   // the first good depth, but the deterministic bucket before any
#pragma unroll
            for (int k = SLOTS - 1; k >= 0; k--)
              if (good[k]) at = 32u * k + (__ffs(good[k]) - 1);
            if (det_good) at = bkt;
            if (at == 0xffffffffu) {     // FAIL
              if constexpr (MANY) mark(tmod + ct);
              else s_mod = 1;
            } else {
              uint64_t idx = 0;
#pragma unroll
              for (int k = 0; k < SLOTS; k++)
                if (at / 32u == (uint32_t)k) idx = __shfl_sync(0xffffffffu, a[k], at & 31u);
              e = edge_of(H, idx);
            }
          }
          if (lane == held) mine = e;
          if (++held == 32) {
            join(mine);
            __syncwarp();
            mine = ~0ull;
            held = 0;
          }
        }
        if (held) join(mine);
        flush_pieces();
        if constexpr (MANY) flush_complement();
      }
      if (!MANY && comp != 0xffffffffu) {
        // one warp's row at a time would queue on the row's L2 lines: combined per block first
        if (t0 < t1) {
#pragma unroll
          for (int k = 0; k < SLOTS; k++) {
            const uint32_t j = lane + 32u * k;
            if (j <= bkt && (ca[k] | cb[k])) {
              atomicXor(&s_row[0][j], (uint32_t)ca[k]);
              atomicXor(&s_row[1][j], (uint32_t)(ca[k] >> 32));
              atomicXor(&s_row[2][j], (uint32_t)cb[k]);
              atomicXor(&s_row[3][j], (uint32_t)(cb[k] >> 32));
            }
          }
        }
        __syncthreads();
        for (uint32_t j = threadIdx.x; j <= bkt; j += kThreads) {
          const uint64_t a = ((uint64_t)s_row[1][j] << 32) | s_row[0][j];
          const uint64_t g = ((uint64_t)s_row[3][j] << 32) | s_row[2][j];
          if (a | g) xor_row(A.acc + (size_t)comp * W, j, a, g);
          s_row[0][j] = s_row[1][j] = s_row[2][j] = s_row[3][j] = 0;
        }
      }
    }
    if (!meet(nullptr)) return;

    // ---- the largest component and those of several pieces: sampled from their rows ----
    const uint32_t nbig = ld_volatile(&c->nbig);
    for (uint32_t k = gwarp; k < nbig; k += gwarps) {
      const uint32_t r = __ldcg(&big[k]);
      GsBucket* row = A.acc + (size_t)r * W;
      uint32_t code;
      uint64_t idx;
      if constexpr (MANY) {
        const uint32_t i = A.vtenant[r];
        const GsBorTenant& M = A.tenants[i];
        const uint32_t b = M.bkt;
        sample_warp(row, row + b, b, M.csmix, &code, &idx);
        if (code == kFail) mark(A.tmod + (round & 1) * A.T1 + i);
        __syncwarp();
        for (uint32_t j = lane; j <= b; j += 32) row[j] = GsBucket{0, 0};
        if (lane == 0 && code == kGood)
          unite_many(A, G, edge_of(Graph{M.vbase, M.V, nullptr, nullptr, nullptr}, idx), A.tmod + (round & 1) * A.T1);
        __syncwarp();
      } else {
        sample_warp(row, row + bkt, bkt, T.csmix, &code, &idx);
        if (code == kFail) s_mod = 1;
        __syncwarp();
        for (uint32_t j = lane; j <= bkt; j += 32) row[j] = GsBucket{0, 0};
        unite(G, lane == 0 && code == kGood ? edge_of(G, idx) : ~0ull, &s_hooked);
      }
    }
  }

  if constexpr (MANY) return;
  if (gtid == 0) { ts[0] = 1; ts[2] = rounds; ts[3] = oos; }
  if (A.out) write_answer(A, G, gtid, gthreads, meet);
  // the first block's counters stay until every block has read them
  if constexpr (CLUSTER) cg::this_cluster().sync();
}

// One graph on a cluster, few graphs in the launch: a round in two phases.
//   accumulate  a warp takes consecutive vertices, walks to their roots (compressing the parents) and XORs their
//               column r and deterministic bucket into the root's accumulator row - in registers while the root
//               stays the same, then by atomics; the warps' last rows are combined per block
//   sample      an octet of lanes per vertex: a root samples its row, zeroes it and unions the sampled edge
// Atomics on rows in L2 are fast (200 per ns) as long as the rows fit there, so nothing is listed, sized or
// complemented: what a small graph's round costs is the chain of phases and their latency, not the bytes.
// Measured (us per query call, against the member lists of k_boruvka on the same cluster): V = 1000 117 -> 80,
// 4096 127 -> 109, 16384 341 -> 285; 8 graphs of up to 65536 vertices 620 -> 418.
template <int SLOTS>
__global__ void __launch_bounds__(threads_of(kWide), 1) k_boruvka_flat(const BorArgs A) {
  constexpr uint32_t kThreads = threads_of(kWide), kWarps = kThreads / 32;
  extern __shared__ __align__(16) GsBucket s_rows[];   // [kWarps][R] the warps' last rows
  __shared__ uint32_t s_flag[2];                       // the first block's: some sample failed or union succeeded
  __shared__ uint32_t s_root[kWarps], s_mod, s_hooked;
  const uint32_t lane = lane_id(), wib = threadIdx.x >> 5;
  cg::cluster_group cl = cg::this_cluster();
  const uint32_t block = cl.block_rank(), blocks = cl.num_blocks();
  volatile uint32_t* const flag = cl.map_shared_rank(s_flag, 0);
  const uint32_t t = A.qlist ? A.qlist[blockIdx.x / blocks] : 0u;
  const GsBorTenant T = A.tenants ? A.tenants[t] : A.t0;
  const uint32_t vlo = T.vbase, span = T.V, vend = T.vbase + T.V;
  const uint32_t bkt = T.bkt, W = A.W, R = A.R;
  const uint32_t gtid = block * kThreads + threadIdx.x, gthreads = blocks * kThreads;
  const uint32_t gwarp = gtid >> 5, gwarps = gthreads >> 5;
  const uint32_t limit = span + 64;
  const GsBucket* const sk = A.sk + T.sk_off;
  uint32_t* const ts = A.tstate + 4 * t;
  const Graph G{vlo, span, A.parent, A.edge, A.status};

  auto meet = [&](volatile uint32_t* f) -> bool {
    if (f) {
      __syncthreads();
      if (threadIdx.x == 0) {
        if (s_mod | s_hooked) *f = 1u;
        if (s_hooked && A.edge) atomicAdd(&A.status[4], s_hooked);
        s_mod = 0;
        s_hooked = 0;
      }
    }
    cg::this_cluster().sync();
    return true;
  };

  if (threadIdx.x == 0) { s_mod = 0; s_hooked = 0; s_flag[0] = 0; s_flag[1] = 0; }
  for (uint32_t v = vlo + gtid; v < vend; v += gthreads) A.parent[v] = v;
  if (A.out && gtid == 0) {   // as in k_boruvka
    A.status[16] = A.status[0];
    A.status[17] = 0;
    for (int i = 0; i < 16; i++) A.status[i] = 0;
  }
  meet(nullptr);
  uint32_t rounds = 0, oos = T.round0_col >= T.ns;
  if (!oos) round_zero(G, sk, T, A.rank, A.complement, gwarp, gwarps, &s_mod, &s_hooked);

  for (uint32_t round = 0; !oos || round;) {
    meet(flag + (round & 1));
    if (!flag[round & 1]) break;
    rounds = ++round;
    oos = rounds >= T.ns;

    // ---- accumulate ----
    {
      constexpr uint32_t kTake = 4;
      const uint32_t take = min(kTake, max(1u, (span + gwarps - 1) / gwarps));
      uint32_t cur = 0xffffffffu;
      uint64_t a[SLOTS] = {}, g[SLOTS] = {};
      for (uint32_t base = gwarp * take; base < span; base += gwarps * take) {
        const uint32_t n = min(take, span - base);
        uint32_t r = 0xffffffffu;
        if (lane < n) {
          const uint32_t v = vlo + base + lane;
          const bool closed = A.complement && __ldcg(&A.rank[v]) == kClosed;
          if (!closed) {
            r = cached_root(A.parent, v, limit, A.status);
            A.parent[v] = r;
          }
          A.size[v] = r == v;   // the roots that sample: a union of the sample phase may hook one before its turn
        }
        if (oos) continue;   // only the labels are still wanted
        const uint32_t open = __ballot_sync(0xffffffffu, r != 0xffffffffu);
        GsBucket b[kTake][SLOTS];
#pragma unroll
        for (uint32_t u = 0; u < kTake; u++) {
          const GsBucket* vb = sk + (size_t)(base + u) * T.nb;
#pragma unroll
          for (int k = 0; k < SLOTS; k++) {
            const uint32_t j = lane + 32u * k;
            b[u][k] = ((open >> u) & 1u) && j <= bkt ? ld_bucket_cg(vb + (j < bkt ? round * bkt + j : T.nb - 1)) : GsBucket{0, 0};
          }
        }
#pragma unroll
        for (uint32_t u = 0; u < kTake; u++) {
          if (!((open >> u) & 1u)) continue;
          const uint32_t root = __shfl_sync(0xffffffffu, r, u);
          if (root != cur) {
            if (cur != 0xffffffffu) {
#pragma unroll
              for (int k = 0; k < SLOTS; k++)
                if (lane + 32u * k <= bkt && (a[k] | g[k])) xor_row(A.acc + (size_t)cur * W, lane + 32u * k, a[k], g[k]);
            }
            cur = root;
#pragma unroll
            for (int k = 0; k < SLOTS; k++) a[k] = g[k] = 0;
          }
#pragma unroll
          for (int k = 0; k < SLOTS; k++) { a[k] ^= b[u][k].alpha; g[k] ^= b[u][k].gamma; }
        }
      }
      // the last rows: most warps hold the largest component's, and its atomics would queue
      if (lane == 0) s_root[wib] = cur;
#pragma unroll
      for (int k = 0; k < SLOTS; k++)
        if (lane + 32u * k <= bkt) s_rows[wib * R + lane + 32u * k] = GsBucket{a[k], g[k]};
      __syncthreads();
      const uint32_t same = __ballot_sync(0xffffffffu, s_root[lane] == cur);
      if (cur != 0xffffffffu && wib == (uint32_t)(__ffs(same) - 1)) {
        for (uint32_t m = same & (same - 1); m; m &= m - 1) {
          const GsBucket* other = s_rows + (__ffs(m) - 1) * R;
#pragma unroll
          for (int k = 0; k < SLOTS; k++)
            if (lane + 32u * k <= bkt) { a[k] ^= other[lane + 32u * k].alpha; g[k] ^= other[lane + 32u * k].gamma; }
        }
#pragma unroll
        for (int k = 0; k < SLOTS; k++)
          if (lane + 32u * k <= bkt && (a[k] | g[k])) xor_row(A.acc + (size_t)cur * W, lane + 32u * k, a[k], g[k]);
      }
    }
    meet(nullptr);
    if (threadIdx.x == 0 && block == 0) flag[(round + 1) & 1] = 0;   // everyone read it before this barrier
    if (oos) break;

    // ---- sample ----
    for (uint32_t base = gwarp * 4; base < span; base += gwarps * 4) {
      const uint32_t sub = lane & 7u, oct = lane >> 3;
      const uint32_t v = vlo + base + oct;
      const bool root = base + oct < span && __ldcg(&A.size[v]) != 0;
      if (!__any_sync(0xffffffffu, root)) continue;
      GsBucket* const row = A.acc + (size_t)(root ? v : vlo) * W;
      const GsBucket det = root ? ld_bucket_cg(row + bkt) : GsBucket{0, 0};
      bool decided = !root;
      uint32_t code = kFail;
      uint64_t idx = 0;
      for (uint32_t j0 = 0; j0 < bkt; j0 += 32) {   // four depths a lane on their way at once
        GsBucket b[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const uint32_t j = j0 + 8 * k + sub;
          b[k] = !decided && j < bkt ? ld_bucket_cg(row + j) : GsBucket{0, 0};
        }
        if (j0 == 0 && root) {
          if (det.alpha == 0 && det.gamma == 0) { code = kZero; decided = true; }
          else if (is_good(det, T.csmix)) { code = kGood; idx = det.alpha; decided = true; }
        }
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const uint32_t j = j0 + 8 * k + sub;
          const uint32_t m = __ballot_sync(0xffffffffu, !decided && j < bkt && is_good(b[k], T.csmix));
          const uint32_t mine = (m >> (8u * oct)) & 0xffu;
          const uint64_t x = __shfl_sync(0xffffffffu, b[k].alpha, mine ? 8u * oct + (uint32_t)(__ffs(mine) - 1) : lane);
          if (!decided && mine) { code = kGood; idx = x; decided = true; }
        }
        if (__all_sync(0xffffffffu, decided)) break;
      }
      __syncwarp();
      if (root) {
        for (uint32_t j = sub; j <= bkt; j += 8) row[j] = GsBucket{0, 0};
        if (sub == 0) {
          if (code == kFail) s_mod = 1;
          if (code == kGood) unite(G, edge_of(G, idx), &s_hooked);
        }
      }
      __syncwarp();
    }
  }

  if (gtid == 0) { ts[0] = 1; ts[2] = rounds; ts[3] = oos; }
  if (A.out) write_answer(A, G, gtid, gthreads, meet);
  cg::this_cluster().sync();   // the first block's flags stay until every block has read them
}

// the edges of the hooked vertices, as (min, max) pairs in any order
__global__ void __launch_bounds__(256) k_forest(const uint32_t* __restrict__ parent, const uint64_t* __restrict__ edge,
                                                uint32_t V, uint32_t* __restrict__ count, uint2* __restrict__ forest) {
  __shared__ uint32_t s_warp[8], s_at;
  const uint32_t lane = lane_id(), w = threadIdx.x >> 5;
  for (uint32_t base = blockIdx.x * 256; base < V; base += gridDim.x * 256) {
    const uint32_t v = base + threadIdx.x;
    const bool hooked = v < V && parent[v] != v;
    const uint32_t m = __ballot_sync(0xffffffffu, hooked);
    if (lane == 0) s_warp[w] = __popc(m);
    __syncthreads();
    uint32_t before = 0, all = 0;
    for (uint32_t i = 0; i < 8; i++) {
      if (i < w) before += s_warp[i];
      all += s_warp[i];
    }
    if (threadIdx.x == 0) s_at = all ? atomicAdd(count, all) : 0u;
    __syncthreads();
    if (hooked) {
      const uint64_t e = edge[v];
      const uint32_t a = (uint32_t)(e >> 32), b = (uint32_t)e;
      forest[s_at + before + __popc(m & ((1u << lane) - 1u))] = make_uint2(min(a, b), max(a, b));
    }
    __syncthreads();
  }
}

template <int SCOPE, int SLOTS, bool MANY>
constexpr auto kernel_of() {
  if constexpr (SCOPE == kWide) return k_boruvka_flat<SLOTS>;
  else return k_boruvka<SCOPE, SLOTS, MANY>;
}

size_t dynamic_bytes(int scope, uint32_t R, uint32_t T1) {
  return (size_t)(threads_of(scope, T1 != 0) / 32) * (scope == kWide ? 1 : kRing) * R * sizeof(GsBucket) + 5 * (size_t)T1;
}

// Launches of more than 48 KB of dynamic shared memory, and clusters of more than 8 blocks, are opted into
// per device and kernel; that it was done, and the cluster size that fits, are remembered per host thread.
template <int SCOPE, int SLOTS, bool MANY = false>
gs_status launch_boruvka(const BorArgs& A, const GsBorLaunch& L, cudaStream_t s) {
  struct Opted { size_t smem = 0; uint32_t blocks = 0; int sms = 0; };
  static thread_local Opted opted[64];
  constexpr auto kernel = kernel_of<SCOPE, SLOTS, MANY>();
  int dev = 0;
  GS_CUDA_TRY(cudaGetDevice(&dev));
  Opted& o = opted[dev & 63];
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  cfg.blockDim = dim3(threads_of(SCOPE, MANY));
  cfg.dynamicSmemBytes = dynamic_bytes(SCOPE, L.R, MANY ? L.T1 : 0);
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (o.smem < cfg.dynamicSmemBytes) {
    GS_TRY(gs_allow_shared_memory(kernel, dev));
    GS_CUDA_TRY(cudaDeviceGetAttribute(&o.sms, cudaDevAttrMultiProcessorCount, dev));
    o.blocks = 8;
    if (SCOPE != kGrid) {
      // 16 blocks where the device can place them
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = 16;
      attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
      cfg.gridDim = dim3(16);
      int n = 0;
      if (cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
          cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) == cudaSuccess && n > 0)
        o.blocks = 16;
      cudaGetLastError();
    }
    o.smem = cfg.dynamicSmemBytes;
  }
  if (SCOPE != kGrid) {
    const uint32_t blocks = std::min(L.scope.blocks, o.blocks);
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = blocks;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(blocks * L.count);
  } else {
    // every block co-resident: cooperative through a launch attribute, so that the launch can also be
    // captured into a CUDA graph
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.gridDim = dim3(o.sms);
    GS_CUDA_TRY(cudaMemsetAsync(A.ctr, 0, kGsBorCounterWords * sizeof(uint32_t), s));
    if (MANY) GS_CUDA_TRY(cudaMemsetAsync(L.many, 0, gs_boruvka_many_bytes(L.T1), s));
  }
  GS_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, A));
  return GS_OK;
}

template <int SLOTS>
gs_status launch_scope(const BorArgs& A, const GsBorLaunch& L, cudaStream_t s) {
  if (L.T1) return launch_boruvka<kGrid, SLOTS, true>(A, L, s);
  if (!L.scope.blocks) return launch_boruvka<kGrid, SLOTS>(A, L, s);
  return L.scope.wide ? launch_boruvka<kWide, SLOTS>(A, L, s) : launch_boruvka<kNarrow, SLOTS>(A, L, s);
}

}  // namespace

static_assert((kGsBorCounterWords - 1) * sizeof(uint32_t) >= 2 * sizeof(BorCounters), "two counter sets and the barrier");

gs_status gs_boruvka_launch(const GsBorLaunch& L, cudaStream_t s) {
  BorArgs A;
  A.sk = L.sk;
  A.tenants = L.tenants;
  A.t0 = L.t0;
  A.qlist = L.qlist;
  A.tenant = L.tenant;
  A.T1 = L.T1;
  A.vtenant = L.vtenant;
  A.vlo = L.vlo;
  A.vhi = L.vhi;
  A.tlargest = static_cast<unsigned long long*>(L.many);
  A.tmod = reinterpret_cast<uint32_t*>(A.tlargest + 2 * (size_t)L.T1);
  A.W = L.W;
  A.R = L.R;
  A.parent = L.parent;
  A.size = L.size;
  const size_t n = L.vertices;
  A.rank = L.members;
  A.off = L.members + n;
  A.list = L.members + 2 * n;
  A.big = L.members + 3 * n;
  A.tasks = L.tasks;
  A.acc = L.acc;
  A.edge = L.edge;
  A.status = L.status;
  A.out = L.out;
  A.labels = L.labels;
  A.tstate = L.tstate;
  A.ctr = reinterpret_cast<BorCounters*>(L.counters);
  A.barrier = L.counters + kGsBorCounterWords - 1;
  A.wait_ns = L.wait_ns;
  A.complement = L.complement;
  if (L.R <= 32) return launch_scope<1>(A, L, s);
  if (L.R <= 64) return launch_scope<2>(A, L, s);
  gs_set_error("more than 63 buckets per column are not supported");
  return GS_ERR_BAD_ARG;
}

gs_status gs_alloc_boruvka(gs_graph* g, uint64_t vertices, uint32_t width, bool forest) {
  // one allocation, cut up by falling alignment
  const uint64_t row = sizeof(uint4) + (forest ? 2 * sizeof(uint64_t) : 0) + 6 * sizeof(uint32_t);
  GS_CUDA_TRY(cudaMalloc(&g->d_bor, vertices * row + kGsBorCounterWords * sizeof(uint32_t)));
  uint8_t* p = static_cast<uint8_t*>(g->d_bor);
  const auto take = [&](uint64_t bytes) { uint8_t* at = p; p += bytes; return at; };
  g->d_tasks = reinterpret_cast<uint4*>(take(vertices * sizeof(uint4)));
  g->d_bor_ctr = reinterpret_cast<uint32_t*>(take(kGsBorCounterWords * sizeof(uint32_t)));
  if (forest) {
    g->d_edge = reinterpret_cast<uint64_t*>(take(vertices * sizeof(uint64_t)));
    g->d_forest = reinterpret_cast<uint32_t*>(take(vertices * 2 * sizeof(uint32_t)));
  }
  g->d_parent = reinterpret_cast<uint32_t*>(take(vertices * sizeof(uint32_t)));
  g->d_size = reinterpret_cast<uint32_t*>(take(vertices * sizeof(uint32_t)));
  g->d_members = reinterpret_cast<uint32_t*>(take(4 * vertices * sizeof(uint32_t)));
  GS_CUDA_TRY(cudaMalloc(&g->d_acc, vertices * width * sizeof(GsBucket)));
  return GS_OK;
}

gs_status gs_gather_forest(gs_graph* g, cudaStream_t s) {
  if (!g->last_forest_edges) return GS_OK;
  GS_CUDA_TRY(cudaMemsetAsync(g->d_bor_ctr, 0, sizeof(uint32_t), s));
  const int grid = std::min<int>((int)((g->V + 255) / 256), g->num_sms * 8);
  GsProfScope ps(g, GS_PROF_QUERY, s, 1);
  k_forest<<<grid, 256, 0, s>>>(g->d_parent, g->d_edge, g->V, g->d_bor_ctr, reinterpret_cast<uint2*>(g->d_forest));
  GS_CUDA_TRY(cudaGetLastError());
  return GS_OK;
}

gs_status gs_boruvka_enqueue(gs_graph* g, uint32_t level, uint32_t round0_col, cudaStream_t s, uint32_t* h_out,
                             uint32_t* h_labels) {
  const uint32_t V = g->V, nb = g->geom.num_buckets, bkt = g->geom.bkt_per_col;
  g->labels_valid = false;
  g->last_forest_edges = 0;

  GsBorLaunch L;
  L.sk = g->d_sk + (size_t)level * V * nb;
  L.t0.sk_off = 0;
  L.t0.vbase = 0;
  L.t0.V = V;
  L.t0.nb = nb;
  L.t0.bkt = bkt;
  L.t0.ns = g->geom.num_samples;
  L.t0.round0_col = round0_col;
  L.t0.csmix = gs_seed_mix(g->seed);
  // a handle with a wait limit of its own keeps the scope whose waits have one
  if (g->wait_ns == kGsDefaultWaitNs) L.scope = gs_boruvka_scope(V);
  L.vertices = V;
  L.W = L.R = bkt + 1;
  L.parent = g->d_parent;
  L.size = g->d_size;
  L.acc = g->d_acc;
  L.members = g->d_members;
  L.tasks = g->d_tasks;
  L.edge = g->d_edge;
  L.status = g->d_status;
  L.tstate = g->d_status + 8;
  L.counters = g->d_bor_ctr;
  L.wait_ns = g->wait_ns;
  L.complement = g->sketches_symmetric ? 1u : 0u;

  // the kernel expects all-zero accumulator rows and leaves them so when it runs to the end
  if (g->acc_dirty) GS_CUDA_TRY(cudaMemsetAsync(g->d_acc, 0, (size_t)V * (bkt + 1) * sizeof(GsBucket), s));
  g->acc_dirty = true;
  // the kernel writes the words when it ends; one that gave up waiting does not
  h_out[0] = GS_DEV_ERR_TIMEOUT;
  L.out = h_out;
  L.labels = h_labels;
  GsProfScope ps(g, GS_PROF_QUERY, s, 1);
  return gs_boruvka_launch(L, s);
}

// One graph: a cluster has 16 SMs and the hardware's barrier, the grid all of them and a barrier of about
// 1.5 us; the two meet above 8192 vertices (us per query call, cluster / grid: V = 1024 88 / 178, 4096
// 109 / 165, 8192 184 / 220, 16384 285 / 207).
GsBorScope gs_boruvka_scope(uint32_t V) { return V <= 8192 ? GsBorScope{16, true} : GsBorScope{}; }

// Several graphs of at most kGsBorClusterV vertices, clusters side by side: the scope of the least estimated
// time.  A graph of V vertices takes about a + b V / blocks us on its cluster (wide: a = 120, b = 0.19;
// narrow: a = 170, b = 0.32, measured on R-MAT and Erdos-Renyi tenants of 256 to 65536 vertices), 148 wide or
// 296 narrow blocks run at once, and the launch ends with its largest graph.  Measured (ms per query, chosen /
// best of all): 256 graphs of 256 to 16384 vertices 1.2 / 1.2, 40 of 1024 to 20000 0.89 / 0.89, 10 of 1024 to
// 8192 0.21 / 0.21.
GsBorScope gs_boruvka_scope(const uint32_t* V, uint32_t graphs) {
  double sum = 0, most = 0;
  for (uint32_t i = 0; i < graphs; i++) {
    sum += V[i];
    most = std::max(most, (double)V[i]);
  }
  GsBorScope best;
  double least = 1e300;
  for (int wide = 0; wide < 2; wide++) {
    const double a = wide ? 120 : 170, b = wide ? 0.19 : 0.32;
    for (uint32_t blocks = 2; blocks <= 16; blocks *= 2) {
      const double at_once = std::floor((wide ? 148.0 : 296.0) / blocks);
      const double t = std::max(a + b * most / blocks, (a * graphs + b * sum / blocks) / at_once);
      if (t < least) {
        least = t;
        best = GsBorScope{blocks, wide != 0};
      }
    }
  }
  return best;
}

// A cluster holds its SMs for about 45 + 0.11 V us however small its graph is, and 148 run at once; one grid launch
// over all graphs takes about 230 us and 1 us for 1000 ids of its range.  Measured (us, clusters / grid): 4096
// graphs of 64 vertices 1574 / 522, of 256 2187 / 1235; 2048 of 64 797 / 324; 1024 of 64 423 / 285, of 256 599 /
// 518, of 1000 1061 / 1256; 512 of 64 238 / 243; 256 of 64 147 / 232.  (The launch before, one grid for all: 834,
// 1771, 568, 534, 793, 1872, 462, 392.)
bool gs_boruvka_shares_grid(uint32_t graphs, uint64_t vertices, uint64_t span) {
  return (45.0 * graphs + 0.11 * (double)vertices) / 148 > 230 + 0.001 * (double)span;
}

gs_status gs_boruvka_finish(gs_graph* g, uint32_t level, uint32_t* st) {
  if (st[0] & GS_DEV_ERR_TIMEOUT) {
    // the words are still on the device, among them the error bits of calls queued behind the query, which stay
    constexpr uint32_t kOwn = GS_DEV_ERR_TIMEOUT | GS_DEV_ERR_DSU_LIMIT;
    GS_CUDA_TRY(cudaMemcpyAsync(st, g->d_status, 18 * sizeof(uint32_t), cudaMemcpyDeviceToHost, g->stream));
    GS_CUDA_TRY(cudaStreamSynchronize(g->stream));
    const uint32_t later = st[0] & ~kOwn;
    GS_CUDA_TRY(cudaMemcpyAsync(g->d_status, &later, sizeof(uint32_t), cudaMemcpyHostToDevice, g->stream));
    GS_CUDA_TRY(cudaStreamSynchronize(g->stream));
    st[0] |= GS_DEV_ERR_TIMEOUT;
    st[16] &= ~kOwn;   // a block gave up before the first one had moved the earlier calls' bits there
  }
  // records skipped by the ingest calls before the query are reported first
  if (st[16]) {
    if (st[16] & GS_DEV_ERR_VERTEX_RANGE) {
      gs_set_error("an edge record named a vertex id >= num_vertices; those records were skipped");
      return GS_ERR_BAD_ARG;
    }
    gs_set_error("device consistency check failed (bits " + std::to_string(st[16]) + ")");
    return GS_ERR_INTERNAL;
  }
  if (st[0] & GS_DEV_ERR_TIMEOUT) {
    gs_set_error("a grid barrier of the Boruvka kernel gave up waiting");
    return GS_ERR_TIMEOUT;
  }
  if (st[0] & GS_DEV_ERR_DSU_LIMIT) {
    gs_set_error("DSU walk exceeded its bound");
    return GS_ERR_INTERNAL;
  }
  g->acc_dirty = false;
  if (st[8 + 3]) {
    gs_set_error("sketch ran out of samples after " + std::to_string(st[8 + 2]) + " Boruvka rounds");
    return GS_ERR_SKETCH_FAIL;
  }
  g->last_rounds = st[8 + 2];
  g->last_forest_edges = st[4] < g->V ? st[4] : g->V - 1;
  g->last_components = st[17];
  g->labels_valid = true;
  g->labels_level = level;
  return GS_OK;
}

gs_status gs_boruvka(gs_graph* g, uint32_t level, uint32_t round0_col, cudaStream_t s, uint32_t* h_labels) {
  GS_TRY(gs_boruvka_enqueue(g, level, round0_col, s, g->h_status, h_labels));
  GS_CUDA_TRY(cudaStreamSynchronize(s));
  return gs_boruvka_finish(g, level, g->h_status);
}
