// Luby-style maximal independent set with goodness priority (indset.cpp) and
// the small shared kernels of the passes: marking, class inheritance,
// expansion, global renumbering.
//
// The star graph is never materialised for the independent set: an edge's
// neighbours are the other edges of the tets around it (up(1,3) then
// down(3,1)), a vertex's neighbours the far ends of its edges (up(0,1)).
// That is exactly the neighbour set of the reference's star(1,3) /
// star(0,1) (star.cpp:135-293); the selection rule depends only on that set.
#include <algorithm>
#include <atomic>
#include <vector>

#include "passes.hpp"

namespace osh {

PassStats& last_pass_stats()
{
  static thread_local PassStats s;
  return s;
}

// a set's control words (mailbox slots 44-50; their layout is given at
// k_indset), which come back with the slots before them
constexpr u32 COOP_CTL_SLOT = 44, COOP_CTL_WORDS = 7;
static_assert(COOP_CTL_SLOT + COOP_CTL_WORDS == INDSET_FETCH_SLOTS, "mailbox slots");

// neighbourhood walks: mode 0 = vertices via edges, mode 1 = edges via
// elements (3D tets or 2D triangles)
struct Nbrs {
  u32 mode;
  u32 const* offs;   // up(ent, via)
  u32 const* uses;
  u32 const* down;   // down(via, ent) or verts_of_edges
  u32 per;           // entities per via-entity
};

// indset_at_vert (indset.cpp:55-84) for entity i: out of the set if a
// neighbour is in it; in the set if no undecided neighbour beats it (higher
// goodness, or equal goodness and a lower global id); undecided otherwise.
// Goodness and id order the candidates strictly, so the set is the same
// whatever the order in which they are decided, as long as each is decided
// on decided neighbours: the lexicographically first independent set, which
// the reference's rounds find. So there are no rounds here, and no barrier:
// a warp keeps the candidates it could not decide, each with its best
// undecided neighbour (its blocker), and looks at their states until they
// are decided; an entity that joins the set puts its undecided neighbours
// out of it. The best undecided candidate can always be decided. (Rounds
// over lists of the undecided, a grid barrier after each, spent 40 to 60 us
// a set on a small mesh, most of it in the barriers and in walking every
// row again: 632 us over a 48^3 adapt and 776 over a 39^3 coarsening, now 290 and 200.)
//
// Words (keys, one per entity): 0 no candidate; an undecided candidate's
// order_key, by which goodness compares as an integer; or decided, below
// KEY_MIN (1 + depth: out of the set) or from KEY_IN on (+ depth: in it).
// One gather tells all of a neighbour, and nothing is written before the
// walks: the kernels that choose the candidates write their keys. The depth
// bounds the reference's round for the entity from above: one more than the
// largest of the better neighbours it joined after (of all its neighbours
// below DEPTH_EXACT, where the bound is far from the cap), or than that of a
// neighbour in the set. Where it passes 100 for some entity, the
// reference's cap of 100 rounds (indset.cpp:33) may have been met, and the
// last block to finish runs rounds as the reference does, alone.
//
// A group of G lanes walks a candidate's upward entries l, l + G, ..., and
// every lane issues the loads of all neighbours of an entry together. (One
// thread per long row issues loads whose lanes are a row apart and fills
// the load/store queue; one neighbour at a time waits for three dependent
// loads each.) Every block must be resident, as warps wait on one another:
// one thread-block cluster or a cooperative launch. The waits are bounded: a
// warp that meets no decided state in ASYNC_SPIN_LIMIT sweeps of its
// candidates sets control word 6 and leaves, and the others leave when they
// see it.
constexpr u32 ASYNC_SPIN_LIMIT = 1u << 22;
constexpr u32 DEPTH_MAX = 127, DEPTH_EXACT = 48;
typedef unsigned long long Key;

__device__ inline bool key_undecided(Key k) { return k - KEY_MIN < KEY_IN - KEY_MIN; }
__device__ inline bool key_in(Key k) { return k >= KEY_IN; }
// (of a decided word)
__device__ inline u32 key_depth(Key k) { return key_in(k) ? (u32)(k - KEY_IN) : (u32)k - 1u; }
__device__ inline Key key_decided(u32 depth, bool in)
{
  return (in ? KEY_IN : (Key)1) + min(depth, DEPTH_MAX);
}

// A word that another warp may be writing, or waiting for: warps wait on one
// another through these words, so they are read and written at device scope
// (a word says all there is to know of its entity: nothing else is ordered
// with it).
__device__ __forceinline__ Key key_read(Key const* p)
{
  Key k;
  asm volatile("ld.relaxed.gpu.u64 %0, [%1];" : "=l"(k) : "l"(p));
  return k;
}
__device__ __forceinline__ void key_write(Key* p, Key k)
{
  asm volatile("st.relaxed.gpu.u64 [%0], %1;" ::"l"(p), "l"(k));
}

// neighbours of an upward entry: 1 (a vertex's edge), 3 or 6 (an edge's
// triangle or tet, the edge itself among them); NB: those a lane takes at once
template <u32 PER>
struct NbrBatch {
  static constexpr u32 USES = PER == 1 ? 2 : 1, NB = PER * USES;
};

// up to NB neighbours of entity i from its entries j, j + G, ... (INV: none;
// swaps in a tangled mesh can leave an edge whose ends are one vertex, which
// is not its own neighbour)
template <int G, u32 PER>
__device__ inline void load_neighbors(Nbrs const& g, u32 i, u32 j, u32 re, u32* o)
{
  if (PER == 1) {
    u32 u[2];
#pragma unroll
    for (u32 k = 0; k < 2; ++k) u[k] = j + k * G < re ? g.uses[j + k * G] : INV;
#pragma unroll
    for (u32 k = 0; k < 2; ++k) o[k] = u[k] != INV ? g.down[u[k] ^ 1u] : INV;
#pragma unroll
    for (u32 k = 0; k < 2; ++k)
      if (o[k] == i) o[k] = INV;
  } else {
    u32 const use = g.uses[j];
    u32 const* ds = g.down + (use - use % PER);
#pragma unroll
    for (u32 k = 0; k < PER; ++k) o[k] = ds[k];
#pragma unroll
    for (u32 k = 0; k < PER; ++k)
      if (o[k] == i) o[k] = INV;
  }
}

struct Walk {
  bool in;       // a neighbour is in the set
  bool worse;    // some undecided neighbour is worse
  u32 depth;     // of a neighbour in the set, else the largest of those out of it
  u32 blocker;   // the best undecided better neighbour, or INV
};

// The first walk of an entity (FRESH false) reads the words through L1, which
// neighbouring entities' walks share: a word that has been decided since
// reads as undecided, which only makes the entity wait. Later ones read past
// L1, or a stale word would block it for good.
template <int G, u32 PER, bool FRESH>
__device__ inline Walk walk_neighbors(Nbrs const& g, u32 i, Key mykey, u32 lg, u32 gmask,
    u32 gbase, Key const* keys, double const* __restrict__ good, u64 const* __restrict__ glob)
{
  constexpr u32 NB = NbrBatch<PER>::NB, STEP = G * NbrBatch<PER>::USES;
  u32 const rb = g.offs[i], re = g.offs[i + 1];
  u32 in_depth = 0, out_depth = 0, blocker = INV;
  Key bk = 0;
  bool in = false, worse = false;
  auto id_of = [&](u32 o) { return glob ? glob[o] : (u64)o; };
  // (numbers that a caller gave twice: by index, so that no two wait for each other)
  auto later = [&](u32 a, u32 b) {
    u64 const x = id_of(a), y = id_of(b);
    return x > y || (x == y && a > b);
  };
  for (u32 j = rb + lg; j < re; j += STEP) {
    u32 o[NB];
    Key ko[NB];
    load_neighbors<G, PER>(g, i, j, re, o);
#pragma unroll
    for (u32 k = 0; k < NB; ++k)
      ko[k] = o[k] == INV ? 0ull : FRESH ? key_read(&keys[o[k]]) : __ldca(&keys[o[k]]);
#pragma unroll
    for (u32 k = 0; k < NB; ++k) {
      if (!ko[k]) continue;
      if (key_undecided(ko[k])) {
        if (ko[k] < mykey || (ko[k] == mykey && later(o[k], i)))
          worse = true;
        else if (blocker == INV || ko[k] > bk || (ko[k] == bk && later(blocker, o[k]))) {
          blocker = o[k];
          bk = ko[k];
        }
        continue;
      }
      u32 const d = key_depth(ko[k]);
      if (key_in(ko[k])) {
        in = true;
        in_depth = d;
      } else if (d > out_depth) {
        bool counts = d < DEPTH_EXACT;
        if (!counts) {
          double const myg = good[i], og = good[o[k]];
          counts = (myg == og && id_of(o[k]) < id_of(i)) || myg < og;
        }
        if (counts) out_depth = d;
      }
    }
  }
  Walk w;
  u32 const ins = (__ballot_sync(gmask, in) & gmask) >> gbase;
  w.in = ins != 0;
  w.worse = (__ballot_sync(gmask, worse) & gmask) != 0;
#pragma unroll
  for (int o = G / 2; o; o >>= 1) {
    out_depth = max(out_depth, __shfl_xor_sync(gmask, out_depth, o));
    u32 const b2 = __shfl_xor_sync(gmask, blocker, o);
    Key const k2 = __shfl_xor_sync(gmask, bk, o);
    if (b2 != INV && b2 != blocker &&
        (blocker == INV || k2 > bk || (k2 == bk && later(blocker, b2)))) {
      blocker = b2;
      bk = k2;
    }
  }
  u32 const d = __shfl_sync(gmask, in_depth, gbase + (ins ? __ffs(ins) - 1 : 0));
  w.depth = w.in ? d : out_depth;
  w.blocker = blocker;
  return w;
}

// The reference's rounds, by one block, over lists of the undecided, in
// place (a state read during a round is the round before's or the final
// one: states only change from undecided to decided). was: the words of
// the kernel above (0: no candidate). wl: two lists of n.
template <int G>
__device__ void indset_rounds(u32 n, Nbrs const& g, Key const* was, u32* st, u32* wl, double const* __restrict__ good, u64 const* __restrict__ glob, u32* ctl)
{
  u32* const wl0 = wl;
  u32* const wl1 = wl + n;
  u32 const lg = threadIdx.x % G, lane = threadIdx.x & 31;
  u32 const gbase = lane & ~(u32)(G - 1);
  u32 const gmask = (G == 32 ? 0xffffffffu : ((1u << G) - 1u)) << gbase;
  for (u64 b = 0; b < n; b += blockDim.x) {
    u64 const i = b + threadIdx.x;
    bool const c = i < n && __ldcg(&was[i]) != 0;
    if (i < n) __stcg(&st[i], c ? (u32)UNKNOWN : (u32)NOT_IN_SET);
    if (c) __stcg(&wl1[atomicAdd(&ctl[2], 1u)], (u32)i);
  }
  __threadfence();
  __syncthreads();
  for (u32 r = 0; r < MAX_INDSET_ROUNDS; ++r) {
    // round 0 walks the candidates, round r > 0 the list round r - 1 left
    u32 const len = *(volatile u32*)&ctl[2 + r % 3];
    u32 const* list = (r % 2 == 1) ? wl0 : wl1;
    u32* next = (r % 2 == 0) ? wl0 : wl1;
    u32* next_len = &ctl[2 + (r + 1) % 3];
    if (threadIdx.x == 0) ctl[2 + (r + 2) % 3] = 0;
    for (u64 t = threadIdx.x; t < (u64)len * G; t += blockDim.x) {
      u32 const i = __ldcg(&list[t / G]);
      u32 const rb = g.offs[i], re = g.offs[i + 1];
      double const myg = good[i];
      u64 const myid = glob ? glob[i] : (u64)i;
      bool in_set = false, beaten = false;
      auto visit = [&](u32 o) {
        u32 so = __ldcg(&st[o]);
        if (so == IN_SET) in_set = true;
        if (so == NOT_IN_SET) return;
        double og = good[o];
        u64 oid = glob ? glob[o] : (u64)o;
        if ((myg == og && oid < myid) || myg < og) beaten = true;
      };
      for (u32 j = rb + lg; j < re; j += G) {
        if (g.mode == 0) {
          visit(g.down[g.uses[j] ^ 1u]);
        } else {
          u32 const* ds = g.down + (g.uses[j] - g.uses[j] % g.per);
          for (u32 k = 0; k < g.per; ++k)
            if (ds[k] != i) visit(ds[k]);
        }
      }
      bool const any_in = (__ballot_sync(gmask, in_set) & gmask) != 0;
      bool const lost = (__ballot_sync(gmask, beaten) & gmask) != 0;
      if (lg) continue;
      if (any_in)
        __stcg(&st[i], (u32)NOT_IN_SET);
      else if (!lost)
        __stcg(&st[i], (u32)IN_SET);
      else
        __stcg(&next[atomicAdd(next_len, 1u)], i);
    }
    __threadfence();
    __syncthreads();
    if (*(volatile u32*)next_len == 0) {
      // settled: the list lengths go back to zero for the next set
      if (threadIdx.x == 0) {
        ctl[5] = r + 1;
        ctl[2] = ctl[3] = ctl[4] = 0;
      }
      return;
    }
  }
  // not settled: the caller reports it, but its next kernels are queued
  // already and count on 0 and 1
  for (u64 i = threadIdx.x; i < n; i += blockDim.x)
    if (__ldcg(&st[i]) == UNKNOWN) __stcg(&st[i], (u32)NOT_IN_SET);
  if (threadIdx.x == 0) ctl[5] = MAX_INDSET_ROUNDS;
}

// Control words, zero on entry but [5]: [0] blocks done, [1] the largest
// depth, [2..4] list lengths of the rounds, [5] rounds (or the largest
// depth), [6] a wait gave up. The listed entities (those whose key is not 0
// are the candidates) are dealt to the lane groups in turn: entry t to group
// t % all groups, so that candidates that lie together are spread evenly.
// (Tiles of the entities dealt to warps left most warps idle where the
// candidates lay together, and every pass read every key.) queue: an entry
// {entity, blocker} per listed entity, 2 n words at least: the last block's
// rounds use it as their lists.
constexpr u32 ITEMS_AHEAD = 4;

// every listed candidate of this warp decided; returns their largest depth
// (item: 32 words of shared memory of the warp's own)
template <int G, u32 PER>
__device__ inline u32 decide_listed(Nbrs const& g, u32 const* __restrict__ list, u32 nitems,
    Key* keys, uint2* queue, double const* __restrict__ good, u64 const* __restrict__ glob,
    u32* __restrict__ out, u32* ctl, u32* item)
{
  constexpr u32 FULL = 0xffffffffu, NG = 32 / G;  // groups of a warp
  u32 const lane = threadIdx.x & 31, lg = lane % G, gi = lane / G;
  u32 const gbase = lane & ~(u32)(G - 1);
  u32 const gmask = (G == 32 ? FULL : ((1u << G) - 1u)) << gbase;
  u32 const below = (1u << lane) - 1u;
  u32 const nwarps = (gridDim.x * blockDim.x) >> 5;
  u32 const w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  u32 len = 0, deepest = 0;
  // entry q of this warp's queue (the places of its list entries, in order)
  auto slot = [&](u32 q) { return queue + ((size_t)(q / NG) * nwarps + w) * NG + q % NG; };
  // an entity found decided, or decided, by this thread
  auto settled = [&](u32 i, Key k) {
    out[i] = key_in(k) ? 1u : 0u;
    deepest = max(deepest, key_depth(k));
  };
  // entity i walked by a group (key: its key as read by the group): decided,
  // or its blocker returned
  auto walk = [&](u32 i, Key mine, bool fresh) -> u32 {
    if (!key_undecided(mine)) {  // put out of the set meanwhile
      if (lg == 0) settled(i, mine);
      return INV;
    }
    Walk const r =
        fresh ? walk_neighbors<G, PER, true>(g, i, mine, lg, gmask, gbase, keys, good, glob)
              : walk_neighbors<G, PER, false>(g, i, mine, lg, gmask, gbase, keys, good, glob);
    if (!r.in && r.blocker != INV) return r.blocker;
    if (lg == 0) {
      Key const k = key_decided(r.depth + 1, !r.in);
      key_write(&keys[i], k);
      settled(i, k);
    }
    if (!r.in && r.worse) {
      // its neighbours are out of the set
      Key const no = key_decided(r.depth + 2, false);
      bool const exact = r.depth + 2 >= DEPTH_EXACT;
      constexpr u32 NB = NbrBatch<PER>::NB, STEP = G * NbrBatch<PER>::USES;
      for (u32 j = g.offs[i] + lg, re = g.offs[i + 1]; j < re; j += STEP) {
        u32 o[NB];
        load_neighbors<G, PER>(g, i, j, re, o);
        Key ko[NB];
#pragma unroll
        for (u32 k = 0; k < NB; ++k) ko[k] = o[k] != INV ? key_read(&keys[o[k]]) : 0ull;
#pragma unroll
        for (u32 k = 0; k < NB; ++k) {
          if (exact && ko[k])  // (the smaller depth stays)
            atomicMin(&keys[o[k]], no);
          else if (key_undecided(ko[k]))
            key_write(&keys[o[k]], no);
        }
      }
    }
    return INV;
  };
  // entities with blockers (one per group, lane 0 of it) onto the queue
  auto append = [&](u32 i, u32 blocker) {
    bool const keep = lg == 0 && blocker != INV;
    u32 const m = __ballot_sync(FULL, keep);
    if (keep) *slot(len + __popc(m & below)) = make_uint2(i, blocker);
    len += __popc(m);
  };
  // every candidate once (ITEMS_AHEAD entries' words loaded together)
  for (u32 q0 = w * NG; q0 < nitems; q0 += nwarps * NG * ITEMS_AHEAD) {
    u32 it[ITEMS_AHEAD];
    Key key[ITEMS_AHEAD];
#pragma unroll
    for (u32 k = 0; k < ITEMS_AHEAD; ++k) {
      size_t const t = (size_t)q0 + (size_t)k * nwarps * NG + gi;
      it[k] = t < nitems ? list[t] : INV;
    }
    // (one lane's reading for the group: a word may change between two)
#pragma unroll
    for (u32 k = 0; k < ITEMS_AHEAD; ++k)
      key[k] = lg == 0 && it[k] != INV ? key_read(&keys[it[k]]) : 0ull;
#pragma unroll
    for (u32 k = 0; k < ITEMS_AHEAD; ++k) {
      Key const mine = __shfl_sync(FULL, key[k], gbase);
      if (!__any_sync(FULL, mine != 0)) continue;
      append(it[k], mine ? walk(it[k], mine, false) : INV);
    }
  }
  // then the undecided, until none is left
  u32 spins = 0;
  while (len) {
    u32 const todo = len;
    bool moved = false;
    __syncwarp();  // the entries written by other lanes
    len = 0;       // entries kept are written at or before the ones being read
    for (u32 q = 0; q < todo; q += 32) {
      uint2 e = make_uint2(0u, INV);
      Key mine = 0, ko = 0;
      if (q + lane < todo) {
        e = *slot(q + lane);
        mine = key_read(&keys[e.x]);
        ko = key_read(&keys[e.y]);
      }
      bool const have = e.y != INV;
      bool const put_out = have && !key_undecided(mine);
      // a decided blocker: in the set, it puts its entity out of it (its own
      // writes may be on their way); out, the entity is walked again
      bool const ready = have && !put_out && !key_undecided(ko);
      bool const again = ready && !key_in(ko);
      __syncwarp();
      if (put_out || (ready && !again)) {
        if (!put_out) {
          mine = key_decided(key_depth(ko) + 1, false);
          key_write(&keys[e.x], mine);
        }
        settled(e.x, mine);
      }
      bool const wait = have && !put_out && !ready;
      u32 const kept = __ballot_sync(FULL, wait);
      if (wait) *slot(len + __popc(kept & below)) = e;
      len += __popc(kept);
      moved = moved || __any_sync(FULL, have && !wait);
      u32 const m = __ballot_sync(FULL, again);
      if (!m) continue;
      if (again) item[__popc(m & below)] = e.x;
      __syncwarp();
      u32 const cnt = __popc(m);
      for (u32 b = 0; b < cnt; b += NG) {
        u32 i = 0, blocker = INV;
        if (b + gi < cnt) {
          i = item[b + gi];
          Key const k = __shfl_sync(gmask, lg == 0 ? key_read(&keys[i]) : 0ull, gbase);
          blocker = walk(i, k, true);
        }
        append(i, blocker);
      }
      __syncwarp();
    }
    if (moved) {
      spins = 0;
      continue;
    }
    if (++spins > ASYNC_SPIN_LIMIT) {
      if (lane == 0) atomicOr(&ctl[6], 1u);
      break;
    }
    if ((spins & 255u) == 0 && *(volatile u32*)&ctl[6]) break;
    __nanosleep(spins < 16 ? 20 : 200);
  }
  return __reduce_max_sync(FULL, deepest);
}

// G: lanes per entity of a long list, where the walks' instructions and
// loads in flight bound the set; a list with a group of WIDE lanes to every
// entity is bound by the chain of one walk, which more lanes shorten (edges'
// rows: 2 lanes 67 us and 8 lanes 222 us on the first list of a 48^3 adapt,
// 17 and 9 us on a late one).
constexpr int WIDE = 8;

template <int G, u32 PER>
__global__ void __launch_bounds__(1024, 1) k_indset(u32 n, Nbrs g,
    u32 const* __restrict__ list, u32 const* nlist, Key* keys, uint2* queue,
    double const* __restrict__ good, u64 const* __restrict__ glob, u32* __restrict__ out,
    u32* ctl)
{
  pdl_wait();
  __shared__ u32 s_item[32][32];
  __shared__ u32 s_depth;
  __shared__ u32 s_last;
  if (threadIdx.x == 0) s_depth = 0;
  __syncthreads();
  u32 const nitems = *(u32 const volatile*)nlist;
  u32* const item = s_item[threadIdx.x >> 5];
  u32 deepest;
  if (G < WIDE && (u64)nitems * WIDE <= (u64)gridDim.x * blockDim.x)
    deepest = decide_listed<(G < WIDE ? WIDE : G), PER>(g, list, nitems, keys, queue, good,
        glob, out, ctl, item);
  else
    deepest = decide_listed<G, PER>(g, list, nitems, keys, queue, good, glob, out, ctl, item);
  if ((threadIdx.x & 31) == 0 && deepest) atomicMax(&s_depth, deepest);
  __syncthreads();
  if (threadIdx.x == 0) {
    if (s_depth) atomicMax(&ctl[1], s_depth);
    __threadfence();
    s_last = atomicAdd(&ctl[0], 1u) + 1u == gridDim.x ? 1u : 0u;
  }
  __syncthreads();
  if (!s_last) return;
  u32 const depth = atomicMax(&ctl[1], 0u);
  __syncthreads();
  if (threadIdx.x == 0) {
    ctl[0] = 0;
    ctl[1] = 0;
    ctl[5] = depth;
  }
  if (depth <= MAX_INDSET_ROUNDS || *(volatile u32*)&ctl[6]) return;
  __threadfence();
  __syncthreads();
  indset_rounds<G>(n, g, keys, out, reinterpret_cast<u32*>(queue), good, glob, ctl);
}

namespace {
// blocks of BLOCK threads a cooperative launch uses on this device: the
// tuning table's indset_blocks per SM, at most as many as are resident
template <int G, u32 PER>
u32 coop_blocks()
{
  static std::atomic<u32> per_sm_of[64];
  static std::atomic<u32> sms_of[64];
  int dev = 0;
  CK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return 0;
  if (!sms_of[dev].load()) {
    int per_sm = 0, sms = 0;
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_indset<G, PER>, BLOCK, 0));
    CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    per_sm_of[dev].store((u32)per_sm);
    sms_of[dev].store((u32)sms);
  }
  u32 per_sm = per_sm_of[dev].load(), want = tuned(TK_INDSET_BLOCKS);
  if (want && want < per_sm) per_sm = want;
  return per_sm * sms_of[dev].load();
}

// A set of at most CLUSTER_ENTS entities goes to one cluster of eight blocks
// of 1024 threads: an ordinary launch, which need not wait for the whole
// device to drain as a cooperative one does.
constexpr u32 CLUSTER_BLOCKS = 8, CLUSTER_ENTS = 8192;

template <int G, u32 PER>
void launch_indset_as(u32 n, Nbrs const& g, IndsetIn const& in, double const* good,
    u64 const* glob, u32* ctl, cudaStream_t s)
{
  bool const one_cluster = n <= CLUSTER_ENTS;
  u32 const threads = one_cluster ? 1024 : BLOCK;
  u32 const most = one_cluster ? CLUSTER_BLOCKS : coop_blocks<G, PER>();
  if (!most) throw Failure(E_CUDA, "independent set: no resident blocks");
  // (the list's length is read on the device; n bounds it)
  u32 const wide = std::max(G, WIDE);
  u32 const blocks =
      one_cluster ? CLUSTER_BLOCKS : std::min<u32>(ceil_div((u64)n * wide, threads), most);
  // a place per listed entity of each group (at either width)
  u64 const all = (u64)blocks * threads;
  auto places = [&](u32 lanes) { return (size_t)ceil_div(n, all / lanes) * (all / lanes); };
  uint2* queue = dalloc<uint2>(std::max(places(G), places(wide)), s);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(threads);
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (one_cluster) {
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CLUSTER_BLOCKS;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
  } else {
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
  }
  CK(cudaLaunchKernelEx(&cfg, k_indset<G, PER>, n, g, in.list, in.nlist, in.keys, queue, good, glob,
      in.out, ctl));
  CK_LAUNCH();
  dev_free(queue, s);
}

template <int G>
void launch_indset(u32 n, Nbrs const& g, IndsetIn const& in, double const* good,
    u64 const* glob, u32* ctl, cudaStream_t s)
{
  if (g.mode == 0) launch_indset_as<G, 1>(n, g, in, good, glob, ctl, s);
  else if (g.per == 3) launch_indset_as<G, 3>(n, g, in, good, glob, ctl, s);
  else launch_indset_as<G, 6>(n, g, in, good, glob, ctl, s);
}
}  // namespace

// number of upward uses (edges of vertices / elements of edges), for the mean
// length of a row
static u32 read_cached_uses(Mesh& m, u32 ent_dim)
{
  return ent_dim == 0 ? 2u * m.counts[1] : deg(m.dim, 1) * m.counts[m.dim];
}

__global__ void __launch_bounds__(BLOCK) k_indset_in(u32 n, u32 const* __restrict__ filter,
    double const* __restrict__ good, Key* __restrict__ keys, u32* __restrict__ list, u32* nlist,
    u32* __restrict__ out)
{
  pdl_wait();
  u32 i = blockIdx.x * blockDim.x + threadIdx.x;
  bool const c = i < n && filter[i];
  if (i < n) {
    keys[i] = c ? indset_key(good[i]) : 0ull;
    out[i] = 0;
  }
  block_append<1>(c ? 1u : 0u, i, list, nlist);
}

void IndsetIn::alloc(u32 n, cudaStream_t s)
{
  keys = dalloc<Key>(n ? n : 1, s);
  own_list = dalloc<u32>(n ? n : 1, s);
  list = own_list;
  out = dalloc<u32>(n ? n : 1, s);
}

void IndsetIn::free(cudaStream_t s)
{
  dev_free(keys, s);
  dev_free(own_list, s);
  dev_free(out, s);
  keys = nullptr;
  list = own_list = out = nullptr;
}

IndsetIn indset_in(Mesh& m, u32 n, u32 const* filter, double const* good)
{
  IndsetIn in;
  in.alloc(n, m.s);
  u32* nlist = m.mb->dev + COOP_CTL_SLOT + COOP_CTL_WORDS;
  in.nlist = nlist;
  CK(cudaMemsetAsync(nlist, 0, sizeof(u32), m.s));
  if (n) {
    CK(launch_kernel(k_indset_in, dim3(grid_for(n)), dim3(BLOCK), 0, m.s, n, filter, good,
        in.keys, in.own_list, nlist, in.out));
    CK_LAUNCH();
  }
  return in;
}

u32* find_indset(Mesh& m, u32 ent_dim, IndsetIn& in, double const* good, bool check)
{
  u32 n = m.count(ent_dim);
  Nbrs g{};
  if (ent_dim == 0) {
    UpAdj const& u = m.ask_up(0, 1, false);
    g.mode = 0;
    g.offs = u.offs;
    g.uses = u.uses;
    g.down = m.ask_down(1, 0);
    g.per = 2;
  } else if (ent_dim == 1 && m.dim >= 2) {
    UpAdj const& u = m.ask_up(1, m.dim, false);
    g.mode = 1;
    g.offs = u.offs;
    g.uses = u.uses;
    g.down = m.ask_down(m.dim, 1);
    g.per = deg(m.dim, 1);
  } else {
    throw Failure(E_ARG, "independent sets are built on vertices or edges");
  }
  // global numbers held as the identity flag are the local index, which is
  // what the kernel compares when it has no array
  u64 const* glob = m.parallel ? m.globals[ent_dim] : nullptr;
  // One launch decides every candidate; its control words (mailbox slots
  // COOP_CTL_SLOT..) come back with slots 1-3, which a caller that left
  // flags there reads after this call without a read-back of its own. With
  // no entity, only the rounds count is zeroed.
  u32* ctl = m.mb->dev + COOP_CTL_SLOT;
  if (n) {
    double nuse = (double)read_cached_uses(m, ent_dim);
    double avg_row = nuse / n;
    u32 lanes = avg_row >= 8.0 ? tuned(TK_INDSET_VERT_GROUP)
              : avg_row >= 3.0 ? tuned(TK_INDSET_EDGE_GROUP) : 1u;
    if (lanes == 16) launch_indset<16>(n, g, in, good, glob, ctl, m.s);
    else if (lanes == 8) launch_indset<8>(n, g, in, good, glob, ctl, m.s);
    else if (lanes == 4) launch_indset<4>(n, g, in, good, glob, ctl, m.s);
    else if (lanes == 2) launch_indset<2>(n, g, in, good, glob, ctl, m.s);
    else launch_indset<1>(n, g, in, good, glob, ctl, m.s);
  } else {
    CK(cudaMemsetAsync(ctl + 5, 0, sizeof(u32), m.s));
  }
  if (check) {
    m.mb->fetch(m.s, INDSET_FETCH_SLOTS);
    indset_check(m);
  }
  u32* a = in.out;
  in.out = nullptr;
  in.free(m.s);
  return a;
}

void indset_check(Mesh& m)
{
  u32 const* hc = m.mb->host + COOP_CTL_SLOT;
  // a set that failed leaves its control words standing: zeroed here for
  // the next set
  auto reset = [&] {
    CK(cudaMemsetAsync(m.mb->dev + COOP_CTL_SLOT, 0, COOP_CTL_WORDS * sizeof(u32), m.s));
  };
  if (hc[6]) {
    reset();
    throw Failure(E_TIMEOUT, "independent set: a wait for a neighbour gave up");
  }
  u32 rounds = hc[5];
  last_pass_stats().indset_rounds = rounds;
  // settled, unless the last block ran rounds and the last of them left some
  // undecided (the list lengths are zero otherwise)
  bool done = rounds == 0 || hc[2 + rounds % 3] == 0;
  if (!done) {
    reset();
    throw Failure(E_NOCONVERGE, "independent set did not settle in 100 rounds");
  }
}

// ---------------------------------------------------------------------------
// expansion and inheritance

template <class T>
__global__ void k_expand_scaled(T const* __restrict__ in, u32 const* __restrict__ offs,
    u32 k, u32 n, u32 width, T* __restrict__ out)
{
  pdl_wait();
  u32 i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  u32 f = offs[i] * k, e = offs[i + 1] * k;
  for (u32 j = f; j < e; ++j)
    for (u32 c = 0; c < width; ++c) out[(size_t)j * width + c] = in[(size_t)i * width + c];
}

void expand_scaled(void const* in, u32 const* offs, u32 k, u32 n, u32 width,
    u32 esz, void* out, cudaStream_t s)
{
  if (!n || !width || !k) return;
  PROBE(P_EXPAND, s, 4.0 * (n + 1) + 2.0 * (double)n * width * esz * k);
  u32 const gb = tuned(TK_GATHER_BLOCK);
  if (esz == 1)
    CK(launch_kernel(k_expand_scaled<unsigned char>, dim3(grid_for(n, gb)), dim3(gb), 0, s,
        (unsigned char const*)in, offs, k, n, width, (unsigned char*)out));
  else if (esz == 4)
    CK(launch_kernel(k_expand_scaled<u32>, dim3(grid_for(n, gb)), dim3(gb), 0, s,
        (u32 const*)in, offs, k, n, width, (u32*)out));
  else
    CK(launch_kernel(k_expand_scaled<unsigned long long>, dim3(grid_for(n, gb)), dim3(gb), 0, s,
        (unsigned long long const*)in, offs, k, n, width, (unsigned long long*)out));
  CK_LAUNCH();
}

// Several row expansions in one launch (the same copy as k_expand_scaled):
// blockIdx.y picks the job, the x blocks stride over its rows. The jobs that
// do not go by words (lists of a pass's few producing entities, wide rows)
// share one y where a y each would not fit the GPU at once: most of those
// blocks had nothing to do (12 -> 8 us a launch in the small passes of a 39^3
// coarsening, 26 -> 15 in a 24^3 warp step's). Where they fit, taking the
// jobs in turn costs more than it saves (7 against 5 us on a 6^3 adapt).
constexpr u32 EXPAND_MAX = 16;  // (a coarsening or refinement pass of a 3D mesh has 11 to 14)
struct ExpandJobs {
  ExpandJob j[EXPAND_MAX];
  u32 nrest;    // the first jobs do not go by words:
  u32 together;  // blockIdx.y 0 takes this many of them in turn
};

template <class T>
__device__ inline void copy_rows(void const* in, void* out, u32 i, u32 f, u32 e, u32 width)
{
  T const* src = static_cast<T const*>(in) + (size_t)i * width;
  for (u32 j = f; j < e; ++j) {
    T* dst = static_cast<T*>(out) + (size_t)j * width;
    for (u32 c = 0; c < width; ++c) dst[c] = src[c];
  }
}

// Jobs over every row with k = 1 -- the survivors' copy, one output row or
// none per row, in order: a stream compaction -- of rows of W 32-bit words
// go by warps: a warp takes EXPAND_CHUNKS runs of 32 consecutive rows,
// loads their offsets (one per lane) and their words coalesced, all before
// any store, and stores each word at its row's place, the row's offsets
// coming by shuffle; the kept rows' words stay consecutive, so the stores
// are coalesced too. (A thread per row read and wrote rows of 2-4 words a
// row apart per lane, with one or two loads in flight: a third of DRAM
// peak.)
constexpr u32 EXPAND_CHUNKS = 2;

template <u32 W>
__device__ inline void expand_same_rows(ExpandJob const& jb, u32 warp, u32 nwarps)
{
  u32 const lane = threadIdx.x & 31;
  u32 const* __restrict__ in = static_cast<u32 const*>(jb.in);
  u32 const* __restrict__ in2 = static_cast<u32 const*>(jb.in2);
  u32* __restrict__ out = static_cast<u32*>(jb.out);
  u32* __restrict__ out2 = static_cast<u32*>(jb.out2);
  bool const two = in2 != nullptr;
  for (u32 base = warp * 32 * EXPAND_CHUNKS; base < jb.n; base += nwarps * 32 * EXPAND_CHUNKS) {
    u32 o0[EXPAND_CHUNKS], o1[EXPAND_CHUNKS], a[EXPAND_CHUNKS][W], b[EXPAND_CHUNKS][W];
#pragma unroll
    for (u32 ch = 0; ch < EXPAND_CHUNKS; ++ch) {
      u32 const cb = base + ch * 32;
      u32 const nrows = cb < jb.n ? min(32u, jb.n - cb) : 0u, nw = nrows * W;
      o0[ch] = o1[ch] = 0;
      if (lane < nrows) {
        o0[ch] = jb.offs[cb + lane];
        o1[ch] = jb.offs[cb + lane + 1];
      }
#pragma unroll
      for (u32 it = 0; it < W; ++it) {
        u32 const q = it * 32 + lane;
        if (q < nw) {
          a[ch][it] = in[(size_t)cb * W + q];
          if (two) b[ch][it] = in2[(size_t)cb * W + q];
        }
      }
    }
#pragma unroll
    for (u32 ch = 0; ch < EXPAND_CHUNKS; ++ch) {
      u32 const cb = base + ch * 32;
      u32 const nw = (cb < jb.n ? min(32u, jb.n - cb) : 0u) * W;
      // 32 rows that all survive (most runs of a pass that changes little)
      // are one run of the output: no row to find for a word
      if (__all_sync(0xffffffffu, o1[ch] == o0[ch] + 1)) {
        size_t const at = (size_t)__shfl_sync(0xffffffffu, o0[ch], 0) * W + lane;
#pragma unroll
        for (u32 it = 0; it < W; ++it) {
          out[at + it * 32] = a[ch][it];
          if (two) out2[at + it * 32] = b[ch][it];
        }
        continue;
      }
#pragma unroll
      for (u32 it = 0; it < W; ++it) {
        u32 const q = it * 32 + lane;
        u32 const row = q / W, c = q - row * W;
        u32 const f = __shfl_sync(0xffffffffu, o0[ch], row & 31);
        u32 const e = __shfl_sync(0xffffffffu, o1[ch], row & 31);
        if (q < nw)
          for (u32 j = f; j < e; ++j) {  // (a row of the survivors' copy has one)
            out[(size_t)j * W + c] = a[ch][it];
            if (two) out2[(size_t)j * W + c] = b[ch][it];
          }
      }
    }
  }
}

// Other jobs (a list of rows, k > 1, wider rows, 1-byte elements): a
// thread per row. (At least three blocks of 512 per SM: at 56 registers
// only four blocks of 256 fit, too few warps to keep the loads in flight.)
__global__ void __launch_bounds__(512, 3) k_expand_many(const __grid_constant__ ExpandJobs jobs)
{
  pdl_wait();
  u32 const t0 = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
  u32 const q0 = blockIdx.y ? blockIdx.y + jobs.together - 1 : 0;
  if (q0 >= jobs.nrest) {
    ExpandJob const jb = jobs.j[q0];
    u32 const warp = t0 / 32, nwarps = stride / 32;
    u32 const words = jb.width * (jb.esz / 4);
    if (words == 1)
      expand_same_rows<1>(jb, warp, nwarps);
    else if (words == 2)
      expand_same_rows<2>(jb, warp, nwarps);
    else if (words == 3)
      expand_same_rows<3>(jb, warp, nwarps);
    else
      expand_same_rows<4>(jb, warp, nwarps);
    return;
  }
  for (u32 q = q0, end = blockIdx.y ? q0 + 1 : jobs.together; q < end; ++q) {
    ExpandJob const jb = jobs.j[q];
    for (u32 t = t0; t < jb.n; t += stride) {
      u32 const i = jb.list ? jb.list[t] : t;
      u32 f = jb.offs[i] * jb.k, e = jb.offs[i + 1] * jb.k;
      if (jb.esz == 4) {
        copy_rows<u32>(jb.in, jb.out, i, f, e, jb.width);
        if (jb.in2) copy_rows<u32>(jb.in2, jb.out2, i, f, e, jb.width);
      } else if (jb.esz == 8) {
        copy_rows<unsigned long long>(jb.in, jb.out, i, f, e, jb.width);
        if (jb.in2) copy_rows<unsigned long long>(jb.in2, jb.out2, i, f, e, jb.width);
      } else {
        copy_rows<unsigned char>(jb.in, jb.out, i, f, e, jb.width);
        if (jb.in2) copy_rows<unsigned char>(jb.in2, jb.out2, i, f, e, jb.width);
      }
    }
  }
}

static bool expand_by_words(ExpandJob const& jb)
{
  u32 const words = jb.esz == 4 ? jb.width : jb.esz == 8 ? 2 * jb.width : 0;
  return words && words <= 4 && !jb.list && jb.k == 1;
}

void expand_many(std::vector<ExpandJob> const& jobs, cudaStream_t s)
{
  std::vector<ExpandJob> live;
  for (u32 words = 0; words < 2; ++words)
    for (ExpandJob const& jb : jobs)
      if (jb.n && jb.width && jb.k && expand_by_words(jb) == (words != 0)) live.push_back(jb);
  u32 const gb = tuned(TK_GATHER_BLOCK);
  for (size_t at = 0; at < live.size(); at += EXPAND_MAX) {
    ExpandJobs pack{};
    u32 cnt = (u32)std::min<size_t>(EXPAND_MAX, live.size() - at), blocks = 0;
    double bytes = 0;
    for (u32 q = 0; q < cnt; ++q) {
      ExpandJob const& jb = pack.j[q] = live[at + q];
      bool const words = expand_by_words(jb);
      if (!words) ++pack.nrest;
      blocks = std::max(blocks, grid_for(jb.n, gb * (words ? EXPAND_CHUNKS : 1u)));
      bytes += 4.0 * (jb.n + 1) + (jb.in2 ? 4.0 : 2.0) *
          (double)jb.n * jb.width * jb.esz * jb.k;
    }
    PROBE(P_EXPAND, s, bytes);
    // a grid-stride loop over at most 16 blocks of 256 threads per SM
    // (measured: a block per 256 rows was twice as slow on the 48^3 adapt)
    blocks = std::min<u32>(blocks, 148u * 16u * 256u / gb);
    bool const fits = blocks * cnt <= resident_blocks(k_expand_many, gb);
    pack.together = fits ? 1u : std::max(pack.nrest, 1u);
    dim3 grid(blocks, cnt - pack.together + 1u);
    CK(launch_kernel(k_expand_many, grid, dim3(gb), 0, s, pack));
    CK_LAUNCH();
  }
}

// class_dim / class_id of the products: every domain of both labels in one
// launch
void inherit_class(Mesh& m, Mesh& out, u32 prod, Doms const& d,
    std::vector<ExpandJob> const* also, std::vector<ExpandJob>* defer)
{
  if (!m.find_tag(0, "class_dim")) {
    if (also && defer)
      defer->insert(defer->end(), also->begin(), also->end());
    else if (also)
      expand_many(*also, m.s);
    return;
  }
  char const* names[2] = {"class_dim", "class_id"};
  u32 nnames = m.find_tag(0, "class_id") ? 2 : 1;
  std::vector<ExpandJob> jobs;
  if (also) jobs = *also;
  u32* data[2] = {nullptr, nullptr};
  u32 nc[2] = {1, 1};
  Tag* t[2] = {nullptr, nullptr};
  for (u32 q = 0; q < nnames; ++q) {
    t[q] = m.find_tag(prod, names[q]);
    if (!t[q]) throw Failure(E_ARG, std::string("missing tag ") + names[q]);
    nc[q] = t[q]->ncomps;
    data[q] = dalloc<u32>((size_t)d.ngo[4] * nc[q], m.s);
  }
  // both labels of a domain dimension in one job when they have the same
  // width (the domain offsets are read once); a domain with a list of its
  // producing entities walks only those
  bool const paired = nnames == 2 && nc[0] == nc[1];
  for (u32 k = 0; k < 4; ++k) {
    if (!d.ndoms[k] || !d.offs[k] || !d.ngen[k]) continue;
    for (u32 q = 0; q < nnames; ++q) {
      Tag* tk = (k == 0) ? t[q] : m.find_tag(k, names[q]);
      if (!tk) continue;
      ExpandJob jb;
      jb.in = tk->data;
      jb.offs = d.offs[k];
      jb.out = data[q] + (size_t)d.ngo[k] * nc[q];
      jb.k = d.scale[k];
      jb.n = d.ndoms[k];
      if (d.list[k]) {
        jb.list = d.list[k];
        jb.n = d.nlist[k];
      }
      jb.width = nc[q];
      jb.esz = 4;
      if (paired && q == 0) {
        Tag* tk2 = (k == 0) ? t[1] : m.find_tag(k, names[1]);
        if (tk2) {
          jb.in2 = tk2->data;
          jb.out2 = data[1] + (size_t)d.ngo[k] * nc[1];
          jobs.push_back(jb);
          break;  // the second label goes with the first
        }
      }
      jobs.push_back(jb);
    }
  }
  if (defer)
    defer->insert(defer->end(), jobs.begin(), jobs.end());
  else
    expand_many(jobs, m.s);
  for (u32 q = 0; q < nnames; ++q) out.add_tag(prod, T_U32, names[q], nc[q], X_NOT, data[q]);
}

void inherit_globals(Mesh& out, u32 d)
{
  out.set_iota_globals(d);
}

__global__ void k_interp_coords(u32 ne, u32 vpe, u32 const* __restrict__ voe,
    double const* __restrict__ x, double* __restrict__ out)
{
  pdl_wait();
  u32 i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= ne) return;
  // average_element_field (element_field.hpp:9-25)
  double o0 = 0, o1 = 0, o2 = 0;
  for (u32 j = 0; j < vpe; ++j) {
    u32 v = voe[(size_t)i * vpe + j];
    o0 += x[v * 3 + 0];
    o1 += x[v * 3 + 1];
    o2 += x[v * 3 + 2];
  }
  out[i * 3 + 0] = o0 / vpe;
  out[i * 3 + 1] = o1 / vpe;
  out[i * 3 + 2] = o2 / vpe;
}

void interp_coords_to_elems(Mesh& m)
{
  u32 ne = m.count(m.dim), vpe = deg(m.dim, 0);
  double* out = dalloc<double>((size_t)ne * 3, m.s);
  if (ne) {
    CK(launch_kernel(k_interp_coords, dim3(grid_for(ne)), dim3(BLOCK), 0, m.s, ne, vpe, m.ask_down(m.dim, 0),
        m.coords(), out));
    CK_LAUNCH();
  }
  m.add_tag(m.dim, T_F64, "coordinates", 3, X_NOT, out);
}

// ---------------------------------------------------------------------------
// marking (mark.cpp)

__global__ void k_mark_down(u32 n, u32 const* __restrict__ offs, u32 const* __restrict__ uses,
    UseDiv div, u32 const* __restrict__ marked, u32* __restrict__ out)
{
  pdl_wait();
  u32 i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  u32 r = 0;
  for (u32 j = offs[i]; j < offs[i + 1]; ++j)
    if (marked[use_high(div, uses[j])]) {
      r = 1;
      break;
    }
  out[i] = r;
}

u32* mark_down(Mesh& m, u32 high, u32 low, u32 const* marked)
{
  u32 n = m.count(low);
  UpAdj const& u = m.ask_up(low, high, false);
  u32* out = dalloc<u32>(n, m.s);
  if (n) {
    CK(launch_kernel(k_mark_down, dim3(grid_for(n)), dim3(BLOCK), 0, m.s, n, u.offs, u.uses, use_div(deg(high, low)), marked, out));
    CK_LAUNCH();
  }
  return out;
}

__global__ void k_mark_up(u32 n, u32 lph, u32 const* __restrict__ loh,
    u32 const* __restrict__ marked, u32* __restrict__ out)
{
  pdl_wait();
  u32 i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  u32 r = 0;
  for (u32 j = 0; j < lph; ++j)
    if (marked[loh[(size_t)i * lph + j]]) {
      r = 1;
      break;
    }
  out[i] = r;
}

u32* mark_up(Mesh& m, u32 low, u32 high, u32 const* marked)
{
  u32 n = m.count(high);
  u32* out = dalloc<u32>(n, m.s);
  if (n) {
    CK(launch_kernel(k_mark_up, dim3(grid_for(n)), dim3(BLOCK), 0, m.s, n, deg(high, low), m.ask_down(high, low),
        marked, out));
    CK_LAUNCH();
  }
  return out;
}

__global__ void k_mark_slivers(u32 n, double const* __restrict__ q, double gq,
    u32 const* __restrict__ voe, u32 vpe, SegView sv, u32* __restrict__ out)
{
  pdl_wait();
  u32 i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = (q[i] < gq && (!sv.active || seg_acts(sv, voe[(size_t)i * vpe]))) ? 1u : 0u;
}

// warp-aggregated per-segment count of flagged entities
__global__ void k_seg_tally(u32 n, u32 const* __restrict__ flags, u32 const* __restrict__ voe,
    u32 vpe, u32 const* __restrict__ seg, u32* __restrict__ out)
{
  pdl_wait();
  u32 i = blockIdx.x * blockDim.x + threadIdx.x;
  bool on = i < n && flags[i] != 0;
  u32 mask = __ballot_sync(0xffffffffu, on);
  if (!on) return;
  u32 sg = seg[voe ? voe[(size_t)i * vpe] : i];
  u32 peers = __match_any_sync(mask, sg);
  if ((threadIdx.x & 31) == (u32)(__ffs(peers) - 1)) atomicAdd(&out[sg], (u32)__popc(peers));
}

void seg_tally(Mesh& m, u32 ent_dim, u32 const* flags)
{
  if (!m.seg || !m.ctl || !m.ctl->selected) return;
  u32 n = m.count(ent_dim);
  if (!n) return;
  u32 const* voe = ent_dim ? m.ask_down(ent_dim, 0) : nullptr;
  CK(launch_kernel(k_seg_tally, dim3(grid_for(n)), dim3(BLOCK), 0, m.s, n, flags, voe, deg(ent_dim, 0), m.seg,
      m.ctl->selected));
  CK_LAUNCH();
}

__global__ void k_dual_layer(u32 n, u32 degr, u32 const* __restrict__ dual,
    u32 const* __restrict__ in, u32* __restrict__ out)
{
  pdl_wait();
  u32 i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  u32 r = in[i];
  for (u32 j = 0; j < degr; ++j) {
    u32 e = dual[(size_t)i * degr + j];
    if (e != INV && in[e]) r = 1;
  }
  out[i] = r;
}

// mesh_mark_slivers + mesh_mark_dual_layers (mark.cpp:101-147,218-243)
u32* mark_slivers(Mesh& m, double gq, u32 nlayers)
{
  u32 n = m.count(m.dim);
  double const* q = m.qualities();
  u32* a = dalloc<u32>(n, m.s);
  if (n) {
    SegView sv = m.segview();
    CK(launch_kernel(k_mark_slivers, dim3(grid_for(n)), dim3(BLOCK), 0, m.s, n, q, gq,
        sv.active ? m.ask_down(m.dim, 0) : nullptr, deg(m.dim, 0), sv, a));
    CK_LAUNCH();
  }
  if (!nlayers) return a;
  u32 const* du = m.ask_dual();
  u32* b = dalloc<u32>(n, m.s);
  u32 degr = deg(m.dim, m.dim - 1);
  for (u32 l = 0; l < nlayers; ++l) {
    if (n) {
      CK(launch_kernel(k_dual_layer, dim3(grid_for(n)), dim3(BLOCK), 0, m.s, n, degr, du, a, b));
      CK_LAUNCH();
    }
    std::swap(a, b);
  }
  dev_free(b, m.s);
  return a;
}

}  // namespace osh
