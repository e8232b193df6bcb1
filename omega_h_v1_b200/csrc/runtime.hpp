// Host-callable device primitives used by every pass: scans, reductions,
// fills, compaction by offsets. All work is issued on the caller's stream.
#pragma once

#include "common.cuh"

namespace osh {

// Launch shapes chosen by the tuner (omega_h_v1_b200/tune.py, which times
// each candidate with CUDA events on a mid-size adapt and writes the table).
// Every key has a default and a set of allowed values; the table is read
// once, from the file named by OSH_B200_TUNING or else tuning.txt beside
// the library ("name value" lines, # comments). Any allowed value gives the
// same meshes: only the launch shapes change.
enum TuneKey : u32 {
  TK_CARRY_GROUP = 0,    // lanes per long carried upward row: 4, 8, 16
  TK_VERT_GROUP,         // lanes per vertex row, coarsening vertex kernels: 4, 8, 16
  TK_INDSET_VERT_GROUP,  // lanes per vertex, independent set, long lists: 4, 8, 16
  TK_INDSET_EDGE_GROUP,  // lanes per edge (3D), the same: 1, 2, 4, 8
  TK_QUALITY_BLOCK,      // threads per block, quality kernels: 64, 128, 256, 512
  TK_GATHER_BLOCK,       // threads per block, carry / search / copy kernels: 128, 256, 512
  TK_SCAN_ITEMS,         // items per thread of a scan tile: 8, 16
  TK_SCAN_THREADS,       // threads per scan tile: 256, 512
  TK_INDSET_BLOCKS,      // blocks per SM of the independent set's cooperative
                         // launch, whose warps wait on one another (0: as many as
                         // fit): 0, 1, 2, 4
  TK_SMALL_MESH_ELEMS,   // concurrent many-mesh adapt: meshes estimated below this
                         // many elements are adapted together in batch unions
                         // (0: none): 0, 25000, 50000 (default), 100000, 200000
  TK_NKEYS
};
u32 tuned(TuneKey k);
char const* tune_name(u32 k);
// 0, or E_ARG for an unknown name or a value the key does not allow
int tune_set(char const* name, u32 value);
int tune_get(char const* name, u32* value);
// reads a table file; 0, E_IO (unreadable) or E_ARG (a bad line: nothing set)
int tune_load(char const* path);

// thread-local error state behind osh_b200_last_error()
void set_error(int code, char const* msg);
int last_error();
char const* last_error_message();
void clear_error();

// Exclusive scan with the total appended: out has n+1 entries and
// out[n] = sum(in). Single-pass decoupled look-back (uints_exscan, ints.cpp).
// total_to (optional, device): receives out[n] as well (a mailbox slot the
// host reads back with other flags, instead of a copy of its own)
// newid (optional, device, n entries; for 0/1 inputs): out[i] where in[i]
// is 1, INV where 0 -- the new id of each entity the flags mark as kept
void exscan_u32(u32 const* in, u32* out, u32 n, cudaStream_t s, u32* total_to = nullptr,
    u32* newid = nullptr);
u32* exscan_new(u32 const* in, u32 n, cudaStream_t s, u32* total_to = nullptr,
    u32* newid = nullptr);

// Independent scans in one launch (their look-back chains overlap): job j
// scans `in` (mode 0) or the survivors of an offsets array in[0..n]
// (mode 1: in[i + 1] == in[i], uints_negate_offsets) into out[0..n], with
// total_to and newid as above. Jobs are launched MAX_SCAN_JOBS at a time.
constexpr u32 MAX_SCAN_JOBS = 8;
struct ScanJob {
  u32 const* in;
  u32* out;
  u32* total_to;
  u32* newid;
  u32 n;
  u32 mode;
  // (optional, 0/1 items: mode 0 with 0/1 items, or mode 2) list[out[i]] = i
  // where item i is 1: the marked items in order
  u32* list = nullptr;
  // (optional, 0/1 items) the scan of the complement,
  // comp[i] = i - out[i] for i <= n (the unmarked items before i), and
  // comp_newid[i] = comp[i] where item i is 0 and INV where it is 1 -- each
  // survivor's new id when the items mark what a pass removes
  u32* comp = nullptr;
  u32* comp_newid = nullptr;
  // mode 2: item i is 1 where in[i] == stamp, else 0 (marks stamped with a
  // generation, see stream_marks)
  u32 stamp = 0;
};
struct ScanJobs {
  u32 njobs;
  u32 tile0[MAX_SCAN_JOBS + 1];
  ScanJob j[MAX_SCAN_JOBS];
};
void exscan_jobs(ScanJob const* jobs, u32 njobs, cudaStream_t s);

// Scratch kept per (device, stream, host thread, key) between calls, zeroed
// when made or grown. stream_zero_scratch: the caller leaves it zero again
// after each use (keys KEPT_ROWS0 and KEPT_ROWS1: the search rows' counts,
// KEPT_USES: the upward rows', which the rows' fill counts back down to
// zero). stream_marks: entries stamped with a generation of the scratch,
// returned in *gen (never 0) and new on every call, so no entry of an earlier use passes for a mark of this one
// (KEPT_MARKS: the products' vertices of a pass's searches; KEPT_FUSED + d:
// the collapses' fused entities of dimension d; KEPT_SPLIT + d: a
// refinement's split domain entities of dimension d).
enum : u32 {
  KEPT_ROWS0 = 1,
  KEPT_ROWS1 = 2,
  KEPT_MARKS = 3,
  KEPT_FUSED = 4,
  KEPT_SPLIT = 8,
  KEPT_USES = 12
};
u32* stream_zero_scratch(u32 key, size_t words, cudaStream_t s);

// blocks of `block` threads (and `smem` bytes of dynamic shared memory) of a
// kernel resident at once on the current device: the occupancy
// calculator's blocks per SM times the SMs, computed once per kernel, shape
// and device (for grids that stride over their work in one wave)
u32 resident_blocks_of(void const* kernel, u32 block, size_t smem);
template <class K>
inline u32 resident_blocks(K kernel, u32 block, size_t smem = 0)
{
  return resident_blocks_of(reinterpret_cast<void const*>(kernel), block, smem);
}
// frees (in the order of s) the scan and kept scratch of stream s on the
// current device; called before a stream is destroyed, so that scratch does
// not outlive its stream (no kernel may use it afterwards)
void release_stream_scratch(cudaStream_t s);

// a non-blocking stream of the current device, and one back (its scratch
// released; its work may still run: the next user's comes after it)
cudaStream_t take_stream();
void give_back_stream(cudaStream_t s);
// a mesh on a stream that is not its own, from its making (or its move there)
// to its end: the blocks kept for a caller's stream go with its last mesh
void begin_stream_use(cudaStream_t s);
void end_stream_use(cudaStream_t s);
u32* stream_marks(u32 key, size_t words, cudaStream_t s, u32* gen);

// The same scan with caller-provided scratch of at least
// exscan_scratch_words(n) 32-bit words (zeroed here); allocates nothing.
size_t exscan_scratch_words(u32 n);
void exscan_u32_scratch(u32 const* in, u32* out, u32 n, u32* scratch, cudaStream_t s);

// throws E_TIMEOUT if a bounded device-side wait gave up since the last check
void check_device_timeouts(cudaStream_t s);
// one scan whose second tile waits for a first tile that never publishes,
// with a wait limit of spin_limit polls: E_TIMEOUT when the wait gave up
int selftest_scan_wait(u32 spin_limit);
// the nth scan issued from now on (0: none) is recorded as one that gave up
void selftest_scan_report(u32 nth);

// out[i] = !(offs[i+1] - offs[i]) scanned (uints_negate_offsets, ints.cpp:227)
// newid (optional): out[i] where entity i is kept, INV where it is not
u32* negate_offsets(u32 const* offs, u32 n, cudaStream_t s, u32* total_to = nullptr,
    u32* newid = nullptr);

void fill_u32(u32* a, u32 n, u32 v, cudaStream_t s);

// device arrays copied to others that they do not overlap, MAX_COPY_JOBS to
// a launch (a mesh's connectivity and tags are a dozen arrays, and a driver
// copy costs the host 8 us whatever its size)
constexpr u32 MAX_COPY_JOBS = 16;
struct CopyJob {
  void const* src;
  void* dst;
  size_t bytes;
};
void copy_many(CopyJob const* jobs, size_t njobs, cudaStream_t s);

// grow the device's memory pool to at least `bytes` now (the pool keeps what
// it holds), so that later passes do not pay for growing it
void pool_reserve(unsigned long long bytes);
void pool_stats(unsigned long long* reserved, unsigned long long* used,
    unsigned long long* used_high, int reset_high);
void iota_u32(u32* a, u32 n, u32 stride, cudaStream_t s);
void iota_u64(u64* a, u32 n, cudaStream_t s);

// expand_array (arrays.cpp:170-192): rows of `width` elements of size esz
// copied to every slot [offs[i], offs[i+1]); output rows start at out.
void expand_rows(void const* in, u32 const* offs, u32 n, u32 width, u32 esz,
    void* out, cudaStream_t s);

// max over a u32 array (uints_max)
u32 max_u32(u32 const* a, u32 n, cudaStream_t s);

// Per-kernel event probes. When a probe is enabled, every launch it wraps is
// bracketed by CUDA events on the launching stream and credited with the
// launch's algorithmic bytes (each input read once, each output written
// once); the pairs are resolved after the timed region by probe_read.
enum ProbeId {
  P_REFLECT_DOWN = 0,
  P_UP_COUNT,
  P_UP_FILL,
  P_UP_RANK,
  P_EXSCAN,
  P_ELEM_QUALITY,
  P_REFINE_CANDIDATES,
  P_REFINE_QUALITY,
  P_INDSET_ROUND,
  P_COARSEN_QUALITY,
  P_SWAP_QUALITY,
  P_REFINE_TOPOLOGY,
  P_COLLAPSE_TO_ENT,
  P_EXPAND,
  P_CARRY,
  P_CARRY_UP,
  P_CARRY_UP_FILL,
  P_NPROBES
};
char const* probe_name(u32 id);
// the single-precision filter's device counters (one buffer per device)
struct Fp32Stats;
Fp32Stats* fp32_stats_dev();
void fp32_stats_read(unsigned long long* decided, unsigned long long* rechecked,
    double* max_err, unsigned* bound_exceeded);
void fp32_stats_reset();
// audit mode (every decision taken on an estimate also taken in double) and
// its counters
void fp32_set_audit(bool on);
void fp32_audit_read(unsigned long long* audited, unsigned long long* flips,
    unsigned long long* checked);
// the filter's estimates for n given tets (12 coordinates each) and edges
// (6 coordinates and 2 sizes each), with the double values (filter.cu)
void fp32_probe_tets(u32 n, double const* host_x, float* est, float* err, double* q64);
void fp32_probe_edges(u32 n, double const* host_x, double const* host_h, double thr,
    int* side, double* ratio64);

void probe_enable(u32 mask);
void probe_reset();
void probe_read(u32 id, u32* launches, double* ms, double* bytes);

struct ProbeScope {
  cudaEvent_t a = nullptr, b = nullptr;
  u32 id;
  double bytes;
  cudaStream_t s;
  ProbeScope(u32 id, cudaStream_t s, double bytes);
  ~ProbeScope();
};
#define PROBE(id, stream, bytes) ::osh::ProbeScope osh_probe_scope_((id), (stream), (double)(bytes))

// number of kernels this library launched in the process, and the number of
// times it waited for the device
unsigned long long launch_count();
unsigned long long sync_count();
// device allocations made so far, and host seconds spent waiting in stream
// synchronisations
void host_stats(unsigned long long* allocs, double* sync_seconds);
void stream_sync(cudaStream_t s);
bool stream_captures(cudaStream_t s);  // (or cannot be asked)
// 64 bytes of pinned host memory owned by the calling host thread, for small
// device-to-host reads (a read into pageable memory is staged by the driver)
void* pinned_scratch();

// small pinned host mailbox for reading several device scalars at once.
// Slots, by the step that writes them (steps of one mesh run one at a time,
// so steps that never overlap share slots):
//   44-50   independent set: blocks done, largest depth, list lengths of the
//           rounds, rounds run (or the largest depth), a wait that gave up
//           (one launch decides the set); 51: candidates listed for a set
//           from a filter
//   0-3     refinement: candidates listed, any good candidate, any inverted
//           child, any candidate
//   4-7     coarsening selection: any collapse kept (4), codes flag, then
//           candidate vertices listed (5, not read), listed edges (7); swap
//           selection: interior candidates (5, not read), any swap kept (6),
//           kept edges listed (7, not read)
//   8-11    refinement build: split entities per domain dimension
//   16-22   coarsening build: products and survivors per dimension, kept
//           vertices (22)
//   20-25   swap build: products and survivors per dimension
//   30-31   size fields (a 64-bit word)
//   59      adjacency derivation: a scan's total
//   60-63   zero but where something is to be told (take puts them back): a
//           star or a dual past its cap (60, 61); classification: a walk
//           past its bound, hinges too close to the angle to call (62, 63)
// fetch: a one-block kernel stores each slot into pinned host memory (mapped
// into the device's address space) with the number of the post beside it;
// the host spins on those words (asking the stream for errors as it waits)
// instead of waiting for a copy and a stream synchronisation, which woke the
// host 6-20 us after the copy ended.
struct Mailbox {
  static constexpr u32 POSTED = 65;  // up to 64 words and the scans' error
  // pinned and mapped, a word of the last post each: its number above its value
  unsigned long long volatile* posted = nullptr;
  unsigned long long* posted_dev = nullptr;  // the device's address of them
  u32* host = nullptr;   // 64 slots and the words of read
  u32* dev = nullptr;    // device, 64 slots
  u32 seq = 0;
  int device = 0;
  // init takes a mailbox another mesh gave back where there is one; release
  // gives it back, so no kernel that writes its slots may be pending then
  void init(cudaStream_t s);
  void release();
  void clear(cudaStream_t s);                 // zero the device slots
  void fetch(cudaStream_t s, u32 nslots = 64);  // the first nslots slots to host
  // after a fetch: the slot's word, its device slot zeroed where it is not
  u32 take(cudaStream_t s, u32 slot);
  // nwords (at most 16) 32-bit words of any device array, the same way,
  // into host[READ_SLOT..]; returns that host address
  static constexpr u32 READ_SLOT = 64;
  static constexpr u32 ERR_SLOT = READ_SLOT + 16;
  u32 const* read(cudaStream_t s, u32 const* src, u32 nwords);
  // nslots words (at most 64) of src into host[at..]; throws E_TIMEOUT where
  // a scan of the stream has given up since the last post or check
  void post(cudaStream_t s, u32 const* src, u32 nslots, u32 at);
};

}  // namespace osh
