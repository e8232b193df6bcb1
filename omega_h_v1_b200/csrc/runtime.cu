// Device runtime for the adaptation pass: error state, stream-ordered
// allocation, the decoupled look-back exclusive scan and small array kernels.
#include <algorithm>
#include <cstdlib>
#include <dlfcn.h>
#include <string>
#include <chrono>
#include <cstdio>
#include <cstring>
#include <atomic>
#include <map>
#include <mutex>
#include <tuple>
#include <vector>

#include "kept_blocks.hpp"
#include "runtime.hpp"

namespace osh {

namespace {

struct TuneSpec {
  char const* name;
  u32 def;
  u32 allowed[5];
};
TuneSpec const g_tune_spec[TK_NKEYS] = {
    {"carry_group", 8, {4, 8, 16, 0, 0}},
    {"vert_group", 8, {4, 8, 16, 0, 0}},
    {"indset_vert_group", 8, {4, 8, 16, 0, 0}},
    {"indset_edge_group", 4, {1, 2, 4, 8, 0}},
    {"quality_block", 256, {64, 128, 256, 512, 0}},
    {"gather_block", 256, {128, 256, 512, 0, 0}},
    {"scan_items", 16, {8, 16, 0, 0, 0}},
    {"scan_threads", 512, {256, 512, 0, 0, 0}},
    {"indset_blocks", 0, {0, 1, 2, 4, 0}},
    {"small_mesh_elems", 50000, {0, 25000, 50000, 100000, 200000}},
};
std::atomic<u32> g_tune[TK_NKEYS];
std::once_flag g_tune_once;

bool tune_allowed(u32 k, u32 v)
{
  // the list ends at the first 0 after its first entry (0 may be a value)
  TuneSpec const& t = g_tune_spec[k];
  for (u32 i = 0; i < 5; ++i) {
    if (i > 0 && t.allowed[i] == 0) break;
    if (t.allowed[i] == v) return true;
  }
  return false;
}

int tune_find(char const* name)
{
  if (!name) return -1;
  for (u32 k = 0; k < TK_NKEYS; ++k)
    if (std::strcmp(name, g_tune_spec[k].name) == 0) return (int)k;
  return -1;
}

int tune_read_file(char const* path, bool apply)
{
  FILE* f = std::fopen(path, "r");
  if (!f) return E_IO;
  std::vector<std::pair<u32, u32>> sets;
  char line[256];
  int rc = E_OK;
  while (std::fgets(line, sizeof line, f)) {
    char* h = std::strchr(line, '#');
    if (h) *h = 0;
    char name[64];
    unsigned v = 0;
    char extra[8];
    int got = std::sscanf(line, "%63s %u %7s", name, &v, extra);
    if (got <= 0) continue;  // blank or comment
    int k = got == 2 ? tune_find(name) : -1;
    if (k < 0 || !tune_allowed((u32)k, v)) {
      rc = E_ARG;
      break;
    }
    sets.emplace_back((u32)k, (u32)v);
  }
  std::fclose(f);
  if (rc == E_OK && apply)
    for (auto const& kv : sets) g_tune[kv.first].store(kv.second);
  return rc;
}

void tune_init()
{
  std::call_once(g_tune_once, [] {
    for (u32 k = 0; k < TK_NKEYS; ++k) g_tune[k].store(g_tune_spec[k].def);
    char const* env = std::getenv("OSH_B200_TUNING");
    if (env && *env) {
      tune_read_file(env, true);
      return;
    }
    Dl_info info;
    if (dladdr(reinterpret_cast<void*>(&tune_init), &info) && info.dli_fname) {
      std::string p(info.dli_fname);
      size_t slash = p.rfind('/');
      p = (slash == std::string::npos ? std::string(".") : p.substr(0, slash)) + "/tuning.txt";
      tune_read_file(p.c_str(), true);
    }
  });
}

}  // namespace

u32 tuned(TuneKey k)
{
  tune_init();
  return g_tune[k].load(std::memory_order_relaxed);
}

char const* tune_name(u32 k) { return k < TK_NKEYS ? g_tune_spec[k].name : nullptr; }

int tune_set(char const* name, u32 value)
{
  tune_init();
  int k = tune_find(name);
  if (k < 0 || !tune_allowed((u32)k, value)) return E_ARG;
  g_tune[k].store(value);
  return E_OK;
}

int tune_get(char const* name, u32* value)
{
  tune_init();
  int k = tune_find(name);
  if (k < 0) return E_ARG;
  if (value) *value = g_tune[k].load();
  return E_OK;
}

int tune_load(char const* path)
{
  tune_init();
  if (!path) return E_ARG;
  return tune_read_file(path, true);
}

bool pdl_enabled()
{
  static bool const on = [] {
    char const* e = std::getenv("OSH_B200_PDL");
    return !(e && e[0] == '0');
  }();
  return on;
}


// ---------------------------------------------------------------------------
// errors

namespace {
thread_local int t_err = 0;
thread_local std::string t_msg;
}  // namespace

void set_error(int code, char const* msg)
{
  t_err = code;
  t_msg = msg ? msg : "";
}
int last_error() { return t_err; }
char const* last_error_message() { return t_msg.c_str(); }
void clear_error()
{
  t_err = 0;
  t_msg.clear();
}

void check_cuda(cudaError_t e, char const* what, char const* file, int line)
{
  if (e == cudaSuccess) return;
  char buf[512];
  snprintf(buf, sizeof(buf), "%s failed: %s (%s:%d)", what, cudaGetErrorString(e),
      file, line);
  throw Failure(e == cudaErrorMemoryAllocation ? E_NOMEM : E_CUDA, buf);
}

// ---------------------------------------------------------------------------
// launch counter (every kernel launch goes through CK_LAUNCH)

namespace {
std::atomic<unsigned long long> g_launches{0};
}
void count_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }
unsigned long long launch_count() { return g_launches.load(); }

namespace {
std::atomic<unsigned long long> g_syncs{0};
std::atomic<unsigned long long> g_sync_ns{0};
std::atomic<unsigned long long> g_allocs{0};
}
unsigned long long sync_count() { return g_syncs.load(); }
void stream_sync(cudaStream_t s)
{
  g_syncs.fetch_add(1, std::memory_order_relaxed);
  auto t0 = std::chrono::steady_clock::now();
  CK(cudaStreamSynchronize(s));
  auto dt = std::chrono::steady_clock::now() - t0;
  g_sync_ns.fetch_add((unsigned long long)std::chrono::duration_cast<std::chrono::nanoseconds>(
      dt).count(), std::memory_order_relaxed);
}
void host_stats(unsigned long long* allocs, double* sync_seconds)
{
  if (allocs) *allocs = g_allocs.load();
  if (sync_seconds) *sync_seconds = g_sync_ns.load() * 1e-9;
}

// ---------------------------------------------------------------------------
// probes

namespace {
struct ProbeState {
  u32 mask = 0;
  struct Rec {
    cudaEvent_t a, b;
    double bytes;
  };
  std::vector<Rec> recs[P_NPROBES];
  u32 launches[P_NPROBES] = {};
  double ms[P_NPROBES] = {};
  double bytes[P_NPROBES] = {};
  std::mutex mu;
};
ProbeState& probes()
{
  static ProbeState p;
  return p;
}
char const* const g_probe_names[P_NPROBES] = {"reflect_down", "up_count", "up_fill",
    "up_rank", "exscan", "elem_quality", "refine_candidates", "refine_quality",
    "indset_round", "coarsen_quality", "swap_quality", "refine_topology",
    "collapse_to_ent", "expand", "carry_down", "carry_up", "carry_up_fill"};
}  // namespace

char const* probe_name(u32 id) { return id < P_NPROBES ? g_probe_names[id] : nullptr; }

namespace {
std::once_flag g_fp32_once[64];
Fp32Stats* g_fp32[64] = {};
}

Fp32Stats* fp32_stats_dev()
{
  int dev = 0;
  CK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) throw Failure(E_ARG, "device index out of range");
  std::call_once(g_fp32_once[dev], [dev]() {
    void* p = nullptr;
    CK(cudaMalloc(&p, sizeof(Fp32Stats)));
    CK(cudaMemset(p, 0, sizeof(Fp32Stats)));
    g_fp32[dev] = static_cast<Fp32Stats*>(p);
  });
  return g_fp32[dev];
}

void fp32_stats_read(unsigned long long* decided, unsigned long long* rechecked,
    double* max_err, unsigned* bound_exceeded)
{
  Fp32Stats h;
  CK(cudaDeviceSynchronize());
  CK(cudaMemcpy(&h, fp32_stats_dev(), sizeof(h), cudaMemcpyDeviceToHost));
  float e;
  std::memcpy(&e, &h.max_err_bits, sizeof(e));
  if (decided) *decided = h.decided;
  if (rechecked) *rechecked = h.rechecked;
  if (max_err) *max_err = e;
  if (bound_exceeded) *bound_exceeded = h.bound_exceeded;
}

void fp32_audit_read(unsigned long long* audited, unsigned long long* flips,
    unsigned long long* checked)
{
  Fp32Stats h;
  CK(cudaDeviceSynchronize());
  CK(cudaMemcpy(&h, fp32_stats_dev(), sizeof(h), cudaMemcpyDeviceToHost));
  if (audited) *audited = h.audited;
  if (flips) *flips = h.flips;
  if (checked) *checked = h.checked;
}

// the counters return to zero; the audit switch is kept
void fp32_stats_reset()
{
  CK(cudaDeviceSynchronize());
  Fp32Stats* d = fp32_stats_dev();
  unsigned audit = 0;
  CK(cudaMemcpy(&audit, &d->audit, sizeof(audit), cudaMemcpyDeviceToHost));
  Fp32Stats z;
  std::memset(&z, 0, sizeof(z));
  z.audit = audit;
  CK(cudaMemcpy(d, &z, sizeof(z), cudaMemcpyHostToDevice));
}

void fp32_set_audit(bool on)
{
  CK(cudaDeviceSynchronize());
  unsigned v = on ? 1u : 0u;
  CK(cudaMemcpy(&fp32_stats_dev()->audit, &v, sizeof(v), cudaMemcpyHostToDevice));
}

void probe_enable(u32 mask) { probes().mask = mask; }

static void probe_resolve(ProbeState& p)
{
  for (u32 i = 0; i < P_NPROBES; ++i) {
    for (auto& r : p.recs[i]) {
      float t = 0;
      CK(cudaEventSynchronize(r.b));
      CK(cudaEventElapsedTime(&t, r.a, r.b));
      p.launches[i] += 1;
      p.ms[i] += t;
      p.bytes[i] += r.bytes;
      cudaEventDestroy(r.a);
      cudaEventDestroy(r.b);
    }
    p.recs[i].clear();
  }
}

void probe_reset()
{
  ProbeState& p = probes();
  std::lock_guard<std::mutex> g(p.mu);
  probe_resolve(p);
  for (u32 i = 0; i < P_NPROBES; ++i) {
    p.launches[i] = 0;
    p.ms[i] = 0;
    p.bytes[i] = 0;
  }
}

void probe_read(u32 id, u32* launches, double* ms, double* bytes)
{
  ProbeState& p = probes();
  std::lock_guard<std::mutex> g(p.mu);
  probe_resolve(p);
  *launches = p.launches[id];
  *ms = p.ms[id];
  *bytes = p.bytes[id];
}

ProbeScope::ProbeScope(u32 i, cudaStream_t st, double by) : id(i), bytes(by), s(st)
{
  if (!((probes().mask >> id) & 1u)) return;
  CK(cudaEventCreate(&a));
  CK(cudaEventCreate(&b));
  CK(cudaEventRecord(a, s));
}

ProbeScope::~ProbeScope()
{
  if (!a) return;
  cudaEventRecord(b, s);
  ProbeState& p = probes();
  std::lock_guard<std::mutex> g(p.mu);
  p.recs[id].push_back({a, b, bytes});
}

// ---------------------------------------------------------------------------
// allocation: the device's default memory pool, never trimmed between passes

namespace {
std::once_flag g_pool_once[64];
}

static void setup_pool()
{
  int dev = 0;
  CK(cudaGetDevice(&dev));
  std::call_once(g_pool_once[dev & 63], [dev]() {
    cudaMemPool_t pool;
    if (cudaDeviceGetDefaultMemPool(&pool, dev) == cudaSuccess) {
      unsigned long long thr = ~0ull;
      cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &thr);
    }
  });
}

namespace {
BlockTable& blocks()
{
  static auto* t = new BlockTable();  // lives to exit
  return *t;
}

// the device's memory pool
struct DriverPool {
  bool full = false;
  void* alloc(size_t bytes, void* s)
  {
    void* p = nullptr;
    cudaError_t const e = cudaMallocAsync(&p, bytes, static_cast<cudaStream_t>(s));
    if (e == cudaSuccess) return p;
    cudaGetLastError();
    full = e == cudaErrorMemoryAllocation;
    return nullptr;
  }
  void free(void* p, void* s) { cudaFreeAsync(p, static_cast<cudaStream_t>(s)); }
  void wait(void* s) { cudaStreamSynchronize(static_cast<cudaStream_t>(s)); }
};

bool capturing(cudaStream_t s)
{
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &st) == cudaSuccess) return st != cudaStreamCaptureStatusNone;
  cudaGetLastError();  // (the legacy stream while another captures)
  return true;
}

// streams and mailboxes that meshes gave back, for the next mesh: a stream
// takes the driver about 70 us to make and 80 to destroy
constexpr size_t SPARE_MAX = 64;
struct Spares {
  std::mutex mu;
  std::map<cudaStream_t, int> made_on;  // the device of each stream made here
  std::map<cudaStream_t, u32> users;    // the meshes on each caller's stream
  std::map<int, std::vector<cudaStream_t>> streams;
  std::map<int, std::vector<Mailbox>> boxes;
};
Spares& spares()
{
  static auto* t = new Spares();
  return *t;
}
}  // namespace

cudaStream_t take_stream()
{
  int dev = 0;
  CK(cudaGetDevice(&dev));
  Spares& sp = spares();
  {
    std::lock_guard<std::mutex> g(sp.mu);
    auto& v = sp.streams[dev];
    if (!v.empty()) {
      cudaStream_t s = v.back();
      v.pop_back();
      return s;
    }
  }
  cudaStream_t s = nullptr;
  CK(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
  std::lock_guard<std::mutex> g(sp.mu);
  sp.made_on[s] = dev;
  return s;
}

void give_back_stream(cudaStream_t s)
{
  release_stream_scratch(s);
  Spares& sp = spares();
  {
    std::lock_guard<std::mutex> g(sp.mu);
    auto it = sp.made_on.find(s);
    if (it != sp.made_on.end()) {
      auto& v = sp.streams[it->second];
      if (v.size() < SPARE_MAX && cudaStreamQuery(s) != cudaErrorInvalidResourceHandle) {
        v.push_back(s);
        return;
      }
      sp.made_on.erase(it);
    }
  }
  cudaStreamDestroy(s);
}

void begin_stream_use(cudaStream_t s)
{
  if (!s || s == cudaStreamLegacy) return;
  Spares& sp = spares();
  std::lock_guard<std::mutex> g(sp.mu);
  if (!sp.made_on.count(s)) ++sp.users[s];
}

void end_stream_use(cudaStream_t s)
{
  if (!s || s == cudaStreamLegacy) return;
  Spares& sp = spares();
  {
    std::lock_guard<std::mutex> g(sp.mu);
    auto it = sp.users.find(s);
    if (it == sp.users.end() || --it->second) return;
    sp.users.erase(it);
  }
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return;
  for (auto const& b : blocks().drop(dev, s)) cudaFreeAsync(b.p, s);
}

// from the pool, with the blocks kept on the device given back to it where
// that is needed (not under capture, where they could not be); E_NOMEM
static void* pool_alloc(size_t bytes, cudaStream_t s)
{
  int dev = 0;
  CK(cudaGetDevice(&dev));
  DriverPool pool;
  void* p = capturing(s) ? pool.alloc(bytes, s) : alloc_or_drop(blocks(), pool, dev, bytes, s);
  if (!p) {
    char buf[128];
    snprintf(buf, sizeof(buf), "device allocation of %zu bytes failed", bytes);
    throw Failure(E_NOMEM, buf);
  }
  return p;
}

// A stream under capture goes to the driver's pool, whose calls are captured.
void* dev_alloc(size_t bytes, cudaStream_t s)
{
  setup_pool();
  if (bytes < 16) bytes = 16;
  g_allocs.fetch_add(1, std::memory_order_relaxed);
  int dev = 0;
  CK(cudaGetDevice(&dev));
  BlockTable& t = blocks();
  bool const small = bytes <= BLOCK_MAX && !capturing(s);
  u32 cls = 0;
  if (small) {
    cls = block_class(bytes, &bytes);
    if (void* p = t.take(dev, s, cls)) return p;
  }
  void* p = pool_alloc(bytes, s);
  if (small)
    t.made(p, dev, cls);
  else
    t.not_a_block(p);
  return p;
}

void pool_reserve(unsigned long long bytes)
{
  setup_pool();
  if (!bytes) return;
  void* p = nullptr;
  try {
    p = pool_alloc(bytes, 0);
  } catch (Failure const&) {
    throw Failure(E_NOMEM, "could not reserve the requested device memory");
  }
  CK(cudaFreeAsync(p, 0));
  CK(cudaStreamSynchronize(0));
}

void pool_stats(unsigned long long* reserved, unsigned long long* used,
    unsigned long long* used_high, int reset_high)
{
  setup_pool();
  int dev = 0;
  CK(cudaGetDevice(&dev));
  cudaMemPool_t pool;
  CK(cudaDeviceGetDefaultMemPool(&pool, dev));
  unsigned long long r = 0, u = 0, h = 0;
  CK(cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &r));
  CK(cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &u));
  CK(cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemHigh, &h));
  if (reserved) *reserved = r;
  // the blocks kept for the next allocations are not in use
  u -= std::min<unsigned long long>(u, blocks().kept_bytes(dev));
  if (used) *used = u;
  if (used_high) *used_high = h;
  if (reset_high) {
    unsigned long long zero = 0;
    CK(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrUsedMemHigh, &zero));
  }
}

void dev_free(void* p, cudaStream_t s)
{
  if (!p) return;
  // (one handle names every thread's own default stream: nothing kept there)
  if (blocks().keep(p, s, s != cudaStreamPerThread && !capturing(s))) return;
  CK(cudaFreeAsync(p, s));
}

void dev_drop(void* p, cudaStream_t s) noexcept
{
  try {
    dev_free(p, s);
  } catch (...) {
    cudaGetLastError();
  }
}

namespace {
// a pinned word per host thread for read_u32: a copy into pageable memory
// goes through the driver's staging buffer and takes several times longer.
// Words go back to a process-wide free list when their thread ends (pinning
// and unpinning memory each take a driver call that can wait for the
// device, which short-lived worker threads would pay every time).
std::mutex g_words_mu;
std::vector<u32*>& free_words()
{
  static std::vector<u32*>* v = new std::vector<u32*>();  // lives to exit
  return *v;
}
struct PinnedWord {
  u32* p = nullptr;
  ~PinnedWord()
  {
    if (!p) return;
    std::lock_guard<std::mutex> g(g_words_mu);
    free_words().push_back(p);
  }
  u32* get()
  {
    if (p) return p;
    {
      std::lock_guard<std::mutex> g(g_words_mu);
      if (!free_words().empty()) {
        p = free_words().back();
        free_words().pop_back();
        return p;
      }
    }
    CK(cudaMallocHost(&p, 64));
    return p;
  }
};
thread_local PinnedWord t_word;
}  // namespace

void* pinned_scratch() { return t_word.get(); }

u32 read_u32(u32 const* d, cudaStream_t s)
{
  u32* h = t_word.get();
  CK(cudaMemcpyAsync(h, d, sizeof(u32), cudaMemcpyDeviceToHost, s));
  stream_sync(s);
  return *h;
}

double read_f64(double const* d, cudaStream_t s)
{
  double* h = static_cast<double*>(pinned_scratch());
  CK(cudaMemcpyAsync(h, d, sizeof(double), cudaMemcpyDeviceToHost, s));
  stream_sync(s);
  return *h;
}

void Mailbox::init(cudaStream_t s)
{
  if (host) return;
  int d = 0;
  CK(cudaGetDevice(&d));
  {
    Spares& sp = spares();
    std::lock_guard<std::mutex> g(sp.mu);
    auto& v = sp.boxes[d];
    if (!v.empty()) {
      *this = v.back();
      v.pop_back();
    }
  }
  if (host) {  // (its numbers go on: the words posted hold the last ones)
    clear(s);
    return;
  }
  device = d;
  void* h = nullptr;
  size_t const bytes = POSTED * sizeof(u64) + (ERR_SLOT + 1) * sizeof(u32);
  CK(cudaMallocHost(&h, bytes));
  std::memset(h, 0, bytes);
  posted = static_cast<unsigned long long volatile*>(h);
  host = reinterpret_cast<u32*>(static_cast<char*>(h) + POSTED * sizeof(u64));
  void* hd = nullptr;
  CK(cudaHostGetDevicePointer(&hd, h, 0));
  posted_dev = static_cast<unsigned long long*>(hd);
  seq = 0;
  // (not one of the kept blocks: it outlives any stream)
  void* p = nullptr;
  CK(cudaMalloc(&p, 64 * sizeof(u32)));
  dev = static_cast<u32*>(p);
  clear(s);
}

void Mailbox::release()
{
  if (host && dev) {
    Spares& sp = spares();
    std::lock_guard<std::mutex> g(sp.mu);
    auto& v = sp.boxes[device];
    if (v.size() < SPARE_MAX) {
      v.push_back(*this);
      host = nullptr;
      posted = nullptr;
      posted_dev = nullptr;
      dev = nullptr;
      return;
    }
  }
  if (host) cudaFreeHost(const_cast<unsigned long long*>(posted));
  if (dev) cudaFree(dev);
  host = nullptr;
  posted = nullptr;
  posted_dev = nullptr;
  dev = nullptr;
}

void Mailbox::clear(cudaStream_t s)
{
  CK(cudaMemsetAsync(dev, 0, 64 * sizeof(u32), s));
}

// Each word goes to the host with the post's number in the same 64-bit store,
// so the host has it when it sees the number: no word waits for another, nor
// for a fence across the bus and a flag after it (6 -> 3 us a post).
// Word n of a post is the stream's scan error (err; null: no scan yet).
__global__ void k_mailbox_post(u32 const* __restrict__ src, u32 n, u32 const* __restrict__ err,
    unsigned long long* dst, u32 seq)
{
  pdl_wait();
  u32 i = threadIdx.x;
  if (i > n) return;
  u32 const w = i < n ? src[i] : err ? *err : 0u;
  reinterpret_cast<volatile unsigned long long*>(dst)[i] = (unsigned long long)seq << 32 | w;
}

namespace {
// the scratch of a stream's scans: [ticket, error, done, pad] then two words
// per tile
struct ScanScratch {
  u32* p = nullptr;
  size_t words = 0;
};
ScanScratch find_scan_scratch(cudaStream_t s);
[[noreturn]] void scan_gave_up(ScanScratch const& sc, cudaStream_t s);
}  // namespace

bool stream_captures(cudaStream_t s) { return capturing(s); }

u32 const* Mailbox::read(cudaStream_t s, u32 const* src, u32 nwords)
{
  if (nwords > 16) throw Failure(E_ARG, "mailbox read: at most 16 words");
  post(s, src, nwords, READ_SLOT);
  return host + READ_SLOT;
}

void Mailbox::fetch(cudaStream_t s, u32 nslots)
{
  post(s, dev, nslots > 64 ? 64 : nslots, 0);
}

u32 Mailbox::take(cudaStream_t s, u32 slot)
{
  u32 const v = host[slot];
  if (v) CK(cudaMemsetAsync(dev + slot, 0, sizeof(u32), s));
  return v;
}

void Mailbox::post(cudaStream_t s, u32 const* src, u32 nslots, u32 at)
{
  u32 const want = ++seq;
  g_syncs.fetch_add(1, std::memory_order_relaxed);
  auto t0 = std::chrono::steady_clock::now();
  ScanScratch const scan = find_scan_scratch(s);
  u32 const* err = scan.p ? scan.p + 1 : nullptr;
  CK(launch_kernel(k_mailbox_post, dim3(1), dim3(96), 0, s, src, nslots, err, posted_dev, want));
  CK_LAUNCH();
  u32 got = 0;
  u32& gave_up = host[ERR_SLOT];
  auto arrived = [&] {
    for (; got <= nslots; ++got) {
      unsigned long long const w = posted[got];
      if ((u32)(w >> 32) != want) return false;
      (got < nslots ? host[at + got] : gave_up) = (u32)w;
    }
    return true;
  };
  for (u64 it = 1; !arrived(); ++it) {
    if ((it & 255) != 0) continue;
    // now and then: a failed stream ends the wait with its error; a drained
    // stream whose words have not arrived (they should have) falls back to a
    // copy and a synchronisation
    cudaError_t st = cudaStreamQuery(s);
    if (st == cudaErrorNotReady) continue;
    CK(st);
    if (arrived()) break;
    gave_up = 0;
    CK(cudaMemcpyAsync(host + at, src, nslots * sizeof(u32), cudaMemcpyDeviceToHost, s));
    if (err) CK(cudaMemcpyAsync(&gave_up, err, sizeof(u32), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    break;
  }
  std::atomic_thread_fence(std::memory_order_acquire);
  auto dt = std::chrono::steady_clock::now() - t0;
  g_sync_ns.fetch_add((unsigned long long)std::chrono::duration_cast<std::chrono::nanoseconds>(
      dt).count(), std::memory_order_relaxed);
  // (what was read may come of a scan that gave up: no pass goes on with it)
  if (gave_up) scan_gave_up(scan, s);
}

// ---------------------------------------------------------------------------
// exclusive scan, single pass with decoupled look-back.
//
// Tiles are claimed through an atomic ticket, so every tile a block waits on
// was claimed (and is running or done) before it. Each tile publishes its
// aggregate, then walks back over predecessors until it meets an inclusive
// prefix. The walk is bounded: after spin_limit empty polls (SCAN_SPIN_LIMIT
// in every scan the passes issue) it sets the scratch's error word, which
// the host reads for that stream (check_device_timeouts), and stops instead
// of spinning forever.

// Tiles of SCAN_T threads (the tuning table's scan_threads, 256 or 512)
// times SCAN_ITEMS items (scan_items, 8 or 16; 256 x 32 where a scan is long,
// see LONG_SCAN). With 8192-element tiles a
// 2M-element scan has 256 tiles, so a tile's look-back meets a published
// prefix within a few steps (with 2048-element tiles the chain of
// look-backs, not bandwidth, set the time of the adapt's scans). Scratch
// is sized for the smallest tile, so every shape fits.
constexpr int SCAN_MIN_TILE = 256 * 8;
constexpr unsigned long long FLAG_AGG = 1ull << 62;
constexpr unsigned long long FLAG_PRE = 2ull << 62;
constexpr u32 SCAN_SPIN_LIMIT = 1u << 24;

// Several independent scans in one launch. Job j scans its `in` (mode 0),
// the survivors of an offsets array, (in[i + 1] == in[i]) (mode 1,
// uints_negate_offsets, ints.cpp:227-235), or the entries stamped with its
// stamp, (in[i] == stamp) (mode 2), into out[0..n] with the total at
// out[n] (and in *total_to when given); newid (optional, for 0/1 items)
// receives out[i] where item i is 1 and INV where it is 0 -- each old
// entity's new id when the items mark survivors. Tiles are numbered across
// the jobs (job j owns tiles tile0[j] .. tile0[j + 1] - 1, one at least) and
// claimed through one ticket, so a look-back, which stops at its job's
// first tile, only waits on tiles claimed before it. Independent scans of a
// pass share a launch, and their look-back chains overlap.
//
// A warp takes CH chunks of 128 consecutive items, a lane 4 consecutive ones
// of each, as one 16-byte word where every array of the job starts on 16
// bytes: loads and stores are coalesced as they stand, the chunks' scans are
// independent shuffles, and nothing is transposed through shared memory
// (which took four shared-memory accesses an item and half the issue slots:
// 28M items 61 us, now 53; 1.5M 8.4, now 7.2). A launch of one tile needs no
// ticket, status or clean-up.
__device__ inline void scan_store4(u32* __restrict__ a, size_t gi, u32 n, bool wide, u32 x0,
    u32 x1, u32 x2, u32 x3)
{
  if (wide && gi + 4 <= n) {
    *reinterpret_cast<uint4*>(a + gi) = make_uint4(x0, x1, x2, x3);
    return;
  }
  if (gi < n) a[gi] = x0;
  if (gi + 1 < n) a[gi + 1] = x1;
  if (gi + 2 < n) a[gi + 2] = x2;
  if (gi + 3 < n) a[gi + 3] = x3;
}

// a count by one, after every write this thread has made before it, for any
// thread on the device that sees the count and fences
__device__ __forceinline__ u32 count_released(u32* n)
{
  u32 was;
  asm volatile("atom.add.release.gpu.u32 %0, [%1], 1;" : "=r"(was) : "l"(n) : "memory");
  return was;
}

template <int SCAN_T, int SCAN_ITEMS>
__global__ void __launch_bounds__(SCAN_T)
k_exscan(const __grid_constant__ ScanJobs jobs, unsigned long long* status,
    u32* ticket_and_err, u32 spin_limit)
{
  pdl_wait();
  constexpr u32 WARPS = SCAN_T / 32, CH = SCAN_ITEMS / 4;
  constexpr u32 SCAN_TILE = SCAN_T * SCAN_ITEMS;
  __shared__ u32 s_tile;
  __shared__ u32 s_warp[WARPS];
  __shared__ u32 s_prefix;
  u32 const ntiles = jobs.tile0[jobs.njobs];
  bool const single = ntiles == 1;
  u32 tile = 0;
  if (!single) {
    if (threadIdx.x == 0) s_tile = atomicAdd(ticket_and_err, 1u);
    __syncthreads();
    tile = s_tile;
    if (tile >= ntiles) return;
  }
  u32 jn = 0;
  while (jn + 1 < jobs.njobs && tile >= jobs.tile0[jn + 1]) ++jn;
  ScanJob const job = jobs.j[jn];
  u32 const first = jobs.tile0[jn], last = jobs.tile0[jn + 1] - 1;
  u32 const* __restrict__ in = job.in;
  u32* __restrict__ out = job.out;
  u32* __restrict__ newid = job.newid;
  u32* __restrict__ list = job.list;
  u32* __restrict__ comp = job.comp;
  u32* __restrict__ comp_newid = job.comp_newid;
  u32 const n = job.n;
  u32 const mode = job.mode, stamp = job.stamp;
  bool const wide = ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out) |
      reinterpret_cast<uintptr_t>(newid) | reinterpret_cast<uintptr_t>(comp) |
      reinterpret_cast<uintptr_t>(comp_newid)) & 15) == 0;
  u32 const lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  size_t const base = (size_t)(tile - first) * SCAN_TILE + warp * (CH * 128) + lane * 4;
  u32 v[CH][4];
#pragma unroll
  for (u32 c = 0; c < CH; ++c) {
    size_t const gi = base + c * 128;
    if (wide && gi + 4 <= n) {
      uint4 const x = *reinterpret_cast<uint4 const*>(in + gi);
      v[c][0] = x.x, v[c][1] = x.y, v[c][2] = x.z, v[c][3] = x.w;
    } else {
#pragma unroll
      for (u32 k = 0; k < 4; ++k) v[c][k] = gi + k < n ? in[gi + k] : 0u;
    }
  }
  if (mode == 1) {
    // (in has n + 1 entries; an item's right neighbour is the next lane's
    // first, or the entry after the chunk)
#pragma unroll
    for (u32 c = 0; c < CH; ++c) {
      size_t const gi = base + c * 128;
      u32 next = __shfl_down_sync(0xffffffffu, v[c][0], 1);
      if (gi + 4 >= n || lane == 31) next = gi + 4 <= n ? in[gi + 4] : 0u;
      u32 const tail = gi < n ? in[n] : 0u;  // the last item's neighbour
#pragma unroll
      for (u32 k = 0; k < 4; ++k) {
        u32 const r = gi + k + 1 == n ? tail : k < 3 ? v[c][k < 3 ? k + 1 : 3] : next;
        v[c][k] = gi + k < n && r == v[c][k] ? 1u : 0u;
      }
    }
  } else if (mode == 2) {
#pragma unroll
    for (u32 c = 0; c < CH; ++c)
#pragma unroll
      for (u32 k = 0; k < 4; ++k) v[c][k] = base + c * 128 + k < n && v[c][k] == stamp ? 1u : 0u;
  }
  u32 excl[CH];  // the lane's first item's prefix within the warp
  {
    u32 x[CH], sum[CH];
#pragma unroll
    for (u32 c = 0; c < CH; ++c) x[c] = sum[c] = v[c][0] + v[c][1] + v[c][2] + v[c][3];
#pragma unroll
    for (u32 o = 1; o < 32; o <<= 1)
#pragma unroll
      for (u32 c = 0; c < CH; ++c) {
        u32 const y = __shfl_up_sync(0xffffffffu, x[c], o);
        if (lane >= o) x[c] += y;
      }
    u32 run = 0;
#pragma unroll
    for (u32 c = 0; c < CH; ++c) {
      excl[c] = run + x[c] - sum[c];
      run += __shfl_sync(0xffffffffu, x[c], 31);
    }
    if (lane == 0) s_warp[warp] = run;
  }
  __syncthreads();
  u32 before = 0, total = 0;  // the warps before this one; the tile
#pragma unroll
  for (u32 w = 0; w < WARPS; ++w) {
    u32 const t = s_warp[w];
    if (w < warp) before += t;
    total += t;
  }
  u32 prefix = 0;
  if (tile != first || !single) {
    if (warp == 0) {
      // warp-cooperative look-back: lane l inspects tile (p - l)
      if (tile == first) {
        if (lane == 0) atomicExch(&status[tile], FLAG_PRE | (unsigned long long)total);
      } else {
        if (lane == 0) atomicExch(&status[tile], FLAG_AGG | (unsigned long long)total);
        int p = (int)tile - 1;
        u32 spins = 0;
        bool gave_up = false;
        for (;;) {
          int idx = p - (int)lane;
          unsigned long long st = FLAG_PRE;  // before the job's first tile: empty
          if (idx >= (int)first) st = *((volatile unsigned long long*)&status[idx]);
          while (__any_sync(0xffffffffu, (st >> 62) == 0)) {
            if (++spins > spin_limit) {
              gave_up = true;
              break;
            }
            if (idx >= (int)first && (st >> 62) == 0)
              st = *((volatile unsigned long long*)&status[idx]);
          }
          if (gave_up) {
            if (lane == 0) atomicOr(&ticket_and_err[1], 1u);
            break;
          }
          u32 pre = __ballot_sync(0xffffffffu, (st & (3ull << 62)) == FLAG_PRE);
          u32 stop = pre ? (u32)(__ffs(pre) - 1) : 31u;
          prefix += __reduce_add_sync(0xffffffffu, lane <= stop ? (u32)st : 0u);
          if (pre) break;
          p -= 32;
        }
        if (lane == 0) atomicExch(&status[tile], FLAG_PRE | (unsigned long long)(prefix + total));
      }
      if (lane == 0) s_prefix = prefix;
    }
    __syncthreads();
    prefix = s_prefix;
  }
  // Counted once the look-back is over; the count is looked at after the
  // stores, so its round trip is not waited for. It is released: the tile's
  // published prefix (this thread's exchange) has been performed when the
  // last tile sees it, so the zeros that one writes come after it. (Without
  // the order an exchange still under way could land on a word already
  // zeroed, and the next scan took the prefix it left for its own: on four
  // busy streams some thousand words in 20,000 launches. It costs 2 us of 53
  // at 28M items and 1 of 13 at 6M.)
  u32 done = 0;
  if (!single && threadIdx.x == 0) done = count_released(&ticket_and_err[2]);
  bool const marks = newid || list || comp_newid;
#pragma unroll
  for (u32 c = 0; c < CH; ++c) {
    size_t const gi = base + c * 128;
    if (gi >= n) break;
    u32 const g = (u32)gi;
    u32 const o0 = prefix + before + excl[c], o1 = o0 + v[c][0], o2 = o1 + v[c][1], o3 = o2 + v[c][2];
    scan_store4(out, gi, n, wide, o0, o1, o2, o3);
    if (comp) scan_store4(comp, gi, n, wide, g - o0, g + 1 - o1, g + 2 - o2, g + 3 - o3);
    if (!marks) continue;
    // (0/1 items)
    if (newid)
      scan_store4(newid, gi, n, wide, v[c][0] ? o0 : INV, v[c][1] ? o1 : INV,
          v[c][2] ? o2 : INV, v[c][3] ? o3 : INV);
    if (comp_newid)
      scan_store4(comp_newid, gi, n, wide, v[c][0] ? INV : g - o0, v[c][1] ? INV : g + 1 - o1,
          v[c][2] ? INV : g + 2 - o2, v[c][3] ? INV : g + 3 - o3);
    if (list) {
      if (v[c][0]) list[o0] = g;
      if (v[c][1]) list[o1] = g + 1;
      if (v[c][2]) list[o2] = g + 2;
      if (v[c][3]) list[o3] = g + 3;
    }
  }
  if (tile == last && threadIdx.x == 0) {
    out[n] = prefix + total;
    if (comp) comp[n] = n - (prefix + total);
    if (job.total_to) *job.total_to = prefix + total;
  }
  // The last tile past its look-back returns the scratch to zero for the
  // next scan on the stream: no look-back reads a status word any more.
  if (!single && warp == 0 && __shfl_sync(0xffffffffu, done, 0) == ntiles - 1) {
    __threadfence();  // after every tile's count, and so after its exchange
    __syncwarp();
    for (u32 t = lane; t < ntiles; t += 32) status[t] = 0ull;
    if (lane == 0) {
      ticket_and_err[0] = 0;
      ticket_and_err[2] = 0;
    }
  }
}

namespace {
// The calling host thread's number: small, its own while it runs, another
// thread's after it. Host threads may share a stream, where each thread's
// kernels run in its order but among the others': what one thread's kernel
// leaves in a scratch for its next (counts, marks) must be out of the others'
// reach, so every scratch is a (stream, host thread)'s. A thread that gets
// another's number after its end comes after it on the stream.
struct HostThread {
  static std::mutex& mu()
  {
    static auto* m = new std::mutex();
    return *m;
  }
  static std::vector<bool>& taken()
  {
    static auto* v = new std::vector<bool>();
    return *v;
  }
  u32 id = 0;
  HostThread()
  {
    std::lock_guard<std::mutex> g(mu());
    while (id < taken().size() && taken()[id]) ++id;
    if (id == taken().size()) taken().push_back(false);
    taken()[id] = true;
  }
  ~HostThread()
  {
    std::lock_guard<std::mutex> g(mu());
    taken()[id] = false;
  }
};
u32 host_thread()
{
  static thread_local HostThread t;
  return t.id;
}

// Scratch of the scans issued on each stream by each host thread ([ticket,
// error, done, pad] then two words per tile), zero between scans: the scan
// kernel's last tile clears it, so no scan pays for a memset. Freed by
// release_stream_scratch when the stream goes.
std::mutex g_scan_mu;
using ScanKey = std::tuple<int, cudaStream_t, u32>;  // device, stream, host thread
std::map<ScanKey, ScanScratch>& scan_scratches()
{
  static auto* m = new std::map<ScanKey, ScanScratch>();
  return *m;
}

u32* stream_scan_scratch(size_t words, cudaStream_t s)
{
  int dev = 0;
  CK(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> g(g_scan_mu);
  auto& all = scan_scratches();
  ScanScratch& sc = all[ScanKey{dev, s, host_thread()}];
  if (sc.words < words) {
    size_t want = std::max(words, (size_t)4096);
    void* q = pool_alloc(want * sizeof(u32), s);
    CK(cudaMemsetAsync(q, 0, want * sizeof(u32), s));
    u32* const old = sc.p;
    sc.p = static_cast<u32*>(q);
    sc.words = want;
    if (old) {
      // (a give-up that nobody has read yet stays recorded)
      CK(cudaMemcpyAsync(sc.p + 1, old + 1, sizeof(u32), cudaMemcpyDeviceToDevice, s));
      CK(cudaFreeAsync(old, s));
    }
  }
  return sc.p;
}

// the calling thread's scan scratch on the stream (p null: it has none)
ScanScratch find_scan_scratch(cudaStream_t s)
{
  int dev = 0;
  CK(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> g(g_scan_mu);
  auto& all = scan_scratches();
  auto it = all.find(ScanKey{dev, s, host_thread()});
  return it != all.end() ? it->second : ScanScratch();
}

// every host thread's
std::vector<ScanScratch> stream_scan_scratches(cudaStream_t s)
{
  int dev = 0;
  CK(cudaGetDevice(&dev));
  std::vector<ScanScratch> v;
  std::lock_guard<std::mutex> g(g_scan_mu);
  auto& all = scan_scratches();
  for (auto it = all.lower_bound(ScanKey{dev, s, 0}); it != all.end() &&
       std::get<0>(it->first) == dev && std::get<1>(it->first) == s; ++it)
    if (it->second.p) v.push_back(it->second);
  return v;
}

// a scan of the stream gave up: its scratch made anew, and the failure
[[noreturn]] void scan_gave_up(ScanScratch const& sc, cudaStream_t s)
{
  CK(cudaMemsetAsync(sc.p, 0, sc.words * sizeof(u32), s));
  throw Failure(E_TIMEOUT, "a bounded device wait gave up (scan look-back)");
}
}  // namespace

namespace {
// Scratch kept between calls, one per stream, host thread and key (what it
// holds); see stream_zero_scratch and stream_marks
struct KeptScratch {
  u32* p = nullptr;
  size_t words = 0;
  u32 gen = 0;
};
std::mutex g_kept_mu;
using KeptKey = std::tuple<int, cudaStream_t, u32, u32>;  // the last two: host thread, key
std::map<KeptKey, KeptScratch>& kept_scratches()
{
  static auto* m = new std::map<KeptKey, KeptScratch>();
  return *m;
}

// at least `words` words for (this device, s, this thread, key), zeroed when
// (re)made
KeptScratch& kept_scratch(u32 key, size_t words, cudaStream_t s)
{
  int dev = 0;
  CK(cudaGetDevice(&dev));
  auto& all = kept_scratches();
  KeptScratch& sc = all[KeptKey{dev, s, host_thread(), key}];
  if (sc.words < words) {
    size_t want = std::max(words + words / 4, (size_t)4096);
    // (the old one stays in place until there is a new one)
    void* q = pool_alloc(want * sizeof(u32), s);
    CK(cudaMemsetAsync(q, 0, want * sizeof(u32), s));
    u32* const old = sc.p;
    sc.p = static_cast<u32*>(q);
    sc.words = want;
    sc.gen = 0;
    if (old) CK(cudaFreeAsync(old, s));
  }
  return sc;
}
}  // namespace

u32 resident_blocks_of(void const* kernel, u32 block, size_t smem)
{
  static std::mutex mu;
  static auto* cache = new std::map<std::tuple<void const*, u32, size_t, int>, u32>();
  int dev = 0;
  CK(cudaGetDevice(&dev));
  auto const key = std::make_tuple(kernel, block, smem, dev);
  std::lock_guard<std::mutex> g(mu);
  auto it = cache->find(key);
  if (it != cache->end()) return it->second;
  int per_sm = 0, sms = 0;
  CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, (int)block, smem));
  CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  u32 const n = (u32)std::max(1, per_sm) * (u32)std::max(1, sms);
  (*cache)[key] = n;
  return n;
}

void release_stream_scratch(cudaStream_t s)
{
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return;
  for (auto const& b : blocks().drop(dev, s)) cudaFreeAsync(b.p, s);
  {
    std::lock_guard<std::mutex> g(g_scan_mu);
    auto& all = scan_scratches();
    for (auto it = all.lower_bound(ScanKey{dev, s, 0}); it != all.end() &&
         std::get<0>(it->first) == dev && std::get<1>(it->first) == s;) {
      if (it->second.p) cudaFreeAsync(it->second.p, s);
      it = all.erase(it);
    }
  }
  std::lock_guard<std::mutex> g(g_kept_mu);
  auto& all = kept_scratches();
  for (auto it = all.lower_bound(KeptKey{dev, s, 0, 0}); it != all.end() &&
       std::get<0>(it->first) == dev && std::get<1>(it->first) == s;) {
    if (it->second.p) cudaFreeAsync(it->second.p, s);
    it = all.erase(it);
  }
}

u32* stream_zero_scratch(u32 key, size_t words, cudaStream_t s)
{
  std::lock_guard<std::mutex> g(g_kept_mu);
  return kept_scratch(key, words, s).p;
}

u32* stream_marks(u32 key, size_t words, cudaStream_t s, u32* gen)
{
  std::lock_guard<std::mutex> g(g_kept_mu);
  KeptScratch& sc = kept_scratch(key, words, s);
  if (++sc.gen == 0) {  // wrapped: no stamp of old may pass for the new one
    CK(cudaMemsetAsync(sc.p, 0, sc.words * sizeof(u32), s));
    sc.gen = 1;
  }
  *gen = sc.gen;
  return sc.p;
}

namespace {
// tiles of a job (one at least: an empty scan still writes out[0] = 0)
u32 job_tiles(u32 n, u32 tile) { return n ? ceil_div(n, (u64)tile) : 1u; }

// a tile's shape: threads (256 or 512) x items per thread (8 or 16, or 32)
struct ScanShape {
  u32 threads, items;
  u32 tile() const { return threads * items; }
};
ScanShape tuned_scan_shape() { return {tuned(TK_SCAN_THREADS), tuned(TK_SCAN_ITEMS)}; }
// A long scan is bound by its tiles' waits on one another rather than by its
// bytes. 256 threads of 32 items have the tile of 512 of 16, 8192 items, but
// three of them fit an SM where two of the others do (28M items: 66 us with
// 512 x 16, 53 with 256 x 32; 6M: 15.5 and 13.6). Below LONG_SCAN items the
// two are level (4.0M: 12.2 both) and the tuning table's shape is taken.
constexpr u64 LONG_SCAN = 4u << 20;
ScanShape scan_shape_for(u64 items)
{
  ScanShape const sh = tuned_scan_shape();
  return items >= LONG_SCAN && sh.items == 16 ? ScanShape{256, 32} : sh;
}

void launch_scan_jobs(ScanJobs const& jobs, ScanShape sh, u32* scratch, u32 spin_limit,
    cudaStream_t s)
{
  u32 const ntiles = jobs.tile0[jobs.njobs];
  auto k = sh.items == 32   ? k_exscan<256, 32>
           : sh.threads == 256 ? (sh.items == 8 ? k_exscan<256, 8> : k_exscan<256, 16>)
                             : (sh.items == 8 ? k_exscan<512, 8> : k_exscan<512, 16>);
  CK(launch_kernel(k, dim3(ntiles), dim3(sh.threads), 0, s, jobs,
      reinterpret_cast<unsigned long long*>(scratch + 4), scratch, spin_limit));
  CK_LAUNCH();
}
}  // namespace

static std::atomic<u32> g_report_scan{0};
void selftest_scan_report(u32 nth) { g_report_scan.store(nth); }

void exscan_jobs(ScanJob const* jobs, u32 njobs, cudaStream_t s)
{
  for (u32 at = 0; at < njobs; at += MAX_SCAN_JOBS) {
    ScanJobs pack;
    pack.njobs = std::min<u32>(MAX_SCAN_JOBS, njobs - at);
    u64 total = 0;
    for (u32 q = 0; q < pack.njobs; ++q) total += jobs[at + q].n;
    ScanShape const sh = scan_shape_for(total);
    u32 const tile = sh.tile();
    pack.tile0[0] = 0;
    double bytes = 0;
    for (u32 q = 0; q < pack.njobs; ++q) {
      pack.j[q] = jobs[at + q];
      pack.tile0[q + 1] = pack.tile0[q] + job_tiles(pack.j[q].n, tile);
      bytes += 8.0 * pack.j[q].n + 4.0 + (pack.j[q].newid ? 4.0 * pack.j[q].n : 0.0) +
          (pack.j[q].comp ? 4.0 * pack.j[q].n : 0.0) + (pack.j[q].comp_newid ? 4.0 * pack.j[q].n : 0.0);
    }
    // [ticket, error, done, pad][status per tile], zero on entry
    u32* scratch = stream_scan_scratch(4 + 2 * (size_t)pack.tile0[pack.njobs], s);
    PROBE(P_EXSCAN, s, bytes);
    launch_scan_jobs(pack, sh, scratch, SCAN_SPIN_LIMIT, s);
    u32 left = g_report_scan.load(std::memory_order_relaxed);
    while (left && !g_report_scan.compare_exchange_weak(left, left - 1)) {
    }
    if (left == 1) CK(cudaMemsetAsync(scratch + 1, 1, sizeof(u32), s));
  }
}

void exscan_u32(u32 const* in, u32* out, u32 n, cudaStream_t s, u32* total_to, u32* newid)
{
  ScanJob j{in, out, total_to, newid, n, 0};
  exscan_jobs(&j, 1, s);
}

// The scans of one stream record a look-back that gave up in word 1 of their
// scratch (the last tile clears words 0 and 2 only), so a stream's check sees
// its own scans' timeouts and no other stream's.
void check_device_timeouts(cudaStream_t s)
{
  u32* h = static_cast<u32*>(pinned_scratch());
  for (ScanScratch const& sc : stream_scan_scratches(s)) {
    CK(cudaMemcpyAsync(h, sc.p + 1, sizeof(u32), cudaMemcpyDeviceToHost, s));
    stream_sync(s);
    if (*h) scan_gave_up(sc, s);
  }
}

int selftest_scan_wait(u32 spin_limit)
{
  // Two tiles, the ticket counter starting at 1: the block that takes tile
  // 1 waits for tile 0, which no block takes, until spin_limit polls have
  // gone by; the block that takes ticket 2 has no tile and returns.
  cudaStream_t s = nullptr;
  CK(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
  u32 const n = 2 * 512 * 16, ntiles = 2;
  size_t words = (size_t)(n + 1) * 2 + 4 + 2 * ntiles + 4;  // + alignment room
  u32* buf = nullptr;
  CK(cudaMalloc(&buf, words * sizeof(u32)));
  u32* in = buf;
  u32* out = buf + n + 1;
  u32* scratch = buf + 2 * (size_t)(n + 1);
  scratch += (4 - (reinterpret_cast<uintptr_t>(scratch) / 4) % 4) % 4;  // 16-byte aligned
  CK(cudaMemsetAsync(buf, 0, words * sizeof(u32), s));
  u32 one = 1;
  CK(cudaMemcpyAsync(scratch, &one, sizeof(u32), cudaMemcpyHostToDevice, s));
  ScanJobs pack;
  pack.njobs = 1;
  pack.tile0[0] = 0;
  pack.tile0[1] = ntiles;
  pack.j[0] = ScanJob{in, out, nullptr, nullptr, n, 0};
  launch_scan_jobs(pack, ScanShape{512, 16}, scratch, spin_limit, s);
  u32 err = 0;
  CK(cudaMemcpyAsync(&err, scratch + 1, sizeof(u32), cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  CK(cudaFree(buf));
  CK(cudaStreamDestroy(s));
  return err ? E_TIMEOUT : E_OK;
}

size_t exscan_scratch_words(u32 n)
{
  return 4 + 2 * (size_t)ceil_div(n ? n : 1, SCAN_MIN_TILE);
}

void exscan_u32_scratch(u32 const* in, u32* out, u32 n, u32* scratch, cudaStream_t s)
{
  if (reinterpret_cast<uintptr_t>(scratch) % 16 != 0)
    throw Failure(E_ARG, "scan scratch must start on a 16-byte boundary");
  ScanShape const sh = tuned_scan_shape();
  CK(cudaMemsetAsync(scratch, 0, exscan_scratch_words(n) * sizeof(u32), s));
  ScanJobs pack;
  pack.njobs = 1;
  pack.tile0[0] = 0;
  pack.tile0[1] = job_tiles(n, sh.tile());
  pack.j[0] = ScanJob{in, out, nullptr, nullptr, n, 0};
  launch_scan_jobs(pack, sh, scratch, SCAN_SPIN_LIMIT, s);
}

u32* exscan_new(u32 const* in, u32 n, cudaStream_t s, u32* total_to, u32* newid)
{
  u32* out = dalloc<u32>((size_t)n + 1, s);
  exscan_u32(in, out, n, s, total_to, newid);
  return out;
}

u32* negate_offsets(u32 const* offs, u32 n, cudaStream_t s, u32* total_to, u32* newid)
{
  u32* o = dalloc<u32>((size_t)n + 1, s);
  ScanJob j{offs, o, total_to, newid, n, 1};
  exscan_jobs(&j, 1, s);
  return o;
}

__global__ void k_fill(u32* a, u32 n, u32 v)
{
  pdl_wait();
  u32 i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) a[i] = v;
}

void fill_u32(u32* a, u32 n, u32 v, cudaStream_t s)
{
  if (!n) return;
  CK(launch_kernel(k_fill, dim3(grid_for(n)), dim3(BLOCK), 0, s, a, n, v));
  CK_LAUNCH();
}

struct CopyJobs {
  CopyJob j[MAX_COPY_JOBS];
};

// blockIdx.y: the job. 16-byte words, COPY_UNROLL to a thread with their
// loads issued together (bound by DRAM); the bytes past the last word, and
// arrays that do not start on 16 bytes, one at a time.
constexpr u32 COPY_UNROLL = 4;

__global__ void __launch_bounds__(BLOCK) k_copy_many(const __grid_constant__ CopyJobs jobs)
{
  pdl_wait();
  CopyJob const jb = jobs.j[blockIdx.y];
  size_t const t0 = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  size_t const stride = (size_t)gridDim.x * blockDim.x;
  bool const wide = ((reinterpret_cast<uintptr_t>(jb.src) | reinterpret_cast<uintptr_t>(jb.dst)) & 15) == 0;
  size_t const nw = wide ? jb.bytes / 16 : 0;
  uint4 const* __restrict__ src = static_cast<uint4 const*>(jb.src);
  uint4* __restrict__ dst = static_cast<uint4*>(jb.dst);
  for (size_t t = t0; t < nw; t += stride * COPY_UNROLL) {
    uint4 v[COPY_UNROLL];
#pragma unroll
    for (u32 k = 0; k < COPY_UNROLL; ++k)
      if (t + k * stride < nw) v[k] = src[t + k * stride];
#pragma unroll
    for (u32 k = 0; k < COPY_UNROLL; ++k)
      if (t + k * stride < nw) dst[t + k * stride] = v[k];
  }
  for (size_t b = nw * 16 + t0; b < jb.bytes; b += stride)
    static_cast<unsigned char*>(jb.dst)[b] = static_cast<unsigned char const*>(jb.src)[b];
}

void copy_many(CopyJob const* jobs, size_t njobs, cudaStream_t s)
{
  for (size_t at = 0; at < njobs;) {
    CopyJobs pack;
    u32 cnt = 0;
    size_t most = 0;
    for (; at < njobs && cnt < MAX_COPY_JOBS; ++at) {
      if (!jobs[at].bytes) continue;
      pack.j[cnt++] = jobs[at];
      most = std::max(most, jobs[at].bytes);
    }
    if (!cnt) return;
    u32 const gx = (u32)std::min<size_t>(ceil_div(most, 16 * COPY_UNROLL * BLOCK), 148 * 8);
    CK(launch_kernel(k_copy_many, dim3(gx, cnt), dim3(BLOCK), 0, s, pack));
    CK_LAUNCH();
  }
}

__global__ void k_iota(u32* a, u32 n, u32 stride)
{
  pdl_wait();
  u32 i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) a[i] = i * stride;
}

void iota_u32(u32* a, u32 n, u32 stride, cudaStream_t s)
{
  if (!n) return;
  CK(launch_kernel(k_iota, dim3(grid_for(n)), dim3(BLOCK), 0, s, a, n, stride));
  CK_LAUNCH();
}

__global__ void k_iota64(u64* a, u32 n)
{
  pdl_wait();
  u32 i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) a[i] = i;
}

void iota_u64(u64* a, u32 n, cudaStream_t s)
{
  if (!n) return;
  CK(launch_kernel(k_iota64, dim3(grid_for(n)), dim3(BLOCK), 0, s, a, n));
  CK_LAUNCH();
}

template <class T>
__global__ void k_expand(T const* __restrict__ in, u32 const* __restrict__ offs,
    u32 n, u32 width, T* __restrict__ out)
{
  pdl_wait();
  u32 i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  u32 f = offs[i], e = offs[i + 1];
  for (u32 j = f; j < e; ++j)
    for (u32 k = 0; k < width; ++k) out[(size_t)j * width + k] = in[(size_t)i * width + k];
}

void expand_rows(void const* in, u32 const* offs, u32 n, u32 width, u32 esz,
    void* out, cudaStream_t s)
{
  if (!n || !width) return;
  PROBE(P_EXPAND, s, 4.0 * (n + 1) + 2.0 * (double)n * width * esz);
  switch (esz) {
    case 1:
      CK(launch_kernel(k_expand<unsigned char>, dim3(grid_for(n)), dim3(BLOCK), 0, s, 
          (unsigned char const*)in, offs, n, width, (unsigned char*)out));
      break;
    case 4:
      CK(launch_kernel(k_expand<u32>, dim3(grid_for(n)), dim3(BLOCK), 0, s, (u32 const*)in, offs, n, width, (u32*)out));
      break;
    default:
      CK(launch_kernel(k_expand<unsigned long long>, dim3(grid_for(n)), dim3(BLOCK), 0, s, 
          (unsigned long long const*)in, offs, n, width, (unsigned long long*)out));
      break;
  }
  CK_LAUNCH();
}

__global__ void k_max_u32(u32 const* __restrict__ a, u32 n, u32* out)
{
  pdl_wait();
  u32 m = 0;
  for (u32 i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    m = max(m, a[i]);
  for (int o = 16; o; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0 && m) atomicMax(out, m);
}

u32 max_u32(u32 const* a, u32 n, cudaStream_t s)
{
  if (!n) return 0;
  u32* d = dalloc<u32>(1, s);
  CK(cudaMemsetAsync(d, 0, sizeof(u32), s));
  u32 g = grid_for(n);
  if (g > 4096) g = 4096;
  CK(launch_kernel(k_max_u32, dim3(g), dim3(BLOCK), 0, s, a, n, d));
  CK_LAUNCH();
  u32 v = read_u32(d, s);
  dev_free(d, s);
  return v;
}

}  // namespace osh
