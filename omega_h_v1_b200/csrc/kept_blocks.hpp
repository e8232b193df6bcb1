// The books of the device blocks kept between allocations (dev_alloc and
// dev_free): which blocks each stream keeps, and which come from the pool by
// which size class. Host code only; the pool itself is the caller's.
//
// Blocks of up to BLOCK_MAX bytes that are freed are kept for the next
// allocation on the same stream, by size class (four to an octave), up to
// KEEP_MAX bytes a stream and KEEP_DEVICE a device: a pass on a small mesh
// makes and drops some forty arrays, and a call into the driver's pool for
// each took longer than its kernels (0.6 to 1.9 us a call, 735 calls in a 6^3
// adapt of 188 launches). Order is the stream's, as the driver's pool keeps
// it. The blocks go back to that pool when the stream's scratch is released,
// past the limits, and, every stream's of the device, when an allocation
// fails (alloc_or_drop).
#pragma once

#include <cstddef>
#include <cstdint>
#include <iterator>
#include <map>
#include <mutex>
#include <unordered_map>
#include <utility>
#include <vector>

namespace osh {

constexpr size_t BLOCK_MAX = 4u << 20, KEEP_MAX = 256u << 20, KEEP_DEVICE = (size_t)2 << 30;
constexpr uint32_t BLOCK_CLASSES = 1 + 13 * 4;  // 512 bytes; then 2^9 .. 2^22 in quarters

// the class of a block of at most BLOCK_MAX bytes, and the bytes it has
inline uint32_t block_class(size_t bytes, size_t* rounded)
{
  if (bytes <= 512) {
    *rounded = 512;
    return 0;
  }
  uint32_t const l = 63 - (uint32_t)__builtin_clzll((unsigned long long)(bytes - 1));  // >= 9
  size_t const base = (size_t)1 << l, step = base / 4;
  uint32_t const k = (uint32_t)((bytes - 1 - base) / step);
  *rounded = base + (k + 1) * step;
  return 1 + (l - 9) * 4 + k;
}

inline size_t class_bytes(uint32_t c)
{
  if (!c) return 512;
  size_t const base = (size_t)1 << (9 + (c - 1) / 4);
  return base + ((c - 1) % 4 + 1) * (base / 4);
}

class BlockTable {
 public:
  struct Block {
    void* p;
    void* stream;
  };

  // a kept block, or null
  void* take(int dev, void* stream, uint32_t cls)
  {
    std::lock_guard<std::mutex> g(mu);
    auto it = kept.find({dev, stream});
    if (it == kept.end() || it->second.free_of[cls].empty()) return nullptr;
    void* p = it->second.free_of[cls].back();
    it->second.free_of[cls].pop_back();
    it->second.bytes -= class_bytes(cls);
    dev_bytes[dev] -= class_bytes(cls);
    return p;
  }

  // p came from the pool as a block of a class
  void made(void* p, int dev, uint32_t cls)
  {
    std::lock_guard<std::mutex> g(mu);
    blocks[p] = {dev, cls};
  }

  // p came from the pool as no block (too large, or under capture)
  void not_a_block(void* p)
  {
    std::lock_guard<std::mutex> g(mu);
    blocks.erase(p);
  }

  // p is freed on a stream: kept (true), or the caller's to give to the pool
  bool keep(void* p, void* stream, bool may_keep)
  {
    std::lock_guard<std::mutex> g(mu);
    auto it = blocks.find(p);
    if (it == blocks.end()) return false;
    int const dev = it->second.first;
    uint32_t const cls = it->second.second;
    size_t const bytes = class_bytes(cls);
    if (may_keep && dev_bytes[dev] + bytes <= KEEP_DEVICE) {
      Stream& k = kept[{dev, stream}];
      if (k.bytes + bytes <= KEEP_MAX) {
        k.free_of[cls].push_back(p);
        k.bytes += bytes;
        dev_bytes[dev] += bytes;
        return true;
      }
    }
    blocks.erase(it);
    return false;
  }

  // every block kept for a stream, or for all streams of a device: the
  // caller's to give to the pool, each on its stream
  std::vector<Block> drop(int dev, void* stream)
  {
    std::vector<Block> out;
    std::lock_guard<std::mutex> g(mu);
    auto it = kept.find({dev, stream});
    if (it != kept.end()) drop(it, out);
    return out;
  }
  std::vector<Block> drop_all(int dev)
  {
    std::vector<Block> out;
    std::lock_guard<std::mutex> g(mu);
    for (auto it = kept.begin(); it != kept.end();)
      it = it->first.first == dev ? drop(it, out) : std::next(it);
    return out;
  }

  size_t kept_bytes(int dev)
  {
    std::lock_guard<std::mutex> g(mu);
    return dev_bytes[dev];
  }

 private:
  struct Stream {
    std::vector<void*> free_of[BLOCK_CLASSES];
    size_t bytes = 0;
  };
  using Kept = std::map<std::pair<int, void*>, Stream>;
  std::mutex mu;
  Kept kept;
  std::unordered_map<void*, std::pair<int, uint32_t>> blocks;  // (device, class) of each
  std::map<int, size_t> dev_bytes;

  Kept::iterator drop(Kept::iterator it, std::vector<Block>& out)
  {
    for (auto const& list : it->second.free_of)
      for (void* p : list) {
        blocks.erase(p);
        out.push_back({p, it->first.second});
      }
    dev_bytes[it->first.first] -= it->second.bytes;
    return kept.erase(it);
  }
};

// An allocation from the pool; where that is out of memory, once more after
// every block kept on the device has gone back to it: the pool's memory is
// free to any stream, a kept block is not. Pool: alloc(bytes, stream), null
// where it failed, with `full` set where memory was what it lacked;
// free(p, stream); and wait(stream) for what was freed on a stream.
template <class Pool>
void* alloc_or_drop(BlockTable& t, Pool& pool, int dev, size_t bytes, void* stream)
{
  void* p = pool.alloc(bytes, stream);
  if (p || !pool.full) return p;
  std::vector<BlockTable::Block> const back = t.drop_all(dev);
  for (auto const& b : back) pool.free(b.p, b.stream);
  for (size_t k = 0; k < back.size(); ++k)  // (a stream's blocks come together)
    if (!k || back[k].stream != back[k - 1].stream) pool.wait(back[k].stream);
  return pool.alloc(bytes, stream);
}

}  // namespace osh
