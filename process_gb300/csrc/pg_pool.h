// Device memory of an engine (included by pg_api.cpp after ck()).
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <map>
#include <vector>

// A small caching pool: freed blocks are kept per engine and reused by size,
// so repeated place/sequence calls do not pay cudaMalloc/cudaFree.  Blocks of
// up to 2 MB are cut from slabs of 128 kB, 512 kB, 4 MB, then 16 MB each: an
// engine with an index takes some 60 of them, at 3 to 10 us for each cudaMalloc
// (from 1 MB on 30 us, whatever the size) and as much again to free them.  (A
// first slab of 2 MB, which no chunk that the driver already has holds, cost a
// small handle beside others 100 us.)  A slab can be given back only when
// none of its blocks is in use, so the slabs take SLABS_MAX together at most; what
// does not fit them (nor a slab the device has no room for) gets an allocation
// of its own.
class Pool {
 public:
  ~Pool() { release_all(); }
  void* get(size_t bytes) {
    if (bytes == 0) bytes = 256;
    bytes = (bytes + 255) & ~size_t(255);
    auto it = free_.lower_bound(bytes);
    if (it != free_.end() && it->first <= 2 * bytes) {
      const Free f = it->second;
      used_[f.p] = {it->first, f.slab};
      if (f.slab != OWN) ++slabs_[f.slab].live;
      free_.erase(it);
      return f.p;
    }
    if (bytes <= SLAB_MAX_BLOCK && room(bytes)) {
      Slab& s = slabs_[cur_];
      void* p = s.p + s.used;
      used_[p] = {bytes, cur_};
      s.used += bytes;
      ++s.live;
      return p;
    }
    void* p = allocate(bytes);
    used_[p] = {bytes, OWN};
    return p;
  }
  void put(void* p) {
    if (!p) return;
    auto it = used_.find(p);
    if (it == used_.end()) return;
    const Block b = it->second;
    free_.emplace(b.size, Free{p, b.slab});
    if (b.slab != OWN) --slabs_[b.slab].live;
    used_.erase(it);
  }
  // gives back every free block, and the slabs none of whose blocks are in use
  void release_free() {
    for (auto it = free_.begin(); it != free_.end();) {
      const Free f = it->second;
      if (f.slab != OWN && slabs_[f.slab].live) { ++it; continue; }
      if (f.slab == OWN) cudaFree(f.p);
      it = free_.erase(it);
    }
    for (Slab& s : slabs_)
      if (!s.live && s.p) { cudaFree(s.p); slab_bytes_ -= s.size; s = Slab(); }
  }
  void release_all() {
    for (auto& kv : free_) if (kv.second.slab == OWN) cudaFree(kv.second.p);
    for (auto& kv : used_) if (kv.second.slab == OWN) cudaFree(kv.first);
    for (Slab& s : slabs_) if (s.p) cudaFree(s.p);
    free_.clear(); used_.clear(); slabs_.clear();
    cur_ = OWN;
    slab_bytes_ = 0;
  }

 private:
  static constexpr uint32_t OWN = 0xffffffffu;             // a block with an allocation of its own
  static constexpr size_t SLAB_MAX_BLOCK = size_t(2) << 20, SLABS_MAX = size_t(64) << 20;
  static constexpr size_t SLAB_SIZE[4] = {size_t(128) << 10, size_t(512) << 10, size_t(4) << 20, size_t(16) << 20};
  struct Slab { char* p = nullptr; size_t size = 0, used = 0; uint32_t live = 0; };
  struct Block { size_t size; uint32_t slab; };
  struct Free { void* p; uint32_t slab; };
  // the current slab has room for a block, perhaps a new one
  bool room(size_t bytes) {
    if (cur_ != OWN && slabs_[cur_].size - slabs_[cur_].used >= bytes) return true;
    Slab s;
    size_t step = std::min<size_t>(slabs_.size(), 3);
    while (SLAB_SIZE[step] < bytes) ++step;
    s.size = SLAB_SIZE[step];
    if (slab_bytes_ + s.size > SLABS_MAX) return false;
    void* p = nullptr;
    if (cudaMalloc(&p, s.size) != cudaSuccess) { cudaGetLastError(); return false; }
    s.p = static_cast<char*>(p);
    slab_bytes_ += s.size;
    slabs_.push_back(s);
    cur_ = uint32_t(slabs_.size() - 1);
    return true;
  }
  void* allocate(size_t bytes) {
    void* p = nullptr;
    if (cudaMalloc(&p, bytes) != cudaSuccess) {
      cudaGetLastError();
      release_free();
      ck(cudaMalloc(&p, bytes), "cudaMalloc");
    }
    return p;
  }
  std::vector<Slab> slabs_;
  size_t slab_bytes_ = 0;
  uint32_t cur_ = OWN;                                     // the slab blocks are cut from
  std::multimap<size_t, Free> free_;
  std::map<void*, Block> used_;
};
