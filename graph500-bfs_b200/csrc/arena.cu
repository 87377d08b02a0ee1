// Device memory of the engines (DeviceArena, engine.h).  Host code only.
#include <algorithm>
#include <string>
#include "engine.h"

namespace b200bfs {
namespace {

// The arenas of the process that may keep blocks.  Never destroyed: an engine
// may be closed by a static object's destructor.
struct OpenArenas {
  std::mutex mu;
  std::vector<DeviceArena*> list;
};
OpenArenas& open_arenas() {
  static OpenArenas* a = new OpenArenas;
  return *a;
}

}  // namespace

DeviceArena::~DeviceArena() {
  OpenArenas& a = open_arenas();
  std::lock_guard<std::mutex> lock(a.mu);
  a.list.erase(std::remove(a.list.begin(), a.list.end(), this), a.list.end());
}

void DeviceArena::open(int device) {
  device_ = device;
  keep_ = budget_ == 0 && shared_ == nullptr;
  OpenArenas& a = open_arenas();
  std::lock_guard<std::mutex> lock(a.mu);
  if (keep_ && std::find(a.list.begin(), a.list.end(), this) == a.list.end())
    a.list.push_back(this);
}

void* DeviceArena::alloc(size_t bytes, const char* what) {
  if (bytes == 0) bytes = 16;
  // (the lock is not held between the tries: other arenas' are taken there,
  // and the owner frees buffers of this one)
  std::string why;
  bool full = false;
  void* p = try_alloc(bytes, what, &why, &full);
  if (!p && full && others_give_back()) p = try_alloc(bytes, what, &why, &full);
  if (!p && give_up_ && give_up_()) p = try_alloc(bytes, what, &why, &full);
  if (!p) throw Error{B200BFS_ERR_OOM, why};
  return p;
}

// Null: why, and whether the device is full (else a budget).
void* DeviceArena::try_alloc(size_t bytes, const char* what, std::string* why, bool* full) {
  std::lock_guard<std::mutex> lock(mu_);
  if (budget_ && in_use_ + bytes > budget_) {
    *why = std::string("HBM budget exceeded allocating ") + what;
    return nullptr;
  }
  if (shared_) {
    const uint64_t before = shared_->used.fetch_add(bytes);
    if (shared_->limit && before + bytes > shared_->limit) {
      shared_->used.fetch_sub(bytes);
      *why = std::string("shared HBM budget exceeded allocating ") + what;
      return nullptr;
    }
  }
  // a kept block that is at most an eighth too large (small ones: up to twice)
  const size_t most = bytes < (size_t(1) << 20) ? 2 * bytes : bytes + bytes / 8;
  size_t best = kept_.size();
  for (size_t i = 0; i < kept_.size(); ++i)
    if (kept_[i].size >= bytes && kept_[i].size <= most &&
        (best == kept_.size() || kept_[i].size < kept_[best].size))
      best = i;
  if (best < kept_.size()) {
    const Block b = kept_[best];
    kept_.erase(kept_.begin() + (int64_t)best);
    kept_bytes_ -= b.size;
    in_use_ += bytes;
    live_.push_back({b.p, bytes, b.size, seq_++});
    return b.p;
  }
  void* p = nullptr;
  cudaError_t e = cudaMalloc(&p, bytes);
  if (e == cudaErrorMemoryAllocation && !kept_.empty()) {
    cudaGetLastError();
    while (!kept_.empty()) drop_oldest();
    e = cudaMalloc(&p, bytes);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    if (shared_) shared_->used.fetch_sub(bytes);
    *full = true;
    *why = std::string("cudaMalloc failed for ") + what + " (" + std::to_string(bytes) + " bytes)";
    return nullptr;
  }
  in_use_ += bytes;
  live_.push_back({p, bytes, bytes, seq_++});
  return p;
}

// What the other arenas on this device keep goes back; false if they keep nothing.
bool DeviceArena::others_give_back() {
  OpenArenas& a = open_arenas();
  std::lock_guard<std::mutex> lock(a.mu);
  bool any = false;
  for (DeviceArena* x : a.list) {
    if (x == this || x->device_ != device_) continue;
    std::lock_guard<std::mutex> lx(x->mu_);
    any |= !x->kept_.empty();
    while (!x->kept_.empty()) x->drop_oldest();
  }
  return any;
}

void DeviceArena::give(const Block& b) {
  in_use_ -= b.bytes;
  if (shared_) shared_->used.fetch_sub(b.bytes);
  if (!keep_ || b.size > limit_) {
    cudaFree(b.p);
    return;
  }
  kept_.push_back(b);
  kept_bytes_ += b.size;
  while (kept_bytes_ > limit_) drop_oldest();
}

void DeviceArena::drop_oldest() {
  cudaFree(kept_.front().p);
  kept_bytes_ -= kept_.front().size;
  kept_.erase(kept_.begin());
}

// What is kept so far goes back: a build's blocks are of no use afterwards.
void DeviceArena::settle(uint64_t spare) {
  std::lock_guard<std::mutex> lock(mu_);
  limit_ = spare;
  while (!kept_.empty()) drop_oldest();
}

void DeviceArena::free(void* p) {
  if (!p) return;
  std::lock_guard<std::mutex> lock(mu_);
  for (size_t i = 0; i < live_.size(); ++i)
    if (live_[i].p == p) {
      const Block b = live_[i];
      live_[i] = live_.back();
      live_.pop_back();
      give(b);
      return;
    }
}

void DeviceArena::rollback(uint64_t m) {
  std::lock_guard<std::mutex> lock(mu_);
  for (size_t i = 0; i < live_.size();) {
    if (live_[i].seq >= m) {
      const Block b = live_[i];
      live_[i] = live_.back();
      live_.pop_back();
      give(b);
    } else {
      ++i;
    }
  }
}

}  // namespace b200bfs
