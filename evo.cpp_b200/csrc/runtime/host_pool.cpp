#include "host_pool.hpp"

#include <algorithm>

namespace evob {

HostPool::HostPool(const Allocate allocate, const Free free, const std::size_t largest)
    : allocate_(allocate), free_memory_(free), largest_(std::min(largest, kLargest)) {
  idle_.reserve(kKept + 1);  // giving back never allocates
}

HostPool::~HostPool() {
  for (const Block &b : idle_) free_memory_(b.data);
  if (slab_ != nullptr) free_memory_(slab_);
}

void HostPool::reserve(const std::size_t bytes, const std::size_t count) {
  const std::size_t rounded = (bytes + 255) / 256 * 256, fitting = std::min(count, kSlabBytes / rounded);
  if (slab_ != nullptr || fitting == 0 || rounded >= kSmallest || bytes > largest_) return;
  small_.reserve(fitting);  // giving back never allocates
  slab_ = allocate_(fitting * rounded);
  if (slab_ == nullptr) return;
  small_bytes_ = rounded;
  for (std::size_t i = 0; i < fitting; ++i) small_.push_back(static_cast<unsigned char *>(slab_) + i * rounded);
}

void *HostPool::take(const std::size_t bytes, std::size_t *const capacity) {
  if (bytes > largest_) return nullptr;
  std::size_t wanted = kSmallest;
  while (wanted < bytes) wanted *= 2;  // few sizes, so that blocks find their next user
  {
    const std::lock_guard<std::mutex> lock(mutex_);
    if (bytes <= small_bytes_ && !small_.empty()) {
      void *const found = small_.back();
      small_.pop_back();
      *capacity = small_bytes_;
      return found;
    }
    auto best = idle_.end();
    for (auto b = idle_.begin(); b != idle_.end(); ++b)
      if (b->capacity >= bytes && b->capacity <= kWaste * wanted && (best == idle_.end() || b->capacity < best->capacity))
        best = b;
    if (best != idle_.end()) {
      const Block found = *best;
      idle_.erase(best);
      idle_bytes_ -= found.capacity;
      *capacity = found.capacity;
      return found.data;
    }
  }
  void *const data = allocate_(wanted);
  if (data != nullptr) *capacity = wanted;
  return data;
}

void HostPool::give(void *const block, const std::size_t capacity) noexcept {
  Block dropped[kKept + 1];
  std::size_t count = 0;
  {
    const std::lock_guard<std::mutex> lock(mutex_);
    if (slab_ != nullptr && capacity == small_bytes_) {
      small_.push_back(block);
      return;
    }
    idle_.push_back({block, capacity});
    idle_bytes_ += capacity;
    while (idle_.size() > kKept || idle_bytes_ > kKeptBytes) {
      dropped[count++] = idle_.front();
      idle_bytes_ -= idle_.front().capacity;
      idle_.erase(idle_.begin());
    }
  }
  for (std::size_t i = 0; i < count; ++i) free_memory_(dropped[i].data);
}

void HostRows::release() noexcept {
  if (block_ != nullptr) pool_->give(block_, capacity_);
  block_ = nullptr;
  pool_.reset();
}

void HostRows::resize(const std::shared_ptr<HostPool> &pool, const std::size_t count) {
  if (block_ == nullptr || pool_ != pool || capacity_ < count * sizeof(float)) {
    release();
    block_ = pool != nullptr ? pool->take(count * sizeof(float), &capacity_) : nullptr;
    if (block_ != nullptr) pool_ = pool;
  }
  if (block_ == nullptr) own_.resize(count);
  count_ = count;
}

void HostRows::assign(const float *const values, const std::size_t count) {
  release();
  own_.assign(values, values + count);
  count_ = count;
}

}  // namespace evob
