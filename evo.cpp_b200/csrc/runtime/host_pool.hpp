// Pinned host memory that results come back through.  Plain C++: the CUDA runtime's calls are handed in.
#pragma once

#include <cstddef>
#include <memory>
#include <mutex>
#include <vector>

namespace evob {

// Shared by the contexts of a model (any thread, any device).  Free blocks stay for the next user, up to kKept of them
// and kKeptBytes; beyond that the one that has been idle longest is given back.
class HostPool {
 public:
  using Allocate = void *(*)(std::size_t);
  using Free = void (*)(void *);
  static constexpr std::size_t kLargest = std::size_t{64} << 20, kSmallest = std::size_t{64} << 10;
  static constexpr std::size_t kKept = 16, kKeptBytes = 4 * kLargest;
  static constexpr std::size_t kSlabBytes = std::size_t{256} << 10;
  static constexpr std::size_t kWaste = 8;  // a block serves what takes an eighth of it or more

  // Nothing above `largest` bytes is pinned.
  HostPool(Allocate allocate, Free free, std::size_t largest = kLargest);
  HostPool(const HostPool &) = delete;
  HostPool &operator=(const HostPool &) = delete;
  ~HostPool();
  // Up to `count` small blocks of `bytes` from one allocation, which lasts as long as the pool: an allocation takes 2 ms
  // and more whatever its size, a context is made in as much.  Once, before the pool is shared; no memory, no blocks.
  void reserve(std::size_t bytes, std::size_t count);
  void *take(std::size_t bytes, std::size_t *capacity);  // nullptr: not to be had
  void give(void *block, std::size_t capacity) noexcept;

 private:
  struct Block {
    void *data;
    std::size_t capacity;
  };
  const Allocate allocate_;
  const Free free_memory_;
  const std::size_t largest_;
  void *slab_ = nullptr;
  std::size_t small_bytes_ = 0;
  std::vector<void *> small_;  // free blocks of the slab, small_bytes_ each (no other block has this capacity)
  std::mutex mutex_;
  std::vector<Block> idle_;  // in the order in which they came back
  std::size_t idle_bytes_ = 0;
};

// Rows of F32 results on the host: a pool's block until the next use or the end of the object, or memory of its own.
class HostRows {
 public:
  HostRows() = default;
  HostRows(const HostRows &) = delete;
  HostRows &operator=(const HostRows &) = delete;
  ~HostRows() { release(); }
  // Room for `count` values, pinned if the pool has it.
  void resize(const std::shared_ptr<HostPool> &pool, std::size_t count);
  void assign(const float *values, std::size_t count);
  bool pinned() const { return block_ != nullptr; }
  float *data() { return block_ != nullptr ? static_cast<float *>(block_) : own_.data(); }
  const float *data() const { return block_ != nullptr ? static_cast<const float *>(block_) : own_.data(); }
  std::size_t size() const { return count_; }

 private:
  void release() noexcept;
  std::shared_ptr<HostPool> pool_;
  void *block_ = nullptr;
  std::size_t capacity_ = 0, count_ = 0;
  std::vector<float> own_;
};

}  // namespace evob
