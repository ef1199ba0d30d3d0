// Device work memory that a finished call leaves for the next one.  Host-only
// (no CUDA: the two calls that reach the device are passed in), so that the rules
// can be tested without a GPU.
//
// Allocating and freeing some GB takes 5-250 ms of host time, varying from call
// to call, against 45 ms for the gradient over 64 steps of 256 x 128 x 128.  So a
// gradient that succeeds leaves its blocks in one list per process, where the
// next one of any handle on the device finds them.  The list is bounded, and
// nobody runs out of memory for its sake:
//   - a call keeps at most a given number of bytes, and what the list holds on
//     the device stays within it (older blocks go first);
//   - an allocation of any handle that fails frees the list's blocks on its
//     device and tries again;
//   - a call that fails frees every block it had;
//   - the blocks a handle's last call left go with the handle, and a release call
//     frees them all (for allocators outside the library).
// Blocks in the list are idle: the call that left them had synchronised.
#pragma once

#include <cstddef>
#include <cstdint>
#include <mutex>

namespace bfx {

struct DeviceMemory {
    int (*allocate)(void** p, size_t n);  // 0, or the device's status
    void (*release)(void* p);
    int out_of_memory;                    // the status of an allocation that does not fit
};

class WorkPool {
  public:
    struct Block {
        void* p;
        size_t bytes;
        int device;
        const void* owner;  // the handle whose call left it
    };
    static constexpr int kMaxBlocks = 64;

    explicit constexpr WorkPool(const DeviceMemory& memory) : memory_(memory) {}
    WorkPool(const WorkPool&) = delete;
    WorkPool& operator=(const WorkPool&) = delete;

    // Allocates n bytes on the (current) device, at the list's cost if need be.
    int allocate(int device, void** p, size_t n) {
        int status = memory_.allocate(p, n);
        if (status == memory_.out_of_memory && drain(device) > 0) status = memory_.allocate(p, n);
        return status;
    }
    void release(void* p) { memory_.release(p); }

    // Takes the smallest block of the device that holds n without wasting a
    // quarter of it out of the list.
    bool take(int device, size_t n, Block* out) {
        std::lock_guard<std::mutex> lock(mutex_);
        int best = -1;
        for (int i = 0; i < count_; ++i)
            if (kept_[i].device == device && kept_[i].bytes >= n && kept_[i].bytes <= n + n / 4 + 4096 &&
                (best < 0 || kept_[i].bytes < kept_[best].bytes))
                best = i;
        if (best < 0) return false;
        *out = kept_[best];
        remove(best);
        return true;
    }

    // Leaves the idle blocks of a finished call in the list, as far as `limit`
    // bytes go.  Freed instead: what is beyond it, the blocks that earlier calls
    // of the same owner left and this one had no use for, and the oldest others
    // while the device's blocks are more than the limit.
    void keep(int device, const void* owner, const Block* blocks, int n, size_t limit) {
        void* freed[2 * kMaxBlocks];
        int nfreed = 0;
        {
            std::lock_guard<std::mutex> lock(mutex_);
            for (int i = count_; i-- > 0;)
                if (kept_[i].owner == owner) freed[nfreed++] = remove(i);
            size_t kept = 0;
            for (int i = 0; i < n && i < kMaxBlocks; ++i) {
                if (blocks[i].bytes > limit - kept) {
                    freed[nfreed++] = blocks[i].p;
                    continue;
                }
                kept += blocks[i].bytes;
                int old;
                while ((old = oldest(device)) >= 0 && bytes_on(device) > limit - blocks[i].bytes)
                    freed[nfreed++] = remove(old);
                if (count_ == kMaxBlocks) freed[nfreed++] = remove(0);
                kept_[count_++] = Block{blocks[i].p, blocks[i].bytes, device, owner};
            }
        }
        for (int i = 0; i < nfreed; ++i) memory_.release(freed[i]);
    }

    // Frees the list's blocks on a device; returns their bytes.
    size_t drain(int device) {
        return free_where([device](const Block& b) { return b.device == device; });
    }
    // Frees what the owner's last call left.
    size_t drop(const void* owner) {
        return free_where([owner](const Block& b) { return b.owner == owner; });
    }
    // Bytes that the owner's last call left.
    size_t held(const void* owner) {
        std::lock_guard<std::mutex> lock(mutex_);
        size_t n = 0;
        for (int i = 0; i < count_; ++i)
            if (kept_[i].owner == owner) n += kept_[i].bytes;
        return n;
    }

  private:
    // (with the lock held; the list is in the order of age)
    void* remove(int i) {
        void* p = kept_[i].p;
        for (--count_; i < count_; ++i) kept_[i] = kept_[i + 1];
        return p;
    }
    int oldest(int device) const {
        for (int i = 0; i < count_; ++i)
            if (kept_[i].device == device) return i;
        return -1;
    }
    size_t bytes_on(int device) const {
        size_t n = 0;
        for (int i = 0; i < count_; ++i)
            if (kept_[i].device == device) n += kept_[i].bytes;
        return n;
    }
    // Releases outside the lock: freeing device memory can wait for the device.
    template <class F>
    size_t free_where(F match) {
        size_t bytes = 0;
        for (;;) {
            void* p = nullptr;
            {
                std::lock_guard<std::mutex> lock(mutex_);
                for (int i = 0; i < count_ && !p; ++i)
                    if (match(kept_[i])) {
                        bytes += kept_[i].bytes;
                        p = remove(i);
                    }
            }
            if (!p) return bytes;
            memory_.release(p);
        }
    }

    const DeviceMemory memory_;
    std::mutex mutex_;
    Block kept_[kMaxBlocks] = {};
    int count_ = 0;
};

// The work memory of one call: blocks from the list or newly allocated, all of
// them freed at its end unless keep() was called first.
class WorkCall {
  public:
    WorkCall(WorkPool& pool, int device, const void* owner) : pool_(pool), device_(device), owner_(owner) {}
    WorkCall(const WorkCall&) = delete;
    WorkCall& operator=(const WorkCall&) = delete;
    ~WorkCall() {
        for (int i = 0; i < count_; ++i) pool_.release(used_[i].p);
    }
    static constexpr int kTooManyBlocks = -1;
    template <class T>
    int get(T** p, size_t n) {
        if (n == 0) n = 16;
        if (count_ == WorkPool::kMaxBlocks) return kTooManyBlocks;
        WorkPool::Block b{};
        if (!pool_.take(device_, n, &b)) {
            const int status = pool_.allocate(device_, &b.p, n);
            if (status != 0) return status;
            b.bytes = n;
            allocated_ = true;
        }
        used_[count_++] = b;
        *p = (T*)b.p;
        bytes_ += n;
        return 0;
    }
    // The call succeeded and nothing uses its blocks any more.
    void keep(size_t limit) {
        pool_.keep(device_, owner_, used_, count_, limit);
        count_ = 0;
    }
    uint64_t bytes() const { return bytes_; }
    // Some of the blocks are new, not from the list.
    bool allocated() const { return allocated_; }

  private:
    WorkPool& pool_;
    const int device_;
    const void* owner_;
    WorkPool::Block used_[WorkPool::kMaxBlocks] = {};
    int count_ = 0;
    uint64_t bytes_ = 0;
    bool allocated_ = false;
};

}  // namespace bfx
