// Host-side copies between a caller's pageable arrays and pinned staging, shared out over a few helper threads.
#pragma once
#include <cstddef>
#include <functional>
#include <memory>

namespace kn {

// Copies of at least this many bytes are worth waking the helpers for (a wake costs some 10 us; one thread moves
// 18 bytes per nanosecond on the B200 hosts, so 256 KB are 14 us).
constexpr size_t kParallelCopyBytes = 256 << 10;

class CopyPool {
   public:
    // The process's pool: started by the first caller, its threads ended when the last holder lets go.
    static std::shared_ptr<CopyPool> shared();
    virtual ~CopyPool() = default;
    // Copies `bytes` bytes, with stores past the caches for a destination that the GPU reads next (not for one that the
    // caller does).  `ready(from, to)`, if given, is called on the calling thread for consecutive ranges as they
    // are complete, so that an upload of the first part runs while the rest is still being copied.  Returns when
    // everything is copied.  Safe from several threads: a caller that finds the helpers taken copies alone.
    virtual void copy(void* dst, const void* src, size_t bytes, bool past_caches, const std::function<void(size_t, size_t)>& ready) = 0;
};

}  // namespace kn
