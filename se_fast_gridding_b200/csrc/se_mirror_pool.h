// se_mirror_pool.h -- idle device buffers kept between calls, by device and
// size.  Host bookkeeping only: the caller supplies the allocation and the
// release of a buffer, so that it is tested without a GPU.
#pragma once

#include <cstddef>
#include <iterator>
#include <map>
#include <mutex>

namespace se {

// Device buffers that stand in for the caller's host arrays, or hold scratch,
// during a call.  A call takes them from this pool and gives them back when it
// returns (its work is finished by then), so a caller that passes new host
// arrays on every call -- spectral_ewald() mallocs its grids per solve --
// reuses the same device memory instead of allocating it again.  A buffer is
// handed out on the device it was allocated on only.  Idle buffers of a device
// beyond `limit` bytes are freed, largest first.
//
// Buffers: static int alloc(void** p, size_t bytes) allocates on the current
// device and returns 0 or an error code; static void free(void* p) releases a
// buffer of any device.
template <typename Buffers>
class MirrorPool {
public:
    explicit MirrorPool(size_t limit) : limit_(limit) {}

    // a buffer of at least `bytes` on `device`, the current one
    int acquire(int device, size_t bytes, void** d, size_t* cap)
    {
        {
            std::lock_guard<std::mutex> lock(mu_);
            Idle& idle = idle_[device];
            auto it = idle.buffers.lower_bound(bytes);
            if (it != idle.buffers.end() && it->first <= 2 * bytes) {   // best fit, at most 2x
                *d = it->second;
                *cap = it->first;
                idle.bytes -= it->first;
                idle.buffers.erase(it);
                return 0;
            }
        }
        void* p = nullptr;
        if (const int e = Buffers::alloc(&p, bytes)) return e;
        *d = p;
        *cap = bytes;
        return 0;
    }

    // device and cap as at acquire
    void release(int device, void* d, size_t cap)
    {
        std::lock_guard<std::mutex> lock(mu_);
        Idle& idle = idle_[device];
        idle.buffers.emplace(cap, d);
        idle.bytes += cap;
        while (idle.bytes > limit_ && !idle.buffers.empty()) {
            auto it = std::prev(idle.buffers.end());
            Buffers::free(it->second);
            idle.bytes -= it->first;
            idle.buffers.erase(it);
        }
    }

private:
    struct Idle {
        std::multimap<size_t, void*> buffers;   // capacity -> buffer
        size_t bytes = 0;
    };
    std::mutex mu_;
    std::map<int, Idle> idle_;   // by device
    const size_t limit_;
};

}  // namespace se
