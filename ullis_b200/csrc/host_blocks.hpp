// The blocks of ullis_cuda_host_alloc: page-locked memory that kernels of any device may write, as long as it is here.
#pragma once
#include <cstddef>
#include <cstdint>
#include <map>
#include <mutex>
#include <new>

namespace ullis {

class HostBlocks {
public:
    // false: no memory for the entry, the block is not here
    bool add(const void* block, size_t bytes) {
        std::lock_guard<std::mutex> held(lock);
        try {
            sizes[reinterpret_cast<uintptr_t>(block)] = bytes;
        } catch (const std::bad_alloc&) {
            return false;
        }
        return true;
    }
    // Before the memory is given back: what lies there next may be ordinary memory.
    void remove(const void* block) {
        std::lock_guard<std::mutex> held(lock);
        sizes.erase(reinterpret_cast<uintptr_t>(block));
    }
    // Whether all of p .. p + bytes lies in one block.
    bool hold(const void* p, size_t bytes) {
        std::lock_guard<std::mutex> held(lock);
        const uintptr_t at = reinterpret_cast<uintptr_t>(p);
        auto it = sizes.upper_bound(at);
        if (it == sizes.begin()) return false;
        --it;
        const size_t before = at - it->first;
        return before <= it->second && bytes <= it->second - before;
    }

private:
    std::mutex lock;
    std::map<uintptr_t, size_t> sizes;
};

}  // namespace ullis
