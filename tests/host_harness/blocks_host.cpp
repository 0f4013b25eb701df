// Host-compiled harness around the register of page-locked blocks (host_blocks.hpp), used only by the CPU tests.  Its memory
// comes from an operator new of its own, which can be told to fail.
#include <cstdlib>

#include "../../ullis_b200/csrc/host_blocks.hpp"

static bool no_memory = false;
void* operator new(size_t n) {
    void* p = no_memory ? nullptr : std::malloc(n);
    if (!p) throw std::bad_alloc();
    return p;
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

static ullis::HostBlocks blocks;
static const void* address(uint64_t p) { return reinterpret_cast<const void*>((uintptr_t)p); }

extern "C" void blocks_no_memory(int fails) { no_memory = fails != 0; }
extern "C" int blocks_add(uint64_t p, uint64_t bytes) { return blocks.add(address(p), bytes); }
extern "C" void blocks_remove(uint64_t p) { blocks.remove(address(p)); }
extern "C" int blocks_hold(uint64_t p, uint64_t bytes) { return blocks.hold(address(p), bytes); }
