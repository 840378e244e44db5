// A host build of the context's buffer growth (dev_buf.h) over an allocator
// with a fixed amount of memory, for tests/test_dev_buf_cpu.py.
#include "dev_buf.h"

#include <map>
#include <vector>

using namespace dmann;

namespace {
struct Mem {
    size_t size = 0, used = 0, calls = 0, changes = 0, next = 1;
    std::map<void *, size_t> held;
    void *alloc(size_t bytes) {
        calls++;
        if (used + bytes > size) return nullptr;
        void *p = (void *)next++;
        held[p] = bytes;
        used += bytes;
        changes++;
        return p;
    }
    void release(void *p) {
        used -= held.at(p);
        held.erase(p);
        changes++;
    }
    size_t available() { return size - used; }
} mem;
std::vector<DevBuf> bufs;
}  // namespace

extern "C" {
void reset(long long size, int n) {
    mem = Mem{};
    mem.size = (size_t)size;
    bufs.assign(n, DevBuf{});
}
int grow_opt(int b, long long bytes) { return grow(mem, bufs[b], (size_t)bytes); }
// every other buffer is optional
int grow_req(int b, long long bytes) {
    std::vector<DevBuf *> opt;
    for (size_t k = 0; k < bufs.size(); k++)
        if ((int)k != b) opt.push_back(&bufs[k]);
    return grow_required(mem, bufs[b], (size_t)bytes, opt);
}
long long share(int b, long long least, long long most, long long beside) {
    return (long long)grow_share(mem, bufs[b], (size_t)least, (size_t)most, (size_t)beside);
}
void free_buf(int b) { drop(mem, bufs[b]); }
long long held(int b) { return (long long)bufs[b].bytes; }
long long used() { return (long long)mem.used; }
long long changes() { return (long long)mem.changes; }
long long trig_cap(int nside, long long held) { return (long long)trig_cap_bytes(nside, (size_t)held); }
long long calls() { return (long long)mem.calls; }
}
