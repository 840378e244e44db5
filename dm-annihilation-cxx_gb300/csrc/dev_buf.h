// dev_buf.h -- the context's device buffers, which grow and are kept, over an
// allocator M with
//     void *alloc(size_t)     null when there is no room
//     void release(void *)
//     size_t available()      bytes free
// in a header a host compiler also takes, so what happens near the end of the
// memory is unit-tested on the CPU.
#pragma once
#include <algorithm>
#include <cstddef>

namespace dmann {

struct DevBuf {
    void *p = nullptr;
    size_t bytes = 0;
};

template <class M>
void drop(M &m, DevBuf &b) {
    if (b.p) m.release(b.p);
    b = DevBuf{};
}

// At least `bytes`, with headroom for slowly growing chunks where there is
// room; false leaves b empty.
template <class M>
bool grow(M &m, DevBuf &b, size_t bytes) {
    if (b.bytes >= bytes) return true;
    drop(m, b);
    for (size_t want : {bytes + bytes / 8, bytes})
        if ((b.p = m.alloc(want))) {
            b.bytes = want;
            return true;
        }
    return false;
}

// The same for a buffer that a call cannot do without: what it cannot have
// beside the optional buffers it has in their place.
template <class M, class Optional>
bool grow_required(M &m, DevBuf &b, size_t bytes, const Optional &optional) {
    if (grow(m, b, bytes)) return true;
    for (DevBuf *o : optional) drop(m, *o);
    return grow(m, b, bytes);
}

// An optional buffer of use from `least` bytes on, and of more up to `most`:
// as many of these as a quarter of the free memory holds (`beside` bytes more
// are about to be taken), so that the caller's other work keeps its room.  One
// that is there is kept until a quarter more can be had: the free memory is not
// the same at every call.  Returns the bytes, 0 for fewer than `least`.
template <class M>
size_t grow_share(M &m, DevBuf &b, size_t least, size_t most, size_t beside) {
    if (b.bytes >= most) return b.bytes;
    const size_t room = m.available() + b.bytes;
    const size_t want = std::min(most + most / 8, room > beside ? (room - beside) / 4 : 0);
    const bool usable = b.bytes >= least;
    if (want < least || (usable && want < b.bytes + b.bytes / 4)) return usable ? b.bytes : 0;
    drop(m, b);
    if ((b.p = m.alloc(want))) b.bytes = want;
    return b.bytes;
}

// The plain form's azimuth table of a cap at one Nside, in bytes: 64 MB at most
// (Nside 1448), and none where a context that renders at many Nside would hold
// more than 256 MB of them (`held` so far); its maps compute the azimuths then.
inline size_t trig_cap_bytes(int nside, size_t held) {
    const size_t bytes = 16 * 2 * (size_t)nside * (size_t)(nside - 1);
    return bytes <= ((size_t)64 << 20) && held + bytes <= ((size_t)256 << 20) ? bytes : 0;
}

}  // namespace dmann
