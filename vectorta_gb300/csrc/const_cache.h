// Where a context's small constant arrays (period lists, per-combo constants)
// lie in its constant buffer.  The buffer is filled front to back; an upload
// whose bytes match an earlier one (hash, then a full compare with the host
// copy) takes its place.  A full buffer starts over, but never under a call
// that already holds a place in it: the call's kernels are enqueued after its
// uploads, so an upload over that place would change what they read.  Such a
// call's uploads get no place, and the next call starts over.  (Kernels of
// earlier calls are ahead of the uploads in the stream.)  Host code only.
#pragma once

#include <cstddef>
#include <cstdint>
#include <cstring>
#include <vector>

namespace vta {

class ConstCache {
   public:
    void init(size_t bytes) { host_.resize(bytes); }

    // A new call: the places handed out before are no longer needed.
    void begin_call() {
        held_ = false;
        if (full_) start_over();
    }

    // The place of an earlier upload of the same bytes.
    bool find(const void* src, size_t bytes, size_t* off) {
        const uint64_t h = hash(src, bytes);
        for (const Entry& e : entries_)
            if (e.hash == h && e.bytes == bytes && std::memcmp(host_.data() + e.off, src, bytes) == 0) {
                *off = e.off;
                held_ = true;
                return true;
            }
        return false;
    }

    // A new place; false: none in this call.
    bool place(const void* src, size_t bytes, size_t* off) {
        const size_t need = (bytes + 255) & ~size_t(255);
        if (need > host_.size()) return false;
        if (used_ + need > host_.size()) {
            if (held_) {
                full_ = true;
                return false;
            }
            start_over();
        }
        std::memcpy(host_.data() + used_, src, bytes);
        *off = used_;
        used_ += need;
        held_ = true;
        return true;
    }

    // The upload to a new place is enqueued: later calls may find it.
    void keep(size_t off, size_t bytes) { entries_.push_back({hash(host_.data() + off, bytes), off, bytes}); }

   private:
    struct Entry {
        uint64_t hash;
        size_t off, bytes;
    };
    static uint64_t hash(const void* src, size_t n) {
        const unsigned char* b = static_cast<const unsigned char*>(src);
        uint64_t h = 0x9E3779B97F4A7C15ull ^ n;
        size_t i = 0;
        for (; i + 8 <= n; i += 8) {
            uint64_t w;
            std::memcpy(&w, b + i, 8);
            h = (h ^ w) * 0xff51afd7ed558ccdull;
            h ^= h >> 32;
        }
        for (; i < n; ++i) h = (h ^ b[i]) * 0x100000001b3ull;
        return h;
    }
    void start_over() {
        entries_.clear();
        used_ = 0;
        full_ = false;
    }

    std::vector<unsigned char> host_;  // host copy of the buffer
    std::vector<Entry> entries_;
    size_t used_ = 0;
    bool held_ = false;  // this call has a place
    bool full_ = false;  // an upload of this call did not fit
};

}  // namespace vta
