// hs_grow.h -- a buffer that its owner keeps and that grows on demand.
#pragma once
#include <cstddef>

namespace hs {

// Mem::get(void**, bytes) and Mem::put(void*) take and give back the memory;
// Mem::ok is get's value on success.
template <class T, class Mem>
struct GrowBuf {
    T* p = nullptr;
    size_t n = 0;
    GrowBuf() = default;
    GrowBuf(const GrowBuf&) = delete;
    GrowBuf& operator=(const GrowBuf&) = delete;
    // room for count elements (contents are not kept); where there is no memory
    // for more, the buffer stays as it was
    auto need(size_t count) -> decltype(Mem::ok) {
        if (count <= n) return Mem::ok;
        void* q = nullptr;
        const auto e = Mem::get(&q, count * sizeof(T));
        if (e != Mem::ok) return e;
        if (p) Mem::put(p);
        p = static_cast<T*>(q);
        n = count;
        return e;
    }
    ~GrowBuf() { if (p) Mem::put(p); }
};

}  // namespace hs
