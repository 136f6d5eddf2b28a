// Arrays of a payload on the host: hundreds of megabytes that are written
// once, from end to end, by a copy from the device or by a loop.  HostArray
// leaves new elements unwritten (std::vector would zero them first) and puts
// arrays of 4 MiB and more on huge pages where the system offers them: the
// page faults of 4 KiB pages cost more than the copies themselves.
#pragma once
#include <sys/mman.h>

#include <cstdlib>
#include <new>
#include <utility>
#include <vector>

namespace nbh {

template <class T>
struct HostAlloc {
    using value_type = T;
    static constexpr size_t kHuge = size_t(2) << 20;
    HostAlloc() = default;
    template <class U>
    HostAlloc(const HostAlloc<U>&) {}
    T* allocate(size_t n) {
        if (n > size_t(-1) / sizeof(T) - kHuge) throw std::bad_alloc();
        const size_t bytes = n * sizeof(T);
        void* p;
        if (bytes < 2 * kHuge) {
            p = std::malloc(bytes ? bytes : 1);
        } else {
            const size_t whole = (bytes + kHuge - 1) / kHuge * kHuge;
            p = std::aligned_alloc(kHuge, whole);
            if (p) madvise(p, whole, MADV_HUGEPAGE);  // a hint: refused where there are none
        }
        if (!p) throw std::bad_alloc();
        return static_cast<T*>(p);
    }
    void deallocate(T* p, size_t) { std::free(p); }
    template <class U>
    void construct(U* p) {
        ::new (static_cast<void*>(p)) U;
    }
    template <class U, class... A>
    void construct(U* p, A&&... a) {
        ::new (static_cast<void*>(p)) U(std::forward<A>(a)...);
    }
    template <class U>
    bool operator==(const HostAlloc<U>&) const {
        return true;
    }
    template <class U>
    bool operator!=(const HostAlloc<U>&) const {
        return false;
    }
};

template <class T>
using HostArray = std::vector<T, HostAlloc<T>>;

}  // namespace nbh
