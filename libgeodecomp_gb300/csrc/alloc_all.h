// Device buffers that are made together, on first use: all of them or none.
#ifndef LGD_ALLOC_ALL_H
#define LGD_ALLOC_ALL_H

#include <stddef.h>

#include <vector>

namespace lgd {

struct BufferRequest {
    void **pointer;         // null before, and after a failure
    size_t bytes;
};

// alloc(pointer, bytes) returns 0 or an error, which ends the attempt: what had
// been allocated is released, every pointer is null again, and the error is
// returned.  A caller's "the buffers are there" is any one of its pointers.
template<typename ALLOC, typename RELEASE>
auto allocate_all(const std::vector<BufferRequest>& buffers, ALLOC alloc, RELEASE release) -> decltype(alloc((void **)nullptr, 0))
{
    for (const BufferRequest& b : buffers) {
        const auto error = alloc(b.pointer, b.bytes);
        if (!error) continue;
        *b.pointer = nullptr;
        for (const BufferRequest& done : buffers) {
            if (*done.pointer) release(*done.pointer);
            *done.pointer = nullptr;
        }
        return error;
    }
    return {};
}

}  // namespace lgd

#endif
