// tess_grow.h -- growing a buffer whose contents need not be kept.
#pragma once
#include <algorithm>
#include <cstddef>

namespace tess {

// Makes *p hold at least `need` elements; cap is what it holds.  alloc(p, n)
// returns 0 or an error and then leaves *p null, release(*p) frees and clears it.
// The old buffer goes first, so that the two need not fit side by side.  Half as
// much again is asked for, so that slowly growing requests do not allocate each
// time; where memory is short, just what is needed.
template <typename T, typename Alloc, typename Release>
auto grow_buffer(T** p, size_t& cap, size_t need, Alloc alloc, Release release) -> decltype(alloc(p, need)) {
    using Status = decltype(alloc(p, need));
    if (*p && need <= cap) return Status(0);
    const size_t ample = std::max(need, cap + cap / 2);
    release(*p);
    cap = 0;
    size_t got = ample;
    Status st = alloc(p, ample);
    if (st != Status(0) && ample > need) {
        got = need;
        st = alloc(p, need);
    }
    if (st == Status(0)) cap = got;
    return st;
}

}  // namespace tess
