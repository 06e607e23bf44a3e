// The host's decisions between paths, apart from the launches they decide on:
// plain C++, so that a host build can hold them to every case.
#pragma once

#include <stddef.h>
#include <stdint.h>

namespace phx {

// Whether a kernel may read or write `p` by 16-byte words.
inline bool aligned16(const void* p) { return ((uintptr_t)p & 15u) == 0u; }

}  // namespace phx
