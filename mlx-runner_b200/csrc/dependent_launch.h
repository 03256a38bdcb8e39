// Programmatic dependent launch, as every kernel family of the library uses it: a kernel may become resident before the
// kernels ahead of it in the stream have finished.
#pragma once

#include <cstdlib>

namespace mlxq {

// MLXQ_PDL=0 launches every kernel as an ordinary one: for hosts that rewrite a layer's tensors with kernels of their own in
// the same stream, which the decode kernels read ahead of everything else.
inline bool pdl_enabled() {
    static const bool v = [] { const char* e = std::getenv("MLXQ_PDL"); return !(e && e[0] == '0'); }();
    return v;
}

}  // namespace mlxq
