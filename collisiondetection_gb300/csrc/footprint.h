// The server's estimate of a request's device memory.
#pragma once

#include <stdint.h>

namespace ccd {

// Estimated device bytes of one request: topology and positions, broad-phase
// buffers (slabs of faces and vertices, tree, Morton keys, about 8 candidate
// face pairs per face and their stencil keys) and the narrow-phase rows and
// refinement scratch of its candidate stencils.
inline int64_t request_footprint(int64_t nfaces, int64_t nverts) {
  // 26 doubles for each vertex that faces use, of at most two a face
  const int64_t slabs = nverts < 2 * nfaces ? nverts : 2 * nfaces;
  return 4096 * nfaces + 64 * nverts + 208 * slabs + ((int64_t)64 << 20);
}

}  // namespace ccd
