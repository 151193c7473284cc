// pure.h — arithmetic of calls and kernels that needs no GPU, in a header of
// its own so that host tests compile the same lines.
#pragma once

#include <stddef.h>

namespace yas {

// Bytes from the first to the last byte of an image of `rows` rows of
// `row_bytes`, `pitch` bytes apart: the padding behind the last row is not the
// image's, and need not be there.
inline size_t image_bytes(size_t row_bytes, size_t pitch, int rows) { return pitch * (size_t)(rows - 1) + row_bytes; }

}  // namespace yas
