// fi_shapes.h — block sizes of the register-line kernels (host code only).
#pragma once

namespace fi {

// Threads of a block of about `lines` register lines of th threads each (th a
// power of two): a power of two of at least a warp and at most `most` threads,
// so that it is a whole number of lines of th threads and of any line with
// fewer.  The kernels take blockDim.x / th lines a block and have no thread
// left over: one would work on a line of the next block, beyond the shared
// memory of this one.
inline int line_block(int lines, int th, int most)
{
    int t = th > 32 ? th : 32;
    while (t < lines * th && 2 * t <= most) t *= 2;
    return t;
}

}  // namespace fi
