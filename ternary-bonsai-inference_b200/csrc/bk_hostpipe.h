// Bulk transfers between pageable caller memory and the device (bk_hostpipe.cpp).
#pragma once

#include "bk_internal.h"

namespace bk {

struct HostSeg {
    void *host;
    void *dev;
    size_t bytes;
};
// BK_ERR_OOM with the name of who ran out; the message is dropped when there is no memory for it either.
bk_status out_of_memory(bk_ctx *ctx, const char *who) noexcept;

// Transfers of less than this are not worth the hand-over to other threads.
constexpr size_t kHostPipeMin = 256 << 10;

// The ranges, in order, after what is on the stream; returns when the bytes are in host memory (and checks the
// context's error word).
bk_status host_pipe_d2h(bk_ctx *ctx, const HostSeg *segs, size_t n_seg);
// The ranges, in order, on the stream; returns when the caller's memory has been read and the copies are through.
bk_status host_pipe_h2d(bk_ctx *ctx, const HostSeg *segs, size_t n_seg);

}  // namespace bk
