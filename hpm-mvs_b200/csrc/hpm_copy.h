/*
 * Copies between a caller's host memory and the device, for the entry points
 * that take whole maps.
 */
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

struct hpm_ctx;

namespace hpm {

struct CopyItem {
    void *dst;
    const void *src;
    size_t bytes;
};

struct HostCopier; /* a context's pinned buffers, made when its copies are worth them */
void host_copier_free(HostCopier *h);

/* Queues the items on the context's stream; sources may be host (pageable or
 * pinned) or device memory.  Pageable sources have been read on return. */
cudaError_t ctx_copy_in(hpm_ctx *c, const CopyItem *items, int n);
/* The same out of device memory; waits for the stream, so that the
 * destinations hold the data on return. */
cudaError_t ctx_copy_out(hpm_ctx *c, const CopyItem *items, int n);

}  // namespace hpm
