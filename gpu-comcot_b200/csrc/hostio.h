/*
 * Field transfers between a caller's ordinary host memory and the device.
 */
#ifndef GC_HOSTIO_H
#define GC_HOSTIO_H

#include "gc_internal.h"

/* nx x ny floats at `h` (contiguous rows) to the pitched device field `d`,
 * in stream order on `s`; they have been read when the call returns, whatever
 * kind of memory `h` is in, device memory included (not on a capturing stream,
 * where the graph reads any but ordinary memory at its launch) */
int gc_field_upload(float *d, size_t pitch_bytes, const float *h, int nx, int ny, cudaStream_t s);
/* the pitched device field `d` after the work queued on `s`, into `h`, in
 * any kind of memory; the data is there when the call returns */
int gc_field_download(void *h, const void *d, size_t pitch_bytes, int nx, int ny, cudaStream_t s);
/* memcpy by several host threads where that is faster */
void gc_copy(void *dst, const void *src, size_t bytes);

#endif
