// When an upload may return before its copy has run.
//
// A copy from pageable memory is staged by the runtime: when the call returns,
// the caller's buffer has been read and may change or go.  That does not hold
// for registered (page-locked or managed) memory, nor on a system whose device
// reads pageable memory itself, where the runtime need not stage.  Api supplies
// unregistered(p) (the CUDA runtime in the library, a fake in the host test).
#ifndef MHD_UPLOAD_H
#define MHD_UPLOAD_H

template <class Api> inline bool upload_source_is_read(const void *src, int device_reads_pageable)
{
    return !device_reads_pageable && Api::unregistered(src);
}

#endif
