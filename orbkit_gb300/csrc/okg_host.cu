// Page-locked host memory for results, and their read-back.
#include "okg_internal.cuh"

using namespace okg;

extern "C" int okg_host_alloc(size_t bytes, void** out)
{
    if (!bytes || !out) return set_error(OKG_ERR_ARG, "okg_host_alloc: bad argument");
    const RelaxedCapture guard;
    return cuda_status(cudaHostAlloc(out, bytes, cudaHostAllocPortable), "okg_host_alloc");
}

extern "C" int okg_host_free(void* p)
{
    const RelaxedCapture guard;
    return p ? cuda_status(cudaFreeHost(p), "okg_host_free") : OKG_OK;
}

extern "C" int okg_read_rows(void* h_dst, size_t pitch, const void* d_src, size_t width, size_t rows, okg_stream stream)
{
    if (!h_dst || !d_src || width > pitch) return set_error(OKG_ERR_ARG, "okg_read_rows: bad argument");
    if (!width || !rows) return OKG_OK;
    cudaStream_t st = (cudaStream_t)stream;
    return cuda_status(width == pitch || rows == 1
                           ? cudaMemcpyAsync(h_dst, d_src, width * rows, cudaMemcpyDeviceToHost, st)
                           : cudaMemcpy2DAsync(h_dst, pitch, d_src, width, width, rows, cudaMemcpyDeviceToHost, st),
                       "okg_read_rows");
}
