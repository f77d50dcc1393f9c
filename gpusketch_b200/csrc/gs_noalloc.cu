// gs_noalloc.cu - edge-record ingest that allocates nothing.
//
// Some callers cannot allocate device memory: their device memory is owned by another allocator
// (a framework's caching allocator, an embedded runtime that forbids allocation once it has
// started), so every cudaMalloc would step outside the budget they were given.  This entry point
// serves them: the caller passes the records and its own sketch buffer.  A call has at most
// GS_NOALLOC_MAX_EDGES records, which the direct update XORs into the sketches without grouping them by
// vertex (65536 records, V = 8191, and the clearing of its buffer: 119 us grouped, 60 direct), so all that
// is kept in device memory is one file-scope error word.
//
// In host code the name g_noalloc_status is only a host-side stand-in for the word: every call asks the
// runtime for its device address on the current device (cudaGetSymbolAddress, with that device current)
// and hands that address to the kernel.  Resolving it per call costs a few microseconds and stays right
// after cudaDeviceReset, which reloads the module at a new address.  All calls share the one word, so
// calls on the same device that overlap on the GPU (different streams, or different host threads) can see
// one another's errors.  A call waits for its own stream before it returns (it reads the error word back),
// so it cannot be made while that stream is being captured into a CUDA graph.
#include "gs_internal.h"

namespace {

static __device__ uint32_t g_noalloc_status;   // zero between calls

// device address of the error word on the current device, and the device's SM count
gs_status word_for_current_device(uint32_t** out, int* sms) {
  int dev = 0;
  GS_CUDA_TRY(cudaGetDevice(&dev));
  void* p = nullptr;
  GS_CUDA_TRY(cudaGetSymbolAddress(&p, g_noalloc_status));
  int n = 0;
  GS_CUDA_TRY(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev));
  *out = static_cast<uint32_t*>(p);
  *sms = n > 0 ? n : 1;
  return GS_OK;
}

}  // namespace

extern "C" gs_status gs_ingest_pairs_noalloc(uint32_t num_vertices, uint64_t seed, double sketches_factor,
                                             const uint32_t* pairs, uint64_t n, gs_bucket* sketches,
                                             void* cuda_stream) {
  if (num_vertices < 2 || num_vertices > GS_NOALLOC_MAX_VERTICES) {
    gs_set_error("gs_ingest_pairs_noalloc: num_vertices must be in [2, " + std::to_string(GS_NOALLOC_MAX_VERTICES) +
                 "], got " + std::to_string(num_vertices));
    return GS_ERR_BAD_ARG;
  }
  if (n > GS_NOALLOC_MAX_EDGES) {
    gs_set_error("gs_ingest_pairs_noalloc: at most " + std::to_string(GS_NOALLOC_MAX_EDGES) +
                 " edge records per call, got " + std::to_string(n));
    return GS_ERR_BAD_ARG;
  }
  if (!sketches || (n && !pairs)) {
    gs_set_error("gs_ingest_pairs_noalloc: null pointer");
    return GS_ERR_BAD_ARG;
  }
  const GsGeom geom = gs_make_geom(num_vertices, sketches_factor > 0 ? sketches_factor : 1.0);
  if (geom.num_columns > 64) {
    gs_set_error("gs_ingest_pairs_noalloc: more than 64 sketch columns are not supported");
    return GS_ERR_BAD_ARG;
  }
  if (n == 0) return GS_OK;

  uint32_t* status = nullptr;
  int sms = 0;
  GS_TRY(word_for_current_device(&status, &sms));
  cudaStream_t s = static_cast<cudaStream_t>(cuda_stream);
  GS_TRY(gs_ingest_pairs_direct(pairs, (uint32_t)n, geom, reinterpret_cast<GsBucket*>(sketches), seed, status, sms, s));
  // the call returns once the update is applied, with the device error word checked (and cleared)
  uint32_t err = 0;
  GS_CUDA_TRY(cudaMemcpyAsync(&err, status, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
  GS_CUDA_TRY(cudaStreamSynchronize(s));
  if (err) {
    GS_CUDA_TRY(cudaMemsetAsync(status, 0, sizeof(uint32_t), s));
    GS_CUDA_TRY(cudaStreamSynchronize(s));
  }
  if (err & GS_DEV_ERR_VERTEX_RANGE) {
    gs_set_error("gs_ingest_pairs_noalloc: a record named a vertex id >= num_vertices; it was skipped and every "
                 "other record of the call was applied");
    return GS_ERR_BAD_ARG;
  }
  if (err) {
    gs_set_error("gs_ingest_pairs_noalloc: device consistency check failed");
    return GS_ERR_INTERNAL;
  }
  return GS_OK;
}
