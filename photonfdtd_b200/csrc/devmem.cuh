// devmem.cuh - memory that outlives one engine: a device pool and pinned error words.
//
// Building an engine takes some 60 allocations, and cudaMalloc / cudaFree of
// them took 3 to 30 ms per run (each cudaFree waits for the device and unmaps),
// as long as a small scene's stepping. A stream-ordered pool keeps up to
// kPoolKeep bytes of freed memory mapped for the next engine; what is above
// that goes back to the driver at the next synchronisation, and everything
// when an allocation of this library fails (pool_trim), a batch sizes itself,
// or the user asks (pf_release_memory). The pool belongs to no engine and is
// never handed pointers of another allocator. Its calls are thread safe, and
// its ordering is per stream: memory freed on one engine's stream reaches
// another only behind the work queued before the free.
//
// Error words are mapped host memory, so that reading one costs no copy; one
// page serves 1024 engines (pinning memory per engine took longer than a small
// run).
//
// Both belong to a CUDA context and end with it (cudaDeviceReset). They are
// kept by the context's id, which no later context repeats, so what a reset
// took is forgotten unseen and never touched again.
#pragma once

#include <cuda_runtime.h>

namespace pfb {

constexpr unsigned long long kPoolKeep = 2ull << 30;

// bytes of device memory in `st`'s order (a stream of device `dev`).
cudaError_t pool_alloc(void** p, size_t bytes, int dev, cudaStream_t st);
void pool_free(void* p, cudaStream_t st);
// Gives back what the pool of the thread's current context holds unused.
void pool_trim();
// cudaMalloc, and once more after pool_trim if there was no memory.
cudaError_t malloc_trim(void** p, size_t bytes);

// An error word (zero) of the context of `st`, or p == nullptr.
struct ErrWord {
  int* p = nullptr;
  unsigned long long ctx = 0;
};
ErrWord err_word(int dev, cudaStream_t st);
void err_word_release(int dev, const ErrWord& w);

}  // namespace pfb
