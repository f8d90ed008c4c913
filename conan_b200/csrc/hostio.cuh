// hostio.cuh -- copies between device memory and the caller's host arrays, and
// device memory and FFT plans for calls without a handle.
//
// A caller's array is usually pageable, and a fresh result array has no pages
// yet: the driver copies those on one thread through its own staging buffer,
// at the speed of that thread's page faults (5 GB/s; the link does 55). Here
// several host threads take chunks in turn, each through a page-locked buffer
// and a stream of its own, so that faults, memory copies and transfers overlap.
// Page-locked arrays go to the driver as they are.
//
// What outlives a call, all bounded and safe to use from several threads:
// HOSTIO_LANES page-locked buffers of HOSTIO_CHUNK bytes with their streams
// per device, a device memory pool that keeps at most HOSTIO_POOL_KEEP idle
// bytes per device, and HOSTIO_PLANS idle plan pairs. conan_release_caches
// gives all of it back.
#pragma once

#include "fft.cuh"

namespace conan {

constexpr int HOSTIO_LANES = 8;
constexpr size_t HOSTIO_CHUNK = (size_t)2 << 20;
constexpr size_t HOSTIO_POOL_KEEP = (size_t)512 << 20;
constexpr int HOSTIO_PLANS = 4;

// Device to host, ordered after the work on st. A pageable destination holds
// the data on return; a page-locked one when st has run.
int copy_to_host(void *dst, const void *src, size_t bytes, cudaStream_t st);
// Host to device, ordered after the work on st and before what follows on it.
// The source may be reused on return (a page-locked one when st has run).
int copy_to_device(void *dst, const void *src, size_t bytes, cudaStream_t st);

// Device memory of one call from the current device's pool, stream-ordered.
cudaError_t pool_alloc(void **p, size_t bytes, cudaStream_t st);
void pool_free(void *p, cudaStream_t st);

// An R2C/C2R pair for one mesh of m's shape on the current device, unbound; the
// caller binds it, and returns it once the work on its stream is done.
int plan_take(const Mesh &m, bool is_double, FFTPair *fft);
void plan_return(const Mesh &m, bool is_double, FFTPair *fft);

}  // namespace conan
