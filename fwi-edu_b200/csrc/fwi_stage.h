/* fwi_stage.h -- copies between pageable host memory and the device by several host threads (internal).
 *
 * A pageable cudaMemcpyAsync runs through the driver's staging buffer on the calling thread, and a fresh
 * destination's page faults besides; the gathers of a survey pass through it on every call of the
 * host-array entry points.  These copies are cut into 1 MB pieces that up to four threads move through
 * page-locked buffers of their own (two each, 8 MB in all), with the device copies on the caller's
 * stream, whose earlier work the caller waits for first.  Page-locked caller memory and jobs below 24 MB go to cudaMemcpyAsync as they are.  Measured
 * (16-core host, B200): 58 MB up in 2.1 ms against 4.1, 115 MB in 3.6 against 9.0; pieces of 256 KB 3.0
 * and 5.7, eight threads 2.7 and 4.1.  The threshold: misfit and step length of gathers of 8 MB (jobs of
 * 8 and 16) take 1.8 ms as they are and 2.3 staged, of 16 MB (16 and 32) 4.2 and 2.7; below, threads
 * that have to wake up only cost (2.2 MB: 0.87 and 1.29 ms).  Down to the host both are the same to 12 MB. */
#ifndef FWI_STAGE_H
#define FWI_STAGE_H

#include <cuda_runtime.h>

#include <cstddef>
#include <vector>

namespace fwi {

struct HostCopy {
    void *dst;
    const void *src;
    size_t bytes;
};
// Host to device: the copies are ordered on st, and the sources may be reused when the call returns
// unless they are page-locked.
cudaError_t stage_to_device(const std::vector<HostCopy> &copies, cudaStream_t st);
// Device to host, after the work on st so far: the data has arrived when the call returns.
cudaError_t stage_to_host(const std::vector<HostCopy> &copies, cudaStream_t st);

}  // namespace fwi
#endif
