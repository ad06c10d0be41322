// upload_source.h -- the host memory of a queued upload.
//
// A copy from pageable memory may still read its source after cudaMemcpyAsync
// has returned: it is staged only where it must be, and a coherent host needs
// no staging.  The source therefore stays with the plan that is uploaded, and
// is written again only once the last copy from it has run.
#pragma once

#include "qg_internal.h"

#include <cuda_runtime.h>
#include <stddef.h>

#include <vector>

namespace qg {

class UploadSource {
public:
    UploadSource() = default;
    UploadSource(const UploadSource&) = delete;
    UploadSource& operator=(const UploadSource&) = delete;
    ~UploadSource() { release(); }
    // n zero bytes to fill; null when the last copy failed
    char* open(size_t n, const char* caller) {
        if (copied_ && QG_CUDA(cudaEventSynchronize(copied_), caller)) return nullptr;
        bytes_.assign(n, 0);
        return bytes_.data();
    }
    // queue their copy to dst
    bool copy(void* dst, cudaStream_t st, const char* caller) {
        if (!copied_ && QG_CUDA(cudaEventCreateWithFlags(&copied_, cudaEventDisableTiming), caller)) return false;
        return !QG_CUDA(cudaMemcpyAsync(dst, bytes_.data(), bytes_.size(), cudaMemcpyHostToDevice, st), caller) &&
               !QG_CUDA(cudaEventRecord(copied_, st), caller);
    }
    void release() {
        if (copied_) {
            (void)cudaEventSynchronize(copied_);
            (void)cudaEventDestroy(copied_);
        }
        copied_ = nullptr;
        std::vector<char>().swap(bytes_);
    }

private:
    std::vector<char> bytes_;
    cudaEvent_t copied_ = nullptr;       // after the last copy
};

}  // namespace qg
