// fused_build.h -- pass operands formed on the device (fused_build.cu).
#pragma once

#include "fused_plan.h"
#include "upload_source.h"

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace qg {

// Where a pass's operands go and in which form; offsets are floats into the
// output, ~0 for a form that is not wanted (the forms of fused_tc.cu's
// ImageLayout, and fused_small.cu's matrix).
struct BuildOutput {
    size_t full = ~(size_t)0, bf16 = ~(size_t)0, compact = ~(size_t)0, f16 = ~(size_t)0;
    size_t small = ~(size_t)0;
    int smallMask = 0;                   // small: the pass's own among the 6 widened qubits
};
// device and host buffers kept from one build to the next (grow-only)
struct BuildScratch {
    void* device = nullptr;
    size_t bytes = 0;
    UploadSource source;
};
void freeBuildScratch(BuildScratch& s);

// whether a pass's product may be left to the device: gates of at most 3
// qubits, no control qubits
bool buildsOnDevice(const FusedPlan& plan, const FusedPass& pass, const std::vector<int>& members);
// queue the products of the passes `which` (their matrices left out) and their
// operands at out; false when a launch or an allocation failed
bool queueBuild(const FusedPlan& plan, const std::vector<int>& which, const std::vector<BuildOutput>& outputs, float* out,
                BuildScratch& scratch, cudaStream_t st, const char* caller);

}  // namespace qg
