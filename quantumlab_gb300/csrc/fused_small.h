// fused_small.h -- plans on small FP32 registers in one launch (fused_small.cu).
#pragma once

#include "fused_plan.h"

#include <cuda_runtime.h>
#include <stddef.h>

namespace qg {

// Whether a plan runs as one program: the library chooses the applier, no
// pass has control qubits, and the register is one where it wins.  Per pass,
// with the launch and its wait, of an 8-layer random circuit, against the
// tensor cores pass by pass: 16 qubits 3.4 us (7.1), 17 4.2 (6.9), 18 5.7
// (7.1), 19 9.3 (8.1); 20 qubits 16.0 (8.5).  19 qubits stay, for sums that
// are nearer to 64 bits than split operands.
constexpr int kSmallMaxQubits = 19;
bool smallPlanFits(const FusedPlan& plan);
// reuse: an earlier program, whose memory is taken over; null when it failed
void* smallPlanUpload(const FusedPlan& plan, void* reuse);
void smallPlanFree(void* program);
size_t smallPlanBytes(const void* program);          // device memory it holds
int smallPlanApply(void* program, float* re, float* im, int first, int last);

}  // namespace qg
