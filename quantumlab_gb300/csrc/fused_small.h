// fused_small.h -- plans on small FP32 registers in one launch (fused_small.cu).
#pragma once

#include "fused_plan.h"

#include <cuda_runtime.h>
#include <stddef.h>

namespace qg {

// Whether a plan runs as one program: the library chooses the applier, no
// pass has control qubits, and the register is one where it wins.  Per pass,
// with the launch and its wait, of an 8-layer random circuit, against the
// tensor cores pass by pass: 16 qubits 3.4 us (10.6), 17 4.2 (10.5), 18 5.7
// (10.5), 19 9.3 (10.6); 20 qubits 16.0 (10.1).
constexpr int kSmallMaxQubits = 19;
bool smallPlanFits(const FusedPlan& plan);
// reuse: an earlier program, whose memory is taken over; null when it failed
void* smallPlanUpload(const FusedPlan& plan, void* reuse);
void smallPlanFree(void* program);
int smallPlanApply(void* program, float* re, float* im, int first, int last);

}  // namespace qg
