// fused_small.h -- plans on small FP32 registers in one launch (fused_small.cu).
#pragma once

#include "fused_plan.h"

#include <cuda_runtime.h>
#include <stddef.h>

namespace qg {

constexpr int kSmallMaxSegs = 8;             // classes of registers in one launch
constexpr size_t kSmallMatrixFloats = 2 * 64 * 64;

struct SmallSeg {                            // one pass of one class (Seg in fused_small.cu)
    uint64_t state, mat;
    uint32_t chunks, each, more;
    int chunkBits, n;
    unsigned char pos[12];
    unsigned short word[12];
};

// A list of steps; the segments [first[s], first[s + 1]) of step s run side
// by side, the steps one after the other.
struct SmallProgram {
    int groups = 16;                         // groups of 64 amplitudes a chunk (8, 16 or 32)
    uint32_t maxChunks = 0;
    unsigned grid = 1;
    std::vector<SmallSeg> segs;
    std::vector<int> first;
    size_t bytes = 0;                        // room in buffer
    void* buffer = nullptr;                  // device: matrices, segments, barrier counters
    float* dMats = nullptr;
    void* dSegs = nullptr;
    int perStep = 1;                         // segments a step, as uploaded
    unsigned* counters = nullptr;            // arrivals at the barrier, ended blocks; zero between launches
};

// groups a chunk for `amps` amplitudes in a pass: the most of 8, 16, 32 that
// leaves at most half the SMs without a chunk
int smallGroups(uint64_t amps);
// whether a pass without control qubits on registers of n qubits can be one of a program
bool smallFits(int n, const std::vector<int>& targets);
// append the pass on `registers` registers, `stateOffset` floats from the base,
// their matrices from `mat` on; returns the end of the matrices
size_t smallAddPass(SmallProgram& p, const FusedPass& pass, int n, size_t stateOffset, int registers, size_t mat);
// the pass's matrix as the kernel reads it (2 x 64 x 64 floats)
void smallMatrix(const FusedPass& pass, int n, float* out);
// mats null: the caller fills p.dMats
bool smallUpload(SmallProgram& p, const float* mats, size_t matFloats, const char* caller);
bool smallLaunch(const SmallProgram& p, float* re, float* im, int step0, int step1, int* errFlag, cudaStream_t st,
                 const char* caller);
void smallReset(SmallProgram& p);
void smallFree(SmallProgram& p);

// Whether a plan runs as one program: the library chooses the applier, no
// pass has control qubits, and the register is one where it wins.  Per pass,
// with the launch and its wait, of an 8-layer random circuit, against the
// tensor cores pass by pass: 16 qubits 3.9 us (14.9), 17 4.7 (14.5), 18 5.8
// (14.5), 19 9.3 (14.7); 20 qubits 16.0 (13.9).
constexpr int kSmallMaxQubits = 19;
bool smallPlanFits(const FusedPlan& plan);
// reuse: an earlier program, whose memory is taken over; null when it failed
void* smallPlanUpload(const FusedPlan& plan, void* reuse);
void smallPlanFree(void* program);
int smallPlanApply(void* program, float* re, float* im, int first, int last);

}  // namespace qg
