// pauli_expec.h -- Pauli-sum expectation values in tiles (expec_tile.cu).
#pragma once

#include "qg_internal.h"

#include <functional>

namespace qg {

// whether terms with X/Y mask x on a state vector of n qubits go by tiles
bool expecTileTakes(int n, uint64_t x);
// queue the groups' reductions, each pass into the slot it is given (a device
// double; null: stop); false when a launch failed
bool queueExpecTiles(SV s, const std::vector<PauliTermGroup>& groups, const Scratch& w, const std::function<double*()>& slot,
                     const char* caller);

}  // namespace qg
