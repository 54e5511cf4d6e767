// Dense gates on 5 and 6 qubits on the CUDA cores (dense_wide.cu).
#pragma once

#include "engine.hpp"

namespace qvdg {

// Launches the gate's pass; false when the gate or the state is not one this
// kernel takes (fewer than 2^11 complex64 or 2^10 complex128 amplitudes
// selected). `mat`: the gate's matrix on the device.
bool launch_dense_wide(StateImpl& s, const PlainGate& g, const void* mat);

}  // namespace qvdg
