// The version of the interface between the library and the sweep kernels of a
// model compiled outside it (ModelKernels): the library fills the parameter
// blocks and the control block, the model's kernels read them, so both sides
// have to agree on their layout.  It is made of their sizes and kModelRevision:
// a field added on one side alone is refused at va_create_model, not read past
// the end of a smaller block.
#pragma once

#include <cstdint>

#include "va_kernels.cuh"
#include "va_registry.h"
#include "va_replay.cuh"

namespace va {

// raised when a field changes its meaning or place and no size changes
constexpr uint32_t kModelRevision = 2;

constexpr uint32_t mix_abi(uint32_t h, uint32_t v) { return (h ^ v) * 0x01000193u; }
constexpr uint32_t kModelAbi =
    mix_abi(mix_abi(mix_abi(mix_abi(mix_abi(mix_abi(0x811c9dc5u, kModelRevision), sizeof(FwdParams)),
                                    sizeof(AdjParams)),
                            sizeof(ReplayParams)),
                    sizeof(Control)),
            sizeof(KernelSet));

} // namespace va
