// Launchers of the doubled-grid assembly passes (k_assemble2.cu), used by the
// assembly in k_assemble.cu.
#pragma once
#include "kernels.h"

namespace simrecon {

// the y (x) axis is doubled and its image length has a two-factor plan
bool asm_y2_supported(const AssembleArgs& a);
bool asm_x2_supported(const AssembleArgs& a);
// y pass of `nslots` slots into a.T; filt: filter the bands as they are loaded
int launch_asm_y2(const AssembleArgs& a, const void* d_slots, int nslots, const FilterArgs* filt, cudaStream_t s);
// x pass of `nplanes` output planes: S with its columns split by parity (the
// ramp table a.ex too), or with `real` (Z = 1) the result itself
int launch_asm_x2(const AssembleArgs& a, const void* d_slots, const int* d_p0, const int* d_pn, const int* d_pz,
                  int nplanes, bool real, cudaStream_t s);

}  // namespace simrecon
