// Factor pairs of the zoomed x transform, part 0 (asm_x2.cuh)
#include "asm_x2.cuh"

namespace simrecon {

bool asm_x2_part0(const AsmX2Launch& l)
{
#define SIMRECON_X2_CASE(R1, R2) \
  if (asm_x2_run<R1, R2>(l)) return true;
  SIMRECON_X2_PAIRS_0(SIMRECON_X2_CASE)
#undef SIMRECON_X2_CASE
  return false;
}

}  // namespace simrecon
