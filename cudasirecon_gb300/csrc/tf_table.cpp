// The two-factor kernels by length (tf_kernels.h).
#include "tf_kernels.h"

namespace simrecon {

#define SIMRECON_TF_PART(i)           \
  extern const TfKernels kTfPart##i[]; \
  extern const int kTfPart##i##Count;
SIMRECON_TF_PART(0)
SIMRECON_TF_PART(1)
SIMRECON_TF_PART(2)
SIMRECON_TF_PART(3)
SIMRECON_TF_PART(4)
SIMRECON_TF_PART(5)
SIMRECON_TF_PART(6)
SIMRECON_TF_PART(7)
#undef SIMRECON_TF_PART

const TfKernels* tf_kernels(int n, TfPlan* plan)
{
  int r1, r2;
  if (!tf_factor(n, &r1, &r2)) return nullptr;
  struct Part {
    const TfKernels* k;
    int n;
  };
  const Part parts[] = {{kTfPart0, kTfPart0Count}, {kTfPart1, kTfPart1Count}, {kTfPart2, kTfPart2Count},
                        {kTfPart3, kTfPart3Count}, {kTfPart4, kTfPart4Count}, {kTfPart5, kTfPart5Count},
                        {kTfPart6, kTfPart6Count}, {kTfPart7, kTfPart7Count}};
  for (const Part& p : parts)
    for (int i = 0; i < p.n; ++i)
      if (p.k[i].r1 == r1 && p.k[i].r2 == r2) return plan && !get_tf_plan(n, plan) ? nullptr : &p.k[i];
  return nullptr;
}

}  // namespace simrecon
