// Two-factor kernels, part 3: every 8th factor pair by length
#include "tf_kernels.cuh"

namespace simrecon {

extern const TfKernels kTfPart3[] = {
    TfEntry<9, 9>::kernels(),
    TfEntry<16, 8>::kernels(),
    TfEntry<15, 12>::kernels(),
    TfEntry<15, 15>::kernels(),
    TfEntry<18, 16>::kernels(),
    TfEntry<20, 18>::kernels(),
    TfEntry<24, 18>::kernels(),
    TfEntry<32, 16>::kernels(),
    TfEntry<25, 25>::kernels(),
    TfEntry<27, 27>::kernels(),
    TfEntry<32, 27>::kernels(),
};
extern const int kTfPart3Count = sizeof(kTfPart3) / sizeof(kTfPart3[0]);

}  // namespace simrecon
