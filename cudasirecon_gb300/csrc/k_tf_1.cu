// Two-factor kernels, part 1: every 8th factor pair by length
#include "tf_kernels.cuh"

namespace simrecon {

extern const TfKernels kTfPart1[] = {
    TfEntry<9, 8>::kernels(),
    TfEntry<12, 10>::kernels(),
    TfEntry<18, 9>::kernels(),
    TfEntry<18, 12>::kernels(),
    TfEntry<18, 15>::kernels(),
    TfEntry<21, 16>::kernels(),
    TfEntry<27, 15>::kernels(),
    TfEntry<25, 20>::kernels(),
    TfEntry<28, 21>::kernels(),
    TfEntry<28, 25>::kernels(),
    TfEntry<30, 27>::kernels(),
};
extern const int kTfPart1Count = sizeof(kTfPart1) / sizeof(kTfPart1[0]);

}  // namespace simrecon
