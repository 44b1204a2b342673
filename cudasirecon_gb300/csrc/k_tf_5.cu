// Two-factor kernels, part 5: every 8th factor pair by length
#include "tf_kernels.cuh"

namespace simrecon {

extern const TfKernels kTfPart5[] = {
    TfEntry<12, 8>::kernels(),
    TfEntry<14, 10>::kernels(),
    TfEntry<16, 12>::kernels(),
    TfEntry<27, 9>::kernels(),
    TfEntry<20, 15>::kernels(),
    TfEntry<21, 18>::kernels(),
    TfEntry<28, 16>::kernels(),
    TfEntry<27, 20>::kernels(),
    TfEntry<32, 20>::kernels(),
    TfEntry<28, 27>::kernels(),
    TfEntry<30, 30>::kernels(),
};
extern const int kTfPart5Count = sizeof(kTfPart5) / sizeof(kTfPart5[0]);

}  // namespace simrecon
