// Two-factor kernels, part 6: every 8th factor pair by length
#include "tf_kernels.cuh"

namespace simrecon {

extern const TfKernels kTfPart6[] = {
    TfEntry<10, 10>::kernels(),
    TfEntry<12, 12>::kernels(),
    TfEntry<14, 14>::kernels(),
    TfEntry<25, 10>::kernels(),
    TfEntry<21, 15>::kernels(),
    TfEntry<24, 16>::kernels(),
    TfEntry<25, 18>::kernels(),
    TfEntry<28, 20>::kernels(),
    TfEntry<27, 24>::kernels(),
    TfEntry<32, 24>::kernels(),
    TfEntry<32, 30>::kernels(),
};
extern const int kTfPart6Count = sizeof(kTfPart6) / sizeof(kTfPart6[0]);

}  // namespace simrecon
