// Two-factor kernels, part 2: every 8th factor pair by length
#include "tf_kernels.cuh"

namespace simrecon {

extern const TfKernels kTfPart2[] = {
    TfEntry<10, 8>::kernels(),
    TfEntry<14, 9>::kernels(),
    TfEntry<14, 12>::kernels(),
    TfEntry<16, 14>::kernels(),
    TfEntry<20, 14>::kernels(),
    TfEntry<25, 14>::kernels(),
    TfEntry<21, 20>::kernels(),
    TfEntry<24, 21>::kernels(),
    TfEntry<25, 24>::kernels(),
    TfEntry<30, 24>::kernels(),
    TfEntry<30, 28>::kernels(),
};
extern const int kTfPart2Count = sizeof(kTfPart2) / sizeof(kTfPart2[0]);

}  // namespace simrecon
