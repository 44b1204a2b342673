// Two-factor kernels, part 4: every 8th factor pair by length
#include "tf_kernels.cuh"

namespace simrecon {

extern const TfKernels kTfPart4[] = {
    TfEntry<10, 9>::kernels(),
    TfEntry<15, 9>::kernels(),
    TfEntry<21, 9>::kernels(),
    TfEntry<16, 15>::kernels(),
    TfEntry<21, 14>::kernels(),
    TfEntry<25, 15>::kernels(),
    TfEntry<21, 21>::kernels(),
    TfEntry<25, 21>::kernels(),
    TfEntry<30, 21>::kernels(),
    TfEntry<30, 25>::kernels(),
    TfEntry<32, 28>::kernels(),
};
extern const int kTfPart4Count = sizeof(kTfPart4) / sizeof(kTfPart4[0]);

}  // namespace simrecon
