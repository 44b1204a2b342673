// Two-factor kernels, part 7: every 8th factor pair by length
#include "tf_kernels.cuh"

namespace simrecon {

extern const TfKernels kTfPart7[] = {
    TfEntry<12, 9>::kernels(),
    TfEntry<15, 10>::kernels(),
    TfEntry<20, 10>::kernels(),
    TfEntry<18, 14>::kernels(),
    TfEntry<20, 16>::kernels(),
    TfEntry<28, 14>::kernels(),
    TfEntry<24, 20>::kernels(),
    TfEntry<27, 21>::kernels(),
    TfEntry<28, 24>::kernels(),
    TfEntry<28, 28>::kernels(),
    TfEntry<32, 32>::kernels(),
};
extern const int kTfPart7Count = sizeof(kTfPart7) / sizeof(kTfPart7[0]);

}  // namespace simrecon
