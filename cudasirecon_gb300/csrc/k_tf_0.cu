// Two-factor kernels, part 0: every 8th factor pair by length
#include "tf_kernels.cuh"

namespace simrecon {

extern const TfKernels kTfPart0[] = {
    TfEntry<8, 8>::kernels(),
    TfEntry<14, 8>::kernels(),
    TfEntry<16, 10>::kernels(),
    TfEntry<15, 14>::kernels(),
    TfEntry<16, 16>::kernels(),
    TfEntry<18, 18>::kernels(),
    TfEntry<20, 20>::kernels(),
    TfEntry<27, 18>::kernels(),
    TfEntry<24, 24>::kernels(),
    TfEntry<27, 25>::kernels(),
    TfEntry<32, 25>::kernels(),
};
extern const int kTfPart0Count = sizeof(kTfPart0) / sizeof(kTfPart0[0]);

}  // namespace simrecon
