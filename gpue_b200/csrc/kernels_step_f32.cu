// kernels_step_f32.cu -- the complex64 resident steppers (stepper.cuh).
//
// (length, radix plan, threads per line, lines per CTA, CTAs per SM).  One CTA per
// SM where the lines have at most 32 threads; the plans are the line passes'
// defaults, so a step is as far from the exact one as they are.  Two others were
// faster and are not used: 8 2 8 at 128 (complex128 rotating 12.4 us per step
// instead of 13.4) is 1.3 to 1.6 times as far from the step in 80-bit arithmetic
// (complex64 1.08 times from complex128), 8 12 8 at 768 (47.6 instead of 51.6) up
// to 1.05 times.  16 16 at 256 and 8 8 8 with 32 threads at 512 were slower (9.4
// -> 10.7, 15.4 -> 16.3).  384 and 512 leave registers for a second CTA, so
// batched solves run side by side (batch.cu).
#include "stepper.cuh"

namespace gpue {

static const StepKernel kTable[] = {
    GPUE_STEP(float, 16, 4, 0, 0, 4, 8, 1),
    GPUE_STEP(float, 32, 4, 2, 0, 8, 4, 1),
    GPUE_STEP(float, 64, 4, 4, 0, 16, 4, 1),
    GPUE_STEP(float, 96, 4, 6, 0, 8, 4, 1),
    GPUE_STEP(float, 128, 4, 8, 0, 16, 4, 1),
    GPUE_STEP(float, 160, 4, 10, 0, 8, 4, 1),
    GPUE_STEP(float, 192, 4, 12, 0, 16, 2, 1),
    GPUE_STEP(float, 256, 8, 4, 0, 32, 4, 1),
    GPUE_STEP(float, 320, 4, 20, 0, 16, 4, 1),
    GPUE_STEP(float, 384, 4, 6, 4, 32, 4, 2),
    GPUE_STEP(float, 512, 8, 8, 0, 64, 4, 2),
    GPUE_STEP(float, 640, 4, 10, 4, 32, 5, 1),
    GPUE_STEP(float, 768, 4, 12, 4, 64, 2, 3),
    GPUE_STEP(float, 1024, 16, 4, 0, 64, 4, 2),
};

const StepKernel* step_table_f32(int* count) {
    *count = (int)(sizeof(kTable) / sizeof(kTable[0]));
    return kTable;
}

}  // namespace gpue
