// kernels_step_f32.cu -- the complex64 resident steppers (stepper.cuh).
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
    GPUE_STEP(float, 320, 4, 5, 4, 16, 4, 1),
    GPUE_STEP(float, 384, 4, 6, 4, 32, 4, 1),
    GPUE_STEP(float, 512, 8, 8, 0, 64, 4, 1),
    GPUE_STEP(float, 640, 4, 10, 4, 32, 5, 1),
    GPUE_STEP(float, 768, 4, 12, 4, 64, 2, 3),
    GPUE_STEP(float, 1024, 16, 4, 0, 64, 4, 2),
};

const StepKernel* step_table_f32(int* count) {
    *count = (int)(sizeof(kTable) / sizeof(kTable[0]));
    return kTable;
}

}  // namespace gpue
