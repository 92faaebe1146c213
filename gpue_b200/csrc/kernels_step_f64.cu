// kernels_step_f64.cu -- the complex128 resident steppers (stepper.cuh).
#include "stepper.cuh"

namespace gpue {

static const StepKernel kTable[] = {
    GPUE_STEP(double, 16, 4, 0, 0, 4, 8, 1),
    GPUE_STEP(double, 32, 4, 2, 0, 8, 4, 1),
    GPUE_STEP(double, 64, 4, 4, 0, 16, 2, 1),
    GPUE_STEP(double, 96, 4, 6, 0, 8, 4, 1),
    GPUE_STEP(double, 128, 4, 8, 0, 16, 2, 1),
    GPUE_STEP(double, 160, 4, 10, 0, 8, 4, 1),
    GPUE_STEP(double, 192, 4, 12, 0, 16, 2, 1),
    GPUE_STEP(double, 256, 8, 4, 0, 32, 2, 1),
    GPUE_STEP(double, 320, 4, 5, 4, 16, 4, 1),
    GPUE_STEP(double, 384, 4, 6, 4, 32, 3, 1),
    GPUE_STEP(double, 512, 8, 8, 0, 64, 2, 2),
    GPUE_STEP(double, 640, 4, 10, 4, 32, 5, 1),
    GPUE_STEP(double, 768, 4, 12, 4, 64, 2, 3),
    GPUE_STEP(double, 1024, 16, 4, 0, 64, 4, 2),
};

const StepKernel* step_table_f64(int* count) {
    *count = (int)(sizeof(kTable) / sizeof(kTable[0]));
    return kTable;
}

}  // namespace gpue
