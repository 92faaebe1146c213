// kernels_tile_f64.cu -- the complex128 TMA tile-stream XY and z passes of the
// 3D step (tstream.cuh), per length; the XY passes from 128 on (plan_xy).
#include "tstream_tables.h"

namespace gpue {

static const ZPassKernel kZPass[] = {
    GPUE_ZPASS(double, 64, 4, 4, 0, 16),
    GPUE_ZPASS(double, 96, 4, 6, 0, 8),
    GPUE_ZPASS(double, 128, 4, 8, 0, 16),
    GPUE_ZPASS(double, 160, 4, 10, 0, 8),
    GPUE_ZPASS(double, 192, 4, 12, 0, 16),
    GPUE_ZPASS(double, 256, 16, 0, 0, 16),
};

static const XYKernel kXY[] = {
    GPUE_XY(double, 128, 4, 8, 0, 16),
    GPUE_XY(double, 160, 4, 10, 0, 8),
    GPUE_XY(double, 192, 4, 12, 0, 16),
    GPUE_XY(double, 256, 16, 0, 0, 16),
};

const ZPassKernel* zpass_table_f64(int* count) {
    *count = (int)(sizeof(kZPass) / sizeof(kZPass[0]));
    return kZPass;
}

const XYKernel* xy_table_f64(int* count) {
    *count = (int)(sizeof(kXY) / sizeof(kXY[0]));
    return kXY;
}

}  // namespace gpue
