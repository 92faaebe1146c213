// kernels_tile_f32.cu -- the complex64 TMA tile-stream XY and z passes of the
// 3D step (tstream.cuh), per length; with the gauge from 192 on (plan_xy).
#include "tstream_tables.h"

namespace gpue {

static const ZPassKernel kZPass[] = {
    GPUE_ZPASS(float, 64, 4, 4, 0, 16),
    GPUE_ZPASS(float, 96, 4, 6, 0, 8),
    GPUE_ZPASS(float, 128, 4, 8, 0, 16),
    GPUE_ZPASS(float, 160, 4, 10, 0, 8),
    GPUE_ZPASS(float, 192, 4, 12, 0, 16),
    GPUE_ZPASS(float, 256, 16, 0, 0, 16),
};

static const XYKernel kXY[] = {
    GPUE_XY_PLAIN(float, 64, 4, 4, 0, 16),
    GPUE_XY_PLAIN(float, 96, 4, 6, 0, 8),
    GPUE_XY_PLAIN(float, 128, 4, 8, 0, 16),
    GPUE_XY_PLAIN(float, 160, 4, 10, 0, 8),
    GPUE_XY(float, 192, 4, 12, 0, 16),
    GPUE_XY(float, 256, 16, 0, 0, 16),
};

const ZPassKernel* zpass_table_f32(int* count) {
    *count = (int)(sizeof(kZPass) / sizeof(kZPass[0]));
    return kZPass;
}

const XYKernel* xy_table_f32(int* count) {
    *count = (int)(sizeof(kXY) / sizeof(kXY[0]));
    return kXY;
}

const XYKernel* find_xy_kernel(int prec, int n) {
    int cnt = 0;
    const XYKernel* t = prec == PREC_F32 ? xy_table_f32(&cnt) : xy_table_f64(&cnt);
    for (int i = 0; i < cnt; ++i)
        if (t[i].n == n) return &t[i];
    return nullptr;
}

const ZPassKernel* find_zpass_kernel(int prec, int n) {
    int cnt = 0;
    const ZPassKernel* t = prec == PREC_F32 ? zpass_table_f32(&cnt) : zpass_table_f64(&cnt);
    for (int i = 0; i < cnt; ++i)
        if (t[i].n == n) return &t[i];
    return nullptr;
}

}  // namespace gpue
