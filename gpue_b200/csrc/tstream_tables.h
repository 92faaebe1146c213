// tstream_tables.h -- table entries of the tile-stream kernels (tstream.cuh).
#pragma once

#include "registry.h"
#include "tstream.cuh"

namespace gpue {

#define GPUE_ZPASS(T, N, RA, RB, RC, P)                                                     \
    ZPassKernel{N, RA, RB, RC, P, TSShape<T, N, RA, RB, P, RC>::THREADS,                     \
                (int)TSShape<T, N, RA, RB, P, RC>::SMEM,                                     \
                (const void*)&k_tstream<T, N, RA, RB, P, RC, TS_Z>}

#define GPUE_XY(T, N, RA, RB, RC, P)                                                        \
    XYKernel{N, RA, RB, RC, P, TSShape<T, N, RA, RB, P, RC>::THREADS,                        \
             (int)TSShape<T, N, RA, RB, P, RC>::SMEM,                                        \
             (const void*)&k_tstream<T, N, RA, RB, P, RC, TS_XY_FWD>,                        \
             (const void*)&k_tstream<T, N, RA, RB, P, RC, TS_XY_INV>,                        \
             (const void*)&k_tstream<T, N, RA, RB, P, RC, TS_XY_INV_GY>,                     \
             (const void*)&k_tstream<T, N, RA, RB, P, RC, TS_YX_INV_GX>}

const ZPassKernel* zpass_table_f32(int* count);
const ZPassKernel* zpass_table_f64(int* count);
const XYKernel* xy_table_f32(int* count);
const XYKernel* xy_table_f64(int* count);

}  // namespace gpue
