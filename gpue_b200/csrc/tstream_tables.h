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

// without the gauge passes (lengths whose rotating steps run as line passes)
#define GPUE_XY_PLAIN(T, N, RA, RB, RC, P)                                                  \
    XYKernel{N, RA, RB, RC, P, TSShape<T, N, RA, RB, P, RC>::THREADS,                        \
             (int)TSShape<T, N, RA, RB, P, RC>::SMEM,                                        \
             (const void*)&k_tstream<T, N, RA, RB, P, RC, TS_XY_FWD>,                        \
             (const void*)&k_tstream<T, N, RA, RB, P, RC, TS_XY_INV>, nullptr, nullptr}

const ZPassKernel* zpass_table_f32(int* count);
const ZPassKernel* zpass_table_f64(int* count);
const XYKernel* xy_table_f32(int* count);
const XYKernel* xy_table_f64(int* count);

}  // namespace gpue
