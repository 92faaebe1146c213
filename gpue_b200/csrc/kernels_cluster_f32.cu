// kernels_cluster_f32.cu -- the complex64 cluster-resident steppers (cluster_step.cuh).
#include "cluster_step.cuh"

namespace gpue {

static const ClusterKernel kTable[] = {
    GPUE_CLUSTER(float, 16, 4, 0, 0, 4),   GPUE_CLUSTER(float, 32, 4, 2, 0, 8),
    GPUE_CLUSTER(float, 64, 4, 4, 0, 16),  GPUE_CLUSTER(float, 96, 4, 6, 0, 8),
    GPUE_CLUSTER(float, 128, 4, 8, 0, 16), GPUE_CLUSTER(float, 160, 4, 10, 0, 8),
    GPUE_CLUSTER(float, 192, 4, 12, 0, 16), GPUE_CLUSTER(float, 256, 8, 4, 0, 32),
    GPUE_CLUSTER(float, 384, 4, 6, 4, 32),
};

const ClusterKernel* cluster_table_f32(int* count) {
    *count = (int)(sizeof(kTable) / sizeof(kTable[0]));
    return kTable;
}

}  // namespace gpue
