// kernels_cluster_f64.cu -- the complex128 cluster-resident steppers (cluster_step.cuh).
#include "cluster_step.cuh"

namespace gpue {

static const ClusterKernel kTable[] = {
    GPUE_CLUSTER(double, 16, 4, 0, 0, 4),   GPUE_CLUSTER(double, 32, 4, 2, 0, 8),
    GPUE_CLUSTER(double, 64, 4, 4, 0, 16),  GPUE_CLUSTER(double, 96, 4, 6, 0, 8),
    GPUE_CLUSTER(double, 128, 4, 8, 0, 16), GPUE_CLUSTER(double, 192, 4, 12, 0, 16),
    GPUE_CLUSTER(double, 256, 16, 0, 0, 16),
};

const ClusterKernel* cluster_table_f64(int* count) {
    *count = (int)(sizeof(kTable) / sizeof(kTable[0]));
    return kTable;
}

}  // namespace gpue
