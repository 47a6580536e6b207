// The y-z solve in clusters, FP32.
#include "slab_cluster.cuh"

namespace c3d {

template int launch_cluster<float>(Handle*, float2*, int, int, int);
template int cluster_setup<float>(Handle*);

}  // namespace c3d
