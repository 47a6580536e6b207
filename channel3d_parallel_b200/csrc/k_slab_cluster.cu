// The y-z solve in clusters, FP64.
#include "slab_cluster.cuh"

namespace c3d {

template int launch_cluster<double>(Handle*, double2*, int, int, int);
template int cluster_setup<double>(Handle*);

}  // namespace c3d
