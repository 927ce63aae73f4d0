// Instances of the cluster recurrence of lstm_forward_cluster.cuh.
#include "lstm_forward_cluster.cuh"

namespace rxmet {
namespace lstm {

template <>
void lstmCluster<true, 256>(const planerec::Problem &p, const LstmPlaneCell<true> &cell, cudaStream_t st) {
    launchLstmCluster<true, 256>(p, cell, st);
}
template <>
void lstmCluster<true, 384>(const planerec::Problem &p, const LstmPlaneCell<true> &cell, cudaStream_t st) {
    launchLstmCluster<true, 384>(p, cell, st);
}

}  // namespace lstm
}  // namespace rxmet
