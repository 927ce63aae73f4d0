// Instances of the cluster recurrence of lstm_forward_cluster.cuh.
#include "lstm_forward_cluster.cuh"

namespace rxmet {
namespace lstm {

template <>
void lstmCluster<false, 256>(const planerec::Problem &p, const LstmPlaneCell<false> &cell, cudaStream_t st) {
    launchLstmCluster<false, 256>(p, cell, st);
}
template <>
void lstmCluster<false, 384>(const planerec::Problem &p, const LstmPlaneCell<false> &cell, cudaStream_t st) {
    launchLstmCluster<false, 384>(p, cell, st);
}

}  // namespace lstm
}  // namespace rxmet
