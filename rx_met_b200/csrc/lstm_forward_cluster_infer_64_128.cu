// Instances of the cluster recurrence of lstm_forward_cluster.cuh.
#include "lstm_forward_cluster.cuh"

namespace rxmet {
namespace lstm {

template <>
void lstmCluster<false, 64>(const planerec::Problem &p, const LstmPlaneCell<false> &cell, cudaStream_t st) {
    launchLstmCluster<false, 64>(p, cell, st);
}
template <>
void lstmCluster<false, 128>(const planerec::Problem &p, const LstmPlaneCell<false> &cell, cudaStream_t st) {
    launchLstmCluster<false, 128>(p, cell, st);
}
template <>
void lstmBytes<64>(const planerec::Problem &p, const LstmPlaneCell<false> &cell, cudaStream_t st) {
    launchLstmBytes<64>(p, cell, st);
}
template <>
void lstmBytes<128>(const planerec::Problem &p, const LstmPlaneCell<false> &cell, cudaStream_t st) {
    launchLstmBytes<128>(p, cell, st);
}

}  // namespace lstm
}  // namespace rxmet
