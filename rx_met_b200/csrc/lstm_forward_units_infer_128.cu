// Instances of the recurrence of lstm_forward_cluster.cuh with a thread per unit.
#include "lstm_forward_cluster.cuh"

namespace rxmet {
namespace lstm {

template <>
void lstmUnits<Saves::None, 128, 1>(const planerec::Problem &p, const LstmPlaneCell<false> &cell, cudaStream_t st) {
    launchLstmUnits<Saves::None, 128, 1>("lstmRecurrent", p, cell, st);
}
template <>
void lstmUnits<Saves::None, 128, 2>(const planerec::Problem &p, const LstmPlaneCell<false> &cell, cudaStream_t st) {
    launchLstmUnits<Saves::None, 128, 2>("lstmRecurrentWide", p, cell, st);
}

}  // namespace lstm
}  // namespace rxmet
