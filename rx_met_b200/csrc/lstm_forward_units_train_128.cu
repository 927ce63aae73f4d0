// Instances of the recurrence of lstm_forward_cluster.cuh with a thread per unit.
#include "lstm_forward_cluster.cuh"

namespace rxmet {
namespace lstm {

template <>
void lstmUnits<Saves::All, 128, 1>(const planerec::Problem &p, const LstmPlaneCell<true> &cell, cudaStream_t st) {
    launchLstmUnits<Saves::All, 128, 1>("lstmRecurrent", p, cell, st);
}
template <>
void lstmUnits<Saves::All, 128, 2>(const planerec::Problem &p, const LstmPlaneCell<true> &cell, cudaStream_t st) {
    launchLstmUnits<Saves::All, 128, 2>("lstmRecurrentWide", p, cell, st);
}

}  // namespace lstm
}  // namespace rxmet
