// Reverse recurrence of the LSTM QAT backward over thread-block clusters: more than 256 hidden units.  A CTA owns 32 of them:
// its weights take 64 columns of tensor memory per 128 units and leave room for the accumulators of 16 rows; nine to sixteen CTAs
// form a cluster.
#include <cuda_runtime.h>

#include "lstm_backward_cluster.cuh"

namespace rxmet {
namespace lstm {
namespace reverse {
namespace {

template <int ROWS>
Variant variantFor(int H) {
    switch (H) {
        case 288: return variant<288, 32, ROWS>();
        case 320: return variant<320, 32, ROWS>();
        case 352: return variant<352, 32, ROWS>();
        case 384: return variant<384, 32, ROWS>();
        case 416: return variant<416, 32, ROWS>();
        case 448: return variant<448, 32, ROWS>();
        case 480: return variant<480, 32, ROWS>();
        default: return variant<512, 32, ROWS>();
    }
}

}  // namespace

Variant wideVariant(int H, int rows) { return rows == 4 ? variantFor<4>(H) : rows == 8 ? variantFor<8>(H) : rows == 16 ? variantFor<16>(H) : variantFor<20>(H); }

}  // namespace reverse
}  // namespace lstm
}  // namespace rxmet
