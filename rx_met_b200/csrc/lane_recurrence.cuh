// One step after another of a recurrence on byte-plane codes for narrow layers (at most 128 hidden units) and few rows, with
// the cells of plane_recurrence_umma.cuh: the product W_hh h on dp4a, four lanes of a warp per hidden unit.
//
// Over a cluster (plane_recurrence_umma.cuh) a step of few rows is a chain of a tensor-core product, copies between SMs and
// three barriers, 1.3 to 1.5 us however little there is to do.  A layer of up to 128 units fits one SM: a lane multiplies a
// quarter of K for all gates (weights in registers, both byte planes combined into one 32-bit sum, which 128 units cannot
// overflow), shuffles add the quarters such that lane g ends with gate g of every row, the operator's linear stage runs
// once per gate and row, further shuffles deal whole rows to lanes for the cell.  ONE barrier per step, hidden codes in two
// buffers by step parity; a step's operands are loaded one step ahead (two register sets, the loop unrolled by two) and
// its outputs are stored under the products of the next step.  Lanes beyond the last unit or row repeat the last one: the
// same values to the same places, no branches.
// T = 98, B = 32, H = 64, 16-bit GRU: 131 -> 77 us; T = 100, B = 1, H = 128, 16-bit LSTM: 0.78 us a step; four rows of 128 units and
// T = 200, B = 128 in both directions of an LSTM at a time, 286 us, are even with the clusters.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "common.h"
#include "plane_recurrence_umma.cuh"

namespace rxmet {
namespace lanerec {

using planerec::Problem;

__device__ __forceinline__ int32_t dotSignedUnsigned(uint32_t signedBytes, uint32_t unsignedBytes, int32_t acc) {
    int32_t d;
    asm("dp4a.s32.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(signedBytes), "r"(unsignedBytes), "r"(acc));
    return d;
}

__host__ __device__ constexpr size_t codeBytes(int KW, int BT, int planes) { return 2 * static_cast<size_t>(BT) * planes * KW * 4; }

// KW: words of a plane row (H <= 4 KW); BT: rows of a CTA.  One plane (8-bit codes) or two.
template <class Cell, int KW, int BT, int PLANES>
__global__ void __launch_bounds__(16 * KW)
laneRecurrence(const __grid_constant__ Problem p, const __grid_constant__ Cell c) {
    constexpr int KL = KW / 4, kGates = Cell::kGates;   // words of a lane's quarter of K
    static_assert(KL % 4 == 0, "a quarter is read in 16-byte pieces");
    extern __shared__ __align__(16) uint8_t smemL[];
    uint32_t *codes = reinterpret_cast<uint32_t *>(smemL);   // [2][BT][PLANES][KW]
    const uint32_t shared = static_cast<uint32_t>(__cvta_generic_to_shared(smemL)) + static_cast<uint32_t>(codeBytes(KW, BT, PLANES));

    const int H = p.H, tid = threadIdx.x, threads = blockDim.x, lane = tid & 3, first = tid & 28;
    const int unit = min(tid >> 2, H - 1), b0 = static_cast<int>(blockIdx.x) * BT;
    const int rowOf = BT == 1 ? 0 : BT == 2 ? lane >> 1 : lane;   // this lane's row in the cell
    constexpr int kLanes = 4 / BT;                                // lanes that hold the same cell
    const int row = min(b0 + rowOf, p.B - 1), part = lane % kLanes;
    const bool good = c.valid();
    const int kWords = (H + 15) / 16 * 4;

    c.init(smemL + codeBytes(KW, BT, PLANES), tid, threads);
    for (int i = tid; i < 2 * BT * PLANES * KW; i += threads) {
        const int kw = i % KW, plane = i / KW % PLANES, r = i / (PLANES * KW) % BT, buffer = i / (PLANES * KW * BT);
        codes[i] = buffer == 0 && kw < kWords ? p.h0[(static_cast<size_t>(min(b0 + r, p.B - 1)) * PLANES + plane) * kWords + kw] : 0u;
    }
    uint32_t w[kGates][KL];
#pragma unroll
    for (int g = 0; g < kGates; ++g)
#pragma unroll
        for (int i = 0; i < KL; ++i) {
            const int kw = lane * KL + i;
            w[g][i] = kw < kWords ? c.weightWord(g, unit, kw) : 0u;
        }
    const typename Cell::Lane mine = c.lane(shared, lane, unit, lane < kGates);
    typename Cell::State state;
    c.begin(shared, state, row, unit);

    struct Operands {
        typename Cell::Fetch a[BT];
        typename Cell::FetchB b;
    };
    typename Cell::Saved saved[BT];
    auto fetch = [&](int t, Operands &to) {
        const size_t at = static_cast<size_t>(t) * p.B;
        if (lane < kGates) {
#pragma unroll
            for (int r = 0; r < BT; ++r) c.fetch(to.a[r], at, min(b0 + r, p.B - 1), lane, unit);
        }
        c.fetchB(to.b, at, row, unit);
    };
    auto store = [&](int t, const Operands &of) {
        const size_t at = static_cast<size_t>(t) * p.B;
        c.template store<kLanes>(state, of.b, at, row, unit, good, part);
        if (Cell::kSaves && lane < kGates) {
#pragma unroll
            for (int r = 0; r < BT; ++r) c.storeLinear(mine, saved[r], at, min(b0 + r, p.B - 1), lane, unit);
        }
    };
    auto step = [&](int t, Operands &now, Operands &other) {
        __syncthreads();   // the codes of step t
        const uint32_t *from = codes + (t & 1) * (BT * PLANES * KW) + lane * KL;
        int32_t sum[BT];
        if (t > 0) store(t - 1, other);
        if (t + 1 < p.T) fetch(t + 1, other);
#pragma unroll
        for (int r = 0; r < BT; ++r) {
            int32_t part[4] = {0, 0, 0, 0};
#pragma unroll
            for (int plane = 0; plane < PLANES; ++plane) {
                int32_t acc[kGates];
#pragma unroll
                for (int g = 0; g < kGates; ++g) acc[g] = 0;
#pragma unroll
                for (int i = 0; i < KL; i += 4) {
                    const uint4 h = *reinterpret_cast<const uint4 *>(from + (r * PLANES + plane) * KW + i);
#pragma unroll
                    for (int g = 0; g < kGates; ++g) {
                        acc[g] = dotSignedUnsigned(w[g][i], h.x, acc[g]);
                        acc[g] = dotSignedUnsigned(w[g][i + 1], h.y, acc[g]);
                        acc[g] = dotSignedUnsigned(w[g][i + 2], h.z, acc[g]);
                        acc[g] = dotSignedUnsigned(w[g][i + 3], h.w, acc[g]);
                    }
                }
#pragma unroll
                for (int g = 0; g < kGates; ++g) part[g] = (part[g] << 8) + acc[g];
            }
            // add the quarters; lane g ends with gate g
            const bool upper = lane & 2, odd = lane & 1;
            int32_t half[2];
#pragma unroll
            for (int i = 0; i < 2; ++i)
                half[i] = (upper ? part[2 + i] : part[i]) + __shfl_xor_sync(0xffffffffu, upper ? part[i] : part[2 + i], 2);
            sum[r] = (odd ? half[1] : half[0]) + __shfl_xor_sync(0xffffffffu, odd ? half[0] : half[1], 1);
        }
        uint32_t linear[BT];
#pragma unroll
        for (int r = 0; r < BT; ++r) {
            const uint32_t acc[2] = {static_cast<uint32_t>(sum[r] >> 8), static_cast<uint32_t>(sum[r] & 255)};
            linear[r] = c.template linear<1>(shared, mine, now.a[r], acc, saved[r]);
        }
        // all gates of a lane's row
        uint32_t v[4];
        if constexpr (BT == 4) {   // a 4 x 4 transposition among the lanes
            const bool upper = lane & 2, odd = lane & 1;
#pragma unroll
            for (int i = 0; i < 4; i += 2) {
                const uint32_t got = __shfl_xor_sync(0xffffffffu, odd ? linear[i] : linear[i + 1], 1);
                v[i] = odd ? got : linear[i];
                v[i + 1] = odd ? linear[i + 1] : got;
            }
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const uint32_t got = __shfl_xor_sync(0xffffffffu, upper ? v[i] : v[i + 2], 2);
                v[i] = upper ? got : v[i];
                v[i + 2] = upper ? v[i + 2] : got;
            }
        } else {
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                v[g] = __shfl_sync(0xffffffffu, linear[0], first | g);
                if constexpr (BT == 2) {
                    const uint32_t second = __shfl_sync(0xffffffffu, linear[1], first | g);
                    v[g] = rowOf ? second : v[g];
                }
            }
        }
        const uint32_t code = c.cell(shared, state, now.b, v);
        uint8_t *to = reinterpret_cast<uint8_t *>(codes + ((t + 1) & 1) * (BT * PLANES * KW) + rowOf * PLANES * KW) + unit;
        if (PLANES == 2) to[0] = static_cast<uint8_t>(code >> 8);
        to[(PLANES - 1) * 4 * KW] = static_cast<uint8_t>(code);
    };
    Operands even, odd;
    fetch(0, even);
    int t = 0;
#pragma unroll 1
    for (; t + 1 < p.T; t += 2) {
        step(t, even, odd);
        step(t + 1, odd, even);
    }
    if (t < p.T) {
        step(t, even, odd);
        store(t, even);
    } else {
        store(t - 1, odd);
    }
    c.finish(state, row, unit, good);
}

// Rows of a CTA for a batch; 0 where other kernels are the better ones.  Two planes: as few as leave half of the GPU to the
// other direction of a layer, and not four rows of 128 units, whose products take as long as the chain of a cluster.  One
// plane: as few as one wave of CTAs holds, and not four rows of 64 units.
template <int KW, int PLANES>
int rowsFor(int B) {
    const int ctas = std::max(1, PLANES == 2 ? currentDevice().sms / 2 : currentDevice().sms);
    for (int rows : {1, 2, 4})
        if ((B + rows - 1) / rows <= ctas) return rows == 4 && KW == (PLANES == 2 ? 32 : 16) ? 0 : rows;
    return 0;
}

template <class Cell, int KW, int PLANES>
bool launch(const char *name, const Problem &p, const Cell &cell, cudaStream_t st) {
    const int rows = rowsFor<KW, PLANES>(p.B);
    auto run = [&](auto kernel, int BT) {
        const size_t smem = codeBytes(KW, BT, PLANES) + cell.sharedBytes();
        if (smem > static_cast<size_t>(currentDevice().smemMax)) return false;
        ensureDynamicSmem(reinterpret_cast<const void *>(kernel), smem);
        {
            KernelTimer timer__(name, st);
            kernel<<<(p.B + BT - 1) / BT, (4 * p.H + 31) / 32 * 32, smem, st>>>(p, cell);
        }
        afterLaunch(name);
        return true;
    };
    if (rows == 1) return run(laneRecurrence<Cell, KW, 1, PLANES>, 1);
    if (rows == 2) return run(laneRecurrence<Cell, KW, 2, PLANES>, 2);
    if constexpr (KW != (PLANES == 2 ? 32 : 16))
        if (rows == 4) return run(laneRecurrence<Cell, KW, 4, PLANES>, 4);
    return false;
}

}  // namespace lanerec
}  // namespace rxmet
