// Float GRU forward and the calibration forward (float forward + min/max statistics).
//
// Same shape as the quantized path: the input projection for all steps is one kernel, the
// recurrence is ONE launch in which each CTA owns a batch tile for the whole sequence with the
// recurrent weights resident in shared memory when they fit.  The 13 activation statistics are
// accumulated in registers across all steps and leave the kernel as one atomic per CTA and
// statistic, so calibration never re-reads the activations from HBM and never returns to the
// host per tensor.
//
// Reference: operators/quant-gru/src/gru_forward_gpu.cu:359-431 (T x (SGEMM + pointwise)),
// src/calibration_gpu.cu:1847-1953 (one reduction + D2H copy per statistic) and the CPU
// definition of what is observed, src/gru_forward_cpu.cc:58-151.
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cstdint>

#include "common.h"
#include "gru_forward_float.h"

namespace rxmet {
namespace gru {
namespace {

constexpr int kRowsPerBlock = 8;

// Order-preserving float atomics (valid for any finite value, -0.0 included, as long as the
// slot starts at +FLT_MAX / -FLT_MAX).
__device__ __forceinline__ void atomicMinFloat(float *addr, float v) {
    if (v >= 0.0f) atomicMin(reinterpret_cast<int *>(addr), __float_as_int(v));
    else atomicMax(reinterpret_cast<unsigned int *>(addr), __float_as_uint(v));
}
__device__ __forceinline__ void atomicMaxFloat(float *addr, float v) {
    if (v >= 0.0f) atomicMax(reinterpret_cast<int *>(addr), __float_as_int(v));
    else atomicMin(reinterpret_cast<unsigned int *>(addr), __float_as_uint(v));
}

struct MinMax {
    float lo = FLT_MAX, hi = -FLT_MAX;
    __device__ __forceinline__ void see(float v) {
        if (isfinite(v)) {  // only finite values are observed (gru_forward_cpu.cc:17-22)
            lo = fminf(lo, v);
            hi = fmaxf(hi, v);
        }
    }
};

__device__ __forceinline__ MinMax warpReduce(MinMax m) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        m.lo = fminf(m.lo, __shfl_xor_sync(0xffffffffu, m.lo, o));
        m.hi = fmaxf(m.hi, __shfl_xor_sync(0xffffffffu, m.hi, o));
    }
    return m;
}

// Block-wide reduce of `count` statistics held per thread, then one atomic pair per statistic.
// scratch: 2 * count * (blockDim/32) floats of shared memory.
template <int N>
__device__ void commitStats(MinMax (&local)[N], const int (&slot)[N], float *mins, float *maxs, float *scratch) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = (blockDim.x + 31) >> 5;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const MinMax m = warpReduce(local[i]);
        if (lane == 0) {
            scratch[(2 * i) * warps + warp] = m.lo;
            scratch[(2 * i + 1) * warps + warp] = m.hi;
        }
    }
    __syncthreads();
    if (threadIdx.x < N) {
        float lo = FLT_MAX, hi = -FLT_MAX;
        for (int w = 0; w < warps; ++w) {
            lo = fminf(lo, scratch[(2 * threadIdx.x) * warps + w]);
            hi = fmaxf(hi, scratch[(2 * threadIdx.x + 1) * warps + w]);
        }
        if (lo <= hi) {
            atomicMinFloat(&mins[slot[threadIdx.x]], lo);
            atomicMaxFloat(&maxs[slot[threadIdx.x]], hi);
        }
    }
    __syncthreads();
}

struct ParameterStats {
    const float *src[4];   // W, R, bw, br
    int rows[4], C;
    float *mins, *maxs;    // packed statistics: kOps scalar slots, then four blocks of C
};
// Per-column min/max of the parameters (blockIdx.y: which one); the scalar slots, which later kernels reach by atomics,
// start empty.
__global__ void observeParameters(const ParameterStats p) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x, which = blockIdx.y;
    if (which == 0 && c < kOps) {
        p.mins[c] = FLT_MAX;
        p.maxs[c] = -FLT_MAX;
    }
    if (c >= p.C) return;
    MinMax m;
    for (int r = 0; r < p.rows[which]; ++r) m.see(p.src[which][static_cast<size_t>(r) * p.C + c]);
    if (m.lo > m.hi) m.lo = m.hi = 0.0f;  // nothing finite: observes 0 (gru_forward_cpu.cc:24)
    p.mins[kOps + which * p.C + c] = m.lo;
    p.maxs[kOps + which * p.C + c] = m.hi;
}

// wx[n, c] = sum_k x[n,k] W[k,c] + bw[c] for all T*B rows.
__global__ void inputLinearFloat(const float *__restrict__ x, int rows, int K, int C, const float *__restrict__ W,
                                 const float *__restrict__ bw, float *__restrict__ out, float *mins, float *maxs) {
    extern __shared__ float smemF[];
    float *xs = smemF;                        // [kRowsPerBlock][K]
    float *scratch = smemF + kRowsPerBlock * K;  // 2 * 2 * warps
    const int row0 = blockIdx.x * kRowsPerBlock;
    const int nRows = min(kRowsPerBlock, rows - row0);
    MinMax m[2];   // wx, x
    for (int i = threadIdx.x; i < kRowsPerBlock * K; i += blockDim.x) {
        const int r = i / K;
        xs[i] = r < nRows ? x[static_cast<size_t>(row0 + r) * K + (i % K)] : 0.0f;
        if (r < nRows) m[1].see(xs[i]);
    }
    __syncthreads();
    for (int c = threadIdx.x; c < C; c += blockDim.x) {
        float acc[kRowsPerBlock];
#pragma unroll
        for (int r = 0; r < kRowsPerBlock; ++r) acc[r] = 0.0f;
        for (int k = 0; k < K; ++k) {
            const float w = W[static_cast<size_t>(k) * C + c];
#pragma unroll
            for (int r = 0; r < kRowsPerBlock; ++r) acc[r] = fmaf(xs[r * K + k], w, acc[r]);
        }
        const float b = bw[c];
#pragma unroll
        for (int r = 0; r < kRowsPerBlock; ++r) {
            if (r < nRows) {
                const float val = acc[r] + b;
                out[static_cast<size_t>(row0 + r) * C + c] = val;
                m[0].see(val);
            }
        }
    }
    if (mins) {
        const int slots[2] = {RXMET_GRU_WEIGHT_IH_LINEAR, RXMET_GRU_X};
        commitStats<2>(m, slots, mins, maxs, scratch);
    }
}

struct FloatRecurrentArgs {
    int T, B, H;
    int weightsInSmem;
    const float *R;   // [H][3H]
    const float *br;  // [3H]
    const float *wx;  // [T][B][3H] = W x + bw
    const float *h0;  // [B][H] or null
    float *h;         // [T+1][B][H]
    float *v;         // [T][B][4H]
    float *mins, *maxs;  // packed statistics or null
    float *trRh, *trPre, *trMul;  // optional [T][B][3H] traces
};

template <int BT>
__global__ void __launch_bounds__(768) recurrentFloat(const __grid_constant__ FloatRecurrentArgs a) {
    const int H = a.H, C = 3 * a.H;
    extern __shared__ float smemF[];
    float *hS = smemF;                 // [BT][H]
    float *rhS = hS + BT * H;          // [BT][C] = R h + br
    float *scratch = rhS + BT * C;     // 2 * 12 * warps
    float *RS = scratch + 2 * 12 * 32; // [H][C] when resident
    const int tid = threadIdx.x, nthreads = blockDim.x;
    const int b0 = blockIdx.x * BT, nb = min(BT, a.B - b0);

    const float *Rsrc = a.R;
    if (a.weightsInSmem) {
        for (int i = tid; i < H * C; i += nthreads) RS[i] = a.R[i];
        Rsrc = RS;
    }
    for (int i = tid; i < BT * H; i += nthreads) {
        const int b = i / H;
        hS[i] = (b < nb && a.h0) ? a.h0[static_cast<size_t>(b0 + b) * H + (i % H)] : 0.0f;
    }
    __syncthreads();
    for (int i = tid; i < nb * H; i += nthreads) a.h[static_cast<size_t>(b0 + i / H) * H + (i % H)] = hS[i];

    // statistic order: h, Rh, z_pre, r_pre, n_pre, z, r, n, r*rec, (1-z)*n, z*h_old  (+ unused)
    MinMax st[12];
    for (int t = 0; t < a.T; ++t) {
        const size_t rowBase = static_cast<size_t>(t) * a.B + b0;
        for (int c = tid; c < C; c += nthreads) {
            float acc[BT];
#pragma unroll
            for (int b = 0; b < BT; ++b) acc[b] = 0.0f;
            for (int k = 0; k < H; ++k) {
                const float w = Rsrc[static_cast<size_t>(k) * C + c];
#pragma unroll
                for (int b = 0; b < BT; ++b) acc[b] = fmaf(hS[b * H + k], w, acc[b]);
            }
            const float bias = a.br[c];
#pragma unroll
            for (int b = 0; b < BT; ++b) {
                const float val = acc[b] + bias;
                rhS[b * C + c] = val;
                if (b < nb) {
                    st[1].see(val);
                    if (a.trRh) a.trRh[(rowBase + b) * C + c] = val;
                }
            }
        }
        __syncthreads();
        for (int i = tid; i < nb * H; i += nthreads) {
            const int b = i / H, j = i % H;
            const size_t row = rowBase + b;
            const float *wx = a.wx + row * C;
            const float *rh = rhS + b * C;
            const float zPre = wx[j] + rh[j];
            const float rPre = wx[H + j] + rh[H + j];
            const float z = 1.0f / (1.0f + expf(-zPre));
            const float r = 1.0f / (1.0f + expf(-rPre));
            const float rec = rh[2 * H + j];
            const float rm = r * rec;
            const float nPre = wx[2 * H + j] + rm;
            const float n = tanhf(nPre);
            const float hOld = hS[b * H + j];
            const float oldC = z * hOld;
            const float newC = (1.0f - z) * n;
            const float hNew = oldC + newC;
            hS[b * H + j] = hNew;
            a.h[(row + a.B) * H + j] = hNew;
            float *vRow = a.v + row * 4 * H;
            vRow[j] = z; vRow[H + j] = r; vRow[2 * H + j] = n; vRow[3 * H + j] = rec;
            if (a.trPre) {
                float *pre = a.trPre + row * C, *mul = a.trMul + row * C;
                pre[j] = zPre; pre[H + j] = rPre; pre[2 * H + j] = nPre;
                mul[j] = rm; mul[H + j] = newC; mul[2 * H + j] = oldC;
            }
            st[0].see(hNew); st[2].see(zPre); st[3].see(rPre); st[4].see(nPre);
            st[5].see(z); st[6].see(r); st[7].see(n); st[8].see(rm); st[9].see(newC); st[10].see(oldC);
        }
        __syncthreads();
    }
    if (a.mins) {
        const int slots[12] = {RXMET_GRU_H, RXMET_GRU_WEIGHT_HH_LINEAR, RXMET_GRU_UPDATE_GATE_INPUT,
                               RXMET_GRU_RESET_GATE_INPUT, RXMET_GRU_NEW_GATE_INPUT, RXMET_GRU_UPDATE_GATE_OUTPUT,
                               RXMET_GRU_RESET_GATE_OUTPUT, RXMET_GRU_NEW_GATE_OUTPUT, RXMET_GRU_MUL_RESET_HIDDEN,
                               RXMET_GRU_MUL_NEW_CONTRIBUTION, RXMET_GRU_MUL_OLD_CONTRIBUTION, RXMET_GRU_H};
        commitStats<12>(st, slots, a.mins, a.maxs, scratch);
    }
}

// Up to 128 hidden units: four lanes of a warp own a unit, as in recurrentLanesI8 (gru_forward_quant.cu).  Each multiplies a
// quarter of K for the three gates - 16 rows of its quarter in registers, the others in shared memory, laid out so that a
// warp reads 512 consecutive bytes - shuffles add the quarters and the cell follows in the same registers: one barrier per
// step instead of two, no thread walks all of K.  Lanes beyond the last unit or row repeat the last one.  The terms of the
// next step are loaded one step ahead, outputs of a step are stored under the products of the next.
// T = 98, B = 32, H = 64 with statistics: 214 -> 68 us.
template <int QUADS, int BT, bool Stats>   // QUADS: groups of four rows in a lane's quarter (H <= 16 QUADS)
__global__ void __launch_bounds__(256 * ((QUADS + 3) / 4))
recurrentFloatLanes(const __grid_constant__ FloatRecurrentArgs a) {
    constexpr int kResident = QUADS < 4 ? QUADS : 4, kLanes = 4 / BT, kPadded = 16 * QUADS;
    __shared__ __align__(16) float hS[2][BT][kPadded];
    __shared__ float scratch[2 * 11 * 32];
    extern __shared__ __align__(16) float smemF[];
    float4 *wS = reinterpret_cast<float4 *>(smemF);   // [QUADS - kResident][3][threads]
    const int H = a.H, C = 3 * a.H, tid = threadIdx.x, threads = blockDim.x;
    const int j = min(tid >> 2, H - 1), lane = tid & 3, row = lane / kLanes, part = lane % kLanes;
    const int b0 = blockIdx.x * BT, batch = min(b0 + row, a.B - 1);

    float4 w[kResident][3];
#pragma unroll
    for (int q = 0; q < QUADS; ++q)
#pragma unroll
        for (int g = 0; g < 3; ++g) {
            float v[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int k = lane * (4 * QUADS) + 4 * q + e;
                v[e] = k < H ? a.R[static_cast<size_t>(k) * C + g * H + j] : 0.0f;
            }
            const float4 packed = make_float4(v[0], v[1], v[2], v[3]);
            if (q < kResident) w[q < kResident ? q : 0][g] = packed;
            else wS[((q - kResident) * 3 + g) * threads + tid] = packed;
        }
    float bias[3];
#pragma unroll
    for (int g = 0; g < 3; ++g) bias[g] = a.br[g * H + j];
    for (int i = tid; i < BT * kPadded; i += threads) {
        const int b = i / kPadded, k = i % kPadded;
        const float v = (k < H && a.h0) ? a.h0[static_cast<size_t>(min(b0 + b, a.B - 1)) * H + k] : 0.0f;
        hS[0][b][k] = v;
        hS[1][b][k] = 0.0f;
        if (k < H && b0 + b < a.B) a.h[static_cast<size_t>(b0 + b) * H + k] = v;
    }
    float hOld = a.h0 ? a.h0[static_cast<size_t>(batch) * H + j] : 0.0f;

    const uint32_t offH = static_cast<uint32_t>(batch) * H + j, offC = static_cast<uint32_t>(batch) * C + j;
    const uint32_t offV = static_cast<uint32_t>(batch) * 4 * H + j;
    const size_t stepH = static_cast<size_t>(a.B) * H;
    const float *wxNext = a.wx;
    float wx[3];
    auto fetch = [&](bool more) {
#pragma unroll
        for (int g = 0; g < 3; ++g) wx[g] = (wxNext + g * H)[offC];
        if (more) wxNext += 3 * stepH;
    };
    fetch(a.T > 1);
    MinMax st[11];   // h, Rh, z_pre, r_pre, n_pre, z, r, n, r*rec, (1-z)*n, z*h_old
    float out[5] = {};   // z, r, n, rec, h of the step before
    size_t stored = 0;
    auto store = [&] {
        if (part == 0) (a.h + stored + stepH)[offH] = out[4];
#pragma unroll
        for (int k = 0; k < 4; k += kLanes) {
            float value = out[k];
#pragma unroll
            for (int l = 1; l < kLanes; ++l) value = part == l ? out[k + l] : value;
            (a.v + 4 * stored + k * H)[offV + part * H] = value;
        }
        stored += stepH;
    };
#pragma unroll 1
    for (int t = 0; t < a.T; ++t) {
        __syncthreads();
        const float *hNow = &hS[t & 1][0][lane * (4 * QUADS)];
        float acc[BT][3];
#pragma unroll
        for (int b = 0; b < BT; ++b)
#pragma unroll
            for (int g = 0; g < 3; ++g) acc[b][g] = 0.0f;
#pragma unroll
        for (int q = 0; q < QUADS; ++q) {
            float4 wq[3];
#pragma unroll
            for (int g = 0; g < 3; ++g) wq[g] = q < kResident ? w[q < kResident ? q : 0][g] : wS[((q - kResident) * 3 + g) * threads + tid];
#pragma unroll
            for (int b = 0; b < BT; ++b) {
                const float4 hv = *reinterpret_cast<const float4 *>(hNow + b * kPadded + 4 * q);
#pragma unroll
                for (int g = 0; g < 3; ++g) {
                    acc[b][g] = fmaf(hv.x, wq[g].x, acc[b][g]);
                    acc[b][g] = fmaf(hv.y, wq[g].y, acc[b][g]);
                    acc[b][g] = fmaf(hv.z, wq[g].z, acc[b][g]);
                    acc[b][g] = fmaf(hv.w, wq[g].w, acc[b][g]);
                }
            }
        }
        if (t > 0) store();
        float rh[3];
#pragma unroll
        for (int g = 0; g < 3; ++g) {
            float s;
            if constexpr (BT == 1) {
                s = acc[0][g] + __shfl_xor_sync(0xffffffffu, acc[0][g], 2);
                s += __shfl_xor_sync(0xffffffffu, s, 1);
            } else if constexpr (BT == 2) {
                s = ((lane & 2) ? acc[1][g] : acc[0][g]) + __shfl_xor_sync(0xffffffffu, (lane & 2) ? acc[0][g] : acc[1][g], 2);
                s += __shfl_xor_sync(0xffffffffu, s, 1);
            } else {
                float half[2];
#pragma unroll
                for (int i = 0; i < 2; ++i)
                    half[i] = ((lane & 2) ? acc[i + 2][g] : acc[i][g]) + __shfl_xor_sync(0xffffffffu, (lane & 2) ? acc[i][g] : acc[i + 2][g], 2);
                s = ((lane & 1) ? half[1] : half[0]) + __shfl_xor_sync(0xffffffffu, (lane & 1) ? half[0] : half[1], 1);
            }
            rh[g] = s + bias[g];
            if (Stats) st[1].see(rh[g]);
        }
        const float zPre = wx[0] + rh[0], rPre = wx[1] + rh[1];
        const float z = 1.0f / (1.0f + expf(-zPre)), r = 1.0f / (1.0f + expf(-rPre));
        // no contraction: the variant with statistics, which needs the products themselves, has to give the same bits
        const float rec = rh[2], rm = __fmul_rn(r, rec), nPre = __fadd_rn(wx[2], rm), n = tanhf(nPre);
        const float oldC = __fmul_rn(z, hOld), newC = __fmul_rn(1.0f - z, n), hNew = __fadd_rn(oldC, newC);
        hS[(t + 1) & 1][row][j] = hNew;
        if (t + 1 < a.T) fetch(t + 2 < a.T);
        hOld = hNew;
        out[0] = z; out[1] = r; out[2] = n; out[3] = rec; out[4] = hNew;
        if (a.trRh || a.trPre) {
            const size_t at = 3 * static_cast<size_t>(t) * stepH + offC;
            if (a.trRh) { a.trRh[at] = rh[0]; a.trRh[at + H] = rh[1]; a.trRh[at + 2 * H] = rh[2]; }
            if (a.trPre) {
                a.trPre[at] = zPre; a.trPre[at + H] = rPre; a.trPre[at + 2 * H] = nPre;
                a.trMul[at] = rm; a.trMul[at + H] = newC; a.trMul[at + 2 * H] = oldC;
            }
        }
        if (Stats) {
            st[0].see(hNew); st[2].see(zPre); st[3].see(rPre); st[4].see(nPre);
            st[5].see(z); st[6].see(r); st[7].see(n); st[8].see(rm); st[9].see(newC); st[10].see(oldC);
        }
    }
    store();
    if (Stats) {
        const int slots[11] = {RXMET_GRU_H, RXMET_GRU_WEIGHT_HH_LINEAR, RXMET_GRU_UPDATE_GATE_INPUT, RXMET_GRU_RESET_GATE_INPUT,
                               RXMET_GRU_NEW_GATE_INPUT, RXMET_GRU_UPDATE_GATE_OUTPUT, RXMET_GRU_RESET_GATE_OUTPUT,
                               RXMET_GRU_NEW_GATE_OUTPUT, RXMET_GRU_MUL_RESET_HIDDEN, RXMET_GRU_MUL_NEW_CONTRIBUTION,
                               RXMET_GRU_MUL_OLD_CONTRIBUTION};
        commitStats<11>(st, slots, a.mins, a.maxs, scratch);
    }
}

template <int QUADS, int BT>
void launchLanes(const FloatRecurrentArgs &a, cudaStream_t st) {
    const int threads = (4 * a.H + 31) / 32 * 32;
    const size_t smem = sizeof(float4) * 3 * std::max(0, QUADS - 4) * threads;
    auto kernel = a.mins ? recurrentFloatLanes<QUADS, BT, true> : recurrentFloatLanes<QUADS, BT, false>;
    ensureDynamicSmem(reinterpret_cast<const void *>(kernel), smem);
    {
        KernelTimer timer__("recurrentFloat", st);
        kernel<<<(a.B + BT - 1) / BT, threads, smem, st>>>(a);
    }
    afterLaunch("recurrentFloat");
}
template <int QUADS>
void launchLanes(const FloatRecurrentArgs &a, int sms, cudaStream_t st) {
    if (a.B > 2 * sms) launchLanes<QUADS, 4>(a, st);
    else if (a.B > sms) launchLanes<QUADS, 2>(a, st);
    else launchLanes<QUADS, 1>(a, st);
}

}  // namespace

size_t statsFloats(int H) { return 2 * (static_cast<size_t>(kOps) + 12 * static_cast<size_t>(H)); }

size_t forwardFloatWorkspaceBytes(int T, int B, int I, int H) {
    (void)I;
    WorkspaceSizer ws;
    ws.take<float>(static_cast<size_t>(T) * B * 3 * H);
    ws.take<float>(statsFloats(H));
    return ws.used() + 1024;
}

void forwardFloat(const ForwardFloatCall &call, void *workspace, size_t workspaceBytes, cudaStream_t st) {
    const int T = call.T, B = call.B, I = call.I, H = call.H, C = 3 * H;
    const size_t rows = static_cast<size_t>(T) * B;
    Workspace ws(workspace, workspaceBytes);
    float *wx = ws.take<float>(rows * C);
    if (call.traceWx) wx = call.traceWx;
    float *mins = nullptr, *maxs = nullptr;
    const size_t half = statsFloats(H) / 2;
    if (call.stats) {
        mins = call.stats;
        maxs = call.stats + half;
        const ParameterStats p{{call.W, call.R, call.bw, call.br}, {I, H, 1, 1}, C, mins, maxs};
        {
            KernelTimer timer__("columnMinMax", st);
            observeParameters<<<dim3((C + 127) / 128, 4), 128, 0, st>>>(p);
        }
        afterLaunch("observeParameters");
    }
    {
        const int block = std::min((C + 31) / 32 * 32, 512);
        const size_t smem = sizeof(float) * (kRowsPerBlock * I + 2 * 2 * (block / 32));   // rows, scratch of two statistics
        {
            KernelTimer timer__("inputLinearFloat", st);
            inputLinearFloat<<<static_cast<int>((rows + kRowsPerBlock - 1) / kRowsPerBlock), block, smem, st>>>(
                call.x, static_cast<int>(rows), I, C, call.W, call.bw, wx, mins, maxs);
        }
        afterLaunch("inputLinearFloat");
    }
    FloatRecurrentArgs a{};
    a.T = T; a.B = B; a.H = H;
    a.R = call.R; a.br = call.br; a.wx = wx; a.h0 = call.h0; a.h = call.h; a.v = call.v;
    a.mins = mins; a.maxs = maxs;
    a.trRh = call.traceRh; a.trPre = call.tracePre; a.trMul = call.traceMul;
    RXMET_REQUIRE((call.tracePre == nullptr) == (call.traceMul == nullptr), "pre-activation and product traces go together");
    const int smemMax = currentDevice().smemMax, sms = currentDevice().sms;
    // offsets inside a step are 32 bits wide
    if (H <= 128 && static_cast<size_t>(B) * H < (size_t{1} << 28)) {
        if (H <= 32) launchLanes<2>(a, sms, st);
        else if (H <= 64) launchLanes<4>(a, sms, st);
        else launchLanes<8>(a, sms, st);
        return;
    }
    const int bt = (B >= 8 * sms) ? 4 : ((B >= 4 * sms) ? 2 : 1);
    const int block = std::min((C + 31) / 32 * 32, 768);
    auto launch = [&](auto kernel, int BT) {
        const size_t base = sizeof(float) * (static_cast<size_t>(BT) * H + static_cast<size_t>(BT) * C + 2 * 12 * 32);
        const size_t full = base + sizeof(float) * static_cast<size_t>(H) * C;
        a.weightsInSmem = full <= static_cast<size_t>(smemMax) ? 1 : 0;
        const size_t smem = a.weightsInSmem ? full : base;
        if (smem > static_cast<size_t>(smemMax))
            fail(RXMET_ERR_UNSUPPORTED, "hidden size %d needs %zu bytes of shared memory per CTA", H, smem);
        ensureDynamicSmem(reinterpret_cast<const void *>(kernel), smem);
        {
            KernelTimer timer__("recurrentFloat", st);
            kernel<<<(B + BT - 1) / BT, block, smem, st>>>(a);
        }
        afterLaunch("recurrentFloat");
    };
    if (bt == 4) launch(recurrentFloat<4>, 4);
    else if (bt == 2) launch(recurrentFloat<2>, 2);
    else launch(recurrentFloat<1>, 1);
}

}  // namespace gru
}  // namespace rxmet
