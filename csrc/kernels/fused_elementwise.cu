// Memory-bound pieces of a decoder layer as single-pass sm_100a kernels (bf16 storage, fp32 math): residual add +
// RMSNorm (forward and backward), SwiGLU (forward and backward) and rotary embedding.  They replace chains of
// framework element-wise kernels around the fused matmul kernels: each tensor is read once and written once.
// The reference has no counterpart (it is a communication library); these serve the TP + SP decoder stack that the
// MC2 kernels are benchmarked in.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>
#include <cstring>
#include "hccl/hccl_fused_ops.h"
#include "../core/log.h"
#include "../core/per_device.h"
#include "dependent_launch.cuh"

namespace hccl {
namespace {

constexpr uint32_t kNormMaxHidden = 8192;      // a row stays in the registers of one group of threads
constexpr uint64_t kNormMaxRows = 0x7FFFFFFF;  // row numbers are 32-bit

__device__ __forceinline__ void Unpack8(const uint4& raw, float* f)
{
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float2 v = __bfloat1622float2(h[k]);
        f[2 * k] = v.x;
        f[2 * k + 1] = v.y;
    }
}
__device__ __forceinline__ uint4 Pack8(const float* f)
{
    uint4 o;
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
    for (int k = 0; k < 4; ++k) h[k] = __floats2bfloat162_rn(f[2 * k], f[2 * k + 1]);
    return o;
}
__device__ __forceinline__ void CopyAsync16(uint32_t smemDst, const void* src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smemDst), "l"(src) : "memory");
}
__device__ __forceinline__ void CopyAsyncCommit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING> __device__ __forceinline__ void CopyAsyncWait() { asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory"); }

// Rows and threads of the two norm kernels.  A row is handled by a GROUP of threads, two 16-byte vectors per thread (32
// threads up to 512 elements, 512 threads at 8192); a CTA holds `nGroups` groups, group g of CTA b works on rows
// b * nGroups + g, + gridDim.x * nGroups, ...  Both kernels are bound by HBM as long as enough bytes are in flight: a row
// is read, reduced over all of its threads and only then written, so a kernel that loads a row into registers between
// its block-wide sums keeps loads in flight for a fraction of the time only.  Here every thread owns a ring of
// kNormSlots rows of its own vectors in shared memory, filled by asynchronous copies three rows ahead of the arithmetic
// (no hand-over between threads: a thread reads what it copied itself).  One barrier of the group per row completes the
// row's sum.  Measured at 4096 x 8192 against one CTA of 256 threads per row (forward) and 296 CTAs that walk the rows
// (backward): forward 51.4 -> 45.2 us (268 MB, 5.9 TB/s), backward with its partial sums 105.6 -> 53.4 us (268 MB);
// 8192 x 4096 45.3 -> 45.8 and 111.6 -> 51.6 us; 8192 x 128 12.4 -> 6.3 and 39.1 -> 8.3 us; 16 x 8192 6.3 -> 4.3 and
// 10.4 -> 8.3 us.
constexpr int kNormSlots = 4;
constexpr int kNormThreads = 512;
constexpr int kNormMaxGroups = kNormThreads / 32;
constexpr uint32_t kNormPartBytes = 2 * kNormMaxGroups * 16 * sizeof(float);      // [row parity][group][warp of the group]

// Sum over the threads of a group.  Two copies of the per-warp sums in turn: slower warps of the group may still be
// reading the previous row's.
__device__ __forceinline__ float GroupSum(float v, uint8_t* smem, int parity, int group, int groupThreads, int tid)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    const int groupWarps = groupThreads / 32;
    if (groupWarps == 1) return v;
    float* part = reinterpret_cast<float*>(smem) + (parity * kNormMaxGroups + group) * 16;
    if ((tid & 31) == 0) part[tid >> 5] = v;
    asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "r"(groupThreads) : "memory");
    float sum = 0.f;
    for (int q = 0; q < groupWarps; q += 2) {
        const float2 two = *reinterpret_cast<const float2*>(part + q);
        sum += two.x + two.y;
    }
    return sum;
}

// xOut = x + delta (DELTA), h = xOut * rstd * w, rstd[row] = rsqrt(mean(xOut^2) + eps).
template <bool DELTA>
__global__ void __launch_bounds__(kNormThreads, 1) AddRmsNormFwdKernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ delta,
                                                                       const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ xOut,
                                                                       __nv_bfloat16* __restrict__ h, float* __restrict__ rstd, int rows, int hidden,
                                                                       int groupThreads, float eps)
{
    DependencyWait();
    AllowDependents();
    extern __shared__ __align__(128) uint8_t smem[];
    const int nVec = hidden / 8;
    const int group = threadIdx.x / groupThreads, nGroups = blockDim.x / groupThreads, tid = threadIdx.x % groupThreads;
    const uint32_t rowBytes = (uint32_t)hidden * 2, slotBytes = rowBytes * (DELTA ? 2 : 1);
    uint8_t* ring = smem + kNormPartBytes + (size_t)group * kNormSlots * slotBytes;
    const uint32_t ringAddr = (uint32_t)__cvta_generic_to_shared(ring);
    const int first = (int)blockIdx.x * nGroups + group, stride = (int)gridDim.x * nGroups;
    const int nMine = first < rows ? (rows - 1 - first) / stride + 1 : 0;
    auto fill = [&](int i) {                          // this thread's vectors of its group's row number i -> slot i % kNormSlots
        if (i < nMine) {
            const size_t off = ((size_t)first + (size_t)i * stride) * hidden;
            const uint32_t slot = ringAddr + (uint32_t)(i % kNormSlots) * slotBytes;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int v = tid + j * groupThreads;
                if (v < nVec) {
                    CopyAsync16(slot + v * 16, x + off + v * 8);
                    if (DELTA) CopyAsync16(slot + rowBytes + v * 16, delta + off + v * 8);
                }
            }
        }
        CopyAsyncCommit();
    };
    for (int i = 0; i < kNormSlots - 1; ++i) fill(i);
    uint4 wv[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int v = tid + j * groupThreads;
        wv[j] = v < nVec ? reinterpret_cast<const uint4*>(w)[v] : make_uint4(0, 0, 0, 0);
    }
    for (int i = 0; i < nMine; ++i) {
        const size_t row = (size_t)first + (size_t)i * stride;
        const uint8_t* slot = ring + (size_t)(i % kNormSlots) * slotBytes;
        fill(i + kNormSlots - 1);                     // into the slot of row i - 1, which this thread has finished with
        CopyAsyncWait<kNormSlots - 1>();              // row i is here
        float vals[2][8];
        float ss = 0.f;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int v = tid + j * groupThreads;
            if (v < nVec) {
                Unpack8(reinterpret_cast<const uint4*>(slot)[v], vals[j]);
                if (DELTA) {
                    float d[8];
                    Unpack8(reinterpret_cast<const uint4*>(slot + rowBytes)[v], d);
#pragma unroll
                    for (int k = 0; k < 8; ++k) vals[j][k] += d[k];
                    // the sum is stored in bf16 and the norm is taken of the stored value, as the unfused ops would
                    const uint4 packed = Pack8(vals[j]);
                    reinterpret_cast<uint4*>(xOut + row * hidden)[v] = packed;
                    Unpack8(packed, vals[j]);
                }
#pragma unroll
                for (int k = 0; k < 8; ++k) ss += vals[j][k] * vals[j][k];
            }
        }
        const float r = rsqrtf(GroupSum(ss, smem, i & 1, group, groupThreads, tid) / (float)hidden + eps);
        if (tid == 0) rstd[row] = r;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int v = tid + j * groupThreads;
            if (v < nVec) {
                float wf[8], o[8];
                Unpack8(wv[j], wf);
#pragma unroll
                for (int k = 0; k < 8; ++k) o[k] = vals[j][k] * r * wf[k];
                reinterpret_cast<uint4*>(h + row * hidden)[v] = Pack8(o);
            }
        }
    }
}

// Backward of h = x * rstd * w (+ the gradient that reaches x through the residual path, dxExtra, when given):
//   dx = rstd * (dh * w) - x * rstd^3 * mean(dh * w * x) + dxExtra
//   dw = sum over rows of dh * x * rstd        (per-CTA partial sums in dwPartial[gridDim.x][hidden], fp32)
//   dxCopy: a second copy of dx, when given (two leaves that each keep a gradient of their own: written from the same registers
//           it costs a store instead of the load and store of a copy kernel: 4096 x 8192 forward and backward 120.6 -> 108.5 us)
//
// Rows are taken from the last to the first: what the kernels in front have read and written last, the stream and the gradient that
// comes in, is still in L2 at the matrix's end.  4096 x 8192 forward and backward, back to back in a graph 101.8 -> 100.1 us, 8192 x 4096
// 104.9 -> 102.1; 4096 x 1024, all of which fits L2, 22.9 -> 23.1.  (Inputs of the forward pass loaded "evict first" made that pass slower,
// 43.0 -> 44.5 us; SwiGLU's backward pass from the end 283.6 -> 283.4.)
//
// dw accumulates in registers over a group's rows, the groups of a CTA are added through shared memory in group order,
// the CTAs' partials by ReducePartialsKernel: the order of the sums depends on the sizes only.
template <bool EXTRA>
__global__ void __launch_bounds__(kNormThreads, 1) RmsNormBwdKernel(const __nv_bfloat16* __restrict__ dh, const __nv_bfloat16* __restrict__ x,
                                                                   const __nv_bfloat16* __restrict__ w, const float* __restrict__ rstd,
                                                                   const __nv_bfloat16* __restrict__ dxExtra, __nv_bfloat16* __restrict__ dx,
                                                                   __nv_bfloat16* __restrict__ dxCopy, float* __restrict__ dwPartial, int rows,
                                                                   int hidden, int groupThreads)
{
    DependencyWait();
    AllowDependents();
    extern __shared__ __align__(128) uint8_t smem[];
    const int nVec = hidden / 8;
    const int group = threadIdx.x / groupThreads, nGroups = blockDim.x / groupThreads, tid = threadIdx.x % groupThreads;
    const uint32_t rowBytes = (uint32_t)hidden * 2, slotBytes = rowBytes * (EXTRA ? 3 : 2);
    uint8_t* ring = smem + kNormPartBytes + (size_t)group * kNormSlots * slotBytes;
    const uint32_t ringAddr = (uint32_t)__cvta_generic_to_shared(ring);
    const int first = (int)blockIdx.x * nGroups + group, stride = (int)gridDim.x * nGroups;
    const int nMine = first < rows ? (rows - 1 - first) / stride + 1 : 0;
    const size_t last = (size_t)rows - 1 - (size_t)first;      // rows are taken from the end (see above)
    auto fill = [&](int i) {                          // this thread's vectors of its group's row number i -> slot i % kNormSlots
        if (i < nMine) {
            const size_t off = (last - (size_t)i * stride) * hidden;
            const uint32_t slot = ringAddr + (uint32_t)(i % kNormSlots) * slotBytes;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int v = tid + j * groupThreads;
                if (v < nVec) {
                    CopyAsync16(slot + v * 16, dh + off + v * 8);
                    CopyAsync16(slot + rowBytes + v * 16, x + off + v * 8);
                    if (EXTRA) CopyAsync16(slot + 2 * rowBytes + v * 16, dxExtra + off + v * 8);
                }
            }
        }
        CopyAsyncCommit();
    };
    for (int i = 0; i < kNormSlots - 1; ++i) fill(i);
    uint4 wv[2];
    float dwAcc[2][8];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int v = tid + j * groupThreads;
        wv[j] = v < nVec ? reinterpret_cast<const uint4*>(w)[v] : make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int k = 0; k < 8; ++k) dwAcc[j][k] = 0.f;
    }
    float rNext = nMine > 0 ? rstd[last] : 0.f;       // one row ahead: its latency is not part of a row's chain
    for (int i = 0; i < nMine; ++i) {
        const size_t row = last - (size_t)i * stride;
        const float r = rNext;
        if (i + 1 < nMine) rNext = rstd[row - stride];
        const uint8_t* slot = ring + (size_t)(i % kNormSlots) * slotBytes;
        fill(i + kNormSlots - 1);                      // into the slot of row i - 1, which this thread has finished with
        CopyAsyncWait<kNormSlots - 1>();               // row i is here
        float g[2][8], xs[2][8];
        float dot = 0.f;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int v = tid + j * groupThreads;
            if (v < nVec) {
                float wf[8];
                Unpack8(reinterpret_cast<const uint4*>(slot)[v], g[j]);
                Unpack8(reinterpret_cast<const uint4*>(slot + rowBytes)[v], xs[j]);
                Unpack8(wv[j], wf);
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    dwAcc[j][k] += g[j][k] * xs[j][k] * r;
                    g[j][k] *= wf[k];
                    dot += g[j][k] * xs[j][k];
                }
            }
        }
        const float c = GroupSum(dot, smem, i & 1, group, groupThreads, tid) / (float)hidden * r * r * r;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int v = tid + j * groupThreads;
            if (v < nVec) {
                float o[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) o[k] = r * g[j][k] - xs[j][k] * c;
                if (EXTRA) {
                    float e[8];
                    Unpack8(reinterpret_cast<const uint4*>(slot + 2 * rowBytes)[v], e);
#pragma unroll
                    for (int k = 0; k < 8; ++k) o[k] += e[k];
                }
                const uint4 packed = Pack8(o);
                reinterpret_cast<uint4*>(dx + row * hidden)[v] = packed;
                if (dxCopy != nullptr) reinterpret_cast<uint4*>(dxCopy + row * hidden)[v] = packed;
            }
        }
    }
    // the ring is idle (every row that was copied has been read): the groups' sums are added there
    __syncthreads();
    float* acc = reinterpret_cast<float*>(smem + kNormPartBytes);
    if (nGroups > 1) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int v = tid + j * groupThreads;
            if (v < nVec) {
                float4* p = reinterpret_cast<float4*>(acc + (size_t)group * hidden + (size_t)v * 8);
                p[0] = make_float4(dwAcc[j][0], dwAcc[j][1], dwAcc[j][2], dwAcc[j][3]);
                p[1] = make_float4(dwAcc[j][4], dwAcc[j][5], dwAcc[j][6], dwAcc[j][7]);
            }
        }
        __syncthreads();
        for (int h = threadIdx.x; h < hidden; h += blockDim.x) {
            float s = 0.f;
            for (int q = 0; q < nGroups; ++q) s += acc[(size_t)q * hidden + h];
            dwPartial[(size_t)blockIdx.x * hidden + h] = s;
        }
    } else {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int v = tid + j * groupThreads;
            if (v < nVec) {
                float4* p = reinterpret_cast<float4*>(dwPartial + (size_t)blockIdx.x * hidden + (size_t)v * 8);
                p[0] = make_float4(dwAcc[j][0], dwAcc[j][1], dwAcc[j][2], dwAcc[j][3]);
                p[1] = make_float4(dwAcc[j][4], dwAcc[j][5], dwAcc[j][6], dwAcc[j][7]);
            }
        }
    }
}

// dw[h] = sum of the CTAs' partials, in a fixed order.  32 columns per block (one 128-byte line of every partial row),
// kReduceRows threads share a column's partials and are added through shared memory; at 148 partials of 8192 columns
// that is 256 blocks of 16 warps instead of one thread per column walking all partials.
constexpr int kReduceRows = 16;
__global__ void __launch_bounds__(32 * kReduceRows) ReducePartialsKernel(const float* __restrict__ partial, __nv_bfloat16* __restrict__ dw, int nPartials, int hidden)
{
    DependencyWait();
    AllowDependents();
    __shared__ float s_sum[kReduceRows][33];
    const int lane = threadIdx.x & 31, r = threadIdx.x >> 5, j = blockIdx.x * 32 + lane;
    float s = 0.f;
    if (j < hidden) {
#pragma unroll 4
        for (int b = r; b < nPartials; b += kReduceRows) s += partial[(size_t)b * hidden + j];
    }
    s_sum[r][lane] = s;
    __syncthreads();
    if (r == 0 && j < hidden) {
        float t = 0.f;
#pragma unroll
        for (int q = 0; q < kReduceRows; ++q) t += s_sum[q][lane];
        dw[j] = __float2bfloat16_rn(t);
    }
}

// SwiGLU on gu [rows, 2 * f] (gate = columns [0, f), up = columns [f, 2f)): out = silu(gate) * up.
//
// Streaming kernels bound by HBM (6 bytes per output element forward, 10 backward).  Every thread takes VECS vectors
// kSwiThreads apart and requests all of them before the first is used (4 resp. 6 16-byte loads in flight); the flat
// vector index is divided by the row length once per thread, not once per vector, in 32 bits where the size allows.
// Measured at 4096 x 28672 against a grid-stride loop with one vector and a 64-bit division per step: forward 137.6 ->
// 102.6 us (705 MB, 6.9 TB/s; 106.7 and 107.2 us with three and four vectors, whose registers leave fewer warps for the
// arithmetic), backward 201.0 -> 172.5 us (1174 MB, 6.8 TB/s); at 4096 x 3584 22.7 -> 16.5 and 28.9 -> 25.5 us.
constexpr int kSwiThreads = 256;
constexpr int kSwiFwdVecs = 2, kSwiBwdVecs = 2;
__device__ __forceinline__ void RowOf(size_t i, uint32_t perRow, bool fits32, size_t* row, uint32_t* v)
{
    if (fits32) {
        const uint32_t r = (uint32_t)i / perRow;
        *row = r;
        *v = (uint32_t)i - r * perRow;
    } else {
        *row = i / perRow;
        *v = (uint32_t)(i - *row * perRow);
    }
}
// n / (1 + e^-x), correctly rounded for every bf16 x and n = x or 1: quotient by an approximate reciprocal, then one
// correction by the exact remainder (P. Markstein, "Computation of elementary functions on the IBM RISC System/6000
// processor", 1990).  Both sides are scaled by a quarter, which keeps the divisor below 2^126, where its reciprocal is a
// normal number: __fdividef(1, 1 + e^-x) is 0 for gates around -88, whose results are normal bf16 numbers.  Zeros and
// infinities have no remainder, their quotient stands.  An exponential that is flushed to zero adds nothing to 1
// anyway.  With the division operator in its place the forward pass at 4096 x 28672, four vectors per thread, takes
// 127.5 instead of 107.2 us.
__device__ __forceinline__ float OverOnePlusExp(float n, float x)
{
    float e, r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(x * -1.44269504f));       // e^-x = 2^(-x log2 e)
    const float d = fmaf(e, 0.25f, 0.25f), n4 = 0.25f * n;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    const float q = n4 * r, t = fmaf(fmaf(-d, q, n4), r, q);
    return fabsf(t) > 0.f ? t : q;
}

template <int VECS>
__global__ void __launch_bounds__(kSwiThreads) SwigluFwdKernel(const __nv_bfloat16* __restrict__ gu, __nv_bfloat16* __restrict__ out, size_t rows, int f)
{
    DependencyWait();
    AllowDependents();
    const uint32_t nVecRow = (uint32_t)f / 8;
    const size_t total = rows * nVecRow;
    size_t i = (size_t)blockIdx.x * (kSwiThreads * VECS) + threadIdx.x, row;
    uint32_t v;
    RowOf(i, nVecRow, total <= 0xFFFFFFFFull, &row, &v);
    uint4 g[VECS], u[VECS];
    uint32_t vs[VECS];
    size_t rs[VECS];
#pragma unroll
    for (int k = 0; k < VECS; ++k, i += kSwiThreads) {
        rs[k] = row;
        vs[k] = v;
        if (i < total) {
            const uint4* p = reinterpret_cast<const uint4*>(gu + row * 2 * f);
            g[k] = p[v];
            u[k] = p[nVecRow + v];
        } else {
            vs[k] = 0xFFFFFFFFu;
        }
        v += kSwiThreads;
        if (v >= nVecRow) { const uint32_t q = v / nVecRow; row += q; v -= q * nVecRow; }
    }
#pragma unroll
    for (int k = 0; k < VECS; ++k) {
        if (vs[k] == 0xFFFFFFFFu) break;
        float fg[8], fu[8], o[8];
        Unpack8(g[k], fg);
        Unpack8(u[k], fu);
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = OverOnePlusExp(fg[e], fg[e]) * fu[e];
        reinterpret_cast<uint4*>(out + rs[k] * f)[vs[k]] = Pack8(o);
    }
}
template <int VECS>
__global__ void __launch_bounds__(kSwiThreads) SwigluBwdKernel(const __nv_bfloat16* __restrict__ gu, const __nv_bfloat16* __restrict__ dout,
                                                               __nv_bfloat16* __restrict__ dgu, size_t rows, int f)
{
    DependencyWait();
    AllowDependents();
    const uint32_t nVecRow = (uint32_t)f / 8;
    const size_t total = rows * nVecRow;
    size_t i = (size_t)blockIdx.x * (kSwiThreads * VECS) + threadIdx.x, row;
    uint32_t v;
    RowOf(i, nVecRow, total <= 0xFFFFFFFFull, &row, &v);
    uint4 g[VECS], u[VECS], d[VECS];
    uint32_t vs[VECS];
    size_t rs[VECS];
#pragma unroll
    for (int k = 0; k < VECS; ++k, i += kSwiThreads) {
        rs[k] = row;
        vs[k] = v;
        if (i < total) {
            const uint4* p = reinterpret_cast<const uint4*>(gu + row * 2 * f);
            g[k] = p[v];
            u[k] = p[nVecRow + v];
            d[k] = reinterpret_cast<const uint4*>(dout + row * f)[v];
        } else {
            vs[k] = 0xFFFFFFFFu;
        }
        v += kSwiThreads;
        if (v >= nVecRow) { const uint32_t q = v / nVecRow; row += q; v -= q * nVecRow; }
    }
#pragma unroll
    for (int k = 0; k < VECS; ++k) {
        if (vs[k] == 0xFFFFFFFFu) break;
        float fg[8], fu[8], fd[8], dg[8], du[8];
        Unpack8(g[k], fg);
        Unpack8(u[k], fu);
        Unpack8(d[k], fd);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const float sig = OverOnePlusExp(1.f, fg[e]);
            const float silu = fg[e] * sig;
            dg[e] = fd[e] * fu[e] * sig * (1.f + fg[e] * (1.f - sig));
            du[e] = fd[e] * silu;
        }
        uint4* q = reinterpret_cast<uint4*>(dgu + rs[k] * 2 * f);
        q[vs[k]] = Pack8(dg);
        q[nVecRow + vs[k]] = Pack8(du);
    }
}

// Rotary embedding of nHeads heads of width d per row ("rotate halves": pairs (i, i + d/2)); cos / sin are fp32
// [rows, d/2].  sign = +1 forward, -1 backward (the transpose of the rotation).  Rows of `in` / `out` are inStride /
// outStride elements apart, so a slice of a wider projection output can be rotated in place or into a packed tensor.
//
// Bound by HBM (4 bytes per element).  A thread takes the same 8 columns of HEADS heads of a row (headGroups apart, so
// that neighbouring threads read neighbouring memory): the row's cosines and sines, four 16-byte loads, are loaded once
// per HEADS heads instead of with every pair, and 2 * HEADS loads of the data are in flight.  A block holds whole rows
// (or one row in several passes), so the index arithmetic is 32-bit.  Measured against one pair of vectors per step and a
// 64-bit division: 4096 x 64 heads x 128 26.7 -> 24.7 us (134 MB), 4096 x 8 x 128 6.3 -> 4.9 us, 8192 x 64 x 128 45.8 ->
// 45.2 us (268 MB, 5.9 TB/s).
constexpr int kRopeThreads = 256;
template <int HEADS>
__global__ void __launch_bounds__(kRopeThreads) RopeKernel(const __nv_bfloat16* __restrict__ in, size_t inStride, __nv_bfloat16* __restrict__ out,
                                                           size_t outStride, const float* __restrict__ cosT, const float* __restrict__ sinT,
                                                           size_t rows, int nHeads, int d, float sign, int rowsPerBlock)
{
    DependencyWait();
    AllowDependents();
    const int half = d / 2, vecHalf = half / 8;
    const int headGroups = (nHeads + HEADS - 1) / HEADS, perRow = headGroups * vecHalf;
    const size_t firstRow = (size_t)blockIdx.x * rowsPerBlock;
    for (int i = threadIdx.x; i < rowsPerBlock * perRow; i += kRopeThreads) {
        const int r = i / perRow, rem = i - r * perRow, hg = rem / vecHalf, v = rem - hg * vecHalf;
        const size_t row = firstRow + r;
        if (row >= rows) break;
        const __nv_bfloat16* src = in + row * inStride;
        __nv_bfloat16* dst = out + row * outStride;
        const float4* cp = reinterpret_cast<const float4*>(cosT + row * half + (size_t)v * 8);
        const float4* sp = reinterpret_cast<const float4*>(sinT + row * half + (size_t)v * 8);
        uint4 ra[HEADS], rb[HEADS];
#pragma unroll
        for (int k = 0; k < HEADS; ++k) {
            const int head = hg + k * headGroups;
            if (head < nHeads) {
                ra[k] = reinterpret_cast<const uint4*>(src + (size_t)head * d)[v];
                rb[k] = reinterpret_cast<const uint4*>(src + (size_t)head * d + half)[v];
            }
        }
        const float4 c0 = cp[0], c1 = cp[1], s0 = sp[0], s1 = sp[1];
        const float c[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
        const float s[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
#pragma unroll
        for (int k = 0; k < HEADS; ++k) {
            const int head = hg + k * headGroups;
            if (head < nHeads) {
                float a[8], b[8], oa[8], ob[8];
                Unpack8(ra[k], a);
                Unpack8(rb[k], b);
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    oa[e] = a[e] * c[e] - sign * b[e] * s[e];
                    ob[e] = b[e] * c[e] + sign * a[e] * s[e];
                }
                reinterpret_cast<uint4*>(dst + (size_t)head * d)[v] = Pack8(oa);
                reinterpret_cast<uint4*>(dst + (size_t)head * d + half)[v] = Pack8(ob);
            }
        }
    }
}

// Gradient of an embedding table.  Bound by the rows it writes, nearly all of them zero: 67 MB for 4096 rows of 8192 beside 17 MB
// of 1024 tokens' gradients, 2.1 GB for 128256.  Two kernels.  The first fills the table with zeros, and some of its blocks meanwhile sort
// the tokens by their ids: a token's place is the number of tokens with a smaller id and of earlier ones with its own, counted against
// all ids in shared memory.  The second writes the rows in use.  Few tokens of one id (nearly all rows): a thread owns a vector of the
// row and adds its tokens in order; a block takes up to 256 vectors of four rows, or more rows if they are short.  More than kEmbLong
// (padding, a separator): a block takes 16 vectors, 16 groups of threads each every 16th token, so that a row is shared by up to 64 SMs.
// Measured against marks of the rows in use and one block per 2048 columns of every row, which went through all ids and added a row's
// tokens alone (tokens, table, us back to back in a graph): 1024, 4096 x 8192 35.3 -> 17.9 (102 MB); 8192, 4096 x 8192 231 -> 93; 8192,
// 128256 x 8192 1042 -> 346 (2.3 GB, 6.6 TB/s); 1024, 128256 x 8192 853 -> 290; 4096, 32000 x 4096 147 -> 54; 8192, 1048576 x 64 1491 -> 38;
// all 8192 tokens of one id 958 -> 110 at 4096 x 8192 and 775 -> 90 at 50000 x 768; 8192, 32 x 8192 (256 tokens of every id) 58.8 -> 62.8.
// With autograd around it a call takes 0.13 .. 1.01 of PyTorch's time at 190 sizes and mixes of ids (1 .. 8192 tokens, 32 .. 16777216 rows);
// with the kernels before it took up to three times as long for large tables of few tokens and for frequent ids.
constexpr int kEmbThreads = 256;
constexpr uint64_t kEmbMaxTokens = 8192;          // sorted by counting: the work grows with the square of the tokens
constexpr int kEmbRanked = 32;                    // tokens that a block finds the places of
constexpr int kEmbFillVecs = 8;                   // 16-byte vectors that a thread fills, 32 KiB per block
constexpr int kEmbLong = 128;
constexpr int kEmbPlaces = 4;                     // places that a thread takes in turn where tokens are not frequent
constexpr int kEmbSlice = 16;                     // vectors of a row that a block takes where a token is frequent

// A place in the order of ids: its token and the id, 0x7FFFFFFF where that is no row of the table.  The blocks that find the places read
// the ids each for itself: ids that another stream is still writing, which a program has no right to, may leave places unwritten, so the
// second kernel takes every number of a place within its bounds.
struct alignas(8) EmbPlace { int token, id; };

__device__ __forceinline__ void EmbeddingRank(const long long* __restrict__ ids, int tokens, int vocab, int base, EmbPlace* __restrict__ places)
{
    constexpr int kWarps = kEmbThreads / 32;
    __shared__ __align__(16) int s_id[kEmbMaxTokens];
    __shared__ int s_before[kWarps][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, padded = (tokens + 3) & ~3;
    constexpr int U = 8;                              // ids that a thread requests at a time
    for (int t0 = threadIdx.x; t0 < padded; t0 += U * kEmbThreads) {
        long long id[U];
#pragma unroll
        for (int u = 0; u < U; ++u) id[u] = t0 + u * kEmbThreads < tokens ? ids[t0 + u * kEmbThreads] : -1;
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (t0 + u * kEmbThreads < padded) s_id[t0 + u * kEmbThreads] = id[u] >= 0 && id[u] < (long long)vocab ? (int)id[u] : 0x7FFFFFFF;
    }
    __syncthreads();
    // lane: a token of this block; warp: an eighth of the ids it is compared with, four at a time (base is a multiple of four).  Ids of
    // tokens in front of the block count if they are no larger, the others if they are smaller.
    const int t = base + lane, mine = t < tokens ? s_id[t] : -1;
    const int quads = padded / 4, q0 = quads * warp / kWarps, q1 = quads * (warp + 1) / kWarps, qBase = min(max(base / 4, q0), q1);
    const int4* quad = reinterpret_cast<const int4*>(s_id);
    int before = 0;
#pragma unroll 4
    for (int q = q0; q < qBase; ++q) {
        const int4 o = quad[q];
        before += (o.x <= mine) + (o.y <= mine) + (o.z <= mine) + (o.w <= mine);
    }
#pragma unroll 4
    for (int q = qBase; q < q1; ++q) {
        const int4 o = quad[q];
        before += (o.x < mine) + (o.y < mine) + (o.z < mine) + (o.w < mine);
    }
    s_before[warp][lane] = before;
    __syncthreads();
    if (warp != 0) return;
    before = __popc(__match_any_sync(0xFFFFFFFFu, mine) & ((1u << lane) - 1u));       // and those of the block itself with the same id
#pragma unroll
    for (int w = 0; w < kWarps; ++w) before += s_before[w][lane];
    if (t < tokens) places[before] = {t, mine};
}
__global__ void __launch_bounds__(kEmbThreads) EmbeddingSortKernel(const long long* __restrict__ ids, uint4* __restrict__ dTable, uint64_t vecs,
                                                                   EmbPlace* __restrict__ places, int tokens, int vocab, int ranking)
{
    DependencyWait();
    AllowDependents();
    if ((int)blockIdx.x < ranking) {
        EmbeddingRank(ids, tokens, vocab, (int)blockIdx.x * kEmbRanked, places);
        return;
    }
    const uint64_t first = (uint64_t)((int)blockIdx.x - ranking) * (kEmbThreads * kEmbFillVecs) + threadIdx.x;
#pragma unroll
    for (int u = 0; u < kEmbFillVecs; ++u) {
        const uint64_t v = first + (uint64_t)u * kEmbThreads;
        if (v < vecs) dTable[v] = make_uint4(0, 0, 0, 0);
    }
}
__device__ __forceinline__ void AddVector(float (&acc)[8], const uint4& raw)
{
    float f[8];
    Unpack8(raw, f);
#pragma unroll
    for (int k = 0; k < 8; ++k) acc[k] += f[k];
}
// acc += vector `v` of every `STEP`-th of the places [at, end).  The tokens of the next eight are requested behind the vectors of these: one
// after the other, in the branches that the ends of a row make of it, eight took 3 us.
template <int STEP>
__device__ __forceinline__ void EmbeddingAdd(float (&acc)[8], const EmbPlace* __restrict__ places, int at, int end, int tokens, const __nv_bfloat16* __restrict__ dy,
                                             int hidden, int v)
{
    constexpr int U = 8;
    int token[U];
    auto request = [&] {
#pragma unroll
        for (int u = 0; u < U; ++u) token[u] = (int)min((unsigned)places[min(at + u * STEP, end - 1)].token, (unsigned)tokens - 1);
    };
    if (at < end) request();
    while (at < end) {
        uint4 raw[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            raw[u] = make_uint4(0, 0, 0, 0);
            if (at + u * STEP < end) raw[u] = reinterpret_cast<const uint4*>(dy + (size_t)token[u] * hidden)[v];
        }
        at += U * STEP;
        if (at < end) request();
#pragma unroll
        for (int u = 0; u < U; ++u) AddVector(acc, raw[u]);
    }
}
// `slots` x `slices` blocks for frequent tokens in front, a slot for every kEmbLong-th place; the others take kEmbPlaces places per `lanes`
// threads, a row of more than kEmbThreads vectors in `chunks` blocks.
__global__ void __launch_bounds__(kEmbThreads, 4) EmbeddingRowsKernel(const EmbPlace* __restrict__ places, const __nv_bfloat16* __restrict__ dy,
                                                                   __nv_bfloat16* __restrict__ dTable, int tokens, int vocab, int hidden, int slots, int slices,
                                                                   int chunks, int lanes)
{
    DependencyWait();
    AllowDependents();
    const int nVec = hidden / 8;
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    int block = (int)blockIdx.x;
    if (block < slots * slices) {
        constexpr int kGroups = kEmbThreads / kEmbSlice;
        __shared__ float s_sum[kGroups][kEmbSlice][8];
        // more than kEmbLong places hold a multiple of it: the first one's blocks take the row, from its first place to its end
        const int at = block / slices * kEmbLong, tid = (int)threadIdx.x, id = places[at].id;
        if ((unsigned)id >= (unsigned)vocab) return;
        const int back = __syncthreads_count(tid < kEmbLong && at - 1 - tid >= 0 && places[at - 1 - tid].id == id);
        if (back == kEmbLong) return;
        const int far = at + 32 * __syncthreads_count(at + 32 * (tid + 1) < tokens && places[at + 32 * (tid + 1)].id == id);
        const int first = at - back, end = far + __syncthreads_count(tid < 32 && far + tid < tokens && places[far + tid].id == id);
        if (end - first <= kEmbLong) return;
        const int lane = threadIdx.x % kEmbSlice, group = threadIdx.x / kEmbSlice, v = block % slices * kEmbSlice + lane;
        if (v < nVec) EmbeddingAdd<kGroups>(acc, places, first + group, end, tokens, dy, hidden, v);
#pragma unroll
        for (int k = 0; k < 8; ++k) s_sum[group][lane][k] = acc[k];
        __syncthreads();
        if (group != 0 || v >= nVec) return;
        for (int g = 1; g < kGroups; ++g) {
#pragma unroll
            for (int k = 0; k < 8; ++k) acc[k] += s_sum[g][lane][k];
        }
        reinterpret_cast<uint4*>(dTable + (size_t)id * hidden)[v] = Pack8(acc);
        return;
    }
    block -= slots * slices;
    const int place = (block / chunks * (kEmbThreads / lanes) + (int)threadIdx.x / lanes) * kEmbPlaces, v = block % chunks * kEmbThreads + (int)threadIdx.x % lanes;
    if (place >= tokens || v >= nVec) return;
    auto at = [&](int i) { return places[min(i, tokens - 1)]; };
    auto vector = [&](int token) { return reinterpret_cast<const uint4*>(dy + (size_t)min((unsigned)token, (unsigned)tokens - 1) * hidden)[v]; };
    EmbPlace p[kEmbPlaces + 1];
    bool mine[kEmbPlaces];                            // a row begins here that is not left to the blocks above
    uint4 raw[kEmbPlaces];
#pragma unroll
    for (int j = 0; j <= kEmbPlaces; ++j) p[j] = at(place + j);
    int previous = place > 0 ? places[place - 1].id : -1;
#pragma unroll
    for (int j = 0; j < kEmbPlaces; ++j) {
        mine[j] = place + j < tokens && p[j].id != previous && (unsigned)p[j].id < (unsigned)vocab && !(place + j + kEmbLong < tokens && at(place + j + kEmbLong).id == p[j].id);
        previous = p[j].id;
        if (mine[j]) raw[j] = vector(p[j].token);
    }
#pragma unroll
    for (int j = 0; j < kEmbPlaces; ++j) {
        if (!mine[j]) continue;
        Unpack8(raw[j], acc);
        bool more = place + j + 1 < tokens && p[j + 1].id == p[j].id;
        for (int i = place + j + 1; more; i += 4) {
            EmbPlace q[4];
            uint4 next[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) q[u] = at(i + u);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                more = i + u < tokens && q[u].id == p[j].id;
                next[u] = make_uint4(0, 0, 0, 0);
                if (more) next[u] = vector(q[u].token);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) AddVector(acc, next[u]);
        }
        reinterpret_cast<uint4*>(dTable + (size_t)p[j].id * hidden)[v] = Pack8(acc);
    }
}

// Lets a norm kernel take the largest ring the norm kernels use.
template <auto KERNEL> HcclResult AllowNormRing()
{
    static OncePerDevice once;
    return once([]() -> HcclResult {
        CHK_CUDA(cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kNormPartBytes + kNormSlots * 3 * 2 * kNormMaxHidden)));
        return HCCL_SUCCESS;
    });
}
// As many groups (rows in work at a time) per CTA as kNormThreads hold, but no more than it takes to give every SM rows
// of its own; one CTA per SM.
struct NormShape { int groupThreads, groups, ctas; };
NormShape ShapeNorm(uint64_t rows, uint32_t hidden)
{
    NormShape n;
    const uint64_t sms = (uint64_t)SmCount();
    n.groupThreads = 32;
    while (n.groupThreads * 16 < (int)hidden) n.groupThreads *= 2;
    n.groups = (int)std::min<uint64_t>((uint64_t)(kNormThreads / n.groupThreads), (rows + sms - 1) / sms);
    n.ctas = (int)std::min<uint64_t>((rows + n.groups - 1) / n.groups, sms);
    return n;
}
bool Aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
HcclResult Launched(cudaError_t e, const char* what)
{
    if (e != cudaSuccess) { HCCL_ERROR("%s launch failed: %s", what, cudaGetErrorString(e)); return HCCL_E_RUNTIME; }
    return HCCL_SUCCESS;
}
// Two vectors per thread only where four blocks per SM remain with them; below that one each, which spreads the work
// over more SMs (128 x 3584: 4.2 us either way, the launch).
bool SwigluBig(size_t vecs) { return vecs >= (size_t)SmCount() * 4 * kSwiThreads * 2; }
size_t SwigluBlocks(size_t vecs, int vecsPerThread) { return (vecs + (size_t)kSwiThreads * vecsPerThread - 1) / ((size_t)kSwiThreads * vecsPerThread); }

}  // namespace
}  // namespace hccl

using namespace hccl;

extern "C" {

HcclResult HcclFusedAddRmsNormFwd(const void* x, const void* delta, const void* w, void* xOut, void* h, void* rstd, uint64_t rows, uint32_t hidden,
                                  float eps, hcclStream_t stream)
{
    CHK_PTR_NULL(x); CHK_PTR_NULL(w); CHK_PTR_NULL(h); CHK_PTR_NULL(rstd);
    if (delta != nullptr) CHK_PTR_NULL(xOut);
    if (hidden == 0 || hidden % 8 != 0 || hidden > kNormMaxHidden || rows > kNormMaxRows) return HCCL_E_PARA;
    if (!Aligned16(x) || !Aligned16(w) || !Aligned16(h) || (delta && (!Aligned16(delta) || !Aligned16(xOut)))) return HCCL_E_PARA;
    if (rows == 0) return HCCL_SUCCESS;
    const NormShape n = ShapeNorm(rows, hidden);
    const size_t smem = kNormPartBytes + (size_t)n.groups * kNormSlots * hidden * 2 * (delta ? 2 : 1);
    auto kernel = delta ? AddRmsNormFwdKernel<true> : AddRmsNormFwdKernel<false>;
    CHK_RET(delta ? AllowNormRing<AddRmsNormFwdKernel<true>>() : AllowNormRing<AddRmsNormFwdKernel<false>>());
    return Launched(LaunchDependent(kernel, n.ctas, n.groups * n.groupThreads, smem, (cudaStream_t)stream, 0, (const __nv_bfloat16*)x,
                                    (const __nv_bfloat16*)delta, (const __nv_bfloat16*)w, (__nv_bfloat16*)xOut, (__nv_bfloat16*)h, (float*)rstd,
                                    (int)rows, (int)hidden, n.groupThreads, eps),
                    "AddRmsNormFwd");
}

uint32_t HcclFusedRmsNormBwdPartials(uint64_t rows)
{
    // the most partial rows that a launch may write: one per row, at most 296.  HcclFusedRmsNormBwd writes one per CTA and
    // runs one CTA per SM, 148 on a B200; callers keep the size that they have always asked for.
    return (uint32_t)(rows < 296 ? (rows < 1 ? 1 : rows) : 296);
}

HcclResult HcclFusedRmsNormBwd(const void* dh, const void* x, const void* w, const void* rstd, const void* dxExtra, void* dx, void* dwPartial,
                               void* dw, uint64_t rows, uint32_t hidden, hcclStream_t stream)
{
    return HcclFusedRmsNormBwdCopy(dh, x, w, rstd, dxExtra, dx, nullptr, dwPartial, dw, rows, hidden, stream);
}

HcclResult HcclFusedRmsNormBwdCopy(const void* dh, const void* x, const void* w, const void* rstd, const void* dxExtra, void* dx, void* dxCopy,
                                   void* dwPartial, void* dw, uint64_t rows, uint32_t hidden, hcclStream_t stream)
{
    CHK_PTR_NULL(dh); CHK_PTR_NULL(x); CHK_PTR_NULL(w); CHK_PTR_NULL(rstd); CHK_PTR_NULL(dx); CHK_PTR_NULL(dwPartial); CHK_PTR_NULL(dw);
    if (hidden == 0 || hidden % 8 != 0 || hidden > kNormMaxHidden || rows > kNormMaxRows) return HCCL_E_PARA;
    if (!Aligned16(dh) || !Aligned16(x) || !Aligned16(w) || !Aligned16(dx) || !Aligned16(dwPartial) || (dxExtra && !Aligned16(dxExtra)) ||
        !Aligned16(dxCopy)) return HCCL_E_PARA;
    if (rows == 0) return HCCL_SUCCESS;
    const NormShape n = ShapeNorm(rows, hidden);
    const uint32_t nPart = std::min<uint32_t>((uint32_t)n.ctas, HcclFusedRmsNormBwdPartials(rows));
    const size_t smem = kNormPartBytes + std::max((size_t)n.groups * kNormSlots * hidden * 2 * (dxExtra ? 3 : 2),
                                                  n.groups > 1 ? (size_t)n.groups * hidden * 4 : (size_t)0);
    auto kernel = dxExtra ? RmsNormBwdKernel<true> : RmsNormBwdKernel<false>;
    CHK_RET(dxExtra ? AllowNormRing<RmsNormBwdKernel<true>>() : AllowNormRing<RmsNormBwdKernel<false>>());
    CHK_RET(Launched(LaunchDependent(kernel, nPart, n.groups * n.groupThreads, smem, (cudaStream_t)stream, 0, (const __nv_bfloat16*)dh,
                                     (const __nv_bfloat16*)x, (const __nv_bfloat16*)w, (const float*)rstd, (const __nv_bfloat16*)dxExtra,
                                     (__nv_bfloat16*)dx, (__nv_bfloat16*)dxCopy, (float*)dwPartial, (int)rows, (int)hidden, n.groupThreads),
                     "RmsNormBwd"));
    return Launched(LaunchDependent(ReducePartialsKernel, (hidden + 31) / 32, 32 * kReduceRows, 0, (cudaStream_t)stream, 0, (const float*)dwPartial,
                                    (__nv_bfloat16*)dw, (int)nPart, (int)hidden),
                    "RmsNormBwd reduce");
}

HcclResult HcclFusedSwigluFwd(const void* gu, void* out, uint64_t rows, uint32_t f, hcclStream_t stream)
{
    CHK_PTR_NULL(gu); CHK_PTR_NULL(out);
    if (f == 0 || f % 8 != 0 || !Aligned16(gu) || !Aligned16(out)) return HCCL_E_PARA;
    if (rows == 0) return HCCL_SUCCESS;
    const size_t vecs = rows * (f / 8);
    const bool big = SwigluBig(vecs);
    const size_t blocks = SwigluBlocks(vecs, big ? kSwiFwdVecs : 1);
    if (blocks > 0x7FFFFFFFull) return HCCL_E_PARA;
    return Launched(LaunchDependent(big ? SwigluFwdKernel<kSwiFwdVecs> : SwigluFwdKernel<1>, (unsigned)blocks, kSwiThreads, 0, (cudaStream_t)stream, 0,
                                    (const __nv_bfloat16*)gu, (__nv_bfloat16*)out, rows, (int)f),
                    "SwigluFwd");
}

HcclResult HcclFusedSwigluBwd(const void* gu, const void* dout, void* dgu, uint64_t rows, uint32_t f, hcclStream_t stream)
{
    CHK_PTR_NULL(gu); CHK_PTR_NULL(dout); CHK_PTR_NULL(dgu);
    if (f == 0 || f % 8 != 0 || !Aligned16(gu) || !Aligned16(dout) || !Aligned16(dgu)) return HCCL_E_PARA;
    if (rows == 0) return HCCL_SUCCESS;
    const size_t vecs = rows * (f / 8);
    const bool big = SwigluBig(vecs);
    const size_t blocks = SwigluBlocks(vecs, big ? kSwiBwdVecs : 1);
    if (blocks > 0x7FFFFFFFull) return HCCL_E_PARA;
    return Launched(LaunchDependent(big ? SwigluBwdKernel<kSwiBwdVecs> : SwigluBwdKernel<1>, (unsigned)blocks, kSwiThreads, 0, (cudaStream_t)stream, 0,
                                    (const __nv_bfloat16*)gu, (const __nv_bfloat16*)dout, (__nv_bfloat16*)dgu, rows, (int)f),
                    "SwigluBwd");
}

HcclResult HcclFusedRope(const void* in, uint64_t inStride, void* out, uint64_t outStride, const void* cosTable, const void* sinTable, uint64_t rows,
                         uint32_t nHeads, uint32_t headDim, int backward, hcclStream_t stream)
{
    CHK_PTR_NULL(in); CHK_PTR_NULL(out); CHK_PTR_NULL(cosTable); CHK_PTR_NULL(sinTable);
    if (headDim == 0 || headDim % 16 != 0 || inStride % 8 != 0 || outStride % 8 != 0) return HCCL_E_PARA;
    if (!Aligned16(in) || !Aligned16(out) || !Aligned16(cosTable) || !Aligned16(sinTable)) return HCCL_E_PARA;
    if (rows == 0 || nHeads == 0) return HCCL_SUCCESS;
    // four heads per thread where there are that many: the cosines and sines are then a quarter of the loads
    const int heads = nHeads >= 4 ? 4 : (nHeads >= 2 ? 2 : 1);
    const uint32_t perRow = (nHeads + heads - 1) / heads * (headDim / 16);
    const uint32_t rowsPerBlock = perRow >= (uint32_t)kRopeThreads ? 1 : kRopeThreads / perRow;
    const uint64_t blocks = (rows + rowsPerBlock - 1) / rowsPerBlock;
    if (blocks > 0x7FFFFFFFull) return HCCL_E_PARA;
    return Launched(LaunchDependent(heads == 4 ? RopeKernel<4> : (heads == 2 ? RopeKernel<2> : RopeKernel<1>), (unsigned)blocks, kRopeThreads, 0,
                                    (cudaStream_t)stream, 0, (const __nv_bfloat16*)in, (size_t)inStride, (__nv_bfloat16*)out, (size_t)outStride,
                                    (const float*)cosTable, (const float*)sinTable, rows, (int)nHeads, (int)headDim, backward ? -1.f : 1.f,
                                    (int)rowsPerBlock),
                    "Rope");
}

HcclResult HcclFusedEmbeddingGrad(const int64_t* ids, const void* dy, void* dTable, void* scratch, uint64_t tokens, uint64_t vocab, uint32_t hidden,
                                  hcclStream_t stream)
{
    CHK_PTR_NULL(ids); CHK_PTR_NULL(dy); CHK_PTR_NULL(dTable); CHK_PTR_NULL(scratch);
    if (hidden == 0 || hidden % 8 != 0 || !Aligned16(dy) || !Aligned16(dTable) || !Aligned16(scratch) || (reinterpret_cast<uintptr_t>(ids) & 7u) != 0) return HCCL_E_PARA;
    const uint64_t nVec = hidden / 8, chunks = (nVec + kEmbThreads - 1) / kEmbThreads;
    if (tokens > kEmbMaxTokens || hidden > 0x7FFFFFFFu || vocab > 0x7FFFFFFFull / chunks) return HCCL_E_NOT_SUPPORT;
    if (vocab == 0) return HCCL_SUCCESS;
    const uint64_t vecs = vocab * nVec, perBlock = (uint64_t)kEmbThreads * kEmbFillVecs, filling = (vecs + perBlock - 1) / perBlock;
    const uint64_t ranking = (tokens + kEmbRanked - 1) / kEmbRanked;
    const uint64_t slots = tokens > kEmbLong ? (tokens + kEmbLong - 1) / kEmbLong : 0, slices = (nVec + kEmbSlice - 1) / kEmbSlice;
    int lanes = 1;
    while (lanes < kEmbThreads && (uint64_t)lanes < nVec) lanes *= 2;
    const uint64_t perRowBlock = (uint64_t)(kEmbThreads / lanes) * kEmbPlaces, rows = (tokens + perRowBlock - 1) / perRowBlock * chunks;
    if (ranking + filling > 0x7FFFFFFFull || slots * slices + rows > 0x7FFFFFFFull) return HCCL_E_NOT_SUPPORT;
    CHK_RET(Launched(LaunchDependent(EmbeddingSortKernel, (unsigned)(ranking + filling), kEmbThreads, 0, (cudaStream_t)stream, 0, reinterpret_cast<const long long*>(ids),
                                     (uint4*)dTable, vecs, (EmbPlace*)scratch, (int)tokens, (int)vocab, (int)ranking), "EmbeddingSort"));
    if (tokens == 0) return HCCL_SUCCESS;
    return Launched(LaunchDependent(EmbeddingRowsKernel, (unsigned)(slots * slices + rows), kEmbThreads, 0, (cudaStream_t)stream, 0, (const EmbPlace*)scratch,
                                    (const __nv_bfloat16*)dy, (__nv_bfloat16*)dTable, (int)tokens, (int)vocab, (int)hidden, (int)slots, (int)slices, (int)chunks, lanes),
                    "EmbeddingRows");
}

HcclResult HcclFusedEmbeddingBwd(const int64_t* ids, const void* dy, void* dTable, void* marks, uint64_t tokens, uint64_t vocab, uint32_t hidden,
                                 hcclStream_t stream)
{
    CHK_PTR_NULL(marks);
    if (!Aligned16(marks)) return HCCL_E_PARA;
    if (tokens > kEmbMaxTokens) return HCCL_E_NOT_SUPPORT;
    void* scratch = nullptr;
    if (const cudaError_t e = cudaMallocAsync(&scratch, std::max<uint64_t>(tokens, 1) * sizeof(EmbPlace), (cudaStream_t)stream); e != cudaSuccess) {
        cudaGetLastError();
        HCCL_ERROR("no scratch for the embedding's gradient: %s", cudaGetErrorString(e));
        return HCCL_E_RUNTIME;
    }
    const HcclResult r = HcclFusedEmbeddingGrad(ids, dy, dTable, scratch, tokens, vocab, hidden, stream);
    CHK_CUDA(cudaFreeAsync(scratch, (cudaStream_t)stream));
    return r;
}

}  // extern "C"
