// dev_kron.cu -- the Kronecker space-time operator on the GPU.
//
// Computes Y = alpha * (K X A^T + M X B^T) + beta * Y, the operator of
// src/kronecker.f90:19-127 (kronspmv / kronspgemv), where X and Y hold the q
// temporal blocks of a space-time vector node-major (row r, block k at
// r*q + k).  The reference runs 2q serial CSR products and then a q^2 p
// mixing loop, so K and M are each streamed q times; here each CSR row is
// streamed once: a team of LANES threads walks the row's nonzeros, every
// nonzero multiplies the q contiguous values of X's column row (one 24 B or
// 48 B gather), the q partial sums of K and of M are reduced across the team
// with shuffles and the q x q temporal mixing with A and B (kept in shared
// memory) is applied in the epilogue before the single store of Y's row.
//
// Roofline: the kernel streams nnz(K)+nnz(M) column indices and values once
// plus the row pointers, and touches X (gathered, L2-resident) and Y once.
// In FP32 it is HBM-bound; in FP64 the GB300's FP64 pipe (about 1.2 TFLOP/s)
// binds first because every nonzero carries q FMAs (k_kron_nb64).
#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "df.cuh"
#include <cuda_bf16.h>

#include "xt_device.h"

namespace xt {

namespace {

__global__ void k_dec_index(int* a, size_t n)
{
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (; i < n; i += stride) a[i] -= 1;
}

__global__ void k_to_f32(const double* a, float* b, size_t n)
{
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (; i < n; i += stride) b[i] = (float)a[i];
}

template <class T, int Q>
__device__ __forceinline__ void load_row(const T* __restrict__ p, T (&v)[Q])
{
#pragma unroll
    for (int b = 0; b < Q; ++b) v[b] = p[b];
}

// 6 contiguous values: three 2-wide loads (rows start 8 B / 16 B aligned)
template <>
__device__ __forceinline__ void load_row<float, 6>(const float* __restrict__ p, float (&v)[6])
{
    const float2* q = reinterpret_cast<const float2*>(p);
    float2 a = __ldg(q), b = __ldg(q + 1), c = __ldg(q + 2);
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y; v[4] = c.x; v[5] = c.y;
}
template <>
__device__ __forceinline__ void load_row<double, 6>(const double* __restrict__ p, double (&v)[6])
{
    const double2* q = reinterpret_cast<const double2*>(p);
    double2 a = __ldg(q), b = __ldg(q + 1), c = __ldg(q + 2);
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y; v[4] = c.x; v[5] = c.y;
}

// value array of the requested precision (host-side selection)
template <class T>
const T* vals(const double* v64, const float* v32);
template <>
const double* vals<double>(const double* v64, const float*) { return v64; }
template <>
const float* vals<float>(const double*, const float* v32) { return v32; }

// stored value -> arithmetic type (BF16 values widen exactly to FP32)
template <class T>
__device__ __forceinline__ T widen(T v) { return v; }
__device__ __forceinline__ float widen(__nv_bfloat16 v) { return __bfloat162float(v); }

template <class T, int Q, int LANES, bool MERGED, class V = T>
__global__ void __launch_bounds__(256)
k_kron_spmm(int p, const int* __restrict__ kptr, const int* __restrict__ kcol,
            const V* __restrict__ kval, const int* __restrict__ mptr,
            const int* __restrict__ mcol, const V* __restrict__ mval,
            const double* __restrict__ dA, const double* __restrict__ dB, T alpha, T beta,
            const T* __restrict__ x, T* __restrict__ y)
{
    __shared__ T sA[Q * Q], sB[Q * Q];
    for (int i = threadIdx.x; i < Q * Q; i += blockDim.x) {
        sA[i] = (T)dA[i];
        sB[i] = (T)dB[i];
    }
    __syncthreads();
    // The loop bound is warp-uniform so that every lane of a warp reaches the
    // shuffles; teams past the last row run with empty ranges.
    constexpr int TPW = 32 / LANES;  // teams per warp
    const int lane = threadIdx.x % LANES;
    const int team = (threadIdx.x % 32) / LANES;
    const int gwarp = (blockIdx.x * blockDim.x + threadIdx.x) / 32;
    const int nwarp = (gridDim.x * blockDim.x) / 32;
    for (int rb = gwarp * TPW; rb < p; rb += nwarp * TPW) {
        const int r = rb + team;
        const bool act = r < p;
        T ak[Q], am[Q];
#pragma unroll
        for (int b = 0; b < Q; ++b) { ak[b] = T(0); am[b] = T(0); }
        const int k0 = act ? kptr[r] : 0, k1 = act ? kptr[r + 1] : 0;
        if constexpr (MERGED) {  // one pattern: one index and one X row for both
#pragma unroll 4
            for (int k = k0 + lane; k < k1; k += LANES) {
                const T vk = widen(kval[k]), vm = widen(mval[k]);
                T xr[Q];
                load_row<T, Q>(x + (size_t)kcol[k] * Q, xr);
#pragma unroll
                for (int b = 0; b < Q; ++b) {
                    ak[b] = fma(vk, xr[b], ak[b]);
                    am[b] = fma(vm, xr[b], am[b]);
                }
            }
        } else {
#pragma unroll 4
            for (int k = k0 + lane; k < k1; k += LANES) {
                const T v = widen(kval[k]);
                T xr[Q];
                load_row<T, Q>(x + (size_t)kcol[k] * Q, xr);
#pragma unroll
                for (int b = 0; b < Q; ++b) ak[b] = fma(v, xr[b], ak[b]);
            }
            const int m0 = act ? mptr[r] : 0, m1 = act ? mptr[r + 1] : 0;
#pragma unroll 4
            for (int k = m0 + lane; k < m1; k += LANES) {
                const T v = widen(mval[k]);
                T xr[Q];
                load_row<T, Q>(x + (size_t)mcol[k] * Q, xr);
#pragma unroll
                for (int b = 0; b < Q; ++b) am[b] = fma(v, xr[b], am[b]);
            }
        }
#pragma unroll
        for (int off = LANES / 2; off > 0; off >>= 1)
#pragma unroll
            for (int b = 0; b < Q; ++b) {
                ak[b] += __shfl_xor_sync(0xffffffffu, ak[b], off, LANES);
                am[b] += __shfl_xor_sync(0xffffffffu, am[b], off, LANES);
            }
        // epilogue: lane a < Q forms output block a of this row (every lane
        // holds all the sums; a branch per a would issue the mixing Q times)
        if (act && lane < Q) {
            T acc = T(0);
#pragma unroll
            for (int b = 0; b < Q; ++b) {
                acc = fma(sA[b * Q + lane], ak[b], acc);
                acc = fma(sB[b * Q + lane], am[b], acc);
            }
            T* yp = y + (size_t)r * Q + lane;
            *yp = (beta == T(0)) ? alpha * acc : fma(beta, *yp, alpha * acc);
        }
    }
}

// XTFEM_KRON_NB=0 keeps the CSR kernels, 2 takes the FP64 node blocks at any
// size (tests compare the two).
bool nb_enabled()
{
    const char* e = std::getenv("XTFEM_KRON_NB");
    return !e || std::atoi(e) != 0;
}

// The node-block copies of CSR value i, at at[i]: FP64 and double-float.
__global__ void k_scatter_blocks(const double* __restrict__ a, const int* __restrict__ at,
                                 double* __restrict__ b64, float2* __restrict__ bdf, size_t n)
{
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x) {
        const double v = a[i];
        const float h = __double2float_rn(v);
        b64[at[i]] = v;
        bdf[at[i]] = make_float2(h, __double2float_rn(v - (double)h));
    }
}

__global__ void k_to_df(const double* __restrict__ a, float2* __restrict__ b, size_t n)
{
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (; i < n; i += stride) {
        const float h = __double2float_rn(a[i]);
        b[i] = make_float2(h, __double2float_rn(a[i] - (double)h));
    }
}

// (hi, lo) += (vh + vl) x for an FP32 x: vh x exactly (fma), vl x in FP32
__device__ __forceinline__ void df_axpy(float& hi, float& lo, float vh, float vl, float x)
{
    const float p = __fmul_rn(vh, x);
    const float e = fmaf(vh, x, -p);
    df_add(hi, lo, p);
    lo = __fadd_rn(lo, fmaf(vl, x, e));
}

// The same row-team structure as k_kron_spmm, with double-float values and
// accumulators, an FP32 X and a double-float Y (alpha = 1, beta = 0).
template <int Q, int LANES, bool MERGED>
__global__ void __launch_bounds__(256)
k_kron_df(int p, const int* __restrict__ kptr, const int* __restrict__ kcol,
          const float2* __restrict__ kval, const int* __restrict__ mptr,
          const int* __restrict__ mcol, const float2* __restrict__ mval,
          const double* __restrict__ dA, const double* __restrict__ dB,
          const float* __restrict__ x, float2* __restrict__ y)
{
    __shared__ float2 sA[Q * Q], sB[Q * Q];
    for (int i = threadIdx.x; i < Q * Q; i += blockDim.x) {
        const float ah = __double2float_rn(dA[i]), bh = __double2float_rn(dB[i]);
        sA[i] = make_float2(ah, __double2float_rn(dA[i] - (double)ah));
        sB[i] = make_float2(bh, __double2float_rn(dB[i] - (double)bh));
    }
    __syncthreads();
    constexpr int TPW = 32 / LANES;
    const int lane = threadIdx.x % LANES;
    const int team = (threadIdx.x % 32) / LANES;
    const int gwarp = (blockIdx.x * blockDim.x + threadIdx.x) / 32;
    const int nwarp = (gridDim.x * blockDim.x) / 32;
    for (int rb = gwarp * TPW; rb < p; rb += nwarp * TPW) {
        const int r = rb + team;
        const bool act = r < p;
        float kh[Q], kl[Q], mh[Q], ml[Q];
#pragma unroll
        for (int b = 0; b < Q; ++b) kh[b] = kl[b] = mh[b] = ml[b] = 0.0f;
        const int k0 = act ? kptr[r] : 0, k1 = act ? kptr[r + 1] : 0;
        if constexpr (MERGED) {
#pragma unroll 4
            for (int k = k0 + lane; k < k1; k += LANES) {
                const float2 vk = kval[k], vm = mval[k];
                float xr[Q];
                load_row<float, Q>(x + (size_t)kcol[k] * Q, xr);
#pragma unroll
                for (int b = 0; b < Q; ++b) {
                    df_axpy(kh[b], kl[b], vk.x, vk.y, xr[b]);
                    df_axpy(mh[b], ml[b], vm.x, vm.y, xr[b]);
                }
            }
        } else {
#pragma unroll 4
            for (int k = k0 + lane; k < k1; k += LANES) {
                const float2 v = kval[k];
                float xr[Q];
                load_row<float, Q>(x + (size_t)kcol[k] * Q, xr);
#pragma unroll
                for (int b = 0; b < Q; ++b) df_axpy(kh[b], kl[b], v.x, v.y, xr[b]);
            }
            const int m0 = act ? mptr[r] : 0, m1 = act ? mptr[r + 1] : 0;
#pragma unroll 4
            for (int k = m0 + lane; k < m1; k += LANES) {
                const float2 v = mval[k];
                float xr[Q];
                load_row<float, Q>(x + (size_t)mcol[k] * Q, xr);
#pragma unroll
                for (int b = 0; b < Q; ++b) df_axpy(mh[b], ml[b], v.x, v.y, xr[b]);
            }
        }
#pragma unroll
        for (int off = LANES / 2; off > 0; off >>= 1)
#pragma unroll
            for (int b = 0; b < Q; ++b) {
                const float a1 = __shfl_xor_sync(0xffffffffu, kh[b], off, LANES);
                const float a2 = __shfl_xor_sync(0xffffffffu, kl[b], off, LANES);
                const float b1 = __shfl_xor_sync(0xffffffffu, mh[b], off, LANES);
                const float b2 = __shfl_xor_sync(0xffffffffu, ml[b], off, LANES);
                df_add_df(kh[b], kl[b], a1, a2);
                df_add_df(mh[b], ml[b], b1, b2);
            }
        if (act && lane < Q) {
            float h = 0.0f, l = 0.0f;
#pragma unroll
            for (int b = 0; b < Q; ++b) {
                df_mul_acc(h, l, sA[b * Q + lane].x, sA[b * Q + lane].y, kh[b], kl[b]);
                df_mul_acc(h, l, sB[b * Q + lane].x, sB[b * Q + lane].y, mh[b], ml[b]);
            }
            y[(size_t)r * Q + lane] = df_norm(h, l);
        }
    }
}

// Node-block double-float apply, Y = K X A^T + M X B^T (even Q): a lane
// owns (node row a, DOF c, temporal pair qp) and accumulates (KX)[3a+c][2qp..]
// and (MX)[3a+c][2qp..] over the node row's blocks: per block one column
// index, row c of K's block, M's scalar and the neighbour's three X pairs.
// The Q/2 lanes of (a, c) then exchange their sums and each finishes its
// two outputs with the q x q temporal mixing.  3 Q/2 lanes per node row,
// 32 / (3 Q/2) node rows per warp.
// This thread block is block bx of a gx-block pass (a batched launch runs
// one such pass per system).
//
// What bounds it is how many bytes of K a warp has in flight: with the blocks
// read where they are used, one block a lane ahead at best, 66 % of the issue
// slots wait for them (1.15 TB/s).  STAGED: a warp copies its node rows'
// blocks, masses and columns -- one contiguous range -- to shared memory at
// once (cp.async, its own part, no block barrier) and keeps kNbAhead X
// slices in flight; then FP32 (packed operations take two cycles) and
// shared-memory reads are each busy half the time.
// Measured (q 6), direct and staged: 25 x 9 x 7 rod 18.7 and 13.3 us, a step of
// 64 rods in 175 and 168 ms a batch.  A system alone of more than kNbStagedNodes
// nodes reads directly all the same: a queue of blocks that hold shared memory
// keeps another system's triangular sweep, which wants most of an SM's, from
// starting.  Eight slab loops at once, slabs/s: 3,751 nodes 295 and 303, 5,239
// nodes 196 and 190, 14,161 nodes 62.3 and 58.2 (one alone the same either way),
// 26,901 nodes 24 and 20.6.  The kernel of a batch, whose sweeps come between
// its steps, is staged up to one round of thread blocks: sixteen rods of 5,239
// nodes 131 and 127 ms, eight of 9,225 nodes 128 and 125.  One or three
// slices ahead, 64 or 256 threads a block are slower.  q 2 and 4, whose 10 or
// 5 rows a warp would take too much shared memory, and 8 read directly.
constexpr int kNbAhead = 2;

constexpr int kNbStagedNodes = 152 * 30;       // two and a half blocks an SM of four warps, three node rows each
constexpr int kNbStagedBatch = 152 * 8 * 12;  // eight

template <bool STAGED>
constexpr int nb_threads()
{
    return STAGED ? 128 : 256;
}

template <class V>
__device__ __forceinline__ void copy_async(V* dst, const V* src)
{
    static_assert(sizeof(V) == 4 || sizeof(V) == 8, "cp.async of 4 or 8 bytes");
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(
                     (unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src), "n"(sizeof(V))
                 : "memory");
}

template <int Q, bool STAGED>
__device__ __forceinline__ void kron_nb_body(int nodes, const int* __restrict__ bptr,
                                             const int* __restrict__ bcol,
                                             const float2* __restrict__ kv,
                                             const float2* __restrict__ mv,
                                             const double* __restrict__ dA,
                                             const double* __restrict__ dB,
                                             const float* __restrict__ x, float2* __restrict__ y,
                                             int bx, int gx)
{
    static_assert(Q % 2 == 0 && Q <= 8, "pairs of temporal blocks");
    constexpr int NP = Q / 2, LPR = 3 * NP, RPW = 32 / LPR;
    [[maybe_unused]] constexpr int WARPS = nb_threads<STAGED>() / 32;
    __shared__ float2 sA[Q * Q], sB[Q * Q];
    for (int i = threadIdx.x; i < Q * Q; i += blockDim.x) {
        const float ah = __double2float_rn(dA[i]), bh = __double2float_rn(dB[i]);
        sA[i] = make_float2(ah, __double2float_rn(dA[i] - (double)ah));
        sB[i] = make_float2(bh, __double2float_rn(dB[i] - (double)bh));
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, slot = lane / LPR, inl = lane - slot * LPR;
    const int c = inl / NP, qp = inl - c * NP;
    const bool lane_ok = slot < RPW;
    const int gwarp = (bx * blockDim.x + threadIdx.x) / 32;
    const int nwarp = (gx * blockDim.x) / 32;
    for (int a0 = gwarp * RPW; a0 < nodes; a0 += nwarp * RPW) {
        const int a = a0 + slot;
        const bool act = lane_ok && a < nodes;
        // (hi, lo) of the lane's two temporal entries, packed: .x entry 2qp,
        // .y entry 2qp+1
        float2 kh = make_float2(0.f, 0.f), kl = kh, mh = kh, ml = kh;
        const int b0 = act ? bptr[a] : 0, b1 = act ? bptr[a + 1] : 0;
        if constexpr (STAGED) {
            constexpr int CAP = 27 * RPW, D = kNbAhead, N = D + 1;
            __shared__ float2 stK[WARPS][CAP * 9], stM[WARPS][CAP];
            __shared__ int stC[WARPS][CAP];
            float2* const sK = stK[threadIdx.x >> 5];
            float2* const sM = stM[threadIdx.x >> 5];
            int* const sC = stC[threadIdx.x >> 5];
            const int r1 = bptr[min(a0 + RPW, nodes)];
            // CAP blocks at a time: all of the warp's rows on a hexahedral mesh
            for (int base = bptr[a0]; base < r1; base += CAP) {
                const int cnt = min(CAP, r1 - base);
                for (int i = lane; i < 9 * cnt; i += 32) copy_async(sK + i, kv + (size_t)base * 9 + i);
                for (int i = lane; i < cnt; i += 32) {
                    copy_async(sM + i, mv + base + i);
                    copy_async(sC + i, bcol + base + i);
                }
                asm volatile("cp.async.wait_all;" ::: "memory");
                __syncwarp();
                const int e1 = min(b1 - base, cnt);
                int e = max(b0 - base, 0);
                const float* xq = x + 2 * qp;
                float2 xs[N][3];
                auto fetch = [&](int at, int u) {
                    const float* xb = xq + (size_t)sC[at] * (3 * Q);
                    xs[u][0] = *reinterpret_cast<const float2*>(xb);
                    xs[u][1] = *reinterpret_cast<const float2*>(xb + Q);
                    xs[u][2] = *reinterpret_cast<const float2*>(xb + 2 * Q);
                };
#pragma unroll
                for (int u = 0; u < D; ++u)
                    if (e + u < e1) fetch(e + u, u);
                for (; e < e1; e += N) {
#pragma unroll
                    for (int u = 0; u < N; ++u) {
                        if (e + u + D < e1) fetch(e + u + D, (u + D) % N);
                        if (e + u < e1) {
                            const float2* kr = sK + (e + u) * 9 + c * 3;
                            const float2 k0 = kr[0], k1 = kr[1], k2 = kr[2], m = sM[e + u];
                            const float2 x0 = xs[u][0], x1 = xs[u][1], x2 = xs[u][2];
                            df2_axpy(kh, kl, k0.x, k0.y, x0);
                            df2_axpy(kh, kl, k1.x, k1.y, x1);
                            df2_axpy(kh, kl, k2.x, k2.y, x2);
                            df2_axpy(mh, ml, m.x, m.y, c == 0 ? x0 : (c == 1 ? x1 : x2));
                        }
                    }
                }
                __syncwarp();  // read before the next copy
            }
        } else {
#pragma unroll 4
            for (int b = b0; b < b1; ++b) {
                const float* xb = x + (size_t)bcol[b] * (3 * Q) + 2 * qp;
                const float2* kr = kv + (size_t)b * 9 + c * 3;
                const float2 k0 = kr[0], k1 = kr[1], k2 = kr[2], m = mv[b];
                const float2 x0 = *reinterpret_cast<const float2*>(xb);
                const float2 x1 = *reinterpret_cast<const float2*>(xb + Q);
                const float2 x2 = *reinterpret_cast<const float2*>(xb + 2 * Q);
                df2_axpy(kh, kl, k0.x, k0.y, x0);
                df2_axpy(kh, kl, k1.x, k1.y, x1);
                df2_axpy(kh, kl, k2.x, k2.y, x2);
                df2_axpy(mh, ml, m.x, m.y, c == 0 ? x0 : (c == 1 ? x1 : x2));
            }
        }
        const float kh0 = kh.x, kl0 = kl.x, kh1 = kh.y, kl1 = kl.y;
        const float mh0 = mh.x, ml0 = ml.x, mh1 = mh.y, ml1 = ml.y;
        // all Q temporal entries of row 3a+c, from the NP lanes of (a, c)
        float KH[Q], KL[Q], MH[Q], ML[Q];
        const int base = slot * LPR + c * NP;
#pragma unroll
        for (int j = 0; j < NP; ++j) {
            const int src = base + j;
            KH[2 * j] = __shfl_sync(0xffffffffu, kh0, src);
            KL[2 * j] = __shfl_sync(0xffffffffu, kl0, src);
            KH[2 * j + 1] = __shfl_sync(0xffffffffu, kh1, src);
            KL[2 * j + 1] = __shfl_sync(0xffffffffu, kl1, src);
            MH[2 * j] = __shfl_sync(0xffffffffu, mh0, src);
            ML[2 * j] = __shfl_sync(0xffffffffu, ml0, src);
            MH[2 * j + 1] = __shfl_sync(0xffffffffu, mh1, src);
            ML[2 * j + 1] = __shfl_sync(0xffffffffu, ml1, src);
        }
        if (act) {
            float2 out[2];
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                const int i = 2 * qp + t;
                float h = 0.0f, l = 0.0f;
#pragma unroll
                for (int j = 0; j < Q; ++j) {
                    df_mul_acc(h, l, sA[j * Q + i].x, sA[j * Q + i].y, KH[j], KL[j]);
                    df_mul_acc(h, l, sB[j * Q + i].x, sB[j * Q + i].y, MH[j], ML[j]);
                }
                out[t] = df_norm(h, l);
            }
            *reinterpret_cast<float4*>(y + (size_t)(3 * a + c) * Q + 2 * qp) =
                make_float4(out[0].x, out[0].y, out[1].x, out[1].y);
        }
    }
}

template <int Q, bool STAGED>
__global__ void __launch_bounds__(nb_threads<STAGED>(), STAGED ? 8 : 1)
k_kron_nb(int nodes, const int* __restrict__ bptr, const int* __restrict__ bcol,
          const float2* __restrict__ kv, const float2* __restrict__ mv,
          const double* __restrict__ dA, const double* __restrict__ dB,
          const float* __restrict__ x, float2* __restrict__ y, const int* __restrict__ skip)
{
    if (skip && skip[0] != 0) return;
    kron_nb_body<Q, STAGED>(nodes, bptr, bcol, kv, mv, dA, dB, x, y, blockIdx.x, gridDim.x);
}

// The node-block operator of table entry blockIdx.y: wfix = op(zfix), nothing
// once the entry's cycle has ended.
template <int Q, bool STAGED>
__global__ void __launch_bounds__(nb_threads<STAGED>(), STAGED ? 8 : 1) kb_kron_nb(const FlexStepItem* __restrict__ t)
{
    const FlexStepItem& e = t[blockIdx.y];
    if (e.ctl[1] != 0) return;
    kron_nb_body<Q, STAGED>(e.nodes, e.bptr, e.bcol, e.kv, e.mv, e.A, e.B, e.zfix, e.wfix, blockIdx.x,
                    gridDim.x);
}

// FP64 node-block apply, Y = alpha (K X A^T + M X B^T) + beta Y: a thread owns
// (node row a, DOF c, temporal entry b) and accumulates (KX)[3a+c][b] and
// (MX)[3a+c][b] over the node row's blocks, four FP64 multiply-adds a block;
// the Q threads of (a, c) exchange their sums through shared memory for the
// q x q mixing.  Threads are dealt to (a, c, b) without a gap, so that the
// multiply-adds are the whole of the FP64 work: this part's FP64 pipe (a warp
// instruction every 19 cycles of an SM) is what bounds the operator, 1.72 M
// warp instructions and 105 us on the 20 x 20 x 60 rod (q = 6).  The CSR
// kernel spends half as much again on row tails and the lanes' tree sums.
//
// A thread keeps nine sums of KX (DOF of the block, block mod 3) and three of
// MX, of nine terms each on a hexahedral mesh, and mixes in four: one sum of 81
// terms in sequence had 1.5 times the rounding of the CSR kernel's eight lanes
// (2.75e-16 of the result in the 2-norm against 1.78e-16; this 1.70e-16).
// Measured on that rod: 132 us (119 with the one sum); figures against the CSR
// kernel at kron_spmm.
template <int Q>
__global__ void __launch_bounds__(256)
k_kron_nb64(int nodes, const int* __restrict__ bptr, const int* __restrict__ bcol,
            const int* __restrict__ mask, const double* __restrict__ kv,
            const double* __restrict__ mv, const double* __restrict__ dA,
            const double* __restrict__ dB, double alpha, double beta,
            const double* __restrict__ x, double* __restrict__ y)
{
    constexpr int TPN = 3 * Q, NPB = 256 / TPN;
    __shared__ double sA[Q * Q], sB[Q * Q], sK[256], sM[256];
    const int t = threadIdx.x;
    for (int i = t; i < Q * Q; i += 256) {
        sA[i] = dA[i];
        sB[i] = dB[i];
    }
    const int nl = t / TPN, rem = t - nl * TPN, c = rem / Q, b = rem - c * Q;
    const int a = blockIdx.x * NPB + nl;
    const bool act = nl < NPB && a < nodes;
    double ak = 0.0, am = 0.0;
    if (act) {
        double s0[3] = {}, s1[3] = {}, s2[3] = {}, sm[3] = {};
        auto block = [&](int k, int u) {
            const double* xb = x + (size_t)bcol[k] * TPN + b;
            const double* kr = kv + (size_t)k * 9 + c * 3;
            const double x0 = xb[0], x1 = xb[Q], x2 = xb[2 * Q];
            const double xc = c == 0 ? x0 : (c == 1 ? x1 : x2);
            const double k0 = kr[0], k1 = kr[1], k2 = kr[2], m = mv[k];
            const int mk = mask[k];
            if (mk == 0xfff) {
                s0[u] = fma(k0, x0, s0[u]);
                s1[u] = fma(k1, x1, s1[u]);
                s2[u] = fma(k2, x2, s2[u]);
                sm[u] = fma(m, xc, sm[u]);
            } else {  // only the entries that K and M have: 0 times an infinite x is no zero
                const int r = mk >> (3 * c);
                if (r & 1) s0[u] = fma(k0, x0, s0[u]);
                if (r & 2) s1[u] = fma(k1, x1, s1[u]);
                if (r & 4) s2[u] = fma(k2, x2, s2[u]);
                if (mk >> 9) sm[u] = fma(m, xc, sm[u]);
            }
        };
        const int b1 = bptr[a + 1];
        int k = bptr[a];
        for (; k + 3 <= b1; k += 3) {
            block(k, 0);
            block(k + 1, 1);
            block(k + 2, 2);
        }
        if (k < b1) block(k, 0);
        if (k + 1 < b1) block(k + 1, 1);
        auto sum = [](const double (&s)[3]) { return (s[0] + s[1]) + s[2]; };
        ak = (sum(s0) + sum(s1)) + sum(s2);
        am = sum(sm);
    }
    sK[t] = ak;
    sM[t] = am;
    __syncthreads();
    if (act) {
        const int base = t - b;
        double pk[2] = {}, pm[2] = {};
#pragma unroll
        for (int j = 0; j < Q; ++j) {
            pk[j & 1] = fma(sA[j * Q + b], sK[base + j], pk[j & 1]);
            pm[j & 1] = fma(sB[j * Q + b], sM[base + j], pm[j & 1]);
        }
        const double acc = (pk[0] + pk[1]) + (pm[0] + pm[1]);
        double* yp = y + (size_t)(3 * a + c) * Q + b;
        *yp = beta == 0.0 ? alpha * acc : fma(beta, *yp, alpha * acc);
    }
}

template <int Q>
int launch_nb64(const DevNodeBlocks& nb, const double* dA, const double* dB, double alpha,
                double beta, const double* x, double* y, cudaStream_t s)
{
    constexpr int NPB = 256 / (3 * Q);
    k_kron_nb64<Q><<<(nb.nodes + NPB - 1) / NPB, 256, 0, s>>>(
        nb.nodes, nb.ptr.p, nb.col.p, nb.mask.p, nb.k64.p, nb.m64.p, dA, dB, alpha, beta, x, y);
    note_launches(1);
    XT_CUDA(cudaGetLastError());
    return XT_OK;
}

template <int Q>
int launch_nb(const DevNodeBlocks& nb, const double* dA, const double* dB, const float* x,
              float2* y, cudaStream_t s, const int* skip)
{
    constexpr int RPW = 32 / (3 * (Q / 2));
    auto launch = [&](auto kernel, int threads) {
        const int rows_per_block = (threads / 32) * RPW;
        const int blocks = std::max(1, (nb.nodes + rows_per_block - 1) / rows_per_block);
        kernel<<<blocks, threads, 0, s>>>(nb.nodes, nb.ptr.p, nb.col.p, nb.kdf.p, nb.mdf.p, dA,
                                          dB, x, y, skip);
    };
    if constexpr (Q == 6) {
        if (nb.nodes <= kNbStagedNodes) launch(k_kron_nb<Q, true>, nb_threads<true>());
        else launch(k_kron_nb<Q, false>, nb_threads<false>());
    } else {
        launch(k_kron_nb<Q, false>, nb_threads<false>());
    }
    note_launches(1);
    XT_CUDA(cudaGetLastError());
    return XT_OK;
}

template <int Q>
int launch_df(const DevCsr& K, const DevCsr& M, const double* dA, const double* dB,
              const float* x, float2* y, cudaStream_t s)
{
    constexpr int LANES = 8;
    const int threads = 256;
    const int rows_per_block = threads / LANES;
    int blocks = (K.n + rows_per_block - 1) / rows_per_block;
    if (blocks < 1) blocks = 1;
    if (M.same_pattern && M.nnz == K.nnz)
        k_kron_df<Q, LANES, true><<<blocks, threads, 0, s>>>(K.n, K.rowptr.p, K.col.p, K.vdf.p,
                                                             M.rowptr.p, M.col.p, M.vdf.p, dA, dB,
                                                             x, y);
    else
        k_kron_df<Q, LANES, false><<<blocks, threads, 0, s>>>(K.n, K.rowptr.p, K.col.p, K.vdf.p,
                                                              M.rowptr.p, M.col.p, M.vdf.p, dA, dB,
                                                              x, y);
    note_launches(1);
    XT_CUDA(cudaGetLastError());
    return XT_OK;
}

__global__ void k_to_bf16(const double* __restrict__ a, __nv_bfloat16* __restrict__ b, size_t n)
{
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (; i < n; i += stride) b[i] = __double2bfloat16(a[i]);  // round to nearest even
}

int ensure_bf16(DevCsr& A, cudaStream_t s)
{
    if (A.v16.p && A.v16.n == (size_t)A.nnz) return XT_OK;
    XT_TRY(A.v16.alloc((size_t)A.nnz));
    if (A.nnz) {
        k_to_bf16<<<1024, 256, 0, s>>>(A.v64.p, A.v16.p, (size_t)A.nnz);
        note_launches(1);
        XT_CUDA(cudaGetLastError());
    }
    return XT_OK;
}

template <int Q>
int launch_bf16(const DevCsr& K, const DevCsr& M, const double* dA, const double* dB,
                double alpha, double beta, const float* x, float* y, cudaStream_t s)
{
    constexpr int LANES = 8;
    const int threads = 256;
    const int rows_per_block = threads / LANES;
    int blocks = (K.n + rows_per_block - 1) / rows_per_block;
    if (blocks < 1) blocks = 1;
    if (M.same_pattern && M.nnz == K.nnz)
        k_kron_spmm<float, Q, LANES, true, __nv_bfloat16><<<blocks, threads, 0, s>>>(
            K.n, K.rowptr.p, K.col.p, K.v16.p, M.rowptr.p, M.col.p, M.v16.p, dA, dB,
            (float)alpha, (float)beta, x, y);
    else
        k_kron_spmm<float, Q, LANES, false, __nv_bfloat16><<<blocks, threads, 0, s>>>(
            K.n, K.rowptr.p, K.col.p, K.v16.p, M.rowptr.p, M.col.p, M.v16.p, dA, dB,
            (float)alpha, (float)beta, x, y);
    note_launches(1);
    XT_CUDA(cudaGetLastError());
    return XT_OK;
}

int ensure_df(DevCsr& A, cudaStream_t s)
{
    if (A.vdf.p && A.vdf.n == (size_t)A.nnz) return XT_OK;
    XT_TRY(A.vdf.alloc((size_t)A.nnz));
    if (A.nnz) {
        k_to_df<<<1024, 256, 0, s>>>(A.v64.p, A.vdf.p, (size_t)A.nnz);
        note_launches(1);
        XT_CUDA(cudaGetLastError());
    }
    return XT_OK;
}

template <class T, int Q>
int launch_q(const DevCsr& K, const DevCsr& M, const double* dA, const double* dB,
             double alpha, double beta, const T* x, T* y, cudaStream_t s)
{
    constexpr int LANES = 8;
    const int threads = 256;
    const int rows_per_block = threads / LANES;
    int blocks = (K.n + rows_per_block - 1) / rows_per_block;
    if (blocks < 1) blocks = 1;
    if (M.same_pattern && M.nnz == K.nnz)
        k_kron_spmm<T, Q, LANES, true><<<blocks, threads, 0, s>>>(
            K.n, K.rowptr.p, K.col.p, vals<T>(K.v64.p, K.v32.p), M.rowptr.p, M.col.p,
            vals<T>(M.v64.p, M.v32.p), dA, dB, (T)alpha, (T)beta, x, y);
    else
        k_kron_spmm<T, Q, LANES, false><<<blocks, threads, 0, s>>>(
            K.n, K.rowptr.p, K.col.p, vals<T>(K.v64.p, K.v32.p), M.rowptr.p, M.col.p,
            vals<T>(M.v64.p, M.v32.p), dA, dB, (T)alpha, (T)beta, x, y);
    note_launches(1);
    XT_CUDA(cudaGetLastError());
    return XT_OK;
}

}  // namespace

int upload_csr(DevCsr& d, int n, const int* ia, const int* ja, const double* a,
               cudaStream_t s)
{
    if (n <= 0 || !ia || !ja || !a) {
        set_error("upload_csr: bad arguments");
        return XT_ERR_ARG;
    }
    const int nnz = ia[n] - ia[0];
    if (nnz < 0 || ia[0] != 1) {
        set_error("upload_csr: row pointers must be 1-based and non-decreasing");
        return XT_ERR_ARG;
    }
    for (int r = 0; r < n; ++r)
        if (ia[r + 1] < ia[r]) {
            set_error("upload_csr: row pointers decrease");
            return XT_ERR_ARG;
        }
    for (int k = 0; k < nnz; ++k)
        if (ja[k] < 1 || ja[k] > n) {
            set_error("upload_csr: column index out of range");
            return XT_ERR_ARG;
        }
    d.n = n;
    d.nnz = nnz;
    d.same_pattern = false;
    d.vdf.release();  // these two are remade from the new values on first use
    d.v16.release();
    d.nb.ok = false;  // rebuilt by csr_build_node_blocks
    XT_TRY(d.rowptr.upload(ia, (size_t)n + 1, s));
    XT_TRY(d.col.upload(ja, (size_t)(nnz > 0 ? nnz : 0), s));
    XT_TRY(d.v64.upload(a, (size_t)nnz, s));
    XT_TRY(d.v32.alloc((size_t)nnz));
    k_dec_index<<<256, 256, 0, s>>>(d.rowptr.p, (size_t)n + 1);
    if (nnz) {
        k_dec_index<<<1024, 256, 0, s>>>(d.col.p, (size_t)nnz);
        k_to_f32<<<1024, 256, 0, s>>>(d.v64.p, d.v32.p, (size_t)nnz);
    }
    note_launches(3);
    XT_CUDA(cudaGetLastError());
    return XT_OK;
}

void csr_mark_shared_pattern(const DevCsr& K, DevCsr& M, const int* ki, const int* kj,
                             const int* mi, const int* mj)
{
    M.same_pattern = false;
    if (K.n != M.n || K.nnz != M.nnz) return;
    if (std::memcmp(ki, mi, sizeof(int) * ((size_t)K.n + 1)) != 0) return;
    if (std::memcmp(kj, mj, sizeof(int) * (size_t)K.nnz) != 0) return;
    M.same_pattern = true;
}

int csr_build_node_blocks(DevCsr& K, int n, const int* ki, const int* kj, const int* mi,
                          const int* mj, const double* mv, cudaStream_t s)
{
    DevNodeBlocks& nb = K.nb;
    nb.ok = false;
    if (n <= 0 || n % 3 != 0 || K.n != n) return XT_OK;
    const int nodes = n / 3;
    std::vector<int> ptr(nodes + 1, 0), col;
    std::vector<double> m64;
    col.reserve((size_t)K.nnz / 9 + nodes);
    m64.reserve((size_t)K.nnz / 9 + nodes);
    std::vector<int> pos(nodes, -1);  // block index of neighbour node b in the current row
    std::vector<int> from_csr((size_t)K.nnz, -1);
    std::vector<int> order, mask;  // mask: the block entries that K (bits 0..8) and M (9..11) have
    mask.reserve((size_t)K.nnz / 9 + nodes);
    for (int a = 0; a < nodes; ++a) {
        const int first = (int)col.size();
        order.clear();
        for (int c = 0; c < 3; ++c)
            for (int k = ki[3 * a + c] - 1; k < ki[3 * a + c + 1] - 1; ++k) {
                const int b = (kj[k] - 1) / 3;
                if (pos[b] < 0) {
                    pos[b] = 0;
                    order.push_back(b);
                }
            }
        // neighbour nodes in ascending order (the CSR columns are sorted)
        std::sort(order.begin(), order.end());
        for (size_t t = 0; t < order.size(); ++t) pos[order[t]] = first + (int)t;
        col.insert(col.end(), order.begin(), order.end());
        mask.resize(col.size(), 0);
        bool fits = true;
        for (int c = 0; c < 3; ++c)
            for (int k = ki[3 * a + c] - 1; k < ki[3 * a + c + 1] - 1; ++k) {
                const int j = kj[k] - 1, b = j / 3;
                const int e = c * 3 + (j - 3 * b);
                const size_t at = (size_t)pos[b] * 9 + e;
                // one entry a place: a column listed twice stays CSR
                if (at >= (size_t)INT32_MAX || (mask[pos[b]] >> e & 1)) fits = false;
                mask[pos[b]] |= 1 << e;
                from_csr[k] = (int)at;
            }
        // M: m_ab on the three diagonal entries of each block, nothing else
        m64.resize(col.size(), 0.0);
        for (int c = 0; c < 3 && fits; ++c)
            for (int k = mi[3 * a + c] - 1; k < mi[3 * a + c + 1] - 1; ++k) {
                const int j = mj[k] - 1, b = j / 3;
                if (j - 3 * b != c || pos[b] < 0) { fits = false; break; }
                int& mk = mask[pos[b]];
                if ((mk >> (9 + c) & 1) || (mk >> 9 && m64[pos[b]] != mv[k])) { fits = false; break; }
                m64[pos[b]] = mv[k];
                mk |= 1 << (9 + c);
            }
        for (size_t t = first; t < col.size() && fits; ++t)
            if (mask[t] >> 9 != 0 && mask[t] >> 9 != 7) fits = false;
        for (int b : order) pos[b] = -1;
        if (!fits) return XT_OK;  // no exact node-block form: the CSR kernel stays
        ptr[a + 1] = (int)col.size();
    }
    nb.nodes = nodes;
    nb.nblocks = (int)col.size();
    const size_t n9 = (size_t)nb.nblocks * 9;
    XT_TRY(nb.ptr.upload(ptr.data(), ptr.size(), s));
    XT_TRY(nb.col.upload(col.data(), col.size(), s));
    XT_TRY(nb.m64.upload(m64.data(), m64.size(), s));
    XT_TRY(nb.mask.upload(mask.data(), mask.size(), s));
    XT_TRY(nb.from_csr.upload(from_csr.data(), from_csr.size(), s));
    XT_TRY(nb.kdf.alloc(n9));
    XT_TRY(nb.k64.alloc(n9));
    XT_TRY(nb.mdf.alloc((size_t)nb.nblocks));
    // K's values from its CSR copy on the device, zero where that has no entry
    XT_CUDA(cudaMemsetAsync(nb.kdf.p, 0, n9 * sizeof(float2), s));
    XT_CUDA(cudaMemsetAsync(nb.k64.p, 0, n9 * sizeof(double), s));
    if (nb.nblocks) {
        k_to_df<<<256, 256, 0, s>>>(nb.m64.p, nb.mdf.p, (size_t)nb.nblocks);
        note_launches(1);
    }
    nb.ok = true;
    XT_TRY(node_blocks_refresh(K, s));
    XT_CUDA(cudaStreamSynchronize(s));  // host staging vectors go out of scope
    return XT_OK;
}

int node_blocks_refresh(DevCsr& K, cudaStream_t s)
{
    if (!K.nb.ok || K.nnz == 0) return XT_OK;
    k_scatter_blocks<<<std::max(1, std::min(4096, (K.nnz + 255) / 256)), 256, 0, s>>>(
        K.v64.p, K.nb.from_csr.p, K.nb.k64.p, K.nb.kdf.p, (size_t)K.nnz);
    note_launches(1);
    XT_CUDA(cudaGetLastError());
    return XT_OK;
}

int to_f32(const double* a, float* b, size_t n, cudaStream_t s)
{
    if (n == 0) return XT_OK;
    size_t blocks = (n + 255) / 256;
    if (blocks > 4096) blocks = 4096;
    k_to_f32<<<(int)blocks, 256, 0, s>>>(a, b, n);
    note_launches(1);
    XT_CUDA(cudaGetLastError());
    return XT_OK;
}

template <class T>
int kron_spmm(const DevCsr& K, const DevCsr& M, int q, const double* dA,
              const double* dB, double alpha, double beta, const T* x, T* y,
              cudaStream_t s)
{
    if (K.n != M.n || q < 1 || q > 8) {
        set_error("kron_spmm: K and M must have the same order and 1 <= q <= 8");
        return XT_ERR_ARG;
    }
    if (K.n == 0) return XT_OK;
    if constexpr (sizeof(T) == 8) {
        // FP64 in node blocks where the rows fill the GPU (a thread follows a
        // node row's blocks alone, 20 us for 27 of them however few the rows:
        // us in CSR form and in blocks, q = 6, at 325 nodes 17.2 and 20.8, 1,539
        // 18.4 and 20.0, 2,080 27.5 and 20.7; q = 3, 3,025 17.3 and 21.1, 3,751
        // 23.1 and 21.0; q = 1, 14,801 27.5 and 29.4, 22,491 36.4 and 29.4) and
        // the blocks hold little but K's own entries (a
        // place without an entry costs its issue all the same: with blocks
        // less than 5/8 full the CSR kernel does less work).  20 x 20 x 60
        // rod, q = 6: 180 us in CSR form, 132 us in blocks (251 us in CSR form
        // with a mixing branch per output); 10 x 10 x 30 rod 38 and 27.5 us.
        const char* e = std::getenv("XTFEM_KRON_NB");
        const bool large = (long long)q * K.nb.nodes >= (q < 3 ? 16000 : 10500) || (e && std::atoi(e) == 2);
        if (K.nb.ok && large && 5LL * 9 * K.nb.nblocks <= 8LL * K.nnz && nb_enabled()) {
            switch (q) {
            case 1: return launch_nb64<1>(K.nb, dA, dB, alpha, beta, x, y, s);
            case 2: return launch_nb64<2>(K.nb, dA, dB, alpha, beta, x, y, s);
            case 3: return launch_nb64<3>(K.nb, dA, dB, alpha, beta, x, y, s);
            case 4: return launch_nb64<4>(K.nb, dA, dB, alpha, beta, x, y, s);
            case 5: return launch_nb64<5>(K.nb, dA, dB, alpha, beta, x, y, s);
            case 6: return launch_nb64<6>(K.nb, dA, dB, alpha, beta, x, y, s);
            case 7: return launch_nb64<7>(K.nb, dA, dB, alpha, beta, x, y, s);
            default: return launch_nb64<8>(K.nb, dA, dB, alpha, beta, x, y, s);
            }
        }
    }
    switch (q) {
    case 1: return launch_q<T, 1>(K, M, dA, dB, alpha, beta, x, y, s);
    case 2: return launch_q<T, 2>(K, M, dA, dB, alpha, beta, x, y, s);
    case 3: return launch_q<T, 3>(K, M, dA, dB, alpha, beta, x, y, s);
    case 4: return launch_q<T, 4>(K, M, dA, dB, alpha, beta, x, y, s);
    case 5: return launch_q<T, 5>(K, M, dA, dB, alpha, beta, x, y, s);
    case 6: return launch_q<T, 6>(K, M, dA, dB, alpha, beta, x, y, s);
    case 7: return launch_q<T, 7>(K, M, dA, dB, alpha, beta, x, y, s);
    default: return launch_q<T, 8>(K, M, dA, dB, alpha, beta, x, y, s);
    }
}

bool kron_nb_batchable(const DevCsr& K, int q)
{
    return K.nb.ok && q % 2 == 0 && q >= 2 && q <= 8 && nb_enabled();
}

int kron_nb_batch(const FlexStepItem* t, int count, int q, const FlexStepDims& d, cudaStream_t s)
{
    if (count <= 0) return XT_OK;
    // a quarter of the largest system's node rows per block pass: each warp
    // loops over about four row groups (any split gives the same rows)
    const int RPW = q == 2 ? 10 : (q == 4 ? 5 : (q == 6 ? 3 : 2));
    const bool staged = q == 6 && d.nodes_max <= kNbStagedBatch;
    const int threads = staged ? nb_threads<true>() : nb_threads<false>();
    const int rows_per_block = threads / 32 * RPW;
    const int gx = std::max(1, (d.nodes_max + 4 * rows_per_block - 1) / (4 * rows_per_block));
    const dim3 grid(gx, count);
    switch (q) {
    case 2: kb_kron_nb<2, false><<<grid, threads, 0, s>>>(t); break;
    case 4: kb_kron_nb<4, false><<<grid, threads, 0, s>>>(t); break;
    case 6:
        if (staged) kb_kron_nb<6, true><<<grid, threads, 0, s>>>(t);
        else kb_kron_nb<6, false><<<grid, threads, 0, s>>>(t);
        break;
    case 8: kb_kron_nb<8, false><<<grid, threads, 0, s>>>(t); break;
    default: set_error("kron_nb_batch: q must be 2, 4, 6 or 8"); return XT_ERR_ARG;
    }
    note_launches(1);
    XT_CUDA(cudaGetLastError());
    return XT_OK;
}

int kron_spmm_df(DevCsr& K, DevCsr& M, int q, const double* dA, const double* dB, const float* x,
                 float2* y, cudaStream_t s, const int* skip)
{
    if (K.n != M.n || q < 1 || q > 8) {
        set_error("kron_spmm_df: K and M must have the same order and 1 <= q <= 8");
        return XT_ERR_ARG;
    }
    if (K.n == 0) return XT_OK;
    // node blocks: y must be 16-byte aligned (one float4 store per lane)
    if (K.nb.ok && q % 2 == 0 && reinterpret_cast<uintptr_t>(y) % 16 == 0 &&
        reinterpret_cast<uintptr_t>(x) % 8 == 0 && nb_enabled()) {
        switch (q) {
        case 2: return launch_nb<2>(K.nb, dA, dB, x, y, s, skip);
        case 4: return launch_nb<4>(K.nb, dA, dB, x, y, s, skip);
        case 6: return launch_nb<6>(K.nb, dA, dB, x, y, s, skip);
        default: return launch_nb<8>(K.nb, dA, dB, x, y, s, skip);
        }
    }
    XT_TRY(ensure_df(K, s));
    XT_TRY(ensure_df(M, s));
    switch (q) {
    case 1: return launch_df<1>(K, M, dA, dB, x, y, s);
    case 2: return launch_df<2>(K, M, dA, dB, x, y, s);
    case 3: return launch_df<3>(K, M, dA, dB, x, y, s);
    case 4: return launch_df<4>(K, M, dA, dB, x, y, s);
    case 5: return launch_df<5>(K, M, dA, dB, x, y, s);
    case 6: return launch_df<6>(K, M, dA, dB, x, y, s);
    case 7: return launch_df<7>(K, M, dA, dB, x, y, s);
    default: return launch_df<8>(K, M, dA, dB, x, y, s);
    }
}

int kron_spmm_bf16(DevCsr& K, DevCsr& M, int q, const double* dA, const double* dB,
                   double alpha, double beta, const float* x, float* y, cudaStream_t s)
{
    if (K.n != M.n || q < 1 || q > 8) {
        set_error("kron_spmm_bf16: K and M must have the same order and 1 <= q <= 8");
        return XT_ERR_ARG;
    }
    if (K.n == 0) return XT_OK;
    XT_TRY(ensure_bf16(K, s));
    XT_TRY(ensure_bf16(M, s));
    switch (q) {
    case 1: return launch_bf16<1>(K, M, dA, dB, alpha, beta, x, y, s);
    case 2: return launch_bf16<2>(K, M, dA, dB, alpha, beta, x, y, s);
    case 3: return launch_bf16<3>(K, M, dA, dB, alpha, beta, x, y, s);
    case 4: return launch_bf16<4>(K, M, dA, dB, alpha, beta, x, y, s);
    case 5: return launch_bf16<5>(K, M, dA, dB, alpha, beta, x, y, s);
    case 6: return launch_bf16<6>(K, M, dA, dB, alpha, beta, x, y, s);
    case 7: return launch_bf16<7>(K, M, dA, dB, alpha, beta, x, y, s);
    default: return launch_bf16<8>(K, M, dA, dB, alpha, beta, x, y, s);
    }
}

template int kron_spmm<double>(const DevCsr&, const DevCsr&, int, const double*,
                               const double*, double, double, const double*, double*,
                               cudaStream_t);
template int kron_spmm<float>(const DevCsr&, const DevCsr&, int, const double*,
                              const double*, double, double, const float*, float*,
                              cudaStream_t);

}  // namespace xt
