// Forward plane kernels for FFT edges above 224 (sm_100a), where one x-plane
// of the grid no longer fits one CTA's shared memory: the two axes of the
// forward plane transform by separate launches through global memory:
//
//   K1r k_rows_fwd   (x-plane p, block of RB voxel rows): build the rows of
//                    the voxel plane (ligand classes + ordered charge sums, or
//                    the receptor grids) and run the pruned forward z-FFT of each row into A[p][y][kz]
//                    for the NG data rows y;
//   K1c k_cols_fwd   (x-plane p, block of CB columns kz): pruned forward y-FFT
//                    of the columns, in place in A -> A[p][ky][kz].
//
// Each launch owns whole rows (K1r) or whole columns (K1c) of a plane: it
// reads every input of its rows or columns before a barrier and writes the
// results after it, so the in-place pass never races.
//
// References (MEGADOCK, akiyamalab): as the plane kernels -- embedding
// src/fft_process.cpp:306-330, FFT :349-396.
#pragma once
#include "dock_kernels.cuh"

namespace mdb {

constexpr int kNTS = 256;   // threads per CTA of the staged kernels
constexpr int kRB = 16;     // voxel rows per CTA of K1r
constexpr int kCB = 16;     // columns per CTA of K1c

// largest edge whose forward plane kernels keep a whole plane in shared memory
constexpr int kMaxResidentN = 224;

template <int N>
constexpr bool staged() {
    return N > kMaxResidentN;
}

// Row layout of K1r: the R1 blocks of R2 elements at an odd stride, so
// that the second pass (lanes = blocks) reads without bank conflicts (an even
// R2 of 16 put all its lanes on one bank: forward planes at N = 256 40.7 -> 27.7
// us per rotation on the B200, with the pruned inputs of both axes 330 102 -> 86).
template <int N>
struct RowPlan {
    static constexpr int R1 = Plan<N>::R1, R2 = Plan<N>::R2, STR = R2 | 1, PZ = R1 * STR;
};
template <int N>
constexpr size_t rows_smem() { return (size_t)kRB * RowPlan<N>::PZ * sizeof(float2); }
constexpr size_t cols_fwd_smem(int N) { return (size_t)N * (kCB + 1) * sizeof(float2); }

// K1r.  Grid (NG planes, ceil(NG / RB) row blocks, nb), kNTS threads.
// MODE 0: ligand classes (K0 bit planes) and charged cells; MODE 1: receptor
// grids src_r / src_i ([NG][NG][NG] floats).
template <int N, int MODE>
__global__ void __launch_bounds__(kNTS)
    k_rows_fwd(LigandView L, GridView G, const uint32_t *__restrict__ vbits, const int2 *__restrict__ qlist,
               const int *__restrict__ qcount, const float *__restrict__ src_r, const float *__restrict__ src_i,
               float2 *__restrict__ A) {
    constexpr int NG = N / 2, OFF = N / 4;
    constexpr int R1 = RowPlan<N>::R1, R2 = RowPlan<N>::R2, STR = RowPlan<N>::STR, PZ = RowPlan<N>::PZ;
    constexpr int W = VoxShared<NG>::W;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2 *Z = reinterpret_cast<float2 *>(smem_raw);   // RB rows x PZ
    const int p = blockIdx.x, q0 = blockIdx.y * kRB, b = blockIdx.z, tid = threadIdx.x;
    const int nr = min(kRB, NG - q0);
    // element of voxel column s in row r
    auto at = [&](int r, int s) -> float2 & {
        const int z = s + OFF;
        return Z[r * PZ + (z / R2) * STR + z % R2];
    };
    if constexpr (MODE == 1) {
        for (int c = tid; c < nr * NG; c += kNTS) {
            const int r = c / NG, s = c % NG;
            const size_t gidx = ((size_t)p * NG + q0 + r) * NG + s;
            at(r, s) = make_float2(src_r[gidx], src_i[gidx]);
        }
        __syncthreads();
    } else {
        const uint32_t *vb = vbits + ((size_t)b * NG + p) * 2 * NG * W;
        // compile-time trip count, both class words loaded unconditionally
        constexpr int CPT = (kRB * NG + kNTS - 1) / kNTS;
#pragma unroll 8
        for (int k = 0; k < CPT; ++k) {
            const int c = tid + k * kNTS;
            const int r = c / NG, s = c % NG, q = q0 + r;
            if (r < nr) {
                const uint32_t bit = 1u << (s & 31);
                const uint32_t w2 = __ldg(&vb[q * W + (s >> 5)]), w1 = __ldg(&vb[NG * W + q * W + (s >> 5)]);
                const float v = (w2 & bit) ? L.delta : (w1 & bit) ? 1.0f : 0.0f;
                at(r, s) = make_float2(v, 0.f);
            }
        }
        __syncthreads();
        // charged cells of this plane whose row falls in the block
        const int nq = qcount[(size_t)b * NG + p];
        const int2 *ql = qlist + ((size_t)b * NG + p) * NG * NG;
        for (int e = tid; e < nq; e += kNTS) {
            const int2 c = ql[e];
            const int r = c.x / NG - q0;
            if ((unsigned)r < (unsigned)nr) at(r, c.x % NG).y = __int_as_float(c.y);
        }
        __syncthreads();
    }
    // z-FFT of the block's rows: phase 1 in place, phase 2 to global (row y = q + OFF)
    for (int it = tid; it < nr * R2; it += kNTS) {
        const int t = it % R2, r = it / R2;
        float2 *row = Z + r * PZ + t;
        float2 v[R1];
        padded_inputs<N, R1, R2>(v, t, [&](int y) { return row[(y + OFF - t) / R2 * STR]; });
        Dft<R1, -1>::run(v);
        static_for<0, R1>([&](auto k1_) {
            constexpr int k1 = decltype(k1_)::value;
            float2 x = v[k1];
            if constexpr (k1 != 0) x = cmul(x, __ldg(&G.tw[t * k1]));
            row[k1 * STR] = x;
        });
    }
    __syncthreads();
    float2 *Ap = A + ((size_t)b * NG + p) * N * N;
    for (int it = tid; it < nr * R1; it += kNTS) {
        const int r = it / R1, u = it % R1;
        float2 o[R2];
        static_for<0, R2>([&](auto n2) { o[n2] = Z[r * PZ + u * STR + n2]; });
        Dft<R2, -1>::run(o);
        float2 *dst = Ap + (size_t)(q0 + r + OFF) * N;
        static_for<0, R2>([&](auto k2) { dst[u + R1 * k2] = o[k2]; });
    }
}

// K1c.  Grid (NG planes, ceil(N / CB) column blocks, nb), kNTS threads.
// Rows y outside [OFF, OFF + NG) of the z-transformed plane are zero (K1r
// writes only the data rows); the pruned pass never reads them.
template <int N>
__global__ void __launch_bounds__(kNTS) k_cols_fwd(GridView G, float2 *__restrict__ A) {
    constexpr int NG = N / 2, OFF = N / 4, PB = kCB + 1;
    constexpr int R1 = Plan<N>::R1, R2 = Plan<N>::R2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2 *Y = reinterpret_cast<float2 *>(smem_raw);   // N rows x PB
    const int p = blockIdx.x, c0 = blockIdx.y * kCB, b = blockIdx.z, tid = threadIdx.x;
    float2 *Ap = A + ((size_t)b * NG + p) * N * N + c0;
    const int c = tid % kCB;
    const bool live = N % kCB == 0 || c0 + c < N;
    for (int t = tid / kCB; t < R2; t += kNTS / kCB) {
        float2 v[R1];
        padded_inputs<N, R1, R2>(v, t, [&](int y) {
            return live ? Ap[(size_t)(y + OFF) * N + c] : make_float2(0.f, 0.f);
        });
        Dft<R1, -1>::run(v);
        static_for<0, R1>([&](auto k1_) {
            constexpr int k1 = decltype(k1_)::value;
            float2 x = v[k1];
            if constexpr (k1 != 0) x = cmul(x, __ldg(&G.tw[t * k1]));
            Y[(k1 * R2 + t) * PB + c] = x;
        });
    }
    __syncthreads();
    for (int u = tid / kCB; u < R1; u += kNTS / kCB) {
        float2 o[R2];
        fft_phase2<N, -1>(Y + c, PB, u, o);
        if (live) static_for<0, R2>([&](auto k2) { Ap[(size_t)(u + R1 * k2) * N + c] = o[k2]; });
    }
}

}  // namespace mdb
