// Inverse plane kernel with a compile-time plan per FFT edge (sm_100a): the
// inverse z-FFT, the fold of the half spectrum, the real inverse along ky and
// the best cells of one x-plane, by one CTA or by a thread-block cluster.  The
// C CTAs of a cluster split the plane by rows for the pass along z and by
// columns for the pass along y; in between every CTA reads its columns from
// the other CTAs' rows through distributed shared memory, so a plane crosses
// global memory once however large it is.
//
// References (MEGADOCK, akiyamalab): inverse FFT src/fft_process.cpp:388,
// top-t :399-458.
#pragma once
#include "dock_kernels.cuh"

namespace mdb {

__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
// Address, in CTA `rank` of the cluster, of this CTA's shared-memory address a.
__device__ __forceinline__ uint32_t cluster_addr(uint32_t a, uint32_t rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ float2 cluster_load(uint32_t a) {
    float2 v;
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a));
    return v;
}

// Split of the inverse plane kernel: z = R1 x R2, ky (N/2) = Q1 x Q2, C CTAs
// of NT threads, OCC of them per SM.
template <int N_, int C_, int R1_, int R2_, int Q1_, int Q2_, int NT_, int OCC_>
struct InvSplit {
    static constexpr int N = N_, C = C_, R1 = R1_, R2 = R2_, Q1 = Q1_, Q2 = Q2_, NT = NT_, OCC = OCC_;
    static constexpr int NH = N / 2;
    static constexpr int RB = (NH + C - 1) / C;   // rows per CTA
    static constexpr int CB = (N + C - 1) / C;    // columns per CTA
    static constexpr int NI = (Q2 + 1) / 2;       // fold items per column
    static constexpr int STR = R2 | 1;            // odd stride of the R2 blocks of a row
    static constexpr int PITCH = R1 * STR;
    static constexpr size_t bytes = sizeof(float2) * ((size_t)RB * PITCH > (size_t)NH * CB ? (size_t)RB * PITCH : (size_t)NH * CB);
    static_assert(R1 * R2 == N && Q1 * Q2 == NH, "splits");
    static constexpr int ITI = (CB * NI + NT - 1) / NT;   // fold items per thread
};

template <class P>
__global__ void __cluster_dims__(P::C, 1, 1) __launch_bounds__(P::NT, P::OCC)
    k_plane_inv(GridView G, const float2 *__restrict__ Gh, int t, int out0, int nsel, Cand *__restrict__ cand) {
    constexpr int N = P::N, NH = P::NH, C = P::C, R1 = P::R1, R2 = P::R2, Q1 = P::Q1, Q2 = P::Q2, NT = P::NT;
    constexpr int RB = P::RB, CB = P::CB, NI = P::NI, STR = P::STR, PITCH = P::PITCH;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2 *S = reinterpret_cast<float2 *>(smem_raw);   // RB rows x PITCH, then NH rows x CB
    auto tw_at = [&](int j) { return __ldg(&G.tw[j]); };
    const int x = blockIdx.x / C, rank = blockIdx.x % C, b = blockIdx.y, tid = threadIdx.x;
    const float2 *Gp = Gh + (((size_t)b * N + x) * NH + (size_t)rank * RB) * N;
    const int rows = min(RB, NH - rank * RB);
    if constexpr (inv_prefetch<N>()) {   // the same rows of the plane one wave ahead
        const unsigned next = blockIdx.y * N + x + (kSMs * P::OCC + C - 1) / C;
        if (tid == 0 && rows > 0 && next < gridDim.y * N)
            prefetch_l2(Gh + ((size_t)next * NH + (size_t)rank * RB) * N, rows * N * (unsigned)sizeof(float2));
    }
    // (1a) inverse kz pass 1 of this CTA's rows, straight from global
    for (int it = tid; it < rows * R2; it += NT) {
        const int row = it / R2, tt = it % R2;
        float2 v[R1];
        static_for<0, R1>([&](auto m_) {
            constexpr int mm = decltype(m_)::value;
            v[mm] = __ldg(&Gp[(size_t)row * N + tt + R2 * mm]);
        });
        Dft<R1, +1>::run(v);
        static_for<0, R1>([&](auto k1_) {
            constexpr int k1 = decltype(k1_)::value;
            float2 xv = v[k1];
            if constexpr (k1 != 0) xv = cmul(xv, conjf2(tw_at(tt * k1)));
            S[row * PITCH + k1 * STR + tt] = xv;
        });
    }
    __syncthreads();
    // (1b) inverse kz pass 2, in place: position u R2 + k2 (column c) holds z = u + R1 k2
    for (int it = tid; it < rows * R1; it += NT) {
        const int row = it / R1, u = it % R1;
        float2 v[R2];
        static_for<0, R2>([&](auto n2) { v[n2] = S[row * PITCH + u * STR + n2]; });
        Dft<R2, +1>::run(v);
        static_for<0, R2>([&](auto k2) { S[row * PITCH + u * STR + k2] = v[k2]; });
    }
    if constexpr (C > 1) cluster_sync();
    else __syncthreads();
    // (2) fold of the half spectrum and pass 1 of the N/2-point inverse along
    // ky for this CTA's columns.  Pass 1 item tt reads rows tt + Q2 m; the fold
    // partner of row k is N/2 - k, so item g takes the row sets g and Q2 - g
    // together, item 0 the sets that pair with themselves (0 and, Q2 even,
    // Q2/2).  The results stay in registers until every CTA of the cluster has
    // read its inputs, then go to this CTA's own buffer.
    float2 va[P::ITI][Q1], vb[P::ITI][Q1];
    auto fold = [&](int it, float2(&a)[Q1], float2(&e)[Q1]) {
        const int cl = it % CB, g = it / CB, c = rank * CB + cl;
        if (g >= NI || c >= N) return;
        const bool two = (Q2 % 2 == 0) || g != 0;
        const int ta = g, tb = g == 0 ? Q2 / 2 : Q2 - g;
        const int pos = c + (c / R2) * (STR - R2);
        const uint32_t col = smem_addr(S) + (uint32_t)pos * 8u;
        auto load = [&](int k) {
            if constexpr (C == 1) return S[k * PITCH + pos];
            const int q = k / RB;
            return cluster_load(cluster_addr(col + (uint32_t)(k - q * RB) * (PITCH * 8u), (uint32_t)q));
        };
        // Z_k = E + i w^k D, E = X_k + conj X_{N/2-k}, D = X_k - conj X_{N/2-k},
        // and its partner; w^{N/2-k} = -conj(w^k)
        auto zpair = [&](float2 &p, float2 &r, int k) {
            const float2 w = conjf2(tw_at(k));
            const float2 w2 = make_float2(-w.x, w.y);
            const float2 e1 = make_float2(p.x + r.x, p.y - r.y), d1 = make_float2(p.x - r.x, p.y + r.y);
            const float2 e2 = make_float2(r.x + p.x, r.y - p.y), d2 = make_float2(r.x - p.x, r.y + p.y);
            const float2 o1 = cmul(w, d1), o2 = cmul(w2, d2);
            p = make_float2(e1.x - o1.y, e1.y + o1.x);
            r = make_float2(e2.x - o2.y, e2.y + o2.x);
        };
        static_for<0, Q1>([&](auto m) { a[m] = load(ta + Q2 * m); });
        if (two) static_for<0, Q1>([&](auto m) { e[m] = load(tb + Q2 * m); });
        if (g == 0) {
            a[0] = make_float2(a[0].x + a[0].y, a[0].x - a[0].y);   // X_0 + i X_{N/2}, both real
            static_for<1, Q1 / 2 + 1>([&](auto m_) {
                constexpr int mm = decltype(m_)::value;
                if constexpr (2 * mm == Q1) {
                    float2 r = a[mm];
                    zpair(a[mm], r, Q2 * mm);
                } else {
                    zpair(a[mm], a[Q1 - mm], Q2 * mm);
                }
            });
            if constexpr (Q2 % 2 == 0) {
                static_for<0, (Q1 + 1) / 2>([&](auto m_) {
                    constexpr int mm = decltype(m_)::value;
                    if constexpr (2 * mm == Q1 - 1) {
                        float2 r = e[mm];
                        zpair(e[mm], r, Q2 / 2 + Q2 * mm);
                    } else {
                        zpair(e[mm], e[Q1 - 1 - mm], Q2 / 2 + Q2 * mm);
                    }
                });
            }
        } else {
            static_for<0, Q1>([&](auto m_) {
                constexpr int mm = decltype(m_)::value;
                zpair(a[mm], e[Q1 - 1 - mm], ta + Q2 * mm);
            });
        }
        Dft<Q1, +1>::run(a);
        if (two) Dft<Q1, +1>::run(e);
        static_for<1, Q1>([&](auto k1_) {
            constexpr int k1 = decltype(k1_)::value;
            a[k1] = cmul(a[k1], conjf2(tw_at(2 * ta * k1)));
            if (two) e[k1] = cmul(e[k1], conjf2(tw_at(2 * tb * k1)));
        });
    };
#pragma unroll
    for (int r = 0; r < P::ITI; ++r) fold(tid + r * NT, va[r], vb[r]);
    if constexpr (C > 1) cluster_sync();
    else __syncthreads();
#pragma unroll
    for (int r = 0; r < P::ITI; ++r) {
        const int it = tid + r * NT, cl = it % CB, g = it / CB;
        if (g < NI && rank * CB + cl < N) {
            const bool two = (Q2 % 2 == 0) || g != 0;
            const int ta = g, tb = g == 0 ? Q2 / 2 : Q2 - g;
            static_for<0, Q1>([&](auto k1) {
                S[(k1 * Q2 + ta) * CB + cl] = va[r][k1];
                if (two) S[(k1 * Q2 + tb) * CB + cl] = vb[r][k1];
            });
        }
    }
    __syncthreads();
    // (3) pass 2 -> scores s[2m], s[2m+1], the column block's best cells
    Cand *out = cand + (((size_t)b * N + x) * C + rank) * t + out0;
    const Cand floor = out0 > 0 ? out[-1] : Cand{0.f, -1};
    if (out0 > 0 && floor.idx < 0) {   // an earlier pass already ran out of cells
        if (tid < nsel) out[tid] = Cand{0.f, -1};
        return;
    }
    const int base = x * N * N;
    select_cells<N, NT, CB * Q1, Q2, 2 * Q1 * N, N % C == 0>(
        [=](int it, float2(&o)[Q2]) {
            const int cc = it % CB, u = it / CB, ccol = rank * CB + cc;
            static_for<0, Q2>([&](auto n2) { o[n2] = S[(u * Q2 + n2) * CB + cc]; });
            Dft<Q2, +1>::run(o);
            const int z = ccol / R2 + R1 * (ccol % R2);
            return (N % C == 0 || ccol < N) ? base + 2 * u * N + z : -1;
        },
        nsel, floor, out);
}

// The plan of every FFT edge but 128 (k_plane_c2r): MDB_INV(N, C, R1, R2, Q1,
// Q2, NT, OCC), the fastest measured.
//
// Bound by instruction issue (ncu, N = 256: 55 % issue active, 18 % of DRAM
// peak), then by the cluster barriers and the loads around them.  C is the
// fewest CTAs that leave room for two or three more clusters on their SMs; a
// plane that fits one CTA three times over is not split.  Leaving the z
// results where pass 2 read them (column c holds z = c / R2 + R1 (c mod R2))
// saves a barrier and a trip through registers, and the two ky passes keep a
// fold item's two row sets in registers across the exchange.  Against the
// forms it replaces (one CTA of 512 threads per plane up to N = 224; a row and
// a column launch through global memory above), us per rotation of the stage
// (B200, one pose): N = 48 0.47 -> 0.27, 96 2.02 -> 1.46, 108 3.09 -> 2.43, 144
// 6.56 -> 5.8, 160 9.1 -> 8.2, 180 16.6 -> 15.0, 224 28.1 -> 26.5, 256 102 ->
// 44, 320 150 -> 116, 330 173 -> 138, 512 677 -> 561 (192 loses, 14.9 -> 15.8,
// and 450 to 504 up to 17 %; the whole calls there gain 53 and 1 to 18 %); ten
// poses at N = 126 9.3 -> 5.7.
template <int N>
struct InvPlan;
#define MDB_INV(N_, ...)                               \
    template <>                                         \
    struct InvPlan<N_> {                                \
        using S = InvSplit<N_, __VA_ARGS__>;            \
    };
MDB_INV(32, 1, 4, 8, 4, 4, 128, 12) MDB_INV(36, 1, 6, 6, 3, 6, 128, 10) MDB_INV(40, 1, 5, 8, 4, 5, 128, 10)
MDB_INV(42, 1, 6, 7, 3, 7, 192, 7) MDB_INV(44, 1, 4, 11, 2, 11, 288, 5) MDB_INV(48, 1, 6, 8, 4, 6, 160, 8)
MDB_INV(50, 1, 5, 10, 5, 5, 160, 8) MDB_INV(54, 1, 6, 9, 3, 9, 288, 5) MDB_INV(56, 1, 7, 8, 4, 7, 224, 7)
MDB_INV(60, 1, 10, 6, 5, 6, 192, 7) MDB_INV(64, 1, 8, 8, 4, 8, 256, 6) MDB_INV(66, 1, 6, 11, 3, 11, 224, 7)
MDB_INV(70, 1, 10, 7, 5, 7, 288, 5) MDB_INV(72, 1, 9, 8, 4, 9, 384, 4) MDB_INV(80, 1, 10, 8, 5, 8, 320, 4)
MDB_INV(84, 1, 12, 7, 7, 6, 256, 5) MDB_INV(88, 1, 8, 11, 4, 11, 288, 5) MDB_INV(90, 1, 9, 10, 5, 9, 256, 5)
MDB_INV(96, 1, 12, 8, 6, 8, 192, 5) MDB_INV(98, 1, 7, 14, 7, 7, 224, 5) MDB_INV(100, 1, 10, 10, 5, 10, 256, 4)
MDB_INV(108, 1, 12, 9, 6, 9, 288, 4) MDB_INV(110, 1, 10, 11, 5, 11, 672, 2) MDB_INV(112, 1, 14, 8, 7, 8, 448, 3)
MDB_INV(120, 1, 12, 10, 5, 12, 384, 3) MDB_INV(126, 1, 9, 14, 7, 9, 320, 3) MDB_INV(132, 1, 11, 12, 6, 11, 416, 2)
MDB_INV(140, 1, 14, 10, 5, 14, 512, 2) MDB_INV(144, 1, 9, 16, 8, 9, 384, 2) MDB_INV(150, 1, 10, 15, 5, 15, 608, 2)
MDB_INV(154, 1, 14, 11, 7, 11, 480, 2) MDB_INV(160, 1, 10, 16, 8, 10, 416, 2) MDB_INV(162, 2, 9, 18, 9, 9, 416, 3)
MDB_INV(168, 2, 14, 12, 7, 12, 256, 3) MDB_INV(176, 2, 11, 16, 8, 11, 544, 2)
MDB_INV(180, 2, 12, 15, 6, 15, 384, 3) MDB_INV(192, 2, 12, 16, 6, 16, 384, 2)
MDB_INV(196, 2, 14, 14, 7, 14, 352, 2) MDB_INV(198, 2, 18, 11, 9, 11, 608, 2)
MDB_INV(200, 2, 20, 10, 5, 20, 512, 2) MDB_INV(210, 2, 15, 14, 7, 15, 448, 2)
MDB_INV(216, 2, 18, 12, 9, 12, 352, 2) MDB_INV(220, 4, 11, 20, 10, 11, 352, 3)
MDB_INV(224, 2, 14, 16, 7, 16, 448, 2) MDB_INV(240, 4, 15, 16, 8, 15, 480, 3)
MDB_INV(242, 4, 11, 22, 11, 11, 384, 3) MDB_INV(250, 4, 10, 25, 5, 25, 416, 2)
MDB_INV(252, 8, 18, 14, 9, 14, 224, 5) MDB_INV(256, 8, 16, 16, 8, 16, 256, 5)
MDB_INV(264, 4, 22, 12, 11, 12, 416, 2) MDB_INV(270, 8, 18, 15, 9, 15, 288, 4)
MDB_INV(280, 8, 14, 20, 10, 14, 256, 4) MDB_INV(288, 4, 18, 16, 9, 16, 576, 2)
MDB_INV(294, 4, 14, 21, 7, 21, 416, 2) MDB_INV(300, 4, 20, 15, 6, 25, 512, 2)
MDB_INV(308, 8, 14, 22, 11, 14, 288, 3) MDB_INV(320, 8, 20, 16, 10, 16, 320, 3)
MDB_INV(324, 8, 18, 18, 9, 18, 384, 3) MDB_INV(330, 8, 22, 15, 11, 15, 352, 3)
MDB_INV(336, 8, 16, 21, 8, 21, 480, 2) MDB_INV(350, 8, 14, 25, 7, 25, 288, 3)
MDB_INV(352, 4, 22, 16, 8, 22, 992, 1) MDB_INV(360, 8, 20, 18, 9, 20, 480, 2)
MDB_INV(378, 8, 18, 21, 9, 21, 544, 2) MDB_INV(384, 4, 24, 16, 12, 16, 768, 1)
MDB_INV(392, 8, 28, 14, 7, 28, 352, 2) MDB_INV(396, 8, 22, 18, 9, 22, 576, 2)
MDB_INV(400, 8, 25, 16, 10, 20, 512, 2) MDB_INV(420, 8, 21, 20, 14, 15, 448, 2)
MDB_INV(432, 4, 18, 24, 12, 18, 992, 1) MDB_INV(440, 8, 22, 20, 11, 20, 576, 2)
MDB_INV(448, 8, 28, 16, 14, 16, 448, 2) MDB_INV(450, 8, 25, 18, 15, 15, 480, 2)
MDB_INV(462, 8, 22, 21, 11, 21, 640, 2) MDB_INV(480, 8, 24, 20, 12, 20, 608, 1)
MDB_INV(484, 8, 22, 22, 11, 22, 672, 1) MDB_INV(486, 8, 18, 27, 9, 27, 864, 1)
MDB_INV(490, 8, 14, 35, 7, 35, 576, 1) MDB_INV(500, 8, 20, 25, 10, 25, 832, 1)
MDB_INV(504, 8, 24, 21, 12, 21, 704, 1) MDB_INV(512, 8, 16, 32, 16, 16, 512, 1)
#undef MDB_INV

// Whether edge N runs k_plane_c2r, whose warp-owned z rows and in-place fold
// still win where the whole plan fits 40 registers (N = 128: 3.2 against 3.4
// us per rotation).
template <int N>
constexpr bool inv_plane_owned() {
    return N == 128;
}

// Forms of the stage that md_set_plan chooses among at edge N; plan 1 is form 1
// where there are two, every other plan form 0.
template <int N>
constexpr int inv_forms() {
    return inv_plane_owned<N>() ? 2 : 1;
}

// Candidate lists per rotation of edge N: one per CTA of each x plane.
template <int N>
constexpr int inv_groups() {
    if constexpr (inv_plane_owned<N>()) return N;
    else return N * InvPlan<N>::S::C;
}

// The inverse plane stage of nb rotations, nsel poses from place out0 on.
template <int N>
cudaError_t set_inv_attrs() {
    auto set = [](const void *f, size_t bytes) {
        return cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    };
    if constexpr (inv_plane_owned<N>()) {
        cudaError_t e = set((const void *)k_plane_c2r<N, 0>, c2r_smem<N, 0>());
        if (e == cudaSuccess) e = set((const void *)k_plane_c2r<N, 1>, c2r_smem<N, 1>());
        return e;
    } else {
        using P = typename InvPlan<N>::S;
        return set((const void *)k_plane_inv<P>, P::bytes);
    }
}
template <int N>
void launch_inv(cudaStream_t s, const GridView &G, const float2 *Gh, int nb, int t, int plan, Cand *cand) {
    for (int out0 = 0; out0 < t; out0 += kSelMax) {
        const int nsel = t - out0 < kSelMax ? t - out0 : kSelMax;
        if constexpr (inv_plane_owned<N>()) {
            if (plan == 1) k_plane_c2r<N, 1><<<dim3(N, nb), kNT, c2r_smem<N, 1>(), s>>>(G, Gh, t, out0, nsel, cand);
            else k_plane_c2r<N, 0><<<dim3(N, nb), kNT, c2r_smem<N, 0>(), s>>>(G, Gh, t, out0, nsel, cand);
        } else {
            using P = typename InvPlan<N>::S;
            k_plane_inv<P><<<dim3(N * P::C, nb), P::NT, P::bytes, s>>>(G, Gh, t, out0, nsel, cand);
        }
    }
}

}  // namespace mdb
