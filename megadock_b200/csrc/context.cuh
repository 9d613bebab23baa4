// Device context shared by the C-ABI translation units: the per-launch work
// sets, the context struct and the per-size pipeline (Sized<N>).  Each FFT
// size's kernels are instantiated in one of the sized_*.cu files, which
// export a SizedOps table; md_b200.cu dispatches through it, so the sizes
// compile in parallel.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <set>
#include <string>
#include <tuple>
#include <vector>

#include "../../include/md_b200.h"
#include "dock_kernels.cuh"
#include "inverse_kernels.cuh"
#include "staged_kernels.cuh"

using namespace mdb;

namespace mdb {

// Candidate lists per rotation of edge N (inv_groups).
inline size_t cand_groups(int N);

// Per-launch intermediates for `cap` rotations of one launch group.
struct WorkSet {
    float2 *A = nullptr;        // [cap][N/2][N][N]    spectrum planes (K1 -> K2)
    float2 *G = nullptr;        // [cap][N][N/2][N]    Hermitian half (K2 -> K3)
    Cand *cand = nullptr;       // [cap][groups][t]    per-plane candidates (K3 -> K4)
    uint32_t *vbits = nullptr;  // [cap][N/2][2][N/2 * words per row] voxel classes (K0 -> K1)
    int2 *qlist = nullptr;      // [cap][N/2][(N/2)^2] charged cells per voxel plane (K0 -> K1)
    int *qcount = nullptr;      // [cap][N/2]
    MarkEntry *srec = nullptr;  // [cap][na]           atom records bucketed by plane (prep -> K0)
    int *sstart = nullptr;      // [cap][N/2 + 2 kReach + 1]
    int2 *cq = nullptr;         // [cap][na]           charge entries bucketed by plane, atom order
    int *cstart = nullptr;      // [cap][N/2 + 1]
    uint32_t *marks = nullptr;  // [cap][N/2][2][N/2 * words per row] core / surface marks (K0m -> K0)

    void release() {
        cudaFree(A);
        cudaFree(G);
        cudaFree(cand);
        cudaFree(vbits);
        cudaFree(qlist);
        cudaFree(qcount);
        cudaFree(srec);
        cudaFree(sstart);
        cudaFree(cq);
        cudaFree(cstart);
        cudaFree(marks);
        *this = WorkSet();
    }
    // Bytes of each buffer for launch groups of `cap` rotations.
    static constexpr int kBufs = 11;
    struct Sizes {
        size_t b[kBufs];
    };
    static Sizes need(size_t cap, size_t N, size_t t, size_t na) {
        const size_t NG = N / 2;
        return Sizes{{sizeof(float2) * cap * NG * N * N, sizeof(float2) * cap * N * (N / 2) * N,
                      sizeof(Cand) * cap * cand_groups((int)N) * t, sizeof(uint32_t) * cap * NG * 2 * NG * ((NG + 31) / 32),
                      sizeof(int2) * cap * NG * NG * NG, sizeof(int) * cap * NG, sizeof(MarkEntry) * cap * na,
                      sizeof(int) * cap * (NG + 2 * kReach + 1), sizeof(int2) * cap * na, sizeof(int) * cap * (NG + 1),
                      sizeof(uint32_t) * cap * NG * 2 * NG * ((NG + 31) / 32)}};
    }
    cudaError_t allocate(const Sizes &z) {
        cudaError_t e = cudaSuccess;
        void **slot[kBufs] = {(void **)&A,    (void **)&G,    (void **)&cand,   (void **)&vbits,
                              (void **)&qlist, (void **)&qcount, (void **)&srec, (void **)&sstart,
                              (void **)&cq,   (void **)&cstart, (void **)&marks};
        for (int k = 0; k < kBufs && e == cudaSuccess; ++k) e = cudaMalloc(slot[k], z.b[k]);
        return e;
    }
};

constexpr int kLanes = 2;
constexpr int kAutoGroup = 64;   // rotations per launch, at most, where the context chooses (group_of)

}  // namespace

struct md_ctx {
    int device = 0;
    // Identity of this context's captured state for other contexts' graph
    // caches: uid is never reused within the process (a later context at the
    // same heap address gets a new one) and gen is bumped whenever a change
    // invalidates this context's own captured graphs (free_graphs).
    uint64_t uid = 0;
    uint64_t gen = 0;
    cudaStream_t own = nullptr;
    cudaStream_t stream = nullptr;
    cudaStream_t side = nullptr;     // second capture stream of the batched form
    cudaEvent_t fork = nullptr, join = nullptr;
    std::string err;
    // grid
    int N = 0, ng = 0;
    float gw = 0.f;
    float gc_step = 0.f;   // grid_coord[1] - grid_coord[0], the cell width the receptor field reads
    float *d_gc = nullptr;
    float2 *d_tw = nullptr;
    // receptor spectrum [kx][ky][kz] and the receptor voxel grids (for the adjoint)
    float2 *d_Rh = nullptr;
    float *d_recv = nullptr;   // [2][ng^3] real, imaginary
    bool have_receptor = false;
    // ligand
    int na = 0, na_cap = 0;
    float delta = 1.0f;
    float4 *d_atom = nullptr;
    float2 *d_rad2 = nullptr;
    bool have_ligand = false;
    // work sets (lane 0 serves every form; lane 1 the batched graph)
    int batch = 0;   // rotations per launch asked for (md_set_batch); 0 = never asked (group_of)
    int auto_most = kAutoGroup;   // 1 once larger automatic groups had no room (reserve_groups)
    int plan = 0;   // md_set_plan's value (inv_forms)
    int lanes = kLanes;   // work sets / capture streams the batched graph alternates over (1 or 2)
    int cap = 0, cap_t = 0, cap_na = 0;
    WorkSet::Sizes have{};           // bytes held by each work-set buffer
    int sets = 0;                    // work sets allocated (1 or kLanes)
    WorkSet ws[kLanes];
    // A caller that captures its stream records the work sets' addresses: from
    // then on they are replaced by larger ones but not freed (`kept`) until
    // md_release_work, another grid edge or the context's end.
    bool lent = false;
    std::vector<WorkSet> kept;
    char *d_scratch = nullptr;   // scratch of the adjoint and pose-scoring calls (grows to the largest call)
    size_t scratch_cap = 0;
    // staging for host-buffer calls
    float *d_rot = nullptr;
    size_t rot_cap = 0;
    DevPose *d_pose = nullptr;
    size_t pose_cap = 0;
    // captured graphs of the batched form: (first_rot, n_rot, t, batch, rot ptr, pose ptr)
    std::map<std::tuple<int, int, int, int, const float *, DevPose *>, cudaGraphExec_t> graphs;
    // captured graphs of md_dock_pairs, keyed by every argument
    std::map<std::vector<uintptr_t>, cudaGraphExec_t> pair_graphs;
};

static_assert(sizeof(md_pose) == sizeof(DevPose), "pose layout");

#define MD_CUDA(call)                                                                          \
    do {                                                                                       \
        cudaError_t e_ = (call);                                                               \
        if (e_ != cudaSuccess) {                                                               \
            ctx->err = std::string(#call) + ": " + cudaGetErrorString(e_);                     \
            return MD_ERR_CUDA;                                                                \
        }                                                                                      \
    } while (0)

namespace mdb {

// Runs `set` once for each device (the current one), also when several threads
// ask at the same time: a kernel's attributes belong to one device's context.
class OncePerDevice {
public:
    template <class Set>
    cudaError_t run(const Set &set) {
        int device = 0;
        cudaError_t e = cudaGetDevice(&device);
        if (e != cudaSuccess) return e;
        std::lock_guard<std::mutex> lock(m_);
        if (done_.count(device)) return cudaSuccess;
        e = set();
        if (e == cudaSuccess) done_.insert(device);
        return e;
    }

private:
    std::mutex m_;
    std::set<int> done_;
};

// ------------------------------------------------------------------ per-size dispatch
template <int N>
struct Sized {
    static constexpr int NG = N / 2;
    static constexpr int TILES = (N + kLT - 1) / kLT;
    // above 224 the plane transforms run as row and column launches
    // (staged_kernels.cuh)
    static constexpr bool kStaged = staged<N>();
    static size_t smem_fwd() { return (size_t)N * (N + 1) * sizeof(float2); }
    static size_t smem_xrec() { return (size_t)N * kLT * sizeof(float2); }
    static size_t smem_vox() { return vox_bits_smem<NG>(); }
    // the column-block forward form: always for MODE 0 where two CTAs fit, and
    // for every mode where the one-CTA plane does not fit
    template <int MODE>
    static constexpr bool use_cb() {
        return !fwd_full_fits<N>() || (MODE == 0 && fwd_cb_fits<N>());
    }
    template <int MODE, class Set>
    static void set_fwd(Set &set) {
        if constexpr (fwd_pipe<N>()) set((const void *)k_plane_fwd_pipe<N, MODE>, FwdPipe<N>::bytes);
        else if constexpr (use_cb<MODE>()) set((const void *)k_plane_fwd_cb<N, MODE>, fwd_cb_smem<N>());
        else set((const void *)k_plane_fwd<N, MODE>, smem_fwd());
    }
    template <int MODE>
    static void plane_fwd(cudaStream_t s, int nb, const LigandView &L, const GridView &G, const uint32_t *vbits,
                          const int2 *qlist, const int *qcount, const float *sr, const float *si, float2 *A) {
        if constexpr (fwd_pipe<N>())
            k_plane_fwd_pipe<N, MODE><<<dim3(NG, nb), FwdPipe<N>::NT, FwdPipe<N>::bytes, s>>>(
                L, G, vbits, qlist, qcount, sr, si, A);
        else if constexpr (use_cb<MODE>())
            k_plane_fwd_cb<N, MODE><<<dim3(NG, nb), kNT1B, fwd_cb_smem<N>(), s>>>(L, G, vbits, qlist, qcount, sr, si, A);
        else
            k_plane_fwd<N, MODE><<<dim3(NG, nb), kNT1, smem_fwd(), s>>>(L, G, vbits, qlist, qcount, sr, si, A);
    }

    static cudaError_t set_attrs() {
        static OncePerDevice once;
        return once.run(&set_device_attrs);
    }
    static cudaError_t set_device_attrs() {
        cudaError_t e = cudaSuccess;
        auto set = [&](const void *f, size_t bytes) {
            if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        };
        if constexpr (kStaged) {
            set((const void *)k_rows_fwd<N, 0>, rows_smem<N>());
            set((const void *)k_rows_fwd<N, 1>, rows_smem<N>());
            set((const void *)k_cols_fwd<N>, cols_fwd_smem(N));
        } else {
            set_fwd<0>(set);
            set_fwd<1>(set);
        }
        if (e == cudaSuccess) e = set_inv_attrs<N>();
        set((const void *)k_xline_rec<N>, smem_xrec());
        set((const void *)k_vox_bits<NG, true>, smem_vox());
        set((const void *)k_xline_fold<N>, xline_smem<N>());
        return e;
    }

    // Forward plane transforms of nb rotations in the staged form: row launch,
    // then column launch.
    template <int MODE>
    static void staged_fwd(cudaStream_t s, int nb, const LigandView &L, const GridView &G, const uint32_t *vbits,
                           const int2 *qlist, const int *qcount, const float *sr, const float *si, float2 *A) {
        k_rows_fwd<N, MODE><<<dim3(NG, (NG + kRB - 1) / kRB, nb), kNTS, rows_smem<N>(), s>>>(L, G, vbits, qlist, qcount,
                                                                                           sr, si, A);
        k_cols_fwd<N><<<dim3(NG, (N + kCB - 1) / kCB, nb), kNTS, cols_fwd_smem(N), s>>>(G, A);
    }
    template <int MODE>
    static void any_fwd(cudaStream_t s, int nb, const LigandView &L, const GridView &G, const uint32_t *vbits,
                        const int2 *qlist, const int *qcount, const float *sr, const float *si, float2 *A) {
        if constexpr (kStaged) staged_fwd<MODE>(s, nb, L, G, vbits, qlist, qcount, sr, si, A);
        else plane_fwd<MODE>(s, nb, L, G, vbits, qlist, qcount, sr, si, A);
    }

    static void receptor(md_ctx *c, const float *d_r, const float *d_i) {
        GridView G{c->ng, c->gw, 0.f, c->d_gc, c->d_tw};
        LigandView L{0, nullptr, nullptr, 1.f};
        any_fwd<1>(c->stream, 1, L, G, nullptr, nullptr, nullptr, d_r, d_i, c->ws[0].A);
        k_xline_rec<N><<<dim3(N * TILES, 1), kNT, smem_xrec(), c->stream>>>(G, c->ws[0].A, c->d_Rh);
    }

    // Voxelizer of one launch group (atom prep + K0).
    static void voxelize(md_ctx *c, const WorkSet &w, const float *d_rot9, int nb, cudaStream_t s) {
        GridView G{c->ng, c->gw, (float)(c->ng * c->gw) / 2, c->d_gc, c->d_tw};
        LigandView L{c->na, c->d_atom, c->d_rad2, c->delta};
        const int nt = prep_threads(c->na);
        k_atom_prep<NG><<<nb, nt, prep_smem<NG>(nt), s>>>(L, G, d_rot9, w.srec, w.sstart, w.cq, w.cstart);
        k_vox_mark<NG><<<dim3(NG, nb), kNT0, 0, s>>>(L, G, w.srec, w.sstart, w.marks);
        k_vox_bits<NG, true><<<dim3(NG, nb), kNT0, smem_vox(), s>>>(L, G, w.srec, w.sstart, w.cq, w.cstart,
                                                                   w.vbits, w.qlist, w.qcount, w.marks);
    }

    // Voxel grids of nb rotations ([nb][ng^3] real, imaginary) into vr / vi.
    static void voxel_chunk(md_ctx *c, const float *d_rot9, int nb, float *d_vr, float *d_vi) {
        GridView G{c->ng, c->gw, (float)(c->ng * c->gw) / 2, c->d_gc, c->d_tw};
        LigandView L{c->na, c->d_atom, c->d_rad2, c->delta};
        const WorkSet &w = c->ws[0];
        voxelize(c, w, d_rot9, nb, c->stream);
        k_vox_store<NG><<<dim3(NG, nb), kNT0, 0, c->stream>>>(L, w.vbits, w.qlist, w.qcount, d_vr, d_vi);
    }

    // One launch group: nb rotations whose matrices start at d_rot9, on work
    // set w and stream s.  With `ev` set, an event is recorded after each of
    // the five stages.
    static void dock(md_ctx *c, const WorkSet &w, cudaStream_t s, const float *d_rot9, int nb, int rot0, int t,
                     DevPose *d_pose, cudaEvent_t *ev) {
        GridView G{c->ng, c->gw, (float)(c->ng * c->gw) / 2, c->d_gc, c->d_tw};
        LigandView L{c->na, c->d_atom, c->d_rad2, c->delta};
        const float nf3f = (float)((long long)N * N * N);
        voxelize(c, w, d_rot9, nb, s);
        if (ev) cudaEventRecord(ev[1], s);
        any_fwd<0>(s, nb, L, G, w.vbits, w.qlist, w.qcount, nullptr, nullptr, w.A);
        if (ev) cudaEventRecord(ev[2], s);
        k_xline_fold<N><<<xline_grid<N>(nb), XPlan<N>::NT, xline_smem<N>(), s>>>(G, w.A, c->d_Rh, w.G);
        if (ev) cudaEventRecord(ev[3], s);
        launch_inv<N>(s, G, w.G, nb, t, c->plan, w.cand);
        if (ev) cudaEventRecord(ev[4], s);
        static_assert(inv_groups<N>() <= kMergeLists, "k_merge's list places");
        k_merge<<<nb, 256, 0, s>>>(w.cand, inv_groups<N>(), t, N, nf3f, rot0, d_pose);
        if (ev) cudaEventRecord(ev[5], s);
    }
};

}  // namespace mdb

namespace mdb {

// The per-size pipeline entry points of one FFT size.
struct SizedOps {
    int N;
    int cand_groups;   // candidate lists per rotation
    int inv_forms;     // kernels that md_set_plan chooses among
    cudaError_t (*set_attrs)();
    void (*receptor)(md_ctx *, const float *, const float *);
    void (*voxel_chunk)(md_ctx *, const float *, int, float *, float *);
    void (*dock)(md_ctx *, const WorkSet &, cudaStream_t, const float *, int, int, int, DevPose *, cudaEvent_t *);
};

template <int N>
const SizedOps *sized_ops_of() {
    static const SizedOps ops{N,
                              inv_groups<N>(),
                              inv_forms<N>(),
                              &Sized<N>::set_attrs,
                              &Sized<N>::receptor,
                              &Sized<N>::voxel_chunk,
                              &Sized<N>::dock};
    return &ops;
}

// Defined by the sized_*.cu files: the table of N, or nullptr.
const SizedOps *sized_ops_a(int N);
const SizedOps *sized_ops_b(int N);
const SizedOps *sized_ops_c(int N);
const SizedOps *sized_ops_d(int N);
const SizedOps *sized_ops_e(int N);
const SizedOps *sized_ops_f(int N);
const SizedOps *sized_ops_g(int N);
const SizedOps *sized_ops_h(int N);
const SizedOps *sized_ops_i(int N);
const SizedOps *sized_ops_j(int N);
const SizedOps *sized_ops_k(int N);
const SizedOps *sized_ops_l(int N);
const SizedOps *sized_ops_m(int N);
const SizedOps *sized_ops_n(int N);
const SizedOps *sized_ops_o(int N);
const SizedOps *sized_ops_p(int N);
const SizedOps *sized_ops_q(int N);
const SizedOps *sized_ops_r(int N);

inline const SizedOps *sized_ops(int N) {
    if (const SizedOps *o = sized_ops_a(N)) return o;
    if (const SizedOps *o = sized_ops_b(N)) return o;
    if (const SizedOps *o = sized_ops_c(N)) return o;
    if (const SizedOps *o = sized_ops_d(N)) return o;
    if (const SizedOps *o = sized_ops_e(N)) return o;
    if (const SizedOps *o = sized_ops_f(N)) return o;
    if (const SizedOps *o = sized_ops_g(N)) return o;
    if (const SizedOps *o = sized_ops_h(N)) return o;
    if (const SizedOps *o = sized_ops_i(N)) return o;
    if (const SizedOps *o = sized_ops_j(N)) return o;
    if (const SizedOps *o = sized_ops_k(N)) return o;
    if (const SizedOps *o = sized_ops_l(N)) return o;
    if (const SizedOps *o = sized_ops_m(N)) return o;
    if (const SizedOps *o = sized_ops_n(N)) return o;
    if (const SizedOps *o = sized_ops_o(N)) return o;
    if (const SizedOps *o = sized_ops_p(N)) return o;
    if (const SizedOps *o = sized_ops_q(N)) return o;
    return sized_ops_r(N);
}

inline size_t cand_groups(int N) { return sized_ops(N)->cand_groups; }

}  // namespace mdb
