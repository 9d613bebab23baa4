// Fused docking kernels (sm_100a).  One rotation's score grid is produced by
// three plane/line passes that never store the full forward spectrum of the
// ligand nor the full score grid:
//
//   K1 plane_fwd   (rotation, voxel x-plane p): rotate the ligand, voxelize
//                  plane p (rPSC real part + charge imaginary part, bit-exact
//                  with MEGADOCK's CPU path), 2D forward FFT over (y, z) in
//                  shared memory, store the plane's spectrum  A[p][ky][kz].
//   K2 xline       (rotation, ky, 16 or 8 kz lines): forward FFT along x of the
//                  ng non-zero planes, multiply by conj(R^), inverse FFT along
//                  x, store G[x][ky][kz].
//   K3 plane_inv   (rotation, x-plane): inverse FFT over (ky, kz) -> real score
//                  plane, per-plane top-t candidates.
//   K4 merge       (rotation): top-t of the per-plane candidates with
//                  MEGADOCK's selection rules -> pose records.
//
// References (MEGADOCK, akiyamalab):
//   rotation           src/docking.cpp:368-396
//   rPSC voxelization  src/ligand.cpp:20-198 (+ precalc :241-260, voxel_init
//                      src/protein.cpp:134-165)
//   charges            src/ligand.cpp:200-239
//   embedding          src/fft_process.cpp:306-330
//   FFT / product      src/fft_process.cpp:333-396 (FFTW) and :537-558 (cuFFT)
//   top-t              src/fft_process.cpp:399-458
#pragma once
#include <climits>

#include "fft_dev.cuh"

namespace mdb {

constexpr int kNT = 512;          // threads per CTA for the plane kernels
#ifndef MDB_K1_NT
#define MDB_K1_NT 1024
#endif
constexpr int kNT1 = MDB_K1_NT;   // threads per CTA of the forward plane kernel (one CTA per SM)
constexpr int kLT = 32;           // lines per CTA in the x-line kernel
constexpr int kMaxLigAtoms = 32768;

struct DevPose {
    float score;
    int rot, i, j, k;
};

struct LigandView {
    int na;
    const float4 *__restrict__ atom;   // centred x, y, z and charge
    const float2 *__restrict__ rad2;   // (R^2 * 1.5, R^2 * 1.0)
    float delta;                       // ligand core value (-b)
};

struct GridView {
    int ng;                            // voxel edge (N/2)
    float gw;                          // grid width (Protein::grid_width)
    float pad;                         // ng * gw / 2 (Ligand::electro)
    const float *__restrict__ gc;      // grid centre coordinates [ng]
    const float2 *__restrict__ tw;     // exp(-2 pi i j / N), j < N
};

// ------------------------------------------------------------------ voxelization
// Shared-memory bit planes for one CTA's x-plane p.
template <int NG>
struct VoxShared {
    static constexpr int W = (NG + 31) / 32;
    uint32_t core[5][NG * W];   // planes p-2 .. p+2
    uint32_t surf[3][NG * W];   // planes p-1 .. p+1
};

__device__ __forceinline__ float rot_x(const float *m, float x, float y, float z) {
    // (m0*x + m1*y) + m2*z in float, no contraction (src/docking.cpp:390-392)
    return __fadd_rn(__fadd_rn(__fmul_rn(m[0], x), __fmul_rn(m[1], y)), __fmul_rn(m[2], z));
}

// (int)(c / gw + ng/2), the atom's nearest-cell search origin (src/ligand.cpp:71-73)
__device__ __forceinline__ int box_origin(float c, float gw, int ng) {
    return __float2int_rz(__fadd_rn(__fdiv_rn(c, gw), (float)(ng / 2)));
}

// clamp((int)((c + pad) / gw)), the charge cell (src/ligand.cpp:219-221)
__device__ __forceinline__ int charge_cell(float c, float pad, float gw, int ng) {
    int v = __float2int_rz(__fdiv_rn(__fadd_rn(c, pad), gw));
    return max(0, min(ng - 1, v));
}

__device__ __forceinline__ float sqdist(float c, float g) {
    const float d = __fsub_rn(c, g);
    return __fmul_rn(d, d);
}

// Per-rotation atom record for the voxelizer: rotated coordinates, the
// search-box origin (src/ligand.cpp:71-73) and both sphere radii squared.
struct MarkEntry {
    float4 pos;   // rotated x, y, z and R^2 * 1.5
    int4 box;     // search-box origin i, j, k and R^2 * 1.0 (as bits)
};

// Shape buckets: atoms are grouped by box origin i, shifted by kReach so that
// origins in [-kReach, ng + kReach) map to [0, ng + 2 kReach).
constexpr int kReach = 4;

// Mark core / surface bits of the planes around p.  The atoms whose box can
// reach those planes are the contiguous bucket range [lo, hi) of the rotation's
// record array; every (atom, plane, row) of their boxes is one task, spread
// evenly over the block; a task tests the row's cells and ORs the bits (the
// marks are ORs, so the order of atoms does not matter).
template <int NG>
__device__ void vox_mark(VoxShared<NG> &vs, const MarkEntry *__restrict__ rec, int lo, int hi, const GridView &G,
                         int p, bool general_delta) {
    constexpr int W = VoxShared<NG>::W;
    const int ng = G.ng;
    const int plo = general_delta ? -2 : -1;
    const int nplanes = general_delta ? 5 : 3;
    const int ntask = (hi - lo) * nplanes * 5;
    for (int task = threadIdx.x; task < ntask; task += blockDim.x) {
        const int e = task / (nplanes * 5);
        const int rem = task % (nplanes * 5);
        const int i = p + plo + rem / 5;
        const MarkEntry me = rec[lo + e];
        const int j = me.box.y - 2 + rem % 5;
        if (i < 0 || i >= ng || i < me.box.x - 2 || i > me.box.x + 2 || j < 0 || j >= ng) continue;
        const float rc2 = me.pos.w, rs2 = __int_as_float(me.box.w);
        const float d2 = __fadd_rn(sqdist(me.pos.x, __ldg(&G.gc[i])), sqdist(me.pos.y, __ldg(&G.gc[j])));
        // d3 = d2 + dz^2 >= d2 and R^2 <= 1.5 R^2: a row outside the core
        // disc has no cell in either sphere
        if (!(d2 < rc2)) continue;
        // the row's (at most 5) cells as bits of a 64-bit window from word wb
        const int ka = max(me.box.z - 2, 0), kb = min(me.box.z + 3, ng);
        const int wb = ka >> 5;
        unsigned long long cm = 0ull, sm = 0ull;
        for (int k = ka; k < kb; ++k) {
            const float d3 = __fadd_rn(d2, sqdist(me.pos.z, __ldg(&G.gc[k])));
            const unsigned long long bit = 1ull << (k - 32 * wb);
            if (d3 < rc2) cm |= bit;
            if (d3 < rs2) sm |= bit;
        }
        const int slot = i - p + 2;
        const bool do_surf = (i >= p - 1 && i <= p + 1);
        uint32_t *crow = &vs.core[slot][j * W + wb];
        if ((uint32_t)cm) atomicOr(crow, (uint32_t)cm);
        if (cm >> 32) atomicOr(crow + 1, (uint32_t)(cm >> 32));
        if (do_surf) {
            uint32_t *srow = &vs.surf[slot - 1][j * W + wb];
            if ((uint32_t)sm) atomicOr(srow, (uint32_t)sm);
            if (sm >> 32) atomicOr(srow + 1, (uint32_t)(sm >> 32));
        }
    }
    __syncthreads();
}

// The class bits of 32 cells (row q, word w) of plane p at once: c2 = "value
// delta" (core), c1 = "value 1.0" (surface).
template <int NG>
__device__ __forceinline__ uint32_t vw_core(const VoxShared<NG> &vs, int slot, int q, int w) {
    constexpr int W = VoxShared<NG>::W;
    return (q < 0 || q >= NG || w < 0 || w >= W) ? 0u : vs.core[slot][q * W + w];
}

template <int NG>
__device__ __forceinline__ uint32_t vw_surf(const VoxShared<NG> &vs, int slot, int q, int w) {
    constexpr int W = VoxShared<NG>::W;
    return (q < 0 || q >= NG || w < 0 || w >= W) ? 0u : vs.surf[slot - 1][q * W + w];
}

// bits s of word w with 1 <= s <= ng - 2
__device__ __forceinline__ uint32_t vw_inner(int w, int ng) {
    uint32_t m = 0xffffffffu;
    const int s0 = 32 * w;
    if (s0 < 1) m &= ~1u;
    const int hi = ng - 2 - s0;   // last kept bit
    if (hi < 0) return 0u;
    if (hi < 31) m &= (2u << hi) - 1u;
    return m;
}

// Core cells of (slot, q, w) that survive the swollen-surface scrape
// (src/ligand.cpp:110-134): interior cells with a 6-neighbour outside the core
// lose their core value.
template <int NG>
__device__ __forceinline__ uint32_t vw_surv(const VoxShared<NG> &vs, int slot, int i, int q, int w, int ng) {
    const uint32_t c = vw_core<NG>(vs, slot, q, w);
    if (!c) return 0u;
    const uint32_t left = (c << 1) | (vw_core<NG>(vs, slot, q, w - 1) >> 31);    // core at s - 1
    const uint32_t right = (c >> 1) | (vw_core<NG>(vs, slot, q, w + 1) << 31);   // core at s + 1
    const uint32_t nb = vw_core<NG>(vs, slot - 1, q, w) & vw_core<NG>(vs, slot + 1, q, w) &
                        vw_core<NG>(vs, slot, q - 1, w) & vw_core<NG>(vs, slot, q + 1, w) & left & right;
    const bool inner_iq = i >= 1 && i <= ng - 2 && q >= 1 && q <= ng - 2;
    const uint32_t interior = inner_iq ? vw_inner(w, ng) : 0u;
    return c & (~interior | nb);
}

// cells of class 0 (neither a surviving core cell nor a surface cell)
template <int NG>
__device__ __forceinline__ uint32_t vw_empty(const VoxShared<NG> &vs, int slot, int i, int q, int w, int ng) {
    return ~(vw_surv<NG>(vs, slot, i, q, w, ng) | vw_surf<NG>(vs, slot, q, w));
}

template <int NG>
__device__ __forceinline__ void vox_code_words(const VoxShared<NG> &vs, int p, int q, int w, int ng,
                                               bool general_delta, uint32_t &c2, uint32_t &c1) {
    const uint32_t surv = vw_surv<NG>(vs, 2, p, q, w, ng);
    c2 = surv;
    c1 = vw_surf<NG>(vs, 2, q, w) & ~surv;
    if (!general_delta || !surv) return;
    if (!(p >= 1 && p <= ng - 2 && q >= 1 && q <= ng - 2)) return;
    const uint32_t e0 = vw_empty<NG>(vs, 2, p, q, w, ng);
    const uint32_t es = (e0 << 1) | (vw_empty<NG>(vs, 2, p, q, w - 1, ng) >> 31) | (e0 >> 1) |
                        (vw_empty<NG>(vs, 2, p, q, w + 1, ng) << 31);
    const uint32_t ez = vw_empty<NG>(vs, 1, p - 1, q, w, ng) | vw_empty<NG>(vs, 3, p + 1, q, w, ng) |
                        vw_empty<NG>(vs, 2, p, q - 1, w, ng) | vw_empty<NG>(vs, 2, p, q + 1, w, ng);
    const uint32_t demote = surv & vw_inner(w, ng) & (es | ez);
    c2 = surv & ~demote;
    c1 |= demote;
}

// ------------------------------------------------------------------ atom prep
// Once per rotation: rotate every atom (src/docking.cpp:386-393), compute its
// search-box origin and its charge cell (src/ligand.cpp:71-73, 219-221) and
// bucket the atoms by x-plane:
//  * shape records rec[b][.] grouped by box origin i (any order inside a
//    bucket), bucket starts sstart[b][0 .. ng + 2 kReach];
//  * charge entries cq[b][.] = (cell j * ng + k, charge bits) grouped by the
//    charge cell's plane, in ascending atom order inside a bucket (the order
//    in which MEGADOCK adds charges), bucket starts cstart[b][0 .. ng].
//
// One CTA per rotation, its latency the whole cost of a small launch group.
// The charge entries are a stable counting sort: warp w owns the w-th run of
// atoms, counts its atoms per plane, and after one scan over (plane, warp)
// writes them in atom order (one warp walking every atom before).  With the
// charge sums from a shared list (k_vox_bits) instead of an array of NG^2 first
// entries, the voxelizer stage went, in us per rotation (B200): N = 128, 1,544
// atoms 0.67 -> 0.63; 160, 3,518 1.84 -> 1.48; 216, 10,074 8.8 -> 5.0; 256,
// 12,000 15.0 -> 6.9; 330, 12,000 (8 rotations per launch) 53 -> 19.5.
constexpr int kNTP = 256;            // threads for ligands of up to kPrepWide atoms
constexpr int kNTPWide = 1024;       // threads above
constexpr int kPrepWide = 3072;
inline int prep_threads(int na) { return na <= kPrepWide ? kNTP : kNTPWide; }

// Exclusive prefix sum of a[0 .. n) in place by the first warp; returns the total.
__device__ __forceinline__ int warp_scan(int *a, int n) {
    const int lane = threadIdx.x & 31;
    int acc = 0;
    for (int i0 = 0; i0 < n; i0 += 32) {
        const int i = i0 + lane;
        const int v = i < n ? a[i] : 0;
        int s = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += u;
        }
        if (i < n) a[i] = acc + s - v;
        acc += __shfl_sync(0xffffffffu, s, 31);
    }
    return acc;
}

template <int NG>
constexpr size_t prep_smem(int threads) {
    return sizeof(int) * (size_t)(threads / 32) * NG;
}

template <int NG>
__global__ void __launch_bounds__(kNTPWide)
    k_atom_prep(LigandView L, GridView G, const float *__restrict__ rotm, MarkEntry *__restrict__ rec,
                int *__restrict__ sstart, int2 *__restrict__ cq, int *__restrict__ cstart) {
    constexpr int NBS = NG + 2 * kReach;
    extern __shared__ __align__(16) int wc[];   // [plane][warp] charge counts, then write positions
    __shared__ int cnt_s[NBS], cnt_c[NG];
    __shared__ float m[9];
    const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
    if (tid < 9) m[tid] = rotm[(size_t)b * 9 + tid];
    for (int i = tid; i < NBS; i += blockDim.x) cnt_s[i] = 0;
    for (int i = tid; i < NG * nw; i += blockDim.x) wc[i] = 0;
    __syncthreads();
    const int run = ((L.na + nw - 1) / nw + 31) & ~31;   // atoms per warp, whole steps of 32
    const int l0 = min(warp * run, L.na), l1 = min(l0 + run, L.na);
    for (int l = l0 + lane; l < l1; l += 32) {
        const float4 a = __ldg(&L.atom[l]);
        const float xr = rot_x(m, a.x, a.y, a.z);
        const int sb = box_origin(xr, G.gw, G.ng) + kReach;
        if (sb >= 0 && sb < NBS) atomicAdd(&cnt_s[sb], 1);
        atomicAdd(&wc[charge_cell(xr, G.pad, G.gw, G.ng) * nw + warp], 1);
    }
    __syncthreads();
    int *ss = sstart + (size_t)b * (NBS + 1);
    int *cs = cstart + (size_t)b * (NG + 1);
    // plane totals, their starts, and each warp's start inside its planes
    for (int i = tid; i < NG; i += blockDim.x) {
        int n = 0;
        for (int w = 0; w < nw; ++w) n += wc[i * nw + w];
        cnt_c[i] = n;
    }
    __syncthreads();
    if (warp == 0) {
        const int n = warp_scan(cnt_s, NBS);
        if (lane == 0) ss[NBS] = n;
        const int nc = warp_scan(cnt_c, NG);
        if (lane == 0) cs[NG] = nc;
    }
    __syncthreads();
    for (int i = tid; i < NBS; i += blockDim.x) ss[i] = cnt_s[i];
    for (int i = tid; i < NG; i += blockDim.x) {
        int at = cnt_c[i];
        cs[i] = at;
        for (int w = 0; w < nw; ++w) {
            const int n = wc[i * nw + w];
            wc[i * nw + w] = at;
            at += n;
        }
    }
    __syncthreads();
    MarkEntry *rb = rec + (size_t)b * L.na;
    int2 *qb = cq + (size_t)b * L.na;
    for (int base = l0; base < l1; base += 32) {
        const int l = base + lane;
        int ie = -1, key = 0;
        float q = 0.f;
        if (l < l1) {
            const float4 a = __ldg(&L.atom[l]);
            const float xr = rot_x(m, a.x, a.y, a.z);
            const float yr = rot_x(m + 3, a.x, a.y, a.z);
            const float zr = rot_x(m + 6, a.x, a.y, a.z);
            const int i2 = box_origin(xr, G.gw, G.ng);
            const int sb = i2 + kReach;
            if (sb >= 0 && sb < NBS) {
                const float2 r2 = __ldg(&L.rad2[l]);
                const int pos = atomicAdd(&cnt_s[sb], 1);
                rb[pos].pos = make_float4(xr, yr, zr, r2.x);
                rb[pos].box = make_int4(i2, box_origin(yr, G.gw, G.ng), box_origin(zr, G.gw, G.ng), __float_as_int(r2.y));
            }
            ie = charge_cell(xr, G.pad, G.gw, G.ng);
            key = charge_cell(yr, G.pad, G.gw, G.ng) * G.ng + charge_cell(zr, G.pad, G.gw, G.ng);
            q = a.w;
        }
        const uint32_t grp = __match_any_sync(0xffffffffu, ie);
        int pos = 0;
        if (ie >= 0) pos = wc[ie * nw + warp] + __popc(grp & ((1u << lane) - 1u));
        __syncwarp();
        if (ie >= 0) {
            qb[pos] = make_int2(key, __float_as_int(q));
            if (lane == 31 - __clz(grp)) wc[ie * nw + warp] += __popc(grp);
        }
        __syncwarp();
    }
}

// ------------------------------------------------------------------ K0
// Ligand grid of one (rotation, x-plane p), everything but the FFT:
//  * real part: core / surface marks of the atoms near p (task-parallel), the
//    swollen-surface scrape and the surface fill (src/ligand.cpp:20-198),
//    stored as two bit planes: vbits[b][p][0] = "value delta",
//    vbits[b][p][1] = "value 1.0";
//  * imaginary part: per-cell charge sums in ascending atom order from 0.0
//    (src/ligand.cpp:200-239), stored as a compact list of the plane's charged
//    cells qlist[b][p][e] = (q * NG + s, sum as bits), qcount[b][p] entries.
constexpr int kNT0 = 256;

// K0m: the core and surface marks of one (rotation, x-plane i), computed once
// per plane and stored for the K0 CTAs of planes i-2 .. i+2 (each of which
// would otherwise mark its neighbour planes itself):
//   marks[b][i][0] = core bits, marks[b][i][1] = surface bits (rows of W words).
// Same tests and rounding as vox_mark, so the bits are the same.
template <int NG>
__global__ void __launch_bounds__(kNT0)
    k_vox_mark(LigandView L, GridView G, const MarkEntry *__restrict__ rec, const int *__restrict__ sstart,
               uint32_t *__restrict__ marks) {
    constexpr int W = VoxShared<NG>::W;
    constexpr int NBS = NG + 2 * kReach;
    __shared__ uint32_t cs[2][NG * W];
    const int i = blockIdx.x, b = blockIdx.y, tid = threadIdx.x;
    for (int w = tid; w < 2 * NG * W; w += blockDim.x) (&cs[0][0])[w] = 0u;
    __syncthreads();
    const int ng = G.ng;
    const int *ss = sstart + (size_t)b * (NBS + 1);
    const int lo = ss[max(i - 2 + kReach, 0)], hi = ss[min(i + 2 + kReach + 1, NBS)];
    const MarkEntry *rb = rec + (size_t)b * L.na;
    for (int task = tid; task < (hi - lo) * 5; task += blockDim.x) {
        const MarkEntry me = rb[lo + task / 5];
        const int j = me.box.y - 2 + task % 5;
        if (i >= ng || i < me.box.x - 2 || i > me.box.x + 2 || j < 0 || j >= ng) continue;
        const float rc2 = me.pos.w, rs2 = __int_as_float(me.box.w);
        const float d2 = __fadd_rn(sqdist(me.pos.x, __ldg(&G.gc[i])), sqdist(me.pos.y, __ldg(&G.gc[j])));
        if (!(d2 < rc2)) continue;
        const int ka = max(me.box.z - 2, 0), kb = min(me.box.z + 3, ng);
        const int wb = ka >> 5;
        unsigned long long cm = 0ull, sm = 0ull;
        for (int k = ka; k < kb; ++k) {
            const float d3 = __fadd_rn(d2, sqdist(me.pos.z, __ldg(&G.gc[k])));
            const unsigned long long bit = 1ull << (k - 32 * wb);
            if (d3 < rc2) cm |= bit;
            if (d3 < rs2) sm |= bit;
        }
        uint32_t *crow = &cs[0][j * W + wb], *srow = &cs[1][j * W + wb];
        if ((uint32_t)cm) atomicOr(crow, (uint32_t)cm);
        if (cm >> 32) atomicOr(crow + 1, (uint32_t)(cm >> 32));
        if ((uint32_t)sm) atomicOr(srow, (uint32_t)sm);
        if (sm >> 32) atomicOr(srow + 1, (uint32_t)(sm >> 32));
    }
    __syncthreads();
    uint32_t *dst = marks + ((size_t)b * NG + i) * 2 * NG * W;
    for (int w = tid; w < 2 * NG * W; w += blockDim.x) dst[w] = (&cs[0][0])[w];
}

// Whether k_vox_bits keeps its bit planes (VoxShared) and output words in
// dynamic shared memory: where their static form would pass 40 KB of the 48 KB
// a kernel may declare statically (NG > 160).
template <int NG>
constexpr bool vox_bits_dyn() {
    return sizeof(VoxShared<NG>) + sizeof(uint32_t) * 2 * NG * VoxShared<NG>::W > 40 * 1024;
}

// Dynamic shared memory of k_vox_bits: the bit planes and the output words
// (vox_bits_dyn).
template <int NG>
constexpr size_t vox_bits_smem() {
    return vox_bits_dyn<NG>() ? sizeof(VoxShared<NG>) + sizeof(uint32_t) * 2 * NG * VoxShared<NG>::W : 0;
}

// Charge entries of a plane k_vox_bits stages in shared memory at once.
constexpr int kVoxQ = 512;

// The charge sums of a plane with more than kVoxQ entries (some 20,000 atoms
// and more, or a ligand that hangs out of the grid, whose charges are clamped to
// the outer cells): the entries pass through shared memory a block's width at a
// time, in atom order, the first of a cell in a step adds that cell's entries
// to the cell's sum, and the sums stay in shared memory, 8 W rows of the plane
// after one another in the bit planes' room (`acc`).  Walking all entries once
// per cell instead takes nq steps a cell, from global memory.  The voxelizer
// stage of one rotation with 32,768 atoms, ms (B200; by that walk, and by a walk
// from an array of first entries per cell before it): N = 128 0.77 (7.4, 1.4),
// with most of them outside 1.4 (32.6, 3.7), N = 64 0.75 (7.9, 1.4).
// A sum of exactly 0 is left out, as the plane is 0 where it lists nothing.
template <int NG>
__device__ __noinline__ void sum_dense_plane(float *acc, int2 *qs, const int2 *__restrict__ qb, int nq,
                                             int2 *__restrict__ ql, int *count) {
    static_assert(kNT0 <= kVoxQ, "a step's entries");
    constexpr int ROWS = 8 * VoxShared<NG>::W, CELLS = ROWS * NG;
    static_assert(sizeof(VoxShared<NG>) >= sizeof(float) * CELLS, "room of the sums");
    const int tid = threadIdx.x;
    for (int c0 = 0; c0 < NG * NG; c0 += CELLS) {
        __syncthreads();   // the bit planes, or the sums before, have been read
        for (int c = tid; c < CELLS; c += kNT0) acc[c] = 0.f;
        for (int e0 = 0; e0 < nq; e0 += kNT0) {
            const int e = e0 + tid, n = min(kNT0, nq - e0);
            const int2 v = e < nq ? qb[e] : make_int2(-1, 0);
            const bool mine = (unsigned)(v.x - c0) < (unsigned)CELLS;
            qs[tid] = v;
            if (__syncthreads_or(mine)) {
                bool first = mine;
                for (int f = 0; f < tid && first; ++f) first = qs[f].x != v.x;
                if (first) {
                    float sum = acc[v.x - c0];
                    for (int f = tid; f < n; ++f) {
                        const int2 u = qs[f];
                        if (u.x == v.x) sum = __fadd_rn(sum, __int_as_float(u.y));
                    }
                    acc[v.x - c0] = sum;
                }
                __syncthreads();
            }
        }
        __syncthreads();
        for (int c = tid; c < CELLS; c += kNT0)
            if (acc[c] != 0.f) ql[atomicAdd(count, 1)] = make_int2(c0 + c, __float_as_int(acc[c]));
    }
    __syncthreads();
}

// CTAs of k_vox_bits per SM that its shared memory allows (1 KB of each is the
// system's): eight leave 32 registers a thread, six 40.  The call for dense
// planes took two registers more than 32 without the bound, 6 % of the
// voxelizer stage at N = 96 and 126.
template <int NG>
constexpr int vox_bits_ctas() {
    constexpr size_t one = sizeof(VoxShared<NG>) + sizeof(uint32_t) * 2 * NG * VoxShared<NG>::W + sizeof(int2) * kVoxQ + 1040;
    constexpr int fit = (int)(228 * 1024 / one);
    return fit >= 8 ? 8 : (fit > 6 ? 6 : fit);
}

// PREMARKED: the marks come from K0m (marks != nullptr) instead of vox_mark.
template <int NG, bool PREMARKED = false>
__global__ void __launch_bounds__(kNT0, vox_bits_ctas<NG>())
    k_vox_bits(LigandView L, GridView G, const MarkEntry *__restrict__ rec, const int *__restrict__ sstart,
               const int2 *__restrict__ cq, const int *__restrict__ cstart, uint32_t *__restrict__ vbits,
               int2 *__restrict__ qlist, int *__restrict__ qcount, const uint32_t *__restrict__ marks = nullptr) {
    constexpr int W = VoxShared<NG>::W;
    constexpr int NBS = NG + 2 * kReach;
    __shared__ int count;
    __shared__ int2 qs[kVoxQ];
    VoxShared<NG> *vsp;
    uint32_t(*ob)[NG * W];
    if constexpr (vox_bits_dyn<NG>()) {
        extern __shared__ __align__(16) unsigned char vox_smem[];
        vsp = reinterpret_cast<VoxShared<NG> *>(vox_smem);
        ob = reinterpret_cast<uint32_t(*)[NG * W]>(vsp + 1);
    } else {
        __shared__ VoxShared<NG> vs_static;
        __shared__ uint32_t ob_static[2][NG * W];
        vsp = &vs_static;
        ob = ob_static;
    }
    VoxShared<NG> &vs = *vsp;
    const int p = blockIdx.x, b = blockIdx.y, tid = threadIdx.x;
    const bool gd = (L.delta != 1.0f);
    if constexpr (PREMARKED) {
        // core of planes p-2 .. p+2 (p-1 .. p+1 unless delta != 1, as vox_mark
        // marks them), surface of p-1 .. p+1; planes outside the grid are 0
        const uint32_t *mb = marks + (size_t)b * NG * 2 * NG * W;
        for (int w = tid; w < 5 * NG * W; w += blockDim.x) {
            const int slot = w / (NG * W), i = p - 2 + slot;
            const bool on = (i >= 0 && i < G.ng && i < NG) && (gd || (slot >= 1 && slot <= 3));
            (&vs.core[0][0])[w] = on ? mb[(size_t)i * 2 * NG * W + w % (NG * W)] : 0u;
        }
        for (int w = tid; w < 3 * NG * W; w += blockDim.x) {
            const int i = p - 1 + w / (NG * W);
            const bool on = (i >= 0 && i < G.ng && i < NG);
            (&vs.surf[0][0])[w] = on ? mb[(size_t)i * 2 * NG * W + NG * W + w % (NG * W)] : 0u;
        }
    } else {
        for (int w = tid; w < 5 * NG * W; w += blockDim.x) (&vs.core[0][0])[w] = 0u;
        for (int w = tid; w < 3 * NG * W; w += blockDim.x) (&vs.surf[0][0])[w] = 0u;
    }
    // this plane's charge entries, in atom order
    const int c0 = cstart[(size_t)b * (NG + 1) + p], nq = cstart[(size_t)b * (NG + 1) + p + 1] - c0;
    const int2 *qb = cq + (size_t)b * L.na + c0;
    for (int e = tid; e < min(nq, kVoxQ); e += blockDim.x) qs[e] = qb[e];
    if (tid == 0) count = 0;
    __syncthreads();
    if constexpr (!PREMARKED) {
        const int reach = gd ? 4 : 3;
        const int *ss = sstart + (size_t)b * (NBS + 1);
        const int lo = ss[max(p - reach + kReach, 0)], hi = ss[min(p + reach + kReach + 1, NBS)];
        vox_mark<NG>(vs, rec + (size_t)b * L.na, lo, hi, G, p, gd);
    }
    for (int c = tid; c < NG * W; c += blockDim.x) {
        const int q = c / W, w = c % W;
        uint32_t c2, c1;
        vox_code_words<NG>(vs, p, q, w, NG, gd, c2, c1);
        const uint32_t valid = (32 * w + 32 <= NG) ? 0xffffffffu : ((1u << (NG - 32 * w)) - 1u);
        ob[0][q * W + w] = c2 & valid;
        ob[1][q * W + w] = c1 & valid;
    }
    // charges of this plane, in atom order: the first entry of each cell sums
    // that cell's entries in order
    int2 *ql = qlist + ((size_t)b * NG + p) * NG * NG;
    if (nq <= kVoxQ) {
        // every thread walks the whole list, the same entry in all lanes at a
        // time (a broadcast from shared memory)
        for (int e = tid; e < nq; e += blockDim.x) {
            const int key = qs[e].x;
            bool later = false;
            float acc = 0.f;
            for (int f = 0; f < nq; ++f) {
                const int2 v = qs[f];
                if (v.x != key) continue;
                if (f < e) {
                    later = true;
                    break;
                }
                acc = __fadd_rn(acc, __int_as_float(v.y));
            }
            if (!later) ql[atomicAdd(&count, 1)] = make_int2(key, __float_as_int(acc));
        }
        __syncthreads();
    } else {
        sum_dense_plane<NG>(reinterpret_cast<float *>(&vs), qs, qb, nq, ql, &count);
    }
    uint32_t *dst = vbits + ((size_t)b * NG + p) * 2 * NG * W;
    for (int w = tid; w < 2 * NG * W; w += blockDim.x) dst[w] = (&ob[0][0])[w];
    __syncthreads();
    if (tid == 0) qcount[(size_t)b * NG + p] = count;
}

// The voxel grids themselves ([nb][NG^3] real, imaginary) from K0's bit planes
// and charge lists, for the adjoint and the direct pose scores: CTA = (x-plane,
// rotation), the plane written once, then its charged cells.  Bound by the
// stores.  The forward plane kernel without its FFT did this through a
// shared-memory plane, one CTA per SM (64 rotations at N = 96 42.8 us); the
// adjoint of 3,600 rotations there, nineteen such chunks, went 1.95 -> 1.78 ms
// (B200).
template <int NG>
__global__ void __launch_bounds__(kNT0)
    k_vox_store(LigandView L, const uint32_t *__restrict__ vbits, const int2 *__restrict__ qlist,
                const int *__restrict__ qcount, float *__restrict__ vox_r, float *__restrict__ vox_i) {
    constexpr int W = VoxShared<NG>::W;
    const int p = blockIdx.x, b = blockIdx.y, tid = threadIdx.x;
    const size_t plane = (size_t)b * NG + p;
    const uint32_t *vb = vbits + plane * 2 * NG * W;
    float *vr = vox_r + plane * NG * NG, *vi = vox_i + plane * NG * NG;
#pragma unroll 4
    for (int c = tid; c < NG * NG; c += kNT0) {
        const int q = c / NG, s = c % NG;
        const uint32_t bit = 1u << (s & 31);
        const uint32_t w2 = __ldg(&vb[q * W + (s >> 5)]), w1 = __ldg(&vb[NG * W + q * W + (s >> 5)]);
        vr[c] = (w2 & bit) ? L.delta : (w1 & bit) ? 1.0f : 0.0f;
        vi[c] = 0.f;
    }
    __syncthreads();   // the zeros before the charges
    const int nq = qcount[plane];
    const int2 *ql = qlist + plane * NG * NG;
    for (int e = tid; e < nq; e += kNT0) {
        const int2 c = ql[e];
        vi[c.x] = __int_as_float(c.y);
    }
}

// ------------------------------------------------------------------ K1
// MODE 0: real part from the K0 bit planes + K0 charge list, store spectrum planes A.
// MODE 1: receptor grids (re, im) loaded from global, store spectrum planes A.
template <int N, int MODE>
__global__ void __launch_bounds__(kNT1, 1)
    k_plane_fwd(LigandView L, GridView G, const uint32_t *__restrict__ vbits, const int2 *__restrict__ qlist,
                const int *__restrict__ qcount, const float *__restrict__ src_r, const float *__restrict__ src_i,
                float2 *__restrict__ A) {
    constexpr int NG = N / 2, OFF = N / 4, PITCH = N + 1;
    constexpr int R1 = Plan<N>::R1, R2 = Plan<N>::R2;
    constexpr int W = VoxShared<NG>::W;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2 *S = reinterpret_cast<float2 *>(smem_raw);   // N x PITCH

    const int p = blockIdx.x;
    const int b = blockIdx.y;
    const int tid = threadIdx.x;

    if (MODE == 1) {
        for (int c = tid; c < NG * NG; c += blockDim.x) {
            const int q = c / NG, s = c % NG;
            const size_t gidx = ((size_t)p * NG + q) * NG + s;
            S[(q + OFF) * PITCH + s + OFF] = make_float2(src_r[gidx], src_i[gidx]);
        }
        __syncthreads();
    } else {
        const uint32_t *vb = vbits + ((size_t)b * NG + p) * 2 * NG * W;
        // compile-time trip count, both class words loaded unconditionally
        constexpr int CPT = (NG * NG + kNT1 - 1) / kNT1;
#pragma unroll
        for (int r = 0; r < CPT; ++r) {
            const int c = tid + r * kNT1;
            if (NG * NG % kNT1 == 0 || c < NG * NG) {
                const int q = c / NG, s = c % NG;
                const uint32_t bit = 1u << (s & 31);
                const uint32_t w2 = __ldg(&vb[q * W + (s >> 5)]), w1 = __ldg(&vb[NG * W + q * W + (s >> 5)]);
                const float v = (w2 & bit) ? L.delta : (w1 & bit) ? 1.0f : 0.0f;
                S[(q + OFF) * PITCH + s + OFF] = make_float2(v, 0.f);
            }
        }
        __syncthreads();
        const int nq = qcount[(size_t)b * NG + p];
        const int2 *ql = qlist + ((size_t)b * NG + p) * NG * NG;
        for (int e = tid; e < nq; e += blockDim.x) {
            const int2 c = ql[e];
            S[(c.x / NG + OFF) * PITCH + c.x % NG + OFF].y = __int_as_float(c.y);
        }
        __syncthreads();
    }

    // z-FFT of the NG non-zero rows (lanes = rows, pruned columns)
    for (int it = tid; it < NG * R2; it += blockDim.x) {
        const int t = it / NG, q = it % NG;
        padded_phase1<N>(S + (q + OFF) * PITCH, 1, t, G.tw);
    }
    __syncthreads();
    {
        constexpr int IPT = (NG * R1 + kNT1 - 1) / kNT1;
        float2 reg[IPT][R2];
#pragma unroll
        for (int r = 0; r < IPT; ++r) {
            const int it = tid + r * kNT1;
            if (it < NG * R1) fft_phase2<N, -1>(S + ((it % NG) + OFF) * PITCH, 1, it / NG, reg[r]);
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < IPT; ++r) {
            const int it = tid + r * kNT1;
            if (it < NG * R1) {
                float2 *row = S + ((it % NG) + OFF) * PITCH;
                const int u = it / NG;
                static_for<0, R2>([&](auto k2) { row[u + R1 * k2] = reg[r][k2]; });
            }
        }
    }
    __syncthreads();
    // y-FFT of all N columns (lanes = columns, pruned rows); phase 2 -> global
    for (int it = tid; it < N * R2; it += blockDim.x) {
        const int t = it / N, c = it % N;
        padded_phase1<N>(S + c, PITCH, t, G.tw);
    }
    __syncthreads();
    float2 *Ab = A + ((size_t)b * NG + p) * N * N;
    for (int it = tid; it < N * R1; it += blockDim.x) {
        const int u = it / N, c = it % N;
        float2 o[R2];
        fft_phase2<N, -1>(S + c, PITCH, u, o);
        static_for<0, R2>([&](auto k2) { Ab[(size_t)(u + R1 * k2) * N + c] = o[k2]; });
    }
}

// K1, pipelined form: the z-FFT results of the NG non-zero rows stay resident
// and the y-FFT runs over blocks of W columns through two block buffers, one
// half of the CTA in pass 1 of a block (resident rows -> buffer) while the
// other is in pass 2 of the block before (buffer -> global memory): one barrier
// per block, an item per thread, and the shared-memory pass overlaps the
// stores.  Rows keep their R1 blocks at the odd stride STR, so the z pass ends
// in place (block u, place k2 holds kz = u + R1 k2) without a trip through
// registers, and lanes over kz read the blocks without bank conflicts.  us per
// rotation against the column-block form below (B200): N = 48 0.25 -> 0.17, 72
// 0.64 -> 0.50, 84 0.93 -> 0.91; the whole graph with two launch groups in
// flight 48 0.79 -> 0.71, 64 1.35 -> 1.29, 72 2.49 -> 2.33, 84 3.86 -> 3.83, 90
// equal, 96 4.85 -> 5.04 (its CTAs leave the other group less room).  From 108
// on two CTAs of 340 to 400 threads lose to two of 512 (1.90 -> 2.14, 128 2.32
// -> 2.70), and as the only CTA of an SM to the one-CTA form (160 6.2 -> 6.6).
constexpr size_t kSmemMax = 227 * 1024;   // dynamic shared memory one CTA may hold

template <int N>
struct FwdPipe {
    static constexpr int R1 = Plan<N>::R1, R2 = Plan<N>::R2, NG = N / 2;
    static constexpr int STR = R2 | 1, PZ = (R1 * STR) | 1;
    static constexpr int W = 16;
    static constexpr int T1 = (W * R2 + 31) / 32 * 32, T2 = (W * R1 + 31) / 32 * 32, NT = T1 + T2;
    static constexpr size_t bytes = ((size_t)NG * PZ + 2 * (size_t)N * (W + 1)) * sizeof(float2);
    static constexpr int OCC_S = (int)((227 * 1024) / (bytes + 1024)), OCC_R = 65536 / (NT * 72), OCC_T = 2048 / NT;
    static constexpr int OCC0 = OCC_S < OCC_R ? OCC_S : OCC_R;
    static constexpr int OCC = (OCC0 < OCC_T ? OCC0 : OCC_T) > 0 ? (OCC0 < OCC_T ? OCC0 : OCC_T) : 1;
};

template <int N>
constexpr bool fwd_pipe() {
    return N <= 84;
}

template <int N, int MODE = 0>
__global__ void __launch_bounds__(FwdPipe<N>::NT, FwdPipe<N>::OCC)
    k_plane_fwd_pipe(LigandView L, GridView G, const uint32_t *__restrict__ vbits, const int2 *__restrict__ qlist,
                     const int *__restrict__ qcount, const float *__restrict__ src_r, const float *__restrict__ src_i,
                     float2 *__restrict__ A) {
    using P = FwdPipe<N>;
    constexpr int NG = N / 2, OFF = N / 4, R1 = P::R1, R2 = P::R2, STR = P::STR, PZ = P::PZ, BW = P::W, PY = BW + 1;
    constexpr int NT = P::NT, W = VoxShared<NG>::W;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2 *Z = reinterpret_cast<float2 *>(smem_raw);   // NG rows x PZ
    float2 *Y = Z + NG * PZ;                             // 2 x N rows x PY
    const int p = blockIdx.x, b = blockIdx.y, tid = threadIdx.x;
    // element of voxel column s in row q
    auto at = [&](int q, int s) -> float2 & {
        const int z = s + OFF;
        return Z[q * PZ + (z / R2) * STR + z % R2];
    };
    if constexpr (MODE == 1) {
        for (int c = tid; c < NG * NG; c += NT) {
            const int q = c / NG, s = c % NG;
            const size_t gidx = ((size_t)p * NG + q) * NG + s;
            at(q, s) = make_float2(src_r[gidx], src_i[gidx]);
        }
        __syncthreads();
    } else {
        const uint32_t *vb = vbits + ((size_t)b * NG + p) * 2 * NG * W;
        // the cells of this thread with a compile-time trip count and both
        // class words loaded unconditionally: the loads of eight are in flight
        constexpr int CPT = (NG * NG + NT - 1) / NT;
#pragma unroll 8
        for (int r = 0; r < CPT; ++r) {
            const int c = tid + r * NT;
            if (NG * NG % NT == 0 || c < NG * NG) {
                const int q = c / NG, s = c % NG;
                const uint32_t bit = 1u << (s & 31);
                const uint32_t w2 = __ldg(&vb[q * W + (s >> 5)]), w1 = __ldg(&vb[NG * W + q * W + (s >> 5)]);
                const float v = (w2 & bit) ? L.delta : (w1 & bit) ? 1.0f : 0.0f;
                at(q, s) = make_float2(v, 0.f);
            }
        }
        __syncthreads();
        const int nq = qcount[(size_t)b * NG + p];
        const int2 *ql = qlist + ((size_t)b * NG + p) * NG * NG;
        for (int e = tid; e < nq; e += NT) {
            const int2 c = ql[e];
            at(c.x / NG, c.x % NG).y = __int_as_float(c.y);
        }
        __syncthreads();
    }
    // z-FFT of the NG rows (lanes = rows), both passes in place
    for (int it = tid; it < NG * R2; it += NT) {
        const int t = it / NG;
        float2 *row = Z + (it % NG) * PZ + t;
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
    for (int it = tid; it < NG * R1; it += NT) {
        float2 *row = Z + (it % NG) * PZ + (it / NG) * STR;
        float2 v[R2];
        static_for<0, R2>([&](auto n2) { v[n2] = row[n2]; });
        Dft<R2, -1>::run(v);
        static_for<0, R2>([&](auto k2) { row[k2] = v[k2]; });
    }
    __syncthreads();
    // y-FFT of the N columns
    float2 *Ab = A + ((size_t)b * NG + p) * N * N;
    constexpr int NB = (N + BW - 1) / BW;
    const bool first = tid < P::T1;
    const int it = first ? tid : tid - P::T1, c = it % BW, k = it / BW;   // k = t (pass 1) or u (pass 2)
    const bool live = first ? k < R2 : k < R1;
    for (int blk = 0; blk <= NB; ++blk) {
        if (first) {
            const int kz = blk * BW + c;
            if (live && blk < NB && (N % BW == 0 || kz < N)) {
                const float2 *col = Z + (kz % R1) * STR + kz / R1;
                float2 *dst = Y + (blk & 1) * N * PY + k * PY + c;
                float2 v[R1];
                padded_inputs<N, R1, R2>(v, k, [&](int q) { return col[q * PZ]; });
                Dft<R1, -1>::run(v);
                static_for<0, R1>([&](auto k1_) {
                    constexpr int k1 = decltype(k1_)::value;
                    float2 x = v[k1];
                    if constexpr (k1 != 0) x = cmul(x, __ldg(&G.tw[k * k1]));
                    dst[k1 * R2 * PY] = x;
                });
            }
        } else {
            const int kz = (blk - 1) * BW + c;
            if (live && blk > 0 && (N % BW == 0 || kz < N)) {
                float2 o[R2];
                fft_phase2<N, -1>(Y + ((blk - 1) & 1) * N * PY + c, PY, k, o);
                static_for<0, R2>([&](auto k2) { Ab[(size_t)(k + R1 * k2) * N + kz] = o[k2]; });
            }
        }
        __syncthreads();
    }
}

// K1, column-block form (84 < N <= 132, two CTAs per SM, and above 168, where
// the one-CTA form does not fit): the resident z-transformed rows (NG x (N+1))
// and one N x (CB+1) block buffer: pruned phase 1 from the resident rows into
// the buffer, phase 2 from the buffer straight to global memory.
constexpr int kNT1B = 512;

template <int N>
constexpr size_t fwd_cb_smem_of(int cb) {
    return ((size_t)(N / 2) * (N + 1) + (size_t)N * (cb + 1)) * sizeof(float2);
}

// Column-block width: 32 where it fits one CTA's shared memory, else 16 or 8.
template <int N>
constexpr int fwd_cb_width() {
    return fwd_cb_smem_of<N>(32) <= kSmemMax ? 32 : (fwd_cb_smem_of<N>(16) <= kSmemMax ? 16 : 8);
}

template <int N>
constexpr size_t fwd_cb_smem() {
    return fwd_cb_smem_of<N>(fwd_cb_width<N>());
}

// two CTAs and their 1 KB system reservations within the SM's 228 KB
template <int N>
constexpr bool fwd_cb_fits() {
    return fwd_cb_smem<N>() <= 113 * 1024;
}

// whether the one-CTA form's N x (N+1) plane fits one CTA (N <= 168); larger
// sizes run every mode in the column-block form
template <int N>
constexpr bool fwd_full_fits() {
    return (size_t)N * (N + 1) * sizeof(float2) <= kSmemMax;
}

// MODE as in k_plane_fwd: 0 ligand bits + charges, 1 receptor grids from global.
template <int N, int MODE = 0>
__global__ void __launch_bounds__(kNT1B, fwd_cb_fits<N>() ? 2 : 1)
    k_plane_fwd_cb(LigandView L, GridView G, const uint32_t *__restrict__ vbits, const int2 *__restrict__ qlist,
                   const int *__restrict__ qcount, const float *__restrict__ src_r, const float *__restrict__ src_i,
                   float2 *__restrict__ A) {
    constexpr int NG = N / 2, OFF = N / 4, PZ = N + 1, CB = fwd_cb_width<N>(), PB = CB + 1;
    constexpr int R1 = Plan<N>::R1, R2 = Plan<N>::R2;
    constexpr int W = VoxShared<NG>::W;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2 *Z = reinterpret_cast<float2 *>(smem_raw);   // NG rows x PZ
    float2 *Y = Z + NG * PZ;                             // N rows x PB
    const int p = blockIdx.x, b = blockIdx.y, tid = threadIdx.x;
    // the plane's NG rows at column offset OFF (the pruned passes read no
    // other column)
    if constexpr (MODE == 1) {
        for (int c = tid; c < NG * NG; c += blockDim.x) {
            const int q = c / NG, s = c % NG;
            const size_t gidx = ((size_t)p * NG + q) * NG + s;
            Z[q * PZ + s + OFF] = make_float2(src_r[gidx], src_i[gidx]);
        }
        __syncthreads();
    } else {
        const uint32_t *vb = vbits + ((size_t)b * NG + p) * 2 * NG * W;
        // the cells of this thread with a compile-time trip count and both
        // class words loaded unconditionally: all loads in flight at once
        constexpr int CPT = (NG * NG + kNT1B - 1) / kNT1B;
#pragma unroll
        for (int r = 0; r < CPT; ++r) {
            const int c = tid + r * kNT1B;
            if (NG * NG % kNT1B == 0 || c < NG * NG) {
                const int q = c / NG, s = c % NG;
                const uint32_t bit = 1u << (s & 31);
                const uint32_t w2 = __ldg(&vb[q * W + (s >> 5)]), w1 = __ldg(&vb[NG * W + q * W + (s >> 5)]);
                const float v = (w2 & bit) ? L.delta : (w1 & bit) ? 1.0f : 0.0f;
                Z[q * PZ + s + OFF] = make_float2(v, 0.f);
            }
        }
        __syncthreads();
        const int nq = qcount[(size_t)b * NG + p];
        const int2 *ql = qlist + ((size_t)b * NG + p) * NG * NG;
        for (int e = tid; e < nq; e += blockDim.x) {
            const int2 c = ql[e];
            Z[(c.x / NG) * PZ + c.x % NG + OFF].y = __int_as_float(c.y);
        }
        __syncthreads();
    }
    // z-FFT of the NG rows (lanes = rows, pruned columns)
    for (int it = tid; it < NG * R2; it += blockDim.x) {
        const int t = it / NG, q = it % NG;
        padded_phase1<N>(Z + q * PZ, 1, t, G.tw);
    }
    __syncthreads();
    {
        constexpr int IPT = (NG * R1 + kNT1B - 1) / kNT1B;
        float2 reg[IPT][R2];
#pragma unroll
        for (int r = 0; r < IPT; ++r) {
            const int it = tid + r * kNT1B;
            if (it < NG * R1) fft_phase2<N, -1>(Z + (it % NG) * PZ, 1, it / NG, reg[r]);
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < IPT; ++r) {
            const int it = tid + r * kNT1B;
            if (it < NG * R1) {
                float2 *row = Z + (it % NG) * PZ;
                const int u = it / NG;
                static_for<0, R2>([&](auto k2) { row[u + R1 * k2] = reg[r][k2]; });
            }
        }
    }
    __syncthreads();
    // y-FFT of the N columns, CB at a time
    float2 *Ab = A + ((size_t)b * NG + p) * N * N;
    for (int cb = 0; cb < N; cb += CB) {
        for (int it = tid; it < CB * R2; it += blockDim.x) {
            const int t = it / CB, c = it % CB;
            if (cb + c >= N) continue;
            float2 v[R1];
            padded_inputs<N, R1, R2>(v, t, [&](int q) { return Z[q * PZ + cb + c]; });   // resident row q
            Dft<R1, -1>::run(v);
            static_for<0, R1>([&](auto k1_) {
                constexpr int k1 = decltype(k1_)::value;
                float2 x = v[k1];
                if constexpr (k1 != 0) x = cmul(x, __ldg(&G.tw[t * k1]));
                Y[(k1 * R2 + t) * PB + c] = x;
            });
        }
        __syncthreads();
        for (int it = tid; it < CB * R1; it += blockDim.x) {
            const int u = it / CB, c = it % CB;
            if (cb + c >= N) continue;
            float2 o[R2];
            fft_phase2<N, -1>(Y + c, PB, u, o);
            static_for<0, R2>([&](auto k2) { Ab[(size_t)(u + R1 * k2) * N + cb + c] = o[k2]; });
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------ K2 (receptor)
// Forward x-FFT of the ng non-zero spectrum planes of the receptor: writes the
// full receptor spectrum R^[kx][ky][kz].  CTA = (ky, 32 kz lines); the last
// tile is partial when N is not a multiple of 32.
template <int N>
__global__ void __launch_bounds__(kNT)
    k_xline_rec(GridView G, const float2 *__restrict__ A, float2 *__restrict__ Rh) {
    constexpr int NG = N / 2, OFF = N / 4;
    constexpr int R1 = Plan<N>::R1, R2 = Plan<N>::R2;
    constexpr int TILES = (N + kLT - 1) / kLT;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2 *X = reinterpret_cast<float2 *>(smem_raw);   // N x kLT
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    const int ky = blockIdx.x / TILES;
    const int kz = (blockIdx.x % TILES) * kLT + lane;
    const bool ok = kz < N;
    for (int pp = warp; pp < NG; pp += nwarp)
        X[(pp + OFF) * kLT + lane] = ok ? A[((size_t)pp * N + ky) * N + kz] : make_float2(0.f, 0.f);
    __syncthreads();
    for (int it = threadIdx.x; it < kLT * R2; it += blockDim.x)
        padded_phase1<N>(X + (it % kLT), kLT, it / kLT, G.tw);
    __syncthreads();
    for (int it = threadIdx.x; it < kLT * R1; it += blockDim.x) {
        const int ln = it % kLT, u = it / kLT;
        float2 o[R2];
        fft_phase2<N, -1>(X + ln, kLT, u, o);
        if (ok)
            static_for<0, R2>([&](auto k2) { Rh[((size_t)(u + R1 * k2) * N + ky) * N + kz] = o[k2]; });
    }
}

// ------------------------------------------------------------------ K2 (docking)
// The score grid s = IFFT(conj(R^) L^) is real, so only its Hermitian part
//   H(k) = (P(k) + conj(P(-k))) / 2,   P = conj(R^) L^,
// contributes: IFFT(H) = Re(IFFT(P)) exactly.  This kernel keeps the rows
// ky in [1, N/2) of the x-inverted H and packs the two self-conjugate rows
// ky = 0 and ky = N/2 into row 0 (row0 = g(ky=0) + i g(ky=N/2)); both become
// real after the inverse along kz, so the plane kernel can unpack them.
//
// One CTA works on tiles of LT kz lines of one row pair: the own tile (ky, kz)
// and the mirror tile (-ky, -kz), F1 threads per line.  Forward split F1 x F2
// (pass 1 a DFT-F1 over stride F2, straight from global memory; pass 2 a
// DFT-F2 whose outputs sit at kx = u + F1 k2): the conjugate partner -kx of
// every output of the own item u is an output of the mirror item (F1 - u) mod
// F1, so one thread transforms both, multiplies both by conj(R^), folds them
// into H in registers and runs the first inverse pass (a DFT-F2 over the same
// stride F1, the inverse split being F2 x F1) before anything is stored: three
// barriers per pass.  CTAs of row 0 run two passes (ky = 0 and ky = N/2) and
// pack them.  Output Gh[x][ky][kz], ky < N/2.
//
// Bound by instruction issue and the latency of the tile loads (ncu, N = 160:
// 65 % issue active, 35 % of DRAM peak; N = 256: 45 % and 33 %), so a plan
// trades radix against warps: F1 near 2 F2 keeps the registers of both passes
// level, F1 threads per line leave none idle in the two larger passes, and LT
// = 8 above N = 196 keeps three or more CTAs per SM.  A form that stored the
// mirror products to shared memory and folded in a pass of its own (five
// barriers, 16 threads per line) took, against this one, in us per rotation
// (B200, random planes, 5 to 128 rotations per launch): N = 60 1.25 -> 0.63,
// 96 2.33 -> 2.06, 108 4.80 -> 3.49, 126 7.6 -> 5.8, 144 8.4 -> 6.7, 160 12.2
// -> 10.5, 180 54 -> 20, 216 93 -> 32, 250 133 -> 56, 330 198 -> 139 (above
// 160 half of that from the block order, xline_rot_fast).
//
// MDB_XPLAN(N, F1, F2, LT, CTAs per SM, SEQ): the fastest measured among the
// splits, at the residencies their registers allow.  SEQ finishes the own
// item's product before it reads the mirror item: without it a radix-16 item
// pair runs out of registers (N = 256 54 -> 47, the older form 50; N = 320 121
// -> 112; slower by up to 9 % elsewhere).  Four sizes lost to the older form's
// shorter items (N = 336 136 -> 145, 352 157 -> 173, 384 187 -> 218, 432 364
// -> 372), though no whole call did: with the other stages those edges gained 10,
// 2, 13 and 1 %; every other one gained here too.
template <int N>
struct XPlan;
#define MDB_XPLAN(N_, F1_, F2_, LT_, OCC_, SEQ_)                               \
    template <>                                                                 \
    struct XPlan<N_> {                                                          \
        static constexpr int F1 = F1_, F2 = F2_, LT = LT_, OCC = OCC_;          \
        static constexpr bool SEQ = SEQ_;                                       \
        static constexpr int NT = F1 * LT, TILES = (N_ + LT - 1) / LT;          \
        static_assert(F1_ * F2_ == N_ && NT <= 1024, "plan");                   \
    };
MDB_XPLAN(32, 8, 4, 16, 8, 0) MDB_XPLAN(36, 6, 6, 16, 8, 0) MDB_XPLAN(40, 10, 4, 16, 6, 0)
MDB_XPLAN(42, 6, 7, 16, 10, 0) MDB_XPLAN(44, 11, 4, 16, 6, 0) MDB_XPLAN(48, 8, 6, 16, 8, 0)
MDB_XPLAN(50, 10, 5, 16, 7, 0) MDB_XPLAN(54, 9, 6, 16, 6, 0) MDB_XPLAN(56, 8, 7, 16, 8, 0)
MDB_XPLAN(60, 12, 5, 16, 6, 0) MDB_XPLAN(64, 8, 8, 16, 7, 0) MDB_XPLAN(66, 11, 6, 16, 6, 0)
MDB_XPLAN(70, 14, 5, 16, 5, 0) MDB_XPLAN(72, 12, 6, 16, 5, 0) MDB_XPLAN(80, 10, 8, 16, 6, 0)
MDB_XPLAN(84, 14, 6, 16, 5, 0) MDB_XPLAN(88, 11, 8, 16, 5, 0) MDB_XPLAN(90, 15, 6, 16, 4, 0)
MDB_XPLAN(96, 12, 8, 16, 5, 0) MDB_XPLAN(98, 14, 7, 16, 4, 0) MDB_XPLAN(100, 10, 10, 16, 4, 0)
MDB_XPLAN(108, 18, 6, 16, 4, 0) MDB_XPLAN(110, 10, 11, 16, 4, 0) MDB_XPLAN(112, 16, 7, 16, 4, 0)
MDB_XPLAN(120, 15, 8, 16, 4, 0) MDB_XPLAN(126, 14, 9, 16, 4, 0) MDB_XPLAN(128, 16, 8, 16, 4, 0)
MDB_XPLAN(132, 12, 11, 16, 4, 0) MDB_XPLAN(140, 20, 7, 16, 3, 0) MDB_XPLAN(144, 12, 12, 16, 4, 0)
MDB_XPLAN(150, 15, 10, 16, 4, 0) MDB_XPLAN(154, 14, 11, 16, 3, 0) MDB_XPLAN(160, 20, 8, 16, 3, 0)
MDB_XPLAN(162, 18, 9, 16, 3, 0) MDB_XPLAN(168, 24, 7, 16, 2, 0) MDB_XPLAN(176, 16, 11, 16, 3, 0)
MDB_XPLAN(180, 20, 9, 16, 3, 0) MDB_XPLAN(192, 24, 8, 16, 3, 0) MDB_XPLAN(196, 28, 7, 16, 2, 0)
MDB_XPLAN(198, 22, 9, 16, 2, 0) MDB_XPLAN(200, 20, 10, 8, 6, 0) MDB_XPLAN(210, 21, 10, 8, 4, 0)
MDB_XPLAN(216, 24, 9, 8, 4, 0) MDB_XPLAN(220, 20, 11, 8, 4, 0) MDB_XPLAN(224, 28, 8, 16, 2, 0)
MDB_XPLAN(240, 24, 10, 16, 2, 0) MDB_XPLAN(242, 22, 11, 8, 4, 0) MDB_XPLAN(250, 25, 10, 8, 4, 0)
MDB_XPLAN(252, 28, 9, 8, 4, 0) MDB_XPLAN(256, 16, 16, 16, 2, 1) MDB_XPLAN(264, 24, 11, 16, 2, 0)
MDB_XPLAN(270, 27, 10, 8, 4, 0) MDB_XPLAN(280, 28, 10, 8, 4, 0) MDB_XPLAN(288, 24, 12, 8, 4, 0)
MDB_XPLAN(294, 21, 14, 8, 4, 0) MDB_XPLAN(300, 30, 10, 8, 3, 0) MDB_XPLAN(308, 28, 11, 8, 3, 0)
MDB_XPLAN(320, 32, 10, 8, 3, 1) MDB_XPLAN(324, 36, 9, 8, 2, 0) MDB_XPLAN(330, 30, 11, 8, 3, 0)
MDB_XPLAN(336, 28, 12, 8, 3, 0) MDB_XPLAN(350, 35, 10, 8, 2, 0) MDB_XPLAN(352, 32, 11, 8, 2, 0)
MDB_XPLAN(360, 30, 12, 8, 3, 0) MDB_XPLAN(378, 27, 14, 8, 3, 0) MDB_XPLAN(384, 32, 12, 8, 3, 0)
MDB_XPLAN(392, 28, 14, 8, 3, 0) MDB_XPLAN(396, 36, 11, 8, 2, 0) MDB_XPLAN(400, 20, 20, 8, 3, 0)
MDB_XPLAN(420, 35, 12, 8, 2, 0) MDB_XPLAN(432, 36, 12, 8, 2, 0) MDB_XPLAN(440, 40, 11, 8, 2, 0)
MDB_XPLAN(448, 32, 14, 8, 3, 0) MDB_XPLAN(450, 30, 15, 8, 2, 0) MDB_XPLAN(462, 33, 14, 8, 2, 0)
MDB_XPLAN(480, 40, 12, 8, 2, 0) MDB_XPLAN(484, 44, 11, 8, 2, 0) MDB_XPLAN(486, 27, 18, 8, 3, 0)
MDB_XPLAN(490, 35, 14, 8, 2, 0) MDB_XPLAN(500, 50, 10, 8, 2, 0) MDB_XPLAN(504, 36, 14, 8, 2, 0)
MDB_XPLAN(512, 32, 16, 8, 2, 1)
#undef MDB_XPLAN

// Twiddles from a shared-memory table instead of the read-only cache, and tile
// addresses formed per access instead of from a running pointer: N = 128,
// whose register budget (64 at four CTAs per SM) the pointer form exceeds
// (4.41 us per rotation against 6.9 with 176 bytes of spills).
template <int N>
constexpr bool xline_tw_smem() {
    return N == 128;
}

// Block order.  Every launch-group rotation reads the same receptor spectrum
// tiles.  Up to N = 144 the spectrum (8 N^3 bytes, 24 MB) stays in L2 beside
// the streamed planes, and neighbouring tiles run together; above, the
// rotation is the fastest-varying block index, so the launch's rotations read
// each (ky, kz-tile) of R^ back to back from L2 instead of streaming all of it
// from HBM once per rotation.  B200, 16-line tiles: N = 128 4.4 us per rotation
// tile-fast, 6.9 rotation-fast; N = 160 equal within 5 %; N = 180 54 against 20.
template <int N>
constexpr bool xline_rot_fast() {
    return N > 144;
}
template <int N>
__device__ __forceinline__ void xline_block(int &tile_id, int &b) {
    if constexpr (xline_rot_fast<N>()) {
        tile_id = blockIdx.y;
        b = blockIdx.x;
    } else {
        tile_id = blockIdx.x;
        b = blockIdx.y;
    }
}
template <int N>
inline dim3 xline_grid(int nb) {
    constexpr int tiles = N / 2 * XPlan<N>::TILES;
    return xline_rot_fast<N>() ? dim3(nb, tiles) : dim3(tiles, nb);
}

// Shared memory: the own and mirror tiles, and the twiddle table where
// xline_tw_smem<N>().
template <int N>
constexpr size_t xline_smem() {
    return (size_t)(2 * N * XPlan<N>::LT + (xline_tw_smem<N>() ? N : 0)) * sizeof(float2);
}

template <int N>
__global__ void __launch_bounds__(XPlan<N>::NT, XPlan<N>::OCC)
    k_xline_fold(GridView G, const float2 *__restrict__ A, const float2 *__restrict__ Rh, float2 *__restrict__ Gh) {
    constexpr int NG = N / 2, NH = N / 2, OFF = N / 4;
    constexpr int F1 = XPlan<N>::F1, F2 = XPlan<N>::F2, LT = XPlan<N>::LT, NT = XPlan<N>::NT;
    constexpr int TILES = XPlan<N>::TILES;
    constexpr bool PTR = !xline_tw_smem<N>();   // running pointers
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2 *X0 = reinterpret_cast<float2 *>(smem_raw);   // own tile   [N][LT]
    float2 *X1 = X0 + N * LT;                           // mirror tile [N][LT]
    float2 *TWs = X1 + N * LT;                          // twiddles W_N^j (xline_tw_smem)
    if constexpr (xline_tw_smem<N>()) {
        for (int e = threadIdx.x; e < N; e += NT) TWs[e] = __ldg(&G.tw[e]);
        __syncthreads();
    }
    auto tw_at = [&](int j) {
        if constexpr (xline_tw_smem<N>()) return TWs[j];
        else return __ldg(&G.tw[j]);
    };
    const int lane = threadIdx.x % LT;
    int tile_id, b;
    xline_block<N>(tile_id, b);
    const int ky = tile_id / TILES;
    const int kz = (tile_id % TILES) * LT + lane;
    const bool ok = N % LT == 0 || kz < N;
    const int kzm = (N - kz) % N;
    const float2 *Ab = A + (size_t)b * NG * N * N;
    float2 *Gb = Gh + (size_t)b * N * NH * N;
    const int passes = (ky == 0) ? 2 : 1;

    for (int pass = 0; pass < passes; ++pass) {
        const int kyo = pass == 0 ? ky : NH;   // own row
        const int kym = (N - kyo) % N;         // mirror row
        // forward pass 1 (DFT-F1 over stride F2) on both tiles, straight from
        // global (padding pruned), every load of a thread issued before its DFTs
        constexpr int IT1 = (2 * LT * F2 + NT - 1) / NT;
        float2 v1[IT1][F1];
#pragma unroll
        for (int r = 0; r < IT1; ++r) {
            const int it = threadIdx.x + r * NT;
            const int s = it / (LT * F2);
            const int t = (it / LT) % F2;
            const int row = s ? kym : kyo, col = s ? kzm : kz;
            const bool live = ok && it < 2 * LT * F2;
            const float2 *src = Ab + (size_t)row * N + col + (ptrdiff_t)(t - OFF) * N * N;
            static_for<0, F1>([&](auto m_) {
                constexpr int mm = decltype(m_)::value;
                constexpr int st = pad_state<N, F2>(mm);
                const int pp = t + F2 * mm - OFF;   // spectrum plane of x = t + F2 mm, if any
                if constexpr (st == 0) {
                    v1[r][mm] = make_float2(-0.f, -0.f);
                } else {
                    const bool in = live && (st == 2 || (unsigned)pp < (unsigned)NG);
                    if constexpr (PTR) v1[r][mm] = in ? src[(size_t)(F2 * mm) * N * N] : make_float2(0.f, 0.f);
                    else v1[r][mm] = in ? Ab[((size_t)pp * N + row) * N + col] : make_float2(0.f, 0.f);
                }
            });
        }
#pragma unroll
        for (int r = 0; r < IT1; ++r) {
            const int it = threadIdx.x + r * NT;
            if ((2 * LT * F2) % NT == 0 || it < 2 * LT * F2) {
                const int s = it / (LT * F2);
                const int t = (it / LT) % F2;
                Dft<F1, -1>::run(v1[r]);
                float2 *X = s ? X1 : X0;
                static_for<0, F1>([&](auto k1_) {
                    constexpr int k1 = decltype(k1_)::value;
                    float2 x = v1[r][k1];
                    if constexpr (k1 != 0) x = cmul(x, tw_at(t * k1));
                    X[(k1 * F2 + t) * LT + lane] = x;
                });
            }
        }
        __syncthreads();
        // forward pass 2 of the own item u and the mirror item (F1 - u) mod F1,
        // conj(R^) products, H = (P_own(kx) + conj P_mirror(-kx)) / 2 and the
        // first inverse pass, in registers (one item per thread)
        const int u = threadIdx.x / LT;
        const int um = (F1 - u) % F1;
        float2 h[F2];
        {
            float2 pm[F2];
            const float2 *ro = Rh + ((size_t)u * N + kyo) * N + kz, *rm = Rh + ((size_t)um * N + kym) * N + kzm;
            auto r_own = [&](int k2) {
                if (!ok) return make_float2(0.f, 0.f);
                if constexpr (PTR) return __ldg(ro + (size_t)(F1 * k2) * N * N);
                else return __ldg(&Rh[((size_t)(u + F1 * k2) * N + kyo) * N + kz]);
            };
            auto r_mirror = [&](int k2) {
                if (!ok) return make_float2(0.f, 0.f);
                if constexpr (PTR) return __ldg(rm + (size_t)(F1 * k2) * N * N);
                else return __ldg(&Rh[((size_t)(um + F1 * k2) * N + kym) * N + kzm]);
            };
            if constexpr (XPlan<N>::SEQ) {
                static_for<0, F2>([&](auto n2) { h[n2] = X0[(u * F2 + n2) * LT + lane]; });
                Dft<F2, -1>::run(h);
                static_for<0, F2>([&](auto k2) { h[k2] = cmulconj(r_own(k2), h[k2]); });
                asm volatile("" ::: "memory");   // the mirror item's loads stay below
                static_for<0, F2>([&](auto n2) { pm[n2] = X1[(um * F2 + n2) * LT + lane]; });
                Dft<F2, -1>::run(pm);
                static_for<0, F2>([&](auto k2) { pm[k2] = cmulconj(r_mirror(k2), pm[k2]); });
            } else {
                static_for<0, F2>([&](auto n2) {
                    h[n2] = X0[(u * F2 + n2) * LT + lane];
                    pm[n2] = X1[(um * F2 + n2) * LT + lane];
                });
                Dft<F2, -1>::run(h);
                Dft<F2, -1>::run(pm);
                static_for<0, F2>([&](auto k2) {
                    const float2 a = r_own(k2), c = r_mirror(k2);
                    h[k2] = cmulconj(a, h[k2]);
                    pm[k2] = cmulconj(c, pm[k2]);
                });
            }
            // the partner of kx = u + F1 k2 is mirror output (F2 - 1 - k2)
            // for u > 0 and (F2 - k2) mod F2 for u = 0
            if (u == 0) {
                static_for<0, F2>([&](auto k2_) {
                    constexpr int k2 = decltype(k2_)::value, j2 = (F2 - k2) % F2;
                    h[k2] = make_float2(0.5f * (h[k2].x + pm[j2].x), 0.5f * (h[k2].y - pm[j2].y));
                });
            } else {
                static_for<0, F2>([&](auto k2_) {
                    constexpr int k2 = decltype(k2_)::value, j2 = F2 - 1 - k2;
                    h[k2] = make_float2(0.5f * (h[k2].x + pm[j2].x), 0.5f * (h[k2].y - pm[j2].y));
                });
            }
            Dft<F2, +1>::run(h);
            static_for<1, F2>([&](auto k1_) {
                constexpr int k1 = decltype(k1_)::value;
                h[k1] = cmul(h[k1], conjf2(tw_at(u * k1)));
            });
        }
        __syncthreads();
        static_for<0, F2>([&](auto k1) { X0[(k1 * F1 + u) * LT + lane] = h[k1]; });
        __syncthreads();
        // inverse pass 2 (DFT-F1 over items u2 < F2) -> Gh (row 0 packs ky = 0 and ky = N/2)
        for (int it = threadIdx.x; it < LT * F2; it += NT) {
            const int u2 = it / LT;
            float2 o[F1];
            static_for<0, F1>([&](auto n2) { o[decltype(n2)::value] = X0[(u2 * F1 + decltype(n2)::value) * LT + lane]; });
            Dft<F1, +1>::run(o);
            if (ok) {
                float2 *dst0 = Gb + ((size_t)u2 * NH + ky) * N + kz;
                static_for<0, F1>([&](auto k2) {
                    float2 *dst = PTR ? dst0 + (size_t)(F2 * k2) * NH * N
                                      : &Gb[((size_t)(u2 + F2 * k2) * NH + ky) * N + kz];
                    if (ky != 0 || pass == 0) {
                        *dst = o[k2];
                    } else {
                        // same thread wrote the ky = 0 value in pass 0
                        const float2 g0 = *dst;
                        *dst = make_float2(g0.x - o[k2].y, g0.y + o[k2].x);
                    }
                });
            }
        }
        if (passes > 1) __syncthreads();
    }
}

// Inverse plane kernels: one thread asks for the rows its CTA's place will need
// one wave of CTAs later to be brought into L2, so that wave's first loads do
// not wait for DRAM.  Worth it where a wave of planes (a few hundred, 64 to 200
// KB each) sits in L2 beside the running one: N = 128 3.31 -> 3.21 us per
// rotation, 144 5.73 -> 5.49, 160 8.12 -> 7.72, 216 29.8 -> 28.4; 96 and 108
// equal, 256 and 330 1.5 % slower (B200).
constexpr int kSMs = 148;
template <int N>
constexpr bool inv_prefetch() {
    return N > 112 && N <= 224;
}
// bytes and the address are multiples of 16 (N is even)
__device__ __forceinline__ void prefetch_l2(const void *p, unsigned bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// ------------------------------------------------------------------ K3
// Selection order for top-t: larger key first, then smaller linear index.
// NaN keys are never selected (they fail every comparison in the reference).
__device__ __forceinline__ bool key_better(float a, int ia, float b, int ib) {
    return (a > b) || (a == b && ia < ib);
}

struct Cand {
    float key;
    int idx;
};

// Order-preserving integer image of a key for the warp reductions of the
// plane kernel (redux.sync reduces integers in one instruction where a
// shuffle tree takes five dependent steps): larger keys map to larger
// integers, -0 and +0 to the same one (they compare equal), NaN below every
// key.
__device__ __forceinline__ int key_ord(float k) {
    if (k != k) return INT_MIN;
    const int b = __float_as_int(k == 0.f ? 0.f : k);
    return b >= 0 ? b : b ^ 0x7FFFFFFF;
}
__device__ __forceinline__ float ord_key(int o) {
    return __int_as_float(o >= 0 ? o : o ^ 0x7FFFFFFF);
}

// The best candidate of a warp's lanes in selection order (larger key, then
// smaller cell index; the lanes' cell indices are distinct), broadcast to
// every lane, and the lane that holds it; idx < 0 when no lane holds one.
// The largest key comes from one integer reduction over the keys'
// order-preserving images, the smallest index among its holders from a
// second.
__device__ __forceinline__ Cand warp_best(Cand c, int &owner) {
    const bool valid = c.idx >= 0;
    const int ko = valid ? key_ord(c.key) : INT_MIN;
    const int kmax = __reduce_max_sync(0xffffffffu, ko);
    const bool tie = valid && ko == kmax;
    const int imin = __reduce_min_sync(0xffffffffu, tie ? c.idx : INT_MAX);
    const unsigned win = __ballot_sync(0xffffffffu, tie && c.idx == imin);
    if (win == 0) {
        owner = 0;
        return Cand{0.f, -1};
    }
    owner = __ffs(win) - 1;
    return Cand{__shfl_sync(0xffffffffu, c.key, owner), imin};
}

// Block-wide best candidate; idx < 0 means "none".
__device__ __forceinline__ Cand block_best(Cand mine, Cand *red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int owner;
    mine = warp_best(mine, owner);
    if (lane == 0) red[warp] = mine;
    __syncthreads();
    if (warp == 0) {
        const int nw = blockDim.x >> 5;
        const Cand c = warp_best((lane < nw) ? red[lane] : Cand{0.f, -1}, owner);
        if (lane == 0) red[32] = c;
    }
    __syncthreads();
    const Cand r = red[32];
    __syncthreads();
    return r;
}

// The nsel best cells of a CTA's scores (nsel <= kSelMax), in selection order,
// to out[0 .. nsel) (index -1 past the last).  item(it, o) computes the
// scores of item it < COUNT -- o[k2].x of cell c0 + STEP k2 and o[k2].y of
// cell c0 + STEP k2 + N -- and returns c0, or -1 when the item holds no cells
// (never, with ALL).
// With a floor (index >= 0) only cells after it in selection order compete.
//
// Every thread keeps the largest of its scores; each such maximum is the key
// of a cell of its own, so the nsel-th largest of them bounds the nsel-th best
// key from below.  Up to kSelLoose poses the bound is the largest over the
// warps of each warp's nsel-th largest lane maximum (one barrier less); a peak
// of the score spreads over the lanes of several warps, so for longer lists
// that bound lets hundreds of cells through and the warps' sorted maxima are
// merged instead.  The few threads that hold a score at or above the bound
// recompute their items (the same bits) and append those cells to a shared
// list; a cell's rank in the list (equal keys by the lower index) is its place
// in the output.  When more cells pass the bound than the list holds, the
// nsel-th best of those it got is a higher bound, and the cells are collected
// again.  Where that does not end (many equal keys) the cells are found round
// by round, every round rescanning the items for the best one after the last.
// Rounds alone, from the first overflow on, took 32 poses at N = 96 7.8 us per
// rotation instead of 3.8, at 144 25.9 instead of 12.3 and at 160 35 instead of
// 16 (B200, stage of 32 or 8 rotations per launch).
constexpr int kSelMax = 32;
constexpr int kSelLoose = 3;
constexpr int kSelCap = 256;
constexpr int kSelRaises = 4;   // times the bound is raised

// What the selection's threads share: the warps' largest lane maxima, then the
// cells at or above the bound.
template <int NW>
struct SelShared {
    union {
        float wtop[NW][kSelMax];
        Cand list[kSelCap];
    };
    float thr_w[NW];
    float thr_all;
    int nlist;
    Cand red[33];
};

// Appends this thread's cells at or above `thr` (after the floor) to the list.
template <int N, int NT, int COUNT, int Q2, int STEP, class Item, class Shared>
__device__ __forceinline__ void collect_cells(const Item &item, const Cand &floor, float thr, Shared &sh) {
#pragma unroll 1
    for (int it = threadIdx.x; it < COUNT; it += NT) {
        float2 o[Q2];
        const int c0 = item(it, o);
        if (c0 < 0) continue;
        auto enter = [&](float key, int idx) {
            if (key >= thr && (floor.idx < 0 || key_better(floor.key, floor.idx, key, idx))) {
                const int e = atomicAdd(&sh.nlist, 1);
                if (e < kSelCap) sh.list[e] = Cand{key, idx};
            }
        };
        static_for<0, Q2>([&](auto k2_) {
            constexpr int k2 = decltype(k2_)::value;
            enter(o[k2].x, c0 + STEP * k2);
            enter(o[k2].y, c0 + STEP * k2 + N);
        });
    }
}

// The list's first n entries at their places in selection order.
template <int NT, class Shared, class Place>
__device__ __forceinline__ void rank_cells(const Shared &sh, int n, const Place &place) {
    for (int e = threadIdx.x; e < n; e += NT) {
        const Cand c = sh.list[e];
        int rank = 0;
        for (int f = 0; f < n; ++f) rank += key_better(sh.list[f].key, sh.list[f].idx, c.key, c.idx) ? 1 : 0;
        place(rank, c);
    }
}

// The nsel best of the list's n entries to out.
template <int NT, class Shared>
__device__ __forceinline__ void write_cells(const Shared &sh, int n, int nsel, Cand *__restrict__ out) {
    rank_cells<NT>(sh, n, [&](int rank, const Cand &c) {
        if (rank < nsel) out[rank] = c;
    });
    const int tid = threadIdx.x;
    if (tid >= n && tid < nsel) out[tid] = Cand{0.f, -1};
}

// The rest of the selection when the list overflowed at the bound `thr`.  A
// function of its own: inlined it took registers from the passes before it.
template <int N, int NT, int COUNT, int Q2, int STEP, class Item, class Shared>
__device__ __noinline__ void select_overflow(Item item, int nsel, Cand floor, Cand *__restrict__ out, float thr,
                                             float tmax, Shared *shp) {
    Shared &sh = *shp;
    const int tid = threadIdx.x;
    for (int raise = 0; raise < kSelRaises; ++raise) {
        rank_cells<NT>(sh, kSelCap, [&](int rank, const Cand &c) {
            if (rank == nsel - 1) sh.thr_all = c.key;
        });
        __syncthreads();
        const float higher = sh.thr_all;
        if (!(higher > thr)) break;
        thr = higher;
        if (tid == 0) sh.nlist = 0;
        __syncthreads();
        if (tmax >= thr) collect_cells<N, NT, COUNT, Q2, STEP>(item, floor, thr, sh);
        __syncthreads();
        if (sh.nlist <= kSelCap) {
            write_cells<NT>(sh, sh.nlist, nsel, out);
            return;
        }
    }
    Cand prev = floor;
    for (int r = 0; r < nsel; ++r) {
        Cand mine{0.f, -1};
#pragma unroll 1
        for (int it = tid; it < COUNT; it += NT) {
            float2 o[Q2];
            const int c0 = item(it, o);
            if (c0 < 0) continue;
            auto look = [&](float key, int idx) {
                if (key != key || (prev.idx >= 0 && !key_better(prev.key, prev.idx, key, idx))) return;
                if (mine.idx < 0 || key_better(key, idx, mine.key, mine.idx)) mine = Cand{key, idx};
            };
            static_for<0, Q2>([&](auto k2_) {
                constexpr int k2 = decltype(k2_)::value;
                look(o[k2].x, c0 + STEP * k2);
                look(o[k2].y, c0 + STEP * k2 + N);
            });
        }
        prev = block_best(mine, sh.red);
        if (tid == 0) out[r] = prev.idx >= 0 ? prev : Cand{0.f, -1};
        if (prev.idx < 0) {
            for (int r2 = r + 1 + tid; r2 < nsel; r2 += NT) out[r2] = Cand{0.f, -1};
            break;
        }
    }
}

template <int N, int NT, int COUNT, int Q2, int STEP, bool ALL, class Item>
__device__ __forceinline__ void select_cells(const Item &item, int nsel, const Cand &floor, Cand *__restrict__ out) {
    static_assert(NT % 32 == 0 && NT <= 1024, "whole warps");
    constexpr int NW = NT / 32;
    __shared__ SelShared<NW> sh;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int TRIPS = (COUNT + NT - 1) / NT;
    const bool fl = floor.idx >= 0;
    if (tid == 0) sh.nlist = 0;
    float tmax = -INFINITY;   // fmaxf drops NaN keys, which are never selected
    if (!fl) {
#pragma unroll
        for (int r = 0; r < TRIPS; ++r) {
            const int it = tid + r * NT;
            if (COUNT % NT == 0 || it < COUNT) {
                float2 o[Q2];
                const int c0 = item(it, o);
                float m = -INFINITY;
                static_for<0, Q2>([&](auto k2_) {
                    constexpr int k2 = decltype(k2_)::value;
                    m = fmaxf(m, fmaxf(o[k2].x, o[k2].y));
                });
                // no branch: the trips' loads overlap
                tmax = fmaxf(tmax, ALL || c0 >= 0 ? m : -INFINITY);
            }
        }
    } else {
#pragma unroll 1
        for (int it = tid; it < COUNT; it += NT) {
            float2 o[Q2];
            const int c0 = item(it, o);
            if (c0 < 0) continue;
            static_for<0, Q2>([&](auto k2_) {
                constexpr int k2 = decltype(k2_)::value;
                if (key_better(floor.key, floor.idx, o[k2].x, c0 + STEP * k2)) tmax = fmaxf(tmax, o[k2].x);
                if (key_better(floor.key, floor.idx, o[k2].y, c0 + STEP * k2 + N)) tmax = fmaxf(tmax, o[k2].y);
            });
        }
    }
    {
        float v = tmax, thw = -INFINITY;
        for (int r = 0; r < nsel; ++r) {
            const int vo = key_ord(v);
            const int mo = __reduce_max_sync(0xffffffffu, vo);
            thw = ord_key(mo);
            if (nsel > kSelLoose && lane == 0) sh.wtop[warp][r] = thw;
            const unsigned holders = __ballot_sync(0xffffffffu, vo == mo);
            if (lane == __ffs(holders) - 1) v = -INFINITY;
        }
        if (lane == 0) sh.thr_w[warp] = thw;
    }
    __syncthreads();
    float thr;
    if (nsel <= kSelLoose) {
        thr = sh.thr_w[0];
#pragma unroll
        for (int w = 1; w < NW; ++w) thr = fmaxf(thr, sh.thr_w[w]);
    } else {
        if (warp == 0) {
            int pos = 0;   // this lane's place in its warp's list
            float best = -INFINITY;
            for (int r = 0; r < nsel; ++r) {
                const int vo = lane < NW && pos < nsel ? key_ord(sh.wtop[lane][pos]) : INT_MIN;
                const int mo = __reduce_max_sync(0xffffffffu, vo);
                best = ord_key(mo);
                const unsigned holders = __ballot_sync(0xffffffffu, vo == mo);
                if (lane == __ffs(holders) - 1) ++pos;
            }
            if (lane == 0) sh.thr_all = best;
        }
        __syncthreads();
        thr = sh.thr_all;
    }
    if (tmax >= thr) collect_cells<N, NT, COUNT, Q2, STEP>(item, floor, thr, sh);
    __syncthreads();
    const int n = sh.nlist;
    if (n <= kSelCap) write_cells<NT>(sh, n, nsel, out);
    else select_overflow<N, NT, COUNT, Q2, STEP>(item, nsel, floor, out, thr, tmax, &sh);
}

// K3: one x-plane of one rotation.  Input Gh[x][ky < N/2][kz] from
// k_xline_fold.  (1) inverse FFT along kz of the N/2 rows, straight from
// global memory; row 0 then holds h0 + i h_{N/2}, both real.  (2) complex-to-
// real inverse along ky for every z column: with X the half spectrum,
//   Z[k] = (X[k] + conj X[N/2-k]) + i w^k (X[k] - conj X[N/2-k]),  w = e^{2 pi i/N},
// the N/2-point inverse FFT of Z gives s[2m] + i s[2m+1].  The plane's best
// cells (select_cells) go to cand[(b*N + x)*t + out0 + j], j < nsel.
// Keys are raw scores: ordering by raw equals ordering by raw / nf3 (a
// positive constant), so the merge kernel divides only the winners.
// Radix plans of this kernel, chosen per context by the autotuner: variant 1
// reverses the kz split, any other is the line plans of N (kz) and N/2 (ky;
// its two factors are equal).  Three CTAs per SM (<= 42 registers) where the
// first kz radix is 8.
constexpr int kC2RPlans = 3;
template <int N, int V>
struct C2RPlan {
    static constexpr int R1 = V == 1 ? Plan<N>::R2 : Plan<N>::R1;
    static constexpr int R2 = V == 1 ? Plan<N>::R1 : Plan<N>::R2;
    static constexpr int Q1 = Plan<N / 2>::R1;
    static constexpr int Q2 = Plan<N / 2>::R2;
};

// Shared memory of k_plane_c2r: the N/2 x PITCH plane.
template <int N, int V>
constexpr size_t c2r_smem() {
    constexpr size_t PA = N + C2RPlan<N, V>::R1, PB = N + 8;
    return (size_t)(N / 2) * (PA > PB ? PA : PB) * sizeof(float2);
}
template <int N, int V = 0>
constexpr int c2r_min_blocks() {
    return C2RPlan<N, V>::R1 <= 8 ? 3 : 2;
}

// The plane kernel's item loops: items tid, tid + kNT, ... below COUNT, with
// a compile-time trip count (blockDim.x is always kNT here) so that each loop
// unrolls (3.4 % less time for this kernel at N = 128 than the runtime-bounded
// loops).
#define MDB_K3_ITEMS(it, COUNT)                                                                 \
    _Pragma("unroll") for (int r_##it = 0; r_##it < ((COUNT) + kNT - 1) / kNT; ++r_##it)       \
        if (const int it = tid + r_##it * kNT; ((COUNT) % kNT == 0) || it < (COUNT))

template <int N, int V = 0>
__global__ void __launch_bounds__(kNT, c2r_min_blocks<N, V>())
    k_plane_c2r(GridView G, const float2 *__restrict__ Gh, int t, int out0, int nsel, Cand *__restrict__ cand) {
    constexpr int NH = N / 2, NT = kNT;
    constexpr int R1 = C2RPlan<N, V>::R1, R2 = C2RPlan<N, V>::R2;
    constexpr int Q1 = C2RPlan<N, V>::Q1, Q2 = C2RPlan<N, V>::Q2;
    constexpr int PA = N + N / R2;   // step-1 layout: one pad per R2 block
    constexpr int PB = N + 8;        // step-2 layout (natural order)
    constexpr int PITCH = PA > PB ? PA : PB;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2 *S = reinterpret_cast<float2 *>(smem_raw);   // NH x PITCH
    auto tw_at = [&](int j) { return __ldg(&G.tw[j]); };
    const int x = blockIdx.x;
    const int b = blockIdx.y;
    const int tid = threadIdx.x;
    const float2 *Gp = Gh + ((size_t)b * N + x) * NH * N;
    if constexpr (inv_prefetch<N>()) {
        const unsigned next = blockIdx.y * N + blockIdx.x + kSMs * c2r_min_blocks<N, V>();
        if (tid == 0 && next < gridDim.y * N) prefetch_l2(Gh + (size_t)next * NH * N, NH * N * sizeof(float2));
    }

    // The z pass works on whole rows: warp w owns rows [w NH/16, (w+1) NH/16) in
    // both of its passes, so the passes are separated by warp barriers only; the
    // plane barrier comes once, before the ky pass reads across rows.
    static_assert(kNT == 512 && NH % 16 == 0 && (NH / 16 * R2) % 32 == 0 && (NH / 16 * R1) % 32 == 0, "warp rows");
    // (1a) inverse kz pass 1, straight from global: item = (row, t), t fastest
    auto z_pass1 = [&](int it) {
        const int row = it / R2, t = it % R2;
        float2 v[R1];
        static_for<0, R1>([&](auto m_) {
            constexpr int mm = decltype(m_)::value;
            v[mm] = __ldg(&Gp[(size_t)row * N + t + R2 * mm]);
        });
        Dft<R1, +1>::run(v);
        static_for<0, R1>([&](auto k1_) {
            constexpr int k1 = decltype(k1_)::value;
            float2 xv = v[k1];
            if constexpr (k1 != 0) xv = cmul(xv, conjf2(tw_at(t * k1)));
            S[row * PITCH + k1 * (R2 + 1) + t] = xv;
        });
    };
    {
        constexpr int IPW = NH / 16 * R2;
#pragma unroll
        for (int r = 0; r < IPW / 32; ++r) z_pass1((tid >> 5) * IPW + (tid & 31) + 32 * r);
        __syncwarp();
    }
    // (1b) inverse kz pass 2: item = (row, u), u fastest; natural order after a warp barrier
    {
        constexpr int IPW = NH / 16 * R1, IPT = IPW / 32;
        float2 reg[IPT][R2];
#pragma unroll
        for (int r = 0; r < IPT; ++r) {
            const int it = (tid >> 5) * IPW + (tid & 31) + 32 * r;
            const int row = it / R1, u = it % R1;
            static_for<0, R2>([&](auto n2_) {
                constexpr int n2 = decltype(n2_)::value;
                reg[r][n2] = S[row * PITCH + u * (R2 + 1) + n2];
            });
            Dft<R2, +1>::run(reg[r]);
        }
        __syncwarp();
#pragma unroll
        for (int r = 0; r < IPT; ++r) {
            const int it = (tid >> 5) * IPW + (tid & 31) + 32 * r;
            const int row = it / R1, u = it % R1;
            static_for<0, R2>([&](auto k2) { S[row * PITCH + u + R1 * k2] = reg[r][k2]; });
        }
    }
    static_assert(Q1 % 2 == 0 && Q2 % 2 == 0, "paired row sets");
    __syncthreads();
    {
        // (2a + 2b) the fold into Z and pass 1 of the N/2-point inverse along
        // ky in one item.  Pass 1 item tt reads and writes the rows
        // tt + Q2 m; the fold partner N/2 - k of row k = tt + Q2 m is row
        // (Q2 - tt) + Q2 (Q1 - 1 - m) for tt > 0, so item g takes the row
        // sets tt = g and Q2 - g, and item 0 the two sets that pair with
        // themselves (tt = 0: Q2 m with Q2 (Q1 - m), row 0 packed; tt = Q2/2).
        // Each item reads and writes only its own rows: no barrier between
        // the fold and the pass.
        // Z_k = E + i w^k D, E = a + conj c, D = a - conj c, a = X_k, c = X_{N/2-k};
        // w^{N/2-k} = -conj(w^k).  The folded rows go back to their own slots
        // (eight values in registers at a time, which keeps the kernel at 40
        // registers without spills) and each row set is then reloaded for its
        // DFT; the empty asm statements with a memory clobber keep the
        // compiler from forwarding those stores to the later loads (which
        // would hold all sixteen values in registers again).  The item's rows
        // are its own, so no barrier is needed between the two.
        // B200, N = 128, 13,824 of the 54,000 rotations at 512 per
        // launch, with the warp-owned z pass above: 274.3 ms per 54,000
        // rotations against 287.7 for the separate fold pass; holding both
        // row sets in registers spilled and took 298.0.
        auto zpair = [&](float2 &a, float2 &c, int k) {
            const float2 w = conjf2(tw_at(k));
            const float2 w2 = make_float2(-w.x, w.y);
            const float2 e1 = make_float2(a.x + c.x, a.y - c.y), d1 = make_float2(a.x - c.x, a.y + c.y);
            const float2 e2 = make_float2(c.x + a.x, c.y - a.y), d2 = make_float2(c.x - a.x, c.y + a.y);
            const float2 o1 = cmul(w, d1), o2 = cmul(w2, d2);
            a = make_float2(e1.x - o1.y, e1.y + o1.x);
            c = make_float2(e2.x - o2.y, e2.y + o2.x);
        };
        MDB_K3_ITEMS(it, N * (Q2 / 2)) {
            const int z = it % N, g = it / N;
            const int ta = g, tb = g == 0 ? Q2 / 2 : Q2 - g;
            auto row = [&](int r) -> float2 & { return S[r * PITCH + z]; };
            if (g == 0) {
                float2 v[Q1];
                static_for<0, Q1>([&](auto m_) { v[decltype(m_)::value] = row(Q2 * decltype(m_)::value); });
                v[0] = make_float2(v[0].x + v[0].y, v[0].x - v[0].y);
                static_for<1, Q1 / 2 + 1>([&](auto m_) {
                    constexpr int mm = decltype(m_)::value;
                    if constexpr (2 * mm == Q1) {
                        float2 c = v[mm];
                        zpair(v[mm], c, Q2 * mm);
                    } else {
                        zpair(v[mm], v[Q1 - mm], Q2 * mm);
                    }
                });
                static_for<0, Q1>([&](auto m_) { row(Q2 * decltype(m_)::value) = v[decltype(m_)::value]; });
                asm volatile("" ::: "memory");
                static_for<0, Q1>([&](auto m_) { v[decltype(m_)::value] = row(Q2 / 2 + Q2 * decltype(m_)::value); });
                static_for<0, Q1 / 2>([&](auto m_) {
                    constexpr int mm = decltype(m_)::value;
                    zpair(v[mm], v[Q1 - 1 - mm], Q2 / 2 + Q2 * mm);
                });
                static_for<0, Q1>([&](auto m_) { row(Q2 / 2 + Q2 * decltype(m_)::value) = v[decltype(m_)::value]; });
            } else {
                static_for<0, 2>([&](auto h_) {
                    constexpr int h = decltype(h_)::value;
                    float2 a[Q1 / 2], c[Q1 / 2];
                    static_for<0, Q1 / 2>([&](auto j_) {
                        constexpr int j = decltype(j_)::value, mm = h * (Q1 / 2) + j;
                        a[j] = row(ta + Q2 * mm);
                        c[j] = row(tb + Q2 * (Q1 - 1 - mm));
                    });
                    static_for<0, Q1 / 2>([&](auto j_) {
                        constexpr int j = decltype(j_)::value, mm = h * (Q1 / 2) + j;
                        zpair(a[j], c[j], ta + Q2 * mm);
                    });
                    static_for<0, Q1 / 2>([&](auto j_) {
                        constexpr int j = decltype(j_)::value, mm = h * (Q1 / 2) + j;
                        row(ta + Q2 * mm) = a[j];
                        row(tb + Q2 * (Q1 - 1 - mm)) = c[j];
                    });
                    asm volatile("" ::: "memory");
                });
            }
            asm volatile("" ::: "memory");
            static_for<0, 2>([&](auto s_) {
                const int tt = decltype(s_)::value == 0 ? ta : tb;
                float2 v[Q1];
                static_for<0, Q1>([&](auto m_) { v[decltype(m_)::value] = row(tt + Q2 * decltype(m_)::value); });
                Dft<Q1, +1>::run(v);
                static_for<0, Q1>([&](auto k1_) {
                    constexpr int k1 = decltype(k1_)::value;
                    float2 xv = v[k1];
                    if constexpr (k1 != 0) xv = cmul(xv, conjf2(tw_at(2 * tt * k1)));
                    row(k1 * Q2 + tt) = xv;
                });
                asm volatile("" ::: "memory");
            });
        }
    }
    __syncthreads();
    // (2c) pass 2 -> scores s[2m], s[2m+1] -> the plane's best cells
    Cand *out = cand + ((size_t)b * N + x) * t + out0;
    const Cand floor = out0 > 0 ? out[-1] : Cand{0.f, -1};
    if (out0 > 0 && floor.idx < 0) {   // an earlier pass already ran out of cells
        if (tid < nsel) out[tid] = Cand{0.f, -1};
        return;
    }
    const int base = x * N * N;
    select_cells<N, NT, N * Q1, Q2, 2 * Q1 * N, true>(
        [=](int it, float2(&o)[Q2]) {
            const int z = it % N, u = it / N;
            static_for<0, Q2>([&](auto n2_) {
                constexpr int n2 = decltype(n2_)::value;
                o[n2] = S[(u * Q2 + n2) * PITCH + z];
            });
            Dft<Q2, +1>::run(o);
            return base + 2 * u * N + z;
        },
        nsel, floor, out);
}

// ------------------------------------------------------------------ K4
// Merge one rotation's `lists` candidate lists of t into t pose records with
// the reference's rules (src/fft_process.cpp:408-458).
//
// Every list is in selection order (select_cells; a longer one pass after
// pass), so a round compares the lists' heads only: a thread holds the best
// head of its lists, and only the round's winner reads again.  Reading all
// lists x t candidates in each of the t rounds took more time with every list
// that a cluster's CTAs add, twice the whole call for 100 poses at N = 162 to
// 224.  100 poses of one rotation, us (B200): N = 160 668 -> 86, 216 3,952 -> 74
// (880 when a plane had one list), 330 23,974 -> 211; one to ten poses equal up
// to N = 200, 10 poses of 8 rotations at 512 53 -> 6.7 per rotation.
constexpr int kMergeLists = 4096;   // N = 512, eight CTAs per plane
static __global__ void __launch_bounds__(256)
    k_merge(const Cand *__restrict__ cand, int lists, int t, int N, float nf3f, int rot0, DevPose *__restrict__ pose) {
    __shared__ Cand red[33];
    __shared__ int pos[kMergeLists];   // place of each list's head; a list belongs to one thread
    const int b = blockIdx.x;
    const Cand *cb = cand + (size_t)b * lists * t;
    for (int g = threadIdx.x; g < lists; g += blockDim.x) pos[g] = 0;
    int from = 0;   // the list of this thread's best head
    auto best_head = [&](auto at_start) {   // at_start: every list is at its first place
        Cand best{0.f, -1};
#pragma unroll 4
        for (int g = threadIdx.x; g < lists; g += blockDim.x) {
            int p = 0;
            if constexpr (!decltype(at_start)::value) p = pos[g];
            const Cand c = p < t ? cb[(size_t)g * t + p] : Cand{0.f, -1};
            if (c.idx >= 0 && (best.idx < 0 || key_better(c.key, c.idx, best.key, best.idx))) {
                best = c;
                from = g;
            }
        }
        return best;
    };
    Cand mine = best_head(std::true_type{});
    const int N2 = N * N;
    for (int round = 0; round < t; ++round) {
        const Cand prev = block_best(mine, red);
        if (round + 1 < t && prev.idx >= 0 && mine.idx == prev.idx) {   // the lists' cells are distinct
            ++pos[from];
            mine = best_head(std::false_type{});
        }
        if (threadIdx.x == 0) {
            DevPose r;
            r.rot = rot0 + b;
            int idx = prev.idx;
            float score;
            if (t == 1) {
                // running maximum from 0.0 with strict '<' (src/fft_process.cpp:433-445)
                if (idx < 0 || !(prev.key > 0.f)) {
                    score = 0.f;
                    idx = 0;
                } else {
                    score = __fdiv_rn(prev.key, nf3f);
                }
            } else {
                // insertion below the -99999 sentinel never happens (:408-431)
                score = idx < 0 ? -99999.0f : __fdiv_rn(prev.key, nf3f);
                if (!(score > -99999.0f)) {
                    score = -99999.0f;
                    idx = 0;
                }
            }
            r.score = score;
            r.i = idx / N2;
            r.j = (idx / N) % N;
            r.k = idx % N;
            pose[(size_t)b * t + round] = r;
        }
        if (prev.idx < 0) {
            if (threadIdx.x == 0)
                for (int r2 = round + 1; r2 < t; ++r2)
                    pose[(size_t)b * t + r2] = DevPose{t == 1 ? 0.f : -99999.0f, rot0 + b, 0, 0, 0};
            break;
        }
    }
}

}  // namespace mdb
