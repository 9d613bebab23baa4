// Receptor grids on the GPU (sm_100a), bit-exact with MEGADOCK's CPU code
// (Receptor::rpscace, src/receptor.cpp:20-254; Receptor::electro, :258-346).
//
//   K_r0 k_rec_prep    per atom: centre cell, squared radii, ACE term, field reach
//   K_r1 k_rec_core    per atom: core bits in the cube of +-reach cells within 1.5 R^2
//   K_r2 k_rec_rays    per line and axis: open space reachable straight from a face
//   K_r3 k_rec_sweep   in-place 6-neighbour propagation sweep (see below), twice,
//   K_r4 k_rec_apply   each followed by the backward neighbours
//   K_r5 k_rec_cells   per cell: shell sum of 1 - 0.8 ACE (double, rounded per add)
//                      and field sum of e beta q / eps(r) / r over the atoms in order
//
// Core, open space and the rest are bit masks, one row of cells along z per
// RowMask, until the last kernel writes the two float grids.  Every float
// operation is an explicitly rounded intrinsic in the reference's association
// order, and every sum runs over atoms in ascending order, so the grids equal
// the sequential CPU result.
//
// The propagation sweep visits cells in linear order c = (i, j, k) and, for an
// open cell with 1 <= i <= ng-2 and 2 <= j, k <= ng-2 ("valid"), opens its zero
// neighbours.  A cell is open when the sweep reaches it iff it was open at the
// start, or it was zero and one of its predecessors (k-1, j-1 or i-1 on the
// same lines) is valid and open when visited:
//     R(c) = O(c) | (Z(c) & OR_p (V(p) & R(p)))
// which depends only on rows (i, j-1) and (i-1, j) and on the row itself, so
// rows on the same anti-diagonal i + j are independent: one CTA walks the
// 2 ng - 1 anti-diagonals, a thread per row, the previous diagonal's masks in
// shared memory and the next one's inputs already on their way.  Zero cells
// next to a valid open successor (k+1, j+1 or i+1) are opened too, after their
// own visit, so they do not propagate in that sweep.
#pragma once
#include <cstdint>

namespace mdb {

constexpr int kRecMaxNg = 256;

struct RecAtom {
    float x, y, z;
    int io, jo, ko;       // centre cell, (int)(c / gw + ng/2)
    int iw, jw, kw;       // centre cell of the field, (int)(c / width + ng/2)
    float core2, shell2;  // 1.5 R^2 and (R + 3.6)^2
    double term;          // 1 + ACE (-0.8) ratio
    float cq;             // e_ratio * -2800 * q
    int reach_e;          // field cube half width (-1: uncharged)
};

struct RecParams {
    int ng, na;
    float gw, width, eps_core, e_ratio, cpg;   // cpg: charge per grid cell
    double ace_ratio;
    int reach_core, reach_shell;
};

// Value of the open-space marker of Receptor::rpscace; a core value (-d) equal
// to it, to 0 or NaN changes what the comparisons with the core value mean.
constexpr float kRecOpen = -7777.0f;

__device__ __forceinline__ float rec_sq(float c, float g) {
    const float d = __fsub_rn(c, g);
    return __fmul_rn(d, d);
}

__global__ void k_rec_prep(RecParams P, const float *__restrict__ xyz, const float *__restrict__ radius,
                           const float *__restrict__ charge, const float *__restrict__ ace, RecAtom *__restrict__ A) {
    const int l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= P.na) return;
    RecAtom a;
    a.x = xyz[3 * l];
    a.y = xyz[3 * l + 1];
    a.z = xyz[3 * l + 2];
    const float half = (float)(P.ng / 2);
    a.io = __float2int_rz(__fadd_rn(__fdiv_rn(a.x, P.gw), half));
    a.jo = __float2int_rz(__fadd_rn(__fdiv_rn(a.y, P.gw), half));
    a.ko = __float2int_rz(__fadd_rn(__fdiv_rn(a.z, P.gw), half));
    a.iw = __float2int_rz(__fadd_rn(__fdiv_rn(a.x, P.width), half));
    a.jw = __float2int_rz(__fadd_rn(__fdiv_rn(a.y, P.width), half));
    a.kw = __float2int_rz(__fadd_rn(__fdiv_rn(a.z, P.width), half));
    const float r = radius[l];
    a.core2 = __fmul_rn(__fmul_rn(r, r), 1.5f);
    const float rd = __fadd_rn(r, 3.6f);
    a.shell2 = __fmul_rn(rd, rd);
    a.term = __dadd_rn(1.0, __dmul_rn(__dmul_rn((double)ace[l], -0.8), P.ace_ratio));
    const float q = charge[l];
    const float aq = fabsf(q);
    a.cq = __fmul_rn(__fmul_rn(P.e_ratio, -2800.0f), q);
    if (aq <= 1.0e-6f) a.reach_e = -1;
    else if ((double)aq < 0.07) a.reach_e = 4;
    else if ((double)aq < 0.21) a.reach_e = 5;
    else a.reach_e = __float2int_rz(__fdiv_rn(aq, P.cpg));
    A[l] = a;
}

// Bits of one row of cells along z, k in [0, ng).
template <int WORDS>
struct RowMask {
    unsigned long long w[WORDS];
};

// bits lo <= k <= hi of word w
__device__ __forceinline__ unsigned long long word_range(int w, int lo, int hi) {
    lo = max(lo - 64 * w, 0);
    hi = min(hi - 64 * w, 63);
    if (hi < lo) return 0ull;
    return ((hi - lo == 63) ? ~0ull : ((1ull << (hi - lo + 1)) - 1ull)) << lo;
}

template <int WORDS>
__global__ void k_rec_core(RecParams P, const RecAtom *__restrict__ A, const float *__restrict__ gc,
                           RowMask<WORDS> *__restrict__ core) {
    const int l = blockIdx.x;
    const RecAtom a = A[l];
    const int ng = P.ng, R = P.reach_core;
    const int i0 = max(a.io - R, 0), i1 = min(a.io + R + 1, ng);
    const int j0 = max(a.jo - R, 0), j1 = min(a.jo + R + 1, ng);
    const int k0 = max(a.ko - R, 0), k1 = min(a.ko + R + 1, ng);
    const int ni = max(i1 - i0, 0), nj = max(j1 - j0, 0);
    for (int t = threadIdx.x; t < ni * nj; t += blockDim.x) {
        const int i = i0 + t / nj, j = j0 + t % nj;
        const float dxy = __fadd_rn(rec_sq(a.x, gc[i]), rec_sq(a.y, gc[j]));
        unsigned long long m = 0ull;
        int w = k0 >> 6;
        for (int k = k0; k < k1; ++k) {
            if ((k >> 6) != w) {
                if (m) atomicOr(&core[i * ng + j].w[w], m);
                m = 0ull;
                w = k >> 6;
            }
            if (__fadd_rn(dxy, rec_sq(a.z, gc[k])) < a.core2) m |= 1ull << (k & 63);
        }
        if (m) atomicOr(&core[i * ng + j].w[w], m);
    }
}

// Open space seen straight from the six faces, ORed into open (zero at the
// start): blockIdx.y = axis; a thread per word column along x and y, per row
// along z.
template <int WORDS>
__global__ void k_rec_rays(RecParams P, const RowMask<WORDS> *__restrict__ core, RowMask<WORDS> *__restrict__ open,
                           int core_open) {
    const int ng = P.ng;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (blockIdx.y == 2) {
        if (t >= ng * ng) return;
        const RowMask<WORDS> c = core[t];
        int first = ng, last = -1;   // first and last core cell of the row
#pragma unroll
        for (int w = WORDS - 1; w >= 0; --w)
            if (c.w[w]) first = 64 * w + __ffsll((long long)c.w[w]) - 1;
#pragma unroll
        for (int w = 0; w < WORDS; ++w)
            if (c.w[w]) last = 64 * w + 63 - __clzll((long long)c.w[w]);
#pragma unroll
        for (int w = 0; w < WORDS; ++w) {
            unsigned long long m = word_range(w, 0, first - 1) | word_range(w, last + 1, ng - 1);
            if (core_open) m |= c.w[w];
            if (m) atomicOr(&open[t].w[w], m);
        }
        return;
    }
    if (t >= ng * WORDS) return;
    const int a = t / WORDS, w = t % WORDS;
    const size_t base = blockIdx.y == 0 ? (size_t)a : (size_t)a * ng, step = blockIdx.y == 0 ? ng : 1;
    const unsigned long long valid = word_range(w, 0, ng - 1);
    unsigned long long run = valid;
#pragma unroll 8
    for (int k = 0; k < ng; ++k) {
        run &= ~core[base + step * k].w[w];
        if (run) atomicOr(&open[base + step * k].w[w], run);
    }
    run = valid;
#pragma unroll 8
    for (int k = ng - 1; k >= 0; --k) {
        run &= ~core[base + step * k].w[w];
        if (run) atomicOr(&open[base + step * k].w[w], run);
    }
}

__device__ __forceinline__ bool rec_vrow(int i, int j, int ng) { return i >= 1 && i <= ng - 2 && j >= 2 && j <= ng - 2; }

// One propagation sweep: R of every row from the open cells and the zero cells
// (neither core nor open).  One CTA, a thread per row of the anti-diagonal.
template <int WORDS>
__global__ void __launch_bounds__(kRecMaxNg)
    k_rec_sweep(RecParams P, const RowMask<WORDS> *__restrict__ core, const RowMask<WORDS> *__restrict__ open,
                RowMask<WORDS> *__restrict__ reach) {
    __shared__ RowMask<WORDS> diag[2][kRecMaxNg];   // R of the last two anti-diagonals, by i
    const int ng = P.ng, i = threadIdx.x;
    RowMask<WORDS> Vk, all;   // positions 2 <= k <= ng - 2 (as a source on the k axis); 0 <= k < ng
#pragma unroll
    for (int w = 0; w < WORDS; ++w) {
        Vk.w[w] = word_range(w, 2, ng - 2);
        all.w[w] = word_range(w, 0, ng - 1);
    }
    auto inside = [&](int d) { return i < ng && d - i >= 0 && d - i < ng; };
    RowMask<WORDS> c{}, o{};
    if (inside(0)) {
        c = core[(size_t)i * ng - i];
        o = open[(size_t)i * ng - i];
    }
    for (int d = 0; d <= 2 * (ng - 1); ++d) {
        const RowMask<WORDS> C = c, O = o;
        if (inside(d + 1)) {
            c = core[(size_t)i * ng + (d + 1 - i)];
            o = open[(size_t)i * ng + (d + 1 - i)];
        }
        if (inside(d)) {
            const int j = d - i;
            RowMask<WORDS> In{};
            if (j > 0 && rec_vrow(i, j - 1, ng)) {
#pragma unroll
                for (int w = 0; w < WORDS; ++w) In.w[w] |= diag[(d + 1) & 1][i].w[w];
            }
            if (i > 0 && rec_vrow(i - 1, j, ng)) {
#pragma unroll
                for (int w = 0; w < WORDS; ++w) In.w[w] |= diag[(d + 1) & 1][i - 1].w[w];
            }
            const bool vr = rec_vrow(i, j, ng);
            // seeds S = O | (Z & In & Vk); k receives from k - 1 when
            // P(k) = Z(k) & Vk(k - 1) & vr.  R = S | (P & (R << 1)) is a
            // carry chain: within a run of P, everything from the first
            // position after a reached cell up to the run's end is reached,
            // i.e. P & (~(P + B) | B) with B = (R << 1) & P restricted to
            // the seeds (the addition carries through the run); a run
            // crossing a word boundary takes the previous word's top bit
            // of R as its carry in.
            RowMask<WORDS> R{};
            unsigned long long carry = 0ull;   // R at bit 63 of the previous word
#pragma unroll
            for (int w = 0; w < WORDS; ++w) {
                const unsigned long long Z = all.w[w] & ~(C.w[w] | O.w[w]);
                const unsigned long long S = O.w[w] | (Z & In.w[w] & Vk.w[w]);
                const unsigned long long vprev = (Vk.w[w] << 1) | (w ? (Vk.w[w ? w - 1 : 0] >> 63) : 0ull);
                const unsigned long long Pm = vr ? (Z & vprev) : 0ull;
                const unsigned long long B = ((S << 1) | carry) & Pm;
                const unsigned long long r = S | (Pm & (~(Pm + B) | B));
                R.w[w] = r;
                carry = r >> 63;
            }
            diag[d & 1][i] = R;
            reach[(size_t)i * ng + j] = R;
        }
        __syncthreads();
    }
}

// After a sweep: the reached cells are open, and so are zero cells with a
// valid reached successor.
template <int WORDS>
__global__ void k_rec_apply(RecParams P, const RowMask<WORDS> *__restrict__ core, RowMask<WORDS> *__restrict__ open,
                            const RowMask<WORDS> *__restrict__ reach) {
    const int ng = P.ng;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= ng * ng) return;
    const int i = t / ng, j = t % ng;
    const RowMask<WORDS> R = reach[t], C = core[t], O = open[t];
    RowMask<WORDS> back{};
    if (rec_vrow(i, j, ng)) {
#pragma unroll
        for (int w = 0; w < WORDS; ++w) {
            const unsigned long long lo = R.w[w] & word_range(w, 2, ng - 2);
            const unsigned long long hi = w + 1 < WORDS ? R.w[w + 1 < WORDS ? w + 1 : w] & word_range(w + 1, 2, ng - 2) : 0ull;
            back.w[w] = (lo >> 1) | (hi << 63);
        }
    }
    if (j + 1 < ng && rec_vrow(i, j + 1, ng)) {
#pragma unroll
        for (int w = 0; w < WORDS; ++w) back.w[w] |= reach[t + 1].w[w] & word_range(w, 2, ng - 2);
    }
    if (i + 1 < ng && rec_vrow(i + 1, j, ng)) {
#pragma unroll
        for (int w = 0; w < WORDS; ++w) back.w[w] |= reach[t + ng].w[w] & word_range(w, 2, ng - 2);
    }
    RowMask<WORDS> out;
#pragma unroll
    for (int w = 0; w < WORDS; ++w) {
        const unsigned long long Z = word_range(w, 0, ng - 1) & ~(C.w[w] | O.w[w]);
        out.w[w] = O.w[w] | R.w[w] | (Z & back.w[w]);
    }
    open[t] = out;
}

// The two grids.  CTA = (i, kRecRows rows j), a warp per row, lane = k modulo
// 32 with KM = ceil(ng / 32) cells each.  The atoms are walked once, in order:
// the CTA collects those whose shell sphere or field cube touches its rows into
// two shared lists (ballot compaction keeps the order), then every warp adds
// the listed atoms' terms to its cells from registers.
//
// Bound by the field terms' issue (a square root and a division per cell of
// every charged atom's cube).  The whole build with 3,661 atoms at ng = 64 takes
// 1.03 ms on the B200 (1.36 with one list of both kinds and the shell's whole
// search cube, 0.81 of it here).
constexpr int kRecRows = 8;
constexpr int kRecList = 512;

struct RecShell {
    double term;
    float x, y, z, shell2;
    int jo, ko;
};
struct RecField {
    float x, y, z;
    float cq, cq4, cq80;   // e_ratio -2800 q, over 4 and over 80 (the two constant dielectrics)
    int jw, kw, reach;
};

template <int WORDS, int KM>
__global__ void __launch_bounds__(32 * kRecRows)
    k_rec_cells(RecParams P, const RecAtom *__restrict__ A, const float *__restrict__ gc,
                const RowMask<WORDS> *__restrict__ core, const RowMask<WORDS> *__restrict__ open, int core_open,
                float *__restrict__ grid_r, float *__restrict__ grid_i) {
    constexpr int NT = 32 * kRecRows;
    __shared__ RecShell shells[kRecList];
    __shared__ RecField fields[kRecList];
    __shared__ int2 wcount[kRecRows];
    const int ng = P.ng, i = blockIdx.x, jb = blockIdx.y * kRecRows;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int j = jb + warp, je = min(jb + kRecRows, ng) - 1;
    const int R = P.reach_shell;
    const float gi = gc[i], gj = gc[min(j, ng - 1)];
    float glo = gc[jb], ghi = glo;   // the rows' coordinates lie between
    for (int r = jb + 1; r <= je; ++r) {
        glo = fminf(glo, gc[r]);
        ghi = fmaxf(ghi, gc[r]);
    }
    float gk[KM], shell[KM], field[KM];
#pragma unroll
    for (int m = 0; m < KM; ++m) {
        gk[m] = gc[min(lane + 32 * m, ng - 1)];
        shell[m] = 0.f;
        field[m] = 0.f;
    }
    int ns = 0, nf = 0;   // entries in the lists (the same in every thread)
    for (int l0 = 0; l0 < P.na; l0 += NT) {
        const int l = l0 + tid;
        bool hs = false, hf = false;
        RecAtom a;
        if (l < P.na) {
            a = A[l];
            // rounding is monotone, so a squared x or y distance above shell2
            // keeps every rounded sum with it above too
            hs = !(i < a.io - R || i > a.io + R || je < a.jo - R || jb > a.jo + R) && !(rec_sq(a.x, gi) > a.shell2) &&
                 !(a.y < glo && rec_sq(a.y, glo) > a.shell2) && !(a.y > ghi && rec_sq(a.y, ghi) > a.shell2);
            hf = a.reach_e >= 0 && !(i < a.iw - a.reach_e || i > a.iw + a.reach_e || je < a.jw - a.reach_e ||
                                     jb > a.jw + a.reach_e);
        }
        const unsigned ms = __ballot_sync(0xffffffffu, hs), mf = __ballot_sync(0xffffffffu, hf);
        if (lane == 0) wcount[warp] = make_int2(__popc(ms), __popc(mf));
        __syncthreads();
        int as = ns, af = nf;
#pragma unroll
        for (int w = 0; w < kRecRows; ++w) {
            const int2 c = wcount[w];
            if (w < warp) {
                as += c.x;
                af += c.y;
            }
            ns += c.x;
            nf += c.y;
        }
        const unsigned below = (1u << lane) - 1u;
        if (hs) shells[as + __popc(ms & below)] = RecShell{a.term, a.x, a.y, a.z, a.shell2, a.jo, a.ko};
        if (hf)
            fields[af + __popc(mf & below)] = RecField{a.x,  a.y,  a.z,  a.cq,     __fdiv_rn(a.cq, 4.0f),
                                                       __fdiv_rn(a.cq, 80.0f), a.jw, a.kw, a.reach_e};
        __syncthreads();
        if (max(ns, nf) + NT <= kRecList && l0 + NT < P.na) continue;   // room for another step
        if (j < ng) {
            for (int f = 0; f < ns; ++f) {
                const RecShell &e = shells[f];
                const float d2 = __fadd_rn(rec_sq(e.x, gi), rec_sq(e.y, gj));
                if (j < e.jo - R || j > e.jo + R || d2 > e.shell2) continue;   // the whole warp
#pragma unroll
                for (int m = 0; m < KM; ++m) {
                    const int k = lane + 32 * m;
                    const float d3 = __fadd_rn(d2, rec_sq(e.z, gk[m]));
                    if (d3 < e.shell2 && k >= e.ko - R && k <= e.ko + R)
                        shell[m] = __double2float_rn(__dadd_rn((double)shell[m], e.term));
                }
            }
            for (int f = 0; f < nf; ++f) {
                const RecField &e = fields[f];
                const int re = e.reach, k0 = e.kw - re, k1 = e.kw + re;
                if (j < e.jw - re || j > e.jw + re) continue;   // the whole warp
                const float d2 = __fadd_rn(rec_sq(e.x, gi), rec_sq(e.y, gj));
#pragma unroll
                for (int m = 0; m < KM; ++m) {
                    if (32 * m > k1 || 32 * m + 31 < k0) continue;
                    const int k = lane + 32 * m;
                    if (k < k0 || k > k1) continue;
                    const float r = __fsqrt_rn(__fadd_rn(d2, rec_sq(e.z, gk[m])));
                    float ce;
                    if (r >= 8.0f) ce = e.cq80;
                    else if (r > 6.0f) ce = __fdiv_rn(e.cq, __fadd_rn(__fmul_rn(38.0f, r), -224.0f));
                    else ce = e.cq4;
                    field[m] = __fadd_rn(field[m], __fdiv_rn(ce, r));
                }
            }
        }
        ns = nf = 0;
        __syncthreads();
    }
    if (j >= ng) return;
#pragma unroll
    for (int m = 0; m < KM; ++m) {
        const int k = lane + 32 * m;
        if (k >= ng) continue;
        const unsigned long long cw = core[i * ng + j].w[k >> 6], ow = open[i * ng + j].w[k >> 6];
        const bool is_open = (ow >> (k & 63)) & 1ull, is_core = (cw >> (k & 63)) & 1ull;
        // cavities (neither core nor open) count as core; a core value equal
        // to the open-space marker makes the core cells open (core_open)
        const bool full = is_core ? !core_open : !is_open;
        const float v = full ? P.eps_core : shell[m];
        const size_t c = ((size_t)i * ng + j) * ng + k;
        grid_r[c] = v;
        grid_i[c] = v < 0.0f ? 0.f : field[m];   // receptor core cells carry no field
    }
}

}  // namespace mdb
