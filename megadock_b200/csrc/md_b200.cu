// Device context and the device half of the C ABI (include/md_b200.h).
//
// Replaces FFTProcess's GPU members (src/fft_process.cpp:79-209 allocation,
// :212-303 receptor FFT, :502-656 per-rotation pipeline, :660-807 ligand
// voxelization and upload).  Differences by design:
//   - one context per device, explicit stream, no cudaDeviceSynchronize inside
//     the pipeline; a call returns after its own copies complete;
//   - no cuFFT: every transform is the project's fused FFT (dock_kernels.cuh);
//   - the batched form is one captured CUDA graph over the whole rotation
//     range, its launch groups alternating between two work sets on two
//     capture streams so that consecutive groups overlap on the GPU;
//   - errors are returned as status codes with a message, never exit().
#include "context.cuh"
#include "adjoint_kernels.cuh"
#include "receptor_kernels.cuh"

#include <atomic>

namespace {

// md_dock_pairs graphs kept per runner context before the cache is emptied
constexpr size_t kMaxPairGraphs = 32;

bool size_supported(int N) { return sized_ops(N) != nullptr; }

cudaError_t set_attrs(int N) {
    const SizedOps *o = sized_ops(N);
    return o ? o->set_attrs() : cudaErrorInvalidValue;
}

void launch_receptor(md_ctx *c, const float *r, const float *i) { sized_ops(c->N)->receptor(c, r, i); }

void launch_voxel_chunk(md_ctx *c, const float *rot, int nb, float *vr, float *vi) {
    sized_ops(c->N)->voxel_chunk(c, rot, nb, vr, vi);
}

void launch_dock_ws(md_ctx *c, const WorkSet &w, cudaStream_t s, const float *rot, int nb, int rot0, int t,
                    DevPose *pose, cudaEvent_t *ev = nullptr) {
    sized_ops(c->N)->dock(c, w, s, rot, nb, rot0, t, pose, ev);
}

void launch_dock(md_ctx *c, int lane, cudaStream_t s, const float *rot, int nb, int rot0, int t, DevPose *pose,
                 cudaEvent_t *ev = nullptr) {
    launch_dock_ws(c, c->ws[lane], s, rot, nb, rot0, t, pose, ev);
}

void free_graphs(md_ctx *c) {
    ++c->gen;   // graphs of md_dock_pairs that captured this context's arguments no longer match
    for (auto &kv : c->graphs) cudaGraphExecDestroy(kv.second);
    c->graphs.clear();
    for (auto &kv : c->pair_graphs) cudaGraphExecDestroy(kv.second);
    c->pair_graphs.clear();
}

void free_scratch(md_ctx *c) {
    cudaFree(c->d_scratch);
    c->d_scratch = nullptr;
    c->scratch_cap = 0;
}

// The work sets go (free), or move to `kept` where a caller's graph holds them.
void drop_sets(md_ctx *c) {
    free_graphs(c);
    for (auto &w : c->ws) {
        if (c->lent && w.A) {
            c->kept.push_back(w);
            w = WorkSet();
        } else {
            w.release();
        }
    }
    c->lent = false;
    c->cap = c->cap_t = c->cap_na = 0;
    c->sets = 0;
    c->have = WorkSet::Sizes{};
}

void release_work(md_ctx *c) {
    drop_sets(c);
    for (auto &w : c->kept) w.release();
    c->kept.clear();
    free_scratch(c);
    c->auto_most = kAutoGroup;
}

// Whether the caller is capturing the context's stream.
bool capture_open(const md_ctx *c) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    return cudaStreamIsCapturing(c->stream, &cs) == cudaSuccess && cs != cudaStreamCaptureStatusNone;
}

// At least `nsets` work sets holding at least `z` bytes per buffer (only the
// batched graph with two launch groups in flight and the pairs runner use the
// second set, so one launch group in flight holds one set on the device).
// Where the device has no room for them, sets that a caller's graph holds stay
// as they are; others are gone already, so that the new ones can take their place.
int ensure_bytes(md_ctx *ctx, const WorkSet::Sizes &z, int nsets) {
    bool ok = ctx->sets >= nsets;
    for (int k = 0; k < WorkSet::kBufs; ++k) ok = ok && z.b[k] <= ctx->have.b[k];
    if (ok) return MD_OK;
    WorkSet::Sizes m = ctx->have;
    for (int k = 0; k < WorkSet::kBufs; ++k) m.b[k] = std::max(m.b[k], z.b[k]);
    const int cap = ctx->cap, t = ctx->cap_t, na = ctx->cap_na;
    free_scratch(ctx);
    if (!ctx->lent) drop_sets(ctx);
    WorkSet fresh[kLanes];
    cudaError_t e = cudaSuccess;
    for (int k = 0; k < nsets && e == cudaSuccess; ++k) e = fresh[k].allocate(m);
    if (e != cudaSuccess) {
        for (auto &w : fresh) w.release();
        cudaGetLastError();
        ctx->err = std::string("work buffers: ") + cudaGetErrorString(e);
        return MD_ERR_CUDA;
    }
    if (ctx->lent) drop_sets(ctx);
    for (int k = 0; k < nsets; ++k) ctx->ws[k] = fresh[k];
    ctx->sets = nsets;
    ctx->have = m;
    ctx->cap = cap;
    ctx->cap_t = t;
    ctx->cap_na = na;
    return MD_OK;
}

// `nsets` work sets for launch groups of `cap` rotations with t poses each.
int ensure_work(md_ctx *ctx, int cap, int t, int nsets = 1) {
    if (cap <= ctx->cap && t <= ctx->cap_t && ctx->na <= ctx->cap_na && nsets <= ctx->sets) return MD_OK;
    cap = std::max({cap, ctx->cap, 1});
    t = std::max({t, ctx->cap_t, 1});
    const int na = std::max({ctx->na, ctx->cap_na, 1});
    int rc = ensure_bytes(ctx, WorkSet::need(cap, ctx->N, t, na), nsets);
    if (rc) return rc;
    ctx->cap = cap;
    ctx->cap_t = t;
    ctx->cap_na = na;
    return MD_OK;
}

// Device scratch of the calls outside the docking graph (receptor build,
// adjoint, pose scores, pose terms, ligand voxels): n sub-buffers of sz[k] bytes,
// 256-byte aligned, carved from one context buffer that grows to the largest
// call, so repeated calls allocate nothing.  A buffer made and freed by each
// call instead took up to 0.7 ms of a 0.1 ms call (one pose's terms at N = 48),
// whenever no other allocation shared its pages.  md_pose_terms, whose grids
// grow with its poses, gives a buffer back that it grew above kScratchKept.
constexpr size_t kScratchKept = size_t(128) << 20;
int carve_scratch(md_ctx *ctx, const size_t *sz, int n, char **out) {
    size_t off[16], total = 0;
    if (n > 16) return MD_ERR_ARG;
    for (int k = 0; k < n; ++k) {
        off[k] = total;
        total += (sz[k] + 255) & ~size_t(255);
    }
    if (total > ctx->scratch_cap) {
        MD_CUDA(cudaStreamSynchronize(ctx->stream));
        free_scratch(ctx);
        MD_CUDA(cudaMalloc(&ctx->d_scratch, total));
        ctx->scratch_cap = total;
    }
    for (int k = 0; k < n; ++k) out[k] = ctx->d_scratch + off[k];
    return MD_OK;
}

// Rotations per launch of a call over n: md_set_batch's value, or, in a context
// that never got one, as many as keep the work set within kAutoBytes, at most
// `auto_most`, in groups of even size.  One rotation leaves most of the GPU
// idle (64 to 2,000 CTAs a kernel at N = 128) and pays seven launches: B200,
// 360 rotations at N = 128, t = 3, from host buffers: 30.5 -> 4.3 ms.
constexpr size_t kAutoBytes = size_t(1) << 30;
int group_of(const md_ctx *ctx, int n, int t, int auto_most) {
    if (ctx->batch) return std::max(1, std::min(ctx->batch, n));
    const WorkSet::Sizes z = WorkSet::need(1, ctx->N, t, std::max(ctx->na, 1));
    size_t one = 0;
    for (size_t b : z.b) one += b;
    const int most = (int)std::max<size_t>(1, std::min<size_t>(auto_most, kAutoBytes / one));
    const int groups = (std::max(n, 1) + most - 1) / most;
    return std::max(1, (n + groups - 1) / groups);
}

// Runs `reserve`, which picks a call's group sizes and allocates for them.  Where
// automatic groups have no room on the device it runs again with groups of one
// rotation, and the context keeps to those until its work buffers are released,
// so that later calls do not repeat the attempt.
template <class Reserve>
int reserve_groups(md_ctx *ctx, bool automatic, const Reserve &reserve) {
    int rc = reserve();
    if (rc == MD_ERR_CUDA && automatic && ctx->auto_most > 1) {
        cudaGetLastError();
        free_scratch(ctx);
        if (!ctx->lent) drop_sets(ctx);
        ctx->auto_most = 1;
        rc = reserve();
        if (rc) ctx->auto_most = kAutoGroup;
    }
    if (rc) cudaGetLastError();   // a refused allocation is reported once, here
    return rc;
}

// The work set and scratch(B) of a call over n in groups of B rotations.
template <class Scratch>
int with_group(md_ctx *ctx, int n, int &B, const Scratch &scratch) {
    return reserve_groups(ctx, ctx->batch == 0, [&]() {
        B = group_of(ctx, n, 1, ctx->auto_most);
        const int rc = ensure_work(ctx, B, 1);
        return rc ? rc : scratch(B);
    });
}

int check_ready(md_ctx *ctx) {
    if (!ctx->N) {
        ctx->err = "md_set_grid has not been called";
        return MD_ERR_STATE;
    }
    if (!ctx->have_receptor) {
        ctx->err = "md_receptor_fft has not been called";
        return MD_ERR_STATE;
    }
    if (!ctx->have_ligand) {
        ctx->err = "md_ligand_data has not been called";
        return MD_ERR_STATE;
    }
    return MD_OK;
}

// The rotation loop of one md_dock call on device buffers.
int run_dock(md_ctx *ctx, const float *d_rot, int first_rot, int n_rot, int t, DevPose *d_pose) {
    int B = 1;
    bool batched = false;
    const bool capturing = capture_open(ctx);
    const int rc = reserve_groups(ctx, ctx->batch == 0 && !capturing, [&]() {
        B = group_of(ctx, n_rot, t, ctx->auto_most);
        // a caller capturing its stream gets the work set that is there: no
        // allocation may fall inside a capture
        if (ctx->batch == 0 && capturing) B = std::min(B, std::max(1, ctx->cap));
        batched = ctx->batch != 0 && B > 1;
        return ensure_work(ctx, B, t, batched ? ctx->lanes : 1);
    });
    if (rc) return rc;
    if (capturing) ctx->lent = true;
    if (!batched) {
        // plain form (one rotation per fused pipeline) and automatic groups,
        // launched back to back
        for (int r = 0; r < n_rot; r += B)
            launch_dock(ctx, 0, ctx->stream, d_rot + 9 * (size_t)r, std::min(B, n_rot - r), first_rot + r, t,
                        d_pose + (size_t)r * t);
        MD_CUDA(cudaGetLastError());
        return MD_OK;
    }
    // batched form: the whole rotation loop as one captured CUDA graph; with
    // two lanes the launch groups alternate between the two work sets and the
    // two capture streams, with one they run back to back on one stream
    auto key = std::make_tuple(first_rot, n_rot, t, B, d_rot, d_pose);
    auto it = ctx->graphs.find(key);
    if (it == ctx->graphs.end()) {
        cudaGraph_t g;
        MD_CUDA(cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
        cudaEventRecord(ctx->fork, ctx->stream);
        cudaStreamWaitEvent(ctx->side, ctx->fork, 0);
        int group = 0;
        for (int r = 0; r < n_rot; r += B, ++group) {
            const int nb = std::min(B, n_rot - r);
            const int lane = group % ctx->lanes;
            launch_dock(ctx, lane, lane ? ctx->side : ctx->stream, d_rot + 9 * (size_t)r, nb, first_rot + r, t,
                        d_pose + (size_t)r * t);
        }
        cudaEventRecord(ctx->join, ctx->side);
        cudaStreamWaitEvent(ctx->stream, ctx->join, 0);
        cudaError_t ce = cudaStreamEndCapture(ctx->stream, &g);
        if (ce != cudaSuccess) {
            ctx->err = std::string("graph capture: ") + cudaGetErrorString(ce);
            return MD_ERR_CUDA;
        }
        cudaGraphExec_t ex;
        ce = cudaGraphInstantiate(&ex, g, 0);
        cudaGraphDestroy(g);
        if (ce != cudaSuccess) {
            ctx->err = std::string("graph instantiate: ") + cudaGetErrorString(ce);
            return MD_ERR_CUDA;
        }
        it = ctx->graphs.emplace(key, ex).first;
    }
    MD_CUDA(cudaGraphLaunch(it->second, ctx->stream));
    return MD_OK;
}

}  // namespace

extern "C" {

int md_fft_size_supported(int nf1) { return size_supported(nf1) ? 1 : 0; }

int md_ctx_create(int device, md_ctx **out) {
    if (!out) return MD_ERR_ARG;
    *out = nullptr;
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess || n == 0) return MD_ERR_CUDA;
    if (device < 0 || device >= n) return MD_ERR_ARG;
    static std::atomic<uint64_t> next_uid{1};
    md_ctx *ctx = new md_ctx;
    ctx->device = device;
    ctx->uid = next_uid.fetch_add(1);
    if (cudaSetDevice(device) != cudaSuccess ||
        cudaStreamCreateWithFlags(&ctx->own, cudaStreamNonBlocking) != cudaSuccess ||
        cudaStreamCreateWithFlags(&ctx->side, cudaStreamNonBlocking) != cudaSuccess ||
        cudaEventCreateWithFlags(&ctx->fork, cudaEventDisableTiming) != cudaSuccess ||
        cudaEventCreateWithFlags(&ctx->join, cudaEventDisableTiming) != cudaSuccess) {
        delete ctx;
        return MD_ERR_CUDA;
    }
    ctx->stream = ctx->own;
    *out = ctx;
    return MD_OK;
}

void md_ctx_destroy(md_ctx *ctx) {
    if (!ctx) return;
    cudaSetDevice(ctx->device);
    cudaStreamSynchronize(ctx->stream);
    cudaStreamSynchronize(ctx->side);
    release_work(ctx);
    cudaFree(ctx->d_gc);
    cudaFree(ctx->d_tw);
    cudaFree(ctx->d_Rh);
    cudaFree(ctx->d_recv);
    cudaFree(ctx->d_atom);
    cudaFree(ctx->d_rad2);
    cudaFree(ctx->d_rot);
    cudaFree(ctx->d_pose);
    if (ctx->fork) cudaEventDestroy(ctx->fork);
    if (ctx->join) cudaEventDestroy(ctx->join);
    if (ctx->side) cudaStreamDestroy(ctx->side);
    if (ctx->own) cudaStreamDestroy(ctx->own);
    delete ctx;
}

const char *md_last_error(const md_ctx *ctx) { return ctx ? ctx->err.c_str() : "null context"; }

int md_set_stream(md_ctx *ctx, void *stream) {
    if (!ctx) return MD_ERR_ARG;
    free_graphs(ctx);
    ctx->stream = stream ? (cudaStream_t)stream : ctx->own;
    return MD_OK;
}

int md_set_grid(md_ctx *ctx, int nf1, float grid_width, const float *grid_coord) {
    if (!ctx || !grid_coord || !(grid_width > 0.f)) return MD_ERR_ARG;
    if (!size_supported(nf1)) {
        ctx->err = "FFT size " + std::to_string(nf1) +
                   " has no built kernel set (built: the default grid table's sizes up to 512; -F picks one)";
        return MD_ERR_SIZE;
    }
    MD_CUDA(cudaSetDevice(ctx->device));
    MD_CUDA(set_attrs(nf1));
    if (ctx->N != nf1) {
        release_work(ctx);
        cudaFree(ctx->d_gc);
        cudaFree(ctx->d_tw);
        cudaFree(ctx->d_Rh);
        cudaFree(ctx->d_recv);
        ctx->d_gc = nullptr;
        ctx->d_tw = nullptr;
        ctx->d_Rh = nullptr;
        ctx->d_recv = nullptr;
        ctx->have_receptor = false;
        const size_t N = nf1;
        MD_CUDA(cudaMalloc(&ctx->d_gc, sizeof(float) * N / 2));
        MD_CUDA(cudaMalloc(&ctx->d_tw, sizeof(float2) * N));
        MD_CUDA(cudaMalloc(&ctx->d_Rh, sizeof(float2) * N * N * N));
        MD_CUDA(cudaMalloc(&ctx->d_recv, sizeof(float) * 2 * (N / 2) * (N / 2) * (N / 2)));
        std::vector<float2> tw(N);
        for (size_t j = 0; j < N; ++j) {
            const double a = -2.0 * M_PI * (double)j / (double)N;
            tw[j] = make_float2((float)std::cos(a), (float)std::sin(a));
        }
        MD_CUDA(cudaMemcpyAsync(ctx->d_tw, tw.data(), sizeof(float2) * N, cudaMemcpyHostToDevice, ctx->stream));
        MD_CUDA(cudaStreamSynchronize(ctx->stream));
        ctx->N = nf1;
        ctx->ng = nf1 / 2;
    }
    if (ctx->gw != grid_width) free_graphs(ctx);   // the grid width is a kernel argument
    ctx->gw = grid_width;
    ctx->gc_step = grid_coord[1] - grid_coord[0];
    MD_CUDA(cudaMemcpyAsync(ctx->d_gc, grid_coord, sizeof(float) * ctx->ng, cudaMemcpyHostToDevice, ctx->stream));
    MD_CUDA(cudaStreamSynchronize(ctx->stream));
    return MD_OK;
}

int md_receptor_fft(md_ctx *ctx, const float *grid_r, const float *grid_i) {
    if (!ctx || !grid_r || !grid_i) return MD_ERR_ARG;
    if (!ctx->N) {
        ctx->err = "md_set_grid has not been called";
        return MD_ERR_STATE;
    }
    MD_CUDA(cudaSetDevice(ctx->device));
    int rc = ensure_work(ctx, std::max(1, ctx->batch), 1);
    if (rc) return rc;
    const size_t ng3 = (size_t)ctx->ng * ctx->ng * ctx->ng;
    float *d_r = ctx->d_recv, *d_i = ctx->d_recv + ng3;
    MD_CUDA(cudaMemcpyAsync(d_r, grid_r, sizeof(float) * ng3, cudaMemcpyHostToDevice, ctx->stream));
    MD_CUDA(cudaMemcpyAsync(d_i, grid_i, sizeof(float) * ng3, cudaMemcpyHostToDevice, ctx->stream));
    launch_receptor(ctx, d_r, d_i);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) {
        ctx->err = std::string("receptor FFT: ") + cudaGetErrorString(e);
        return MD_ERR_CUDA;
    }
    ctx->have_receptor = true;
    return MD_OK;
}

int md_receptor_build(md_ctx *ctx, int na, const float *xyz_centred, const float *radius, const float *charge,
                      const float *ace, float rec_core, float ace_ratio, float elec_ratio, int make_receptor,
                      float *grid_r, float *grid_i) {
    if (!ctx || na < 1 || !xyz_centred || !radius || !charge || !ace) return MD_ERR_ARG;
    if (!ctx->N) {
        ctx->err = "md_set_grid has not been called";
        return MD_ERR_STATE;
    }
    const int ng = ctx->ng;
    if (ng > kRecMaxNg) {
        ctx->err = "receptor grids on the device are built for ng1 <= " + std::to_string(kRecMaxNg);
        return MD_ERR_SIZE;
    }
    MD_CUDA(cudaSetDevice(ctx->device));
    if (make_receptor) {
        int rc = ensure_work(ctx, std::max(1, ctx->batch), 1);
        if (rc) return rc;
    }
    const size_t ng3 = (size_t)ng * ng * ng;
    RecParams P;
    P.ng = ng;
    P.na = na;
    P.gw = ctx->gw;
    P.width = ctx->gc_step;
    P.eps_core = rec_core;
    P.e_ratio = elec_ratio;
    P.cpg = -1 * P.width * 80.0f / (-2800.0f * elec_ratio);
    P.ace_ratio = (double)ace_ratio;
    P.reach_core = (int)((2.4 + ctx->gw - 0.01) / ctx->gw);
    P.reach_shell = (int)((12 + ctx->gw - 0.01) / ctx->gw);
    const int words = (ng + 63) / 64;
    const size_t mask = sizeof(unsigned long long) * words * ng * ng;
    const size_t sz[6] = {sizeof(float) * 6 * na, sizeof(RecAtom) * na, mask, mask, mask,
                          make_receptor ? 0 : sizeof(float) * 2 * ng3};
    char *p[6];
    int rc = carve_scratch(ctx, sz, 6, p);
    if (rc) return rc;
    const float *d_in = reinterpret_cast<float *>(p[0]);
    RecAtom *d_atoms = reinterpret_cast<RecAtom *>(p[1]);
    float *d_r = make_receptor ? ctx->d_recv : reinterpret_cast<float *>(p[5]);
    float *d_i = d_r + ng3;
    cudaStream_t s = ctx->stream;
    // one upload: coordinates, radii, charges, ACE values
    std::vector<float> in(6 * (size_t)na);
    std::copy(xyz_centred, xyz_centred + 3 * (size_t)na, in.begin());
    std::copy(radius, radius + na, in.begin() + 3 * (size_t)na);
    std::copy(charge, charge + na, in.begin() + 4 * (size_t)na);
    std::copy(ace, ace + na, in.begin() + 5 * (size_t)na);
    cudaError_t e = cudaSuccess;
    auto step = [&](cudaError_t x) {
        if (e == cudaSuccess) e = x;
    };
    step(cudaMemcpyAsync(p[0], in.data(), sizeof(float) * in.size(), cudaMemcpyHostToDevice, s));
    // a core value of 0 makes every cell of the zeroed grid compare equal to
    // the core, NaN none; equal to the open-space marker, core cells are open
    step(cudaMemsetAsync(p[2], rec_core == 0.0f ? 0xff : 0, mask, s));
    step(cudaMemsetAsync(p[3], 0, mask, s));
    const bool draw_core = rec_core != 0.0f && !std::isnan(rec_core);
    const int core_open = rec_core == kRecOpen;
    auto build = [&](auto words_, auto km_) {
        constexpr int W = decltype(words_)::value, KM = decltype(km_)::value;
        RowMask<W> *core = reinterpret_cast<RowMask<W> *>(p[2]), *open = reinterpret_cast<RowMask<W> *>(p[3]),
                   *reach = reinterpret_cast<RowMask<W> *>(p[4]);
        k_rec_prep<<<(na + 255) / 256, 256, 0, s>>>(P, d_in, d_in + 3 * (size_t)na, d_in + 4 * (size_t)na,
                                                    d_in + 5 * (size_t)na, d_atoms);
        if (draw_core) k_rec_core<W><<<na, 32, 0, s>>>(P, d_atoms, ctx->d_gc, core);
        k_rec_rays<W><<<dim3((ng * ng + 63) / 64, 3), 64, 0, s>>>(P, core, open, core_open);
        for (int k = 0; k < 2; ++k) {
            k_rec_sweep<W><<<1, (ng + 31) & ~31, 0, s>>>(P, core, open, reach);
            k_rec_apply<W><<<(ng * ng + 127) / 128, 128, 0, s>>>(P, core, open, reach);
        }
        k_rec_cells<W, KM><<<dim3(ng, (ng + kRecRows - 1) / kRecRows), 32 * kRecRows, 0, s>>>(
            P, d_atoms, ctx->d_gc, core, open, core_open, d_r, d_i);
    };
    if (e == cudaSuccess) {
        if (ng <= 32) build(std::integral_constant<int, 1>{}, std::integral_constant<int, 1>{});
        else if (ng <= 64) build(std::integral_constant<int, 1>{}, std::integral_constant<int, 2>{});
        else if (ng <= 128) build(std::integral_constant<int, 2>{}, std::integral_constant<int, 4>{});
        else if (ng <= 192) build(std::integral_constant<int, 3>{}, std::integral_constant<int, 6>{});
        else build(std::integral_constant<int, 4>{}, std::integral_constant<int, 8>{});
        if (make_receptor) launch_receptor(ctx, d_r, d_i);
        step(cudaGetLastError());
        if (grid_r) step(cudaMemcpyAsync(grid_r, d_r, sizeof(float) * ng3, cudaMemcpyDeviceToHost, s));
        if (grid_i) step(cudaMemcpyAsync(grid_i, d_i, sizeof(float) * ng3, cudaMemcpyDeviceToHost, s));
    }
    step(cudaStreamSynchronize(s));
    if (e != cudaSuccess) {
        ctx->err = std::string("receptor grids: ") + cudaGetErrorString(e);
        return MD_ERR_CUDA;
    }
    if (make_receptor) ctx->have_receptor = true;
    return MD_OK;
}

int md_receptor_spectrum(md_ctx *ctx, float *re, float *im) {
    if (!ctx || !re || !im) return MD_ERR_ARG;
    if (!ctx->have_receptor) {
        ctx->err = "no receptor spectrum";
        return MD_ERR_STATE;
    }
    const size_t n3 = (size_t)ctx->N * ctx->N * ctx->N;
    std::vector<float2> h(n3);
    MD_CUDA(cudaMemcpyAsync(h.data(), ctx->d_Rh, sizeof(float2) * n3, cudaMemcpyDeviceToHost, ctx->stream));
    MD_CUDA(cudaStreamSynchronize(ctx->stream));
    for (size_t i = 0; i < n3; ++i) {
        re[i] = h[i].x;
        im[i] = h[i].y;
    }
    return MD_OK;
}

int md_ligand_data(md_ctx *ctx, int na, const float *xyz, const float *radius, const float *charge,
                   float lig_core) {
    if (!ctx || na <= 0 || !xyz || !radius || !charge) return MD_ERR_ARG;
    if (na > kMaxLigAtoms) {
        ctx->err = "ligand has " + std::to_string(na) + " atoms; at most " + std::to_string(kMaxLigAtoms) +
                   " are supported";
        return MD_ERR_SIZE;
    }
    if (lig_core == 0.0f || lig_core == -8888.0f) {
        ctx->err = "ligand core value (-b) 0 or -8888 collides with the voxelizer's markers";
        return MD_ERR_ARG;
    }
    MD_CUDA(cudaSetDevice(ctx->device));
    std::vector<float4> atom(na);
    std::vector<float2> rad(na);
    for (int l = 0; l < na; ++l) {
        atom[l] = make_float4(xyz[3 * l], xyz[3 * l + 1], xyz[3 * l + 2], charge[l]);
        // Ligand::precalc (src/ligand.cpp:251-254): R*R*1.5 and R*R*1.0 in float
        const float r = radius[l];
        rad[l] = make_float2(r * r * 1.5f, r * r * 1.0f);
    }
    if (na > ctx->na_cap) {
        free_graphs(ctx);
        cudaFree(ctx->d_atom);
        cudaFree(ctx->d_rad2);
        ctx->d_atom = nullptr;
        ctx->d_rad2 = nullptr;
        ctx->na_cap = 0;
        MD_CUDA(cudaMalloc(&ctx->d_atom, sizeof(float4) * na));
        MD_CUDA(cudaMalloc(&ctx->d_rad2, sizeof(float2) * na));
        ctx->na_cap = na;
    }
    // captured graphs hold the atom count and core value as kernel arguments;
    // new coordinates in the same buffers keep them valid
    if (na != ctx->na || lig_core != ctx->delta) free_graphs(ctx);
    MD_CUDA(cudaMemcpyAsync(ctx->d_atom, atom.data(), sizeof(float4) * na, cudaMemcpyHostToDevice, ctx->stream));
    MD_CUDA(cudaMemcpyAsync(ctx->d_rad2, rad.data(), sizeof(float2) * na, cudaMemcpyHostToDevice, ctx->stream));
    MD_CUDA(cudaStreamSynchronize(ctx->stream));
    ctx->na = na;
    ctx->delta = lig_core;
    ctx->have_ligand = true;
    return MD_OK;
}

int md_set_batch(md_ctx *ctx, int b) {
    if (!ctx || b < 1) return MD_ERR_ARG;
    ctx->batch = b;
    return MD_OK;
}

int md_release_work(md_ctx *ctx) {
    if (!ctx) return MD_ERR_ARG;
    MD_CUDA(cudaSetDevice(ctx->device));
    MD_CUDA(cudaStreamSynchronize(ctx->stream));
    MD_CUDA(cudaStreamSynchronize(ctx->side));
    release_work(ctx);
    return MD_OK;
}

int md_set_lanes(md_ctx *ctx, int lanes) {
    if (!ctx || lanes < 1 || lanes > kLanes) return MD_ERR_ARG;
    if (lanes != ctx->lanes) {
        free_graphs(ctx);
        ctx->lanes = lanes;
    }
    return MD_OK;
}

// Every size runs the x-line tile that measured fastest for it (XPlan): the
// value is checked and selects nothing.
int md_set_tile(md_ctx *ctx, int lines) {
    if (!ctx || (lines != 8 && lines != 16 && lines != 32)) return MD_ERR_ARG;
    return MD_OK;
}

int md_set_plan(md_ctx *ctx, int plan) {
    if (!ctx || plan < 0 || plan >= kC2RPlans) return MD_ERR_ARG;
    // captured launches name the kernels; without a grid nothing is captured
    const bool forms = ctx->N && sized_ops(ctx->N)->inv_forms > 1;
    if (forms && (plan == 1) != (ctx->plan == 1)) free_graphs(ctx);
    ctx->plan = plan;
    return MD_OK;
}

int md_dock_device(md_ctx *ctx, const float *d_rot, int first_rot, int n_rot, int t, md_pose *d_out) {
    if (!ctx || !d_rot || !d_out || n_rot < 0 || t < 1) return MD_ERR_ARG;
    int rc = check_ready(ctx);
    if (rc) return rc;
    if (n_rot == 0) return MD_OK;
    MD_CUDA(cudaSetDevice(ctx->device));
    return run_dock(ctx, d_rot, first_rot, n_rot, t, reinterpret_cast<DevPose *>(d_out));
}

int md_dock(md_ctx *ctx, const float *rotmat, int first_rot, int n_rot, int t, md_pose *out) {
    if (!ctx || !rotmat || !out || n_rot < 0 || t < 1) return MD_ERR_ARG;
    int rc = check_ready(ctx);
    if (rc) return rc;
    if (n_rot == 0) return MD_OK;
    MD_CUDA(cudaSetDevice(ctx->device));
    if ((size_t)n_rot * 9 > ctx->rot_cap) {
        free_graphs(ctx);
        cudaFree(ctx->d_rot);
        ctx->d_rot = nullptr;
        ctx->rot_cap = 0;
        MD_CUDA(cudaMalloc(&ctx->d_rot, sizeof(float) * 9 * n_rot));
        ctx->rot_cap = (size_t)n_rot * 9;
    }
    if ((size_t)n_rot * t > ctx->pose_cap) {
        free_graphs(ctx);
        cudaFree(ctx->d_pose);
        ctx->d_pose = nullptr;
        ctx->pose_cap = 0;
        MD_CUDA(cudaMalloc(&ctx->d_pose, sizeof(DevPose) * n_rot * t));
        ctx->pose_cap = (size_t)n_rot * t;
    }
    MD_CUDA(cudaMemcpyAsync(ctx->d_rot, rotmat, sizeof(float) * 9 * n_rot, cudaMemcpyHostToDevice, ctx->stream));
    rc = run_dock(ctx, ctx->d_rot, first_rot, n_rot, t, ctx->d_pose);
    if (rc) return rc;
    MD_CUDA(cudaMemcpyAsync(out, ctx->d_pose, sizeof(DevPose) * n_rot * t, cudaMemcpyDeviceToHost, ctx->stream));
    MD_CUDA(cudaStreamSynchronize(ctx->stream));
    return MD_OK;
}

int md_dock_profile(md_ctx *ctx, const float *d_rot, int first_rot, int n_rot, int t, md_pose *d_out,
                    float *stage_ms, int *launches) {
    if (!ctx || !d_rot || !d_out || !stage_ms || n_rot < 1 || t < 1) return MD_ERR_ARG;
    int rc = check_ready(ctx);
    if (rc) return rc;
    MD_CUDA(cudaSetDevice(ctx->device));
    int B = 1;
    rc = reserve_groups(ctx, ctx->batch == 0, [&]() {
        B = group_of(ctx, n_rot, t, ctx->auto_most);
        return ensure_work(ctx, B, t);
    });
    if (rc) return rc;
    cudaEvent_t ev[6];
    for (auto &e : ev) MD_CUDA(cudaEventCreate(&e));
    double acc[5] = {0, 0, 0, 0, 0};
    int nl = 0;
    // atom prep, marks, voxelizer, forward planes, x lines, one top-t pass per
    // kSelMax poses, merge
    const int per_group = 6 + (t + kSelMax - 1) / kSelMax;
    for (int r = 0; r < n_rot; r += B) {
        const int nb = std::min(B, n_rot - r);
        MD_CUDA(cudaEventRecord(ev[0], ctx->stream));
        launch_dock(ctx, 0, ctx->stream, d_rot + 9 * (size_t)r, nb, first_rot + r, t,
                    reinterpret_cast<DevPose *>(d_out) + (size_t)r * t, ev);
        nl += per_group;
        MD_CUDA(cudaEventSynchronize(ev[5]));
        for (int k = 0; k < 5; ++k) {
            float ms = 0.f;
            MD_CUDA(cudaEventElapsedTime(&ms, ev[k], ev[k + 1]));
            acc[k] += ms;
        }
    }
    for (auto &e : ev) cudaEventDestroy(e);
    for (int k = 0; k < 5; ++k) stage_ms[k] = (float)acc[k];
    if (launches) *launches = nl;
    MD_CUDA(cudaGetLastError());
    return MD_OK;
}

int md_dock_pairs(md_ctx *runner, md_ctx *const *pairs, int npairs, const float *const *d_rotmat, const int *n_rot,
                  int t, md_pose *const *d_out) {
    md_ctx *ctx = runner;
    if (!ctx || !pairs || !d_rotmat || !n_rot || !d_out || npairs < 0 || t < 1) return MD_ERR_ARG;
    MD_CUDA(cudaSetDevice(ctx->device));
    bool automatic = false;   // a pair whose groups are chosen here
    for (int p = 0; p < npairs; ++p) {
        md_ctx *c = pairs[p];
        if (!c || !d_rotmat[p] || !d_out[p] || n_rot[p] < 0) return MD_ERR_ARG;
        if (c->device != ctx->device) {
            ctx->err = "md_dock_pairs: pair " + std::to_string(p) + " is on another device";
            return MD_ERR_ARG;
        }
        int rc = check_ready(c);
        if (rc) {
            ctx->err = "md_dock_pairs: pair " + std::to_string(p) + ": " + c->err;
            return rc;
        }
        MD_CUDA(set_attrs(c->N));
        automatic = automatic || c->batch == 0;
    }
    // shared work sets: the largest launch group of any pair
    std::vector<int> group_size(npairs);
    std::vector<uintptr_t> key;
    const bool capturing = capture_open(ctx);
    int rc = reserve_groups(ctx, automatic && !capturing, [&]() {
        WorkSet::Sizes z{};
        key = {(uintptr_t)npairs, (uintptr_t)t};
        for (int p = 0; p < npairs; ++p) {
            const md_ctx *c = pairs[p];
            const int B = group_size[p] = group_of(c, n_rot[p], t, ctx->auto_most);
            const WorkSet::Sizes zp = WorkSet::need(B, c->N, t, std::max(c->na, 1));
            for (int k = 0; k < WorkSet::kBufs; ++k) z.b[k] = std::max(z.b[k], zp.b[k]);
            // the pair's (uid, gen) stands for every argument the capture takes
            // from it: grid width, core value, atom count, plan, tile and buffers
            key.insert(key.end(), {(uintptr_t)c->uid, (uintptr_t)c->gen, (uintptr_t)d_rotmat[p], (uintptr_t)n_rot[p],
                                   (uintptr_t)d_out[p], (uintptr_t)B, (uintptr_t)c->na, (uintptr_t)c->N});
        }
        return ensure_bytes(ctx, z, kLanes);
    });
    if (rc) return rc;
    if (capturing) ctx->lent = true;
    auto it = ctx->pair_graphs.find(key);
    if (it == ctx->pair_graphs.end()) {
        // keys of changed or destroyed pair contexts never match again: bound the cache
        if (ctx->pair_graphs.size() >= kMaxPairGraphs) {
            MD_CUDA(cudaStreamSynchronize(ctx->stream));
            for (auto &kv : ctx->pair_graphs) cudaGraphExecDestroy(kv.second);
            ctx->pair_graphs.clear();
        }
        cudaGraph_t g;
        MD_CUDA(cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
        cudaEventRecord(ctx->fork, ctx->stream);
        cudaStreamWaitEvent(ctx->side, ctx->fork, 0);
        int group = 0;
        for (int p = 0; p < npairs; ++p) {
            md_ctx *c = pairs[p];
            const int B = group_size[p];
            DevPose *out = reinterpret_cast<DevPose *>(d_out[p]);
            for (int r = 0; r < n_rot[p]; r += B, ++group) {
                const int nb = std::min(B, n_rot[p] - r);
                const int lane = group % kLanes;
                launch_dock_ws(c, ctx->ws[lane], lane ? ctx->side : ctx->stream, d_rotmat[p] + 9 * (size_t)r, nb, r,
                               t, out + (size_t)r * t);
            }
        }
        cudaEventRecord(ctx->join, ctx->side);
        cudaStreamWaitEvent(ctx->stream, ctx->join, 0);
        cudaError_t ce = cudaStreamEndCapture(ctx->stream, &g);
        if (ce != cudaSuccess) {
            ctx->err = std::string("graph capture: ") + cudaGetErrorString(ce);
            return MD_ERR_CUDA;
        }
        cudaGraphExec_t ex;
        ce = cudaGraphInstantiate(&ex, g, 0);
        cudaGraphDestroy(g);
        if (ce != cudaSuccess) {
            ctx->err = std::string("graph instantiate: ") + cudaGetErrorString(ce);
            return MD_ERR_CUDA;
        }
        it = ctx->pair_graphs.emplace(key, ex).first;
    }
    MD_CUDA(cudaGraphLaunch(it->second, ctx->stream));
    return MD_OK;
}

namespace {

// Shared body of the adjoint entry points: per-pose rotation matrices (9 each),
// translations and weights dL/ds on the host; host outputs (any may be null).
int adjoint_core(md_ctx *ctx, const float *rotmat, int n, const int4 *shift, const float *w, float *d_rec_r,
                 float *d_rec_i, float *d_charge, const int *lig_sel, int n_lig, float *d_lig_r, float *d_lig_i,
                 float alpha, double *d_alpha) {
    MD_CUDA(cudaSetDevice(ctx->device));
    const int N = ctx->N, ng = ctx->ng;
    const size_t ng3 = (size_t)ng * ng * ng;
    int B = 1;
    char *p[9];
    int rc = with_group(ctx, n, B, [&](int b) {
        const size_t sz[9] = {sizeof(float) * 9 * n,       sizeof(float) * n,
                              sizeof(int4) * n,            sizeof(float) * 2 * ng3,
                              sizeof(float) * 2 * ng3 * b, sizeof(float) * std::max(ctx->na, 1),
                              sizeof(int) * std::max(n_lig, 1), sizeof(float) * 2 * ng3 * std::max(n_lig, 0),
                              sizeof(double) * kAdjBlocks};
        return carve_scratch(ctx, sz, 9, p);
    });
    if (rc) return rc;
    float *d_rot = reinterpret_cast<float *>(p[0]), *d_w = reinterpret_cast<float *>(p[1]);
    int4 *d_shift = reinterpret_cast<int4 *>(p[2]);
    float *d_grad = reinterpret_cast<float *>(p[3]), *d_vox = reinterpret_cast<float *>(p[4]);
    float *d_dq = reinterpret_cast<float *>(p[5]);
    int *d_sel = reinterpret_cast<int *>(p[6]);
    float *d_lg = reinterpret_cast<float *>(p[7]);
    cudaError_t e = cudaSuccess;
    auto step = [&](cudaError_t x) {
        if (e == cudaSuccess) e = x;
    };
    cudaStream_t s = ctx->stream;
    step(cudaMemcpyAsync(d_rot, rotmat, sizeof(float) * 9 * n, cudaMemcpyHostToDevice, s));
    step(cudaMemcpyAsync(d_w, w, sizeof(float) * n, cudaMemcpyHostToDevice, s));
    step(cudaMemcpyAsync(d_shift, shift, sizeof(int4) * n, cudaMemcpyHostToDevice, s));
    step(cudaMemsetAsync(d_grad, 0, sizeof(float) * 2 * ng3, s));
    if (e != cudaSuccess) {
        ctx->err = std::string("adjoint: ") + cudaGetErrorString(e);
        return MD_ERR_CUDA;
    }
    const int thr = 256;
    const int blocks = (int)((ng3 + thr - 1) / thr);
    // receptor gradient: voxel grids of each chunk of poses, then the gather
    for (int r0 = 0; r0 < n; r0 += B) {
        const int nb = std::min(B, n - r0);
        launch_voxel_chunk(ctx, d_rot + 9 * (size_t)r0, nb, d_vox, d_vox + ng3 * B);
        k_adj_receptor<<<blocks, thr, 0, s>>>(N, ng, nb, d_vox, d_vox + ng3 * B, d_shift + r0, d_w + r0, d_grad,
                                              d_grad + ng3);
    }
    // charge gradient through the charge-cell assignment
    GridView G{ng, ctx->gw, (float)(ng * ctx->gw) / 2, ctx->d_gc, ctx->d_tw};
    LigandView L{ctx->na, ctx->d_atom, ctx->d_rad2, ctx->delta};
    k_adj_charge<<<(ctx->na + 3) / 4, 128, 0, s>>>(L, G, N, n, d_rot, d_shift, d_w, ctx->d_recv + ng3, d_dq);
    if (n_lig > 0) {
        step(cudaMemcpyAsync(d_sel, lig_sel, sizeof(int) * n_lig, cudaMemcpyHostToDevice, s));
        k_adj_ligand<<<dim3(blocks, n_lig), thr, 0, s>>>(N, ng, n_lig, d_sel, ctx->d_recv, ctx->d_recv + ng3,
                                                         d_shift, d_w, d_lg, d_lg + ng3 * n_lig);
    }
    // the receptor's imaginary grid is alpha times a fixed-support unit grid
    double *d_part = reinterpret_cast<double *>(p[8]), part[kAdjBlocks];
    if (d_alpha) k_adj_dot<<<kAdjBlocks, 256, 0, s>>>(ng3, d_grad + ng3, ctx->d_recv + ng3, d_part);
    step(cudaGetLastError());
    if (d_rec_r) step(cudaMemcpyAsync(d_rec_r, d_grad, sizeof(float) * ng3, cudaMemcpyDeviceToHost, s));
    if (d_rec_i) step(cudaMemcpyAsync(d_rec_i, d_grad + ng3, sizeof(float) * ng3, cudaMemcpyDeviceToHost, s));
    if (d_alpha) step(cudaMemcpyAsync(part, d_part, sizeof(part), cudaMemcpyDeviceToHost, s));
    if (d_charge) step(cudaMemcpyAsync(d_charge, d_dq, sizeof(float) * ctx->na, cudaMemcpyDeviceToHost, s));
    if (n_lig > 0) {
        step(cudaMemcpyAsync(d_lig_r, d_lg, sizeof(float) * ng3 * n_lig, cudaMemcpyDeviceToHost, s));
        step(cudaMemcpyAsync(d_lig_i, d_lg + ng3 * n_lig, sizeof(float) * ng3 * n_lig, cudaMemcpyDeviceToHost, s));
    }
    step(cudaStreamSynchronize(s));
    if (e != cudaSuccess) {
        ctx->err = std::string("adjoint: ") + cudaGetErrorString(e);
        return MD_ERR_CUDA;
    }
    if (d_alpha) {
        double acc = 0.0;
        for (double v : part) acc += v;
        *d_alpha = alpha != 0.f ? acc / alpha : std::nan("");
    }
    return MD_OK;
}

int check_lig_sel(md_ctx *ctx, int n, const int *lig_sel, int n_lig, const float *a, const float *b) {
    if (n_lig < 0 || (n_lig > 0 && (!lig_sel || !a || !b))) return MD_ERR_ARG;
    for (int m = 0; m < n_lig; ++m)
        if (lig_sel[m] < 0 || lig_sel[m] >= n) {
            ctx->err = "ligand-grid selection outside the pose list";
            return MD_ERR_ARG;
        }
    return MD_OK;
}

}  // namespace

int md_adjoint_lse(md_ctx *ctx, const float *rotmat, int n_rot, const md_pose *top1, float temperature, float alpha,
                   double *loss, float *d_rec_r, float *d_rec_i, float *d_charge, double *d_alpha,
                   const int *lig_rot, int n_lig_rot, float *d_lig_r, float *d_lig_i) {
    if (!ctx || !rotmat || !top1 || n_rot < 1 || !(temperature > 0.f)) return MD_ERR_ARG;
    int rc = check_lig_sel(ctx, n_rot, lig_rot, n_lig_rot, d_lig_r, d_lig_i);
    if (rc) return rc;
    if ((rc = check_ready(ctx))) return rc;
    // loss and weights in double on the host: w_r = softmax(s_r / T); rotations
    // whose score was clamped to 0 (no positive cell) have no parameter gradient
    double smax = -1e300;
    for (int r = 0; r < n_rot; ++r) smax = std::max(smax, (double)top1[r].score);
    double z = 0.0;
    for (int r = 0; r < n_rot; ++r) z += std::exp(((double)top1[r].score - smax) / temperature);
    if (loss) *loss = smax + temperature * std::log(z);
    std::vector<float> w(n_rot);
    std::vector<int4> shift(n_rot);
    for (int r = 0; r < n_rot; ++r) {
        if (top1[r].i < 0 || top1[r].i >= ctx->N || top1[r].j < 0 || top1[r].j >= ctx->N || top1[r].k < 0 ||
            top1[r].k >= ctx->N) {
            ctx->err = "pose translation outside [0, nf1)";
            return MD_ERR_ARG;
        }
        const bool live = top1[r].score > 0.f;
        w[r] = live ? (float)(std::exp(((double)top1[r].score - smax) / temperature) / z) : 0.f;
        shift[r] = make_int4(top1[r].i, top1[r].j, top1[r].k, 0);
    }
    // only rotations with a nonzero float weight (or a requested ligand grid)
    // contribute: compact them, keeping their order
    std::vector<int> idx, remap(n_rot, -1);
    std::vector<char> want(n_rot, 0);
    for (int m = 0; m < n_lig_rot; ++m) want[lig_rot[m]] = 1;
    for (int r = 0; r < n_rot; ++r)
        if (w[r] != 0.f || want[r]) {
            remap[r] = (int)idx.size();
            idx.push_back(r);
        }
    if (idx.empty()) {   // no live rotation: every gradient is zero
        const size_t ng3 = (size_t)ctx->ng * ctx->ng * ctx->ng;
        if (d_rec_r) std::fill(d_rec_r, d_rec_r + ng3, 0.f);
        if (d_rec_i) std::fill(d_rec_i, d_rec_i + ng3, 0.f);
        if (d_charge) std::fill(d_charge, d_charge + ctx->na, 0.f);
        if (d_alpha) *d_alpha = 0.0;
        return MD_OK;
    }
    const int nc = (int)idx.size();
    std::vector<float> mc(9 * (size_t)nc), wc(nc);
    std::vector<int4> sc(nc);
    for (int c = 0; c < nc; ++c) {
        std::copy(rotmat + 9 * (size_t)idx[c], rotmat + 9 * (size_t)idx[c] + 9, mc.begin() + 9 * (size_t)c);
        wc[c] = w[idx[c]];
        sc[c] = shift[idx[c]];
    }
    std::vector<int> lc(n_lig_rot);
    for (int m = 0; m < n_lig_rot; ++m) lc[m] = remap[lig_rot[m]];
    return adjoint_core(ctx, mc.data(), nc, sc.data(), wc.data(), d_rec_r, d_rec_i, d_charge, lc.data(), n_lig_rot,
                        d_lig_r, d_lig_i, alpha, d_alpha);
}

int md_adjoint_poses(md_ctx *ctx, const float *rotmat, int n, const md_pose *poses, const float *dl_ds,
                     float *d_rec_r, float *d_rec_i, float *d_charge, const int *lig_pose, int n_lig,
                     float *d_lig_r, float *d_lig_i) {
    if (!ctx || !rotmat || !poses || !dl_ds || n < 1) return MD_ERR_ARG;
    int rc = check_lig_sel(ctx, n, lig_pose, n_lig, d_lig_r, d_lig_i);
    if (rc) return rc;
    if ((rc = check_ready(ctx))) return rc;
    std::vector<int4> shift(n);
    for (int r = 0; r < n; ++r) {
        if (poses[r].i < 0 || poses[r].i >= ctx->N || poses[r].j < 0 || poses[r].j >= ctx->N || poses[r].k < 0 ||
            poses[r].k >= ctx->N) {
            ctx->err = "pose translation outside [0, nf1)";
            return MD_ERR_ARG;
        }
        shift[r] = make_int4(poses[r].i, poses[r].j, poses[r].k, 0);
    }
    return adjoint_core(ctx, rotmat, n, shift.data(), dl_ds, d_rec_r, d_rec_i, d_charge, lig_pose, n_lig, d_lig_r,
                        d_lig_i, 0.f, nullptr);
}

int md_pose_scores(md_ctx *ctx, const float *rotmat, int n, const md_pose *poses, float *scores) {
    if (!ctx || !rotmat || !poses || !scores || n < 1) return MD_ERR_ARG;
    int rc = check_ready(ctx);
    if (rc) return rc;
    MD_CUDA(cudaSetDevice(ctx->device));
    const int N = ctx->N, ng = ctx->ng;
    const size_t ng3 = (size_t)ng * ng * ng;
    std::vector<int4> shift(n);
    for (int r = 0; r < n; ++r) {
        if (poses[r].i < 0 || poses[r].i >= N || poses[r].j < 0 || poses[r].j >= N || poses[r].k < 0 ||
            poses[r].k >= N) {
            ctx->err = "pose translation outside [0, nf1)";
            return MD_ERR_ARG;
        }
        shift[r] = make_int4(poses[r].i, poses[r].j, poses[r].k, 0);
    }
    int B = 1;
    char *p[4];
    rc = with_group(ctx, n, B, [&](int b) {
        const size_t sz[4] = {sizeof(float) * 9 * n, sizeof(int4) * n, sizeof(float) * n, sizeof(float) * 2 * ng3 * b};
        return carve_scratch(ctx, sz, 4, p);
    });
    if (rc) return rc;
    float *d_rot = reinterpret_cast<float *>(p[0]), *d_sc = reinterpret_cast<float *>(p[2]);
    int4 *d_shift = reinterpret_cast<int4 *>(p[1]);
    float *d_vox = reinterpret_cast<float *>(p[3]);
    cudaError_t e = cudaSuccess;
    auto step = [&](cudaError_t x) {
        if (e == cudaSuccess) e = x;
    };
    cudaStream_t s = ctx->stream;
    step(cudaMemcpyAsync(d_rot, rotmat, sizeof(float) * 9 * n, cudaMemcpyHostToDevice, s));
    step(cudaMemcpyAsync(d_shift, shift.data(), sizeof(int4) * n, cudaMemcpyHostToDevice, s));
    if (e == cudaSuccess) {
        for (int r0 = 0; r0 < n; r0 += B) {
            const int nb = std::min(B, n - r0);
            launch_voxel_chunk(ctx, d_rot + 9 * (size_t)r0, nb, d_vox, d_vox + ng3 * B);
            k_pose_dot<<<nb, 512, 0, s>>>(N, ng, ctx->d_recv, ctx->d_recv + ng3, d_vox, d_vox + ng3 * B,
                                          d_shift + r0, d_sc + r0);
        }
        step(cudaGetLastError());
        step(cudaMemcpyAsync(scores, d_sc, sizeof(float) * n, cudaMemcpyDeviceToHost, s));
        step(cudaStreamSynchronize(s));
    }
    if (e != cudaSuccess) {
        ctx->err = std::string("pose scores: ") + cudaGetErrorString(e);
        return MD_ERR_CUDA;
    }
    return MD_OK;
}

int md_pose_terms(md_ctx *ctx, const float *rec_rpsc, const float *rotmat, int n, const int *tem3, float *terms) {
    if (!ctx || !rec_rpsc || !rotmat || !tem3 || !terms || n < 1) return MD_ERR_ARG;
    int rc = check_ready(ctx);
    if (rc) return rc;
    const int ng = ctx->ng;
    for (int p = 0; p < 3 * n; ++p)
        if (tem3[p] < 0 || tem3[p] >= 2 * ng) {
            ctx->err = "pose offset outside [0, nf1)";
            return MD_ERR_ARG;
        }
    if (ng > kPoseTermMaxNg) {
        ctx->err = "pose terms: grid edge above " + std::to_string(kPoseTermMaxNg);
        return MD_ERR_SIZE;
    }
    MD_CUDA(cudaSetDevice(ctx->device));
    const size_t ng3 = (size_t)ng * ng * ng;
    // poses per launch: their voxel grids within about 1 GB
    const int P = (int)std::max<size_t>(1, std::min<size_t>((size_t)n, ((size_t)1 << 30) / (8 * ng3)));
    const size_t held = ctx->scratch_cap;
    int B = 1;
    char *p[5];
    rc = with_group(ctx, P, B, [&](int) {
        const size_t sz[5] = {sizeof(float) * 9 * n, sizeof(int4) * n, sizeof(float) * 9 * n, sizeof(float) * ng3,
                              sizeof(float) * 2 * ng3 * P};
        return carve_scratch(ctx, sz, 5, p);
    });
    if (rc) return rc;
    float *d_rot = reinterpret_cast<float *>(p[0]), *d_terms = reinterpret_cast<float *>(p[2]);
    float *d_rpsc = reinterpret_cast<float *>(p[3]), *d_vox = reinterpret_cast<float *>(p[4]);
    int4 *d_tem = reinterpret_cast<int4 *>(p[1]);
    cudaError_t e = cudaSuccess;
    auto step = [&](cudaError_t x) {
        if (e == cudaSuccess) e = x;
    };
    std::vector<int4> tem(n);
    for (int p = 0; p < n; ++p) tem[p] = make_int4(tem3[3 * p], tem3[3 * p + 1], tem3[3 * p + 2], 0);
    cudaStream_t s = ctx->stream;
    step(cudaMemcpyAsync(d_rot, rotmat, sizeof(float) * 9 * n, cudaMemcpyHostToDevice, s));
    step(cudaMemcpyAsync(d_tem, tem.data(), sizeof(int4) * n, cudaMemcpyHostToDevice, s));
    step(cudaMemcpyAsync(d_rpsc, rec_rpsc, sizeof(float) * ng3, cudaMemcpyHostToDevice, s));
    if (e == cudaSuccess) {
        for (int p0 = 0; p0 < n; p0 += P) {
            const int np = std::min(P, n - p0);
            for (int b0 = 0; b0 < np; b0 += B) {
                const int nb = std::min(B, np - b0);
                // the chunk's grids at [b0, b0 + nb) of the P-pose buffers
                launch_voxel_chunk(ctx, d_rot + 9 * (size_t)(p0 + b0), nb, d_vox + ng3 * b0,
                                   d_vox + ng3 * ((size_t)P + b0));
            }
            k_pose_terms<<<(np + kPoseTermWarps - 1) / kPoseTermWarps, 32 * kPoseTermWarps, 0, s>>>(
                ng, np, d_tem + p0, ctx->d_recv, d_rpsc, ctx->d_recv + ng3, d_vox, d_vox + ng3 * P,
                d_terms + 9 * (size_t)p0);
        }
        step(cudaGetLastError());
        step(cudaMemcpyAsync(terms, d_terms, sizeof(float) * 9 * n, cudaMemcpyDeviceToHost, s));
        step(cudaStreamSynchronize(s));
    }
    // a call over hundreds of poses gives its grids back
    if (ctx->scratch_cap > std::max(held, kScratchKept)) free_scratch(ctx);
    if (e != cudaSuccess) {
        ctx->err = std::string("pose terms: ") + cudaGetErrorString(e);
        return MD_ERR_CUDA;
    }
    return MD_OK;
}

int md_ligand_voxels(md_ctx *ctx, const float *rotmat9, float *grid_r, float *grid_i) {
    if (!ctx || !rotmat9 || !grid_r || !grid_i) return MD_ERR_ARG;
    if (!ctx->N || !ctx->have_ligand) {
        ctx->err = "grid and ligand must be set first";
        return MD_ERR_STATE;
    }
    MD_CUDA(cudaSetDevice(ctx->device));
    int rc = ensure_work(ctx, std::max(1, ctx->batch), 1);
    if (rc) return rc;
    const size_t ng3 = (size_t)ctx->ng * ctx->ng * ctx->ng;
    const size_t sz[2] = {sizeof(float) * 9, sizeof(float) * 2 * ng3};
    char *p[2];
    if ((rc = carve_scratch(ctx, sz, 2, p))) return rc;
    float *d_rot = reinterpret_cast<float *>(p[0]), *d_vr = reinterpret_cast<float *>(p[1]), *d_vi = d_vr + ng3;
    cudaError_t e = cudaMemcpyAsync(d_rot, rotmat9, sizeof(float) * 9, cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess) {
        launch_voxel_chunk(ctx, d_rot, 1, d_vr, d_vi);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(grid_r, d_vr, sizeof(float) * ng3, cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(grid_i, d_vi, sizeof(float) * ng3, cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) {
        ctx->err = std::string("voxelization: ") + cudaGetErrorString(e);
        return MD_ERR_CUDA;
    }
    return MD_OK;
}

}  // extern "C"
