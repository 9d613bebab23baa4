// Launch tables for the fake runtime: the docking and voxel entries of each FFT
// size note the work set they were handed instead of launching kernels.
#include <vector>

#include "../../megadock_b200/csrc/context.cuh"

extern "C" size_t fake_block(uintptr_t addr);

namespace {

struct Launch {
    WorkSet w;
    int rotations, t;
};
std::vector<Launch> launches;
int short_buffers = 0;   // launches whose work set was freed or too small

bool live(const WorkSet &w) {
    const void *p[] = {w.A, w.G, w.cand, w.vbits, w.qlist, w.qcount, w.srec, w.sstart, w.cq, w.cstart, w.marks};
    for (const void *q : p)
        if (!fake_block((uintptr_t)q)) return false;
    return true;
}

template <int N>
bool room(const WorkSet &w, size_t nb, size_t t, size_t na) {
    const size_t ng = N / 2;
    return fake_block((uintptr_t)w.A) >= sizeof(float2) * nb * ng * N * N &&
           fake_block((uintptr_t)w.G) >= sizeof(float2) * nb * ng * N * N &&
           fake_block((uintptr_t)w.cand) >= sizeof(Cand) * nb * inv_groups<N>() * t &&
           fake_block((uintptr_t)w.srec) >= sizeof(MarkEntry) * nb * na &&
           fake_block((uintptr_t)w.qlist) >= sizeof(int2) * nb * ng * ng * ng;
}

template <int N>
struct Fake {
    static void note(md_ctx *c, const WorkSet &w, int nb, int t) {
        launches.push_back({w, nb, t});
        if (!live(w) || !room<N>(w, nb, t, c->na)) ++short_buffers;
    }
    static void receptor(md_ctx *, const float *, const float *) {}
    static void voxel_chunk(md_ctx *c, const float *, int nb, float *, float *) { note(c, c->ws[0], nb, 1); }
    static void dock(md_ctx *c, const WorkSet &w, cudaStream_t, const float *, int nb, int, int t, DevPose *,
                     cudaEvent_t *) {
        note(c, w, nb, t);
    }
    static const SizedOps *ops() {
        static const SizedOps o = [] {
            SizedOps x = *sized_ops_of<N>();
            x.receptor = &receptor;
            x.voxel_chunk = &voxel_chunk;
            x.dock = &dock;
            return x;
        }();
        return &o;
    }
};

}  // namespace

namespace mdb {

const SizedOps *sized_ops_a(int N) {
    switch (N) {
    case 48: return Fake<48>::ops();
    case 128: return Fake<128>::ops();
    case 256: return Fake<256>::ops();
    default: return nullptr;
    }
}
#define NONE(x) \
    const SizedOps *sized_ops_##x(int) { return nullptr; }
NONE(b) NONE(c) NONE(d) NONE(e) NONE(f) NONE(g) NONE(h) NONE(i) NONE(j) NONE(k) NONE(l) NONE(m) NONE(n) NONE(o)
NONE(p) NONE(q) NONE(r)
#undef NONE

}  // namespace mdb

extern "C" {

int fake_launches() { return (int)launches.size(); }
int fake_rotations(int k) { return launches[k].rotations; }
int fake_live(int k) { return live(launches[k].w) ? 1 : 0; }
int fake_short() { return short_buffers; }
void fake_forget() { launches.clear(); }

}  // extern "C"
