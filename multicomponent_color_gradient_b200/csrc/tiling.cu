// tiling.cu - launch shape of the fused step and its dispatch by row pitch.
#include <algorithm>
#include <cstdlib>

#include "fused.cuh"

namespace mcg {

// The marches in one launch, on request only (MCG_FUSED_PIPE=0: k_fused, 1:
// k_fused_pipe; with MCG_FUSED_BULK=1 k_fused_bulk, rows of 128 columns): each
// is slower than the split step at every size measured, and they are kept as
// independent forms of the same arithmetic that the tests compare.
static void march_tiling(const Geometry &g, int max_smem, FusedTiling &t) {
    const int rpt = kFusedThreads / t.tpr;
    const bool f16 = g.storage == kStoreF16, pipe = t.march != kMarchBlock;
    t.threads = kFusedThreads;
    if (pipe) max_smem = std::max(max_smem, 112 * 1024);
    // rows per tile: whole rounds of rows in parallel, fewer if shared memory does not fit
    int ty = std::max(4, rpt);
    if (pipe && !f16) ty = t.tpr == 256 ? 1 : std::max(2, rpt);
    auto smem_of = [&](int h) {
        return (pipe ? kPipeRing * (h + 2) + kPipeStage * kMomCount * h : 3 * (h + 2) + 2 * kMomCount * h) * t.tpr * 4;
    };
    while (ty > 1 && smem_of(ty) > max_smem) --ty;
    if (ty > rpt) ty -= ty % rpt;
    t.ty = ty;
    t.smem_bytes = smem_of(ty);
    t.ny_tiles = (g.NY - 2 + ty - 1) / ty;
    if (t.march == kMarchBulk)
        t.smem_bytes = f16 ? bulk_smem_for<CodecF16>(ty) : bulk_smem_for<CodecF32>(ty);
    // z chunks: about thirteen CTAs per SM over the launch
    const int chunks = std::max(1, (13 * 148 + t.ny_tiles - 1) / t.ny_tiles);
    t.lz = std::max(4, (g.NZ - 2 + chunks - 1) / chunks);
    if (const char *v = std::getenv("MCG_FUSED_LZ")) t.lz = std::max(1, std::atoi(v));
    t.nz_chunks = (g.NZ - 2 + t.lz - 1) / t.lz;
    t.alternate = 1;
}

// The split step: a warp per piece of 32 columns, a plane per blockIdx.y.
static void split_tiling(const Geometry &g, FusedTiling &t) {
    const int ppr = g.storage == kStoreF16 ? pieces_per_row<CodecF16>(g) : pieces_per_row<CodecF32>(g);
    const int warps = kSplitThreads / 32;
    t.threads = kSplitThreads;
    t.ty = std::max(1, warps / ppr);
    t.lz = 1;
    t.ny_tiles = (ppr * (g.NY - 2) + warps - 1) / warps;
    t.nz_chunks = g.NZ - 2;
    // one wave of the interface launch, at most one warp per piece
    const long long per = kInterfaceThreads / 32, pieces = (long long)ppr * (g.NY - 2) * (g.NZ - 2);
    t.interface_ctas = int(std::min<long long>((pieces + per - 1) / per, 148 * kInterfaceBlocks));
    const long long columns = 2ll * (g.NX - 2) * (g.NZ - 2);
    t.boundary_ctas = int(std::min<long long>((columns + kInterfaceThreads - 1) / kInterfaceThreads, 148));
}

static int compiled_pitch(const Geometry &g) { return g.px % 32 == 0 ? g.px : 0; }

void retile_plain_rows(const Geometry &g, FusedTiling &t) {
    // a march's shape does not depend on the pitch
    if (t.march != kMarchSplit) return;
    split_tiling(g, t);
    t.pitch = 0;
}

FusedTiling fused_tiling(const Geometry &g, int max_smem) {
    FusedTiling t{};
    t.tpr = ((g.NX + 31) / 32) * 32;
    t.fixed_nx = (g.NX == kFusedNX || g.NX == kFusedNX2) ? g.NX : 0;
    if (const char *v = std::getenv("MCG_FUSED_FIXED_NX"))  // tests
        if (std::atoi(v) == 0) t.fixed_nx = 0;
    t.wait_limit = kBulkWaitLimit;
    t.march = kMarchSplit;
    if (const char *v = std::getenv("MCG_FUSED_PIPE")) t.march = std::atoi(v) != 0 ? kMarchPipe : kMarchBlock;
    if (const char *v = std::getenv("MCG_FUSED_BULK"))
        if (std::atoi(v) != 0 && t.march != kMarchBlock && t.fixed_nx == kFusedNX) t.march = kMarchBulk;
    // planes are blockIdx.y of the split step, whose extent ends at 65535; such a
    // grid can be set by mcg_set_populations, stepped and summed
    if (t.march == kMarchSplit && g.NZ - 2 > 65535) t.march = kMarchBlock;
    if (t.march == kMarchSplit)
        split_tiling(g, t);
    else
        march_tiling(g, max_smem, t);
    // the row pitch the kernels are compiled for (the marches: whole rows)
    t.pitch = t.march == kMarchSplit ? compiled_pitch(g) : t.fixed_nx;
    if (const char *v = std::getenv("MCG_FUSED_FIXED_NX"))  // tests
        if (std::atoi(v) == 0) t.pitch = 0;
    // the jet's inlet and outlet columns within the step's launches, instead of
    // a k_boundary launch after them
    t.boundary = g.boundary == kBoundaryJet;
    if (const char *v = std::getenv("MCG_FUSED_BOUNDARY")) t.boundary = t.boundary && std::atoi(v) != 0;  // tests
    return t;
}

// One object per row pitch instantiates these (fused.cu).
#define MCG_EACH_PITCH(F) F(0) F(32) F(64) F(96) F(128) F(160) F(192) F(224) F(256)
#define MCG_EXTERN(P)                                                                          \
    extern template cudaError_t fused_configure_pitch<P>(const Geometry &, const FusedTiling &); \
    extern template cudaError_t fused_launch_pitch<P>(const DeviceState &, const FusedTiling &, int, int64_t, bool, \
                                                      cudaStream_t);                           \
    extern template cudaError_t moments_launch_pitch<P>(const DeviceState &, int, int64_t, int, int, cudaStream_t); \
    extern template cudaError_t collide_launch_pitch<P>(const DeviceState &, int, int64_t, cudaStream_t);
MCG_EACH_PITCH(MCG_EXTERN)

cudaError_t fused_configure(const Geometry &g, const FusedTiling &t) {
    switch (t.pitch) {
#define MCG_CASE(P) \
    case P: return fused_configure_pitch<P>(g, t);
        MCG_EACH_PITCH(MCG_CASE)
#undef MCG_CASE
    }
    return cudaErrorInvalidValue;
}

cudaError_t launch_fused(const DeviceState &s, const FusedTiling &t_in, int cur, int64_t step, bool stats,
                         cudaStream_t st) {
    FusedTiling t = t_in;
    if (t.boundary) {
        t.bnd_dst = s.pops[cur ^ 1];
        t.bnd_psi = s.psi[(step + 1) & 1];
        t.bnd_step = step;
    }
    switch (t.pitch) {
#define MCG_CASE(P) \
    case P: return fused_launch_pitch<P>(s, t, cur, step, stats, st);
        MCG_EACH_PITCH(MCG_CASE)
#undef MCG_CASE
    }
    return cudaErrorInvalidValue;
}

cudaError_t launch_moments_planes(const DeviceState &s, int cur, int64_t step, int first, int planes, cudaStream_t st) {
    switch (compiled_pitch(s.g)) {
#define MCG_CASE(P) \
    case P: return moments_launch_pitch<P>(s, cur, step, first, planes, st);
        MCG_EACH_PITCH(MCG_CASE)
#undef MCG_CASE
    }
    return cudaErrorInvalidValue;
}

cudaError_t launch_moments(const DeviceState &s, int cur, int64_t step, bool stats, cudaStream_t st) {
    const cudaError_t e = launch_moments_planes(s, cur, step, 1, s.g.NZ - 2, st);
    if (e != cudaSuccess || !stats) return e;
    return launch_accumulate_radial(s, st);
}

cudaError_t launch_collide(const DeviceState &s, int cur, int64_t step, cudaStream_t st) {
    switch (compiled_pitch(s.g)) {
#define MCG_CASE(P) \
    case P: return collide_launch_pitch<P>(s, cur, step, st);
        MCG_EACH_PITCH(MCG_CASE)
#undef MCG_CASE
    }
    return cudaErrorInvalidValue;
}

}  // namespace mcg
