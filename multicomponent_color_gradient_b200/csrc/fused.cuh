// fused.cuh - the D3Q27 colour-gradient step on B200 (sm_100a).
//
// The step pulls f(t) of every interior node (row-blocked layout, so a pulled
// row is nine contiguous segments), forms rho_r, rho_b, u, Pi^neq
// (lbm.cuh:82-165) and psi, accumulates the radial statistics
// (kernels.cu:188-233) with warp segmented reductions, relaxes (lbm.cuh:184-293):
// Hermite-regularised BGK and, at interface nodes, colour-gradient perturbation
// and recolouring, and stores the post-collision values at the node (pull
// layout, coalesced rows).  The jet's inlet (jet/boundary_conditions.cuh:17-85)
// and convective outlet (:163-233) columns go into the y ghost planes of the
// new buffer.  Moments do not go through the moment planes in HBM.
//   k_step_pull, k_step_interface
//              the step in two launches: a node is relaxed where it is pulled
//              unless an interface needs psi of its neighbours.
//   k_fused, k_fused_pipe, k_fused_bulk
//              the step as a march over z in one launch, on request: a CTA
//              owns a tile of rows, pulls its rows and a one-row halo plane by
//              plane, keeps psi in shared memory and relaxes behind the march
//              front.  Kept as independent forms of the same arithmetic that
//              the tests compare bit for bit.
//   k_boundary the boundary as a launch of its own, one thread per column,
//              from the fluid-plane moments the step leaves in bmom (the
//              granular sequence, and MCG_FUSED_BOUNDARY=0).
// The reference's in-place push buffer becomes a ping-pong pull pair; the
// populations a reference step never rewrites (y=1 slots fed by non-jet
// inlet columns, y=NY-2 slots fed by ghost columns) are ghost-plane values of
// both buffers that no kernel writes, so results are the same.
#pragma once
#include "step.cuh"

namespace mcg {
namespace {

// ------------------------------------------------------------------ marches

constexpr int kFusedThreads = 256;
// Row lengths the fused kernels are specialised for (the 128-column rows of
// the 128x256x128 jet, the 256-column rows of the 256x512x256 one); other
// row lengths take the runtime-geometry kernels.
constexpr int kFusedNX = 128;
constexpr int kFusedNX2 = 256;

#ifndef MCG_FUSED_MIN_BLOCKS
#define MCG_FUSED_MIN_BLOCKS 3  // CTAs per SM the register budget is sized for
#endif

// First row of this CTA's y-tile.  With the jet boundary in the step the
// tiles are numbered from the outlet end: the outlet tile's CTAs, which also
// write the outlet columns, then start first in each chunk instead of last.
// Neighbouring CTAs still hold neighbouring tiles.
__device__ __forceinline__ int tile_y0(const FusedTiling &T) {
    const int t = T.boundary ? T.ny_tiles - 1 - int(blockIdx.x) : int(blockIdx.x);
    return 1 + t * T.ty;
}

// Own-row results of a pulled node that leave the march: the fluid-plane
// moments for the boundary (fused_boundary or k_boundary) and the adjoint's
// moment record.
__device__ __forceinline__ void tile_record_moments(const DeviceState &s, int x, int y, int zp, const NodeMoments &m,
                                                    float ps) {
    const Geometry &g = s.g;
    if (g.boundary == kBoundaryJet && (y == 1 || y == g.NY - 2)) {
        // fluid-plane moments for the boundary launch
        float *b = s.bmom + ((size_t(y == 1 ? 0 : 1) * g.NZ + zp) * kMomCount) * g.NX + x;
        const float v[kMomCount] = {m.rr, m.rb, m.ux, m.uy, m.uz, m.pxx, m.pxy, m.pyy, m.pyz, m.pzz, m.pxz};
#pragma unroll
        for (int k = 0; k < kMomCount; ++k) b[size_t(k) * g.NX] = v[k];
    }
    if (s.tape) {
        // moment record of the pulled state (the adjoint sweep reads it)
        float *t = s.tape + (uint32_t(x) + uint32_t(g.sy) * uint32_t(y) + uint32_t(g.sz) * uint32_t(zp));
        const size_t N = g.N;
        const float v[kTapePlanes] = {m.rr, m.rb, m.ux, m.uy, m.uz, m.pxx, m.pxy, m.pyy, m.pyz, m.pzz, m.pxz, ps};
#pragma unroll
        for (int k = 0; k < kTapePlanes; ++k) t[size_t(k) * N] = v[k];
    }
}

// The moments into the stage row, for a relaxation in a later iteration.
__device__ __forceinline__ void tile_stage_moments(int x, const NodeMoments &m, float *msm_row, int tpr) {
    float *q = msm_row + x;
    q[kMomRR * tpr] = m.rr;
    q[kMomRB * tpr] = m.rb;
    q[kMomUX * tpr] = m.ux;
    q[kMomUY * tpr] = m.uy;
    q[kMomUZ * tpr] = m.uz;
    q[kMomPXX * tpr] = m.pxx;
    q[kMomPXY * tpr] = m.pxy;
    q[kMomPYY * tpr] = m.pyy;
    q[kMomPYZ * tpr] = m.pyz;
    q[kMomPZZ * tpr] = m.pzz;
    q[kMomPXZ * tpr] = m.pxz;
}

template <class C>
__device__ __forceinline__ void tile_store_moments(const DeviceState &s, int x, int y, int zp, const NodeMoments &m,
                                                   float ps, float *msm_row, int tpr) {
    tile_stage_moments(x, m, msm_row, tpr);
    tile_record_moments(s, x, y, zp, m, ps);
}

// One node of a tile row in plane zp, pulled in two halves.  tile_pull_issue
// loads the node's words (at a position that is not pulled, its psi);
// tile_pull_finish puts psi into `ring_row` (all columns, halo rows
// included), and for own rows the moments into `msm_row`, the fluid-plane
// moments for the boundary launch, the adjoint's moment record, and the
// radial statistics.  tile_pull_finish is warp-collective when kStats: all
// 32 lanes of a warp (one row) call it together.  TilePull holds the loads
// between the two.
template <class C>
struct TilePull {
    RawPull<C> raw;  // the node's pulled words, when `pull`
    float ps;        // psi of a position that is not pulled (ghost)
    bool pull;
};

template <class C, bool kPeriodic>
__device__ __forceinline__ void tile_pull_issue(const DeviceState &s, const C &codec, const float *__restrict__ psi_g,
                                                int x, int y, int zp, TilePull<C> &t) {
    const Geometry &g = s.g;
    t.pull = false;
    if (x >= g.NX) return;
    int xn = x, yn = y, zn = zp;
    if constexpr (kPeriodic) {
        xn = wrap_interior(x, g.NX);
        yn = wrap_interior(y, g.NY);
        zn = wrap_interior(zp, g.NZ);
        t.pull = true;
    } else {
        t.pull = x >= 1 && x <= g.NX - 2 && y >= 1 && y <= g.NY - 2 && zp >= 1 && zp <= g.NZ - 2;
    }
    if (t.pull)
        pull_issue<C, kPeriodic>(g, codec, xn, yn, zn, t.raw);
    else
        t.ps = psi_g[uint32_t(x) + uint32_t(g.sy) * uint32_t(y) + uint32_t(g.sz) * uint32_t(zp)];
}

// A node's statistics sample held for a later radial_accumulate_warp call.
struct RadialSample {
    float ux, uy, uz;
    int y, z;
    bool active;
};

template <class C, bool kStats, bool kPeriodic>
__device__ __forceinline__ void tile_pull_finish(const DeviceState &s, const C &codec, int x, int y, int zp,
                                                 bool own_row, const TilePull<C> &t, float *ring_row, float *msm_row,
                                                 int tpr, RadialSample *defer = nullptr) {
    const Geometry &g = s.g;
    const bool xin = x >= 1 && x <= g.NX - 2;
    NodeMoments m{};
    bool have = false;
    if (x < g.NX) {
        float ps;
        if (t.pull && own_row) {  // own_row is uniform per warp: a warp covers part of one row
            m = moments_from(RawSource<C>{codec, t.raw});
            have = true;
            ps = psi_of(m.rr, m.rb);
        } else if (t.pull) {
            float rr, rb;
            densities_from(RawSource<C>{codec, t.raw}, rr, rb);
            ps = psi_of(rr, rb);
        } else {
            ps = t.ps;
        }
        ring_row[x] = ps;
        if (own_row && xin) tile_store_moments<C>(s, x, y, zp, m, ps, msm_row, tpr);
    }
    if constexpr (kStats) {
        if (defer) {
            *defer = RadialSample{m.ux, m.uy, m.uz, y, zp, have && xin};
        } else if (own_row) {
            radial_accumulate_warp(s, x, y, zp, have && xin, m.ux, m.uy, m.uz);
        }
    }
}

// One node of a tile row in plane zp: psi into `ring_row` (all columns, halo
// rows included), and for own rows the moments into `msm_row`, the fluid-plane
// moments for the boundary, the adjoint's moment record, and the radial
// statistics.  The own-row / halo branch comes before the loads, so each
// branch consumes its loads as they arrive (issuing all of them before the
// branch keeps every word live at once and spills at 80 registers).
template <class C, bool kStats, bool kPeriodic>
__device__ __forceinline__ void tile_pull(const DeviceState &s, const C &codec, const float *__restrict__ psi_g, int x,
                                          int y, int zp, bool own_row, float *ring_row, float *msm_row, int tpr) {
    const Geometry &g = s.g;
    const bool xin = x >= 1 && x <= g.NX - 2;
    NodeMoments m{};
    bool have = false;
    if (x < g.NX) {
        int xn = x, yn = y, zn = zp;
        bool pull;
        if constexpr (kPeriodic) {
            xn = wrap_interior(x, g.NX);
            yn = wrap_interior(y, g.NY);
            zn = wrap_interior(zp, g.NZ);
            pull = true;
        } else {
            pull = xin && y >= 1 && y <= g.NY - 2 && zp >= 1 && zp <= g.NZ - 2;
        }
        float ps;
        if (pull && own_row) {  // uniform per warp: a warp covers part of one row
            m = pull_moments<C, kPeriodic>(g, codec, xn, yn, zn);
            have = true;
            ps = psi_of(m.rr, m.rb);
        } else if (pull) {
            float rr, rb;
            pull_densities<C, kPeriodic>(g, codec, xn, yn, zn, rr, rb);
            ps = psi_of(rr, rb);
        } else {
            ps = psi_g[uint32_t(x) + uint32_t(g.sy) * uint32_t(y) + uint32_t(g.sz) * uint32_t(zp)];
        }
        ring_row[x] = ps;
        if (own_row && xin) tile_store_moments<C>(s, x, y, zp, m, ps, msm_row, tpr);
    }
    if constexpr (kStats) {
        if (own_row) radial_accumulate_warp(s, x, y, zp, have && xin, m.ux, m.uy, m.uz);
    }
}

// Hides how the moments were formed from the compiler, at no instruction: it
// may otherwise contract their last operations with the collision's first ones
// differently in each kernel, and a node relaxed from registers would differ
// in the last bit from one relaxed from the stage.
__device__ __forceinline__ void opaque(NodeMoments &m) {
    asm volatile("" : "+f"(m.rr), "+f"(m.rb), "+f"(m.ux), "+f"(m.uy), "+f"(m.uz));
    asm volatile("" : "+f"(m.pxx), "+f"(m.pxy), "+f"(m.pyy), "+f"(m.pyz), "+f"(m.pzz), "+f"(m.pxz));
}

// Relax interior node (x, y, zc) of a tile: moments from the stage row
// `msm_row`, psi of planes zc-1, zc, zc+1 from the ring planes pm, p0, pp at
// ring row r.
template <class C>
__device__ __forceinline__ void tile_collide(const DeviceState &s, const C &codec, int x, int y, int zc, int r,
                                             const float *msm_row, const float *pm, const float *p0, const float *pp,
                                             int tpr) {
    const Geometry &g = s.g;
    const float *q = msm_row + x;
    NodeMoments m;
    m.rr = q[kMomRR * tpr];
    m.rb = q[kMomRB * tpr];
    m.ux = q[kMomUX * tpr];
    m.uy = q[kMomUY * tpr];
    m.uz = q[kMomUZ * tpr];
    m.pxx = q[kMomPXX * tpr];
    m.pxy = q[kMomPXY * tpr];
    m.pyy = q[kMomPYY * tpr];
    m.pyz = q[kMomPYZ * tpr];
    m.pzz = q[kMomPZZ * tpr];
    m.pxz = q[kMomPXZ * tpr];
    const int base = r * tpr + x;
    auto psi_at = [&](int cx, int cy, int cz) {
        const float *pl = cz < 0 ? pm : (cz > 0 ? pp : p0);
        return pl[base + cy * tpr + cx];
    };
    collide_node<false>(g, s.ph, codec, pop_row(g, y, zc), x, y, zc, m, psi_at);
}

// The jet boundary of a fused step, from the CTAs whose tile holds fluid row
// 1 (inlet) or NY-2 (outlet), once their march is over: every column of the
// chunk from the fluid-plane moments the march left in bmom (written by this
// CTA's threads, visible after the barrier), into the ghost planes of the
// buffer the step writes and the next step's psi.  A column touches only its
// own ghost nodes and the outlet state it carries, which no other CTA of the
// launch reads.  Kept out of the march, where it added its instructions to
// every row.  The condition is uniform over the CTA.
template <class C>
__device__ __forceinline__ void fused_boundary(const DeviceState &s, const FusedTiling &T, int y0, int ty, int z0,
                                               int lz) {
    const Geometry &g = s.g;
    const bool inlet = y0 == 1, outlet = y0 + ty - 1 == g.NY - 2;
    if (!T.boundary || !(inlet || outlet)) return;
    __syncthreads();
    const int nx = g.NX - 2;
    for (int side = 0; side < 2; ++side) {
        if (!(side == 0 ? inlet : outlet)) continue;
        for (int i = threadIdx.x; i < lz * nx; i += blockDim.x) {
            const int x = 1 + i % nx, z = z0 + i / nx;
            const NodeMoments m =
                load_moments(s.bmom + (size_t(side) * g.NZ + z) * kMomCount * g.NX, size_t(g.NX), size_t(x));
            if (side == 0)
                inlet_column<C>(s, T.bnd_dst, T.bnd_psi, x, z, int64_t(T.bnd_step), m);
            else
                outlet_column<C>(s, T.bnd_dst, T.bnd_psi, x, z, m);
        }
    }
}

// Geometry of a fused launch: with kNX > 0 (rows of exactly kNX columns, one
// thread per column) the row length and slot counts are compile-time
// constants, so population, slot and shared-memory offsets fold into the
// loads' immediate offsets.
template <class C, int kNX>
__device__ __forceinline__ DeviceState fused_state(const DeviceState &s) {
    DeviceState l = s;
    if constexpr (kNX > 0) {
        l.g.NX = kNX;
        l.g.px = kNX;
        l.g.sy = kNX;
        l.g.slots = 9 * C::kGroupSlots;
    }
    return l;
}
template <class C, int kNX>
__device__ __forceinline__ C fused_codec(const DeviceState &s, int cur) {
    C c = make_codec<C>(s, cur);
    if constexpr (kNX > 0) c.px = kNX;
    return c;
}
// The same with only the row pitch of the populations compiled in (rows of up
// to kPX columns).
template <class C, int kPX>
__device__ __forceinline__ DeviceState pitch_state(const DeviceState &s) {
    DeviceState l = s;
    if constexpr (kPX > 0) {
        l.g.px = kPX;
        l.g.slots = 9 * C::kGroupSlots;
    }
    return l;
}
// Brings the parameters of a step into the constant cache while the launch before
// runs (8^3 5.7 us a step without, 5.1 with, together with relax_flagged).
__device__ __forceinline__ void touch_params(const DeviceState &s) {
    asm volatile("" ::"f"(s.ph.omega), "r"(s.ph.sponge), "l"(s.piece_flags), "l"(s.tape));
}
template <class C, int kPX>
__device__ __forceinline__ C pitch_codec(const DeviceState &s, int cur) {
    return fused_codec<C, kPX>(s, cur);
}

template <class C, bool kStats, bool kPeriodic, int kNX>
__global__ void __launch_bounds__(kFusedThreads, MCG_FUSED_MIN_BLOCKS) k_fused(const DeviceState s_arg,
                                                                              const FusedTiling T, int cur,
                                                                              int64_t step) {
    extern __shared__ float sm[];
    const DeviceState s = fused_state<C, kNX>(s_arg);
    const Geometry &g = s.g;
    const int tpr = kNX > 0 ? kNX : T.tpr;
    const int rpt = kFusedThreads / tpr;
    // row group of this thread; groups beyond rpt (when tpr does not divide
    // the block) start past every row and only take part in the barriers
    const int lr0 = threadIdx.x / tpr;
    const int lr = lr0 < rpt ? lr0 : T.ty + 2;
    const int x = threadIdx.x - lr0 * tpr;
    const int y0 = tile_y0(T);
    const int ty = min(T.ty, g.NY - 1 - y0);
    const int z0 = 1 + int(blockIdx.y) * T.lz;
    const int lz = min(T.lz, g.NZ - 1 - z0);
    const int pstride = (T.ty + 2) * tpr;  // one psi plane of the ring
    float *ring = sm;                      // [3][ty+2][tpr]
    float *msm = sm + 3 * pstride;         // [2][ty][11][tpr]
    const int mplane = T.ty * kMomCount * tpr;
    const C codec = fused_codec<C, kNX>(s_arg, cur);
    const float *__restrict__ psi_g = s_arg.psi[step & 1];  // indexed on the parameter, not the local copy
    const bool xin = x >= 1 && x <= g.NX - 2;
    // Odd chunks march down: the plane two neighbouring chunks both pull (one
    // as its halo, one as its own) is then pulled by both at the same end of
    // their marches, close in time, and the second pull finds it in L2.
    const bool down = T.alternate && (blockIdx.y & 1);
    for (int k = 0; k <= lz + 1; ++k) {
        const int zp = down ? z0 + lz - k : z0 - 1 + k;
        float *ringp = ring + (zp % 3) * pstride;
        float *msmp = msm + (zp & 1) * mplane;
        const bool own_plane = zp >= z0 && zp < z0 + lz;
        // ---- pull plane zp: psi for rows y0-1 .. y0+ty, moments for own rows
        for (int r = lr; r < ty + 2; r += rpt) {
            tile_pull<C, kStats, kPeriodic>(s, codec, psi_g, x, y0 - 1 + r, zp, own_plane && r >= 1 && r <= ty,
                                            ringp + r * tpr, msmp + (r - 1) * kMomCount * tpr, tpr);
        }
        __syncthreads();
        // ---- relax the plane behind the march front, whose neighbours are all pulled
        const int zc = down ? zp + 1 : zp - 1;
        if (zc >= z0 && zc < z0 + lz) {
            const float *pm = ring + ((zc + 2) % 3) * pstride;  // plane zc-1
            const float *p0 = ring + (zc % 3) * pstride;        // plane zc
            const float *pp = ring + ((zc + 1) % 3) * pstride;  // plane zc+1
            const float *mc = msm + (zc & 1) * mplane;
            for (int r = 1 + lr; r <= ty; r += rpt) {
                if (!xin) continue;
                tile_collide(s, codec, x, y0 - 1 + r, zc, r, mc + (r - 1) * kMomCount * tpr, pm, p0, pp, tpr);
            }
        }
        __syncthreads();
    }
    fused_boundary<C>(s, T, y0, ty, z0, lz);
}

// ------------------------------------------------------------------ software-pipelined fused step

// The tile march of k_fused with the pull and the relaxation in the same
// phase: iteration k pulls march plane k and relaxes march plane k-2, whose
// psi neighbours (planes k-3 .. k-1) and moments were pulled in earlier
// iterations.  The pull writes ring slot k mod 4 and stage slot k mod 3; the
// relaxation reads ring slots k-3 .. k-1 and stage slot k-2 - all different -
// so one __syncthreads per iteration suffices.  Between barriers the warps of
// a CTA drift apart, and the memory-bound pull of one warp overlaps the
// ALU-bound relaxation of another.
constexpr int kPipeRing = 4, kPipeStage = 3;
// CTAs per SM the pipelined kernel's register budget is sized for: float32
// (3-row tiles, 3 CTAs, 80 registers) measured faster than 2 CTAs at 128
// registers; float16 keeps 2 (its words in flight across the relaxation need
// the registers).
template <class C>
struct PipeBlocks {
    static constexpr int value = std::is_same<C, CodecF16>::value ? 2 : 3;
};

template <class C, bool kStats, bool kPeriodic, int kNX>
__global__ void __launch_bounds__(kFusedThreads, PipeBlocks<C>::value) k_fused_pipe(const DeviceState s_arg,
                                                                                  const FusedTiling T, int cur,
                                                                                  int64_t step) {
    extern __shared__ float sm[];
    const DeviceState s = fused_state<C, kNX>(s_arg);
    const Geometry &g = s.g;
    const int tpr = kNX > 0 ? kNX : T.tpr;
    const int rpt = kFusedThreads / tpr;
    const int lr0 = threadIdx.x / tpr;
    const int lr = lr0 < rpt ? lr0 : T.ty + 2;  // idle groups (tpr not dividing the block) skip every row
    const int x = threadIdx.x - lr0 * tpr;
    const int pstride = (T.ty + 2) * tpr;
    const int mplane = T.ty * kMomCount * tpr;
    float *ring = sm;                        // [4][ty+2][tpr]
    float *msm = sm + kPipeRing * pstride;   // [3][ty][11][tpr]
    const C codec = fused_codec<C, kNX>(s_arg, cur);
    const float *__restrict__ psi_g = s_arg.psi[step & 1];  // indexed on the parameter, not the local copy
    const bool xin = x >= 1 && x <= g.NX - 2;
    // Float16 words (27 registers a node) stay in flight across the relaxation
    // of another row: measured +4 % on 128x256x128.  Float32 (27 float2, 54
    // registers) pulls then relaxes: its 3-CTA, 80-register default is faster
    // than the overlap, which spills there.
    constexpr bool kOverlap = std::is_same<C, CodecF16>::value;
    // One CTA per y-tile (blockIdx.x) and z chunk (blockIdx.y): CTAs of
    // neighbouring y-tiles run the same planes at about the same time, so the
    // halo rows one pulls are the own rows another pulled and hit L2.  Odd
    // chunks march down: two neighbouring chunks then pull their shared
    // boundary plane at the same end of their marches (L2 again).
    {
        const int y0 = tile_y0(T);
        const int z0 = 1 + int(blockIdx.y) * T.lz;
        const int lz = min(T.lz, g.NZ - 1 - z0);
        const bool down = T.alternate && (blockIdx.y & 1);
        const int ty = min(T.ty, g.NY - 1 - y0);
        auto plane = [&](int k) { return down ? z0 + lz - k : z0 - 1 + k; };
        RadialSample held{};   // statistics of this warp's last own row, taken
        bool pending = false;  // after the next row's loads are issued
        for (int k = 0; k <= lz + 2; ++k) {
            const bool do_pull = k <= lz + 1;
            const int c = k - 2;  // march index of the plane relaxed in this iteration
            const bool do_relax = c >= 1 && c <= lz;
            const int zp = plane(k);
            float *ringp = ring + (k % kPipeRing) * pstride;
            float *msmp = msm + (k % kPipeStage) * mplane;
            const bool own_plane = k >= 1 && k <= lz;
            const int zc = plane(c);
            const float *pm = ring + (((down ? c + 1 : c - 1) + kPipeRing) % kPipeRing) * pstride;  // plane zc-1
            const float *p0 = ring + ((c + kPipeRing) % kPipeRing) * pstride;                       // plane zc
            const float *pp = ring + (((down ? c - 1 : c + 1) + kPipeRing) % kPipeRing) * pstride;  // plane zc+1
            const float *mc = msm + ((c + kPipeStage) % kPipeStage) * mplane;
            // rows of this thread: pull rows lr, lr+rpt, ... (< ty+2) and relax rows
            // 1+lr, 1+lr+rpt, ... (<= ty), interleaved so that a warp has loads of
            // one row in flight while it relaxes another.  With one row group (rows
            // of 256 columns) the upper half of the row's threads takes the rows in
            // a rotated order, so that one half pulls while the other relaxes, as
            // two row groups do; the order of the rows within an iteration is free.
            // (split at a warp boundary: the statistics are warp-collective)
            const int rot = (rpt == 1 && x >= (tpr / 64) * 32) ? (ty + 2) / 2 : 0;
            for (int ri = lr; ri < ty + 2; ri += rpt) {
                const int r = rot ? (ri + rot) % (ty + 2) : ri;
                const bool own = own_plane && r >= 1 && r <= ty;
                const int rc = r + 1;
                if constexpr (kOverlap) {
                    // the loads of row r are in flight while this warp takes the
                    // statistics of its previous own row and relaxes row r+1
                    TilePull<C> tp;
                    if (do_pull) tile_pull_issue<C, kPeriodic>(s, codec, psi_g, x, y0 - 1 + r, zp, tp);
                    if constexpr (kStats) {
                        if (pending) {  // warp-uniform
                            radial_accumulate_warp(s, x, held.y, held.z, held.active, held.ux, held.uy, held.uz);
                            pending = false;
                        }
                    }
                    if (do_relax && rc <= ty && xin)
                        tile_collide(s, codec, x, y0 - 1 + rc, zc, rc, mc + (rc - 1) * kMomCount * tpr, pm, p0, pp,
                                     tpr);
                    if (do_pull) {
                        tile_pull_finish<C, kStats, kPeriodic>(s, codec, x, y0 - 1 + r, zp, own, tp, ringp + r * tpr,
                                                               msmp + (r - 1) * kMomCount * tpr, tpr,
                                                               kStats && own ? &held : nullptr);
                        if (kStats && own) pending = true;
                    }
                } else {
                    if (do_pull)
                        tile_pull<C, kStats, kPeriodic>(s, codec, psi_g, x, y0 - 1 + r, zp, own, ringp + r * tpr,
                                                        msmp + (r - 1) * kMomCount * tpr, tpr);
                    if (do_relax && rc <= ty && xin)
                        tile_collide(s, codec, x, y0 - 1 + rc, zc, rc, mc + (rc - 1) * kMomCount * tpr, pm, p0, pp,
                                     tpr);
                }
            }
            __syncthreads();
        }
        if constexpr (kStats) {
            if (pending) radial_accumulate_warp(s, x, held.y, held.z, held.active, held.ux, held.uy, held.uz);
        }
        fused_boundary<C>(s, T, y0, ty, z0, lz);
    }
}

// ------------------------------------------------------------------ the split step

// The step in two launches, neither with a march, a halo or shared memory:
//   k_step_pull       one warp per piece of 32 columns of a row: pulls its 32
//                     nodes, forms moments, psi and statistics, and, when all
//                     32 are bulk, relaxes and stores them at once.  A piece
//                     (float16: a quarter of one) with an interface node
//                     leaves its moments in the slots it will store (of the
//                     buffer the step writes, which no one reads yet) and sets
//                     its flag.
//   k_step_interface  relaxes the flagged pieces, with the colour gradient
//                     from the psi the first launch wrote for every node, and
//                     writes the jet's inlet and outlet columns.
// Bound by HBM: a node's 27 elements are read and written once; psi adds 4 B
// written, an interface piece 48 B written and read again, and psi read, mostly
// in L2.  A march forms psi of the halo rows and planes of its tile by pulling
// them (2.3 pulls a node on 2-row tiles of 13 planes), holds its warps at
// barriers and leaves columns 0 and NX-1 unwritten (see store_columns); the
// pull launch runs at the rate of a plain copy of the same elements.
// us a step, this against the marches chosen before (fraction of the measured
// copy peak at 432 or 216 B a node): jet 128x256x128 float32 296 (0.90) against
// 352 (0.76), 256x512x256 2264 (0.96) against 2984 (0.73), 200x301x183 769
// (0.92) against 1541 (0.46), 64x128x64 39 against 76, 24x40x24 6.6 against 29;
// float16 jet 128x400x128 258 (0.81) against 441, 256x512x256 1216 (0.89)
// against 2073 (0.52).  With an interface at every node, which no flow keeps, float32
// 128x256x128 takes 358 against 351 and float16 256^3 1256 against 1228; other
// sizes gain there too (float16 128x256x128 316 against 324, float32 256^3 1450
// against 1558, 200x301x183 1052 against 1556, 64x128x64 42 against 77).

// Threads and CTAs per SM the register budgets are sized for: k_step_pull 72
// registers (64, with spills in float32, to 96 measured within 1 % in float32;
// the float16 jet 128x256x128 takes 171 us a step at 72, 175 at 64 and 189 at
// 80), k_step_interface 96 (at 80 a periodic float16 run of 128^2 x 256 was 12 %
// slower, at 2 CTAs of 256 threads a float16 jet 13 %).
constexpr int kSplitThreads = 128, kSplitBlocks = 7;
constexpr int kInterfaceThreads = 128, kInterfaceBlocks = 5;
// Neighbouring pieces that one CTA of k_step_interface takes together: whole
// rows of 128 columns (4 against 1: 174 against 196 us a step for the
// 128x256x128 float16 jet, 2250 against 2328 for 256x512x256 float32).
constexpr int kPieceGroup = 4;

// Float16, whose pull issues in 73 % of the cycles (float32: 33 %), parks and relaxes
// quarters of 8 columns (32 bytes of a row): fewer bulk nodes go through the
// interface launch (64x128x64 jet 28.0 us a step against 31.6 by pieces, periodic
// drops 128x256x128 181 against 195).  Float32 is bound by HBM and takes whole
// pieces (318 by quarters against 313 for the same drops).
template <class C>
constexpr bool relax_by_quarters() { return std::is_same<C, CodecF16>::value; }

// Moments of a node to and from its own element slots in the row it will
// store: two floats an element in float32, one in float16.
__device__ __forceinline__ void park_moments(float2 *wrow, int px, const NodeMoments &m) {
    wrow[0 * px] = make_float2(m.rr, m.rb);
    wrow[1 * px] = make_float2(m.ux, m.uy);
    wrow[2 * px] = make_float2(m.uz, m.pxx);
    wrow[3 * px] = make_float2(m.pxy, m.pyy);
    wrow[4 * px] = make_float2(m.pyz, m.pzz);
    wrow[5 * px] = make_float2(m.pxz, 0.0f);
}
__device__ __forceinline__ void unpark_moments(const float2 *wrow, int px, NodeMoments &m) {
    const float2 a = wrow[0 * px], b = wrow[1 * px], c = wrow[2 * px], d = wrow[3 * px], e = wrow[4 * px];
    m.pxz = wrow[5 * px].x;
    m.rr = a.x; m.rb = a.y;
    m.ux = b.x; m.uy = b.y; m.uz = c.x;
    m.pxx = c.y; m.pxy = d.x; m.pyy = d.y; m.pyz = e.x; m.pzz = e.y;
}
__device__ __forceinline__ void park_moments(__half2 *wrow, int px, const NodeMoments &m) {
    float *w = reinterpret_cast<float *>(wrow);
    const float v[kMomCount] = {m.rr, m.rb, m.ux, m.uy, m.uz, m.pxx, m.pxy, m.pyy, m.pyz, m.pzz, m.pxz};
#pragma unroll
    for (int k = 0; k < kMomCount; ++k) w[k * px] = v[k];
}
__device__ __forceinline__ void unpark_moments(const __half2 *wrow, int px, NodeMoments &m) {
    const float *w = reinterpret_cast<const float *>(wrow);
    float v[kMomCount];
#pragma unroll
    for (int k = 0; k < kMomCount; ++k) v[k] = w[k * px];
    m = NodeMoments{v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7], v[8], v[9], v[10]};
}

template <class C, bool kStats, bool kPeriodic, int kPX>
__global__ void __launch_bounds__(kSplitThreads, kSplitBlocks) k_step_pull(const DeviceState s_arg, int cur, int64_t step) {
    const DeviceState s = pitch_state<C, kPX>(s_arg);
    const Geometry &g = s.g;
    C codec = pitch_codec<C, kPX>(s_arg, cur);
    // blockIdx.y: plane; along x, pieces of its rows, neighbours in one block
    // so that their x-shifted loads meet in L1
    const int ppr = pieces_per_row<C>(g);
    const int piece = int(blockIdx.x) * (kSplitThreads / 32) + int(threadIdx.x >> 5);
    const int row = piece / ppr;
    // Planes go up in one step and down in the next, and k_step_interface the
    // other way round: the elements written last are read first, while L2
    // (126 MB) still holds them (128x256x128 float16: 174 us a step against 189
    // always upwards; 64x128x64 float32 42 against 46; no change where the
    // buffers are many times L2).
    const int y = 1 + row, zi = (step & 1) ? g.NZ - 3 - int(blockIdx.y) : int(blockIdx.y), z = 1 + zi;
    const float *psi = s_arg.psi[step & 1];
    const bool small = gridDim.x * gridDim.y <= kSmallLaunch;
    if (!small) allow_next_launch();
    touch_params(s_arg);
    wait_for_previous_launch(codec, psi);
    if (small) allow_next_launch();
    if (y > g.NY - 2) return;
    const int w = piece - row * ppr;
    const int x = w * 32 + int(threadIdx.x & 31);
    const bool xin = x >= 1 && x <= g.NX - 2;
    const bool xst = x < store_columns<C>(g);
    const int xn = min(max(x, 1), g.NX - 2);  // a column that is only stored repeats its interior neighbour
    const NodeMoments m = [&] {
        NodeMoments v = pull_moments<C, kPeriodic>(g, codec, xn, y, z);
        opaque(v);
        return v;
    }();
    const float ps = psi_of(m.rr, m.rb);
    if (xin) {
        const_cast<float *>(psi)[uint32_t(x) + uint32_t(g.sy) * uint32_t(y) + uint32_t(g.sz) * uint32_t(z)] = ps;
        tile_record_moments(s, x, y, z, m, ps);
    }
    if constexpr (kStats) radial_accumulate_warp(s, x, y, z, xin, m.ux, m.uy, m.uz);
    const unsigned interface = __ballot_sync(kFull, xin && !is_bulk(m.rr, m.rb));
    if ((x & 31) == 0) s.piece_flags[(size_t(zi) * (g.NY - 2) + row) * ppr + w] = piece_flag(g, w, interface);
    const size_t at = pop_row(g, y, z);
    if (interface & (relax_by_quarters<C>() ? 0xffu << (x & 24) : kFull)) {
        if (xin) park_moments(codec.wr + at + x, g.px, m);
    } else if (xst) {
        collide_node<true>(g, s.ph, codec, at, x, y, z, m, [](int, int, int) { return 0.0f; });
    }
}

// psi of the neighbours of interior node (x, y, z); a periodic box wraps.
template <bool kPeriodic>
struct PsiAround {
    const float *psi;
    int xs[3], ys[3], zs[3];
    __device__ __forceinline__ PsiAround(const Geometry &g, const float *p, int x, int y, int z)
        : psi(p),
          xs{kPeriodic ? wrap_interior(x - 1, g.NX) : x - 1, x, kPeriodic ? wrap_interior(x + 1, g.NX) : x + 1},
          ys{g.sy * (kPeriodic ? wrap_interior(y - 1, g.NY) : y - 1), g.sy * y,
             g.sy * (kPeriodic ? wrap_interior(y + 1, g.NY) : y + 1)},
          zs{g.sz * (kPeriodic ? wrap_interior(z - 1, g.NZ) : z - 1), g.sz * z,
             g.sz * (kPeriodic ? wrap_interior(z + 1, g.NZ) : z + 1)} {}
    __device__ __forceinline__ float operator()(int cx, int cy, int cz) const {
        return psi[xs[cx + 1] + ys[cy + 1] + zs[cz + 1]];
    }
};

// The same read at once, for use after other loads have been waited for.
struct PsiNear {
    float v[27];
    template <bool kPeriodic>
    __device__ __forceinline__ explicit PsiNear(const PsiAround<kPeriodic> &around) {
#pragma unroll
        for (int k = 0; k < 27; ++k) v[k] = k == 13 ? 0.0f : around(k % 3 - 1, k / 3 % 3 - 1, k / 9 - 1);
    }
    __device__ __forceinline__ float operator()(int cx, int cy, int cz) const {
        return v[cx + 1 + 3 * (cy + 1) + 9 * (cz + 1)];
    }
};

// One piece of k_step_interface, or four quarters, one per 8 lanes: moments from
// where k_step_pull parked them, psi of the neighbours, relaxation and stores.
// Float16 reads psi together with the moments, one latency instead of two: with
// an interface at every node 128x256x128 takes 316 us a step against 325,
// 256^3 1256 against 1302, jets of little interface the same.  In float32 the 26
// words spill (373 against 357).
template <class C, bool kPeriodic>
__device__ __forceinline__ void relax_parked(const DeviceState &s, const C &codec, const float *psi, bool on, int x,
                                               int y, int z) {
    const Geometry &g = s.g;
    const bool xst = on && x < store_columns<C>(g);
    const int xn = min(max(x, 1), g.NX - 2);
    const size_t at = pop_row(g, y, z);
    NodeMoments m{};
    if (xst) unpark_moments(codec.wr + at + xn, g.px, m);
    const PsiAround<kPeriodic> around(g, psi, xn, y, z);
    const std::conditional_t<std::is_same<C, CodecF16>::value, PsiNear, const PsiAround<kPeriodic> &> psi_at(around);
    __syncwarp();  // every lane has its moments before one of them stores over them
    if (xst) collide_node<false>(g, s.ph, codec, at, x, y, z, m, psi_at);
}

// The same for the piece that a warp of a small grid has to itself, which is bound
// by latency: moments and psi are read while the flag is on the way, one round
// trip to L2 in the place of three and no list (16x24x16 jet 5.5 us a step
// against 6.4 with the list, 24x40x24 6.5 against 6.9).
template <class C, bool kPeriodic>
__device__ __forceinline__ void relax_flagged(const DeviceState &s, const C &codec, const float *psi,
                                              const uint8_t *flag, int x, int y, int z) {
    const Geometry &g = s.g;
    const int xn = min(max(x, 1), g.NX - 2);
    const size_t at = pop_row(g, y, z);
    const unsigned f = *flag;
    NodeMoments m;
    unpark_moments(codec.wr + at + xn, g.px, m);
    const PsiNear psi_at(PsiAround<kPeriodic>(g, psi, xn, y, z));
    __syncwarp();  // every lane has its moments before one of them stores over them
    const bool on = relax_by_quarters<C>() ? (f >> (4 + (x >> 3 & 3))) & 1u : f & 1u;
    if (on && x < store_columns<C>(g)) collide_node<false>(g, s.ph, codec, at, x, y, z, m, psi_at);
}

// Blocks [0, T.interface_ctas) relax what is flagged; each looks at every
// interface_ctas-th group of neighbouring pieces, so that the pieces of one
// interface, which lie together, go to different SMs, and its warps share what
// it finds.  Where every piece has a warp of its own, each warp takes its piece
// (relax_flagged).  The blocks after them write the jet's inlet and outlet columns from
// the fluid-plane moments in bmom.
template <class C, bool kPeriodic, int kPX>
__global__ void __launch_bounds__(kInterfaceThreads, kInterfaceBlocks) k_step_interface(const DeviceState s_arg,
                                                                                       const FusedTiling T, int cur,
                                                                                       int64_t step) {
    constexpr bool kQuarters = relax_by_quarters<C>();
    __shared__ uint32_t list[(kQuarters ? 4 : 1) * kInterfaceThreads];  // pieces, or 4 * piece + quarter
    __shared__ int found;
    const DeviceState s = pitch_state<C, kPX>(s_arg);
    const Geometry &g = s.g;
    C codec = pitch_codec<C, kPX>(s_arg, cur);
    const float *psi = s_arg.psi[step & 1];
    const int lane = int(threadIdx.x & 31), warp = int(threadIdx.x >> 5);
    const uint32_t ctas = uint32_t(T.interface_ctas), ppr = uint32_t(pieces_per_row<C>(g));
    const uint32_t pieces = ppr * uint32_t(g.NY - 2) * uint32_t(g.NZ - 2);
    allow_next_launch();
    touch_params(s_arg);
    const uint32_t own = blockIdx.x * (kInterfaceThreads / 32) + uint32_t(warp);
    const uint32_t own_row = own / ppr, own_zi = own_row / uint32_t(g.NY - 2);
    wait_for_previous_launch(codec, psi);
    if (blockIdx.x < ctas && pieces <= ctas * (kInterfaceThreads / 32)) {
        if (own < pieces)
            relax_flagged<C, kPeriodic>(s, codec, psi, s.piece_flags + own, int(own - own_row * ppr) * 32 + lane,
                                        1 + int(own_row - own_zi * uint32_t(g.NY - 2)), 1 + int(own_zi));
        return;
    }
    if (blockIdx.x < ctas) {
        for (uint32_t first = 0; first < pieces; first += ctas * kInterfaceThreads) {
            if (threadIdx.x == 0) found = 0;
            __syncthreads();
            const uint64_t at = (uint64_t(threadIdx.x / kPieceGroup) * ctas + blockIdx.x) * kPieceGroup +
                                threadIdx.x % kPieceGroup + first;
            // against the planes' order of k_step_pull (see there)
            const uint32_t mine = (step & 1) ? uint32_t(at) : pieces - 1 - uint32_t(at);
            const unsigned flag = at < pieces ? unsigned(s.piece_flags[mine]) : 0u;
            if (flag) {
                unsigned quarters = kQuarters ? flag >> 4 : 1u;
                int k = atomicAdd(&found, __popc(quarters));
                for (; quarters; quarters &= quarters - 1)
                    list[k++] = kQuarters ? 4 * mine + uint32_t(__ffs(int(quarters)) - 1) : mine;
            }
            __syncthreads();
            constexpr int kTake = kQuarters ? 4 : 1;  // entries a warp takes together
            for (int i = kTake * warp; i < found; i += kTake * (kInterfaceThreads / 32)) {
                const int k = kQuarters ? i + (lane >> 3) : i;
                const uint32_t entry = list[k < found ? k : i], piece = kQuarters ? entry >> 2 : entry, row = piece / ppr;
                const uint32_t zi = row / uint32_t(g.NY - 2);
                const int column = kQuarters ? int(entry & 3) * 8 + (lane & 7) : lane;
                relax_parked<C, kPeriodic>(s, codec, psi, k < found, int(piece - row * ppr) * 32 + column,
                                           1 + int(row - zi * uint32_t(g.NY - 2)), 1 + int(zi));
                __syncwarp();
            }
            __syncthreads();
        }
    } else if constexpr (!kPeriodic) {
        const uint32_t nx = uint32_t(g.NX - 2), columns = nx * uint32_t(g.NZ - 2);
        for (uint32_t i = (blockIdx.x - ctas) * kInterfaceThreads + threadIdx.x; i < 2 * columns;
             i += (gridDim.x - ctas) * kInterfaceThreads) {
            const int side = i >= columns ? 1 : 0;
            const uint32_t c = i - (side ? columns : 0u);
            const int z = 1 + int(c / nx), x = 1 + int(c % nx);
            const NodeMoments m =
                load_moments(s.bmom + (size_t(side) * g.NZ + z) * kMomCount * g.NX, size_t(g.NX), size_t(x));
            if (side == 0)
                inlet_column<C>(s, T.bnd_dst, T.bnd_psi, x, z, int64_t(T.bnd_step), m);
            else
                outlet_column<C>(s, T.bnd_dst, T.bnd_psi, x, z, m);
        }
    }
}

// ------------------------------------------------------------------ granular sequence

// launch_Macros and launch_collistream as the reference drives them, by the
// pieces of the split step: moments and psi of every interior node to HBM
// (planes first .. first + planes - 1;
// 216 or 108 B read, 48 written a node), and the relaxation from there (48 B
// read, 216 or 108 written, whole sectors).  A step of the five launchers of the
// 64x128x64 jet takes 56 us (86 with kernels of runtime pitch that stored the
// rows in part, each launch after the end of the one before).
template <class C, bool kPeriodic, int kPX>
__global__ void __launch_bounds__(kSplitThreads, kSplitBlocks) k_moments(const DeviceState s_arg, int cur, int64_t step,
                                                                           int first, int planes) {
    const DeviceState s = pitch_state<C, kPX>(s_arg);
    const Geometry &g = s.g;
    C codec = pitch_codec<C, kPX>(s_arg, cur);
    const int ppr = pieces_per_row<C>(g);
    const int piece = int(blockIdx.x) * (kSplitThreads / 32) + int(threadIdx.x >> 5);
    const int row = piece / ppr, y = 1 + row;
    const int z = first + ((step & 1) ? planes - 1 - int(blockIdx.y) : int(blockIdx.y));
    const int x = (piece - row * ppr) * 32 + int(threadIdx.x & 31);
    const float *psi_at = s_arg.psi[step & 1];
    allow_next_launch();
    wait_for_previous_launch(codec, psi_at);
    if (y > g.NY - 2 || x < 1 || x > g.NX - 2) return;
    const uint32_t id = uint32_t(x) + uint32_t(g.sy) * uint32_t(y) + uint32_t(g.sz) * uint32_t(z);
    const NodeMoments m = pull_moments<C, kPeriodic>(g, codec, x, y, z);
    const float v[kMomCount] = {m.rr, m.rb, m.ux, m.uy, m.uz, m.pxx, m.pxy, m.pyy, m.pyz, m.pzz, m.pxz};
#pragma unroll
    for (int k = 0; k < kMomCount; ++k) s.mom[size_t(k) * g.N + id] = v[k];
    const float ps = psi_of(m.rr, m.rb);
    float *psi = const_cast<float *>(psi_at);
    psi[id] = ps;
    if constexpr (kPeriodic) {
        // ghost mirrors so the unwrapped gradient stencil sees a periodic field
        const int xs[2] = {x, x == 1 ? g.NX - 1 : (x == g.NX - 2 ? 0 : -1)};
        const int ys[2] = {y, y == 1 ? g.NY - 1 : (y == g.NY - 2 ? 0 : -1)};
        const int zs[2] = {z, z == 1 ? g.NZ - 1 : (z == g.NZ - 2 ? 0 : -1)};
#pragma unroll
        for (int k = 1; k < 8; ++k) {
            const int xx = xs[k & 1], yy = ys[(k >> 1) & 1], zz = zs[(k >> 2) & 1];
            if (xx >= 0 && yy >= 0 && zz >= 0)
                psi[uint32_t(xx) + uint32_t(g.sy) * uint32_t(yy) + uint32_t(g.sz) * uint32_t(zz)] = ps;
        }
    }
}

template <class C, int kPX>
__global__ void __launch_bounds__(kInterfaceThreads, kInterfaceBlocks) k_collide(const DeviceState s_arg, int cur,
                                                                                int64_t step) {
    const DeviceState s = pitch_state<C, kPX>(s_arg);
    const Geometry &g = s.g;
    C codec = pitch_codec<C, kPX>(s_arg, cur);
    const int ppr = pieces_per_row<C>(g);
    const int piece = int(blockIdx.x) * (kInterfaceThreads / 32) + int(threadIdx.x >> 5);
    const int row = piece / ppr, y = 1 + row;
    const int zi = (step & 1) ? int(blockIdx.y) : g.NZ - 3 - int(blockIdx.y), z = 1 + zi;  // against k_moments
    const int x = (piece - row * ppr) * 32 + int(threadIdx.x & 31);
    const float *psi = s_arg.psi[step & 1];
    allow_next_launch();
    wait_for_previous_launch(codec, psi);
    if (y > g.NY - 2 || x >= store_columns<C>(g)) return;
    const int xn = min(max(x, 1), g.NX - 2);
    const uint32_t id = uint32_t(xn) + uint32_t(g.sy) * uint32_t(y) + uint32_t(g.sz) * uint32_t(z);
    float v[kMomCount];
#pragma unroll
    for (int k = 0; k < kMomCount; ++k) v[k] = s.mom[size_t(k) * g.N + id];
    const NodeMoments m{v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7], v[8], v[9], v[10]};
    auto psi_at = [&](int cx, int cy, int cz) { return psi[int(id) + cx + g.sy * cy + g.sz * cz]; };
    collide_node<false>(g, s.ph, codec, pop_row(g, y, z), x, y, z, m, psi_at);
}

// ------------------------------------------------------------------ bulk-staged pipelined fused step

// One-dimensional bulk copies (cp.async.bulk, no multicast) into shared
// memory, completed on an mbarrier; one GPU, the CTA's own shared memory.
__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void bulk_copy_g2s(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}
// Waits for the phase of parity `parity` of `bar` to complete: at most
// `limit` tries, each suspending the thread for about a microsecond at most.
// Returns false when the limit ran out (limit 0: at once).
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, uint32_t limit) {
    for (uint32_t i = 0; i < limit; ++i) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(smem_u32(bar)), "r"(parity), "r"(1000u)
            : "memory");
        if (done) return true;
    }
    return false;
}
// Barrier of the `count` threads of one row group (named barrier `id` > 0);
// returns the OR of `pred` over them.
__device__ __forceinline__ bool group_barrier_or(int id, int count, bool pred) {
    uint32_t out;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "bar.red.or.pred q, %2, %3, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(out)
        : "r"(uint32_t(pred)), "r"(id), "r"(count)
        : "memory");
    return out != 0;
}

// Row image of a staged pull: the 9 (cy, cz) source segments of row (y, z)
// (3 slots x NX elements each, group g = dir_group at g*3*NX), copied
// verbatim from the population buffer.  Direction I of node x reads slot
// (g, cx+1) at column x - cx, with the lateral wrap of PullMap: columns 1
// and NX-2 wrap for cx = +1 / -1, except in a segment that comes from a y
// ghost plane (the boundary's unwrapped slots).
template <class C, int kNX>
struct StagedRow {
    const typename C::Elem *img;
    int x;
    int wxp, wxm;
    bool gy_p, gy_m;
    __device__ __forceinline__ StagedRow(const typename C::Elem *img_, int x_, int y, const Geometry &g, bool periodic)
        : img(img_), x(x_) {
        wxp = (x == 1) ? (kNX - 2) : 0;
        wxm = (x == kNX - 2) ? -(kNX - 2) : 0;
        gy_p = !periodic && y == 1;
        gy_m = !periodic && y == g.NY - 2;
    }
    template <int I>
    __device__ __forceinline__ typename C::Raw load() const {
        using D = Dir<I>;
        int xc = 0;
        if constexpr (D::cx == 1) xc = wxp;
        if constexpr (D::cx == -1) xc = wxm;
        if constexpr (D::cy == 1) xc = gy_p ? 0 : xc;
        if constexpr (D::cy == -1) xc = gy_m ? 0 : xc;
        return img[(dir_group(I) * C::kGroupSlots + D::cx + 1) * kNX + x - D::cx + xc];
    }
};

// Issues the 9 segment copies of pulled row (y, z) (own coordinates, wrapped
// for the periodic box) into `img`, completing on `bar`.
template <class C, int kNX>
__device__ __forceinline__ void stage_row(const Geometry &g, const C &codec, bool periodic, int y, int z,
                                          typename C::Elem *img, uint64_t *bar) {
    constexpr uint32_t seg = uint32_t(C::kGroupSlots * kNX * sizeof(typename C::Elem));
    mbar_expect_tx(bar, 9 * seg);
    for (int grp = 0; grp < 9; ++grp) {
        const int cy = grp / 3 - 1, cz = grp % 3 - 1;
        int ys = y - cy, zs = z - cz;
        const bool ghost = !periodic && (ys == 0 || ys == g.NY - 1);
        if (!ghost) {
            zs = wrap_interior(zs, g.NZ);
            if (periodic) ys = wrap_interior(ys, g.NY);
        }
        const typename C::Elem *src =
            codec.rd + ((size_t(zs) * g.NY + ys) * kQ + size_t(grp) * C::kGroupSlots) * kNX;
        bulk_copy_g2s(img + grp * C::kGroupSlots * kNX, src, seg, bar);
    }
}

// The pipelined march of k_fused_pipe with each pulled row staged: the 9
// source segments of a row (3 KB each in float32 at 128 columns) arrive in
// shared memory by bulk copies while the row group (the 128 threads of one
// row, 4 warps) finishes its previous row and relaxes another.  Each row
// group owns one row image and one mbarrier; after its threads have read the
// image into registers (a barrier of the group), its first thread issues the
// copies of the group's next pulled row.  Pulls therefore hold no global
// loads in registers.  Ghost rows and planes are not pulled (psi from HBM).
// The pulled words, their order and the arithmetic are those of
// k_fused_pipe, so the results are bit-identical.
// Every wait has an iteration limit (T.wait_limit tries of about 1 us): when
// it runs out, the group sets flag[1], issues nothing more and finishes the
// march on whatever its image holds; before it exits, the group's first
// thread waits (again bounded) for the copies it has in flight.
constexpr int kBulkBarBytes = 128;  // mbarriers at the start of the shared memory
template <class C>
constexpr int bulk_image_bytes() { return kQ * kFusedNX * int(sizeof(typename C::Elem)); }

template <class C, bool kStats, bool kPeriodic>
__global__ void __launch_bounds__(kFusedThreads, 2) k_fused_bulk(const DeviceState s_arg, const FusedTiling T,
                                                                 int cur, int64_t step) {
    constexpr int kNX = kFusedNX;
    constexpr int tpr = kNX;
    constexpr int rpt = kFusedThreads / tpr;  // row groups
    using E = typename C::Elem;
    extern __shared__ __align__(128) unsigned char smb[];
    const DeviceState s = fused_state<C, kNX>(s_arg);
    const Geometry &g = s.g;
    const int grp = threadIdx.x / tpr;
    const int x = threadIdx.x - grp * tpr;
    const bool leader = x == 0;
    const int pstride = (T.ty + 2) * tpr;
    const int mplane = T.ty * kMomCount * tpr;
    uint64_t *bar = reinterpret_cast<uint64_t *>(smb) + grp;
    E *img = reinterpret_cast<E *>(smb + kBulkBarBytes) + grp * (kQ * kNX);
    float *ring = reinterpret_cast<float *>(smb + kBulkBarBytes + rpt * bulk_image_bytes<C>());  // [4][ty+2][tpr]
    float *msm = ring + kPipeRing * pstride;                                                    // [3][ty][11][tpr]
    const C codec = fused_codec<C, kNX>(s_arg, cur);
    const float *__restrict__ psi_g = s_arg.psi[step & 1];
    const bool xin = x >= 1 && x <= kNX - 2;
    const int y0 = tile_y0(T);
    const int z0 = 1 + int(blockIdx.y) * T.lz;
    const int lz = min(T.lz, g.NZ - 1 - z0);
    const bool down = T.alternate && (blockIdx.y & 1);
    const int ty = min(T.ty, g.NY - 1 - y0);
    auto plane = [&](int k) { return down ? z0 + lz - k : z0 - 1 + k; };
    // a row of the march that is pulled (the periodic box pulls every row,
    // ghost rows as their wrapped interior rows)
    auto pulled = [&](int k, int r) {
        if constexpr (kPeriodic) return true;
        const int y = y0 - 1 + r, z = plane(k);
        return y >= 1 && y <= g.NY - 2 && z >= 1 && z <= g.NZ - 2;
    };
    // the group's next pulled row after (k, r); k > lz+1 when there is none
    auto next_pull = [&](int &k, int &r) {
        do {
            r += rpt;
            if (r >= ty + 2) {
                r = grp;
                ++k;
            }
        } while (k <= lz + 1 && !pulled(k, r));
    };
    auto issue = [&](int k, int r) {
        int y = y0 - 1 + r, z = plane(k);
        if constexpr (kPeriodic) {
            y = wrap_interior(y, g.NY);
            z = wrap_interior(z, g.NZ);
        }
        stage_row<C, kNX>(g, codec, kPeriodic, y, z, img, bar);
    };
    if (threadIdx.x == 0) {
        for (int k = 0; k < rpt; ++k) mbar_init(reinterpret_cast<uint64_t *>(smb) + k, 1);
        mbar_fence_init();
    }
    __syncthreads();
    const uint32_t limit = uint32_t(T.wait_limit);
    bool failed = false;    // uniform over the row group
    bool in_flight = false; // leader: copies issued and not yet waited for
    uint32_t parity = 0;     // of the next phase this thread waits for
    if (leader && grp < ty + 2) {
        int k = 0, r = grp;
        if (!pulled(k, r)) next_pull(k, r);
        if (k <= lz + 1) {
            issue(k, r);
            in_flight = true;
        }
    }
    for (int k = 0; k <= lz + 2; ++k) {
        const bool do_pull = k <= lz + 1;
        const int c = k - 2;
        const bool do_relax = c >= 1 && c <= lz;
        const int zp = plane(k);
        float *ringp = ring + (k % kPipeRing) * pstride;
        float *msmp = msm + (k % kPipeStage) * mplane;
        const bool own_plane = k >= 1 && k <= lz;
        const int zc = plane(c);
        const float *pm = ring + (((down ? c + 1 : c - 1) + kPipeRing) % kPipeRing) * pstride;
        const float *p0 = ring + ((c + kPipeRing) % kPipeRing) * pstride;
        const float *pp = ring + (((down ? c - 1 : c + 1) + kPipeRing) % kPipeRing) * pstride;
        const float *mc = msm + ((c + kPipeStage) % kPipeStage) * mplane;
        for (int r = grp; r < ty + 2; r += rpt) {
            const bool own = own_plane && r >= 1 && r <= ty;
            const int y = y0 - 1 + r;
            if (do_pull) {
                if (pulled(k, r)) {
                    bool late = false;
                    if (!failed) {
                        late = !mbar_wait(bar, parity, limit);
                        if (!late) {
                            parity ^= 1u;
                            if (leader) in_flight = false;  // the copies have landed
                        }
                    }
                    int xn = x, yn = y, zn = zp;
                    if constexpr (kPeriodic) {
                        xn = wrap_interior(x, kNX);
                        yn = wrap_interior(y, g.NY);
                        zn = wrap_interior(zp, g.NZ);
                    }
                    const bool pull = kPeriodic || xin;
                    RawPull<C> raw;
                    if (pull) {
                        const StagedRow<C, kNX> src(img, xn, yn, g, kPeriodic);
                        static_for<kQ>([&](auto I) {
                            constexpr int i = decltype(I)::value;
                            raw.v[i] = src.template load<i>();
                        });
                    }
                    // every thread of the group has read the image
                    const bool now_failed = group_barrier_or(1 + grp, tpr, late);
                    if (now_failed && !failed) {
                        failed = true;
                        if (leader) atomicExch(s.flag + 1, 1);
                    }
                    if (leader && !failed) {
                        int kn = k, rn = r;
                        next_pull(kn, rn);
                        if (kn <= lz + 1) {
                            issue(kn, rn);
                            in_flight = true;
                        }
                    }
                    NodeMoments m{};
                    float ps = 0.0f;
                    if (pull && own) {  // own is uniform per warp
                        m = moments_from(RawSource<C>{codec, raw});
                        ps = psi_of(m.rr, m.rb);
                    } else if (pull) {
                        float rr, rb;
                        densities_from(RawSource<C>{codec, raw}, rr, rb);
                        ps = psi_of(rr, rb);
                    } else {
                        ps = psi_g[uint32_t(x) + uint32_t(g.sy) * uint32_t(y) + uint32_t(g.sz) * uint32_t(zp)];
                    }
                    ringp[r * tpr + x] = ps;
                    if (own && xin)
                        tile_store_moments<C>(s, x, y, zp, m, ps, msmp + (r - 1) * kMomCount * tpr, tpr);
                    if constexpr (kStats) {
                        if (own) radial_accumulate_warp(s, x, y, zp, pull && xin, m.ux, m.uy, m.uz);
                    }
                } else {
                    ringp[r * tpr + x] =
                        psi_g[uint32_t(x) + uint32_t(g.sy) * uint32_t(y) + uint32_t(g.sz) * uint32_t(zp)];
                }
            }
            const int rc = r + 1;
            if (do_relax && rc <= ty && xin)
                tile_collide(s, codec, x, y0 - 1 + rc, zc, rc, mc + (rc - 1) * kMomCount * tpr, pm, p0, pp, tpr);
        }
        __syncthreads();
    }
    // copies still in flight after a wait ran out land before the CTA exits
    if (leader && in_flight) mbar_wait(bar, parity, limit > 0 ? limit : kBulkDrainLimit);
    fused_boundary<C>(s, T, y0, ty, z0, lz);
}

// Shared memory of k_fused_bulk with `ty`-row tiles: mbarriers, one row image
// per row group, the psi ring and the moment stage of k_fused_pipe.
template <class C>
constexpr int bulk_smem_for(int ty) {
    return kBulkBarBytes + (kFusedThreads / kFusedNX) * bulk_image_bytes<C>() +
           (kPipeRing * (ty + 2) + kPipeStage * kMomCount * ty) * kFusedNX * 4;
}
// rows per tile of k_fused_bulk: float32 2 (3 KB segments, 27 KB images),
// float16 4; both fit two CTAs per SM
template <class C>
constexpr int bulk_rows() { return std::is_same<C, CodecF16>::value ? 4 : 2; }
template <class C>
constexpr int bulk_smem_bytes() { return bulk_smem_for<C>(bulk_rows<C>()); }

}  // namespace

// ------------------------------------------------------------------ launches of one row pitch

// The kernels are instantiated per row pitch (fused.cu, one object per pitch).
template <class C, bool kStats, bool kPeriodic, int kPX>
cudaError_t fused_configure_one(const FusedTiling &t) {
    if constexpr (kPX == kFusedNX) {
        if (t.march == kMarchBulk)
            return cudaFuncSetAttribute(k_fused_bulk<C, kStats, kPeriodic>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        t.smem_bytes);
    }
    if constexpr (kPX == 0 || kPX == kFusedNX || kPX == kFusedNX2) {
        if (t.march == kMarchBlock)
            return cudaFuncSetAttribute(k_fused<C, kStats, kPeriodic, kPX>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        t.smem_bytes);
        if (t.march == kMarchPipe)
            return cudaFuncSetAttribute(k_fused_pipe<C, kStats, kPeriodic, kPX>,
                                        cudaFuncAttributeMaxDynamicSharedMemorySize, t.smem_bytes);
    }
    return cudaSuccess;
}

template <class C, bool kStats, bool kPeriodic, int kPX>
cudaError_t fused_launch_one(const DeviceState &s, const FusedTiling &t, int cur, int64_t step, cudaStream_t st) {
    const dim3 grid(t.ny_tiles, t.nz_chunks), block(t.threads);
    const size_t smem = size_t(t.smem_bytes);
    if constexpr (kPX == kFusedNX) {
        if (t.march == kMarchBulk) {
            k_fused_bulk<C, kStats, kPeriodic><<<grid, block, smem, st>>>(s, t, cur, step);
            return cudaGetLastError();
        }
    }
    if constexpr (kPX == 0 || kPX == kFusedNX || kPX == kFusedNX2) {
        if (t.march == kMarchBlock) {
            k_fused<C, kStats, kPeriodic, kPX><<<grid, block, smem, st>>>(s, t, cur, step);
            return cudaGetLastError();
        }
        if (t.march == kMarchPipe) {
            k_fused_pipe<C, kStats, kPeriodic, kPX><<<grid, block, smem, st>>>(s, t, cur, step);
            return cudaGetLastError();
        }
    }
    const cudaError_t e = launch_overlapped(k_step_pull<C, kStats, kPeriodic, kPX>, grid, block, st, s, cur, step);
    if (e != cudaSuccess) return e;
    return launch_overlapped(k_step_interface<C, kPeriodic, kPX>,
                             dim3(t.interface_ctas + (t.boundary ? t.boundary_ctas : 0)), dim3(kInterfaceThreads), st, s,
                             t, cur, step);
}

template <int kPX>
cudaError_t fused_configure_pitch(const Geometry &g, const FusedTiling &t) {
    cudaError_t e = cudaSuccess;
    auto both = [&](auto codec, auto periodic) {
        using C = decltype(codec);
        constexpr bool kP = decltype(periodic)::value;
        e = fused_configure_one<C, false, kP, kPX>(t);
        if (e == cudaSuccess) e = fused_configure_one<C, true, kP, kPX>(t);
    };
    const bool per = g.boundary == kBoundaryPeriodic;
    if (g.storage == kStoreF16)
        per ? both(CodecF16{}, std::true_type{}) : both(CodecF16{}, std::false_type{});
    else
        per ? both(CodecF32{}, std::true_type{}) : both(CodecF32{}, std::false_type{});
    return e;
}

template <int kPX>
cudaError_t fused_launch_pitch(const DeviceState &s, const FusedTiling &t, int cur, int64_t step, bool stats,
                               cudaStream_t st) {
    auto go = [&](auto codec, auto periodic) {
        using C = decltype(codec);
        constexpr bool kP = decltype(periodic)::value;
        return stats ? fused_launch_one<C, true, kP, kPX>(s, t, cur, step, st)
                     : fused_launch_one<C, false, kP, kPX>(s, t, cur, step, st);
    };
    const bool per = s.g.boundary == kBoundaryPeriodic;
    if (s.g.storage == kStoreF16)
        return per ? go(CodecF16{}, std::true_type{}) : go(CodecF16{}, std::false_type{});
    return per ? go(CodecF32{}, std::true_type{}) : go(CodecF32{}, std::false_type{});
}

template <int kPX>
cudaError_t moments_launch_pitch(const DeviceState &s, int cur, int64_t step, int first, int planes, cudaStream_t st) {
    constexpr int kWarps = kSplitThreads / 32;
    auto go = [&](auto codec) {
        using C = decltype(codec);
        const dim3 grid((pieces_per_row<C>(s.g) * (s.g.NY - 2) + kWarps - 1) / kWarps, planes);
        return s.g.boundary == kBoundaryPeriodic
                   ? launch_overlapped(k_moments<C, true, kPX>, grid, dim3(kSplitThreads), st, s, cur, step, first, planes)
                   : launch_overlapped(k_moments<C, false, kPX>, grid, dim3(kSplitThreads), st, s, cur, step, first, planes);
    };
    return s.g.storage == kStoreF16 ? go(CodecF16{}) : go(CodecF32{});
}

template <int kPX>
cudaError_t collide_launch_pitch(const DeviceState &s, int cur, int64_t step, cudaStream_t st) {
    constexpr int kWarps = kInterfaceThreads / 32;
    auto go = [&](auto codec) {
        using C = decltype(codec);
        const dim3 grid((pieces_per_row<C>(s.g) * (s.g.NY - 2) + kWarps - 1) / kWarps, s.g.NZ - 2);
        return launch_overlapped(k_collide<C, kPX>, grid, dim3(kInterfaceThreads), st, s, cur, step);
    };
    return s.g.storage == kStoreF16 ? go(CodecF16{}) : go(CodecF32{});
}

}  // namespace mcg
