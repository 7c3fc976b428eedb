// kernels.cu - the kernels around the fused step (fused.cuh) on B200 (sm_100a):
// the granular launch sequence of the reference (k_moments, k_collide,
// k_boundary, k_accumulate_radial) for callers that drive the launchers one by
// one, which writes the moment planes to HBM like the reference; initial
// states, state transfer, diagnostics, outputs and the discrete adjoint.
#include "step.cuh"

namespace mcg {
namespace {

// ------------------------------------------------------------------ granular sequence

constexpr int kBX = 32, kBY = 8;
constexpr int kRedThreads = 256;

// Jet boundary of step `step`: blockIdx.z == 0 is the inlet (y=0 plane), 1 the
// outlet (y=NY-1 plane), unless `which` selects one.  Values go to the ghost
// planes of buffer `wbuf` (the one the collision of this step writes) and to
// the psi buffer of the next step.
template <class C>
__global__ void __launch_bounds__(256) k_boundary(const DeviceState s, int wbuf, int64_t step, int which,
                                                  int from_bmom) {
    const Geometry &g = s.g;
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int z = blockIdx.y * blockDim.y + threadIdx.y;
    allow_next_launch();
    wait_for_previous_launch();
    if (x < 1 || x > g.NX - 2 || z < 1 || z > g.NZ - 2) return;
    const int side = which >= 0 ? which : int(blockIdx.z);
    float *psi_next = s.psi[(step + 1) & 1];
    NodeMoments m;
    if (from_bmom) {
        m = load_moments(s.bmom + (size_t(side) * g.NZ + z) * kMomCount * g.NX, size_t(g.NX), size_t(x));
    } else {
        const int yF = side == 0 ? 1 : g.NY - 2;
        m = load_moments(s.mom, size_t(g.N), size_t(x) + size_t(g.sy) * size_t(yF) + size_t(g.sz) * size_t(z));
    }
    if (side == 0) inlet_column<C>(s, s.pops[wbuf], psi_next, x, z, step, m);
    else outlet_column<C>(s, s.pops[wbuf], psi_next, x, z, m);
}

__global__ void __launch_bounds__(kBX * kBY) k_accumulate_radial(const DeviceState s) {
    const Geometry &g = s.g;
    const int x = blockIdx.x * kBX + threadIdx.x;
    const int y = blockIdx.y * kBY + threadIdx.y;
    const int z = blockIdx.z;
    allow_next_launch();
    wait_for_previous_launch();
    const bool active = x >= 1 && x <= g.NX - 2 && y >= 1 && y <= g.NY - 2 && z >= 1 && z <= g.NZ - 2;
    float ux = 0, uy = 0, uz = 0;
    if (active) {
        const uint32_t id = uint32_t(x) + uint32_t(g.sy) * uint32_t(y) + uint32_t(g.sz) * uint32_t(z);
        ux = s.mom[kMomUX * size_t(g.N) + id];
        uy = s.mom[kMomUY * size_t(g.N) + id];
        uz = s.mom[kMomUZ * size_t(g.N) + id];
    }
    radial_accumulate_warp(s, x, y, z, active, ux, uy, uz);
}

// ------------------------------------------------------------------ initial state

// Densities of every node (jet/jetIn.cuh:13-62 or bubble/bubbleIn.cuh:10-22).
__global__ void k_init_fields(const DeviceState s, int mode, int red_inside, float r2, float bx, float by, float bz) {
    const Geometry &g = s.g;
    const Physics &ph = s.ph;
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y * blockDim.y + threadIdx.y;
    const int z = blockIdx.z;
    if (x >= g.NX || y >= g.NY) return;
    const uint32_t id = uint32_t(x) + uint32_t(g.sy) * uint32_t(y) + uint32_t(g.sz) * uint32_t(z);
    float rr, rb;
    if (mode == 0) {
        rr = ph.rhor0;
        rb = 0.0f;
        if (y == 0 && x >= 1 && x <= g.NX - 2 && z >= 1 && z <= g.NZ - 2) {
            const float j = is_jet_column(ph, x, z) ? 1.0f : 0.0f;
            rr = (1.0f - j) * ph.rhor0;
            rb = j * ph.rhob0;
        }
    } else {
        int xx = x, yy = y, zz = z;
        if (g.boundary == kBoundaryPeriodic) {  // ghosts mirror the opposite interior node
            xx = wrap_interior(x, g.NX);
            yy = wrap_interior(y, g.NY);
            zz = wrap_interior(z, g.NZ);
        }
        const float dx = float(xx) - bx, dy = float(yy) - by, dz = float(zz) - bz;
        const float in = ((dx * dx) + (dy * dy) + (dz * dz)) <= r2 ? 1.0f : 0.0f;
        if (red_inside) {
            rr = in * ph.rhor0;
            rb = (1.0f - in) * ph.rhob0;
        } else {
            rr = (1.0f - in) * ph.rhor0;
            rb = in * ph.rhob0;
        }
    }
    const size_t N = g.N;
    s.mom[kMomRR * N + id] = rr;
    s.mom[kMomRB * N + id] = rb;
    for (int k = kMomUX; k < kMomCount; ++k) s.mom[size_t(k) * N + id] = 0.0f;
}

// Populations of every interior node, written at their pull sources.  The
// current buffer takes every slot; the other one only the slots on a y ghost
// plane, which no step rewrites (they must hold the initial value in both
// buffers).  Every other slot of the other buffer is written by the first
// step before anything reads it.  Directions are unrolled, so the pull
// source and the equilibrium take compile-time lattice constants.
// By pieces of 32 columns, the ghost columns of the rows filled with zeros to
// complete their sectors (store_columns): an initial jet of 128x256x128 float32
// takes 226 us in all (384 on 32x8 blocks that left them partly written).
template <class C>
__global__ void __launch_bounds__(kRedThreads) k_init_pops(const DeviceState s, const C codec, int mode, float noise) {
    const Geometry &g = s.g;
    const int ppr = pieces_per_row<C>(g);
    const int piece = int(blockIdx.x) * (kRedThreads / 32) + int(threadIdx.x >> 5);
    const int row = piece / ppr, y = 1 + row, z = 1 + int(blockIdx.y);
    const int x = (piece - row * ppr) * 32 + int(threadIdx.x & 31);
    if (y > g.NY - 2 || x >= store_columns<C>(g)) return;
    const bool node = x >= 1 && x <= g.NX - 2;
    const uint32_t id = uint32_t(x) + uint32_t(g.sy) * uint32_t(y) + uint32_t(g.sz) * uint32_t(z);
    const size_t N = g.N;
    float rr = 0.f, rb = 0.f, ux = 0.f, uy = 0.f, uz = 0.f;
    if (node) {
        rr = s.mom[kMomRR * N + id];
        rb = s.mom[kMomRB * N + id];
        ux = s.mom[kMomUX * N + id];
        uy = s.mom[kMomUY * N + id];
        uz = s.mom[kMomUZ * N + id];
    }
    const float usq = fmaf(uz, uz, fmaf(ux, ux, uy * uy));  // one order of rounding in every build
    const bool periodic = g.boundary == kBoundaryPeriodic;
    const PullMap<C> pm(g, x, y, z, periodic);
    typename C::Elem *const other = const_cast<typename C::Elem *>(codec.rd);  // the other buffer
    static_for<kQ>([&](auto I) {
        constexpr int i = decltype(I)::value;
        using D = Dir<i>;
        const bool ghost = (D::cy == 1 && pm.gy_p) || (D::cy == -1 && pm.gy_m);  // a slot of a y ghost plane
        if (!node && ghost) return;
        float fr, fb;
        if (mode == 3) {
            // per colour, the third-order equilibrium at the node's velocity (lbm.cuh:16-35)
            const float cu = D::fx * ux + D::fy * uy + D::fz * uz;
            const float A2 = (cu * cu) * kInv2Cs4 - usq * kInv2Cs2 + cu * kInvCs2;
            const float A3 = cu * ((cu * cu) * kInv6Cs6 - usq * kInv2Cs4);
            const float e = D::w * (1.0f + A2 + A3);
            fr = e * rr;
            fb = e * rb;
        } else {
            // jetDensity: feq(rho, 0) = w rho; bubble: w rho (jetIn.cuh:26-34, bubbleIn.cuh:25-39)
            fr = D::w * rr;
            fb = D::w * rb;
            if (noise != 0.0f) {
                const float u = hash_uniform(s.ph.seed, 0x1D17ull, id, uint64_t(i));
                const float f = 1.0f + (2.0f * u - 1.0f) * noise;
                fr = fr * f;
                fb = fb * f;
            }
        }
        size_t grow;
        int xs;
        pm.template src<i>(node ? x : x + D::cx, grow, xs);
        const size_t at = grow + size_t(D::cx + 1) * g.px + xs;
        const typename C::Elem v = codec.template pack<i>(fr, fb);
        codec.wr[at] = v;
        if (ghost) other[at] = v;
    });
}

__global__ void k_refresh_psi(const DeviceState s) {
    const Geometry &g = s.g;
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y * blockDim.y + threadIdx.y;
    const int z = blockIdx.z;
    if (x >= g.NX || y >= g.NY) return;
    int xx = x, yy = y, zz = z;
    if (g.boundary == kBoundaryPeriodic) {
        xx = wrap_interior(x, g.NX);
        yy = wrap_interior(y, g.NY);
        zz = wrap_interior(z, g.NZ);
    }
    const uint32_t id = uint32_t(x) + uint32_t(g.sy) * uint32_t(y) + uint32_t(g.sz) * uint32_t(z);
    const uint32_t src = uint32_t(xx) + uint32_t(g.sy) * uint32_t(yy) + uint32_t(g.sz) * uint32_t(zz);
    const size_t N = g.N;
    const float p = psi_of(s.mom[kMomRR * N + src], s.mom[kMomRB * N + src]);
    s.psi[0][id] = p;
    s.psi[1][id] = p;
}

// Host state transfer in z-chunks of the reference layout f[i*Ncells + id].
// A chunk holds planes [z0, z0 + nz) of both colours, staged as
// stage[colour][i][id - z0*NX*NY] with `pitch` elements per direction row, so
// that the host copy of each colour is one 2-D copy of 27 rows.
//
// Scatter: the populations of the chunk's interior nodes go to their pull
// sources in buffer `wbuf` (the sources of planes z0 and z0+nz-1 lie in the
// neighbouring chunks' planes; every source is written by exactly one node).
template <class C>
__global__ void __launch_bounds__(kRedThreads) k_scatter_chunk(const DeviceState s, const C codec,
                                                              const float *__restrict__ stage, size_t pitch, int z0) {
    const Geometry &g = s.g;
    const int ppr = pieces_per_row<C>(g);
    const int piece = int(blockIdx.x) * (kRedThreads / 32) + int(threadIdx.x >> 5);
    const int row = piece / ppr, y = 1 + row, z = z0 + int(blockIdx.y);
    const int x = (piece - row * ppr) * 32 + int(threadIdx.x & 31);
    if (y > g.NY - 2 || z < 1 || z > g.NZ - 2 || x >= store_columns<C>(g)) return;
    const bool node = x >= 1 && x <= g.NX - 2;
    const size_t lid = size_t(x) + size_t(g.sy) * size_t(y) + size_t(g.sz) * size_t(blockIdx.y);
    const float *fr = stage, *fb = stage + size_t(kQ) * pitch;
    const PullMap<C> pm(g, x, y, z, g.boundary == kBoundaryPeriodic);
    static_for<kQ>([&](auto I) {
        constexpr int i = decltype(I)::value;
        using D = Dir<i>;
        if (!node && ((D::cy == 1 && pm.gy_p) || (D::cy == -1 && pm.gy_m))) return;
        float r = 0.f, b = 0.f;
        if (node) {
            r = fr[size_t(i) * pitch + lid];
            b = fb[size_t(i) * pitch + lid];
        }
        size_t grow;
        int xs;
        pm.template src<i>(node ? x : x + D::cx, grow, xs);
        codec.wr[grow + size_t(D::cx + 1) * g.px + xs] = codec.template pack<i>(r, b);
    });
}

// Gather: f(t) = pops[cur] pulled at the chunk's nodes into the stage; ghost
// nodes give 0.
template <class C, bool kPeriodic>
__global__ void __launch_bounds__(kRedThreads) k_gather_chunk(const DeviceState s, const C codec,
                                                             float *__restrict__ stage, size_t pitch, int z0) {
    const Geometry &g = s.g;
    const int ppr = (g.NX + 31) / 32;
    const int piece = int(blockIdx.x) * (kRedThreads / 32) + int(threadIdx.x >> 5);
    const int y = piece / ppr, z = z0 + int(blockIdx.y);
    const int x = (piece - y * ppr) * 32 + int(threadIdx.x & 31);
    if (y >= g.NY || x >= g.NX) return;
    const size_t lid = size_t(x) + size_t(g.sy) * size_t(y) + size_t(g.sz) * size_t(blockIdx.y);
    float *fr = stage, *fb = stage + size_t(kQ) * pitch;
    if (!(x >= 1 && x <= g.NX - 2 && y >= 1 && y <= g.NY - 2 && z >= 1 && z <= g.NZ - 2)) {
        for (int i = 0; i < kQ; ++i) fr[size_t(i) * pitch + lid] = fb[size_t(i) * pitch + lid] = 0.0f;
        return;
    }
    RawPull<C> raw;
    pull_issue<C, kPeriodic>(g, codec, x, y, z, raw);
    static_for<kQ>([&](auto I) {
        constexpr int i = decltype(I)::value;
        float r, b;
        codec.template unpack<i>(raw.v[i], r, b);
        fr[size_t(i) * pitch + lid] = r;
        fb[size_t(i) * pitch + lid] = b;
    });
}

template <class E>
__global__ void k_unpad_rows(const E *__restrict__ src, E *__restrict__ dst, int NX, int px, size_t rows) {
    const size_t warps = size_t(gridDim.x) * (blockDim.x / 32);
    for (size_t r = size_t(blockIdx.x) * (blockDim.x / 32) + threadIdx.x / 32; r < rows; r += warps)
        for (int x = int(threadIdx.x & 31); x < NX; x += 32) dst[r * size_t(NX) + x] = src[r * size_t(px) + x];
}

// ------------------------------------------------------------------ reductions

template <int NT>
__device__ __forceinline__ double block_sum(double v, double *sh) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(kFull, v, o);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) sh[wid] = v;
    __syncthreads();
    double r = 0.0;
    if (threadIdx.x == 0)
        for (int k = 0; k < NT / 32; ++k) r += sh[k];
    return r;
}


// Sum of 0.5|u|^2 over interior nodes (kernels.cu:136-152), float64.
__global__ void __launch_bounds__(kRedThreads) k_tke(const DeviceState s, double *out) {
    __shared__ double sh[kRedThreads / 32];
    const Geometry &g = s.g;
    const size_t N = g.N;
    double acc = 0.0;
    for (size_t id = size_t(blockIdx.x) * blockDim.x + threadIdx.x; id < N; id += size_t(gridDim.x) * blockDim.x) {
        const int x = int(id % g.NX), y = int((id / g.NX) % g.NY), z = int(id / (size_t(g.NX) * g.NY));
        if (x < 1 || x > g.NX - 2 || y < 1 || y > g.NY - 2 || z < 1 || z > g.NZ - 2) continue;
        const float vx = s.mom[kMomUX * N + id], vy = s.mom[kMomUY * N + id], vz = s.mom[kMomUZ * N + id];
        acc += double(0.5f * (vx * vx + vy * vy + vz * vz));
    }
    const double r = block_sum<kRedThreads>(acc, sh);
    if (threadIdx.x == 0) atomicAdd(out, r);
}

// Running mean of uy per interior node (kernels.cu:168-186).
__global__ void k_uy_average(const DeviceState s, uint32_t samples) {
    const Geometry &g = s.g;
    const size_t N = g.N;
    const float c = float(samples);
    for (size_t id = size_t(blockIdx.x) * blockDim.x + threadIdx.x; id < N; id += size_t(gridDim.x) * blockDim.x) {
        const int x = int(id % g.NX), y = int((id / g.NX) % g.NY), z = int(id / (size_t(g.NX) * g.NY));
        if (x < 1 || x > g.NX - 2 || y < 1 || y > g.NY - 2 || z < 1 || z > g.NZ - 2) continue;
        s.uy_avg[id] = (s.uy_avg[id] * c + s.mom[kMomUY * N + id]) / (c + 1.0f);
    }
}

constexpr int kConsBlocksMax = 3 * 148;  // one wave at 3 blocks per SM

// Row pieces of 32 columns over all interior rows, one warp each, for the
// diagnostics that pull every interior node once: no integer division per
// node, and the piece's lanes share the pull maps of the step.
template <class F>
__device__ __forceinline__ void for_row_pieces(const Geometry &g, F &&f) {
    const int per_row = (g.NX + 31) / 32;
    const int pieces = per_row * (g.NY - 2) * (g.NZ - 2);
    const int warps = int(gridDim.x) * (kRedThreads / 32);
    for (int t = int(blockIdx.x) * (kRedThreads / 32) + int(threadIdx.x >> 5); t < pieces; t += warps) {
        const int row = t / per_row;
        const int x = (t - row * per_row) * 32 + int(threadIdx.x & 31);
        const int z = row / (g.NY - 2);
        if (x >= 1 && x <= g.NX - 2) f(x, 1 + row - z * (g.NY - 2), 1 + z);
    }
}

// Pass 1: per-block float64 partial sums of f(t) over interior nodes.
// Bound by the pulls (216 or 108 B a node).  The directions are unrolled, so a
// node's 27 elements are in flight together and the momentum sums add or
// subtract; a loop over the directions with runtime lattice vectors and four
// divisions a node kept its tables in local memory: 10.2 ms a call on
// 128x256x128 float32, 0.165 ms now (5.5 TB/s, the synchronisation included).
template <class C, bool kPeriodic>
__global__ void __launch_bounds__(kRedThreads, 3) k_conservation_partials(const DeviceState s, const C codec,
                                                                          double *partials) {
    __shared__ double sh[kRedThreads / 32];
    const Geometry &g = s.g;
    double acc[5] = {0, 0, 0, 0, 0};
    for_row_pieces(g, [&](int x, int y, int z) {
        RawPull<C> raw;
        pull_issue<C, kPeriodic>(g, codec, x, y, z, raw);
        static_for<kQ>([&](auto I) {
            constexpr int i = decltype(I)::value;
            float r, b;
            codec.template unpack<i>(raw.v[i], r, b);
            const double a = r, c = b, t = a + c;
            acc[0] += a;
            acc[1] += c;
            if constexpr (Dir<i>::cx != 0) acc[2] += Dir<i>::cx > 0 ? t : -t;
            if constexpr (Dir<i>::cy != 0) acc[3] += Dir<i>::cy > 0 ? t : -t;
            if constexpr (Dir<i>::cz != 0) acc[4] += Dir<i>::cz > 0 ? t : -t;
        });
    });
    for (int k = 0; k < 5; ++k) {
        const double r = block_sum<kRedThreads>(acc[k], sh);
        if (threadIdx.x == 0) partials[size_t(k) * gridDim.x + blockIdx.x] = r;
    }
}

// Pass 2: one block folds the partials in a fixed order (deterministic).
__global__ void __launch_bounds__(kRedThreads) k_conservation_final(const double *partials, int nblocks, double *out) {
    __shared__ double sh[kRedThreads / 32];
    for (int k = 0; k < 5; ++k) {
        double acc = 0.0;
        for (int b = threadIdx.x; b < nblocks; b += blockDim.x) acc += partials[size_t(k) * nblocks + b];
        const double r = block_sum<kRedThreads>(acc, sh);
        if (threadIdx.x == 0) out[k] = r;
    }
}

// Whether any moment plane or population of an interior node is not finite;
// the same row pieces and unrolled pulls (10.0 ms -> 0.18 ms on
// 128x256x128 float32).
template <class C, bool kPeriodic>
__global__ void __launch_bounds__(kRedThreads, 3) k_check_finite(const DeviceState s, const C codec, int *flag) {
    const Geometry &g = s.g;
    const size_t N = g.N;
    bool bad = false;
    for_row_pieces(g, [&](int x, int y, int z) {
        RawPull<C> raw;
        pull_issue<C, kPeriodic>(g, codec, x, y, z, raw);
        const uint32_t id = uint32_t(x) + uint32_t(g.sy) * uint32_t(y) + uint32_t(g.sz) * uint32_t(z);
#pragma unroll
        for (int k = 0; k < kMomCount; ++k) bad |= !isfinite(s.mom[size_t(k) * N + id]);
        static_for<kQ>([&](auto I) {
            constexpr int i = decltype(I)::value;
            float r, b;
            codec.template unpack<i>(raw.v[i], r, b);
            bad |= !isfinite(r) || !isfinite(b);
        });
    });
    if (__any_sync(kFull, bad) && (threadIdx.x & 31) == 0) atomicOr(flag, 1);
}

dim3 grid3(const Geometry &g) { return dim3((g.NX + kBX - 1) / kBX, (g.NY + kBY - 1) / kBY, g.NZ); }
dim3 grid_plane(const Geometry &g) { return dim3((g.NX + 31) / 32, (g.NZ + 7) / 8, 1); }
unsigned grid1(const Geometry &g) {
    const size_t want = (size_t(g.N) + kRedThreads - 1) / kRedThreads;
    return unsigned(want < size_t(8 * 148) ? want : size_t(8 * 148));
}


template <class C>
cudaError_t boundary_dispatch(const DeviceState &s, int wbuf, int64_t step, int which, bool from_bmom,
                              cudaStream_t st) {
    dim3 grid = grid_plane(s.g);
    grid.z = which >= 0 ? 1 : 2;
    return launch_overlapped(k_boundary<C>, grid, dim3(32, 8), st, s, wbuf, step, which, from_bmom ? 1 : 0);
}

// ------------------------------------------------------------------ discrete adjoint

// Adjoint of one step of the periodic box, float32 populations.  The forward
// step maps the stored post-collision values S_t to S_{t+1}:
//   f_i(x) = S_t,i(x - c_i); M(x) = moments(f(x)); psi(x) = psi(M(x));
//   F(x) = (1/cs2) sum_j w_j c_j psi(x + c_j);  S_{t+1},i(x) = C_i(M(x), F(x)).
// Given lambda_{t+1} = dJ/dS_{t+1} the adjoint forms lambda_t = dJ/dS_t in two
// node-parallel parts: adj_collide_node takes C's Jacobian (moments and F of the
// node), adj_moments_node gathers the F-adjoints of the neighbours into the
// node's psi-adjoint, goes back through the moments and scatters along the
// transposed streaming.  The bulk/interface switch (I <= 1e-4) and the
// |F| <= 1e-4 cut-off are taken as in the forward step (derivatives inside
// the branch the forward state selects).
//
// Every pass reads the state S_t only through its moment record M: the 11
// moment planes of the pulled populations and psi (plane kTapePsi), interior
// nodes; neighbours are addressed with the periodic wrap.

__device__ __forceinline__ double block_sum_any(double v, double *sh, int nthreads) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(kFull, v, o);
    const int t = threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z);
    const int lane = t & 31, wid = t >> 5;
    __syncthreads();
    if (lane == 0) sh[wid] = v;
    __syncthreads();
    double r = 0.0;
    if (t == 0)
        for (int k = 0; k < nthreads / 32; ++k) r += sh[k];
    __syncthreads();
    return r;
}

// block_sum_any of three values in one pass: two barriers instead of nine.
// Each value is summed in the same order as block_sum_any sums it.  sh holds
// 3 * (threads / 32) doubles; the sums are valid in thread 0.
__device__ __forceinline__ void block_sum3(double (&v)[3], double *sh, int nthreads) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
        for (int k = 0; k < 3; ++k) v[k] += __shfl_down_sync(kFull, v[k], o);
    }
    const int t = threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z);
    const int lane = t & 31, wid = t >> 5, nw = nthreads / 32;
    __syncthreads();
    if (lane == 0)
        for (int k = 0; k < 3; ++k) sh[k * nw + wid] = v[k];
    __syncthreads();
    if (t == 0) {
        for (int k = 0; k < 3; ++k) {
            double r = 0.0;
            for (int j = 0; j < nw; ++j) r += sh[k * nw + j];
            v[k] = r;
        }
    }
}

// J = sum over interior nodes of (psi_T - psi*)^2 and lambda_T = dJ/dS_T.
__global__ void __launch_bounds__(kBX * kBY) k_adj_terminal(const DeviceState s, const float *__restrict__ M,
                                                           const float *__restrict__ target, float *lam, double *J) {
    __shared__ double sh[kBX * kBY / 32];
    const Geometry &g = s.g;
    const int x = blockIdx.x * kBX + threadIdx.x;
    const int y = blockIdx.y * kBY + threadIdx.y;
    const int z = blockIdx.z;
    const bool in = x >= 1 && x <= g.NX - 2 && y >= 1 && y <= g.NY - 2 && z >= 1 && z <= g.NZ - 2;
    double jloc = 0.0;
    if (in) {
        const uint32_t id = uint32_t(x) + uint32_t(g.sy) * uint32_t(y) + uint32_t(g.sz) * uint32_t(z);
        const size_t N = g.N;
        const float rr = M[kMomRR * N + id], rb = M[kMomRB * N + id];
        const float rho = rr + rb;
        const float d = M[kTapePsi * N + id] - target[id];
        jloc = double(d) * double(d);
        const float lpsi = 2.0f * d;
        const float inv2 = 1.0f / (rho * rho);
        const float lrr = lpsi * 2.0f * rb * inv2, lrb = -lpsi * 2.0f * rr * inv2;
        const PullMap<CodecF32> pm(g, x, y, z, true);
        static_for<kQ>([&](auto I) {
            constexpr int i = decltype(I)::value;
            size_t grow;
            int xs;
            pm.template src<i>(x, grow, xs);
            reinterpret_cast<float2 *>(lam)[grow + size_t(dir_cx(i) + 1) * g.px + xs] = make_float2(lrr, lrb);
        });
    }
    const double r = block_sum_any(jloc, sh, kBX * kBY);
    if (threadIdx.x == 0 && threadIdx.y == 0) atomicAdd(J, r);
}

// Exponents (a, b, c) of the 17 monomials cx^a cy^b cz^c of the collision
// polynomial (collision_poly): per-axis degree <= 2, total degree <= 3.
__host__ __device__ constexpr int poly_exp(int k, int axis) {
    constexpr int e[17][3] = {{0, 0, 0}, {1, 0, 0}, {0, 1, 0}, {0, 0, 1}, {2, 0, 0}, {0, 2, 0},
                              {0, 0, 2}, {1, 1, 0}, {1, 0, 1}, {0, 1, 1}, {2, 1, 0}, {2, 0, 1},
                              {1, 2, 0}, {1, 0, 2}, {0, 2, 1}, {0, 1, 2}, {1, 1, 1}};
    return e[k][axis];
}
__host__ __device__ constexpr int ipow1(int c, int e) { return e == 0 ? 1 : (e == 1 ? c : c * c); }
enum PolyTerm { kT000, kT100, kT010, kT001, kT200, kT020, kT002, kT110, kT101, kT011,
                kT210, kT201, kT120, kT102, kT021, kT012, kT111 };

// Adjoint of the bulk value g_i = w_i P(c_i) over the collision polynomial's
// coefficients, from the moments T_k = sum_i v_i m_k(c_i) of per-direction
// weights v (v = w lambda_g): Phi = (feq polynomial)/rho dotted with T, its
// u-gradient, and Psi = (fneq polynomial) dotted with T, with the S2 / S3
// Hermite sums Psi is made of.
struct PolyAdjoint {
    float S2[6], S3[7];
    float Phi, dPhi[3], Psi;
};
__device__ __forceinline__ PolyAdjoint poly_adjoint(const float (&T)[17], float ux, float uy, float uz,
                                                    const NeqTerms &n) {
    PolyAdjoint r;
    r.S2[0] = T[kT200] - kCs2 * T[kT000];
    r.S2[1] = T[kT110];
    r.S2[2] = T[kT020] - kCs2 * T[kT000];
    r.S2[3] = T[kT011];
    r.S2[4] = T[kT002] - kCs2 * T[kT000];
    r.S2[5] = T[kT101];
    r.S3[0] = T[kT210] - kCs2 * T[kT010];
    r.S3[1] = T[kT201] - kCs2 * T[kT001];
    r.S3[2] = T[kT120] - kCs2 * T[kT100];
    r.S3[3] = T[kT102] - kCs2 * T[kT100];
    r.S3[4] = T[kT021] - kCs2 * T[kT001];
    r.S3[5] = T[kT012] - kCs2 * T[kT010];
    r.S3[6] = T[kT111];
    r.Psi = kInv2Cs4 * (n.pxx * r.S2[0] + 2.0f * n.pxy * r.S2[1] + n.pyy * r.S2[2] + 2.0f * n.pyz * r.S2[3] +
                        n.pzz * r.S2[4] + 2.0f * n.pxz * r.S2[5]) +
            kInv2Cs6 * (n.a3xxy * r.S3[0] + n.a3xxz * r.S3[1] + n.a3xyy * r.S3[2] + n.a3xzz * r.S3[3] +
                        n.a3yyz * r.S3[4] + n.a3yzz * r.S3[5] + 2.0f * n.a3xyz * r.S3[6]);
    // feq_i / (w_i rho) = 1 + q cu + (q^2/2) cu^2 - (q/2) |u|^2 + (q^3/6) cu^3 - (q^2/2) |u|^2 cu, q = 1/cs^2
    const float usq = ux * ux + uy * uy + uz * uz;
    const float uTc = ux * T[kT100] + uy * T[kT010] + uz * T[kT001];
    const float lin = kInvCs2 - kInv2Cs4 * usq;
    const float t2x = T[kT200] * ux + T[kT110] * uy + T[kT101] * uz;
    const float t2y = T[kT110] * ux + T[kT020] * uy + T[kT011] * uz;
    const float t2z = T[kT101] * ux + T[kT011] * uy + T[kT002] * uz;
    // (1/3) d(cu^3)/du_a summed against T (c^3 = c on the lattice)
    const float cx3 = ux * ux * T[kT100] + 2.0f * ux * uy * T[kT210] + 2.0f * ux * uz * T[kT201] + uy * uy * T[kT120] +
                      uz * uz * T[kT102] + 2.0f * uy * uz * T[kT111];
    const float cy3 = uy * uy * T[kT010] + 2.0f * uy * ux * T[kT120] + 2.0f * uy * uz * T[kT021] + ux * ux * T[kT210] +
                      uz * uz * T[kT012] + 2.0f * ux * uz * T[kT111];
    const float cz3 = uz * uz * T[kT001] + 2.0f * uz * ux * T[kT102] + 2.0f * uz * uy * T[kT012] + ux * ux * T[kT201] +
                      uy * uy * T[kT021] + 2.0f * ux * uy * T[kT111];
    r.Phi = T[kT000] * (1.0f - kInv2Cs2 * usq) + lin * uTc + kInv2Cs4 * (ux * t2x + uy * t2y + uz * t2z) +
            kInv6Cs6 * (ux * cx3 + uy * cy3 + uz * cz3);
    const float q2 = 2.0f * kInv2Cs4, q3h = 3.0f * kInv6Cs6;
    r.dPhi[0] = -kInvCs2 * ux * T[kT000] - q2 * ux * uTc + lin * T[kT100] + q2 * t2x + q3h * cx3;
    r.dPhi[1] = -kInvCs2 * uy * T[kT000] - q2 * uy * uTc + lin * T[kT010] + q2 * t2y + q3h * cy3;
    r.dPhi[2] = -kInvCs2 * uz * T[kT000] - q2 * uz * uTc + lin * T[kT001] + q2 * t2z + q3h * cz3;
    return r;
}

// Adjoints of a node's moments (moment order) and of its colour gradient.
struct NodeAdjoint {
    float rr, rb, ux, uy, uz, pxx, pxy, pyy, pyz, pzz, pxz;
    float Fx, Fy, Fz;
};

// Relaxation part of a node: lambda_post (54 values at the node) -> adjoints of
// the node's moments and colour gradient; float64 parts of dJ/domega, dJ/d(A/2)
// and J.  kInterface false: the caller knows that the node is bulk.
//
// Per direction the stored pair is r_i = aR g_i + D_i, b_i = aB g_i - D_i, so
// with lg_i = aR lr_i + aB lb_i and ld_i = lr_i - lb_i the node's sums are
//   d/d(aR - aB)-part  sum ld_i g_i,   d/drho  sum lg_i feq_i / rho,
//   d/du     sum lg_i w rho (c P_i - u Q_i)  (dfeq/du),
//   d/dPi    oms sum lg_i w H2_i / 2cs4 and the third-order a3 chain,
//   d/domega -sum lg_i fneq_i,  d/dF from Omega2 and D,  d/dK from D.
// Opposite directions i, i+1 are taken together: feq and fneq split into even
// and odd parts, Omega2 is even and D odd, so every sum needs only
// lg_i + lg_o, lg_i - lg_o, ld_i + ld_o and ld_i - ld_o.
template <bool kPeriodic, bool kInterface>
__device__ __forceinline__ void adj_collide_node(const DeviceState &s, const float *M, const float *lam,
                                                 const AdjObjective &obj, int x, int y, int z, NodeAdjoint &o,
                                                 double &a_omega, double &a_Ah, double &a_J) {
    const Geometry &g = s.g;
    const Physics &ph = s.ph;
    const uint32_t id = uint32_t(x) + uint32_t(g.sy) * uint32_t(y) + uint32_t(g.sz) * uint32_t(z);
    const size_t N = g.N;
    const float *mom = M;
    const float rr = mom[kMomRR * N + id], rb = mom[kMomRB * N + id];
    const float ux = mom[kMomUX * N + id], uy = mom[kMomUY * N + id], uz = mom[kMomUZ * N + id];
    const NeqTerms n = make_neq(mom[kMomPXX * N + id], mom[kMomPXY * N + id], mom[kMomPYY * N + id],
                                mom[kMomPYZ * N + id], mom[kMomPZZ * N + id], mom[kMomPXZ * N + id], ux, uy, uz);
    const float rho = rr + rb;
    const float invr = 1.0f / rho;
    const float aR = rr * invr, aB = rb * invr;
    const float oms = 1.0f - omega_at(ph, y);
    const bool interface = kInterface && !is_bulk(rr, rb);
    float Fx = 0.f, Fy = 0.f, Fz = 0.f, absF = 0.f, K = 0.f;
    bool has_dir = false;
    if (interface) {
        // periodic box: neighbours wrap over the interior; jet: the record's
        // psi plane holds the ghost values the forward step read unwrapped
        const float *psi = M + size_t(kTapePsi) * N;
        const int xn[3] = {kPeriodic ? wrap_interior(x - 1, g.NX) : x - 1, x,
                           kPeriodic ? wrap_interior(x + 1, g.NX) : x + 1};
        const int yn[3] = {g.sy * (kPeriodic ? wrap_interior(y - 1, g.NY) : y - 1), g.sy * y,
                           g.sy * (kPeriodic ? wrap_interior(y + 1, g.NY) : y + 1)};
        const int zn[3] = {g.sz * (kPeriodic ? wrap_interior(z - 1, g.NZ) : z - 1), g.sz * z,
                           g.sz * (kPeriodic ? wrap_interior(z + 1, g.NZ) : z + 1)};
        float sx = 0.f, sy = 0.f, sz = 0.f;
        static_for<kQ - 1>([&](auto I) {
            constexpr int i = decltype(I)::value + 1;
            using D = Dir<i>;
            const float wp = D::w * psi[xn[D::cx + 1] + yn[D::cy + 1] + zn[D::cz + 1]];
            if constexpr (D::cx != 0) sx += D::fx * wp;
            if constexpr (D::cy != 0) sy += D::fy * wp;
            if constexpr (D::cz != 0) sz += D::fz * wp;
        });
        Fx = kInvCs2 * sx;
        Fy = kInvCs2 * sy;
        Fz = kInvCs2 * sz;
        absF = sqrtf(Fx * Fx + Fy * Fy + Fz * Fz);
        has_dir = !(absF <= 1.0e-4f);
        K = ph.beta * ((rr * rb) / (rho * rho)) * rho;
    }
    const float invF = has_dir ? 1.0f / absF : 0.0f;
    const float invF2 = invF * invF;
    [[maybe_unused]] const float Ah = ph.Ah;
    const size_t row = pop_row(g, y, z);
    // (lambda_r, lambda_b) of a direction: one float2, as the populations
    auto lam_at = [&](int slot) {
        return reinterpret_cast<const float2 *>(lam)[row + size_t(slot) * size_t(g.px) + size_t(x)];
    };
    // Bulk part: g_i = w_i P(c_i) with P the collision polynomial, so the
    // sums over directions are the polynomial's coefficients dotted with
    // the moments T_k = sum_i w_i lambda_g,i m_k(c_i) (and U_k with
    // lambda_r - lambda_b for the colour split).  The moments are formed
    // group by group: per (cy, cz) the three cx values reduce to
    // (sum, sum cx, sum cx^2), which add into the 17 moments with the
    // weights cy^b cz^c.
    float Tm[17], Um[17];
    #pragma unroll
    for (int k = 0; k < 17; ++k) Tm[k] = Um[k] = 0.f;
    static_for<9>([&](auto G) {
        constexpr int cy = decltype(G)::value / 3 - 1, cz = decltype(G)::value % 3 - 1;
        float mv[3], nv[3];
        static_for<3>([&](auto X) {
            constexpr int cx = decltype(X)::value - 1;
            constexpr int i = dir_of(cx, cy, cz);
            const float2 l = lam_at(slot_pair(i));
            mv[cx + 1] = Dir<i>::w * (aR * l.x + aB * l.y);
            nv[cx + 1] = Dir<i>::w * (l.x - l.y);
        });
        const float m2 = mv[2] + mv[0], n2 = nv[2] + nv[0];
        const float ms[3] = {m2 + mv[1], mv[2] - mv[0], m2};
        const float ns[3] = {n2 + nv[1], nv[2] - nv[0], n2};
        static_for<17>([&](auto K) {
            constexpr int k = decltype(K)::value;
            constexpr int wgt = ipow1(cy, poly_exp(k, 1)) * ipow1(cz, poly_exp(k, 2));
            constexpr int a = poly_exp(k, 0);
            if constexpr (wgt == 1) {
                Tm[k] += ms[a];
                Um[k] += ns[a];
            } else if constexpr (wgt == -1) {
                Tm[k] -= ms[a];
                Um[k] -= ns[a];
            }
        });
    });
    const PolyAdjoint pT = poly_adjoint(Tm, ux, uy, uz, n);
    const PolyAdjoint pU = poly_adjoint(Um, ux, uy, uz, n);
    const float(&S2)[6] = pT.S2;
    const float(&S3)[7] = pT.S3;
    const float l_rhoeq = rho * pT.Phi;  // sum lambda_g feq (feq is proportional to rho)
    const float l_oms = pT.Psi;          // sum lambda_g fneq
    float l_d = rho * pU.Phi + oms * pU.Psi;  // sum (lambda_r - lambda_b) g
    // interface nodes: the perturbation and recolouring terms, direction by direction
    float sAx = 0.f, sAy = 0.f, sAz = 0.f, sB = 0.f, sDx = 0.f, sDy = 0.f, sDz = 0.f, sE = 0.f, sBB = 0.f,
          l_Ah = 0.f;
    if (interface) {
        {  // rest direction: even only
            const float2 l0 = lam_at(slot_pair(0));
            const float lg = aR * l0.x + aB * l0.y, ld = l0.x - l0.y;
            const float o2A = -absF * Dir<0>::B;  // Omega2 / (A/2)
            l_d += ld * (Ah * o2A);
            sBB += lg * Dir<0>::B;
            l_Ah += lg * o2A;
        }
        static_for<(kQ - 1) / 2>([&](auto P) {
            constexpr int i = 2 * decltype(P)::value + 1;
            using D = Dir<i>;
            const float2 li = lam_at(slot_pair(i)), lo = lam_at(slot_pair(i + 1));
            const float lgi = aR * li.x + aB * li.y, lgo = aR * lo.x + aB * lo.y;
            const float ldi = li.x - li.y, ldo = lo.x - lo.y;
            const float gs = lgi + lgo, ds = ldi + ldo, dd = ldi - ldo;
            float fc = 0.f;
            if constexpr (D::cx != 0) fc += D::fx * Fx;
            if constexpr (D::cy != 0) fc += D::fy * Fy;
            if constexpr (D::cz != 0) fc += D::fz * Fz;
            const float o2A = absF * (D::w * (fc * fc) * invF2 - D::B);  // Omega2 / (A/2), even
            l_d += ds * (Ah * o2A);
            sBB += gs * D::B;
            l_Ah += gs * o2A;
            const float a = gs * D::w * fc, d = dd * D::w * D::invc;
            if constexpr (D::cx != 0) { sAx += D::fx * a; sDx += D::fx * d; }
            if constexpr (D::cy != 0) { sAy += D::fy * a; sDy += D::fy * d; }
            if constexpr (D::cz != 0) { sAz += D::fz * a; sDz += D::fz * d; }
            sB += a * fc;
            sE += d * fc;
        });
    }
    // fneq: Pi enters directly (H2) and through the third-order terms a3
    const float c2 = oms * kInv2Cs4, c3 = oms * kInv2Cs6;
    float lPxx = S2[0] * c2, lPxy = 2.0f * S2[1] * c2, lPyy = S2[2] * c2;
    float lPyz = 2.0f * S2[3] * c2, lPzz = S2[4] * c2, lPxz = 2.0f * S2[5] * c2;
    const float la_xxy = S3[0] * c3, la_xxz = S3[1] * c3, la_xyy = S3[2] * c3, la_xzz = S3[3] * c3;
    const float la_yyz = S3[4] * c3, la_yzz = S3[5] * c3, la_xyz = 2.0f * S3[6] * c3;
    lPxx += la_xxy * uy + la_xxz * uz;
    lPyy += la_xyy * ux + la_yyz * uz;
    lPzz += la_xzz * ux + la_yzz * uy;
    lPxy += 2.0f * la_xxy * ux + 2.0f * la_xyy * uy + la_xyz * uz;
    lPxz += 2.0f * la_xxz * ux + 2.0f * la_xzz * uz + la_xyz * uy;
    lPyz += 2.0f * la_yyz * uy + 2.0f * la_yzz * uz + la_xyz * ux;
    float lux = 2.0f * la_xxy * n.pxy + 2.0f * la_xxz * n.pxz + la_xyy * n.pyy + la_xzz * n.pzz + la_xyz * n.pyz;
    float luy = la_xxy * n.pxx + 2.0f * la_xyy * n.pxy + 2.0f * la_yyz * n.pyz + la_yzz * n.pzz + la_xyz * n.pxz;
    float luz = la_xxz * n.pxx + 2.0f * la_xzz * n.pxz + la_yyz * n.pyy + 2.0f * la_yzz * n.pyz + la_xyz * n.pxy;
    // feq: rho times the u-gradient of the feq polynomial against T
    lux += rho * pT.dPhi[0];
    luy += rho * pT.dPhi[1];
    luz += rho * pT.dPhi[2];
    // colour gradient: perturbation and recolouring
    float lFx = 0.f, lFy = 0.f, lFz = 0.f, lK = 0.f;
    if (interface) {
        if (has_dir) {
            const float i3 = invF2 * invF;
            lFx = Ah * (2.0f * invF * sAx - Fx * i3 * sB - Fx * invF * sBB) + K * (sDx * invF - Fx * i3 * sE);
            lFy = Ah * (2.0f * invF * sAy - Fy * i3 * sB - Fy * invF * sBB) + K * (sDy * invF - Fy * i3 * sE);
            lFz = Ah * (2.0f * invF * sAz - Fz * i3 * sB - Fz * invF * sBB) + K * (sDz * invF - Fz * i3 * sE);
            lK = sE * invF;
        } else if (absF > 0.0f) {
            const float q = -Ah * sBB / absF;
            lFx = q * Fx;
            lFy = q * Fy;
            lFz = q * Fz;
        }
    }
    const float inv2 = invr * invr;
    const float l_rho = l_rhoeq * invr;  // feq is proportional to rho
    o.rr = l_rho + l_d * rb * inv2 + lK * ph.beta * rb * rb * inv2;
    o.rb = l_rho - l_d * rr * inv2 + lK * ph.beta * rr * rr * inv2;
    // the objective's source: J_t = (w/2) sum uy^2 over nodes with y >= y_obs,
    // or the profile objective's dJ/duy of the node's radial bin (the bin of
    // radial_accumulate_warp, same float arithmetic)
    float lobj = 0.f;
    if (obj.table) {
        const float dx = float(x) - ph.jet_x0, dz = float(z) - ph.jet_z0;
        const unsigned rbin = unsigned(sqrtf(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dz, dz))));
        if (rbin < unsigned(ph.NRB)) lobj = obj.table[size_t(y) * ph.NRB + rbin];
    } else if (obj.weight != 0.0f && y >= obj.y_obs) {
        lobj = obj.weight * uy;
        a_J += 0.5 * double(obj.weight) * double(uy) * double(uy);
    }
    o.ux = lux;
    o.uy = luy + lobj;
    o.uz = luz;
    o.pxx = lPxx; o.pxy = lPxy; o.pyy = lPyy; o.pyz = lPyz; o.pzz = lPzz; o.pxz = lPxz;
    o.Fx = lFx; o.Fy = lFy; o.Fz = lFz;
    a_omega -= double(l_oms);  // oms = 1 - omega
    if constexpr (kInterface) a_Ah += double(l_Ah);
}

// Moment part of a node: the psi-adjoint lpsi and the adjoints of its moments
// back through the moments to the 54 pulled populations, stored at their pull
// sources (transposed streaming) in lam_out.  `node` false: a column that is
// only stored (store_columns), to complete the sectors of the rows.
template <bool kPeriodic>
__device__ __forceinline__ void adj_moments_node(const DeviceState &s, const float *M, const NodeAdjoint &o,
                                                 float lpsi, float *lam_out, int x, int y, int z, bool node) {
    const Geometry &g = s.g;
    const size_t N = g.N;
    float lrr = 0.f, lrb = 0.f, k0 = 0.f, ljx = 0.f, ljy = 0.f, ljz = 0.f;
    float lPxx = 0.f, lPxy = 0.f, lPyy = 0.f, lPyz = 0.f, lPzz = 0.f, lPxz = 0.f;
    if (node) {
        const uint32_t id = uint32_t(x) + uint32_t(g.sy) * uint32_t(y) + uint32_t(g.sz) * uint32_t(z);
        const float rr = M[kMomRR * N + id], rb = M[kMomRB * N + id];
        const float ux = M[kMomUX * N + id], uy = M[kMomUY * N + id], uz = M[kMomUZ * N + id];
        const float rho = rr + rb;
        const float inv2 = 1.0f / (rho * rho);
        lrr = o.rr + lpsi * 2.0f * rb * inv2;
        lrb = o.rb - lpsi * 2.0f * rr * inv2;
        lPxx = o.pxx; lPxy = o.pxy; lPyy = o.pyy;
        lPyz = o.pyz; lPzz = o.pzz; lPxz = o.pxz;
        // Pi = A - rho u u
        const float lux = o.ux - rho * (2.0f * ux * lPxx + uy * lPxy + uz * lPxz);
        const float luy = o.uy - rho * (2.0f * uy * lPyy + ux * lPxy + uz * lPyz);
        const float luz = o.uz - rho * (2.0f * uz * lPzz + ux * lPxz + uy * lPyz);
        float lrho = -(lPxx * ux * ux + lPxy * ux * uy + lPyy * uy * uy + lPyz * uy * uz + lPzz * uz * uz + lPxz * ux * uz);
        // u = j / rho
        const float invr = 1.0f / rho;
        ljx = lux * invr; ljy = luy * invr; ljz = luz * invr;
        lrho -= (lux * ux + luy * uy + luz * uz) * invr;
        // lambda_g,i = lrho + lj.c_i + lP:H2(c_i) is a quadratic polynomial in c_i:
        // evaluated at the 27 directions by sum factorisation (per cz, then cy,
        // then cx) instead of a Hermite sum per direction
        k0 = lrho - kCs2 * (lPxx + lPyy + lPzz);
    }
    const PullMap<CodecF32> pm(g, x, y, z, kPeriodic);
    static_for<3>([&](auto CZ) {
        constexpr int cz = decltype(CZ)::value - 1;
        const float az = cz == 0 ? k0 : (cz > 0 ? k0 + ljz + lPzz : k0 - ljz + lPzz);
        const float bxz = cz == 0 ? ljx : (cz > 0 ? ljx + lPxz : ljx - lPxz);  // coefficient of cx
        const float byz = cz == 0 ? ljy : (cz > 0 ? ljy + lPyz : ljy - lPyz);  // coefficient of cy
        static_for<3>([&](auto CY) {
            constexpr int cy = decltype(CY)::value - 1;
            const float c0 = cy == 0 ? az : (cy > 0 ? az + byz + lPyy : az - byz + lPyy);
            const float c1 = cy == 0 ? bxz : (cy > 0 ? bxz + lPxy : bxz - lPxy);
            const float c2 = c0 + lPxx;
            static_for<3>([&](auto CX) {
                constexpr int cx = decltype(CX)::value - 1;
                constexpr int i = dir_of(cx, cy, cz);
                const float lgi = cx == 0 ? c0 : (cx > 0 ? c2 + c1 : c2 - c1);
                // lanes of columns that are only stored write 0 to their own
                // column of the rows, never to a y ghost plane
                if (!node && !kPeriodic && ((cy == 1 && pm.gy_p) || (cy == -1 && pm.gy_m))) return;
                size_t grow;
                int xs;
                pm.template src<i>(node ? x : x + cx, grow, xs);
                reinterpret_cast<float2 *>(lam_out)[grow + size_t(dir_cx(i) + 1) * g.px + xs] =
                    make_float2(lrr + lgi, lrb + lgi);
            });
        });
    });
}

__device__ __forceinline__ void adj_write(const NodeAdjoint &o, float *lmom, size_t N, uint32_t id) {
    const float v[kMomCount] = {o.rr, o.rb, o.ux, o.uy, o.uz, o.pxx, o.pxy, o.pyy, o.pyz, o.pzz, o.pxz};
#pragma unroll
    for (int k = 0; k < kMomCount; ++k) lmom[size_t(k) * N + id] = v[k];
}
__device__ __forceinline__ void adj_read(NodeAdjoint &o, const float *lmom, size_t N, uint32_t id) {
    float v[kMomCount];
#pragma unroll
    for (int k = 0; k < kMomCount; ++k) v[k] = lmom[size_t(k) * N + id];
    o = NodeAdjoint{v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7], v[8], v[9], v[10], 0.f, 0.f, 0.f};
}

// The reverse step in the pieces of 32 columns of the split step (fused.cuh),
// with the flags of the pieces that hold an interface node of the state.  Only
// an interface node has a colour-gradient adjoint F, and a node's psi-adjoint
// gathers F of its 26 neighbours, so a piece with no flagged piece around it is
// taken from lambda_in to lambda_out in one pass:
//   k_adj_relax  unflagged pieces: the relaxation part, and where no interface
//                node is around the moment part too; otherwise the moments'
//                adjoints go to lmom, and the piece is marked as left over.
//                Flagged pieces: the relaxation part, to lmom and lf.
//   k_adj_near   pieces left over: psi-adjoint from lf of the interface nodes
//                around, moment part.
// (The jet's boundary adjoint, between the two, adds to lmom in rows 1 and
// NY-2, which are always left over.)
// Bound by HBM: lambda 216 B read and 216 written, the moment record 48 read a
// node; lmom and lf (56 B written and read) only near interfaces, where the
// two-pass form moved them for every node.  Reverse step, before and after:
// 96^3 bubble (a third of the pieces left over) 124 -> 109 us, jet 64x128x64
// 101 -> 79 us (its boundary adjoint 26 -> 7 us of that).
// CTAs per SM: 20 warps of 96 registers for k_adj_relax (which spill a little:
// 9.33 ms for the 96^3 bubble's 40 steps against 9.86 at 16 warps that do not
// and 9.44 at 24), 24 of 80 for k_adj_near (9.29 ms against 9.33 at 20).
constexpr int kAdjThreads = 128, kAdjRelaxBlocks = 5, kAdjNearBlocks = 6;

__host__ __device__ __forceinline__ int adj_pieces_per_row(const Geometry &g) { return pieces_per_row<CodecF32>(g); }

// What piece (w, y, z) sees of the flags around it: bit 3 r + d, r = 3 (dy + 1)
// + dz + 1 over the rows; d = 1: the row's piece at w holds an interface node;
// d = 0, 2: the node before its first or after its last column is one.  The box
// wraps when periodic; outside it nothing is flagged.  Warp-collective.
template <bool kPeriodic>
__device__ __forceinline__ unsigned flags_around(const Geometry &g, const uint8_t *flags, int w, int y, int z) {
    const int ppr = adj_pieces_per_row(g), lane = int(threadIdx.x & 31);
    bool hit = false;
    if (lane < 27) {
        int yy = y + lane / 9 - 1, zz = z + (lane / 3) % 3 - 1, ww = w + lane % 3 - 1;
        if constexpr (kPeriodic) {
            yy = wrap_interior(yy, g.NY);
            zz = wrap_interior(zz, g.NZ);
            // the piece of column NX-2 lies before column 1's, and after it
            ww = ww < 0 ? (g.NX - 2) >> 5 : (ww * 32 > g.NX - 2 ? 0 : ww);
        }
        if (yy >= 1 && yy <= g.NY - 2 && zz >= 1 && zz <= g.NZ - 2 && ww >= 0 && ww < ppr)
            hit = (flags[(size_t(zz - 1) * (g.NY - 2) + (yy - 1)) * ppr + ww] >> (lane % 3 == 1 ? 0 : lane % 3 == 0 ? 2 : 1)) & 1;
    }
    return __ballot_sync(kFull, hit);
}

// Calls f(w, y, z) with a whole warp for every piece set in `flags`, the pieces
// spread over blocks 0 .. ctas-1 as in k_step_interface.
template <class F>
__device__ __forceinline__ void for_flagged_pieces(const Geometry &g, const uint8_t *flags, uint32_t ctas, F &&f) {
    __shared__ uint32_t list[kAdjThreads];
    __shared__ int found;
    constexpr uint32_t kGroup = 4;
    const int lane = int(threadIdx.x & 31), warp = int(threadIdx.x >> 5);
    const uint32_t ppr = uint32_t(adj_pieces_per_row(g));
    const uint32_t pieces = ppr * uint32_t(g.NY - 2) * uint32_t(g.NZ - 2);
    for (uint32_t first = 0; first < pieces; first += ctas * kAdjThreads) {
        if (threadIdx.x == 0) found = 0;
        __syncthreads();
        const uint64_t mine = (uint64_t(threadIdx.x / kGroup) * ctas + blockIdx.x) * kGroup + threadIdx.x % kGroup + first;
        const bool flagged = mine < pieces && flags[mine];
        const unsigned hits = __ballot_sync(kFull, flagged);
        int base = 0;
        if (lane == 0 && hits) base = atomicAdd(&found, __popc(hits));
        base = __shfl_sync(kFull, base, 0);
        if (flagged) list[base + __popc(hits & ((1u << lane) - 1u))] = uint32_t(mine);
        __syncthreads();
        for (int i = warp; i < found; i += kAdjThreads / 32) {
            const uint32_t piece = list[i], row = piece / ppr, zi = row / uint32_t(g.NY - 2);
            f(int(piece - row * ppr), 1 + int(row - zi * uint32_t(g.NY - 2)), 1 + int(zi));
        }
        __syncthreads();
    }
}

// The two roles share a launch: its first `list_blocks` blocks take the flagged
// pieces, each other block the unflagged ones among kAdjThreads / 32 neighbours.
template <bool kPeriodic>
__global__ void __launch_bounds__(kAdjThreads, kAdjRelaxBlocks) k_adj_relax(const DeviceState s,
                                                                           const float *M, const uint8_t *flags,
                                                                           uint8_t *near_flags, const float *lam,
                                                                           float *lmom, float *lf, float *lam_out,
                                                                           double *acc, AdjObjective obj,
                                                                           int list_blocks, int plane_blocks) {
    __shared__ double sh[3 * (kAdjThreads / 32)];
    const Geometry &g = s.g;
    double a_omega = 0.0, a_Ah = 0.0, a_J = 0.0;
    wait_then_allow_if_small();
    if (int(blockIdx.x) < list_blocks) {
        for_flagged_pieces(g, flags, uint32_t(list_blocks), [&](int w, int y, int z) {
            const int x = w * 32 + int(threadIdx.x & 31);
            if (x < 1 || x > g.NX - 2) return;
            NodeAdjoint o;
            adj_collide_node<kPeriodic, true>(s, M, lam, obj, x, y, z, o, a_omega, a_Ah, a_J);
            const uint32_t id = uint32_t(x) + uint32_t(g.sy) * uint32_t(y) + uint32_t(g.sz) * uint32_t(z);
            adj_write(o, lmom, g.N, id);
            lf[id] = o.Fx;
            lf[size_t(g.N) + id] = o.Fy;
            lf[size_t(2) * g.N + id] = o.Fz;
        });
    } else {
        const int ppr = adj_pieces_per_row(g), block = int(blockIdx.x) - list_blocks, zi = block / plane_blocks;
        const int piece = (block - zi * plane_blocks) * (kAdjThreads / 32) + int(threadIdx.x >> 5);
        const int row = piece / ppr, y = 1 + row, z = 1 + zi;
        if (y <= g.NY - 2) {  // uniform over the warp
            const int w = piece - row * ppr, x = w * 32 + int(threadIdx.x & 31);
            const unsigned around = flags_around<kPeriodic>(g, flags, w, y, z);
            const bool near_one = around != 0 || (!kPeriodic && (y == 1 || y == g.NY - 2));
            if ((x & 31) == 0) near_flags[(size_t(zi) * (g.NY - 2) + row) * ppr + w] = near_one ? 1 : 0;
            const bool node = x >= 1 && x <= g.NX - 2;
            if (!((around >> 13) & 1u)) {
                NodeAdjoint o{};
                if (node) adj_collide_node<kPeriodic, false>(s, M, lam, obj, x, y, z, o, a_omega, a_Ah, a_J);
                if (!near_one) {
                    if (x < store_columns<CodecF32>(g)) adj_moments_node<kPeriodic>(s, M, o, 0.0f, lam_out, x, y, z, node);
                } else if (node) {
                    const uint32_t id = uint32_t(x) + uint32_t(g.sy) * uint32_t(y) + uint32_t(g.sz) * uint32_t(z);
                    adj_write(o, lmom, g.N, id);
                    if (!kPeriodic && y == g.NY - 2)  // read by the boundary adjoint
                        for (int k = 0; k < 3; ++k) lf[size_t(k) * g.N + id] = 0.0f;
                }
            }
        }
    }
    double r[3] = {a_omega, a_Ah, obj.J ? a_J : 0.0};
    block_sum3(r, sh, kAdjThreads);
    if (threadIdx.x == 0) {
        if (r[0] != 0.0) atomicAdd(acc, r[0]);
        if (r[1] != 0.0) atomicAdd(acc + 1, r[1]);
        if (r[2] != 0.0) atomicAdd(obj.J, r[2]);
    }
}

template <bool kPeriodic>
__global__ void __launch_bounds__(kAdjThreads, kAdjNearBlocks) k_adj_near(const DeviceState s, const float *M,
                                                                             const uint8_t *flags,
                                                                             const uint8_t *near_flags,
                                                                             const float *lmom, const float *lf,
                                                                             float *lam_out) {
    const Geometry &g = s.g;
    const size_t N = g.N;
    wait_then_allow_if_small();
    for_flagged_pieces(g, near_flags, gridDim.x, [&](int w, int y, int z) {
        const unsigned around = flags_around<kPeriodic>(g, flags, w, y, z);
        const int x = w * 32 + int(threadIdx.x & 31);
        if (x >= store_columns<CodecF32>(g)) return;
        const bool node = x >= 1 && x <= g.NX - 2;
        NodeAdjoint o{};
        float lpsi = 0.f;
        if (node) {
            // psi(y) enters F(y - c_j) with weight w_j c_j / cs2
            const int xs[3] = {kPeriodic ? wrap_interior(x - 1, g.NX) : x - 1, x,
                               kPeriodic ? wrap_interior(x + 1, g.NX) : x + 1};
            // the piece of the node before and after: bit offsets in a row of `around`
            const int px[3] = {(x & 31) == 0 || x == 1 ? 0 : 1, 1, (x & 31) == 31 || x == g.NX - 2 ? 2 : 1};
            static_for<kQ - 1>([&](auto I) {
                constexpr int i = decltype(I)::value + 1;
                using D = Dir<i>;
                constexpr int r = 3 * (1 - D::cy) + (1 - D::cz);  // row (y - cy, z - cz)
                float v0 = 0.f, v1 = 0.f, v2 = 0.f;
                if ((around >> (3 * r + px[1 - D::cx])) & 1u) {
                    const int yn = kPeriodic ? wrap_interior(y - D::cy, g.NY) : y - D::cy;
                    const int zn = kPeriodic ? wrap_interior(z - D::cz, g.NZ) : z - D::cz;
                    const uint32_t nid = uint32_t(xs[1 - D::cx]) + uint32_t(g.sy) * uint32_t(yn) + uint32_t(g.sz) * uint32_t(zn);
                    if constexpr (D::cx != 0) v0 = lf[nid];
                    if constexpr (D::cy != 0) v1 = lf[N + nid];
                    if constexpr (D::cz != 0) v2 = lf[2 * N + nid];
                }
                float dot = 0.f;
                if constexpr (D::cx != 0) dot += D::fx * v0;
                if constexpr (D::cy != 0) dot += D::fy * v1;
                if constexpr (D::cz != 0) dot += D::fz * v2;
                lpsi += D::w * dot;
            });
            lpsi *= kInvCs2;
            const uint32_t id = uint32_t(x) + uint32_t(g.sy) * uint32_t(y) + uint32_t(g.sz) * uint32_t(z);
            adj_read(o, lmom, N, id);
        }
        adj_moments_node<kPeriodic>(s, M, o, lpsi, lam_out, x, y, z, node);
    });
}

// One wave of blocks over the flagged pieces, at most a warp each.
unsigned adj_list_blocks(const Geometry &g, int per_sm) {
    const long long per = kAdjThreads / 32, pieces = (long long)adj_pieces_per_row(g) * (g.NY - 2) * (g.NZ - 2);
    return unsigned(std::min<long long>((pieces + per - 1) / per, 148ll * per_sm));
}

// Flags of the pieces of a moment record (k_step_pull sets those of the states
// it records).
__global__ void __launch_bounds__(kRedThreads) k_piece_flags(const DeviceState s, const float *__restrict__ M,
                                                            uint8_t *flags) {
    const Geometry &g = s.g;
    const int ppr = adj_pieces_per_row(g);
    const int piece = int(blockIdx.x) * (kRedThreads / 32) + int(threadIdx.x >> 5);
    const int row = piece / ppr, y = 1 + row, z = 1 + int(blockIdx.y);
    if (y > g.NY - 2) return;
    const int w = piece - row * ppr, x = w * 32 + int(threadIdx.x & 31);
    bool interface = false;
    if (x >= 1 && x <= g.NX - 2) {
        const uint32_t id = uint32_t(x) + uint32_t(g.sy) * uint32_t(y) + uint32_t(g.sz) * uint32_t(z);
        interface = !is_bulk(M[kMomRR * size_t(g.N) + id], M[kMomRB * size_t(g.N) + id]);
    }
    const unsigned lanes = __ballot_sync(kFull, interface);
    if ((x & 31) == 0) flags[(size_t(blockIdx.y) * (g.NY - 2) + row) * ppr + w] = piece_flag(g, w, lanes);
}

// Adjoint of the regularised non-equilibrium part over a set of directions:
// S2 = sum mu_i H2_i, S3 = sum mu_i H3_i with mu_i = (1-omega) lambda_i w_i give
// the adjoints of Pi (pxx, pxy, pyy, pyz, pzz, pxz) and the u added through
// the third-order terms a3 (lbm.cuh:38-78).
__device__ __forceinline__ void neq_adjoint(const float (&S2)[6], const float (&S3)[7], const NeqTerms &n, float ux,
                                            float uy, float uz, float (&lP)[6], float (&lu)[3]) {
    const float c2 = kInv2Cs4, c3 = kInv2Cs6;
    float lPxx = S2[0] * c2, lPxy = 2.0f * S2[1] * c2, lPyy = S2[2] * c2;
    float lPyz = 2.0f * S2[3] * c2, lPzz = S2[4] * c2, lPxz = 2.0f * S2[5] * c2;
    const float la_xxy = S3[0] * c3, la_xxz = S3[1] * c3, la_xyy = S3[2] * c3, la_xzz = S3[3] * c3;
    const float la_yyz = S3[4] * c3, la_yzz = S3[5] * c3, la_xyz = 2.0f * S3[6] * c3;
    lPxx += la_xxy * uy + la_xxz * uz;
    lPyy += la_xyy * ux + la_yyz * uz;
    lPzz += la_xzz * ux + la_yzz * uy;
    lPxy += 2.0f * la_xxy * ux + 2.0f * la_xyy * uy + la_xyz * uz;
    lPxz += 2.0f * la_xxz * ux + 2.0f * la_xzz * uz + la_xyz * uy;
    lPyz += 2.0f * la_yyz * uy + 2.0f * la_yzz * uz + la_xyz * ux;
    lu[0] += 2.0f * la_xxy * n.pxy + 2.0f * la_xxz * n.pxz + la_xyy * n.pyy + la_xzz * n.pzz + la_xyz * n.pyz;
    lu[1] += la_xxy * n.pxx + 2.0f * la_xyy * n.pxy + 2.0f * la_yyz * n.pyz + la_yzz * n.pzz + la_xyz * n.pxz;
    lu[2] += la_xxz * n.pxx + 2.0f * la_xzz * n.pxz + la_yyz * n.pyy + 2.0f * la_yzz * n.pyz + la_xyz * n.pxy;
    lP[0] = lPxx; lP[1] = lPxy; lP[2] = lPyy; lP[3] = lPyz; lP[4] = lPzz; lP[5] = lPxz;
}

template <int I>
__device__ __forceinline__ void neq_accumulate(float mu, float (&S2)[6], float (&S3)[7]) {
    using D = Dir<I>;
    S2[0] += mu * D::Hxx; S2[1] += mu * D::Hxy; S2[2] += mu * D::Hyy;
    S2[3] += mu * D::Hyz; S2[4] += mu * D::Hzz; S2[5] += mu * D::Hxz;
    if constexpr (D::Hxxy != 0.0f) S3[0] += mu * D::Hxxy;
    if constexpr (D::Hxxz != 0.0f) S3[1] += mu * D::Hxxz;
    if constexpr (D::Hxyy != 0.0f) S3[2] += mu * D::Hxyy;
    if constexpr (D::Hxzz != 0.0f) S3[3] += mu * D::Hxzz;
    if constexpr (D::Hyyz != 0.0f) S3[4] += mu * D::Hyyz;
    if constexpr (D::Hyzz != 0.0f) S3[5] += mu * D::Hyzz;
    if constexpr (D::Hxyz != 0.0f) S3[6] += mu * D::Hxyz;
}

__device__ __forceinline__ float inlet_noise_factor(const Physics &ph, int64_t step, int x, int z) {
    if (ph.inlet_noise == 0.0f) return 1.0f;
    const float u = hash_uniform(ph.seed, 0x1A1E7ull ^ uint64_t(step), uint64_t(x), uint64_t(z));
    return 1.0f + (2.0f * u - 1.0f) * ph.inlet_noise;
}

// One thread per interior column (x, z): the outlet at y = NY-1 (blockIdx.z 0)
// or, in a jet column, the inlet at y = 0 (1).  A ghost-plane slot enters only if an interior
// node pulls it (the boundary also writes slots nothing reads).
__global__ void __launch_bounds__(32) k_adj_boundary(const DeviceState s, int64_t step, const float *M,
                                                      const float *Bt, const float *lam,
                                                      const float *lf, float *lmom,
                                                      const float *LB_in, float *LB_out,
                                                      const float *bessel, int nb, double *dJdc) {
    const Geometry &g = s.g;
    const Physics &ph = s.ph;
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int z = blockIdx.y * blockDim.y + threadIdx.y;
    wait_then_allow_if_small();
    const bool col = x >= 1 && x <= g.NX - 2 && z >= 1 && z <= g.NZ - 2;
    const size_t N = g.N;
    const int NP = g.NX * g.NZ;
    const int ic = x + g.NX * z;
    float dc[kInletBesselMax];
#pragma unroll
    for (int k = 0; k < kInletBesselMax; ++k) dc[k] = 0.f;
    auto pulled = [&](int xp, int zp) { return xp >= 1 && xp <= g.NX - 2 && zp >= 1 && zp <= g.NZ - 2; };
    // The values a side reads from memory come first, all in flight together;
    // one after the other behind the branches they took 26 us a launch.
    auto pulled_lambda = [&](auto CY, int y, float2 (&l)[9]) {
        constexpr int cy = decltype(CY)::value;
        static_for<9>([&](auto K) {
            constexpr int k = decltype(K)::value, i = dir_of(k / 3 - 1, cy, k % 3 - 1);
            l[k] = pulled(x + Dir<i>::cx, z + Dir<i>::cz)
                       ? reinterpret_cast<const float2 *>(lam)[pop_index(g, slot_pair(i), x, y, z)]
                       : make_float2(0.f, 0.f);
        });
    };
    auto add_to = [&](uint32_t id, const float (&v)[kMomCount]) {
        float m[kMomCount];
#pragma unroll
        for (int k = 0; k < kMomCount; ++k) m[k] = lmom[size_t(k) * N + id];
#pragma unroll
        for (int k = 0; k < kMomCount; ++k) lmom[size_t(k) * N + id] = m[k] + v[k];
    };
    if (col && blockIdx.z == 0) {
        // ---------------- outlet (boundary_conditions.cuh:163-233)
        const uint32_t idF = uint32_t(x) + uint32_t(g.sy) * uint32_t(g.NY - 2) + uint32_t(g.sz) * uint32_t(z);
        const float phi[5] = {M[kMomRR * N + idF], M[kMomRB * N + idF], M[kMomUX * N + idF], M[kMomUY * N + idF],
                              M[kMomUZ * N + idF]};
        const NeqTerms nF = make_neq(M[kMomPXX * N + idF], M[kMomPXY * N + idF], M[kMomPYY * N + idF],
                                     M[kMomPYZ * N + idF], M[kMomPZZ * N + idF], M[kMomPXZ * N + idF], phi[2], phi[3],
                                     phi[4]);
        float2 l9[9];
        pulled_lambda(std::integral_constant<int, -1>{}, g.NY - 1, l9);
        // colour-gradient adjoints of the nodes (x - cx, NY-2, z - cz)
        float f9[9][3];
        static_for<9>([&](auto K) {
            constexpr int k = decltype(K)::value, cx = k / 3 - 1, cz = k % 3 - 1;
            const bool in = pulled(x - cx, z - cz);
            const uint32_t nid = in ? uint32_t(x - cx) + uint32_t(g.sy) * uint32_t(g.NY - 2) + uint32_t(g.sz) * uint32_t(z - cz)
                                    : idF;
            for (int c = 0; c < 3; ++c) f9[k][c] = in ? lf[size_t(c) * N + nid] : 0.f;
        });
        float B[5], Bn[5];
        const float uc = clamp01(phi[3]);
#pragma unroll
        for (int c = 0; c < 5; ++c) {
            B[c] = Bt[c * NP + ic];
            Bn[c] = B[c] - uc * (B[c] - phi[c]);
        }
        const float rho = Bn[0] + Bn[1];
        const float inv = 1.0f / rho;
        const float aR = Bn[0] * inv, aB = Bn[1] * inv;
        const float oms = 1.0f - omega_at(ph, g.NY - 2);
        const EqTerms e = make_eq(Bn[2], Bn[3], Bn[4]);
        float lrho = 0.f, le[3] = {0.f, 0.f, 0.f}, laR = 0.f, laB = 0.f;
        float S2[6] = {0, 0, 0, 0, 0, 0}, S3[7] = {0, 0, 0, 0, 0, 0, 0};
        static_for<kQ>([&](auto I) {
            constexpr int i = decltype(I)::value;
            using D = Dir<i>;
            if constexpr (D::cy == -1) {
                const float2 l = l9[(D::cx + 1) * 3 + D::cz + 1];
                const float lr = l.x, lb = l.y;
                const float fe = feq<i>(rho, e), fn = fneq<i>(nF);
                const float gi = fe + oms * fn;
                const float lg = aR * lr + aB * lb;
                laR += lr * gi;
                laB += lb * gi;
                lrho += lg * fe * inv;
                float cu = 0.f;
                if constexpr (D::cx != 0) cu += D::fx * e.ux;
                cu += D::fy * e.uy;
                if constexpr (D::cz != 0) cu += D::fz * e.uz;
                const float P = kInvCs2 + cu * (2.0f * kInv2Cs4) + (cu * cu) * (3.0f * kInv6Cs6) - e.usq * kInv2Cs4;
                const float Q = kInvCs2 + cu * (2.0f * kInv2Cs4);
                const float wl = lg * D::w * rho;
                if constexpr (D::cx != 0) le[0] += wl * P * D::fx;
                le[1] += wl * P * D::fy;
                if constexpr (D::cz != 0) le[2] += wl * P * D::fz;
                const float q = wl * Q;
                le[0] -= q * e.ux;
                le[1] -= q * e.uy;
                le[2] -= q * e.uz;
                neq_accumulate<i>(oms * lg * D::w, S2, S3);
            }
        });
        const float inv2 = inv * inv;
        float lBn[5];
        lBn[0] = lrho + (laR - laB) * Bn[1] * inv2;
        lBn[1] = lrho - (laR - laB) * Bn[0] * inv2;
        lBn[2] = le[0];
        lBn[3] = le[1];
        lBn[4] = le[2];
        float luc = 0.f, lphi[5], lB[5];
#pragma unroll
        for (int c = 0; c < 5; ++c) {
            lBn[c] += LB_in[c * NP + ic];
            luc += lBn[c] * (phi[c] - B[c]);
            lphi[c] = uc * lBn[c];
            lB[c] = (1.0f - uc) * lBn[c];
        }
        if (phi[3] > 0.0f && phi[3] < 1.0f) lphi[3] += luc;  // d clamp01 / d uy
        float lP[6], lu[3] = {0.f, 0.f, 0.f};
        neq_adjoint(S2, S3, nF, phi[2], phi[3], phi[4], lP, lu);
        add_to(idF, {lphi[0], lphi[1], lphi[2] + lu[0], lphi[3] + lu[1], lphi[4] + lu[2], lP[0], lP[1], lP[2], lP[3],
                     lP[4], lP[5]});
        // psi(B) at (x, NY-1, z) entered the colour gradient of the step's
        // interior nodes (x, NY-2, z) - c over the cy = +1 directions
        float lpsi = 0.f;
        static_for<kQ>([&](auto I) {
            constexpr int i = decltype(I)::value;
            using D = Dir<i>;
            if constexpr (D::cy == 1) {
                const float(&v)[3] = f9[(D::cx + 1) * 3 + D::cz + 1];
                float dot = D::fy * v[1];
                if constexpr (D::cx != 0) dot += D::fx * v[0];
                if constexpr (D::cz != 0) dot += D::fz * v[2];
                lpsi += D::w * dot;
            }
        });
        lpsi *= kInvCs2;
        const float rB = B[0] + B[1];
        const float i2 = 1.0f / (rB * rB);
        lB[0] += lpsi * 2.0f * B[1] * i2;
        lB[1] -= lpsi * 2.0f * B[0] * i2;
#pragma unroll
        for (int c = 0; c < 5; ++c) LB_out[c * NP + ic] = lB[c];
    }
    if (col && blockIdx.z == 1) {
        // ---------------- inlet (boundary_conditions.cuh:17-85): jet columns only
        if (is_jet_column(ph, x, z)) {
            float2 l9[9];
            pulled_lambda(std::integral_constant<int, 1>{}, 0, l9);
            const uint32_t id1 = uint32_t(x) + uint32_t(g.sy) * 1u + uint32_t(g.sz) * uint32_t(z);
            const float u1x = M[kMomUX * N + id1], u1y = M[kMomUY * N + id1], u1z = M[kMomUZ * N + id1];
            const NeqTerms n1 = make_neq(M[kMomPXX * N + id1], M[kMomPXY * N + id1], M[kMomPYY * N + id1],
                                         M[kMomPYZ * N + id1], M[kMomPZZ * N + id1], M[kMomPXZ * N + id1], u1x, u1y,
                                         u1z);
            const float rT = ph.rhob0;  // the mask: red 0, blue rhob0 (aR = 0, aB = 1)
            const float U = inlet_velocity(s, step, x, z);
            const float omsb = 1.0f - ph.omega_b;
            float lU = 0.f;
            float T2[6] = {0, 0, 0, 0, 0, 0}, T3[7] = {0, 0, 0, 0, 0, 0, 0};
            static_for<kQ>([&](auto I) {
                constexpr int i = decltype(I)::value;
                using D = Dir<i>;
                if constexpr (D::cy == 1) {
                    const float lg = l9[(D::cx + 1) * 3 + D::cz + 1].y;  // red = 0 * g
                    // d feq_i / d uy at u = (0, U, 0): w rho (c_y P - U Q), c.u = U
                    const float P = kInvCs2 + U * (2.0f * kInv2Cs4) + (U * U) * (3.0f * kInv6Cs6) - (U * U) * kInv2Cs4;
                    const float Q = kInvCs2 + U * (2.0f * kInv2Cs4);
                    lU += lg * D::w * rT * (P - U * Q);
                    neq_accumulate<i>(omsb * lg * D::w, T2, T3);
                }
            });
            float lP1[6], lu1[3] = {0.f, 0.f, 0.f};
            neq_adjoint(T2, T3, n1, u1x, u1y, u1z, lP1, lu1);
            add_to(id1, {0.f, 0.f, lu1[0], lu1[1], lu1[2], lP1[0], lP1[1], lP1[2], lP1[3], lP1[4], lP1[5]});
            // U = U0 (1 + sum_k c_k J0_k) (1 + noise): dU/dc_k = U0 (1 + noise) J0_k
            if (bessel) {
                const float dU = ph.jet_velocity * inlet_noise_factor(ph, step, x, z);
                for (int k = 0; k < nb; ++k) dc[k] = lU * dU * bessel[k * NP + ic];
            }
        }
    }
    if (bessel) {
        for (int k = 0; k < nb; ++k) {
            double v = dc[k];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(kFull, v, o);
            if ((threadIdx.x & 31) == 0 && v != 0.0) atomicAdd(dJdc + k, v);
        }
    }
}

// The inverse: outlet state from src[5][NX*NZ] back to y = NY-1, with the psi
// the next step reads there (what the boundary launch writes).
__global__ void __launch_bounds__(256) k_restore_outlet_state(const DeviceState s, const float *src, float *psi) {
    const Geometry &g = s.g;
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int z = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= g.NX || z >= g.NZ) return;
    const uint32_t idB = uint32_t(x) + uint32_t(g.sy) * uint32_t(g.NY - 1) + uint32_t(g.sz) * uint32_t(z);
    const int NP = g.NX * g.NZ;
#pragma unroll
    for (int c = 0; c < 5; ++c) s.mom[size_t(c) * g.N + idB] = src[c * NP + x + g.NX * z];
    if (x >= 1 && x <= g.NX - 2 && z >= 1 && z <= g.NZ - 2)
        psi[idB] = psi_of(src[0 * NP + x + g.NX * z], src[1 * NP + x + g.NX * z]);
}

// Outlet state (rr, rb, ux, uy, uz at y = NY-1) of interior columns to dst[5][NX*NZ].
__global__ void __launch_bounds__(256) k_copy_outlet_state(const DeviceState s, float *dst) {
    const Geometry &g = s.g;
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int z = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= g.NX || z >= g.NZ) return;
    const uint32_t idB = uint32_t(x) + uint32_t(g.sy) * uint32_t(g.NY - 1) + uint32_t(g.sz) * uint32_t(z);
    const int NP = g.NX * g.NZ;
#pragma unroll
    for (int c = 0; c < 5; ++c) dst[c * NP + x + g.NX * z] = s.mom[size_t(c) * g.N + idB];
}

// What a jet record needs of the state beside what the step writes into it: the
// psi plane with its ghost values (plane kTapePsi of rec; the step rewrites the
// interior) and the outlet state (5 planes behind the record's).
__global__ void __launch_bounds__(256) k_record_state(const DeviceState s, const float *psi, float *rec, float *outlet) {
    const Geometry &g = s.g;
    const uint32_t NP = uint32_t(g.NX) * uint32_t(g.NZ), stride = gridDim.x * 256;
    wait_then_allow_if_small();
    for (uint32_t i = blockIdx.x * 256 + threadIdx.x; i < g.N; i += stride) rec[size_t(kTapePsi) * g.N + i] = psi[i];
    for (uint32_t i = blockIdx.x * 256 + threadIdx.x; i < NP; i += stride) {
        const uint32_t z = i / uint32_t(g.NX), x = i - z * uint32_t(g.NX);
        const uint32_t idB = x + uint32_t(g.sy) * uint32_t(g.NY - 1) + uint32_t(g.sz) * z;
#pragma unroll
        for (int c = 0; c < 5; ++c) outlet[size_t(c) * NP + i] = s.mom[size_t(c) * g.N + idB];
    }
}

// dJ/du0 for an initial state f0_c,i = feq_i(rho_c, u0): pulls lambda_0 like
// the forward step pulls populations.
__global__ void __launch_bounds__(kBX * kBY) k_adj_initial(const DeviceState s, const float *__restrict__ M,
                                                          const float *lam0, float *du0) {
    const Geometry &g = s.g;
    const int x = blockIdx.x * kBX + threadIdx.x;
    const int y = blockIdx.y * kBY + threadIdx.y;
    const int z = blockIdx.z;
    if (x >= g.NX || y >= g.NY) return;
    const uint32_t id = uint32_t(x) + uint32_t(g.sy) * uint32_t(y) + uint32_t(g.sz) * uint32_t(z);
    const size_t N = g.N;
    if (!(x >= 1 && x <= g.NX - 2 && y >= 1 && y <= g.NY - 2 && z >= 1 && z <= g.NZ - 2)) {
        du0[id] = du0[N + id] = du0[2 * N + id] = 0.0f;
        return;
    }
    const float *mom = M;
    const float rr = mom[kMomRR * N + id], rb = mom[kMomRB * N + id];
    const float ux = mom[kMomUX * N + id], uy = mom[kMomUY * N + id], uz = mom[kMomUZ * N + id];
    const EqTerms e = make_eq(ux, uy, uz);
    const PullMap<CodecF32> pm(g, x, y, z, true);
    float gx = 0.f, gy = 0.f, gz = 0.f, gq = 0.f;
    static_for<kQ>([&](auto I) {
        constexpr int i = decltype(I)::value;
        using D = Dir<i>;
        size_t grow;
        int xs;
        pm.template src<i>(x, grow, xs);
        const float2 l = reinterpret_cast<const float2 *>(lam0)[grow + size_t(dir_cx(i) + 1) * g.px + xs];
        const float lr = l.x, lb = l.y;
        float cu = 0.f;
        if constexpr (D::cx != 0) cu += D::fx * ux;
        if constexpr (D::cy != 0) cu += D::fy * uy;
        if constexpr (D::cz != 0) cu += D::fz * uz;
        const float P = kInvCs2 + cu * (2.0f * kInv2Cs4) + (cu * cu) * (3.0f * kInv6Cs6) - e.usq * kInv2Cs4;
        const float Q = kInvCs2 + cu * (2.0f * kInv2Cs4);
        const float wl = D::w * (lr * rr + lb * rb);
        if constexpr (D::cx != 0) gx += wl * P * D::fx;
        if constexpr (D::cy != 0) gy += wl * P * D::fy;
        if constexpr (D::cz != 0) gz += wl * P * D::fz;
        gq += wl * Q;
    });
    du0[id] = gx - ux * gq;
    du0[N + id] = gy - uy * gq;
    du0[2 * N + id] = gz - uz * gq;
}

}  // namespace

// ---------------------------------------------------------------------- host side

cudaError_t launch_boundary(const DeviceState &s, int wbuf, int64_t step, int which, bool from_bmom,
                            cudaStream_t st) {
    if (s.g.storage == kStoreF16) return boundary_dispatch<CodecF16>(s, wbuf, step, which, from_bmom, st);
    return boundary_dispatch<CodecF32>(s, wbuf, step, which, from_bmom, st);
}

cudaError_t launch_accumulate_radial(const DeviceState &s, cudaStream_t st) {
    return launch_overlapped(k_accumulate_radial, grid3(s.g), dim3(kBX, kBY), st, s);
}

cudaError_t launch_init_fields(const DeviceState &s, int mode, int red_inside, float r2, float bx, float by, float bz,
                               cudaStream_t st) {
    k_init_fields<<<grid3(s.g), dim3(kBX, kBY), 0, st>>>(s, mode, red_inside, r2, bx, by, bz);
    return cudaGetLastError();
}

cudaError_t launch_init_pops(const DeviceState &s, int mode, float noise, cudaStream_t st) {
    auto go = [&](auto made) {
        using C = decltype(made);
        const dim3 grid((pieces_per_row<C>(s.g) * (s.g.NY - 2) + kRedThreads / 32 - 1) / (kRedThreads / 32), s.g.NZ - 2);
        k_init_pops<C><<<grid, kRedThreads, 0, st>>>(s, made, mode, noise);
        return cudaGetLastError();
    };
    return s.g.storage == kStoreF16 ? go(make_codec<CodecF16>(s, 1)) : go(make_codec<CodecF32>(s, 1));
}

cudaError_t launch_refresh_psi(const DeviceState &s, cudaStream_t st) {
    k_refresh_psi<<<grid3(s.g), dim3(kBX, kBY), 0, st>>>(s);
    return cudaGetLastError();
}

cudaError_t launch_scatter_chunk(const DeviceState &s, int wbuf, const float *stage, size_t pitch, int z0, int nz,
                                 cudaStream_t st) {
    auto go = [&](auto made) {
        using C = decltype(made);
        const dim3 grid((pieces_per_row<C>(s.g) * (s.g.NY - 2) + kRedThreads / 32 - 1) / (kRedThreads / 32), nz);
        k_scatter_chunk<C><<<grid, kRedThreads, 0, st>>>(s, made, stage, pitch, z0);
        return cudaGetLastError();
    };
    return s.g.storage == kStoreF16 ? go(make_codec<CodecF16>(s, wbuf ^ 1)) : go(make_codec<CodecF32>(s, wbuf ^ 1));
}

cudaError_t launch_gather_chunk(const DeviceState &s, int cur, float *stage, size_t pitch, int z0, int nz,
                                cudaStream_t st) {
    const dim3 grid(((s.g.NX + 31) / 32 * s.g.NY + kRedThreads / 32 - 1) / (kRedThreads / 32), nz);
    auto go = [&](auto made) {
        using C = decltype(made);
        if (s.g.boundary == kBoundaryPeriodic)
            k_gather_chunk<C, true><<<grid, kRedThreads, 0, st>>>(s, made, stage, pitch, z0);
        else
            k_gather_chunk<C, false><<<grid, kRedThreads, 0, st>>>(s, made, stage, pitch, z0);
        return cudaGetLastError();
    };
    return s.g.storage == kStoreF16 ? go(make_codec<CodecF16>(s, cur)) : go(make_codec<CodecF32>(s, cur));
}

cudaError_t launch_unpad_rows(const DeviceState &s, int cur, cudaStream_t st) {
    const size_t rows = size_t(s.g.NY) * s.g.NZ * kQ;
    const void *src = s.pops[cur];
    void *dst = s.pops[cur ^ 1];
    if (s.g.storage == kStoreF16)
        k_unpad_rows<<<8 * 148, 256, 0, st>>>(static_cast<const __half2 *>(src), static_cast<__half2 *>(dst), s.g.NX,
                                              s.g.px, rows);
    else
        k_unpad_rows<<<8 * 148, 256, 0, st>>>(static_cast<const float2 *>(src), static_cast<float2 *>(dst), s.g.NX, s.g.px,
                                              rows);
    return cudaGetLastError();
}

cudaError_t launch_tke(const DeviceState &s, double *out, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(out, 0, sizeof(double), st);
    if (e != cudaSuccess) return e;
    k_tke<<<grid1(s.g), kRedThreads, 0, st>>>(s, out);
    return cudaGetLastError();
}

cudaError_t launch_uy_average(const DeviceState &s, uint32_t samples, cudaStream_t st) {
    k_uy_average<<<grid1(s.g), kRedThreads, 0, st>>>(s, samples);
    return cudaGetLastError();
}

// ---- VTI text (base64, RFC 4648 alphabet, '=' padding) ----------------------

__device__ __forceinline__ uint32_t b64_char(uint32_t v) {
    return v < 26 ? 'A' + v : v < 52 ? 'a' + (v - 26) : v < 62 ? '0' + (v - 52) : v == 62 ? '+' : '/';
}

// Word e of array a's float32 payload.
__device__ __forceinline__ uint32_t vti_word(const float *__restrict__ m, uint64_t N, int a, uint64_t e) {
    if (a < 2) return __float_as_uint(m[a * N + e]);
    if (a == 2) return __float_as_uint(__fadd_rn(m[e], m[N + e]));
    const uint64_t node = e / 3;
    return __float_as_uint(m[(2 + (e - 3 * node)) * N + node]);
}

// One thread per 3-byte group of [count][payload] -> one 4-character word.
// blockIdx.y selects the array; stores are 4-byte words, coalesced per warp.
__global__ void __launch_bounds__(256) k_vti_encode(const float *__restrict__ m, uint64_t N, char *__restrict__ text,
                                                    VtiText L) {
    const int a = blockIdx.y;
    const uint64_t payload = (a == 3 ? 3 : 1) * N * 4, total = payload + 8, groups = (total + 2) / 3;
    uint32_t *out = reinterpret_cast<uint32_t *>(text + L.off[a]);
    for (uint64_t g = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; g < groups;
         g += uint64_t(gridDim.x) * blockDim.x) {
        uint32_t v = 0, cw = 0;
        uint64_t ce = ~uint64_t(0);
        for (int k = 0; k < 3; ++k) {
            const uint64_t p = 3 * g + k;
            uint32_t b = 0;
            if (p < 8) {
                b = uint32_t(payload >> (8 * p)) & 0xffu;
            } else if (p < total) {
                const uint64_t q = p - 8, e = q >> 2;
                if (e != ce) {
                    ce = e;
                    cw = vti_word(m, N, a, e);
                }
                b = (cw >> (8 * (q & 3))) & 0xffu;
            }
            v = (v << 8) | b;
        }
        const uint64_t rest = total - 3 * g;
        const uint32_t valid = rest >= 3 ? 4u : uint32_t(rest) + 1u;  // characters that carry data
        uint32_t w = 0;
        for (uint32_t c = 0; c < 4; ++c) w |= (c < valid ? b64_char((v >> (18 - 6 * c)) & 63u) : uint32_t('=')) << (8 * c);
        out[g] = w;
    }
}

cudaError_t launch_vti_encode(const DeviceState &s, char *text, cudaStream_t st) {
    const uint64_t N = uint64_t(s.g.N);
    const VtiText L = vti_text_layout(N);
    const uint64_t groups = (8 + 3 * N * 4 + 2) / 3;
    const uint64_t want = (groups + 255) / 256;
    const unsigned bx = unsigned(want < uint64_t(8 * 148) ? want : uint64_t(8 * 148));
    k_vti_encode<<<dim3(bx, 4), 256, 0, st>>>(s.mom, N, text, L);
    return cudaGetLastError();
}

uint32_t conservation_blocks(const Geometry &g) {
    const size_t want = (size_t(g.N) + kRedThreads - 1) / kRedThreads;
    return uint32_t(want < size_t(kConsBlocksMax) ? want : size_t(kConsBlocksMax));
}

namespace {
template <class C>
cudaError_t conservation_dispatch(const DeviceState &s, int cur, double *partials, cudaStream_t st) {
    const C codec = make_codec<C>(s, cur);
    const uint32_t nb = conservation_blocks(s.g);
    if (s.g.boundary == kBoundaryPeriodic)
        k_conservation_partials<C, true><<<nb, kRedThreads, 0, st>>>(s, codec, partials);
    else
        k_conservation_partials<C, false><<<nb, kRedThreads, 0, st>>>(s, codec, partials);
    return cudaGetLastError();
}
template <class C>
cudaError_t check_finite_dispatch(const DeviceState &s, int cur, int *flag, cudaStream_t st) {
    const C codec = make_codec<C>(s, cur);
    const uint32_t nb = conservation_blocks(s.g);
    if (s.g.boundary == kBoundaryPeriodic)
        k_check_finite<C, true><<<nb, kRedThreads, 0, st>>>(s, codec, flag);
    else
        k_check_finite<C, false><<<nb, kRedThreads, 0, st>>>(s, codec, flag);
    return cudaGetLastError();
}
}  // namespace

cudaError_t launch_conservation(const DeviceState &s, int cur, double *partials, double *out5, cudaStream_t st) {
    cudaError_t e = s.g.storage == kStoreF16 ? conservation_dispatch<CodecF16>(s, cur, partials, st)
                                             : conservation_dispatch<CodecF32>(s, cur, partials, st);
    if (e != cudaSuccess) return e;
    k_conservation_final<<<1, kRedThreads, 0, st>>>(partials, int(conservation_blocks(s.g)), out5);
    return cudaGetLastError();
}

cudaError_t launch_check_finite(const DeviceState &s, int cur, int *flag, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(flag, 0, sizeof(int), st);
    if (e != cudaSuccess) return e;
    return s.g.storage == kStoreF16 ? check_finite_dispatch<CodecF16>(s, cur, flag, st)
                                    : check_finite_dispatch<CodecF32>(s, cur, flag, st);
}

cudaError_t launch_adj_terminal(const DeviceState &s, const float *M, const float *target, float *lam, double *J,
                                cudaStream_t st) {
    k_adj_terminal<<<grid3(s.g), dim3(kBX, kBY), 0, st>>>(s, M, target, lam, J);
    return cudaGetLastError();
}

namespace {
template <bool kPeriodic>
cudaError_t adj_relax(const DeviceState &s, const float *M, const uint8_t *flags, uint8_t *near_flags, const float *lam_in,
                      float *lmom, float *lf, float *lam_out, double *acc, const AdjObjective &obj, cudaStream_t st) {
    constexpr int kWarps = kAdjThreads / 32;
    const int plane = (adj_pieces_per_row(s.g) * (s.g.NY - 2) + kWarps - 1) / kWarps;
    const int list = int(adj_list_blocks(s.g, kAdjRelaxBlocks));
    return launch_overlapped(k_adj_relax<kPeriodic>, dim3(list + plane * (s.g.NZ - 2)), dim3(kAdjThreads), st, s, M, flags,
                             near_flags, lam_in, lmom, lf, lam_out, acc, obj, list, plane);
}
}  // namespace

cudaError_t launch_adj_relax(const DeviceState &s, const float *M, const uint8_t *flags, uint8_t *near_flags,
                             const float *lam_in, float *lmom, float *lf, float *lam_out, double *acc,
                             const AdjObjective &obj, cudaStream_t st) {
    return s.g.boundary == kBoundaryPeriodic
               ? adj_relax<true>(s, M, flags, near_flags, lam_in, lmom, lf, lam_out, acc, obj, st)
               : adj_relax<false>(s, M, flags, near_flags, lam_in, lmom, lf, lam_out, acc, obj, st);
}

cudaError_t launch_adj_near(const DeviceState &s, const float *M, const uint8_t *flags, const uint8_t *near_flags,
                            const float *lmom, const float *lf, float *lam_out, cudaStream_t st) {
    const unsigned n = adj_list_blocks(s.g, kAdjNearBlocks);
    return s.g.boundary == kBoundaryPeriodic
               ? launch_overlapped(k_adj_near<true>, dim3(n), dim3(kAdjThreads), st, s, M, flags, near_flags, lmom, lf, lam_out)
               : launch_overlapped(k_adj_near<false>, dim3(n), dim3(kAdjThreads), st, s, M, flags, near_flags, lmom, lf,
                                   lam_out);
}

cudaError_t launch_piece_flags(const DeviceState &s, const float *M, uint8_t *flags, cudaStream_t st) {
    constexpr int kWarps = kRedThreads / 32;
    const int pieces = adj_pieces_per_row(s.g) * (s.g.NY - 2);
    k_piece_flags<<<dim3((pieces + kWarps - 1) / kWarps, s.g.NZ - 2), kRedThreads, 0, st>>>(s, M, flags);
    return cudaGetLastError();
}

cudaError_t launch_adj_boundary(const DeviceState &s, int64_t step, const float *M, const float *Bt,
                                const float *lam_next, const float *lf, float *lmom, const float *LB_in,
                                float *LB_out, const float *bessel, int nb, double *dJdc, cudaStream_t st) {
    // one warp per block: a column is a long chain of dependent work, and blocks
    // of 8 warps put the 62 x 62 columns of a 64-wide jet on 16 SMs
    const dim3 block(32, 1), grid((s.g.NX + 31) / 32, s.g.NZ, 2);
    return launch_overlapped(k_adj_boundary, grid, block, st, s, step, M, Bt, lam_next, lf, lmom, LB_in, LB_out, bessel, nb,
                             dJdc);
}

cudaError_t launch_restore_outlet_state(const DeviceState &s, const float *src, float *psi, cudaStream_t st) {
    const dim3 block(32, 8), grid((s.g.NX + 31) / 32, (s.g.NZ + 7) / 8);
    k_restore_outlet_state<<<grid, block, 0, st>>>(s, src, psi);
    return cudaGetLastError();
}

cudaError_t launch_record_state(const DeviceState &s, const float *psi, float *rec, float *outlet, cudaStream_t st) {
    const unsigned blocks = unsigned(std::min<uint32_t>((s.g.N + 255) / 256, 4 * 148));
    return launch_overlapped(k_record_state, dim3(blocks), dim3(256), st, s, psi, rec, outlet);
}

cudaError_t launch_copy_outlet_state(const DeviceState &s, float *dst, cudaStream_t st) {
    const dim3 block(32, 8), grid((s.g.NX + 31) / 32, (s.g.NZ + 7) / 8);
    k_copy_outlet_state<<<grid, block, 0, st>>>(s, dst);
    return cudaGetLastError();
}

cudaError_t launch_adj_initial(const DeviceState &s, const float *M, const float *lam0, float *du0, cudaStream_t st) {
    k_adj_initial<<<grid3(s.g), dim3(kBX, kBY), 0, st>>>(s, M, lam0, du0);
    return cudaGetLastError();
}

}  // namespace mcg
