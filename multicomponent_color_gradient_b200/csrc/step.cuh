// step.cuh - device code the kernels of the step share: storage codecs, pull
// maps, moments, collision, radial statistics and the jet boundary columns.
#pragma once

#include <type_traits>
#include <cuda_fp16.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>

#include "kernels.cuh"
#include "lattice.cuh"

namespace mcg {
namespace {

constexpr unsigned kFull = 0xffffffffu;

// ------------------------------------------------------------------ storage codecs

// Float32 element per (direction, node): the pair (fr, fb), so a pull or a
// store of both colours is one 8-byte access.
struct CodecF32 {
    using Elem = float2;
    static constexpr int kGroupSlots = 3;
    static constexpr bool kSumDiff = false;  // pulls form sum fr and sum fb (reference order)
    // store_bulk takes P_i itself (collision_poly without a shift)
    static constexpr bool kShiftPoly = false;
    __device__ __forceinline__ float poly_shift() const { return 0.0f; }
    const float2 *__restrict__ rd;
    float2 *__restrict__ wr;
    int px;  // row pitch
    int l2_resident;
    // store through `wrow` = the node's row in the written buffer, offset by x
    template <int I>
    __device__ __forceinline__ void store_row(float2 *wrow, float r, float b) const {
        wrow[slot_pair(I) * px] = make_float2(r, b);
    }
    // bulk node: fr_i = aR w_i P_i, fb_i = aB w_i P_i (lbm.cuh:216-247)
    __device__ __forceinline__ void store_bulk(float2 *wrow, float aR, float aB, const float (&P)[kQ]) const {
        static_for<kQ>([&](auto I) {
            constexpr int i = decltype(I)::value;
            // both colours in one packed multiply and one store
            wrow[slot_pair(i) * px] = __fmul2_rn(make_float2(aR * Dir<i>::w, aB * Dir<i>::w), make_float2(P[i], P[i]));
        });
    }
    // pull in two halves: the raw pair at `p` = the source node's element of
    // direction I, then the pair the colour sums add and the total gi
    using Raw = float2;
    template <int I>
    __device__ __forceinline__ Raw load_raw(const float2 *p) const {
        // a plain load, not the read-only path: the split step's launches are
        // resident before the launch that writes these elements has ended
        float2 v;
        asm("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
        return v;
    }
    template <int I>
    __device__ __forceinline__ Raw load_raw(const float2 *p, uint64_t policy) const {
        float2 v;
        asm("ld.global.L2::cache_hint.v2.f32 {%0, %1}, [%2], %3;" : "=f"(v.x), "=f"(v.y) : "l"(p), "l"(policy));
        return v;
    }
    template <int I>
    __device__ __forceinline__ float2 decode(Raw v, float &gi) const {
        gi = v.x + v.y;
        return v;
    }
    template <int I>
    __device__ __forceinline__ void store(size_t row, int x, float r, float b) const {
        wr[row + size_t(slot_pair(I)) * px + x] = make_float2(r, b);
    }
    __device__ __forceinline__ static void store_to(void *buf, const Geometry &g, int i, int x, int y, int z, float r,
                                                    float b, float) {
        static_cast<float2 *>(buf)[pop_index(g, slot_pair(i), x, y, z)] = make_float2(r, b);
    }
    template <int I>
    __device__ __forceinline__ Elem pack(float r, float b) const {
        return make_float2(r, b);
    }
    // the colour pair of a pulled element
    template <int I>
    __device__ __forceinline__ void unpack(Raw v, float &r, float &b) const {
        r = v.x;
        b = v.y;
    }
};

// F16 word per (direction, node): x = g/w_i - rho0 (total offset by the rest
// equilibrium and scaled by 1/w_i), y = q, the minority-colour fraction
// 2 min(fr,fb)/g carrying the sign of fr-fb.  Pure nodes store q = +-0
// exactly, so a single-colour region keeps exactly zero of the other colour.
__device__ __forceinline__ __half2 f16_encode(float r, float b, float inv_w, float rho0) {
    // rounded operation by operation, so that every kernel that inlines it
    // (the jet boundary is written from several) gives the same word
    const float g = __fadd_rn(r, b);
    const float h0 = __fsub_rn(__fmul_rn(g, inv_w), rho0);
    const float mn = fminf(r, b);
    float q = (g > 0.0f) ? __fdividef(2.0f * mn, g) : 0.0f;
    q = copysignf(fmaxf(q, 0.0f), r - b);
    return __floats2half2_rn(h0, q);
}
__device__ __forceinline__ void f16_decode(__half2 h, float w, float rho0, float &r, float &b) {
    const float2 v = __half22float2(h);
    const float g = w * (rho0 + v.x);
    const float minor = 0.5f * g * fabsf(v.y);
    const bool red_major = !signbit(v.y);
    r = red_major ? g - minor : minor;
    b = red_major ? minor : g - minor;
}

struct CodecF16 {
    using Elem = __half2;
    static constexpr int kGroupSlots = 3;
    static constexpr bool kSumDiff = true;  // pulls form sum (fr+fb) and sum (fr-fb)
    // store_bulk takes P_i - rho0, formed by collision_poly's constant term
    static constexpr bool kShiftPoly = true;
    __device__ __forceinline__ float poly_shift() const { return rho0; }
    const __half2 *__restrict__ rd;
    __half2 *__restrict__ wr;
    int px;  // row pitch
    int l2_resident;
    float rho0;
    template <int I>
    __device__ __forceinline__ void store_row(__half2 *wrow, float r, float b) const {
        wrow[slot_pair(I) * px] = f16_encode(r, b, 1.0f / Dir<I>::w, rho0);
    }
    // bulk node: every direction splits its total g_i = w_i P_i in the same
    // proportion aR : aB, so the word is (P_i - rho0, q) (Ps = P - rho0 from
    // collision_poly) with one signed
    // minority fraction q = 2 min(aR, aB) for the node - the value f16_encode
    // forms from fr_i, fb_i up to float rounding, and exactly +-0 at a pure
    // node (aB or aR is exactly 0 there).
    __device__ __forceinline__ void store_bulk(__half2 *wrow, float aR, float aB, const float (&Ps)[kQ]) const {
        const float q = copysignf(fmaxf(2.0f * fminf(aR, aB), 0.0f), aR - aB);
        static_for<kQ>([&](auto I) {
            constexpr int i = decltype(I)::value;
            wrow[slot_pair(i) * px] = __floats2half2_rn(Ps[i], q);
        });
    }
    // pull in two halves: the raw word, then the total g = fr + fb and the
    // difference d = fr - fb.  With q the signed minority fraction, fr - fb =
    // g (1 - q) when red is the majority and -g (1 + q) otherwise, i.e.
    // g (sign(q) - q).
    // The load asks L2 to fetch 256-byte blocks on a miss: the words
    // of a pulled row segment are then in L2 for the neighbouring warps'
    // loads (measured +0.3 % on the 128x256x128 jet, +1.2 % on 256-column
    // rows; no change in float32).
    using Raw = __half2;
    template <int I>
    __device__ __forceinline__ Raw load_raw(const __half2 *p) const {
        uint32_t u;
        asm("ld.global.L2::256B.b32 %0, [%1];" : "=r"(u) : "l"(p));
        __half2 h;
        memcpy(&h, &u, sizeof h);
        return h;
    }
    template <int I>
    __device__ __forceinline__ Raw load_raw(const __half2 *p, uint64_t policy) const {
        uint32_t u;
        asm("ld.global.L2::cache_hint.L2::256B.b32 %0, [%1], %2;" : "=r"(u) : "l"(p), "l"(policy));
        __half2 h;
        memcpy(&h, &u, sizeof h);
        return h;
    }
    template <int I>
    __device__ __forceinline__ float2 decode(Raw h, float &gi) const {
        const float2 v = __half22float2(h);
        const float gs = fmaf(Dir<I>::w, v.x, Dir<I>::w * rho0);
        gi = gs;
        return make_float2(gs, fmaf(-gs, v.y, copysignf(gs, v.y)));
    }
    template <int I>
    __device__ __forceinline__ void store(size_t row, int x, float r, float b) const {
        wr[row + size_t(slot_pair(I)) * px + x] = f16_encode(r, b, 1.0f / Dir<I>::w, rho0);
    }
    __device__ __forceinline__ static void store_to(void *buf, const Geometry &g, int i, int x, int y, int z, float r,
                                                    float b, float rho0) {
        static_cast<__half2 *>(buf)[pop_index(g, slot_pair(i), x, y, z)] = f16_encode(r, b, 1.0f / dir_w(i), rho0);
    }
    template <int I>
    __device__ __forceinline__ Elem pack(float r, float b) const {
        return f16_encode(r, b, 1.0f / Dir<I>::w, rho0);
    }
    template <int I>
    __device__ __forceinline__ void unpack(Raw h, float &r, float &b) const {
        f16_decode(h, Dir<I>::w, rho0, r, b);
    }
};

template <class C>
__host__ __device__ C make_codec(const DeviceState &s, int cur);
template <>
__host__ __device__ CodecF32 make_codec<CodecF32>(const DeviceState &s, int cur) {
    return CodecF32{static_cast<const float2 *>(s.pops[cur]), static_cast<float2 *>(s.pops[cur ^ 1]), s.g.px,
                    s.l2_resident};
}
template <>
__host__ __device__ CodecF16 make_codec<CodecF16>(const DeviceState &s, int cur) {
    return CodecF16{static_cast<const __half2 *>(s.pops[cur]), static_cast<__half2 *>(s.pops[cur ^ 1]), s.g.px,
                    s.l2_resident, s.ph.f16_rho0};
}

// ------------------------------------------------------------------ helpers

__device__ __forceinline__ float psi_of(float a, float b) { return (a - b) / (a + b); }  // mathUtilities.cuh:24-28

__device__ __forceinline__ float clamp01(float v) { return fminf(fmaxf(v, 0.0f), 1.0f); }

// Relaxation rate at height y (mathUtilities.cuh:56-90); constant when K == 0.
__device__ __forceinline__ float omega_at(const Physics &ph, int y) {
    if (!ph.sponge) return ph.omega;
    const float s = clamp01((float(y) - ph.sponge_y_start) * ph.sponge_inv_width);
    const float nus = ph.nu * (1.0f + ph.sponge_K * (s * s * s));
    return 1.0f / (0.5f + nus * kInvCs2);
}

__device__ __forceinline__ bool is_jet_column(const Physics &ph, int x, int z) {  // mathUtilities.cuh:14-21
    const float dx = float(x) - ph.jet_x0, dz = float(z) - ph.jet_z0;
    return __fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dz, dz)) <= ph.jet_r2;
}

// Inlet velocity of jet column (x, z): the top-hat U (boundary_conditions.cuh:62),
// times the column's profile multiplier when a radial profile is set, times
// the seeded perturbation when inlet_noise != 0.
__device__ __forceinline__ float inlet_velocity(const DeviceState &s, int64_t step, int x, int z) {
    const Physics &ph = s.ph;
    float U = ph.jet_velocity;
    if (s.inlet_profile) U *= s.inlet_profile[x + s.g.NX * z];
    if (ph.inlet_noise == 0.0f) return U;
    const float u = hash_uniform(ph.seed, 0x1A1E7ull ^ uint64_t(step), uint64_t(x), uint64_t(z));
    return __fmul_rn(U, __fadd_rn(1.0f, __fmul_rn(__fsub_rn(2.0f * u, 1.0f), ph.inlet_noise)));
}

__host__ __device__ __forceinline__ int wrap_interior(int v, int n) { return v == 0 ? n - 2 : (v == n - 1 ? 1 : v); }

// Pull sources of interior node (x,y,z).  x and z are periodic over the
// interior through the ghost shell (the push side wraps with
// bounds.cuh:23-60); y sources on a ghost plane are the boundary's slots and
// are not wrapped laterally (boundary writes are unwrapped,
// boundary_conditions.cuh:73,137); in the periodic box y wraps too.
template <class C>
struct PullMap {
    long long own_row;              // offset of row (y,z)
    long long step_y, step_z;       // row offsets of y+1, z+1
    long long wzp, wzm, wyp, wym;   // wrap corrections (row offsets)
    int wxp, wxm;                   // wrap corrections (x)
    int px;                         // row pitch
    bool gy_p, gy_m;
    __device__ __forceinline__ PullMap(const Geometry &g, int x, int y, int z, bool periodic) {
        px = g.px;
        own_row = (long long)pop_row(g, y, z);
        step_y = (long long)g.slots * g.px;
        step_z = step_y * g.NY;
        wxp = (x == 1) ? (g.NX - 2) : 0;
        wxm = (x == g.NX - 2) ? -(g.NX - 2) : 0;
        wzp = (z == 1) ? step_z * (g.NZ - 2) : 0;
        wzm = (z == g.NZ - 2) ? -step_z * (g.NZ - 2) : 0;
        wyp = (periodic && y == 1) ? step_y * (g.NY - 2) : 0;
        wym = (periodic && y == g.NY - 2) ? -step_y * (g.NY - 2) : 0;
        gy_p = !periodic && y == 1;
        gy_m = !periodic && y == g.NY - 2;
    }
    // offset of the group segment of direction I's source row, and source x
    template <int I>
    __device__ __forceinline__ void src(int x, size_t &grow, int &xs) const {
        using D = Dir<I>;
        const long long o = own_row - D::cy * step_y - D::cz * step_z;
        bool ghost = false;
        if constexpr (D::cy == 1) ghost = gy_p;
        if constexpr (D::cy == -1) ghost = gy_m;
        int xc = 0;
        long long oc = 0;
        if constexpr (D::cx == 1) xc = wxp;
        if constexpr (D::cx == -1) xc = wxm;
        if constexpr (D::cz == 1) oc = wzp;
        if constexpr (D::cz == -1) oc = wzm;
        if (ghost) {
            xc = 0;
            oc = 0;
        }
        if constexpr (D::cy == 1) oc += wyp;
        if constexpr (D::cy == -1) oc += wym;
        grow = size_t(o + oc) + size_t(dir_group(I) * C::kGroupSlots) * size_t(px);
        xs = x - D::cx + xc;
    }
    // the source's first slot of direction I (red for float32)
    template <int I>
    __device__ __forceinline__ const typename C::Elem *ptr(const C &codec, int x) const {
        size_t grow;
        int xs;
        src<I>(x, grow, xs);
        return codec.rd + grow + size_t(dir_cx(I) + 1) * size_t(px) + xs;
    }
};

// Pull sources of a node in rows y = 2 .. NY-3: no source lies on a y ghost
// plane or wraps in y, so the only corrections are the z wrap, the same for
// all directions of one cz, and the x wrap of columns 1 and NX-2.  One base
// pointer per cz (z wrap applied, offset by x) then serves nine directions,
// each a load at a constant offset from it, plus the x wrap for cx = +-1.
// The addresses are those of PullMap.
template <class C>
struct FastPullMap {
    const typename C::Elem *base[3];  // cz = -1, 0, +1
    long long step_y;
    int xwp, xwm;  // x wrap of cx = +1 (column 1) and cx = -1 (column NX-2)
    int px;
    __device__ __forceinline__ FastPullMap(const Geometry &g, const C &codec, int x, int y, int z) {
        px = g.px;
        step_y = (long long)g.slots * g.px;
        const long long step_z = step_y * g.NY;
        const typename C::Elem *own = codec.rd + pop_row(g, y, z) + x;
        base[0] = own + step_z + ((z == g.NZ - 2) ? -step_z * (g.NZ - 2) : 0);  // cz = -1: source plane z+1
        base[1] = own;
        base[2] = own - step_z + ((z == 1) ? step_z * (g.NZ - 2) : 0);          // cz = +1: source plane z-1
        xwp = (x == 1) ? (g.NX - 2) : 0;
        xwm = (x == g.NX - 2) ? -(g.NX - 2) : 0;
    }
    template <int I>
    __device__ __forceinline__ const typename C::Elem *ptr(const C &, int) const {
        using D = Dir<I>;
        const typename C::Elem *b = base[D::cz + 1];
        if constexpr (D::cx == 1) b += xwp;
        if constexpr (D::cx == -1) b += xwm;
        return b + (-(long long)D::cy * step_y + (long long)(dir_group(I) * C::kGroupSlots + D::cx + 1) * px - D::cx);
    }
};

// ------------------------------------------------------------------ per-node pieces

// First of the opposite pairs (i, i+1), i = 2p+1, whose direction has a
// nonzero c_a c_b (a == b: c_a != 0); the moment sums start there.
__host__ __device__ constexpr int dir_comp(int i, int a) { return a == 0 ? dir_cx(i) : (a == 1 ? dir_cy(i) : dir_cz(i)); }
__host__ __device__ constexpr int first_pair(int a, int b) {
    for (int p = 0; p < (kQ - 1) / 2; ++p)
        if (dir_comp(2 * p + 1, a) * dir_comp(2 * p + 1, b) != 0) return p;
    return (kQ - 1) / 2;
}
template <bool kFirst>
__device__ __forceinline__ void moment_add(float &acc, float v) {
    if constexpr (kFirst)
        acc = v;
    else
        acc += v;
}

// A node's pull in two halves: pull_issue loads the 27 raw elements (float2
// or half2) into registers; densities_from / moments_from decode and sum them.
// Between the two a warp can do other work while the loads are in flight.
template <class C>
struct RawPull {
    typename C::Raw v[kQ];
};

template <class C, class Map>
__device__ __forceinline__ void pull_issue_map(const Map &pm, const C &codec, int x, RawPull<C> &raw) {
    static_for<kQ>([&](auto I) {
        constexpr int i = decltype(I)::value;
        raw.v[i] = codec.template load_raw<i>(pm.template ptr<i>(codec, x));
    });
}

// Colour densities only of interior node (x,y,z): the colour sums of
// pull_moments below in the same order (direction index), so psi formed from
// either is bit-identical.  Nodes whose psi is all that is needed (halo rows
// and planes of a tile) take this.
// The pulled pairs come from `src.get<I>(gi)`: decoded from words already in
// registers (RawSource) or loaded and decoded on the spot (DecodedPull).
template <class C>
struct RawSource {
    const C &codec;
    const RawPull<C> &raw;
    template <int I>
    __device__ __forceinline__ float2 get(float &gi) const {
        return codec.template decode<I>(raw.v[I], gi);
    }
};

template <class Src>
__device__ __forceinline__ void densities_from(const Src &src, float &rr, float &rb) {
    using C = std::remove_cv_t<std::remove_reference_t<decltype(src.codec)>>;
    float2 sum = make_float2(0.f, 0.f);  // (sum fr, sum fb); C::kSumDiff: (sum fr+fb, sum fr-fb)
    static_for<kQ>([&](auto I) {
        constexpr int i = decltype(I)::value;
        float gi;
        sum = __fadd2_rn(sum, src.template get<i>(gi));  // both colours in one packed add
    });
    if constexpr (C::kSumDiff) {
        rr = 0.5f * (sum.x + sum.y);
        rb = 0.5f * (sum.x - sum.y);
    } else {
        rr = sum.x;
        rb = sum.y;
    }
}

// Pull the 54 populations of interior node (x,y,z) and form its moments
// (lbm.cuh:106-164: densities, velocity, second-order Hermite moments minus
// the equilibrium part).  The loads are issued in direction-index order
// (measured: issuing them group by group was 5-20 % slower) into registers;
// the moments are then formed from the sums and differences of opposite
// pairs, about 100 operations instead of one multiply-add per direction and
// moment.
template <class Src>
__device__ __forceinline__ NodeMoments moments_from(const Src &src) {
    using C = std::remove_cv_t<std::remove_reference_t<decltype(src.codec)>>;
    float2 sum = make_float2(0.f, 0.f);  // (sum fr, sum fb); C::kSumDiff: (sum fr+fb, sum fr-fb)
    float gv[kQ];                        // totals fr + fb per direction
    static_for<kQ>([&](auto I) {
        constexpr int i = decltype(I)::value;
        sum = __fadd2_rn(sum, src.template get<i>(gv[i]));
    });
    // Moments over the 13 opposite pairs (i, i+1), i odd: d = g_i - g_opp
    // carries the first moments, s = g_i + g_opp the second.  Near equilibrium
    // the two members of a pair are within a factor of two, so d is exact and
    // the momentum sums add small numbers.  The diagonal stresses take s times
    // the Hermite constants H_aa = c_a^2 - cs^2 (multiply-adds, as lbm.cuh
    // forms them): the rounding of the two constants cancels at rest, whereas
    // sum c_a^2 g - rho * float(1/3) is biased by 1e-8 rho at every node and
    // step, which accumulated to 3x the float32 error of the reference's
    // arithmetic in the kinetic energy.  (Summing whole (cy, cz) groups
    // before differencing lost digits of the momentum.)
    float Jx, Jy, Jz, Qxy, Qxz, Qyz;
    float Axx = gv[0] * Dir<0>::Hxx, Ayy = gv[0] * Dir<0>::Hyy, Azz = gv[0] * Dir<0>::Hzz;
    static_for<(kQ - 1) / 2>([&](auto P) {
        constexpr int p = decltype(P)::value, i = 2 * p + 1;
        using D = Dir<i>;
        static_assert(Dir<i + 1>::cx == -D::cx && Dir<i + 1>::cy == -D::cy && Dir<i + 1>::cz == -D::cz,
                      "directions i, i+1 (i odd) are opposite");
        const float d = gv[i] - gv[i + 1], sp = gv[i] + gv[i + 1];
        if constexpr (D::cx != 0) moment_add<p == first_pair(0, 0)>(Jx, D::cx > 0 ? d : -d);
        if constexpr (D::cy != 0) moment_add<p == first_pair(1, 1)>(Jy, D::cy > 0 ? d : -d);
        if constexpr (D::cz != 0) moment_add<p == first_pair(2, 2)>(Jz, D::cz > 0 ? d : -d);
        Axx = fmaf(sp, D::Hxx, Axx);
        Ayy = fmaf(sp, D::Hyy, Ayy);
        Azz = fmaf(sp, D::Hzz, Azz);
        if constexpr (D::cx * D::cy != 0) moment_add<p == first_pair(0, 1)>(Qxy, D::cx * D::cy > 0 ? sp : -sp);
        if constexpr (D::cx * D::cz != 0) moment_add<p == first_pair(0, 2)>(Qxz, D::cx * D::cz > 0 ? sp : -sp);
        if constexpr (D::cy * D::cz != 0) moment_add<p == first_pair(1, 2)>(Qyz, D::cy * D::cz > 0 ? sp : -sp);
    });
    float sumr = sum.x, sumb = sum.y;
    if constexpr (C::kSumDiff) {
        sumr = 0.5f * (sum.x + sum.y);
        sumb = 0.5f * (sum.x - sum.y);
    }
    NodeMoments m;
    const float rho = sumr + sumb;
    const float inv = 1.0f / rho;
    m.rr = sumr;
    m.rb = sumb;
    m.ux = Jx * inv;
    m.uy = Jy * inv;
    m.uz = Jz * inv;
    m.pxx = Axx - rho * m.ux * m.ux;
    m.pxy = Qxy - rho * m.ux * m.uy;
    m.pyy = Ayy - rho * m.uy * m.uy;
    m.pyz = Qyz - rho * m.uy * m.uz;
    m.pzz = Azz - rho * m.uz * m.uz;
    m.pxz = Qxz - rho * m.ux * m.uz;
    return m;
}

// Rows 2 .. NY-3 take FastPullMap, the two edge rows PullMap (ghost planes,
// y wrap); y is uniform over a warp at every call site, so the branch is too.
template <class C, bool kPeriodic>
__device__ __forceinline__ void pull_issue(const Geometry &g, const C &codec, int x, int y, int z, RawPull<C> &raw) {
    if (y >= 2 && y <= g.NY - 3)
        pull_issue_map(FastPullMap<C>(g, codec, x, y, z), codec, x, raw);
    else
        pull_issue_map(PullMap<C>(g, x, y, z, kPeriodic), codec, x, raw);
}
// One-piece pulls: each load is decoded where it is issued, which lets the
// compiler consume the words as they arrive (measured 2 % faster at 80
// registers than issuing all of them first).  The arithmetic and its order
// are the same either way, so the results are bit-identical.
template <class C, class Map>
struct DecodedPull {
    const Map &pm;
    const C &codec;
    int x;
    template <int I>
    __device__ __forceinline__ float2 get(float &gi) const {
        return codec.template decode<I>(codec.template load_raw<I>(pm.template ptr<I>(codec, x)), gi);
    }
};
// The same, of a buffer that fits L2: the pulled sectors, which the step reads
// once, leave L2 before those that it writes, which the next step reads.
// 64^3 19.9 -> 19.3 us, 97 x 75 x 131 float16 54.9 -> 52.8.  In larger grids the
// sectors that neighbouring warps share would leave before they have met
// (128x256x128 297 -> 304 us, float16 at 256x512x256 1221 -> 1283).
template <class C, class Map>
struct DecodedPullOnce {
    const Map &pm;
    const C &codec;
    int x;
    uint64_t first;
    template <int I>
    __device__ __forceinline__ float2 get(float &gi) const {
        return codec.template decode<I>(codec.template load_raw<I>(pm.template ptr<I>(codec, x), first), gi);
    }
};
template <class C, class Map>
__device__ __forceinline__ void pull_densities_map(const Map &pm, const C &codec, int x, float &rr, float &rb) {
    densities_from(DecodedPull<C, Map>{pm, codec, x}, rr, rb);
}
template <class C, class Map>
__device__ __forceinline__ NodeMoments pull_moments_map(const Map &pm, const C &codec, int x) {
    if (codec.l2_resident) {
        uint64_t first;
        asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(first));
        return moments_from(DecodedPullOnce<C, Map>{pm, codec, x, first});
    }
    return moments_from(DecodedPull<C, Map>{pm, codec, x});
}
template <class C, bool kPeriodic>
__device__ __forceinline__ void pull_densities(const Geometry &g, const C &codec, int x, int y, int z, float &rr,
                                               float &rb) {
    if (y >= 2 && y <= g.NY - 3)
        pull_densities_map(FastPullMap<C>(g, codec, x, y, z), codec, x, rr, rb);
    else
        pull_densities_map(PullMap<C>(g, x, y, z, kPeriodic), codec, x, rr, rb);
}
template <class C, bool kPeriodic>
__device__ __forceinline__ NodeMoments pull_moments(const Geometry &g, const C &codec, int x, int y, int z) {
    if (y >= 2 && y <= g.NY - 3) return pull_moments_map(FastPullMap<C>(g, codec, x, y, z), codec, x);
    return pull_moments_map(PullMap<C>(g, x, y, z, kPeriodic), codec, x);
}

// Launches that follow one another on a stream overlap by programmatic dependent
// launch: each starts while the one before it drains, and everything before the
// wait reads only kernel parameters.  Every thread of a kernel launched this way
// waits, so that the end of a launch is also the end of all before it.
__device__ __forceinline__ void wait_for_previous_launch() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// The same, renewing the pointers behind the wait, so that no load of theirs can
// be moved above it.
template <class C>
__device__ __forceinline__ void wait_for_previous_launch(C &codec, const float *&psi) {
    wait_for_previous_launch();
    auto rd = codec.rd;
    auto wr = codec.wr;
    asm volatile("" : "+l"(rd), "+l"(wr), "+l"(psi)::"memory");
    codec.rd = rd;
    codec.wr = wr;
}
__device__ __forceinline__ void allow_next_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Blocks up to which a launch lets the next one start only when it runs itself:
// half of the blocks of k_step_pull that fit the chip, so that it and the next
// one fit together.  Launches that each let the next one start at once go on to
// pile up, waiting, several deep, and fill the SMs unevenly (k_step_pull: 32x48x32
// jet 8.6 us a step so and 10.4 at once, float16 24x40x24 jet 7.9 and 11.2; the
// adjoint kernels: a 32x48x32 jet gradient 1500 us and 1605).  For larger ones at
// once is the faster: the next launch's blocks fill the last wave (float16
// 128x256x128 jet 168.8 us a step against 172.7).
constexpr unsigned kSmallLaunch = 148 * 7 / 2;

__device__ __forceinline__ void wait_then_allow_if_small() {
    const bool small = gridDim.x * gridDim.y * gridDim.z <= kSmallLaunch;
    if (!small) allow_next_launch();
    wait_for_previous_launch();
    if (small) allow_next_launch();
}

template <class... P, class... A>
cudaError_t launch_overlapped(void (*kernel)(P...), dim3 grid, dim3 block, cudaStream_t st, const A &...args) {
    cudaLaunchAttribute overlap{};
    overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    overlap.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.stream = st;
    cfg.attrs = &overlap;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// Columns of a lattice row whose slots a kernel that relaxes the row stores:
// the interior ones, ghost column 0 and the columns that complete the last 64
// bytes (the pitch allowing).  Nothing reads the ghost and pad columns of an
// interior row (pulls wrap over the interior), but a 32-byte sector written in
// part makes L2 fetch the rest of it from HBM: with columns 0 and NX-1 left
// out, a copy with the step's access pattern ran at 0.83 (float32) and 0.73
// (float16) of the measured copy peak on 128x256x128, with them at 1.00.
template <class C>
__host__ __device__ __forceinline__ int store_columns(const Geometry &g) {
    constexpr int kPiece = 64 / int(sizeof(typename C::Elem));
    const int c = (g.NX - 1 + kPiece - 1) / kPiece * kPiece;
    return c < g.px ? c : g.px;
}

// Pieces of 32 columns that hold the stored columns of a row.
template <class C>
__host__ __device__ __forceinline__ int pieces_per_row(const Geometry &g) {
    return (store_columns<C>(g) + 31) / 32;
}

// Flag of piece w of a row from the lanes that hold interface nodes: bit 0 any,
// bit 1 its first interior column, bit 2 its last, bits 4 to 7 its quarters of 8
// columns.
__device__ __forceinline__ uint8_t piece_flag(const Geometry &g, int w, unsigned lanes) {
    const int first = w == 0 ? 1 : 0, last = min(31, g.NX - 2 - 32 * w);
    unsigned f = (lanes != 0 ? 1u : 0u) | (((lanes >> first) & 1u) << 1) | (((lanes >> last) & 1u) << 2);
#pragma unroll
    for (int q = 0; q < 4; ++q) f |= ((lanes >> (8 * q)) & 0xffu) != 0 ? 16u << q : 0u;
    return uint8_t(f);
}

// A node whose interface indicator (lbm.cuh:214-216) is at most 1e-4 takes the
// bulk branch, which reads no psi.  A NaN is not bulk.
__device__ __forceinline__ bool is_bulk(float rr, float rb) {
    const float invrT = 1.0f / (rr + rb);
    return 4.0f * rr * rb * invrT * invrT <= 1e-4f;
}
// Relax one node and store its 54 post-collision values (lbm.cuh:184-293).
// The bulk part feq + (1-omega) fneq of all 27 directions comes from
// collision_poly (lattice.cuh).  At interface nodes the perturbation Omega2
// (even in c: one evaluation per opposite pair) and the recolouring Delta
// (odd) are added per direction.  psi_at(cx,cy,cz) returns the neighbour's
// psi, read unwrapped like forces.cuh:31 (ghost psi is what the reference
// sees there).
// kBulk: the caller knows that the node is_bulk (psi_at is not called).
template <bool kBulk, class C, class PsiAt>
__device__ __forceinline__ void collide_node(const Geometry &g, const Physics &ph, const C &codec, size_t row, int x,
                                             int y, int z, const NodeMoments &m, PsiAt &&psi_at) {
    const NeqTerms n = make_neq(m.pxx, m.pxy, m.pyy, m.pyz, m.pzz, m.pxz, m.ux, m.uy, m.uz);
    const float rr = m.rr, rb = m.rb;
    const float rT = rr + rb;
    const float invrT = 1.0f / rT;
    const float aR = rr * invrT, aB = rb * invrT;
    const float oms = 1.0f - omega_at(ph, y);
    float P[kQ];  // P_i - shift, shift = 0 (float32) or rho0 (float16)
    const float shift = codec.poly_shift();
    collision_poly(rT, m.ux, m.uy, m.uz, n, oms, P, shift);
    typename C::Elem *const wrow = codec.wr + row + x;
    if (kBulk || is_bulk(rr, rb)) {  // bulk (lbm.cuh:216-247)
        codec.store_bulk(wrow, aR, aB, P);
        return;
    }
    auto full = [&](float p) {  // P_i from P_i - shift
        if constexpr (C::kShiftPoly)
            return p + shift;
        else
            return p;
    };
    // interface (lbm.cuh:249-292): colour gradient over the 26 neighbours
    float sx = 0.f, sy = 0.f, sz = 0.f;
    static_for<kQ - 1>([&](auto I) {
        constexpr int i = decltype(I)::value + 1;
        using D = Dir<i>;
        const float wp = D::w * psi_at(D::cx, D::cy, D::cz);
        if constexpr (D::cx == 1) sx += wp;
        if constexpr (D::cx == -1) sx -= wp;
        if constexpr (D::cy == 1) sy += wp;
        if constexpr (D::cy == -1) sy -= wp;
        if constexpr (D::cz == 1) sz += wp;
        if constexpr (D::cz == -1) sz -= wp;
    });
    InterfaceTerms t;
    t.Fx = kInvCs2 * sx;
    t.Fy = kInvCs2 * sy;
    t.Fz = kInvCs2 * sz;
    t.absF = sqrtf(t.Fx * t.Fx + t.Fy * t.Fy + t.Fz * t.Fz);
    t.has_dir = !(t.absF <= 1.0e-4f);
    t.inv_absF = 1.0f / t.absF;
    t.inv_absF2 = 1.0f / (t.absF * t.absF);
    t.Ah_absF = ph.Ah * t.absF;
    t.coeff_rho = ph.beta * ((rr * rb) / (rT * rT)) * rT;
    {
        const float g0 = Dir<0>::w * full(P[0]) + omega2<0>(t);
        codec.template store_row<0>(wrow, aR * g0, aB * g0);
    }
    static_for<(kQ - 1) / 2>([&](auto Q) {
        constexpr int i = 2 * decltype(Q)::value + 1;
        const float o2 = omega2<i>(t);  // even: the same for i and its opposite
        const float gi = Dir<i>::w * full(P[i]) + o2, go = Dir<i + 1>::w * full(P[i + 1]) + o2;
        const float d = recolour<i>(t);  // odd: -d for the opposite
        codec.template store_row<i>(wrow, aR * gi + d, aB * gi - d);
        codec.template store_row<i + 1>(wrow, aR * go - d, aB * go + d);
    });
}

// ------------------------------------------------------------------ radial statistics

// Warp-collective: one warp = 32 consecutive x at fixed (y,z).  Lanes with the
// same radial bin form contiguous runs once split by the side of the jet axis
// (the bin is monotone in |x - x0| on each side), so a segmented scan leaves
// each run's sums in its last lane, which issues one float64 atomic per sum.
// Counts are not accumulated per node: every sample adds the fixed number of
// interior columns of a bin, so they are materialised on read.
__device__ __forceinline__ void radial_accumulate_warp(const DeviceState &s, int x, int y, int z, bool active,
                                                       float ux, float uy, float uz) {
    const Physics &ph = s.ph;
    const int lane = threadIdx.x & 31;
    unsigned key = 0xffffffffu;
    float v0 = 0.f, v1 = 0.f, v2 = 0.f, v3 = 0.f, v4 = 0.f;
    if (active) {
        const float dx = float(x) - ph.jet_x0, dz = float(z) - ph.jet_z0;
        const float r = sqrtf(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dz, dz)));
        const unsigned rb = unsigned(r);
        if (rb < unsigned(ph.NRB)) {
            key = (rb << 1) | (dx < 0.0f ? 1u : 0u);
            float ur = 0.0f;
            // rounded as written, whatever kernel this is part of
            if (r > 1.0e-12f) ur = fmaf(ux, dx, __fmul_rn(uz, dz)) / r;
            v0 = uy;
            v1 = __fmul_rn(uy, uy);
            v2 = ur;
            v3 = __fmul_rn(ur, ur);
            v4 = __fmul_rn(ur, uy);
        }
    }
    if (__all_sync(kFull, key == 0xffffffffu)) return;
    // run sums in float32 (a run is at most 32 nodes of one row); the run
    // totals go into the float64 accumulators
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const unsigned ok = __shfl_up_sync(kFull, key, d);
        const float o0 = __shfl_up_sync(kFull, v0, d);
        const float o1 = __shfl_up_sync(kFull, v1, d);
        const float o2 = __shfl_up_sync(kFull, v2, d);
        const float o3 = __shfl_up_sync(kFull, v3, d);
        const float o4 = __shfl_up_sync(kFull, v4, d);
        if (lane >= d && ok == key) {
            v0 += o0; v1 += o1; v2 += o2; v3 += o3; v4 += o4;
        }
    }
    const unsigned next = __shfl_down_sync(kFull, key, 1);
    const bool tail = (lane == 31) || (next != key);
    if (tail && key != 0xffffffffu) {
        const size_t M = size_t(s.g.NY) * ph.NRB;
        const size_t mi = size_t(y) * ph.NRB + (key >> 1);
        atomicAdd(s.radial + mi, double(v0));
        atomicAdd(s.radial + M + mi, double(v1));
        atomicAdd(s.radial + 2 * M + mi, double(v2));
        atomicAdd(s.radial + 3 * M + mi, double(v3));
        atomicAdd(s.radial + 4 * M + mi, double(v4));
    }
}

// ------------------------------------------------------------------ boundary arithmetic

// The jet boundary columns are written from every fused kernel (and from
// k_boundary).  Their arithmetic is rounded operation by operation (no
// contraction into fused multiply-adds, which the compiler chooses per
// kernel), so that every kernel writes the same bits.  Same formulas as
// make_eq, make_neq, feq and fneq (lbm.cuh:16-78).
__device__ __forceinline__ float rmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float radd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float rsub(float a, float b) { return __fsub_rn(a, b); }

__device__ __forceinline__ EqTerms bnd_eq(float ux, float uy, float uz) {
    return EqTerms{ux, uy, uz, radd(radd(rmul(ux, ux), rmul(uy, uy)), rmul(uz, uz))};
}
__device__ __forceinline__ NeqTerms bnd_neq(const NodeMoments &m) {
    NeqTerms n;
    n.pxx = m.pxx; n.pxy = m.pxy; n.pyy = m.pyy; n.pyz = m.pyz; n.pzz = m.pzz; n.pxz = m.pxz;
    n.a3xxy = radd(rmul(m.pxx, m.uy), rmul(2.0f * m.pxy, m.ux));
    n.a3xxz = radd(rmul(m.pxx, m.uz), rmul(2.0f * m.pxz, m.ux));
    n.a3xyy = radd(rmul(m.pyy, m.ux), rmul(2.0f * m.pxy, m.uy));
    n.a3xzz = radd(rmul(m.pzz, m.ux), rmul(2.0f * m.pxz, m.uz));
    n.a3yyz = radd(rmul(m.pyy, m.uz), rmul(2.0f * m.pyz, m.uy));
    n.a3yzz = radd(rmul(m.pzz, m.uy), rmul(2.0f * m.pyz, m.uz));
    n.a3xyz = radd(radd(rmul(m.pxy, m.uz), rmul(m.pxz, m.uy)), rmul(m.pyz, m.ux));
    return n;
}
template <int I>
__device__ __forceinline__ float bnd_feq(float rho, const EqTerms &e) {
    using D = Dir<I>;
    float cu = 0.0f;
    if constexpr (D::cx != 0) cu = radd(cu, D::fx * e.ux);
    if constexpr (D::cy != 0) cu = radd(cu, D::fy * e.uy);
    if constexpr (D::cz != 0) cu = radd(cu, D::fz * e.uz);
    const float cu2 = rmul(cu, cu);
    const float A2 = radd(rsub(rmul(cu2, kInv2Cs4), rmul(e.usq, kInv2Cs2)), rmul(cu, kInvCs2));
    const float A3 = rmul(cu, rsub(rmul(cu2, kInv6Cs6), rmul(e.usq, kInv2Cs4)));
    return rmul(rmul(D::w, rho), radd(radd(1.0f, A2), A3));
}
template <int I>
__device__ __forceinline__ float bnd_fneq(const NeqTerms &n) {
    using D = Dir<I>;
    float A2 = 0.0f;
    if constexpr (D::Hxx != 0.0f) A2 = radd(A2, rmul(n.pxx, D::Hxx));
    if constexpr (D::Hxy != 0.0f) A2 = radd(A2, rmul(2.0f * n.pxy, D::Hxy));
    if constexpr (D::Hyy != 0.0f) A2 = radd(A2, rmul(n.pyy, D::Hyy));
    if constexpr (D::Hyz != 0.0f) A2 = radd(A2, rmul(2.0f * n.pyz, D::Hyz));
    if constexpr (D::Hzz != 0.0f) A2 = radd(A2, rmul(n.pzz, D::Hzz));
    if constexpr (D::Hxz != 0.0f) A2 = radd(A2, rmul(2.0f * n.pxz, D::Hxz));
    A2 = rmul(A2, kInv2Cs4);
    float A3 = 0.0f;
    if constexpr (D::Hxxy != 0.0f) A3 = radd(A3, rmul(n.a3xxy, D::Hxxy));
    if constexpr (D::Hxxz != 0.0f) A3 = radd(A3, rmul(n.a3xxz, D::Hxxz));
    if constexpr (D::Hxyy != 0.0f) A3 = radd(A3, rmul(n.a3xyy, D::Hxyy));
    if constexpr (D::Hxzz != 0.0f) A3 = radd(A3, rmul(n.a3xzz, D::Hxzz));
    if constexpr (D::Hyyz != 0.0f) A3 = radd(A3, rmul(n.a3yyz, D::Hyyz));
    if constexpr (D::Hyzz != 0.0f) A3 = radd(A3, rmul(n.a3yzz, D::Hyzz));
    if constexpr (D::Hxyz != 0.0f) A3 = radd(A3, rmul(2.0f * n.a3xyz, D::Hxyz));
    return rmul(D::w, radd(A2, rmul(A3, kInv2Cs6)));
}
// omega_at with the same rounding rule (the outlet's fluid plane)
__device__ __forceinline__ float bnd_omega_at(const Physics &ph, int y) {
    if (!ph.sponge) return ph.omega;
    const float s = clamp01(rmul(float(y) - ph.sponge_y_start, ph.sponge_inv_width));
    const float nus = rmul(ph.nu, radd(1.0f, rmul(ph.sponge_K, rmul(rmul(s, s), s))));
    return 1.0f / radd(0.5f, rmul(nus, kInvCs2));
}

__device__ __forceinline__ NodeMoments load_moments(const float *m, size_t stride, size_t id) {
    NodeMoments r;
    r.rr = m[kMomRR * stride + id]; r.rb = m[kMomRB * stride + id];
    r.ux = m[kMomUX * stride + id]; r.uy = m[kMomUY * stride + id]; r.uz = m[kMomUZ * stride + id];
    r.pxx = m[kMomPXX * stride + id]; r.pxy = m[kMomPXY * stride + id]; r.pyy = m[kMomPYY * stride + id];
    r.pyz = m[kMomPYZ * stride + id]; r.pzz = m[kMomPZZ * stride + id]; r.pxz = m[kMomPXZ * stride + id];
    return r;
}

// ------------------------------------------------------------------ boundary pieces

// Inlet column (x,z): density mask at y=0 and, for disc columns, the nine
// cy=+1 populations entering y=1 (jet/boundary_conditions.cuh:17-85).  They
// are stored in the ghost plane y=0 of `dst` at (x,0,z), where the y=1 nodes
// (x+cx, 1, z+cz) pull them.  `m` are the moments of fluid node (x,1,z).
template <class C>
__device__ __forceinline__ void inlet_column(const DeviceState &s, void *dst, float *psi_dst, int x, int z,
                                             int64_t step, const NodeMoments &m) {
    const Geometry &g = s.g;
    const Physics &ph = s.ph;
    const uint32_t idB = uint32_t(x) + uint32_t(g.sz) * uint32_t(z);
    const bool jet = is_jet_column(ph, x, z);
    const float rrB = (1.0f - (jet ? 1.0f : 0.0f)) * ph.rhor0;
    const float rbB = (jet ? 1.0f : 0.0f) * ph.rhob0;
    s.mom[size_t(kMomRR) * g.N + idB] = rrB;
    s.mom[size_t(kMomRB) * g.N + idB] = rbB;
    psi_dst[idB] = psi_of(rrB, rbB);
    if (!jet) return;
    const float rT = radd(rrB, rbB);
    const float aR = rmul(rrB, 1.0f / rT), aB = rmul(rbB, 1.0f / rT);
    const float oms = rsub(1.0f, ph.omega_b);
    const EqTerms e = bnd_eq(0.0f, inlet_velocity(s, step, x, z), 0.0f);
    const NeqTerms n = bnd_neq(m);
    static_for<kQ>([&](auto I) {
        constexpr int i = decltype(I)::value;
        if constexpr (Dir<i>::cy == 1) {
            const float gi = radd(bnd_feq<i>(rT, e), rmul(oms, bnd_fneq<i>(n)));
            C::store_to(dst, g, i, x, 0, z, rmul(aR, gi), rmul(aB, gi), ph.f16_rho0);
        }
    });
}

// Outlet column (x,z): convective update of the y=NY-1 state from fluid node
// F=(x,NY-2,z) and the nine cy=-1 populations entering y=NY-2
// (jet/boundary_conditions.cuh:163-233), stored in ghost plane y=NY-1 of dst.
template <class C>
__device__ __forceinline__ void outlet_column(const DeviceState &s, void *dst, float *psi_dst, int x, int z,
                                              const NodeMoments &m) {
    const Geometry &g = s.g;
    const Physics &ph = s.ph;
    const uint32_t idB = uint32_t(x) + uint32_t(g.sy) * uint32_t(g.NY - 1) + uint32_t(g.sz) * uint32_t(z);
    float *mom = s.mom;
    const size_t N = g.N;
    const float uc = clamp01(m.uy);
    auto conv = [uc](float b, float f) { return rsub(b, rmul(uc, rsub(b, f))); };
    const float rrB = conv(mom[kMomRR * N + idB], m.rr);
    const float rbB = conv(mom[kMomRB * N + idB], m.rb);
    const float uxB = conv(mom[kMomUX * N + idB], m.ux);
    const float uyB = conv(mom[kMomUY * N + idB], m.uy);
    const float uzB = conv(mom[kMomUZ * N + idB], m.uz);
    mom[kMomRR * N + idB] = rrB;
    mom[kMomRB * N + idB] = rbB;
    mom[kMomUX * N + idB] = uxB;
    mom[kMomUY * N + idB] = uyB;
    mom[kMomUZ * N + idB] = uzB;
    psi_dst[idB] = psi_of(rrB, rbB);
    const float rhoT = radd(rrB, rbB);
    const float inv = 1.0f / rhoT;
    const float aR = rmul(rrB, inv), aB = rmul(rbB, inv);
    const float oms = rsub(1.0f, bnd_omega_at(ph, g.NY - 2));
    const EqTerms e = bnd_eq(uxB, uyB, uzB);
    const NeqTerms n = bnd_neq(m);
    static_for<kQ>([&](auto I) {
        constexpr int i = decltype(I)::value;
        if constexpr (Dir<i>::cy == -1) {
            const float gi = radd(bnd_feq<i>(rhoT, e), rmul(oms, bnd_fneq<i>(n)));
            C::store_to(dst, g, i, x, g.NY - 1, z, rmul(aR, gi), rmul(aB, gi), ph.f16_rho0);
        }
    });
}

}  // namespace
}  // namespace mcg
