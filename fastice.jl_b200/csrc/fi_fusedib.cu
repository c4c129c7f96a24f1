// fi_fusedib.cu -- immersed-boundary PT iteration in one pass: the plane march of
// fi_sweep3d.cuh over the part of the box that holds ice.
//
// Reference semantics: src/Models/ImmersedBoundaryFullStokes/Isothermal/Isothermal.jl:
// 100-122 with kernels_3d.jl:3-74 and boundary_conditions.jl, operation by operation as
// the in-place kernels of fi_reference.cu (a no-FMA build matches the CPU oracle bit for
// bit).
//
// Work list.  Once two full iterations have run, a point without an activity bit holds a
// value that never moves (zero, or what a boundary batch puts there), in both state
// buffers after they have been made equal.  A job is a 32x8 column of positions and a run
// of planes [kb, ke) in which the column has an active point or a neighbour of one; a CTA
// runs one job, and nothing outside the jobs is read or written except as the constant
// ring of one.
//
// Fractions.  They are read from global memory, all of a point's at once (in FP32 ahead of the
// wait or barrier before their use), and their lines are brought into the L2 cache two planes
// earlier.  Where every fraction that the updates of an index read is exactly 1 (IBF_FULL:
// all of the ice except the layers cut by bed and surface) or where nothing is active, none
// is read and the weights are 1: the masked update is then the plain one bit for bit.
//
// What bounds it.  In place, the two masked kernels and six boundary batches moved 344
// bytes per active FP64 point in dependent loads; one pass without fractions moves 176 and
// the ring.  After that the code itself is the limit: beyond some 100 KB of it the warps
// wait for instructions, so there is one body for interior and boundary columns and no
// second one for unmasked points (FP32, 383^3: 949 us with both, 742 without).  In FP64 it is
// registers and the wait for fractions: values spilled to local memory miss every time, as next
// to no L1 is left beside this much shared memory (2118 us with 36 bytes spilled), so the loads
// stand where they are used and three blocks fit an SM with 8 bytes spilled (see sweep_ib).
// Measured per iteration, in place and now: FP64 383^3 1599 -> 1066-1154 us by the box, 191^3
// 260 -> 188 us; FP32 383^3 1209 -> 695 us, 191^3 215 -> 129 us; a box a quarter full of ice
// under rough beds, FP64 383^3 1355-1645 -> 1232-1559 us, 191^3 233-265 -> 166-193 us.
#include <algorithm>
#include <cstring>
#include <vector>

#include "fi_fusedib.h"
#include "fi_sweep3d.cuh"

namespace fi {

namespace {

constexpr int IX = 32, IY = 8;
constexpr unsigned IBF_ANY = 0x7fu;
constexpr unsigned IBF_V_ANY = IBF_V_VCC | IBF_V_CVC | IBF_V_CCV;

// Volume fractions around a point that the stress updates of step s read (plane s: suffix
// none, r right, l left, d below, t above in y; u: plane s + 1).  need: not all of them are 1.
template <typename T>
struct StressW {
    T nx, nxr, nxd, nxu, ny, nyl, nyt, nyu, nz, nzu, nzul, nzud;
};
template <typename T>
__device__ __forceinline__ StressW<T> stress_w(const Ptrs<T> &in, long long I, long long sx, long long sxy, bool need) {
    const T o = T(1);
    StressW<T> w{o, o, o, o, o, o, o, o, o, o, o, o};
    if (need) {
        const T *x = in.wns[W_VCC] + I, *y = in.wns[W_CVC] + I, *z = in.wns[W_CCV] + I;
        w.nx = __ldg(x), w.nxr = __ldg(x + 1), w.nxd = __ldg(x - sx), w.nxu = __ldg(x + sxy);
        w.ny = __ldg(y), w.nyl = __ldg(y - 1), w.nyt = __ldg(y + sx), w.nyu = __ldg(y + sxy);
        w.nz = __ldg(z), w.nzu = __ldg(z + sxy), w.nzul = __ldg(z + sxy - 1), w.nzud = __ldg(z + sxy - sx);
    }
    return w;
}
// and those of the velocity updates (na: c centre, xy, xz, yz edges; ns at the faces)
template <typename T>
struct VelocityW {
    T c, cl, cd, cz, xy, xyt, xyr, xz, xzu, xzr, yz, yzu, yzt, nx, ny, nz;
};
template <typename T>
__device__ __forceinline__ VelocityW<T> velocity_w(const Ptrs<T> &in, long long I, long long sx, long long sxy, bool need) {
    const T o = T(1);
    VelocityW<T> w{o, o, o, o, o, o, o, o, o, o, o, o, o, o, o, o};
    if (need) {
        const T *c = in.wna[W_CCC] + I, *xy = in.wna[W_VVC] + I, *xz = in.wna[W_VCV] + I, *yz = in.wna[W_CVV] + I;
        w.c = __ldg(c), w.cl = __ldg(c - 1), w.cd = __ldg(c - sx), w.cz = __ldg(c - sxy);
        w.xy = __ldg(xy), w.xyt = __ldg(xy + sx), w.xyr = __ldg(xy + 1);
        w.xz = __ldg(xz), w.xzu = __ldg(xz + sxy), w.xzr = __ldg(xz + 1);
        w.yz = __ldg(yz), w.yzu = __ldg(yz + sxy), w.yzt = __ldg(yz + sx);
        w.nx = __ldg(in.wns[W_VCC] + I), w.ny = __ldg(in.wns[W_CVC] + I), w.nz = __ldg(in.wns[W_CCV] + I);
    }
    return w;
}

__device__ __forceinline__ void prefetch_l2(const void *a) { asm volatile("prefetch.global.L2 [%0];" ::"l"(a)); }

// ---- masked values: new where the activity bit is set, else what the point holds -------
template <int mask, typename T, int TX, int TY>
__device__ __forceinline__ Centre<T> centre_masked(const Ctx<T, TX, TY> &c, const KParams &p, const TConst<T> &q,
                                                   const Ptrs<T> &in, int li, int lj, long long I, const StressW<T> &w, bool on) {
    constexpr int BV = FBox<T, TX, TY, M_VX>::bw;
    const T *vx = EL(M_VX, c.V0), *vy = EL(M_VY, c.V0), *vz = EL(M_VZ, c.V0), *vzp = EL(M_VZ, c.V1);
    const T e2 = T(2.0) * *EL(M_ET, c.V0);
    const T s[3] = {diff_r(w.nxr, vx[1], w.nx, vx[0]), diff_r(w.nyt, vy[BV], w.ny, vy[0]), diff_r(w.nzu, vzp[0], w.nz, vz[0])};
    T d[3];
    const T divV = rates_r<3, sizeof(T) == 4>(s, q.inv_dx, d);
    const T dv = p.p_forcing && on ? divV + __ldg(in.fP + I) : divV;
    auto pick = [&](T o, T r, int k) { return on ? relax_r(o, e2, r, q.dt_tau[k]) : o; };
    Centre<T> r;
    const T oP = *EL(M_P, c.C);
    r.P = on ? fma_r(-mul_r(dv, *EL(M_ET, c.V0)), q.dt_P, oP) : oP;
    r.xx = (mask & F_XX) ? pick(*EL(M_XX, c.C), d[0], 0) : T(0);
    r.yy = (mask & F_YY) ? pick(*EL(M_YY, c.C), d[1], 1) : T(0);
    r.zz = (mask & F_ZZ) ? pick(*EL(M_ZZ, c.C), d[2], 2) : T(0);
    return r;
}
template <typename T, int TX, int TY>
__device__ __forceinline__ T xy_masked(const Ctx<T, TX, TY> &c, const TConst<T> &q, int li, int lj, const StressW<T> &w, bool on) {
    constexpr int BV = FBox<T, TX, TY, M_VX>::bw;
    const T o = *EL(M_XY, c.C);
    const T *vx = EL(M_VX, c.V0), *vy = EL(M_VY, c.V0), *et = EL(M_ET, c.V0);
    const T exy = h(sum_r(diff_r(w.ny, vy[0], w.nyl, vy[-1]), q.inv_dx[0], diff_r(w.nx, vx[0], w.nxd, vx[-BV]), q.inv_dx[1]));
    const T e_xy = h(h(et[-1 - BV] + et[-BV]) + h(et[-1] + et[0]));
    return on ? relax_r(o, T(2.0) * e_xy, exy, q.dt_tau[3]) : o;
}
template <typename T, int TX, int TY>
__device__ __forceinline__ T xz_masked(const Ctx<T, TX, TY> &c, const TConst<T> &q, int li, int lj, const StressW<T> &w, bool on) {
    const T o = *EL(M_XZ, c.V1);
    const T *vx = EL(M_VX, c.V1), *vxm = EL(M_VX, c.V0), *vz = EL(M_VZ, c.V1);
    const T *et = EL(M_ET, c.V1), *etm = EL(M_ET, c.V0);
    const T exz = h(sum_r(diff_r(w.nzu, vz[0], w.nzul, vz[-1]), q.inv_dx[0], diff_r(w.nxu, vx[0], w.nx, vxm[0]), q.inv_dx[2]));
    const T e_xz = h(h(etm[-1] + etm[0]) + h(et[-1] + et[0]));
    return on ? relax_r(o, T(2.0) * e_xz, exz, q.dt_tau[4]) : o;
}
template <typename T, int TX, int TY>
__device__ __forceinline__ T yz_masked(const Ctx<T, TX, TY> &c, const TConst<T> &q, int li, int lj, const StressW<T> &w, bool on) {
    constexpr int BV = FBox<T, TX, TY, M_VX>::bw;
    const T o = *EL(M_YZ, c.V1);
    const T *vy = EL(M_VY, c.V1), *vym = EL(M_VY, c.V0), *vz = EL(M_VZ, c.V1);
    const T *et = EL(M_ET, c.V1), *etm = EL(M_ET, c.V0);
    const T eyz = h(sum_r(diff_r(w.nzu, vz[0], w.nzud, vz[-BV]), q.inv_dx[1], diff_r(w.nyu, vy[0], w.ny, vym[0]), q.inv_dx[2]));
    const T e_yz = h(h(etm[-BV] + etm[0]) + h(et[-BV] + et[0]));
    return on ? relax_r(o, T(2.0) * e_yz, eyz, q.dt_tau[5]) : o;
}

// Velocity from the weighted differences: P and τ_dd along it (spacing 1/i), then the two
// shear stresses.  unit: no lane of the warp divides by a fraction other than 1.
template <typename T>
__device__ __forceinline__ T v_masked(T o, T dP, T dt, T i, T d1, T i1, T d2, T i2, T g, T eta, T w, T dtV, bool on, bool unit) {
    T r = div_fast(fma_r(d2, i2, fma_r(d1, i1, sum_r(dt, i, -dP, i))) - g, eta);
    if (!unit) r = div_fast(r, w);
    return on ? fma_r(r, dtV, o) : o;
}
template <typename T, int TX, int TY>
__device__ __forceinline__ T vx_masked(const Ctx<T, TX, TY> &c, const TConst<T> &q, int li, int lj, const VelocityW<T> &w, bool on,
                                       bool unit, T gx) {
    constexpr int BY = FBox<T, TX, TY, M_XY>::bw;
    const T *P = EL(M_P, c.C), *xx = EL(M_XX, c.C), *xy = EL(M_XY, c.C), *et = EL(M_ET, c.V0);
    return v_masked(*EL(M_VX, c.V0), diff_r(w.c, P[0], w.cl, P[-1]), diff_r(w.c, xx[0], w.cl, xx[-1]), q.inv_dx[0],
                    diff_r(w.xyt, xy[BY], w.xy, xy[0]), q.inv_dx[1], diff_r(w.xzu, *EL(M_XZ, c.V1), w.xz, *EL(M_XZ, c.V0)),
                    q.inv_dx[2], gx, h(et[-1] + et[0]), w.nx, q.dt_V[0], on, unit);
}
template <typename T, int TX, int TY>
__device__ __forceinline__ T vy_masked(const Ctx<T, TX, TY> &c, const TConst<T> &q, int li, int lj, const VelocityW<T> &w, bool on,
                                       bool unit, T gy) {
    constexpr int BP = FBox<T, TX, TY, M_P>::bw, BYY = FBox<T, TX, TY, M_YY>::bw, BV = FBox<T, TX, TY, M_ET>::bw;
    const T *P = EL(M_P, c.C), *yy = EL(M_YY, c.C), *xy = EL(M_XY, c.C), *et = EL(M_ET, c.V0);
    return v_masked(*EL(M_VY, c.V0), diff_r(w.c, P[0], w.cd, P[-BP]), diff_r(w.c, yy[0], w.cd, yy[-BYY]), q.inv_dx[1],
                    diff_r(w.xyr, xy[1], w.xy, xy[0]), q.inv_dx[0], diff_r(w.yzu, *EL(M_YZ, c.V1), w.yz, *EL(M_YZ, c.V0)),
                    q.inv_dx[2], gy, h(et[-BV] + et[0]), w.ny, q.dt_V[1], on, unit);
}
template <typename T, int TX, int TY>
__device__ __forceinline__ T vz_masked(const Ctx<T, TX, TY> &c, const TConst<T> &q, int li, int lj, const VelocityW<T> &w, bool on,
                                       bool unit, T gz, const Carry<T> &k) {
    constexpr int BYZ = FBox<T, TX, TY, M_YZ>::bw;
    const T *xz = EL(M_XZ, c.V0), *yz = EL(M_YZ, c.V0);
    return v_masked(*EL(M_VZ, c.V0), diff_r(w.c, k.P, w.cz, k.Pm), diff_r(w.c, k.zz, w.cz, k.zzm), q.inv_dx[2],
                    diff_r(w.xzr, xz[1], w.xz, xz[0]), q.inv_dx[0], diff_r(w.yzt, yz[BYZ], w.yz, yz[0]), q.inv_dx[1], gz,
                    h(k.etm + *EL(M_ET, c.V0)), w.nz, q.dt_V[2], on, unit);
}

// Ring stresses of step s (sigma_ring of the plain sweep) under the activity bits f0, f1 of
// the ring thread's point at planes s and s + 1.  A side of the domain has no ring below or
// left of it (no periodic dimensions): its ghosts come from the cells beside them.
template <typename T, int TX, int TY>
__device__ __forceinline__ void ring_masked(const Ctx<T, TX, TY> &c, const KParams &p, const TConst<T> &q, const Ptrs<T> &in,
                                            const Ptrs<T> &out, int s, int zf, bool write, int role, int li, int lj, unsigned f0,
                                            unsigned f1) {
    const int i = c.i0 + li, j = c.j0 + lj, lane = threadIdx.x % 32;
    const long long I = c.sxy * s + c.col(li, lj);
    if (role == 0 || role == 2) {  // P with τyy (row below) or τxx (column left)
        if (!(f0 & IBF_S_CCC) || s < 1) return;
        const StressW<T> w = stress_w(in, I, c.sx, c.sxy, !(f0 & IBF_FULL));
        if (role == 0) {
            const Centre<T> v = centre_masked<F_P | F_YY>(c, p, q, in, li, lj, I, w, true);
            *EL(M_P, c.C) = v.P;
            *EL(M_YY, c.C) = v.yy;
            if (j == c.n1 && p.bc_kind[1][1] == FI_BC_TRACTION) traction_y(c, q, out, s, 1, li, v.P, v.yy, write);
        } else {
            const Centre<T> v = centre_masked<F_P | F_XX>(c, p, q, in, li, lj, I, w, true);
            *EL(M_P, c.C) = v.P;
            *EL(M_XX, c.C) = v.xx;
            if (i == c.n0 && p.bc_kind[0][1] == FI_BC_TRACTION) traction_x(c, q, out, s, 1, lj, v.P, v.xx, write);
        }
        return;
    }
    // τxy with τyz (row above) or τxz (column right; its corner has τxy alone)
    const bool on_xy = f0 & IBF_S_VVC, on_z = f1 & (role == 1 ? IBF_S_CVV : IBF_S_VCV), has_z = role == 1 || lane < TY;
    if (!on_xy && !on_z) return;  // both keep what they hold
    const StressW<T> w = stress_w(in, I, c.sx, c.sxy, !(f0 & f1 & IBF_FULL));
    const unsigned f = shear_flags(c, p, i, j);
    *EL(M_XY, c.C) = fix_xy(q, xy_masked(c, q, li, lj, w, on_xy), f);
    if (role == 1) {
        const T yz = fix_yz(q, yz_masked(c, q, li, lj, w, on_z), f);
        *EL(M_YZ, c.V1) = zf >= 0 ? q.bc_val[2][zf][1] : yz;
    } else if (has_z) {
        const T xz = fix_xz(q, xz_masked(c, q, li, lj, w, on_z), f);
        *EL(M_XZ, c.V1) = zf >= 0 ? q.bc_val[2][zf][0] : xz;
    }
}

// activity bytes of a point at planes s, s + 1, s + 2
template <bool PACKED>
struct PlaneBits {
    unsigned f0, f1, f2;
    __device__ __forceinline__ PlaneBits(unsigned a, unsigned b, unsigned c) : f0(a), f1(b), f2(c) {}
    __device__ __forceinline__ unsigned at0() const { return f0; }
    __device__ __forceinline__ unsigned at1() const { return f1; }
    __device__ __forceinline__ unsigned at2() const { return f2; }
    __device__ __forceinline__ void up(unsigned next) { f0 = f1, f1 = f2, f2 = next; }
};
template <>
struct PlaneBits<true> {
    unsigned v;
    __device__ __forceinline__ PlaneBits(unsigned a, unsigned b, unsigned c) : v(a | b << 8 | c << 16) {}
    __device__ __forceinline__ unsigned at0() const { return v & 0xffu; }
    __device__ __forceinline__ unsigned at1() const { return v >> 8 & 0xffu; }
    __device__ __forceinline__ unsigned at2() const { return v >> 16; }
    __device__ __forceinline__ void up(unsigned next) { v = v >> 8 | next << 16; }
};

// The plane march of one job.  TIGHT: the fractions and the body force are loaded where they
// are used instead of ahead of the wait or barrier, and the activity bytes share a register,
// so that FP64 fits three blocks a multiprocessor at 80 registers (383^3: 1221 us an
// iteration with two blocks and 120 registers, 1066 so; 191^3 214 and 188.5).
template <bool TIGHT, typename T>
__device__ __forceinline__ void sweep_ib(Ctx<T, IX, IY> &c, const KParams &p, const TConst<T> &q, const Ptrs<T> &in,
                                         const Ptrs<T> &out, const InMaps &maps, uint64_t *bars, unsigned *released, int *err) {
    constexpr int TX = IX, TY = IY, NW = Layout<T, IX, IY>::NW;
    const int tid = threadIdx.x, lane = tid % 32;
    const int li = tid % TX, lj = tid / TX;
    const int first = c.kb - 1;
    const int gmax = min(c.ke - 1, c.n2) + 1;
    if (tid == 0) {
        issue_group(c, maps, first, 0, bars);
        issue_group(c, maps, first + 1, 1, bars);
        if (first + 2 <= gmax) issue_group(c, maps, first + 2, 2, bars);
    }
    const unsigned fl = column_flags(c, p, c.i0 + li, c.j0 + lj);
    const bool inside = fl & CF_IN;
    // the ring point of the last four warps: row below, row above, column left, column right
    const int role = tid / 32 - (NW - 4);
    const int rli = role == 2 ? -1 : role == 3 ? TX : lane, rlj = role == 0 ? -1 : role == 1 ? TY : lane;
    const int ri = c.i0 + rli, rj = c.j0 + rlj;
    const bool ring = role >= 0 && (role < 2 || lane < TY + (role == 3 ? 1 : 0)) && ri >= 1 && rj >= 1 && ri <= c.n0 + 1 &&
                      rj <= c.n1 + 1;
    const unsigned char *own_bits = in.ibf + c.col(li, lj), *ring_bits = in.ibf + (ring ? c.col(rli, rlj) : 0u);
    auto bits = [&](const unsigned char *at, int bi, int bj, bool on, int k) -> unsigned {
        if (!on || k < 1 || k > c.n2 + 1) return 0u;
        if constexpr (TIGHT) return (unsigned)__ldg(in.ibf + (c.sxy * k + c.col(bi, bj)));
        return (unsigned)__ldg(at + c.sxy * k);
    };
    PlaneBits<TIGHT> own_at(bits(own_bits, li, lj, inside, first), bits(own_bits, li, lj, inside, first + 1), bits(own_bits, li, lj, inside, first + 2));
    PlaneBits<TIGHT> ring_at(bits(ring_bits, rli, rlj, ring, first), bits(ring_bits, rli, rlj, ring, first + 1), bits(ring_bits, rli, rlj, ring, first + 2));
    uint32_t phase = 0;
    auto wait_group = [&](int g) -> bool {
        const int b = g % 3;
        const bool ok = mbar_wait(&bars[b], (phase >> b) & 1u);
        phase ^= 1u << b;
        return __all_sync(0xffffffffu, ok);  // (a warp leaves the march as one)
    };
    Carry<T> k{T(0), T(0), T(0), T(0), T(0)};
    long long I = c.sxy * first + c.col(li, lj);
    bool ok = wait_group(first);
    for (int s = first; s < c.ke && ok; s++, I += c.sxy) {
        c.set_plane(s);
        const unsigned f0 = own_at.at0(), f1 = own_at.at1(), f2 = own_at.at2();
        const bool own = s >= c.kb;
        const int zf = z_fixed(c, p, s + 1);
        if (s <= c.n2) {
            const bool any = (f0 | f1) & IBF_ANY;
            const bool need = any && !(f0 & f1 & IBF_FULL);
            StressW<T> sw;
            if constexpr (!TIGHT) sw = stress_w(in, I, c.sx, c.sxy, need);
            if ((f2 & IBF_ANY) && !(f2 & IBF_FULL)) {
                const long long N = I + 2 * c.sxy;
                for (int w : {W_CCC, W_VVC, W_VCV, W_CVV}) prefetch_l2(in.wna[w] + N);
                for (int w : {W_VCC, W_CVC, W_CCV}) prefetch_l2(in.wns[w] + N);
            }
            ok = wait_group(s + 1);
            if (!ok) break;
            if (__any_sync(0xffffffffu, any)) {
                if constexpr (TIGHT) sw = stress_w(in, I, c.sx, c.sxy, need);
                const Centre<T> v = centre_masked<F_P | F_XX | F_YY | F_ZZ>(c, p, q, in, li, lj, I, sw, f0 & IBF_S_CCC);
                const T xy = xy_masked(c, q, li, lj, sw, f0 & IBF_S_VVC);
                const T xz = xz_masked(c, q, li, lj, sw, f1 & IBF_S_VCV), yz = yz_masked(c, q, li, lj, sw, f1 & IBF_S_CVV);
                sigma_store<true>(c, p, q, out, s, li, lj, fl, zf, own, s + 1 < c.ke, I, v, xy, xz, yz, k);
            } else {  // all keep what they hold
                k.P = *EL(M_P, c.C);
                k.zz = *EL(M_ZZ, c.C);
                if (s == 1 && p.bc_kind[2][0] == FI_BC_TRACTION) {
                    const T tv = T(2.0) * q.bc_val[2][0][2];
                    k.Pm = tv - k.P;
                    k.zzm = tv - k.zz;
                }
            }
            if (ring) ring_masked(c, p, q, in, out, s, zf, own, role, rli, rlj, ring_at.at0(), ring_at.at1());
        } else if (inside && p.bc_kind[2][1] == FI_BC_TRACTION) {
            // the top plane of vertices has no stresses: the ghosts over a traction top
            const T tv = T(2.0) * q.bc_val[2][1][2];
            k.P = tv - k.Pm;
            k.zz = tv - k.zzm;
            if ((fl & CF_CX) && (fl & CF_CY)) {
                out.P[I] = k.P;
                out.tzz[I] = k.zz;
            }
        }
        if (own) {
            const bool need = (f0 & IBF_V_ANY) && !(f0 & IBF_FULL);
            const bool unit = __all_sync(0xffffffffu, !need);
            VelocityW<T> vw;
            T g[3];
            auto force = [&](const T *field, int d) {
                return TIGHT ? (inside ? body_force(p, q, field, d, I) : q.g_val[d]) : g[d];
            };
            if constexpr (!TIGHT) {
                g[0] = q.g_val[0], g[1] = q.g_val[1], g[2] = q.g_val[2];
                if (inside) {
                    g[0] = body_force(p, q, in.gx, 0, I);
                    g[1] = body_force(p, q, in.gy, 1, I);
                    g[2] = body_force(p, q, in.gz, 2, I);
                }
                vw = velocity_w(in, I, c.sx, c.sxy, need);
            }
            __syncthreads();
            if constexpr (TIGHT) vw = velocity_w(in, I, c.sx, c.sxy, need);
            const T vx = vx_masked(c, q, li, lj, vw, f0 & IBF_V_VCC, unit, force(in.gx, 0));
            const T vy = vy_masked(c, q, li, lj, vw, f0 & IBF_V_CVC, unit, force(in.gy, 1));
            const T vz = vz_masked(c, q, li, lj, vw, f0 & IBF_V_CCV, unit, force(in.gz, 2), k);
            v_store<true, true>(c, p, q, in, out, s, li, lj, fl, I, k, vx, vy, vz);
        }
        k.Pm = k.P;
        k.zzm = k.zz;
        k.etm = *EL(M_ET, c.V0);
        own_at.up(bits(own_bits, li, lj, inside, s + 3));
        ring_at.up(bits(ring_bits, rli, rlj, ring, s + 3));
        __syncwarp();
        if (s + 3 <= gmax && lane == 0) {
            unsigned n;
            asm volatile("atom.add.acq_rel.cta.shared::cta.u32 %0, [%1], 1;" : "=r"(n) : "r"(smem_u32(released)) : "memory");
            if (n % NW == NW - 1) {
                fence_proxy_async();
                issue_group(c, maps, s + 3, 2, bars);
            }
        }
    }
    if (ok) return;
    atomicExch(err, (int)FI_ERR_TIMEOUT);
    for (int b = 0; b < kBars; b++) mbar_wait(&bars[b], (phase >> b) & 1u);
}

// one job: x = tile x | tile y << 16, y = kb, z = ke
template <bool TIGHT, typename T>
__device__ __forceinline__ void run_job(const Geom &g, const KParams &p, const TConst<T> &q, const Ptrs<T> &in,
                                        const Ptrs<T> &out, const InMaps &maps, unsigned char *smem, int4 job, int *err) {
    using Lay = Layout<T, IX, IY>;
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + (size_t)Lay::ELEMS * sizeof(T));
    unsigned *released = reinterpret_cast<unsigned *>(bars + kBars);
    if (threadIdx.x == 0) {
        for (int b = 0; b < kBars; b++) mbar_init(&bars[b], 1);
        *released = 0u;
        mbar_fence_init();
    }
    __syncthreads();
    Ctx<T, IX, IY> c;
    c.sm = reinterpret_cast<T *>(smem);
    c.i0 = 1 + (job.x & 0xffff) * IX;
    c.j0 = 1 + (job.x >> 16) * IY;
    c.kb = job.y;
    c.ke = job.z;
    c.n0 = g.n[0];
    c.n1 = g.n[1];
    c.n2 = g.n[2];
    c.sx = g.pitch;
    c.sxy = g.sxy;
    c.hx0 = c.hx1 = c.hy0 = c.hy1 = false;
    chain_launches();
    sweep_ib<TIGHT>(c, p, q, in, out, maps, bars, released, err);
}

template <typename T>
__global__ void __launch_bounds__(Layout<T, IX, IY>::NT, Layout<T, IX, IY>::MINB)
    fusedib_kernel(Geom g, KParams p, TConst<T> q, Ptrs<T> in, Ptrs<T> out, const __grid_constant__ InMaps maps,
                   const int4 *__restrict__ jobs, int *err) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    run_job<sizeof(T) == 8>(g, p, q, in, out, maps, smem_raw, jobs[blockIdx.x], err);
}

// jobs of several models: w = member; the block copies its member's parameters and pointers
// into shared memory (e: the roles of its buffers).  With them there, FP64 at three blocks a
// multiprocessor spills (12 glaciers of 16^3-48^3: 71 us an iteration against 63 at two).
template <typename T>
__global__ void __launch_bounds__(Layout<T, IX, IY>::NT, sizeof(T) == 8 ? 2 : Layout<T, IX, IY>::MINB)
    fusedib_batched(const IbFusedMember<T> *__restrict__ members, const int4 *__restrict__ jobs, int e) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ __align__(16) IbFusedHead<T> sm;
    const int4 job = jobs[blockIdx.x];
    const IbFusedMember<T> &m = members[job.w];
    const unsigned *src = reinterpret_cast<const unsigned *>(&m.head);
    unsigned *dst = reinterpret_cast<unsigned *>(&sm);
    for (int w = threadIdx.x; w < (int)(sizeof(IbFusedHead<T>) / 4); w += blockDim.x) dst[w] = __ldg(src + w);
    __syncthreads();
    run_job<false>(sm.g, sm.p, sm.q, sm.f[e], sm.f[2 + e], reinterpret_cast<const InMaps &>(m.maps[e]), smem_raw, job, sm.err);
}

// 1 where a tile column has, in this plane, a point next to an active one (or active)
__global__ void __launch_bounds__(IX *IY) ib_tiles_kernel(Geom g, const unsigned char *__restrict__ flags, unsigned char *tiles) {
    const int i = 1 + blockIdx.x * IX + threadIdx.x, j = 1 + blockIdx.y * IY + threadIdx.y, k = 1 + blockIdx.z;
    unsigned any = 0;
    if (i <= g.n[0] + 1 && j <= g.n[1] + 1)
        for (int c = max(k - 1, 1); c <= min(k + 1, g.n[2] + 1); c++)
            for (int b = max(j - 1, 1); b <= min(j + 1, g.n[1] + 1); b++)
                for (int a = max(i - 1, 1); a <= min(i + 1, g.n[0] + 1); a++)
                    any |= flags[(long long)a + g.pitch * ((long long)b + g.rows * (long long)c)];
    const int on = __syncthreads_or(any != 0);
    if (threadIdx.x == 0 && threadIdx.y == 0)
        tiles[blockIdx.x + gridDim.x * (blockIdx.y + (size_t)gridDim.y * blockIdx.z)] = on ? 1 : 0;
}

// The kernels' shared memory, once per device.  (Internal linkage: a static of an exported
// template would be one object for all builds of this library loaded in a process.)
template <typename T, bool BATCHED>
cudaError_t lift_smem() {
    static bool set[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || (dev < 64 && set[dev])) return e;
    const int bytes = (int)Layout<T, IX, IY>::SMEM;
    e = BATCHED ? cudaFuncSetAttribute(fusedib_batched<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes)
                : cudaFuncSetAttribute(fusedib_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess && dev < 64) set[dev] = true;
    return e;
}

template <typename T>
cudaLaunchConfig_t launch_config(int blocks, cudaStream_t s, bool chained, cudaLaunchAttribute *attr) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(Layout<T, IX, IY>::NT);
    cfg.dynamicSmemBytes = Layout<T, IX, IY>::SMEM;
    cfg.stream = s;
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = chained ? 1 : 0;
    return cfg;
}

}  // namespace

cudaError_t ib_runs(const Geom &g, const unsigned char *flags, std::vector<IbRun> *runs, cudaStream_t s) {
    const int ntx = (g.n[0] + IX) / IX, nty = (g.n[1] + IY) / IY, np = g.n[2] + 1;
    unsigned char *d = nullptr;
    const size_t bytes = (size_t)ntx * nty * np;
    cudaError_t e = cudaMalloc(&d, bytes);
    if (e != cudaSuccess) return e;
    ib_tiles_kernel<<<dim3(ntx, nty, np), dim3(IX, IY), 0, s>>>(g, flags, d);
    std::vector<unsigned char> t(bytes);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(t.data(), d, bytes, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    cudaFree(d);
    if (e != cudaSuccess) return e;
    runs->clear();
    for (int y = 0; y < nty; y++)
        for (int x = 0; x < ntx; x++) {
            int k0 = 0, k1 = 0;  // the open run [k0, k1)
            for (int k = 1; k <= np; k++) {
                if (!t[x + (size_t)ntx * (y + (size_t)nty * (k - 1))]) continue;
                if (k0 && k <= k1 + 2) {  // a gap of two planes costs less than another run
                    k1 = k + 1;
                    continue;
                }
                if (k0) runs->push_back({x, y, k0, k1});
                k0 = k, k1 = k + 1;
            }
            if (k0) runs->push_back({x, y, k0, k1});
        }
    return cudaSuccess;
}

// z-blocks as fused3d_default_variant chooses them, over the planes of the runs
int ib_job_depth(const std::vector<const std::vector<IbRun> *> &all) {
    int best = 32;
    double cost = 0.0;
    for (int zb : {1, 2, 4, 8, 12, 16, 24, 32}) {
        long long jobs = 0;
        for (const auto *r : all)
            for (const IbRun &u : *r) jobs += (u.k1 - u.k0 + zb - 1) / zb;
        const double c = (zb + 1) * (1.25 * jobs / 148.0 + 1.6);
        if (cost == 0.0 || c < cost) best = zb, cost = c;
    }
    return best;
}

void ib_make_jobs(const std::vector<IbRun> &runs, int zb, int member, std::vector<int4> *jobs) {
    for (const IbRun &u : runs) {
        // equal parts rather than a short last one
        const int n = u.k1 - u.k0, parts = (n + zb - 1) / zb;
        for (int q = 0; q < parts; q++)
            jobs->push_back(make_int4(u.x | (u.y << 16), u.k0 + n * q / parts, u.k0 + n * (q + 1) / parts, member));
    }
}

template <typename T>
cudaError_t launch_fusedib(const Geom &g, const KParams &p, const Ptrs<T> &in, const Ptrs<T> &out, const void *maps11,
                           const int4 *jobs, int njobs, int *err, cudaStream_t s, bool chained) {
    if (njobs <= 0) return cudaSuccess;
    if (cudaError_t r = lift_smem<T, false>(); r != cudaSuccess) return r;
    cudaLaunchAttribute attr[1];
    const cudaLaunchConfig_t cfg = launch_config<T>(njobs, s, chained, attr);
    return cudaLaunchKernelEx(&cfg, fusedib_kernel<T>, g, p, make_tconst<T>(p), in, out, *reinterpret_cast<const InMaps *>(maps11),
                              jobs, err);
}

template <typename T>
cudaError_t launch_fusedib_batched(const IbFusedMember<T> *members, const int4 *jobs, int njobs, int e, cudaStream_t s, bool chained) {
    if (njobs <= 0) return cudaSuccess;
    if (cudaError_t r = lift_smem<T, true>(); r != cudaSuccess) return r;
    cudaLaunchAttribute attr[1];
    const cudaLaunchConfig_t cfg = launch_config<T>(njobs, s, chained, attr);
    return cudaLaunchKernelEx(&cfg, fusedib_batched<T>, members, jobs, e);
}

#define FI_INST(T)                                                                                                     \
    template cudaError_t launch_fusedib<T>(const Geom &, const KParams &, const Ptrs<T> &, const Ptrs<T> &, const void *, \
                                           const int4 *, int, int *, cudaStream_t, bool);                                  \
    template cudaError_t launch_fusedib_batched<T>(const IbFusedMember<T> *, const int4 *, int, int, cudaStream_t, bool);
FI_INST(double)
FI_INST(float)
#undef FI_INST

}  // namespace fi
