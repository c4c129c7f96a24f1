// fi_sweep3d.cuh -- the plane march of the fused 3D sweep: shared-memory layout, group
// loads, stress and velocity updates, boundary values.  fi_fused3d.cu describes the
// design and launches it on FullStokes models, fi_fusedib.cu on immersed-boundary ones.
#pragma once

#include <cuda.h>

// Layout and box constants of shapes a precision does not launch are still instantiated by
// the host-side box tables: their unreferenced members are expected.
#pragma nv_diag_suppress 177

#include "fi_device.cuh"
#include "fi_tma.cuh"

namespace fi {

namespace {

// input fields in map order
enum { M_P = 0, M_XX, M_YY, M_ZZ, M_XY, M_XZ, M_YZ, M_VX, M_VY, M_VZ, M_ET, M_COUNT };

constexpr int kBars = 3;
constexpr int kSmemPerSM = 233472;  // bytes of shared memory per SM (228 KB)

// x positions a box starts left of the column so that its global x coordinate times
// the element size is a multiple of 16 bytes
template <typename T>
constexpr int box_xb() { return 16 / (int)sizeof(T); }

// Box of input field F relative to the column origin (i0, j0): x from i0 + ox, width
// bw; y from j0 + oy, height bh.  A plane's boxes lie together in shared memory: two
// slots of the five centre stresses (P .. τxy), then three of the six face fields (τxz,
// τyz, V, η); OFF is the box's element offset inside its slot (128-byte aligned).
template <typename T, int TX, int TY, int F>
struct FBox {
    static constexpr int XB = box_xb<T>();
    static constexpr bool full = F >= M_VX;
    static constexpr bool left = full || F == M_P || F == M_XX, right = full || F == M_XY || F == M_XZ;
    static constexpr bool below = full || F == M_P || F == M_YY, above = full || F == M_XY || F == M_YZ;
    static constexpr int ox = left ? -XB : 0;
    static constexpr int bw = TX + (left ? XB : 0) + (right ? XB : 0);
    static constexpr int oy = below ? -1 : 0;
    static constexpr int bh = TY + (below ? 1 : 0) + (above ? 1 : 0);
    static constexpr int bytes = bw * bh * (int)sizeof(T);
    static constexpr int elems = ((bytes + 127) / 128) * 128 / (int)sizeof(T);
    static constexpr int off() {
        if constexpr (F == M_P || F == M_XZ) return 0;
        else return FBox<T, TX, TY, F - 1>::off() + FBox<T, TX, TY, F - 1>::elems;
    }
    static constexpr int OFF = off();
    static_assert((bw * (int)sizeof(T)) % 16 == 0, "TMA box rows are whole 16-byte units");
};

template <typename T, int TX, int TY>
struct Layout {
    static constexpr int NT = TX * TY;
    static constexpr int NW = NT / 32;
    static constexpr int CS = FBox<T, TX, TY, M_XY>::OFF + FBox<T, TX, TY, M_XY>::elems;  // a slot of centre stresses
    static constexpr int VS = FBox<T, TX, TY, M_ET>::OFF + FBox<T, TX, TY, M_ET>::elems;  // a slot of face fields
    static constexpr int ELEMS = 2 * CS + 3 * VS;
    static constexpr size_t SMEM = (size_t)ELEMS * sizeof(T) + 64;  // + mbarriers and the release counter
    static constexpr int FIT = kSmemPerSM / (int)(SMEM + 1024);
    // resident CTAs asked of the compiler: as many as the shared memory holds, up to
    // 24 warps (80 registers a thread) in FP64 and 32 (64 registers) in FP32
    static constexpr int WANT = (sizeof(T) == 8 ? 768 : 1024) / NT;
    static constexpr int MINB = FIT < 1 ? 1 : (WANT < 1 ? 1 : (FIT < WANT ? FIT : WANT));
};

// the input maps of one sweep, in map order
struct InMaps {
    CUtensorMap m[M_COUNT];
};

// What a boundary column's thread has to do beyond the update, from its position alone
// (computed once per march).
enum ColFlag : unsigned {
    CF_IN = 1u << 0,                                           // inside the vertex range
    CF_CX = 1u << 1, CF_CY = 1u << 2,                          // centre stresses exist along x / y
    CF_X0 = 1u << 3, CF_X1 = 1u << 4, CF_Y0 = 1u << 5, CF_Y1 = 1u << 6,      // fixed shear nodes
    CF_TX0 = 1u << 7, CF_TX1 = 1u << 8, CF_TY0 = 1u << 9, CF_TY1 = 1u << 10, // traction ghosts beside
    CF_VX0 = 1u << 11, CF_VX1 = 1u << 12, CF_VY0 = 1u << 13, CF_VY1 = 1u << 14,  // fixed velocity nodes
    CF_ONX = 1u << 15, CF_ONY = 1u << 16, CF_ONC = 1u << 17,   // V.x / V.y / V.z and η exist here
    CF_IMG = 1u << 18,                                         // values here have images
    CF_XIMG = 1u << 20, CF_YIMG = 1u << 21,                    // along x or y alone
    CF_DUP = 1u << 19                                          // some have two along one dimension
};
constexpr unsigned CF_SHEAR = CF_X0 | CF_X1 | CF_Y0 | CF_Y1, CF_TRAC = CF_TX0 | CF_TX1 | CF_TY0 | CF_TY1;

template <typename T, int TX, int TY>
struct Ctx {
    using Lay = Layout<T, TX, TY>;
    T *sm;
    int i0, j0, kb, ke;
    int n0, n1, n2;
    long long sx, sxy;
    // the ghost layer on the low / high side of x / y comes from elsewhere: a periodic
    // image, or a neighbouring subdomain's halo (FI_BC_PERIODIC / FI_BC_HALO)
    bool hx0, hx1, hy0, hy1;
    // byte offsets of the slots of the step's planes: centre stresses of plane s, face
    // fields of s and s + 1
    unsigned C, V0, V1;

    __device__ __forceinline__ void set_plane(int s) {
        const unsigned p0 = (unsigned)s % 3u, p1 = p0 == 2u ? 0u : p0 + 1u;
        C = (s & 1) * (unsigned)(Lay::CS * sizeof(T));
        V0 = (unsigned)(2 * Lay::CS * sizeof(T)) + p0 * (unsigned)(Lay::VS * sizeof(T));
        V1 = (unsigned)(2 * Lay::CS * sizeof(T)) + p1 * (unsigned)(Lay::VS * sizeof(T));
    }
    __device__ __forceinline__ unsigned col(int li, int lj) const {
        return (unsigned)(i0 + li) + (unsigned)sx * (unsigned)(j0 + lj);
    }
};

// element of field F at the position (li, lj) from the column origin, in the slot at a
// byte offset: the boxes have three row pitches, so a step's addresses are a few byte
// offsets per thread plus constants
template <int F, int TX, int TY, typename T>
__device__ __forceinline__ T *el(unsigned slot, int li, int lj) {
    using B = FBox<T, TX, TY, F>;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    constexpr int K = (B::OFF - (B::oy * B::bw + B::ox)) * (int)sizeof(T);
    return reinterpret_cast<T *>(smem_raw + (slot + (unsigned)((lj * B::bw + li) * (int)sizeof(T))) + K);
}
#define EL(F, slot) (el<F, TX, TY, T>(slot, li, lj))

// A launch chained to the one before it (programmatic stream serialization) starts when that
// one's last blocks run: wait for its results, and let the next launch start likewise.  Set-up
// and launch latency then overlap the sweep before (47x33x29 FP64: 11.5 -> 9.3 us an
// iteration; 12 glaciers of 16^3-48^3 68 -> 63 us; nothing at 511^3).
__device__ __forceinline__ void chain_launches() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <typename T>
__device__ __forceinline__ T h(T x) { return T(0.5) * x; }

// issue the copies of group g: V, η of plane g; from kind 1 on the face stresses of
// plane g and P, τzz of plane g - 1; kind 2: all centre stresses of plane g - 1
template <typename T, int TX, int TY>
__device__ __forceinline__ void issue_group(const Ctx<T, TX, TY> &c, const InMaps &mp, int g, int kind, uint64_t *bars) {
    using Lay = Layout<T, TX, TY>;
    constexpr uint32_t vb = 4u * FBox<T, TX, TY, M_VX>::bytes;
    constexpr uint32_t fb = FBox<T, TX, TY, M_XZ>::bytes + FBox<T, TX, TY, M_YZ>::bytes + FBox<T, TX, TY, M_P>::bytes +
                            FBox<T, TX, TY, M_ZZ>::bytes;
    constexpr uint32_t cb = FBox<T, TX, TY, M_XX>::bytes + FBox<T, TX, TY, M_YY>::bytes + FBox<T, TX, TY, M_XY>::bytes;
    const int q = g % 3;
    uint64_t *bar = &bars[q];
    T *V = c.sm + 2 * Lay::CS + q * Lay::VS, *C = c.sm + ((g - 1) & 1) * Lay::CS;
    mbar_expect_tx(bar, vb + (kind > 0 ? fb : 0u) + (kind > 1 ? cb : 0u));
#define FI_LOAD(F, slot, plane)                                                                                  \
    tma_load_3d(slot + FBox<T, TX, TY, F>::OFF, &mp.m[F], (int)kXOff + c.i0 + FBox<T, TX, TY, F>::ox, \
                c.j0 + FBox<T, TX, TY, F>::oy, plane, bar)
    FI_LOAD(M_VX, V, g);
    FI_LOAD(M_VY, V, g);
    FI_LOAD(M_VZ, V, g);
    FI_LOAD(M_ET, V, g);
    if (kind > 0) {
        FI_LOAD(M_XZ, V, g);
        FI_LOAD(M_YZ, V, g);
        FI_LOAD(M_P, C, g - 1);
        FI_LOAD(M_ZZ, C, g - 1);
    }
    if (kind > 1) {
        FI_LOAD(M_XX, C, g - 1);
        FI_LOAD(M_YY, C, g - 1);
        FI_LOAD(M_XY, C, g - 1);
    }
#undef FI_LOAD
}

// ---- new stresses at (li, lj): values only, stored by the caller ----------------------
enum { F_P = 1, F_XX = 2, F_YY = 4, F_ZZ = 8 };

template <typename T>
struct Centre {
    T P, xx, yy, zz;
};

// P and the components of `mask` at plane s
template <int mask, typename T, int TX, int TY>
__device__ __forceinline__ Centre<T> centre_raw(const Ctx<T, TX, TY> &c, const KParams &p, const TConst<T> &q, int s, int li,
                                                int lj, const Ptrs<T> &out) {
    constexpr int BV = FBox<T, TX, TY, M_VX>::bw;
    const T *vx = EL(M_VX, c.V0), *vy = EL(M_VY, c.V0), *vz = EL(M_VZ, c.V0), *vzp = EL(M_VZ, c.V1);
    const T etac = *EL(M_ET, c.V0);
    Centre<T> r;
    const T oP = *EL(M_P, c.C);
    T oXX = T(0), oYY = T(0), oZZ = T(0);
    if (mask & F_XX) oXX = *EL(M_XX, c.C);
    if (mask & F_YY) oYY = *EL(M_YY, c.C);
    if (mask & F_ZZ) oZZ = *EL(M_ZZ, c.C);
    const T exx = (vx[1] - vx[0]) * q.inv_dx[0];
    const T eyy = (vy[BV] - vy[0]) * q.inv_dx[1];
    const T ezz = (vzp[0] - vz[0]) * q.inv_dx[2];
    const T divV = exx + eyy + ezz;
    r.P = oP - (p.p_forcing ? divV + __ldg(out.fP + c.sxy * s + c.col(li, lj)) : divV) * etac * q.dt_P;
    r.xx = oXX - (oXX - T(2.0) * etac * (exx - third(divV))) * q.dt_tau[0];
    r.yy = oYY - (oYY - T(2.0) * etac * (eyy - third(divV))) * q.dt_tau[1];
    r.zz = oZZ - (oZZ - T(2.0) * etac * (ezz - third(divV))) * q.dt_tau[2];
    return r;
}

// τxy at plane s
template <typename T, int TX, int TY>
__device__ __forceinline__ T xy_raw(const Ctx<T, TX, TY> &c, const TConst<T> &q, int li, int lj) {
    constexpr int BV = FBox<T, TX, TY, M_VX>::bw;
    const T *vx = EL(M_VX, c.V0), *vy = EL(M_VY, c.V0), *et = EL(M_ET, c.V0);
    const T o = *EL(M_XY, c.C);
    const T exy = T(0.5) * ((vy[0] - vy[-1]) * q.inv_dx[0] + (vx[0] - vx[-BV]) * q.inv_dx[1]);
    const T e_xy = h(h(et[-1 - BV] + et[-BV]) + h(et[-1] + et[0]));
    return o - (o - T(2.0) * e_xy * exy) * q.dt_tau[3];
}

// τxz and τyz at plane s + 1
template <typename T, int TX, int TY>
__device__ __forceinline__ T xz_raw(const Ctx<T, TX, TY> &c, const TConst<T> &q, int li, int lj) {
    const T *vx = EL(M_VX, c.V1), *vxm = EL(M_VX, c.V0), *vz = EL(M_VZ, c.V1);
    const T *et = EL(M_ET, c.V1), *etm = EL(M_ET, c.V0);
    const T o = *EL(M_XZ, c.V1);
    const T exz = T(0.5) * ((vz[0] - vz[-1]) * q.inv_dx[0] + (vx[0] - vxm[0]) * q.inv_dx[2]);
    const T e_xz = h(h(etm[-1] + etm[0]) + h(et[-1] + et[0]));
    return o - (o - T(2.0) * e_xz * exz) * q.dt_tau[4];
}
template <typename T, int TX, int TY>
__device__ __forceinline__ T yz_raw(const Ctx<T, TX, TY> &c, const TConst<T> &q, int li, int lj) {
    constexpr int BV = FBox<T, TX, TY, M_VX>::bw;
    const T *vy = EL(M_VY, c.V1), *vym = EL(M_VY, c.V0), *vz = EL(M_VZ, c.V1);
    const T *et = EL(M_ET, c.V1), *etm = EL(M_ET, c.V0);
    const T o = *EL(M_YZ, c.V1);
    const T eyz = T(0.5) * ((vz[0] - vz[-BV]) * q.inv_dx[1] + (vy[0] - vym[0]) * q.inv_dx[2]);
    const T e_yz = h(h(etm[-BV] + etm[0]) + h(et[-BV] + et[0]));
    return o - (o - T(2.0) * e_yz * eyz) * q.dt_tau[5];
}

// ---- boundary values of the shear stresses ------------------------------------------
__device__ __forceinline__ bool stress_fixed(int kind) { return kind == FI_BC_TRACTION || kind == FI_BC_SLIP; }

// fixed-node bits of a position
template <typename T, int TX, int TY>
__device__ __forceinline__ unsigned shear_flags(const Ctx<T, TX, TY> &c, const KParams &p, int i, int j) {
    unsigned f = 0;
    if (i == 1 && stress_fixed(p.bc_kind[0][0])) f |= CF_X0;
    if (i == c.n0 + 1 && stress_fixed(p.bc_kind[0][1])) f |= CF_X1;
    if (j == 1 && stress_fixed(p.bc_kind[1][0])) f |= CF_Y0;
    if (j == c.n1 + 1 && stress_fixed(p.bc_kind[1][1])) f |= CF_Y1;
    return f;
}
// x faces, then y faces, then z faces (a later dimension's value wins)
template <typename T>
__device__ __forceinline__ T fix_xy(const TConst<T> &q, T v, unsigned f) {
    if (f & CF_X0) v = q.bc_val[0][0][1];
    if (f & CF_X1) v = q.bc_val[0][1][1];
    if (f & CF_Y0) v = q.bc_val[1][0][0];
    if (f & CF_Y1) v = q.bc_val[1][1][0];
    return v;
}
template <typename T>
__device__ __forceinline__ T fix_xz(const TConst<T> &q, T v, unsigned f) {
    if (f & CF_X0) v = q.bc_val[0][0][2];
    if (f & CF_X1) v = q.bc_val[0][1][2];
    return v;
}
template <typename T>
__device__ __forceinline__ T fix_yz(const TConst<T> &q, T v, unsigned f) {
    if (f & CF_Y0) v = q.bc_val[1][0][2];
    if (f & CF_Y1) v = q.bc_val[1][1][2];
    return v;
}
// the side of plane k's z face with fixed shear stresses, or -1
template <typename T, int TX, int TY>
__device__ __forceinline__ int z_fixed(const Ctx<T, TX, TY> &c, const KParams &p, int k) {
    if (k == 1 && stress_fixed(p.bc_kind[2][0])) return 0;
    if (k == c.n2 + 1 && stress_fixed(p.bc_kind[2][1])) return 1;
    return -1;
}

// The ghosts of P and τxx (τyy) beside a traction side, from the values at the cell next
// to it; written by the thread that computed those, where the ghost lies in this CTA's
// column (or is its low ring).
template <typename T, int TX, int TY>
__device__ __forceinline__ void traction_x(const Ctx<T, TX, TY> &c, const TConst<T> &q, const Ptrs<T> &out, int s, int side,
                                           int lj, T P, T xx, bool write) {
    const int li = side == 0 ? -1 : c.n0 + 1 - c.i0;
    const T tv = T(2.0) * q.bc_val[0][side][0];
    *EL(M_P, c.C) = tv - P;
    *EL(M_XX, c.C) = tv - xx;
    if (write) {
        const long long I = c.sxy * s + c.col(li, lj);
        out.P[I] = tv - P;
        out.txx[I] = tv - xx;
    }
}
template <typename T, int TX, int TY>
__device__ __forceinline__ void traction_y(const Ctx<T, TX, TY> &c, const TConst<T> &q, const Ptrs<T> &out, int s, int side,
                                           int li, T P, T yy, bool write) {
    const int lj = side == 0 ? -1 : c.n1 + 1 - c.j0;
    const T tv = T(2.0) * q.bc_val[1][side][1];
    *EL(M_P, c.C) = tv - P;
    *EL(M_YY, c.C) = tv - yy;
    if (write) {
        const long long I = c.sxy * s + c.col(li, lj);
        out.P[I] = tv - P;
        out.tyy[I] = tv - yy;
    }
}

// Ring stresses of step s, one side per warp on the last warps (one per scheduler for
// 32-wide tiles): the row below (P, τyy), the row above (τxy, τyz), the column left
// (P, τxx), the column right (τxy, τxz) with the corner above it (τxy).
template <bool BND, typename T, int TX, int TY>
__device__ __forceinline__ void sigma_ring(const Ctx<T, TX, TY> &c, const KParams &p, const TConst<T> &q, const Ptrs<T> &out,
                                           int s, int zf, bool write) {
    constexpr int RW = TX / 32, NW = Layout<T, TX, TY>::NW;
    static_assert(TY < 32 && NW >= 2 * RW + 2, "one ring side per warp");
    const int w = (int)(threadIdx.x / 32) - (NW - 2 * RW - 2), lane = threadIdx.x % 32;
    const bool cz = s >= 1;  // s <= n2 in every step with stresses
    if (w < 0) return;
    if (w < RW) {
        const int li = lane + 32 * w, lj = -1, i = c.i0 + li, j = c.j0 - 1;
        if (cz && (!BND || ((i <= c.n0 || (c.hx1 && i == c.n0 + 1)) && (j >= 1 || c.hy0)))) {
            const Centre<T> v = centre_raw<F_P | F_YY>(c, p, q, s, li, lj, out);
            *EL(M_P, c.C) = v.P;
            *EL(M_YY, c.C) = v.yy;
            if (BND && j == 0 && write) {
                const long long I = c.sxy * s + c.col(li, lj);
                out.P[I] = v.P;
                out.tyy[I] = v.yy;
            }
            if (BND && j == c.n1 && p.bc_kind[1][1] == FI_BC_TRACTION) traction_y(c, q, out, s, 1, li, v.P, v.yy, write);
        }
    } else if (w < 2 * RW) {
        const int li = lane + 32 * (w - RW), lj = TY, i = c.i0 + li, j = c.j0 + TY;
        if (!BND || (i <= c.n0 + 1 && j <= c.n1 + 1)) {
            T xy = xy_raw(c, q, li, lj), yz = yz_raw(c, q, li, lj);
            if (BND) {
                const unsigned f = shear_flags(c, p, i, j);
                xy = fix_xy(q, xy, f);
                yz = fix_yz(q, yz, f);
            }
            if (zf >= 0) yz = q.bc_val[2][zf][1];
            *EL(M_XY, c.C) = xy;
            *EL(M_YZ, c.V1) = yz;
        }
    } else if (w == 2 * RW) {
        const int li = -1, lj = lane, i = c.i0 - 1, j = c.j0 + lane;
        if (lane < TY && cz && (!BND || ((i >= 1 || c.hx0) && (j <= c.n1 || (c.hy1 && j == c.n1 + 1))))) {
            const Centre<T> v = centre_raw<F_P | F_XX>(c, p, q, s, li, lj, out);
            *EL(M_P, c.C) = v.P;
            *EL(M_XX, c.C) = v.xx;
            if (BND && i == 0 && write) {
                const long long I = c.sxy * s + c.col(li, lj);
                out.P[I] = v.P;
                out.txx[I] = v.xx;
            }
            if (BND && i == c.n0 && p.bc_kind[0][1] == FI_BC_TRACTION) traction_x(c, q, out, s, 1, lj, v.P, v.xx, write);
        }
    } else {
        const int li = TX, lj = lane, i = c.i0 + TX, j = c.j0 + lane;
        if (lane <= TY && (!BND || (i <= c.n0 + 1 && j <= c.n1 + 1))) {
            T xy = xy_raw(c, q, li, lj), xz = T(0);
            if (lane < TY) xz = xz_raw(c, q, li, lj);
            if (BND) {
                const unsigned f = shear_flags(c, p, i, j);
                xy = fix_xy(q, xy, f);
                xz = fix_xz(q, xz, f);
            }
            if (zf >= 0) xz = q.bc_val[2][zf][0];
            *EL(M_XY, c.C) = xy;
            if (lane < TY) *EL(M_XZ, c.V1) = xz;
        }
    }
}

// values of the thread's column that V.z needs from plane to plane
template <typename T>
struct Carry {
    T P, zz;    // new values of the step's plane
    T Pm, zzm;  // of the plane below
    T etm;      // η of the plane below
};

// New stresses of step s at the thread's position, stored with their boundary values.  wc:
// the centre stresses and τxy of plane s belong to this z-block; wf: τxz, τyz of plane
// s + 1 do.
template <bool BND, typename T, int TX, int TY>
__device__ __forceinline__ void sigma_store(const Ctx<T, TX, TY> &c, const KParams &p, const TConst<T> &q, const Ptrs<T> &out,
                                            int s, int li, int lj, unsigned fl, int zf, bool wc, bool wf, long long I,
                                            const Centre<T> &v, T xy, T xz, T yz, Carry<T> &k) {
    const bool cz = s >= 1;
    const bool cx = !BND || (fl & CF_CX), cy = !BND || (fl & CF_CY);
    if (BND && (fl & CF_SHEAR)) {
        xy = fix_xy(q, xy, fl);
        xz = fix_xz(q, xz, fl);
        yz = fix_yz(q, yz, fl);
    }
    if (zf >= 0) {
        xz = q.bc_val[2][zf][0];
        yz = q.bc_val[2][zf][1];
    }
    const bool dc = cx && cy && cz;
    if (dc) {
        *EL(M_P, c.C) = v.P;
        *EL(M_XX, c.C) = v.xx;
        *EL(M_YY, c.C) = v.yy;
    }
    *EL(M_XY, c.C) = xy;
    *EL(M_XZ, c.V1) = xz;
    *EL(M_YZ, c.V1) = yz;
    k.P = v.P;
    k.zz = v.zz;
    if (wc) {
        if (dc) {
            out.P[I] = v.P;
            out.txx[I] = v.xx;
            out.tyy[I] = v.yy;
            out.tzz[I] = v.zz;
        }
        if (!BND || (fl & CF_IN)) out.txy[I] = xy;
    }
    if (wf && (!BND || (fl & CF_IN))) {
        if (cy) out.txz[I + c.sxy] = xz;
        if (cx) out.tyz[I + c.sxy] = yz;
    }
    if (BND && dc && (fl & CF_TRAC)) {
        if (fl & CF_TX0) traction_x(c, q, out, s, 0, lj, v.P, v.xx, wc);
        if (fl & CF_TX1) traction_x(c, q, out, s, 1, lj, v.P, v.xx, wc);
        if (fl & CF_TY0) traction_y(c, q, out, s, 0, li, v.P, v.yy, wc);
        if (fl & CF_TY1) traction_y(c, q, out, s, 1, li, v.P, v.yy, wc);
    }
    // the ghosts under a traction bottom
    if (s == 1 && p.bc_kind[2][0] == FI_BC_TRACTION) {
        const T tv = T(2.0) * q.bc_val[2][0][2];
        k.Pm = tv - v.P;
        k.zzm = tv - v.zz;
        if (wc && dc) {
            out.P[I - c.sxy] = k.Pm;
            out.tzz[I - c.sxy] = k.zzm;
        }
    }
}

template <bool BND, typename T, int TX, int TY>
__device__ __forceinline__ void sigma_column(const Ctx<T, TX, TY> &c, const KParams &p, const TConst<T> &q, const Ptrs<T> &out,
                                             int s, int li, int lj, unsigned fl, int zf, bool wc, bool wf, long long I,
                                             Carry<T> &k) {
    const Centre<T> v = centre_raw<F_P | F_XX | F_YY | F_ZZ>(c, p, q, s, li, lj, out);
    const T xy = xy_raw(c, q, li, lj), xz = xz_raw(c, q, li, lj), yz = yz_raw(c, q, li, lj);
    sigma_store<BND>(c, p, q, out, s, li, lj, fl, zf, wc, wf, I, v, xy, xz, yz, k);
}

// ---- ghost / image writes ---------------------------------------------------------------
template <typename T>
struct Img {
    int d;     // offset along the dimension of the value's image beside it (0: none)
    int d2;    // of a second one, a copy: next to one physical and one foreign side
    bool dir;  // the first is a Dirichlet ghost 2c - v (else a copy)
    T c;
};

// Center-located value at index q (1..N) along a dim with BC kinds kl/kr; lo / hi: the
// low / high ghost comes from elsewhere (a periodic image of this model's own value,
// which a subdomain's halo exchange replaces with its neighbour's).  neumann: copies
// (η_next); else Velocity-BC ghosts 2c - v of a velocity component.  Dimensions have 3
// or more cells.
template <typename T>
__device__ __forceinline__ Img<T> img_center(int q, int N, bool lo, bool hi, int kl, int kr, T cl, T cr, bool neumann) {
    Img<T> r{0, 0, false, T(0)};
    if (q == 1 && !lo && (neumann || kl == FI_BC_VELOCITY)) r = {-1, 0, !neumann, cl};
    if (q == N && !hi && (neumann || kr == FI_BC_VELOCITY)) r = {1, 0, !neumann, cr};
    const int away = (q == N && lo) ? -N : (q == 1 && hi) ? N : 0;
    (r.d ? r.d2 : r.d) = away;
    return r;
}
template <typename T>
__device__ __forceinline__ Img<T> img_vertex(int q, int N, bool lo, bool hi) {
    Img<T> r{0, 0, false, T(0)};
    if (lo && q == N) r.d = -N;
    if (hi && (q == 1 || q == 2)) r.d = N;
    return r;
}

// the images of v (x, then y, then z: an image of an image follows both rules)
template <typename T>
__device__ __forceinline__ T img_value(const Img<T> &m, T v) { return m.dir ? T(2.0) * m.c - v : v; }

template <typename T>
__device__ __forceinline__ void put_images(T *f, T v, const Img<T> &x, const Img<T> &y, long long sx, const Img<T> &z,
                                           long long sxy, bool dup) {
    const T vx = img_value(x, v);
    if (x.d) f[x.d] = vx;
    if (y.d) {
        T *fy = f + sx * y.d;
        fy[0] = img_value(y, v);
        if (x.d) fy[x.d] = img_value(y, vx);
    }
    if (z.d) {
        T *fz = f + sxy * z.d;
        fz[0] = img_value(z, v);
        if (x.d) fz[x.d] = img_value(z, vx);
        if (y.d) {
            fz[sx * y.d] = img_value(z, img_value(y, v));
            if (x.d) fz[sx * y.d + x.d] = img_value(z, img_value(y, vx));
        }
    }
    if (!dup) return;
    // second images (a physical and a foreign side): copies, with the first images of the
    // other dimensions
#pragma unroll 1
    for (int e = 0; e < 18; e++) {
        const int a = e % 3, b = (e / 3) % 3, g = e / 9;
        const int da = a == 0 ? 0 : a == 1 ? x.d : x.d2, db = b == 0 ? 0 : b == 1 ? y.d : y.d2, dg = g ? z.d : 0;
        if ((a != 2 && b != 2) || (a && !da) || (b && !db) || (g && !dg)) continue;
        T u = a == 1 ? img_value(x, v) : v;
        u = b == 1 ? img_value(y, u) : u;
        u = g == 1 ? img_value(z, u) : u;
        f[da + sx * db + sxy * dg] = u;
    }
}

// ---- velocity / η_next update of plane t on the column ----------------------------------
// The thread's neighbours in shared memory; P, τzz and η of the plane below from Carry.
template <typename T, int TX, int TY>
__device__ __forceinline__ T vx_raw(const Ctx<T, TX, TY> &c, const TConst<T> &q, int li, int lj, T gx) {
    constexpr int BY = FBox<T, TX, TY, M_XY>::bw;
    const T *P = EL(M_P, c.C), *xx = EL(M_XX, c.C), *xy = EL(M_XY, c.C), *et = EL(M_ET, c.V0);
    const T ex = h(et[-1] + et[0]);
    return *EL(M_VX, c.V0) +
           div_fast(-(P[0] - P[-1]) * q.inv_dx[0] + (xx[0] - xx[-1]) * q.inv_dx[0] + (xy[BY] - xy[0]) * q.inv_dx[1] +
                        (*EL(M_XZ, c.V1) - *EL(M_XZ, c.V0)) * q.inv_dx[2] - gx,
                    ex) *
               q.dt_V[0];
}
template <typename T, int TX, int TY>
__device__ __forceinline__ T vy_raw(const Ctx<T, TX, TY> &c, const TConst<T> &q, int li, int lj, T gy) {
    constexpr int BP = FBox<T, TX, TY, M_P>::bw, BYY = FBox<T, TX, TY, M_YY>::bw, BV = FBox<T, TX, TY, M_ET>::bw;
    const T *P = EL(M_P, c.C), *yy = EL(M_YY, c.C), *xy = EL(M_XY, c.C), *et = EL(M_ET, c.V0);
    const T ey = h(et[-BV] + et[0]);
    return *EL(M_VY, c.V0) +
           div_fast(-(P[0] - P[-BP]) * q.inv_dx[1] + (yy[0] - yy[-BYY]) * q.inv_dx[1] + (xy[1] - xy[0]) * q.inv_dx[0] +
                        (*EL(M_YZ, c.V1) - *EL(M_YZ, c.V0)) * q.inv_dx[2] - gy,
                    ey) *
               q.dt_V[1];
}
template <typename T, int TX, int TY>
__device__ __forceinline__ T vz_raw(const Ctx<T, TX, TY> &c, const TConst<T> &q, int li, int lj, T gz, const Carry<T> &k) {
    constexpr int BYZ = FBox<T, TX, TY, M_YZ>::bw;
    const T *xz = EL(M_XZ, c.V0), *yz = EL(M_YZ, c.V0);
    const T ez = h(k.etm + *EL(M_ET, c.V0));
    return *EL(M_VZ, c.V0) +
           div_fast(-(k.P - k.Pm) * q.inv_dx[2] + (k.zz - k.zzm) * q.inv_dx[2] + (xz[1] - xz[0]) * q.inv_dx[0] +
                        (yz[BYZ] - yz[0]) * q.inv_dx[1] - gz,
                    ez) *
               q.dt_V[2];
}
template <bool IB, typename T, int TX, int TY>
__device__ __forceinline__ T eta_raw(const Ctx<T, TX, TY> &c, const KParams &p, const TConst<T> &q, const Ptrs<T> &in, int li,
                                     int lj, long long I, T zz) {
    // a linear viscosity without regularisation or relaxation does not read the stresses
    if (linear_unrelaxed(p)) return p.rheo_eta_is_field ? in.eta_lin[I] : T(p.rheo_eta);
    constexpr int BY = FBox<T, TX, TY, M_XY>::bw, BYZ = FBox<T, TX, TY, M_YZ>::bw;
    const T xx = *EL(M_XX, c.C), yy = *EL(M_YY, c.C);
    const T *xy = EL(M_XY, c.C);
    const T *xz = EL(M_XZ, c.V0), *xzp = EL(M_XZ, c.V1), *yz = EL(M_YZ, c.V0), *yzp = EL(M_YZ, c.V1);
    const T lxy = h(h(xy[0] + xy[1]) + h(xy[BY] + xy[BY + 1]));
    const T lxz = h(h(xz[0] + xz[1]) + h(xzp[0] + xzp[1]));
    const T lyz = h(h(yz[0] + yz[BYZ]) + h(yzp[0] + yzp[BYZ]));
    T s2;
    if constexpr (IB) s2 = fma_r(lyz, lyz, fma_r(lxz, lxz, fma_r(lxy, lxy, h(fma_r(zz, zz, sum_r(xx, xx, yy, yy))))));
    else s2 = T(0.5) * (xx * xx + yy * yy + zz * zz) + lxy * lxy + lxz * lxz + lyz * lyz;
    return rheology_s2(p, q.rheo_A, q.rheo_inv_eta_reg, in.eta_lin, in.A, *EL(M_ET, c.V0), I, s2);
}

__device__ __forceinline__ bool node_fixed(int kind) { return kind == FI_BC_SLIP || kind == FI_BC_VELOCITY; }

// the ghost images of the four values at (t, i, j)
template <typename T, int TX, int TY>
__device__ __forceinline__ void v_images(const Ctx<T, TX, TY> &c, const KParams &p, const TConst<T> &q, const Ptrs<T> &out,
                                         int t, int li, int lj, unsigned fl, long long I, T vx, T vy, T vz, T et) {
    const int n0 = c.n0, n1 = c.n1, n2 = c.n2, i = c.i0 + li, j = c.j0 + lj;
    const int xl = p.bc_kind[0][0], xr = p.bc_kind[0][1], yl = p.bc_kind[1][0], yr = p.bc_kind[1][1];
    const int zl = p.bc_kind[2][0], zr = p.bc_kind[2][1];
    const bool cz = t <= n2, dup = fl & CF_DUP;
    const bool y_node = fl & (CF_VY0 | CF_VY1), z_node = (t == 1 && node_fixed(zl)) || (t == n2 + 1 && node_fixed(zr));
    // A value on a fixed node of its own dim d is written there last by the
    // reference's dim-d node assignment, which spans the ghosts of the dims before
    // d: its images along those dims are copies, not mirrors (as_copies).
    auto as_copies = [](Img<T> m, bool yes) {
        m.dir = m.dir && !yes;
        return m;
    };
    const Img<T> none{0, 0, false, T(0)};
    if ((fl & CF_ONX) && cz)  // V.x at (V, C, C)
        put_images(out.Vx + I, vx, img_vertex<T>(i, n0, c.hx0, c.hx1),
                   img_center<T>(j, n1, c.hy0, c.hy1, yl, yr, q.bc_val[1][0][0], q.bc_val[1][1][0], false), c.sx,
                   img_center<T>(t, n2, false, false, zl, zr, q.bc_val[2][0][0], q.bc_val[2][1][0], false), c.sxy, dup);
    if ((fl & CF_ONY) && cz)  // V.y at (C, V, C)
        put_images(out.Vy + I, vy,
                   as_copies(img_center<T>(i, n0, c.hx0, c.hx1, xl, xr, q.bc_val[0][0][1], q.bc_val[0][1][1], false), y_node),
                   img_vertex<T>(j, n1, c.hy0, c.hy1), c.sx,
                   img_center<T>(t, n2, false, false, zl, zr, q.bc_val[2][0][1], q.bc_val[2][1][1], false), c.sxy, dup);
    if (fl & CF_ONC)  // V.z at (C, C, V)
        put_images(out.Vz + I, vz,
                   as_copies(img_center<T>(i, n0, c.hx0, c.hx1, xl, xr, q.bc_val[0][0][2], q.bc_val[0][1][2], false), z_node),
                   as_copies(img_center<T>(j, n1, c.hy0, c.hy1, yl, yr, q.bc_val[1][0][2], q.bc_val[1][1][2], false), z_node),
                   c.sx, none, c.sxy, dup);
    if (!p.freeze_eta && (fl & CF_ONC) && cz)  // η_next at (C, C, C), Neumann / periodic ghosts
        put_images(out.eta_next + I, et, img_center<T>(i, n0, c.hx0, c.hx1, xl, xr, T(0), T(0), true),
                   img_center<T>(j, n1, c.hy0, c.hy1, yl, yr, T(0), T(0), true), c.sx,
                   img_center<T>(t, n2, false, false, zl, zr, T(0), T(0), true), c.sxy, dup);
}

// The images of a cell beside one x or y side (dim) away from all others: the general path
// costs every warp of a column along an x side its length at every plane (127^3 FP64 walls:
// 104 us an iteration without this path, 98 with it).
template <typename T, int TX, int TY>
__device__ __forceinline__ void v_images_one(const Ctx<T, TX, TY> &c, const KParams &p, const TConst<T> &q, const Ptrs<T> &out,
                                             int dim, int li, int lj, long long I, T vx, T vy, T vz, T et) {
    const int at = dim ? c.j0 + lj : c.i0 + li, n = dim ? c.n1 : c.n0;
    const bool foreign = dim ? c.hy0 : c.hx0;
    const int side = at == n, kind = p.bc_kind[dim][side];
    const long long d = (foreign ? (side ? -n : n) : (side ? 1 : -1)) * (dim ? c.sx : 1LL);
    T *along = dim ? out.Vy : out.Vx, *across = dim ? out.Vx : out.Vy;
    if (foreign) along[I + d] = dim ? vy : vx;
    if (foreign && at == 2) return;  // (a second node beside the side, not a second cell)
    if (foreign || kind == FI_BC_VELOCITY) {
        const T v = dim ? vx : vy;
        across[I + d] = foreign ? v : T(2.0) * q.bc_val[dim][side][dim ? 0 : 1] - v;
        out.Vz[I + d] = foreign ? vz : T(2.0) * q.bc_val[dim][side][2] - vz;
    }
    if (!p.freeze_eta) out.eta_next[I + d] = et;
}

// V and η_next of plane t.  Every value is computed (its operands lie in the boxes even
// where no such point exists), then replaced at fixed nodes and stored where it exists.
template <bool BND, bool IB = false, typename T, int TX, int TY>
__device__ __forceinline__ void v_store(const Ctx<T, TX, TY> &c, const KParams &p, const TConst<T> &q, const Ptrs<T> &in,
                                        const Ptrs<T> &out, int t, int li, int lj, unsigned fl, long long I, const Carry<T> &k,
                                        T vxn, T vyn, T vzn) {
    const bool cz = t <= c.n2;
    const bool on_c = !BND || (fl & CF_ONC);
    T etn = T(0);
    if (!p.freeze_eta && on_c && cz) etn = eta_raw<IB>(c, p, q, in, li, lj, I, k.zz);
    if (BND) {
        if (fl & CF_VX0) vxn = q.bc_val[0][0][0];
        if (fl & CF_VX1) vxn = q.bc_val[0][1][0];
        if (fl & CF_VY0) vyn = q.bc_val[1][0][1];
        if (fl & CF_VY1) vyn = q.bc_val[1][1][1];
    }
    if (t == 1 && node_fixed(p.bc_kind[2][0])) vzn = q.bc_val[2][0][2];
    if (!cz && node_fixed(p.bc_kind[2][1])) vzn = q.bc_val[2][1][2];
    if (cz) {
        if (!BND || (fl & CF_ONX)) out.Vx[I] = vxn;
        if (!BND || (fl & CF_ONY)) out.Vy[I] = vyn;
        if (!p.freeze_eta && on_c) out.eta_next[I] = etn;
    }
    if (on_c) out.Vz[I] = vzn;
    const bool ends = t == 1 || t >= c.n2;
    if (BND && (fl & (CF_XIMG | CF_YIMG)) && !ends) v_images_one(c, p, q, out, fl & CF_YIMG ? 1 : 0, li, lj, I, vxn, vyn, vzn, etn);
    else if (ends || (BND && (fl & CF_IMG))) v_images(c, p, q, out, t, li, lj, fl, I, vxn, vyn, vzn, etn);
}

template <bool BND, typename T, int TX, int TY>
__device__ __forceinline__ void v_column(const Ctx<T, TX, TY> &c, const KParams &p, const TConst<T> &q, const Ptrs<T> &in,
                                         const Ptrs<T> &out, int t, int li, int lj, unsigned fl, long long I, const Carry<T> &k,
                                         T gx, T gy, T gz) {
    const T vxn = vx_raw(c, q, li, lj, gx), vyn = vy_raw(c, q, li, lj, gy), vzn = vz_raw(c, q, li, lj, gz, k);
    v_store<BND>(c, p, q, in, out, t, li, lj, fl, I, k, vxn, vyn, vzn);
}

// body force at a point of V; loaded ahead of the step's barrier
template <typename T>
__device__ __forceinline__ T body_force(const KParams &p, const TConst<T> &q, const T *g, int d, long long I) {
    return p.g_kind[d] == FI_G_FIELD ? __ldg(g + I) : q.g_val[d];
}

template <typename T, int TX, int TY>
__device__ __forceinline__ unsigned column_flags(const Ctx<T, TX, TY> &c, const KParams &p, int i, int j) {
    if (i > c.n0 + 1 || j > c.n1 + 1) return 0u;
    unsigned f = CF_IN | shear_flags(c, p, i, j);
    const int xl = p.bc_kind[0][0], xr = p.bc_kind[0][1], yl = p.bc_kind[1][0], yr = p.bc_kind[1][1];
    if (i <= c.n0 || c.hx1) f |= CF_CX;
    if (j <= c.n1 || c.hy1) f |= CF_CY;
    if (xl == FI_BC_TRACTION && i == 1) f |= CF_TX0;
    if (xr == FI_BC_TRACTION && i == c.n0 && c.n0 + 1 < c.i0 + TX) f |= CF_TX1;
    if (yl == FI_BC_TRACTION && j == 1) f |= CF_TY0;
    if (yr == FI_BC_TRACTION && j == c.n1 && c.n1 + 1 < c.j0 + TY) f |= CF_TY1;
    if (!c.hx0 && i == 1 && node_fixed(xl)) f |= CF_VX0;
    if (!c.hx1 && i == c.n0 + 1 && node_fixed(xr)) f |= CF_VX1;
    if (!c.hy0 && j == 1 && node_fixed(yl)) f |= CF_VY0;
    if (!c.hy1 && j == c.n1 + 1 && node_fixed(yr)) f |= CF_VY1;
    if (j <= c.n1 && !(c.hx1 && i == c.n0 + 1)) f |= CF_ONX;
    if (i <= c.n0 && !(c.hy1 && j == c.n1 + 1)) f |= CF_ONY;
    if (i <= c.n0 && j <= c.n1) f |= CF_ONC;
    const bool xi = i == 1 || i == c.n0 || (c.hx1 && i == 2), yi = j == 1 || j == c.n1 || (c.hy1 && j == 2);
    if (xi || yi) f |= CF_IMG;
    if (xi != yi && i <= c.n0 && j <= c.n1 && c.hx0 == c.hx1 && c.hy0 == c.hy1) f |= xi ? CF_XIMG : CF_YIMG;
    if (c.hx0 != c.hx1 || c.hy0 != c.hy1) f |= CF_DUP;
    return f;
}

// the plane march of one CTA (BND: the column touches an x or y boundary)
template <bool BND, typename T, int TX, int TY>
__device__ __forceinline__ void sweep(Ctx<T, TX, TY> &c, const KParams &p, const TConst<T> &q, const Ptrs<T> &in,
                                      const Ptrs<T> &out, const InMaps &maps, uint64_t *bars, unsigned *released, int *err) {
    constexpr int NW = Layout<T, TX, TY>::NW;
    const int tid = threadIdx.x;
    const int li = tid % TX, lj = tid / TX;
    const int first = c.kb - 1;
    const int last = min(c.ke - 1, c.n2);  // last step that computes stresses
    const int gmax = last + 1;             // last group it needs
    if (tid == 0) {
        issue_group(c, maps, first, 0, bars);
        issue_group(c, maps, first + 1, 1, bars);
        if (first + 2 <= gmax) issue_group(c, maps, first + 2, 2, bars);
    }
    const unsigned fl = BND ? column_flags(c, p, c.i0 + li, c.j0 + lj) : (CF_ONX | CF_ONY | CF_ONC);
    const bool inside = !BND || (fl & CF_IN);
    uint32_t phase = 0;  // bit b: parity of the next completion of bars[b]
    auto wait_group = [&](int g) -> bool {
        const int b = g % 3;
        const bool ok = mbar_wait(&bars[b], (phase >> b) & 1u);
        phase ^= 1u << b;
        return ok;
    };
    Carry<T> k{T(0), T(0), T(0), T(0), T(0)};
    long long I = c.sxy * first + c.col(li, lj);
    bool ok = wait_group(first);
    for (int s = first; s <= last && ok; s++, I += c.sxy) {
        c.set_plane(s);
        const bool own = s >= c.kb;
        const int zf = z_fixed(c, p, s + 1);
        ok = wait_group(s + 1);
        if (!ok) break;
        sigma_column<BND>(c, p, q, out, s, li, lj, fl, zf, own, s + 1 < c.ke, I, k);
        sigma_ring<BND>(c, p, q, out, s, zf, own);
        if (own) {
            T gx = q.g_val[0], gy = q.g_val[1], gz = q.g_val[2];
            if (inside) {
                gx = body_force(p, q, in.gx, 0, I);
                gy = body_force(p, q, in.gy, 1, I);
                gz = body_force(p, q, in.gz, 2, I);
            }
            __syncthreads();
            v_column<BND>(c, p, q, in, out, s, li, lj, fl, I, k, gx, gy, gz);
        }
        k.Pm = k.P;
        k.zzm = k.zz;
        k.etm = *EL(M_ET, c.V0);
        // the warp is done with the slots of this step; the last one to say so refills them
        __syncwarp();
        if (s + 3 <= gmax && tid % 32 == 0) {
            unsigned n;
            asm volatile("atom.add.acq_rel.cta.shared::cta.u32 %0, [%1], 1;" : "=r"(n) : "r"(smem_u32(released)) : "memory");
            if (n % NW == NW - 1) {
                fence_proxy_async();
                issue_group(c, maps, s + 3, 2, bars);
            }
        }
    }
    if (ok) {
        if (c.ke - 1 == c.n2 + 1) {
            // the top plane of vertices: V.z, and the ghosts over a traction top
            const int t = c.n2 + 1;
            c.set_plane(t);
            if (c.kb == t) __syncthreads();  // no step before this one had a barrier
            if (inside && p.bc_kind[2][1] == FI_BC_TRACTION) {
                const T tv = T(2.0) * q.bc_val[2][1][2];
                k.P = tv - k.Pm;
                k.zz = tv - k.zzm;
                if (!BND || ((fl & CF_CX) && (fl & CF_CY))) {
                    out.P[I] = k.P;
                    out.tzz[I] = k.zz;
                }
            }
            const T gz = inside ? body_force(p, q, in.gz, 2, I) : T(0);
            v_column<BND>(c, p, q, in, out, t, li, lj, fl, I, k, T(0), T(0), gz);
        }
        return;
    }
    // bounded wait expired: record it and drain this CTA's own copies (bounded) before leaving
    atomicExch(err, (int)FI_ERR_TIMEOUT);
    for (int b = 0; b < kBars; b++) mbar_wait(&bars[b], (phase >> b) & 1u);
}

}  // namespace

}  // namespace fi
