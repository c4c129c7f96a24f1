// fi_tile2d.cu -- several PT iterations of a 2D model in one launch.
//
// Reference semantics: advance_iteration! of the 2D IsothermalFullStokesModel
// (src/Models/FullStokes/Isothermal/Isothermal.jl:91-112, kernels_2d.jl:3-29,
// boundary_conditions.jl:26-47 and :104-115), operation by operation as the
// reference-shaped kernels (fi_reference.cu) do it, so the no-FMA build matches the CPU
// oracle bit for bit.
//
// A 2D state is small (the 1021 x 509 FP64 section holds 33 MB, 128^2 one) and an
// iteration as six launches is bound by their latency (13.8 us at 128^2, 21.9 us at
// 1021 x 509).  Here a CTA loads a region of RX x RY positions into shared memory, runs k
// whole iterations on it and writes the inner (RX - 2k) x (RY - 2k) positions to the
// model's other state buffer.  V at a point depends on the old V one position away, so
// what is wrong at the region's edge moves inwards by one position an iteration: the k
// layers around the tile are recomputed by the neighbouring CTAs and thrown away here.
// No CTA waits for another.  A thread owns PY consecutive rows of one column: its own
// values and the neighbours above and below inside the strip stay in registers.
//
// Boundary values are applied by the thread that computes the value next to them: fixed
// nodes replace it, ghosts (traction mirrors of P and τ, Velocity mirrors of V, Neumann
// copies of η) go to the neighbouring shared-memory positions.  A periodic dimension has
// no ghosts inside a launch: the region wraps around.
//
// What bounds it.  Small grids: the launch and the load latency, then the two barriers and
// the FP64 chains of an iteration.  Large grids: FP64 issue and shared-memory bandwidth
// over 1.5-1.8 times the points (recomputed layers); the state stays in L2.
#include "fi_device.cuh"
#include "fi_model.h"

namespace fi {
namespace {

template <typename T>
__device__ __forceinline__ T h(T x) { return T(0.5) * x; }

enum PointFlag : unsigned {
    PF_C = 1u << 0,                                                   // centre values exist
    PF_XY = 1u << 1,                                                  // τxy exists
    PF_X0 = 1u << 2, PF_X1 = 1u << 3, PF_Y0 = 1u << 4, PF_Y1 = 1u << 5,      // τxy fixed by a side
    PF_TX0 = 1u << 6, PF_TX1 = 1u << 7, PF_TY0 = 1u << 8, PF_TY1 = 1u << 9,  // traction ghosts beside
    PF_VX = 1u << 10, PF_VY = 1u << 11,                               // V.x, V.y exist
    PF_FX0 = 1u << 12, PF_FX1 = 1u << 13, PF_FY0 = 1u << 14, PF_FY1 = 1u << 15,  // fixed velocity nodes
    PF_GX0 = 1u << 16, PF_GX1 = 1u << 17, PF_GY0 = 1u << 18, PF_GY1 = 1u << 19   // ghosts beside, per side
};
constexpr unsigned PF_SHEAR = PF_X0 | PF_X1 | PF_Y0 | PF_Y1, PF_TRAC = PF_TX0 | PF_TX1 | PF_TY0 | PF_TY1;
constexpr unsigned PF_NODE = PF_FX0 | PF_FX1 | PF_FY0 | PF_FY1, PF_GHOST = PF_GX0 | PF_GX1 | PF_GY0 | PF_GY1;

template <typename T, int RX, int RY, int PY>
struct Region {
    static constexpr int NT = RX * RY / PY;
    static constexpr int PW = RX + 2;                 // row pitch: one position of padding on each side
    static constexpr int PLANE = PW * (RY + 2);
    static constexpr size_t SMEM = 7 * (size_t)PLANE * sizeof(T);
};

struct TileArgs {
    int k;           // iterations of this launch
    int tx, ty;      // inner tile
    int write_prev;  // the last launch of an advance: also write η of the iteration before
};

__device__ __forceinline__ bool t2_fixed(int kind) { return kind == FI_BC_SLIP || kind == FI_BC_VELOCITY; }
__device__ __forceinline__ bool t2_shear(int kind) { return kind == FI_BC_TRACTION || kind == FI_BC_SLIP; }

// storage index of position g along a dimension of n cells: itself, or wrapped into 1..n
__device__ __forceinline__ int t2_wrap(int g, int n, bool per) {
    if (!per) return g;
    int m = (g - 1) % n;
    return (m < 0 ? m + n : m) + 1;
}

// the values of a thread's strip
template <typename T, int PY>
struct Strip {
    T P[PY], xx[PY], yy[PY], xy[PY], vx[PY], vy[PY], et[PY], ep[PY];
    T gx[PY], gy[PY];  // body force, where it is a field
    unsigned fl[PY];
    unsigned at[PY];  // storage index of the point (the first position where there is none)
};

// The k iterations of a region.  EDGE: it touches a side that is not periodic.  Every point
// computes; where no such value exists the result is not stored, and what the strip keeps
// of it is replaced by the ghost that another thread has put there.
template <bool EDGE, bool GF, bool BATCH, typename T, int RX, int RY, int PY>
__device__ __forceinline__ void iterate(const KParams &p, const TConst<T> &q, const Ptrs<T> &in, Strip<T, PY> &v, T *sP, int a0,
                                        int k) {
    using R = Region<T, RX, RY, PY>;
    constexpr int PW = R::PW;
    T *sXX = sP + R::PLANE, *sYY = sXX + R::PLANE, *sXY = sYY + R::PLANE;
    T *sVx = sXY + R::PLANE, *sVy = sVx + R::PLANE, *sE = sVy + R::PLANE;
    const T idx = q.inv_dx[0], idy = q.inv_dx[1];
    const bool linear = linear_unrelaxed(p), frozen = p.freeze_eta, forced = p.p_forcing;
#pragma unroll 1
    for (int it = 0; it < k; it++) {
        // ---- update_σ! (kernels_2d.jl:3-18): V and η of the iteration before ----
        T etl[PY], etd[PY];
        T vxd = sVx[a0 - PW], ed = sE[a0 - PW], edl = sE[a0 - PW - 1];  // the row below the strip
#pragma unroll
        for (int r = 0; r < PY; r++) {
            const int a = a0 + r * PW;
            const T vyu = r + 1 < PY ? v.vy[r + 1] : sVy[a + PW];
            const T el = sE[a - 1];
            etl[r] = el;
            etd[r] = ed;
            const T s[3] = {sVx[a + 1] - v.vx[r], vyu - v.vy[r], T(0)};
            T d[3];
            const T divV = rates_r<2, BATCH || sizeof(T) == 4>(s, q.inv_dx, d);
            const T exy = h(sum_r(v.vy[r] - sVy[a - 1], idx, v.vx[r] - vxd, idy));
            const T dv = forced ? divV + __ldg(in.fP + v.at[r]) : divV;
            const T nP = fma_r(-mul_r(dv, v.et[r]), q.dt_P, v.P[r]);
            const T nxx = relax_r(v.xx[r], T(2.0) * v.et[r], d[0], q.dt_tau[0]);
            const T nyy = relax_r(v.yy[r], T(2.0) * v.et[r], d[1], q.dt_tau[1]);
            const T e_xy = h(h(edl + ed) + h(el + v.et[r]));
            T nxy = relax_r(v.xy[r], T(2.0) * e_xy, exy, q.dt_tau[3]);
            vxd = v.vx[r];
            ed = v.et[r];
            edl = el;
            const unsigned f = v.fl[r];
            if (EDGE && (f & PF_SHEAR)) {
                if (f & PF_X0) nxy = q.bc_val[0][0][1];
                if (f & PF_X1) nxy = q.bc_val[0][1][1];
                if (f & PF_Y0) nxy = q.bc_val[1][0][0];
                if (f & PF_Y1) nxy = q.bc_val[1][1][0];
            }
            v.P[r] = nP, v.xx[r] = nxx, v.yy[r] = nyy, v.xy[r] = nxy;
            if (!EDGE || (f & PF_C)) {
                sP[a] = nP;
                sXX[a] = nxx;
                sYY[a] = nyy;
            }
            if (!EDGE || (f & PF_XY)) sXY[a] = nxy;
            if (EDGE && (f & PF_TRAC)) {
                for (int s = 0; s < 2; s++) {
                    if (f & (s ? PF_TX1 : PF_TX0)) {
                        const T tv = T(2.0) * q.bc_val[0][s][0];
                        sP[a + (s ? 1 : -1)] = tv - nP;
                        sXX[a + (s ? 1 : -1)] = tv - nxx;
                    }
                    if (f & (s ? PF_TY1 : PF_TY0)) {
                        const T tv = T(2.0) * q.bc_val[1][s][1];
                        sP[a + (s ? PW : -PW)] = tv - nP;
                        sYY[a + (s ? PW : -PW)] = tv - nyy;
                    }
                }
            }
        }
        __syncthreads();
        // a position may hold the ghost of another thread's cell, or a value that does not move
        if (EDGE) {
#pragma unroll
            for (int r = 0; r < PY; r++)
                if (!(v.fl[r] & PF_C)) v.P[r] = sP[a0 + r * PW], v.xx[r] = sXX[a0 + r * PW], v.yy[r] = sYY[a0 + r * PW];
        }
        // ---- update_V! (kernels_2d.jl:20-29) and the viscosity ----
        T Pd = sP[a0 - PW], yyd = sYY[a0 - PW];  // the row below the strip
        T xyr = sXY[a0 + 1];                     // τxy right of the point
#pragma unroll
        for (int r = 0; r < PY; r++) {
            const int a = a0 + r * PW;
            const T xyu = r + 1 < PY ? v.xy[r + 1] : sXY[a + PW];
            const T xyru = sXY[a + PW + 1];
            const T fx = fma_r(xyu - v.xy[r], idy, sum_r(v.xx[r] - sXX[a - 1], idx, -(v.P[r] - sP[a - 1]), idx));
            const T fy = fma_r(xyr - v.xy[r], idx, sum_r(v.yy[r] - yyd, idy, -(v.P[r] - Pd), idy));
            T nvx = fma_r(div_fast(fx - (GF ? v.gx[r] : q.g_val[0]), h(etl[r] + v.et[r])), q.dt_V[0], v.vx[r]);
            T nvy = fma_r(div_fast(fy - (GF ? v.gy[r] : q.g_val[1]), h(etd[r] + v.et[r])), q.dt_V[1], v.vy[r]);
            T ne = v.et[r];
            if (!frozen) {
                if (linear) {
                    ne = p.rheo_eta_is_field ? __ldg(in.eta_lin + v.at[r]) : T(p.rheo_eta);
                } else {
                    const T lxy = h(h(v.xy[r] + xyr) + h(xyu + xyru));
                    const T s2 = h(sum_r(v.xx[r], v.xx[r], v.yy[r], v.yy[r])) + mul_r(lxy, lxy);
                    ne = rheology_s2(p, q.rheo_A, q.rheo_inv_eta_reg, in.eta_lin, in.A, v.et[r], (long long)v.at[r], s2);
                }
            }
            Pd = v.P[r];
            yyd = v.yy[r];
            xyr = xyru;
            const unsigned f = v.fl[r];
            if (EDGE && (f & PF_NODE)) {
                if (f & PF_FX0) nvx = q.bc_val[0][0][0];
                if (f & PF_FX1) nvx = q.bc_val[0][1][0];
                if (f & PF_FY0) nvy = q.bc_val[1][0][1];
                if (f & PF_FY1) nvy = q.bc_val[1][1][1];
            }
            v.ep[r] = v.et[r];
            v.vx[r] = nvx, v.vy[r] = nvy, v.et[r] = ne;
            if (!EDGE || (f & PF_VX)) sVx[a] = nvx;
            if (!EDGE || (f & PF_VY)) sVy[a] = nvy;
            if (!EDGE || (f & PF_C)) sE[a] = ne;
            if (EDGE && (f & PF_GHOST)) {
                if (f & PF_VX) {
                    if ((f & PF_GY0) && p.bc_kind[1][0] == FI_BC_VELOCITY) sVx[a - PW] = T(2.0) * q.bc_val[1][0][0] - nvx;
                    if ((f & PF_GY1) && p.bc_kind[1][1] == FI_BC_VELOCITY) sVx[a + PW] = T(2.0) * q.bc_val[1][1][0] - nvx;
                }
                if (f & PF_VY) {
                    // on a fixed node of y, whose assignment runs last and spans the x ghosts, the
                    // image is a copy
                    const bool node = f & (PF_FY0 | PF_FY1);
                    if ((f & PF_GX0) && p.bc_kind[0][0] == FI_BC_VELOCITY) sVy[a - 1] = node ? nvy : T(2.0) * q.bc_val[0][0][1] - nvy;
                    if ((f & PF_GX1) && p.bc_kind[0][1] == FI_BC_VELOCITY) sVy[a + 1] = node ? nvy : T(2.0) * q.bc_val[0][1][1] - nvy;
                }
                if ((f & PF_C) && !frozen) {
                    const int dx = (f & PF_GX0) ? -1 : (f & PF_GX1) ? 1 : 0, dy = (f & PF_GY0) ? -PW : (f & PF_GY1) ? PW : 0;
                    if (dx) sE[a + dx] = ne;
                    if (dy) sE[a + dy] = ne;
                    if (dx && dy) sE[a + dx + dy] = ne;
                }
            }
        }
        __syncthreads();
        // (τxy at a node reads the ghosts of V and η at its own position)
        if (EDGE) {
#pragma unroll
            for (int r = 0; r < PY; r++) {
                const int a = a0 + r * PW;
                if (!(v.fl[r] & PF_VX)) v.vx[r] = sVx[a];
                if (!(v.fl[r] & PF_VY)) v.vy[r] = sVy[a];
                if (!(v.fl[r] & PF_C)) v.et[r] = sE[a];
                if (!(v.fl[r] & PF_XY)) v.xy[r] = sXY[a];
            }
        }
    }
}

// one region, the one around the tile that starts at (bx0, by0)
template <typename T, int RX, int RY, int PY, bool GF, bool BATCH>
__device__ __forceinline__ void run_region(const Geom &g, const KParams &p, const TConst<T> &q, const Ptrs<T> &in,
                                           const Ptrs<T> &out, T *eta_prev, const TileArgs &ta, int bx0, int by0,
                                           unsigned char *t2_smem) {
    using R = Region<T, RX, RY, PY>;
    constexpr int PW = R::PW;
    T *sP = reinterpret_cast<T *>(t2_smem), *sXX = sP + R::PLANE, *sYY = sXX + R::PLANE, *sXY = sYY + R::PLANE;
    T *sVx = sXY + R::PLANE, *sVy = sVx + R::PLANE, *sE = sVy + R::PLANE;
    const int w = threadIdx.x / 32, x = threadIdx.x % 32 + 32 * (w % (RX / 32)), y0 = (w / (RX / 32)) * PY;
    const int n0 = g.n[0], n1 = g.n[1];
    // (a batch has no periodic members)
    const bool px = !BATCH && p.bc_kind[0][0] == FI_BC_PERIODIC, py = !BATCH && p.bc_kind[1][0] == FI_BC_PERIODIC;
    const int i0 = bx0 - ta.k, j0 = by0 - ta.k;
    const int gi = i0 + x;
    const int a0 = (y0 + 1) * PW + x + 1;
    const bool edge = (!px && (i0 <= 1 || i0 + RX > n0)) || (!py && (j0 <= 1 || j0 + RY > n1));
    Strip<T, PY> v;
    const int si = t2_wrap(gi, n0, px);
    const int xl = p.bc_kind[0][0], xr = p.bc_kind[0][1], yl = p.bc_kind[1][0], yr = p.bc_kind[1][1];
#pragma unroll
    for (int r = 0; r < PY; r++) {
        const int gj = j0 + y0 + r, sj = t2_wrap(gj, n1, py);
        const bool ok = si >= 0 && si <= n0 + 2 && sj >= 0 && sj <= n1 + 2;
        v.at[r] = ok ? (unsigned)(si + (int)g.pitch * sj) : 0u;
        unsigned f = PF_C | PF_XY | PF_VX | PF_VY;
        if (edge) {
            const bool cx = px || (gi >= 1 && gi <= n0), cy = py || (gj >= 1 && gj <= n1);
            const bool ux = px || (gi >= 1 && gi <= n0 + 1), uy = py || (gj >= 1 && gj <= n1 + 1);
            f = 0;
            if (cx && cy) f |= PF_C;
            if (ux && uy) f |= PF_XY;
            if (ux && cy) f |= PF_VX;
            if (cx && uy) f |= PF_VY;
            if (!px && ux) {
                if (gi == 1 && t2_shear(xl)) f |= PF_X0;
                if (gi == n0 + 1 && t2_shear(xr)) f |= PF_X1;
                if (gi == 1 && xl == FI_BC_TRACTION && cy) f |= PF_TX0;
                if (gi == n0 && xr == FI_BC_TRACTION && cy) f |= PF_TX1;
                if (gi == 1 && t2_fixed(xl)) f |= PF_FX0;
                if (gi == n0 + 1 && t2_fixed(xr)) f |= PF_FX1;
                if (gi == 1) f |= PF_GX0;
                if (gi == n0) f |= PF_GX1;
            }
            if (!py && uy) {
                if (gj == 1 && t2_shear(yl)) f |= PF_Y0;
                if (gj == n1 + 1 && t2_shear(yr)) f |= PF_Y1;
                if (gj == 1 && yl == FI_BC_TRACTION && cx) f |= PF_TY0;
                if (gj == n1 && yr == FI_BC_TRACTION && cx) f |= PF_TY1;
                if (gj == 1 && t2_fixed(yl)) f |= PF_FY0;
                if (gj == n1 + 1 && t2_fixed(yr)) f |= PF_FY1;
                if (gj == 1) f |= PF_GY0;
                if (gj == n1) f |= PF_GY1;
            }
        }
        v.fl[r] = f;
    }
    // everything above may run while the launch before this one finishes
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const bool gfx = p.g_kind[0] == FI_G_FIELD, gfy = p.g_kind[1] == FI_G_FIELD;
#pragma unroll
    for (int r = 0; r < PY; r++) {
        const unsigned I = v.at[r];
        v.P[r] = in.P[I];
        v.xx[r] = in.txx[I];
        v.yy[r] = in.tyy[I];
        v.xy[r] = in.txy[I];
        v.vx[r] = in.Vx[I];
        v.vy[r] = in.Vy[I];
        v.et[r] = in.eta[I];
        v.ep[r] = v.et[r];
        if (GF) v.gx[r] = gfx ? __ldg(in.gx + I) : q.g_val[0];
        if (GF) v.gy[r] = gfy ? __ldg(in.gy + I) : q.g_val[1];
    }
#pragma unroll
    for (int r = 0; r < PY; r++) {
        const int a = a0 + r * PW;
        sP[a] = v.P[r];
        sXX[a] = v.xx[r];
        sYY[a] = v.yy[r];
        sXY[a] = v.xy[r];
        sVx[a] = v.vx[r];
        sVy[a] = v.vy[r];
        sE[a] = v.et[r];
    }
    __syncthreads();
    if (edge) iterate<true, GF, BATCH, T, RX, RY, PY>(p, q, in, v, sP, a0, ta.k);
    else iterate<false, GF, BATCH, T, RX, RY, PY>(p, q, in, v, sP, a0, ta.k);
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    // ---- the inner tile (with the ghosts beside it) to the other buffer ----
    const auto &P = v.P, &xx = v.xx, &yy = v.yy, &xy = v.xy, &vx = v.vx, &vy = v.vy, &et = v.et;
    if (!t2_owned(gi, bx0, ta.tx, n0, px)) return;
    // periodic images of centre (c) and vertex (v) values along a dimension: 0 = none
    auto image_c = [](int gq, int n, bool per) { return !per ? 0 : gq == n ? -n : gq == 1 ? n : 0; };
    auto image_v = [](int gq, int n, bool per) { return !per ? 0 : gq == n ? -n : gq <= 2 ? n : 0; };
    const int xc = image_c(gi, n0, px), xv = image_v(gi, n0, px);
#pragma unroll
    for (int r = 0; r < PY; r++) {
        const int gj = j0 + y0 + r;
        if (!t2_owned(gj, by0, ta.ty, n1, py)) continue;
        const int a = a0 + r * PW;
        const long long I = (long long)gi + g.pitch * (long long)gj;
        const long long yc = g.pitch * image_c(gj, n1, py), yv = g.pitch * image_v(gj, n1, py);
        auto put = [&](T *f, T v, int dx, long long dy) {
            f[I] = v;
            if (dx) f[I + dx] = v;
            if (dy) f[I + dy] = v;
            if (dx && dy) f[I + dx + dy] = v;
        };
        put(out.P, edge ? sP[a] : P[r], xc, yc);
        put(out.txx, edge ? sXX[a] : xx[r], xc, yc);
        put(out.tyy, edge ? sYY[a] : yy[r], xc, yc);
        put(out.txy, edge ? sXY[a] : xy[r], xv, yv);
        put(out.Vx, edge ? sVx[a] : vx[r], xv, yc);
        put(out.Vy, edge ? sVy[a] : vy[r], xc, yv);
        if (!p.freeze_eta) {
            put(out.eta, edge ? sE[a] : et[r], xc, yc);
            if (ta.write_prev && (v.fl[r] & PF_C)) eta_prev[I] = v.ep[r];
        }
    }
}

template <typename T, int RX, int RY, int PY, int MINB, bool GF>
__global__ void __launch_bounds__(RX *RY / PY, MINB)
    tile2d_kernel(Geom g, KParams p, TConst<T> q, Ptrs<T> in, Ptrs<T> out, T *eta_prev, TileArgs ta, int x0, int y0) {
    extern __shared__ __align__(16) unsigned char t2_smem[];
    run_region<T, RX, RY, PY, GF, false>(g, p, q, in, out, eta_prev, ta, x0 + (int)blockIdx.x * ta.tx, y0 + (int)blockIdx.y * ta.ty,
                                              t2_smem);
}

// The regions of several models, a block each; blocks past the end of the work list leave.
// The list does not change while chained launches run.  The members come as kernel arguments:
// copied from a device table into shared memory they cost the iterations' loads and registers
// (48 members of 63^2-511^2, FP32: 60.6 us an iteration; a persistent grid that copies the
// next member ahead 67.4), as uniform operands from the constant bank 42.6.
template <typename T, int RX, int RY, int PY, int MINB, bool GF>
__global__ void __launch_bounds__(RX *RY / PY, MINB)
    tile2d_batched(const __grid_constant__ Tile2DTable<T> members, int first, int end, const int4 *__restrict__ tiles,
                   const int *__restrict__ start, int src, int k, int tile) {
    extern __shared__ __align__(16) unsigned char t2_smem[];
    const int w = start[first] + (int)blockIdx.x;
    if (w >= start[end]) {
        // Also a block without work waits: a group with no active member would otherwise be a
        // grid that ends at once, and the launch chained to it would run beside the one before.
        asm volatile("griddepcontrol.wait;" ::: "memory");
        return;
    }
    const int4 d = tiles[w];
    // (a reduction's result is known to be the same in all lanes: the member's values are
    // read as uniform operands)
    const Tile2DMember<T> &c = members.m[__reduce_max_sync(0xffffffffu, (unsigned)(d.x - first))];
    Geom g{};
    KParams p{};
    TConst<T> q{};
    Ptrs<T> in{}, out{};
    p.freeze_eta = 1;
    p.p_forcing = c.forced;
    q.dt_P = c.dt_P;
    q.dt_tau[0] = c.dt_tau[0], q.dt_tau[1] = c.dt_tau[1], q.dt_tau[3] = c.dt_tau[2];
    g.pitch = c.pitch;
#pragma unroll
    for (int a = 0; a < 2; a++) {
        g.n[a] = c.n[a];
        p.g_kind[a] = c.g_kind[a];
        q.inv_dx[a] = c.inv_dx[a], q.dt_V[a] = c.dt_V[a], q.g_val[a] = c.g_val[a];
#pragma unroll
        for (int e = 0; e < 2; e++) {
            p.bc_kind[a][e] = c.bc_kind[a][e];
            q.bc_val[a][e][0] = c.bc_val[a][e][0], q.bc_val[a][e][1] = c.bc_val[a][e][1];
        }
    }
    in.P = c.f[src][0], in.txx = c.f[src][1], in.tyy = c.f[src][2], in.txy = c.f[src][3], in.Vx = c.f[src][4], in.Vy = c.f[src][5];
    in.eta = const_cast<T *>(c.eta), in.gx = c.gx, in.gy = c.gy, in.fP = const_cast<T *>(c.fP);
    const int dst = src ^ 1;
    out.P = c.f[dst][0], out.txx = c.f[dst][1], out.tyy = c.f[dst][2], out.txy = c.f[dst][3], out.Vx = c.f[dst][4],
    out.Vy = c.f[dst][5];
    const TileArgs ta{k, tile, tile, 0};
    run_region<T, RX, RY, PY, GF, true>(g, p, q, in, out, nullptr, ta, d.y, d.z, t2_smem);
}

template <typename T, int RX, int RY, int PY, int MINB, bool GF>
cudaError_t launch_region(const Geom &g, const KParams &p, const Ptrs<T> &in, const Ptrs<T> &out, T *eta_prev, int k,
                          bool write_prev, cudaStream_t s) {
    using R = Region<T, RX, RY, PY>;
    auto *kern = tile2d_kernel<T, RX, RY, PY, MINB, GF>;
    int dev = 0;
    cudaGetDevice(&dev);
    static bool attr_set[64] = {};
    if (dev < 64 && !attr_set[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)R::SMEM);
        if (e != cudaSuccess) return e;
        attr_set[dev] = true;
    }
    const bool px = p.bc_kind[0][0] == FI_BC_PERIODIC, py = p.bc_kind[1][0] == FI_BC_PERIODIC;
    const TileArgs ta{k, RX - 2 * k, RY - 2 * k, write_prev ? 1 : 0};
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(t2_tiles(g.n[0], ta.tx, px), t2_tiles(g.n[1], ta.ty, py));
    cfg.blockDim = dim3(R::NT);
    cfg.dynamicSmemBytes = R::SMEM;
    cfg.stream = s;
    // the launch may start while the one before it drains (griddepcontrol.wait orders them)
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, g, p, make_tconst<T>(p), in, out, eta_prev, ta, 1 - t2_shift(g.n[0], ta.tx, px),
                              1 - t2_shift(g.n[1], ta.ty, py));
}

template <typename T, bool GF>
cudaError_t launch_batched_regions(const Tile2DTable<T> &members, int first, int end, const int4 *tiles, const int *start,
                                   int blocks, int src, int k, int tile, bool chained, cudaStream_t s) {
    using R = Region<T, 32, 32, 2>;
    auto *kern = tile2d_batched<T, 32, 32, 2, 2, GF>;
    int dev = 0;
    cudaGetDevice(&dev);
    static bool attr_set[64] = {};
    if (dev < 64 && !attr_set[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)R::SMEM);
        if (e != cudaSuccess) return e;
        attr_set[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(R::NT);
    cfg.dynamicSmemBytes = R::SMEM;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = chained ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, members, first, end, tiles, start, src, k, tile);
}

}  // namespace

template <typename T, bool GF>
static cudaError_t launch_shape(const Geom &g, const KParams &p, const Ptrs<T> &in, const Ptrs<T> &out, T *eta_prev, int shape,
                                int k, bool write_prev, cudaStream_t s) {
    switch (shape) {
        case 0: return launch_region<T, 32, 16, 1, 1, GF>(g, p, in, out, eta_prev, k, write_prev, s);
        case 1: return launch_region<T, 32, 32, 2, 1, GF>(g, p, in, out, eta_prev, k, write_prev, s);
        default: return launch_region<T, 32, 32, 2, 2, GF>(g, p, in, out, eta_prev, k, write_prev, s);
    }
}

template <typename T>
cudaError_t launch_tile2d(const Geom &g, const KParams &p, const Ptrs<T> &in, const Ptrs<T> &out, T *eta_prev, int shape,
                          int k, bool write_prev, cudaStream_t s) {
    const bool gf = p.g_kind[0] == FI_G_FIELD || p.g_kind[1] == FI_G_FIELD;
    return gf ? launch_shape<T, true>(g, p, in, out, eta_prev, shape, k, write_prev, s)
              : launch_shape<T, false>(g, p, in, out, eta_prev, shape, k, write_prev, s);
}

template <typename T>
cudaError_t launch_tile2d_batched(const Tile2DTable<T> &members, int first, int end, const int4 *tiles, const int *start,
                                  int blocks, int src, int k, int tile, bool gf, bool chained, cudaStream_t s) {
    return gf ? launch_batched_regions<T, true>(members, first, end, tiles, start, blocks, src, k, tile, chained, s)
              : launch_batched_regions<T, false>(members, first, end, tiles, start, blocks, src, k, tile, chained, s);
}

template cudaError_t launch_tile2d_batched<double>(const Tile2DTable<double> &, int, int, const int4 *, const int *, int, int, int,
                                                   int, bool, bool, cudaStream_t);
template cudaError_t launch_tile2d_batched<float>(const Tile2DTable<float> &, int, int, const int4 *, const int *, int, int, int,
                                                  int, bool, bool, cudaStream_t);
template cudaError_t launch_tile2d<double>(const Geom &, const KParams &, const Ptrs<double> &, const Ptrs<double> &, double *,
                                           int, int, bool, cudaStream_t);
template cudaError_t launch_tile2d<float>(const Geom &, const KParams &, const Ptrs<float> &, const Ptrs<float> &, float *, int,
                                          int, bool, cudaStream_t);

}  // namespace fi
