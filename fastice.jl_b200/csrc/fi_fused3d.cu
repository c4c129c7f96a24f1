// fi_fused3d.cu -- fused single-pass 3D PT iteration (update_σ! + stress BCs +
// update_V! + velocity/η_next BCs in one kernel), TMA-staged.
//
// Reference semantics: src/Models/FullStokes/Isothermal/Isothermal.jl:91-112
// with kernels_3d.jl:3-40 and boundary_conditions.jl.  The two reference
// kernels touch the state twice per iteration (33 array passes); this sweep
// reads P, τ(6), V(3), η once and writes P, τ(6), V(3), η_next once (22 passes).
//
// Work decomposition.  A CTA owns a TX x TY column of grid positions (x, y), one
// thread each, and a block of z planes [kb, ke).  It marches up in z.  Step s
// computes the new P, τxx, τyy, τzz, τxy of plane s and the new τxz, τyz of plane
// s + 1 (their staggered position is the face between the two planes), then V and
// η_next of plane s: everything V(s) reads is then at hand in the same step, so the
// centre stresses live in two shared-memory slots and a z-block re-reads one plane
// of its neighbour below and one above.  P, τzz and η of the plane below, which V.z
// needs in the thread's own column only, stay in registers.  A step s = kb - 1
// before the march provides them and τxz, τyz of plane kb.
//
// Loads.  The tensor-memory accelerator copies an (x, y) box of each input field
// into shared-memory plane slots, one step ahead, signalled by an mbarrier.  Group g
// holds V, η, τxz, τyz of plane g and P, τxx, τyy, τzz, τxy of plane g - 1.  V and η
// come with a one-position ring on every side; a stress component comes only with
// the ring sides the velocity update reads: P and τxx left of the column, P and τyy
// below it, τxy and τxz right of it, τxy and τyz above it, τzz with none.  A group's
// slots are refilled as soon as every warp has left the velocity update that read
// them: the last warp to arrive (an atomic counter) issues the copies, so no warp
// waits for another there and a step has one block barrier.
//
// The new stresses are computed in place in shared memory, over the column and over
// the ring sides above (neighbouring CTAs recompute each other's ring: no grid-wide
// synchronisation).
//
// Clusters.  A launch shape may group CTAs into thread-block clusters (2x2, ...)
// purely for co-scheduling.  There is no cross-CTA communication and no multicast;
// a CTA may leave the cluster at any time.
//
// What bounds it.  At 511^3 FP64 DRAM: 1.11 times the field bytes are read (the rings;
// 64-byte L2 promotion) and the launch takes 4.25 ms, 5.7 TB/s of traffic; FP32 2.55 ms, bound
// by instruction issue (78 % active).  Three FP64 CTAs fit an SM (70 KB of slots,
// 80 registers), 24 warps; a form with 37 slots, two barriers a step, the boundary values
// applied in passes over the plane and two CTAs per SM took 5.45 and 3.46 ms on the same
// box.  Small grids are bound by the latency of a step (2.5-3 us alone on an SM), hence
// the short z-blocks of fused3d_default_variant and the chained launches: 127^3 with walls
// 240 -> 98 us, 47x33x29 138 -> 9.3 us, 259x193x125 399 -> 248 us.
//
// Double buffering.  Stresses and velocities are read from `in` and written to
// `out` (distinct buffers), so the pointwise in-place updates of the reference
// are reproduced exactly.  With a no-FMA build the sweep matches the CPU oracle
// bit for bit.
//
// Boundary conditions.  They are applied in registers by the thread that computes
// the value: fixed shear stresses at boundary nodes replace the value (x, then y,
// then z faces, a later dimension's value wins, as the CPU oracle applies them),
// and the thread that computes a P or τ_dd next to a traction side also writes its
// ghost 2c - v.  Velocity Dirichlet values are written at the boundary nodes; ghost
// values (Velocity BC ghosts 2c - v, η_next Neumann copies, periodic images) are
// written by the thread that computes the interior value they derive from.  Periodic
// x / y need no stress fix-up: the ghost-layer stresses (the ring of the first
// column, written back by its ring threads) follow from the wrapped ghosts of V and
// η of the previous iteration.  Stress ghosts that no update or residual reads are
// not maintained.
//
// Waits.  Every mbarrier wait is bounded (about one second of SM clock); on
// expiry the CTA records FI_ERR_TIMEOUT in the model's error word, waits once
// more (bounded) for its own copies in flight, and returns.
#include <cudaTypedefs.h>

#include <cstdio>
#include <cstdlib>

#include "fi_sweep3d.cuh"

namespace fi {

namespace {

// Launch shapes: tile width and height, z-block depth, cluster shape (x, y).  The trim flag
// only marks names, which callers choose by: every shape loads the trimmed boxes, and the
// autotuner does not time the same launch twice (fused3d_same_launch).  Shapes whose
// shared memory does not fit a CTA for a precision are not offered for it.
// fused3d_default_variant picks a 32x8 shape by the grid; the others stay for the
// autotuner (511^3 on one box, before the direct path for ghosts: FP64 32x8 tiles 4.37 ms,
// 32x16 5.45, 1x4 clusters 4.48; FP32 2.72, 2.86, 2.86 and 64x8 2.98 ms).
struct Variant {
    int tx, ty, zb, cx, cy, trim;
};
constexpr Variant kVariants[] = {
    {32, 8, 32, 1, 1, 0},  {32, 8, 64, 1, 1, 0},  {32, 8, 128, 1, 1, 0}, {32, 4, 64, 1, 1, 0},
    {32, 16, 32, 1, 1, 0}, {32, 16, 64, 1, 1, 0}, {32, 16, 128, 1, 1, 0},
    {32, 8, 32, 1, 1, 1},  {32, 8, 32, 1, 4, 1},  {32, 8, 32, 2, 2, 0},
    {64, 8, 32, 1, 1, 0},  {64, 8, 32, 1, 1, 1},
    // short z-blocks: grids too small to fill the GPU with long columns
    {32, 8, 1, 1, 1, 0},   {32, 8, 2, 1, 1, 0},   {32, 8, 4, 1, 1, 0},   {32, 8, 8, 1, 1, 0},
    {32, 8, 12, 1, 1, 0},  {32, 8, 16, 1, 1, 0},  {32, 8, 24, 1, 1, 0}};
constexpr int kNumVariants = sizeof(kVariants) / sizeof(kVariants[0]);

// Tiles of one launch along a split dimension: a launch runs either every tile, or
// part of them (the overlapped halo exchange runs the tiles next to the split faces
// first and the others while the halo moves).  Along `dim`, grid block b stands for
// tile b + base + (b >= nlow ? shift : 0).
struct TileMap {
    int dim;  // 0: x, 1: y, -1: every tile
    int base, nlow, shift;
};

__device__ __forceinline__ int tile_x(const TileMap &tm) {
    const int b = (int)blockIdx.x;
    return tm.dim == 0 ? b + tm.base + (b >= tm.nlow ? tm.shift : 0) : b;
}
__device__ __forceinline__ int tile_y(const TileMap &tm) {
    const int b = (int)blockIdx.y;
    return tm.dim == 1 ? b + tm.base + (b >= tm.nlow ? tm.shift : 0) : b;
}

template <typename T, int TX, int TY>
__device__ __forceinline__ void init_ctx(Ctx<T, TX, TY> &c, const Geom &g, const KParams &p, unsigned char *smem, int zb,
                                         const TileMap &tm) {
    c.sm = reinterpret_cast<T *>(smem);
    c.i0 = 1 + tile_x(tm) * TX;
    c.j0 = 1 + tile_y(tm) * TY;
    c.kb = 1 + blockIdx.z * zb;
    c.n0 = g.n[0];
    c.n1 = g.n[1];
    c.n2 = g.n[2];
    c.ke = min(c.kb + zb, c.n2 + 2);
    c.sx = g.pitch;
    c.sxy = g.sxy;
    auto away = [](int k) { return k == FI_BC_PERIODIC || k == FI_BC_HALO; };
    c.hx0 = away(p.bc_kind[0][0]);
    c.hx1 = away(p.bc_kind[0][1]);
    c.hy0 = away(p.bc_kind[1][0]);
    c.hy1 = away(p.bc_kind[1][1]);
}

template <typename T, int TX, int TY>
__global__ void __launch_bounds__(Layout<T, TX, TY>::NT, Layout<T, TX, TY>::MINB)
    fused3d_kernel(Geom g, KParams p, TConst<T> q, Ptrs<T> in, Ptrs<T> out, const __grid_constant__ InMaps maps, int zb,
                   TileMap tm, int *err) {
    using Lay = Layout<T, TX, TY>;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    // the grid is padded to whole clusters: columns past the vertex range have no work
    if (1 + tile_x(tm) * TX > g.n[0] + 1 || 1 + tile_y(tm) * TY > g.n[1] + 1) return;
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem_raw + (size_t)Lay::ELEMS * sizeof(T));
    unsigned *released = reinterpret_cast<unsigned *>(bars + kBars);
    if (threadIdx.x == 0) {
        for (int b = 0; b < kBars; b++) mbar_init(&bars[b], 1);
        *released = 0u;
        mbar_fence_init();
    }
    __syncthreads();
    Ctx<T, TX, TY> c;
    init_ctx(c, g, p, smem_raw, zb, tm);
    chain_launches();
    // Interior columns need no range tests, no x or y boundary values and no images, but in
    // FP64 a body of their own costs more in instruction fetches than it saves (259x193x125:
    // 268 us an iteration with it, 251 without; 511^3 4.37 and 4.26 ms).  FP32 code is
    // shorter: 2.72 ms with it at 511^3, 2.77 without.
    if (sizeof(T) == 4 && c.i0 > 2 && c.i0 + TX <= c.n0 && c.j0 > 2 && c.j0 + TY <= c.n1) sweep<false>(c, p, q, in, out, maps, bars, released, err);
    else sweep<true>(c, p, q, in, out, maps, bars, released, err);
}

template <typename T, int TX, int TY>
cudaError_t launch_variant(const Geom &g, const KParams &p, const Ptrs<T> &in, const Ptrs<T> &out, const InMaps &maps,
                           Variant v, int *err, cudaStream_t s, int part_dim, int part, bool chained) {
    using Lay = Layout<T, TX, TY>;
    int dev = 0;
    cudaGetDevice(&dev);
    static bool attr_set[64] = {};
    if (dev < 64 && !attr_set[dev]) {
        cudaError_t e =
            cudaFuncSetAttribute(fused3d_kernel<T, TX, TY>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Lay::SMEM);
        if (e != cudaSuccess) return e;
        attr_set[dev] = true;
    }
    auto up = [](int a, int b) { return (a + b - 1) / b * b; };
    TileMap tm{-1, 0, 1 << 30, 0};
    const int nbx = (g.n[0] + 1 + TX - 1) / TX, nby = (g.n[1] + 1 + TY - 1) / TY;
    int gx = nbx, gy = nby;
    if (part_dim == 0 || part_dim == 1) {
        // part 0: the tiles of the split faces -- tile 0 (positions 1 and 2) and the
        // tile of position n: the layers a slab sends and the ghost images it
        // writes; part 1: every other tile.  No clusters in partial launches.
        const int T_d = part_dim == 0 ? TX : TY, nb = part_dim == 0 ? nbx : nby;
        const int last = (g.n[part_dim] - 1) / T_d;
        int cnt;
        if (part == 0) {
            tm = {part_dim, 0, 1, last - 1};
            cnt = last > 0 ? 2 : 1;
        } else {
            // tiles 1 .. last-1, then last+1 .. nb-1
            tm = last > 0 ? TileMap{part_dim, 1, last - 1, 1} : TileMap{part_dim, 1, 1 << 30, 0};
            cnt = nb - (last > 0 ? 2 : 1);
            if (cnt <= 0) return cudaSuccess;
        }
        (part_dim == 0 ? gx : gy) = cnt;
        v.cx = v.cy = 1;
    }
    dim3 grd(up(gx, v.cx), up(gy, v.cy), (g.n[2] + 1 + v.zb - 1) / v.zb);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grd;
    cfg.blockDim = dim3(Lay::NT);
    cfg.dynamicSmemBytes = Lay::SMEM;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    if (v.cx * v.cy > 1) {
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = v.cx;
        attr[0].val.clusterDim.y = v.cy;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    } else if (chained) {
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    }
    const TConst<T> q = make_tconst<T>(p);
    return cudaLaunchKernelEx(&cfg, fused3d_kernel<T, TX, TY>, g, p, q, in, out, maps, v.zb, tm, err);
}

template <typename T>
size_t variant_smem(const Variant &v) {
    if (v.tx == 64) return Layout<T, 64, 8>::SMEM;
    return v.ty == 4 ? Layout<T, 32, 4>::SMEM : v.ty == 16 ? Layout<T, 32, 16>::SMEM : Layout<T, 32, 8>::SMEM;
}

PFN_cuTensorMapEncodeTiled_v12000 get_encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    if (!fn) {
        cudaDriverEntryPointQueryResult q;
        void *ptr = nullptr;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (PFN_cuTensorMapEncodeTiled_v12000)ptr;
    }
    return fn;
}

// box (width, height) of input field f for tile tx x ty
template <typename T, int TX, int TY>
void box_of(int f, int *bw, int *bh) {
#define FI_BOX_CASE(F)                 \
    case F:                            \
        *bw = FBox<T, TX, TY, F>::bw;  \
        *bh = FBox<T, TX, TY, F>::bh;  \
        return;
    switch (f) {
        FI_BOX_CASE(M_P)
        FI_BOX_CASE(M_XX)
        FI_BOX_CASE(M_YY)
        FI_BOX_CASE(M_ZZ)
        FI_BOX_CASE(M_XY)
        FI_BOX_CASE(M_XZ)
        FI_BOX_CASE(M_YZ)
        default: FI_BOX_CASE(M_VX)
    }
#undef FI_BOX_CASE
}

template <typename T>
void variant_box(const Variant &v, int f, int *bw, int *bh) {
    if (v.tx == 64) box_of<T, 64, 8>(f, bw, bh);
    else if (v.ty == 4) box_of<T, 32, 4>(f, bw, bh);
    else if (v.ty == 16) box_of<T, 32, 16>(f, bw, bh);
    else box_of<T, 32, 8>(f, bw, bh);
}

}  // namespace

int fused3d_num_variants() { return kNumVariants; }
const char *fused3d_variant_name(int v) {
    static char buf[kNumVariants][48];
    if (v < 0 || v >= kNumVariants) return "?";
    const Variant &w = kVariants[v];
    int n = snprintf(buf[v], sizeof(buf[v]), "tile%dx%d_zb%d", w.tx, w.ty, w.zb);
    if (w.trim) n += snprintf(buf[v] + n, sizeof(buf[v]) - n, "_trim");
    if (w.cx * w.cy > 1) snprintf(buf[v] + n, sizeof(buf[v]) - n, "_cl%dx%d", w.cx, w.cy);
    return buf[v];
}
int fused3d_variant_key(int v) {
    const Variant &w = kVariants[(v < 0 || v >= kNumVariants) ? 0 : v];
    return w.tx * 1000 + w.ty;
}
int fused3d_same_launch(int v) {
    const Variant &w = kVariants[v];
    for (int u = 0; u < v; u++) {
        const Variant &o = kVariants[u];
        if (o.tx == w.tx && o.ty == w.ty && o.zb == w.zb && o.cx == w.cx && o.cy == w.cy) return u;
    }
    return v;
}
bool fused3d_variant_fits(int v, int esz) {
    if (v < 0 || v >= kNumVariants) return false;
    const size_t smem = esz == 8 ? variant_smem<double>(kVariants[v]) : variant_smem<float>(kVariants[v]);
    // 64-wide FP64 tiles would hold one CTA per SM: not offered
    if (esz == 8 && kVariants[v].tx == 64) return false;
    return smem <= 227 * 1024;
}

// The 32x8 shape whose z-blocks take least time on this grid.  A z-block of zb planes is
// zb + 1 steps; with b blocks to each of the 148 SMs a step of all of them takes about
// 1.25 b + 1.6 us (fitted to FP64 and FP32 runs of 47x33x29 to 511^3: the first term is
// the throughput of three or four resident CTAs, the second the latency of a step that
// nothing else hides).  Short blocks pay the extra step, long ones leave SMs idle (measured
// before launches were chained and ghosts beside one side had their own path):
// 259x193x125 FP64 measures 403, 273, 262, 285, 422 us at zb = 1, 8, 16, 32, 128 (the rule
// takes 16), 127^3 walls 147, 117, 116, 138 at 1, 4, 8, 32 (8), 47x33x29 10, 16, 86 at
// 1, 4, 32 (1), and 511^3 4.37 and 4.91 ms at 32 and 64 (32, the longest it considers).
int fused3d_default_variant(const Geom &g) {
    const double cols = (double)((g.n[0] + 32) / 32) * ((g.n[1] + 8) / 8);
    int best = 0;
    double cost = 0.0;
    for (int v = 0; v < kNumVariants; v++) {
        const Variant &w = kVariants[v];
        if (w.tx != 32 || w.ty != 8 || w.cx * w.cy > 1 || w.trim || w.zb > 32) continue;
        const double b = cols * ((g.n[2] + w.zb) / w.zb) / 148.0;
        const double c = (w.zb + 1) * (1.25 * b + 1.6);
        if (cost == 0.0 || c < cost) best = v, cost = c;
    }
    return best;
}

template <typename T>
bool fused3d_supported(const Geom &g, const KParams &p, bool ib) {
    if (g.nd != 3 || ib) return false;
    if (p.bc_kind[2][0] == FI_BC_PERIODIC) return false;
    return g.pitch >= kXOff + g.n[0] + 3;
}

// a 2D or 3D tiled tensor map (no interleave, no swizzle, zero fill out of range)
// over `nd` dims of a field allocation; strides in bytes (dims 1..nd-1)
bool tma_encode(void *raw_base, int nd, const unsigned long long *dims, const unsigned long long *strides,
                const unsigned *box, int esz, void *map_out) {
    PFN_cuTensorMapEncodeTiled_v12000 enc = get_encoder();
    if (!enc || nd < 1 || nd > 3) return false;
    cuuint64_t d[3], st[2];
    cuuint32_t bx[3], estr[3] = {1, 1, 1};
    for (int k = 0; k < nd; k++) {
        d[k] = dims[k];
        bx[k] = box[k];
        if (k > 0) st[k - 1] = strides[k - 1];
    }
    CUresult r = enc((CUtensorMap *)map_out, esz == 8 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32,
                     nd, raw_base, d, st, bx, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

// the 3D tensor map of input field f (map order) over a field allocation (raw
// base, aligned) for a launch shape: box = one plane of the field's box
bool fused3d_encode_map(void *raw_base, const Geom &g, int esz, int variant, int field, void *map_out) {
    PFN_cuTensorMapEncodeTiled_v12000 enc = get_encoder();
    if (!enc || variant < 0 || variant >= kNumVariants || field < 0 || field >= M_COUNT) return false;
    int bw = 0, bh = 0;
    if (esz == 8) variant_box<double>(kVariants[variant], field, &bw, &bh);
    else variant_box<float>(kVariants[variant], field, &bw, &bh);
    cuuint64_t dims[3] = {(cuuint64_t)g.pitch, (cuuint64_t)g.rows, (cuuint64_t)g.planes};
    cuuint64_t strides[2] = {(cuuint64_t)(g.pitch * esz), (cuuint64_t)(g.sxy * esz)};
    cuuint32_t box[3] = {(cuuint32_t)bw, (cuuint32_t)bh, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    // L2 promotion of the box rows: 64 bytes (511^3 FP64 4.35 ms against 4.49 at 256, whose
    // wider fetches of a box's ring sectors raise the DRAM reads from 1.11 to 1.24 times the
    // field bytes); FI_TMA_L2_PROMOTION=0/64/128/256 overrides
    CUtensorMapL2promotion promo = CU_TENSOR_MAP_L2_PROMOTION_L2_64B;
    if (const char *e = getenv("FI_TMA_L2_PROMOTION")) {
        int v = atoi(e);
        promo = v == 0 ? CU_TENSOR_MAP_L2_PROMOTION_NONE
                       : v == 64 ? CU_TENSOR_MAP_L2_PROMOTION_L2_64B
                                 : v == 128 ? CU_TENSOR_MAP_L2_PROMOTION_L2_128B : CU_TENSOR_MAP_L2_PROMOTION_L2_256B;
    }
    CUresult r = enc((CUtensorMap *)map_out, esz == 8 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32,
                     3, raw_base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                     promo, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

template <typename T>
cudaError_t launch_fused3d(const Geom &g, const KParams &p, const Ptrs<T> &in, const Ptrs<T> &out, const void *maps11,
                           int variant, int *err, cudaStream_t s, int part_dim, int part, bool chained) {
    if (variant < 0 || variant >= kNumVariants) variant = 0;
    const Variant v = kVariants[variant];
    if (!fused3d_variant_fits(variant, (int)sizeof(T))) return cudaErrorInvalidConfiguration;
    const InMaps &mp = *reinterpret_cast<const InMaps *>(maps11);
    if (v.tx == 64) {
        if constexpr (sizeof(T) == 4) {
            return launch_variant<T, 64, 8>(g, p, in, out, mp, v, err, s, part_dim, part, chained);
        }
        return cudaErrorInvalidConfiguration;
    }
    switch (v.ty) {
        case 4: return launch_variant<T, 32, 4>(g, p, in, out, mp, v, err, s, part_dim, part, chained);
        case 16: return launch_variant<T, 32, 16>(g, p, in, out, mp, v, err, s, part_dim, part, chained);
        default: return launch_variant<T, 32, 8>(g, p, in, out, mp, v, err, s, part_dim, part, chained);
    }
}

template bool fused3d_supported<double>(const Geom &, const KParams &, bool);
template bool fused3d_supported<float>(const Geom &, const KParams &, bool);
template cudaError_t launch_fused3d<double>(const Geom &, const KParams &, const Ptrs<double> &, const Ptrs<double> &,
                                            const void *, int, int *, cudaStream_t, int, int, bool);
template cudaError_t launch_fused3d<float>(const Geom &, const KParams &, const Ptrs<float> &, const Ptrs<float> &,
                                           const void *, int, int *, cudaStream_t, int, int, bool);

}  // namespace fi
