// Fused right-hand side of a regular (uncut) box, ideal gas, FP64 form.
//
// Replaces the per-box kernel chain of EBR::compute_dSdt (Source/Advance.cpp:
// 231-329): c2prim over the grown box, then per direction flux_split (full
// grown box), reconstruction (WENO-Z, per face and component), compute_visc,
// and finally divop - fused into one launch (rhs_regular_kernel.cuh).
#include <cuda.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include "rhs_regular_kernel.cuh"

namespace ocfd {

ocfd_status configure_rhs_regular() { return configure_all<double>(); }

bool regular_tile_fits(int tile, bool visc) { return tile_fits<double>(tile, visc); }

// whether an SM holds two CTAs of the FP64 tile
static bool regular_tile_pairs(int tile, bool visc) {
    switch (tile) {
#define OCFD_PAIRS(I, X, Y, Z, XS)                                                              \
    case I:                                                                                     \
        return visc ? regular_min_blocks<double, X, Y, Z, true, false>() > 1                    \
                    : regular_min_blocks<double, X, Y, Z, false, false>() > 1;
        OCFD_REGULAR_TILES(OCFD_PAIRS)
#undef OCFD_PAIRS
    }
    return false;
}

const TileShape kRegularTiles[] = {{8, 8, 8, 0},  {8, 8, 4, 0}, {16, 8, 4, 0}, {16, 16, 2, 0}, {32, 8, 2, 0},
                                   {16, 8, 2, 0}, {8, 8, 8, 1}, {8, 8, 4, 1}, {16, 8, 4, 1}, {8, 4, 4, 0}, {4, 4, 4, 0},  {4, 4, 2, 0}, {8, 2, 2, 0}};
const int kNumRegularTiles = sizeof(kRegularTiles) / sizeof(kRegularTiles[0]);
const int kNumPublicTiles = 9;

ocfd_status launch_rhs_regular(int tile, bool visc, const RegBoxArgs* d_boxes,
                               const int* d_tile_start, int nbox, const RegBoxArgs& single,
                               int ntiles, const DevParm& P, cudaStream_t st, int sched, unsigned* queue) {
    return launch_any<double>(tile, visc, d_boxes, d_tile_start, nbox, single, ntiles, P, st, sched, queue);
}

// Warp instructions a tile takes on the pipe that bounds its form (FP64: FP64
// instructions; FP32: all), from its counts of work items per sweep: WENO-Z runs of
// three faces x component (FP64) or faces x component (FP32), split cells of the
// pencils, primitives (of the cross, or of each pencil and the ring with viscosity)
// and viscous faces.  The weights are the kernels' instruction counts at the time the
// tile shapes were measured (FP64 run 80, split 41; today's 60 and 27, and the integer
// chain that runs beside them, are not in them): they rank the shapes, and the shapes
// were measured with them.  The counts of today would choose otherwise for few sizes.
static double tile_work(const TileShape& s, bool visc, bool f32) {
    const int T[3] = {s.x, s.y, s.z};
    auto warps = [](int items) { return (items + 31) / 32; };
    const double weno = f32 ? 150 : 80, split = f32 ? 70 : 41, prim = f32 ? 60 : 25, vface = f32 ? 120 : 95;
    double w = (f32 ? 200 : 65) * warps(T[0] * T[1] * T[2]);  // divergence and update
    int cross = T[0] * T[1] * T[2];
    for (int d = 0; d < 3; ++d) {
        const int line = T[(d + 1) % 3] * T[(d + 2) % 3], faces = T[d] + 1, pencil = (T[d] + 6) * line;
        w += weno * warps(5 * line * (f32 ? faces : (faces + 2) / 3)) + split * warps(pencil);
        if (visc || f32) w += prim * warps(pencil);
        if (visc) w += vface * warps(faces * line);
        cross += 6 * line;
    }
    if (visc) w += prim * warps((T[0] + 2) * (T[1] + 2) * (T[2] + 2));
    else if (!f32) w += prim * warps(cross);
    return w;
}

// Time of a tile shape over a set of boxes on `sms` SMs.  The pipe that bounds a tile
// is shared by the CTAs of an SM: large tiles have the least halo work per cell,
// small ones spread a small box over more SMs and leave a shorter last wave.
//   FP64  one tile's work while every tile has an SM of its own; else the cells' share
//         of an SM (tiles that overhang the box skip what lies outside) and half a
//         tile's work for the last wave.  Tiles of which an SM holds two keep its
//         FP64 pipe busier (one's barriers are the other's work), hence the factor.
//   FP32  three and more tiles share an SM and overhanging ones do all their work.
// The constants (0.5, 0.91, 0.35, 1.05 and the two rules of small shapes) are fitted to
// the boxes below and some ten others of 20x12x8 to 128x96x64 cells.
// Measured (us, the best shape of nine unless said; the rule takes these or is within
// 3 %): FP64 viscous box of 20x12x8 cells 33 in 60 tiles of 4x4x2, 190 in six 8^3;
// 13x97x5 45 in 8x2x2, 52 in 4x4x4; with the arithmetic before the split's and the
// correction's last regrouping (1.1 times these) 175 in 8^3, 32^3 127 in 8x8x4, 192 in
// 8^3, 61x45x37 339 in 8x8x4, 371 in 8^3, inviscid 128x96x64 1422 in 8^3, 1427 in
// 8x8x4, 1898 in 8x4x4.
// FP32 viscous 32^3 16 in 4x4x4, 22 in 8x8x4, 27 in 8^3; inviscid 128x96x64 128 in
// 8^3, 133 in 8x8x4.  FP32 boxes take the pencil tiles: TMA staging of the same shape
// is slower (a box of 128x96x64 cells with face fluxes 183 us staged, 158 us not; two
// CTAs per SM against three).
static double tile_cost(int t, const int (*n)[3], int nbox, bool visc, bool f32, int sms) {
    const TileShape& s = kRegularTiles[t];
    long long tiles = 0;
    double cells = 0;
    for (int b = 0; b < nbox; ++b) {
        tiles += (long long)((n[b][0] + s.x - 1) / s.x) * ((n[b][1] + s.y - 1) / s.y) * ((n[b][2] + s.z - 1) / s.z);
        cells += (double)n[b][0] * n[b][1] * n[b][2];
    }
    const double work = tile_work(s, visc, f32);
    if (f32) return work * ((double)tiles / sms + 0.35);
    if (tiles <= sms) return t == 12 ? 1.05 * work : work;  // 8x2x2: 256 threads (34.9 us against 32.8)
    // an SM holds one 4x4x2 tile (480 threads), and all take alike
    if (t == 11) return work * (double)((tiles + sms - 1) / sms);
    return work * (cells / ((double)s.x * s.y * s.z * sms) + 0.5) * (regular_tile_pairs(t, visc) ? 0.91 : 1.0);
}

int pick_regular_tile(const int n[3], bool visc, bool f32, int sms) {
    const int one[1][3] = {{n[0], n[1], n[2]}};
    int best = 1;
    double best_cost = 1e300;
    for (int t = 0; t < kNumRegularTiles; ++t) {
        if (!regular_tile_fits(t, visc) || kRegularTiles[t].staged || (f32 && t == 12)) continue;  // 8x2x2: FP64's
        const double cost = tile_cost(t, one, 1, visc, f32, sms);
        if (cost < best_cost * 0.999) {
            best_cost = cost;
            best = t;
        }
    }
    return best;
}

// A level's tile serves its FP64 and its FP32 steps: the shape with the least padded
// work, where the FP32 form is fastest too, but 8x8x4 for 16x8x4 (slabs of at most
// four cells) where that ends sooner in FP64; the FP32 form takes either alike.
int pick_level_tile(const int (*n)[3], int nbox, int sms) {
    int best = 1;
    double best_cost = 1e300;
    for (int t = 0; t < kNumPublicTiles; ++t) {
        if (!regular_tile_fits(t, true) || kRegularTiles[t].staged) continue;
        const TileShape& s = kRegularTiles[t];
        double cost = 0;
        for (int b = 0; b < nbox; ++b) {
            const long long tiles = (long long)((n[b][0] + s.x - 1) / s.x) * ((n[b][1] + s.y - 1) / s.y) * ((n[b][2] + s.z - 1) / s.z);
            cost += tiles * ((double)s.x * s.y * s.z * 3.0 + 6.0 * ((double)s.y * s.z + (double)s.x * s.z + (double)s.x * s.y));
        }
        if (cost < best_cost * 0.999) {
            best_cost = cost;
            best = t;
        }
    }
    constexpr int T884 = 1, T1684 = 2;
    return best == T1684 && tile_cost(T884, n, nbox, true, false, sms) < tile_cost(T1684, n, nbox, true, false, sms) ? T884 : best;
}

void fill_regular_args(RegBoxArgs& a, const ocfd_array4* S, const ocfd_array4* dSdt,
                       const ocfd_array4* flux, const ocfd_box& bx, const double dxinv[3],
                       int tile) {
    a.S = view_of<const double>(S);
    if (dSdt) a.dsdt = view_of<double>(dSdt);
    a.has_flux = flux != nullptr ? FLUX_WRITE : 0;
    a.flux_w = 0.0;
    for (int d = 0; d < 3; ++d) {
        if (flux) a.flux[d] = view_of<double>(&flux[d]);
        a.lo[d] = bx.lo[d];
        a.hi[d] = bx.hi[d];
        a.dxinv[d] = dxinv[d];
        a.dxinv_f[d] = (float)dxinv[d];
    }
    const TileShape& s = kRegularTiles[tile];
    const int T[3] = {s.x, s.y, s.z};
    for (int d = 0; d < 3; ++d) a.ntile[d] = (bx.hi[d] - bx.lo[d] + T[d]) / T[d];
    a.mode = RHS_WRITE_DSDT;
    a.dt_ptr = nullptr;
    a.cfl_min = nullptr;
    encode_regular_tmaps(a, S, tile);
}

static bool g_regular_tma = true;

void set_regular_tma(bool on) { g_regular_tma = on; }

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link
// against the driver library); null when the driver does not offer it
static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) !=
                cudaSuccess ||
            q != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            p = nullptr;
        }
        return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    }();
    return fn;
}

// The four box shapes of a tile's cross (centre, x halo 4 wide, y halo 3 deep,
// z halo 3 deep) over S as a (x, y, z, component) tensor of doubles.  TMA wants
// a 16-byte aligned base, strides that are multiples of 16 bytes and an x
// offset times 8 bytes that is a multiple of 16 for every box: the tiles start
// at lo + t TX with TX even and the x halo box at 4 cells before a tile, so
// (lo - begin) must be even.  Only tiles of depth >= 4 are staged this way.
bool encode_regular_tmaps(RegBoxArgs& a, const ocfd_array4* S, int tile) {
    a.use_tma = 0;
    if (!g_regular_tma || !S || tile < 0 || tile >= kNumRegularTiles) return false;
    const TileShape& t = kRegularTiles[tile];
    if (!t.staged || t.z < 4 || t.x % 2 != 0 || S->ncomp < 5) return false;
    const uintptr_t base = reinterpret_cast<uintptr_t>(S->p);
    if (base % 16 != 0 || S->jstride % 2 != 0 || S->kstride % 2 != 0 || S->nstride % 2 != 0) return false;
    if (((a.lo[0] - S->begin[0]) & 1) != 0) return false;
    PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
    if (!enc) return false;
    const cuuint64_t dim[4] = {(cuuint64_t)(S->end[0] - S->begin[0]), (cuuint64_t)(S->end[1] - S->begin[1]),
                               (cuuint64_t)(S->end[2] - S->begin[2]), 5};
    const cuuint64_t stride[3] = {(cuuint64_t)S->jstride * 8, (cuuint64_t)S->kstride * 8,
                                  (cuuint64_t)S->nstride * 8};
    const cuuint32_t box[4][4] = {{(cuuint32_t)t.x, (cuuint32_t)t.y, (cuuint32_t)t.z, 5},
                                  {4, (cuuint32_t)t.y, (cuuint32_t)t.z, 5},
                                  {(cuuint32_t)t.x, 3, (cuuint32_t)t.z, 5},
                                  {(cuuint32_t)t.x, (cuuint32_t)t.y, 3, 5}};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    for (int m = 0; m < 4; ++m) {
        if (enc(&a.tmap[m], CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 4, S->p, dim, stride, box[m], estr,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return false;
    }
    a.use_tma = 1;
    return true;
}

}  // namespace ocfd

using namespace ocfd;

extern "C" ocfd_status ocfd_rhs_regular_box_f64(ocfd_context* ctx, const ocfd_array4* S,
                                                const ocfd_array4* dSdt, const ocfd_array4* flux,
                                                ocfd_box bx, const double dxinv[3],
                                                unsigned flags, void* stream) {
    if (!ctx || !dxinv) return fail(OCFD_BAD_ARG, "ocfd_rhs_regular_box_f64: null argument");
    for (int d = 0; d < 3; ++d)
        if (bx.hi[d] < bx.lo[d]) return fail(OCFD_BAD_ARG, "ocfd_rhs_regular_box_f64: empty box");
    if (!covers(S, bx, 3, 5)) return fail(OCFD_BAD_ARG, "ocfd_rhs_regular_box_f64: S must cover grow(bx,3) with 5 components");
    if (!covers(dSdt, bx, 0, 5)) return fail(OCFD_BAD_ARG, "ocfd_rhs_regular_box_f64: dSdt must cover bx with 5 components");
    if (flux)
        for (int d = 0; d < 3; ++d)
            if (!covers(&flux[d], bx, 0, 5, d))
                return fail(OCFD_BAD_ARG, "ocfd_rhs_regular_box_f64: flux[d] must cover surroundingNodes(bx,d)");
    if (flags & ~(unsigned)(OCFD_VISC | OCFD_FLUX_FP32 | OCFD_GRAVITY))
        return fail(OCFD_BAD_ARG, "ocfd_rhs_regular_box_f64: unknown flags");
    if (flags & OCFD_FLUX_FP32) return rhs_regular_box_f32(ctx, S, dSdt, flux, bx, dxinv, flags, stream);
    DevParm P = ctx->parm;
    P.grav = (flags & OCFD_GRAVITY) ? kGravity : 0.0;
    const int n[3] = {bx.hi[0] - bx.lo[0] + 1, bx.hi[1] - bx.lo[1] + 1, bx.hi[2] - bx.lo[2] + 1};
    const int tile = pick_regular_tile(n, (flags & OCFD_VISC) != 0, false, ctx->num_sms);
    RegBoxArgs a{};
    fill_regular_args(a, S, dSdt, flux, bx, dxinv, tile);
    const int ntiles = a.ntile[0] * a.ntile[1] * a.ntile[2];
    return launch_rhs_regular(tile, (flags & OCFD_VISC) != 0, nullptr, nullptr, 1, a, ntiles,
                              P, static_cast<cudaStream_t>(stream));
}

extern "C" void ocfd_set_tma_staging(int32_t on) { ocfd::set_regular_tma(on != 0); }
