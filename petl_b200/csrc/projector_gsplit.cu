// Split forward projector for any psi with voxel height equal to the u1 bin
// pitch, the counterpart of the shear-warp split kernels (projector_split.cu)
// for orientations whose rays are not parallel to a volume axis; and, further
// down, for unequal height and pitch at psi = 0 and 90 (k_uz in place of k_gz)
// with its exact transpose (k_backproject_uz).
//
// The reference footprint (src/projectors.cu:11-238) of a ray at its
// driving plane p (y = const for a y-driven view, x = const for an
// x-driven one, |r_x| < |r_y| deciding per view v0) is the product of a u0
// box overlap that depends on the ray parameter t and the in-plane voxel
// index a, and a u1 box overlap that depends on t, the slope v1 and the
// voxel row z.  t = (coordinate of plane p - p-coordinate of u0) / r_p
// depends on (v0, u0, p) only.  So
//   g[v1][v0][u1][u0] = l_phi rs sum_p sum_z w1(t, v1, u1, z) X[v0][p][z][u0],
//   X[v0][p][z][u0]   = sum_a w0(t, a, u0) f(z, p, a),
// and the two sums run as two kernels:
//
// * k_gx: a block stages 32 volume rows of plane p (8 of long axes; from the
//   volume, or from its x/y-transposed copy for x-driven views) in shared
//   memory for all views of the chunk; a thread per column u0 evaluates the u0
//   taps of its ray on plane p once (the reference's tap range and box
//   overlaps, taps with a positive weight) and applies them to the rows.
// * k_gz: CTA = one view x 16 slopes x 64 rows x 32 columns, 16 warps of
//   2 slopes x 32 rows, one column per lane (a last block of at most 8
//   slopes as 8 slopes x 128 rows).  With equal pitch the u1 taps
//   of row u1 are voxel rows u1 + s and u1 + s + 1 with weights 1 - fr and
//   fr, where s + fr = (u1_0 - z_0 - t v1) / T_u1 depends on the lane's t
//   and the slope but not on the row.  The lanes' shifts differ, so each
//   lane reads its own rows of the staged plane: the rows every lane and
//   slope of the tile needs (bounded on the host) for 32 columns, row-major,
//   so a lane's column is its bank whatever its row.  They arrive per plane
//   by a tiled TMA copy (no multicast; rows outside the scratch read zero)
//   into a ring of three planes with full/empty mbarriers and a rotating
//   issuer; every wait is bounded (a wait that gives up sets the device
//   error word, the CTA drains its copies and writes nothing).
// Epilogue: scale l_phi * rs, the reference's ray masks, optional MLEM
// ratio.
//
// The sums are associated differently from the reference's (u0 taps summed
// before the z taps), so results agree with it to float rounding, not bit
// for bit.
#include <algorithm>
#include <cmath>
#include <string>

#include "common.cuh"
#include "gsplit.cuh"
#include "projector.cuh"
#include "storage.cuh"
#include "tma.cuh"
#include "ztaps.cuh"

namespace petl {

namespace {

// Volume rows per k_gx block: a column's taps are evaluated once per block, and
// with 8 rows their evaluation bounded the pass (psi = 30, 256x256x128: 3.4 ms
// for 4.3 GB of scratch); 32 rows of axes up to 512 voxels (64 KB of shared
// memory), 8 of longer ones.
constexpr int GXZ = 32, GXZ_LONG = 8, GXZ_AXIS = 512;
constexpr int GZS = 16;       // slopes per k_gz CTA (2 per warp), main shape
constexpr int GZR = 64;       // rows per k_gz CTA (32 per warp), main shape
constexpr int GZS_T = 8;      // slopes per CTA of the tail shape (a last slope block of at most 8)
constexpr int GZR_T = 128;    // rows per CTA of the tail shape
constexpr int GZC = 32;       // columns per k_gz CTA (one per lane)
constexpr int GZT = 512;      // threads per k_gz CTA
constexpr int GJS = 2;        // slopes per warp
constexpr int GRW = 32;       // rows per warp (GZS / GJS x GZR / GRW = 16 warps; GZS_T / GJS x GZR_T / GRW the same;
                              // 16 rows per warp: 10 % slower at psi = 30, 256x256x128)
constexpr int GZRMAX = 224;   // staged rows per plane at most (TMA box rows <= 256)
constexpr int GZNS = 3;       // ring stages (one plane each) at most

struct GxArgs {
    petl_geom G;
    ViewRange vr;
    int vi0;    // first view of the chunk (index in vr)
    int nvc;    // views of the chunk
    int NPmax;  // planes per view slot of the scratch
    int NUc;    // scratch row pitch
};

struct GzArgs {
    petl_geom G;
    ViewRange vr;
    int vi0;
    int NPmax;
    int NUc;
    int n_colblk, n_rowblk;
    int nrows;  // staged rows per plane (32 + shift range + margins, <= GZRMAX)
    int ns;     // ring stages
    int* err;
    unsigned wait_limit;  // bound of the waits on staged data (wait_limit(): kWaitLimit or 0)
};

// First and last of n bins that a warp-wide test holds for, (1 << 30, -1) if none.
template <class F>
__device__ __forceinline__ int2 visible_range(int n, int lane, F test)
{
    int lo = 1 << 30, hi = -1;
    for (int i = lane; i < n; i += 32)
        if (test(i)) {
            lo = min(lo, i);
            hi = i;
        }
    return make_int2(__reduce_min_sync(0xffffffffu, lo), __reduce_max_sync(0xffffffffu, hi));
}

__device__ __forceinline__ bool view_xdriven(const petl_geom& G, int iv0)
{
    return ray_geom(G, 0, iv0, 0, 0).xdriven;
}

// X[vi][p][z][u0] for ZB rows z of plane p, for the views of the chunk that are
// driven along one axis (grid.z even: y, odd: x; above two, every n-th of
// them).  The rows are staged once for all views: a block per view read the
// volume anew for each (4.3 GB at 256x256x128 and 129 views, as much as the
// scratch it wrote) and waited for it.  A column's taps are evaluated once for
// all rows of the block; columns whose rays are all masked are left out.  AXIS
// (psi = 0 and 90, unequal pitch): the taps in double, for bins hundreds of
// voxels from the origin leave a float's fraction five digits, and a sharp image
// shows it.  Grid
// (ceil(NZ / ZB), NPmax, x_parts()); dynamic shared memory ZB rows of the
// longest in-plane axis.
template <int ZB, bool AXIS>
__global__ void __launch_bounds__(256) k_gx(const float* __restrict__ f, const float* __restrict__ fT,
                                           float* __restrict__ X, const GxArgs A)
{
    extern __shared__ float rowbuf[];
    const petl_geom& G = A.G;
    const int z0 = blockIdx.x * ZB, p = blockIdx.y;
    const bool xd = blockIdx.z & 1;  // this block's views: driven along x or along y
    const int part = blockIdx.z >> 1, nparts = (gridDim.z + 1) >> 1;
    const int NP = xd ? G.numX : G.numY, NA = xd ? G.numY : G.numX;
    if (p >= NP) return;
    const float* __restrict__ src = xd ? fT : f;  // [z][p][a]
    const int nz = min(ZB, G.numZ - z0);
    bool staged = false;
    for (int vi = part; vi < A.nvc; vi += nparts) {
        const int iv0 = A.vr.iv0_first + (A.vi0 + vi) * A.vr.iv0_step;
        if (view_xdriven(G, iv0) != xd) continue;
        if (!staged) {
            for (int e = threadIdx.x; e < nz * NA; e += blockDim.x) {
                const int r = e / NA, a = e - r * NA;
                rowbuf[r * NA + a] = src[(size_t(z0 + r) * NP + p) * NA + a];
            }
            __syncthreads();
            staged = true;
        }
        float* Xv = X + (size_t(vi) * A.NPmax + p) * G.numZ * A.NUc;
        for (int iu0 = threadIdx.x; iu0 < G.N_u0; iu0 += blockDim.x) {
            if (!u0_visible(G, iv0, iu0)) continue;
            float acc[ZB];
#pragma unroll
            for (int k = 0; k < ZB; k++) acc[k] = 0.0f;
            RayGeom r;
            PlaneTaps pt;
            double ua = 0.0, a0 = 0.0;  // AXIS: in-plane position of the ray, of voxel 0
            const double Tx = double(G.T_x), Tu = double(G.T_u0), fw = 0.5 * Tx / Tu;
            if (AXIS) {
                const double t = ((xd ? double(G.x_0) : double(G.y_0)) + p * Tx) * (xd ? -1.0 : 1.0);
                a0 = xd ? double(G.y_0) : double(G.x_0);
                ua = (double(G.u0_0) + iu0 * Tu) - t * (double(G.v0_0) + iv0 * double(G.T_v0));
                const double half = 0.5 * (Tu + Tx);
                pt.a_min = max(0, int(ceil((ua - half - a0) / Tx)));
                pt.a_max = min(NA - 1, int(floor((ua + half - a0) / Tx)));
            } else {
                r = ray_geom(G, 0, iv0, 0, iu0);
                pt = xd ? plane_taps_x(G, r, p) : plane_taps_y(G, r, p);
            }
            for (int a = pt.a_min; a <= pt.a_max; a++) {
                float w0;
                if (AXIS) {
                    const double c = (a0 + a * Tx - ua) / Tu;  // voxel centre in bins from the ray
                    w0 = float(fmin(0.5, c + fw) - fmax(-0.5, c - fw));
                } else {
                    w0 = xd ? tap_w0_x(G, r, pt.t, a, iu0) : tap_w0_y(G, r, pt.t, a, iu0);
                }
                if (!(w0 > 0.0f)) continue;
#pragma unroll
                for (int k = 0; k < ZB; k++) acc[k] = fmaf(w0, rowbuf[k * NA + a], acc[k]);
            }
#pragma unroll
            for (int k = 0; k < ZB; k++)
                if (k < nz) Xv[size_t(z0 + k) * A.NUc + iu0] = acc[k];
        }
    }
}


// NQ slope pairs x (16 / NQ) row groups of 32 per CTA: NQ = 8 is the main
// shape (16 slopes x 64 rows), NQ = 4 the tail shape (8 slopes x 128 rows)
// for a last block of few slopes, which would leave most warps of a
// 16-slope CTA idle.
template <int NQ>
__global__ void __launch_bounds__(GZT, 1) k_gz(const __grid_constant__ CUtensorMap xmap, float* __restrict__ g,
                                                const float* __restrict__ meas, const GzArgs A)
{
    constexpr int SZ = NQ * GJS, RZ = (GZT / 32 / NQ) * GRW;
    extern __shared__ __align__(128) unsigned char gsm[];
    const petl_geom& G = A.G;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int q = warp % NQ, rg = warp / NQ;
    int t_ = blockIdx.x;
    const int colblk = t_ % A.n_colblk;
    t_ /= A.n_colblk;
    const int rowblk = t_ % A.n_rowblk;
    const int v1blk = t_ / A.n_rowblk;
    const int vi = blockIdx.y;
    const int iv0 = A.vr.iv0_first + (A.vi0 + vi) * A.vr.iv0_step;
    const int v1c = A.vr.iv1_begin + v1blk * SZ;           // first slope of the CTA
    const int v1c_last = min(v1c + SZ, A.vr.iv1_end) - 1;  // last slope of the CTA
    // tiles start at the first visible row of the CTA's slopes and the first
    // visible column of the view; the tiles at the edge write the zeros of
    // the masked rays around them
    const int2 cvis = visible_range(G.N_u0, lane, [&](int c) { return u0_visible(G, iv0, c); });
    int2 rvis = make_int2(1 << 30, -1);
    for (int v = v1c; v <= v1c_last; v++) {
        const int2 x = visible_range(G.N_u1, lane, [&](int u) { return u1_visible(G, v, u); });
        rvis = make_int2(min(rvis.x, x.x), max(rvis.y, x.y));
    }
    const bool any = cvis.x <= cvis.y && rvis.x <= rvis.y;
    const int clo = any ? cvis.x & ~3 : 0, rlo = any ? rvis.x : 0;
    const int ncol = any ? (cvis.y - clo) / GZC + 1 : 1, nrow = any ? (rvis.y - rlo) / RZ + 1 : 1;
    if (colblk >= ncol || rowblk >= nrow) return;
    const int col0 = clo + colblk * GZC, iu0 = col0 + lane;
    const int row0c = rlo + rowblk * RZ, row0 = row0c + rg * GRW;
    const int v1w = v1c + q * GJS;                          // first slope of the warp
    const int nrows = A.nrows, ns = A.ns;
    const float Tu1_inv = __frcp_rn(G.T_u1);
    const float K = fmul(fsub(G.u1_0, G.z_0), Tu1_inv);  // -(row 0 position) at t = 0
    // the lane's ray geometry on this view (t depends on v0, u0 and the plane)
    const RayGeom r = ray_geom(G, 0, iv0, 0, min(iu0, G.N_u0 - 1));
    const int NP = r.xdriven ? G.numX : G.numY;
    float v1s[GJS];
#pragma unroll
    for (int j = 0; j < GJS; j++) v1s[j] = fmul(ffma(float(min(v1w + j, A.vr.iv1_end - 1)), G.T_v1, G.v1_0), Tu1_inv);

    float* ring = reinterpret_cast<float*>(gsm);                        // [ns][nrows][32]
    uint64_t* full = reinterpret_cast<uint64_t*>(ring + size_t(ns) * nrows * GZC);
    uint64_t* empty = full + GZNS;
    int* s_wr = reinterpret_cast<int*>(empty + GZNS);  // [GZNS] first staged row of the slot's plane
    int* s_round = s_wr + GZNS;                        // [GZNS] round of the copy last started in a slot
    volatile int* s_abort = s_round + GZNS;
    int* s_live = const_cast<int*>(s_abort) + 1;       // planes [s_live[0], s_live[1])
    if (tid == 0) {
        for (int k = 0; k < ns; k++) {
            mbar_init(&full[k], 1);
            mbar_init(&empty[k], GZT / 32);
            s_round[k] = -1;
        }
        *s_abort = 0;
        fence_barrier_init();
    }

    // first staged row of plane p: the smallest shift at the tile's corners
    // (monotone in t and in v1), less one row of margin
    const float v1lo = fmul(ffma(float(v1c), G.T_v1, G.v1_0), Tu1_inv);
    const float v1hi = fmul(ffma(float(v1c_last), G.T_v1, G.v1_0), Tu1_inv);
    auto first_row = [&](int p) {
        const RayGeom ra = ray_geom(G, 0, iv0, 0, col0);
        const RayGeom rb = ray_geom(G, 0, iv0, 0, min(col0 + GZC - 1, G.N_u0 - 1));
        const float ta = plane_t(G, ra, p), tb = plane_t(G, rb, p);
        const float m = fminf(fminf(fmaf(-ta, v1lo, K), fmaf(-ta, v1hi, K)), fminf(fmaf(-tb, v1lo, K), fmaf(-tb, v1hi, K)));
        return row0c + int(floorf(m)) - 1;
    };
    // planes on which a ray of the tile meets the volume (the tile's rays lie
    // between its first and last column's, and its staged rows; a voxel of
    // margin)
    if (warp == 0) {
        const RayGeom ra = ray_geom(G, 0, iv0, 0, col0);
        const RayGeom rb = ray_geom(G, 0, iv0, 0, min(col0 + GZC - 1, G.N_u0 - 1));
        const int NA = r.xdriven ? G.numY : G.numX;
        const float a0 = r.xdriven ? G.y_0 : G.x_0, half = ra.width + 1.5f * G.T_x;
        int lo = NP, hi = 0;
        if (any)
            for (int p = lane; p < NP; p += 32) {
                const float ta = plane_t(G, ra, p), tb = plane_t(G, rb, p);
                const float pa = r.xdriven ? ffma(ta, ra.ry, ra.py) : ffma(ta, ra.rx, ra.px);
                const float pb = r.xdriven ? ffma(tb, rb.ry, rb.py) : ffma(tb, rb.rx, rb.px);
                const int wr = first_row(p);
                if (fmaxf(pa, pb) + half > a0 - 0.5f * G.T_x && fminf(pa, pb) - half < a0 + (NA - 0.5f) * G.T_x &&
                    wr + nrows > 0 && wr < G.numZ) {
                    lo = min(lo, p);
                    hi = p + 1;
                }
            }
        lo = __reduce_min_sync(0xffffffffu, lo);
        hi = __reduce_max_sync(0xffffffffu, hi);
        if (lane == 0) {
            s_live[0] = min(lo, hi);
            s_live[1] = hi;
        }
    }
    __syncthreads();
    const int pl0 = s_live[0], npl = s_live[1] - s_live[0];
    // slopes and rows of this warp with a visible ray
    bool have = false;
    for (int v = v1w; v < min(v1w + GJS, v1c_last + 1); v++)
        have |= __any_sync(0xffffffffu, row0 + lane < G.N_u1 && lane < GRW && u1_visible(G, v, row0 + lane));

    const uint32_t box_bytes = uint32_t(nrows) * GZC * 4u;
    auto issue = [&](int i) {
        const int p = pl0 + i, slot = i % ns, round = i / ns;
        if (round > 0 && !mbar_wait(&empty[slot], uint32_t((round - 1) & 1), A.err, A.wait_limit)) return false;
        if (*s_abort) return false;
        fence_proxy_async_smem();
        const int wr = first_row(p);
        s_wr[slot] = wr;
        mbar_arrive_expect_tx(&full[slot], box_bytes);
        tma_load_3d(ring + size_t(slot) * nrows * GZC, &xmap, &full[slot], col0, wr, vi * A.NPmax + p);
        s_round[slot] = round;
        return true;
    };
    if (tid == 0)
        for (int i = 0; i < ns - 1 && i < npl; i++) issue(i);
    // the next plane this warp starts: the first i >= ns - 1 with i % 16 == warp
    constexpr int NW = GZT / 32;
    int my_next = warp + NW * ((ns - 1 - warp + NW - 1) / NW);
    if (my_next < ns - 1) my_next += NW;

    float acc[GJS][GRW];
#pragma unroll
    for (int j = 0; j < GJS; j++)
#pragma unroll
        for (int k = 0; k < GRW; k++) acc[j][k] = 0.0f;

    bool dead = false;
    int slot = 0;
    uint32_t phase = 0;
    for (int i = 0; i < npl; i++) {
        if (i + ns - 1 == my_next) {
            if (lane == 0 && !dead && my_next < npl && !issue(my_next)) dead = true;
            my_next += NW;
        }
        if (!dead) dead = !mbar_wait(&full[slot], phase, A.err, A.wait_limit);
        if (dead) *s_abort = 1;  // before this warp releases the slot
        if (!dead && have) {
            const float tt = plane_t(G, r, pl0 + i);
            const float* B = ring + size_t(slot) * nrows * GZC + lane;
            const int wr = s_wr[slot];
#pragma unroll
            for (int j = 0; j < GJS; j++) {
                const float nc = fmaf(-tt, v1s[j], K);
                const float sf = floorf(nc);
                const float fr = nc - sf, w0 = 1.0f - fr;
                int base = row0 + int(sf) - wr;  // staged row of tap 0 of the warp's first row
                if (base < 0 || base + GRW + 1 > nrows) {  // outside the staged rows: the host bound failed
                    atomicOr(A.err, kErrLayout);
                    base = 0;
                }
                float W[GRW + 1];
#pragma unroll
                for (int k = 0; k < GRW + 1; k++) W[k] = B[(base + k) * GZC];
#pragma unroll
                for (int k = 0; k < GRW; k++) acc[j][k] = fmaf(fr, W[k + 1], fmaf(w0, W[k], acc[j][k]));
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[slot]);
        if (++slot == ns) {
            slot = 0;
            phase ^= 1u;
        }
    }
    if (__syncthreads_or(dead)) {
        // a wait gave up: drain the copies still in flight, write nothing
        if (tid == 0)
            for (int k = 0; k < ns; k++)
                if (s_round[k] >= 0) mbar_wait(&full[k], uint32_t(s_round[k] & 1), nullptr);
        return;
    }

    // epilogue: scale, ray masks, optional MLEM ratio
    const bool ok0 = iu0 < G.N_u0 && u0_visible(G, iv0, iu0);
    const int cz0 = colblk == 0 ? 0 : col0, cz1 = colblk == ncol - 1 ? G.N_u0 : min(col0 + GZC, G.N_u0);
    const int row1 = min(row0 + GRW, G.N_u1);
    const int rz0 = rowblk == 0 && rg == 0 ? 0 : row0;
    const int rz1 = rowblk == nrow - 1 && rg == GZT / 32 / NQ - 1 ? G.N_u1 : row1;
#pragma unroll
    for (int j = 0; j < GJS; j++) {
        const int iv1 = v1w + j;
        if (iv1 > v1c_last) continue;
        const RayGeom rr = ray_geom(G, iv1, iv0, 0, min(iu0, G.N_u0 - 1));
        const size_t o0 = (size_t(iv1) * G.N_v0 + iv0) * G.N_u1 * G.N_u0;
        if (iu0 < G.N_u0) {
#pragma unroll
            for (int k = 0; k < GRW; k++) {
                if (row0 + k >= G.N_u1) break;
                const float val = ok0 && u1_visible(G, iv1, row0 + k) ? fmul(fmul(acc[j][k], rr.l_phi), rr.rs) : 0.0f;
                const size_t o = o0 + size_t(row0 + k) * G.N_u0 + iu0;
                g[o] = meas ? ratio_rule(__ldg(&meas[o]), val) : val;
            }
        }
        if (cz0 < col0 || cz1 > col0 + GZC || rz0 < row0 || rz1 > row1)
#pragma unroll 1
            for (int u = rz0; u < rz1; u++) {
                const bool inside = u >= row0 && u < row1;
#pragma unroll 1
                for (int c = cz0 + lane; c < cz1; c += 32)
                    if (!inside || c < col0 || c >= col0 + GZC) g[o0 + size_t(u) * G.N_u0 + c] = 0.0f;
            }
    }
}

// ---------------------------------------------------------------------------
// Unequal voxel height and u1 pitch on an axis-aligned planogram (psi = 0 and
// 90: PET/X's 1.6 mm bins over 0.5 mm voxels).  The ray parameter of a plane is
// the same for every column, so the edges of a ray's u1 bin cut the voxel
// column at the same heights in every column: edge k of a slope lies at
//   e_k = ((u1_0 + (iu1 - 1/2) T_u1) - t v1 - z_0) / T_z + 1/2,  iu1 = row0 + k
// in voxels, and bin k sums X over [e_k, e_k+1): the voxel of its lower edge by
// (1 - frac e_k), the whole voxels, the voxel of its upper edge by
// frac e_k+1 (all times T_z / T_u1).
//
// CTA = one view x 16 slopes (one per warp) x 32 bins x 64 columns (two per
// lane).  The voxel rows that the tile needs on a plane arrive by a tiled TMA
// copy (no multicast) into a ring of three planes; lane k of a warp places edge
// k (in double: the heights reach a hundred voxels, and their fractions are the
// weights) and the warp reads the edges back as broadcasts.  Planes on which no
// ray of the tile meets the volume are left out: with panels four times as
// long as the field of view that is most of them.  Bound by shared-memory
// loads (T_u1 / T_z + 1 rows per bin).  The general kernel recomputed both
// footprints' weights per tap and read every tap from global memory: one
// subset of 8 of PET/X's two planograms into 120x120x120 took it 27.2 ms.
constexpr int UZS = 16;              // slopes per CTA, one per warp
constexpr int UZR = 32;              // bins (rows) per CTA
constexpr int UZC = 64;              // columns per CTA
constexpr int UZT = 32 * UZS;        // threads per CTA
constexpr int UZRMAX = 250;          // staged rows per plane at most (TMA box rows <= 256)

struct UzArgs {
    petl_geom G;
    ViewRange vr;
    int vi0;
    int NPmax;
    int n_colblk, n_rowblk;
    int nrows;  // staged rows per plane
    int ns;     // ring stages (one plane each)
    int xd;     // driving planes of constant x (psi = 90), else of constant y
    int* err;
    unsigned wait_limit;
};

struct __align__(8) UEdge {
    int row;  // staged row that holds the edge
    float f;  // its fraction below the edge
};

// NI: whole voxels of a bin at most (floor of T_u1 / T_z), or -1 for any number.
template <int NI>
__global__ void __launch_bounds__(UZT, 1) k_uz(const __grid_constant__ CUtensorMap xmap, float* __restrict__ g,
                                               const float* __restrict__ meas, const UzArgs A)
{
    extern __shared__ __align__(128) unsigned char usm[];
    const petl_geom& G = A.G;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int t_ = blockIdx.x;
    const int colblk = t_ % A.n_colblk;
    t_ /= A.n_colblk;
    const int rowblk = t_ % A.n_rowblk;
    const int v1blk = t_ / A.n_rowblk;
    const int vi = blockIdx.y;
    const int iv0 = A.vr.iv0_first + (A.vi0 + vi) * A.vr.iv0_step;
    const int col0 = colblk * UZC, row0 = rowblk * UZR;
    const int v1c = A.vr.iv1_begin + v1blk * UZS, v1e = min(v1c + UZS, A.vr.iv1_end);
    const int iv1 = v1c + warp;  // the warp's slope
    const int nrows = A.nrows, ns = A.ns, NP = A.xd ? G.numX : G.numY, NA = A.xd ? G.numY : G.numX;

    float* ring = reinterpret_cast<float*>(usm);  // [ns][nrows][64]
    UEdge* edge = reinterpret_cast<UEdge*>(ring + size_t(ns) * nrows * UZC) + warp * (UZR + 1);
    uint64_t* full = reinterpret_cast<uint64_t*>(reinterpret_cast<UEdge*>(ring + size_t(ns) * nrows * UZC) +
                                                 UZS * (UZR + 1));
    uint64_t* empty = full + GZNS;
    int* s_wr = reinterpret_cast<int*>(empty + GZNS);  // [GZNS] first staged row of the slot's plane
    int* s_round = s_wr + GZNS;                        // [GZNS] round of the copy last started in a slot
    int* s_live = s_round + GZNS;                      // planes [s_live[0], s_live[1])
    volatile int* s_abort = s_live + 2;
    if (tid == 0) {
        for (int k = 0; k < ns; k++) {
            mbar_init(&full[k], 1);
            mbar_init(&empty[k], UZS);
            s_round[k] = -1;
        }
        *s_abort = 0;
        fence_barrier_init();
    }

    // the ray parameter of plane p and the height of edge k of a slope there
    const double Tz = double(G.T_z), Tu1 = double(G.T_u1), rho = Tu1 / Tz;
    const double sign = A.xd ? -double(G.sin_psi) : double(G.cos_psi);  // r_p = +-1
    const double s0 = A.xd ? double(G.x_0) : double(G.y_0);
    auto plane_par = [&](int p) { return (s0 + p * double(G.T_x)) * sign; };
    const double e0 = ((double(G.u1_0) + (row0 - 0.5) * Tu1) - double(G.z_0)) / Tz + 0.5;
    auto slope = [&](int i) { return (double(G.v1_0) + i * double(G.T_v1)) / Tz; };
    const double va = slope(v1c), vb = slope(v1e - 1);
    auto first_row = [&](int p) {
        const double t = plane_par(p);
        return int(floor(e0 - fmax(t * va, t * vb))) - 1;
    };
    // planes whose staged rows meet the volume and on which a column of the
    // tile does (a voxel of margin)
    if (warp == 0) {
        bool rows = false;
        for (int i = lane; i < (v1e - v1c) * UZR; i += 32)
            rows |= row0 + i % UZR < G.N_u1 && u1_visible(G, v1c + i / UZR, row0 + i % UZR);
        bool cols = false;
        for (int c = col0 + lane; c < min(col0 + UZC, G.N_u0); c += 32) cols |= u0_visible(G, iv0, c);
        int lo = NP, hi = 0;
        if (__any_sync(0xffffffffu, rows) && __any_sync(0xffffffffu, cols)) {
            const double v0 = double(ffma(float(iv0), G.T_v0, G.v0_0));
            const double a0 = A.xd ? double(G.y_0) : double(G.x_0), Tx = double(G.T_x);
            const double half = 0.5 * (double(G.T_u0) + Tx) + Tx;
            // in-plane position of a ray: u0 - t v0 (psi = 0), u0 - t v0 with
            // y as the in-plane axis (psi = 90)
            for (int p = lane; p < NP; p += 32) {
                const double t = plane_par(p);
                const double ua = double(G.u0_0) + col0 * double(G.T_u0), ub = ua + (UZC - 1) * double(G.T_u0);
                const double off = -t * v0;
                const bool in = ub + off + half > a0 - 0.5 * Tx && ua + off - half < a0 + (NA - 0.5) * Tx;
                const int wr = first_row(p);
                if (in && wr + nrows > 0 && wr < G.numZ) {
                    lo = min(lo, p);
                    hi = p + 1;
                }
            }
        }
        lo = __reduce_min_sync(0xffffffffu, lo);
        hi = __reduce_max_sync(0xffffffffu, hi);
        if (lane == 0) {
            s_live[0] = min(lo, hi);
            s_live[1] = hi;
        }
    }
    __syncthreads();
    const int pa = s_live[0], np = s_live[1] - s_live[0];

    const uint32_t box_bytes = uint32_t(nrows) * UZC * 4u;
    auto issue = [&](int i) {
        const int slot = i % ns, round = i / ns;
        if (round > 0 && !mbar_wait(&empty[slot], uint32_t((round - 1) & 1), A.err, A.wait_limit)) return false;
        if (*s_abort) return false;
        fence_proxy_async_smem();
        const int wr = first_row(pa + i);
        s_wr[slot] = wr;
        mbar_arrive_expect_tx(&full[slot], box_bytes);
        tma_load_3d(ring + size_t(slot) * nrows * UZC, &xmap, &full[slot], col0, wr, vi * A.NPmax + pa + i);
        s_round[slot] = round;
        return true;
    };
    if (tid == 0)
        for (int i = 0; i < ns - 1 && i < np; i++) issue(i);
    // the next plane this warp starts: the first i >= ns - 1 with i % 16 == warp
    int my_next = warp + UZS * ((ns - 1 - warp + UZS - 1) / UZS);
    if (my_next < ns - 1) my_next += UZS;

    using shear::f2x;
    f2x acc[UZR];
#pragma unroll
    for (int k = 0; k < UZR; k++) acc[k] = 0ull;
    const double v1z = slope(min(iv1, A.vr.iv1_end - 1));
    // a bin of the warp's slope is visible
    const bool have = iv1 < v1e && __any_sync(0xffffffffu, row0 + lane < G.N_u1 && u1_visible(G, iv1, row0 + lane));
    bool dead = false;
    int slot = 0;
    uint32_t phase = 0;
    for (int i = 0; i < np; i++) {
        if (i + ns - 1 == my_next) {
            if (lane == 0 && !dead && my_next < np && !issue(my_next)) dead = true;
            my_next += UZS;
        }
        if (!dead) dead = !mbar_wait(&full[slot], phase, A.err, A.wait_limit);
        dead = __any_sync(0xffffffffu, dead);
        if (dead) *s_abort = 1;  // before this warp releases the slot
        const double ez = e0 - plane_par(pa + i) * v1z;  // edge 0
        if (!dead && have && ez < G.numZ && ez + UZR * rho > 0.0) {
            const double eb = ez - s_wr[slot];
            bool bad = false;
            for (int k = lane; k <= UZR; k += 32) {
                const double e = fma(double(k), rho, eb), fl = floor(e);
                const int row = int(fl);
                bad |= row < 0 || row >= nrows;
                edge[k] = UEdge{min(max(row, 0), nrows - 1), float(e - fl)};
            }
            if (bad) atomicOr(A.err, kErrLayout);  // outside the staged rows: the host bound failed
            __syncwarp();
            const f2x* B = reinterpret_cast<const f2x*>(ring + size_t(slot) * nrows * UZC) + lane;
            UEdge a = edge[0];
            f2x xa = B[a.row * (UZC / 2)];
#pragma unroll
            for (int k = 0; k < UZR; k++) {
                const UEdge b = edge[k + 1];
                const int n = b.row - a.row;
                acc[k] = shear::f2_fma(shear::f2_dup(n > 0 ? 1.0f - a.f : b.f - a.f), xa, acc[k]);
                if constexpr (NI >= 0) {
#pragma unroll
                    for (int j = 1; j <= NI; j++)
                        if (j < n) acc[k] = shear::f2_add(acc[k], B[(a.row + j) * (UZC / 2)]);
                } else {
                    for (int j = 1; j < n; j++) acc[k] = shear::f2_add(acc[k], B[(a.row + j) * (UZC / 2)]);
                }
                xa = B[b.row * (UZC / 2)];
                if (n > 0 && b.f > 0.0f) acc[k] = shear::f2_fma(shear::f2_dup(b.f), xa, acc[k]);
                a = b;
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[slot]);
        if (++slot == ns) {
            slot = 0;
            phase ^= 1u;
        }
    }
    if (__syncthreads_or(dead)) {
        // a wait gave up: drain the copies still in flight, write nothing
        if (tid == 0)
            for (int k = 0; k < ns; k++)
                if (s_round[k] >= 0) mbar_wait(&full[k], uint32_t(s_round[k] & 1), nullptr);
        return;
    }

    // epilogue: scale, ray masks, optional MLEM ratio
    const int iu0 = col0 + 2 * lane;
    if (iv1 >= v1e || iu0 >= G.N_u0) return;
    const RayGeom rr = ray_geom(G, iv1, iv0, 0, iu0);
    const float c = float(Tz / Tu1);
    const bool two = iu0 + 1 < G.N_u0;
    const bool ok0 = u0_visible(G, iv0, iu0), ok1 = two && u0_visible(G, iv0, iu0 + 1);
#pragma unroll
    for (int k = 0; k < UZR; k++) {
        const int iu1 = row0 + k;
        if (iu1 >= G.N_u1) break;
        const bool rv = u1_visible(G, iv1, iu1);
        const float2 v = shear::f2_unpack(acc[k]);
        float2 o = make_float2(rv && ok0 ? fmul(fmul(fmul(v.x, c), rr.l_phi), rr.rs) : 0.0f,
                               rv && ok1 ? fmul(fmul(fmul(v.y, c), rr.l_phi), rr.rs) : 0.0f);
        const size_t at = ((size_t(iv1) * G.N_v0 + iv0) * G.N_u1 + iu1) * G.N_u0 + iu0;
        if (meas) o = make_float2(ratio_rule(__ldg(meas + at), o.x), two ? ratio_rule(__ldg(meas + at + 1), o.y) : 0.0f);
        g[at] = o.x;
        if (two) g[at + 1] = o.y;
    }
}

// grid.z of k_gx: both driving axes, and the views split over more blocks
// where rows and planes alone give an SM less than about eight blocks.
unsigned x_parts(unsigned blocks, int nviews)
{
    const unsigned want = ceil_div(8ll * sm_count(), blocks);
    return 2u * std::max(1u, std::min(want, unsigned(nviews)));
}

bool aligned_90(const petl_geom& G) { return std::fabs(G.cos_psi) < 1e-6f && G.sin_psi == 1.0f; }

// Whether the views of a call on a geometry with unequal voxel height and u1
// pitch take the edges in double: along one axis, and staged rows that fit.
// The forward and its adjoint ask the same, so that they take the same
// weights.
struct UPlan {
    bool xd;    // driving planes of constant x
    int nrows;  // staged rows per plane
};

bool usplit_applies(const petl_geom& G, const ViewRange& vr, UPlan& P)
{
    const int n_v0 = vr.n_v0(G.N_v0);
    if (G.N_u0 > 4096 || G.numX > 4096 || G.numY > 4096) return false;
    P.xd = aligned_90(G);
    if (!P.xd && !(G.cos_psi == 1.0f && G.sin_psi == 0.0f)) return false;
    for (int k = 0; k < n_v0; k++)
        if (host_view(G, vr.iv0_first + k * vr.iv0_step).xd != P.xd) return false;
    const int NP = P.xd ? G.numX : G.numY;
    const double rho = double(G.T_u1) / double(G.T_z);
    const double first = P.xd ? double(G.x_0) : double(G.y_0);
    const double tmax = std::max(std::fabs(first), std::fabs(first + (NP - 1) * double(G.T_x)));
    const double spread = (UZS - 1) * std::fabs(double(G.T_v1)) * tmax / double(G.T_z);
    // the rows of 32 bins, the slopes' spread and a row on either side
    const double need = UZR * rho + spread * (1.0 + 1e-6) + 4.0;
    if (!(need <= UZRMAX)) return false;
    P.nrows = int(std::ceil(need));
    return true;
}

// The same sums a ray per thread, for calls too small for k_uz (uz_rays): no
// scratch, one launch, the weights of k_gx and k_uz.  Grid (ceil(N_u0 / 32),
// ceil(N_u1 / 4), slopes x views), 32 x 4 threads.
__global__ void __launch_bounds__(128)
k_project_uz_rays(const float* __restrict__ f, float* __restrict__ g, const float* __restrict__ meas, const petl_geom G,
                  const ViewRange vr, int n_v0, int xd)
{
    const int iu0 = blockIdx.x * 32 + threadIdx.x, iu1 = blockIdx.y * 4 + threadIdx.y;
    const int iv1 = vr.iv1_begin + blockIdx.z / n_v0, iv0 = vr.iv0_first + blockIdx.z % n_v0 * vr.iv0_step;
    if (iu0 >= G.N_u0 || iu1 >= G.N_u1) return;
    float val = 0.0f;
    if (ray_visible(G, iv1, iv0, iu1, iu0)) {
        const double Tx = double(G.T_x), Tu0 = double(G.T_u0), Tz = double(G.T_z), Tu1 = double(G.T_u1), rho = Tu1 / Tz;
        const int NP = xd ? G.numX : G.numY, NA = xd ? G.numY : G.numX;
        const size_t sa = xd ? size_t(G.numX) : 1, sp = xd ? 1 : size_t(G.numX), sz = size_t(G.numX) * G.numY;
        // in-plane position of the ray in voxels and its lower edge in rows, at t = 0 and per t
        const double a0 = (double(G.u0_0) + iu0 * Tu0 - (xd ? double(G.y_0) : double(G.x_0))) / Tx;
        const double e0 = ((double(G.u1_0) + (iu1 - 0.5) * Tu1) - double(G.z_0)) / Tz + 0.5;
        const double da = (double(G.v0_0) + iv0 * double(G.T_v0)) / Tx, de = (double(G.v1_0) + iv1 * double(G.T_v1)) / Tz;
        const double half = 0.5 * (Tu0 / Tx + 1.0), hu = 0.5 * Tu0 / Tx, q = Tx / Tu0;
        for (int p = 0; p < NP; p++) {
            const double t = ((xd ? double(G.x_0) : double(G.y_0)) + p * Tx) * (xd ? -1.0 : 1.0);
            const double ua = a0 - t * da, e = e0 - t * de, eh = e + rho;
            const int z0 = max(0, int(floor(e))), z1 = min(G.numZ - 1, int(floor(eh)));
            if (z0 > z1) continue;
            const int i0 = max(0, int(ceil(ua - half))), i1 = min(NA - 1, int(floor(ua + half)));
            const float* fp = f + size_t(p) * sp;
            for (int a = i0; a <= i1; a++) {
                // overlap of the bin and the voxel's tent of the plane, in bins
                const float w0 = float((fmin(ua + hu, a + 0.5) - fmax(ua - hu, a - 0.5)) * q);
                if (!(w0 > 0.0f)) continue;
                float s = 0.0f;
                for (int z = z0; z <= z1; z++) {
                    const float w1 = float(fmin(eh, z + 1.0) - fmax(e, double(z)));
                    s = ffma(w1, __ldg(fp + size_t(a) * sa + size_t(z) * sz), s);
                }
                val = ffma(w0, s, val);
            }
        }
        const RayGeom r = ray_geom(G, iv1, iv0, iu1, iu0);
        val = fmul(fmul(fmul(val, float(Tz / Tu1)), r.l_phi), r.rs);
    }
    const size_t o = ((size_t(iv1) * G.N_v0 + iv0) * G.N_u1 + iu1) * G.N_u0 + iu0;
    g[o] = meas ? ratio_rule(__ldg(&meas[o]), val) : val;
}

// The exact transpose of k_gx<.., true> + k_uz, one thread per voxel: the same
// bin edges and u0 positions in double, so that the two agree to the rounding
// of their sums.  (The general adjoint's float edges differ by up to 1e-5 of
// a bin for bins a hundred voxels from the origin.)  Grid as the general
// kernel's: (ceil(numX / 32), ceil(numY / 4), numZ), 32 x 4 threads.  Per slope
// the voxel's u1 bins are the same for every view: their weights are formed
// once, four at a time.  120x120x120 voxels of 0.5 mm from one of 8 subsets of
// PET/X's planograms: 9.4 ms (psi = 0) and 31.8 ms (psi = 90); the general
// kernel, which forms both weights anew for every candidate ray, 182 and 709.
__global__ void __launch_bounds__(128)
k_backproject_uz(const float* __restrict__ g, float* __restrict__ f, const petl_geom G, const ViewRange vr, int xd,
                 int accumulate, float scale)
{
    constexpr int NW = 4;  // u1 bins at a time
    const int ix = blockIdx.x * 32 + threadIdx.x, iy = blockIdx.y * 4 + threadIdx.y, iz = blockIdx.z;
    if (ix >= G.numX || iy >= G.numY) return;
    const double Tx = double(G.T_x), Tu0 = double(G.T_u0), Tz = double(G.T_z), Tu1 = double(G.T_u1), rho = Tu1 / Tz;
    // ray parameter of the voxel's plane, in-plane position in bins at v0 = 0
    const double t = xd ? -(double(G.x_0) + ix * Tx) : double(G.y_0) + iy * Tx;
    const double a = xd ? double(G.y_0) + iy * Tx : double(G.x_0) + ix * Tx;
    const double c00 = (a - double(G.u0_0)) / Tu0, tu = t / Tu0, fw = 0.5 * Tx / Tu0;
    const double e00 = ((double(G.u1_0) - 0.5 * Tu1) - double(G.z_0)) / Tz + 0.5 - iz;
    const float c = float(Tz / Tu1), l_phi = G.T_x;
    float acc = 0.0f;
    for (int iv1 = vr.iv1_begin; iv1 < vr.iv1_end; iv1++) {
        // edge k of the slope's bins lies at e0 + k rho above the voxel's lower face
        const double e0 = e00 - t * ((double(G.v1_0) + iv1 * double(G.T_v1)) / Tz);
        const int k0 = max(0, int(floor(-e0 / rho))), k1 = min(G.N_u1 - 1, int(floor((1.0 - e0) / rho)));
        const float v1 = ffma(float(iv1), G.T_v1, G.v1_0);
        for (int kb = k0; kb <= k1; kb += NW) {
            float w1[NW];
            bool any = false;
#pragma unroll
            for (int i = 0; i < NW; i++) {
                const double lo = fmax(0.0, fma(double(kb + i), rho, e0));
                const double hi = fmin(1.0, fma(double(kb + i + 1), rho, e0));
                const bool ok = kb + i <= k1 && hi > lo && u1_visible(G, iv1, kb + i);
                w1[i] = ok ? float(hi - lo) : 0.0f;
                any |= ok;
            }
            if (!any) continue;
            for (int iv0 = vr.iv0_first; iv0 < G.N_v0; iv0 += vr.iv0_step) {
                const double cc = fma(tu, double(G.v0_0) + iv0 * double(G.T_v0), c00);  // voxel centre in bins
                const int j0 = max(0, int(ceil(cc - fw - 0.5))), j1 = min(G.N_u0 - 1, int(floor(cc + fw + 0.5)));
                const float* gv = g + ((size_t(iv1) * G.N_v0 + iv0) * G.N_u1 + kb) * G.N_u0;
                float sview = 0.0f;
                for (int j = j0; j <= j1; j++) {
                    const float w0 = float(fmin(0.5, cc - j + fw) - fmax(-0.5, cc - j - fw));
                    if (!(w0 > 0.0f) || !u0_visible(G, iv0, j)) continue;
                    float sk = 0.0f;
#pragma unroll
                    for (int i = 0; i < NW; i++)
                        if (w1[i] > 0.0f) sk = ffma(w1[i], __ldg(gv + size_t(i) * G.N_u0 + j), sk);
                    sview = ffma(w0, sk, sview);
                }
                const float v0 = ffma(float(iv0), G.T_v0, G.v0_0);
                const float rs = __frsqrt_rn(ffma(v0, v0, ffma(v1, v1, 1.0f)));
                acc = fadd(acc, fmul(fmul(fmul(sview, c), l_phi), rs));
            }
        }
    }
    const size_t o = (size_t(iz) * G.numY + iy) * G.numX + ix;
    const float r = acc * scale;
    f[o] = accumulate ? f[o] + r : r;
}

// Whether a call is too small for k_gx + k_uz: fewer taps on a plane (rays times
// the voxels that a bin meets) than 7e5.  Their time is then the latency of two
// launches and of the planes of a few CTAs.  Median of 6300 random calls at psi =
// 0 and 90, general kernel / k_gx + k_uz / rays, us: below 5e4 taps 32 / 36 / 27,
// 2e5 to 4e5 79 / 80 / 68, 4e5 to 7e5 101 / 92 / 88, 7e5 to 1.2e6 137 / 108 / 130,
// 2.5e6 to 1e7 508 / 149 / 478.
bool uz_rays(const petl_geom& G, int nv1, int n_v0)
{
    const double views = double(nv1) * n_v0;
    const double taps = views * G.N_u1 * G.N_u0 * (double(G.T_u1) / double(G.T_z) + 1.0) * (double(G.T_u0) / double(G.T_x) + 1.0);
    return views <= 65535.0 && taps < 7.0e5;
}

// The split forward for unequal voxel height and u1 pitch; kNotApplicable (-2)
// off the axes and where the staged rows would not fit.
int project_usplit(const petl_geom& G, const float* f, float* g, const ViewRange& vr, const float* meas,
                   cudaStream_t st)
{
    constexpr int kNotApplicable = -2;
    const int n_v0 = vr.n_v0(G.N_v0), nv1 = vr.iv1_end - vr.iv1_begin;
    UPlan P;
    if (!usplit_applies(G, vr, P)) return kNotApplicable;
    const bool xd = P.xd;
    const int NP = xd ? G.numX : G.numY, NA = xd ? G.numY : G.numX, nrows = P.nrows;
    const double rho = double(G.T_u1) / double(G.T_z);
    if (uz_rays(G, nv1, n_v0)) {
        k_project_uz_rays<<<dim3(ceil_div(G.N_u0, 32), ceil_div(G.N_u1, 4), unsigned(nv1) * unsigned(n_v0)), dim3(32, 4), 0,
                            st>>>(f, g, meas, G, vr, n_v0, xd);
        PETL_LAUNCH_CHECK("project_uz_rays");
        return 0;
    }
    int* err = device_error_ptr();
    if (!err) return kNotApplicable;
    const int NUc = (G.N_u0 + 3) & ~3;
    const size_t per_view = size_t(NP) * G.numZ * NUc * 4;
    int nv = int(std::max<size_t>(1, std::min<size_t>(size_t(n_v0), gsplit_scratch_budget() / per_view)));
    nv = std::min(nv, 65535);
    if (NP > 65535) return kNotApplicable;
    const int nchunks = (n_v0 + nv - 1) / nv;
    nv = (n_v0 + nchunks - 1) / nchunks;
    const size_t stage = size_t(nrows) * UZC * 4;
    UzArgs Z{};
    Z.G = G;
    Z.vr = vr;
    Z.NPmax = NP;
    Z.n_colblk = int(ceil_div(G.N_u0, UZC));
    Z.n_rowblk = int(ceil_div(G.N_u1, UZR));
    Z.nrows = nrows;
    Z.ns = int(std::min<size_t>(GZNS, (200 * 1024) / stage));
    Z.xd = xd;
    Z.err = err;
    Z.wait_limit = wait_limit();
    if (Z.ns < 2) return kNotApplicable;
    const size_t smem = size_t(Z.ns) * stage + size_t(UZS) * (UZR + 1) * sizeof(UEdge) + GZNS * 16 + GZNS * 8 + 16;
    float* X = nullptr;
    float* fT = nullptr;
    if (scratch_alloc(reinterpret_cast<void**>(&X), per_view * nv, st) != cudaSuccess ||
        (xd && scratch_alloc(reinterpret_cast<void**>(&fT), size_t(G.numX) * G.numY * G.numZ * 4, st) != cudaSuccess)) {
        cudaGetLastError();
        if (X) cudaFreeAsync(X, st);
        return kNotApplicable;
    }
    CUtensorMap map;
    const uint64_t dims[3] = {uint64_t(NUc), uint64_t(G.numZ), uint64_t(NP) * uint64_t(nv)};
    const uint64_t strides[2] = {uint64_t(NUc) * 4, uint64_t(NUc) * G.numZ * 4};
    const uint32_t box[3] = {uint32_t(UZC), uint32_t(nrows), 1u};
    if (!encode_tensor_map(&map, X, 3, dims, strides, box, 4)) {
        cudaFreeAsync(X, st);
        if (fT) cudaFreeAsync(fT, st);
        return kNotApplicable;
    }
    if (xd) {
        k_transpose_xy<<<dim3(ceil_div(G.numX, 32), ceil_div(G.numY, 32), unsigned(G.numZ)), dim3(32, 8), 0, st>>>(
            f, fT, G.numX, G.numY);
        note_launch();
    }
    const int xzb = NA <= GXZ_AXIS ? GXZ : GXZ_LONG;
    auto kx = xzb == GXZ ? k_gx<GXZ, true> : k_gx<GXZ_LONG, true>;
    const size_t xsmem = size_t(xzb) * NA * 4;
    const int ni = int(std::floor(rho));
    auto kz = ni == 0 ? k_uz<0> : ni == 1 ? k_uz<1> : ni == 2 ? k_uz<2> : ni == 3 ? k_uz<3> : k_uz<-1>;
    cudaError_t e = cudaFuncSetAttribute(kx, cudaFuncAttributeMaxDynamicSharedMemorySize, int(xsmem));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kz, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    for (int c = 0; c < nchunks && e == cudaSuccess; c++) {
        const int vi0 = c * nv, nvc = std::min(nv, n_v0 - vi0);
        const GxArgs XA{G, vr, vi0, nvc, NP, NUc};
        kx<<<dim3(ceil_div(G.numZ, xzb), unsigned(NP), x_parts(ceil_div(G.numZ, xzb) * unsigned(NP), nvc)), 256, xsmem,
             st>>>(f, fT, X, XA);
        note_launch();
        Z.vi0 = vi0;
        kz<<<dim3(unsigned(Z.n_colblk) * unsigned(Z.n_rowblk) * ceil_div(nv1, UZS), unsigned(nvc)), UZT, smem, st>>>(
            map, g, meas, Z);
        note_launch();
        e = cudaGetLastError();
    }
    cudaFreeAsync(X, st);
    if (fT) cudaFreeAsync(fT, st);
    if (e != cudaSuccess) {
        set_error(std::string("project_usplit: ") + cudaGetErrorString(e));
        return int(e);
    }
    return 0;
}

}  // namespace


__global__ void k_transpose_xy(const float* __restrict__ in, float* __restrict__ out, int nx, int ny)
{
    __shared__ float tile[32][33];
    const int z = blockIdx.z, x0 = blockIdx.x * 32, y0 = blockIdx.y * 32;
    const float* fz = in + size_t(z) * nx * ny;
    float* tz = out + size_t(z) * nx * ny;
    for (int j = threadIdx.y; j < 32; j += blockDim.y) {
        const int y = y0 + j, x = x0 + threadIdx.x;
        if (y < ny && x < nx) tile[j][threadIdx.x] = fz[size_t(y) * nx + x];
    }
    __syncthreads();
    for (int j = threadIdx.y; j < 32; j += blockDim.y) {
        const int x = x0 + j, y = y0 + threadIdx.x;
        if (x < nx && y < ny) tz[size_t(x) * ny + y] = tile[threadIdx.x][j];
    }
}

int backproject_usplit_adjoint(const petl_geom& G, const float* g, float* f, int accumulate, float scale,
                               const ViewRange& vr, cudaStream_t st)
{
    UPlan P;
    if (G.T_z == G.T_u1 || G.numZ > 65535 || !usplit_applies(G, vr, P)) return -2;
    const dim3 grid(ceil_div(G.numX, 32), ceil_div(G.numY, 4), unsigned(G.numZ));
    k_backproject_uz<<<grid, dim3(32, 4), 0, st>>>(g, f, G, vr, P.xd, accumulate, scale);
    PETL_LAUNCH_CHECK("backproject_usplit_adjoint");
    return 0;
}

// kNotApplicable when the layout rules fail (the caller then runs the
// general kernel): voxel height != u1 pitch off the axes, a view whose shift
// range over a tile exceeds the staged rows, or scratch that cannot be
// allocated.
int project_gsplit(const petl_geom& G, const float* f, float* g, const ViewRange& vr, const float* meas,
                   cudaStream_t st)
{
    constexpr int kNotApplicable = -2;
    const int n_v0 = vr.n_v0(G.N_v0);
    const int nv1 = vr.iv1_end - vr.iv1_begin;
    if (n_v0 <= 0 || nv1 <= 0) return 0;
    if (G.N_u0 > 4096 || G.numX > 4096 || G.numY > 4096) return kNotApplicable;
    if (G.T_z != G.T_u1) return project_usplit(G, f, g, vr, meas, st);
    // staged rows per plane: the CTA's rows + the range of floor(-c0) over a
    // tile's 32 columns and its slopes + margins.  -c0 = (u1_0 - z_0 + t v1)
    // / T_u1 with t = (coordinate of the plane - u0 pscale) * inv: bounded
    // with the extremes of |t| and of its change over 32 columns.
    const double vmax = std::max(std::fabs(double(G.v1_0)), std::fabs(double(G.v1_0) + (G.N_v1 - 1) * double(G.T_v1)));
    const double xext = std::max(std::fabs(double(G.x_0)), std::fabs(double(G.x_0) + (G.numX - 1) * double(G.T_x)));
    const double yext = std::max(std::fabs(double(G.y_0)), std::fabs(double(G.y_0) + (G.numY - 1) * double(G.T_x)));
    const double uext = std::max(std::fabs(double(G.u0_0)), std::fabs(double(G.u0_0) + (G.N_u0 - 1) * double(G.T_u0)));
    double tmax = 0, dtmax = 0;
    bool any_xd = false;
    for (int k = 0; k < n_v0; k++) {
        const HostView h = host_view(G, vr.iv0_first + k * vr.iv0_step);
        any_xd = any_xd || h.xd;
        tmax = std::max(tmax, (std::max(xext, yext) + uext * h.pscale) * std::fabs(h.inv));
        dtmax = std::max(dtmax, GZC * double(G.T_u0) * h.pscale * std::fabs(h.inv));
    }
    auto staged_rows = [&](int slopes, int rows) {
        const double dv1 = (slopes - 1) * std::fabs(double(G.T_v1));
        const double spread = (dtmax * vmax + tmax * dv1 + dtmax * dv1) / double(G.T_u1);
        return rows + int(std::ceil(spread * (1.0 + 1e-6))) + 5;  // + floors and the one-row margins
    };
    const int nrows = staged_rows(GZS, GZR);
    if (nrows > GZRMAX) return kNotApplicable;
    // a last block of at most 8 slopes runs in the tail shape
    const int rem = nv1 % GZS;
    const int nrows_t = staged_rows(GZS_T, GZR_T);
    const bool tail = rem > 0 && rem <= GZS_T && nrows_t <= GZRMAX && G.N_u1 > GZR;
    const int nv1_main = tail ? nv1 - rem : nv1;
    int* err = device_error_ptr();
    if (!err) return kNotApplicable;

    const int NPmax = any_xd ? std::max(G.numX, G.numY) : G.numY;
    const int NUc = (G.N_u0 + 3) & ~3;
    const size_t per_view = size_t(NPmax) * G.numZ * NUc * 4;
    int nv = int(std::max<size_t>(1, std::min<size_t>(size_t(n_v0), gsplit_scratch_budget() / per_view)));
    nv = std::min(nv, 65535);
    const int nchunks = (n_v0 + nv - 1) / nv;
    nv = (n_v0 + nchunks - 1) / nchunks;
    float* X = nullptr;
    float* fT = nullptr;
    if (scratch_alloc(reinterpret_cast<void**>(&X), per_view * nv, st) != cudaSuccess ||
        (any_xd && scratch_alloc(reinterpret_cast<void**>(&fT), size_t(G.numX) * G.numY * G.numZ * 4, st) !=
                       cudaSuccess)) {
        cudaGetLastError();
        if (X) cudaFreeAsync(X, st);
        return kNotApplicable;
    }
    cudaError_t e = cudaSuccess;
    if (any_xd) {
        k_transpose_xy<<<dim3(ceil_div(G.numX, 32), ceil_div(G.numY, 32), unsigned(G.numZ)), dim3(32, 8), 0, st>>>(
            f, fT, G.numX, G.numY);
        note_launch();
    }
    const int NAmax = any_xd ? std::max(G.numX, G.numY) : G.numX;
    const int xzb = NAmax <= GXZ_AXIS ? GXZ : GXZ_LONG;
    auto kx = xzb == GXZ ? k_gx<GXZ, false> : k_gx<GXZ_LONG, false>;
    const size_t xsmem = size_t(xzb) * NAmax * 4;
    e = cudaFuncSetAttribute(kx, cudaFuncAttributeMaxDynamicSharedMemorySize, int(xsmem));
    // one z launch shape: its argument block, tensor map (boxes of 32
    // columns x its staged rows; TMA, no multicast; rows outside read zero)
    // and shared memory
    struct ZLaunch {
        GzArgs Z;
        CUtensorMap map;
        size_t smem;
        unsigned nblk;
    };
    auto z_setup = [&](ZLaunch& L, int rows_cta, int slopes_cta, int staged, int v1b, int v1e) -> cudaError_t {
        const size_t stage = size_t(staged) * GZC * 4;
        const int ns = int(std::min<size_t>(GZNS, (200 * 1024) / stage));
        if (ns < 2) return cudaErrorInvalidValue;
        L.smem = size_t(ns) * stage + GZNS * 16 + GZNS * 8 + 16;  // ring, barriers, slot words, abort and live planes
        L.Z = GzArgs{};
        L.Z.G = G;
        L.Z.vr = vr;
        L.Z.vr.iv1_begin = v1b;
        L.Z.vr.iv1_end = v1e;
        L.Z.NPmax = NPmax;
        L.Z.NUc = NUc;
        L.Z.n_colblk = int(ceil_div(G.N_u0, GZC));
        L.Z.n_rowblk = int(ceil_div(G.N_u1, rows_cta));
        L.Z.nrows = staged;
        L.Z.ns = ns;
        L.Z.err = err;
        L.Z.wait_limit = wait_limit();
        L.nblk = unsigned(L.Z.n_colblk) * unsigned(L.Z.n_rowblk) * ceil_div(v1e - v1b, slopes_cta);
        const uint64_t dims[3] = {uint64_t(NUc), uint64_t(G.numZ), uint64_t(NPmax) * uint64_t(nv)};
        const uint64_t strides[2] = {uint64_t(NUc) * 4, uint64_t(NUc) * G.numZ * 4};
        const uint32_t box[3] = {uint32_t(GZC), uint32_t(staged), 1u};
        return encode_tensor_map(&L.map, X, 3, dims, strides, box, 4) ? cudaSuccess : cudaErrorInvalidValue;
    };
    ZLaunch zm{}, zt{};
    if (e == cudaSuccess && nv1_main > 0) e = z_setup(zm, GZR, GZS, nrows, vr.iv1_begin, vr.iv1_begin + nv1_main);
    if (e == cudaSuccess && tail) e = z_setup(zt, GZR_T, GZS_T, nrows_t, vr.iv1_begin + nv1_main, vr.iv1_end);
    if (e == cudaSuccess && nv1_main > 0)
        e = cudaFuncSetAttribute(k_gz<GZS / GJS>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(zm.smem));
    if (e == cudaSuccess && tail)
        e = cudaFuncSetAttribute(k_gz<GZS_T / GJS>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(zt.smem));
    for (int c = 0; c < nchunks && e == cudaSuccess; c++) {
        const int vi0 = c * nv, nvc = std::min(nv, n_v0 - vi0);
        const GxArgs XA{G, vr, vi0, nvc, NPmax, NUc};
        kx<<<dim3(ceil_div(G.numZ, xzb), unsigned(NPmax), x_parts(ceil_div(G.numZ, xzb) * unsigned(NPmax), nvc)), 256,
             xsmem, st>>>(f, fT, X, XA);
        note_launch();
        if (nv1_main > 0) {
            zm.Z.vi0 = vi0;
            k_gz<GZS / GJS><<<dim3(zm.nblk, unsigned(nvc)), GZT, zm.smem, st>>>(zm.map, g, meas, zm.Z);
            note_launch();
        }
        if (tail) {
            zt.Z.vi0 = vi0;
            k_gz<GZS_T / GJS><<<dim3(zt.nblk, unsigned(nvc)), GZT, zt.smem, st>>>(zt.map, g, meas, zt.Z);
            note_launch();
        }
        e = cudaGetLastError();
    }
    cudaFreeAsync(X, st);
    if (fT) cudaFreeAsync(fT, st);
    if (e != cudaSuccess) {
        set_error(std::string("project_gsplit: ") + cudaGetErrorString(e));
        return int(e);
    }
    return 0;
}

}  // namespace petl
