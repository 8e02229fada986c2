// Split forward projector (psi = 0, voxel pitch equal to the bin pitch).
//
// The shear-warp form of the reference footprint (src/projectors.cu:131-185,
// see projector_shear.cu) adds, for every plane y,
//   g[v1][v0][iu1][iu0] += wz0 X[iu1 + dz][iu0] + wz1 X[iu1 + dz + 1][iu0]
// where X is plane y of the volume interpolated in x by the shift of view v0:
//   X_v0[y][z][c] = (1 - wx) f[z][y][c + dx] + wx f[z][y][c + dx + 1].
// project_tma computes X inside every CTA (stage A) between two CTA barriers
// per plane pair.  Here the two stages are separate kernels:
//
// * k_xshift writes X for a chunk of views into FP32 scratch, [view][y][z][c]
//   (memory bound: one write of a volume per view; each volume row is read
//   once per chunk);
// * k_fwd_zsum applies the z taps: persistent CTAs of twelve consumer warps
//   and a producer warp that stages planes by tiled TMA copies (no multicast)
//   into a ring with full/empty mbarriers, across tile borders.  The tap
//   offsets of a warp's four consecutive slopes move by at most one row from
//   slope to slope, so they form one of 15 monotone patterns: one dispatch per
//   run of planes with the same one selects a fully unrolled form.
//
// 256x256x128, planogram (65, 129, 128, 256): 7.88 ms, of which 6.8 the z taps
// (before: 10.9 and 10.0, with one 16-warp CTA per tile, tables built by every
// CTA, scalar FMAs on 8 rows per warp and tiles that started at bin 0).  What the steps gave on the z taps: twelve warps x 12 rows against
// eight x 16 9 %, tiles handed out by a counter against a fixed stride 18 % (the
// stride of 148 met the period of the column blocks, whose last is often
// empty), a rolled epilogue 10 %, twelve rows at a time against four 4 %, runs of
// planes with one pattern 7 %, and the epilogue's
// loads in batches another 25 % where the MLEM ratio is computed.
//
// Both kernels do the float operations of project_tma in the same order (x
// taps fmaf(w1, b, w0 * a); per ray, the z taps of the live planes in
// ascending y, tap 0 then tap 1), so the two paths agree bit for bit.
//
// A launch serves the views of one call or, for the server's batched steps,
// of up to kMaxMembers requests of one geometry (Members: per-member
// volumes, planograms and view subsets; member b's views in scratch slots
// b * nvm + v).  The kernels are compiled for one member (plain calls) and
// for up to kMaxMembers.
//
// Every wait is bounded: a wait that gives up sets the device error word,
// the CTA drains its copies in flight and returns without writing.
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>

#include "common.cuh"
#include "projector.cuh"
#include "shear.cuh"
#include "storage.cuh"
#include "tma.cuh"
#include "ztaps.cuh"

namespace petl {
namespace shear {

namespace {

constexpr int ZSLOPES = 16;           // slopes per block at most (a table record holds 16 weights)
constexpr int XZB = 8;                // volume rows z per k_xshift block
constexpr int XMAXNX = 1024;          // longest volume row k_xshift stages

// Table record of one (slope block, plane), staged with the plane: the second
// tap's weight of each slope, and per slope group (warp) the tap offsets (2
// bits per slope) and the window's first staged row << 8.
struct __align__(16) ZRec {
    float w[ZSLOPES];
    uint32_t code[kZWarps];
};

// Blocks of slopes that share a launch shape: sg slope groups (warps along
// v1) x rg row groups (warps along u1).
struct ZKind {
    int v1_first, v1_end;
    int sg, rg, rows;  // rows = NK * rg
    int nblk;          // slope blocks
    int n_rowblk;      // row blocks at most (the visible rows of a block need fewer)
    int nrb;           // staged rows per plane (rows + shift spread of the block + 1)
    int pstride;       // floats per staged plane (nrb + kZSpread rows of 64)
    int pps;           // planes per stage
    int blk0;          // index of the first block in the tables
    int ntile;
};

struct ZsumArgs {
    petl_geom G;
    int step;       // view step of the members' view ranges
    int nw;         // consumer warps
    int nslot;      // view slots of all members
    int n_colblk;   // column blocks at most
    int ns;         // ring stages
    int stage;      // bytes per stage (planes, then their records)
    int rec_off;    // the records' offset in a stage
    int pairs;      // the planograms take column-pair accesses (pair_access)
    ZKind k[2];     // full blocks, and the tail of at most half a block
    ZRec* rec;      // [block][plane]
    int* dz;        // [block][plane] smallest shift of the block
    int* next;      // tiles handed out beyond one per CTA
    Tables T;
    int* err;
    unsigned wait_limit;  // bound of the waits on staged data (wait_limit(): kWaitLimit or 0)
    Members M;            // planograms (out), measured planograms (meas) and views of the chunk
};

struct ZMaps {
    CUtensorMap m[2];  // X with the box of each kind
};

struct XshiftArgs {
    petl_geom G;
    int step;  // view step of the members' view ranges
    int NXc;   // scratch row pitch (columns, a multiple of 4)
    Tables T;
    Members M;  // volumes (in) and views of the chunk
    ZKind k[2];
    int nv;     // slopes per group
    ZRec* rec;
    int* dz;
    int* next;
    int* err;
};

// Table records of plane y for every slope block of the call.
__device__ void z_records(const XshiftArgs& A, int y)
{
    const int NY = A.G.numY, nv = A.nv;
    const int nblk = A.k[0].nblk + A.k[1].nblk;
    for (int e = threadIdx.x; e < nblk * kZWarps; e += blockDim.x) {
        const int blk = e / kZWarps, q = e - blk * kZWarps;
        const ZKind& K = A.k[blk < A.k[0].nblk ? 0 : 1];
        const int v1a = K.v1_first + (blk - K.blk0) * nv * K.sg;
        const int v1b = min(v1a + nv * K.sg, K.v1_end);
        // the shifts are monotone in v1
        const int da = A.T.zt[size_t(v1a) * NY + y].d, db = A.T.zt[size_t(v1b - 1) * NY + y].d;
        const int dmin = min(da, db);
        ZRec* R = A.rec + size_t(blk) * NY + y;
        uint32_t code = 0;
        const int j0 = v1a + q * nv, j1 = min(j0 + nv, v1b);
        if (j0 < v1b) {
            int base = 1 << 30;
            for (int j = j0; j < j1; j++) base = min(base, A.T.zt[size_t(j) * NY + y].d);
            int xoff = base - dmin;
            bool bad = xoff < 0 || max(da, db) - dmin + K.rows + 1 > K.nrb;
            for (int j = j0; j < j1; j++) {
                const Shift zs = A.T.zt[size_t(j) * NY + y];
                if (zs.d - base > kZSpread) bad = true;
                // four slopes: neighbours a row apart at most, else no unrolled form has the pattern
                if (nv == 4 && j > j0 && abs(zs.d - A.T.zt[size_t(j - 1) * NY + y].d) > 1) bad = true;
                code |= uint32_t(min(zs.d - base, kZSpread)) << (2 * (j - j0));
                R->w[q * nv + j - j0] = zs.w;
            }
            if (bad) {  // a host-side bound does not hold: stay inside the staged rows
                atomicOr(A.err, kErrLayout);
                xoff = 0;
            }
            // slopes beyond the last one: a pattern of the present ones, no weight
            for (int j = j1; j < j0 + nv; j++) {
                code |= ((code >> (2 * (j1 - 1 - j0))) & 3u) << (2 * (j - j0));
                R->w[q * nv + j - j0] = 0.0f;
            }
            code |= uint32_t(xoff) << 8;
        }
        if (q < K.sg) R->code[q] = code;
        if (q == 0) A.dz[size_t(blk) * NY + y] = dmin;
    }
}

// X rows of a chunk of views.  A block stages rows z0..z0+7 of plane y of
// one member's volume in shared memory once and writes them shifted for
// every view of that member in the chunk, one float4 of columns per thread
// and step; columns whose rays are all masked are left out.  Bound by its
// writes of the scratch.  The first block of a plane also writes the plane's
// table records.  Grid (ceil(NZ / 8), NY, members).
template <class TF, int NM>
__global__ void __launch_bounds__(256) k_xshift(float* __restrict__ X, const XshiftArgs A)
{
    __shared__ float rowbuf[XZB * XMAXNX];
    const petl_geom& G = A.G;
    const int NY = G.numY, NX = G.numX, NZ = G.numZ;
    const int y = blockIdx.y, z0 = blockIdx.x * XZB;
    const int b = NM == 1 ? 0 : int(blockIdx.z);
    const int nz = min(XZB, NZ - z0);
    const TF* __restrict__ f = static_cast<const TF*>(member_pick<NM>(A.M.in, b));
    for (int e = threadIdx.x; e < nz * NX; e += blockDim.x) {
        const int r = e / NX, x = e - r * NX;
        rowbuf[r * NX + x] = Store<TF>::ld(f[(size_t(z0 + r) * NY + y) * NX + x]);
    }
    __syncthreads();
    const int first = member_pick<NM>(A.M.first, b), nvb = member_pick<NM>(A.M.nv, b);
    for (int iv = 0; iv < nvb; iv++) {
        const int v0 = first + iv * A.step;
        const Shift xs = A.T.xt[size_t(v0) * NY + y];
        const int2 ub0 = A.T.ub0[v0];
        const int c0 = ub0.x & ~3;
        const int nq = ub0.y < ub0.x ? 0 : ((ub0.y - c0) >> 2) + 1;  // float4 columns per row
        const float w1 = xs.w, w0 = 1.0f - xs.w;
        float* Xv = X + (size_t(b * A.M.nvm + iv) * NY + y) * NZ * A.NXc;
        for (int e = threadIdx.x; e < nz * nq; e += blockDim.x) {
            const int r = e / nq, c = c0 + (e - r * nq) * 4;
            const float* fr = rowbuf + r * NX;
            float v[5];
#pragma unroll
            for (int i = 0; i < 5; i++) {
                const int ix = c + xs.d + i;
                v[i] = unsigned(ix) < unsigned(NX) ? fr[ix] : 0.0f;
            }
            const float4 o = make_float4(fmaf(w1, v[1], w0 * v[0]), fmaf(w1, v[2], w0 * v[1]),
                                         fmaf(w1, v[3], w0 * v[2]), fmaf(w1, v[4], w0 * v[3]));
            // streaming store: the scratch is read once, by the next kernel
            __stcs(reinterpret_cast<float4*>(Xv + size_t(z0 + r) * A.NXc + c), o);
        }
    }
    if (blockIdx.x == 0 && b == 0) z_records(A, y);
    if (blockIdx.x == 0 && y == 0 && b == 0 && threadIdx.x == 0) *A.next = 0;
}

// The z taps: g[v1][v0][iu1][c] = S sum_y (1 - w) X[y][iu1 + d] + w X[y][iu1 + d + 1].
//
// Persistent CTAs of nw consumer warps and a producer warp.  A tile is one
// view x one slope block x rows x 64 columns, placed at the first visible row
// of the block and the first visible column of the view (masked rays are
// written as zeros by the tiles at the edge, not computed); a warp sums NV
// slopes x NK rows x 2 columns per lane over the planes.  The producer walks
// the tiles and stages their planes two or four at a time, rows by a tiled TMA copy
// (no multicast) and the planes' table records by a bulk copy, ahead of the
// consumers across tile borders, so set-up and epilogue of a warp overlap the
// sums of the others.
//
// Bound by the FMA pipe and what three warps per scheduler cannot hide: a plane
// costs a warp 96 packed FMAs (192 cycles of its scheduler, which holds three
// such warps) and 16 eight-byte window loads (32 cycles of the SM's shared
// memory, of which twelve warps take 384 of the 576 cycles the FMAs take).
// The FMA pipe is active on 44-48 % of cycles (256x256x128, 26 views): the
// dispatch, the window's first loads, the ring's waits and the masked parts of
// tiles are not covered.  4 slopes x 16 rows in eight warps need fewer loads
// per FMA but ran 9 % slower; 8 rows and 16 warps are bound by the loads.
// TG: planogram storage (float or bfloat16); X and the arithmetic are FP32.
template <class TG, int NM, int NV, int NK>
__global__ void __launch_bounds__(kZThreads, 1)
k_fwd_zsum(const __grid_constant__ ZMaps maps, const __grid_constant__ ZsumArgs A)
{
    extern __shared__ __align__(128) unsigned char smem[];
    ZCtl* ctl = reinterpret_cast<ZCtl*>(smem + size_t(A.ns) * A.stage);
    ZStage* s_info = ctl->info;
    uint64_t *full = ctl->full, *empty = ctl->empty;
    volatile int* s_abort = &ctl->abort;
    const petl_geom& G = A.G;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int NY = G.numY, NZ = G.numZ, NX = G.numX, ns = A.ns;
    if (tid == 0) {
        *s_abort = 0;
        for (int s = 0; s < ns; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], A.nw);
        }
        fence_barrier_init();
    }
    __syncthreads();

    if (warp >= A.nw) {
        producer_registers();
        if (warp > A.nw) {
            __syncthreads();
            return;
        }
        int j = 0;       // stages started
        bool dead = false;
        const int ntile = A.k[0].ntile + A.k[1].ntile;
        // waits until the slot of stage j is free (lane 0)
        auto claim = [&]() {
            const int slot = j % ns, round = j / ns;
            if (round > 0 && !ring_wait(&empty[slot], uint32_t((round - 1) & 1), A.err, s_abort, A.wait_limit))
                return false;
            return *s_abort == 0;
        };
        // The next tile is taken when this one is staged, not ahead of it: tiles
        // without visible rays cost nothing, and a CTA that held a tile in
        // reserve worked on two while others had none left (43 slopes, 29
        // views, 42 rows, 40 planes: busiest SM 170k cycles, 64k on average)
        auto next_tile = [&]() {
            int t = 0;
            if (lane == 0) t = int(gridDim.x) + atomicAdd(A.next, 1);
            return __shfl_sync(0xffffffffu, t, 0);
        };
        for (int tile = blockIdx.x; tile < ntile && !dead; tile = next_tile()) {
            const int kind = tile < A.k[0].ntile ? 0 : 1;
            const ZKind& K = A.k[kind];
            int t = tile - (kind ? A.k[0].ntile : 0);
            const int colblk = t % A.n_colblk;
            t /= A.n_colblk;
            const int rowblk = t % K.n_rowblk;
            t /= K.n_rowblk;
            const int blk = t % K.nblk, vi = t / K.nblk;  // slope block, view slot
            const int mb = NM == 1 ? 0 : vi / A.M.nvm, mv = vi - mb * A.M.nvm;
            if (mv >= member_pick<NM>(A.M.nv, mb)) continue;  // a member with fewer views than the slots
            const int iv0 = member_pick<NM>(A.M.first, mb) + mv * A.step;
            const int nsl = NV * K.sg, v1a = K.v1_first + blk * nsl, v1b = min(v1a + nsl, K.v1_end);
            // visible columns of the view and visible rows of the block
            const int2 ub0 = A.T.ub0[iv0];
            int lo = 1 << 30, hi = -1;
            if (v1a + lane < v1b) {
                const int2 u = A.T.ub1[v1a + lane];
                if (u.x <= u.y) lo = u.x, hi = u.y;
            }
            lo = __reduce_min_sync(0xffffffffu, lo);
            hi = __reduce_max_sync(0xffffffffu, hi);
            const bool vis = lo <= hi && ub0.x <= ub0.y;
            const int rlo = vis ? lo : 0, clo = vis ? ub0.x & ~3 : 0;
            const int nrow = vis ? (hi - rlo) / K.rows + 1 : 1, ncol = vis ? (ub0.y - clo) / kZCols + 1 : 1;
            if (rowblk >= nrow || colblk >= ncol) continue;
            const int row0 = rlo + rowblk * K.rows, col0 = clo + colblk * kZCols;
            // planes whose staged window meets the volume
            int ya = NY, ye = 0;
            const int* dz = A.dz + size_t(K.blk0 + blk) * NY;
            if (vis)
                for (int yb = 0; yb < NY; yb += 32) {
                    const int y = yb + lane;
                    if (y < NY) {
                        const int cx = col0 + A.T.xt[size_t(iv0) * NY + y].d, wlo = row0 + dz[y];
                        if (cx + kZCols >= 0 && cx < NX && wlo + K.nrb > 0 && wlo < NZ) {
                            ya = min(ya, y);
                            ye = y + 1;
                        }
                    }
                }
            ya = __reduce_min_sync(0xffffffffu, ya);
            ye = __reduce_max_sync(0xffffffffu, ye);
            const int edge = (kind ? kZTail : 0) | (rowblk == 0 ? kZRow0 : 0) | (rowblk == nrow - 1 ? kZRowN : 0) |
                             (colblk == 0 ? kZCol0 : 0) | (colblk == ncol - 1 ? kZColN : 0);
            const int nst = max(1, (ye - ya + K.pps - 1) / K.pps);  // a tile without planes still writes its zeros
            if (lane == 0) {
                const uint32_t box = uint32_t(K.nrb) * kZCols * 4u;
                for (int i = 0; i < nst; i++) {
                    if (!claim()) {
                        dead = true;
                        break;
                    }
                    const int slot = j % ns, y = ya + K.pps * i, np = max(0, min(K.pps, ye - y));
                    unsigned char* st = smem + size_t(slot) * A.stage;
                    s_info[slot] =
                        ZStage{y, np | edge | (i == nst - 1 ? kZLast : 0), v1a, vi, row0, col0, 0.0f, 0.0f};
                    fence_proxy_async_smem();
                    mbar_arrive_expect_tx(&full[slot], uint32_t(np) * (box + uint32_t(sizeof(ZRec))));
                    for (int h = 0; h < np; h++)
                        tma_load_4d(st + size_t(h) * K.pstride * 4, &maps.m[kind], &full[slot], col0, row0 + dz[y + h],
                                    y + h, vi);
                    if (np)
                        bulk_load(st + A.rec_off, A.rec + size_t(K.blk0 + blk) * NY + y,
                                  uint32_t(np) * uint32_t(sizeof(ZRec)), &full[slot]);
                    j++;
                }
            }
            dead = __shfl_sync(0xffffffffu, int(dead), 0) != 0;
        }
        if (lane == 0) {
            if (!dead && claim()) {
                const int slot = j % ns;
                s_info[slot].flags = kZEnd;
                mbar_arrive(&full[slot]);
                j++;
            } else {
                *s_abort = 1;
            }
        }
        __syncthreads();
        // a wait gave up: drain the copies still in flight
        if (lane == 0 && *s_abort)
            for (int i = max(0, j - ns); i < j; i++) mbar_wait(&full[i % ns], uint32_t((i / ns) & 1), nullptr);
        return;
    }

    {
        consumer_registers();
        int slot = 0;
        uint32_t phase = 0;
        auto wait = [&]() {
            return __all_sync(0xffffffffu, ring_wait(&full[slot], phase, A.err, s_abort, A.wait_limit)) != 0;
        };
        bool dead = !wait();
        while (!dead) {  // tiles
            const ZStage in = s_info[slot];
            if (in.flags & kZEnd) break;
            const ZKind& K = A.k[in.flags & kZTail ? 1 : 0];
            const int gv = warp % K.sg, gr = warp / K.sg, row0 = in.row0 + gr * NK;
            bool have = false;  // some slope of this warp has visible rows in the tile
            if (gr < K.rg)
                for (int v1 = in.a + gv * NV; v1 < min(in.a + (gv + 1) * NV, K.v1_end); v1++) {
                    const int2 u = A.T.ub1[v1];
                    have |= row0 <= u.y && row0 + NK - 1 >= u.x;
                }
            f2x acc[NV][NK];
#pragma unroll
            for (int j = 0; j < NV; j++)
#pragma unroll
                for (int k = 0; k < NK; k++) acc[j][k] = 0ull;
            const int pbytes = K.pstride * 4;
            for (;;) {  // stages
                const int flags = s_info[slot].flags;
                if (have) {
                    const unsigned char* st = smem + size_t(slot) * A.stage;
                    const ZRec* rec = reinterpret_cast<const ZRec*>(st + A.rec_off);
                    const f2x* W;
                    f2x wa[NV], wb[NV];
                    uint32_t code;
                    int left = flags & kZCount;  // planes of the stage still to sum
                    auto load = [&]() {
                        code = rec->code[gv];
                        W = reinterpret_cast<const f2x*>(st) + (int((code >> 8) & 0xffu) + gr * NK) * (kZCols / 2) + lane;
#pragma unroll
                        for (int j = 0; j < NV; j++) {
                            const float w = rec->w[gv * NV + j];
                            wa[j] = f2_dup(1.0f - w);
                            wb[j] = f2_dup(w);
                        }
                    };
                    // on to the next plane; whether it has the same pattern
                    auto next = [&](uint32_t pattern) {
                        rec++;
                        st += pbytes;
                        if (--left <= 0) return false;
                        load();
                        return (code & 0xffu) == pattern;
                    };
                    if (left > 0) load();
                    // the offsets of consecutive slopes are monotone and (four
                    // slopes) at most one row apart: one dispatch over the
                    // patterns that occur for each run of planes with the same
                    // one (forward at 256x256x128 8.4 ms with a jump per plane, 7.8 so)
                    while (left > 0) {
#define PETL_ZCASE(PC)                        \
    case PC:                                  \
        do                                    \
            z_taps<PC, true>(acc, W, wa, wb); \
        while (next(PC));                     \
        break;
                        if constexpr (NV == 4) {
                            switch (code & 0xffu) {
                                PETL_ZCASE(0x00) PETL_ZCASE(0x40) PETL_ZCASE(0x50) PETL_ZCASE(0x90) PETL_ZCASE(0x54)
                                PETL_ZCASE(0x94) PETL_ZCASE(0xA4) PETL_ZCASE(0xE4) PETL_ZCASE(0x01) PETL_ZCASE(0x05)
                                PETL_ZCASE(0x15) PETL_ZCASE(0x06) PETL_ZCASE(0x16) PETL_ZCASE(0x1A) PETL_ZCASE(0x1B)
                                default: next(0x100u);  // no such pattern: z_records reported a layout error
                            }
                        } else {
                            switch (code & 0xffu) {
                                PETL_ZCASE(0x0) PETL_ZCASE(0x4) PETL_ZCASE(0x8) PETL_ZCASE(0xC) PETL_ZCASE(0x1)
                                PETL_ZCASE(0x2) PETL_ZCASE(0x3)
                                default: next(0x100u);
                            }
                        }
#undef PETL_ZCASE
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&empty[slot]);
                if (++slot == ns) {
                    slot = 0;
                    phase ^= 1u;
                }
                if (flags & kZLast) break;
                if (!wait()) {
                    dead = true;
                    break;
                }
            }
            if (dead) break;
            if (gr < K.rg) {
            // epilogue: scale, ray masks, optional MLEM ratio; zeros for the
            // masked rays beyond the tiles
            const int mb = NM == 1 ? 0 : in.b / A.M.nvm, mv = in.b - mb * A.M.nvm;
            const int iv0 = member_pick<NM>(A.M.first, mb) + mv * A.step;
            TG* __restrict__ g = static_cast<TG*>(member_pick<NM>(A.M.out, mb));
            const TG* __restrict__ meas = static_cast<const TG*>(member_pick<NM>(A.M.meas, mb));
            const int2 ub0 = A.T.ub0[iv0];
            const int colA = in.col0 + 2 * lane;
            const int row1 = min(row0 + NK, G.N_u1);
            const bool ok0 = colA >= ub0.x && colA <= ub0.y, ok1 = colA + 1 >= ub0.x && colA + 1 <= ub0.y;
            f2x* out = ctl->out[warp][0] + lane;
#pragma unroll 1
            for (int i = 0; i < NV * NK / kZOut; i++) {
                out_rows(acc, out, i);
                const int v1 = in.a + gv * NV + i / (NK / kZOut), r0 = row0 + i % (NK / kZOut) * kZOut;
                if (v1 >= min(in.a + NV * K.sg, K.v1_end)) break;
                const float S = A.T.S[size_t(v1) * G.N_v0 + iv0];
                const int2 u1r = A.T.ub1[v1];
                const size_t o0 = (size_t(v1) * G.N_v0 + iv0) * G.N_u1 * G.N_u0;
#pragma unroll 1
                for (int kk = 0; kk < kZOut; kk += 4) {
                    if (A.pairs && colA + 1 < G.N_u0) {
                        float2 m[4];
                        if (meas)
#pragma unroll
                            for (int k = 0; k < 4; k++)
                                if (r0 + kk + k < G.N_u1)
                                    m[k] = Store<TG>::ld2(meas + o0 + size_t(r0 + kk + k) * G.N_u0 + colA);
#pragma unroll
                        for (int k = 0; k < 4; k++) {
                            const int iu1 = r0 + kk + k;
                            if (iu1 >= G.N_u1) break;
                            const bool rv = iu1 >= u1r.x && iu1 <= u1r.y;
                            const float2 a = f2_unpack(out[(kk + k) * 32]);
                            float2 val = make_float2(rv && ok0 ? a.x * S : 0.0f, rv && ok1 ? a.y * S : 0.0f);
                            if (meas) val = make_float2(ratio_rule(m[k].x, val.x), ratio_rule(m[k].y, val.y));
                            Store<TG>::st2(g + o0 + size_t(iu1) * G.N_u0 + colA, val);
                        }
                    } else {  // no pairs, or the row's last column
#pragma unroll 1
                        for (int k = kk; k < min(kk + 4, G.N_u1 - r0); k++) {
                            const bool rv = r0 + k >= u1r.x && r0 + k <= u1r.y;
                            const size_t o = o0 + size_t(r0 + k) * G.N_u0 + colA;
                            const float2 a = f2_unpack(out[k * 32]);
                            const float2 val = make_float2(rv && ok0 ? a.x * S : 0.0f, rv && ok1 ? a.y * S : 0.0f);
                            if (colA < G.N_u0) g[o] = Store<TG>::st(meas ? ratio_rule(Store<TG>::ld(meas[o]), val.x) : val.x);
                            if (colA + 1 < G.N_u0)
                                g[o + 1] = Store<TG>::st(meas ? ratio_rule(Store<TG>::ld(meas[o + 1]), val.y) : val.y);
                        }
                    }
                }
            }
            // masked rays around the tiles
            const int cz0 = in.flags & kZCol0 ? 0 : in.col0;
            const int cz1 = in.flags & kZColN ? G.N_u0 : min(in.col0 + kZCols, G.N_u0);
            const int rz0 = (in.flags & kZRow0) && gr == 0 ? 0 : row0;
            const int rz1 = (in.flags & kZRowN) && gr == K.rg - 1 ? G.N_u1 : row1;
            if (cz0 < in.col0 || cz1 > in.col0 + kZCols || rz0 < row0 || rz1 > row1)
#pragma unroll 1
                for (int v1 = in.a + gv * NV; v1 < min(in.a + (gv + 1) * NV, K.v1_end); v1++)
#pragma unroll 1
                    for (int r = rz0; r < rz1; r++) {
                        TG* row = g + ((size_t(v1) * G.N_v0 + iv0) * G.N_u1 + r) * G.N_u0;
                        const bool inside = r >= row0 && r < row1;
#pragma unroll 1
                        for (int c = cz0 + lane; c < cz1; c += 32)
                            if (!inside || c < in.col0 || c >= in.col0 + kZCols) row[c] = Store<TG>::st(0.0f);
                    }
            }
            dead = !wait();
        }
        if (dead) *s_abort = 1;
    }
    __syncthreads();
}

// Launch shape of the z kernel for a call: false when a layout rule fails.
struct ZPlan {
    ZsumArgs A;
    int nv, nk;        // slopes and rows per warp
    int ctas;          // CTAs per SM
    size_t smem;
    size_t table_bytes;
};

bool zsum_plan(const petl_geom& G, const ViewRange& vr, const ShiftStep& step, int nslot, ZPlan& P)
{
    ZsumArgs& A = P.A;
    A = ZsumArgs{};
    A.G = G;
    A.step = vr.iv0_step;
    A.nslot = nslot;
    A.n_colblk = int(ceil_div(G.N_u0, kZCols));
    A.wait_limit = wait_limit();
    // four slopes share a window of 16 rows where their shifts move by less
    // than a row per slope; steeper slopes (a volume
    // that reaches beyond the panels) take two per warp and a window of 28
    // rows, whose loads then bound them; steps of three rows and more are left
    // to the first-generation kernel.  192x192x96 at 1.1 to 1.4 rows per
    // slope: 3.3 ms for 67 views here, 6.0 on the first-generation kernel
    P.nv = four_per_window(step) ? 4 : 2;
    P.nk = P.nv == 4 ? 12 : 24;
    if (shift_spread(P.nv - 1, step) > kZSpread) return false;
    const int nv1 = vr.iv1_end - vr.iv1_begin;
    const int ngrp = int(ceil_div(nv1, P.nv));
    // twelve consumer warps, or four where these have few tiles (ztwelve)
    int tiles = 0;
    for (A.nw = kZWarps;; A.nw = 4) {
        const int sg = P.nv == 4 || A.nw == 4 ? 4 : 6;
        // full blocks of sg slope groups; a tail of at most half a block
        // takes fewer slope groups over more rows instead of idle warps
        const int ntail = ngrp % sg;
        const int tail_sg = ntail == 0 ? 0 : ntail == 1 ? 1 : 2 * ntail <= sg ? sg / 2 : 0;
        const int v1_split = tail_sg ? vr.iv1_begin + (ngrp - ntail) * P.nv : vr.iv1_end;
        tiles = 0;
        for (int i = 0; i < 2; i++) {
            ZKind& K = A.k[i];
            K.v1_first = i ? v1_split : vr.iv1_begin;
            K.v1_end = i ? vr.iv1_end : v1_split;
            K.sg = i ? std::max(tail_sg, 1) : sg;
            K.nblk = int(ceil_div(K.v1_end - K.v1_first, P.nv * K.sg));
            // staged rows: the tile's, the spread of the block's shifts and
            // the second tap's.  They fit a TMA box and, with the window's
            // margin, the 8 bits of a window row: a tail of one group of two
            // slopes on a tall panel takes fewer warps (192x192x128, 256 rows,
            // 79 views, 1.2 rows per slope: 72 slopes 5.9 ms and 74 slopes 6.4
            // here, 18.8 and 19.0 on the first-generation kernel)
            const int extra = shift_spread(P.nv * K.sg - 1, step) + 1;
            K.rg = std::min(A.nw / K.sg, int(ceil_div(G.N_u1, P.nk)));
            K.rg = std::min(K.rg, (256 - kZSpread - extra) / P.nk);
            if (K.rg < 1 && K.nblk == 0) K.rg = 1;  // no such blocks
            if (K.rg < 1) return false;
            K.rows = P.nk * K.rg;
            K.n_rowblk = int(ceil_div(G.N_u1, K.rows));
            K.nrb = K.rows + extra;
            K.pstride = (K.nrb + kZSpread) * kZCols;
            K.blk0 = i ? A.k[0].nblk : 0;
            const long long nt = (long long)nslot * K.nblk * K.n_rowblk * A.n_colblk;
            if (nt > (1 << 30)) return false;
            K.ntile = int(nt);
            tiles += K.ntile;
        }
        if (A.nw == 4 || ztwelve(tiles)) break;
    }
    // four planes per stage (longer runs of one pattern, fewer waits) where
    // three stages fit, else two; the tail's tall planes one or two at a time.
    // A ring that does not fit half an SM takes the whole
    for (P.ctas = zctas(A.nw, tiles);; P.ctas = 1) {
        for (int pps = 4;; pps = 2) {
            A.k[0].pps = pps;
            A.k[1].pps = std::max(1, std::min(pps, A.k[0].nblk ? pps * A.k[0].pstride / A.k[1].pstride : 2));
            A.rec_off = 0;
            for (const ZKind& K : A.k)
                if (K.nblk > 0) A.rec_off = std::max(A.rec_off, K.pstride * K.pps * 4);
            A.stage = (A.rec_off + pps * int(sizeof(ZRec)) + 127) & ~127;
            A.ns = std::min(kZStages, (zsmem(P.ctas) - zctl_bytes(A.nw)) / A.stage);
            if (A.ns >= 3 || pps == 2) break;
        }
        if (A.ns >= 2 || P.ctas == 1) break;
    }
    if (A.ns < 2) return false;
    P.smem = size_t(A.ns) * A.stage + zctl_bytes(A.nw);
    const size_t nrec = size_t(A.k[0].nblk + A.k[1].nblk) * G.numY;
    P.table_bytes = nrec * (sizeof(ZRec) + sizeof(int)) + sizeof(int);
    return true;
}

}  // namespace

// Scratch budget of the x-shift pass (bytes of FP32 X per chunk of views);
// PETL_SPLIT_SCRATCH_MB overrides it.
size_t split_scratch_budget()
{
    static const long long env_mb = [] {
        const char* e = std::getenv("PETL_SPLIT_SCRATCH_MB");
        return e ? std::atoll(e) : 0LL;
    }();
    if (env_mb > 0) return size_t(env_mb) << 20;
    // the device's memory size, looked up once per device (a query per call
    // would cost host time on the launch path)
    static std::mutex mu;
    static size_t total[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
        cudaGetLastError();
        return size_t(1) << 30;
    }
    std::lock_guard<std::mutex> lk(mu);
    if (!total[dev]) {
        cudaDeviceProp prop;
        if (cudaGetDeviceProperties(&prop, dev) != cudaSuccess) {
            cudaGetLastError();
            return size_t(1) << 30;
        }
        total[dev] = prop.totalGlobalMem;
    }
    return std::min(size_t(5) << 30, total[dev] / 8);
}

// Forward projection of the members' views.  One member: its views in
// chunks of at most the scratch budget (and chunk_cap); several: one chunk,
// else kNotApplicable.
template <class TF, class TG>
int project_split_m(const petl_geom& G, const Members& M0, const ViewRange& vr, const Tables& T, cudaStream_t st,
                    int chunk_cap, const ChunkHook* hook)
{
    const int nb = M0.nb;
    if (nb < 1 || nb > kMaxMembers) return kNotApplicable;
    int nvmax = 0;
    for (int b = 0; b < nb; b++) nvmax = std::max(nvmax, M0.nv[b]);
    const int nv1 = vr.iv1_end - vr.iv1_begin;
    if (nvmax <= 0 || nv1 <= 0) return 0;
    // the x pass writes a volume per view whatever the slope count: below
    // about ten slopes the single-pass kernel is cheaper than that round trip
    if (nv1 < kSplitMinSlopes) return kNotApplicable;
    const ShiftStep step = slope_step(G);
    int* err = device_error_ptr();
    if (!err) return kNotApplicable;

    // chunks of views whose X fits the scratch budget, balanced in size
    const int NXc = (G.N_u0 + 3) & ~3;
    const size_t per_view = size_t(G.numY) * G.numZ * NXc * 4;
    if (G.numX > XMAXNX || G.numY > 65535) return kNotApplicable;  // k_xshift row buffer, grid.y
    const size_t fit = std::max<size_t>(1, split_scratch_budget() / per_view);
    int nv, nchunks;
    if (nb == 1) {
        nv = int(std::min<size_t>(size_t(nvmax), fit));
        if (chunk_cap > 0) nv = std::min(nv, chunk_cap);
        nchunks = (nvmax + nv - 1) / nv;
        nv = (nvmax + nchunks - 1) / nchunks;
    } else {
        if (size_t(nb) * nvmax > fit || chunk_cap > 0) return kNotApplicable;
        nv = nvmax;
        nchunks = 1;
    }
    ZPlan P;
    if (!zsum_plan(G, vr, step, nv * nb, P)) return kNotApplicable;

    // X, then the table records and the blocks' smallest shifts
    float* X = nullptr;
    const size_t x_bytes = per_view * nv * nb;  // a multiple of 16
    if (scratch_alloc(reinterpret_cast<void**>(&X), x_bytes + P.table_bytes, st) != cudaSuccess) {
        cudaGetLastError();  // out of memory is not sticky: the caller takes the fused kernel
        return kNotApplicable;
    }
    ZsumArgs& A = P.A;
    A.T = T;
    A.err = err;
    A.pairs = 1;
    for (int b = 0; b < nb; b++)
        if (!pair_access<TG>(G, M0.out[b], M0.meas[b])) A.pairs = 0;
    A.rec = reinterpret_cast<ZRec*>(reinterpret_cast<unsigned char*>(X) + x_bytes);
    A.dz = reinterpret_cast<int*>(A.rec + size_t(A.k[0].nblk + A.k[1].nblk) * G.numY);
    A.next = A.dz + size_t(A.k[0].nblk + A.k[1].nblk) * G.numY;
    ZMaps maps;
    std::memset(&maps, 0, sizeof(maps));
    const uint64_t dims[4] = {uint64_t(NXc), uint64_t(G.numZ), uint64_t(G.numY), uint64_t(nv * nb)};
    const uint64_t strides[3] = {uint64_t(NXc) * 4, uint64_t(NXc) * G.numZ * 4, uint64_t(NXc) * G.numZ * G.numY * 4};
    bool ok = true;
    for (int i = 0; i < 2 && ok; i++) {
        if (A.k[i].nblk == 0) continue;
        const uint32_t box[4] = {uint32_t(kZCols), uint32_t(A.k[i].nrb), 1u, 1u};
        ok = encode_tensor_map(&maps.m[i], X, 4, dims, strides, box, 4);
    }
    if (!ok) {
        cudaFreeAsync(X, st);
        return kNotApplicable;
    }
    // kernels compiled for one member where there is one
    auto kz = nb == 1 ? (P.nv == 4 ? k_fwd_zsum<TG, 1, 4, 12> : k_fwd_zsum<TG, 1, 2, 24>)
                      : (P.nv == 4 ? k_fwd_zsum<TG, kMaxMembers, 4, 12> : k_fwd_zsum<TG, kMaxMembers, 2, 24>);
    auto kx = nb == 1 ? k_xshift<TF, 1> : k_xshift<TF, kMaxMembers>;
    cudaError_t e = cudaFuncSetAttribute(kz, cudaFuncAttributeMaxDynamicSharedMemorySize, int(P.smem));
    for (int c = 0; c < nchunks && e == cudaSuccess; c++) {
        Members M = M0;
        const int vi0 = c * nv;
        int nvc = nv;
        if (nb == 1) {
            nvc = std::min(nv, nvmax - vi0);
            M.first[0] = M0.first[0] + vi0 * vr.iv0_step;
            M.nv[0] = nvc;
        }
        M.nvm = nvc;
        XshiftArgs XA{G, vr.iv0_step, NXc, T, M, {A.k[0], A.k[1]}, P.nv, A.rec, A.dz, A.next, err};
        kx<<<dim3(ceil_div(G.numZ, XZB), unsigned(G.numY), unsigned(nb)), 256, 0, st>>>(X, XA);
        note_launch();
        A.M = M;
        A.nslot = nvc * nb;
        int tiles = 0;
        for (ZKind& K : A.k) tiles += K.ntile = A.nslot * K.nblk * K.n_rowblk * A.n_colblk;
        kz<<<std::min(tiles, P.ctas * sm_count()), 32 * (A.nw + 4), P.smem, st>>>(maps, A);
        note_launch();
        e = cudaGetLastError();
        if (e == cudaSuccess && hook && hook->fn) hook->fn(hook->ctx, vi0, nvc);
    }
    cudaFreeAsync(X, st);
    if (e != cudaSuccess) {
        set_error(std::string("project_split: ") + cudaGetErrorString(e));
        return int(e);
    }
    return 0;
}

template <class TF, class TG>
int project_split_t(const petl_geom& G, const TF* f, TG* g, const ViewRange& vr, const TG* meas, const Tables& T,
                    cudaStream_t st, int chunk_cap, const ChunkHook* hook)
{
    Members M;
    M.nb = 1;
    M.first[0] = vr.iv0_first;
    M.nv[0] = vr.n_v0(G.N_v0);
    M.in[0] = f;
    M.out[0] = g;
    M.meas[0] = meas;
    if (M.nv[0] <= 0 || vr.iv1_end <= vr.iv1_begin) return 0;
    return project_split_m<TF, TG>(G, M, vr, T, st, chunk_cap, hook);
}

int project_split(const petl_geom& G, const float* f, float* g, const ViewRange& vr, const float* meas,
                  const Tables& T, cudaStream_t st, int chunk_cap, const ChunkHook* hook)
{
    return project_split_t<float, float>(G, f, g, vr, meas, T, st, chunk_cap, hook);
}

int project_split_bf16(const petl_geom& G, const __nv_bfloat16* f, __nv_bfloat16* g, const ViewRange& vr,
                       const __nv_bfloat16* meas, const Tables& T, cudaStream_t st)
{
    return project_split_t<__nv_bfloat16, __nv_bfloat16>(G, f, g, vr, meas, T, st, 0, nullptr);
}

int project_split_members(const petl_geom& G, const Members& M, const ViewRange& vr, const Tables& T,
                          cudaStream_t st)
{
    return project_split_m<float, float>(G, M, vr, T, st, 0, nullptr);
}

}  // namespace shear
}  // namespace petl
