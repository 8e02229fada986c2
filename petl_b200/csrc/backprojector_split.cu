// Split backprojector (psi = 0, voxel pitch equal to the bin pitch): the
// transpose of the split forward (projector_split.cu), in the gather form of
// k_bwd_tma (projector_shear_tma.cu) for the reference semantics of
// src/projectors.cu:240-377 and for the exact adjoint.
//
// The voxel (x, y, z) receives, from view v0 and slope v1 on plane y,
//   S (1 - wz) g[v1][v0][z - dz][x - dx] + S wz g[v1][v0][z - dz - 1][x - dx]
// interpolated in x by (1 - wx, wx) over columns x - dx and x - dx - 1.  The
// two interpolations are separate kernels:
//
// * k_bwd_zgather sums the z taps over the slopes of one view into FP32
//   scratch B[view][y][z][c] (c = planogram column): persistent CTAs of twelve
//   consumer warps and a producer warp that stages the slopes' planogram rows
//   into a ring with full/empty mbarriers, by tiled TMA copies (no multicast)
//   or, where rows are no multiple of 16 bytes, by copies of column pairs;
//   k_gather_records tabulates window offsets, masks and weights once per call.
// * k_bwd_xgather applies the x taps and sums the views of a chunk into the
//   volume (or an FP32 partial sum between chunks).
//
// Both do the float operations of k_bwd_tma in the same order (per voxel:
// z taps over the live slopes in ascending v1, tap 0 then tap 1; x taps over
// the views in order; the scale last), so the two paths agree bit for bit.
// As in the forward, a launch serves one call or up to kMaxMembers requests
// of one geometry (one tensor map per member's planogram).  A single slope
// at v1 = 0 (the rebinned planogram of FBP) takes k_bwd_zflat: its z sums
// do not depend on the plane.
//
// 256x256x128, planogram (65, 129, 128, 256): 8.82 ms, of which 7.8 the z taps
// (before: 13.4 and 12.5, with one 16-warp CTA per tile, tables built by every
// CTA and scalar FMAs).  FBP's single slope: 0.46 ms (0.73 with a thread per x).
// Every wait is bounded: a wait that gives up sets the device error word, the
// CTA drains its copies in flight and returns without writing.
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <string>
#include <type_traits>

#include "common.cuh"
#include "projector.cuh"
#include "shear.cuh"
#include "storage.cuh"
#include "tma.cuh"
#include "ztaps.cuh"

namespace petl {
namespace shear {

namespace {

constexpr int GPLMAX = 16;          // planes per block at most (a table record holds 16 weights)
constexpr int GV1MAX = 128;         // slopes per call at most

// Table record of one (plane block, row block, slope), staged with the slope:
// the second tap's weight of each plane; per warp a code word (window offsets,
// 2 bits per plane; kind << 8: 0 no rows, 1 every row, 2 edge of the visible
// range; the window's first staged row << 16) and a mask for the edge: the
// output rows of each plane that receive the slope (64 / NV bits per plane;
// reference semantics) or the window rows that hold visible bins (adjoint).
struct __align__(16) GRec {
    float w[GPLMAX];
    uint32_t code[kZWarps];
    unsigned long long mask[kZWarps];
};

struct ZgatherArgs {
    petl_geom G;
    ViewRange vr;   // slopes and view step (the members hold their views)
    int nw;         // consumer warps
    int pg, rg;     // plane groups x row groups of a CTA (pg * rg = nw)
    int planes, rows;  // planes and rows per tile
    int nslot;      // view slots of all members
    int n_plblk, n_rowblk, n_colblk;
    int nrb;        // staged planogram rows per slope (rows + 1 + shift spread of the planes)
    int ns;         // ring stages, two slopes each
    int sbytes;     // bytes per staged slope (nrb + kZSpread rows of 64, a multiple of 128)
    int stage;      // bytes per stage (slopes, then two records)
    int NUc;        // scratch row pitch (columns)
    int nv1;        // slopes of the call
    int ntile;
    GRec* rec;      // [plane block][row block][nv1], the slopes that reach the tile first
    int2* list;     // same layout: (v1, first staged row)
    int* cnt;       // [plane block][row block] slopes that reach the tile
    int* next;      // tiles handed out beyond one per CTA, per chunk
    int nchunks;
    Tables T;
    int* err;
    unsigned wait_limit;  // bound of the waits on staged data (wait_limit(): kWaitLimit or 0)
    Members M;            // planograms (in) and views of the chunk
};

// tensor maps of the members' planograms
template <int NM>
struct GMaps {
    CUtensorMap m[NM];
};

// The slopes that reach each tile of planes and rows, compacted in order, and
// their records.  Grid (plane blocks, row blocks), 256 threads.
template <bool ADJ>
__global__ void __launch_bounds__(256) k_gather_records(const ZgatherArgs A, int NV, int NK)
{
    const petl_geom& G = A.G;
    const int NY = G.numY, NU1 = G.N_u1;
    const int p0 = blockIdx.x * A.planes, r0 = blockIdx.y * A.rows;
    const size_t base = (size_t(blockIdx.x) * gridDim.y + blockIdx.y) * A.nv1;
    __shared__ int s_n;
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        int n = 0;
        for (int vb = A.vr.iv1_begin; vb < A.vr.iv1_end; vb += 32) {
            const int v1 = vb + lane;
            bool ok = false;
            int grow = 0;
            if (v1 < A.vr.iv1_end) {
                int dmin = 1 << 30, dmax = -(1 << 30);
                const int2 ub1 = A.T.ub1[v1];
                for (int p = 0; p < A.planes && p0 + p < NY; p++) {
                    const int d = A.T.zt[size_t(v1) * NY + p0 + p].d;
                    dmin = min(dmin, d);
                    dmax = max(dmax, d);
                    // planogram rows that the tile touches on plane p
                    const int lo = r0 - d - 1, hi = r0 + A.rows - 1 - d;
                    if (hi < 0 || lo >= NU1) continue;
                    if (ADJ) {
                        ok |= !(hi < ub1.x || lo > ub1.y);
                    } else {
                        const int2 zv = A.T.zvis[size_t(v1) * NY + p0 + p];
                        ok |= !(r0 + A.rows - 1 < zv.x || r0 > zv.y);
                    }
                }
                grow = r0 - dmax - 1;
                if (ok && dmax - dmin + A.rows + 1 > A.nrb) {  // a host-side bound does not hold
                    atomicOr(A.err, kErrLayout);
                    ok = false;
                }
            }
            const unsigned bal = __ballot_sync(0xffffffffu, ok);
            if (ok) A.list[base + n + __popc(bal & ((1u << lane) - 1u))] = make_int2(v1, grow);
            n += __popc(bal);
        }
        if (lane == 0) {
            s_n = n;
            A.cnt[blockIdx.x * gridDim.y + blockIdx.y] = n;
        }
    }
    __syncthreads();
    if (blockIdx.x == 0 && blockIdx.y == 0)
        for (int i = threadIdx.x; i < A.nchunks; i += blockDim.x) A.next[i] = 0;
    const int nlive = s_n;
    for (int e = threadIdx.x; e < nlive * kZWarps; e += blockDim.x) {
        const int li = e / kZWarps, w = e - li * kZWarps;
        if (w >= A.pg * A.rg) continue;
        const int2 sl = A.list[base + li];
        const int v1 = sl.x, grow = sl.y;
        GRec* R = A.rec + base + li;
        const int q = w % A.pg, zr = r0 + (w / A.pg) * NK;  // first row of the warp
        const int2 ub1 = A.T.ub1[v1];
        int dmx = -(1 << 30);
        for (int u = 0; u < NV; u++) dmx = max(dmx, A.T.zt[size_t(v1) * NY + min(p0 + q * NV + u, NY - 1)].d);
        uint32_t offs = 0;
        unsigned long long rows = 0;
        int full = 0, some = 0;
        bool bad = false;
        for (int u = 0; u < NV; u++) {
            const int yq = p0 + q * NV + u, y = min(yq, NY - 1);
            const Shift zs = A.T.zt[size_t(v1) * NY + y];
            const int o = dmx - zs.d;
            bad |= o > kZSpread;
            // four planes: neighbours a row apart at most, else no unrolled form has the pattern
            if (NV == 4 && u > 0) bad |= abs(zs.d - A.T.zt[size_t(v1) * NY + min(yq - 1, NY - 1)].d) > 1;
            offs |= uint32_t(min(o, kZSpread)) << (2 * u);
            if (w < A.pg) R->w[q * NV + u] = zs.w;
            if (yq >= NY) continue;
            const int lo = zr - zs.d - 1, hi = zr + NK - 1 - zs.d;  // planogram rows touched
            if (hi < 0 || lo >= NU1) continue;
            if (ADJ) {
                if (hi < ub1.x || lo > ub1.y) continue;
                some++;
                full += lo >= ub1.x && hi <= ub1.y;
            } else {
                const int2 zv = A.T.zvis[size_t(v1) * NY + y];
                const int ka = max(zv.x - zr, 0), kb = min(zv.y - zr, NK - 1);
                if (kb < ka) continue;
                some++;
                full += ka == 0 && kb == NK - 1;
                const unsigned long long bits = ((~0ull >> (63 - kb)) >> ka) << ka;
                rows |= bits << (64 / NV * u);
            }
        }
        const int wfirst = zr - dmx - 1, wrow = wfirst - grow;  // planogram row and staged row of window row 0
        if (ADJ)
            for (int i = 0; i < NK + kZSpread + 1; i++)
                if (wfirst + i >= ub1.x && wfirst + i <= ub1.y) rows |= 1ull << i;
        bad |= wrow < 0 || wrow + NK + 1 > A.nrb;
        if (bad) atomicOr(A.err, kErrLayout);
        R->code[w] = bad || !some ? 0u : offs | uint32_t(full == NV ? 1 : 2) << 8 | uint32_t(wrow) << 16;
        R->mask[w] = rows;
    }
}

// The z taps of the transpose: B[view][y][z][c] = sum over the slopes of
// S (1 - w) g[v1][v0][z - d][c] + S w g[v1][v0][z - d - 1][c].
//
// Persistent CTAs as in k_fwd_zsum, with planes and slopes exchanged: a tile
// is one view x a block of planes x rows x 64 columns (from the first column
// that a voxel of those planes reads), a warp sums NV planes x NK rows x 2
// columns per lane over the slopes that reach the tile, and the producer
// stages the planogram rows of two slopes at a time with their table records.
// Bound as k_fwd_zsum (FMA pipe active on 44 % of cycles, issue slots on 58 %).
// At the edges of the visible range the taps are predicated per output row
// (reference semantics) or take zeros for masked window rows (adjoint), a
// plane at a time.
//
// TG: planogram storage (float or bfloat16); B and the arithmetic are FP32.
// BULK: planogram rows are multiples of 16 bytes and arrive by a tiled TMA copy
// (no multicast); else the producer's lanes copy a column pair each.
template <bool ADJ, class TG, int NM, bool BULK, int NV, int NK>
__global__ void __launch_bounds__(kZThreads, 1)
k_bwd_zgather(const __grid_constant__ GMaps<NM> gmaps, float* __restrict__ B, const __grid_constant__ ZgatherArgs A)
{
    extern __shared__ __align__(128) unsigned char smem[];
    ZCtl* ctl = reinterpret_cast<ZCtl*>(smem + size_t(A.ns) * A.stage);
    ZStage* s_info = ctl->info;
    uint64_t *full = ctl->full, *empty = ctl->empty;
    volatile int* s_abort = &ctl->abort;
    const petl_geom& G = A.G;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int NY = G.numY, NZ = G.numZ, NX = G.numX, ns = A.ns;
    constexpr int EB = int(sizeof(TG));
    if (tid == 0) {
        *s_abort = 0;
        for (int s = 0; s < ns; s++) {
            mbar_init(&full[s], BULK ? 1 : 1 + 128);  // or the stage's words, and each lane's copies
            mbar_init(&empty[s], A.nw);
        }
        fence_barrier_init();
    }
    __syncthreads();

    if (warp >= A.nw) {
        // the first of these warps is the producer; column pairs keep all four
        // busy, each with every fourth row (one warp took 2.3 ms for what the
        // consumers sum in 0.8: 31 slopes, 69 views, 150x141x75, 162 columns)
        producer_registers();
        const int pw = warp - A.nw;
        if (BULK && pw > 0) {
            __syncthreads();
            return;
        }
        int j = 0;  // stages started
        bool dead = false;
        auto claim = [&]() {
            const int slot = j % ns, round = j / ns;
            const bool ok = round == 0 || ring_wait(&empty[slot], uint32_t((round - 1) & 1), A.err, s_abort, A.wait_limit);
            return __all_sync(0xffffffffu, ok && *s_abort == 0) != 0;
        };
        int turn = 0;
        // the next tile, taken when this one is staged (k_fwd_zsum), or -1 once
        // a wait gave up.  Several producer warps meet here after every tile,
        // a warp that gave up included (each gets here in bounded time), and
        // leave together.
        auto next_tile = [&]() {
            if constexpr (BULK) {
                int t = -1;
                if (lane == 0 && !dead) t = int(gridDim.x) + atomicAdd(A.next, 1);
                return __shfl_sync(0xffffffffu, t, 0);
            } else {
                if (dead) *s_abort = 1;
                turn ^= 1;
                if (pw == 0 && lane == 0) ctl->tile[turn] = int(gridDim.x) + atomicAdd(A.next, 1);
                if (producers_or(dead)) {
                    dead = true;
                    return -1;
                }
                return ctl->tile[turn];
            }
        };
        for (int tile = blockIdx.x; unsigned(tile) < unsigned(A.ntile); tile = next_tile()) {
            int t = tile;
            const int colblk = t % A.n_colblk;
            t /= A.n_colblk;
            const int rowblk = t % A.n_rowblk;
            t /= A.n_rowblk;
            const int plblk = t % A.n_plblk, vi = t / A.n_plblk;  // view slot
            const int mb = NM == 1 ? 0 : vi / A.M.nvm, mv = vi - mb * A.M.nvm;
            if (mv >= member_pick<NM>(A.M.nv, mb)) continue;  // a member with fewer views than the slots
            const int v0 = member_pick<NM>(A.M.first, mb) + mv * A.vr.iv0_step;
            const int p0 = plblk * A.planes, r0 = rowblk * A.rows;
            // columns that a voxel of the tile's planes reads (and, for the
            // adjoint, that are visible)
            const int da = A.T.xt[size_t(v0) * NY + p0].d;
            const int db = A.T.xt[size_t(v0) * NY + min(p0 + A.planes, NY) - 1].d;
            int clo = max(-max(da, db) - 1, 0), chi = min(NX - 1 - min(da, db), G.N_u0 - 1);
            if (ADJ) {
                const int2 u = A.T.ub0[v0];
                clo = max(clo, u.x);
                chi = min(chi, u.y);
            }
            clo &= ~(16 / EB - 1);  // a TMA copy starts on a 16-byte boundary
            const int col0 = clo + colblk * kZCols;
            if (col0 > chi) continue;
            const size_t tb = size_t(plblk) * A.n_rowblk + rowblk;
            const int nlive = A.cnt[tb];
            const int2* list = A.list + tb * A.nv1;
            // the slopes' ray scales, a slope per lane and register
            float S[GV1MAX / 32];
#pragma unroll
            for (int i = 0; i < GV1MAX / 32; i++)
                S[i] = 32 * i + lane < nlive ? A.T.S[size_t(list[32 * i + lane].x) * G.N_v0 + v0] : 0.0f;
            auto scale = [&](int i) {
                const float s = i < 32 ? S[0] : i < 64 ? S[1] : i < 96 ? S[2] : S[3];
                return __shfl_sync(0xffffffffu, s, i & 31);
            };
            const int nst = max(1, (nlive + 1) / 2);  // a tile without slopes still writes its zeros
            for (int i = 0; i < nst; i++) {
                if (!claim()) {
                    dead = true;
                    if (!BULK) *s_abort = 1;  // the other producer warps stop as well
                    break;
                }
                const int slot = j % ns, np = max(0, min(2, nlive - 2 * i));
                unsigned char* st = smem + size_t(slot) * A.stage;
                const float s0 = scale(2 * i), s1 = scale(min(2 * i + 1, GV1MAX - 1));
                if (lane == 0 && pw == 0) {
                    s_info[slot] = ZStage{2 * i, np | (i == nst - 1 ? kZLast : 0), p0, vi, r0, col0, s0, s1};
                    if (BULK) {
                        fence_proxy_async_smem();
                        mbar_arrive_expect_tx(&full[slot], uint32_t(np) * (uint32_t(sizeof(GRec)) +
                                                                           uint32_t(A.nrb) * uint32_t(kZCols * EB)));
                        const CUtensorMap* gmap = &gmaps.m[0];
#pragma unroll
                        for (int m = 1; m < NM; m++)
                            if (mb == m) gmap = &gmaps.m[m];
                        for (int h = 0; h < np; h++) {
                            const int2 sl = list[2 * i + h];
                            tma_load_4d(st + size_t(h) * A.sbytes, gmap, &full[slot], col0, sl.y, v0, sl.x);
                        }
                        if (np)
                            bulk_load(st + A.stage - 2 * sizeof(GRec), A.rec + tb * A.nv1 + 2 * i,
                                      uint32_t(np) * uint32_t(sizeof(GRec)), &full[slot]);
                    } else {
                        mbar_arrive(&full[slot]);
                    }
                }
                if (!BULK) {
                    const TG* g = static_cast<const TG*>(member_pick<NM>(A.M.in, mb));
                    const int c = col0 + 2 * lane;
                    const bool cok = c < G.N_u0;  // N_u0 is even: both columns of the pair
                    static_assert(sizeof(GRec) % 16 == 0 && 2 * sizeof(GRec) <= 32 * 16, "a lane per 16 bytes");
                    if (pw == 0 && lane < np * int(sizeof(GRec) / 16))
                        pair_load<16>(smem_addr(st + A.stage - 2 * sizeof(GRec)) + 16u * lane,
                                      reinterpret_cast<const unsigned char*>(A.rec + tb * A.nv1 + 2 * i) + 16 * lane, true);
                    for (int h = 0; h < np; h++) {
                        const int2 sl = list[2 * i + h];
                        const TG* src = g + ((size_t(sl.x) * G.N_v0 + v0) * G.N_u1 + sl.y + pw) * G.N_u0 + c;
                        uint32_t dst = smem_addr(st + size_t(h) * A.sbytes) + uint32_t((pw * kZCols + 2 * lane) * EB);
#pragma unroll 4
                        for (int r = pw; r < A.nrb; r += 4) {
                            const bool ok = cok && unsigned(sl.y + r) < unsigned(G.N_u1);
                            pair_load<2 * EB>(dst, ok ? src : g, ok);
                            src += 4 * G.N_u0;
                            dst += uint32_t(4 * kZCols * EB);
                        }
                    }
                    pair_arrive(&full[slot]);
                }
                __syncwarp();
                j++;
            }
        }
        if (!dead && claim()) {
            const int slot = j % ns;
            if (lane == 0 && pw == 0) {
                s_info[slot].flags = kZEnd;
                mbar_arrive(&full[slot]);
            }
            if (!BULK) mbar_arrive(&full[slot]);
            j++;
        } else if (lane == 0) {
            *s_abort = 1;
        }
        __syncthreads();
        // a wait gave up: drain the copies still in flight
        if (*s_abort) {
            if (!BULK)
                pair_drain();
            else if (lane == 0)
                for (int i = max(0, j - ns); i < j; i++) mbar_wait(&full[i % ns], uint32_t((i / ns) & 1), nullptr);
        }
        return;
    }

    {
        consumer_registers();
        const int q = warp % A.pg, gr = warp / A.pg;
        int slot = 0;
        uint32_t phase = 0;
        auto wait = [&]() {
            return __all_sync(0xffffffffu, ring_wait(&full[slot], phase, A.err, s_abort, A.wait_limit)) != 0;
        };
        bool dead = !wait();
        while (!dead) {  // tiles
            const ZStage in = s_info[slot];
            if (in.flags & kZEnd) break;
            f2x acc[NV][NK];
#pragma unroll
            for (int u = 0; u < NV; u++)
#pragma unroll
                for (int k = 0; k < NK; k++) acc[u][k] = 0ull;
            for (;;) {  // stages
                const int flags = s_info[slot].flags;
                const unsigned char* st = smem + size_t(slot) * A.stage;
                const GRec* rec = reinterpret_cast<const GRec*>(st + A.stage - 2 * sizeof(GRec));
                const float* sc = &s_info[slot].s0;
#pragma unroll 1
                for (int h = flags & kZCount; h > 0; h--, rec++, sc++, st += A.sbytes) {
                    const uint32_t code = rec->code[warp];
                    if (!(code & 0x300u)) continue;
                    const auto* W = reinterpret_cast<const typename Pair<TG>::type*>(st) +
                                    int(code >> 16) * (kZCols / 2) + lane;
                    f2x wa[NV], wb[NV];
#pragma unroll
                    for (int u = 0; u < NV; u++) {
                        const float w = rec->w[q * NV + u], S = *sc;
                        wa[u] = f2_dup(S * (1.0f - w));
                        wb[u] = f2_dup(S * w);
                    }
                    if ((code & 0x300u) == 0x100u) {
                        if constexpr (NV == 4) {
                            switch (code & 0xffu) {
#define PETL_ZCASE(PC) case PC: z_taps<PC, false>(acc, W, wa, wb); break;
                                PETL_ZCASE(0x00) PETL_ZCASE(0x40) PETL_ZCASE(0x50) PETL_ZCASE(0x90) PETL_ZCASE(0x54)
                                PETL_ZCASE(0x94) PETL_ZCASE(0xA4) PETL_ZCASE(0xE4) PETL_ZCASE(0x01) PETL_ZCASE(0x05)
                                PETL_ZCASE(0x15) PETL_ZCASE(0x06) PETL_ZCASE(0x16) PETL_ZCASE(0x1A) PETL_ZCASE(0x1B)
                            }
                        } else {
                            switch (code & 0xfu) {
                                PETL_ZCASE(0x0) PETL_ZCASE(0x4) PETL_ZCASE(0x8) PETL_ZCASE(0xC) PETL_ZCASE(0x1)
                                PETL_ZCASE(0x2) PETL_ZCASE(0x3)
#undef PETL_ZCASE
                            }
                        }
                    } else {
                        const unsigned long long m = rec->mask[warp];
#pragma unroll
                        for (int u = 0; u < NV; u++) {
                            const int o = int((code >> (2 * u)) & 3u);
                            z_taps_edge<ADJ>(acc[u], W + o * (kZCols / 2), wa[u], wb[u],
                                             uint32_t(m >> (ADJ ? o : 64 / NV * u)));
                        }
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
            // the z sums of the tile
            const int c = in.col0 + 2 * lane, z0 = in.row0 + gr * NK;
            f2x* out = ctl->out[warp][0] + lane;
#pragma unroll 1
            for (int i = 0; i < NV * NK / kZOut; i++) {
                out_rows(acc, out, i);
                const int y = in.a + q * NV + i / (NK / kZOut), zr = z0 + i % (NK / kZOut) * kZOut;
                if (y >= NY) break;
                float* dst = B + ((size_t(in.b) * NY + y) * NZ + zr) * A.NUc + c;
                if (c < G.N_u0)  // N_u0 is even: both columns of the pair
#pragma unroll 4
                    for (int k = 0; k < min(kZOut, NZ - zr); k++)
                        __stcs(reinterpret_cast<float2*>(dst + size_t(k) * A.NUc), f2_unpack(out[k * 32]));
            }
            dead = !wait();
        }
        if (dead) *s_abort = 1;
    }
    __syncthreads();
}

struct XgatherArgs {
    petl_geom G;
    int step;        // view step of the members' view ranges
    int NUc;         // scratch row pitch
    int first;       // first chunk: the view sums start at zero, else at the partial sum
    int last;        // last chunk: write the volume, else the partial sum
    int accumulate;  // add to the volume instead of overwriting it
    float scale;
    Tables T;
    Members M;       // volumes (out) and views of the chunk
};

// x shift of a view on a plane and the scratch columns that count
struct __align__(16) XView {
    int d;
    float w;
    int lo, n;
};

constexpr int XR = 4;         // volume rows z per k_bwd_xgather thread
constexpr int XMAXN = 1024;   // longest scratch / volume row

// x taps of a chunk of views into the volume: thread = column x of rows
// z0..z0+3 of plane y of one member, reading the two scratch taps of every
// view of that member straight from global memory (neighbouring threads
// share them through L1).  Grid (ceil(numX / 256), ceil(numZ / 4), numY x
// members).
template <bool ADJ, int NM>
__global__ void __launch_bounds__(256) k_bwd_xgather(const float* __restrict__ B, float* __restrict__ part,
                                                     const XgatherArgs A)
{
    extern __shared__ __align__(16) unsigned char s_views[];
    Shift* s_xs = reinterpret_cast<Shift*>(s_views);                     // [views of the member] x shifts of plane y
    int2* s_vis = reinterpret_cast<int2*>(s_views) + A.M.nvm;             // and (adjoint) visible columns
    const petl_geom& G = A.G;
    const int NY = G.numY, NZ = G.numZ, NX = G.numX, NU0 = G.N_u0, NUc = A.NUc;
    const int mb = NM == 1 ? 0 : blockIdx.z / NY, y = blockIdx.z - mb * NY;
    const int x = blockIdx.x * 256 + threadIdx.x, z0 = blockIdx.y * XR;
    const int first = member_pick<NM>(A.M.first, mb), nvb = member_pick<NM>(A.M.nv, mb);
    float* __restrict__ f = static_cast<float*>(member_pick<NM>(A.M.out, mb));
    for (int vi = threadIdx.x; vi < nvb; vi += 256) {
        const int v0 = first + vi * A.step;
        s_xs[vi] = A.T.xt[size_t(v0) * NY + y];
        if (ADJ) s_vis[vi] = A.T.ub0[v0];
    }
    __syncthreads();
    if (x >= NX) return;
    const int nz = min(XR, NZ - z0);
    float acc[XR];
#pragma unroll
    for (int r = 0; r < XR; r++)
        acc[r] = (!A.first && r < nz) ? part[(size_t(z0 + r) * NY + y) * NX + x] : 0.0f;
    const int rlast = nz - 1;
    const float* Bm = B + size_t(mb) * A.M.nvm * NY * NZ * NUc;
#pragma unroll 4
    for (int vi = 0; vi < nvb; vi++) {
        const Shift xs = s_xs[vi];
        const float wx1 = xs.w, wx0 = 1.0f - xs.w;
        const int j0 = x - xs.d;  // scratch column of tap 0
        // the adjoint counts the view's visible columns only (the scratch holds no others)
        const int2 u = ADJ ? s_vis[vi] : make_int2(0, NU0 - 1);
        const bool okm = j0 - 1 >= u.x && j0 - 1 <= u.y, ok0 = j0 >= u.x && j0 <= u.y;
        // in-bounds addresses for every tap; the out-of-range ones are selected away
        const int jm = min(max(j0 - 1, 0), NU0 - 1), jz = min(max(j0, 0), NU0 - 1);
        const float* Bv = Bm + ((size_t(vi) * NY + y) * NZ + z0) * NUc;
#pragma unroll
        for (int r = 0; r < XR; r++) {
            const int rr = min(r, rlast);
            const float vm = __ldg(Bv + rr * NUc + jm), vz = __ldg(Bv + rr * NUc + jz);
            acc[r] = acc[r] + fmaf(wx1, okm ? vm : 0.0f, wx0 * (ok0 ? vz : 0.0f));
        }
    }
#pragma unroll
    for (int r = 0; r < XR; r++) {
        if (r >= nz) break;
        const size_t o = (size_t(z0 + r) * NY + y) * NX + x;
        if (!A.last)
            part[o] = acc[r];
        else
            f[o] = A.accumulate ? f[o] + A.scale * acc[r] : A.scale * acc[r];
    }
}

// One slope with v1 = 0 (the rebinned planogram of FBP): its z taps and
// visible rows are the same on every plane.  k_bwd_zflat writes the z sums
// once per view, B[view][c][z] = S (1 - w) g[z - d][c] then + S w g[z - d - 1][c],
// the operations and masks of k_bwd_zgather for a single slope (rows outside
// the planogram read zero; the adjoint zeroes rows outside the visible u1
// range, the reference semantics leave rows z outside the voxel test at
// zero).  A block transposes 32 columns x 32 rows of one view.  Grid
// (ceil(N_u0 / 32), ceil(NZc / 32), views), 32 x 8 threads.
struct FlatArgs {
    petl_geom G;
    int iv1;         // the slope
    int first;       // first view
    int step;        // view step
    int nv;          // views
    int NZc;         // scratch row pitch (rows z, even)
    int accumulate;  // add to the volume instead of overwriting it
    float scale;
    Tables T;
};

template <bool ADJ>
__global__ void __launch_bounds__(256) k_bwd_zflat(const float* __restrict__ g, float* __restrict__ B, const FlatArgs A)
{
    __shared__ float tile[32][33];
    const petl_geom& G = A.G;
    const int c0 = blockIdx.x * 32, z0 = blockIdx.y * 32, vi = blockIdx.z;
    const int v0 = A.first + vi * A.step;
    const Shift zs = A.T.zt[size_t(A.iv1) * G.numY];  // plane 0: every plane has the same
    const float S = A.T.S[size_t(A.iv1) * G.N_v0 + v0];
    const float w0 = S * (1.0f - zs.w), w1 = S * zs.w;
    const int2 ub1 = A.T.ub1[A.iv1], zv = A.T.zvis[size_t(A.iv1) * G.numY];
    const int c = c0 + threadIdx.x;
    for (int r = threadIdx.y; r < 32; r += 8) {
        const int z = z0 + r;
        auto row = [&](int i) {
            const bool in = i >= 0 && i < G.N_u1 && c < G.N_u0 && (!ADJ || (i >= ub1.x && i <= ub1.y));
            return in ? g[((size_t(A.iv1) * G.N_v0 + v0) * G.N_u1 + i) * G.N_u0 + c] : 0.0f;
        };
        const bool live = z < G.numZ && (ADJ || (z >= zv.x && z <= zv.y));
        tile[r][threadIdx.x] = live ? fmaf(w1, row(z - zs.d - 1), fmaf(w0, row(z - zs.d), 0.0f)) : 0.0f;
    }
    __syncthreads();
    const int z = z0 + threadIdx.x;
    for (int r = threadIdx.y; r < 32; r += 8)
        if (c0 + r < G.N_u0 && z < A.NZc) B[(size_t(vi) * G.N_u0 + c0 + r) * A.NZc + z] = tile[threadIdx.x][r];
}

// x taps of the flat z sums into the volume.  LZ lanes take 2 LZ rows z (two
// per lane, so every tap is a coalesced eight-byte load whatever the shift) of
// FX neighbouring x on one plane: FX + 1 loads per view for 2 FX taps.  The
// block's FW warps take neighbouring planes, whose taps meet in L1, FVB views'
// shifts staged at a time.  With a thread per x the taps cost two four-byte
// loads each, and FBP's backprojection at 256x256x128 (129 views) was bound by
// them (0.70 ms).  The operations of k_bwd_xgather in its order.  Grid
// (ceil(numX / FX), ceil(numY / FPL), ceil(numZ / (2 LZ))), 32 FW threads.
//
// Large volumes: 8 x, 8 planes, 64 rows.  Where such blocks number fewer than
// the SMs the kernel waits on a view's loads after the other's: 2 x, 8 planes
// of half a warp each, 32 rows, four views' loads in flight (whole
// backprojection of 65 views, large shape / this one / a thread per x:
// 48x48x24 46 / 32 / 41 us, 63x63x28 48 / 32 / 41, 80x80x40 49 / 39 / 43,
// 96x96x32 47 / 35 / 43; 96x96x96, 288 blocks of the large shape, 56 / 58 / 79).
template <bool ADJ, int FX, int FW, int LZ, int FVB, int UNROLL>
__global__ void __launch_bounds__(32 * FW) k_bwd_flat_gather(const float* __restrict__ B, float* __restrict__ f,
                                                        const FlatArgs A)
{
    constexpr int FPL = FW * 32 / LZ;  // planes per block
    __shared__ XView s_xs[FVB][FPL];
    const petl_geom& G = A.G;
    const int NY = G.numY, NZ = G.numZ, NX = G.numX, NU0 = G.N_u0;
    const int lane = threadIdx.x % LZ, pl = threadIdx.x / LZ;
    const int x0 = blockIdx.x * FX, y = blockIdx.y * FPL + pl, z = blockIdx.z * (2 * LZ) + 2 * lane;
    const bool zok = z < A.NZc;
    const f2x* Bz = reinterpret_cast<const f2x*>(B + (zok ? z : 0));
    const int pitch = A.NZc / 2;
    f2x acc[FX];
#pragma unroll
    for (int k = 0; k < FX; k++) acc[k] = 0ull;
    for (int vb = 0; vb < A.nv; vb += FVB) {
        __syncthreads();
#pragma unroll 4
        for (int r = 0; r < FVB * FPL / (32 * FW); r++) {  // by four: by eight and one by one ran 7 us slower
            const int e = r * (32 * FW) + threadIdx.x, i = e / FPL, p = e % FPL;
            const int v0 = A.first + (vb + i) * A.step;
            if (vb + i < A.nv && blockIdx.y * FPL + p < NY) {
                const Shift xs = A.T.xt[size_t(v0) * NY + blockIdx.y * FPL + p];
                const int2 u = ADJ ? A.T.ub0[v0] : make_int2(0, NU0 - 1);
                s_xs[i][p] = XView{xs.d, xs.w, u.x, max(0, u.y - u.x + 1)};
            }
        }
        __syncthreads();
        if (y >= NY) continue;
        const int n = min(FVB, A.nv - vb);
#pragma unroll UNROLL
        for (int i = 0; i < n; i++) {
            const XView xs = s_xs[i][pl];
            const f2x w1 = f2_dup(xs.w), w0 = f2_dup(1.0f - xs.w);
            const int cb = x0 - xs.d - 1;  // scratch column of tap 1 of x0
            const f2x* Bv = Bz + size_t(vb + i) * NU0 * pitch;
            f2x t[FX + 1];
#pragma unroll
            for (int k = 0; k <= FX; k++)
                t[k] = unsigned(cb + k - xs.lo) < unsigned(xs.n) ? __ldg(Bv + size_t(cb + k) * pitch) : 0ull;
#pragma unroll
            for (int k = 0; k < FX; k++) acc[k] = f2_add(acc[k], f2_fma(w1, t[k], f2_mul(w0, t[k + 1])));
        }
    }
    if (y >= NY) return;
    const bool quads = (NX & 3) == 0 && (reinterpret_cast<uintptr_t>(f) & 15) == 0;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        if (z + h >= NZ) break;
        float v[FX < 4 ? 4 : FX];
#pragma unroll
        for (int k = 0; k < FX; k++) {
            const float2 a = f2_unpack(acc[k]);
            v[k] = h ? a.y : a.x;
        }
        float* row = f + (size_t(z + h) * NY + y) * NX + x0;
#pragma unroll
        for (int k = 0; k < FX; k += 4) {
            if (FX % 4 == 0 && quads && x0 + k + 4 <= NX) {
                float4* o = reinterpret_cast<float4*>(row + k);
                if (A.accumulate) {
                    const float4 p = *o;
                    *o = make_float4(fmaf(A.scale, v[k], p.x), fmaf(A.scale, v[k + 1], p.y),
                                     fmaf(A.scale, v[k + 2], p.z), fmaf(A.scale, v[k + 3], p.w));
                } else {
                    *o = make_float4(A.scale * v[k], A.scale * v[k + 1], A.scale * v[k + 2], A.scale * v[k + 3]);
                }
            } else {
#pragma unroll
                for (int i = k; i < (k + 4 < FX ? k + 4 : FX); i++)
                    if (x0 + i < NX) row[i] = A.accumulate ? fmaf(A.scale, v[i], row[i]) : A.scale * v[i];
            }
        }
    }
}

int backproject_flat(const petl_geom& G, const float* g, float* f, int mode, int accumulate, float scale,
                     const ViewRange& vr, const Tables& T, cudaStream_t st)
{
    const int n_v0 = vr.n_v0(G.N_v0);
    if (n_v0 <= 0 || n_v0 > 65535 || G.N_u0 > XMAXN || G.numZ > 65535 || G.numY > 65535) return kNotApplicable;
    const int NZc = (G.numZ + 1) & ~1;
    float* B = nullptr;
    if (scratch_alloc(reinterpret_cast<void**>(&B), size_t(n_v0) * G.N_u0 * NZc * 4, st) != cudaSuccess) {
        cudaGetLastError();
        return kNotApplicable;
    }
    const FlatArgs FA{G, vr.iv1_begin, vr.iv0_first, vr.iv0_step, n_v0, NZc, accumulate, scale, T};
    const dim3 grid(ceil_div(G.N_u0, 32), ceil_div(NZc, 32), unsigned(n_v0));
    const bool adj = mode == PETL_BP_ADJOINT;
    const bool small = (long long)ceil_div(G.numX, 8) * ceil_div(G.numY, 8) * ceil_div(G.numZ, 64) < sm_count();
    const dim3 ggrid = small ? dim3(ceil_div(G.numX, 2), ceil_div(G.numY, 8), ceil_div(G.numZ, 32))
                             : dim3(ceil_div(G.numX, 8), ceil_div(G.numY, 8), ceil_div(G.numZ, 64));
    auto kz = adj ? k_bwd_zflat<true> : k_bwd_zflat<false>;
    auto kg = adj ? (small ? k_bwd_flat_gather<true, 2, 4, 16, 128, 4> : k_bwd_flat_gather<true, 8, 8, 32, 32, 2>)
                  : (small ? k_bwd_flat_gather<false, 2, 4, 16, 128, 4> : k_bwd_flat_gather<false, 8, 8, 32, 32, 2>);
    kz<<<grid, dim3(32, 8), 0, st>>>(g, B, FA);
    kg<<<ggrid, small ? 128 : 256, 0, st>>>(B, f, FA);
    note_launch();
    note_launch();
    const cudaError_t e = cudaGetLastError();
    cudaFreeAsync(B, st);
    if (e != cudaSuccess) {
        set_error(std::string("backproject_flat: ") + cudaGetErrorString(e));
        return int(e);
    }
    return 0;
}

}  // namespace

// Backprojection of the members' views.  One member: its views in chunks of
// at most the scratch budget (and chunk_cap); several: one chunk, else
// kNotApplicable.  Member b reads planogram M0.in[b] and writes (or adds to)
// volume M0.out[b].
template <class TG>
int backproject_split_m(const petl_geom& G, const Members& M0, int mode, int accumulate, float scale,
                        const ViewRange& vr, const Tables& T, cudaStream_t st, int chunk_cap, const ChunkHook* hook)
{
    constexpr int EB = int(sizeof(TG));
    const int nb = M0.nb;
    if (nb < 1 || nb > kMaxMembers) return kNotApplicable;
    int nvmax = 0;
    for (int b = 0; b < nb; b++) nvmax = std::max(nvmax, M0.nv[b]);
    const int nv1 = vr.iv1_end - vr.iv1_begin;
    if (nvmax <= 0 || nv1 <= 0 || nv1 > GV1MAX) return kNotApplicable;
    // one slope at v1 = 0 (FBP's rebinned planogram): z sums without a plane
    // dimension
    if (std::is_same<TG, float>::value && nb == 1 && nv1 == 1 && M0.first[0] == vr.iv0_first &&
        M0.nv[0] == vr.n_v0(G.N_v0) && std::fmaf(float(vr.iv1_begin), G.T_v1, G.v1_0) == 0.0f)
        return backproject_flat(G, static_cast<const float*>(M0.in[0]), static_cast<float*>(M0.out[0]), mode,
                                accumulate, scale, vr, T, st);
    // the scratch holds a volume per view whatever the slope count: below
    // about ten slopes (the 2-D backprojection of FBP has one) the
    // single-pass kernel is cheaper than that round trip
    if (nv1 < kSplitMinSlopes) return kNotApplicable;
    // staged rows: tiled copies of rows of a multiple of 16 bytes from a
    // 16-byte aligned base, else lanes copy column pairs (even N_u0)
    bool bulk = (G.N_u0 * EB) % 16 == 0;
    if (G.N_u0 & 1) return kNotApplicable;
    for (int b = 0; b < nb; b++) {
        const uintptr_t p = reinterpret_cast<uintptr_t>(M0.in[b]);
        bulk = bulk && (p & 15) == 0;
        if ((p & (2 * EB - 1)) != 0) return kNotApplicable;
    }
    if (G.N_u0 > XMAXN || G.numY > 65535 || G.numZ > 65535 * XR) return kNotApplicable;
    if (size_t(G.numY) * nb > 65535) return kNotApplicable;  // k_bwd_xgather grid.z
    const ShiftStep step = plane_step(G);
    // four planes share a window of 16 rows where their shifts move by less
    // than a row per plane, else two planes a window of 28 rows, as in the
    // forward
    const int NV = four_per_window(step) ? 4 : 2, NK = NV == 4 ? 12 : 24;
    if (shift_spread(NV - 1, step) > kZSpread) return kNotApplicable;
    int* err = device_error_ptr();
    if (!err) return kNotApplicable;

    // chunks of views whose scratch fits the budget, balanced in size
    const int NUc = (G.N_u0 + 3) & ~3;
    const size_t per_view = size_t(G.numY) * G.numZ * NUc * 4;
    const size_t fit = std::max<size_t>(1, split_scratch_budget() / per_view);
    int nv, nchunks;
    if (nb == 1) {
        nv = int(std::min<size_t>(size_t(nvmax), fit));
        nv = std::min(nv, 3072);  // k_bwd_xgather stages the chunk's x shifts in shared memory
        if (chunk_cap > 0) nv = std::min(nv, chunk_cap);
        nchunks = (nvmax + nv - 1) / nv;
        nv = (nvmax + nchunks - 1) / nchunks;
    } else {
        if (size_t(nb) * nvmax > fit || nvmax > 3072 || chunk_cap > 0) return kNotApplicable;
        nv = nvmax;
        nchunks = 1;
    }

    ZgatherArgs A{};
    A.G = G;
    A.vr = vr;
    A.n_colblk = int(ceil_div(G.N_u0, kZCols));
    A.NUc = NUc;
    A.nv1 = nv1;
    A.T = T;
    A.err = err;
    A.wait_limit = wait_limit();
    // twelve consumer warps, or four where these have few tiles (ztwelve)
    for (A.nw = kZWarps;; A.nw = 4) {
        A.pg = NV == 4 || A.nw == 4 ? 4 : 6;
        A.rg = A.nw / A.pg;
        A.planes = NV * A.pg;
        A.rows = NK * A.rg;
        A.n_plblk = int(ceil_div(G.numY, A.planes));
        A.n_rowblk = int(ceil_div(G.numZ, A.rows));
        const long long nt = (long long)nv * nb * A.n_plblk * A.n_rowblk * A.n_colblk;
        if (nt > (1 << 30)) return kNotApplicable;
        A.ntile = int(nt);
        if (A.nw == 4 || ztwelve(A.ntile)) break;
    }
    if (A.n_rowblk > 65535) return kNotApplicable;  // k_gather_records grid.y
    A.nrb = A.rows + 1 + shift_spread(A.planes - 1, step);
    if (A.nrb > 250) return kNotApplicable;  // TMA box rows
    A.sbytes = (A.nrb + kZSpread) * kZCols * EB;  // a multiple of 128
    A.stage = (2 * A.sbytes + 2 * int(sizeof(GRec)) + 127) & ~127;
    int ctas = zctas(A.nw, A.ntile);  // a ring that does not fit half an SM takes the whole
    for (;; ctas = 1) {
        A.ns = std::min(kZStages, (zsmem(ctas) - zctl_bytes(A.nw)) / A.stage);
        if (A.ns >= 2 || ctas == 1) break;
    }
    if (A.ns < 2) return kNotApplicable;
    const size_t smem = size_t(A.ns) * A.stage + zctl_bytes(A.nw);

    GMaps<kMaxMembers> maps;
    std::memset(&maps, 0, sizeof(maps));
    if (bulk) {
        const uint64_t dims[4] = {uint64_t(G.N_u0), uint64_t(G.N_u1), uint64_t(G.N_v0), uint64_t(G.N_v1)};
        const uint64_t strides[3] = {uint64_t(G.N_u0) * EB, uint64_t(G.N_u0) * G.N_u1 * EB,
                                     uint64_t(G.N_u0) * G.N_u1 * G.N_v0 * EB};
        const uint32_t box[4] = {uint32_t(kZCols), uint32_t(A.nrb), 1u, 1u};
        for (int b = 0; b < nb; b++)
            if (!encode_tensor_map(&maps.m[b], M0.in[b], 4, dims, strides, box, EB)) return kNotApplicable;
    }

    // B, then the table records, the lists and the counts
    float* B = nullptr;
    float* part = nullptr;
    const size_t nvox = size_t(G.numX) * G.numY * G.numZ;
    const size_t b_bytes = per_view * nv * nb;  // a multiple of 16
    const size_t ntab = size_t(A.n_plblk) * A.n_rowblk;
    const size_t t_bytes = ntab * nv1 * (sizeof(GRec) + sizeof(int2)) + (ntab + nchunks) * sizeof(int);
    if (scratch_alloc(reinterpret_cast<void**>(&B), b_bytes + t_bytes, st) != cudaSuccess ||
        (nchunks > 1 && scratch_alloc(reinterpret_cast<void**>(&part), nvox * 4, st) != cudaSuccess)) {
        cudaGetLastError();  // out of memory is not sticky: the caller takes the single-pass kernel
        if (B) cudaFreeAsync(B, st);
        return kNotApplicable;
    }
    A.rec = reinterpret_cast<GRec*>(reinterpret_cast<unsigned char*>(B) + b_bytes);
    A.list = reinterpret_cast<int2*>(A.rec + ntab * nv1);
    A.cnt = reinterpret_cast<int*>(A.list + ntab * nv1);
    A.next = A.cnt + ntab;
    A.nchunks = nchunks;
    const bool adj = mode == PETL_BP_ADJOINT;
    const dim3 rgrid(unsigned(A.n_plblk), unsigned(A.n_rowblk));
    if (adj)
        k_gather_records<true><<<rgrid, 256, 0, st>>>(A, NV, NK);
    else
        k_gather_records<false><<<rgrid, 256, 0, st>>>(A, NV, NK);
    note_launch();
    auto launch = [&](auto bulk_c, auto nv_c, auto nk_c, unsigned grid) {
        constexpr bool BULK = decltype(bulk_c)::value;
        constexpr int V = decltype(nv_c)::value, K = decltype(nk_c)::value;
        const unsigned threads = 32u * unsigned(A.nw + 4);
        cudaError_t r;
        if (nb == 1) {  // kernels compiled for one member where there is one
            GMaps<1> map1;
            map1.m[0] = maps.m[0];
            auto kz = adj ? k_bwd_zgather<true, TG, 1, BULK, V, K> : k_bwd_zgather<false, TG, 1, BULK, V, K>;
            r = cudaFuncSetAttribute(kz, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
            if (r == cudaSuccess) kz<<<grid, threads, smem, st>>>(map1, B, A);
        } else {
            auto kz = adj ? k_bwd_zgather<true, TG, kMaxMembers, BULK, V, K>
                          : k_bwd_zgather<false, TG, kMaxMembers, BULK, V, K>;
            r = cudaFuncSetAttribute(kz, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
            if (r == cudaSuccess) kz<<<grid, threads, smem, st>>>(maps, B, A);
        }
        return r;
    };
    auto kx = adj ? (nb == 1 ? k_bwd_xgather<true, 1> : k_bwd_xgather<true, kMaxMembers>)
                  : (nb == 1 ? k_bwd_xgather<false, 1> : k_bwd_xgather<false, kMaxMembers>);
    cudaError_t e = cudaGetLastError();
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
        if (hook && hook->fn) hook->fn(hook->ctx, vi0, nvc);
        A.M = M;
        A.nslot = nvc * nb;
        A.ntile = A.nslot * A.n_plblk * A.n_rowblk * A.n_colblk;
        const unsigned grid = unsigned(std::min(A.ntile, ctas * sm_count()));
        using std::integral_constant;
        if (bulk)
            e = NV == 4 ? launch(std::true_type{}, integral_constant<int, 4>{}, integral_constant<int, 12>{}, grid)
                        : launch(std::true_type{}, integral_constant<int, 2>{}, integral_constant<int, 24>{}, grid);
        else
            e = NV == 4 ? launch(std::false_type{}, integral_constant<int, 4>{}, integral_constant<int, 12>{}, grid)
                        : launch(std::false_type{}, integral_constant<int, 2>{}, integral_constant<int, 24>{}, grid);
        if (e != cudaSuccess) break;
        note_launch();
        A.next++;
        XgatherArgs X{G, vr.iv0_step, A.NUc, c == 0, c == nchunks - 1, accumulate, scale, T, M};
        kx<<<dim3(ceil_div(G.numX, 256), ceil_div(G.numZ, XR), unsigned(G.numY) * unsigned(nb)), 256,
                        size_t(nvc) * (adj ? 2 : 1) * sizeof(Shift), st>>>(B, part, X);
        note_launch();
        e = cudaGetLastError();
    }
    cudaFreeAsync(B, st);
    if (part) cudaFreeAsync(part, st);
    if (e != cudaSuccess) {
        set_error(std::string("backproject_split: ") + cudaGetErrorString(e));
        return int(e);
    }
    return 0;
}

template <class TG>
int backproject_split_t(const petl_geom& G, const TG* g, float* f, int mode, int accumulate, float scale,
                        const ViewRange& vr, const Tables& T, cudaStream_t st, int chunk_cap, const ChunkHook* hook)
{
    Members M;
    M.nb = 1;
    M.first[0] = vr.iv0_first;
    M.nv[0] = vr.n_v0(G.N_v0);
    M.in[0] = g;
    M.out[0] = f;
    return backproject_split_m<TG>(G, M, mode, accumulate, scale, vr, T, st, chunk_cap, hook);
}

int backproject_split(const petl_geom& G, const float* g, float* f, int mode, int accumulate, float scale,
                      const ViewRange& vr, const Tables& T, cudaStream_t st, int chunk_cap, const ChunkHook* hook)
{
    return backproject_split_t<float>(G, g, f, mode, accumulate, scale, vr, T, st, chunk_cap, hook);
}

int backproject_split_bf16(const petl_geom& G, const __nv_bfloat16* g, float* f, int mode, int accumulate,
                           float scale, const ViewRange& vr, const Tables& T, cudaStream_t st)
{
    return backproject_split_t<__nv_bfloat16>(G, g, f, mode, accumulate, scale, vr, T, st, 0, nullptr);
}

int backproject_split_members(const petl_geom& G, const Members& M, int mode, int accumulate, float scale,
                              const ViewRange& vr, const Tables& T, cudaStream_t st)
{
    return backproject_split_m<float>(G, M, mode, accumulate, scale, vr, T, st, 0, nullptr);
}

}  // namespace shear
}  // namespace petl
