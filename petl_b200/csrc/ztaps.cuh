// Pieces shared by the split z kernels (projector_split.cu,
// backprojector_split.cu): packed column-pair FMAs, the unrolled z taps over a
// register window, and the ring of staged planes / slopes that one producer
// warp fills for the consumer warps of a persistent CTA.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "common.cuh"
#include "tma.cuh"

namespace petl {
namespace shear {

// A column pair of two FP32 values in one 64-bit register.  The packed FMA
// rounds each half as the scalar FMA does, so results equal the scalar form
// bit for bit.  It takes half the issue slots: a loop of shared-memory window
// loads and z taps ran at 29.5-32 TFMA/s packed against 24-25 scalar (4 to 16
// warps per SM, 2 x 16 or 4 x 8 accumulator pairs; the FP32 peak is 37.2).
typedef unsigned long long f2x;

__device__ __forceinline__ f2x f2_pack(float x, float y)
{
    f2x r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ f2x f2_dup(float a) { return f2_pack(a, a); }
__device__ __forceinline__ float2 f2_unpack(f2x a)
{
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
    return r;
}
__device__ __forceinline__ f2x f2_fma(f2x a, f2x b, f2x c)
{
    f2x r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

__device__ __forceinline__ f2x f2_mul(f2x a, f2x b)
{
    f2x r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2x f2_add(f2x a, f2x b)
{
    f2x r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// Staged column pairs of either storage type as FP32 pairs.
__device__ __forceinline__ f2x pair_get(f2x v) { return v; }
__device__ __forceinline__ f2x pair_get(uint32_t v)
{
    return f2_pack(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u));
}
template <class T>
struct Pair;
template <>
struct Pair<float> {
    using type = f2x;
};
template <>
struct Pair<__nv_bfloat16> {
    using type = uint32_t;
};

// z taps of N accumulator blocks of NK rows with compile-time window offsets
// (PC: 2 bits per block): acc[j][k] takes first its first tap, then its
// second, from window rows k + o and k + o + 1 (FWD: in this order; else the
// other way round).  The window rows stream from shared memory (row pitch:
// 64 columns) in the order that keeps each accumulator's taps in order, so
// few of them are live at a time: a window held in registers next to 128
// accumulator registers spilled.
template <int PC, bool FWD, int N, int NK, class P>
__device__ __forceinline__ void z_taps(f2x (&acc)[N][NK], const P* __restrict__ W, const f2x (&wa)[N],
                                       const f2x (&wb)[N])
{
    constexpr int o0 = PC & 3, o1 = N > 1 ? (PC >> 2) & 3 : o0, o2 = N > 2 ? (PC >> 4) & 3 : o0,
                  o3 = N > 3 ? (PC >> 6) & 3 : o0;
    constexpr int omin = o0 < o1 ? (o0 < o2 ? (o0 < o3 ? o0 : o3) : (o2 < o3 ? o2 : o3))
                                 : (o1 < o2 ? (o1 < o3 ? o1 : o3) : (o2 < o3 ? o2 : o3));
    constexpr int omax = o0 > o1 ? (o0 > o2 ? (o0 > o3 ? o0 : o3) : (o2 > o3 ? o2 : o3))
                                 : (o1 > o2 ? (o1 > o3 ? o1 : o3) : (o2 > o3 ? o2 : o3));
    constexpr int rows = NK + 1 + omax - omin;
#pragma unroll
    for (int s = 0; s < rows; s++) {
        const int i = FWD ? omin + s : omin + rows - 1 - s;  // window row
        const f2x w = pair_get(W[i * 32]);
#pragma unroll
        for (int j = 0; j < N; j++) {
            const int o = (PC >> (2 * j)) & 3;
            const int ka = FWD ? i - o : i - o - 1, kb = FWD ? i - o - 1 : i - o;
            if (ka >= 0 && ka < NK) acc[j][ka] = f2_fma(wa[j], w, acc[j][ka]);
            if (kb >= 0 && kb < NK) acc[j][kb] = f2_fma(wb[j], w, acc[j][kb]);
        }
    }
}

// Backward z taps of one plane at the edge of the visible range: window rows
// outside mask m read zero (ADJ), or output rows outside m take nothing.
template <bool ADJ, int NK, class P>
__device__ __forceinline__ void z_taps_edge(f2x (&acc)[NK], const P* __restrict__ W, f2x wa, f2x wb, uint32_t m)
{
#pragma unroll
    for (int i = NK; i >= 0; i--) {
        f2x w = pair_get(W[i * 32]);
        if (ADJ && !((m >> i) & 1u)) w = 0ull;
        if (i >= 1 && (ADJ || ((m >> (i - 1)) & 1u))) acc[i - 1] = f2_fma(wa, w, acc[i - 1]);
        if (i < NK && (ADJ || ((m >> i) & 1u))) acc[i] = f2_fma(wb, w, acc[i]);
    }
}

// A lane's copy of a column pair into shared memory (zeros unless ok), and the
// lane's arrival on the stage's barrier once its copies are done.
template <int BYTES>
__device__ __forceinline__ void pair_load(uint32_t dst, const void* src, bool ok)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(dst), "l"(src), "n"(BYTES), "r"(ok ? BYTES : 0)
                 : "memory");
}
__device__ __forceinline__ void pair_arrive(uint64_t* bar)
{
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void pair_drain() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Shape of a consumer warp's tile: NV slopes (forward) or planes (backward)
// x NK rows x 64 columns (two per lane), 48 packed accumulators per lane.
// Four slopes x 12 rows share one register window where their shifts differ
// by at most kZSpread rows; two slopes x 24 rows serve steeper shifts (a
// window of 28 rows feeds 96 packed FMAs, against 16 rows in the 4 x 12 form).
constexpr int kZSpread = 3;    // largest shift difference within a warp's tile
constexpr int kZCols = 64;     // columns per tile
constexpr int kZWarps = 12;    // consumer warps of a CTA at most
constexpr int kZStages = 8;    // ring stages at most (of up to four planes or two slopes)
// A CTA's last four warps give up registers to the consumer warps: a launch
// of 16 warps has 128 registers a thread (four warps per scheduler), 12 x 160
// + 4 x 32 is the same total.  The first of the four is the producer.
constexpr int kZThreads = 32 * (kZWarps + 4);
__device__ __forceinline__ void consumer_registers() { asm volatile("setmaxnreg.inc.sync.aligned.u32 160;"); }
__device__ __forceinline__ void producer_registers() { asm volatile("setmaxnreg.dec.sync.aligned.u32 32;"); }

// Whether any of the four producer warps (128 threads) passes true; all of
// them call it the same number of times.
__device__ __forceinline__ bool producers_or(bool v)
{
    uint32_t any;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "bar.red.or.pred q, 1, 128, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(any)
        : "r"(uint32_t(v))
        : "memory");
    return any != 0;
}

// What the producer tells the consumers about a stage.
struct __align__(16) ZStage {
    // first plane (forward) or position in the slope list (backward).  Nothing
    // reads it; without it, or with the others in another order, the compiler
    // spills twice as much in the plane loop of one z kernel or the other
    // (256x256x128: forward 7.86 -> 10.5 ms, or backward 8.83 -> 10.0)
    int y;
    int flags;  // staged planes / slopes | kZLast | ...
    int a, b;   // tile: first slope / plane, view slot
    int row0, col0;
    float s0, s1;  // backward: ray scale of the staged slopes
};
constexpr int kZCount = 7;   // planes / slopes of the stage
constexpr int kZLast = 16;   // last stage of a tile
constexpr int kZEnd = 1024;  // no more tiles
constexpr int kZRow0 = 32, kZRowN = 64, kZCol0 = 128, kZColN = 256;  // tile at an edge of the output
constexpr int kZTail = 512;  // tile of the tail launch shape

constexpr int kZOut = 12;

// Ring control block, after the stages in shared memory.
struct ZCtl {
    ZStage info[kZStages];
    uint64_t full[kZStages], empty[kZStages];
    int abort;  // a warp gave up a wait: start no further copies
    int tile[2];  // the producer warps' next tile, by turns
    // (the CTA's consumer warps only) a warp's epilogue passes its accumulators through here, twelve rows at a
    // time, so that the code that scales, masks and stores them is one rolled
    // loop: unrolled over all accumulators it was tens of KB of straight code
    // per tile, and its instruction fetches took a fifth of the forward's time
    f2x out[kZWarps][kZOut][32];
};
constexpr int zctl_bytes(int nw) { return int(sizeof(ZCtl)) - (kZWarps - nw) * kZOut * 32 * int(sizeof(f2x)); }

// Whether a launch of so many tiles of twelve-warp CTAs takes these, or tiles
// of a third of the rows in four-warp CTAs, two of which share an SM where
// there are more of them than SMs (registers: 256 threads of 128; shared memory:
// 228 KB per SM, 1 KB per CTA reserved).  A tile's time is latency below a full
// chip, so smaller tiles on more SMs win until twelve-warp tiles fill about
// two thirds of them.  Forward of 4000 panels at psi = 0, time of twelve-warp
// tiles over four-warp ones by number of tiles: 20-40 1.09, 60-80 1.07, 80-100
// 1.04, 100-120 1.02, 120-148 0.97, 200-296 0.96, 400 0.88; two CTAs per SM
// against one, where four-warp tiles outnumber SMs: 1.06 at 80-100 tiles, 1.13
// at 120-148.
inline bool ztwelve(int tiles) { return 3 * tiles >= 2 * sm_count(); }
inline int zctas(int nw, int tiles) { return nw == 4 && tiles > sm_count() ? 2 : 1; }
constexpr int zsmem(int ctas) { return (228 / ctas - 1) * 1024; }

// Rows 12 * (i % (NK / 12)) .. + 11 of accumulator block i / (NK / 12) to the
// warp's lane slots.
template <int N, int NK>
__device__ __forceinline__ void out_rows(const f2x (&acc)[N][NK], f2x* out, int i)
{
    static_assert(N * NK == 4 * kZOut, "four groups of twelve rows");
    switch (i) {
#define PETL_ZOUT(I)                                                                       \
    case I:                                                                                \
        _Pragma("unroll") for (int k = 0; k < kZOut; k++) out[k * 32] =                    \
            acc[I / (NK / kZOut)][I % (NK / kZOut) * kZOut + k];                           \
        break;
        PETL_ZOUT(0) PETL_ZOUT(1) PETL_ZOUT(2) PETL_ZOUT(3)
#undef PETL_ZOUT
    }
}

// Bounded wait that also ends when another warp of the CTA gave up (*abort).
// limit 0 (petl_force_wait_timeout) gives up without polling.
__device__ __forceinline__ bool ring_wait(uint64_t* bar, uint32_t parity, int* err, const volatile int* abort,
                                          unsigned limit)
{
    if (limit != 0) return mbar_wait_abortable(bar, parity, err, abort);
    if (err) atomicOr(err, kErrWaitTimeout);
    return false;
}

}  // namespace shear
}  // namespace petl
