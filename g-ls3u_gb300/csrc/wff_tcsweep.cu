// wff_tcsweep.cu -- WFF2 column sweep on the tensor cores (FP32 form).
//
// The demodulated form of the sweep: for one x-frequency plane R and every wy
//     U = (R e^{-j wy y}) (*)_y g,   T = U . [ |U| >= thr N ],
//     C += e^{+j wy y} (T (*)_y g)
// with g the real, truncated window of 2s+1 taps.  Each of the two
// convolutions is a banded Toeplitz product.  The image columns are the M
// rows of the MMA (64 columns, real and imaginary parts in lanes of their
// own: M = 128), 16 image rows are its K, and the N outputs they reach --
// 2s + 16, rounded up to a multiple of 16 -- its N.  The B operand is one
// constant block B[n][j] = g(n - j - s) for every K step; the accumulator
// window of a step starts 16 TMEM columns after that of the step before.
//
// FP32 in 11-bit operands: each value and each tap is split into two FP16
// parts, x = hi + lo with |x - hi - lo| <= 2^-22 |x| (lo below 2^-10 of x, see
// split2; taps to 2^-24 of the largest), and a K step is three MMAs, lo.hi +
// hi.lo + hi.hi, accumulated in FP32 (the dropped lo.lo is at most 2^-21 of the
// product with the largest tap, of either sign in turns).  Powers of two keep both parts in FP16's normal
// range: R is scaled to at most 2^15, the taps by 2^6, T by tscale to at most
// 2^15.  An input of unit modulus (DPRA) has one scale, which the row pass
// applies (d_kr); for any other the B warps scale each column of a tile by its
// own largest finite value, so that a large value leaves its mark, 2^-40 of
// itself, on its own columns and tiles only.  (Where the direct kernel's shorter
// reach is to be kept, wff_tc_local_kernel does such columns of a tile again.)
//
// One CTA of seven warpgroups per SM walks a list of (plane, 64 columns, Rw
// rows) tiles; the tile of R (Rw + 4s rows) stays in shared memory for all
// wy.  Per 32 rows (two K steps):
//   A  (2 x 4 warps)  R . e^{-j wy y}, split, tcgen05.st into an A1 slot
//   M  (2 warps)      pass 1: A1 x B into U; pass 2: A2 x B into C
//   B  (2 x 4 warps)  U from TMEM, threshold (in FP64 where it is close), split,
//                     into an A2 slot
//   C  (2 x 4 warps)  finished rows from TMEM, times e^{+j wy y}, into registers
// The operands never pass through shared memory: tcgen05.ld .16x256b and
// tcgen05.st .16x128b give a thread the same image column and the same rows
// on both sides, real part in lane i and imaginary in lane i + 8.
//
// TMEM holds all of a wy's rows of U and C (24 blocks of 16 columns) beside
// the operand slots; the windows are cut to the blocks in which a needed row
// lies.  A drained block is refilled with zeros, so every MMA accumulates, and
// each accumulator sees the same K steps in the same order whatever the tile:
// a row's bits do not depend on the tile height, the batch or a tile mask.
//
// Bound: instruction issue, and the waits between the stages.  At 1024^2, sigma
// 10, 21 x 21 frequencies the sweep takes 1.49 ms (the FFT sweep 3.18): 3.0
// instructions a clock per SM, 76% of the issue slots, about 170 per 16 x 64 block, wy
// and pass for the splitting and thresholding, a quarter of them waiting; tensor pipe
// 30%.  In an earlier form of 1.39 ms, with nearly all of A's, B's and C's arithmetic
// taken out 1.0 was left: the chain slot, MMAs, commit, next slot.  A third A warpgroup, up to four A1 slots, filling a slot in
// halves, skipping empty blocks and sleeping waits each left the time as it was
// or made it longer.  The MMAs alone would take 0.5 ms (N/2 cycles each at M =
// 128, K = 16, A in TMEM); the DRAM is at 3%.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include <cuda_fp16.h>

#include "glsu_internal.cuh"
#include "ptx_sm103.cuh"
#include "wff_common.cuh"

namespace glsu {
namespace {

constexpr int kBlocks = 24;       // blocks of 16 TMEM columns for the accumulators U and C
constexpr int kCols = 64;         // image columns per CTA
constexpr int kChunkRows = 64;    // rows of R per TMA chunk
constexpr int kMaxChunks = 6;     // 384 rows of R in shared memory
constexpr int kPhRing = 4;        // wy phasor tables in flight
constexpr int kPhPairs = kMaxChunks * kChunkRows / 2;
constexpr int kPairs = 8;         // pairs of blocks of either
// Half-sizes.  Error against 64 bits over that of the FFT sweep, median of 15 to 24
// fields (sigma = half-size / 3, thresholds 0.1 to 0.5, unit modulus and not): 0.75 to
// 0.99 up to 31, 0.97 to 1.07 from 32 to 42, 1.2 at 45 and 48 (large fields are closer:
// values near the threshold decide there, see kThrBand); over the direct kernel's 1.1 to
// 1.45 at 3 to 20, where that is 0.6 to 1.0e-7 of the norm.
constexpr int kMaxTcHalf = 48;
constexpr int kMaxN = 112;
static_assert(16 * kBlocks + 2 * 2 * 32 <= 512, "TMEM columns");
constexpr int kChunkBytes = kChunkRows * kCols * 8;
constexpr int kPhBytes = kPhPairs * 16;
constexpr int kMaxTapBytes = 2 * kMaxN * 32;  // hi and lo B operands
constexpr int kTapShift = 6;                // taps scaled by 2^6
constexpr int kScaleBytes = 6 * kCols * 4;  // column scales of two tiles; column maxima and smallest block maxima
constexpr int kSmem = kMaxChunks * kChunkBytes + kPhRing * kPhBytes + kMaxTapBytes + 768 + kScaleBytes + 1024;
static_assert(kSmem <= 227 * 1024, "column tile exceeds shared memory");

// One sequence of the sweep.
struct TcSeq {
    CUtensorMap tm;      // R: {4 pitch floats, row pairs, planes}
    const float4 *ey2;   // phasors of row pairs, [nfy][eys2], kTcPad pairs of padding in front
    float2 *C;
    const float *thr;
    const float *kr;     // scale that R carries
    uint8_t *wide;       // per tile and column: its values' range is wide (nullptr: not asked for)
    const float *R;      // the planes that tm maps, [plane][row pair][pitch](re, re', im, im')
    double thr_exact;    // thr_mul without what the accumulation's truncation takes
    int H, W, pitch, nfy, eys2, ncg, nty, item0;
    float thr_mul, out_mul;
};
template <int NS> struct TcTable {
    TcSeq seq[NS];
};
constexpr int kTcPad = 64;  // row pairs of padding in front of a phasor table

// Geometry of one tile.  R row of pass-1 step q: ra + 16 q; U row of block p:
// ra - s + 16 p; C row of block p: y0 + 16 (p - m).
struct TcTile {
    int plane, x0, y0, ra, q0, q1, p0, p1, nc;
};

__device__ __forceinline__ int fdiv16(int v) { return v >> 4; }  // floor

__device__ __forceinline__ TcTile tc_tile(const TcSeq &q, int plane, int g, int ty, int s, int m, int rw)
{
    TcTile t;
    t.plane = plane;
    t.x0 = g * kCols;
    t.y0 = ty * rw;
    t.ra = t.y0 + 2 * s - 16 * m;
    const int y1 = min(t.y0 + rw, q.H);
    // steps go in pairs, the small products of both first: pairs start at the same image rows in every tile
    t.q0 = fdiv16(max(0, t.y0 - 2 * s) - t.ra) & ~1;
    t.q1 = fdiv16(min(q.H, y1 + 2 * s) - t.ra + 15);
    const int pi = fdiv16(16 * m - 2 * s);  // p0 of a tile inside the image
    t.p0 = pi + ((fdiv16(max(0, t.y0 - s) - t.ra + s) - pi) & ~1);
    t.p1 = fdiv16(min(q.H, y1 + s) - t.ra + s + 15);
    t.nc = (y1 - t.y0 + 15) >> 4;
    return t;
}

// The products of one K step (A hi at TMEM column a, lo at a + 8) into the
// accumulators at d: the two small ones, or hi.hi.  One asm statement with its own
// elect, in code that a whole warp walks with warp-uniform operands: 3 MMAs with a
// wait before them then issue in 190 cycles; with an elected thread walking the same
// loop it is 305.
__device__ __forceinline__ void umma_cross(uint32_t d, uint32_t a, uint64_t bhi, uint64_t blo, uint32_t idesc)
{
    asm volatile(
        "{\n\t.reg .pred p, e;\n\t.reg .b32 alo;\n\t"
        "elect.sync _|e, 0xffffffff;\n\tsetp.ne.b32 p, 1, 0;\n\tadd.u32 alo, %1, 8;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [alo], %2, %4, p;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %3, %4, p;\n\t}" ::"r"(d),
        "r"(a), "l"(bhi), "l"(blo), "r"(idesc)
        : "memory");
}
__device__ __forceinline__ void umma_main(uint32_t d, uint32_t a, uint64_t bhi, uint32_t idesc)
{
    asm volatile(
        "{\n\t.reg .pred p, e;\n\telect.sync _|e, 0xffffffff;\n\tsetp.ne.b32 p, 1, 0;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d),
        "r"(a), "l"(bhi), "r"(idesc)
        : "memory");
}
// The same by a whole warp: arrive on bar when the MMAs that its elected thread issued have completed.
__device__ __forceinline__ void umma_commit_warp(uint64_t *bar)
{
    asm volatile(
        "{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\t"
        "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes, uint64_t *bar)
{
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

// 16 lanes x 16 columns: r[4j + {0,1}] rows (lanes) t/4, columns 8j + 2(t%4) + {0,1}; r[4j + {2,3}] lane t/4 + 8.
__device__ __forceinline__ void tmem_ld_16x256b_x2(uint32_t a, float *r)
{
    uint32_t u[8];
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7])
                 : "r"(a));
#pragma unroll
    for (int i = 0; i < 8; i++) r[i] = __uint_as_float(u[i]);
}
// 16 lanes x 16 columns: r[2j] lane t/4, column 4j + t%4; r[2j + 1] lane t/4 + 8.
__device__ __forceinline__ void tmem_st_16x128b_x4(uint32_t a, const uint32_t *r)
{
    asm volatile("tcgen05.st.sync.aligned.16x128b.x4.b32 [%8], {%0,%1,%2,%3,%4,%5,%6,%7};" ::"r"(r[0]), "r"(r[1]),
                 "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(a)
                 : "memory");
}
__device__ __forceinline__ void tmem_zero16(uint32_t a)
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1};" ::"r"(a),
                 "r"(0)
                 : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// The loaded registers may be read only after the wait: tie them to it.
__device__ __forceinline__ void tie8(float *r)
{
    asm volatile("" : "+f"(r[0]), "+f"(r[1]), "+f"(r[2]), "+f"(r[3]), "+f"(r[4]), "+f"(r[5]), "+f"(r[6]), "+f"(r[7]));
}

template <int N> __device__ __forceinline__ void reg_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N> __device__ __forceinline__ void reg_dec()  // from 72
{
    if constexpr (N < 72) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
}

// v = (v.x, v.y) as FP16 pairs hi and lo (v.x in the lower half), hi rounded
// towards zero for v.x and, but for powers of two, away from it for v.y: of two
// neighbouring rows one lo has its value's sign and the other the opposite.  The
// tensor core cuts the products lo.g off below the accumulator's bits; of one sign
// down a smooth column those cuts add up (half-size 45, a constant column:
// 4.3e-7 of a pass with hi rounded to nearest, 1.3e-7 as here).
__device__ __forceinline__ void split2(float2 v, uint32_t &hi, uint32_t &lo)
{
    __half2 h;
    asm("cvt.rz.f16x2.f32 %0, %1, %2;" : "=r"(*reinterpret_cast<uint32_t *>(&h)) : "f"(v.y), "f"(v.x));
    h = __hfma2(h, __halves2half2(__ushort_as_half(0), __ushort_as_half(0x1000)), h);  // (1, 1 + 2^-11)
    const float2 hf = __half22float2(h);
    const float2 d = __ffma2_rn(hf, make_float2(-1.f, -1.f), v);
    const __half2 l = __floats2half2_rn(d.x, d.y);
    hi = *reinterpret_cast<const uint32_t *>(&h);
    lo = *reinterpret_cast<const uint32_t *>(&l);
}

__device__ __forceinline__ float finite_abs(float v)
{
    const float a = fabsf(v);
    return a <= 3.402823466e38f ? a : 0.f;
}
// A column of a tile is wide where its largest value passes that of one of its
// 16-row blocks by more: what the parts drop (2^-40 of the largest) is then more than
// 2^-24 of that block.  Wide too is one with a value that is not finite.
constexpr float kWide = 65536.f;
// The power of two by which a column of R whose parts' largest magnitude is mx is multiplied: its
// values times a phasor then stay below 2^15.
__device__ __forceinline__ float column_scale(float mx)
{
    const int e = (int)(__float_as_uint(mx * 1.4143f) >> 23) - 126;  // below 2^e
    return mx > 0.f ? __uint_as_float((uint32_t)(127 + min(100, 15 - e)) << 23) : 1.f;
}
__device__ __forceinline__ float reciprocal_pow2(float k)
{
    return __uint_as_float((254u << 23) - __float_as_uint(k));
}

struct TcBars {
    uint64_t rfull[kMaxChunks], rfree[kMaxChunks], phfull[kPhRing], phfree[kPhRing];
    uint64_t a1full[2], a1free[2], a2full[2], a2free[2];
    uint64_t ufull[kPairs], ufree[kPairs], cfull[kPairs], cfree[kPairs];  // per pair of blocks
    uint64_t kfull[2], kfree[2], rscaled;  // column scales, R scaled by them
    uint64_t drain;
    uint32_t tmem;
};
static_assert(sizeof(TcBars) <= 768, "barriers");

// Whether U at image row y, column x, frequency k reaches the threshold, from R
// itself in FP64, for the values that lie within kThrBand of it, where the
// rounding of the split products would decide.  450 random fields against 64 bits,
// counted where one decision on the other side showed (error over 1e-6 and over
// 1.5 times the other sweep's): the FFT sweep 4, this one 2, those shared with the
// direct kernel; without the FP64 decisions 3 in 150.  They cost 4% of a frame
// (1024^2: 1662 -> 1734 us).  A whole warp works on one value, its taps over the
// lanes: one thread's loop over them made the sweep there 1.3 ms longer.  N, tb:
// the B operand's height and its place in shared memory (its first column is the
// taps).
constexpr float kThrBand = 1e-5f;  // of |U|^2
__device__ __forceinline__ bool tc_reaches(const TcSeq &q, const unsigned char *tb, int N, int s, int plane, int y,
                                           int x, int k, float kr)
{
    const float *R = q.R + ((size_t)plane * ((q.H + 1) >> 1) * q.pitch + x) * 4;
    const float *P = reinterpret_cast<const float *>(q.ey2 + (size_t)k * q.eys2 + kTcPad);
    const int r1 = min(q.H - 1, y + s);
    double sr = 0, si = 0;
#pragma unroll 1
    for (int r = max(0, y - s) + (threadIdx.x & 31); r <= r1; r += 32) {
        const float *e = R + (size_t)(r >> 1) * q.pitch * 4 + (r & 1), *c = P + (r >> 1) * 4 + (r & 1);
        const int n = y + s - r;
        const __half *g = reinterpret_cast<const __half *>(tb) + (n >> 3) * 128 + (n & 7) * 8;
        const double w = (double)__half2float(g[0]) + (double)__half2float(g[N * 16]);  // to 2^-24 of the largest
        const double re = e[0], im = e[2], pr = c[0], pi = c[2];
        sr += w * (re * pr - im * pi);
        si += w * (re * pi + im * pr);
    }
#pragma unroll 1
    for (int o = 16; o > 0; o >>= 1) {
        sr += __shfl_xor_sync(0xffffffffu, sr, o);
        si += __shfl_xor_sync(0xffffffffu, si, o);
    }
    const double thr = (double)*q.thr * q.thr_exact * (double)kr;
    return sr * sr + si * si >= thr * thr;
}

// The value of lane 0.
__device__ __forceinline__ int uniform(int v) { return __shfl_sync(0xffffffffu, v, 0); }

constexpr uint32_t kTcWaitCycles = 1u << 31;
// Bounded wait, the clock in 32 bits, as its copies in every role count towards the
// size of the code.  After a timeout (ok false) waits return at once: the roles then
// run to their ends, within their buffers, and the results are not used.
__device__ __forceinline__ void wait_ok(uint64_t *bar, uint32_t parity, bool &ok)
{
    if (!ok) return;
    const uint32_t t0 = (uint32_t)clock();
    while (!mbar_try_wait(bar, parity))
        if ((uint32_t)clock() - t0 > kTcWaitCycles) {
            ok = false;
            break;
        }
}

// The same with a warp-uniform verdict.
__device__ __forceinline__ void warp_wait(uint64_t *bar, uint32_t parity, bool &ok)
{
    if (!ok) return;
    bool w = true;
    wait_ok(bar, parity, w);
    ok = __all_sync(0xffffffffu, w);
}

// Seven warpgroups: loads and MMAs, two A, two B, two C.  A tile is RB pairs of
// 16-row blocks.  RM, RA, RT, RC: registers a thread of each kind keeps of the
// 72 at launch; the shares sum to the launch's.
template <int RB_, int RM_, int RA_, int RT_, int RC_> struct TcCfg {
    static constexpr int RB = RB_, RM = RM_, RA = RA_, RT = RT_, RC = RC_;
    static_assert(RM + 2 * (RA + RT + RC) <= 7 * 72, "register shares");
    static_assert(RM <= 72 && RA <= 72 && RT <= 72 && RC >= 72, "a share is given up or taken, not both");
};
constexpr int kThreads = 7 * 128;

// Walks the CTA's items: fills t and the sequence index; false past the end.
template <int NS>
__device__ __forceinline__ int tc_item(const TcTable<NS> &tab, int nseq, int item, const int2 *list, int listn, int s,
                                       int m, int rw, TcTile &t)
{
    int k = 0;
    if (NS > 1) {
        int hi = nseq - 1;  // the last sequence with item0 <= item
        while (k < hi) {
            const int mid = (k + hi + 1) >> 1;
            if (tab.seq[mid].item0 <= item) k = mid;
            else hi = mid - 1;
        }
    }
    const TcSeq &q = tab.seq[k];
    int local = item - q.item0;
    if (list) {
        const int2 e = list[local % listn];
        t = tc_tile(q, local / listn, e.x, e.y, s, m, rw);
    } else {
        const int g = local % q.ncg;
        local /= q.ncg;
        t = tc_tile(q, local / q.nty, g, local % q.nty, s, m, rw);
    }
    return k;
}

// UNIT: the row pass has scaled R (an input of unit modulus).
template <class Cfg, int NS, bool UNIT>
__global__ void __launch_bounds__(kThreads, 1)
    wff_tc_kernel(const __grid_constant__ TcTable<NS> tab, int nseq, int nitems_full, int s, int m, int N, float tscale,
                  const uint4 *__restrict__ taps, int *__restrict__ err, const int2 *__restrict__ list,
                  const int *__restrict__ list_count)
{
    constexpr int RB = Cfg::RB, RW = 32 * RB;
    extern __shared__ unsigned char sm_raw[];
    unsigned char *sm = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(sm_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char *Rs = sm;
    float4 *ph = reinterpret_cast<float4 *>(Rs + kMaxChunks * kChunkBytes);
    unsigned char *tb = reinterpret_cast<unsigned char *>(ph + kPhRing * kPhPairs);
    TcBars &bar = *reinterpret_cast<TcBars *>(tb + kMaxTapBytes);
    float(*kcol)[kCols] = reinterpret_cast<float(*)[kCols]>(tb + kMaxTapBytes + 768);  // of two tiles, in turns
    float(*kmax)[kCols] = kcol + 2, (*kmin)[kCols] = kcol + 4;  // by the two warpgroups that scale

    // by a shuffle, as everything that the operands of the tcgen05 instructions derive from
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31, wg = warp >> 2, w4 = warp & 3;
    const int nchunks = (RW + 16 * m + kChunkRows - 1) / kChunkRows;
    int nitems = nitems_full, listn = 0;
    if (list) {
        listn = *list_count;
        nitems = nitems_full * listn;  // nitems_full planes
    }
    if ((int)blockIdx.x >= nitems) return;  // uniform, before any barrier or allocation

    if (tid == 0) {
        for (int i = 0; i < kMaxChunks; i++) {
            mbar_init(&bar.rfull[i], 1);
            mbar_init(&bar.rfree[i], 8);
        }
        for (int i = 0; i < kPhRing; i++) {
            mbar_init(&bar.phfull[i], 1);
            mbar_init(&bar.phfree[i], 16);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(&bar.a1full[i], 4);
            mbar_init(&bar.a1free[i], 1);
            mbar_init(&bar.a2full[i], 4);
            mbar_init(&bar.a2free[i], 1);
        }
        for (int i = 0; i < kPairs; i++) {
            mbar_init(&bar.ufull[i], 1);
            mbar_init(&bar.ufree[i], i == 0 ? 8 : 4);  // pair 0: both B warpgroups
            mbar_init(&bar.cfull[i], 1);
            mbar_init(&bar.cfree[i], 8);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(&bar.kfull[i], 4);
            mbar_init(&bar.kfree[i], 8);
        }
        mbar_init(&bar.rscaled, 8);
        mbar_init(&bar.drain, 2);
        fence_mbar_init();
    }
    if (warp == 0) tmem_alloc(&bar.tmem, 512);
    for (int e = tid; e < N * 4; e += kThreads) reinterpret_cast<uint4 *>(tb)[e] = taps[e];  // hi, then lo
    fence_proxy_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, bar.tmem, 0);
    const uint32_t tU = tmem, tC = tmem + 16 * (kBlocks - 2 * RB), tA1 = tmem + 16 * kBlocks, tA2 = tA1 + 64;
    if (wg == 1) {
        for (int c = 0; c < 16 * kBlocks; c += 16) tmem_zero16(tmem + c + ((uint32_t)w4 << 21));
        tmem_wait_st();
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();

    // fragment coordinates: first row pair within a block, image column within 8
    const int frow = lane & 3, fi = lane >> 2, fcol = (fi >> 1) | ((fi & 1) << 2);
    const uint32_t lanes = (uint32_t)w4 << 21;
    bool ok = true;

    if (wg == 0) {
        reg_dec<Cfg::RM>();
        if (warp == 1 && elect_one()) {
            // ---- loads: R chunks of each tile, one phasor table per wy ----
            uint32_t nk = 0, nit = 0;
            for (int item = blockIdx.x; item < nitems; item += gridDim.x, nit++) {
                TcTile t;
                const TcSeq &q = tab.seq[tc_item<NS>(tab, nseq, item, list, listn, s, m, RW, t)];
                for (int ch = 0; ch < nchunks && ok; ch++) {
                    if (nit > 0) wait_ok(&bar.rfree[ch], (nit - 1) & 1, ok);
                    if (!ok) break;
                    if (4 * ch + 3 < t.q0 || 4 * ch >= t.q1) {
                        mbar_arrive(&bar.rfull[ch]);  // outside the image: not read
                        continue;
                    }
                    mbar_expect_tx(&bar.rfull[ch], kChunkBytes);
                    for (int p = 0; p < 8; p++)
                        tma_load_3d(Rs + ch * kChunkBytes + p * (kChunkBytes / 8), &q.tm, &bar.rfull[ch],
                                    (t.x0 + 8 * p) * 4, (t.ra >> 1) + ch * (kChunkRows / 2), t.plane);
                }
                const float4 *src = q.ey2 + kTcPad + (t.ra >> 1);
                for (int k = 0; k < q.nfy && ok; k++, nk++) {
                    const int b = nk % kPhRing;
                    if (nk >= kPhRing) wait_ok(&bar.phfree[b], ((nk / kPhRing) - 1) & 1, ok);
                    if (!ok) break;
                    mbar_expect_tx(&bar.phfull[b], kPhBytes);
                    bulk_load(ph + b * kPhPairs, src + (size_t)k * q.eys2, kPhBytes, &bar.phfull[b]);
                }
                if (!ok) break;
            }
            if (!ok) atomicExch(err, GLSU_ERR_TIMEOUT);
            // every load has landed before the CTA exits
            for (uint32_t j = nk > kPhRing ? nk - kPhRing : 0; j < nk; j++)
                mbar_wait_bounded(&bar.phfull[j % kPhRing], (j / kPhRing) & 1);
            if (!ok)
                for (int ch = 0; ch < nchunks; ch++) mbar_wait_bounded(&bar.rfull[ch], nit & 1);
        } else if (warp == 0 || warp == 2) {
            // ---- MMA issuers: pass 1 (warp 0) and pass 2 (warp 2) ----
            const int W = N >> 4;                           // blocks of a window
            const uint32_t idesc = (1u << 4) | (8u << 24);  // FP16 x FP16 -> FP32, M = 128; N / 8 goes to bit 17
            const uint64_t bhi = umma_desc(smem_u32(tb), 128, 256), blo = umma_desc(smem_u32(tb) + N * 32, 128, 256);
            auto issue = [&](const bool second, uint32_t tD, uint32_t tA, uint64_t *full, uint64_t *fre, uint64_t *afull,
                             uint64_t *afree) {
                uint32_t n = 0;                 // operand slots used
                uint32_t parity = 0, used = 0;  // per pair of blocks: parity of its next use, used before
                for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
                    TcTile t;
                    const int nfy = uniform(tab.seq[tc_item<NS>(tab, nseq, item, list, listn, s, m, RW, t)].nfy);
                    // steps from..to, outputs in blocks b0 .. b0 + nb
                    const int from = uniform(second ? t.p0 : t.q0), to = uniform(second ? t.p1 : t.q1);
                    const int b0 = second ? m : uniform(t.p0), nb = uniform(second ? t.nc : t.p1 - t.p0);
                    for (int k = 0; k < nfy; k++) {
                        int taken = 0, done = 0;  // pairs of blocks
                        for (int st = from; st < to; st += 2, n++) {
                            const uint32_t slot = n & 1;
                            const int nst = min(2, to - st), top = min(st + nst - 1 + W - b0, nb);
                            uint32_t d[2], off[2], id[2];
#pragma unroll
                            for (int h = 0; h < 2; h++) {
                                const int lo = max(st + h - b0, 0), hi = min(st + h + W - b0, nb);
                                off[h] = (uint32_t)(lo + b0 - st - h) * 32;  // 16 outputs: 512 bytes
                                d[h] = tD + 16 * lo;
                                id[h] = idesc | ((uint32_t)(hi - lo) << 18);
                            }
                            for (; 2 * taken < top; taken++)
                                if ((used >> taken) & 1) warp_wait(&fre[taken], ((parity >> taken) & 1) ^ 1, ok);
                            warp_wait(&afull[slot], (n >> 1) & 1, ok);
                            tc_fence_after();
                            // the small products of both steps, then the large ones
                            const uint32_t a = tA + 32 * slot;
                            umma_cross(d[0], a, bhi + off[0], blo + off[0], id[0]);
                            if (nst > 1) umma_cross(d[1], a + 16, bhi + off[1], blo + off[1], id[1]);
                            umma_main(d[0], a, bhi + off[0], id[0]);
                            if (nst > 1) umma_main(d[1], a + 16, bhi + off[1], id[1]);
                            umma_commit_warp(&afree[slot]);
                            // pairs with all their products
                            const int fin = st + 2 < to ? min(st + 2 - b0, nb) : nb;
                            for (; 2 * done + 1 < fin || (fin == nb && 2 * done < nb); done++)
                                umma_commit_warp(&full[done]);
                        }
                        const uint32_t mask = (1u << ((nb + 1) >> 1)) - 1;
                        parity ^= mask;
                        used |= mask;
                    }
                }
            };
            const bool p2 = warp == 2;
            issue(p2, p2 ? tC : tU, p2 ? tA2 : tA1, p2 ? bar.cfull : bar.ufull, p2 ? bar.cfree : bar.ufree,
                  p2 ? bar.a2full : bar.a1full, p2 ? bar.a2free : bar.a1free);
            if (!ok) atomicExch(err, GLSU_ERR_TIMEOUT);
            umma_commit_warp(&bar.drain);  // every MMA has completed before TMEM is released
            mbar_wait_bounded(&bar.drain, 0);
        }
    } else if (wg <= 2) {
        // ---- A: demodulate and split 32 rows of R per slot; each warpgroup its own slot ----
        reg_dec<Cfg::RA>();
        const uint32_t slot = wg - 1;
        const uint32_t a0 = tA1 + 32 * slot + lanes;
        const unsigned char *Rw = Rs + (2 * w4) * (kChunkBytes / 8) + frow * 128;
        uint32_t n = 0, mine = 0, nk = 0, nit = 0;  // n: slots used by both; mine: by this warpgroup
        for (int item = blockIdx.x; item < nitems; item += gridDim.x, nit++) {
            TcTile t;
            const int nfy = tab.seq[tc_item<NS>(tab, nseq, item, list, listn, s, m, RW, t)].nfy;
            if constexpr (UNIT) {
                for (int ch = t.q0 >> 2; ch <= (t.q1 - 1) >> 2; ch++) wait_ok(&bar.rfull[ch], nit & 1, ok);
            } else {
                wait_ok(&bar.rscaled, nit & 1, ok);
            }
            for (int k = 0; k < nfy; k++, nk++) {
                wait_ok(&bar.phfull[nk % kPhRing], (nk / kPhRing) & 1, ok);
                const float4 *P = ph + (nk % kPhRing) * kPhPairs + frow;
                for (int q = t.q0; q < t.q1; q += 2, n++) {
                    if ((n & 1) != slot) continue;
                    uint32_t o[2][8];
                    auto half = [&](int st) {
                        const unsigned char *base = Rw + (st >> 2) * kChunkBytes + (st & 3) * 1024;
#pragma unroll
                        for (int j = 0; j < 2; j++) {
                            const float4 p = P[8 * st + 4 * j];
                            const float2 px = make_float2(p.x, p.y), py = make_float2(p.z, p.w);
                            const float2 ny = __fmul2_rn(py, make_float2(-1.f, -1.f));
                            const int xo = (fcol ^ (4 * j + frow)) * 16 + 512 * j;
#pragma unroll
                            for (int h = 0; h < 2; h++) {
                                const float4 x = *reinterpret_cast<const float4 *>(base + h * (kChunkBytes / 8) + xo);
                                const float2 re = make_float2(x.x, x.y), im = make_float2(x.z, x.w);
                                const float2 dr = __ffma2_rn(im, ny, __fmul2_rn(re, px));
                                const float2 di = __ffma2_rn(im, px, __fmul2_rn(re, py));
                                split2(dr, o[h][2 * j], o[h][4 + 2 * j]);
                                split2(di, o[h][2 * j + 1], o[h][5 + 2 * j]);
                            }
                        }
                    };
                    half(q);
                    if (mine > 0) wait_ok(&bar.a1free[slot], (mine - 1) & 1, ok);
                    mine++;
                    tc_fence_after();
                    __syncwarp();
                    tmem_st_16x128b_x4(a0, o[0]);
                    tmem_st_16x128b_x4(a0 + (1u << 20), o[1]);
                    if (q + 1 < t.q1) {
                        half(q + 1);
                        tmem_st_16x128b_x4(a0 + 16, o[0]);
                        tmem_st_16x128b_x4(a0 + 16 + (1u << 20), o[1]);
                    }
                    tmem_wait_st();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&bar.a1full[slot]);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&bar.phfree[nk % kPhRing]);
            }
            if (lane == 0)
                for (int ch = 0; ch < nchunks; ch++) mbar_arrive(&bar.rfree[ch]);
        }
        if (!ok) atomicExch(err, GLSU_ERR_TIMEOUT);
    } else if (wg <= 4) {
        // ---- B: threshold and split the finished rows of U, 32 per slot ----
        reg_dec<Cfg::RT>();
        const uint32_t slot = wg - 3;
        const uint32_t a0 = tA2 + 32 * slot + lanes;
        const float2 ts = make_float2(tscale, tscale);
        uint32_t n = 0, mine = 0, parity = 0, nit = 0;
        for (int item = blockIdx.x; item < nitems; item += gridDim.x, nit++) {
            TcTile t;
            const TcSeq &q = tab.seq[tc_item<NS>(tab, nseq, item, list, listn, s, m, RW, t)];
            const int nfy = q.nfy, H = q.H, urow = t.ra - s + 2 * frow, nb = t.p1 - t.p0;
            const float kr = *q.kr, thr = *q.thr * q.thr_mul * kr;
            float thr2[2] = {thr, thr};  // of the thread's two columns
            if constexpr (!UNIT) {
                // scale the tile's columns in place, each by a power of two to at most 2^15; the steps in
                // turns between the warpgroups
                for (int ch = t.q0 >> 2; ch <= (t.q1 - 1) >> 2; ch++) wait_ok(&bar.rfull[ch], nit & 1, ok);
                unsigned char *Rm = Rs + (2 * w4) * (kChunkBytes / 8) + frow * 128;
                float mx[2] = {0.f, 0.f}, mn[2] = {3.402823466e38f, 3.402823466e38f};
#pragma unroll 1
                for (int st = t.q0 + (int)slot; st < t.q1; st += 2) {
                    float bm[2] = {0.f, 0.f};  // of the step's 16 rows
                    const unsigned char *base = Rm + (st >> 2) * kChunkBytes + (st & 3) * 1024;
#pragma unroll
                    for (int j = 0; j < 2; j++)
#pragma unroll
                        for (int h = 0; h < 2; h++) {
                            const float4 x = *reinterpret_cast<const float4 *>(base + h * (kChunkBytes / 8) +
                                                                               (fcol ^ (4 * j + frow)) * 16 + 512 * j);
                            bm[h] = fmaxf(fmaxf(bm[h], finite_abs(x.x)), finite_abs(x.y));
                            bm[h] = fmaxf(fmaxf(bm[h], finite_abs(x.z)), finite_abs(x.w));
                            if (!(isfinite(x.x) && isfinite(x.y) && isfinite(x.z) && isfinite(x.w))) mn[h] = 0.f;
                        }
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        bm[h] = fmaxf(bm[h], __shfl_xor_sync(0xffffffffu, bm[h], 1));
                        bm[h] = fmaxf(bm[h], __shfl_xor_sync(0xffffffffu, bm[h], 2));
                        mx[h] = fmaxf(mx[h], bm[h]);
                        if (bm[h] > 0.f) mn[h] = fminf(mn[h], bm[h]);
                    }
                }
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    mn[h] = fminf(mn[h], __shfl_xor_sync(0xffffffffu, mn[h], 1));
                    mn[h] = fminf(mn[h], __shfl_xor_sync(0xffffffffu, mn[h], 2));
                    if (frow == 0) {
                        kmax[slot][16 * w4 + 8 * h + fcol] = mx[h];
                        kmin[slot][16 * w4 + 8 * h + fcol] = mn[h];
                    }
                }
                asm volatile("bar.sync 1, 256;" ::: "memory");
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int c = 16 * w4 + 8 * h + fcol;
                    const float top = fmaxf(kmax[0][c], kmax[1][c]);
                    if (q.wide && slot == 0 && frow == 0)
                        q.wide[(size_t)item * kCols + c] = top > kWide * fminf(kmin[0][c], kmin[1][c]);
                    mx[h] = column_scale(top);
                }
#pragma unroll 1
                for (int st = t.q0 + (int)slot; st < t.q1; st += 2) {
                    unsigned char *base = Rm + (st >> 2) * kChunkBytes + (st & 3) * 1024;
#pragma unroll
                    for (int j = 0; j < 2; j++)
#pragma unroll
                        for (int h = 0; h < 2; h++) {
                            float4 &x = *reinterpret_cast<float4 *>(base + h * (kChunkBytes / 8) +
                                                                    (fcol ^ (4 * j + frow)) * 16 + 512 * j);
                            x = make_float4(x.x * mx[h], x.y * mx[h], x.z * mx[h], x.w * mx[h]);
                        }
                }
                fence_proxy_async_smem();  // the scaled values before a later tile's loads over them
                if (slot == 0) {
                    if (nit >= 2) wait_ok(&bar.kfree[nit & 1], ((nit >> 1) - 1) & 1, ok);
                    if (frow == 0) {
                        kcol[nit & 1][16 * w4 + fcol] = mx[0];
                        kcol[nit & 1][16 * w4 + 8 + fcol] = mx[1];
                    }
                }
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(&bar.rscaled);
                    if (slot == 0) mbar_arrive(&bar.kfull[nit & 1]);
                }
                thr2[0] *= mx[0];
                thr2[1] *= mx[1];
            }
            thr2[0] *= thr2[0];
            thr2[1] *= thr2[1];
            for (int k = 0; k < nfy; k++) {
                for (int i = 0; 2 * i < nb; i++, n++) {
                    if ((n & 1) != slot) {
                        // Where a wy has one pair only, this warpgroup waits for nothing of it: it
                        // follows the pair by its phase, which it holds until it has seen it.
                        if (i == 0) {
                            wait_ok(&bar.ufull[0], parity & 1, ok);
                            __syncwarp();
                            if (lane == 0) mbar_arrive(&bar.ufree[0]);
                        }
                        continue;
                    }
                    wait_ok(&bar.ufull[i], (parity >> i) & 1, ok);
                    tc_fence_after();
                    __syncwarp();
                    uint32_t o[2][8];
                    auto half = [&](int blk) {
                        const uint32_t u = tU + 16 * blk + lanes;
                        float r[2][8];
                        tmem_ld_16x256b_x2(u, r[0]);
                        tmem_ld_16x256b_x2(u + (1u << 20), r[1]);
                        tmem_wait_ld();
                        tie8(r[0]);
                        tie8(r[1]);
                        tmem_zero16(u);
                        const int row = urow + 16 * (t.p0 + blk);
                        float2 a[2][2];
                        float near[2] = {3.402823466e38f, 3.402823466e38f};
#pragma unroll
                        for (int j = 0; j < 2; j++)
#pragma unroll
                            for (int h = 0; h < 2; h++) {
                                const float2 re = make_float2(r[h][4 * j], r[h][4 * j + 1]);
                                const float2 im = make_float2(r[h][4 * j + 2], r[h][4 * j + 3]);
                                a[j][h] = __ffma2_rn(im, im, __fmul2_rn(re, re));
                                const float2 d = __fadd2_rn(a[j][h], make_float2(-thr2[h], -thr2[h]));
                                near[h] = fminf(near[h], fminf(fabsf(d.x), fabsf(d.y)));
                            }
                        if (__any_sync(0xffffffffu, near[0] < kThrBand * thr2[0] || near[1] < kThrBand * thr2[1])) {
                            // what lies too near is decided in FP64, value by value
#pragma unroll 1
                            for (int e = 0; e < 8; e++) {
                                const int j = e >> 2, h = (e >> 1) & 1;
                                const float2 v = j ? (h ? a[1][1] : a[1][0]) : (h ? a[0][1] : a[0][0]);
                                const int y = row + 8 * j + (e & 1), x = t.x0 + 16 * w4 + 8 * h + fcol;
                                const float th = h ? thr2[1] : thr2[0];
                                const bool mine_ = fabsf((e & 1 ? v.y : v.x) - th) < kThrBand * th &&
                                                   (unsigned)y < (unsigned)H && x < q.W;
                                uint32_t todo = __ballot_sync(0xffffffffu, mine_);
                                bool over = false;
                                while (todo) {
                                    const int src = __ffs(todo) - 1;
                                    todo &= todo - 1;
                                    const bool o1 = tc_reaches(q, tb, N, s, t.plane, __shfl_sync(0xffffffffu, y, src),
                                                               __shfl_sync(0xffffffffu, x, src), k, kr);
                                    if (lane == src) over = o1;
                                }
                                const float f = over ? 3.402823466e38f : -1.f;
#pragma unroll
                                for (int c = 0; c < 4; c++) {
                                    if (mine_ && e == 2 * c) a[c >> 1][c & 1].x = f;
                                    if (mine_ && e == 2 * c + 1) a[c >> 1][c & 1].y = f;
                                }
                            }
                        }
#pragma unroll
                        for (int j = 0; j < 2; j++) {
                            const int y = row + 8 * j;  // rows outside the image carry no T
                            const bool in0 = (unsigned)y < (unsigned)H, in1 = (unsigned)(y + 1) < (unsigned)H;
#pragma unroll
                            for (int h = 0; h < 2; h++) {
                                float2 re = make_float2(r[h][4 * j], r[h][4 * j + 1]);
                                float2 im = make_float2(r[h][4 * j + 2], r[h][4 * j + 3]);
                                const bool k0 = in0 && a[j][h].x >= thr2[h], k1 = in1 && a[j][h].y >= thr2[h];
                                re = make_float2(k0 ? re.x : 0.f, k1 ? re.y : 0.f);
                                im = make_float2(k0 ? im.x : 0.f, k1 ? im.y : 0.f);
                                split2(__fmul2_rn(re, ts), o[h][2 * j], o[h][4 + 2 * j]);
                                split2(__fmul2_rn(im, ts), o[h][2 * j + 1], o[h][5 + 2 * j]);
                            }
                        }
                        __syncwarp();
                    };
                    // one body for both halves: every SM sub-partition runs all roles, and the time follows the
                    // size of their code together (a 1024^2 frame by the kernel's size in KB: 60 1.75 ms,
                    // 71 1.79, 77 1.92, 84 2.17)
#pragma unroll 1
                    for (int hb = 0; hb < 2 && 2 * i + hb < nb; hb++) {
                        half(2 * i + hb);
                        if (hb == 0) {
                            if (mine > 0) wait_ok(&bar.a2free[slot], (mine - 1) & 1, ok);
                            mine++;
                            tc_fence_after();
                        }
                        __syncwarp();
                        tmem_st_16x128b_x4(a0 + 16 * hb, o[0]);
                        tmem_st_16x128b_x4(a0 + 16 * hb + (1u << 20), o[1]);
                    }
                    tmem_wait_st();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        mbar_arrive(&bar.a2full[slot]);
                        mbar_arrive(&bar.ufree[i]);
                    }
                }
                parity ^= (1u << ((nb + 1) >> 1)) - 1;
            }
        }
        if (!ok) atomicExch(err, GLSU_ERR_TIMEOUT);
    } else {
        // ---- C: modulate and sum the finished rows over wy; one block of each pair per warpgroup ----
        reg_inc<Cfg::RC>();
        const int par = wg - 5;
        uint32_t nk = 0, parity = 0, nit = 0;
        for (int item = blockIdx.x; item < nitems; item += gridDim.x, nit++) {
            TcTile t;
            const TcSeq &q = tab.seq[tc_item<NS>(tab, nseq, item, list, listn, s, m, RW, t)];
            const int nfy = q.nfy, poff = ((t.y0 - t.ra) >> 1) + frow;
            float2 are[RB][2][2], aim[RB][2][2];
#pragma unroll
            for (int c = 0; c < RB; c++)
#pragma unroll
                for (int e = 0; e < 4; e++) are[c][e >> 1][e & 1] = aim[c][e >> 1][e & 1] = make_float2(0.f, 0.f);
            for (int k = 0; k < nfy; k++, nk++) {
                const float4 *P = ph + (nk % kPhRing) * kPhPairs + poff;
                wait_ok(&bar.phfull[nk % kPhRing], (nk / kPhRing) & 1, ok);
#pragma unroll
                for (int c = 0; c < RB; c++) {
                    if (2 * c < t.nc) {
                        wait_ok(&bar.cfull[c], (parity >> c) & 1, ok);
                        tc_fence_after();
                        __syncwarp();
                        if (2 * c + par < t.nc) {
                            const uint32_t u = tC + 16 * (2 * c + par) + lanes;
                            float r[2][8];
                            tmem_ld_16x256b_x2(u, r[0]);
                            tmem_ld_16x256b_x2(u + (1u << 20), r[1]);
                            tmem_wait_ld();
                            tie8(r[0]);
                            tie8(r[1]);
                            tmem_zero16(u);
#pragma unroll
                            for (int j = 0; j < 2; j++) {
                                const float4 p = P[8 * (2 * c + par) + 4 * j];
                                const float2 px = make_float2(p.x, p.y), py = make_float2(p.z, p.w);
                                const float2 ny = __fmul2_rn(py, make_float2(-1.f, -1.f));
#pragma unroll
                                for (int h = 0; h < 2; h++) {
                                    const float2 re = make_float2(r[h][4 * j], r[h][4 * j + 1]);
                                    const float2 im = make_float2(r[h][4 * j + 2], r[h][4 * j + 3]);
                                    are[c][h][j] = __ffma2_rn(px, re, __ffma2_rn(py, im, are[c][h][j]));
                                    aim[c][h][j] = __ffma2_rn(px, im, __ffma2_rn(ny, re, aim[c][h][j]));
                                }
                            }
                            tmem_wait_st();
                        }
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&bar.cfree[c]);
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&bar.phfree[nk % kPhRing]);
                parity ^= (1u << ((t.nc + 1) >> 1)) - 1;
            }
            const float mul = q.out_mul / *q.kr;
            float inv[2] = {1.f, 1.f};  // of the columns' scales
            if constexpr (!UNIT) {
                const uint32_t b = nit & 1;
                wait_ok(&bar.kfull[b], (nit >> 1) & 1, ok);
                inv[0] = reciprocal_pow2(kcol[b][16 * w4 + fcol]);
                inv[1] = reciprocal_pow2(kcol[b][16 * w4 + 8 + fcol]);
                __syncwarp();
                if (lane == 0) mbar_arrive(&bar.kfree[b]);
            }
            float2 *Cp = q.C + (size_t)t.plane * q.H * q.pitch + t.x0 + 16 * w4 + fcol;
#pragma unroll
            for (int c = 0; c < RB; c++)
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    const int y = t.y0 + 16 * (2 * c + par) + 8 * j + 2 * frow;
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const float2 re = are[c][h][j], im = aim[c][h][j];
                        if (y < q.H)
                            Cp[(size_t)y * q.pitch + 8 * h] = make_float2(re.x * mul * inv[h], im.x * mul * inv[h]);
                        if (y + 1 < q.H)
                            Cp[(size_t)(y + 1) * q.pitch + 8 * h] = make_float2(re.y * mul * inv[h], im.y * mul * inv[h]);
                    }
                }
        }
        if (!ok) atomicExch(err, GLSU_ERR_TIMEOUT);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) tmem_dealloc(tmem, 512);
}

// The wide columns of a tile once more, directly in FP32 from R, as the direct
// column kernel does them: a value then acts on the 2s rows around it only.  Runs
// where AUTO would take the direct kernel but for this file (WffPlan::tc_local) and
// the input is not of unit modulus.  With no wide column, the rule on measured fields,
// it costs its launch.  A CTA takes four wide columns of a tile at a time, 64 threads
// each, four rows a thread (eight FMAs for a tap and a value read from shared memory).
// Whole calls, one pixel of 1e12 (direct kernel): 512 x 512 with sigma 3 0.40 ms (0.46),
// 733 x 1021 with sigma 5 0.77 (1.35); every column wide: 1.54 (0.46) and 2.65 (1.35),
// 2.85 and 5.05 with a column at a time and a row a thread.
constexpr int kLocalCols = 4, kLocalThreads = 64 * kLocalCols;

// Element i of D and T stands at local_at(i): threads four rows apart then meet no bank twice.
__device__ __forceinline__ int local_at(int i) { return i + (i >> 2); }

// Four outputs i0 .. i0 + 3, i0 = 4 lt, of sum_j g[j] v[i + j], j = 0 .. 2s; taps beyond the window do not
// meet a value (0 times NaN), and v is readable to i0 + 2s + 3.
__device__ __forceinline__ void local_filter4(const float *g, const float2 *v, int s, int lt, float2 (&u)[4])
{
    v += 5 * lt;
#pragma unroll
    for (int r = 0; r < 4; r++) u[r] = make_float2(0.f, 0.f);
    const auto edge = [&](int j) {
        const float2 x = v[local_at(j)];
#pragma unroll
        for (int r = 0; r < 4; r++)
            if (j >= r && j - r <= 2 * s) u[r] = make_float2(fmaf(g[j - r], x.x, u[r].x), fmaf(g[j - r], x.y, u[r].y));
    };
    for (int j = 0; j < 3; j++) edge(j);
    if (s < 2) {
        for (int j = 3; j < 2 * s + 4; j++) edge(j);
        return;
    }
    float t1 = g[2], t2 = g[1], t3 = g[0];
#pragma unroll 4
    for (int j = 3; j <= 2 * s; j++) {
        const float2 x = v[local_at(j)];
        const float t0 = g[j];
        u[0] = make_float2(fmaf(t0, x.x, u[0].x), fmaf(t0, x.y, u[0].y));
        u[1] = make_float2(fmaf(t1, x.x, u[1].x), fmaf(t1, x.y, u[1].y));
        u[2] = make_float2(fmaf(t2, x.x, u[2].x), fmaf(t2, x.y, u[2].y));
        u[3] = make_float2(fmaf(t3, x.x, u[3].x), fmaf(t3, x.y, u[3].y));
        t3 = t2;
        t2 = t1;
        t1 = t0;
    }
    for (int j = 2 * s + 1; j < 2 * s + 4; j++) edge(j);
}

__global__ void __launch_bounds__(kLocalThreads, 4) wff_tc_local_kernel(const __grid_constant__ TcTable<1> tab, int nitems,
                                                                     int s, int m, int rw,
                                                                     const __grid_constant__ Taps<float, 60> gA,
                                                                     const __grid_constant__ Taps<float, 60> gB)
{
    constexpr int kRows = kMaxChunks * kChunkRows + 4, kRowsT = 260 + 2 * kMaxTcHalf;
    __shared__ float2 Rc[kLocalCols][kRows], D[kLocalCols][kRows + kRows / 4], T[kLocalCols][kRowsT + kRowsT / 4];
    __shared__ float a[2 * kMaxTcHalf + 1], b[2 * kMaxTcHalf + 1];
    const TcSeq &q = tab.seq[0];
    const int tid = threadIdx.x, grp = tid >> 6, lt = tid & 63;
    for (int j = tid; j <= 2 * s; j += kLocalThreads) {
        a[j] = gA.g[60 - s + j];
        b[j] = gB.g[60 - s + j];
    }
    const float thr = *q.thr, thr2 = thr * thr;
    const int pairs = (q.H + 1) >> 1;
    constexpr int kLook = kLocalThreads / 16;  // items whose 64 flags are looked at together
    for (int first = blockIdx.x; first < nitems; first += kLook * gridDim.x) {
        const int mine = first + (tid >> 4) * gridDim.x;
        const bool some =
            mine < nitems && reinterpret_cast<const uint32_t *>(q.wide)[(size_t)mine * (kCols / 4) + (tid & 15)];
        if (!__syncthreads_or(some)) continue;
        for (int item = first, n = 0; n < kLook && item < nitems; n++, item += gridDim.x) {
            const uint8_t *flag = q.wide + (size_t)item * kCols + (tid & 31);
            // the same in every warp
            uint64_t todo = __ballot_sync(0xffffffffu, flag[0]) | (uint64_t)__ballot_sync(0xffffffffu, flag[32]) << 32;
            if (!todo) continue;
            TcTile t;
            tc_item<1>(tab, 1, item, nullptr, 0, s, m, rw, t);
            if (q.W - t.x0 < kCols) todo &= (1ull << (q.W - t.x0)) - 1;
            const int y1 = min(t.y0 + rw, q.H), nu = y1 - t.y0 + 2 * s, nr = nu + 2 * s;
            while (todo) {
                int c = -1;  // the group's column
                for (int g = 0; g < kLocalCols; g++) {
                    if (g == grp && todo) c = __ffsll((long long)todo) - 1;
                    todo &= todo - 1;
                }
                const float *R = q.R + ((size_t)t.plane * pairs * q.pitch + t.x0 + max(c, 0)) * 4;
                for (int i = lt; i < nr + 3 && c >= 0; i += 64) {
                    const int y = t.y0 - 2 * s + i;
                    const float *e = R + (size_t)(y >> 1) * q.pitch * 4 + (y & 1);
                    Rc[grp][i] = (unsigned)y < (unsigned)q.H && i < nr ? make_float2(e[0], e[2]) : make_float2(0.f, 0.f);
                }
                float2 acc[4];  // of rows t.y0 + 4 lt ..: rw <= 256
#pragma unroll
                for (int r = 0; r < 4; r++) acc[r] = make_float2(0.f, 0.f);
                for (int k = 0; k < q.nfy; k++) {
                    const float *P = reinterpret_cast<const float *>(q.ey2 + (size_t)k * q.eys2 + kTcPad);
                    for (int i = lt; i < nr + 3 && c >= 0; i += 64) {
                        // rows outside the image are zeros times some row's phasor
                        const int y = min(max(t.y0 - 2 * s + i, 0), q.H - 1);
                        const float *p = P + (y >> 1) * 4 + (y & 1);
                        const float2 r = Rc[grp][i];
                        D[grp][local_at(i)] = make_float2(r.x * p[0] - r.y * p[2], r.x * p[2] + r.y * p[0]);
                    }
                    __syncthreads();
                    if (c >= 0 && 4 * lt < nu) {
                        float2 u[4];
                        local_filter4(a, D[grp], s, lt, u);
#pragma unroll
                        for (int r = 0; r < 4; r++) {
                            const int i = 4 * lt + r, y = t.y0 - s + i;
                            const bool keep = i < nu && (unsigned)y < (unsigned)q.H &&
                                              u[r].x * u[r].x + u[r].y * u[r].y >= thr2;
                            T[grp][local_at(i)] = keep ? u[r] : make_float2(0.f, 0.f);
                        }
                    }
                    __syncthreads();
                    if (c >= 0 && t.y0 + 4 * lt < y1) {
                        float2 v[4];
                        local_filter4(b, T[grp], s, lt, v);
#pragma unroll
                        for (int r = 0; r < 4; r++) {
                            const int y = min(t.y0 + 4 * lt + r, q.H - 1);
                            const float *p = P + (y >> 1) * 4 + (y & 1);
                            acc[r].x += p[0] * v[r].x + p[2] * v[r].y;
                            acc[r].y += p[0] * v[r].y - p[2] * v[r].x;
                        }
                    }
                }
                __syncthreads();
                if (c >= 0)
#pragma unroll
                    for (int r = 0; r < 4; r++) {
                        const int y = t.y0 + 4 * lt + r;
                        if (y < y1) q.C[(size_t)t.plane * q.H * q.pitch + (size_t)y * q.pitch + t.x0 + c] = acc[r];
                    }
            }
        }
    }
}

// Tile heights (in pairs of blocks) whose accumulators fit the TMEM and whose
// rows of R fit the shared memory at half-size s, largest first.
int tc_row_blocks(int s, int *rb)
{
    int n = 0;
    for (int r : {5, 4, 2})
        if (4 * r + (s + 7) / 8 <= kBlocks && 32 * r + 16 * ((s + 3) / 4) <= kMaxChunks * kChunkRows) rb[n++] = r;
    return n;
}

// Steps (16 image rows through one of the two passes) of one tile and wy.
int tc_steps(int H, int s, int rw, int ty)
{
    const int y0 = ty * rw, y1 = std::min(H, y0 + rw);
    const int r = std::min(H, y1 + 2 * s) - std::max(0, y0 - 2 * s), u = std::min(H, y1 + s) - std::max(0, y0 - s);
    return (r + 31) / 16 + (u + 31) / 16;
}

// A tap's FP16 parts, hi a multiple of 2^grain (the largest tap is 2^6).
void tap_parts(double g, int grain, __half &hi, __half &lo)
{
    g = std::ldexp(g, kTapShift);
    const double h = std::ldexp(std::nearbyint(std::ldexp(g, -grain)), grain);
    hi = __float2half((float)h);
    lo = __float2half((float)(g - h));
}

// The grain of the taps and what a pass then comes out smaller by, of itself.  The
// tensor core adds the 16 products of an MMA and the accumulator in fixed point,
// cutting each off (towards zero) two bits below the last of the largest's 24, and
// cuts the sum off to 24 bits: with that this reproduces measured sweeps to 4e-8,
// FP32's rounding of the output.  A coarse hi leaves hi.hi no bits below those the
// accumulator keeps, but grows lo; how that falls out depends on the window, so the
// better of two grains is taken (-5 keeps the largest tap within 11 bits).  Data: real
// parts of waves from the window's centre frequency to 1.2 / sigma off it, without and
// with noise, amplitudes over a power of two.  Bit patterns instead of half and math
// functions, as this runs at a handle's creation (half-size 30: 1.3 ms, 48: 1.9).
int tc_pass_grain(const double *gy, int s, double &shrink)
{
    constexpr int kGrains = 2, kGrain[kGrains] = {-4, -5};
    const auto bits = [](double x) {
        uint64_t u;
        std::memcpy(&u, &x, 8);
        return u;
    };
    const auto of_bits = [](uint64_t u) {
        double x;
        std::memcpy(&x, &u, 8);
        return x;
    };
    const auto exponent = [&](double x) { return (int)((bits(x) >> 52) & 2047) - 1023; };
    const auto pow2 = [&](int e) { return of_bits((uint64_t)(e + 1023) << 52); };
    const auto to11 = [&](double x) {  // nearest with 11 bits
        const double c = 1.5 * pow2(exponent(x) + 42);
        return x == 0 ? 0 : (x + c) - c;
    };
    const int taps = 2 * s + 1;
    std::vector<double> g(taps), ghi[kGrains], glo[kGrains], part[kGrains][3];  // part: lo.g, hi.g', hi.g
    for (int v = 0; v < kGrains; v++)
        for (int k = 0; k < taps; k++) {
            __half hi, lo;
            tap_parts(gy[k], kGrain[v], hi, lo);
            ghi[v].push_back(__half2float(hi));
            glo[v].push_back(__half2float(lo));
            g[k] = std::ldexp(gy[k], kTapShift);
        }
    uint64_t rng = 88172645463325252ull;
    const auto uniform = [&] {  // xorshift64
        rng ^= rng << 13;
        rng ^= rng >> 7;
        rng ^= rng << 17;
        return (double)(rng >> 11) * 0x1p-53;
    };
    double ee = 0, er[kGrains] = {}, rr[kGrains] = {};  // sums of exact^2, exact x loss, loss^2
    for (int n = 0; n < 384; n++) {
        const int off = n & 15, kind = (n >> 4) & 7, steps = (off + taps + 15) / 16;
        const double amp = std::exp2(9 + uniform()), phase = 2 * M_PI * uniform();
        const double slope = 0.4 * (kind & 3) * 3.0 / std::max(s, 1), noise = kind & 4 ? 4.0 : 0.0;
        const double cs = std::cos(slope), sn = std::sin(slope);
        double wr = amp * std::cos(phase), wi = amp * std::sin(phase), exact = 0;  // the wave, row by row
        for (auto &v : part)
            for (auto &p : v) p.assign((size_t)steps * 16, 0.0);
        for (int k = 0; k < taps; k++) {
            const double x = (float)(wr + noise * amp * (uniform() - 0.5));
            const double r = wr * cs - wi * sn;
            wi = wr * sn + wi * cs;
            wr = r;
            double h = of_bits(bits(x) & ~((1ull << 42) - 1));
            if (((off + k) & 1) && (bits(h) << 12)) h = of_bits(bits(h) + (1ull << 42));
            const double l = to11(x - h);
            for (int v = 0; v < kGrains; v++) {
                part[v][0][off + k] = l * ghi[v][k];
                part[v][1][off + k] = h * glo[v][k];
                part[v][2][off + k] = h * ghi[v][k];
            }
            exact += x * g[k];
        }
        ee += exact * exact;
        for (int v = 0; v < kGrains; v++) {
            double acc = 0;
            const auto mma = [&](const double *p) {
                double mx = std::fabs(acc), sum = 0;
                for (int k = 0; k < 16; k++) mx = std::max(mx, std::fabs(p[k]));
                if (mx == 0) return;
                const int e = exponent(mx) - 25;
                const double per = pow2(-e);
                for (int k = 0; k < 16; k++) sum += (double)(int64_t)(p[k] * per);
                sum = (sum + (double)(int64_t)(acc * per)) * pow2(e);
                const int f = exponent(sum) - 23;
                acc = sum == 0 ? 0 : (double)(int64_t)(sum * pow2(-f)) * pow2(f);
            };
            for (int q = 0; q < steps; q += 2) {
                const int q1 = std::min(q + 2, steps);
                for (int h = q; h < q1; h++) {
                    mma(&part[v][0][16 * h]);
                    mma(&part[v][1][16 * h]);
                }
                for (int h = q; h < q1; h++) mma(&part[v][2][16 * h]);
            }
            er[v] += exact * (exact - acc);
            rr[v] += (exact - acc) * (exact - acc);
        }
    }
    int best = 0;
    for (int v = 1; v < kGrains; v++)
        if (rr[v] - er[v] * er[v] / ee < rr[best] - er[best] * er[best] / ee) best = v;
    shrink = er[best] / ee;
    return kGrain[best];
}

// Modelled cost of a sweep of these plans with 32 rb-row tiles, in steps of
// the busiest SM: half whole rounds of mean tiles (tiles are dealt out round robin, so
// a few more than the SMs cost a round), half an even share, as tiles at the image's
// ends are short and let their SM go ahead.  Over nine shapes (200 x 300 to 1024^2,
// sigma 5 to 15) the height with the least cost took the least time of 5, 4 and 2 or
// up to 2% more: 1024^2, sigma 10 1503, 1556 and 2183 us; 256^2 184, 178 and 190;
// 733 x 1021, sigma 7 418, 459 and 575; 384 x 512 356, 348 and 427 with equal costs.
double tc_cost(const WffPlan *const *plans, int n, int rb, int sms)
{
    double total = 0, items = 0, mx = 0;
    for (int k = 0; k < n; k++) {
        const WffPlan &P = *plans[k];
        const int nty = (P.H + 32 * rb - 1) / (32 * rb), ncg = (P.W + kCols - 1) / kCols;
        for (int ty = 0; ty < nty; ty++) {
            const double st = (double)tc_steps(P.H, P.sy, 32 * rb, ty) * P.nfy;
            total += st * ncg * P.nfx;
            mx = std::max(mx, st);
        }
        items += (double)nty * ncg * P.nfx;
    }
    return std::ceil(items / sms) * (total / items) * 0.5 + std::max(total / sms, mx) * 0.5;
}

using Tc5 = TcCfg<5, 40, 48, 72, 112>;
using Tc4 = TcCfg<4, 40, 56, 72, 104>;
using Tc2 = TcCfg<2, 40, 64, 72, 88>;

template <class Cfg, int NS, bool UNIT>
int tc_launch(const TcTable<NS> &tab, int nseq, int nitems, int grid, const WffPlan &P, const int2 *list,
              const int *count, cudaStream_t s)
{
    GLSU_TRY(raise_smem_limit((const void *)wff_tc_kernel<Cfg, NS, UNIT>, kSmem));
    const int N = (2 * P.sy + 16 + 15) / 16 * 16;
    wff_tc_kernel<Cfg, NS, UNIT><<<grid, kThreads, kSmem, s>>>(tab, nseq, nitems, P.sy, (P.sy + 3) / 4, N,
                                                              P.tc_tscale, (const uint4 *)P.d_tctaps, P.d_err, list,
                                                              count);
    GLSU_CUDA_TRY(cudaGetLastError());
    return GLSU_OK;
}

template <int NS, bool UNIT>
int tc_launch_rb(int rb, const TcTable<NS> &tab, int nseq, int nitems, int grid, const WffPlan &P, const int2 *list,
                 const int *count, cudaStream_t s)
{
    switch (rb) {
    case 5: return tc_launch<Tc5, NS, UNIT>(tab, nseq, nitems, grid, P, list, count, s);
    case 4: return tc_launch<Tc4, NS, UNIT>(tab, nseq, nitems, grid, P, list, count, s);
    default: return tc_launch<Tc2, NS, UNIT>(tab, nseq, nitems, grid, P, list, count, s);
    }
}

int tc_launch_one(int rb, const TcTable<1> &tab, int nitems, int grid, const WffPlan &P, const int2 *list,
                  const int *count, cudaStream_t s)
{
    return P.unit_input ? tc_launch_rb<1, true>(rb, tab, 1, nitems, grid, P, list, count, s)
                        : tc_launch_rb<1, false>(rb, tab, 1, nitems, grid, P, list, count, s);
}

void tc_seq(TcSeq &q, const WffPlan &P, int rw, int item0)
{
    q.tm = P.tmT;
    q.ey2 = (const float4 *)P.d_ey2;
    q.C = (float2 *)P.d_C;
    q.thr = (const float *)P.d_thr;
    q.kr = (const float *)P.d_kr;
    q.wide = P.tc_local ? P.d_tcwide : nullptr;
    q.R = (const float *)P.d_R;
    q.H = P.H;
    q.W = P.W;
    q.pitch = P.pitch;
    q.nfy = P.nfy;
    q.eys2 = kTcPad + (P.H + 1) / 2 + kPhPairs;
    q.ncg = (P.W + kCols - 1) / kCols;
    q.nty = (P.H + rw - 1) / rw;
    q.item0 = item0;
    // U = 2^kTapShift kr N u; T = tscale U; C = 2^kTapShift sum T
    const double taps = std::ldexp(1.0, kTapShift);
    const double shrink = P.tc_shrink;
    q.thr_exact = taps / P.inv_norm;
    q.thr_mul = (float)(q.thr_exact * (1.0 - shrink));
    q.out_mul = (float)(P.inv_norm / (taps * taps * (double)P.tc_tscale) * (1.0 + 2.0 * shrink));
}

}  // namespace

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
bool WffPlan::tc_supported() const { return prec == GLSU_F32 && !external_scratch && sy <= kMaxTcHalf; }

// Tables of the tensor-core sweep: the B operand (K-major core matrices of 8
// outputs x 8 inputs, hi then lo), the phasors of row pairs, the tensor map of
// the row-pair layout of R, and the scales.
int WffPlan::init_tc()
{
    if (!tc_supported()) return GLSU_OK;
    const int N = (2 * sy + 16 + 15) / 16 * 16, eys2 = kTcPad + (H + 1) / 2 + kPhPairs;
    std::vector<__half> tb((size_t)2 * N * 16);
    double sum = 0, sumx = 0;
    for (int k = 0; k <= 2 * sy; k++) sum += gy[k];
    for (int k = 0; k <= 2 * sx; k++) sumx += gx[k];
    const int grain = tc_pass_grain(gy, sy, tc_shrink);
    for (int n = 0; n < N; n++)
        for (int j = 0; j < 16; j++) {
            const int k = n - j;
            __half hi, lo;
            tap_parts((k >= 0 && k <= 2 * sy) ? gy[k] : 0.0, grain, hi, lo);
            const size_t at = (size_t)(n / 8) * 128 + (size_t)(j / 8) * 64 + (n % 8) * 8 + j % 8;
            tb[at] = hi;
            tb[(size_t)N * 16 + at] = lo;
        }
    // T = tscale U stays below 2^15 as R does
    tc_tscale = (float)std::ldexp(1.0, -(kTapShift + std::max(0, (int)std::ceil(std::log2(sum)))));
    std::vector<float> ey((size_t)nfy * eys2 * 4);
    for (int k = 0; k < nfy; k++) {
        const double wy = p.wyl + (double)k * p.wyi;
        for (int i = 0; i < eys2; i++)
            for (int r = 0; r < 2; r++) {
                const double y = 2.0 * (i - kTcPad) + r;
                ey[((size_t)k * eys2 + i) * 4 + r] = (float)std::cos(wy * y);
                ey[((size_t)k * eys2 + i) * 4 + 2 + r] = (float)-std::sin(wy * y);
            }
    }
    if (cudaMalloc(&d_tctaps, tb.size() * 2) != cudaSuccess || cudaMalloc(&d_ey2, ey.size() * 4) != cudaSuccess ||
        cudaMalloc(&d_kr, sizeof(float)) != cudaSuccess ||
        (!unit_input && cudaMalloc(&d_tcwide, (size_t)nfx * ((H + 63) / 64) * ((W + kCols - 1) / kCols) * kCols) !=
                            cudaSuccess))
        return fail(GLSU_ERR_ALLOC, "cudaMalloc of the tensor-core sweep's tables failed");
    GLSU_CUDA_TRY(cudaMemcpy(d_tctaps, tb.data(), tb.size() * 2, cudaMemcpyHostToDevice));
    GLSU_CUDA_TRY(cudaMemcpy(d_ey2, ey.data(), ey.size() * 4, cudaMemcpyHostToDevice));
    // an input of unit modulus (DPRA) is scaled by the row pass, others by column and tile in the sweep
    const float kr = unit_input ? (float)std::ldexp(1.0, 15 - std::ilogb((float)(1.4143f * sumx)) - 1) : 1.f;
    GLSU_CUDA_TRY(cudaMemcpy(d_kr, &kr, sizeof(kr), cudaMemcpyHostToDevice));
    auto enc = get_encode_fn();
    if (!enc) return fail(GLSU_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
    const cuuint64_t pairs = (cuuint64_t)(H + 1) / 2;
    cuuint64_t dims[3] = {(cuuint64_t)pitch * 4, pairs, (cuuint64_t)nfx};
    cuuint64_t strides[2] = {(cuuint64_t)pitch * 16, pairs * pitch * 16};
    cuuint32_t box[3] = {32, kChunkRows / 2, 1}, es[3] = {1, 1, 1};
    if (enc(&tmT, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, d_R, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return fail(GLSU_ERR_CUDA, "cuTensorMapEncodeTiled failed");
    return GLSU_OK;
}

void WffPlan::release_tc()
{
    cudaFree(d_tctaps);
    cudaFree(d_ey2);
    cudaFree(d_kr);
    cudaFree(d_tcwide);
    d_tctaps = d_ey2 = nullptr;
    d_tcwide = nullptr;
    d_kr = nullptr;
}

// Modelled time (ms): the steps of the busiest SM at 250 cycles each (measured
// 265 at sigma 10 and 15 on large frames: 1.38 ms modelled at 1024^2, 1.50 measured),
// plus launch and tail.
double tc_model_ms(const WffPlan &P)
{
    int rb[4];
    const int n = tc_row_blocks(P.sy, rb);
    const WffPlan *pp = &P;
    double best = 1e30;
    for (int k = 0; k < n; k++) best = std::min(best, tc_cost(&pp, 1, rb[k], 152));
    return best * 250.0 / 1.9e6 + 0.05;
}

// The sweep of n plans of one window (half-size and sigma) as one persistent
// launch (per 64 plans); n = 1 honours the plan's tile mask.
int launch_tc_sweep(const WffPlan *const *plans, int n, cudaStream_t s)
{
    if (n <= 0) return GLSU_OK;
    const int sms = device_sm_count();
    int rbs[4], rb = 2;
    const int nrb = tc_row_blocks(plans[0]->sy, rbs);
    double best = 1e30;
    for (int k = 0; k < nrb; k++) {
        const double c = tc_cost(plans, n, rbs[k], sms);
        if (c < best) {
            best = c;
            rb = rbs[k];
        }
    }
    if (n == 1) {
        const WffPlan &P = *plans[0];
        TcTable<1> tab;
        tc_seq(tab.seq[0], P, 32 * rb, 0);
        const int tiles = tab.seq[0].ncg * tab.seq[0].nty;
        if (!P.mask.flags) {
            const int items = tiles * P.nfx;
            GLSU_TRY(tc_launch_one(rb, tab, items, std::min(items, sms), P, nullptr, nullptr, s));
            if (!tab.seq[0].wide) return GLSU_OK;
            wff_tc_local_kernel<<<std::min(items, 4 * sms), kLocalThreads, 0, s>>>(
                tab, items, P.sy, (P.sy + 3) / 4, 32 * rb, make_taps<float, 60>(P.gy, P.sy, P.inv_norm),
                make_taps<float, 60>(P.gy, P.sy, 1.0));
            GLSU_CUDA_TRY(cudaGetLastError());
            return GLSU_OK;
        }
        // tile-masked run: the tiles whose outputs, grown by sx columns, meet a
        // flagged tile.  A tile's results depend on its own rows of R only, and
        // ring positions on image rows, so they are the full frame's bits.
        if (!P.d_list) return fail(GLSU_ERR_INVALID, "tile-masked run without a tile list buffer");
        tab.seq[0].wide = nullptr;
        TileMask mk = P.mask;
        mk.my = 0;
        mk.mx = P.sx;
        GLSU_TRY(launch_mask_list(mk, tab.seq[0].ncg, tab.seq[0].nty, 32 * rb, kCols, P.d_list, P.d_list_count, s));
        return tc_launch_one(rb, tab, P.nfx, std::min(tiles * P.nfx, sms), P, P.d_list, P.d_list_count, s);
    }
    constexpr int NS = 64;
    static thread_local TcTable<NS> tab;
    for (int i0 = 0; i0 < n; i0 += NS) {
        const int c = std::min(n - i0, NS);
        int items = 0;
        for (int k = 0; k < c; k++) {
            const WffPlan &P = *plans[i0 + k];
            if (P.sy != plans[0]->sy || P.p.sigma_y != plans[0]->p.sigma_y || P.mask.flags || !P.use_tc() ||
                !P.unit_input)
                return fail(GLSU_ERR_INVALID, "batched column sweep: plans of one window and unit modulus only");
            tc_seq(tab.seq[k], P, 32 * rb, items);
            items += tab.seq[k].ncg * tab.seq[k].nty * P.nfx;
        }
        GLSU_TRY((tc_launch_rb<NS, true>(rb, tab, c, items, std::min(items, sms), *plans[i0], nullptr, nullptr, s)));
    }
    return GLSU_OK;
}

}  // namespace glsu
