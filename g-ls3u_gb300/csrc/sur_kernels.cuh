// sur_kernels.cuh -- kernels of the learned WFF2 surrogate on sm_103a
// (compiled in sur_host.cu).
//
// Network: 8 layers of 3x3 convolutions with per-layer dilation, 32 hidden
// channels, ReLU after layers 0..6; input and output 2 channels (re, im):
//     x   = (Re z, Im z)                 z = exp(j dphi) of the DPRA LS stage
//     a0  = relu(conv0(x))               2 -> 32   CUDA cores, FP32 math
//     a_l = relu(conv_l(a_{l-1}))        32 -> 32  tcgen05, l = 1..6
//     y   = x + conv7(a6)                32 -> 2   tcgen05, N padded to 16
//     out = y / |y|                      the stand-in for WFF2(z) / |WFF2(z)|
// Weights and activations are BF16, accumulation FP32 (TMEM for the
// tensor-core layers).  Activations are NHWC [B][H][W][32] BF16, 64 bytes a
// pixel.
//
// Tensor-core layer (sur_conv_tc_kernel): the MMA tile is 128 consecutive
// pixels of one row (M = 128), K = 16 input channels per tcgen05.mma.  The
// input rows are loaded by TMA through a 4-D tensor map {32 channels, W, H,
// B} with box {32, 128 + 2d, 1, 1} and 64-byte swizzle: each pixel's 64
// bytes arrive as one line, and in shared memory they form the K-major
// SWIZZLE_64B operand layout (rows of 64 bytes, 8-row groups 512 bytes
// apart, the 16-byte chunks of a row permuted by address bits 7-8).  A tap's
// horizontal offset dx * d is a shift of the descriptor start by 64 * dx * d
// bytes, the second K = 16 half a shift by 32 bytes, with the base offset
// field left at 0: the tensor core applies the swizzle to the absolute
// shared-memory address, as TMA does (measured: every dilation 1..16 and odd
// shifts agree with the oracle), so no im2col copy is needed, and TMA
// zero-fills the image border.  The epilogue writes each warp's 32 output pixels into a
// staging tile in the same swizzled layout (conflict-free 16-byte stores)
// and one thread stores the tile with a TMA tensor store.
// Work items are chunks of kSurRows output rows of one chain y = r, r + d,
// r + 2d, ... (the rows that share input rows under dilation d).  Input row j
// of an item (j = 0 .. nout + 1) feeds output rows j - 2, j - 1, j through
// the vertical taps dy = 2, 1, 0, so each input row is consumed by ONE MMA
// per (dx, K half) with N = 96: the B operand stacks the three vertical taps'
// weights [dy = 2 | dy = 1 | dy = 0] and the D columns are the three output
// rows' accumulators, which sit side by side in TMEM (output row k of the
// item at columns 32k .. 32k + 31).  At the ends of an item N shrinks to 64
// or 32.  Every MMA accumulates: the epilogue fills each accumulator with the
// bias before its first use and again after draining it.  A row's 18 K = 16
// products are thus 6 MMAs of up to N = 96 instead of 18 of N = 32 (an N = 32
// MMA costs nearly as much as an N = 96 one).
// The kernel is persistent and warp-specialised: one thread streams every
// item's input rows through a ring of slots by TMA, one thread issues the
// MMAs, four warps drain the accumulators.
#pragma once

#include <cuda_bf16.h>

#include <algorithm>
#include <atomic>
#include <cmath>

#include "dpra_ls_ff.cuh"
#include "glsu_internal.cuh"
#include "ptx_sm103.cuh"

namespace glsu {

constexpr int kSurSlots = 8;     // input-row ring of the tensor-core conv (TMA loads in flight)
constexpr int kSurRows = 8;      // output rows per work item = TMEM accumulators
constexpr int kSurWBytes = 9 * 4 * 32 * 16;  // packed B operand of a 32 -> 32 layer
constexpr int kSurStageBytes = 32 * 64;      // one epilogue warp's output tile

// Geometry of a tensor-core layer with NOUT output channels per accumulator:
// 32 for the hidden layers, 16 for the last layer (its 2 outputs padded with
// zero weights to the smallest N of an M = 128 MMA).  The packed B operand
// is [dx][K half kc][8-channel chunk h][3 NOUT rows][8 channels], row
// n = NOUT (2 - dy) + output channel.
template <int NOUT> struct SurTc {
    static constexpr int BROWS = 3 * NOUT;
    static constexpr int BHALF = BROWS * 16;  // bytes between the two 8-channel chunks of one K = 16 step
    static constexpr int BSTEP = 2 * BHALF;   // bytes of one (dx, kc) operand
    static constexpr int WBYTES = 6 * BSTEP;  // 3 dx x 2 kc operands (a 1024-byte multiple)
    static constexpr int TMEM_COLS = kSurRows * NOUT;
    static constexpr int STAGE = NOUT == 32 ? 4 * kSurStageBytes : 0;
    static constexpr int NBIAS = NOUT == 32 ? 32 : 2;
};
static_assert(SurTc<32>::WBYTES == kSurWBytes && SurTc<16>::WBYTES % 1024 == 0, "B operand layout");
constexpr int kSurPk7Bytes = SurTc<16>::WBYTES;  // packed B operand of the last layer

// out = y / |y| with the same rounding wherever it is evaluated (the last
// layer's epilogue in inference, the loss kernel in training).
__device__ __forceinline__ void sur_unit(float yr, float yi, float &orr, float &oii, float &inv)
{
    const float nrm = __fsqrt_rn(__fadd_rn(__fmul_rn(yr, yr), __fmul_rn(yi, yi)));
    inv = nrm > 1e-20f ? __fdiv_rn(1.f, nrm) : 0.f;
    orr = __fmul_rn(yr, inv);
    oii = __fmul_rn(yi, inv);
}

__device__ __forceinline__ float bf2f(uint16_t v) { return __uint_as_float((uint32_t)v << 16); }

// A float-float sum in FP32; where the sum is not finite its low part is NaN.
__device__ __forceinline__ float ff_value(ff a) { return isfinite(a.hi) ? a.hi + a.lo : a.hi; }

__device__ __forceinline__ uint32_t pack_bf2(float lo, float hi)
{
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&h);
}

__device__ __forceinline__ void unpack8(const uint4 u, float *f)
{
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int i = 0; i < 4; i++) {
        f[2 * i] = __uint_as_float(w[i] << 16);
        f[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
    }
}

// ---------------------------------------------------------------------------
// tensor-core 32 -> 32 conv (forward, or backward-data with flipped weights)
// ---------------------------------------------------------------------------
// Work item: (image b, 128-pixel segment, residue r mod d, chunk of the
// chain r, r+d, r+2d, ...), up to kSurRows output rows with 2 halo rows.
struct SurItem {
    int b, x0, r, kbeg, nout;
};

__device__ __forceinline__ SurItem sur_item(const SurConvArgs &a, int item)
{
    const int nsx = (a.W + 127) / 128;
    const int nch = ((a.H + a.dil - 1) / a.dil + kSurRows - 1) / kSurRows;
    SurItem it;
    const int ch = item % nch;
    item /= nch;
    it.r = item % a.dil;
    item /= a.dil;
    it.x0 = (item % nsx) * 128;
    it.b = item / nsx;
    it.kbeg = ch * kSurRows;
    const int chain_len = (a.H - it.r + a.dil - 1) / a.dil;  // rows r, r+d, ... below H
    it.nout = max(0, min(kSurRows, chain_len - it.kbeg));
    return it;
}

// Persistent, warp-specialised: thread 0 of warp 0 issues the TMA row loads
// into a ring of kSurSlots slots, thread 0 of warp 1 issues the MMAs, warps
// 4-7 drain the accumulators.  All three walk the same item list
// (blockIdx.x, + gridDim.x, ...); input rows are numbered across items and
// each accumulator completes one phase of its two mbarriers per item (a
// block that an item leaves unused gets an empty phase), which keeps the
// mbarrier parities consistent.  NOUT = 32: a hidden layer (ReLU / mask,
// BF16 NHWC by TMA store through tmo); NOUT = 16: the last layer (y = z +
// conv + bias from the first two accumulator columns; out = y / |y| into
// a.cout, or y itself into a.yout).
template <int NOUT>
__global__ void __launch_bounds__(256, 2) sur_conv_tc_kernel(const __grid_constant__ CUtensorMap tm,
                                                             const __grid_constant__ CUtensorMap tmo, SurConvArgs a,
                                                             int nitems)
{
    using L = SurTc<NOUT>;
    extern __shared__ __align__(1024) unsigned char sm[];
    const int BW = 128 + 2 * a.dil;
    const int slot_bytes = (BW * 64 + 1023) & ~1023;
    unsigned char *wsm = sm;
    unsigned char *slots = sm + L::WBYTES;
    unsigned char *stage = slots + kSurSlots * slot_bytes;  // [4 warps][32 px][64 B], 64-byte swizzle
    uint64_t *full = reinterpret_cast<uint64_t *>(stage + L::STAGE);
    uint64_t *sfree = full + kSurSlots;
    uint64_t *accf = sfree + kSurSlots;  // [kSurRows] accumulator complete
    uint64_t *acce = accf + kSurRows;    // [kSurRows] accumulator drained and refilled with the bias
    uint64_t *drain = acce + kSurRows;
    float *bias_s = reinterpret_cast<float *>(drain + 1);
    uint32_t *tslot = reinterpret_cast<uint32_t *>(bias_s + 32);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int s = 0; s < kSurSlots; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&sfree[s], 1);
        }
        for (int b = 0; b < kSurRows; b++) {
            mbar_init(&accf[b], 1);
            mbar_init(&acce[b], 128);
        }
        mbar_init(drain, 1);
        fence_mbar_init();
    }
    if (warp == 0) tmem_alloc(tslot, L::TMEM_COLS);
    for (int e = tid; e < L::WBYTES / 16; e += 256)
        reinterpret_cast<uint4 *>(wsm)[e] = reinterpret_cast<const uint4 *>(a.wpack)[e];
    if (tid < 32) bias_s[tid] = (a.bias && tid < L::NBIAS) ? a.bias[tid] : 0.f;
    fence_proxy_async_smem();  // the weight image was written by generic stores
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot;

    if (warp == 0 && elect_one()) {
        // ---- producer: TMA loads of every item's nout + 2 input rows ----
        uint32_t g = 0;
        bool ok = true;
        for (int item = blockIdx.x; item < nitems && ok; item += gridDim.x) {
            const SurItem it = sur_item(a, item);
            for (int j = 0; j < it.nout + 2 && it.nout > 0; j++, g++) {
                const int s = g % kSurSlots;
                if (g >= kSurSlots && !mbar_wait_bounded(&sfree[s], ((g / kSurSlots) - 1) & 1)) {
                    ok = false;
                    break;
                }
                mbar_expect_tx(&full[s], (uint32_t)BW * 64);
                tma_load_4d(slots + s * slot_bytes, &tm, &full[s], 0, it.x0 - a.dil, it.r + (it.kbeg + j - 1) * a.dil,
                            it.b);
            }
        }
        if (!ok) atomicExch(a.err, GLSU_ERR_TIMEOUT);
        // every load has landed before the CTA exits
        for (uint32_t j = g > (uint32_t)kSurSlots ? g - kSurSlots : 0; j < g; j++)
            mbar_wait_bounded(&full[j % kSurSlots], (j / kSurSlots) & 1);
    } else if (warp == 1 && elect_one()) {
        // ---- MMA issuer ----
        const uint32_t wbase = smem_u32(wsm), sbase = smem_u32(slots);
        uint32_t g = 0, li = 0;
        bool ok = true;
        for (int item = blockIdx.x; item < nitems && ok; item += gridDim.x, li++) {
            const SurItem it = sur_item(a, item);
            if (it.nout <= 0) {
                li--;
                continue;
            }
            const uint32_t par = li & 1;
            for (int j = 0; j < it.nout + 2 && ok; j++, g++) {
                const int s = g % kSurSlots;
                if (!mbar_wait_bounded(&full[s], (g / kSurSlots) & 1)) ok = false;
                // output row j is first written by this input row: its accumulator must hold the bias
                if (ok && j < it.nout && !mbar_wait_bounded(&acce[j], par)) ok = false;
                if (!ok) break;
                tc_fence_after();
                const int klo = max(0, j - 2), khi = min(it.nout - 1, j);
                const uint32_t id = khi == klo       ? umma_idesc_bf16(128, NOUT)
                                    : khi == klo + 1 ? umma_idesc_bf16(128, 2 * NOUT)
                                                     : umma_idesc_bf16(128, 3 * NOUT);
                const uint32_t d = tmem + (uint32_t)(klo * NOUT);
                const uint32_t srow = sbase + (uint32_t)(s * slot_bytes);
                const uint32_t brow = wbase + (uint32_t)((2 - j + klo) * NOUT * 16);
#pragma unroll
                for (int dx = 0; dx < 3; dx++) {
#pragma unroll
                    for (int kc = 0; kc < 2; kc++) {
                        const uint32_t astart = srow + (uint32_t)(dx * a.dil * 64 + kc * 32);
                        const uint64_t ad = umma_desc_sw64(astart, 0);
                        const uint64_t bd = umma_desc(brow + (uint32_t)((dx * 2 + kc) * L::BSTEP), L::BHALF, 128);
                        umma_bf16(d, ad, bd, id, 1u);
                    }
                }
                umma_commit(&sfree[s]);              // input row g is not read again
                if (j >= 2) umma_commit(&accf[j - 2]);  // output row j - 2 has all its products
            }
            // accumulators this item leaves unused: an empty phase
            for (int b = it.nout; b < kSurRows && ok; b++) {
                if (!mbar_wait_bounded(&acce[b], par)) ok = false;
                else umma_commit(&accf[b]);
            }
        }
        if (!ok) atomicExch(a.err, GLSU_ERR_TIMEOUT);
        umma_commit(drain);  // every MMA has completed before TMEM is released
        mbar_wait_bounded(drain, 0);
    } else if (warp >= 4 && NOUT == 16) {
        // ---- last-layer epilogue: y = z + h, out = y / |y|; refill with the bias ----
        const int q = warp - 4;
        const uint32_t lane_base = tmem + ((uint32_t)(q * 32) << 16);
        float bias[16];
#pragma unroll
        for (int c = 0; c < 16; c++) bias[c] = bias_s[c];
        for (int b = 0; b < kSurRows; b++) tmem_st16(lane_base + b * NOUT, bias);
        tc_fence_before();
        for (int b = 0; b < kSurRows; b++) mbar_arrive(&acce[b]);
        uint32_t li = 0;
        bool ok = true;
        for (int item = blockIdx.x; item < nitems && ok; item += gridDim.x) {
            const SurItem it = sur_item(a, item);
            if (it.nout <= 0) continue;
            const int x = it.x0 + q * 32 + lane;
            // the residual input z of the item's rows, loaded before the first
            // accumulator wait so that the loads overlap the MMAs
            float2 zr[kSurRows];
#pragma unroll
            for (int k = 0; k < kSurRows; k++) {
                zr[k] = make_float2(0.f, 0.f);
                if (k < it.nout && x < a.W)
                    zr[k] = a.z[((size_t)it.b * a.H + it.r + (size_t)(it.kbeg + k) * a.dil) * a.W + x];
            }
#pragma unroll
            for (int k = 0; k < kSurRows; k++) {
                if (!__all_sync(0xffffffffu, mbar_wait_bounded(&accf[k], li & 1))) {
                    if (lane == 0) atomicExch(a.err, GLSU_ERR_TIMEOUT);
                    ok = false;
                    break;
                }
                tc_fence_after();
                float h[2] = {0.f, 0.f};
                if (k < it.nout) {
                    tmem_ld2(lane_base + k * NOUT, h);
                    tmem_st16(lane_base + k * NOUT, bias);
                }
                tc_fence_before();
                mbar_arrive(&acce[k]);
                if (k >= it.nout || x >= a.W) continue;
                const size_t p = ((size_t)it.b * a.H + it.r + (size_t)(it.kbeg + k) * a.dil) * a.W + x;
                const float2 zv = zr[k];
                const float yr = __fadd_rn(zv.x, h[0]), yi = __fadd_rn(zv.y, h[1]);
                if (a.yout) {
                    a.yout[p] = make_float2(yr, yi);
                } else {
                    float orr, oii, inv;
                    sur_unit(yr, yi, orr, oii, inv);
                    a.cout[p] = make_float2(orr, oii);
                }
            }
            li++;
        }
    } else if (warp >= 4 && NOUT == 32) {
        // ---- epilogue: TMEM -> ReLU, mask -> BF16 NHWC; refill with the bias ----
        const int q = warp - 4;
        const uint32_t lane_base = tmem + ((uint32_t)(q * 32) << 16);
        unsigned char *my_stage = stage + q * kSurStageBytes;
        float bias[32];
#pragma unroll
        for (int c = 0; c < 32; c++) bias[c] = bias_s[c];
        for (int b = 0; b < kSurRows; b++) tmem_st32(lane_base + b * 32, bias);
        tc_fence_before();
        for (int b = 0; b < kSurRows; b++) mbar_arrive(&acce[b]);
        uint32_t li = 0;
        bool ok = true;
        for (int item = blockIdx.x; item < nitems && ok; item += gridDim.x) {
            const SurItem it = sur_item(a, item);
            if (it.nout <= 0) continue;
            const int x = it.x0 + q * 32 + lane;
            // the mask of a row is asked for while the row before it is stored
            // (the first one while the item's MMAs run): loaded after the
            // accumulator's wait, its latency made a masked layer 46 us where an
            // unmasked one takes 30 at 16 x 256 x 256; 39 us as here
            const bool masked = a.mask && x < a.W;
            uint4 mk[4];
            auto load_mask = [&](int k) {
                if (!masked || k >= it.nout) return;
                const int y = it.r + (it.kbeg + k) * a.dil;
                const uint4 *mp =
                    reinterpret_cast<const uint4 *>(a.mask + (((size_t)it.b * a.H + y) * a.W + x) * 32);
#pragma unroll
                for (int g = 0; g < 4; g++) mk[g] = mp[g];
            };
            load_mask(0);
            for (int k = 0; k < kSurRows; k++) {
                // warp-uniform: tcgen05.ld / st below are warp-collective instructions
                if (!__all_sync(0xffffffffu, mbar_wait_bounded(&accf[k], li & 1))) {
                    if (lane == 0) atomicExch(a.err, GLSU_ERR_TIMEOUT);
                    ok = false;
                    break;
                }
                tc_fence_after();
                float v[32];
                if (k < it.nout) {
                    tmem_ld32(lane_base + k * 32, v);
                    tmem_st32(lane_base + k * 32, bias);
                }
                tc_fence_before();
                mbar_arrive(&acce[k]);
                if (k >= it.nout) continue;
                const int y = it.r + (it.kbeg + k) * a.dil;
                if (a.relu) {
#pragma unroll
                    for (int c = 0; c < 32; c++) v[c] = fmaxf(v[c], 0.f);
                }
                if (masked) {
#pragma unroll
                    for (int g = 0; g < 4; g++) {
                        float mv[8];
                        unpack8(mk[g], mv);
#pragma unroll
                        for (int i = 0; i < 8; i++)
                            if (!(mv[i] > 0.f)) v[8 * g + i] = 0.f;
                    }
                    load_mask(k + 1);
                }
                // the previous tile of this warp has been read by its TMA store
                if (lane == 0) bulk_wait_read0();
                __syncwarp();
#pragma unroll
                for (int g = 0; g < 4; g++)
                    *reinterpret_cast<uint4 *>(my_stage + lane * 64 + ((g ^ ((lane >> 1) & 3)) * 16)) =
                        make_uint4(pack_bf2(v[8 * g], v[8 * g + 1]), pack_bf2(v[8 * g + 2], v[8 * g + 3]),
                                   pack_bf2(v[8 * g + 4], v[8 * g + 5]), pack_bf2(v[8 * g + 6], v[8 * g + 7]));
                fence_proxy_async_smem();
                __syncwarp();
                // columns beyond W are clipped by the store
                if (lane == 0 && it.x0 + q * 32 < a.W) {
                    tma_store_4d(&tmo, my_stage, 0, it.x0 + q * 32, y, it.b);
                    bulk_commit();
                }
            }
            li++;
        }
        if (lane == 0) bulk_wait0();  // every output tile has been written
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) tmem_dealloc(tmem, L::TMEM_COLS);
}

template <int NOUT> static int sur_conv_smem_bytes(int dil)
{
    const int BW = 128 + 2 * dil;
    const int slot_bytes = (BW * 64 + 1023) & ~1023;
    return SurTc<NOUT>::WBYTES + kSurSlots * slot_bytes + SurTc<NOUT>::STAGE +
           (2 * kSurSlots + 2 * kSurRows + 1) * 8 + 32 * 4 + 16;
}

int sur_conv_items(int B, int H, int W, int dil)
{
    const int nsx = (W + 127) / 128;
    const int nch = ((H + dil - 1) / dil + kSurRows - 1) / kSurRows;
    return B * nsx * dil * nch;
}

// 4-D map {32 channels, W, H, B} of a [B][H][W][32] BF16 activation tensor
// (strides 64 B, W*64 B, H*W*64 B) with box {32, box_px, 1, 1} and 64-byte
// swizzle: the conv's input rows (box_px = 128 + 2d) and output tiles
// (box_px = 32).
static int sur_make_map_box(CUtensorMap *tm, const void *act, int B, int H, int W, int box_px)
{
    auto enc = get_encode_fn();
    if (!enc) return fail(GLSU_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
    cuuint64_t dims[4] = {32, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)B};
    cuuint64_t strides[3] = {64, (cuuint64_t)W * 64, (cuuint64_t)H * W * 64};
    cuuint32_t box[4] = {32, (cuuint32_t)box_px, 1, 1};
    cuuint32_t es[4] = {1, 1, 1, 1};
    CUresult r = enc(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void *>(act), dims, strides, box, es,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(GLSU_ERR_CUDA, "cuTensorMapEncodeTiled failed for an activation map");
    return GLSU_OK;
}

int sur_make_map(CUtensorMap *tm, const void *act, int B, int H, int W, int dil)
{
    if (dil < 1 || 128 + 2 * dil > 256) return fail(GLSU_ERR_INVALID, "surrogate dilation must be 1..64");
    return sur_make_map_box(tm, act, B, H, W, 128 + 2 * dil);
}

int sur_make_out_map(CUtensorMap *tm, const void *act, int B, int H, int W)
{
    return sur_make_map_box(tm, act, B, H, W, 32);
}

template <int NOUT>
static int launch_sur_conv_t(const CUtensorMap &tm, const CUtensorMap &tmo, const SurConvArgs &a, cudaStream_t s)
{
    // registers per thread are a property of the binary (the same on every device)
    static std::atomic<int> regs_cached{0};
    const int smem = sur_conv_smem_bytes<NOUT>(a.dil);
    GLSU_TRY(raise_smem_limit((const void *)sur_conv_tc_kernel<NOUT>, sur_conv_smem_bytes<NOUT>(64),
                              (int)cudaSharedmemCarveoutMaxShared));
    const int sms = device_sm_count();
    int regs = regs_cached.load();
    if (!regs) {
        cudaFuncAttributes fa;
        GLSU_CUDA_TRY(cudaFuncGetAttributes(&fa, sur_conv_tc_kernel<NOUT>));
        regs = std::max(1, fa.numRegs);
        regs_cached.store(regs);
    }
    // persistent: as many CTAs as are resident at once, each walking a
    // strided list of items.  Residency is bounded by registers (per-warp
    // allocation in units of 256), shared memory (1 KB reserved per CTA) and
    // the 512 TMEM columns.
    const int warp_regs = (regs * 32 + 255) / 256 * 256;
    const int by_regs = 65536 / (8 * warp_regs);
    const int by_smem = (228 * 1024) / (smem + 1024);
    const int by_tmem = 512 / SurTc<NOUT>::TMEM_COLS;
    int per_sm = std::max(1, std::min(std::min(by_regs, by_smem), by_tmem));
    if (a.max_ctas_per_sm > 0) per_sm = std::min(per_sm, a.max_ctas_per_sm);
    const int items = sur_conv_items(a.B, a.H, a.W, a.dil);
    const int grid = std::min(items, per_sm * sms);
    sur_conv_tc_kernel<NOUT><<<grid, 256, smem, s>>>(tm, tmo, a, items);
    GLSU_CUDA_TRY(cudaGetLastError());
    return GLSU_OK;
}

int launch_sur_conv(const CUtensorMap &tm, const CUtensorMap &tmo, const SurConvArgs &a, cudaStream_t s)
{
    return launch_sur_conv_t<32>(tm, tmo, a, s);
}

int launch_sur_last(const CUtensorMap &tm, const SurConvArgs &a, cudaStream_t s)
{
    if (!a.z || (!a.cout && !a.yout)) return fail(GLSU_ERR_INVALID, "last surrogate layer without input or output");
    return launch_sur_conv_t<16>(tm, tm, a, s);
}

// ---------------------------------------------------------------------------
// layer 0 (2 -> 32) on CUDA cores, the training loss
// ---------------------------------------------------------------------------
// Layer 0 (2 -> 32, ReLU); z: complex [B][H][W].  The weights are kernel
// parameters, so every FMA takes its weight from the parameter bank.
__global__ void __launch_bounds__(256) sur_l0_kernel(const float2 *__restrict__ z, int B, int H, int W, int dil,
                                                     const __grid_constant__ SurL0W wp, uint16_t *__restrict__ out)
{
    for (int row = blockIdx.x; row < B * H; row += gridDim.x)
        for (int x = threadIdx.x; x < W; x += 256) {
            const int y = row % H;
            const size_t p = (size_t)row * W + x;
            const size_t img = (size_t)(row - y) * W;
            float in[18];
#pragma unroll
            for (int t = 0; t < 9; t++) {
                const int yy = y + (t / 3 - 1) * dil, xx = x + (t % 3 - 1) * dil;
                float2 v = make_float2(0.f, 0.f);
                if (yy >= 0 && yy < H && xx >= 0 && xx < W) v = z[img + (size_t)yy * W + xx];
                in[t] = v.x;
                in[9 + t] = v.y;
            }
            float acc[32];
#pragma unroll
            for (int c = 0; c < 32; c++) {
                float s = wp.b[c];
#pragma unroll
                for (int k = 0; k < 18; k++) s = fmaf(wp.w[c * 18 + k], in[k], s);
                acc[c] = fmaxf(s, 0.f);
            }
            uint4 *op = reinterpret_cast<uint4 *>(out + p * 32);
#pragma unroll
            for (int g = 0; g < 4; g++)
                op[g] = make_uint4(pack_bf2(acc[8 * g], acc[8 * g + 1]), pack_bf2(acc[8 * g + 2], acc[8 * g + 3]),
                                   pack_bf2(acc[8 * g + 4], acc[8 * g + 5]), pack_bf2(acc[8 * g + 6], acc[8 * g + 7]));
        }
}

// Training loss of the last layer's output: from y = z + conv7(a6) (written
// by the tensor-core last layer), out = y / |y| (the same rounding as the
// inference epilogue), per pixel loss wgt |out - t|^2 with wgt =
// min(wscale |target|, 1) and t = target / |target|, the gradient dL/dh7 of
// the mean loss into dh
// and per-block loss sums (fixed order) into part.
__global__ void __launch_bounds__(256) sur_l7_loss_kernel(const float2 *__restrict__ yv,
                                                          const float2 *__restrict__ target, size_t n,
                                                          float2 *__restrict__ out, float2 *__restrict__ dh,
                                                          double *__restrict__ part, float wscale)
{
    __shared__ double red[256];
    const int tid = threadIdx.x;
    const double inv_n = 1.0 / (double)n;
    double lsum = 0;
    for (size_t p = (size_t)blockIdx.x * 256 + tid; p < n; p += (size_t)gridDim.x * 256) {
        const float2 y = yv[p];
        float orr, oii, inv;
        sur_unit(y.x, y.y, orr, oii, inv);
        out[p] = make_float2(orr, oii);
        const float2 tv = target[p];
        const float tn = sqrtf(tv.x * tv.x + tv.y * tv.y);
        const float wgt = fminf(tn * wscale, 1.f);
        const float ti = tn > 1e-20f ? 1.f / tn : 0.f;
        const float er = orr - tv.x * ti, ei = oii - tv.y * ti;
        lsum += (double)(wgt * (er * er + ei * ei)) * inv_n;
        // d out: 2 wgt e / n; through out = y/|y|: (g - out (out.g)) / |y|
        const float gr = (float)(2.0 * inv_n) * wgt * er, gi = (float)(2.0 * inv_n) * wgt * ei;
        const float dot = orr * gr + oii * gi;
        dh[p] = make_float2((gr - orr * dot) * inv, (gi - oii * dot) * inv);
    }
    red[tid] = lsum;
    __syncthreads();
    for (int s = 128; s > 0; s >>= 1) {
        if (tid < s) red[tid] += red[tid + s];
        __syncthreads();
    }
    if (tid == 0) part[blockIdx.x] = red[0];
}

// ---------------------------------------------------------------------------
// weight gradients
// ---------------------------------------------------------------------------
// 32 -> 32 layer on the tensor cores.  With d the dilation and g the
// gradient w.r.t. the layer's output,
//   dW[co][ci][ky][kx] = sum_{b, y', x} g[b, y' - (ky-1) d, x, co] a[b, y', x + (kx-1) d, ci]
// (y' = y + (ky-1) d: each activation row y' meets the gradient rows y' + d,
// y', y' - d).  A work item is one 128-pixel segment of `rows` activation rows
// d apart, taken downwards: with its rows + 2 gradient rows in consecutive
// slots (slot j: the top activation row + d - j d) the i-th activation row
// meets the three slots i, i + 1, i + 2.  Per 16 pixels and activation row one
// MMA D[M = 128][N = 96] += A[M][K = 16] B[K][N]:
//   A: those three gradient rows, M = ky * 32 + co (the slot after them pads M
//      to 128, zeros behind the last: lanes 96-127 are not read);
//   B: the activation row, N = kx * 32 + ci, its three kx blocks d pixels
//      apart.
// Both operands are the pixel-major rows that TMA writes with 64-byte
// swizzle, read MN-major: per pixel the 32 channels (64 bytes, the M or N
// direction), pixels 64 bytes apart and 8-pixel groups 512 bytes apart (K),
// the 32-channel blocks LBO apart (the gradient slot stride for A, 64 d bytes
// for B).  The accumulator stays in TMEM across all of a CTA's items; the
// epilogue writes it once as the CTA's partial, part[blk][t = ky*3+kx][ci][co]
// with co along the lanes.
// The bias gradient, the sum of g, comes from the same shared-memory rows: the
// four warps that wait for the epilogue add up each item's centre slots,
// compensated from item to item, into part[blk][9216 + co].
// What bounds it is the L2 traffic of the operands, (2 rows + 2) row segments
// per `rows`: one row an item, as this kernel had, reads every gradient row
// three times.  A training pass at 16 x 256 x 256: 1522 us with one row an item,
// a bias pass over g of 21 us a layer and FP64 reductions, 1212 us as here.
constexpr int kWgMaxRows = 4;
constexpr int kWgMaxStages = 4;
constexpr int kWgSlot = 128 * 64;          // one 128-pixel gradient row segment
constexpr int kWgPad = 16 * 1024;          // slack after the stages
constexpr int kWgTail = 1024;              // barriers and the bias sums of four warps
constexpr int kWgSmemMax = 232448;
constexpr uint32_t kWgTmemCols = 128;
constexpr int kWgCols = kSurL32Params;     // columns of a partial: weights, then biases

__host__ __device__ inline int sur_wgrad_act_bytes(int dil) { return ((128 + 2 * dil) * 64 + 1023) & ~1023; }
// gradient slots, the zero slot, activation rows
__host__ __device__ inline int sur_wgrad_stage_bytes(int dil, int rows)
{
    return (rows + 3) * kWgSlot + rows * sur_wgrad_act_bytes(dil);
}
inline int sur_wgrad_stages(int dil, int rows)
{
    return std::min(kWgMaxStages, (kWgSmemMax - kWgPad - kWgTail) / sur_wgrad_stage_bytes(dil, rows));
}
inline int sur_wgrad_smem_bytes(int dil, int rows)
{
    return sur_wgrad_stages(dil, rows) * sur_wgrad_stage_bytes(dil, rows) + kWgPad + kWgTail;
}
// First activation row of an item (0 .. rows) that is inside the image; those
// above it in the item's order are neither loaded nor multiplied.
__host__ __device__ inline int sur_wgrad_first(int top, int H, int dil, int rows)
{
    if (top < H) return 0;
    const int j = (top - H) / dil + 1;
    return j < rows ? j : rows;
}
// Items of a batch: rows of a residue class mod d, `rows` at a time, by segments.
inline int sur_wgrad_items(int B, int H, int W, int dil, int rows)
{
    const int classes = std::min(dil, H), chain = (H + dil - 1) / dil;
    return B * classes * ((chain + rows - 1) / rows) * ((W + 127) / 128);
}

// MN-major operand in the 64-byte swizzle layout: 32-element blocks `lbo`
// bytes apart, 8-row (K) groups 512 bytes apart.
__device__ __forceinline__ uint64_t umma_desc_mn_sw64(uint32_t saddr, uint32_t lbo)
{
    return (uint64_t)((saddr >> 4) & 0x3FFF) | ((uint64_t)((lbo >> 4) & 0x3FFF) << 16) |
           ((uint64_t)(512 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)4 << 61);
}

struct SurWgradArgs {
    int B = 0, H = 0, W = 0, dil = 1;
    float *part = nullptr;  // [gridDim.x][kWgCols]
    int *err = nullptr;
};

__global__ void __launch_bounds__(256, 1) sur_wgrad_tc_kernel(const __grid_constant__ CUtensorMap tma,
                                                              const __grid_constant__ CUtensorMap tmg,
                                                              SurWgradArgs a, int nitems, int rows, int stages)
{
    extern __shared__ __align__(1024) unsigned char sm[];
    const int stage_bytes = sur_wgrad_stage_bytes(a.dil, rows), act_bytes = sur_wgrad_act_bytes(a.dil);
    uint64_t *full = reinterpret_cast<uint64_t *>(sm + stages * stage_bytes + kWgPad);
    uint64_t *sfree = full + kWgMaxStages;
    uint64_t *done = sfree + kWgMaxStages;
    uint32_t *tslot = reinterpret_cast<uint32_t *>(done + 1);
    float *bsum = reinterpret_cast<float *>(full) + 64;  // [4 warps][32]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nsx = (a.W + 127) / 128;
    if (tid == 0) {
        for (int s = 0; s < stages; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&sfree[s], 1 + 4);  // the MMAs' commit and the four bias warps
        }
        mbar_init(done, 1);
        fence_mbar_init();
    }
    if (warp == 0) tmem_alloc(tslot, kWgTmemCols);
    // the slot after the gradient rows of every stage stays zero
    for (int s = 0; s < stages; s++)
        for (int e = tid; e < kWgSlot / 16; e += 256)
            reinterpret_cast<uint4 *>(sm + s * stage_bytes + (rows + 2) * kWgSlot)[e] = make_uint4(0, 0, 0, 0);
    fence_proxy_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot;
    // every MMA accumulates
    if (warp >= 4) {
        const float z[32] = {};
        for (int c = 0; c < 96; c += 32) tmem_st32(tmem + ((uint32_t)((warp - 4) * 32) << 16) + c, z);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();

    // the top (last) activation row of an item
    const int classes = min(a.dil, a.H), groups = ((a.H + a.dil - 1) / a.dil + rows - 1) / rows;
    auto top_of = [&](int item) {
        const int i = item / nsx;
        return i % classes + ((i / classes % groups + 1) * rows - 1) * a.dil;
    };

    if (warp == 0 && elect_one()) {
        // ---- producer: per item up to rows + 2 gradient rows and `rows` activation rows ----
        uint32_t s = 0, lap = 0;
        bool ok = true;
        for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
            const int sx = item % nsx, b = item / nsx / classes / groups, top = top_of(item);
            const int j0 = sur_wgrad_first(top, a.H, a.dil, rows);
            const uint32_t bytes =
                (uint32_t)(rows + 2 - j0) * kWgSlot + (uint32_t)((rows - j0) * (128 + 2 * a.dil)) * 64;
            if (lap > 0 && !mbar_wait_bounded(&sfree[s], (lap - 1) & 1)) {
                ok = false;
                break;
            }
            unsigned char *st = sm + s * stage_bytes, *sa = st + (rows + 3) * kWgSlot;
            mbar_expect_tx(&full[s], bytes);
            // rows outside the image arrive as zeros
            for (int j = j0; j < rows + 2; j++)
                tma_load_4d(st + j * kWgSlot, &tmg, &full[s], 0, sx * 128, top + (1 - j) * a.dil, b);
            for (int j = j0; j < rows; j++)
                tma_load_4d(sa + j * act_bytes, &tma, &full[s], 0, sx * 128 - a.dil, top - j * a.dil, b);
            if (++s == (uint32_t)stages) {
                s = 0;
                lap++;
            }
        }
        if (!ok) atomicExch(a.err, GLSU_ERR_TIMEOUT);
        // no copy is in flight when the CTA ends: each stage's last one
        for (uint32_t j = 0; j < (uint32_t)stages; j++) {
            const uint32_t uses = lap + (j < s ? 1 : 0);
            if (uses > 0) mbar_wait_bounded(&full[j], (uses - 1) & 1);
        }
    } else if (warp == 1 && elect_one()) {
        // ---- MMA issuer ----
        const uint32_t idesc = umma_idesc_bf16(128, 96) | (1u << 15) | (1u << 16);  // A and B MN-major
        uint32_t s = 0, lap = 0;
        bool ok = true;
        for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
            if (!mbar_wait_bounded(&full[s], lap & 1)) {
                ok = false;
                break;
            }
            tc_fence_after();
            const int j0 = sur_wgrad_first(top_of(item), a.H, a.dil, rows);
            const uint32_t st = smem_u32(sm + s * stage_bytes);
            uint32_t gb = st + j0 * kWgSlot, ab = st + (rows + 3) * kWgSlot + j0 * act_bytes;
            for (int j = j0; j < rows; j++, gb += kWgSlot, ab += act_bytes) {
#pragma unroll
                for (int k = 0; k < 8; k++)
                    umma_bf16(tmem, umma_desc_mn_sw64(gb + k * 1024, kWgSlot),
                              umma_desc_mn_sw64(ab + k * 1024, (uint32_t)a.dil * 64), idesc, 1);
            }
            umma_commit(&sfree[s]);
            if (++s == (uint32_t)stages) {
                s = 0;
                lap++;
            }
        }
        if (!ok) atomicExch(a.err, GLSU_ERR_TIMEOUT);
        umma_commit(done);  // every MMA has completed before the epilogue reads and TMEM is released
        mbar_wait_bounded(done, 0);
    } else if (warp >= 4) {
        // ---- bias sums: thread = (8-channel group, pixel lane 0..31) of the centre rows ----
        const int cg = tid & 3, pl = (tid - 128) >> 2;
        ff acc[8];
#pragma unroll
        for (int c = 0; c < 8; c++) acc[c] = {0.f, 0.f};
        uint32_t s = 0, lap = 0;
        bool ok = true;
        for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
            if (!__all_sync(0xffffffffu, mbar_wait_bounded(&full[s], lap & 1))) {
                ok = false;
                break;
            }
            float sum[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            for (int j = sur_wgrad_first(top_of(item), a.H, a.dil, rows) + 1; j <= rows; j++) {
                const unsigned char *row = sm + s * stage_bytes + j * kWgSlot;
                float v[4][8];
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int px = pl + 32 * i;
                    unpack8(*reinterpret_cast<const uint4 *>(row + px * 64 + ((cg ^ ((px >> 1) & 3)) << 4)), v[i]);
                }
#pragma unroll
                for (int c = 0; c < 8; c++) sum[c] += (v[0][c] + v[1][c]) + (v[2][c] + v[3][c]);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&sfree[s]);
#pragma unroll
            for (int c = 0; c < 8; c++) {
                const ff t = ff_two_sum(acc[c].hi, sum[c]);
                acc[c] = {t.hi, acc[c].lo + t.lo};
            }
            if (++s == (uint32_t)stages) {
                s = 0;
                lap++;
            }
        }
        // the 8 lanes of a channel group, then the four warps in order
#pragma unroll
        for (int c = 0; c < 8; c++) {
#pragma unroll
            for (int o = 4; o < 32; o <<= 1) {
                const ff t = ff_two_sum(acc[c].hi, __shfl_xor_sync(0xffffffffu, acc[c].hi, o));
                acc[c] = {t.hi, acc[c].lo + __shfl_xor_sync(0xffffffffu, acc[c].lo, o) + t.lo};
            }
            if (lane < 4) bsum[(warp - 4) * 32 + cg * 8 + c] = ff_value(acc[c]);
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");
        // ---- epilogue: lanes 0-95 (ky = warp - 4, co = lane) -> the CTA's partial ----
        float *pp = a.part + (size_t)blockIdx.x * kWgCols + lane;
        if (warp == 7) pp[9216] = ((bsum[lane] + bsum[32 + lane]) + bsum[64 + lane]) + bsum[96 + lane];
        if (!__all_sync(0xffffffffu, mbar_wait_bounded(done, 0))) ok = false;
        if (!ok && lane == 0) atomicExch(a.err, GLSU_ERR_TIMEOUT);
        tc_fence_after();
        if (warp < 7) {
            const int ky = warp - 4;
#pragma unroll
            for (int kx = 0; kx < 3; kx++) {
                float v[32];
                tmem_ld32(tmem + ((uint32_t)(ky * 32) << 16) + (uint32_t)(kx * 32), v);
#pragma unroll
                for (int ci = 0; ci < 32; ci++) pp[((ky * 3 + kx) * 32 + ci) * 32] = ok ? v[ci] : 0.f;
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) tmem_dealloc(tmem, kWgTmemCols);
}

// Rows of an item: as many as fit two stages and still leave an item for every
// SM (a small image is faster by a row at a time than with SMs idle).
int launch_sur_wgrad(const CUtensorMap &tma, const CUtensorMap &tmg, const SurWgradArgs &a, cudaStream_t s,
                     int *nblocks)
{
    if (a.dil < 1 || a.dil > 64) return fail(GLSU_ERR_INVALID, "surrogate dilation must be 1..64");
    GLSU_TRY(raise_smem_limit((const void *)sur_wgrad_tc_kernel, kWgSmemMax, (int)cudaSharedmemCarveoutMaxShared));
    const int sms = device_sm_count();
    int rows = kWgMaxRows;
    while (rows > 1 && (sur_wgrad_stages(a.dil, rows) < 2 || sur_wgrad_items(a.B, a.H, a.W, a.dil, rows) < sms))
        rows /= 2;
    const int items = sur_wgrad_items(a.B, a.H, a.W, a.dil, rows);
    const int grid = std::min(items, sms);
    sur_wgrad_tc_kernel<<<grid, 256, sur_wgrad_smem_bytes(a.dil, rows), s>>>(tma, tmg, a, items, rows,
                                                                             sur_wgrad_stages(a.dil, rows));
    GLSU_CUDA_TRY(cudaGetLastError());
    *nblocks = grid;
    return GLSU_OK;
}

// Backward of the two layers between 2 and 32 channels, on CUDA cores.  With u
// the 32-channel BF16 side and v the complex side, both sum
//   dW[t] += u[p] v[p + s off_t],  off_t = ((ky-1) d, (kx-1) d),
// layer 0 (LAST false) with u = g0, v = z, s = +1, layer 7 with u = a6, v = dh,
// s = -1; layer 7 also needs, of the same values,
//   g6[p][ci] = [a6 > 0] * sum_t sum_co w7[co][ci][t] dh[p - off_t][co].
// A CTA takes items of kNwRows rows of a 128-pixel segment: v's rows y - d, y,
// y + d with the dilated halo are staged in shared memory as (x, x, y, y), u
// is read once, straight from global memory (the next item's asked into L2
// meanwhile), a warp's step being PX pixels with CH channels a lane.  The nine
// v that a lane reads (one 16-byte broadcast load each, for PX pixels) meet
// its channel pairs in 9 CH packed FMAs, 18 CH with g6.  What bounds it is
// latency: accumulators and weights take 72 registers, so three CTAs of four
// warps with 168 registers a thread fit, and the FMA pipe is busy 40 % of the
// time.  A thread's FP32 chain is at most 512 products long.
// part[blk][co][ci][t], then the biases part[blk][576 + co].
// 16 x 256 x 256 (under the profiler): 116 + 111 us of layer 7 and 91 us of
// layer 0 with weights, values and gradients all read from shared memory; 108
// and 62 us with scalar FMAs and two CTAs of eight warps at 128 registers; the
// training pass 1060 us with those, 1036 us as here (1061 with packed FMAs
// alone, 1048 with four rows an item).
constexpr int kNwSeg = 128, kNwRows = 2, kNwWarps = 4, kNwThreads = 32 * kNwWarps;
constexpr int kNwCtas = 3;                            // per SM
constexpr int kNwItems = 8 * kNwWarps / kNwRows;      // of a CTA, at most: chains of 512 products
constexpr int kNwCols = 576 + 32;  // columns of a partial, at most

__device__ __forceinline__ void prefetch_l2(const void *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

template <bool LAST>
__global__ void __launch_bounds__(kNwThreads, kNwCtas)
    sur_narrow_bwd_kernel(const uint16_t *__restrict__ wide, const float2 *__restrict__ narrow, int B, int H, int W,
                          int dil, int nitems, const float *__restrict__ w7, uint16_t *__restrict__ g6,
                          float *__restrict__ part)
{
    constexpr int CH = LAST ? 2 : 4, PX = CH, LP = 32 / PX;  // channels a lane, pixels a step, lanes a pixel
    constexpr int C2 = CH / 2, ST = kNwWarps * PX;           // channel pairs; pixels between a warp's steps
    constexpr int Q = 4;                                     // steps whose u are loaded together
    constexpr int GR = kNwSeg / (ST * Q);                    // such groups a row
    extern __shared__ __align__(16) float4 vs[];  // (x, x, y, y) [3][kNwRows][SW]; at the end the warps' sums
    const int SW = kNwSeg + 2 * dil;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, cl = lane % LP, hp = lane / LP;
    const int nsx = (W + kNwSeg - 1) / kNwSeg, nby = (H + kNwRows - 1) / kNwRows;
    float2 w[LAST ? 9 : 1][2];
    if (LAST) {
#pragma unroll
        for (int t = 0; t < 9; t++)
#pragma unroll
            for (int k = 0; k < 2; k++)
                w[t][k] = make_float2(w7[k * 288 + cl * 18 + t], w7[k * 288 + cl * 18 + 9 + t]);
    }
    float2 acc[9][2][C2], bias[C2];
#pragma unroll
    for (int c = 0; c < C2; c++) {
        bias[c] = make_float2(0.f, 0.f);
#pragma unroll
        for (int t = 0; t < 9; t++) acc[t][0][c] = acc[t][1][c] = make_float2(0.f, 0.f);
    }
    const int off = warp * PX + hp;  // the lane's pixel in a step

    for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
        const int sx = item % nsx, by = item / nsx % nby, b = item / nsx / nby;
        const int x0 = sx * kNwSeg, y0 = by * kNwRows, nr = min(kNwRows, H - y0);
        const size_t img = (size_t)b * H * W, first = (img + (size_t)y0 * W + x0 + off) * 32 + cl * CH;
        const int left = W - x0 - off;  // the lane's steps at or beyond it lie right of the image
        auto load = [&](int q, uint32_t(&u)[Q][C2]) {
            const uint16_t *src = wide + first + ((size_t)(q / GR) * W + q % GR * (Q * ST)) * 32;
#pragma unroll
            for (int i = 0; i < Q; i++) {
                const bool in = (q % GR * Q + i) * ST < left;
                if constexpr (C2 == 1) {
                    u[i][0] = in ? *reinterpret_cast<const uint32_t *>(src + i * ST * 32) : 0;
                } else {
                    const uint2 v = in ? *reinterpret_cast<const uint2 *>(src + i * ST * 32) : make_uint2(0, 0);
                    u[i][0] = v.x;
                    u[i][C2 - 1] = v.y;
                }
            }
        };
        uint32_t cur[Q][C2], nxt[Q][C2];
        load(0, cur);
        __syncthreads();
        constexpr int V = 6;  // of v a thread loads together
        for (int e0 = tid; e0 < 3 * kNwRows * SW; e0 += V * kNwThreads) {
            float2 v[V];
#pragma unroll
            for (int i = 0; i < V; i++) {
                const int e = e0 + i * kNwThreads, r = e / SW;
                const int ys = y0 + r % kNwRows + (r / kNwRows - 1) * dil, xs = x0 - dil + e - r * SW;
                const bool in = r < 3 * kNwRows && ys >= 0 && ys < H && xs >= 0 && xs < W;
                v[i] = in ? narrow[img + (size_t)ys * W + xs] : make_float2(0.f, 0.f);
            }
#pragma unroll
            for (int i = 0; i < V; i++)
                if (e0 + i * kNwThreads < 3 * kNwRows * SW)
                    vs[e0 + i * kNwThreads] = make_float4(v[i].x, v[i].x, v[i].y, v[i].y);
        }
        // the next item's u on its way into L2, lines of two pixels
        if (item + gridDim.x < nitems) {
            const int ni = item + gridDim.x, nx = ni % nsx * kNwSeg, ny = ni / nsx % nby * kNwRows;
            const uint16_t *src = wide + (size_t)(ni / nsx / nby) * H * W * 32;
#pragma unroll
            for (int e = tid; e < kNwRows * kNwSeg / 2; e += kNwThreads) {
                const int y = ny + e / (kNwSeg / 2), x = nx + e % (kNwSeg / 2) * 2;
                if (y < H && x < W) prefetch_l2(src + ((size_t)y * W + x) * 32);
            }
        }
        __syncthreads();
        const int nq = nr * GR;
#pragma unroll 1
        for (int q = 0; q < nq; q++) {
            if (q + 1 < nq) load(q + 1, nxt);
            const float4 *vr = vs + q / GR * SW + q % GR * (Q * ST) + off;
#pragma unroll
            for (int i = 0; i < Q; i++) {
                float2 a[C2], g = make_float2(0.f, 0.f);
#pragma unroll
                for (int c = 0; c < C2; c++)
                    a[c] = make_float2(__uint_as_float(cur[i][c] << 16),
                                       __uint_as_float(cur[i][c] & 0xFFFF0000u));
#pragma unroll
                for (int t = 0; t < 9; t++) {
                    const int k = LAST ? 8 - t : t;  // the staged neighbour: rows k / 3, columns k % 3
                    const float4 v = (vr + (k / 3) * kNwRows * SW + (k % 3) * dil)[i * ST];
                    const float2 vx = make_float2(v.x, v.y), vy = make_float2(v.z, v.w);
#pragma unroll
                    for (int c = 0; c < C2; c++) {
                        acc[t][0][c] = __ffma2_rn(vx, a[c], acc[t][0][c]);
                        acc[t][1][c] = __ffma2_rn(vy, a[c], acc[t][1][c]);
                    }
                    if (LAST) {
                        g = __ffma2_rn(w[t][0], vx, __ffma2_rn(w[t][1], vy, g));
                        if (t == 4) bias[0] = make_float2(bias[0].x + v.x, bias[0].y + v.z);
                    }
                }
                if constexpr (LAST) {
                    if ((q % GR * Q + i) * ST < left)
                        *reinterpret_cast<uint32_t *>(g6 + first + ((size_t)(q / GR) * W + q % GR * (Q * ST)) * 32 +
                                                      i * ST * 32) =
                            pack_bf2(a[0].x > 0.f ? g.x : 0.f, a[0].y > 0.f ? g.y : 0.f);
                } else {
#pragma unroll
                    for (int c = 0; c < C2; c++) bias[c] = __fadd2_rn(bias[c], a[c]);
                }
            }
#pragma unroll
            for (int i = 0; i < Q; i++)
#pragma unroll
                for (int c = 0; c < C2; c++) cur[i][c] = nxt[i][c];
        }
    }
    // the lanes of a channel, then the warps in order
    __syncthreads();
    float *red = reinterpret_cast<float *>(vs) + warp * kNwCols;
    auto lanes = [&](float x) {
#pragma unroll
        for (int o = LP; o < 32; o <<= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        return x;
    };
#pragma unroll
    for (int t = 0; t < 9; t++)
#pragma unroll
        for (int k = 0; k < 2; k++)
#pragma unroll
            for (int c = 0; c < CH; c++) {
                const float x = lanes(c & 1 ? acc[t][k][c / 2].y : acc[t][k][c / 2].x);
                const int ch = cl * CH + c;
                if (hp == 0) red[(LAST ? k * 32 + ch : ch * 2 + k) * 9 + t] = x;
            }
#pragma unroll
    for (int c = 0; c < CH; c++) {
        const float x = lanes(c & 1 ? bias[c / 2].y : bias[c / 2].x);
        if (hp == 0 && (!LAST || cl == 0)) red[576 + (LAST ? c : cl * CH + c)] = x;
    }
    __syncthreads();
    constexpr int cols = LAST ? kSurL7Params : kSurL0Params;
    const float *rp = reinterpret_cast<const float *>(vs);
    for (int c = tid; c < cols; c += kNwThreads) {
        float x = rp[c];
        for (int k = 1; k < kNwWarps; k++) x += rp[k * kNwCols + c];
        part[(size_t)blockIdx.x * cols + c] = x;
    }
}

int sur_narrow_items(int B, int H, int W) { return B * ((H + kNwRows - 1) / kNwRows) * ((W + kNwSeg - 1) / kNwSeg); }
// One wave of CTAs, more where a thread's chain would pass kNwItems items.
int sur_narrow_blocks(int B, int H, int W)
{
    const int items = sur_narrow_items(B, H, W);
    return std::min(items, std::max(kNwCtas * device_sm_count(), (items + kNwItems - 1) / kNwItems));
}
int sur_narrow_smem(int dil)
{
    return std::max(3 * kNwRows * (kNwSeg + 2 * dil) * 16, kNwWarps * kNwCols * 4);  // at most 48 KB
}

// Deterministic column sums of per-block partials: sum_b part[b][c].  A block
// takes 32 columns; its warps (blockDim.x / 32 of them) sum every nw-th
// partial, then warp 0 adds the warps' sums in order, all in float-float (two
// FP64 operations an element made it FP64-bound).  WGRAD: the columns are
// those of sur_wgrad_tc_kernel, [t][ci][co] then the biases; out has the
// parameters' order W[co][ci][t], b[co].
template <bool WGRAD>
__global__ void __launch_bounds__(1024) sur_reduce_kernel(const float *__restrict__ part, int nblocks, int ncols,
                                                          float *__restrict__ out)
{
    __shared__ float2 s[32][32];
    const int nw = blockDim.x >> 5, w = threadIdx.x >> 5, l = threadIdx.x & 31;
    const int c = blockIdx.x * 32 + l;
    ff acc = {0.f, 0.f};
    if (c < ncols) {
        int b = w;
        for (; b + 3 * nw < nblocks; b += 4 * nw) {
            float v[4];
#pragma unroll
            for (int i = 0; i < 4; i++) v[i] = part[(size_t)(b + i * nw) * ncols + c];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const ff t = ff_two_sum(acc.hi, v[i]);
                acc = {t.hi, acc.lo + t.lo};
            }
        }
        for (; b < nblocks; b += nw) {
            const ff t = ff_two_sum(acc.hi, part[(size_t)b * ncols + c]);
            acc = {t.hi, acc.lo + t.lo};
        }
    }
    s[w][l] = make_float2(acc.hi, acc.lo);
    __syncthreads();
    if (w == 0 && c < ncols) {
        for (int k = 1; k < nw; k++) {
            const ff t = ff_two_sum(acc.hi, s[k][l].x);
            acc = {t.hi, acc.lo + s[k][l].y + t.lo};
        }
        const int o = !WGRAD || c >= 9216 ? c : (c & 31) * 288 + ((c >> 5) & 31) * 9 + (c >> 10);
        out[o] = ff_value(acc);
    }
}

// Threads of a reduction: more warps when there are many partials.
inline int sur_reduce_threads(int nblocks) { return nblocks >= 1024 ? 1024 : nblocks >= 128 ? 512 : 256; }

__global__ void sur_sum_kernel(const double *__restrict__ part, int n, double *__restrict__ out)
{
    double s = 0;
    for (int i = threadIdx.x; i < n; i += 32) s += part[i];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) *out = s;
}

// ---------------------------------------------------------------------------
// Adam and weight packing
// ---------------------------------------------------------------------------
__global__ void sur_adam_kernel(float *__restrict__ w, const float *__restrict__ grad, float *__restrict__ m,
                                float *__restrict__ v, int n, float lr, float b1, float b2, float eps, float c1,
                                float c2)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = grad[i];
    const float mi = b1 * m[i] + (1 - b1) * gi;
    const float vi = b2 * v[i] + (1 - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    w[i] -= lr * (mi * c1) / (sqrtf(vi * c2) + eps);
}

__device__ __forceinline__ float bf16_round(float f) { return __bfloat162float(__float2bfloat16_rn(f)); }

// Element index in the packed B operand (layout of SurTc<NOUT>): tap
// t = 3 dy + dx, K index k (input channel of the layer), N index n (output
// channel): [dx][kc = k / 16][h = (k / 8) % 2][row NOUT (2 - dy) + n][k % 8].
template <int NOUT> __device__ __forceinline__ int sur_bpack_index(int t, int k, int n)
{
    const int dy = t / 3, dx = t % 3;
    return ((dx * 2 + k / 16) * 2 + (k / 8) % 2) * SurTc<NOUT>::BROWS * 8 + (NOUT * (2 - dy) + n) * 8 + k % 8;
}

// From the FP32 master parameters (per layer W[co][ci][3][3] then b[co]):
//   pk_fwd[l] with B[n = co][k = ci] and pk_bwd[l] with B[n = ci][k = co] of
//   the flipped tap 8 - t (the transposed, flipped kernel of the
//   backward-data pass) for the six tensor-core layers; pk7 (if not null,
//   zeroed beforehand) with B[n = co < 2][k = ci] of the last layer; BF16-
//   rounded FP32 copies of layers 0 and 7.
__global__ void sur_pack_kernel(const float *__restrict__ master, uint16_t *__restrict__ pk_fwd,
                                uint16_t *__restrict__ pk_bwd, float *__restrict__ w0r, float *__restrict__ w7r,
                                uint16_t *__restrict__ pk7)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < 576) w0r[i] = bf16_round(master[i]);
    const int off7 = kSurL0Params + 6 * kSurL32Params;
    if (i < 576) {
        w7r[i] = bf16_round(master[off7 + i]);
        if (pk7) {
            const __nv_bfloat16 h = __float2bfloat16_rn(master[off7 + i]);
            pk7[sur_bpack_index<16>(i % 9, (i / 9) % 32, i / 288)] = *reinterpret_cast<const uint16_t *>(&h);
        }
    }
    if (i >= 6 * 9216) return;
    const int l = i / 9216, e = i % 9216;
    const int co = e / 288, ci = (e / 9) % 32, t = e % 9;
    const float wv = master[kSurL0Params + l * kSurL32Params + e];
    const __nv_bfloat16 h = __float2bfloat16_rn(wv);
    const uint16_t bits = *reinterpret_cast<const uint16_t *>(&h);
    // forward: B[n = 32 (2 - dy) + co][k = ci] of tap t = 3 dy + dx
    pk_fwd[(size_t)l * 9216 + sur_bpack_index<32>(t, ci, co)] = bits;
    // backward data: B[n = 32 (2 - dy') + ci][k = co] of the flipped tap t' = 8 - t
    pk_bwd[(size_t)l * 9216 + sur_bpack_index<32>(8 - t, co, ci)] = bits;
}

// Gather training crops: x[b] = pool_x[idx[b]][oy:oy+h, ox:ox+w] (complex),
// same for the target.  The crop list travels as a kernel parameter, so a
// step needs no copy and no synchronisation.
constexpr int kSurMaxBatch = 512;
struct SurCrops {
    int4 c[kSurMaxBatch];  // (pool index, oy, ox, unused)
};

__global__ void sur_gather_kernel(const float2 *__restrict__ px, const float2 *__restrict__ pt, int PH, int PW,
                                  const __grid_constant__ SurCrops crops, int B, int h, int w,
                                  float2 *__restrict__ x, float2 *__restrict__ t)
{
    const size_t n = (size_t)B * h * w;
    for (size_t p = (size_t)blockIdx.x * 256 + threadIdx.x; p < n; p += (size_t)gridDim.x * 256) {
        const int xx = (int)(p % w), yy = (int)((p / w) % h), b = (int)(p / ((size_t)w * h));
        const int4 c = crops.c[b];
        const size_t src = ((size_t)c.x * PH + c.y + yy) * PW + c.z + xx;
        x[p] = px[src];
        t[p] = pt[src];
    }
}

}  // namespace glsu
