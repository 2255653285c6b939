// wff_colfft64.cu -- WFF2 column sweep with FFTs in FP64.
//
// The sweep of wff_colfft.cuh (per column S = FFT(R); per wy an inverse
// transform of S . H_k, the threshold, a forward transform, an accumulation;
// one inverse transform at the end) for FP64 handles.  GB300 runs an FP64
// instruction at 1/64 of the FP32 rate, so only their number counts: the
// direct kernel takes 2 (2s + 1) multiply-adds per part, pixel and wy, with
// the first filter repeated over the 2s-row halo of its 64-row tiles; the
// transforms take about 3.2 log2 L instructions per element each.  Window and
// spectrum being symmetric and real (H_k is the real spectrum of the real,
// symmetric window shifted by wy_k), the products take 2 instructions per
// element, not 4.  WFF2 in FP64, 21 x 21 frequencies: 256 x 256 with sigma 10
// 27.6 ms by the direct kernel, 7.6 by this one; 1200 x 20 with sigma 15
// 141 and 5.1 (the direct kernel also works on the padding to 128 columns).
// The error against 64-bit FFTs is no larger (9.2e-16 and 9.9e-16 of the norm
// at 256 x 256).
//
// A transform spreads a value's rounding, and a value that is not finite, over the
// whole column, where the direct kernel's reach is 2s rows.  Columns of R that hold
// such a value, or whose 16-row blocks differ by more than 2^12 in size (so that the
// transform's 2^-52 would pass 2^-40 of the smallest), are noted by the sweep and done
// again directly by wff_local64_kernel.  On 8 noisy and unit-modulus fields none was;
// without any it costs its launch (256 x 256: 6.38 ms either way).
//
// The working transform sits in registers, S and the accumulator in shared
// memory beside the exchange buffer: at this rate one or two warps per SM
// sub-partition already fill the FP64 pipe, so occupancy is given up for
// registers.
#include <cmath>
#include <vector>

#include "wff_colfft.cuh"
#include "wff_common.cuh"

namespace glsu {
namespace colfft {
namespace {

using D256 = Plan<256, 32, 8, 8, 4>;
using D384 = Plan<384, 16, 8, 8, 2, 3>;
using D512 = Plan<512, 64, 8, 8, 8>;
using D640 = Plan<640, 32, 4, 4, 4, 2, 5>;
using D768 = Plan<768, 32, 8, 8, 4, 3>;
using D1024 = Plan<1024, 64, 8, 8, 4, 4>;
using D1280 = Plan<1280, 64, 4, 4, 4, 4, 5>;
using D1536 = Plan<1536, 64, 8, 8, 8, 3>;
using D2048 = Plan<2048, 128, 8, 8, 8, 4>;
using D3072 = Plan<3072, 128, 8, 8, 4, 4, 3>;
using D4096 = Plan<4096, 256, 8, 8, 8, 8>;

constexpr int kRange = 12, kAnyRange = 4096;  // of the exponents of a column's blocks

template <class P> constexpr size_t smem64_per_column() { return sizeof(double2) * (size_t)(P::XBUF + 2 * P::L); }

template <class P, int NCOL>
__global__ void __launch_bounds__(P::T *NCOL)
    wff_colfft64_kernel(const double2 *__restrict__ R, double2 *__restrict__ Cout, int H, int pitch, int nfy,
                        const double *__restrict__ hk, const double2 *__restrict__ tw,
                        const double *__restrict__ thr_ptr, double LN, double out_scale, int range,
                        uint8_t *__restrict__ wide)
{
    constexpr int L = P::L, T = P::T, Q = P::Q;
    extern __shared__ __align__(16) double2 cd_smem[];
    const int col = threadIdx.x / T, t = threadIdx.x % T;
    double2 *xb = cd_smem + (size_t)col * (P::XBUF + 2 * L);
    double2 *S = xb + P::XBUF, *ch = S + L;  // both only ever touched by the thread that owns the element
    const size_t plane = (size_t)H * pitch;
    const int x = blockIdx.x * NCOL + col;
    const double thr = LN * (*thr_ptr), thr2 = thr * thr;
    const int nit = 2 * nfy + 2;
    double2 v[Q];
#pragma unroll 1
    for (int it = 0; it < nit; it++) {
        const double *h = hk + (size_t)((it - 1) >> 1) * L;  // of the pair it belongs to (0 < it < nit - 1)
        if (it == 0) {
#pragma unroll
            for (int m = 0; m < Q; m++) {
                const int row = t + T * m;
                v[m] = row < H ? R[blockIdx.y * plane + (size_t)row * pitch + x] : mkv<double2>(0, 0);
            }
        } else if (it == nit - 1) {
#pragma unroll
            for (int m = 0; m < Q; m++) v[m] = conjf2(ch[t + T * m]);
        } else if (it & 1) {
#pragma unroll
            for (int m = 0; m < Q; m++) {
                const double2 s = S[t + T * m];
                const double g = __ldg(h + t + T * m);
                v[m] = mkv<double2>(s.x * g, -s.y * g);
            }
        }
        if (it == 0) {
            // the upper words of the 16-row blocks' largest parts: their order is that of the magnitudes
            uint32_t *bm = reinterpret_cast<uint32_t *>(xb), *ends = bm + L / 16;
            for (int e = t; e < L / 16 + 2; e += T) bm[e] = e <= L / 16 ? 0u : ~0u;
            col_sync<T>(col);
#pragma unroll
            for (int m = 0; m < Q; m++) {
                const uint32_t u = max((uint32_t)__double2hiint(v[m].x) & 0x7fffffffu,
                                       (uint32_t)__double2hiint(v[m].y) & 0x7fffffffu);
                if (u) atomicMax(&bm[(t + T * m) / 16], u);
            }
            col_sync<T>(col);
            for (int e = t; e < L / 16; e += T)
                if (bm[e]) {
                    atomicMax(&ends[0], bm[e]);
                    atomicMin(&ends[1], bm[e]);
                }
            col_sync<T>(col);
            if (t == 0) {
                const int top = (int)(ends[0] >> 20), low = (int)(ends[1] >> 20);
                wide[(size_t)blockIdx.y * pitch + x] = top >= 2047 || (ends[0] && top - low > range);
            }
            col_sync<T>(col);
        }
        fft<P>(v, xb, tw, t, col);
        if (it == 0) {
#pragma unroll
            for (int m = 0; m < Q; m++) {
                S[t + T * m] = v[m];
                ch[t + T * m] = mkv<double2>(0, 0);
            }
        } else if (it == nit - 1) {
#pragma unroll
            for (int m = 0; m < Q; m++) {
                const int row = t + T * m;
                if (row < H)
                    Cout[blockIdx.y * plane + (size_t)row * pitch + x] =
                        mkv<double2>(v[m].x * out_scale, -v[m].y * out_scale);
            }
        } else if (it & 1) {
            // u = conj(v): hard threshold, rows >= H dropped
#pragma unroll
            for (int m = 0; m < Q; m++) {
                const bool keep = t + T * m < H && v[m].x * v[m].x + v[m].y * v[m].y >= thr2;
                v[m] = keep ? conjf2(v[m]) : mkv<double2>(0, 0);
            }
        } else {
#pragma unroll
            for (int m = 0; m < Q; m++) {
                const double g = __ldg(h + t + T * m);
                double2 a = ch[t + T * m];
                a.x = fma(v[m].x, g, a.x);
                a.y = fma(v[m].y, g, a.y);
                ch[t + T * m] = a;
            }
        }
    }
}

template <class P, int NCOL> int launch64(const WffPlan &Pl, cudaStream_t s)
{
    static_assert(NCOL * smem64_per_column<P>() <= 227 * 1024 && 128 % NCOL == 0, "CTA width");
    const size_t smem = NCOL * smem64_per_column<P>();
    GLSU_TRY(raise_smem_limit((const void *)wff_colfft64_kernel<P, NCOL>, (int)smem));
    const double N = 1.0 / Pl.inv_norm;
    // pitch is a multiple of 128; the columns beyond W are not read by the final pass
    wff_colfft64_kernel<P, NCOL><<<dim3((Pl.W + NCOL - 1) / NCOL, Pl.nfx), P::T * NCOL, smem, s>>>(
        (const double2 *)Pl.d_R, (double2 *)Pl.d_C, Pl.H, Pl.pitch, Pl.nfy, (const double *)Pl.d_h64,
        (const double2 *)Pl.d_tw64, (const double *)Pl.d_thr, P::L * N, 1.0 / ((double)P::L * P::L * N),
        Pl.unit_input ? kAnyRange : kRange, Pl.d_wide64);
    GLSU_CUDA_TRY(cudaGetLastError());
    return GLSU_OK;
}

// The wide columns of R directly: a CTA takes 128 rows of those among 32 columns of a
// plane, one after another, all wy of each.
constexpr int kLocRows = 128, kLocThreads = 256, kLocMaxHalf = 60;
__global__ void __launch_bounds__(kLocThreads)
    wff_local64_kernel(const double2 *__restrict__ R, double2 *__restrict__ Cout, int W, int H, int pitch,
                       const double2 *__restrict__ ey, int nfy, int s, const __grid_constant__ Taps<double, 60> gA,
                       const __grid_constant__ Taps<double, 60> gB, const double *__restrict__ thr_ptr,
                       const uint8_t *__restrict__ wide)
{
    __shared__ double2 D[kLocRows + 4 * kLocMaxHalf], T[kLocRows + 2 * kLocMaxHalf];
    __shared__ double a[2 * kLocMaxHalf + 1], b[2 * kLocMaxHalf + 1];
    const int tid = threadIdx.x, x0 = blockIdx.x * 32, y0 = blockIdx.y * kLocRows, y1 = min(y0 + kLocRows, H);
    const size_t plane = (size_t)blockIdx.z * H * pitch;
    const int xl = x0 + (tid & 31);
    uint32_t todo = __ballot_sync(0xffffffffu, xl < W && wide[(size_t)blockIdx.z * pitch + xl]);  // the same in every warp
    if (!todo) return;
    for (int j = tid; j <= 2 * s; j += kLocThreads) {
        a[j] = gA.g[60 - s + j];
        b[j] = gB.g[60 - s + j];
    }
    const double thr = *thr_ptr;
    const size_t eys = (size_t)H + 2 * kPhasorPad;
    const int nu = y1 - y0 + 2 * s, nr = nu + 2 * s;
    for (; todo; todo &= todo - 1) {
        const int x = x0 + __ffs(todo) - 1;
        const double2 *Rx = R + plane + x;
        double2 acc = make_double2(0, 0);
        for (int k = 0; k < nfy; k++) {
            const double2 *p = ey + k * eys + kPhasorPad;
            for (int i = tid; i < nr; i += kLocThreads) {
                const int y = y0 - 2 * s + i;
                double2 d = make_double2(0, 0);
                if (y >= 0 && y < H) {
                    const double2 r = Rx[(size_t)y * pitch];
                    d = make_double2(r.x * p[y].x - r.y * p[y].y, r.x * p[y].y + r.y * p[y].x);
                }
                D[i] = d;
            }
            __syncthreads();
            for (int i = tid; i < nu; i += kLocThreads) {
                const int y = y0 - s + i;
                double2 u = make_double2(0, 0);
                for (int j = 0; j <= 2 * s; j++) cfma(u, a[j], D[i + j]);
                const bool keep = y >= 0 && y < H && sqrt(u.x * u.x + u.y * u.y) >= thr;
                T[i] = keep ? u : make_double2(0, 0);
            }
            __syncthreads();
            if (y0 + tid < y1) {
                double2 c = make_double2(0, 0);
                for (int j = 0; j <= 2 * s; j++) cfma(c, b[j], T[tid + j]);
                const double2 q = p[y0 + tid];
                acc.x += q.x * c.x + q.y * c.y;
                acc.y += q.x * c.y - q.y * c.x;
            }
        }
        if (y0 + tid < y1) Cout[plane + (size_t)(y0 + tid) * pitch + x] = acc;
        __syncthreads();
    }
}

int launch_local64(const WffPlan &P, cudaStream_t s)
{
    if (P.sy > kLocMaxHalf) return fail(GLSU_ERR_INVALID, "half-size above the compiled ones");
    wff_local64_kernel<<<dim3((P.W + 31) / 32, (P.H + kLocRows - 1) / kLocRows, P.nfx), kLocThreads, 0, s>>>(
        (const double2 *)P.d_R, (double2 *)P.d_C, P.W, P.H, P.pitch, (const double2 *)P.d_ey, P.nfy, P.sy,
        make_taps<double, 60>(P.gy, P.sy, P.inv_norm), make_taps<double, 60>(P.gy, P.sy, 1.0),
        (const double *)P.d_thr, P.d_wide64);
    GLSU_CUDA_TRY(cudaGetLastError());
    return GLSU_OK;
}

constexpr int kLengths64[] = {256, 384, 512, 640, 768, 1024, 1280, 1536, 2048, 3072, 4096};
// FP64 instructions of a transform per element and log2 L (a count of the passes' adds, multiplies and FMAs).
constexpr double kFft64Instr = 3.2;

}  // namespace
}  // namespace colfft

// FP64 instructions per column of the two sweeps (rows of all wy).
static double direct64_instr(const WffPlan &P)
{
    const int S = P.syi, ty = S <= 30 ? 64 : 32;
    return (double)P.H * P.nfy * (2.0 * (2 * S + 1) * (2.0 + 2.0 * S / ty) + 4.0 * (ty + 4.0 * S) / ty + 8.0);
}
static double fft64_instr(int L, int nfy)
{
    return (double)L * (colfft::kFft64Instr * std::log2((double)L) * (2.0 * nfy + 2.0) + 7.0 * nfy);
}

// AUTO for an FP64 handle: the FFT sweep at the shortest compiled length >=
// H + 2s when it takes less than 0.8 of the direct kernel's instructions.
int WffPlan::init_colfft64()
{
    int L = 0;
    for (int l : colfft::kLengths64)
        if (!L && l >= H + 2 * sy) L = l;
    if (prec != GLSU_F64 || !L || fft64_instr(L, nfy) > 0.8 * direct64_instr(*this)) return GLSU_OK;
    // H_k(w) = sum_m g(m) cos((wy_k - 2 pi w / L) m), by the addition theorem from two tables
    std::vector<double> h((size_t)nfy * L), tw(2 * (size_t)L), cw(L), sw(L);
    for (int j = 0; j < L; j++) {
        cw[j] = std::cos(2.0 * M_PI * j / L);
        sw[j] = std::sin(2.0 * M_PI * j / L);
        tw[2 * j] = cw[j];
        tw[2 * j + 1] = -sw[j];
    }
    std::vector<double> ck(sy + 1), sk(sy + 1);
    for (int k = 0; k < nfy; k++) {
        const double wy = p.wyl + (double)k * p.wyi;
        for (int m = 1; m <= sy; m++) {
            ck[m] = 2.0 * gy[sy + m] * std::cos(wy * m);
            sk[m] = 2.0 * gy[sy + m] * std::sin(wy * m);
        }
        for (int w = 0; w < L; w++) {
            double a = gy[sy];
            for (int m = 1, j = w; m <= sy; m++) {
                a += ck[m] * cw[j] + sk[m] * sw[j];
                j += w;
                if (j >= L) j -= L;
            }
            h[(size_t)k * L + w] = a;
        }
    }
    if (cudaMalloc(&d_h64, h.size() * sizeof(double)) != cudaSuccess ||
        cudaMalloc(&d_tw64, tw.size() * sizeof(double)) != cudaSuccess ||
        cudaMalloc((void **)&d_wide64, (size_t)nfx * pitch) != cudaSuccess)
        return fail(GLSU_ERR_ALLOC, "cudaMalloc of the FP64 column FFT tables failed");
    GLSU_CUDA_TRY(cudaMemcpy(d_h64, h.data(), h.size() * sizeof(double), cudaMemcpyHostToDevice));
    GLSU_CUDA_TRY(cudaMemcpy(d_tw64, tw.data(), tw.size() * sizeof(double), cudaMemcpyHostToDevice));
    fft64_L = L;
    return GLSU_OK;
}

static int launch_any64(const WffPlan &P, cudaStream_t s)
{
    using namespace colfft;
    switch (P.fft64_L) {
    case 256: return launch64<D256, 4>(P, s);
    case 384: return launch64<D384, 4>(P, s);
    case 512: return launch64<D512, 2>(P, s);
    case 640: return launch64<D640, 2>(P, s);
    case 768: return launch64<D768, 2>(P, s);
    case 1024: return launch64<D1024, 2>(P, s);
    case 1280: return launch64<D1280, 2>(P, s);
    case 1536: return launch64<D1536, 1>(P, s);
    case 2048: return launch64<D2048, 1>(P, s);
    case 3072: return launch64<D3072, 1>(P, s);
    default: return launch64<D4096, 1>(P, s);
    }
}

int launch_colfft64(const WffPlan &P, cudaStream_t s)
{
    GLSU_TRY(launch_any64(P, s));
    return colfft::launch_local64(P, s);
}

}  // namespace glsu
