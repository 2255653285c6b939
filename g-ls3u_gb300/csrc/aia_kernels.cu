// aia_kernels.cu -- AIA (advanced iterative algorithm) on sm_103a.
//
// Reference: AIA/aia_cpu.cpp:16-263 (CPU) and AIA/aia_cudaf.cu:308-505 (GPU);
// MATLAB definition MatLab/fp_aia.m:50-121.  Each iteration alternates
//   phi-step: per pixel, A1 x = [sum I, sum I cos d, sum I sin d] with A1 built
//             from the frame shifts d only, phi = atan2(-x3, x2);
//   d-step:   per frame, A2 y = [sum I, sum I cos phi, sum I sin phi] with A2
//             built from cos/sin phi summed over all pixels, d = atan2(-y3, y2).
// One launch per iteration: every block does the phi-step of its pixels and
// sums what the d-step needs; the block that finishes last reduces the blocks'
// partials in a fixed order in FP64, solves the 3x3 d-step, prepares the next
// iteration's tables and raises a done flag when the shifts have settled or
// the iteration cap is hit.  The host enqueues all iterations without
// synchronising; launches after the done flag return at once.
//
// The pixels' work is in float-float (pairs of FP32, about 48 bits): an FP64
// instruction takes 64 times an FP32 one here.  With the unit vector, the
// moments and 3M sums in FP64 a pass over 5 frames of 1024^2 took 190 us (its
// bytes 3 us) and the one-block solve behind it 46 us; in float-float, with
// the solve in the last block, an iteration takes 55 us (all three profiled).
// Phases and shifts are as far from 64 bits as before (3.3e-8 of their norm:
// the FP32 sums b and the FP32 result decide), on the frames measured to the
// bit.  Bound now: the float-float chains' latency, then the last block's
// FP64 solve (about 10 us).
#include <cmath>

#include "dpra_ls_ff.cuh"
#include "glsu_internal.cuh"

namespace glsu {

constexpr int kAiaMaxM = 32;
constexpr int kAiaThreads = 256;

// state layout (doubles): [0,M) deltas, [M,2M) old deltas, [2M] err, [2M+1] iterations,
// [2M+2] status (0 ok, else GLSU_ERR_NOT_POSDEF)

// What the phi-step needs of the shifts: their cosines and sines, and rows 2
// and 3 of adj(A1), signed by det(A1) and scaled by a power of two so that a row's
// products with finite sums of intensities stay finite, as float-float.
struct AiaTables {
    float c[kAiaMaxM], s[kAiaMaxM];
    ff adj[2][3];
};

__device__ __forceinline__ ff ff_of(double v)
{
    const float hi = (float)v;
    return {hi, (float)(v - (double)hi)};
}

// Tables of the shifts in state[0, M), by one block (trig in parallel, cs: 2 M doubles of shared memory).
__device__ void aia_tables(const double *__restrict__ state, int M, double *cs, AiaTables *__restrict__ tab)
{
    const int tid = threadIdx.x;
    if (tid < M) {
        double s, c;
        sincos(state[tid], &s, &c);
        cs[2 * tid] = c;
        cs[2 * tid + 1] = s;
        tab->c[tid] = (float)c;
        tab->s[tid] = (float)s;
    }
    __syncthreads();
    if (tid == 0) {
        double a3 = 0, a4 = 0, a6 = 0, a7 = 0, a8 = 0;
        for (int i = 0; i < M; i++) {
            const double c = cs[2 * i], s = cs[2 * i + 1];
            a3 += c; a4 += c * c; a6 += s; a7 += c * s; a8 += s * s;
        }
        const double A[3][3] = {{(double)M, a3, a6}, {a3, a4, a7}, {a6, a7, a8}};
        // cofactor rows 2,3 of the inverse: x = adj(A) b / det(A)
        const double c10 = -(A[0][1] * A[2][2] - A[0][2] * A[2][1]);
        const double c11 = (A[0][0] * A[2][2] - A[0][2] * A[2][0]);
        const double c12 = -(A[0][0] * A[2][1] - A[0][1] * A[2][0]);
        const double c20 = (A[0][1] * A[1][2] - A[0][2] * A[1][1]);
        const double c21 = -(A[0][0] * A[1][2] - A[0][2] * A[1][0]);
        const double c22 = (A[0][0] * A[1][1] - A[0][1] * A[1][0]);
        const double det = A[0][0] * (A[1][1] * A[2][2] - A[1][2] * A[2][1]) -
                           A[0][1] * (A[1][0] * A[2][2] - A[1][2] * A[2][0]) +
                           A[0][2] * (A[1][0] * A[2][1] - A[1][1] * A[2][0]);
        const double top = fmax(fmax(fmax(fabs(c10), fabs(c11)), fabs(c12)), fmax(fmax(fabs(c20), fabs(c21)), fabs(c22)));
        const double sg = ldexp(det < 0 ? -1.0 : 1.0, top > 0 ? -2 - ilogb(top) : 0);
        tab->adj[0][0] = ff_of(sg * c10); tab->adj[0][1] = ff_of(sg * c11); tab->adj[0][2] = ff_of(sg * c12);
        tab->adj[1][0] = ff_of(sg * c20); tab->adj[1][1] = ff_of(sg * c21); tab->adj[1][2] = ff_of(sg * c22);
    }
}

// (X, -Y) / hypot(X, Y) in float-float; (1, 0) where both vanish.  False where
// that is not finite, with no number in *c and *s.
__device__ __forceinline__ bool aia_unit(ff X, ff Y, ff *c, ff *s)
{
    // scaled by a power of two so that the larger part is in [1, 2)
    const float mx = fmaxf(fabsf(X.hi), fabsf(Y.hi));
    const int e = min(126, (int)(__float_as_uint(mx) >> 23) - 127);
    const float sc = __uint_as_float((uint32_t)(127 - e) << 23);
    X = ff{X.hi * sc, X.lo * sc};
    Y = ff{Y.hi * sc, Y.lo * sc};
    const float n = fmaf(X.hi, X.hi, Y.hi * Y.hi);
    if (!(n > 0.f && n <= 3.402823466e38f)) {
        *c = ff{n == 0.f ? 1.f : n - n, 0.f};
        *s = ff{n == 0.f ? 0.f : n - n, 0.f};
        return n == 0.f;
    }
    const float r = rsqrtf(n);
    const ff u = ff_mul_f(X, r), v = ff_mul_f(Y, r);  // within 2^-22 of unit length
    const ff t = ff_add(ff_mul(u, u), ff_mul(v, v));
    const float d = (1.f - t.hi) - t.lo;              // 1 - |(u, v)|^2, the first difference exact
    const float k = d * fmaf(0.375f, d, 0.5f);        // (1 - d)^(-1/2) - 1
    *c = ff_fast_two_sum(u.hi, fmaf(u.hi, k, u.lo));
    *s = ff_neg(ff_fast_two_sum(v.hi, fmaf(v.hi, k, v.lo)));
    return true;
}

// The d-step by the block that finished last (AIA/aia_cpu.cpp:172-263): reduce
// the partials in a fixed order, solve A2 y = b for every frame (Cholesky, as
// LAPACKE_dposv at AIA/aia_cpu.cpp:235), update the deltas.  The convergence
// measure is max_i |delta_i - old_i| (AIA_CUDAF, AIA/aia_cpu.cpp:249-263), or
// with rel != 0 the change of the shifts relative to the first, max_i |(delta_i
// - delta_0) - (old_i - old_0)| (AIA_CUDAF_YC2, AIA/aia_cudaf_v2.cu:665-677),
// which does not see the common rotation the two steps leave free.
__device__ void aia_solve(const double *__restrict__ part, int nblocks, int M, int N, double *__restrict__ state,
                          int *__restrict__ done, int max_iter, double max_err, int rel, AiaTables *__restrict__ tab)
{
    __shared__ double red[kAiaThreads / 32][32], tot[5 + 3 * kAiaMaxM], dnew[kAiaMaxM], cs[2 * kAiaMaxM];
    __shared__ double U[3][3];
    __shared__ int bad;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nv = 5 + 3 * M;
    for (int v0 = 0; v0 < nv; v0 += 32) {
        double t = 0;
        if (v0 + lane < nv)
#pragma unroll 8
            for (int b = wid; b < nblocks; b += kAiaThreads / 32) t += __ldcg(&part[(size_t)b * nv + v0 + lane]);
        red[wid][lane] = t;
        __syncthreads();
        if (wid == 0 && v0 + lane < nv) {
            double a = 0;
            for (int w = 0; w < kAiaThreads / 32; w++) a += red[w][lane];
            tot[v0 + lane] = a;
        }
        __syncthreads();
    }
    if (tid == 0) {
        const double A[3][3] = {{(double)N, tot[0], tot[2]}, {tot[0], tot[1], tot[3]}, {tot[2], tot[3], tot[4]}};
        bad = 0;
        for (int j = 0; j < 3 && !bad; j++) {
            double s = A[j][j];
            for (int k = 0; k < j; k++) s -= U[k][j] * U[k][j];
            if (!(s > 0)) {
                state[2 * M + 2] = (double)GLSU_ERR_NOT_POSDEF;
                *done = 1;
                bad = 1;
                break;
            }
            U[j][j] = sqrt(s);
            for (int i = j + 1; i < 3; i++) {
                double t = A[j][i];
                for (int k = 0; k < j; k++) t -= U[k][j] * U[k][i];
                U[j][i] = t / U[j][j];
            }
        }
    }
    __syncthreads();
    if (bad) return;
    if (tid < M) {
        double b[3] = {tot[5 + 3 * tid], tot[6 + 3 * tid], tot[7 + 3 * tid]};
        double y[3];
        for (int i = 0; i < 3; i++) {
            double t = b[i];
            for (int k = 0; k < i; k++) t -= U[k][i] * y[k];
            y[i] = t / U[i][i];
        }
        for (int i = 2; i >= 0; i--) {
            double t = y[i];
            for (int k = i + 1; k < 3; k++) t -= U[i][k] * b[k];
            b[i] = t / U[i][i];
        }
        dnew[tid] = atan2(-b[2], b[1]);
    }
    __syncthreads();
    if (tid == 0) {
        double err = 0;
        const double new0 = dnew[0], old0 = state[0];
        for (int m = 0; m < M; m++) {
            const double e = rel ? fabs((dnew[m] - new0) - (state[m] - old0)) : fabs(dnew[m] - state[m]);
            err = e > err ? e : err;
        }
        for (int m = 0; m < M; m++) {
            state[M + m] = state[m];
            state[m] = dnew[m];
        }
        const double it = state[2 * M + 1] + 1;
        state[2 * M + 1] = it;
        state[2 * M] = err;
        if (!(err > max_err) || it >= max_iter) *done = 1;
    }
    __syncthreads();
    aia_tables(state, M, cs, tab);
}

template <typename IMG, int MM, bool FINAL>
__global__ void __launch_bounds__(kAiaThreads)
    aia_pass_kernel(const IMG *__restrict__ f, int M, int N, double *__restrict__ state, int *__restrict__ done,
                    double *__restrict__ part, AiaTables *__restrict__ tab, unsigned *__restrict__ count, int max_iter,
                    double max_err, int rel, float *__restrict__ phi)
{
    if (!FINAL && *done) return;
    __shared__ AiaTables T;
    __shared__ ff red[kAiaThreads / 32][5 + 3 * MM];
    __shared__ bool last;
    __shared__ ff d0;  // FINAL: delta_0 in [-pi, pi]; the shifts given by a caller may be any
    const int tid = threadIdx.x;
    if (FINAL && tid == 0) {
        double sn, cs;
        sincos(state[0], &sn, &cs);
        d0 = ff_of(atan2(sn, cs));
    }
    for (int e = tid; e < (int)(sizeof(AiaTables) / 4); e += kAiaThreads)
        reinterpret_cast<float *>(&T)[e] = __ldcg(reinterpret_cast<const float *>(tab) + e);
    __syncthreads();
    ff acc[FINAL ? 1 : 5 + 3 * MM];
    if constexpr (!FINAL) {
#pragma unroll
        for (int v = 0; v < 5 + 3 * MM; v++) acc[v] = ff{0.f, 0.f};
    }
    for (int j = blockIdx.x * kAiaThreads + tid; j < N; j += gridDim.x * kAiaThreads) {
        float I[MM];
        float b0 = 0, b1 = 0, b2 = 0;
#pragma unroll
        for (int i = 0; i < MM; i++) {
            I[i] = 0;
            if (i < M) {
                I[i] = (float)f[(size_t)i * N + j];
                b0 += I[i];
                b1 = fmaf(I[i], T.c[i], b1);
                b2 = fmaf(I[i], T.s[i], b2);
            }
        }
        const ff X = ff_add(ff_add(ff_mul_f(T.adj[0][0], b0), ff_mul_f(T.adj[0][1], b1)), ff_mul_f(T.adj[0][2], b2));
        const ff Y = ff_add(ff_add(ff_mul_f(T.adj[1][0], b0), ff_mul_f(T.adj[1][1], b1)), ff_mul_f(T.adj[1][2], b2));
        ff c, s;  // cos and sin of phi = atan2(-Y, X), X ~ x2, Y ~ x3
        if (!aia_unit(X, Y, &c, &s)) {
            // an intensity, or a sum of them, is not finite: as 64 bits make it of infinities and NaN
            const float x = fmaf(T.adj[0][0].hi, b0, fmaf(T.adj[0][1].hi, b1, T.adj[0][2].hi * b2));
            const float y = fmaf(T.adj[1][0].hi, b0, fmaf(T.adj[1][1].hi, b1, T.adj[1][2].hi * b2));
            if constexpr (FINAL) {
                const float p = atan2f(-y, x) + d0.hi;
                phi[j] = p > 3.14159274f ? p - 6.28318531f : p < -3.14159274f ? p + 6.28318531f : p;
                continue;
            } else if (!isinf(x) && !isinf(y)) {  // hypot is NaN, not infinite
                c = ff{1.f, 0.f};
                s = ff{0.f, 0.f};
            }
        }
        if constexpr (FINAL) {
            // phi + delta_0 in (-pi, pi]: atan2f, corrected by the sine of what it is off
            const float p0 = atan2f(s.hi, c.hi);
            ff sp, cm1;
            ff_sincos_m1(ff_from(p0), &sp, &cm1);
            const ff cp = ff_add(cm1, ff_from(1.f));
            const ff off = ff_sub(ff_mul(s, cp), ff_mul(c, sp));
            ff p = ff_add(ff_add(ff_from(p0), off), d0);
            const ff pi = {3.14159274101257324f, -8.74227800036e-8f}, two_pi = {6.28318548202514648f, -1.74845560007e-7f};
            const ff over = ff_sub(p, pi), under = ff_add(p, pi);
            if (over.hi > 0.f) p = ff_sub(p, two_pi);
            else if (under.hi < 0.f) p = ff_add(p, two_pi);
            phi[j] = p.hi;
        } else {
            acc[0] = ff_add(acc[0], c);
            acc[1] = ff_add(acc[1], ff_mul(c, c));
            acc[2] = ff_add(acc[2], s);
            acc[3] = ff_add(acc[3], ff_mul(c, s));
            acc[4] = ff_add(acc[4], ff_mul(s, s));
#pragma unroll
            for (int i = 0; i < MM; i++) {
                if (i < M) {
                    acc[5 + 3 * i] = ff_add(acc[5 + 3 * i], ff_from(I[i]));
                    acc[6 + 3 * i] = ff_add(acc[6 + 3 * i], ff_mul_f(c, I[i]));
                    acc[7 + 3 * i] = ff_add(acc[7 + 3 * i], ff_mul_f(s, I[i]));
                }
            }
        }
    }
    if constexpr (!FINAL) {
        const int lane = tid & 31, wid = tid >> 5;
        const int nv = 5 + 3 * M;
#pragma unroll
        for (int v = 0; v < 5 + 3 * MM; v++) {
            if (v < nv) {
                ff t = acc[v];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1)
                    t = ff_add(t, ff{__shfl_down_sync(0xffffffffu, t.hi, o), __shfl_down_sync(0xffffffffu, t.lo, o)});
                if (lane == 0) red[wid][v] = t;
            }
        }
        __syncthreads();
        for (int v = tid; v < nv; v += kAiaThreads) {
            double t = 0;
            for (int w = 0; w < kAiaThreads / 32; w++) t += (double)red[w][v].hi + (double)red[w][v].lo;
            part[(size_t)blockIdx.x * nv + v] = t;
        }
        __threadfence();  // the partials before the ticket
        __syncthreads();
        if (tid == 0) last = atomicInc(count, gridDim.x - 1) == gridDim.x - 1;  // wraps to 0 for the next launch
        __syncthreads();
        if (last) {
            __threadfence();
            aia_solve(part, gridDim.x, M, N, state, done, max_iter, max_err, rel, tab);
        }
    }
}

// Start of a run: the shifts are in state[0, M); clears the rest and makes the first tables.
__global__ void aia_init_kernel(double *__restrict__ state, int M, int *__restrict__ done, unsigned *__restrict__ count,
                                AiaTables *__restrict__ tab)
{
    __shared__ double cs[2 * kAiaMaxM];
    for (int e = M + threadIdx.x; e < 2 * M + 3; e += blockDim.x) state[e] = 0;
    if (threadIdx.x == 0) {
        *done = 0;
        *count = 0;
    }
    aia_tables(state, M, cs, tab);
}

// Normalise the deltas relative to the first one (AIA/aia_cpu.cpp:95-99).
__global__ void aia_norm_kernel(double *__restrict__ state, int M)
{
    const int i = threadIdx.x;
    const double d0 = state[0];
    const double v = i < M ? state[i] - d0 : 0.0;
    __syncthreads();
    if (i < M) state[i] = atan2(sin(v), cos(v));
}

size_t aia_tables_bytes() { return sizeof(AiaTables) + sizeof(unsigned); }

template <typename IMG, bool FINAL>
static int pass_t(const AiaDev &a, const void *d_frames, int max_iter, double max_err, float *d_phi, cudaStream_t s)
{
    const IMG *f = (const IMG *)d_frames;
    AiaTables *tab = (AiaTables *)a.d_tab;
#define GLSU_AIA(MMV)                                                                                                 \
    aia_pass_kernel<IMG, MMV, FINAL><<<a.nblocks, kAiaThreads, 0, s>>>(                                               \
        f, a.M, a.N, a.d_state, a.d_done, a.d_part, tab, (unsigned *)(tab + 1), max_iter, max_err,                    \
        a.err_mode == GLSU_AIA_ERR_RELATIVE ? 1 : 0, d_phi)
    if (a.M <= 4) GLSU_AIA(4);
    else if (a.M <= 8) GLSU_AIA(8);
    else if (a.M <= 16) GLSU_AIA(16);
    else GLSU_AIA(32);
#undef GLSU_AIA
    GLSU_CUDA_TRY(cudaGetLastError());
    return GLSU_OK;
}

int aia_launch_iteration(const AiaDev &a, int img_type, const void *d_frames, int max_iter, double max_err,
                         cudaStream_t s)
{
    if (img_type == GLSU_U8) return pass_t<uint8_t, false>(a, d_frames, max_iter, max_err, nullptr, s);
    if (img_type == GLSU_F32) return pass_t<float, false>(a, d_frames, max_iter, max_err, nullptr, s);
    return fail(GLSU_ERR_INVALID, "AIA frames must be GLSU_U8 or GLSU_F32");
}

int aia_launch_init(const AiaDev &a, const double *h_deltas, cudaStream_t s)
{
    GLSU_CUDA_TRY(cudaMemcpyAsync(a.d_state, h_deltas, sizeof(double) * a.M, cudaMemcpyHostToDevice, s));
    AiaTables *tab = (AiaTables *)a.d_tab;
    aia_init_kernel<<<1, 64, 0, s>>>(a.d_state, a.M, a.d_done, (unsigned *)(tab + 1), tab);
    GLSU_CUDA_TRY(cudaGetLastError());
    return GLSU_OK;
}

int aia_launch_finalize(const AiaDev &a, int img_type, const void *d_frames, float *d_phi, cudaStream_t s)
{
    if (img_type == GLSU_U8) GLSU_TRY((pass_t<uint8_t, true>(a, d_frames, 0, 0, d_phi, s)));
    else if (img_type == GLSU_F32) GLSU_TRY((pass_t<float, true>(a, d_frames, 0, 0, d_phi, s)));
    else return fail(GLSU_ERR_INVALID, "AIA frames must be GLSU_U8 or GLSU_F32");
    aia_norm_kernel<<<1, 32, 0, s>>>(a.d_state, a.M);
    GLSU_CUDA_TRY(cudaGetLastError());
    return GLSU_OK;
}

}  // namespace glsu
