// evp_vox.cuh -- device helpers shared by the per-voxel kernels: block reductions, field loads and
// stores, the power law and the constitutive law (evp_kernels.cu, evp_newton.cu).
#pragma once
#include "evp_dev.cuh"
#include "evp_math.cuh"

namespace evp {

constexpr int kBlock = 256;
constexpr int kC0Block = 64;

// ---------------------------------------------------------------- reductions
// NS sums then NM maxima per thread -> one partial per block (stored field-major,
// partials[f * nblocks + block], in the body's block coordinates) -> the last block to finish
// folds them: lane l of a field's warp adds blocks l, l + 32, ... in order, then a fixed shuffle
// tree, so the result does not depend on timing.
//
// On small grids this is most of a pass, and it is all latency, so nothing goes one field at a
// time: a warp reduces 32 fields by halving exchanges (31 shuffles instead of 160; lane f ends
// with field f), the block's warps are added by a thread per field, and the last block's warps
// fold four fields each at once.  Event-timed launches, with blocks of 64 at 16^3 instead of 256:
// k_corr 15.9 -> 13.8 us, k_fft_x_inv 15.8 -> 13.8, k_c0 (72 sums) 74 -> 47 (an empty launch reads
// 5 us); at 64^3 k_corr 31.6 -> 25.4, k_fft_x_inv 39 -> 36, k_c0 500 -> 434, and k_diag 240 -> 132,
// whose block pairs one thread used to fold.
template <bool MAX>
__device__ __forceinline__ double red_op(double a, double b) { return MAX ? fmax(a, b) : a + b; }

// W (a power of two, at most 32) values over the warp: lane l ends with value l >> (5 - log2 W)
template <int W, bool MAX>
__device__ __forceinline__ double warp_reduce_many(double (&x)[W], int lane) {
    int dist = 16;
#pragma unroll
    for (int h = W / 2; h >= 1; h /= 2, dist /= 2) {
        const bool up = lane & dist;
#pragma unroll
        for (int f = 0; f < h; f++) {
            const double send = up ? x[f] : x[f + h], keep = up ? x[f + h] : x[f];
            x[f] = red_op<MAX>(keep, __shfl_xor_sync(0xffffffffu, send, dist));
        }
    }
    double y = x[0];
    for (; dist >= 1; dist /= 2) y = red_op<MAX>(y, __shfl_xor_sync(0xffffffffu, y, dist));
    return y;
}
__host__ __device__ constexpr int pow2_at_least(int n) { return n <= 1 ? 1 : 2 * pow2_at_least((n + 1) / 2); }
__host__ __device__ constexpr int log2_of(int n) { return n <= 1 ? 0 : 1 + log2_of(n / 2); }
// fields [F0, F0 + NF) of the thread's values into sh[f] (one row per warp)
template <int NF, bool MAX, int F0 = 0>
__device__ __forceinline__ void warp_fields(const double* vals, double* sh, int lane, int stride = 1) {
    if constexpr (F0 < NF) {
        constexpr int n = NF - F0 < 32 ? NF - F0 : 32, W = pow2_at_least(n);
        double x[W];
#pragma unroll
        for (int f = 0; f < W; f++) x[f] = f < n ? vals[(F0 + f) * stride] : (MAX ? -EVP_HUGE : 0.0);
        const double y = warp_reduce_many<W, MAX>(x, lane);
        constexpr int sft = 5 - log2_of(W);
        if ((lane & ((1 << sft) - 1)) == 0 && (lane >> sft) < n) sh[F0 + (lane >> sft)] = y;
        warp_fields<NF, MAX, F0 + 32>(vals, sh, lane, stride);
    }
}
// fold of fields f0, f0 + step, f0 + 2 step, f0 + 3 step (below nf) over the block partials by one warp
template <bool MAX>
__device__ __forceinline__ void fold_four(const double* partials, int nblk, int f0, int step, int nf, double* out, int lane) {
    double s[4];
    const double* q[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        s[i] = MAX ? -EVP_HUGE : 0.0;
        q[i] = partials + (size_t)(f0 + i * step < nf ? f0 + i * step : f0) * nblk;
    }
    int b = lane;
    for (; b + 3 * 32 < nblk; b += 4 * 32) {
        double x[4][4];
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) x[i][j] = __ldcg(q[i] + b + 32 * j);
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) s[i] = red_op<MAX>(s[i], x[i][j]);
    }
    for (; b < nblk; b += 32)
#pragma unroll
        for (int i = 0; i < 4; i++) s[i] = red_op<MAX>(s[i], __ldcg(q[i] + b));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int i = 0; i < 4; i++) s[i] = red_op<MAX>(s[i], __shfl_down_sync(0xffffffffu, s[i], o));
    if (lane == 0)
#pragma unroll
        for (int i = 0; i < 4; i++)
            if (f0 + i * step < nf) out[f0 + i * step] = s[i];
}

// Returns true in every thread of the block that folded (out is then written, visible to the
// block after a __syncthreads); blocks of at most 8 warps, whole warps.  stride: between a thread's sums.
template <int NS, int NM>
__device__ bool reduce_store(const double* sums, const double* maxs, double* partials, double* out, unsigned int* counter,
                             const VB& vb, int stride = 1) {
    constexpr int NF = NS + NM;
    __shared__ double sh[8][NF];
    __shared__ bool last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    warp_fields<NS, false>(sums, sh[warp], lane, stride);
    warp_fields<NM, true>(maxs, sh[warp] + NS, lane);
    __syncthreads();
    for (int f = threadIdx.x; f < NF; f += blockDim.x) {
        double x = sh[0][f];
        for (int w = 1; w < nw; w++) x = f < NS ? x + sh[w][f] : fmax(x, sh[w][f]);
        partials[(size_t)f * vb.nx + vb.x] = x;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = (atomicAdd(counter, 1u) == (unsigned)vb.nx - 1u);
    __syncthreads();
    if (!last) return false;
    __threadfence();
    for (int f = warp; f < NS; f += 4 * nw) fold_four<false>(partials, vb.nx, f, nw, NS, out, lane);
    for (int f = NS + warp; f < NF; f += 4 * nw) fold_four<true>(partials, vb.nx, f, nw, NF, out, lane);
    if (threadIdx.x == 0) *counter = 0;
    return true;
}

__device__ __forceinline__ void set_err(int* err, int bit) { atomicOr(err, bit); }

__device__ __forceinline__ void ld9(const double* __restrict__ a, long long N, long long v, double* o) {
#pragma unroll
    for (int c = 0; c < 9; c++) o[c] = a[c * N + v];
}
__device__ __forceinline__ void st9(double* __restrict__ a, long long N, long long v, const double* o) {
#pragma unroll
    for (int c = 0; c < 9; c++) a[c * N + v] = o[c];
}
__device__ __forceinline__ void ld6(const double* __restrict__ a, long long N, long long v, double* o) {
#pragma unroll
    for (int c = 0; c < 6; c++) o[c] = a[c * N + v];
}
__device__ __forceinline__ void st6(double* __restrict__ a, long long N, long long v, const double* o) {
#pragma unroll
    for (int c = 0; c < 6; c++) a[c * N + v] = o[c];
}
__device__ __forceinline__ void eye9(double* a) {
#pragma unroll
    for (int c = 0; c < 9; c++) a[c] = (c % 4 == 0) ? 1.0 : 0.0;
}

// 1 / x by Newton-Raphson from the hardware's approximation (rcp.approx.ftz.f64, 20 bits: two steps
// of y += y (1 - x y) reach FP64 rounding).  Branch free, so that independent reciprocals overlap:
// the compiler's division tests for its slow path one quotient after the other.  For normal x whose
// reciprocal is normal; 1 / 0 gives NaN.
__device__ __forceinline__ double rcp_nr(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    y = fma(y, fma(-x, y, 1.0), y);
    return fma(y, fma(-x, y, 1.0), y);
}

__host__ __device__ constexpr int tri(int i, int j) { return i >= j ? i * (i + 1) / 2 + j : j * (j + 1) / 2 + i; }

// the general inverse, for a matrix that the symmetric one refuses
__device__ __noinline__ inline int inv_general6(const double* h21, double* x21) {
    double J[36];
#pragma unroll
    for (int i = 0; i < 6; i++)
#pragma unroll
        for (int j = 0; j < 6; j++) J[6 * i + j] = h21[tri(i, j)];
    const int info = inv_unrolled<6>(J);
#pragma unroll
    for (int i = 0; i < 6; i++)
#pragma unroll
        for (int j = 0; j <= i; j++) x21[tri(i, j)] = J[6 * i + j];
    return info;
}
// Inverse of a symmetric positive definite 6x6 matrix (packed lower triangles) from its L D L^T
// factors: M = L^-1, X = M^T D^-1 M, 21 entries instead of 36 and no pivoting.  A pivot that is not
// positive sends it to the general elimination.  Returns nonzero for a singular matrix.
__device__ __forceinline__ int inv_sym6(const double (&h)[21], double (&x)[21]) {
    double a[21], inv[6];
    bool spd = true;
#pragma unroll
    for (int i = 0; i < 21; i++) a[i] = h[i];
#pragma unroll
    for (int k = 0; k < 6; k++) {
        spd = spd && a[tri(k, k)] > 0.0;
        inv[k] = rcp_nr(a[tri(k, k)]);
        double l[6];
#pragma unroll
        for (int i = k + 1; i < 6; i++) l[i] = a[tri(i, k)] * inv[k];
#pragma unroll
        for (int i = k + 1; i < 6; i++) {
#pragma unroll
            for (int j = k + 1; j <= i; j++) a[tri(i, j)] -= l[i] * a[tri(j, k)];
        }
#pragma unroll
        for (int i = k + 1; i < 6; i++) a[tri(i, k)] = l[i];  // L below the diagonal
    }
    if (!spd) {
        double hh[21], xx[21];
#pragma unroll
        for (int i = 0; i < 21; i++) hh[i] = h[i];
        const int info = inv_general6(hh, xx);
#pragma unroll
        for (int i = 0; i < 21; i++) x[i] = xx[i];
        return info;
    }
#pragma unroll
    for (int j = 0; j < 6; j++)
#pragma unroll
        for (int i = j + 1; i < 6; i++) {  // column j of M below the diagonal, in place of L's rows used up
            double t = a[tri(i, j)];
#pragma unroll
            for (int k = j + 1; k < i; k++) t += a[tri(i, k)] * x[tri(k, j)];
            x[tri(i, j)] = -t;
        }
#pragma unroll
    for (int i = 0; i < 6; i++)
#pragma unroll
        for (int j = 0; j <= i; j++) {  // X_ij = sum over k >= i of M_ki M_kj / d_k, rows in rising order
            double t = i == j ? inv[i] : inv[i] * x[tri(i, j)];
#pragma unroll
            for (int k = i + 1; k < 6; k++) t += inv[k] * x[tri(k, i)] * x[tri(k, j)];
            a[tri(i, j)] = t;
        }
#pragma unroll
    for (int i = 0; i < 21; i++) x[i] = a[i];
    return 0;
}

// |x|^e for the power law: integer exponents by binary powering, else pow().
__device__ __forceinline__ double powabs(double x, double e, int int_exp) {
    double a = fabs(x);
    if (int_exp) {
        int k = (int)e;
        double r = 1.0, b = a;
        while (k) {
            if (k & 1) r *= b;
            b *= b;
            k >>= 1;
        }
        return r;
    }
    return pow(a, e);
}

// ---------------------------------------------------------------- local constitutive solve
// plastic_strain_rate (various_functions.f90:1367-1419) + elastic_strain_rate (1422-1436)
template <int NS>
__device__ __forceinline__ void constitutive(const PhaseDev& ph, const double* __restrict__ sch, long long N, long long v,
                                             const double (&tt)[NS][2], const double (&sg)[6], double (&edotp)[6],
                                             double (&dd)[15], double (&gamdot)[NS]) {
#pragma unroll
    for (int i = 0; i < 6; i++) edotp[i] = 0.0;
#pragma unroll
    for (int i = 0; i < 15; i++) dd[i] = 0.0;
#pragma unroll
    for (int is = 0; is < NS; is++) {
        if (is < ph.nsyst) {
            double sc[5];
#pragma unroll
            for (int c = 0; c < 5; c++) sc[c] = sch[(is * 5 + c) * N + v];
            double rss = sc[0] * sg[0] + sc[1] * sg[1] + sc[2] * sg[2] + sc[3] * sg[3] + sc[4] * sg[4];
            const double tau = (rss - 0.0 < 0.0) ? tt[is][1] : tt[is][0];  // kin(is) == 0
            rss = (rss - 0.0) / tau;
            const double dum = ph.gamd0[is] * powabs(rss, ph.nrs[is] - 1.0, ph.int_exp);
            const double rss1 = ph.nrs[is] * dum / tau;
            const double rss2 = rss * dum;
            gamdot[is] = rss2;
            int q = 0;
#pragma unroll
            for (int jj = 0; jj < 5; jj++) {
                edotp[jj] = edotp[jj] + sc[jj] * rss2;
#pragma unroll
                for (int ii = 0; ii <= jj; ii++) dd[q++] += sc[ii] * sc[jj] * rss1;
            }
        } else {
            gamdot[is] = 0.0;
        }
    }
}
__device__ __forceinline__ double dd_at(const double (&dd)[15], int i, int j) {
    if (i > 4 || j > 4) return 0.0;
    int a = i < j ? i : j, b = i < j ? j : i;
    return dd[b * (b + 1) / 2 + a];
}

// harden (various_functions.f90:1439-1491)
template <int NS>
__device__ __forceinline__ void harden(const PhaseDev& ph, const double* __restrict__ crss, long long N, long long v,
                                       const double (&gamdot)[NS], double gamma0, double tdot, double (&tau)[NS][2], double& gamma1) {
    double deltgam = 0.0;
#pragma unroll
    for (int is = 0; is < NS; is++)
        if (is < ph.nsyst) deltgam = deltgam + fabs(gamdot[is]) * tdot;
    gamma1 = gamma0 + deltgam;
#pragma unroll
    for (int is = 0; is < NS; is++) { tau[is][0] = 0.0; tau[is][1] = 0.0; }
    int is = 0;
    for (int mode = 0; mode < ph.nmodes; mode++) {
        const double tau1 = ph.tau1[mode], thet0 = ph.thet0[mode], thet1 = ph.thet1[mode];
        const double fact = fabs(thet0 / tau1);
        const double exp0 = exp(-fact * gamma0), exp1 = exp(-fact * gamma1);
        const double voce = deltgam * thet1 + tau1 * (exp0 - exp1) + thet1 * (gamma0 * exp0 - gamma1 * exp1);
        for (int ism = 0; ism < ph.nsm[mode]; ism++, is++) {
            double dtau = 0.;
#pragma unroll
            for (int js = 0; js < NS; js++)
                if (js < ph.nsyst) dtau = dtau + ph.hard[is * kMaxSysDev + js] * fabs(gamdot[js]);
#pragma unroll
            for (int q = 0; q < NS; q++)
                if (q == is) {
                    tau[q][0] = crss[(2 * q) * N + v] + dtau * voce * tdot / deltgam;
                    tau[q][1] = crss[(2 * q + 1) * N + v] + dtau * voce * tdot / deltgam;
                }
        }
    }
}

}  // namespace evp
