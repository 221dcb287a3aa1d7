// evp_newton.cu -- the local constitutive solve of every equilibrium iteration.
//   k_newton    solve_res / plastic_strain_rate / elastic_strain_rate / harden
//               (various_functions.f90:1142-1491) + the stress sums of calc_velgradavg_corr (1556-1578)
#include "evp_dev.cuh"
#include "evp_math.cuh"
#include "evp_vox.cuh"

#include <mutex>

namespace evp {

// ---------------------------------------------------------------- k_newton: one voxel per thread, operators on chip
// The local solve with one thread per voxel and everything an evaluation reads kept in the
// block's shared memory, one column per thread (entry i of a lane at [32 i + lane] of its warp's columns, so
// every access of a warp is conflict free).  With dedot = dd + S / dt the Jacobian of solve_res is
//   J = I - C~ G + C~ (S / dt + dd) = C~ H,   H = B + S / dt + dd,   B = C~^-1 - G,
// where G = Gamma~r is the modified augmented Lagrangian's operator (zero without --modal 1;
// k_prologue_modal leaves C~ G in cG and subtracts G from the stored C~^-1), C~ (c066mod) and S
// (sg66) are symmetric positive definite, G is symmetric and dd is positive semi-definite.  So
// the Newton step J^-1 res equals H^-1 rho with rho = C~^-1 res formed directly,
//   rho = H0 sg + edotp - q',  H0 = B + S / dt,  q' = B lam + (S / dt) sgt + D - eth,
// and res = C~ rho gives the residual norm that drives the step halving.  H is factored as
// L D L^T in its 21 entries; a pivot that is not positive (G can only cause that with --modal 1)
// sends the voxel to the pivoted elimination of the general system.
// The resistances are used as reciprocals, formed where they change (at the start and at each
// hardening update, 1.2 per voxel) instead of at each evaluation (3 per voxel); the resistances
// themselves go to their output array at each update, and the old ones, for the norm of the change, are the
// reciprocals inverted.
//
// What bounds it: latency (global loads of the batch, FP64 chains) at 8 warps per SM: 255 registers
// a thread and the 840 B column both allow 256 threads per SM with 12 systems, 128 with 24; the
// systems of an evaluation give each warp independent work, which replaces occupancy.  Against six
// lanes per voxel, which exchanged every vector between lanes (243 M warp instructions per launch
// at 64^3, now 64 M), a launch takes 231 us instead of 621 (64^3, 12 systems, n = 20, 3.0
// evaluations per voxel; 0.50 GB of DRAM traffic, FP64 pipe 28 % busy), 167 instead of 347 (40^3,
// 24 systems), 32 instead of 105 (32^3, --modal 1), and 29 instead of 31 at 16^3, where each SM has one
// warp and its chain is all there is.  32 voxels of a warp wait for the slowest: 84 % of the slots
// work.  Measured without gain at 64^3: L2 prefetch of the next batch (290 -> 322 us: two batches of
// 51 kB per warp do not fit the L2), its asynchronous copies issued before this batch's closing sums
// (240 -> 243), 12 systems per step (242 -> 324: spills), C~ loaded ahead of the systems (268).
//
// SYM false: a phase whose stiffness was given as an asymmetric matrix.  C~, S, G and H are then asymmetric
// too; every operator is taken with its 36 entries and H goes to the pivoted elimination.  The wider column
// leaves room for 128 threads per SM: 485 us at 64^3 (630 with six lanes per voxel, 1600 with every operator
// re-read from memory), 231 at 40^3 with 24 systems (365), 42 at 16^3 (36).
// column entries of a thread: Schmid vectors, 1 / resistance (forward, backward), H0 (packed lower triangle, or all of it)
template <int NS, bool SYM>
struct ColV {
    static constexpr int sch = 0, itau = 5 * NS, h0 = 7 * NS, n = 7 * NS + (SYM ? 21 : 36);
};
template <int NS, bool SYM>
__host__ __device__ constexpr int newtonv_threads_per_sm() { return NS <= 12 && SYM ? 256 : 128; }

// Loads and stores of fields that the kernel writes, ordered among themselves and known to be global
// memory (the compiler would otherwise order every shared-memory access around them).
__device__ __forceinline__ double ld_rw(const double* p) {
    double x;
    asm volatile("ld.global.f64 %0, [%1];" : "=d"(x) : "l"(p));
    return x;
}
__device__ __forceinline__ void st_rw(double* p, double x) { asm volatile("st.global.f64 [%0], %1;" ::"l"(p), "d"(x)); }

// the general system by pivoted elimination (rare: see above)
__device__ __noinline__ int solve_general6(const double* h21, double* b6) {
    double J[36], b[6];
#pragma unroll
    for (int i = 0; i < 6; i++) {
        b[i] = b6[i];
#pragma unroll
        for (int j = 0; j < 6; j++) J[6 * i + j] = h21[tri(i, j)];
    }
    const int info = solve6(J, b);
#pragma unroll
    for (int i = 0; i < 6; i++) b6[i] = b[i];
    return info;
}

// x = H^-1 b in place (H packed, symmetric); returns nonzero when H is singular
__device__ __forceinline__ int solve_sym6(double (&h)[21], double (&b)[6]) {
    double a[21], y[6], inv[6];
    bool spd = true;
#pragma unroll
    for (int i = 0; i < 21; i++) a[i] = h[i];
#pragma unroll
    for (int i = 0; i < 6; i++) y[i] = b[i];
#pragma unroll
    for (int k = 0; k < 6; k++) {
        spd = spd && a[tri(k, k)] > 0.0;
        inv[k] = rcp_nr(a[tri(k, k)]);
#pragma unroll
        for (int i = k + 1; i < 6; i++) {
            const double l = a[tri(i, k)] * inv[k];
#pragma unroll
            for (int j = k + 1; j <= i; j++) a[tri(i, j)] -= l * a[tri(j, k)];
            y[i] -= l * y[k];
        }
    }
    if (!spd) {
        double hh[21], bb[6];
#pragma unroll
        for (int i = 0; i < 21; i++) hh[i] = h[i];
#pragma unroll
        for (int i = 0; i < 6; i++) bb[i] = b[i];
        const int info = solve_general6(hh, bb);
#pragma unroll
        for (int i = 0; i < 6; i++) b[i] = bb[i];
        return info;
    }
    // a(i, k) below the diagonal still holds l_ik d_k
#pragma unroll
    for (int i = 5; i >= 0; i--) {
        double s = y[i];
#pragma unroll
        for (int j = i + 1; j < 6; j++) s -= a[tri(j, i)] * b[j];
        b[i] = s * inv[i];
    }
    return 0;
}
// y = A x of a packed symmetric A
__device__ __forceinline__ void sym6_mv(const double (&A)[21], const double (&x)[6], double (&y)[6]) {
#pragma unroll
    for (int i = 0; i < 6; i++) {
        double t = 0.0;
#pragma unroll
        for (int j = 0; j < 6; j++) t += A[tri(i, j)] * x[j];
        y[i] = t;
    }
}
// the upper triangle of a 6x6 operator's planes
__device__ __forceinline__ void ld_sym6(const double* __restrict__ A, long long N, long long v, double (&a)[21]) {
#pragma unroll
    for (int i = 0; i < 6; i++)
#pragma unroll
        for (int j = 0; j <= i; j++) a[tri(i, j)] = __ldg(A + (6 * j + i) * N + v);
}
// an operator: packed and symmetric, or all of its rows
template <bool SYM>
struct Op6 {
    static constexpr int n = SYM ? 21 : 36;
    static __host__ __device__ constexpr int at(int i, int j) { return SYM ? tri(i, j) : 6 * i + j; }
    static __host__ __device__ constexpr int plane(int i, int j) { return SYM ? 6 * j + i : 6 * i + j; }  // entry (i, j <= i if SYM)
    static __host__ __device__ constexpr int cols(int i) { return SYM ? i + 1 : 6; }  // stored entries of row i
    static __device__ __forceinline__ void load(const double* __restrict__ A, long long N, long long v, double (&a)[n]) {
        if constexpr (SYM) {
            ld_sym6(A, N, v, a);
        } else {
#pragma unroll
            for (int c = 0; c < 36; c++) a[c] = __ldg(A + c * N + v);
        }
    }
    static __device__ __forceinline__ void mv(const double (&A)[n], const double (&x)[6], double (&y)[6]) {
        if constexpr (SYM) {
            sym6_mv(A, x, y);
        } else {
#pragma unroll
            for (int i = 0; i < 6; i++) {
                double t = 0.0;
#pragma unroll
                for (int j = 0; j < 6; j++) t += A[6 * i + j] * x[j];
                y[i] = t;
            }
        }
    }
    static __device__ __forceinline__ int solve(double (&h)[n], double (&b)[6]) {
        if constexpr (SYM) return solve_sym6(h, b);
        else return solve6(h, b);
    }
};
template <int M>
__device__ __forceinline__ void ldg_n(const double* __restrict__ a, long long N, long long v, double* o) {
#pragma unroll
    for (int c = 0; c < M; c++) o[c] = __ldg(a + c * N + v);
}
__device__ __forceinline__ void cp_async8(double* dst, const double* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

// dummy gas voxel: closed-form stress update (various_functions.f90:1165-1185)
__device__ __forceinline__ void gas_voxel(const Dev& d, const NewtonParams& p, long long v, double (&s6v)[6]) {
    const long long N = d.N;
    double lam[6], t[6], a[6], res[6], out[6], vg[9], vs[9];
    ld9(d.velgrad, N, v, vg);
    sym33(vg, vs);
    t2_to_b6(vs, t);
    ld6(d.sgt, N, v, a);
    s6_to_b6(a, out);
#pragma unroll
    for (int i = 0; i < 6; i++) t[i] = t[i] + out[i] / p.tdot * p.complgas;
    ld6(d.sg, N, v, a);
    s6_to_b6(a, lam);
    for (int i = 0; i < 6; i++) {
        double x = 0.0;
        for (int j = 0; j < 6; j++) x += d.c066mod[(6 * i + j) * N + v] * t[j];
        res[i] = lam[i] + x;
    }
    if (p.modal) {
        for (int i = 0; i < 6; i++) {
            double x = 0.0;
            for (int j = 0; j < 6; j++) x += d.cG[(6 * i + j) * N + v] * lam[j];
            res[i] -= x;
        }
    }
    for (int i = 0; i < 6; i++) {
        double x = 0.0;
        for (int j = 0; j < 6; j++) x += d.cgas[(6 * i + j) * N + v] * res[j];
        out[i] = x;
    }
    b6_to_s6(out, s6v);
    st6(d.sg, N, v, s6v);
#pragma unroll
    for (int c = 0; c < 6; c++) d.edotp[c * N + v] = 0.0;
    for (int q = 0; q < d.nsys; q++) d.gamdot[q * N + v] = 0.0;
}

// Every warp of the block has put its 14 sums into sh -> one partial per block -> the last block
// folds them in block order (reduce_store's second half, with running sums per warp before it).
constexpr int kNewtonSums = 14;
__device__ __forceinline__ void reduce_newton(const double (*sh)[kNewtonSums], double* partials, double* out, unsigned int* counter,
                                              const VB& vb) {
    __shared__ bool last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    __syncthreads();
    if (threadIdx.x < kNewtonSums) {
        double x = sh[0][threadIdx.x];
        for (int w = 1; w < nw; w++) x += sh[w][threadIdx.x];
        partials[(size_t)threadIdx.x * vb.nx + vb.x] = x;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = (atomicAdd(counter, 1u) == (unsigned)vb.nx - 1u);
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int f = warp; f < kNewtonSums; f += 4 * nw) fold_four<false>(partials, vb.nx, f, nw, kNewtonSums, out, lane);
    if (threadIdx.x == 0) *counter = 0;
}

// Resolved shears over resistance rs and powers |rs|^(n-1) of G systems (Schmid vectors cs,
// reciprocal resistances ci, (gamd0, n) pairs ng), each step on all of them so that their chains overlap.
template <int G, bool UNI>
__device__ __forceinline__ void slip_powers(const double* cs, const double* ci, const double* ng, int kuni,
                                            const double (&sg)[6], double (&rs)[G], double (&pw)[G]) {
#pragma unroll
    for (int q = 0; q < G; q++) {
        double x = cs[5 * q * 32] * sg[0];
#pragma unroll
        for (int c = 1; c < 5; c++) x += cs[(5 * q + c) * 32] * sg[c];
        rs[q] = x * ci[2 * q * 32 + (x < 0.0 ? 32 : 0)];
    }
    if (UNI || kuni >= 0) {  // one integer exponent: binary powering of the systems together
        double b[G];
#pragma unroll
        for (int q = 0; q < G; q++) {
            b[q] = fabs(rs[q]);
            pw[q] = (kuni & 1) ? b[q] : 1.0;
        }
        for (int k = kuni >> 1; k; k >>= 1) {
#pragma unroll
            for (int q = 0; q < G; q++) b[q] *= b[q];
            if (k & 1)
#pragma unroll
                for (int q = 0; q < G; q++) pw[q] *= b[q];
        }
    } else {
#pragma unroll
        for (int q = 0; q < G; q++) pw[q] = pow(fabs(rs[q]), ng[2 * q + 1] - 1.0);
    }
}

// UNI: every phase has one integer exponent for its systems; the kernel then holds no pow(), which
// would take registers and instruction cache from the common case.
template <int NS, bool UNI, bool SYM>
__device__ __forceinline__ void body_newtonv(const Dev& d, const NewtonParams& p, const VB& vb) {
    using Col = ColV<NS, SYM>;
    using Op = Op6<SYM>;
    extern __shared__ __align__(16) double dyn_smem[];
    PhaseV<NS>* const sph = reinterpret_cast<PhaseV<NS>*>(dyn_smem);
    const int nph = d.nph;  // at most kMaxPhaseSmem
    for (int e = threadIdx.x; e < nph * (int)(sizeof(PhaseV<NS>) / 8); e += blockDim.x) dyn_smem[e] = d.phv[e];
    __syncthreads();
    const int lane = threadIdx.x & 31;
    double* const col = reinterpret_cast<double*>(sph + nph) + (threadIdx.x >> 5) * (Col::n * 32) + lane;
    const long long N = d.N;
    const int qlast = 2 * d.nsys - 1, slast = 5 * d.nsys - 1;
    constexpr int kG = 6;  // systems per step of an evaluation (of 12 the kernel spills)
    const double tolt = fmax(p.error, p.erroral), idt = 1.0 / p.tdot;
    const bool stats = d.nstats != nullptr;
    unsigned c_pass = 0, c_eval = 0, c_nr = 0, c_tau = 0, c_vox = 0, c_npass = 0;
    double mine = 0.0, mineg = 0.0;  // running sum lane / 4 of this warp: dsg and ddg norms, stress (solid; gas)
    const long long stride = (long long)vb.nx * blockDim.x;
    for (long long v0 = (long long)vb.x * blockDim.x + (threadIdx.x & ~31); v0 < N; v0 += stride) {  // warp-uniform
        const long long v = v0 + lane;
        double sums[8], gsum[8];
#pragma unroll
        for (int c = 0; c < 8; c++) {
            sums[c] = 0.0;
            gsum[c] = 0.0;
        }
        if (v < N) {
            const bool gas = __ldg(d.gas + v);
            const PhaseV<NS>& ph = sph[__ldg(d.phase + v)];
            // The batch's inputs are all in flight together: the resistances, B and the Schmid vectors go
            // to the column by asynchronous copies (no registers wait for them), the rest to registers.
            double l6[6], t6[6], vg[9], e9[9], sm[Op::n], a[9];
            {
                const double* q = d.trialtau + v;
#pragma unroll
                for (int i = 0; i < 2 * NS; i++) {
                    cp_async8(col + (Col::itau + i) * 32, q);
                    q += i < qlast ? N : 0;
                }
                q = d.c066inv + v;
#pragma unroll
                for (int i = 0; i < 6; i++)
#pragma unroll
                    for (int j = 0; j < Op::cols(i); j++) cp_async8(col + (Col::h0 + Op::at(i, j)) * 32, q + Op::plane(i, j) * N);
                q = d.sch + v;
#pragma unroll 10
                for (int i = 0; i < 5 * NS; i++) {
                    cp_async8(col + (Col::sch + i) * 32, q);
                    q += i < slast ? N : 0;
                }
            }
            Op::load(d.sg66, N, v, sm);
#pragma unroll
            for (int c = 0; c < 6; c++) l6[c] = ld_rw(d.sg + c * N + v);
            ldg_n<6>(d.sgt, N, v, t6);
            ldg_n<9>(d.velgrad, N, v, vg);
            if (p.thermo) ldg_n<9>(d.eth, N, v, e9);
            const double w = __ldg(d.wgtc + v);
            double s6v[6];
            if (gas) {
                asm volatile("cp.async.wait_all;" ::: "memory");
                gas_voxel(d, p, v, s6v);
#pragma unroll
                for (int c = 0; c < 6; c++) gsum[2 + c] = s6v[c] * w;
            } else {
                const int nsyst = ph.nsyst;
                double sg[6], qp[6], taun = 0.0;
                {
                    double sgt[6];
                    s6_to_b6(l6, sg);
                    s6_to_b6(t6, sgt);
                    sym33(vg, a);
                    t2_to_b6(a, qp);
                    if (p.thermo) {
                        t2_to_b6(e9, a);
#pragma unroll
                        for (int i = 0; i < 6; i++) qp[i] = qp[i] - a[i];
                    }
                    asm volatile("cp.async.wait_all;" ::: "memory");
#pragma unroll
                    for (int i = 0; i < 6; i++)
#pragma unroll
                        for (int j = 0; j < Op::cols(i); j++) {
                            const double bi = col[(Col::h0 + Op::at(i, j)) * 32], si = sm[Op::at(i, j)] * idt;
                            col[(Col::h0 + Op::at(i, j)) * 32] = bi + si;
                            qp[i] += bi * sg[j] + si * sgt[j];
                            if (SYM && j != i) qp[j] += bi * sg[i] + si * sgt[i];
                        }
#pragma unroll
                    for (int q = 0; q < 2 * NS; q++) {
                        const double t = q <= qlast ? col[(Col::itau + q) * 32] : 0.0, i = rcp_nr(t);
                        taun += t * t;
                        col[(Col::itau + q) * 32] = q < 2 * nsyst ? i : 0.0;
                    }
                    for (int i = 5 * nsyst; i < 5 * NS; i++) col[(Col::sch + i) * 32] = 0.0;
                }
                taun = sqrt(taun);
                double sgnorm2 = 0.0;
#pragma unroll
                for (int i = 0; i < 6; i++) sgnorm2 += sg[i] * sg[i];
                const double sgnorm = sqrt(sgnorm2);
                const double errlim2 = (p.erroral * sgnorm) * (p.erroral * sgnorm);
                double sgold[6] = {0, 0, 0, 0, 0, 0}, ep[5] = {0, 0, 0, 0, 0};
                bool halved = false;  // the last evaluation's stress is in edotp, not in sgold
                double errtau = 2.0 * tolt;
                c_vox++;
                for (int itertau = 0; itertau < 10 && errtau > tolt; itertau++) {
                    double resold2 = 1.0;
                    bool more = true;
                    c_tau++;
                    for (int iterNR = 0; iterNR < 100 && more; iterNR++) {
                        // residual norms and the Newton correction are compared as squares (no square
                        // roots on the chain): res2 = |res|^2, and the loop runs while |dsg|^2 > (erroral |sg_in|)^2
                        double res2 = 4.0 * resold2, rho[6], dd[15];
                        for (int icut = 0; icut < 10 && res2 > resold2; icut++) {
                            if (stats) {
                                c_eval++;
                                if (lane == __ffs(__activemask()) - 1) c_pass++;
                            }
                            // plastic_strain_rate and its derivative: resolved shears, powers and sums of
                            // kG systems at a time, each step on all of them so that their chains overlap
#pragma unroll
                            for (int c = 0; c < 5; c++) ep[c] = 0.0;
#pragma unroll
                            for (int c = 0; c < 15; c++) dd[c] = 0.0;
#pragma unroll 1
                            for (int s0 = 0; s0 < NS; s0 += kG) {
                                const double* const cs = col + (Col::sch + 5 * s0) * 32;
                                const double* const ci = col + (Col::itau + 2 * s0) * 32;
                                double rs[kG], pw[kG];
                                slip_powers<kG, UNI>(cs, ci, &ph.ng[2 * s0], ph.kuni, sg, rs, pw);
#pragma unroll
                                for (int q = 0; q < kG; q++) {
                                    const double2 ng = *reinterpret_cast<const double2*>(&ph.ng[2 * (s0 + q)]);
                                    const double dum = ng.x * pw[q], g = rs[q] * dum;
                                    if constexpr (!UNI)
                                        if (2 * (s0 + q) < qlast) st_rw(d.gamdot + (s0 + q) * N + v, g);
                                    const double r1 = ng.y * dum * ci[2 * q * 32 + (rs[q] < 0.0 ? 32 : 0)];
                                    double sc[5];
#pragma unroll
                                    for (int c = 0; c < 5; c++) sc[c] = cs[(5 * q + c) * 32];
                                    int e = 0;
#pragma unroll
                                    for (int jj = 0; jj < 5; jj++) {
                                        ep[jj] += sc[jj] * g;
                                        const double t = sc[jj] * r1;
#pragma unroll
                                        for (int ii = 0; ii <= jj; ii++) dd[e++] += sc[ii] * t;
                                    }
                                }
                            }
#pragma unroll
                            for (int i = 0; i < 6; i++) rho[i] = (i < 5 ? ep[i < 5 ? i : 0] : 0.0) - qp[i];
#pragma unroll
                            for (int i = 0; i < 6; i++)
#pragma unroll
                                for (int j = 0; j < Op::cols(i); j++) {
                                    const double h = col[(Col::h0 + Op::at(i, j)) * 32];
                                    rho[i] += h * sg[j];
                                    if (SYM && j != i) rho[j] += h * sg[i];
                                }
                            double rn[6], cm[Op::n];
                            Op::load(d.c066mod, N, v, cm);
                            Op::mv(cm, rho, rn);
                            res2 = (rn[0] * rn[0] + rn[1] * rn[1]) + (rn[2] * rn[2] + rn[3] * rn[3]) + (rn[4] * rn[4] + rn[5] * rn[5]);
                            if (iterNR == 0) resold2 = res2;
                            halved = false;
                            if (res2 > resold2) {
                                if (icut == 9) {
                                    halved = true;
#pragma unroll
                                    for (int i = 0; i < 6; i++) st_rw(d.edotp + i * N + v, sg[i]);
                                }
#pragma unroll
                                for (int i = 0; i < 6; i++) sg[i] = sgold[i] + (sg[i] - sgold[i]) * 0.5;
                            }
                        }
                        resold2 = res2;
                        if (stats) {
                            c_nr++;
                            if (lane == __ffs(__activemask()) - 1) c_npass++;
                        }
                        double h[Op::n], dsg2 = 0.0;
#pragma unroll
                        for (int i = 0; i < 6; i++)
#pragma unroll
                            for (int j = 0; j < Op::cols(i); j++)
                                h[Op::at(i, j)] = col[(Col::h0 + Op::at(i, j)) * 32] + dd_at(dd, i, j);
                        if (Op::solve(h, rho) != 0) set_err(d.err, 1);
#pragma unroll
                        for (int i = 0; i < 6; i++) {
                            sgold[i] = sg[i];
                            sg[i] = sg[i] - rho[i];
                            dsg2 += (sg[i] - sgold[i]) * (sg[i] - sgold[i]);
                        }
                        more = sgnorm > 0.0 ? dsg2 > errlim2 : dsg2 > 0.0;
                    }
                    // The slip rates at the last evaluation's stress.  With an integer exponent they are formed
                    // again (a third of an evaluation) instead of kept in registers; where each power is a
                    // call of pow() the evaluations left them in their output array (50x45x36, n = 12.6:
                    // 201 -> 180 us per launch).
                    double gd[NS], dg = 0.0;
                    if constexpr (UNI) {
                        double se[6], *out = d.gamdot + v;
#pragma unroll
                        for (int i = 0; i < 6; i++) se[i] = sgold[i];
                        if (halved)
#pragma unroll
                            for (int i = 0; i < 6; i++) se[i] = ld_rw(d.edotp + i * N + v);
#pragma unroll
                        for (int s0 = 0; s0 < NS; s0 += kG) {
                            double rs[kG], pw[kG];
                            slip_powers<kG, UNI>(col + (Col::sch + 5 * s0) * 32, col + (Col::itau + 2 * s0) * 32, &ph.ng[2 * s0], ph.kuni, se,
                                                  rs, pw);
#pragma unroll
                            for (int q = 0; q < kG; q++) {
                                const double g = rs[q] * (ph.ng[2 * (s0 + q)] * pw[q]);
                                gd[s0 + q] = fabs(g);
                                if (2 * (s0 + q) < qlast) st_rw(out, g);
                                out += N;
                            }
                        }
                    } else {
                        const double* q = d.gamdot + v;
#pragma unroll
                        for (int s = 0; s < NS; s++) {
                            gd[s] = ld_rw(q);
                            q += 2 * s < qlast - 1 ? N : 0;
                        }
#pragma unroll
                        for (int s = 0; s < NS; s++) gd[s] = s < nsyst ? fabs(gd[s]) : 0.0;
                    }
#pragma unroll
                    for (int s = 0; s < NS; s++) dg += gd[s];
                    if (!p.iuphard) break;
                    // harden (various_functions.f90:1439-1491).  The new resistances go to their output array;
                    // the old ones, for the norm of the change, are the column's reciprocals inverted.
                    double e2 = 0.0, fm[3];
                    const double gamma0 = __ldg(d.gacumgr + v);
                    const double deltgam = dg * p.tdot, gamma1 = gamma0 + deltgam;
#pragma unroll
                    for (int m = 0; m < 3; m++) {  // the Voce factor of each mode
                        fm[m] = 0.0;
                        if (m < ph.nmodes) {
                            const double tau1 = ph.tau1[m], thet0 = ph.thet0[m], thet1 = ph.thet1[m];
                            const double fact = fabs(thet0 / tau1);
                            const double exp0 = exp(-fact * gamma0), exp1 = exp(-fact * gamma1);
                            const double voce = deltgam * thet1 + tau1 * (exp0 - exp1) + thet1 * (gamma0 * exp0 - gamma1 * exp1);
                            fm[m] = voce * p.tdot / deltgam;
                        }
                    }
                    const int m1 = ph.nsm[0], m2 = m1 + ph.nsm[1];
#pragma unroll 1
                    for (int s0 = 0; s0 < NS; s0 += 12) {
                        // every load before the first store: the compiler keeps shared-memory loads behind
                        // shared-memory stores, which would run the twelve systems one after the other
                        double cr[24], dtau[12], *out = d.trialtau + 2 * s0 * N + v;
                        double* const ci = col + (Col::itau + 2 * s0) * 32;
                        const double* qc = d.crss + (long long)min(2 * s0, qlast) * N + v;
#pragma unroll
                        for (int i = 0; i < 24; i++) {
                            cr[i] = __ldg(qc);
                            qc += 2 * s0 + i < qlast ? N : 0;
                        }
#pragma unroll
                        for (int q = 0; q < 12; q++) dtau[q] = 0.0;
#pragma unroll
                        for (int js = 0; js < NS; js += 2)
#pragma unroll
                            for (int q = 0; q < 12; q++) {
                                const double2 hh = *reinterpret_cast<const double2*>(&ph.hard[(s0 + q) * NS + js]);
                                dtau[q] += hh.x * gd[js] + hh.y * gd[js + 1];
                            }
#pragma unroll
                        for (int q = 0; q < 12; q++) {
                            const int s = s0 + q;
                            const bool own = s < nsyst;
                            const double x = dtau[q] * (s < m1 ? fm[0] : (s < m2 ? fm[1] : fm[2]));
                            // systems beyond the phase's own get zero resistance, as harden leaves them
                            const double n0 = own ? cr[2 * q] + x : 0.0, n1 = own ? cr[2 * q + 1] + x : 0.0;
                            const double i0 = rcp_nr(n0), i1 = rcp_nr(n1), t0 = rcp_nr(ci[2 * q * 32]), t1 = rcp_nr(ci[(2 * q + 1) * 32]);
                            const double d0 = own ? t0 - n0 : 0.0, d1 = own ? t1 - n1 : 0.0;
                            e2 += d0 * d0 + d1 * d1;
                            ci[2 * q * 32] = own ? i0 : 0.0;
                            ci[(2 * q + 1) * 32] = own ? i1 : 0.0;
                            if (2 * s < qlast) {
                                st_rw(out, n0);
                                st_rw(out + N, n1);
                            }
                            out += 2 * N;
                        }
                    }
                    errtau = sqrt(e2) / taun;
                }
                // |sg - lam|^2 at the final stress; |edot - D|^2 at the last evaluation, with
                // edot = edotp + S (sg - sgt) / dt + eth as elastic_strain_rate forms it
                double x6[6], e6[6], D[6], e6v[6], dsg = 0.0, ddg = 0.0;
                Op::load(d.sg66, N, v, sm);
                ldg_n<6>(d.sgt, N, v, t6);
                ldg_n<9>(d.velgrad, N, v, vg);
                if (p.thermo) ldg_n<9>(d.eth, N, v, e9);
#pragma unroll
                for (int c = 0; c < 6; c++) l6[c] = ld_rw(d.sg + c * N + v);
                if (halved)
#pragma unroll
                    for (int i = 0; i < 6; i++) sgold[i] = ld_rw(d.edotp + i * N + v);
                s6_to_b6(t6, x6);
#pragma unroll
                for (int i = 0; i < 6; i++) x6[i] = (sgold[i] - x6[i]) * idt;
                Op::mv(sm, x6, e6);
                sym33(vg, a);
                t2_to_b6(a, D);
                if (p.thermo) t2_to_b6(e9, a);
                s6_to_b6(l6, x6);
#pragma unroll
                for (int i = 0; i < 6; i++) {
                    double x = (i < 5 ? ep[i < 5 ? i : 0] : 0.0) + e6[i];
                    if (p.thermo) x = x + a[i];
                    ddg += (x - D[i]) * (x - D[i]);
                    dsg += (sg[i] - x6[i]) * (sg[i] - x6[i]);
                }
                if (!(dsg == dsg) || !(ddg == ddg)) set_err(d.err, 2);
                b6_to_s6(sg, s6v);
#pragma unroll
                for (int i = 0; i < 6; i++) e6[i] = i < 5 ? ep[i < 5 ? i : 0] : 0.0;
                b6_to_s6(e6, e6v);
#pragma unroll
                for (int c = 0; c < 6; c++) {
                    st_rw(d.sg + c * N + v, s6v[c]);
                    st_rw(d.edotp + c * N + v, e6v[c]);
                    sums[2 + c] = w * s6v[c];
                }
                sums[0] = dsg * w;
                sums[1] = ddg * w;
            }
        }
        __syncwarp();
        mine += warp_reduce_many<8, false>(sums, lane);
        if (d.cgas) mineg += warp_reduce_many<8, false>(gsum, lane);
    }
    if (stats) {
        unsigned c[6] = {c_pass, c_eval, c_nr, c_tau, c_vox, c_npass};
#pragma unroll
        for (int i = 0; i < 6; i++) {
            const unsigned x = __reduce_add_sync(0xffffffffu, c[i]);
            if (lane == 0) atomicAdd(d.nstats + i, (unsigned long long)x);
        }
    }
    // dsg and ddg norms, the solid's stress sum and the whole cell's
    __shared__ double sh[8][kNewtonSums];
    if ((lane & 3) == 0) {
        const int f = lane >> 2;
        sh[threadIdx.x >> 5][f] = mine;
        if (f >= 2) sh[threadIdx.x >> 5][f + 6] = mine + mineg;
    }
    reduce_newton(sh, d.partials, d.red + OFF_NEWTON, d.counters + CNT_NEWTON, vb);
}

// The local-solve kernel of a solve: 0/1 body_newtonv<12/24> for integer exponents, 2/3 for others, 4/5 for
// any with a phase of asymmetric stiffness.
static int newton_kernel(const Dev& d) { return (!d.symel ? 4 : (d.uniexp ? 0 : 2)) + (d.nsys > 12 ? 1 : 0); }
constexpr int newton_sm_threads(int kernel) {
    return kernel >= 4 ? newtonv_threads_per_sm<12, false>() : (kernel & 1 ? newtonv_threads_per_sm<24, true>() : newtonv_threads_per_sm<12, true>());
}
// Block size: as many threads as an SM holds (one block per SM, the fewest partial
// sums to fold) unless that leaves SMs without a block; then halved until every SM has one, down
// to one warp.
static int newton_threads(const Dev& d, int kernel) {
    int t = newton_sm_threads(kernel);
    while (t > 32 && (d.N + t - 1) / t < 148) t /= 2;
    return t;
}
static int newton_grid(const Dev& d, int kernel) {
    const long long t = newton_threads(d, kernel), g = (d.N + t - 1) / t;
    // one wave, every warp taking every (blocks x warps)-th batch of 32 voxels
    const long long wave = 148LL * (newton_sm_threads(kernel) / t);
    return (int)(g < wave ? g : wave);
}
static size_t newton_smem(const Dev& d, int kernel) {
    const size_t t = newton_threads(d, kernel);
    const size_t entries = kernel >= 4 ? (kernel & 1 ? ColV<24, false>::n : ColV<12, false>::n) : (kernel & 1 ? ColV<24, true>::n : ColV<12, true>::n);
    return d.nph * (kernel & 1 ? sizeof(PhaseV<24>) : sizeof(PhaseV<12>)) + sizeof(double) * entries * t;
}
// dynamic shared memory that a block may take beside the kernel's own (the SM's limit of 227 KB less 5)
constexpr int kNewtonSmemMost = 222 * 1024;
static_assert(kMaxPhaseSmem * sizeof(PhaseV<12>) + sizeof(double) * ColV<12, true>::n * newtonv_threads_per_sm<12, true>() <= kNewtonSmemMost &&
              kMaxPhaseSmem * sizeof(PhaseV<24>) + sizeof(double) * ColV<24, true>::n * newtonv_threads_per_sm<24, true>() <= kNewtonSmemMost &&
              kMaxPhaseSmem * sizeof(PhaseV<12>) + sizeof(double) * ColV<12, false>::n * newtonv_threads_per_sm<12, false>() <= kNewtonSmemMost &&
              kMaxPhaseSmem * sizeof(PhaseV<24>) + sizeof(double) * ColV<24, false>::n * newtonv_threads_per_sm<24, false>() <= kNewtonSmemMost,
              "the phases' tables and the columns fit");
template <int V>
__global__ void __launch_bounds__(newton_sm_threads(V), 1) kb_newton(const __grid_constant__ BatchParams P);
static void newton_configure() {
    static std::once_flag once;
    std::call_once(once, [] {
        const void* const ks[] = {(const void*)kb_newton<0>, (const void*)kb_newton<1>, (const void*)kb_newton<2>,
                                  (const void*)kb_newton<3>, (const void*)kb_newton<4>, (const void*)kb_newton<5>};
        for (const void* k : ks) cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kNewtonSmemMost);
    });
}

template <int V>
__global__ void __launch_bounds__(newton_sm_threads(V), 1) kb_newton(const __grid_constant__ BatchParams P) {
    __shared__ NewtonParams ps;
    __shared__ int go;
    const Job& jb = batch_job(P);
    const BatchSolve& m = P.E[jb.solve];
    if (threadIdx.x == 0) {
        go = m.ctl->active;
        ps = m.ctl->newton;
    }
    __syncthreads();
    if (!go) return;
    const NewtonParams p = ps;  // in registers, as a single-solve launch's parameter
    const VB vb = job_vb(jb);
    if constexpr (V == 0) body_newtonv<12, true, true>(m.d, p, vb);
    else if constexpr (V == 1) body_newtonv<24, true, true>(m.d, p, vb);
    else if constexpr (V == 2) body_newtonv<12, false, true>(m.d, p, vb);
    else if constexpr (V == 3) body_newtonv<24, false, true>(m.d, p, vb);
    else if constexpr (V == 4) body_newtonv<12, false, false>(m.d, p, vb);
    else body_newtonv<24, false, false>(m.d, p, vb);
}

// Launch shape of a solve's local solve.  Members of one block size share a batched launch:
// variant = kernel + 8 * (block size / 32).
NewtonShape newton_shape(const Dev& d) {
    newton_configure();
    const int k = newton_kernel(d), t = newton_threads(d, k);
    return NewtonShape{newton_grid(d, k), t, k + 8 * (t / 32), newton_smem(d, k)};
}
void launch_batched_newton(const BatchLaunch& L, const BatchParams& P, cudaStream_t st) {
    switch (L.variant & 7) {
        case 0: kb_newton<0><<<L.blocks, L.threads, L.smem, st>>>(P); break;
        case 1: kb_newton<1><<<L.blocks, L.threads, L.smem, st>>>(P); break;
        case 2: kb_newton<2><<<L.blocks, L.threads, L.smem, st>>>(P); break;
        case 3: kb_newton<3><<<L.blocks, L.threads, L.smem, st>>>(P); break;
        case 4: kb_newton<4><<<L.blocks, L.threads, L.smem, st>>>(P); break;
        default: kb_newton<5><<<L.blocks, L.threads, L.smem, st>>>(P); break;
    }
}

}  // namespace evp
