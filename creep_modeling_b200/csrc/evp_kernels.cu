// evp_kernels.cu -- per-voxel sm_100a kernels of the LS-EVPFFT solve.
//
// One thread per voxel (grid-stride), SoA FP64 state (layout in evp_dev.cuh).
// Every reduction is a fixed-order tree: warp shuffles, one partial per block,
// and the last block to finish sums the partials in block order, so results
// are reproducible run to run.  Kernel <-> reference routine map:
//   k_init      data_grain + Hall-Petch init + initial_guess (IO_functions.f90:722-812, 107-199;
//               various_functions.f90:8-53) and the start-up c066 sum (LS-EVPFFT.f90:156-165)
//   k_sgavg     stress average before the PK1 prologue (LS-EVPFFT.f90:238-254)
//   k_prologue  update_schmid + calc_c066mod_Goperr066mod (various_functions.f90:472-539, 812-906)
//   k_gas_compl calc_gas_compl (various_functions.f90:909-951)
//   k_corr      correction_to_current pass 2 + velgrad mixing (various_functions.f90:1103-1139;
//               LS-EVPFFT.f90:277-311)
//   (the local solve, k_newton: evp_newton.cu)
//   k_upd1      accepted-step commit (LS-EVPFFT.f90:432-446) + update_plastic_defgrad + update_defgrad
//   k_upd2      update_elstic_defgrad + update_el_stiff + update_tensor_config pass 1
//   k_upd3      update_tensor_config pass 2 + update_hardening + macro averages (LS-EVPFFT.f90:460-523)
//   k_diag      update_diagnostics (types.f90:345-692)
//   k_c0        calc_c0 voxel part (various_functions.f90:2537-2634)
//   k_kinematic kinematic_increments (various_functions.f90:2766-2837)
//   k_goperr0   real-space Green operator at the origin (various_functions.f90:798-807)
//   k_cell2node cell2node_tensor1 + nodal update (various_functions.f90:2026-2054, 2652-2691)
#include "evp_dev.cuh"
#include "evp_math.cuh"
#include "evp_vox.cuh"

namespace evp {

// ---------------------------------------------------------------- k_init
struct InitParams {
    double udot[9];
    double u6t[6];  // b6(udot) * tdot of process 1
    int keepF;       // F, F^-1, det F and w J come from k_dispini
    double detFavg;  // sum of w J (divides the weights when keepF)
};

__global__ void __launch_bounds__(kBlock) k_init(Dev d, const double* __restrict__ euler, const int* __restrict__ grain,
                                                   const double* __restrict__ hp, InitParams ip) {
    const long long N = d.N;
    double sums[36];
#pragma unroll
    for (int c = 0; c < 36; c++) sums[c] = 0.0;
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < N; v += (long long)gridDim.x * blockDim.x) {
        const int p = d.phase[v];
        const PhaseDev& ph = d.ph[p];
        double I9[9];
        eye9(I9);
        if (!ip.keepF) {
            st9(d.F, N, v, I9);
            st9(d.Finv, N, v, I9);
            d.detF[v] = 1.0;
        }
        st9(d.Fe, N, v, I9); st9(d.Fp, N, v, I9);
        st9(d.Finc, N, v, I9); st9(d.Feinc, N, v, I9);
        const double w = ip.keepF ? d.wgtc[v] / ip.detFavg : d.wgt;  // wgtc (IO_functions.f90:917, 934)
        d.wgtc[v] = w;
        d.epvm[v] = 0.0;
        d.gacumgr[v] = 0.0;
        st9(d.velgrad, N, v, ip.udot);
        double z[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
        st9(d.velgradold, N, v, z);
        st9(d.dvr, N, v, z);
        st6(d.sgt, N, v, z); st6(d.edotp, N, v, z); st6(d.ept, N, v, z); st6(d.disgradsym, N, v, z);
        for (int s = 0; s < d.nsys; s++) {
            d.gamdot[s * N + v] = 0.0;
            d.crss[(2 * s) * N + v] = 0.0; d.crss[(2 * s + 1) * N + v] = 0.0;
            d.trialtau[(2 * s) * N + v] = 0.0; d.trialtau[(2 * s + 1) * N + v] = 0.0;
            for (int c = 0; c < 5; c++) d.sch[(s * 5 + c) * N + v] = 0.0;
        }
        if (ph.igas) {
            st6(d.sg, N, v, z);
            st9(d.ag, N, v, z);
            for (int c = 0; c < 36; c++) d.sg66[c * N + v] = 0.0;
            continue;
        }
        double aa[9], ag[9];
        const double deg = EVP_PI / 180.0;
        euler2(euler[3 * v] * deg, euler[3 * v + 1] * deg, euler[3 * v + 2] * deg, aa);
        for (int j = 0; j < 3; j++)
            for (int k = 0; k < 3; k++) ag[3 * j + k] = aa[3 * k + j];
        st9(d.ag, N, v, ag);
        double c4[81], cg66[36];
        rotate4(ag, ph.C, c4);
        t4_to_b66(c4, cg66);
        for (int c = 0; c < 36; c++) sums[c] += cg66[c] * w;
        double sg6[6], s6[6];
        for (int i = 0; i < 6; i++) {
            double s = 0.0;
            for (int j = 0; j < 6; j++) s += cg66[6 * i + j] * ip.u6t[j];
            sg6[i] = s;
        }
        b6_to_s6(sg6, s6);
        st6(d.sg, N, v, s6);
        if (inv_unrolled<6>(cg66) != 0) set_err(d.err, 1);
        for (int c = 0; c < 36; c++) d.sg66[c * N + v] = cg66[c];
        const double hps = hp[v];
        for (int s = 0; s < ph.nsyst; s++) {
            double c1 = ph.tau0f[s] + hps, c2 = ph.tau0b[s] + hps;
            double db1 = ag[3] * ph.dbca[3 * s] + ag[4] * ph.dbca[3 * s + 1] + ag[5] * ph.dbca[3 * s + 2];
            double cosalpha = fabs(db1);
            c1 = c1 + ph.hpfac[s] * sqrt(cosalpha);
            c2 = c2 + ph.hpfac[s] * sqrt(cosalpha);
            d.crss[(2 * s) * N + v] = c1;
            d.crss[(2 * s + 1) * N + v] = c2;
            d.trialtau[(2 * s) * N + v] = c2;  // both columns start from the backward CRSS (IO_functions.f90:193-194)
            d.trialtau[(2 * s + 1) * N + v] = c2;
        }
    }
    reduce_store<36, 0>(sums, nullptr, d.partials, d.red + OFF_INIT, d.counters + CNT_INIT, hw_vb());
}

void launch_init(const Dev& d, const double* euler, const int* grain, const double* hp, const double* udot9, const double* u6t,
                 int keepF, double detFavg, cudaStream_t st) {
    InitParams ip;
    for (int c = 0; c < 9; c++) ip.udot[c] = udot9[c];
    for (int c = 0; c < 6; c++) ip.u6t[c] = u6t[c];
    ip.keepF = keepF;
    ip.detFavg = detFavg;
    k_init<<<d.grid, d.block, 0, st>>>(d, euler, grain, hp, ip);
}

// ---------------------------------------------------------------- k_dispini
// init_defgrad per voxel (IO_functions.f90:893-921).  Sums, in OFF_DISP order: F^-1 w J over all
// voxels (9), the solid ones (9), the gas ones (9); w J over solid and gas voxels; J w.
__global__ void __launch_bounds__(kBlock) k_dispini(Dev d, const double* __restrict__ grad, double delt) {
    const long long N = d.N;
    double sums[30];
#pragma unroll
    for (int c = 0; c < 30; c++) sums[c] = 0.0;
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < N; v += (long long)gridDim.x * blockDim.x) {
        double F[9], Fi[9];
        for (int l = 0; l < 3; l++)
            for (int m = 0; m < 3; m++) F[3 * l + m] = grad[(size_t)(3 * m + l) * N + v] + (l == m ? delt : 0.0);
        const double J = det33(F);
        if (inv3u(F, Fi) != 0) set_err(d.err, 1);
        st9(d.F, N, v, F);
        st9(d.Fini, N, v, F);
        st9(d.Finv, N, v, Fi);
        d.detF[v] = J;
        d.wgtc[v] = d.wgt * J;
        const int gas = d.gas[v];
#pragma unroll
        for (int c = 0; c < 9; c++) {
            const double t = Fi[c] * d.wgt * J;
            sums[c] += t;
            sums[9 + c] += gas ? 0.0 : t;
            sums[18 + c] += gas ? t : 0.0;
        }
        sums[27] += gas ? 0.0 : d.wgt * J;
        sums[28] += gas ? d.wgt * J : 0.0;
        sums[29] += J * d.wgt;
    }
    reduce_store<30, 0>(sums, nullptr, d.partials, d.red + OFF_DISP, d.counters + CNT_DISP, hw_vb());
}
void launch_dispini(const Dev& d, const double* grad, double delt, cudaStream_t st) {
    k_dispini<<<d.grid, d.block, 0, st>>>(d, grad, delt);
}

// ---------------------------------------------------------------- k_sgavg
__device__ __forceinline__ void body_sgavg(const Dev& d, const VB& vb) {
    const long long N = d.N;
    double s[6] = {0, 0, 0, 0, 0, 0};
    for (long long v = vb.x * (long long)blockDim.x + threadIdx.x; v < N; v += (long long)vb.nx * blockDim.x) {
        double w = d.wgtc[v];
#pragma unroll
        for (int c = 0; c < 6; c++) s[c] += d.sg[c * N + v] * w;
    }
    reduce_store<6, 0>(s, nullptr, d.partials, d.red + OFF_SGAVG, d.counters + CNT_SGAVG, vb);
}
__global__ void __launch_bounds__(kBlock) k_sgavg(Dev d) { body_sgavg(d, hw_vb()); }
void launch_sgavg(const Dev& d, cudaStream_t st) { k_sgavg<<<d.grid, d.block, 0, st>>>(d); }

// ---------------------------------------------------------------- b-basis congruence
// For a 3x3 matrix M, T(M)_ag = <B^a, B^g M^T> (Frobenius product; B^0..B^5 the orthonormal
// b-basis of chg_basis).  A fourth-order tensor with minor symmetries, c = sum B^g c66_gd B^d,
// pulled back as p_ijkl = sum_mn c_imkn M_jm M_ln has the b-basis components T c66 T^T, so the
// 3x3x3x3 expansion and its contraction (81 x 9 products) reduce to two 6x6 products.
__device__ __forceinline__ void basis_T(const double* M, double* T) {
    double Bg[9], P[9], col[6];
#pragma unroll
    for (int g = 0; g < 6; g++) {
#pragma unroll
        for (int c = 0; c < 9; c++) Bg[c] = 0.0;
        if (g == 0) { Bg[0] = -EVP_RSQ2; Bg[4] = EVP_RSQ2; }
        else if (g == 1) { Bg[0] = -EVP_RSQ6; Bg[4] = -EVP_RSQ6; Bg[8] = EVP_RSQ23; }
        else if (g == 2) { Bg[5] = EVP_RSQ2; Bg[7] = EVP_RSQ2; }
        else if (g == 3) { Bg[2] = EVP_RSQ2; Bg[6] = EVP_RSQ2; }
        else if (g == 4) { Bg[1] = EVP_RSQ2; Bg[3] = EVP_RSQ2; }
        else { Bg[0] = EVP_RSQ3; Bg[4] = EVP_RSQ3; Bg[8] = EVP_RSQ3; }
        mm3_bt(Bg, M, P);  // B^g M^T
        t2_to_b6(P, col);
#pragma unroll
        for (int a = 0; a < 6; a++) T[6 * a + g] = col[a];
    }
}
// out = s * T A T^T (6x6)
// (a row of T A at a time: six live values instead of 36, each sum in the same order)
__device__ __forceinline__ void congruence6(const double* T, const double* A, double s, double* out) {
#pragma unroll
    for (int i = 0; i < 6; i++) {
        double ta[6];
#pragma unroll
        for (int j = 0; j < 6; j++) {
            double x = 0.0;
#pragma unroll
            for (int k = 0; k < 6; k++) x += T[6 * i + k] * A[6 * k + j];
            ta[j] = x;
        }
#pragma unroll
        for (int j = 0; j < 6; j++) {
            double x = 0.0;
#pragma unroll
            for (int k = 0; k < 6; k++) x += ta[k] * T[6 * j + k];
            out[6 * i + j] = s * x;
        }
    }
}

// ---------------------------------------------------------------- k_prologue
// One block of 256 per SM at most (200 registers): the C~ congruence and its LU factors stay in
// registers, where a two-block bound of 128 registers spilled ~0.5 kB per thread to local memory
// (its write-back nearly doubled the kernel's DRAM writes).
__global__ void __launch_bounds__(kBlock, 1) k_prologue(Dev d, const double* __restrict__ c0g, const double* __restrict__ g0g,
                                                       int do_schmid, int modal) {
    __shared__ double c0[81], g0[81], c0b[36];
    for (int i = threadIdx.x; i < 81; i += blockDim.x) {
        c0[i] = c0g[i];
        g0[i] = modal ? g0g[i] : 0.0;
    }
    __syncthreads();
    if (threadIdx.x == 0) t4_to_b66(c0, c0b);
    __syncthreads();
    const long long N = d.N;
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < N; v += (long long)gridDim.x * blockDim.x) {
        const bool gas = d.gas[v];
        if (do_schmid && !gas) {
            const PhaseDev& ph = d.ph[d.phase[v]];
            double Fe[9], ag[9], aa[9], ai[9];
            ld9(d.Fe, N, v, Fe);
            ld9(d.ag, N, v, ag);
            mm3(Fe, ag, aa);
            if (inv3u(aa, ai) != 0) set_err(d.err, 1);
            for (int s = 0; s < ph.nsyst; s++) {
                double S[9], t[9], r[9], rs[9], b5[5];
#pragma unroll
                for (int i = 0; i < 3; i++)
#pragma unroll
                    for (int j = 0; j < 3; j++) S[3 * i + j] = ph.dbca[3 * s + i] * ph.dnca[3 * s + j];
                mm3(aa, S, t);
                mm3(t, ai, r);
                sym33(r, rs);
                t2_to_b5(rs, b5);
#pragma unroll
                for (int c = 0; c < 5; c++) d.sch[(s * 5 + c) * N + v] = b5[c];
            }
        }
        double F[9], detF = d.detF[v];
        ld9(d.F, N, v, F);
        // calc_c066mod: cm_ijkl = sum_mn c0_imkn F_jm F_ln / J, quarter-symmetrized, in the b-basis;
        // c0 has the minor symmetries, so this is (1/J) T(F) c0_66 T(F)^T
        double c66[36], TF[36];
        basis_T(F, TF);
        congruence6(TF, c0b, 1.0 / detF, c66);
#pragma unroll
        for (int c = 0; c < 36; c++) d.c066mod[c * N + v] = c66[c];
        // its inverse, for the symmetric form of the local Newton system, a column at a time from
        // the LU factors (the bits of inv_unrolled without its identity block in registers)
        int piv[6];
        if (lu_unrolled<6>(c66, piv) != 0 && !gas) set_err(d.err, 1);
#pragma unroll
        for (int j = 0; j < 6; j++) {
            double x[6];
            lu_inverse_column<6>(c66, piv, j, x);
#pragma unroll
            for (int i = 0; i < 6; i++) d.c066inv[(6 * i + j) * N + v] = x[i];
        }
    }
}
// calc_c066mod_Goperr066mod, the modified augmented Lagrangian part (various_functions.f90:866-900):
// cG = C~ : Gamma~r with Gamma~r = sym(J Gamma^r(0) F^-1 F^-1), for --modal 1 only (a kernel of its
// own, so that its 3x3x3x3 work arrays do not burden the common prologue's registers)
__global__ void __launch_bounds__(kBlock, 2) k_prologue_modal(Dev d, const double* __restrict__ g0g) {
    __shared__ double g0[81];
    for (int i = threadIdx.x; i < 81; i += blockDim.x) g0[i] = g0g[i];
    __syncthreads();
    const long long N = d.N;
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < N; v += (long long)gridDim.x * blockDim.x) {
        const double detF = d.detF[v];
        double c66[36];
#pragma unroll
        for (int c = 0; c < 36; c++) c66[c] = d.c066mod[c * N + v];
        {
            double Fi[9], g66[36], cm[81], cs[81];
            ld9(d.Finv, N, v, Fi);
            for (int ii = 0; ii < 3; ii++)
                for (int jj = 0; jj < 3; jj++)
                    for (int kk = 0; kk < 3; kk++)
                        for (int ll = 0; ll < 3; ll++) {
                            double dum = 0.0;
                            for (int m = 0; m < 3; m++)
                                for (int n = 0; n < 3; n++) dum += g0[((ii * 3 + m) * 3 + kk) * 3 + n] * Fi[3 * m + jj] * Fi[3 * n + ll];
                            cm[((ii * 3 + jj) * 3 + kk) * 3 + ll] = dum * detF;
                        }
            for (int ii = 0; ii < 3; ii++)
                for (int jj = 0; jj < 3; jj++)
                    for (int kk = 0; kk < 3; kk++)
                        for (int ll = 0; ll < 3; ll++)
                            cs[((ii * 3 + jj) * 3 + kk) * 3 + ll] =
                                0.25 * (cm[((ii * 3 + jj) * 3 + kk) * 3 + ll] + cm[((jj * 3 + ii) * 3 + kk) * 3 + ll] +
                                        cm[((ii * 3 + jj) * 3 + ll) * 3 + kk] + cm[((jj * 3 + ii) * 3 + ll) * 3 + kk]);
            t4_to_b66(cs, g66);
            for (int i = 0; i < 6; i++)
                for (int j = 0; j < 6; j++) {
                    double s = 0.0;
                    for (int k = 0; k < 6; k++) s += c66[6 * i + k] * g66[6 * k + j];
                    d.cG[(6 * i + j) * N + v] = s;
                    d.c066inv[(6 * i + j) * N + v] -= g66[6 * i + j];  // B of the local Newton system
                }
        }
    }
}
void launch_prologue(const Dev& d, const double* c0, const double* goperr0, int do_schmid, int modal, cudaStream_t st) {
    k_prologue<<<d.grid, d.block, 0, st>>>(d, c0, goperr0, do_schmid, modal);
    if (modal) k_prologue_modal<<<d.grid, d.block, 0, st>>>(d, goperr0);
}

// ---------------------------------------------------------------- k_gas_compl
__global__ void __launch_bounds__(kBlock) k_gas_compl(Dev d, double tdot, double complgas, int modal) {
    const long long N = d.N;
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < N; v += (long long)gridDim.x * blockDim.x) {
        if (!d.gas[v]) {
            for (int c = 0; c < 36; c++) d.cgas[c * N + v] = 0.0;
            continue;
        }
        double a[36];
        for (int i = 0; i < 6; i++)
            for (int j = 0; j < 6; j++) {
                a[6 * i + j] = ((i == j) ? 1.0 : 0.0) + d.c066mod[(6 * i + j) * N + v] / tdot * complgas;
                if (modal) a[6 * i + j] = a[6 * i + j] - d.cG[(6 * i + j) * N + v];
            }
        if (inv_unrolled<6>(a) != 0) set_err(d.err, 1);
        for (int c = 0; c < 36; c++) d.cgas[c * N + v] = a[c];
    }
}
void launch_gas_compl(const Dev& d, double tdot, double complgas, int modal, cudaStream_t st) {
    k_gas_compl<<<d.grid, d.block, 0, st>>>(d, tdot, complgas, modal);
}

// ---------------------------------------------------------------- k_corr
// velgrad += (dvelgradref + du) F^{-1}; averages; dL statistics; mixing.
// GAS false: a solve without a gas phase (no cgas, no gas voxels), whose gas sums stay zero; the
// kernel then holds eleven fewer running sums and runs without spills (-12 % at 64^3).
template <bool GAS>
__device__ __forceinline__ void body_corr(const Dev& d, const CorrParams& p, const VB& vb) {
    const long long N = d.N;
    __shared__ double du[9];
    if (threadIdx.x < 9) du[threadIdx.x] = __ldcg(&d.red[OFF_DU + threadIdx.x]);
    __syncthreads();
    double s[31];
#pragma unroll
    for (int c = 0; c < 31; c++) s[c] = 0.0;
    for (long long v = vb.x * (long long)blockDim.x + threadIdx.x; v < N; v += (long long)vb.nx * blockDim.x) {
        double t[9], fi[9], u[9], vg[9], vo[9];
        ld9(d.dvr, N, v, t);
        ld9(d.Finv, N, v, fi);
#pragma unroll
        for (int c = 0; c < 9; c++) t[c] = t[c] + du[c];
        mm3(t, fi, u);
        ld9(d.velgrad, N, v, vg);
        ld9(d.velgradold, N, v, vo);
        const double w = d.wgtc[v];
        const bool gas = GAS && d.gas[v];
#pragma unroll
        for (int c = 0; c < 9; c++) {
            vg[c] = vg[c] + u[c];
            s[c] += vg[c] * w;
            if (gas) s[9 + c] += vg[c] * w;
            else s[18 + c] += vg[c] * w;
        }
        if (!p.kinematic) {
            double dl = 0.0;
#pragma unroll
            for (int c = 0; c < 9; c++) dl += (vg[c] - vo[c]) * (vg[c] - vo[c]);
            dl = sqrt(dl);
            double rel = dl / p.Lscale;
            if (gas) { s[29] += (rel * rel) * w; s[30] += w; }
            else { s[27] += (rel * rel) * w; s[28] += w; }
        }
#pragma unroll
        for (int c = 0; c < 9; c++) vg[c] = p.do_mix ? p.mix * vg[c] + (1.0 - p.mix) * vo[c] : p.mix * vg[c];
        st9(d.velgrad, N, v, vg);
        st9(d.velgradold, N, v, vg);
    }
    reduce_store<31, 0>(s, nullptr, d.partials, d.red + OFF_CORR, d.counters + CNT_CORR, vb);
}

// ---------------------------------------------------------------- batched launches of the iteration's voxel passes
// Each block finds its member in the launch's parameter (binary search on blk0), reads
// the member's control block and runs the same body as the member's single-solve
// launch, on the member's own block coordinates.  Blocks of members that are not
// iterating (converged, waiting for the host) exit at once.
template <bool GAS>
__global__ void __launch_bounds__(kBlock, 2) kb_corr(const __grid_constant__ BatchParams P) {
    __shared__ CorrParams p;
    __shared__ int go;
    const Job& jb = batch_job(P);
    const BatchSolve& m = P.E[jb.solve];
    if (threadIdx.x == 0) {
        go = m.ctl->active;
        p = m.ctl->corr;
    }
    __syncthreads();
    if (!go) return;
    body_corr<GAS>(m.d, p, job_vb(jb));
}
void member_jobs_voxel(const Dev& d, MemberJobs& mj) {
    auto one_d = [&](int k, int grid, int thr, size_t sm, int variant) {
        mj.job[0][k] = Job{0, 0, grid, 1, 1, 0};
        mj.threads[0][k] = thr;
        mj.smem[0][k] = sm;
        mj.variant[0][k] = variant;
    };
    // k_corr: fewer blocks than the other voxel kernels, so that each thread's several voxels spread the
    // 31-field block reduction over more loads; members of one block size share a launch:
    // variant = (no gas phase) + 2 * (block size / 32)
    one_d(BK_CORR, d.grid < 148 * 2 ? d.grid : 148 * 2, d.block, 0, (d.cgas ? 0 : 1) + 2 * (d.block / 32));
    const NewtonShape n = newton_shape(d);
    one_d(BK_NEWTON, n.grid, n.threads, n.smem, n.variant);
}

void launch_batched_voxel(const BatchLaunch& L, const BatchParams& P, cudaStream_t st) {
    switch (L.kind) {
        case BK_CORR:
            if ((L.variant & 1) == 0) kb_corr<true><<<L.blocks, L.threads, 0, st>>>(P);
            else kb_corr<false><<<L.blocks, L.threads, 0, st>>>(P);
            break;
        case BK_NEWTON:
            launch_batched_newton(L, P, st);
            break;
        default: break;
    }
}

// ---------------------------------------------------------------- k_upd1
template <int NS>
__global__ void __launch_bounds__(kBlock) k_upd1(Dev d, Upd1Params p) {
    const long long N = d.N;
    double s[39], mx[1] = {0.0};
#pragma unroll
    for (int c = 0; c < 39; c++) s[c] = 0.0;
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < N; v += (long long)gridDim.x * blockDim.x) {
        const bool gas = d.gas[v];
        // accepted-step commit (LS-EVPFFT.f90:432-446)
        double e6[6], a6[6], vg[9], vs[9];
        ld6(d.edotp, N, v, e6);
        ld6(d.ept, N, v, a6);
#pragma unroll
        for (int c = 0; c < 6; c++) a6[c] = a6[c] + e6[c] * p.tdot;
        st6(d.ept, N, v, a6);
        ld6(d.sg, N, v, a6);
        st6(d.sgt, N, v, a6);
        ld9(d.velgrad, N, v, vg);
        sym33(vg, vs);
        ld6(d.disgradsym, N, v, a6);
        double vs6[6];
        t2_to_s6(vs, vs6);
#pragma unroll
        for (int c = 0; c < 6; c++) a6[c] = a6[c] + vs6[c] * p.tdot;
        st6(d.disgradsym, N, v, a6);
        double e9[9];
        s6_to_t2(e6, e9);
        d.epvm[v] = d.epvm[v] + vm_strain(e9) * p.tdot;
        const double evm = vm_strain(vs);
        if (!gas) mx[0] = fmax(mx[0], evm);
        if (!p.iupdate) continue;
        if (!gas) {  // update_plastic_defgrad (various_functions.f90:1748-1827)
            const PhaseDev& ph = d.ph[d.phase[v]];
            double ag[9], Lp[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
            ld9(d.ag, N, v, ag);
            for (int is = 0; is < ph.nsyst; is++) {
                double dn[3], db[3];
                for (int i = 0; i < 3; i++) {
                    dn[i] = ag[3 * i] * ph.dnca[3 * is] + ag[3 * i + 1] * ph.dnca[3 * is + 1] + ag[3 * i + 2] * ph.dnca[3 * is + 2];
                    db[i] = ag[3 * i] * ph.dbca[3 * is] + ag[3 * i + 1] * ph.dbca[3 * is + 1] + ag[3 * i + 2] * ph.dbca[3 * is + 2];
                }
                const double gd = d.gamdot[is * N + v];
                for (int i = 0; i < 3; i++)
                    for (int j = 0; j < 3; j++) Lp[3 * i + j] = Lp[3 * i + j] + db[i] * dn[j] * gd;
            }
            double dl[9], ex[9], fp[9];
            for (int c = 0; c < 9; c++) dl[c] = Lp[c] * p.tdot;
            if (expm_adaptive(dl, ex) != 0) set_err(d.err, 1);
            ld9(d.Fp, N, v, fp);
            mm3(ex, fp, fp);
            st9(d.Fp, N, v, fp);
        }
        // update_defgrad (various_functions.f90:2152-2282)
        double dl[9], ex[9], F[9], Fi[9];
        for (int c = 0; c < 9; c++) dl[c] = vg[c] * p.tdot;
        if (expm_adaptive(dl, ex) != 0) set_err(d.err, 1);
        ld9(d.F, N, v, F);
        mm3(ex, F, F);
        const double detF = det33(F);
        if (inv3u(F, Fi) != 0) set_err(d.err, 1);
        st9(d.F, N, v, F);
        st9(d.Finv, N, v, Fi);
        st9(d.Finc, N, v, ex);
        d.detF[v] = detF;
        d.wgtc[v] = d.wgt * detF;
#pragma unroll
        for (int c = 0; c < 9; c++) {
            s[c] += F[c] * d.wgt;
            s[9 + c] += Fi[c] * d.wgt * detF;
            if (gas) s[27 + c] += Fi[c] * d.wgt * detF;
            else s[18 + c] += Fi[c] * d.wgt * detF;
        }
        if (gas) s[37] += d.wgt * detF;
        else s[36] += d.wgt * detF;
        s[38] += detF * d.wgt;
    }
    reduce_store<39, 1>(s, mx, d.partials, d.red + OFF_UPD1, d.counters + CNT_UPD1, hw_vb());
}
void launch_upd1(const Dev& d, const Upd1Params& p, cudaStream_t st) {
    if (d.nsys <= 12) k_upd1<12><<<d.grid, d.block, 0, st>>>(d, p);
    else k_upd1<24><<<d.grid, d.block, 0, st>>>(d, p);
}

// ---------------------------------------------------------------- k_upd2
// SYM: every phase's stiffness is symmetric, so its rotation and inverse are formed in 21 entries.
template <bool SYM>
__global__ void __launch_bounds__(kBlock) k_upd2(Dev d, Upd2Params p) {
    const long long N = d.N;
    const double dav = __ldcg(&d.red[OFF_UPD1 + 38]);
    double s[9];
#pragma unroll
    for (int c = 0; c < 9; c++) s[c] = 0.0;
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < N; v += (long long)gridDim.x * blockDim.x) {
        const bool gas = d.gas[v];
        const double w = d.wgtc[v] / dav;
        d.wgtc[v] = w;
        double Finc[9], Feinc[9];
        ld9(d.Finc, N, v, Finc);
        if (!gas) {
            // update_elstic_defgrad (various_functions.f90:2285-2324): Fe = F (Fp Fini)^-1, Fini = I
            // unless an initial displacement field was given
            const PhaseDev& ph = d.ph[d.phase[v]];
            double Fe[9], Feo[9], Fp[9], Fpi[9], F[9];
            ld9(d.Fe, N, v, Fe);
            if (inv3u(Fe, Feo) != 0) set_err(d.err, 1);
            ld9(d.Fp, N, v, Fp);
            if (d.Fini) {
                double Fi0[9], FpFi[9];
                ld9(d.Fini, N, v, Fi0);
                mm3(Fp, Fi0, FpFi);
                if (inv3u(FpFi, Fpi) != 0) set_err(d.err, 1);
            } else if (inv3u(Fp, Fpi) != 0) {
                set_err(d.err, 1);
            }
            ld9(d.F, N, v, F);
            mm3(F, Fpi, Fe);
            mm3(Fe, Feo, Feinc);
            st9(d.Fe, N, v, Fe);
            st9(d.Feinc, N, v, Feinc);
            // update_el_stiff (various_functions.f90:2327-2402)
            // (the rotation of the crystal stiffness by aa = Fe ag as two 6x6 products in the
            // b-basis, Q c Q^T with Q = rot_b66(aa), instead of index by index over 3x3x3x3 and
            // chg_basis: the same tensor, rounding apart)
            double ag[9], aa[9], Q[36];
            ld9(d.ag, N, v, ag);
            mm3(Fe, ag, aa);
            const double idet = 1.0 / det33(Fe);
            rot_b66(aa, Q);
            if constexpr (SYM) {
                double c66[21], s66[21];
#pragma unroll
                for (int i = 0; i < 6; i++) {
                    double ta[6];
#pragma unroll
                    for (int j = 0; j < 6; j++) {
                        double x = 0.0;
#pragma unroll
                        for (int k = 0; k < 6; k++) x += Q[6 * i + k] * ph.C66[6 * k + j];
                        ta[j] = x;
                    }
#pragma unroll
                    for (int j = 0; j <= i; j++) {
                        double x = 0.0;
#pragma unroll
                        for (int k = 0; k < 6; k++) x += ta[k] * Q[6 * j + k];
                        c66[tri(i, j)] = idet * x;
                    }
                }
                if (inv_sym6(c66, s66) != 0) set_err(d.err, 1);
#pragma unroll
                for (int c = 0; c < 36; c++) d.sg66[c * N + v] = s66[tri(c / 6, c % 6)];
            } else {
                double c66[36];
                congruence6(Q, ph.C66, idet, c66);
                if (inv_unrolled<6>(c66) != 0) set_err(d.err, 1);
#pragma unroll
                for (int c = 0; c < 36; c++) d.sg66[c * N + v] = c66[c];
            }
        } else {
            ld9(d.Feinc, N, v, Feinc);
        }
        // update_tensor_config pass 1 (various_functions.f90:2425-2466)
        const double detei = det33(Feinc);
        double Fii[9];
        if (inv3u(Finc, Fii) != 0) set_err(d.err, 1);
        if (!gas) {
            double R[9], U[9], t[9], m[9], a6[6];
            polar(Finc, R, U);
            ld6(d.disgradsym, N, v, a6);
            s6_to_t2(a6, m);
            mm3(R, m, t);
            mm3_bt(t, R, m);
            t2_to_s6(m, a6);
            st6(d.disgradsym, N, v, a6);
            ld6(d.ept, N, v, a6);
            s6_to_t2(a6, m);
            mm3(R, m, t);
            mm3_bt(t, R, m);
            t2_to_s6(m, a6);
            st6(d.ept, N, v, a6);
            ld6(d.sgt, N, v, a6);
            s6_to_t2(a6, m);
            mm3(Feinc, m, t);
            mm3_bt(t, Feinc, m);
            for (int c = 0; c < 9; c++) m[c] = m[c] / detei;
            t2_to_s6(m, a6);
            st6(d.sgt, N, v, a6);
        }
        double vg[9];
        ld9(d.velgrad, N, v, vg);
        mm3(vg, Fii, vg);
        st9(d.velgrad, N, v, vg);
#pragma unroll
        for (int c = 0; c < 9; c++) s[c] += vg[c] * w;
    }
    // the last block forms du2 = (<L>_prev - <L>) inv(<F^{-1}>_c)
    __shared__ double fsum[9];
    if (!reduce_store<9, 0>(s, nullptr, d.partials, fsum, d.counters + CNT_UPD2, hw_vb())) return;
    __syncthreads();
    if (threadIdx.x == 0) {
        double fc[9], di[9], dd[9], du[9];
        for (int f = 0; f < 9; f++) fc[f] = __ldcg(&d.red[OFF_UPD1 + 9 + f]) / dav;
        if (inv3u(fc, di) != 0) set_err(d.err, 1);
        for (int f = 0; f < 9; f++) dd[f] = p.velgradavg[f] - fsum[f];
        mm3(dd, di, du);
        for (int f = 0; f < 9; f++) d.red[OFF_DU2 + f] = du[f];
    }
}
void launch_upd2(const Dev& d, const Upd2Params& p, cudaStream_t st) {
    if (d.symel) k_upd2<true><<<d.grid, d.block, 0, st>>>(d, p);
    else k_upd2<false><<<d.grid, d.block, 0, st>>>(d, p);
}

// ---------------------------------------------------------------- k_upd3
template <int NS>
__global__ void __launch_bounds__(kBlock, 2) k_upd3(Dev d, Upd3Params p) {
    const long long N = d.N;
    __shared__ double du[9];
    if (threadIdx.x < 9) du[threadIdx.x] = p.iupdate ? __ldcg(&d.red[OFF_DU2 + threadIdx.x]) : 0.0;
    __syncthreads();
    double s[30];
#pragma unroll
    for (int c = 0; c < 30; c++) s[c] = 0.0;
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < N; v += (long long)gridDim.x * blockDim.x) {
        const bool gas = d.gas[v];
        if (p.iupdate) {
            double fi[9], t[9], vg[9];
            ld9(d.Finv, N, v, fi);
            mm3(du, fi, t);
            ld9(d.velgrad, N, v, vg);
#pragma unroll
            for (int c = 0; c < 9; c++) vg[c] = vg[c] + t[c];
            st9(d.velgrad, N, v, vg);
        }
        if (gas) continue;
        const PhaseDev& ph = d.ph[d.phase[v]];
        double gd[NS];
#pragma unroll
        for (int q = 0; q < NS; q++) gd[q] = (q < d.nsys) ? d.gamdot[q * N + v] : 0.0;
        if (p.iuphard) {  // update_hardening (various_functions.f90:1493-1523)
            double tn[NS][2], g1;
            harden<NS>(ph, d.crss, N, v, gd, d.gacumgr[v], p.tdot, tn, g1);
#pragma unroll
            for (int q = 0; q < NS; q++)
                if (q < d.nsys) {
                    d.crss[(2 * q) * N + v] = tn[q][0];
                    d.crss[(2 * q + 1) * N + v] = tn[q][1];
                    d.trialtau[(2 * q) * N + v] = tn[q][0];
                    d.trialtau[(2 * q + 1) * N + v] = tn[q][1];
                }
            d.gacumgr[v] = g1;
        }
        const double w = d.wgtc[v];
        double a[6];
        ld6(d.ept, N, v, a);
#pragma unroll
        for (int c = 0; c < 6; c++) s[c] += a[c] * w;
        if (v == p.vlast) {
            for (int c = 0; c < 6; c++) d.red[OFF_UPD3 + 36 + c] = a[c];
        }
        ld6(d.disgradsym, N, v, a);
#pragma unroll
        for (int c = 0; c < 6; c++) s[6 + c] += a[c] * w;
        if (v == p.vlast) {
            for (int c = 0; c < 6; c++) d.red[OFF_UPD3 + 30 + c] = a[c];
            d.red[OFF_UPD3 + 42] = w;
        }
        ld6(d.edotp, N, v, a);
#pragma unroll
        for (int c = 0; c < 6; c++) s[12 + c] += a[c] * w;
        ld6(d.sgt, N, v, a);
#pragma unroll
        for (int c = 0; c < 6; c++) s[18 + c] += a[c] * w;
        s[24] += d.gacumgr[v];
        s[25] += 1.0;
#pragma unroll
        for (int q = 0; q < NS; q++)
            if (q < ph.nsyst) {
                const double gs = 0.5 * (d.crss[(2 * q) * N + v] + d.crss[(2 * q + 1) * N + v]);
                s[26] += gs;
                s[27] += 1.0;
                s[28] += fabs(gd[q]);
                s[29] += fabs(gd[q]) * gs;
            }
    }
    reduce_store<30, 0>(s, nullptr, d.partials, d.red + OFF_UPD3, d.counters + CNT_UPD3, hw_vb());
}
void launch_upd3(const Dev& d, const Upd3Params& p, cudaStream_t st) {
    if (d.nsys <= 12) k_upd3<12><<<d.grid, d.block, 0, st>>>(d, p);
    else k_upd3<24><<<d.grid, d.block, 0, st>>>(d, p);
}

// ---------------------------------------------------------------- k_diag
// sums: s2a swa s2s sws s2g swg | maxes: mxa mxs mxg vms vmg rms rmg sms smg ccs ccg cgg
// min detF (all), and (min, last index) for solid and gas voxels.
struct MinIdx {
    double v;
    long long i;
};
__device__ __forceinline__ MinIdx min_last(MinIdx a, MinIdx b) {
    if (b.v < a.v) return b;
    if (a.v < b.v) return a;
    return (b.i > a.i) ? b : a;
}
__global__ void __launch_bounds__(kBlock, 2) k_diag(Dev d, double Lfloor) {
    const long long N = d.N;
    double s[6] = {0, 0, 0, 0, 0, 0};
    double m[13];
#pragma unroll
    for (int c = 0; c < 12; c++) m[c] = 0.0;
    m[12] = -EVP_HUGE;  // max of -detF
    MinIdx ms = {EVP_HUGE, -1}, mg = {EVP_HUGE, -1};
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < N; v += (long long)gridDim.x * blockDim.x) {
        const bool gas = d.gas[v];
        double vg[9], vs[9], Fi[9];
        ld9(d.velgrad, N, v, vg);
        ld9(d.s_velgrad, N, v, vs);
        double dl = 0.0, l0 = 0.0;
#pragma unroll
        for (int c = 0; c < 9; c++) { dl += (vg[c] - vs[c]) * (vg[c] - vs[c]); l0 += vs[c] * vs[c]; }
        dl = sqrt(dl);
        l0 = sqrt(l0);
        const double rel = dl / fmax(l0, Lfloor);
        const double w = d.wgtc[v];
        s[0] += (rel * rel) * w; s[1] += w; m[0] = fmax(m[0], rel);
        const double detF = d.detF[v];
        m[12] = fmax(m[12], -detF);
        ld9(d.Finc, N, v, Fi);
        double vi, ro, st, Ji;
        stretch_rot(Fi, true, vi, ro, st, Ji);
        double c66[36];
        for (int c = 0; c < 36; c++) c66[c] = d.c066mod[c * N + v];
        const double cc = cond1_est_6x6(c66);
        if (gas) {
            MinIdx t = {detF, v};
            mg = min_last(mg, t);
            s[4] += (rel * rel) * w; s[5] += w; m[2] = fmax(m[2], rel);
            m[4] = fmax(m[4], vi); m[6] = fmax(m[6], ro); m[8] = fmax(m[8], st);
            m[10] = fmax(m[10], cc);
            for (int c = 0; c < 36; c++) c66[c] = d.cgas[c * N + v];
            m[11] = fmax(m[11], cond1_est_6x6(c66));
        } else {
            MinIdx t = {detF, v};
            ms = min_last(ms, t);
            s[2] += (rel * rel) * w; s[3] += w; m[1] = fmax(m[1], rel);
            m[3] = fmax(m[3], vi); m[5] = fmax(m[5], ro); m[7] = fmax(m[7], st);
            m[9] = fmax(m[9], cc);
        }
    }
    // (min, last index) pairs reduced first, by a fixed-order warp/block tree
    __shared__ MinIdx shm[2][8];
    __shared__ bool lastblk;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    auto block_min = [&](MinIdx& x, MinIdx& y) {  // the result is in thread 0
        for (int o = 16; o > 0; o >>= 1) {
            x = min_last(x, MinIdx{__shfl_down_sync(0xffffffffu, x.v, o), __shfl_down_sync(0xffffffffu, x.i, o)});
            y = min_last(y, MinIdx{__shfl_down_sync(0xffffffffu, y.v, o), __shfl_down_sync(0xffffffffu, y.i, o)});
        }
        __syncthreads();
        if (lane == 0) { shm[0][warp] = x; shm[1][warp] = y; }
        __syncthreads();
        if (threadIdx.x == 0)
            for (int q = 0; q < nw; q++) { x = min_last(x, shm[0][q]); y = min_last(y, shm[1][q]); }
    };
    block_min(ms, mg);
    MinIdx* pm = reinterpret_cast<MinIdx*>(d.partials + (size_t)gridDim.x * 19);
    if (threadIdx.x == 0) {
        pm[2 * blockIdx.x] = ms;
        pm[2 * blockIdx.x + 1] = mg;
    }
    __syncthreads();
    reduce_store<6, 13>(s, m, d.partials, d.red + OFF_DIAG, d.counters + CNT_DIAG, hw_vb());
    // reduce_store reset the counter; use a second counter pass for the pairs
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) lastblk = (atomicAdd(d.counters + CNT_DIAG2, 1u) == gridDim.x - 1);
    __syncthreads();
    if (!lastblk) return;
    // the block pairs: every thread folds some (any order gives the same pair: the smallest value, and
    // of its voxels the last), then the block
    __threadfence();
    ms = MinIdx{EVP_HUGE, -1};
    mg = MinIdx{EVP_HUGE, -1};
    for (unsigned q = threadIdx.x; q < gridDim.x; q += blockDim.x) {
        ms = min_last(ms, MinIdx{__ldcg(&pm[2 * q].v), __ldcg(&pm[2 * q].i)});
        mg = min_last(mg, MinIdx{__ldcg(&pm[2 * q + 1].v), __ldcg(&pm[2 * q + 1].i)});
    }
    block_min(ms, mg);
    if (threadIdx.x == 0) {
        d.red[OFF_DIAG + 19] = ms.v;
        d.red[OFF_DIAG + 20] = (double)ms.i;
        d.red[OFF_DIAG + 21] = mg.v;
        d.red[OFF_DIAG + 22] = (double)mg.i;
        d.counters[CNT_DIAG2] = 0;
    }
}
void launch_diag(const Dev& d, double Lfloor, cudaStream_t st) { k_diag<<<d.grid, d.block, 0, st>>>(d, Lfloor); }

// ---------------------------------------------------------------- k_c0
// SYM: every phase's stiffness is symmetric, and with it both tangents.
__host__ __device__ constexpr int c0_sums(bool sym) { return sym ? 42 : 72; }
template <int NS, bool SYM>
__global__ void __launch_bounds__(kC0Block) k_c0(Dev d, double tdot, double tdotref) {
    const long long N = d.N;
    // each thread's running sums (both tangents, their lower triangles if SYM) in a shared-memory column,
    // entry c of thread t at [c * kC0Block + t]: conflict free, and registers hold the per-voxel work
    constexpr int kSums = c0_sums(SYM);
    extern __shared__ double c0acc[];
    double* const s = c0acc + threadIdx.x;
    for (int c = 0; c < kSums; c++) s[c * kC0Block] = 0.0;
    const double itr = 1.0 / tdotref;
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < N; v += (long long)gridDim.x * blockDim.x) {
        if (d.gas[v]) continue;
        const PhaseDev& ph = d.ph[d.phase[v]];
        double a6[6], sg[6];
        ld6(d.sg, N, v, a6);
        s6_to_b6(a6, sg);
        double tt[NS][2], ep[6], dd[15], gd[NS];
#pragma unroll
        for (int q = 0; q < NS; q++) {
            tt[q][0] = (q < d.nsys) ? d.trialtau[(2 * q) * N + v] : 1.0;
            tt[q][1] = (q < d.nsys) ? d.trialtau[(2 * q + 1) * N + v] : 1.0;
        }
        constitutive<NS>(ph, d.sch, N, v, tt, sg, ep, dd, gd);
        // de/dsg = S / tdotref + dd (symmetric positive definite if SYM) and its inverse dsg in the b-basis
        // (summed here, expanded to 3x3x3x3 on the host); the PK1 tangent dpg_ijkl = J sum_mn dsg_imkn Fi_jm
        // Fi_ln has the b-basis components J T(Fi) dsg T(Fi)^T
        double Fi[9], T[36];
        if constexpr (SYM) {
            double h[21], tr[21];
#pragma unroll
            for (int i = 0; i < 6; i++)
#pragma unroll
                for (int j = 0; j <= i; j++) h[tri(i, j)] = d.sg66[(6 * j + i) * N + v] * itr + dd_at(dd, i, j);
            if (inv_sym6(h, tr) != 0) set_err(d.err, 1);
            ld9(d.Finv, N, v, Fi);
            const double detF = d.detF[v], w = d.wgtc[v];
            basis_T(Fi, T);
#pragma unroll
            for (int c = 0; c < 21; c++) s[c * kC0Block] += tr[c] * w;
#pragma unroll
            for (int i = 0; i < 6; i++) {
                double ta[6];
#pragma unroll
                for (int j = 0; j < 6; j++) {
                    double x = 0.0;
#pragma unroll
                    for (int k = 0; k < 6; k++) x += T[6 * i + k] * tr[tri(k, j)];
                    ta[j] = x;
                }
#pragma unroll
                for (int j = 0; j <= i; j++) {
                    double x = 0.0;
#pragma unroll
                    for (int k = 0; k < 6; k++) x += ta[k] * T[6 * j + k];
                    s[(21 + tri(i, j)) * kC0Block] += (detF * x) * d.wgt;
                }
            }
        } else {
            double tr[36], dp6[36];
#pragma unroll
            for (int i = 0; i < 6; i++)
#pragma unroll
                for (int j = 0; j < 6; j++) tr[6 * i + j] = d.sg66[(6 * i + j) * N + v] * itr + dd_at(dd, i, j);
            if (inv_unrolled<6>(tr) != 0) set_err(d.err, 1);
            ld9(d.Finv, N, v, Fi);
            const double detF = d.detF[v], w = d.wgtc[v];
            basis_T(Fi, T);
            congruence6(T, tr, detF, dp6);
#pragma unroll
            for (int c = 0; c < 36; c++) {
                s[c * kC0Block] += tr[c] * w;
                s[(36 + c) * kC0Block] += dp6[c] * d.wgt;
            }
        }
    }
    __shared__ double fs[kSums];
    if (!reduce_store<kSums, 0>(s, nullptr, d.partials, fs, d.counters + CNT_C0, hw_vb(), kC0Block)) return;
    __syncthreads();
    for (int c = threadIdx.x; c < 72; c += blockDim.x) {
        const int e = c % 36;
        d.red[OFF_C0 + c] = SYM ? fs[(c / 36) * 21 + tri(e / 6, e % 6)] : fs[c];
    }
}
template <int NS, bool SYM>
static void c0_launch(const Dev& d, int grid, double tdot, double tdotref, cudaStream_t st) {
    const size_t sm = (size_t)kC0Block * c0_sums(SYM) * sizeof(double);
    cudaFuncSetAttribute(k_c0<NS, SYM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    k_c0<NS, SYM><<<grid, kC0Block, sm, st>>>(d, tdot, tdotref);
}
void launch_c0(const Dev& d, double tdot, double tdotref, cudaStream_t st) {
    // four blocks per SM (the 255-register bound allows four of 64 threads): one wave, each
    // thread several voxels, and a fold of 592 block partials per field instead of 2368.
    // At 64^3 (event-timed) 434 us with 72 sums a thread side by side (16-way bank conflicts),
    // the general inverse and two divisions for each entry of S / tdotref; 142 now.
    const long long g = (d.N + kC0Block - 1) / kC0Block;
    const int grid = (int)(g < 148LL * 4 ? g : 148LL * 4);
    if (d.symel) d.nsys <= 12 ? c0_launch<12, true>(d, grid, tdot, tdotref, st) : c0_launch<24, true>(d, grid, tdot, tdotref, st);
    else d.nsys <= 12 ? c0_launch<12, false>(d, grid, tdot, tdotref, st) : c0_launch<24, false>(d, grid, tdot, tdotref, st);
}

// ---------------------------------------------------------------- k_kinematic
__global__ void __launch_bounds__(kBlock) k_kinematic(Dev d, double tdot_step) {
    const long long N = d.N;
    double m[4] = {0.0, 0.0, 0.0, -EVP_HUGE};
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < N; v += (long long)gridDim.x * blockDim.x) {
        double L[9], Fi[9];
        ld9(d.velgrad, N, v, L);
        for (int c = 0; c < 9; c++) L[c] = L[c] * tdot_step;
        if (expm_adaptive(L, Fi) != 0) set_err(d.err, 1);
        double vi, ro, st, Ji;
        stretch_rot(Fi, false, vi, ro, st, Ji);
        m[0] = fmax(m[0], vi);
        m[1] = fmax(m[1], ro);
        m[2] = fmax(m[2], st);
        m[3] = fmax(m[3], -(d.detF[v] * Ji));
    }
    reduce_store<0, 4>(nullptr, m, d.partials, d.red + OFF_KIN, d.counters + CNT_KIN, hw_vb());
}
void launch_kinematic(const Dev& d, double tdot_step, cudaStream_t st) { k_kinematic<<<d.grid, d.block, 0, st>>>(d, tdot_step); }

// ---------------------------------------------------------------- k_cell2node
__global__ void __launch_bounds__(kBlock) k_cell2node(Dev d, double tdot, int ideriv) {
    const int n1 = d.n1, n2 = d.n2, n3 = d.n3;
    const long long nn1 = n1 + 1, nn2 = n2 + 1;
    const long long nnode = nn1 * nn2 * d.n3node;
    __shared__ double va[9];
    if (threadIdx.x < 9) va[threadIdx.x] = __ldcg(&d.red[OFF_DC + 2 * threadIdx.x]) * d.wgt;
    __syncthreads();
    const long long N = d.N;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < nnode; q += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(q % nn1) + 1, j = (int)((q / nn1) % nn2) + 1, k = (int)(q / (nn1 * nn2)) + 1;
        double dn[3];
        if (ideriv != 2) {
            int k1 = k - 1, k2 = k, j1 = j - 1, j2 = j, i1 = i - 1, i2 = i;
            if (k1 == 0) k1 = n3;
            if (k2 == n3 + 1) k2 = 1;
            if (j1 == 0) j1 = n2;
            if (j2 == n2 + 1) j2 = 1;
            if (i1 == 0) i1 = n1;
            if (i2 == n1 + 1) i2 = 1;
            auto c = [&](int a, int b, int e, int l) {
                return d.dv3[l * N + (a - 1) + (long long)n1 * ((b - 1) + (long long)n2 * (e - 1))];
            };
            for (int l = 0; l < 3; l++)
                dn[l] = (c(i2, j2, k2, l) + c(i1, j2, k2, l) + c(i2, j1, k2, l) + c(i2, j2, k1, l) + c(i1, j1, k2, l) +
                         c(i1, j2, k1, l) + c(i2, j1, k1, l) + c(i1, j1, k1, l)) * 0.125;
        } else {
            long long vv = ((i - 1) % n1) + (long long)n1 * (((j - 1) % n2) + (long long)n2 * ((k - 1) % n3));
            for (int l = 0; l < 3; l++) dn[l] = d.dv3[l * N + vv];
        }
        const double x[3] = {(double)i - 0.5, (double)j - 0.5, (d.n3node == 1) ? 0.0 : (double)k - 0.5};
        for (int l = 0; l < 3; l++) {
            const double sv = va[3 * l] * x[0] + va[3 * l + 1] * x[1] + va[3 * l + 2] * x[2];
            d.xnode[3 * q + l] = d.xnode[3 * q + l] + (sv + dn[l]) * tdot;
        }
    }
}
void launch_cell2node(const Dev& d, double tdot, int ideriv, cudaStream_t st) {
    k_cell2node<<<d.grid, d.block, 0, st>>>(d, tdot, ideriv);
}

// ---------------------------------------------------------------- k_interleave
// One thread per output value: writes are contiguous, and the reads of a warp take whole 32-byte
// sectors of each plane.  Bound by the copy to the host that follows (PCIe), not by HBM.
struct InterleaveMap {
    unsigned char c[kMaxInterleave];
};
__global__ void __launch_bounds__(kBlock) k_interleave(const double* __restrict__ in, InterleaveMap map, int nout, long long N,
                                                        long long total, double* __restrict__ out) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const long long v = i / nout;
        out[i] = in[(long long)map.c[(int)(i - v * nout)] * N + v];
    }
}
void launch_interleave(const Dev& d, const double* in, const int* map, int nout, long long v0, long long nv, double* out,
                       cudaStream_t st) {
    InterleaveMap m{};
    for (int c = 0; c < nout; c++) m.c[c] = (unsigned char)map[c];
    const long long total = nv * nout, blocks = (total + kBlock - 1) / kBlock;
    k_interleave<<<(int)(blocks < 148LL * 64 ? blocks : 148LL * 64), kBlock, 0, st>>>(in + v0, m, nout, d.N, total, out);
}

// ---------------------------------------------------------------- k_goperr0
__device__ __forceinline__ void spatial_freq(int kx, int ky, int kz, int n1, int n2, int n3, double* xi) {
    const double twopi = 2.0 * EVP_PI;
    xi[0] = (kx + 1 <= n1 / 2) ? twopi * (double)kx / (double)n1 : twopi * (double)(kx - n1) / (double)n1;
    xi[1] = (ky + 1 <= n2 / 2) ? twopi * (double)ky / (double)n2 : twopi * (double)(ky - n2) / (double)n2;
    if (n3 == 1) xi[2] = 0.0;
    else xi[2] = (kz + 1 <= n3 / 2) ? twopi * (double)kz / (double)n3 : twopi * (double)(kz - n3) / (double)n3;
}
// Green operator at one frequency point, all three forms of form_G (various_functions.f90:640-785):
// IGAMMA 0 continuous (Nyquist planes: -s0), 1 discrete central differences followed by four
// projections g <- -g1 : c0 : g, 2 rotated scheme (zero where two Nyquist planes meet).
// kx, ky, kz are 0-based indices of the full spectrum.  Returns 1 for a singular acoustic tensor
// or a complex rotated-scheme D (the reference stops there).
__device__ int goper_at(int igamma, int kx, int ky, int kz, int n1, int n2, int n3, const double* c0, const double* s0,
                        double* g) {
    const bool nx = (n1 % 2 == 0 && kx == n1 / 2), ny = (n2 % 2 == 0 && ky == n2 / 2), nz = (n3 % 2 == 0 && kz == n3 / 2);
    if ((nx || ny || (nz && n3 > 1)) && igamma == 0) {
        for (int c = 0; c < 81; c++) g[c] = -s0[c];
        return 0;
    }
    if (((nx && ny) || (nx && nz) || (ny && nz)) && igamma >= 2) {
        for (int c = 0; c < 81; c++) g[c] = 0.0;
        return 0;
    }
    int bad = 0;
    double xk[3], D[9];
    spatial_freq(kx, ky, kz, n1, n2, n3, xk);
    if (igamma == 0) {
        for (int i = 0; i < 3; i++)
            for (int j = 0; j < 3; j++) D[3 * i + j] = xk[i] * xk[j];
    } else if (igamma == 1) {
        const double twopi = 2.0 * EVP_PI;
        const double xi = twopi * (double)kx / (double)n1, xj = twopi * (double)ky / (double)n2,
                     xz = twopi * (double)kz / (double)n3;
        D[0] = 2.0 * (cos(xi) - 1.0);
        D[4] = 2.0 * (cos(xj) - 1.0);
        D[8] = 2.0 * (cos(xz) - 1.0);
        D[3] = -sin(xi) * sin(xj);
        D[6] = -sin(xi) * sin(xz);
        D[7] = -sin(xj) * sin(xz);
        D[1] = D[3];
        D[2] = D[6];
        D[5] = D[7];
    } else {
        // kmod = i/4 (1 + e^{i xk1})(1 + e^{i xk2})(1 + e^{i xk3}) tan(xk/2); D = Re(kmod kmod^*)
        double br = 0.0, bi = 0.25;
        for (int l = 0; l < 3; l++) {
            const double fr = 1.0 + cos(xk[l]), fi = sin(xk[l]);
            const double r = br * fr - bi * fi, im = br * fi + bi * fr;
            br = r;
            bi = im;
        }
        double kr[3], ki[3];
        for (int l = 0; l < 3; l++) {
            const double t = tan(xk[l] / 2.0);
            kr[l] = t * br;
            ki[l] = t * bi;
        }
        double im2 = 0.0;
        for (int i = 0; i < 3; i++)
            for (int j = 0; j < 3; j++) {
                D[3 * i + j] = kr[i] * kr[j] + ki[i] * ki[j];
                const double dim = ki[i] * kr[j] - kr[i] * ki[j];
                im2 += dim * dim;
            }
        if (sqrt(im2) > 1.0e-7) bad = 1;
    }
    double a[9];
    if (kx == 0 && ky == 0 && kz == 0) {
        for (int c = 0; c < 9; c++) a[c] = 0.0;
    } else {
        double A[9];
        for (int i = 0; i < 3; i++)
            for (int k = 0; k < 3; k++) {
                double x = 0.0;
                for (int j = 0; j < 3; j++)
                    for (int l = 0; l < 3; l++) x += c0[((i * 3 + j) * 3 + k) * 3 + l] * D[3 * j + l];
                A[3 * i + k] = x;
            }
        if (inv3u(A, a) != 0) bad = 1;
    }
    for (int p = 0; p < 3; p++)
        for (int q = 0; q < 3; q++)
            for (int i = 0; i < 3; i++)
                for (int j = 0; j < 3; j++) g[((p * 3 + q) * 3 + i) * 3 + j] = -a[3 * p + i] * D[3 * q + j];
    if (igamma == 1) {
        // g <- -g1 : (c0 : g) four times, as two 9x9 products (the four-fold sum regrouped)
        double g1[81], t[81];
        for (int c = 0; c < 81; c++) g1[c] = g[c];
        for (int itt = 0; itt < 4; itt++) {
            for (int mn = 0; mn < 9; mn++)
                for (int kl = 0; kl < 9; kl++) {
                    double x = 0.0;
                    for (int op = 0; op < 9; op++) x += c0[mn * 9 + op] * g[op * 9 + kl];
                    t[mn * 9 + kl] = x;
                }
            for (int ij = 0; ij < 9; ij++)
                for (int kl = 0; kl < 9; kl++) {
                    double x = 0.0;
                    for (int mn = 0; mn < 9; mn++) x += g1[ij * 9 + mn] * t[mn * 9 + kl];
                    g[ij * 9 + kl] = -x;
                }
        }
    }
    return bad;
}

// Real-space origin value of the Green operator (mean over the full spectrum), used by the
// modified augmented Lagrangian (various_functions.f90:798-807).
__global__ void __launch_bounds__(kBlock) k_goperr0(Dev d, const double* __restrict__ c0g, const double* __restrict__ s0g,
                                                    int igamma) {
    __shared__ double c0[81], s0[81];
    for (int i = threadIdx.x; i < 81; i += blockDim.x) { c0[i] = c0g[i]; s0[i] = s0g[i]; }
    __syncthreads();
    const long long N = d.N;
    const int n1 = d.n1, n2 = d.n2, n3 = d.n3;
    double s[81];
#pragma unroll
    for (int c = 0; c < 81; c++) s[c] = 0.0;
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < N; v += (long long)gridDim.x * blockDim.x) {
        const int kx = (int)(v % n1), ky = (int)((v / n1) % n2), kz = (int)(v / ((long long)n1 * n2));
        if (igamma != 0) {
            double g[81];
            if (goper_at(igamma, kx, ky, kz, n1, n2, n3, c0, s0, g) != 0) set_err(d.err, 4);
            for (int c = 0; c < 81; c++) s[c] += g[c];
            continue;
        }
        const bool nyq = (n1 % 2 == 0 && kx == n1 / 2) || (n2 % 2 == 0 && ky == n2 / 2) || (n3 % 2 == 0 && kz == n3 / 2 && n3 > 1);
        if (nyq) {
            for (int c = 0; c < 81; c++) s[c] += -s0[c];
            continue;
        }
        if (v == 0) continue;
        double xi[3], A[9], a[9];
        spatial_freq(kx, ky, kz, n1, n2, n3, xi);
        for (int i = 0; i < 3; i++)
            for (int k = 0; k < 3; k++) {
                double x = 0.0;
                for (int j = 0; j < 3; j++)
                    for (int l = 0; l < 3; l++) x += c0[((i * 3 + j) * 3 + k) * 3 + l] * (xi[j] * xi[l]);
                A[3 * i + k] = x;
            }
        if (inv3u(A, a) != 0) set_err(d.err, 1);
        for (int p = 0; p < 3; p++)
            for (int q = 0; q < 3; q++)
                for (int i = 0; i < 3; i++)
                    for (int j = 0; j < 3; j++) s[((p * 3 + q) * 3 + i) * 3 + j] += -a[3 * p + i] * (xi[q] * xi[j]);
    }
    reduce_store<81, 0>(s, nullptr, d.partials, d.red + OFF_G0, d.counters + CNT_G0, hw_vb());
}
void launch_goperr0(const Dev& d, const double* c0, const double* s0, int igamma, cudaStream_t st) {
    k_goperr0<<<d.grid, d.block, 0, st>>>(d, c0, s0, igamma);
}

// form_G for IGAMMA 1 and 2 on the half spectrum, once per increment (c0 changes per increment)
__global__ void __launch_bounds__(kBlock) k_goper_tab(Dev d, const double* __restrict__ c0g, const double* __restrict__ s0g,
                                                      int igamma) {
    __shared__ double c0[81], s0[81];
    for (int i = threadIdx.x; i < 81; i += blockDim.x) { c0[i] = c0g[i]; s0[i] = s0g[i]; }
    __syncthreads();
    const int n1h = d.n1h, n2 = d.n2, n3 = d.n3;
    const long long P = (long long)n1h * n2 * n3;
    for (long long pt = blockIdx.x * (long long)blockDim.x + threadIdx.x; pt < P; pt += (long long)gridDim.x * blockDim.x) {
        const int kx = (int)(pt % n1h), j = (int)((pt / n1h) % n2), k3 = (int)(pt / ((long long)n1h * n2));
        double g[81];
        if (goper_at(igamma, kx, j, k3, d.n1, n2, n3, c0, s0, g) != 0) set_err(d.err, 4);
        for (int c = 0; c < 81; c++) d.goper[c * P + pt] = g[c];
    }
}
void launch_goper_tab(const Dev& d, const double* c0, const double* s0, int igamma, cudaStream_t st) {
    k_goper_tab<<<d.grid, d.block, 0, st>>>(d, c0, s0, igamma);
}

}  // namespace evp
