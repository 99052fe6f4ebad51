// Derivatives of the Kim functional and of the converged OMM energy.
//
// Functional gradient (libOMM's calc_G, omm_ops.F90:17-39): for
//     Omega(C) = tr[(2I - S_W) H_W],  H_W = C H C^H,  S_W = C S C^H,
// dOmega/dC = G = 4 HC - 2 S_W HC - 2 H_W SC  (HC = C H, SC = C S).
//
// Energy adjoint: the converged energy E(theta) = min_C Omega(C; H(theta))
// with H(theta) = H0 + sum_k theta_k V_k is stationary in C, so
//     dE/dtheta_k = dOmega/dtheta_k |_{C*} = Re sum_ij conj(D_ij) (V_k)_ij,
//     D = C^H (2I - S_W) C
// (the density matrix that omm() returns, omm.F90:575-582).  D is m x m and
// dense.  With CD = (2I - S_W) C (n x m), conj(D_ij) = sum_a C_ai conj(CD_aj),
// and there are two ways to the sum over the nonzeros (i, j, v) of the V_k:
//   * SDDMM: each nonzero contributes v * <C(:,i), conj(CD(:,j))>.  One column j of
//     V per CTA, CD(:,j) in shared memory, a warp per nonzero.  Bound by the n-vector
//     of C that every nonzero reads from L2 (about 9.5 TB/s).
//   * density panels: the upper triangle of D in column panels of at most 1 GiB as
//     FP64-accurate products on the tensor cores, then one gather of v conj(D_ij) over
//     the nonzeros of all V_k.  Its cost does not grow with the nonzeros.
#include "internal.h"

#include <algorithm>
#include <cmath>

namespace ommgpu {

namespace {

const double ONE[2] = {1.0, 0.0}, ZERO[2] = {0.0, 0.0}, MONE[2] = {-1.0, 0.0};

DView make_view(DevBuf& b, int rows, int cols, bool real, bool zero = false) {
    const size_t bytes = std::max<size_t>(1, (size_t)rows * cols) * (real ? 8 : 16);
    if (zero) b.alloc_zero(bytes);
    else b.alloc(bytes);
    return DView{b.p, rows, cols, std::max(1, rows), real};
}

// A * M for M = H or S (dense or CSC); out n x m
void apply(const DView& A, const msw_matrix* M, DView& out, int m) {
    if (M->dense()) {
        Staged s;
        stage_in(M, s);
        gemm('n', 'n', A.rows, m, m, ONE, A, s.v, ZERO, out);
        if (M->loc == Loc::Host) sync();  // the staged copy goes out of scope
    } else {
        spmm_dense_csc(A, M, out, ONE, ZERO);
    }
}

// out = C (the S half of a product stack when there is no S); out is written in full
void copy_into(const DView& C, DView& out) {
    const size_t es = C.is_real ? 8 : 16;
    if (C.rows && C.cols)
        OMM_CK(cudaMemcpy2DAsync(out.p, (size_t)out.ld * es, C.p, (size_t)C.ld * es, (size_t)C.rows * es, C.cols,
                                 cudaMemcpyDeviceToDevice, rt().stream));
}

constexpr int kAdjThreads = 256;

// grad partial per CTA: sum over nonzeros (i, v) of column j of V of
// Re( v * sum_a C(a,i) * conj(CD(a,j)) ).
template <bool REAL>
__global__ void __launch_bounds__(kAdjThreads) adjoint_sddmm_kernel(int n, const double* __restrict__ C, int ldc,
                                                                   const double* __restrict__ CD, int ldcd,
                                                                   const int* __restrict__ colptr,
                                                                   const int* __restrict__ rowind,
                                                                   const double* __restrict__ val, double* part) {
    extern __shared__ double s_cd[];  // n (real) or 2n (complex) values of CD(:, j)
    const int j = blockIdx.x;
    const int w = REAL ? 1 : 2;
    for (int a = threadIdx.x; a < n * w; a += blockDim.x) s_cd[a] = CD[(size_t)j * ldcd * w + a];
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    double acc = 0.0;
    for (int l = colptr[j] + warp; l < colptr[j + 1]; l += nw) {
        const int i = rowind[l];
        const double* ci = C + (size_t)i * ldc * w;
        double re = 0.0, im = 0.0;
        if (REAL) {
            for (int a = lane; a < n; a += 32) re = fma(ci[a], s_cd[a], re);
        } else {
            for (int a = lane; a < n; a += 32) {
                double cr = ci[2 * a], cim = ci[2 * a + 1], dr = s_cd[2 * a], di = s_cd[2 * a + 1];
                re += cr * dr + cim * di;  // C * conj(CD)
                im += cim * dr - cr * di;
            }
        }
        for (int o = 16; o > 0; o >>= 1) {
            re += __shfl_down_sync(0xffffffffu, re, o);
            im += __shfl_down_sync(0xffffffffu, im, o);
        }
        if (lane == 0) {
            if (REAL) acc += val[l] * re;
            else acc += val[2 * l] * re - val[2 * l + 1] * im;  // Re(v * z)
        }
    }
    __shared__ double s_acc[kAdjThreads / 32];
    if (lane == 0) s_acc[warp] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int q = 0; q < nw; ++q) s += s_acc[q];
        part[j] = s;
    }
}

// The CSC arrays of up to kVBatch perturbations, for the kernels that take all of them in one launch
constexpr int kVBatch = 32;
struct VList {
    const int* colptr[kVBatch];
    const int* rowind[kVBatch];
    const double* val[kVBatch];
};

// part[k m + j] (+)= sum over the nonzeros (i, v) of column j of V_k with c0 <= max(i, j) < c1 of
// Re(v conj(D_ij)), D's columns c0 .. c1 - 1 given down to the diagonal at least (D is Hermitian: below
// it D_ij = conj(D_ji)).  One warp per column.
template <bool REAL>
__global__ void __launch_bounds__(kAdjThreads) adjoint_gather_kernel(int m, int c0, int c1,
                                                                    const double* __restrict__ D, int ldd,
                                                                    const __grid_constant__ VList V, int first,
                                                                    double* __restrict__ part) {
    const int j = blockIdx.x * (kAdjThreads / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31, k = blockIdx.y;
    if (j >= m) return;
    const int* __restrict__ rowind = V.rowind[k];
    const double* __restrict__ val = V.val[k];
    const int e = V.colptr[k][j + 1];
    double acc = 0.0;
    for (int l = V.colptr[k][j] + lane; l < e; l += 32) {
        const int i = rowind[l], lo = min(i, j), hi = max(i, j);
        if (hi < c0 || hi >= c1) continue;
        const size_t at = (size_t)lo + (size_t)(hi - c0) * ldd;
        if (REAL) {
            acc = fma(val[l], D[at], acc);
        } else {
            const double2 d = reinterpret_cast<const double2*>(D)[at];
            const double2 v = reinterpret_cast<const double2*>(val)[l];
            acc += v.x * d.x + (i > j ? -v.y : v.y) * d.y;
        }
    }
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if (lane == 0) {
        double* p = part + (size_t)k * m + j;
        *p = first ? acc : *p + acc;
    }
}

// out[k] = sum of part[k n .. k n + n - 1], one block per k: Neumaier sums of strided shares, combined
// in a fixed tree order
__global__ void __launch_bounds__(256) sum_partials(const double* part, int n, double* out) {
    const double* p = part + (size_t)blockIdx.x * n;
    auto add = [](double& s, double& c, double v) {
        const double t = s + v;
        c += (fabs(s) >= fabs(v)) ? ((s - t) + v) : ((v - t) + s);
        s = t;
    };
    double s = 0.0, c = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) add(s, c, p[i]);
    auto tree = [&]() {
        for (int o = 16; o > 0; o >>= 1) {
            const double s2 = __shfl_down_sync(0xffffffffu, s, o), c2 = __shfl_down_sync(0xffffffffu, c, o);
            add(s, c, s2);
            c += c2;
        }
    };
    __shared__ double ss[8], sc[8];
    tree();
    if ((threadIdx.x & 31) == 0) {
        ss[threadIdx.x >> 5] = s;
        sc[threadIdx.x >> 5] = c;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        s = threadIdx.x < 8 ? ss[threadIdx.x] : 0.0;
        c = threadIdx.x < 8 ? sc[threadIdx.x] : 0.0;
        tree();
        if (threadIdx.x == 0) out[blockIdx.x] = s + c;
    }
}

// The density panels or the SDDMM for perturbations of nnz nonzeros together, by their estimated times:
// the SDDMM reads n values of C per nonzero from L2 (measured 9.5 TB/s: 335,000 complex nonzeros with
// n = 512 in 283 us); a panel's product runs at about 90 TFLOP/s FP64-equivalent (complex: four real
// ones), a little over half of it formed, and its reconstruction and gather take about 1 us per
// 250,000 elements (four passes for complex).  m = 4,096, n = 512, 16 complex V_k of 2 %: 0.7 ms
// against 4.6; one such V_k: 0.7 against 0.29.
bool adjoint_by_panels(double m, double n, double nnz, bool real) {
    if (!fp64_emu_enabled() || !fp64_emu_worth((int)m, (int)m, (int)n, !real)) return false;
    const double z = real ? 1.0 : 4.0;
    const double panels = 0.55 * z * 2.0 * m * m * n / 90e12 + z * m * m / 250e9 + 30e-6;
    return nnz * n * (real ? 8.0 : 16.0) / 9.5e12 > panels;
}

}  // namespace

// d E / d theta_k for sparse perturbations, given C and CD = (2I - S_W) C on the device
void adjoint_sparse(const DView& C, const DView& CD, const std::vector<const msw_matrix*>& V, double* grad) {
    const int m = C.cols, n = C.rows, nv = (int)V.size();
    const bool real = C.is_real;
    cudaStream_t st = rt().stream;
    const size_t smem = (size_t)n * (real ? 8 : 16);
    if (smem > 200 * 1024) fail(OMM_ERR_UNSUPPORTED, "energy adjoint: n too large for one CD column in shared memory");
    double nnz = 0.0;
    for (const msw_matrix* v : V) {
        ensure_csc_device(v);
        nnz += v->nnz;
    }
    DevBuf part;
    part.alloc(((size_t)nv * m + nv) * sizeof(double));
    double* sums = part.as<double>() + (size_t)nv * m;
    if (adjoint_by_panels(m, n, nnz, real)) {
        // D(0 .. c1 - 1, c0 .. c1 - 1) = C(:, 0 .. c1 - 1)^H CD(:, c0 .. c1 - 1), panel by panel
        const size_t es = real ? 8 : 16;
        const int pc = (int)std::min<size_t>(m, std::max<size_t>(256, (((size_t)1 << 30) / ((size_t)m * es)) / 256 * 256));
        DevBuf bD;
        bD.alloc((size_t)m * pc * es);
        for (int c0 = 0; c0 < m; c0 += pc) {
            const int c1 = std::min(m, c0 + pc);
            DView A = C, B = CD, D{bD.p, c1, c1 - c0, c1, real};
            A.cols = c1;
            B.p = (char*)CD.p + (size_t)c0 * CD.ld * es;
            B.cols = c1 - c0;
            const int herm = c0 == 0 && c1 == m ? m : 0;  // one panel: only the tiles reaching the upper triangle
            if (real) gemm_f64_emu('t', 'n', c1, c1 - c0, n, 1.0, A, B, 0.0, D, herm);
            else gemm_z_emu('c', 'n', c1, c1 - c0, n, 1.0, A, B, 0.0, D, herm);
            for (int k0 = 0; k0 < nv; k0 += kVBatch) {
                const int nk = std::min(kVBatch, nv - k0);
                VList L{};
                for (int k = 0; k < nk; ++k) {
                    L.colptr[k] = V[k0 + k]->d_colptr.as<int>();
                    L.rowind[k] = V[k0 + k]->d_rowind.as<int>();
                    L.val[k] = V[k0 + k]->d_val.as<double>();
                }
                const dim3 grid((m + kAdjThreads / 32 - 1) / (kAdjThreads / 32), nk);
                double* p = part.as<double>() + (size_t)k0 * m;
                if (real)
                    adjoint_gather_kernel<true><<<grid, kAdjThreads, 0, st>>>(m, c0, c1, D.as<double>(), D.ld, L, c0 == 0, p);
                else
                    adjoint_gather_kernel<false><<<grid, kAdjThreads, 0, st>>>(m, c0, c1, D.as<double>(), D.ld, L, c0 == 0, p);
                OMM_KCHECK();
            }
        }
    } else {
        // the kernel's static shared memory comes on top of the column: opt in for every size
        OMM_CK(cudaFuncSetAttribute(real ? adjoint_sddmm_kernel<true> : adjoint_sddmm_kernel<false>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        for (int k = 0; k < nv; ++k) {
            auto kernel = real ? adjoint_sddmm_kernel<true> : adjoint_sddmm_kernel<false>;
            kernel<<<m, kAdjThreads, smem, st>>>(n, (const double*)C.p, C.ld, (const double*)CD.p, CD.ld,
                                                 V[k]->d_colptr.as<int>(), V[k]->d_rowind.as<int>(),
                                                 V[k]->d_val.as<double>(), part.as<double>() + (size_t)k * m);
            OMM_KCHECK();
        }
    }
    sum_partials<<<nv, 256, 0, st>>>(part.as<double>(), m, sums);
    OMM_KCHECK();
    OMM_CK(cudaMemcpyAsync(grad, sums, (size_t)nv * sizeof(double), cudaMemcpyDeviceToHost, st));
    sync();
}

}  // namespace ommgpu

using namespace ommgpu;

extern "C" {

int omm_gpu_functional_grad(int m, int n, const msw_matrix* H, const msw_matrix* S, const msw_matrix* C,
                            msw_matrix* G, double* omega) {
    try {
        if (!H || !C || !G || !omega) fail(OMM_ERR_ARG, "functional_grad: null argument");
        bool real = C->is_real;
        if (C->dim1 != n || C->dim2 != m || G->dim1 != n || G->dim2 != m || H->dim1 != m || H->dim2 != m)
            fail(OMM_ERR_ARG, "functional_grad: dimensions do not match");
        if (S && (S->dim1 != m || S->dim2 != m)) fail(OMM_ERR_ARG, "functional_grad: S has wrong dimensions");
        Staged sc, sg;
        stage_in(C, sc, true);
        stage_in(G, sg, false);
        // X = [HC; SC] and W = [HW; SW] = X C^H stacked (as omm's step does), so that the residues of C
        // and the columns of C are read once for both halves, and G = [4I - 2SW, -2HW] X is one product
        DevBuf bX, bW, bL;
        DView X = make_view(bX, 2 * n, m, real), W = make_view(bW, 2 * n, n, real), L = make_view(bL, n, 2 * n, real);
        const size_t es = real ? 8 : 16;
        auto half = [&](const DView& v, int h) {
            DView o = v;
            o.rows = n;
            o.p = (char*)v.p + (size_t)h * n * es;
            return o;
        };
        DView HC = half(X, 0), SC = half(X, 1), HW = half(W, 0), SW = half(W, 1);
        if (S && !H->dense() && !S->dense() && same_pattern(H, S)) {
            spmm_dense_csc(sc.v, H, HC, ONE, ZERO, S, &SC);
        } else {
            apply(sc.v, H, HC, m);
            if (S) apply(sc.v, S, SC, m);
            else copy_into(sc.v, SC);
        }
        gemm('n', 'c', 2 * n, n, m, ONE, X, sc.v, ZERO, W);
        double trh[2], trhs[2];
        r_trace(HW, trh);
        r_dot(HW, SW, trhs);
        *omega = 2.0 * trh[0] - trhs[0];  // coeff(0), omm_ops.F90:213
        k_calcG_left(SW, HW, L);
        gemm('n', 'n', n, m, 2 * n, ONE, L, X, ZERO, sg.v);
        stage_out(G, sg);
        sync();
    } catch (const Error& e) {
        set_last_error(e.msg);
        return e.code;
    }
    set_last_error("");
    return OMM_OK;
}

int omm_gpu_energy_adjoint(int m, int n, const msw_matrix* S, const msw_matrix* C, int nv, const msw_matrix* const* V,
                           double* grad) {
    try {
        if (!C || (nv > 0 && (!V || !grad))) fail(OMM_ERR_ARG, "energy_adjoint: null argument");
        if (C->dim1 != n || C->dim2 != m) fail(OMM_ERR_ARG, "energy_adjoint: C must be n x m");
        bool real = C->is_real;
        Staged sc;
        stage_in(C, sc, true);
        for (int k = 0; k < nv; ++k)
            if (!V[k] || V[k]->dim1 != m || V[k]->dim2 != m || V[k]->is_real != real)
                fail(OMM_ERR_ARG, "energy_adjoint: V_k must be m x m with the type of C");
        DevBuf bSC, bSW, bQ, bCD;
        DView SC = make_view(bSC, n, m, real), SW = make_view(bSW, n, n, real);
        DView Q = make_view(bQ, n, n, real), CD = make_view(bCD, n, m, real);
        if (S) apply(sc.v, S, SC, m);
        else copy_into(sc.v, SC);
        gemm('n', 'c', n, n, m, ONE, SC, sc.v, ZERO, SW);   // S_W = C S C^H
        double two[2] = {2.0, 0.0};
        k_set(Q, 'a', ZERO, two);
        k_axpby(SW, 'n', Q, MONE, ONE);                     // Q = 2I - S_W
        gemm('n', 'n', n, m, n, ONE, Q, sc.v, ZERO, CD);    // CD = Q C
        std::vector<const msw_matrix*> sparse;
        std::vector<int> at;
        for (int k = 0; k < nv; ++k) {
            const msw_matrix* Vk = V[k];
            if (Vk->dense()) {
                // dense V: tr(Q C V C^H) through two GEMMs
                DevBuf bCV, bW;
                DView CV = make_view(bCV, n, m, real), W = make_view(bW, n, n, real);
                Staged sv;
                stage_in(Vk, sv);
                gemm('n', 'n', n, m, m, ONE, sc.v, sv.v, ZERO, CV);
                gemm('n', 'c', n, n, m, ONE, CV, sc.v, ZERO, W);
                double t[2];
                r_dot(Q, W, t);
                grad[k] = t[0];
            } else {
                sparse.push_back(Vk);
                at.push_back(k);
            }
        }
        if (!sparse.empty()) {
            std::vector<double> g(sparse.size());
            adjoint_sparse(sc.v, CD, sparse, g.data());
            for (size_t i = 0; i < at.size(); ++i) grad[at[i]] = g[i];
        }
        sync();
    } catch (const Error& e) {
        set_last_error(e.msg);
        return e.code;
    }
    set_last_error("");
    return OMM_OK;
}

}  // extern "C"
