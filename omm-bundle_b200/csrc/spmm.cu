// Dense x CSC products (pspBLAS psp_gemspm local update, pspMspm_nn.F90:191-198;
// MatrixSwitch serial loop MatrixSwitch_mm_multiply.F90:263-327):
//     C(:, j) = beta*C(:, j) + alpha * sum_{l in column j of B} B_l * A(:, row_l)
// A is n x K column-major, so A(:, row) is a contiguous n-vector: every kernel
// here reads whole contiguous column segments of A (coalesced) and writes
// contiguous column segments of C.
//
// Two kernels:
//  * gather  : one CTA per (row chunk, output column); generic CSC.
//  * cgu     : "column-group union", on the FP64 tensor cores (complex ones as
//              two value sets).  Output columns are cut into groups of G
//              consecutive columns; a group's nonzeros live in the union U_g
//              of their row indices, and the group is the dense product
//              A(:, U_g) * B_g with B_g the |U_g| x G block of B (zero filled).
//              For the block-sparse H and S of atom-centred bases (24 x 24
//              atom blocks, all columns of an atom share one pattern) the
//              union adds no fill at G = block size, and the product is a
//              tiled dense GEMM with K = |U_g|.  A second value array
//              with the same pattern (S beside H) is multiplied in the same
//              pass, so A is read once for both.
// The plan (groups, union rows, dense blocks) is built once per matrix on the
// host and kept on the device.
#include "internal.h"

#include <algorithm>
#include <atomic>
#include <cstring>
#include <deque>
#include <map>
#include <mutex>
#include <numeric>

namespace ommgpu {

struct SpmmPlan {
    int G = 0;          // group width
    int ngroups = 0;
    double efficiency = 0.0;  // nnz / sum(|U_g| * G)
    bool cgu = false;
    bool full = false;  // no zero cell: every column of a group holds each of its union's rows once
    std::vector<int> h_gptr;    // ngroups+1 offsets into union rows
    std::vector<int> h_urows;   // union rows
    int maxK = 0;               // the largest union
    bool too_long = false;      // column groups that fill_blocks_kernel cannot form: maxK over kMaxUnion
    DevBuf gptr, urows;
    DevBuf bvals;               // sum(|U_g|*G) values, row-major per group (k, c)
    const msw_matrix* owner = nullptr;
    DevBuf bvals32;             // FP32 copy of bvals for the reduced-precision solver stages
};

namespace {

constexpr int kGatherThreads = 128;

__device__ inline zdbl zfma(zdbl a, zdbl b, zdbl c) {  // a*b + c
    return {fma(a.x, b.x, fma(-a.y, b.y, c.x)), fma(a.x, b.y, fma(a.y, b.x, c.y))};
}

template <typename T> struct Ar;
template <> struct Ar<double> {
    __device__ static double fmaa(double a, double b, double c) { return fma(a, b, c); }
    __device__ static double mulz(zdbl s, double v) { return s.x * v; }
    __device__ static double add(double a, double b) { return a + b; }
    __device__ static double zero() { return 0.0; }
};
template <> struct Ar<zdbl> {
    __device__ static zdbl fmaa(zdbl a, zdbl b, zdbl c) { return zfma(a, b, c); }
    __device__ static zdbl mulz(zdbl s, zdbl v) { return {s.x * v.x - s.y * v.y, s.x * v.y + s.y * v.x}; }
    __device__ static zdbl add(zdbl a, zdbl b) { return {a.x + b.x, a.y + b.y}; }
    __device__ static zdbl zero() { return {0.0, 0.0}; }
};

// C(r, j) = beta*C(r,j) + alpha*sum_l val_l*A(r, row_l); blockIdx.y = column j.  With only_if, nothing
// unless that flag is set.
// R rows per thread, as many as leave the last row block fullest; the column segments of four nonzeros are
// fetched before the first is used (one at a time, with four rows per thread whatever n: 2,501 x 2,501
// complex of 2 %, n = 333, 48 us; now 39).
template <typename T, int R>
__global__ void __launch_bounds__(kGatherThreads) gather_kernel(int n, const T* __restrict__ A, int lda,
                                                                  const int* __restrict__ colptr,
                                                                  const int* __restrict__ rowind,
                                                                  const T* __restrict__ val, T* __restrict__ C,
                                                                  int ldc, zdbl alpha, zdbl beta, int beta_zero,
                                                                  const int* __restrict__ only_if) {
    if (only_if && *only_if == 0) return;
    constexpr int U = 4;
    int j = blockIdx.y;
    int r0 = blockIdx.x * (kGatherThreads * R) + threadIdx.x;
    int s = colptr[j], e = colptr[j + 1];
    T acc[R];
#pragma unroll
    for (int q = 0; q < R; ++q) acc[q] = Ar<T>::zero();
    __shared__ int s_row[kGatherThreads];
    __shared__ T s_val[kGatherThreads];
    for (int base = s; base < e; base += kGatherThreads) {
        int cnt = min(kGatherThreads, e - base);
        __syncthreads();
        if (threadIdx.x < cnt) {
            s_row[threadIdx.x] = rowind[base + threadIdx.x];
            s_val[threadIdx.x] = val[base + threadIdx.x];
        }
        __syncthreads();
        int l = 0;
        for (; l + U <= cnt; l += U) {
            T a[U][R];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const T* col = A + (size_t)s_row[l + u] * lda;
#pragma unroll
                for (int q = 0; q < R; ++q) {
                    const int r = r0 + q * kGatherThreads;
                    if (r < n) a[u][q] = col[r];
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const T v = s_val[l + u];
#pragma unroll
                for (int q = 0; q < R; ++q)
                    if (r0 + q * kGatherThreads < n) acc[q] = Ar<T>::fmaa(a[u][q], v, acc[q]);
            }
        }
        for (; l < cnt; ++l) {
            const T* col = A + (size_t)s_row[l] * lda;
            const T v = s_val[l];
#pragma unroll
            for (int q = 0; q < R; ++q) {
                const int r = r0 + q * kGatherThreads;
                if (r < n) acc[q] = Ar<T>::fmaa(col[r], v, acc[q]);
            }
        }
    }
#pragma unroll
    for (int q = 0; q < R; ++q) {
        int r = r0 + q * kGatherThreads;
        if (r < n) {
            T* c = C + r + (size_t)j * ldc;
            T out = Ar<T>::mulz(alpha, acc[q]);
            if (!beta_zero) out = Ar<T>::add(Ar<T>::mulz(beta, *c), out);
            *c = out;
        }
    }
}

// ---- FP64 column-group kernel on the FP64 tensor cores (mma.sync m8n8k4 f64; tcgen05 has no
// FP64 kind).  Per CTA 32 MT rows of A (4 warps x 8 MT) x one column group (G = 8..32 columns, NM
// value sets).  K (the group's union rows) runs in 8-row chunks through a ring of four stages: the
// chunk's column segments of A and rows of B come by cp.async (16 bytes where the source allows),
// three chunks ahead of the one being multiplied, one barrier per chunk.  Per 4-k step a warp issues
// MT (row tiles) x G/8 (column tiles) x NM DMMAs; the A fragments serve both value sets.
// Fragment layouts (m8n8k4, f64): A(r, k) at lane 4r + k, B(k, c) at lane 4c + k,
// D(r, 2q + i) at lane 4r + q, element i.
// The rows of both shared tiles are padded to 4 (mod 16) doubles -- or 12, its mirror -- so that the
// 16 lanes of a half-warp's fragment load (4 rows x 4 k) fall in 32 distinct banks.  With the padding
// of 8 doubles used before, every fragment load took two passes and the L1 path (85 % busy)
// held the DMMA pipe at 64 %.
// lattice_8x8x8 (n = 1,536): H alone 1.30 -> 1.10 ms with that, 0.98 with the copies' addresses formed once
// and five CTAs per SM (30.6 TFLOP/s; the gathers then move about 6 TB/s from L2), H and S fused
// 2.21 -> 1.82 ms (32.8 TFLOP/s, near cuBLAS DGEMM's 36).  Within 3 %: three or five stages, 16-row chunks in
// two or three stages.
//
// Complex matrices (CPLX) take the same kernel: A, interleaved, is a real matrix of 2n rows; B_re
// and B_im are the two value sets; and with P = A [B_re | B_im], Re C(r, c) = P(2r, c) - P(2r+1, G+c),
// Im C(r, c) = P(2r, G+c) + P(2r+1, c): one lane exchange in the epilogue.
__device__ __forceinline__ void cp_async8(uint32_t dst, const double* src, int bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const double* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(a), "d"(b));
}

constexpr int kDmmaBK = 8, kDmmaStages = 4;
template <int G, int NM, int MT>
constexpr int dmma_stage() {  // doubles of one stage
    return kDmmaBK * ((32 * MT + 4) + NM * (G + 4));
}

struct DmmaArgs {
    int n, N;  // rows of A and C in doubles (2 x the matrix rows for complex matrices), columns
    const double* A;
    long long lda;  // doubles between A's columns
    const int *gptr, *urows;
    const double *B0, *B1;  // value sets (B1 unused for complex ones: B0 holds re, im pairs)
    double *C0, *C1;
    long long rs, cs, cs1;  // strides of C in doubles: row (of the complex matrix), column of C0 and of C1
    double alpha, alpha_im, beta, beta_im;
    int beta_zero;
    int stage_k;  // the group's union rows are staged in shared memory once (else read from global)
    int vec;      // A's column segments are 16-byte aligned
};

// CTAs per SM the registers are held to (0: no bound), from groups of 24 columns.  One value set, 128 rows: five
// CTAs 978 us, four 1,020; 64 rows: eight 992, six 1,076; two value sets, 64 rows: five 1,820, four 1,936; 128 rows:
// three of 154 registers 1,822, four of 128 1,927.  With groups of 32 the first bound spills 40 bytes (6 x 6 x 6
// atoms, 1,536 rows: 783 us; the kernel without the bound and the copies' fixed addresses took 894).
constexpr int dmma_ctas(int nm, int mt, bool cplx) {
    return cplx ? 0 : nm == 1 ? (mt == 4 ? 5 : mt == 2 ? 8 : 0) : (mt == 2 ? 5 : 0);
}
template <int G, int NM, int MT, bool CPLX>
__global__ void __launch_bounds__(128, dmma_ctas(NM, MT, CPLX)) cgu_dmma_kernel(const __grid_constant__ DmmaArgs p) {
    static_assert(MT <= 4, "the copies cover at most 128 rows");
    constexpr int BM = 32 * MT, BK = kDmmaBK, AS = BM + 4, GS = G + 4, NT = G / 8, ST = kDmmaStages;
    constexpr int STAGE = dmma_stage<G, NM, MT>();
    extern __shared__ __align__(16) double dsm[];  // [ST] stages: A [BK][AS], B [NM][BK][GS]
    int* s_ur = (int*)(dsm + ST * STAGE);          // [K] when stage_k
    const int g = blockIdx.y, r0 = blockIdx.x * BM;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int kb = p.gptr[g], K = p.gptr[g + 1] - kb;
    if (p.stage_k) {
        for (int i = threadIdx.x; i < K; i += 128) s_ur[i] = p.urows[kb + i];
        __syncthreads();
    }
    const int* ur = p.stage_k ? s_ur : p.urows + kb;

    double acc[NM][MT][NT][2];
#pragma unroll
    for (int s = 0; s < NM; ++s)
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) acc[s][mt][nt][0] = acc[s][mt][nt][1] = 0.0;

    // A thread's copies of a chunk: places and bytes are formed once, the rows' column comes from the union.
    // Of A, with 16-byte copies, two rows (place mm) of the k kk0, kk0 + KS, ...; with 8-byte ones one row.
    // Of B, a vector per turn of the value sets' contiguous chunk (complex: an element, re and im apart).
    const int nk = (K + BK - 1) / BK, nfull = K / BK;
    constexpr int VR = BM / 2, KS = 128 / VR, NV = BK / KS;                       // 16-byte copies
    constexpr int KS1 = BM >= 128 ? 1 : 128 / BM, NV1 = BK * BM / 128;            // 8-byte copies
    const int kk0 = p.vec ? (int)threadIdx.x / VR : (int)threadIdx.x / BM;
    const int mm = p.vec ? 2 * ((int)threadIdx.x % VR) : (int)threadIdx.x % BM;
    const int abytes = 8 * max(0, min(p.vec ? 2 : 1, p.n - (r0 + mm)));
    const double* acol = abytes ? p.A + r0 + mm : p.A;
    const long long alda = abytes ? p.lda : 0;
    const uint32_t ad = (uint32_t)__cvta_generic_to_shared(dsm + kk0 * AS + mm);
    constexpr int BV = CPLX ? 2 * BK * G : BK * G / 2, NB = (BV + 127) / 128;     // copies of B's chunk (per set)
    uint32_t bd[NB];
    int bk[NB];
#pragma unroll
    for (int u = 0; u < NB; ++u) {
        const int e = threadIdx.x + 128 * u;
        const int kk = CPLX ? e / (2 * G) : e / (G / 2), c = CPLX ? e % (2 * G) / 2 : 2 * (e % (G / 2));
        bk[u] = e < BV ? kk : 1 << 30;
        bd[u] = (uint32_t)__cvta_generic_to_shared(dsm + BK * AS + ((CPLX ? (e & 1) * BK : 0) + kk) * GS + c);
    }
    const double* bsrc[NM] = {};
    bsrc[0] = p.B0 + (size_t)kb * G * (CPLX ? 2 : 1) + (CPLX ? 1 : 2) * threadIdx.x;
    if constexpr (NM == 2 && !CPLX) bsrc[NM - 1] = p.B1 + (size_t)kb * G + 2 * threadIdx.x;
    auto load = [&](int t, uint32_t off) {
        const int k0 = t * BK;
        const bool full = t < nfull;
        if (p.vec) {
#pragma unroll
            for (int u = 0; u < NV; ++u) {
                const int k = k0 + kk0 + KS * u;
                const bool in = full || k < K;
                cp_async16(ad + off + u * KS * AS * 8, acol + (in ? ur[k] * alda : 0), in ? abytes : 0);
            }
        } else {
#pragma unroll
            for (int u = 0; u < NV1; ++u) {
                const int kk = BM >= 128 ? u : kk0 + KS1 * u, k = k0 + kk;
                const bool in = full || k < K;
                cp_async8(ad + off + (BM >= 128 ? u : u * KS1) * AS * 8, acol + (in ? ur[k] * alda : 0), in ? abytes : 0);
            }
        }
#pragma unroll
        for (int u = 0; u < NB; ++u) {
            if (NB * 128 != BV && bk[u] == 1 << 30) continue;  // no copy of this thread
            const bool in = full || k0 + bk[u] < K;
            if constexpr (CPLX) {
                cp_async8(bd[u] + off, in ? bsrc[0] + 128 * u : p.B0, in ? 8 : 0);
            } else {
#pragma unroll
                for (int s = 0; s < NM; ++s)
                    cp_async16(bd[u] + off + s * BK * GS * 8, in ? bsrc[s] + 256 * u : p.B0, in ? 16 : 0);
            }
        }
#pragma unroll
        for (int s = 0; s < (CPLX ? 1 : NM); ++s) bsrc[s] += BK * G * (CPLX ? 2 : 1);
    };

    const double* fa = dsm + (lane & 3) * AS + warp * 8 * MT + (lane >> 2);
    const double* fb = dsm + BK * AS + (lane & 3) * GS + (lane >> 2);
    auto multiply = [&](int stage) {
#pragma unroll
        for (int k4 = 0; k4 < BK; k4 += 4) {
            double af[MT];
#pragma unroll
            for (int mt = 0; mt < MT; ++mt) af[mt] = fa[stage * STAGE + k4 * AS + mt * 8];
#pragma unroll
            for (int s = 0; s < NM; ++s)
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) {
                    const double bf = fb[stage * STAGE + (s * BK + k4) * GS + nt * 8];
#pragma unroll
                    for (int mt = 0; mt < MT; ++mt) dmma(acc[s][mt][nt], af[mt], bf);
                }
        }
    };
#pragma unroll
    for (int t = 0; t < ST - 1; ++t) {
        if (t < nk) load(t, t * STAGE * 8);
        cp_async_commit();
    }
    for (int t0 = 0; t0 < nk; t0 += ST) {
#pragma unroll
        for (int s = 0; s < ST; ++s) {
            const int t = t0 + s;
            if (t < nk) {
                cp_async_wait<ST - 2>();  // chunk t has landed (this thread's part)
                __syncthreads();          // everyone's part, and the slot of chunk t - 1 is free
                if (t + ST - 1 < nk) load(t + ST - 1, (s + ST - 1) % ST * STAGE * 8);
                cp_async_commit();
                multiply(s);
            }
        }
    }
    cp_async_wait<0>();
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
        const int r = r0 + warp * 8 * MT + mt * 8 + (lane >> 2);
        if constexpr (CPLX) {
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    // lane's row 2r' (+1) holds A_re (A_im) times B_re in set 0 and B_im in set 1; the
                    // row of the other parity is four lanes away
                    const double re = acc[0][mt][nt][i], im = acc[1][mt][nt][i];
                    const double ore = __shfl_xor_sync(0xffffffffu, re, 4), oim = __shfl_xor_sync(0xffffffffu, im, 4);
                    const bool odd = (lane >> 2) & 1;
                    const double zr = odd ? ore - im : re - oim;  // Re C = P(2r', c) - P(2r'+1, G+c)
                    const double zi = odd ? oim + re : im + ore;  // Im C = P(2r', G+c) + P(2r'+1, c)
                    const int col = g * G + nt * 8 + (lane & 3) * 2 + i;
                    const bool in = r < p.n && col < p.N;  // the same for both lanes of a row (n is even)
                    // the even lane writes the real part, the odd one the imaginary part
                    double out = odd ? p.alpha * zi + p.alpha_im * zr : p.alpha * zr - p.alpha_im * zi;
                    double* c = p.C0 + (size_t)(r >> 1) * p.rs + (size_t)col * p.cs;
                    if (in && !p.beta_zero) {
                        const double cr = c[0], ci = c[1];
                        out += odd ? p.beta * ci + p.beta_im * cr : p.beta * cr - p.beta_im * ci;
                    }
                    __syncwarp();  // both parts are read before either is written
                    if (in) c[odd ? 1 : 0] = out;
                }
        } else {
            if (r >= p.n) continue;
#pragma unroll
            for (int s = 0; s < NM; ++s)
#pragma unroll
                for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const int col = g * G + nt * 8 + (lane & 3) * 2 + i;
                        if (col >= p.N) continue;
                        double* c = (s == 0 ? p.C0 : p.C1) + (size_t)r * p.rs + (size_t)col * (s == 0 ? p.cs : p.cs1);
                        double out = p.alpha * acc[s][mt][nt][i];
                        if (!p.beta_zero) out += p.beta * *c;
                        *c = out;
                    }
        }
    }
}

template <int G, int NM, int MT, bool CPLX>
void launch_cgu_dmma_t(const DmmaArgs& a, int ngroups, int extra) {
    const int SM = kDmmaStages * dmma_stage<G, NM, MT>() * (int)sizeof(double) + extra;
    static int attr = 0;
    if (SM > attr) {
        OMM_CK(cudaFuncSetAttribute(cgu_dmma_kernel<G, NM, MT, CPLX>, cudaFuncAttributeMaxDynamicSharedMemorySize, SM));
        attr = SM;
    }
    dim3 grid((a.n + 32 * MT - 1) / (32 * MT), ngroups);
    cgu_dmma_kernel<G, NM, MT, CPLX><<<grid, 128, SM, rt().stream>>>(a);
}
template <int G, int NM, bool CPLX>
void launch_cgu_dmma_m(const DmmaArgs& a, int ngroups, int extra, int mt) {
    if (mt == 4) launch_cgu_dmma_t<G, NM, 4, CPLX>(a, ngroups, extra);
    else if (mt == 2) launch_cgu_dmma_t<G, NM, 2, CPLX>(a, ngroups, extra);
    else launch_cgu_dmma_t<G, NM, 1, CPLX>(a, ngroups, extra);
}
template <int G>
void launch_cgu_dmma_g(const DmmaArgs& a, int ngroups, int extra, int mt, bool two, bool cplx) {
    if (cplx) launch_cgu_dmma_m<G, 2, true>(a, ngroups, extra, mt);
    else if (two) launch_cgu_dmma_m<G, 2, false>(a, ngroups, extra, mt);
    else launch_cgu_dmma_m<G, 1, false>(a, ngroups, extra, mt);
}

// Rows of A per CTA: 128 (MT = 4) read each B row once per 128 rows and have the most DMMAs per
// fragment load; 64 and 32 pay where they leave less of the last row block empty, or where the
// grid of 128-row blocks would not give every SM its CTAs (all at the same k order, so the
// results are the same bits).
int dmma_row_tiles(int n, int ngroups) {
    int best = 4;
    double cost = 0.0;
    for (int mt : {4, 2, 1}) {
        const long long blocks = (long long)((n + 32 * mt - 1) / (32 * mt)) * ngroups;
        const double waves = std::ceil((double)blocks / 148.0);
        const double c = waves * mt * (mt == 4 ? 1.0 : mt == 2 ? 1.01 : 1.15);
        if (mt == 4 || c < cost) {
            best = mt;
            cost = c;
        }
    }
    return best;
}

// C (+ C2 for the second value set) = alpha A B + beta C; with trans, C is the transpose of the
// product's layout: element (r, j) at C[j + r ldc]
void launch_cgu_dmma(const DView& A, const SpmmPlan& P, const SpmmPlan* P2, DView& C, DView* C2, const double al[2],
                     const double be[2], int bz, int N, bool trans) {
    const bool cplx = !A.is_real;
    const int w = cplx ? 2 : 1;
    DmmaArgs a{};
    a.n = A.rows * w;
    a.N = N;
    a.A = A.as<double>();
    a.lda = (long long)A.ld * w;
    a.gptr = P.gptr.as<int>();
    a.urows = P.urows.as<int>();
    a.B0 = P.bvals.as<double>();
    a.B1 = P2 ? P2->bvals.as<double>() : nullptr;
    a.C0 = C.as<double>();
    a.C1 = P2 ? C2->as<double>() : nullptr;
    a.rs = trans ? (long long)C.ld * w : w;
    a.cs = trans ? w : (long long)C.ld * w;
    a.cs1 = P2 ? (trans ? w : (long long)C2->ld * w) : 0;
    a.alpha = al[0];
    a.alpha_im = cplx ? al[1] : 0.0;
    a.beta = be[0];
    a.beta_im = cplx ? be[1] : 0.0;
    a.beta_zero = bz;
    a.stage_k = (P.maxK > 0 && P.maxK <= 4096) ? 1 : 0;  // at most 16 KB of indices beside the ring
    a.vec = (a.lda % 2 == 0 && (reinterpret_cast<uintptr_t>(a.A) & 15) == 0) ? 1 : 0;
    const int extra = a.stage_k ? (P.maxK * (int)sizeof(int) + 15) / 16 * 16 : 0;
    const int mt = dmma_row_tiles(a.n, P.ngroups);
    ktime_begin();
    switch (P.G) {
        case 8: launch_cgu_dmma_g<8>(a, P.ngroups, extra, mt, P2 != nullptr, cplx); break;
        case 16: launch_cgu_dmma_g<16>(a, P.ngroups, extra, mt, P2 != nullptr, cplx); break;
        case 24: launch_cgu_dmma_g<24>(a, P.ngroups, extra, mt, P2 != nullptr, cplx); break;
        default: launch_cgu_dmma_g<32>(a, P.ngroups, extra, mt, P2 != nullptr, cplx); break;
    }
    OMM_KCHECK();
    // FP64 flops of the dense group blocks (= 2 nnz n per product for atom-block patterns)
    ktime_end("cgu_dmma_kernel", 2.0 * a.n * (double)P.h_urows.size() * P.G * (P2 || cplx ? 2 : 1));
}

// FP32 variant of the column-group kernel for the reduced-precision solver stages:
// A and the group blocks in FP32, FP32 accumulation, FP64 output (C = A*B).
template <int TM, int TN, int NM>
__global__ void __launch_bounds__(64) cgu32_kernel(int n, int N, const float* __restrict__ A, int lda,
                                                   const int* __restrict__ gptr, const int* __restrict__ urows,
                                                   const float* __restrict__ B0, const float* __restrict__ B1,
                                                   double* __restrict__ C0, int ldc0, double* __restrict__ C1,
                                                   int ldc1) {
    constexpr int BM = 16 * TM;
    constexpr int G = 4 * TN;
    constexpr int BK = 8;
    constexpr int A_PER = BK * BM / 64;
    constexpr int B_PER = (BK * G + 63) / 64;
    __shared__ float As[BK][BM];
    __shared__ float Bs[NM][BK][G];
    const int g = blockIdx.y;
    const int r0 = blockIdx.x * BM;
    const int tid = threadIdx.x;
    const int tm = tid & 15, tn = tid >> 4;
    const int k_begin = gptr[g], K = gptr[g + 1] - k_begin;
    const float* Bg[2] = {B0 + (size_t)k_begin * G, (NM == 2) ? B1 + (size_t)k_begin * G : nullptr};
    float acc[NM][TM][TN];
#pragma unroll
    for (int s = 0; s < NM; ++s)
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int q = 0; q < TN; ++q) acc[s][i][q] = 0.0f;
    float ra[A_PER];
    float rb[NM][B_PER];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int u = 0; u < A_PER; ++u) {
            int e = tid + 64 * u;
            int kk = e / BM, mm = e % BM;
            int r = r0 + mm;
            ra[u] = 0.0f;
            if (k0 + kk < K && r < n) ra[u] = A[(size_t)__ldg(urows + k_begin + k0 + kk) * lda + r];
        }
#pragma unroll
        for (int s = 0; s < NM; ++s)
#pragma unroll
            for (int u = 0; u < B_PER; ++u) {
                int e = tid + 64 * u;
                rb[s][u] = 0.0f;
                if (e < BK * G && k0 + e / G < K) rb[s][u] = Bg[s][(size_t)k0 * G + e];
            }
    };
    auto stash = [&]() {
#pragma unroll
        for (int u = 0; u < A_PER; ++u) {
            int e = tid + 64 * u;
            As[e / BM][e % BM] = ra[u];
        }
#pragma unroll
        for (int s = 0; s < NM; ++s)
#pragma unroll
            for (int u = 0; u < B_PER; ++u) {
                int e = tid + 64 * u;
                if (e < BK * G) Bs[s][e / G][e % G] = rb[s][u];
            }
    };
    const int nk = (K + BK - 1) / BK;
    if (nk > 0) {
        fetch(0);
        stash();
        __syncthreads();
    }
    for (int t = 0; t < nk; ++t) {
        if (t + 1 < nk) fetch((t + 1) * BK);
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            float a[TM];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = As[kk][tm + 16 * i];
#pragma unroll
            for (int s = 0; s < NM; ++s) {
                float b[TN];
#pragma unroll
                for (int q = 0; q < TN; ++q) b[q] = Bs[s][kk][tn * TN + q];
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int q = 0; q < TN; ++q) acc[s][i][q] = fmaf(a[i], b[q], acc[s][i][q]);
            }
        }
        __syncthreads();
        if (t + 1 < nk) {
            stash();
            __syncthreads();
        }
    }
#pragma unroll
    for (int s = 0; s < NM; ++s) {
        double* Cs = (s == 0) ? C0 : C1;
        int ldc = (s == 0) ? ldc0 : ldc1;
#pragma unroll
        for (int q = 0; q < TN; ++q) {
            int col = g * G + tn * TN + q;
            if (col >= N) continue;
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                int r = r0 + tm + 16 * i;
                if (r < n) Cs[r + (size_t)col * ldc] = (double)acc[s][i][q];
            }
        }
    }
}

// *flag = 1 when a (rows x cols, column stride lda) holds an Inf or NaN
__global__ void nonfinite_kernel(int rows, int cols, const double* __restrict__ a, long long lda, int* flag) {
    bool bad = false;
    for (Walk w(rows, cols); w.e < w.total; w.next()) bad |= !(fabs(a[w.i + (size_t)w.j * lda]) <= 1.7976931348623157e308);
    if (bad) *flag = 1;
}

__global__ void f64_to_f32_kernel(size_t n, const double* __restrict__ a, float* __restrict__ b) {
    for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x)
        b[e] = (float)a[e];
}

// ----------------------------------------------------------------------- plan
struct Candidate {
    int G;
    long long cells;
    std::vector<int> gptr, urows;
};

Candidate build_groups(const msw_matrix* B, int G) {
    Candidate c;
    c.G = G;
    int N = B->dim2;
    int ng = (N + G - 1) / G;
    c.gptr.assign(ng + 1, 0);
    std::vector<int> mark(B->dim1, -1);
    std::vector<int> rows;
    for (int g = 0; g < ng; ++g) {
        rows.clear();
        for (int j = g * G; j < std::min(N, (g + 1) * G); ++j)
            for (int l = B->h_colptr[j]; l < B->h_colptr[j + 1]; ++l) {
                int r = B->h_rowind[l];
                if (mark[r] != g) { mark[r] = g; rows.push_back(r); }
            }
        std::sort(rows.begin(), rows.end());
        c.urows.insert(c.urows.end(), rows.begin(), rows.end());
        c.gptr[g + 1] = (int)c.urows.size();
    }
    c.cells = (long long)c.urows.size() * G;
    return c;
}

// The plan is built once per matrix, but an SCF caller registers a new H every cycle, so the
// group blocks are filled on the device, from B's CSC arrays: one CTA per group, its union rows in shared
// memory, a warp per column whose lanes find each nonzero's row in the (ascending) union by binary
// search and add the value into its block cell (duplicate entries add up, as the reference's
// loops would sum them).
__device__ __forceinline__ void add_to(double* d, const double* v, long long l) { atomicAdd(d, v[l]); }
__device__ __forceinline__ void add_to(zdbl* d, const zdbl* v, long long l) {
    atomicAdd(&d->x, v[l].x);
    atomicAdd(&d->y, v[l].y);
}
constexpr int kMaxUnion = 200 * 1024 / (int)sizeof(int);  // the union rows lie in its shared memory
template <typename T>
__global__ void __launch_bounds__(256) fill_blocks_kernel(int G, int N, const int* __restrict__ gptr,
                                                          const int* __restrict__ urows, const int* __restrict__ colptr,
                                                          const int* __restrict__ rowind, const T* __restrict__ val,
                                                          T* __restrict__ out) {
    extern __shared__ int su[];
    const int g = blockIdx.x, kb = gptr[g], nk = gptr[g + 1] - kb;
    for (int i = threadIdx.x; i < nk; i += blockDim.x) su[i] = urows[kb + i];
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int jj = warp; jj < G; jj += 8) {
        const int j = g * G + jj;
        if (j >= N) break;
        for (int l = colptr[j] + lane; l < colptr[j + 1]; l += 32) {
            const int r = rowind[l];
            int lo = 0, hi = nk - 1;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (su[mid] < r) lo = mid + 1;
                else hi = mid;
            }
            add_to(out + (size_t)(kb + lo) * G + jj, val, l);
        }
    }
}

// the dense blocks of the groups (which finish_plan has put on the device) with B's values
void upload_blocks(const msw_matrix* B, SpmmPlan& P, DevBuf& dst) {
    ensure_csc_device(B);
    const size_t cells = std::max<size_t>(1, P.h_urows.size() * (size_t)P.G);
    const int smem = std::max(1, P.maxK) * (int)sizeof(int);
    if (B->is_real) {
        dst.alloc_zero(cells * sizeof(double));
        if (smem > 48 * 1024)
            OMM_CK(cudaFuncSetAttribute(fill_blocks_kernel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        fill_blocks_kernel<double><<<P.ngroups, 256, smem, rt().stream>>>(
            P.G, B->dim2, P.gptr.as<int>(), P.urows.as<int>(), B->d_colptr.as<int>(), B->d_rowind.as<int>(),
            B->d_val.as<double>(), dst.as<double>());
    } else {
        dst.alloc_zero(cells * sizeof(zdbl));
        if (smem > 48 * 1024)
            OMM_CK(cudaFuncSetAttribute(fill_blocks_kernel<zdbl>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        fill_blocks_kernel<zdbl><<<P.ngroups, 256, smem, rt().stream>>>(
            P.G, B->dim2, P.gptr.as<int>(), P.urows.as<int>(), B->d_colptr.as<int>(), B->d_rowind.as<int>(),
            B->d_val.as<zdbl>(), dst.as<zdbl>());
    }
    OMM_KCHECK();
    OMM_CK(cudaStreamSynchronize(rt().stream));  // the caller may change the plan's host arrays
}

// Column groups of recently planned patterns, by content: a caller that registers a matrix
// with a pattern seen before (H and S of the same basis, or H afresh every SCF cycle) skips the
// search over group widths.  A hit needs equal dimensions, column pointers and row indices.
struct GroupsOfPattern {
    int dim1 = 0, dim2 = 0, nnz = 0;
    HostVec<int> colptr, rowind;
    int G = 0;
    double efficiency = 0.0;
    bool cgu = false, full = false;
    std::vector<int> gptr, urows;
};
std::mutex g_groups_mu;
std::deque<std::shared_ptr<const GroupsOfPattern>> g_groups;  // most recent first
constexpr size_t kGroupsKept = 2;

bool same_ints(const int* a, const int* b, long long n) {
    std::atomic<int> diff{0};
    host_parallel(n, [&](long long i0, long long i1) {
        if (std::memcmp(a + i0, b + i0, (size_t)(i1 - i0) * sizeof(int)) != 0) diff = 1;
    });
    return !diff;
}

std::shared_ptr<const GroupsOfPattern> find_groups(const msw_matrix* B) {
    std::deque<std::shared_ptr<const GroupsOfPattern>> kept;
    {
        std::lock_guard<std::mutex> lk(g_groups_mu);
        kept = g_groups;
    }
    for (auto& e : kept)
        if (e->dim1 == B->dim1 && e->dim2 == B->dim2 && e->nnz == B->nnz &&
            same_ints(e->colptr.data(), B->h_colptr.data(), (long long)B->dim2 + 1) &&
            same_ints(e->rowind.data(), B->h_rowind.data(), B->nnz))
            return e;
    return nullptr;
}

void keep_groups(const msw_matrix* B, const SpmmPlan& P) {
    auto e = std::make_shared<GroupsOfPattern>();
    e->dim1 = B->dim1;
    e->dim2 = B->dim2;
    e->nnz = B->nnz;
    e->colptr = B->h_colptr;
    e->rowind.resize(B->h_rowind.size());
    const int* src = B->h_rowind.data();
    int* dst = e->rowind.data();
    host_parallel((long long)B->h_rowind.size(), [&](long long i0, long long i1) {
        std::memcpy(dst + i0, src + i0, (size_t)(i1 - i0) * sizeof(int));
    });
    e->G = P.G;
    e->efficiency = P.efficiency;
    e->cgu = P.cgu;
    e->full = P.full;
    e->gptr = P.h_gptr;
    e->urows = P.h_urows;
    std::lock_guard<std::mutex> lk(g_groups_mu);
    g_groups.push_front(std::move(e));
    while (g_groups.size() > kGroupsKept) g_groups.pop_back();
}

void finish_plan(const msw_matrix* B, SpmmPlan& P);

// Whether every column of a group holds each row of its union exactly once.  As many nonzeros as cells do not
// say so: duplicate entries (which add up) count several times and can make up for zero cells.
bool no_zero_cell(const msw_matrix* B, const SpmmPlan& P) {
    std::atomic<bool> all{true};
    host_parallel(B->dim2, [&](long long j0, long long j1) {
        std::vector<int> rows;
        for (long long j = j0; j < j1 && all; ++j) {
            const int* u = P.h_urows.data() + P.h_gptr[j / P.G];
            const int nu = P.h_gptr[j / P.G + 1] - P.h_gptr[j / P.G];
            const int* r = B->h_rowind.data() + B->h_colptr[j];
            bool same = B->h_colptr[j + 1] - B->h_colptr[j] == nu;
            if (same && !std::equal(r, r + nu, u)) {  // the same rows in another order, perhaps
                rows.assign(r, r + nu);
                std::sort(rows.begin(), rows.end());
                same = std::equal(rows.begin(), rows.end(), u);
            }
            if (!same) all = false;
        }
    });
    return all;
}

// The matrix's plan, whether its column groups can be formed or not (too_long)
SpmmPlan& any_plan(const msw_matrix* B) {
    msw_matrix* Bm = const_cast<msw_matrix*>(B);
    if (Bm->plan) return *Bm->plan;
    auto P = std::make_shared<SpmmPlan>();
    P->owner = B;
    if (auto hit = find_groups(B)) {
        P->G = hit->G;
        P->ngroups = (int)hit->gptr.size() - 1;
        P->efficiency = hit->efficiency;
        P->cgu = hit->cgu;
        P->full = hit->full;
        P->h_gptr = hit->gptr;
        P->h_urows = hit->urows;
        finish_plan(B, *P);
        Bm->plan = P;
        return *P;
    }
    // choose the widest group width whose fill is within 5 % of the best one
    std::vector<Candidate> cands(4);
    {
        const int widths[4] = {8, 16, 24, 32};
        host_shares(4, [&](int i) { cands[i] = build_groups(B, widths[i]); });
    }
    long long nnz = std::max(1, B->nnz);
    double best = 0.0;
    for (auto& c : cands) best = std::max(best, (double)nnz / std::max<long long>(1, c.cells));
    Candidate* pick = &cands[0];
    for (auto& c : cands) {
        double eff = (double)nnz / std::max<long long>(1, c.cells);
        if (eff >= 0.95 * best) pick = &c;
    }
    P->G = pick->G;
    P->ngroups = (int)pick->gptr.size() - 1;
    P->efficiency = (double)nnz / std::max<long long>(1, pick->cells);
    // the dense-union form pays off when most of its cells are real nonzeros and
    // columns are long enough for the tile loop
    double avg = (double)B->nnz / std::max(1, B->dim2);
    P->cgu = (P->efficiency >= 0.5) && (avg >= 16.0);
    P->h_gptr.swap(pick->gptr);
    P->h_urows.swap(pick->urows);
    P->full = P->cgu && nnz == pick->cells && no_zero_cell(B, *P);
    finish_plan(B, *P);
    keep_groups(B, *P);
    Bm->plan = P;
    return *P;
}

// The plan for the paths that have no other way to a matrix with column groups
SpmmPlan& get_plan(const msw_matrix* B) {
    SpmmPlan& P = any_plan(B);
    if (P.too_long) fail(OMM_ERR_UNSUPPORTED, "spmm plan: a column group's row union is too long");
    return P;
}

void clear_kept_groups() {
    std::lock_guard<std::mutex> lk(g_groups_mu);
    g_groups.clear();
}

// device copies of the groups and the dense blocks of the values
void finish_plan(const msw_matrix* B, SpmmPlan& Pl) {
    SpmmPlan* P = &Pl;
    P->maxK = 0;
    for (size_t g = 0; g + 1 < P->h_gptr.size(); ++g) P->maxK = std::max(P->maxK, P->h_gptr[g + 1] - P->h_gptr[g]);
    P->too_long = P->cgu && P->maxK > kMaxUnion;
    if (P->cgu && !P->too_long) {
        P->gptr.alloc(P->h_gptr.size() * sizeof(int));
        P->urows.alloc(std::max<size_t>(1, P->h_urows.size()) * sizeof(int));
        OMM_CK(cudaMemcpyAsync(P->gptr.p, P->h_gptr.data(), P->h_gptr.size() * sizeof(int), cudaMemcpyHostToDevice,
                               rt().stream));
        if (!P->h_urows.empty())
            OMM_CK(cudaMemcpyAsync(P->urows.p, P->h_urows.data(), P->h_urows.size() * sizeof(int),
                                   cudaMemcpyHostToDevice, rt().stream));
        upload_blocks(B, *P, P->bvals);
    }
}

// The plan of a matrix with P's pattern.  It is complete (groups on the device too): the matrix may be
// multiplied by itself next.
SpmmPlan& plan_of_pattern(const msw_matrix* B2, const SpmmPlan& P) {
    msw_matrix* Bm = const_cast<msw_matrix*>(B2);
    if (!Bm->plan) {
        auto Q = std::make_shared<SpmmPlan>();
        Q->G = P.G;
        Q->ngroups = P.ngroups;
        Q->efficiency = P.efficiency;
        Q->cgu = P.cgu;
        Q->full = P.full;
        Q->h_gptr = P.h_gptr;
        Q->h_urows = P.h_urows;
        Q->owner = B2;
        finish_plan(B2, *Q);
        Bm->plan = Q;
    }
    return *Bm->plan;
}

}  // namespace

void spmm_plan_cache_clear() { clear_kept_groups(); }

unsigned long long next_pattern_id() {
    static std::atomic<unsigned long long> next{1};
    return next.fetch_add(1);
}

// Comparing two patterns walks nnz row indices (milliseconds at 10^7 nonzeros), and the
// solver asks once per CG step, so results are memoised by the pair of pattern ids.
bool same_pattern(const msw_matrix* A, const msw_matrix* B) {
    if (!A || !B || A->fmt != Fmt::CSC || B->fmt != Fmt::CSC) return false;
    if (A->dim1 != B->dim1 || A->dim2 != B->dim2 || A->nnz != B->nnz || A->is_real != B->is_real) return false;
    if (A == B) return true;
    static std::mutex mu;
    static std::map<std::pair<unsigned long long, unsigned long long>, bool> memo;
    auto key = std::minmax(A->pattern_id, B->pattern_id);
    {
        std::lock_guard<std::mutex> lk(mu);
        auto it = memo.find(key);
        if (it != memo.end()) return it->second;
    }
    const bool eq = A->h_colptr.size() == B->h_colptr.size() && A->h_rowind.size() == B->h_rowind.size() &&
                    same_ints(A->h_colptr.data(), B->h_colptr.data(), (long long)A->h_colptr.size()) &&
                    same_ints(A->h_rowind.data(), B->h_rowind.data(), (long long)A->h_rowind.size());
    std::lock_guard<std::mutex> lk(mu);
    if (memo.size() > 4096) memo.clear();
    memo[key] = eq;
    return eq;
}

static void launch_gather(const DView& A, const msw_matrix* B, DView& C, const double alpha[2], const double beta[2],
                          const int* only_if) {
    ensure_csc_device(B);
    int n = A.rows, N = B->dim2;
    if (n == 0 || N == 0) return;
    zdbl al{alpha[0], alpha[1]}, be{beta[0], beta[1]};
    int bz = (beta[0] == 0.0 && beta[1] == 0.0) ? 1 : 0;
    const int nb = (n + kGatherThreads * 4 - 1) / (kGatherThreads * 4);
    const int R = (n + kGatherThreads * nb - 1) / (kGatherThreads * nb);  // 1 .. 4
    dim3 grid((n + kGatherThreads * R - 1) / (kGatherThreads * R), N);
    auto launch = [&](auto tag, auto kernel) {
        using T = decltype(tag);
        kernel<<<grid, kGatherThreads, 0, rt().stream>>>(n, A.as<T>(), A.ld, B->d_colptr.as<int>(),
                                                         B->d_rowind.as<int>(), B->d_val.as<T>(), C.as<T>(), C.ld, al,
                                                         be, bz, only_if);
    };
    if (A.is_real) launch(double{}, R == 1 ? gather_kernel<double, 1> : R == 2 ? gather_kernel<double, 2>
                                     : R == 3 ? gather_kernel<double, 3> : gather_kernel<double, 4>);
    else launch(zdbl{}, R == 1 ? gather_kernel<zdbl, 1> : R == 2 ? gather_kernel<zdbl, 2>
                         : R == 3 ? gather_kernel<zdbl, 3> : gather_kernel<zdbl, 4>);
    OMM_KCHECK();
}
void spmm_dense_csc_gather(const DView& A, const msw_matrix* B, DView& C, const double alpha[2],
                           const double beta[2]) {
    launch_gather(A, B, C, alpha, beta, nullptr);
}

// Whether a look at 16 of the matrix's 8-column groups, evenly spaced, already rules the column-group
// kernels out: their fill is below half of what a plan needs (a wider group of the same columns is
// emptier still).  Saves a matrix with an irregular pattern the search over group widths, which takes
// the host milliseconds per 10^5 nonzeros; a sample near the limit leaves the decision to the plan.
bool rules_out_groups(const msw_matrix* B) {
    msw_matrix* Bm = const_cast<msw_matrix*>(B);
    if (Bm->plan) return false;
    if (Bm->no_groups < 0) {
        const int ng = B->dim2 / 8, take = std::min(ng, 16);
        long long nnz = 0, cells = 0;
        std::vector<int> seen(B->dim1, -1);
        for (int s = 0; s < take; ++s) {
            const int j = (int)((long long)s * ng / take) * 8;
            for (int l = B->h_colptr[j]; l < B->h_colptr[j + 8]; ++l) {
                int& mark = seen[B->h_rowind[l]];
                cells += mark != s ? 8 : 0;
                mark = s;
            }
            nnz += B->h_colptr[j + 8] - B->h_colptr[j];
        }
        Bm->no_groups = take == 16 && nnz * 4 < cells ? 1 : 0;
    }
    return Bm->no_groups == 1;
}

void spmm_dense_csc(const DView& A, const msw_matrix* B, DView& C, const double alpha[2], const double beta[2],
                    const msw_matrix* B2, DView* C2) {
    if (A.rows == 0 || B->dim2 == 0) return;
    if (rules_out_groups(B)) {
        spmm_dense_csc_gather(A, B, C, alpha, beta);
        if (B2 && C2) spmm_dense_csc(A, B2, *C2, alpha, beta);
        return;
    }
    SpmmPlan& P = get_plan(B);
    bool fuse = B2 && C2 && same_pattern(B, B2);
    if (!P.cgu) {
        spmm_dense_csc_gather(A, B, C, alpha, beta);
        if (B2 && C2) spmm_dense_csc_gather(A, B2, *C2, alpha, beta);
        return;
    }
    SpmmPlan* P2 = nullptr;
    if (fuse) {
        P2 = &plan_of_pattern(B2, P);
        if (P2->G != P.G || P2->h_gptr != P.h_gptr) fuse = false, P2 = nullptr;
    }
    const int bz = (beta[0] == 0.0 && beta[1] == 0.0) ? 1 : 0;
    fuse = fuse && A.is_real;  // a complex matrix's two parts take both value sets of the kernel
    launch_cgu_dmma(A, P, fuse ? P2 : nullptr, C, fuse ? C2 : nullptr, alpha, beta, bz, B->dim2, false);
    if (B2 && C2 && !fuse) spmm_dense_csc(A, B2, *C2, alpha, beta);
}

namespace {
void ensure_f32_values(SpmmPlan& P) {
    if (P.bvals32.p) return;
    size_t cnt = P.bvals.bytes / sizeof(double);
    P.bvals32.alloc(std::max<size_t>(1, cnt) * sizeof(float));
    size_t b = std::min<size_t>((cnt + 255) / 256, 148 * 32);
    f64_to_f32_kernel<<<(int)std::max<size_t>(b, 1), 256, 0, rt().stream>>>(cnt, P.bvals.as<double>(),
                                                                             P.bvals32.as<float>());
    OMM_KCHECK();
}
template <int TM, int TN>
void launch_cgu32(const float* A, int lda, int n, const SpmmPlan& P, const SpmmPlan* P2, DView& C, DView* C2, int N) {
    constexpr int BM = 16 * TM;
    dim3 grid((n + BM - 1) / BM, P.ngroups);
    if (P2)
        cgu32_kernel<TM, TN, 2><<<grid, 64, 0, rt().stream>>>(n, N, A, lda, P.gptr.as<int>(), P.urows.as<int>(),
                                                              P.bvals32.as<float>(), P2->bvals32.as<float>(),
                                                              C.as<double>(), C.ld, C2->as<double>(), C2->ld);
    else
        cgu32_kernel<TM, TN, 1><<<grid, 64, 0, rt().stream>>>(n, N, A, lda, P.gptr.as<int>(), P.urows.as<int>(),
                                                              P.bvals32.as<float>(), nullptr, C.as<double>(), C.ld,
                                                              nullptr, 0);
    OMM_KCHECK();
}
}  // namespace

bool spmm32_available(const msw_matrix* B) { return B && B->fmt == Fmt::CSC && B->is_real && get_plan(B).cgu; }

// C (FP64) = A (FP32, n x K column-major) * B (CSC, FP32 values); fused second matrix when the
// patterns agree (B2 / C2).  Requires a column-group plan (spmm32_available).
void spmm32_dense_csc(const float* A, int lda, int n, const msw_matrix* B, DView& C, const msw_matrix* B2,
                      DView* C2) {
    SpmmPlan& P = get_plan(B);
    if (!P.cgu) fail(OMM_ERR_UNSUPPORTED, "spmm32: matrix has no column-group plan");
    ensure_f32_values(P);
    SpmmPlan* P2 = nullptr;
    if (B2 && C2 && same_pattern(B, B2)) {
        P2 = &plan_of_pattern(B2, P);  // the second value set
        if (P2->G != P.G || P2->h_gptr != P.h_gptr) P2 = nullptr;
        else ensure_f32_values(*P2);
    }
    int N = B->dim2;
    switch (P.G) {
        case 8: launch_cgu32<8, 2>(A, lda, n, P, P2, C, P2 ? C2 : nullptr, N); break;
        case 16: launch_cgu32<8, 4>(A, lda, n, P, P2, C, P2 ? C2 : nullptr, N); break;
        case 24: launch_cgu32<8, 6>(A, lda, n, P, P2, C, P2 ? C2 : nullptr, N); break;
        default: launch_cgu32<8, 8>(A, lda, n, P, P2, C, P2 ? C2 : nullptr, N); break;
    }
    if (B2 && C2 && !P2) spmm32_dense_csc(A, lda, n, B2, *C2, nullptr, nullptr);
}

SpmmPlanView spmm_plan_view(const msw_matrix* B) {
    SpmmPlan& P = get_plan(B);
    SpmmPlanView v;
    v.cgu = P.cgu;
    v.G = P.G;
    v.ngroups = P.ngroups;
    v.gptr = P.h_gptr.data();
    v.urows = P.h_urows.data();
    v.d_gptr = P.gptr.as<int>();
    v.d_bvals = P.bvals.as<double>();
    return v;
}

bool spmm_tc_available(const msw_matrix* B) {
    if (!B || B->fmt != Fmt::CSC || !B->is_real) return false;
    return spmm_tc_plan(B, spmm_plan_view(B)) != nullptr;
}

SpmmInfo spmm_info(const msw_matrix* B) {
    SpmmPlan& P = get_plan(B);
    return SpmmInfo{P.G, P.ngroups, P.efficiency, (long long)P.h_urows.size(), P.cgu};
}

}  // namespace ommgpu

extern "C" int omm_gpu_spmm_plan_info(const msw_matrix* B, int* G, int* ngroups, double* fill, int* column_groups) {
    using namespace ommgpu;
    try {
        if (!B || B->fmt != Fmt::CSC) fail(OMM_ERR_ARG, "spmm_plan_info: B must be a CSC matrix");
        SpmmInfo info = spmm_info(B);
        if (G) *G = info.group_width;
        if (ngroups) *ngroups = info.ngroups;
        if (fill) *fill = info.efficiency;
        if (column_groups) *column_groups = info.cgu ? 1 : 0;
    } catch (const Error& e) {
        set_last_error(e.msg);
        return e.code;
    }
    set_last_error("");
    return OMM_OK;
}

namespace ommgpu {

// psp_gemspm with every op combination (pspMspm.F90:58-120 dispatch to _nn/_nt/_tn/_tt):
// C = alpha*op(A)*op(B) + beta*C.  op(A) != 'n' is materialised with a transpose;
// op(B) != 'n' uses the CSC of B^T (conjugated values for 'c').
void gemspm(char opA, const DView& A, char opB, const msw_matrix* B, DView& C, const double alpha[2],
            const double beta[2]) {
    DevBuf tA;
    DView Aop = A;
    bool trA = !(opA == 'n' || opA == 'N');
    if (trA) {
        Aop.rows = A.cols;
        Aop.cols = A.rows;
        Aop.ld = (A.cols + 1) & ~1;  // even: 16-byte column segments for the column-group kernel
        tA.alloc(std::max<size_t>(1, (size_t)Aop.ld * Aop.cols) * (A.is_real ? 8 : 16));
        Aop.p = tA.p;
        transpose_into(A, opA, Aop);
    }
    const msw_matrix* Bop = B;
    if (!(opB == 'n' || opB == 'N')) {
        Bop = csc_transpose(B);
        if (!B->is_real && (opB == 'c' || opB == 'C')) {
            // conjugated copy of the transpose, kept beside it
            msw_matrix* Bm = const_cast<msw_matrix*>(B);
            if (!Bm->conj_transposed) {
                auto Cj = std::make_shared<msw_matrix>();
                Cj->dim1 = Bop->dim1; Cj->dim2 = Bop->dim2; Cj->is_real = false; Cj->fmt = Fmt::CSC;
                Cj->loc = Loc::Device; Cj->nnz = Bop->nnz;
                Cj->h_colptr = Bop->h_colptr; Cj->h_rowind = Bop->h_rowind; Cj->h_val = Bop->h_val;
                for (int l = 0; l < Cj->nnz; ++l) Cj->h_val[2 * l + 1] = -Cj->h_val[2 * l + 1];
                Bm->conj_transposed = Cj;
            }
            Bop = Bm->conj_transposed.get();
        }
    }
    spmm_dense_csc(Aop, Bop, C, alpha, beta);
}

// psp_gespmm (pspSpmm.F90:61-123): C = alpha*op(A)*op(B) + beta*C with A CSC, evaluated as
// C^T = op(B)^T op(A)^T with the dense x CSC kernels.  op(A)^T is A^T's CSC for 'n' and A itself
// otherwise; where 'c' asks for conj(A), the dense operand is conjugated instead and so is the
// product: conj(conj(X) A) = X conj(A).  The column-group kernel writes the product transposed, in
// place of a second matrix and a transposing add (5 x 5 x 5 atoms of 24 orbitals, 375 columns: 109 us
// with the transposed copy of B and C's read; the gather kernel, which took every pattern before, 500 us).
void gespmm(char opA, const msw_matrix* A, char opB, const DView& B, DView& C, const double alpha[2],
            const double beta[2]) {
    const bool real = B.is_real;
    const int M = C.rows, N = C.cols;
    const bool aN = (opA == 'n' || opA == 'N'), aC = !real && (opA == 'c' || opA == 'C');
    const bool bN = (opB == 'n' || opB == 'N'), bC = !real && (opB == 'c' || opB == 'C');
    const bool conj = aC != bC;  // X = op(B)^T, conjugated once more when op(A) is 'c'
    const size_t es = real ? 8 : 16;
    DevBuf tX, tmp;
    DView X = B;
    if (bN) {
        X.rows = B.cols; X.cols = B.rows;
        X.ld = std::max(2, (B.cols + 1) & ~1);  // even: 16-byte column segments for the column-group kernel
        tX.alloc((size_t)X.ld * std::max(1, X.cols) * es);
        X.p = tX.p;
        transpose_into(B, conj ? 'c' : 't', X);
    } else if (conj) {
        // conj(B) = (B^H)^T: two transposes keep this on existing kernels
        DView Th{nullptr, B.cols, B.rows, std::max(1, B.cols), false};
        tmp.alloc(std::max<size_t>(1, (size_t)B.rows * B.cols) * 16);
        Th.p = tmp.p;
        transpose_into(B, 'c', Th);
        X.ld = std::max(1, B.rows);
        tX.alloc(std::max<size_t>(1, (size_t)X.rows * X.cols) * 16);
        X.p = tX.p;
        transpose_into(Th, 't', X);
    }
    const msw_matrix* Y = aN ? csc_transpose(A) : A;
    if (N == 0 || M == 0) return;
    const double one[2] = {1.0, 0.0}, zero[2] = {0.0, 0.0};
    const SpmmPlan* P = rules_out_groups(Y) ? nullptr : &any_plan(Y);
    if (P && (!P->cgu || P->too_long)) P = nullptr;
    // every cell of the groups' blocks is a nonzero (atom blocks): nothing is multiplied that the sparse
    // product leaves out
    const bool full = P && P->full;
    // the direct form writes C while it reads X, which is B itself for 't': where they share memory (C = op(A)
    // B^T in place) the product goes through Z
    if (full && !aC && !overlap(X, C)) {
        // beta multiplies C even when it is 0 (an Inf or NaN of C stays), as in the last pass of the other routes
        launch_cgu_dmma(X, *P, nullptr, C, nullptr, alpha, beta, 0, M, true);
        return;
    }
    // Z = X * Y  (N x M), then C = alpha*Z^T (or Z^H) + beta*C
    DevBuf tZ, flag;
    DView Z{nullptr, N, M, N, real};
    tZ.alloc((size_t)N * M * es);
    Z.p = tZ.p;
    if (P) {
        launch_cgu_dmma(X, *P, nullptr, Z, nullptr, one, zero, 1, M, false);
        if (!full) {
            // a zero cell times an Inf or NaN of X is a NaN that the sparse product does not have: when X
            // holds any, the gather kernel forms the product again from the nonzeros alone
            flag.alloc_zero(sizeof(int));
            nonfinite_kernel<<<(int)std::min<size_t>(((size_t)X.rows * X.cols + 255) / 256, 148 * 8), 256, 0,
                               rt().stream>>>(X.rows * (real ? 1 : 2), X.cols, X.as<double>(),
                                              (long long)X.ld * (real ? 1 : 2), flag.as<int>());
            OMM_KCHECK();
            launch_gather(X, Y, Z, one, zero, flag.as<int>());
        }
    } else {
        spmm_dense_csc_gather(X, Y, Z, one, zero);
    }
    k_axpby(Z, aC ? 'c' : 't', C, alpha, beta);
}

}  // namespace ommgpu
