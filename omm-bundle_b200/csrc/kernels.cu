// Elementwise, reduction and initialisation kernels of the libOMM CG loop, plus
// the dispatch of the FP64 dense products (gemm()).
//
// All matrices are column-major views (pointer, rows, cols, leading dimension).
// Real matrices are double, complex ones zdbl (interleaved re, im).
#include "internal.h"
#include "line_search.h"

#include <algorithm>
#include <cmath>

namespace ommgpu {

namespace {

constexpr int kThreads = 256;

__host__ __device__ inline zdbl zmul(zdbl a, zdbl b) { return {a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x}; }
__host__ __device__ inline zdbl zadd(zdbl a, zdbl b) { return {a.x + b.x, a.y + b.y}; }
__host__ __device__ inline zdbl zconj(zdbl a) { return {a.x, -a.y}; }

// ---- generic scalar helpers: real matrices use only the .x part of the complex scalars
template <typename T> struct Sc;
template <> struct Sc<double> {
    __device__ static double load(const double* p, size_t i) { return p[i]; }
    __device__ static void store(double* p, size_t i, double v) { p[i] = v; }
    __device__ static double conj(double v) { return v; }
    __device__ static double mul(zdbl a, double v) { return a.x * v; }
    __device__ static double add(double a, double b) { return a + b; }
    __device__ static double from(zdbl a) { return a.x; }
};
template <> struct Sc<zdbl> {
    __device__ static zdbl load(const zdbl* p, size_t i) { return p[i]; }
    __device__ static void store(zdbl* p, size_t i, zdbl v) { p[i] = v; }
    __device__ static zdbl conj(zdbl v) { return zconj(v); }
    __device__ static zdbl mul(zdbl a, zdbl v) { return zmul(a, v); }
    __device__ static zdbl add(zdbl a, zdbl b) { return zadd(a, b); }
    __device__ static zdbl from(zdbl a) { return a; }
};

inline int grid_for(size_t elems, int per_thread = 4) {
    size_t b = (elems + (size_t)kThreads * per_thread - 1) / ((size_t)kThreads * per_thread);
    if (b < 1) b = 1;
    if (b > 148 * 32) b = 148 * 32;
    return (int)b;
}

constexpr int kAhead = 4;  // elements whose loads a thread issues before it uses the first

// C = beta*C + alpha*A  (MatrixSwitch_m_add.F90:95-175: C=beta*C first, then += alpha*op(A)).
// Bound by memory: two reads and a write per element.
template <typename T>
__global__ void axpby_kernel(int rows, int cols, const T* __restrict__ A, int lda, T* __restrict__ C, int ldc,
                             zdbl alpha, zdbl beta, int beta_zero, const double* __restrict__ beta_at,
                             const int* __restrict__ stop) {
    if (stop && *stop) return;
    if (beta_at) beta = zdbl{*beta_at, 0.0};
    Walk w(rows, cols);
    while (w.e < w.total) {
        T a[kAhead], cin[kAhead];
        T* at[kAhead];
        int cnt = 0;
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            at[u] = nullptr;
            if (w.e < w.total) {
                a[u] = A[w.i + (size_t)w.j * lda];
                at[u] = C + w.i + (size_t)w.j * ldc;
                cin[u] = *at[u];
                ++cnt;
                w.next();
            }
        }
#pragma unroll
        for (int u = 0; u < kAhead; ++u)
            if (u < cnt) {
                T c = beta_zero ? T{} : Sc<T>::mul(beta, cin[u]);
                *at[u] = Sc<T>::add(c, Sc<T>::mul(alpha, a[u]));
            }
    }
}

// C = beta*C + alpha*A^T or alpha*A^H: one 32 x 32 tile per block turn, A's tile staged through shared
// memory so that its reads run down its columns.  2049 x 1537 complex: 23 us where the element walk,
// one 32-byte sector per element of A, took 45.
template <typename T>
__global__ void axpby_trans_kernel(int rows, int cols, const T* __restrict__ A, int lda, int conj, T* __restrict__ C,
                                   int ldc, zdbl alpha, zdbl beta, int beta_zero) {
    __shared__ T tile[32][33];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
    const int tr = (rows + 31) / 32, tc = (cols + 31) / 32;
    for (long long t = blockIdx.x; t < (long long)tr * tc; t += gridDim.x) {
        const int r0 = (int)(t % tr) * 32, c0 = (int)(t / tr) * 32;
        T cin[4];
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int yy = ty + 8 * q;
            const int j = c0 + tx, i = r0 + yy;  // A(j, i)
            if (i < rows && j < cols) tile[yy][tx] = A[j + (size_t)i * lda];
            const int ci = r0 + tx, cj = c0 + yy;
            if (ci < rows && cj < cols) cin[q] = C[ci + (size_t)cj * ldc];
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int yy = ty + 8 * q, i = r0 + tx, j = c0 + yy;
            if (i < rows && j < cols) {
                T a = tile[tx][yy];
                if (conj) a = Sc<T>::conj(a);
                T c = beta_zero ? T{} : Sc<T>::mul(beta, cin[q]);
                C[i + (size_t)j * ldc] = Sc<T>::add(c, Sc<T>::mul(alpha, a));
            }
        }
    }
}

template <typename T>
__global__ void scale_kernel(int rows, int cols, T* C, int ldc, zdbl beta) {
    for (Walk w(rows, cols); w.e < w.total; w.next()) {
        T* c = C + w.i + (size_t)w.j * ldc;
        *c = Sc<T>::mul(beta, *c);
    }
}

// m_set (MatrixSwitch_m_set.F90:19-75): lu 0 all, 1 upper (j>=i), 2 lower (j<=i)
template <typename T>
__global__ void set_kernel(int rows, int cols, T* C, int ldc, int lu, zdbl alpha, zdbl beta) {
    for (Walk w(rows, cols); w.e < w.total; w.next()) {
        if (lu == 1 && w.j < w.i) continue;
        if (lu == 2 && w.j > w.i) continue;
        C[w.i + (size_t)w.j * ldc] = Sc<T>::from(w.i == w.j ? beta : alpha);
    }
}

template <typename T>
__global__ void set_element_kernel(T* C, size_t idx, zdbl alpha, zdbl beta) {
    C[idx] = Sc<T>::add(Sc<T>::from(alpha), Sc<T>::mul(beta, C[idx]));
}

// C(j,i) = conj(C(i,j)) for j > i and a real diagonal  (omm_ops.F90:483-487 / :590-594).  One 32 x 32 tile of the
// lower triangle per block, its source tile of the upper triangle staged through shared memory
// so that both the reads and the writes run down columns (coalesced).
template <typename T>
__global__ void fill_lower_kernel(int n, T* C, int ldc) {
    const int bi = blockIdx.x, bj = blockIdx.y;  // destination tile: rows 32*bi.., columns 32*bj..
    if (bi < bj) return;
    __shared__ T tile[32][33];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
    for (int yy = ty; yy < 32; yy += 8) {
        int r = 32 * bj + tx, c = 32 * bi + yy;  // source C(r, c) in the upper triangle
        if (r < n && c < n) tile[yy][tx] = C[r + (size_t)c * ldc];
    }
    __syncthreads();
    for (int yy = ty; yy < 32; yy += 8) {
        int r = 32 * bi + tx, c = 32 * bj + yy;  // destination C(r, c) = conj(C(c, r))
        if (r < n && c < n && r > c) C[r + (size_t)c * ldc] = Sc<T>::conj(tile[tx][yy]);
        if constexpr (sizeof(T) == 16)
            if (r < n && r == c) C[r + (size_t)c * ldc].y = 0.0;  // as herk leaves a Hermitian diagonal
    }
}

// W += x*(Wd^H + Wd) + x^2*Wdd  (omm.F90:499-501, :514-516, :168-170), applied as the
// reference's three m_add calls in order.  One 32 x 32 tile per block turn, Wd's mirror tile staged
// through shared memory (read element by element it cost a 32-byte sector per element).
template <typename T>
__global__ void w_update_kernel(int n, T* W, int ldw, const T* __restrict__ Wd, int ldd, const T* __restrict__ Wdd,
                                int lddd, double x) {
    __shared__ T tile[32][33];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
    const int tiles = (n + 31) / 32;
    zdbl xz{x, 0.0}, x2{x * x, 0.0};
    for (long long t = blockIdx.x; t < (long long)tiles * tiles; t += gridDim.x) {
        const int r0 = (int)(t % tiles) * 32, c0 = (int)(t / tiles) * 32;
        T w[4], d[4], dd[4];
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int yy = ty + 8 * q;
            if (c0 + tx < n && r0 + yy < n) tile[yy][tx] = Wd[c0 + tx + (size_t)(r0 + yy) * ldd];
            const int i = r0 + tx, j = c0 + yy;
            if (i < n && j < n) {
                w[q] = W[i + (size_t)j * ldw];
                d[q] = Wd[i + (size_t)j * ldd];
                dd[q] = Wdd[i + (size_t)j * lddd];
            }
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int yy = ty + 8 * q, i = r0 + tx, j = c0 + yy;
            if (i < n && j < n) {
                T v = w[q];
                v = Sc<T>::add(v, Sc<T>::mul(xz, Sc<T>::conj(tile[tx][yy])));
                v = Sc<T>::add(v, Sc<T>::mul(xz, d[q]));
                v = Sc<T>::add(v, Sc<T>::mul(x2, dd[q]));
                W[i + (size_t)j * ldw] = v;
            }
        }
    }
}

// ---- reference C0: BSD LCG under NORAND (omm_rand.F90:19-55), element order of
// omm.F90:331-341: element e = j + i*n (column-major) uses draws 2e+1 and 2e+2.
__device__ inline void lcg_jump(unsigned long long t, unsigned long long& A, unsigned long long& Cc) {
    // affine map x -> a x + c (mod 2^31) raised to the power t
    const unsigned long long M = (1ull << 31) - 1;  // mask
    unsigned long long ra = 1, rc = 0;              // result map
    unsigned long long ba = 1103515245ull, bc = 12345ull;
    while (t) {
        if (t & 1ull) {  // result = base o result
            rc = (ba * rc + bc) & M;
            ra = (ba * ra) & M;
        }
        // base = base o base
        bc = (ba * bc + bc) & M;
        ba = (ba * ba) & M;
        t >>= 1;
    }
    A = ra;
    Cc = rc;
}
template <typename T>
__global__ void lcg_kernel(int n, int m, T* C, int ldc, double scale) {
    // a thread's elements are a fixed number of draws apart: the jump to its first one and the jump
    // from one to the next are formed once each
    Walk w(n, m);
    if (w.e >= w.total) return;
    const unsigned long long M = (1ull << 31) - 1;
    unsigned long long A, Cc, As, Cs;
    lcg_jump(2ull * w.e + 1ull, A, Cc);
    lcg_jump(2ull * w.step, As, Cs);
    unsigned long long x1 = (A * 123456ull + Cc) & M;
    for (; w.e < w.total; w.next()) {
        unsigned long long x2 = (1103515245ull * x1 + 12345ull) & M;
        double r1 = (double)x1 / 2147483648.0, r2 = (double)x2 / 2147483648.0;
        double h = 0.5 * r1;
        double el = (r2 - 0.5 >= 0.0) ? fabs(h) : -fabs(h);
        el = el * scale;
        zdbl v{el, 0.0};
        C[w.i + (size_t)w.j * ldc] = Sc<T>::from(v);
        x1 = (As * x1 + Cs) & M;
    }
}

// ---- reductions ------------------------------------------------------------------
// (s, c) + (s2, c2) for compensated sums: s + s2 split exactly into t + e (Knuth's TwoSum),
// the rounding errors carried in c
__device__ inline void comp_add(double& s, double& c, double s2, double c2) {
    const double t = s + s2, z = t - s;
    const double e = (s - (t - z)) + (s2 - z);
    s = t;
    c += c2 + e;
}

// blocks of the running reduction that have stored their partial sums; the last one sets it back to
// zero (reductions follow each other on the library's one stream)
__device__ unsigned g_reduce_done;

// Every block stores its K partial sums; the block that arrives last adds the nb records up with
// compensation, in a fixed order (a warp per value: each lane strided shares, then a tree over the
// lanes), so the result does not depend on timing, and writes it to `out` (pinned
// host memory, or device memory for sums the host does not need).  True in that block.  (A second kernel
// for the sum and a copy of its result cost 4 + 3 us and their gaps in each of a CG step's two
// reductions; all 13 values in every thread's registers, 4 us of the coefficients' last block.)
template <int K>
__device__ inline bool block_reduce_finish(double (&v)[K], double* part, double* out) {
    __shared__ double sm[K][kThreads / 32];
    __shared__ bool last;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nb = (int)gridDim.x;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        double a = v[k];
        for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
        if (lane == 0) sm[k][w] = a;
    }
    __syncthreads();
    if (threadIdx.x < K) {
        double s = 0.0;
        for (int i = 0; i < (int)(blockDim.x / 32); ++i) s += sm[threadIdx.x][i];
        part[(size_t)blockIdx.x * K + threadIdx.x] = s;
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) last = atomicInc(&g_reduce_done, (unsigned)nb - 1u) == (unsigned)nb - 1u;
    __syncthreads();
    if (!last) return false;
    __threadfence();
    // warp w takes the values w, w + 8: its lanes strided shares of the records, four in flight, then a tree
#pragma unroll
    for (int k = w; k < K; k += kThreads / 32) {
        double s[4] = {0.0, 0.0, 0.0, 0.0}, c[4] = {0.0, 0.0, 0.0, 0.0};
        for (int b0 = lane; b0 < nb; b0 += 128) {
            double x[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) x[u] = b0 + 32 * u < nb ? __ldcg(part + (size_t)(b0 + 32 * u) * K + k) : 0.0;
#pragma unroll
            for (int u = 0; u < 4; ++u) comp_add(s[u], c[u], x[u], 0.0);
        }
        comp_add(s[0], c[0], s[1], c[1]);
        comp_add(s[2], c[2], s[3], c[3]);
        comp_add(s[0], c[0], s[2], c[2]);
        for (int o = 16; o > 0; o >>= 1) {
            const double s2 = __shfl_down_sync(0xffffffffu, s[0], o), c2 = __shfl_down_sync(0xffffffffu, c[0], o);
            comp_add(s[0], c[0], s2, c2);
        }
        if (lane == 0) out[k] = s[0] + c[0];
    }
    return true;
}

template <typename T>
__device__ inline void dot_acc(T a, T b, double& re, double& im);
template <>
__device__ inline void dot_acc<double>(double a, double b, double& re, double&) { re += a * b; }
template <>
__device__ inline void dot_acc<zdbl>(zdbl a, zdbl b, double& re, double& im) {
    re += a.x * b.x + a.y * b.y;  // conj(a)*b
    im += a.x * b.y - a.y * b.x;
}

// Bound by memory (two reads per element); kAhead pairs of loads in flight per thread.
template <typename T>
__global__ void dot_kernel(int rows, int cols, const T* __restrict__ A, int lda, const T* __restrict__ B, int ldb,
                           double* part, double* out) {
    double v[2] = {0.0, 0.0};
    Walk w(rows, cols);
    while (w.e < w.total) {
        T a[kAhead], b[kAhead];
        int cnt = 0;
#pragma unroll
        for (int u = 0; u < kAhead; ++u)
            if (w.e < w.total) {
                a[u] = A[w.i + (size_t)w.j * lda];
                b[u] = B[w.i + (size_t)w.j * ldb];
                ++cnt;
                w.next();
            }
#pragma unroll
        for (int u = 0; u < kAhead; ++u)
            if (u < cnt) dot_acc<T>(a[u], b[u], v[0], v[1]);
    }
    block_reduce_finish<2>(v, part, out);
}

template <typename T>
__global__ void trace_kernel(int n, const T* A, int lda, double* part, double* out) {
    double v[2] = {0.0, 0.0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        T a = A[i + (size_t)i * lda];
        zdbl z;
        if constexpr (sizeof(T) == 8) { z.x = *(const double*)&a; z.y = 0.0; }
        else { z = *(const zdbl*)&a; }
        v[0] += z.x;
        v[1] += z.y;
    }
    block_reduce_finish<2>(v, part, out);
}

// The 13 traces of calc_coeff (omm_ops.F90:194-211) in one pass over the six n x n
// matrices.  TrHdSd needs SWd^H, read through a shared-memory transposed tile.
// Index: 0 TrH 1 TrHS 2 TrHd 3 TrHdS 4 TrHSd 5 TrHdd 6 TrHddS 7 TrHSdd 8 TrHdSd
//        9 TrHdSdH 10 TrHddSd 11 TrHdSdd 12 TrHddSdd
template <typename T>
__device__ inline double re_dot(T a, T b) {
    double re = 0.0, im = 0.0;
    dot_acc<T>(a, b, re, im);
    return re;
}
template <typename T>
__device__ inline double re_of(T a) {
    if constexpr (sizeof(T) == 8) return *(const double*)&a;
    else return ((const zdbl*)&a)->x;
}
__host__ __device__ inline void coeff_of_traces(const double t[13], double coeff[5]) {  // omm_ops.F90:213-217
    coeff[0] = 2.0 * t[0] - t[1];
    coeff[1] = 2.0 * (2.0 * t[2] - t[3] - t[4]);
    coeff[2] = 2.0 * (t[5] - t[8] - t[9]) - t[6] - t[7];
    coeff[3] = -2.0 * (t[10] + t[11]);
    coeff[4] = -t[12];
}
template <typename T>
__global__ void coeff_kernel(int n, const T* __restrict__ HW, int l0, const T* __restrict__ SW, int l1,
                             const T* __restrict__ HWd, int l2, const T* __restrict__ SWd, int l3,
                             const T* __restrict__ HWdd, int l4, const T* __restrict__ SWdd, int l5, double* part,
                             double* out, const LineSearch ls) {
    if (ls.stop && *ls.stop) return;
    __shared__ T tileT[32][33];
    double v[13];
#pragma unroll
    for (int k = 0; k < 13; ++k) v[k] = 0.0;
    int tiles = (n + 31) / 32;
    int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
    for (int t = blockIdx.x; t < tiles * tiles; t += gridDim.x) {
        int bi = t % tiles, bj = t / tiles;
        // load SWd tile (rows bj*32.., cols bi*32..) so that tileT[c][r] = SWd(bj*32+r, bi*32+c)
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            int yy = ty + 8 * q, r = bj * 32 + tx, c = bi * 32 + yy;
            T val{};
            if (r < n && c < n) val = SWd[r + (size_t)c * l3];
            tileT[yy][tx] = val;
        }
        // two rounds of two elements each, the loads of a round (twelve) before its sums
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            T hw[2], sw[2], hwd[2], swd[2], hwdd[2], swdd[2];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int i = bi * 32 + tx, j = bj * 32 + ty + 8 * (2 * h + q);
                if (i < n && j < n) {
                    hw[q] = HW[i + (size_t)j * l0];
                    sw[q] = SW[i + (size_t)j * l1];
                    hwd[q] = HWd[i + (size_t)j * l2];
                    swd[q] = SWd[i + (size_t)j * l3];
                    hwdd[q] = HWdd[i + (size_t)j * l4];
                    swdd[q] = SWdd[i + (size_t)j * l5];
                }
            }
            if (h == 0) __syncthreads();  // tileT is complete
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int yy = ty + 8 * (2 * h + q), i = bi * 32 + tx, j = bj * 32 + yy;
                if (i >= n || j >= n) continue;
                T swdT = tileT[tx][yy];  // SWd(j, i)
                if (i == j) {
                    v[0] += re_of(hw[q]);
                    v[2] += re_of(hwd[q]);
                    v[5] += re_of(hwdd[q]);
                }
                v[1] += re_dot(hw[q], sw[q]);
                v[3] += re_dot(sw[q], hwd[q]);
                v[4] += re_dot(hw[q], swd[q]);
                v[6] += re_dot(hwdd[q], sw[q]);
                v[7] += re_dot(hw[q], swdd[q]);
                v[8] += re_dot(Sc<T>::conj(swdT), hwd[q]);  // mm_trace(SWd^H, HWd): conj((SWd^H)_ij) = SWd_ji
                v[9] += re_dot(swd[q], hwd[q]);
                v[10] += re_dot(hwdd[q], swd[q]);
                v[11] += re_dot(swdd[q], hwd[q]);
                v[12] += re_dot(hwdd[q], swdd[q]);
            }
        }
    }
    const bool last = block_reduce_finish<13>(v, part, out);
    if (!last || !ls.record) return;
    __syncthreads();
    if (threadIdx.x == 0) {
        double c[5], x = 0.0;
        coeff_of_traces(out, c);
        bool fail = false, finite = true;
        for (int k = 0; k < 5; ++k) finite = finite && isfinite(c[k]);
        if (finite) solve_quartic(c, &x, &fail);
        const double old = ls.state[2], e = quartic_energy(c, x), number = ls.state[3] + 1.0;
        const double diff = 2.0 * fabs((e - old) / (e + old));
        const bool stop = !finite || fail || diff <= ls.tol || number >= ls.most;
        volatile double* q = ls.record + 16 * ((long long)ls.state[3] % kStepRecords);
        for (int k = 0; k < 5; ++k) q[k] = c[k];
        q[5] = x;
        q[6] = e;
        q[7] = diff;
        q[8] = stop ? 1.0 : 0.0;
        __threadfence_system();
        q[9] = number;  // the host polls it: last
        ls.state[1] = x;
        ls.state[2] = e;
        ls.state[3] = number;
        if (stop) *ls.stop = 1;
    }
}

// Polak-Ribiere lambda = v0 / v1 for the next direction, left in device memory: the host has no use for
// it, and waiting for it cost a round trip per CG step.
// SAME: no preconditioner, PG is G and PG_p is G_p (two reads per element instead of four)
template <typename T, bool SAME>
__global__ void lambda_kernel(int rows, int cols, const T* __restrict__ PG, int l0, const T* __restrict__ G, int l1,
                              const T* __restrict__ Gp, int l2, const T* __restrict__ PGp, int l3, double* part,
                              double* out, double* lambda, const int* __restrict__ stop) {
    if (stop && *stop) return;
    double v[2] = {0.0, 0.0};
    Walk w(rows, cols);
    while (w.e < w.total) {
        T g[kAhead], gp[kAhead], pg[SAME ? 1 : kAhead], pgp[SAME ? 1 : kAhead];
        int cnt = 0;
#pragma unroll
        for (int u = 0; u < kAhead; ++u)
            if (w.e < w.total) {
                g[u] = G[w.i + (size_t)w.j * l1];
                gp[u] = Gp[w.i + (size_t)w.j * l2];
                if constexpr (!SAME) {
                    pg[u] = PG[w.i + (size_t)w.j * l0];
                    pgp[u] = PGp[w.i + (size_t)w.j * l3];
                }
                ++cnt;
                w.next();
            }
#pragma unroll
        for (int u = 0; u < kAhead; ++u)
            if (u < cnt) {
                T w2;
                if constexpr (sizeof(T) == 8) w2 = g[u] - gp[u];
                else w2 = zdbl{((zdbl*)&g[u])->x - ((zdbl*)&gp[u])->x, ((zdbl*)&g[u])->y - ((zdbl*)&gp[u])->y};
                if constexpr (SAME) {
                    v[0] += re_dot(g[u], w2);
                    v[1] += re_dot(gp[u], gp[u]);
                } else {
                    v[0] += re_dot(pg[u], w2);    // mm_trace(PG, work2), work2 = G - G_p
                    v[1] += re_dot(pgp[u], gp[u]);  // mm_trace(PG_p, G_p)
                }
            }
    }
    if (block_reduce_finish<2>(v, part, out)) {
        __syncthreads();
        if (threadIdx.x == 0) *lambda = out[0] / out[1];
    }
}

// The updates of a CG step that do not wait for anything of it but x, in one launch (a small solve spent
// five launches of 2 to 3 us and their gaps on them): C += x D, X += x Y (flat arrays; bX = 0: X is
// updated elsewhere), both W updates of w_update_kernel, and with L the left factor of calc_G from the new
// W matrices.  Blocks [0, bC) take C, [bC, bC + bX) X, the rest 32 x 32 tiles of the W matrices.
template <typename T>
struct CgUpdate {
    size_t nc, nx;
    T* C;
    const T* D;
    T* X;
    const T* Y;
    T *HW, *SW, *L;      // n x n, n x n, n x 2n
    const T *Wd, *Wdd;   // [HWd; SWd], [HWdd; SWdd], leading dimension 2n
    int n, bC, bX;
    double x;
    const double* x_at;
    const int* stop;
};
template <typename T>
__global__ void __launch_bounds__(kThreads) cg_update_kernel(const __grid_constant__ CgUpdate<T> p) {
    if (p.stop && *p.stop) return;
    const double x = p.x_at ? *p.x_at : p.x;
    const zdbl xz{x, 0.0}, x2{x * x, 0.0};
    int b = blockIdx.x;
    if (b < p.bC + p.bX) {
        const bool c = b < p.bC;
        T* __restrict__ y = c ? p.C : p.X;
        const T* __restrict__ a = c ? p.D : p.Y;
        const size_t total = c ? p.nc : p.nx, step = (size_t)(c ? p.bC : p.bX) * blockDim.x;
        for (size_t e = (size_t)(c ? b : b - p.bC) * blockDim.x + threadIdx.x; e < total; e += kAhead * step) {
            T av[kAhead], yv[kAhead];
#pragma unroll
            for (int u = 0; u < kAhead; ++u)
                if (e + u * step < total) {
                    av[u] = a[e + u * step];
                    yv[u] = y[e + u * step];
                }
#pragma unroll
            for (int u = 0; u < kAhead; ++u)
                if (e + u * step < total) y[e + u * step] = Sc<T>::add(yv[u], Sc<T>::mul(xz, av[u]));
        }
        return;
    }
    b -= p.bC + p.bX;
    __shared__ T tile[2][32][33];
    const int n = p.n, tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
    const int tiles = (n + 31) / 32, nb = gridDim.x - p.bC - p.bX;
    for (long long t = b; t < (long long)tiles * tiles; t += nb) {
        const int r0 = (int)(t % tiles) * 32, c0 = (int)(t / tiles) * 32;
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int yy = ty + 8 * q;
            if (c0 + tx < n && r0 + yy < n) {
                tile[0][yy][tx] = p.Wd[c0 + tx + (size_t)(r0 + yy) * 2 * n];
                tile[1][yy][tx] = p.Wd[n + c0 + tx + (size_t)(r0 + yy) * 2 * n];
            }
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int yy = ty + 8 * q, i = r0 + tx, j = c0 + yy;
            if (i >= n || j >= n) continue;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                T* W = h ? p.SW : p.HW;
                const size_t at = (size_t)h * n + i + (size_t)j * 2 * n;
                T v = W[i + (size_t)j * n];
                v = Sc<T>::add(v, Sc<T>::mul(xz, Sc<T>::conj(tile[h][tx][yy])));
                v = Sc<T>::add(v, Sc<T>::mul(xz, p.Wd[at]));
                v = Sc<T>::add(v, Sc<T>::mul(x2, p.Wdd[at]));
                W[i + (size_t)j * n] = v;
                if (p.L) {
                    T l = Sc<T>::mul(zdbl{-2.0, 0.0}, v);
                    if (h && i == j) l = Sc<T>::add(Sc<T>::from(zdbl{4.0, 0.0}), l);
                    p.L[i + (size_t)(h ? j : n + j) * n] = l;
                }
            }
        }
    }
}

// L = [4I - 2 SW, -2 HW] (n x 2n), the left factor of calc_G as one product
template <typename T>
__global__ void calcG_left_kernel(int n, const T* __restrict__ SW, int lds, const T* __restrict__ HW, int ldh,
                                  T* __restrict__ L, int ldl) {
    for (Walk w(n, 2 * n); w.e < w.total; w.next()) {
        const bool left = w.j < n;
        T v = left ? SW[w.i + (size_t)w.j * lds] : HW[w.i + (size_t)(w.j - n) * ldh];
        v = Sc<T>::mul(zdbl{-2.0, 0.0}, v);
        if (left && w.i == w.j) v = Sc<T>::add(Sc<T>::from(zdbl{4.0, 0.0}), v);
        L[w.i + (size_t)w.j * ldl] = v;
    }
}

template <typename T>
__global__ void transpose_kernel(int rows, int cols, const T* A, int lda, int conj, T* Tm, int ldt) {
    // Tm (cols x rows) = op(A), A rows x cols
    __shared__ T tile[32][33];
    int bx = blockIdx.x * 32, by = blockIdx.y * 32;
    int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    for (int yy = ty; yy < 32; yy += 8) {
        int r = bx + tx, c = by + yy;
        if (r < rows && c < cols) tile[yy][tx] = A[r + (size_t)c * lda];
    }
    __syncthreads();
    for (int yy = ty; yy < 32; yy += 8) {
        int r = by + tx, c = bx + yy;  // Tm(r, c) = A(c, r)
        if (r < cols && c < rows) {
            T v = tile[tx][yy];
            Tm[r + (size_t)c * ldt] = conj ? Sc<T>::conj(v) : v;
        }
    }
}

inline int op_code(char op) {
    if (op == 'n' || op == 'N') return 0;
    if (op == 't' || op == 'T') return 1;
    if (op == 'c' || op == 'C') return 2;
    fail(OMM_ERR_ARG, std::string("process_opM: invalid opM '") + op + "'");
}

double* scratch_partials(size_t nrec, int K) {
    rt().scratch.ensure((nrec * K + 64) * sizeof(double));
    return rt().scratch.as<double>();
}

// the reduction's result, which its last block wrote to the pinned buffer
void finish_reduce(int K, double* out) {
    sync();
    for (int k = 0; k < K; ++k) out[k] = rt().host_pinned[k];
}

// blocks of a reduction: eight elements per thread, at most six blocks per SM (a block's own sums, its
// fence and its record cost as much as some 30 elements per thread)
inline int reduce_grid(size_t elems) { return std::min(grid_for(elems, 8), 148 * 6); }

// blocks of a kernel that takes 32 x 32 tiles in turn
inline int tile_grid(int rows, int cols) {
    const long long t = (long long)((rows + 31) / 32) * ((cols + 31) / 32);
    return (int)std::max<long long>(1, std::min<long long>(t, 148 * 8));
}

}  // namespace

// ------------------------------------------------------------------ host wrappers
void k_axpby(const DView& A, char op, DView& C, const double alpha[2], const double beta[2], const double* beta_at,
             const int* stop) {
    int oc = op_code(op);
    if (A.is_real && oc == 2) oc = 1;
    size_t tot = (size_t)C.rows * C.cols;
    if (tot == 0) return;
    zdbl a{alpha[0], alpha[1]}, b{beta[0], beta[1]};
    int bz = 0;  // the reference multiplies C by beta even when beta == 0 (NaN propagates); keep that
    if (oc == 0) {
        if (C.is_real)
            axpby_kernel<double><<<grid_for(tot), kThreads, 0, rt().stream>>>(C.rows, C.cols, A.as<double>(), A.ld,
                                                                                C.as<double>(), C.ld, a, b, bz, beta_at, stop);
        else
            axpby_kernel<zdbl><<<grid_for(tot), kThreads, 0, rt().stream>>>(C.rows, C.cols, A.as<zdbl>(), A.ld,
                                                                              C.as<zdbl>(), C.ld, a, b, bz, beta_at, stop);
    } else {
        if (beta_at || stop) fail(OMM_ERR_ARG, "axpby: a device scalar with a transposed operand");
        const int grid = tile_grid(C.rows, C.cols);
        if (C.is_real)
            axpby_trans_kernel<double><<<grid, kThreads, 0, rt().stream>>>(C.rows, C.cols, A.as<double>(), A.ld, 0,
                                                                             C.as<double>(), C.ld, a, b, bz);
        else
            axpby_trans_kernel<zdbl><<<grid, kThreads, 0, rt().stream>>>(C.rows, C.cols, A.as<zdbl>(), A.ld, oc == 2,
                                                                           C.as<zdbl>(), C.ld, a, b, bz);
    }
    OMM_KCHECK();
}

void k_scale(DView& C, const double beta[2]) {
    size_t tot = (size_t)C.rows * C.cols;
    if (tot == 0) return;
    zdbl b{beta[0], beta[1]};
    if (C.is_real) scale_kernel<double><<<grid_for(tot), kThreads, 0, rt().stream>>>(C.rows, C.cols, C.as<double>(), C.ld, b);
    else scale_kernel<zdbl><<<grid_for(tot), kThreads, 0, rt().stream>>>(C.rows, C.cols, C.as<zdbl>(), C.ld, b);
    OMM_KCHECK();
}

void k_set(DView& C, char seC, const double alpha[2], const double beta[2]) {
    int lu = (seC == 'u' || seC == 'U') ? 1 : (seC == 'l' || seC == 'L') ? 2 : 0;  // process_seM
    size_t tot = (size_t)C.rows * C.cols;
    if (tot == 0) return;
    zdbl a{alpha[0], alpha[1]}, b{beta[0], beta[1]};
    if (C.is_real) set_kernel<double><<<grid_for(tot), kThreads, 0, rt().stream>>>(C.rows, C.cols, C.as<double>(), C.ld, lu, a, b);
    else set_kernel<zdbl><<<grid_for(tot), kThreads, 0, rt().stream>>>(C.rows, C.cols, C.as<zdbl>(), C.ld, lu, a, b);
    OMM_KCHECK();
}

void k_set_element(DView& C, int i, int j, const double alpha[2], const double beta[2]) {
    size_t idx = (size_t)i + (size_t)j * C.ld;
    zdbl a{alpha[0], alpha[1]}, b{beta[0], beta[1]};
    if (C.is_real) set_element_kernel<double><<<1, 1, 0, rt().stream>>>(C.as<double>(), idx, a, b);
    else set_element_kernel<zdbl><<<1, 1, 0, rt().stream>>>(C.as<zdbl>(), idx, a, b);
    OMM_KCHECK();
}

void k_fill_lower_from_upper(DView& C) {
    if (C.rows == 0) return;
    int nt = (C.rows + 31) / 32;
    dim3 grid(nt, nt);
    if (C.is_real) fill_lower_kernel<double><<<grid, kThreads, 0, rt().stream>>>(C.rows, C.as<double>(), C.ld);
    else fill_lower_kernel<zdbl><<<grid, kThreads, 0, rt().stream>>>(C.rows, C.as<zdbl>(), C.ld);
    OMM_KCHECK();
}

void k_w_update(DView& W, const DView& Wd, const DView& Wdd, double x) {
    const int grid = tile_grid(W.rows, W.rows);
    if (W.is_real)
        w_update_kernel<double><<<grid, kThreads, 0, rt().stream>>>(W.rows, W.as<double>(), W.ld,
                                                                               Wd.as<double>(), Wd.ld,
                                                                               Wdd.as<double>(), Wdd.ld, x);
    else
        w_update_kernel<zdbl><<<grid, kThreads, 0, rt().stream>>>(W.rows, W.as<zdbl>(), W.ld, Wd.as<zdbl>(),
                                                                             Wd.ld, Wdd.as<zdbl>(), Wdd.ld, x);
    OMM_KCHECK();
}

void k_calcG_left(const DView& SW, const DView& HW, DView& L) {
    const int n = L.rows;
    const size_t tot = (size_t)n * 2 * n;
    if (L.is_real)
        calcG_left_kernel<double><<<grid_for(tot), kThreads, 0, rt().stream>>>(n, SW.as<double>(), SW.ld,
                                                                                 HW.as<double>(), HW.ld, L.as<double>(),
                                                                                 L.ld);
    else
        calcG_left_kernel<zdbl><<<grid_for(tot), kThreads, 0, rt().stream>>>(n, SW.as<zdbl>(), SW.ld, HW.as<zdbl>(),
                                                                               HW.ld, L.as<zdbl>(), L.ld);
    OMM_KCHECK();
}

void k_lcg_init(DView& C) {
    // the scale 1e-2/sqrt(m) of omm.F90:342 is applied by the caller through m_scale
    size_t tot = (size_t)C.rows * C.cols;
    if (C.is_real) lcg_kernel<double><<<grid_for(tot), kThreads, 0, rt().stream>>>(C.rows, C.cols, C.as<double>(), C.ld, 1.0);
    else lcg_kernel<zdbl><<<grid_for(tot), kThreads, 0, rt().stream>>>(C.rows, C.cols, C.as<zdbl>(), C.ld, 1.0);
    OMM_KCHECK();
}

void r_trace(const DView& A, double out[2]) {
    int nb = 64;
    double* part = scratch_partials(nb + 1, 2);
    if (A.is_real) trace_kernel<double><<<nb, kThreads, 0, rt().stream>>>(A.rows, A.as<double>(), A.ld, part,
                                                                          rt().host_pinned);
    else trace_kernel<zdbl><<<nb, kThreads, 0, rt().stream>>>(A.rows, A.as<zdbl>(), A.ld, part, rt().host_pinned);
    OMM_KCHECK();
    finish_reduce(2, out);
}

void r_dot(const DView& A, const DView& B, double out[2]) {
    size_t tot = (size_t)A.rows * A.cols;
    int nb = reduce_grid(tot);
    double* part = scratch_partials(nb + 1, 2);
    if (A.is_real)
        dot_kernel<double><<<nb, kThreads, 0, rt().stream>>>(A.rows, A.cols, A.as<double>(), A.ld, B.as<double>(), B.ld, part,
                                                            rt().host_pinned);
    else
        dot_kernel<zdbl><<<nb, kThreads, 0, rt().stream>>>(A.rows, A.cols, A.as<zdbl>(), A.ld, B.as<zdbl>(), B.ld, part,
                                                          rt().host_pinned);
    OMM_KCHECK();
    finish_reduce(2, out);
}

void r_coeff(const DView& HW, const DView& SW, const DView& HWd, const DView& SWd, const DView& HWdd, const DView& SWdd,
             double coeff[5], const LineSearch* lsp) {
    int n = HW.rows;
    const LineSearch ls = lsp ? *lsp : LineSearch{};
    int tiles = (n + 31) / 32;
    int nb = tiles * tiles;
    if (nb > 148 * 8) nb = 148 * 8;
    double* part = scratch_partials(nb + 1, 13);
    double* out = lsp ? part + (size_t)nb * 13 : rt().host_pinned;
    if (HW.is_real)
        coeff_kernel<double><<<nb, kThreads, 0, rt().stream>>>(n, HW.as<double>(), HW.ld, SW.as<double>(), SW.ld,
                                                                 HWd.as<double>(), HWd.ld, SWd.as<double>(), SWd.ld,
                                                                 HWdd.as<double>(), HWdd.ld, SWdd.as<double>(),
                                                                 SWdd.ld, part, out, ls);
    else
        coeff_kernel<zdbl><<<nb, kThreads, 0, rt().stream>>>(n, HW.as<zdbl>(), HW.ld, SW.as<zdbl>(), SW.ld,
                                                               HWd.as<zdbl>(), HWd.ld, SWd.as<zdbl>(), SWd.ld,
                                                               HWdd.as<zdbl>(), HWdd.ld, SWdd.as<zdbl>(), SWdd.ld,
                                                               part, out, ls);
    OMM_KCHECK();
    if (lsp) return;
    double t[13];
    finish_reduce(13, t);
    coeff_of_traces(t, coeff);
}

void r_lambda(const DView& PG, const DView& G, const DView& Gp, const DView& PGp, double* lambda,
              const int* stop) {
    size_t tot = (size_t)G.rows * G.cols;
    int nb = reduce_grid(tot);
    double* part = scratch_partials(nb + 1, 2);
    const bool same = PG.p == G.p && PG.ld == G.ld && PGp.p == Gp.p && PGp.ld == Gp.ld;
    auto launch = [&](auto tag, auto kernel) {
        using T = decltype(tag);
        kernel<<<nb, kThreads, 0, rt().stream>>>(G.rows, G.cols, PG.as<T>(), PG.ld, G.as<T>(), G.ld, Gp.as<T>(), Gp.ld,
                                                 PGp.as<T>(), PGp.ld, part, part + (size_t)nb * 2, lambda, stop);
    };
    if (G.is_real) launch(double{}, same ? lambda_kernel<double, true> : lambda_kernel<double, false>);
    else launch(zdbl{}, same ? lambda_kernel<zdbl, true> : lambda_kernel<zdbl, false>);
    OMM_KCHECK();
}

void k_cg_update(int n, int m, double x, DView& C, const DView& D, DView* X, const DView* Y, DView& HW, DView& SW,
                 const DView& Wd, const DView& Wdd, DView* L, const double* x_at, const int* stop) {
    auto launch = [&](auto tag) {
        using T = decltype(tag);
        CgUpdate<T> p{};
        p.n = n;
        p.x = x;
        p.x_at = x_at;
        p.stop = stop;
        p.C = C.as<T>();
        p.D = D.as<T>();
        p.nc = (size_t)n * m;
        p.bC = grid_for(p.nc);
        if (X) {
            p.X = X->as<T>();
            p.Y = Y->as<T>();
            p.nx = (size_t)2 * n * m;
            p.bX = grid_for(p.nx);
        }
        p.HW = HW.as<T>();
        p.SW = SW.as<T>();
        p.Wd = Wd.as<T>();
        p.Wdd = Wdd.as<T>();
        p.L = L ? L->as<T>() : nullptr;
        cg_update_kernel<T><<<p.bC + p.bX + tile_grid(n, n), kThreads, 0, rt().stream>>>(p);
    };
    if (C.is_real) launch(double{});
    else launch(zdbl{});
    OMM_KCHECK();
}

void gemm(char opA, char opB, int M, int N, int K, const double alpha[2], const DView& A, const DView& B,
          const double beta[2], DView& C) {
    auto cop = [&](char o, bool real) {
        int c = op_code(o);
        if (c == 0) return CUBLAS_OP_N;
        if (c == 1 || real) return CUBLAS_OP_T;
        return CUBLAS_OP_C;
    };
    if (M == 0 || N == 0) return;
    if (alpha[0] == 0.0 && alpha[1] == 0.0) {
        // C = beta C, and 0 whatever C holds for beta = 0 (as BLAS has it): A and B are not read
        if (beta[0] == 0.0 && beta[1] == 0.0) k_set(C, 'a', beta, beta);
        else if (beta[0] != 1.0 || beta[1] != 0.0) k_scale(C, beta);
        return;
    }
    if (fp64_emu_enabled()) {
        const char ops[3] = {'n', 't', 'c'};
        const bool cplx = !C.is_real, real_scalars = !cplx || (alpha[1] == 0.0 && beta[1] == 0.0);
        // the emulation reads its operands before it writes the result, the FP64 kernel while it does: products
        // whose result shares any memory with an operand never take the latter
        const bool in_place = overlap(C, A) || overlap(C, B);
        // real operands with odd leading dimensions are copied 8 bytes at a time: 1,001 x 515 x 2,003 109 us on the
        // FP64 tensor cores, 85 emulated
        const auto wide16 = [](const DView& v) { return v.ld % 2 == 0 && (reinterpret_cast<uintptr_t>(v.p) & 15) == 0; };
        const bool wide = cplx || (wide16(A) && wide16(B));
        if (real_scalars && (in_place ? fp64_emu_fits(M, N, K) : fp64_emu_worth(M, N, K, cplx, wide))) {
            // FP64-accurate product on the int8 tensor cores (ozaki.cu); 'c' is 't' for real data, complex
            // ones are one product of the stacked parts
            if (cplx) gemm_z_emu(ops[op_code(opA)], ops[op_code(opB)], M, N, K, alpha[0], A, B, beta[0], C);
            else gemm_f64_emu(op_code(opA) ? 't' : 'n', op_code(opB) ? 't' : 'n', M, N, K, alpha[0], A, B, beta[0], C);
            return;
        }
        if (!in_place && gemm_dmma_takes(A) && gemm_dmma_takes(B) && gemm_dmma_takes(C) &&
            !gemm_dmma_slower(cplx, M, N, K)) {
            gemm_dmma(ops[op_code(opA)], ops[op_code(opB)], M, N, K, alpha, &A, &B, beta, &C);
            return;
        }
    }
    OMM_CKB(cublasSetStream(rt().blas, rt().stream));
    if (C.is_real) {
        OMM_CKB(cublasDgemm(rt().blas, cop(opA, true), cop(opB, true), M, N, K, &alpha[0], A.as<double>(), A.ld,
                            B.as<double>(), B.ld, &beta[0], C.as<double>(), C.ld));
    } else {
        cuDoubleComplex a = make_cuDoubleComplex(alpha[0], alpha[1]), b = make_cuDoubleComplex(beta[0], beta[1]);
        OMM_CKB(cublasZgemm(rt().blas, cop(opA, false), cop(opB, false), M, N, K, &a, A.as<cuDoubleComplex>(), A.ld,
                            B.as<cuDoubleComplex>(), B.ld, &b, C.as<cuDoubleComplex>(), C.ld));
    }
}

void transpose_into(const DView& A, char op, DView& Tm) {
    int oc = op_code(op);
    if (oc == 0) {  // plain copy
        double one[2] = {1.0, 0.0}, zero[2] = {0.0, 0.0};
        k_axpby(A, 'n', Tm, one, zero);
        return;
    }
    dim3 grid((A.rows + 31) / 32, (A.cols + 31) / 32);
    if (A.is_real)
        transpose_kernel<double><<<grid, kThreads, 0, rt().stream>>>(A.rows, A.cols, A.as<double>(), A.ld, 0,
                                                                      Tm.as<double>(), Tm.ld);
    else
        transpose_kernel<zdbl><<<grid, kThreads, 0, rt().stream>>>(A.rows, A.cols, A.as<zdbl>(), A.ld, oc == 2,
                                                                    Tm.as<zdbl>(), Tm.ld);
    OMM_KCHECK();
}

}  // namespace ommgpu
