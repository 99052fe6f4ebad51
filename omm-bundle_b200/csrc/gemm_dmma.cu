// FP64 (real and complex) matrix products on the FP64 tensor cores (mma.sync m8n8k4 f64; tcgen05 has no
// FP64 kind), for the products too small for the int8 emulation of ozaki.cu to pay: MatrixSwitch products
// of a few hundred rows, and every product of the CG step of a small problem.
//
//   C_z = alpha * op(A_z) op(B_z) + beta * C_z,  op in {n, t, c},  z = 0 .. nz - 1 (nz <= 2)
//
// A CTA of four warps forms one 32 x 32 tile, a 16 x 16 quarter each; its K runs in 16-k (complex: 8-k) chunks
// through a ring of three (two) stages filled by cp.async ahead, one barrier per chunk, and an unsplit tile is
// written from the accumulators.  Warps that share the chunk's k instead (each the whole tile by its own four
// k, the partial tiles added at the end) load half as many fragments but were slower at every unsplit size
// and most split ones: 3,000 x 3,000 x 16 74 us against 26, 1,895 x 415 x 160 19 against 12, 1,500 x 800 x 300
// 33 against 26, 256 x 128 x 832 9.5 against 8.5.  Taller tiles (64 x 64, 64 x 32) were slower too.
// What bounds small products is latency -- one or two CTAs per SM, each a serial chain over K -- so
//   * a chunk is few instructions: copies from pointers formed once, stages as immediate offsets of an
//     unrolled turn (with addresses formed per chunk it was 200 instructions a warp, at five clocks each,
//     for 16 DMMAs: 128 x 832 x 832 twice 31 us, now 21);
//   * K is split over the CTAs of a cluster (up to 8): the partial tiles are added through distributed
//     shared memory in rank order (the same bits every time), and each CTA writes its part of the tile;
//   * two products of one shape run in one launch (D [H, S] and [X; Y] D^H of a CG step);
//   * a Hermitian product forms its upper tiles only and writes both triangles.
// Operands keep their global order in shared memory (rows or k contiguous, whichever the op makes of
// them), padded so that the 16 lanes of a half-warp's fragment load (8 lanes for complex elements) fall
// in distinct banks.  Complex products take four DMMAs per fragment pair.
// A call through the entry point, with cuBLAS's in brackets (with their waits, microseconds): 256 x 128 x 832 20
// (22), 500^3 25 (26), 1,895 x 415 x 161 29 (26), 3,000 x 3,000 x 16 37 (39), 1,500 x 800 x 300 42 (42), 512 x
// 512 x 4,096 99 (91), complex 500^3 57 (55), 2,500 x 900 x 120 96 (93); with a third of cuBLAS's rounding error
// (Sums below), and in a launch that a graph can hold.
#include "internal.h"

#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>
#include <type_traits>

namespace cg = cooperative_groups;

namespace ommgpu {

namespace {


struct DgArgs {
    int M, N, K;
    const double *A[2], *B[2];
    double* C[2];
    long long lda, ldb, ldc;  // elements
    zdbl alpha, beta;
    int beta_zero;
    int conj_a, conj_b;
    int vec;      // 16-byte copies of A and B (real: even leading dimensions and 16-byte addresses)
    int herm[2];  // rows per Hermitian block of C_z (0: none): both triangles from the upper tiles
    int kper;     // k per CTA of the cluster (a multiple of the chunk)
    const int* stop;
};

template <bool CPLX> struct El { using T = double; };
template <> struct El<true> { using T = double2; };

// copy of 16 (WIDE) or 8 bytes to shared memory, `bytes` of them from src and zeros beyond
template <bool WIDE>
__device__ __forceinline__ void cp(uint32_t dst, const void* src, int bytes) {
    if constexpr (WIDE)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(a), "d"(b));
}

__device__ __forceinline__ double flip(double v, int sign) {
    return __hiloint2double(__double2hiint(v) ^ sign, __double2loint(v));
}

template <bool CPLX, int R>
constexpr int stride_rows() { return CPLX ? R + 2 : R + 4; }  // [k][r]
template <bool CPLX>
constexpr int chunk() { return CPLX ? 8 : 16; }
template <bool CPLX>
constexpr int stride_k() { return chunk<CPLX>() + 4; }  // [r][k]
template <bool CPLX, int R, bool KC>
constexpr int tile_elems() { return KC ? R * stride_k<CPLX>() : chunk<CPLX>() * stride_rows<CPLX, R>(); }
template <bool CPLX, int BM, int BN, int ST, bool TA, bool TB>
constexpr int smem_bytes() {
    const int es = CPLX ? 16 : 8;
    const int ring = ST * (tile_elems<CPLX, BM, TA>() + tile_elems<CPLX, BN, !TB>()) * es;
    const int part = BM * BN * es;  // the partial tile of a split K
    return ring > part ? ring : part;
}

// A thread's copies of an operand's chunks into shared memory: R rows (of op(A), or columns of op(B)) from
// row r0 (of n), k from k_lo on.  KC: k contiguous in memory, element (r, k) at S[k + r ld], kept as
// [r][k]; else rows contiguous, at S[r + k ld], kept as [k][r].  Source, place and bytes of every copy are
// formed once: a chunk then costs an add and a copy each -- forming them per chunk took a warp longer than
// its DMMAs, which at one or two CTAs per SM nothing hides.
template <bool CPLX, int R, bool KC, int NTHR, bool VEC>
struct Loader {
    using T = typename El<CPLX>::T;
    static constexpr int BK = chunk<CPLX>(), W = CPLX ? 2 : 1, PER = VEC && !CPLX ? 2 : 1;  // elements per copy
    static constexpr int NU = BK * R / PER / NTHR;
    const double* src[NU];
    uint32_t dst[NU];
    int bytes[NU], kk[NU];
    long long step;
    __device__ __forceinline__ Loader(T* ring, const double* S, long long ld, int r0, int n, int k_lo) {
        step = (KC ? (long long)BK : BK * ld) * W;
#pragma unroll
        for (int u = 0; u < NU; ++u) {
            const int e = threadIdx.x + NTHR * u;
            const int k = KC ? PER * (e % (BK / PER)) : e / (R / PER);
            const int rr = KC ? e / (BK / PER) : PER * (e % (R / PER)), r = r0 + rr;
            kk[u] = k;
            const int rows = KC ? (r < n ? PER : 0) : max(0, min(PER, n - r));
            bytes[u] = rows * 8 * W;
            // a copy of no bytes reads nothing: any address does
            src[u] = S + (bytes[u] ? (KC ? (long long)(k_lo + k) + r * ld : (long long)r + (k_lo + k) * ld) * W : 0);
            dst[u] = (uint32_t)__cvta_generic_to_shared(ring + (KC ? rr * stride_k<CPLX>() + k : k * stride_rows<CPLX, R>() + rr));
        }
    }
    // the next chunk into the stage at `off` bytes
    __device__ __forceinline__ void copy(uint32_t off) {
#pragma unroll
        for (int u = 0; u < NU; ++u) {
            cp<CPLX || VEC>(dst[u] + off, src[u], bytes[u]);
            src[u] += step;
        }
    }
    // the last chunk, of which only krem k are left
    __device__ __forceinline__ void copy_tail(uint32_t off, int krem) {
#pragma unroll
        for (int u = 0; u < NU; ++u) {
            const int left = KC ? max(0, min(PER, krem - kk[u])) * 8 * W : (kk[u] < krem ? bytes[u] : 0);
            cp<CPLX || VEC>(dst[u] + off, src[u], bytes[u] ? left : 0);
        }
    }
};

// A warp's part of the tile: NP parts (real; re and im) of MT x NT fragments.
template <int NP, int MT, int NT>
struct Sums {
    double v[NP][MT][NT][2];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int s = 0; s < NP; ++s)
#pragma unroll
            for (int i = 0; i < MT; ++i)
#pragma unroll
                for (int j = 0; j < NT; ++j) v[s][i][j][0] = v[s][i][j][1] = 0.0;
    }
    // adds the sums o and sets them to zero
    __device__ __forceinline__ void take(Sums& o) {
#pragma unroll
        for (int s = 0; s < NP; ++s)
#pragma unroll
            for (int i = 0; i < MT; ++i)
#pragma unroll
                for (int j = 0; j < NT; ++j) {
                    v[s][i][j][0] += o.v[s][i][j][0];
                    v[s][i][j][1] += o.v[s][i][j][1];
                }
        o.clear();
    }
};
// RUN > 0: K is added up in runs of RUN chunks (16 products each) in the DMMAs' accumulators, and those -- with
// THIRD in eights first -- because the rounding errors of one chain grow with its length.  Rms error over
// sqrt(sum |a|^2 |b|^2), and time: 512 x 512 x 4,096 in one chain 2.0e-15 and 94 us, in runs of 32 products 2.4e-16
// and 99 us (of 64: 3.8e-16 and 96; of 16, which wait for their DMMAs too often: 2.4e-16 and 137).
constexpr int RUNS = 8;  // runs of the second level

// TA: A is K-contiguous (op 't' / 'c'); TB: B is column-contiguous (op 't' / 'c')
template <bool CPLX, int BM, int BN, int WM, int WN, int ST, bool TA, bool TB, bool VEC, int RUN, bool THIRD>
__global__ void __launch_bounds__(32 * WM * WN) gemm_dmma_kernel(const __grid_constant__ DgArgs p) {
    using T = typename El<CPLX>::T;
    constexpr int BK = chunk<CPLX>(), MT = BM / (8 * WM), NT = BN / (8 * WN), NP = CPLX ? 2 : 1, NTHR = 32 * WM * WN;
    constexpr int AE = tile_elems<CPLX, BM, TA>(), BE = tile_elems<CPLX, BN, !TB>();
    if (p.stop && *p.stop) return;
    extern __shared__ __align__(16) unsigned char raw[];
    T* ring = reinterpret_cast<T*>(raw);
    const int tm = (p.M + BM - 1) / BM;
    const int m0 = (blockIdx.x % tm) * BM, n0 = (blockIdx.x / tm) * BN, z = blockIdx.y;
    const int S = gridDim.z, rank = blockIdx.z;  // the cluster is the z dimension
    const int herm = p.herm[z];
    if (herm > 0) {
        const int last = min(m0 + BM, p.M) - 1;
        if (m0 / herm == last / herm && m0 % herm > n0 + BN - 1) return;  // below the diagonal: the same for the cluster
    }
    const int k_lo = min(p.K, rank * p.kper), k_hi = min(p.K, k_lo + p.kper);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wm = (warp % WM) * (BM / WM), wn = (warp / WM) * (BN / WN);
    const double *A = p.A[z], *B = p.B[z];

    Sums<NP, MT, NT> acc, runs, total;  // runs: RUN > 0 only, total: THIRD only
    acc.clear();
    runs.clear();
    total.clear();

    constexpr uint32_t STAGE = (AE + BE) * sizeof(T);
    Loader<CPLX, BM, TA, NTHR, VEC> la(ring, A, p.lda, m0, p.M, k_lo);
    Loader<CPLX, BN, !TB, NTHR, VEC> lb(ring + AE, B, p.ldb, n0, p.N, k_lo);
    const int kspan = k_hi - k_lo, nfull = kspan / BK, nk = (kspan + BK - 1) / BK;
    auto load = [&](int t, uint32_t off) {
        if (t < nfull) {
            la.copy(off);
            lb.copy(off);
        } else if (t < nk) {
            la.copy_tail(off, kspan - t * BK);
            lb.copy_tail(off, kspan - t * BK);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int t = 0; t < ST - 1; ++t) load(t, t * STAGE);
    // a conjugate's sign bit: integer work, which leaves the FP64 pipe to the DMMAs
    const int sa = p.conj_a ? 0x80000000 : 0, sb = p.conj_b ? 0x80000000 : 0;
    // this lane's elements of a stage's fragments; the stages of an unrolled turn are immediate offsets
    const int fk = lane & 3, fr = lane >> 2;
    const T* fa = ring + (TA ? (wm + fr) * stride_k<CPLX>() + fk : fk * stride_rows<CPLX, BM>() + wm + fr);
    const T* fb = ring + AE + (TB ? fk * stride_rows<CPLX, BN>() + wn + fr : (wn + fr) * stride_k<CPLX>() + fk);
    auto multiply = [&](int stage) {
#pragma unroll
        for (int k4 = 0; k4 < BK / 4; ++k4) {
            T a[MT], b[NT];
#pragma unroll
            for (int i = 0; i < MT; ++i)
                a[i] = fa[stage * (AE + BE) + (TA ? 8 * i * stride_k<CPLX>() + 4 * k4
                                                  : 4 * k4 * stride_rows<CPLX, BM>() + 8 * i)];
#pragma unroll
            for (int j = 0; j < NT; ++j)
                b[j] = fb[stage * (AE + BE) + (TB ? 4 * k4 * stride_rows<CPLX, BN>() + 8 * j
                                                  : 8 * j * stride_k<CPLX>() + 4 * k4)];
            if constexpr (CPLX) {
#pragma unroll
                for (int i = 0; i < MT; ++i) {
                    const double ai = flip(a[i].y, sa), nai = flip(ai, 0x80000000);
#pragma unroll
                    for (int j = 0; j < NT; ++j) {
                        const double bi = flip(b[j].y, sb);
                        dmma(acc.v[0][i][j], a[i].x, b[j].x);
                        dmma(acc.v[NP - 1][i][j], a[i].x, bi);
                        dmma(acc.v[0][i][j], nai, bi);
                        dmma(acc.v[NP - 1][i][j], ai, b[j].x);
                    }
                }
            } else {
#pragma unroll
                for (int i = 0; i < MT; ++i)
#pragma unroll
                    for (int j = 0; j < NT; ++j) dmma(acc.v[0][i][j], a[i], b[j]);
            }
        }
    };
    for (int t0 = 0; t0 < nk; t0 += ST) {
#pragma unroll
        for (int s = 0; s < ST; ++s) {
            const int t = t0 + s;
            if (t < nk) {
                asm volatile("cp.async.wait_group %0;" ::"n"(ST - 2) : "memory");  // chunk t, this thread's part
                __syncthreads();  // everyone's part, and the stage of chunk t - 1 is free
                load(t + ST - 1, ((s + ST - 1) % ST) * STAGE);
                multiply(s);
                if constexpr (RUN > 0) {
                    if (t % RUN == RUN - 1) {
                        runs.take(acc);
                        if constexpr (THIRD)
                            if (t % (RUN * RUNS) == RUN * RUNS - 1) total.take(runs);
                    }
                }
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if constexpr (RUN > 0) {
        runs.take(acc);
        if constexpr (THIRD) {
            total.take(runs);
            acc = total;
        } else {
            acc = runs;
        }
    }

    // C(i, j) = alpha v + beta C(i, j), and the mirrored element of a Hermitian block
    auto emit = [&](int i, int j, T v) {
        if (i >= p.M || j >= p.N) return;
        int ii = i, base = 0;
        if (herm > 0) {
            base = i / herm * herm;
            ii = i - base;
            if (ii > j) return;  // written by its mirror
        }
        T* C = reinterpret_cast<T*>(p.C[z]);
        T* c = C + i + (long long)j * p.ldc;
        if constexpr (CPLX) {
            double re = p.alpha.x * v.x - p.alpha.y * v.y, im = p.alpha.x * v.y + p.alpha.y * v.x;
            if (!p.beta_zero) {
                const T o = *c;
                re += p.beta.x * o.x - p.beta.y * o.y;
                im += p.beta.x * o.y + p.beta.y * o.x;
            }
            if (herm > 0 && ii == j) im = 0.0;
            *c = make_double2(re, im);
            if (herm > 0 && ii < j) C[base + j + (long long)ii * p.ldc] = make_double2(re, -im);
        } else {
            double o = p.alpha.x * v;
            if (!p.beta_zero) o += p.beta.x * *c;
            *c = o;
            if (herm > 0 && ii < j) C[base + j + (long long)ii * p.ldc] = o;
        }
    };
    auto value = [&](int i, int j, int h) -> T {
        if constexpr (CPLX) return make_double2(acc.v[0][i][j][h], acc.v[NP - 1][i][j][h]);
        else return acc.v[0][i][j][h];
    };
    if (S == 1) {
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int i = 0; i < MT; ++i)
                    emit(m0 + wm + 8 * i + (lane >> 2), n0 + wn + 8 * j + 2 * (lane & 3) + h, value(i, j, h));
        return;
    }
    // the CTA's partial tile, column-major, in the ring's memory; then each CTA of the cluster adds up and
    // writes its part of the tile
    cg::cluster_group cl = cg::this_cluster();
    __syncthreads();
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h)
                ring[wm + 8 * i + (lane >> 2) + (wn + 8 * j + 2 * (lane & 3) + h) * BM] = value(i, j, h);
    cl.sync();
    for (int e = rank * NTHR + threadIdx.x; e < BM * BN; e += S * NTHR) {
        T sum{};
        for (int s = 0; s < S; ++s) {
            const T v = cl.map_shared_rank(ring, s)[e];
            if constexpr (CPLX) {
                sum.x += v.x;
                sum.y += v.y;
            } else {
                sum += v;
            }
        }
        emit(m0 + e % BM, n0 + e / BM, sum);
    }
    cl.sync();  // no CTA leaves while another reads its partial tile
}

template <bool CPLX, int BM, int BN, int WM, int WN, int ST, bool TA, bool TB, bool VEC, int RUN, bool THIRD>
void launch_t(const DgArgs& a, int nz, int split) {
    constexpr int SM = smem_bytes<CPLX, BM, BN, ST, TA, TB>();
    auto kernel = gemm_dmma_kernel<CPLX, BM, BN, WM, WN, ST, TA, TB, VEC, RUN, THIRD>;
    static bool attr = false;
    if (!attr) {
        OMM_CK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SM));
        attr = true;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(((a.M + BM - 1) / BM) * ((a.N + BN - 1) / BN), nz, split);
    cfg.blockDim = dim3(32 * WM * WN);
    cfg.dynamicSmemBytes = SM;
    cfg.stream = rt().stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim = {1, 1, (unsigned)split};
    cfg.attrs = at;
    cfg.numAttrs = split > 1 ? 1 : 0;
    OMM_CK(cudaLaunchKernelEx(&cfg, kernel, a));
    OMM_KCHECK();
}
template <bool CPLX, int BM, int BN, int WM, int WN, int ST, bool VEC, int RUN, bool THIRD>
void launch_ops(const DgArgs& a, bool ta, bool tb, int nz, int split) {
    if (ta && tb) launch_t<CPLX, BM, BN, WM, WN, ST, true, true, VEC, RUN, THIRD>(a, nz, split);
    else if (ta) launch_t<CPLX, BM, BN, WM, WN, ST, true, false, VEC, RUN, THIRD>(a, nz, split);
    else if (tb) launch_t<CPLX, BM, BN, WM, WN, ST, false, true, VEC, RUN, THIRD>(a, nz, split);
    else launch_t<CPLX, BM, BN, WM, WN, ST, false, false, VEC, RUN, THIRD>(a, nz, split);
}

// Split of K by an estimate of the time in SM clocks: the CTAs of the busiest SM in turn, each with a
// fixed cost (start, filling of the ring, and for a split the exchange) and a cost per chunk, which is the
// DMMAs' 256 (complex: 450) clocks and what they leave idle, or the chunk's own latency where a CTA has the
// SM to itself.  Fitted to 15 shapes from 37 x 53 x 61 to 3,000 x 30 x 3,000 (within 15 %).
struct Config {
    int split;
    double us;
};
Config pick(bool cplx, int M, int N, int K, int nz, bool herm, bool wide = true) {
    const double chunk_k = cplx ? 8.0 : 16.0, busy = cplx ? 590.0 : wide ? 315.0 : 405.0, alone = cplx ? 830.0 : 440.0;
    const double tiles = (double)((M + 31) / 32) * ((N + 31) / 32) * nz * (herm ? 0.6 : 1.0);
    Config best{1, 1e300};
    for (int s = 1; s <= 8; s *= 2) {
        if (s > 1 && K < 48 * s) break;
        const double chunks = std::ceil(K / (s * chunk_k)), turns = std::ceil(tiles * s / 148.0);
        const double fixed = s > 1 ? 2400.0 : 900.0;
        const double clocks = std::max(turns * (fixed + chunks * busy), fixed + chunks * alone);
        const double us = 4.0 + clocks / 1850.0;
        if (us < 0.97 * best.us) best = Config{s, us};
    }
    return best;
}

}  // namespace

// Products cuBLAS has the better split for, left to it where the emulation never took them (a call, microseconds,
// cuBLAS / this kernel): complex ones with a long K (64 x 64 x 3,000 27 / 37, 64 x 3,000 x 3,000 160 / 208; with
// more than 32 tiles from K = 1,000 on: 300 x 150 x 1,000 34 / 40, 257 x 259 x 1,001 43 / 49; 64 x 200 x 1,300
// leads with 24 / 25), and real ones of one or two rows of tiles with a long K (64 x 3,000 x 3,000 59 / 64; 100 x
// 1,000 x 3,000 47 / 50, 130 x 260 x 3,000 32 / 29).  Complex ones large enough for the emulation to be had
// (fp64_emu_fits) take it or this kernel although cuBLAS is faster (300 x 150 x 3,000 61 / 80, 130 x 700 x 2,000
// 73 / 102): cuBLAS's rounding error there is 7.0e-16, this kernel's 2.5e-16, the emulation's below 1e-16.
bool gemm_dmma_slower(bool cplx, int M, int N, int K) {
    if (!cplx) return K >= 2500 && std::min(M, N) <= 64 && std::max(M, N) >= 1500;
    if (fp64_emu_fits(M, N, K)) return false;
    return K >= 1500 || (K >= 1000 && ((M + 31) / 32) * (long long)((N + 31) / 32) > 32);
}

double gemm_dmma_us(bool cplx, int M, int N, int K, int nz, bool wide) { return pick(cplx, M, N, K, nz, false, wide).us; }

bool gemm_dmma_takes(const DView& v) { return v.is_real || (reinterpret_cast<uintptr_t>(v.p) & 15) == 0; }

void gemm_dmma(char opA, char opB, int M, int N, int K, const double alpha[2], const DView* A, const DView* B,
               const double beta[2], DView* C, int nz, const int* herm, const int* stop) {
    if (M == 0 || N == 0) return;
    const bool cplx = !C[0].is_real;
    auto code = [](char o) { return o == 'n' || o == 'N' ? 0 : o == 't' || o == 'T' ? 1 : 2; };
    const bool ta = code(opA) != 0, tb = code(opB) != 0;
    DgArgs a{};
    a.M = M;
    a.N = N;
    a.K = K;
    a.stop = stop;
    a.lda = A[0].ld;
    a.ldb = B[0].ld;
    a.ldc = C[0].ld;
    a.alpha = {alpha[0], cplx ? alpha[1] : 0.0};
    a.beta = {beta[0], cplx ? beta[1] : 0.0};
    a.beta_zero = a.beta.x == 0.0 && a.beta.y == 0.0;
    a.conj_a = cplx && code(opA) == 2;
    a.conj_b = cplx && code(opB) == 2;
    a.vec = a.lda % 2 == 0 && a.ldb % 2 == 0;
    bool any = false;
    for (int z = 0; z < nz; ++z) {
        a.A[z] = A[z].as<double>();
        a.B[z] = B[z].as<double>();
        a.C[z] = C[z].as<double>();
        a.vec = a.vec && (reinterpret_cast<uintptr_t>(A[z].p) & 15) == 0 && (reinterpret_cast<uintptr_t>(B[z].p) & 15) == 0;
        a.herm[z] = herm ? herm[z] : 0;
        any = any || a.herm[z] > 0;
        if (A[z].ld != A[0].ld || B[z].ld != B[0].ld || C[z].ld != C[0].ld)
            fail(OMM_ERR_ARG, "gemm_dmma: the products of one launch share their leading dimensions");
    }
    const Config c = pick(cplx, M, N, K, nz, any && nz == 1);
    const int bk = cplx ? 8 : 16;
    a.kper = std::max(bk, ((K + c.split - 1) / c.split + bk - 1) / bk * bk);
    auto launch = [&](auto run, auto third) {
        constexpr int RUN = decltype(run)::value;
        constexpr bool THIRD = decltype(third)::value;
        if (cplx) launch_ops<true, 32, 32, 2, 2, 2, true, RUN, (RUN > 0)>(a, ta, tb, nz, c.split);
        else if (a.vec) launch_ops<false, 32, 32, 2, 2, 3, true, RUN, THIRD>(a, ta, tb, nz, c.split);
        else launch_ops<false, 32, 32, 2, 2, 3, false, RUN, THIRD>(a, ta, tb, nz, c.split);
    };
    // At most 64 real products or 16 complex ones are one chain: as accurate as cuBLAS's, and the sums cost
    // registers (3,000 x 3,000 x 16 38 us, 44 with all three).  Runs of 32 where the emulation was had before this
    // kernel (fp64_emu_fits), whose 2.0e-16 to 2.5e-16 they keep, and for short complex products (37 x 53 x 61
    // 2.1e-16 as cuBLAS, in runs of 64 2.6e-16); elsewhere cuBLAS's 3.4e-16 to 7e-16 are the measure, and runs of 64
    // do: 500^3 24.0 -> 24.4 us, 7.1e-16 -> 2.8e-16; complex 51 -> 52, 1.0e-15 -> 2.9e-16; 256 x 128 x 832 18.3 us
    // either way, 4.7e-16 -> 2.8e-16.  The third level's registers let five CTAs of a
    // real product share an SM: where a few more are to be run, and at most 32 runs, two levels are faster (900^3,
    // 841 CTAs, 72 us against 85, 65 in one chain; 1,100 x 900 x 700, 1,015, 67 against 72), elsewhere slower
    // (1,500 x 800 x 300, 1,175, 47 against 41; 512 x 512 x 4,096 118 against 99).
    const long long ctas = (long long)((M + 31) / 32) * ((N + 31) / 32) * nz;
    const bool crowded = !cplx && c.split == 1 && ctas > 148 * 5 && ctas <= 148 * 7 && a.kper <= 1024;
    if (a.kper <= (cplx ? 16 : 64)) launch(std::integral_constant<int, 0>{}, std::false_type{});
    else if (!fp64_emu_fits(M, N, K) && !(cplx && K <= 128)) launch(std::integral_constant<int, 4>{}, std::true_type{});
    else if (crowded) launch(std::integral_constant<int, 2>{}, std::false_type{});
    else launch(std::integral_constant<int, 2>{}, std::true_type{});
}

}  // namespace ommgpu
