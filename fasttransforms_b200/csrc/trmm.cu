// Triangular multiplies of the connection stage, FP64 on the tensor pipe.
//
// The reference applies its dense upper-triangular connection matrices with
// cblas_dtrmm, in place (src/drivers.c:836-863, 924-956, 992-1019).  Here the
// product is computed out of place, Out = op(U) * In (left) or Out = In * op(U)
// (right), as a tiled GEMM with mma.sync.m8n8k4.f64 (DMMA) whose K loop only
// visits the nonzero triangle.  Up to four column classes (the stride-4N
// classes of sph / disk, each with its own U) share one launch.
//
// Three tile shapes (TileShape), chosen per launch by trmm_shape: 128 x 64 outputs with 8 warps of
// 32 x 32 where the tiles fill the chip several times over, 64 x 64 with 4 such warps where they do
// not, 32 x 32 with 4 warps of 16 x 16 for the smallest.  K slabs of 16 are staged in shared memory
// by a cp.async pipeline; the layouts are padded so every fragment load is conflict-free.
//
// Summation: the accumulators sum one chunk of 256 consecutive k (k / 256 equal) at a time; at the
// end of each chunk a thread adds them into its outputs in C (which it alone writes) and starts the
// next chunk from zero.  The additions are reductions at L2: reading the sums back held the warps for
// a round trip every 16 slabs (sph degree 4095 4752 -> 4511 us, 2047 630 -> 594).  A single
// accumulation over all n terms lets the rounding error grow with n; chunked sums, like a BLAS's K
// panels, keep it near that of 256 terms plus n / 256 additions (the reference's round trips, which
// amplify this error in the ill-conditioned triangle transforms, then match its BLAS build).  The
// chunks do not depend on the tile, so every shape gives the same bits.  C must not alias the inputs
// (every caller multiplies out of place).

#include <algorithm>
#include <atomic>
#include <vector>

#include "ft_internal.h"

namespace ftb {

void trmm_tile(int shape, int * rows, int * cols) {
    static const int r[3] = {128, 64, 32}, c[3] = {64, 64, 32};
    *rows = r[shape];
    *cols = c[shape];
}

// A launch takes about its slabs' time over the SMs plus the tail in which the longest tiles run
// alone, which is where the smaller tiles win: they are more and shorter, but load more per flop.
// Per slab of 16 k, in us: with the chip full, 1.18, 0.62 and 0.18 (128 x 64, 64 x 64, 32 x 32: 30.5,
// 30.0 and 25.7 TFLOP/s at sph degree 4095; 0.20 with odd n, whose copies are single doubles); of the
// longest tile, 0.75, 0.5 and 0.25.  Measured per launch (us; 128 x 64 / 64 x 64 / 32 x 32): sph 64
// 13 / 11 / 8, 301 40 / 29 / 16, 512 54 / 37 / 25, 1024 127 / 106 / 97, 1501 291 / 282 / 345, 2048
// 604 / 595 / 688, 4096 4515 / 4598 / 5371; tri 1001 115 / 89 / 66, 2048 321 / 313 / 340.
int trmm_shape(const std::vector<TrmmExtent> & x) {
    static const double full[3] = {1.18, 0.623, 0.184}, tail[3] = {0.75, 0.5, 0.25};
    int best = 0;
    double least = 0.0;
    for (int s = 0; s < 3; ++s) {
        int bm, bn;
        trmm_tile(s, &bm, &bn);
        double slabs = 0.0, longest = 0.0;
        for (const TrmmExtent & e : x) {
            const int tm = (e.mrows + bm - 1) / bm, tn = (e.ncols + bn - 1) / bn;
            // a tile's K runs from its place on the diagonal to the matrix's end: half of it on average
            slabs += 0.5 * tm * tn * (e.n + (e.mode < 2 ? bm : bn)) / 16.0 * (s == 2 && e.n % 2 ? 1.1 : 1.0);
            longest = std::max(longest, e.n / 16.0);
        }
        const double t = slabs * full[s] / 148.0 + longest * tail[s];
        if (s == 0 || t < least) { least = t; best = s; }
    }
    return best;
}

namespace {

constexpr int BK = 16;
constexpr int KCHUNK = 256;   // consecutive k summed before a partial sum is added into C

template <int S> struct TileShape;
template <> struct TileShape<0> { static constexpr int BM = 128, BN = 64, WM = 32, WN = 32, STAGES = 3, CTAS = 2; };
template <> struct TileShape<1> { static constexpr int BM = 64, BN = 64, WM = 32, WN = 32, STAGES = 3, CTAS = 3; };
template <> struct TileShape<2> { static constexpr int BM = 32, BN = 32, WM = 16, WN = 16, STAGES = 4, CTAS = 5; };

template <int S, bool A_MC, bool B_KC>
struct TileLayout : TileShape<S> {
    using T = TileShape<S>;
    static constexpr int THREADS = 32 * (T::BM / T::WM) * (T::BN / T::WN);
    static constexpr int FA = T::WM / 8, FB = T::WN / 8;             // fragments of a warp
    static constexpr int LDA = A_MC ? T::BM + 4 : BK + 4;            // [k][m] or [m][k]
    static constexpr int LDB = B_KC ? BK + 4 : T::BN + 4;            // [n][k] or [k][n]
    static constexpr int ASZ = A_MC ? BK * LDA : T::BM * LDA;
    static constexpr int BSZ = B_KC ? T::BN * LDB : BK * LDB;
    static constexpr size_t bytes = sizeof(double) * T::STAGES * (ASZ + BSZ);
};

__device__ __forceinline__ void cp_async16(void * smem, const void * gmem, bool valid) {
    unsigned sa = (unsigned) __cvta_generic_to_shared(smem);
    int sz = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" :: "r"(sa), "l"(gmem), "r"(sz));
}
__device__ __forceinline__ void cp_async8(void * smem, const void * gmem, bool valid) {
    unsigned sa = (unsigned) __cvta_generic_to_shared(smem);
    int sz = valid ? 8 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" :: "r"(sa), "l"(gmem), "r"(sz));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;\n" :: "n"(N)); }

__device__ __forceinline__ void dmma(double & d0, double & d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(d0), "+d"(d1) : "d"(a), "d"(b));
}

// Operand descriptions.  A(m, k) = a[m * a_sm + k * a_sk]; B(k, n) = b[k * b_sk + n * b_sn].
// A_MC: A contiguous in m (a_sm == 1), else in k.  B_KC: B contiguous in k, else in n.
// Triangle: TRI_SIDE 0 = A is the triangular operand, 1 = B is.
struct GemmClass {
    const double * a; const double * b; double * c;
    long long a_ld, b_ld, c_ld;   // leading dims (the non-unit stride of each operand / of C)
    int mrows, ncols;
};
struct GemmParams {
    GemmClass cls[4];
    int nclasses;
    int n;              // order of the triangular matrix (also the K extent)
    int tiles_m, tiles_n;
    int mode;           // 0: left N (k >= i), 1: left T (k <= i), 2: right N (k <= j), 3: right T (k >= j)
};

// A thread's accumulators (rows m0 + 8a, columns n0 + 8b + {0, 1}) into C: C = acc (first chunk) or
// C + acc (a reduction, which the thread does not wait for; only this thread adds to its outputs, so
// the order of the additions is its own), then acc = 0 when more chunks follow.
__device__ __forceinline__ void add_to(double * p, double v) {
    asm volatile("red.relaxed.gpu.global.add.f64 [%0], %1;\n" :: "l"(p), "d"(v) : "memory");
}
template <int FA, int FB>
__device__ __forceinline__ void flush_partial(const GemmClass & C, const int m0, const int n0, double (&acc)[FA][FB][2],
                                              const bool add, const bool restart) {
#pragma unroll
    for (int a = 0; a < FA; ++a) {
        const int m = m0 + a * 8;
#pragma unroll
        for (int b = 0; b < FB; ++b) {
            const int nn = n0 + b * 8;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (m < C.mrows && nn + h < C.ncols) {
                    double * const p = C.c + (long long) (nn + h) * C.c_ld + m;
                    if (add) add_to(p, acc[a][b][h]); else *p = acc[a][b][h];
                }
                if (restart) acc[a][b][h] = 0.0;
            }
        }
    }
}

// One output tile of class C: rows [tm*BM, ...), columns [tn*BN, ...).
template <int S, bool A_MC, bool B_KC, bool VEC16>
__device__ __forceinline__ void tri_tile(const GemmClass & C, const int n, const int mode, const int tm, const int tn) {
    using T = TileLayout<S, A_MC, B_KC>;
    constexpr int BM = T::BM, BN = T::BN, NSTAGE = T::STAGES, NTHREADS = T::THREADS, FA = T::FA, FB = T::FB, LDA = T::LDA, LDB = T::LDB,
                  ASZ = T::ASZ, BSZ = T::BSZ;
    extern __shared__ double sm[];
    double * As = sm;
    double * Bs = sm + NSTAGE * ASZ;
    const int i0 = tm * BM, j0 = tn * BN;
    if (i0 >= C.mrows || j0 >= C.ncols) return;
    int klo, khi;
    if (mode == 0)      { klo = i0; khi = n; }
    else if (mode == 1) { klo = 0; khi = min(i0 + BM, n); }
    else if (mode == 2) { klo = 0; khi = min(j0 + BN, n); }
    else                { klo = j0; khi = n; }
    klo = (klo / BK) * BK;
    const int nslab = (khi - klo + BK - 1) / BK;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int wm = warp / (BN / T::WN) * T::WM, wn = warp % (BN / T::WN) * T::WN;

    auto load_slab = [&](int slab, int stage) {
        const int k0 = klo + slab * BK;
        double * as = As + stage * ASZ;
        double * bs = Bs + stage * BSZ;
        if (VEC16) {
            // A: BM * BK doubles, in pairs
#pragma unroll
            for (int r = 0; r < (BM * BK / 2) / NTHREADS; ++r) {
                const int p = r * NTHREADS + tid;
                int m, k;
                if (A_MC) { k = p / (BM / 2); m = (p % (BM / 2)) * 2; }
                else      { m = p / (BK / 2); k = (p % (BK / 2)) * 2; }
                const int gm = i0 + m, gk = k0 + k;
                const bool ok = gm < C.mrows && gk < n;
                const double * g = A_MC ? C.a + (long long) gk * C.a_ld + gm : C.a + (long long) gm * C.a_ld + gk;
                double * s = A_MC ? as + k * LDA + m : as + m * LDA + k;
                cp_async16(s, ok ? g : C.a, ok);
            }
#pragma unroll
            for (int r = 0; r < (BK * BN / 2) / NTHREADS; ++r) {
                const int p = r * NTHREADS + tid;
                int k, nn;
                if (B_KC) { nn = p / (BK / 2); k = (p % (BK / 2)) * 2; }
                else      { k = p / (BN / 2); nn = (p % (BN / 2)) * 2; }
                const int gk = k0 + k, gn = j0 + nn;
                const bool ok = gk < n && gn < C.ncols;
                const double * g = B_KC ? C.b + (long long) gn * C.b_ld + gk : C.b + (long long) gk * C.b_ld + gn;
                double * s = B_KC ? bs + nn * LDB + k : bs + k * LDB + nn;
                cp_async16(s, ok ? g : C.b, ok);
            }
        } else {
#pragma unroll
            for (int r = 0; r < (BM * BK) / NTHREADS; ++r) {
                const int p = r * NTHREADS + tid;
                int m, k;
                if (A_MC) { k = p / BM; m = p % BM; }
                else      { m = p / BK; k = p % BK; }
                const int gm = i0 + m, gk = k0 + k;
                const bool ok = gm < C.mrows && gk < n;
                const double * g = A_MC ? C.a + (long long) gk * C.a_ld + gm : C.a + (long long) gm * C.a_ld + gk;
                double * s = A_MC ? as + k * LDA + m : as + m * LDA + k;
                cp_async8(s, ok ? g : C.a, ok);
            }
#pragma unroll
            for (int r = 0; r < (BK * BN) / NTHREADS; ++r) {
                const int p = r * NTHREADS + tid;
                int k, nn;
                if (B_KC) { nn = p / BK; k = p % BK; }
                else      { k = p / BN; nn = p % BN; }
                const int gk = k0 + k, gn = j0 + nn;
                const bool ok = gk < n && gn < C.ncols;
                const double * g = B_KC ? C.b + (long long) gn * C.b_ld + gk : C.b + (long long) gk * C.b_ld + gn;
                double * s = B_KC ? bs + nn * LDB + k : bs + k * LDB + nn;
                cp_async8(s, ok ? g : C.b, ok);
            }
        }
    };

    double acc[FA][FB][2];
#pragma unroll
    for (int a = 0; a < FA; ++a)
#pragma unroll
        for (int b = 0; b < FB; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;
    bool flushed = false;   // C holds the sum of the chunks before the current one

#pragma unroll
    for (int s = 0; s < NSTAGE - 1; ++s) {
        if (s < nslab) load_slab(s, s);
        cp_commit();
    }
    const int fr = lane >> 2, fc = lane & 3;   // fragment row (m or n) and k index
    for (int slab = 0; slab < nslab; ++slab) {
        cp_wait<NSTAGE - 2>();
        __syncthreads();
        {
            const int nxt = slab + NSTAGE - 1;
            if (nxt < nslab) load_slab(nxt, nxt % NSTAGE);
            cp_commit();
        }
        const double * as = As + (slab % NSTAGE) * ASZ;
        const double * bs = Bs + (slab % NSTAGE) * BSZ;
#pragma unroll
        for (int kk = 0; kk < BK; kk += 4) {
            double af[FA], bf[FB];
#pragma unroll
            for (int a = 0; a < FA; ++a) {
                const int m = wm + a * 8 + fr, k = kk + fc;
                af[a] = A_MC ? as[k * LDA + m] : as[m * LDA + k];
            }
#pragma unroll
            for (int b = 0; b < FB; ++b) {
                const int nn = wn + b * 8 + fr, k = kk + fc;
                bf[b] = B_KC ? bs[nn * LDB + k] : bs[k * LDB + nn];
            }
#pragma unroll
            for (int a = 0; a < FA; ++a)
#pragma unroll
                for (int b = 0; b < FB; ++b) dmma(acc[a][b][0], acc[a][b][1], af[a], bf[b]);
        }
        if ((klo + (slab + 1) * BK) % KCHUNK == 0 && slab + 1 < nslab) {   // end of a chunk: into C, restart from zero
            flush_partial(C, i0 + wm + fr, j0 + wn + fc * 2, acc, flushed, true);
            flushed = true;
        }
    }
    cp_wait<0>();

    // epilogue: C(m, n) at c[n * c_ld + m] (plus the earlier chunks' sum)
    flush_partial(C, i0 + wm + fr, j0 + wn + fc * 2, acc, flushed, false);
}

template <int S, bool A_MC, bool B_KC, bool VEC16>
__global__ void __launch_bounds__(TileLayout<S, A_MC, B_KC>::THREADS, TileShape<S>::CTAS)
gemm_tri_kernel(const __grid_constant__ GemmParams P) {
    allow_next();
    wait_for_previous();
    // block -> (tile along the triangle, class, other tile): tiles with the most K work first,
    // whatever their class
    const int along = P.mode < 2 ? P.tiles_m : P.tiles_n, across = P.mode < 2 ? P.tiles_n : P.tiles_m;
    int t = blockIdx.x / (P.nclasses * across);
    const int rest = blockIdx.x % (P.nclasses * across), cl = rest / across, x = rest % across;
    if (P.mode == 1 || P.mode == 2) t = along - 1 - t;   // long K at large i (j); else at small i (j)
    tri_tile<S, A_MC, B_KC, VEC16>(P.cls[cl], P.n, P.mode, P.mode < 2 ? t : x, P.mode < 2 ? x : t);
}

// Batched multiplies over many fields: the tile list (longest K first) and the
// pointer-free class table live in device memory; pointers come by value.
// MODE 0/1: left, op(U) = U / U^T; MODE 2/3: right, op(U) = U / U^T.
template <int S, int MODE, bool VEC16>
__global__ void __launch_bounds__(TileLayout<S, MODE != 1, MODE != 3>::THREADS, TileShape<S>::CTAS)
gemm_tri_batched_kernel(const __grid_constant__ TrmmBatch P) {
    allow_next();
    wait_for_previous();
    const TrmmTile t = P.tiles[blockIdx.x];
    const TrmmBatchClass c = P.classes[t.cls];
    GemmClass C;
    const double * X = P.in[c.field] + (long long) c.r * c.n;
    const double * U = P.U[c.field][c.u];
    C.c = P.out[c.field] + (long long) c.r * c.n;
    C.c_ld = c.ld;
    C.mrows = c.mrows;
    C.ncols = c.ncols;
    if (MODE < 2) { C.a = U; C.a_ld = c.n; C.b = X; C.b_ld = c.ld; }
    else          { C.a = X; C.a_ld = c.ld; C.b = U; C.b_ld = c.n; }
    tri_tile<S, MODE != 1, MODE != 3, VEC16>(C, c.n, MODE, t.tm, t.tn);
}

// One launch; the kernel's shared-memory limit is raised once per device.
template <class P>
cudaError_t launch_tiles(void (*kern)(P), const P & p, int blocks, int threads, size_t shm, std::atomic<unsigned> & ready, cudaStream_t st) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const unsigned bit = dev < 32 ? 1u << dev : 0u;
    if (!(ready.load(std::memory_order_acquire) & bit)) {
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) shm);
        if (e != cudaSuccess) return e;
        ready.fetch_or(bit, std::memory_order_release);
    }
    count_launch();
    return launch_overlapped(kern, dim3(blocks), threads, shm, st, p);
}

template <int S, int MODE, bool VEC16>
cudaError_t run_batched(const TrmmBatch & P, int ntiles, cudaStream_t st) {
    using T = TileLayout<S, MODE != 1, MODE != 3>;
    static std::atomic<unsigned> ready{0};
    return launch_tiles(gemm_tri_batched_kernel<S, MODE, VEC16>, P, ntiles, T::THREADS, T::bytes, ready, st);
}
template <int MODE>
cudaError_t run_batched(const TrmmBatch & P, int ntiles, bool vec16, int shape, cudaStream_t st) {
    if (shape == 0) return vec16 ? run_batched<0, MODE, true>(P, ntiles, st) : run_batched<0, MODE, false>(P, ntiles, st);
    if (shape == 1) return vec16 ? run_batched<1, MODE, true>(P, ntiles, st) : run_batched<1, MODE, false>(P, ntiles, st);
    return vec16 ? run_batched<2, MODE, true>(P, ntiles, st) : run_batched<2, MODE, false>(P, ntiles, st);
}

template <int S, bool A_MC, bool B_KC, bool VEC16>
cudaError_t run_gemm(GemmParams P, int rows, int cols, cudaStream_t st) {
    using T = TileLayout<S, A_MC, B_KC>;
    P.tiles_m = (rows + T::BM - 1) / T::BM;
    P.tiles_n = (cols + T::BN - 1) / T::BN;
    const int blocks = P.nclasses * P.tiles_m * P.tiles_n;
    if (blocks == 0) return cudaSuccess;
    static std::atomic<unsigned> ready{0};
    return launch_tiles(gemm_tri_kernel<S, A_MC, B_KC, VEC16>, P, blocks, T::THREADS, T::bytes, ready, st);
}
template <bool A_MC, bool B_KC>
cudaError_t run_gemm(const GemmParams & P, int rows, int cols, bool vec16, cudaStream_t st) {
    std::vector<TrmmExtent> x;
    for (int c = 0; c < P.nclasses; ++c) x.push_back({P.cls[c].mrows, P.cls[c].ncols, P.n, P.mode});
    const int shape = trmm_shape(x);
    if (shape == 0) return vec16 ? run_gemm<0, A_MC, B_KC, true>(P, rows, cols, st) : run_gemm<0, A_MC, B_KC, false>(P, rows, cols, st);
    if (shape == 1) return vec16 ? run_gemm<1, A_MC, B_KC, true>(P, rows, cols, st) : run_gemm<1, A_MC, B_KC, false>(P, rows, cols, st);
    return vec16 ? run_gemm<2, A_MC, B_KC, true>(P, rows, cols, st) : run_gemm<2, A_MC, B_KC, false>(P, rows, cols, st);
}

inline bool aligned16(const void * p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

struct NormLaunch {
    double * A[kMaxFields];
    int N[kMaxFields], M[kMaxFields];
};
__global__ void cheb_norm_kernel(const __grid_constant__ NormLaunch L, double r, double g) {
    allow_next();
    wait_for_previous();
    // src/drivers.c:6-24: first column and first row scaled by r (entry (0,0) twice), all by g
    double * const A = L.A[blockIdx.y];
    const int N = L.N[blockIdx.y];
    const long long total = (long long) N * L.M[blockIdx.y];
    for (long long e = blockIdx.x * (long long) blockDim.x + threadIdx.x; e < total; e += (long long) gridDim.x * blockDim.x) {
        double v = A[e];
        if (e < N) v *= r;
        if (e % N == 0) v *= r;
        A[e] = v * g;
    }
}

}  // namespace

cudaError_t launch_trmm(const TrmmLaunch & L, cudaStream_t st) {
    GemmParams P{};
    P.nclasses = L.nclasses;
    P.n = L.n;
    int maxcols = 0;
    bool vec = (L.n % 2 == 0) && (L.ld_in % 2 == 0);
    for (int c = 0; c < L.nclasses; ++c) {
        GemmClass & g = P.cls[c];
        g.a = L.cls[c].U; g.b = L.cls[c].in; g.c = L.cls[c].out;
        g.a_ld = L.n; g.b_ld = L.ld_in; g.c_ld = L.ld_out;
        g.mrows = L.n; g.ncols = L.cls[c].ncols;
        maxcols = std::max(maxcols, g.ncols);
        vec = vec && aligned16(g.a) && aligned16(g.b);
    }
    P.mode = L.trans ? 1 : 0;
    return L.trans ? run_gemm<false, true>(P, L.n, maxcols, vec, st) : run_gemm<true, true>(P, L.n, maxcols, vec, st);
}

cudaError_t launch_trmm_batched(const TrmmBatch & P, int ntiles, bool vec16, int mode, int shape, cudaStream_t st) {
    if (ntiles == 0) return cudaSuccess;
    switch (mode) {
        case 0: return run_batched<0>(P, ntiles, vec16, shape, st);
        case 1: return run_batched<1>(P, ntiles, vec16, shape, st);
        case 2: return run_batched<2>(P, ntiles, vec16, shape, st);
        case 3: return run_batched<3>(P, ntiles, vec16, shape, st);
    }
    return cudaErrorInvalidValue;
}


cudaError_t launch_trmm_right(const double * U, const double * in, double * out, int n, int nrows,
                              long long ld, bool trans, cudaStream_t st) {
    // Out(row, j) = sum_k In(row, k) op(U)(k, j): A = In (contiguous in rows), B = op(U)
    GemmParams P{};
    P.nclasses = 1;
    P.n = n;
    GemmClass & g = P.cls[0];
    g.a = in; g.b = U; g.c = out;
    g.a_ld = ld; g.b_ld = n; g.c_ld = ld;
    g.mrows = nrows; g.ncols = n;
    P.mode = trans ? 3 : 2;
    const bool vec = (n % 2 == 0) && (ld % 2 == 0) && aligned16(in) && aligned16(U);
    // op(U) = U: B(k, j) = U[k + j n] contiguous in k; op(U) = U^T: B(k, j) = U[j + k n] contiguous in j
    return trans ? run_gemm<true, false>(P, nrows, n, vec, st) : run_gemm<true, true>(P, nrows, n, vec, st);
}

cudaError_t launch_cheb_normalize(double * const * A, const int * N, const int * M, int nf, bool transposed, cudaStream_t st) {
    const double r = transposed ? 1.41421356237309504880 : 0.70710678118654752440;   // M_SQRT2, M_SQRT1_2
    const double g = transposed ? 1.57079632679489661923 : 0.63661977236758134308;   // M_PI_2, M_2_PI
    static thread_local NormLaunch L;
    long long most = 0;
    for (int f = 0; f < nf; ++f) {
        L.A[f] = A[f];
        L.N[f] = N[f];
        L.M[f] = M[f];
        most = std::max(most, (long long) N[f] * M[f]);
    }
    // four elements a thread, up to four CTAs per SM over all fields
    const int blocks = (int) std::max(1LL, std::min((most + 1023) / 1024, (long long) (592 / nf + 1)));
    count_launch();
    return launch_overlapped(cheb_norm_kernel, dim3(blocks, nf), 256, 0, st, L, r, g);
}

}  // namespace ftb
