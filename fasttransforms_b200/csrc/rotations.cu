// Givens-rotation sweeps (hi2lo / lo2hi) for the sph, tri and disk families on
// sm_100a, in FP64 with the reference's FMA arithmetic:
//   hi2lo: x' = fma(c, x, s*y),  y' = fma(c, y, -(s*x))
//   lo2hi: x' = fma(c, x, -(s*y)), y' = fma(c, y, s*x)
// (src/rotations/rotations_AVX512F.c:4-15; x is row k, y is row k+d).
//
// Two kernels apply them, each element meeting its rotations in the same order, so that every launch
// shape gives the same bits.
//
// rot_kernel: columns streamed from global memory
// -----------------------------------------------
// A task is a group of columns that receive the same sweeps (sph: 16 orders of one parity, cos and
// sin column each; disk: 32 orders of one parity, cos and sin each; tri: 32 consecutive orders).
// Orders in a group differ, so a sweep j is applied to the columns whose order m satisfies
// j <= m - STEP and is an exact no-op (sin 0, cos 1) for the others.  Tasks, or single passes of
// W x B sweeps of a task (the pass pipeline), are pulled from a queue by persistent CTAs.
//
// Inside a CTA the sweeps of a pass run as a wavefront.  Warp q (a "stage") owns B consecutive
// sweeps.  Each lane owns one chain of the columns of one order and keeps, per column, a window of
// 2B consecutive chain positions in registers.  At every step the window slides by one position:
// one element enters, B independent rotations are applied (sweep b at window slots 2b, 2b+1), one
// element leaves, into a ring in shared memory that the next stage reads.  A loading warp copies
// chunks of E positions from global memory into the first ring (cp.async), a storing warp writes
// the last ring back, so one pass reads and writes each column once.  The lanes that carry the same
// chain use the same (sin, cos) pair at each rotation, read as a broadcast 16-byte shared-memory
// load; a stage's pairs of a chunk are contiguous in a skewed copy of the table (Geo::skew_at) and
// arrive by one bulk copy a few chunks ahead.
//
// Warps meet only through mbarriers per ring slot, and every warp goes on to the next pass or queue
// entry by itself: the stages never drain between passes.  What bounds the kernel: the FP64 pipe
// (4 instructions a rotation, 2 cycles each on a sub-partition; the inner step alone, without
// global traffic, reaches 80 % of it) and, next, instruction fetch.  The unrolled steps are 21 KB
// of code (16 steps of 8 sweeps on 2 columns), which the stages run at different places at the
// same time: with unrolled loading and storing loops beside them (register staging, about 50 KB in
// all) the instruction cache missed and the launch took 10.8 ms at sph degree 4095; with the
// compact loops 7.97 ms (9.8 ms for the former kernel, whose stages met at a barrier per chunk).
//
// rot_resident_kernel: columns resident in shared memory
// ------------------------------------------------------
// For chains that fit; see there.
//
// Every wait is bounded, after which the launch leaves a status to report and its other waits end at
// once; later launches start afresh.  Every global access is bounds-checked against the field's N, M.

#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <type_traits>

#include <map>
#include <mutex>
#include <tuple>
#include <string>

#include "ft_internal.h"
#include "tc05.h"

namespace ftb {
namespace {

// NC: sequences a lane carries, all those of an order (1 or 2) or one.
constexpr int order_sequences(int kind) { return kind == TRI || kind == RECT ? 1 : 2; }
template <int KIND, int NC = order_sequences(KIND)>
struct KT {
    static constexpr int CH = (KIND == SPH || KIND == SPIN || KIND == RECT) ? 2 : 1;   // chains per column
    static constexpr int STEP = KIND == TRI ? 1 : 2;      // order step between sweeps
    // sequences per order sharing the rotations: cos, sin columns (sph, disk), the column
    // (tri, rect), or the real and imaginary parts of the column of -m or of m (spin)
    static constexpr int SEQ = order_sequences(KIND);
    static constexpr int NCOL = NC;
    static constexpr int ES = KIND == SPIN ? 2 : 1;       // doubles per element (interleaved complex)
    static constexpr int ORD = 32 * NC / (CH * SEQ);      // orders per group of 32 lanes
    static constexpr int COLS = ORD * SEQ;                // sequences of those, both chains as one
    // a step's elements in a ring: lanes with all sequences read theirs next to each other, chain by
    // chain; lanes with one sequence read element [lane]
    static constexpr int CPAD = COLS + 1;
    static constexpr int ROWD = NC == SEQ ? CH * CPAD : 33;
    __host__ __device__ static constexpr int place(int c, int cl) { return NC == SEQ ? c * CPAD + cl : cl * CH + c; }
    __host__ __device__ static constexpr int lane_order(int lane) { return NC == SEQ ? lane / CH : lane / (CH * SEQ); }
    __host__ __device__ static constexpr int lane_place(int lane) { return NC == SEQ ? lane % CH * CPAD + lane / CH * NC : lane; }
};

// Builds the skewed table (Geo::skew_at): CTA (beta, p) fills block beta of parity p.
__global__ void skew_table_kernel(const double2 * __restrict__ sc, double2 * __restrict__ out, int kind, int N) {
    const int beta = blockIdx.x, p = blockIdx.y, ch = Geo::chains(kind);
    if (beta >= Geo::skew_blocks(kind, N, p)) return;
    double2 * const block = out + Geo::skew_at(kind, N, p, beta);
    const int row_len = Geo::kSkewLen * ch, chunk = Geo::kSkewRows * row_len;
    const int total = (Geo::skew_chunks(kind, N, p, beta) + 1) * chunk;
    for (int e = threadIdx.x; e < total; e += blockDim.x) {
        const int kappa = e / chunk, i = (e % chunk) / row_len, jj = e % row_len;
        const int j = p + Geo::step(kind) * (Geo::kSkewRows * beta + i);
        const int pos = Geo::kSkewLen * kappa - 2 - 2 * i + jj / ch, c = jj % ch;
        const bool rotates = j < Geo::table_cols(kind, N) && pos >= 0 && pos <= Geo::top(kind, N, j, c);
        block[e] = rotates ? sc[Geo::table_base(kind, N, j) + ch * pos + c] : make_double2(0.0, 1.0);
    }
}

__device__ __forceinline__ void rot_hi2lo(double & x, double & y, double s, double c) {
    const double sy = __dmul_rn(s, y), sx = __dmul_rn(s, x);
    const double xn = __fma_rn(c, x, sy);
    const double yn = __fma_rn(c, y, -sx);
    x = xn; y = yn;
}
__device__ __forceinline__ void rot_lo2hi(double & x, double & y, double s, double c) {
    const double sy = __dmul_rn(s, y), sx = __dmul_rn(s, x);
    const double xn = __fma_rn(c, x, -sy);
    const double yn = __fma_rn(c, y, sx);
    x = xn; y = yn;
}

// Report word of the rotation kernels: nonzero once a bounded wait ran out (that launch's output is
// not valid).  Read and replaced by rotation_status(); no wait looks at it, so a launch that gave up
// leaves no trace in the launches after it.
__device__ int g_rot_status;

// Progress of a pass over its columns: hi2lo, -X where every position >= X is final for the pass;
// lo2hi, X where every position <= X is final.  A finished pass publishes INT_MAX.
//
// Pipelined launches keep one word per pass in global memory (cleared by the launcher to a value
// below any position).  The storing warp publishes after a __syncwarp: that orders all its lanes'
// stores before lane 0's release, and a release is cumulative.  A release reduction (max: the
// words only rise) does not hold the thread the way a fence does.
__device__ __forceinline__ void publish_progress(int * p, int v) {
    asm volatile("red.release.gpu.global.max.s32 [%0], %1;\n" :: "l"(p), "r"(v) : "memory");
}
// The word in which a launch (resident kernel: a CTA) keeps that one of its waits ran out: its other
// waits then return at once, so one failed wait costs the launch about that long, not that long per
// unit.  Streaming launches hold it behind their work counter, reset by the same fill.
// Where it is stands in shared memory, written before the CTA's first barrier: the waits are calls from
// many places, which then pass nothing, and only a wait that is polling looks (with the pointer as an
// argument and a look before the first poll sph degree 4095 took 0.7 % longer).
struct GiveUp { int * word; int clean; };
__shared__ GiveUp s_giveup;
// true once the wait that began at t0 is to end: about 2^32 SM cycles later, or when another one ran out
__device__ __forceinline__ bool gave_up(long long t0, int code) {
    if (*(volatile int *) s_giveup.word != s_giveup.clean) return true;
    if (clock64() - t0 <= (1LL << 32)) return false;
    atomicExch(s_giveup.word, s_giveup.clean + 1);
    atomicCAS(&g_rot_status, 0, code);
    return true;
}
// Waits until *p >= need and returns the value read (a smaller one if the wait ended before).
// (The launch's word is a read of global memory, as slow as the progress word's own: only every 64th
// poll looks at it.)
__device__ __noinline__ int wait_progress(const int * p, int need) {
    const long long t0 = clock64();
    for (unsigned i = 1;; ++i) {
        int v;
        asm volatile("ld.acquire.gpu.global.s32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory");
        if (v >= need) return v;
        if (i % 64 == 0 && gave_up(t0, 3)) return v;
    }
}
// Whole-task launches run a task's passes one after another in one CTA, whose loading warp waits
// for its own storing warp: one 64-bit word in shared memory holds (pass counter of the CTA,
// progress + 2^31), which only rises.
__device__ __forceinline__ unsigned long long local_word(unsigned seq, int v) {
    return ((unsigned long long) seq << 32) | (unsigned) (v ^ 0x80000000);
}
__device__ __forceinline__ void publish_local(unsigned long long * p, unsigned long long w) {
    asm volatile("st.release.cta.shared::cta.u64 [%0], %1;\n" :: "r"(tc::smem_addr(p)), "l"(w) : "memory");
}
__device__ __noinline__ unsigned long long wait_local(const unsigned long long * p, unsigned long long need) {
    const long long t0 = clock64();
    for (unsigned i = 1;; ++i) {
        unsigned long long v;
        asm volatile("ld.acquire.cta.shared::cta.u64 %0, [%1];\n" : "=l"(v) : "r"(tc::smem_addr(p)) : "memory");
        if (v >= need) return v;
        if (i % 64 == 0 && gave_up(t0, 3)) return v;
        __nanosleep(32);
    }
}
// Bounded mbarrier wait: false once a wait of the launch ran out; the loops over queue entries then
// end, and the kernel with them.
// (The slow path is a call: the kernel's warps run different code at the same time, and what they
// run between them has to stay small to be served from the instruction cache.)
__device__ __noinline__ bool wait_bar_slow(uint64_t * bar, uint32_t parity) {
    const long long t0 = clock64();
    while (!tc::mbar_try_wait(bar, parity))
        if (gave_up(t0, 5)) return false;
    return true;
}
__device__ __forceinline__ bool wait_bar(uint64_t * bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok) : "r"(tc::smem_addr(bar)), "r"(parity) : "memory");
    return ok || wait_bar_slow(bar, parity);
}

// Asynchronous 8-byte copy global -> shared (0 bytes read, zeros written when !valid), and the
// arrival of this thread on a barrier once its copies so far have landed.
__device__ __forceinline__ void copy_async8(uint32_t dst, const double * src, bool valid) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" :: "r"(dst), "l"(src), "r"(valid ? 8 : 0) : "memory");
}
__device__ __forceinline__ void copy_async_arrive(uint64_t * bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];\n" :: "r"(tc::smem_addr(bar)) : "memory");
}

// Geometry of one pass of W x B sweeps of a task, the same for every warp of the CTA.  The
// sweeps are numbered i = (j - parity) / STEP; a pass holds i0 .. i0 + W B - 1 (the last one
// fewer), aligned with the task's lowest sweep, so that the B sweeps of a stage are rows of one
// block of the skewed table.  The pass moves positions 0 .. emax of every chain as a stream of
// nchunk chunks of E positions (hi2lo: from the top down, lo2hi: from the bottom up); chunk k
// covers positions pmin(k) .. pmin(k) + E - 1, those outside 0 .. emax read as zero and are not
// written.  The chunks are aligned so that the pairs of a stage's chunk are whole chunks of the
// skewed table.
template <int KIND, bool HI2LO, int W, int B, int E>
struct Pass {
    int i0, stages;   // lowest sweep, stages with a sweep
    int emax, nchunk;
    __host__ __device__ __forceinline__ Pass(int N, int nsw, int npass, int jpar, int jlo, int r, bool copy_all) {
        const int at = HI2LO ? npass - 1 - r : r;
        const int left = nsw - at * W * B;
        i0 = (jlo - jpar) / KT<KIND>::STEP + at * W * B;
        stages = (left >= W * B ? W * B : left) / B + ((left < W * B && left % B) ? 1 : 0);
        const int top = Geo::top(KIND, N, jpar + KT<KIND>::STEP * i0, 0), last = Geo::chain_len(KIND, N, 0) - 1;
        emax = top + 1;
        if (copy_all || emax > last) emax = last;
        if (emax < 0) emax = 0;
        nchunk = HI2LO ? emax / E + 1 : (emax + 1) / E + 1;
    }
    __host__ __device__ __forceinline__ int pmin(int k) const { return HI2LO ? (nchunk - 1 - k) * E : k * E - 1; }
    // lowest sweep of stage q
    __host__ __device__ __forceinline__ int stage_sweep(int q) const { return i0 + (HI2LO ? stages - 1 - q : q) * B; }
    // chunk of the skewed table (in units of E positions) that a stage meets at its chunk k
    __host__ __device__ __forceinline__ int kappa(int k) const { return HI2LO ? nchunk - 1 + 2 * B / E - k : k; }
};

// A task's sweeps and passes.
template <int KIND, int NC, int W, int B>
struct TaskGeo {
    int N, M, mbase, mlast, jpar, nsw, jlo, jhi, npass;
    __host__ __device__ __forceinline__ TaskGeo(const RotField & F, const RotTask & t) {   // t: a group of KT<KIND, NC>::ORD orders
        N = F.N; M = F.M; mbase = t.mbase;
        mlast = Geo::last_order(KIND, M);
        // lowest sweep of every column (spin: the parity of the effective orders |m - s|)
        jpar = KIND == TRI ? 0 : (KIND == SPIN ? ((mbase + F.spin) & 1) : (mbase & 1));
        nsw = mbase > mlast ? 0 : Geo::task_sweeps(KIND, M, mbase, F.blk, &jlo, &jhi, F.spin, KT<KIND, NC>::ORD);
        npass = (nsw + W * B - 1) / (W * B);
    }
};

// The elements of one chunk as a warp moves them between global memory and a ring slot.  A column's
// part of a chunk is a segment of E * CH * ES consecutive doubles; a lane takes, in each of PH
// phases, the same double of every SSTEP-th segment, so that its addresses advance by constants.
template <int KIND, int NC, bool HI2LO, int E>
struct Mover {
    using T = KT<KIND, NC>;
    static constexpr int RPC = E * T::CH * T::ES;                  // doubles of a segment
    static constexpr int SEGS = T::COLS / T::ES;                   // segments (columns) of a task
    static constexpr int PER = T::COLS * E * T::CH / 32;           // elements of a lane
    static constexpr int RB = RPC >= 32 ? RPC / 32 : 1;            // instructions per segment
    static constexpr int SP = RPC >= 32 ? 1 : 32 / RPC;            // segments per instruction
    static constexpr bool PAIRED = KIND == SPH || KIND == DISK;    // two columns an order, side by side
    static constexpr int PH = RB > 1 ? RB : (PAIRED && SP == 1) ? 2 : 1;
    static constexpr int NV = PER / PH;                            // elements of a lane in a phase
    static constexpr int SSTEP = RB > 1 ? 1 : SP * PH;
    static constexpr int SLOT_STEP = T::place(0, SSTEP * T::ES);   // ring slot doubles between them
    static_assert(RPC % 32 == 0 || 32 % RPC == 0, "a segment must split evenly over the lanes");
    static_assert(!PAIRED || SSTEP % 2 == 0, "a lane's segments must be whole orders apart");
    long long base;     // double offset, at chain position 0, of the column of this lane's segment 0
    long long lda2;     // doubles between columns
    int nseg, seg0;     // the task's valid segments, less this lane's own (spin: order 0 has one column)
    int N, lane;
    __host__ __device__ __forceinline__ static int lane_seg(int lane) { return RPC < 32 ? lane / RPC : 0; }
    __host__ __device__ __forceinline__ static int rr(int ph, int lane) { return RB > 1 ? ph * 32 + lane : lane % RPC; }
    __host__ __device__ __forceinline__ static constexpr int seg(int ph) { return RB > 1 ? 0 : ph * SP; }
    // columns from the task's first one to segment s's
    __host__ __device__ __forceinline__ static constexpr int col_of(int s) {
        return KIND == TRI ? s : KIND == RECT ? 2 * s : KIND == SPIN ? 4 * s : 4 * (s >> 1) + (s & 1);
    }
    __host__ __device__ __forceinline__ Mover(const RotField & F, const RotTask & t, int mlast, int lane_) : lane(lane_) {
        N = F.N;
        lda2 = (long long) T::ES * F.lda;
        const int orders = t.mbase > mlast ? 0 : min(T::ORD, (mlast - t.mbase) / T::STEP + 1);
        const int ls = lane_seg(lane);
        nseg = orders * (SEGS / T::ORD) - ls;
        seg0 = 0;
        long long col0;
        if (KIND == TRI || KIND == RECT) col0 = t.mbase;
        else if (KIND == SPIN) {
            col0 = 2LL * t.mbase - (t.side ? 0 : 1);    // side 0: order -m in column 2m - 1; 1: order m in 2m
            if (col0 < 0) seg0 = 1 - ls;
            // the matrix may end before the last order's column
            const long long most = (F.M - 1 - col0) / 4 + 1;
            if (nseg + ls > most) nseg = (int) most - ls;
        } else col0 = 2LL * t.mbase - 1;
        base = (col0 + col_of(ls)) * lda2;
    }
    // element v of phase ph belongs to a column of the task
    __host__ __device__ __forceinline__ bool seg_ok(int ph, int v) const {
        const int s = seg(ph) + v * SSTEP;
        return s < nseg && s >= seg0;
    }
    __host__ __device__ __forceinline__ bool row_ok(int ph, int pmin, int emax) const {
        const int r = rr(ph, lane), p = pmin + r / (T::ES * T::CH);
        return p >= 0 && p <= emax && T::CH * p + (r / T::ES) % T::CH < N;
    }
    // double offset of element 0 of a phase in the chunk that starts at position pmin, and between elements
    __host__ __device__ __forceinline__ long long at(int ph, int pmin) const {
        return base + (long long) col_of(seg(ph)) * lda2 + (long long) T::ES * T::CH * pmin + rr(ph, lane);
    }
    __host__ __device__ __forceinline__ long long step() const { return (long long) col_of(SSTEP) * lda2; }
    // place of element 0 of a phase in a ring slot
    __host__ __device__ __forceinline__ int slot_at(int ph) const {
        const int r = rr(ph, lane), pos = r / (T::ES * T::CH), c = (r / T::ES) % T::CH, part = r % T::ES;
        const int u = HI2LO ? E - 1 - pos : pos;
        return u * T::ROWD + T::place(c, (seg(ph) + lane_seg(lane)) * T::ES + part);
    }
};

// E steps of a stage.  The window is circular: at step u, window position x lives in register
// slot (u - x) mod 2B.  The element leaving (position 2B - 1 of the previous step) sits in slot
// u mod 2B, which the entering element (position 0) takes over.  OFF: step number of the chunk's
// first step mod 2B.  Without rotations (ROTATE false) every element leaves as it entered.
// has_in / has_out are the same for the warp; elements are read and written in groups of SUB steps,
// a branch a group (2 - 4 % faster than a condition on each access).
template <bool HI2LO, int NCOL, int B, int E, int OFF, int STRIDE, int PAIR, int ROWLEN, int SUB, bool ROTATE>
__device__ __forceinline__ void stage_steps(double (&win)[NCOL][2 * B], const double * bin, double * bout, bool has_in, bool has_out,
                                            const double2 * const (&sc)[B]) {
    constexpr int W2 = 2 * B;
#pragma unroll
    for (int e0 = 0; e0 < E; e0 += SUB) {
        double in[SUB][NCOL], out[SUB][NCOL];
#pragma unroll
        for (int e = 0; e < SUB; ++e)
#pragma unroll
            for (int h = 0; h < NCOL; ++h) in[e][h] = 0.0;
        if (has_in) {
#pragma unroll
            for (int e = 0; e < SUB; ++e)
#pragma unroll
                for (int h = 0; h < NCOL; ++h) in[e][h] = bin[(e0 + e) * STRIDE + h];
        }
#pragma unroll
        for (int e = 0; e < SUB; ++e) {
            const int u = OFF + e0 + e, pn = u % W2;
#pragma unroll
            for (int h = 0; h < NCOL; ++h) {
                out[e][h] = win[h][pn];
                win[h][pn] = in[e][h];
            }
            if (ROTATE) {
                // PAIR: pairs between positions of a row; rows of a chunk of kSkewLen positions are
                // ROWLEN pairs long and a chunk of them kSkewRows rows
                constexpr int SL = Geo::kSkewLen;
                const int pos = HI2LO ? E - 1 - e0 - e : e0 + e;
#pragma unroll
                for (int b = 0; b < B; ++b) {
                    const double2 p = sc[b][pos / SL * Geo::kSkewRows * ROWLEN + pos % SL * PAIR];
                    const int xl = (u - 2 * b + 2 * W2) % W2;       // window position 2b
                    const int xu = (u - 2 * b - 1 + 2 * W2) % W2;   // window position 2b+1
#pragma unroll
                    for (int h = 0; h < NCOL; ++h) {
                        if (HI2LO) rot_hi2lo(win[h][xl], win[h][xu], p.x, p.y);
                        else       rot_lo2hi(win[h][xu], win[h][xl], p.x, p.y);
                    }
                }
            }
        }
        if (has_out) {
#pragma unroll
            for (int e = 0; e < SUB; ++e)
#pragma unroll
                for (int h = 0; h < NCOL; ++h) bout[(e0 + e) * STRIDE + h] = out[e][h];
        }
    }
}

// Progress of a warp of the resident kernel, in shared memory (it only rises).
__device__ __forceinline__ void publish_word(int * p, int v) {
    asm volatile("st.release.cta.shared::cta.s32 [%0], %1;\n" :: "r"(tc::smem_addr(p)), "r"(v) : "memory");
}
__device__ __noinline__ int wait_word_slow(const int * p, int need) {
    const long long t0 = clock64();
    for (unsigned i = 1;; ++i) {
        int v;
        asm volatile("ld.acquire.cta.shared::cta.s32 %0, [%1];\n" : "=r"(v) : "r"(tc::smem_addr(p)) : "memory");
        if (v >= need) return v;
        if (i % 256 == 0 && gave_up(t0, 3)) return v;
    }
}
__device__ __forceinline__ int wait_word(const int * p, int need) {
    int v;
    asm volatile("ld.acquire.cta.shared::cta.s32 %0, [%1];\n" : "=r"(v) : "r"(tc::smem_addr(p)) : "memory");
    return v >= need ? v : wait_word_slow(p, need);
}

// E steps of one sequence of the resident kernel (stage_steps with the columns in place; a branch an
// access here: groups measured 7 % slower).  ROTATE false: the window only shifts.
template <bool HI2LO, int CH, int B, int E, int OFF, int ROW, bool ROTATE>
__device__ __forceinline__ void resident_steps(double (&win)[2 * B], const double * bin, double * bout, bool has_in, bool has_out,
                                               const double2 * const (&sc)[B]) {
    constexpr int W2 = 2 * B;
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int u = OFF + e, pn = u % W2, at = HI2LO ? -e * ROW : e * ROW;
        const double in = has_in ? bin[at] : 0.0;
        if (has_out) bout[at] = win[pn];
        win[pn] = in;
        if (ROTATE) {
#pragma unroll
            for (int b = 0; b < B; ++b) {
                const double2 p = sc[b][(HI2LO ? E - 1 - e : e) * CH];
                const int xl = (u - 2 * b + 2 * W2) % W2, xu = (u - 2 * b - 1 + 2 * W2) % W2;
                if (HI2LO) rot_hi2lo(win[xl], win[xu], p.x, p.y);
                else       rot_lo2hi(win[xu], win[xl], p.x, p.y);
            }
        }
    }
}

// Compile-time layout of a launch shape.
template <int KIND, int NC, int W, int B, int E>
struct Shape {
    using T = KT<KIND, NC>;
    static constexpr int SPLIT = KT<KIND>::ORD / T::ORD;  // groups of a task of the list
    static constexpr int D = 2 * B / E;                  // chunks an element spends in a stage's window
    static constexpr int SL = 2;                         // slots of a ring
    static constexpr int SCS = E >= 16 ? 2 : 3;          // staged (sin, cos) chunks of a stage
    static constexpr int WARPS = W + 2;                  // and a loading and a storing warp
    static constexpr int SLOT = E * T::ROWD;     // doubles of a ring slot
    static constexpr int SCLEN = B * E * T::CH;          // pairs of a stage's chunk
    static constexpr int IDLEN = (E / Geo::kSkewLen - 1) * Geo::kSkewRows * Geo::kSkewLen * T::CH + Geo::kSkewLen * T::CH;   // a row's span in one
    static constexpr int UR = 4;                         // queue entries in flight in a CTA
    static constexpr size_t doubles = (size_t) (W + 1) * SL * SLOT;
    static constexpr size_t pairs = (size_t) W * SCS * SCLEN + IDLEN;
    static constexpr size_t bytes = (doubles * sizeof(double) + 15) / 16 * 16 + pairs * sizeof(double2);
    static_assert(D >= 1 && D * E == 2 * B, "a window must hold whole chunks");
    static_assert(E % Geo::kSkewLen == 0, "a chunk must be whole chunks of the skewed table");
    static_assert(B == Geo::kSkewRows, "a stage's sweeps must be the rows of one block of the skewed table");
};

// Columns without sweeps, in to out (one CTA a field; nothing when in place).
__device__ __forceinline__ void copy_lead(const RotLaunch & L) {
    for (int f = blockIdx.x; f < L.nfields; f += gridDim.x) {
        const RotField & F = L.fields[f];
        if (F.in == F.out) continue;
        for (int c = L.lead0; c < min(L.lead, F.M); ++c)
            for (int i = threadIdx.x; i < F.N; i += blockDim.x) F.out[c * F.lda + i] = __ldcg(F.in + c * F.lda + i);
    }
}

template <int KIND, int NC, bool HI2LO, int W, int B, int E, int MINB>
__global__ void __launch_bounds__(Shape<KIND, NC, W, B, E>::WARPS * 32, MINB)
rot_kernel(const __grid_constant__ RotLaunch L) {
    using T = KT<KIND, NC>;
    using SH = Shape<KIND, NC, W, B, E>;
    using MV = Mover<KIND, NC, HI2LO, E>;
    constexpr int SUBS = 2;   // 4 measured the same, 8 (more registers) 10 % slower
    constexpr int CH = T::CH, STEP = T::STEP, NCOL = T::NCOL, D = SH::D, SL = SH::SL, SCS = SH::SCS, SLOT = SH::SLOT,
                  SCLEN = SH::SCLEN, UR = SH::UR;
    extern __shared__ __align__(16) double smem[];
    double * const rings = smem;                                  // ring q: input of stage q; ring W: output of the last stage
    double2 * const pairs = reinterpret_cast<double2 *>(reinterpret_cast<unsigned char *>(smem) + (SH::doubles * sizeof(double) + 15) / 16 * 16);
    double2 * const ident = pairs + (size_t) W * SCS * SCLEN; // identity pairs, for sweeps a lane's order does not have
    __shared__ __align__(8) uint64_t full[(W + 1) * SL], empt[(W + 1) * SL], scbar[W * SCS], ufull[UR], uempt[UR];
    __shared__ unsigned long long s_local;
    __shared__ int s_unit[UR];

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = threadIdx.x; i < SH::IDLEN; i += blockDim.x) ident[i] = make_double2(0.0, 1.0);
    if (threadIdx.x == 0) {
        for (int i = 0; i < (W + 1) * SL; ++i) { tc::mbar_init(&full[i], i < SL ? 32 : 1); tc::mbar_init(&empt[i], 1); }
        for (int i = 0; i < W * SCS; ++i) tc::mbar_init(&scbar[i], 1);
        for (int i = 0; i < UR; ++i) { tc::mbar_init(&ufull[i], 1); tc::mbar_init(&uempt[i], SH::WARPS - 1); }
        s_local = 0;
        s_giveup = GiveUp{L.counter + 1, L.counter0};
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncthreads();

    if (L.lead > L.lead0) copy_lead(L);

    const bool pipe = L.chains != nullptr;
    const int nwork = pipe ? L.nchains : L.ntasks * SH::SPLIT;
    // group g of the list: orders g % SPLIT of its task
    auto group = [&](int g) {
        RotTask t = L.tasks[g / SH::SPLIT];
        t.mbase += T::STEP * T::ORD * (g % SH::SPLIT);
        return t;
    };
    unsigned nunit = 0;        // queue entries taken so far
    unsigned seq = 0;          // passes begun so far
    // The loading warp takes an entry from the queue and hands it to the other warps, which
    // take it up as they finish the one before: nothing in the CTA stands still between entries.
    auto next_unit = [&]() -> int {
        const int slot = nunit % UR;
        const uint32_t ph = (nunit / UR) & 1;
        ++nunit;
        int id = 0;
        if (warp == W) {
            if (!__all_sync(0xffffffffu, wait_bar(&uempt[slot], ph ^ 1))) return -1;
            if (lane == 0) {
                id = atomicAdd(L.counter, 1) - L.counter0;
                if (id >= nwork) id = -1;
                s_unit[slot] = id;
                tc::mbar_arrive(&ufull[slot]);
            }
            id = __shfl_sync(0xffffffffu, id, 0);
        } else {
            if (!__all_sync(0xffffffffu, wait_bar(&ufull[slot], ph))) return -1;
            id = *(volatile int *) &s_unit[slot];
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&uempt[slot]);
        }
        return id;
    };

    if (warp < W) {
        // ---------------- a stage: B consecutive sweeps of each pass ----------------
        const int q = warp;
        const int o_lane = T::lane_order(lane), c_lane = lane % CH, lane_off = T::lane_place(lane);
        uint64_t * const in_full = full + q * SL, * const in_empty = empt + q * SL;
        uint64_t * const out_full = full + (q + 1) * SL, * const out_empty = empt + (q + 1) * SL;
        double * const in_ring = rings + (size_t) q * SL * SLOT, * const out_ring = in_ring + (size_t) SL * SLOT;
        double2 * const sc_ring = pairs + (size_t) q * SCS * SCLEN;
        unsigned nin = 0, nout = 0;           // chunks taken and passed on
        unsigned sc_issued = 0, sc_used = 0;  // (sin, cos) chunks staged and used
        double win[NCOL][2 * B];
        for (;;) {
            const int id = next_unit();
            if (id < 0) break;
            const RotChain chain = pipe ? L.chains[id] : RotChain{id, 0, 0, 1};
            const RotTask task = group(chain.task);
            const RotField & F = L.fields[task.field];
            const TaskGeo<KIND, NC, W, B> G(F, task);
            const int N = G.N;
            const int jpar = G.jpar;
            // the order whose sweeps this lane runs (spin: |m - s|), and its lowest sweep: with
            // F.blk > 0 a column of order m runs only the (m - jpar)/STEP mod blk sweeps above its
            // last whole block of blk sweeps
            const int m_lane = G.mbase + STEP * o_lane;
            const int me_lane = KIND == SPIN ? abs(m_lane - F.spin) : m_lane;
            const int jcut = F.blk > 0 ? m_lane - STEP * (((m_lane - jpar) / STEP) % F.blk) : jpar;
            for (int r = chain.first; r < G.npass; r += chain.stride) {
                const Pass<KIND, HI2LO, W, B, E> P(N, G.nsw, G.npass, G.jpar, G.jlo, r, r == 0 && F.in != F.out);
                if (q >= P.stages) {
                    // no sweep of the pass: hand the chunks on
                    for (int k = 0; k < P.nchunk; ++k) {
                        wait_bar(&in_full[nin % SL], (nin / SL) & 1);
                        wait_bar(&out_empty[nout % SL], ((nout / SL) & 1) ^ 1);
                        const double * const bin = in_ring + (nin % SL) * SLOT + lane_off;
                        double * const bout = out_ring + (nout % SL) * SLOT + lane_off;
#pragma unroll
                        for (int e = 0; e < E; ++e)
#pragma unroll
                            for (int h = 0; h < NCOL; ++h) bout[e * T::ROWD + h] = bin[e * T::ROWD + h];
                        __syncwarp();
                        if (lane == 0) { tc::mbar_arrive(&in_empty[nin % SL]); tc::mbar_arrive(&out_full[nout % SL]); }
                        ++nin; ++nout;
                    }
                    continue;
                }
                const int i0 = P.stage_sweep(q);
                unsigned lane_mask = 0;   // sweeps this lane's order has (hi2lo applies the highest first)
#pragma unroll
                for (int b = 0; b < B; ++b) {
                    const int j = jpar + STEP * (HI2LO ? i0 + B - 1 - b : i0 + b);
                    if (j <= me_lane - STEP && j >= jcut) lane_mask |= 1u << b;
                }
                // The (sin, cos) pairs of chunk k: one bulk copy of the skewed table's chunk of the stage's
                // block, whose entries are the identity where a sweep has no rotation, so every chunk runs the same straight-line code and those
                // rotations are exact no-ops.  Returns false, staging nothing, when no sweep of the
                // stage rotates in the chunk.
                const int K = P.nchunk + D;
                const int beta = i0 / Geo::kSkewRows;
                const int nk = beta < Geo::skew_blocks(KIND, N, jpar) ? Geo::skew_chunks(KIND, N, jpar, beta) : 0;
                const double2 * const rows = F.sc + Geo::skew_at(KIND, N, jpar, beta);
                auto stage_sc = [&](int k) -> bool {
                    const int kappa = P.kappa(k) * (E / Geo::kSkewLen);
                    if (k >= K || kappa >= nk) return false;
                    if (lane == 0) {
                        const int slot = sc_issued % SCS;
                        uint64_t * const bar = &scbar[q * SCS + slot];
                        tc::mbar_arrive_expect_tx(bar, (uint32_t) (SCLEN * sizeof(double2)));
                        tc::bulk_g2s(sc_ring + slot * SCLEN, rows + kappa * Geo::skew_chunk(KIND), (uint32_t) (SCLEN * sizeof(double2)), bar);
                    }
                    ++sc_issued;
                    return true;
                };
                unsigned live = 0;        // bit i: chunk k + i is staged
#pragma unroll
                for (int i = 0; i + 1 < SCS; ++i) live |= stage_sc(i) ? 1u << i : 0u;
#pragma unroll
                for (int h = 0; h < NCOL; ++h)
#pragma unroll
                    for (int x = 0; x < 2 * B; ++x) win[h][x] = 0.0;
                // element entering at chunk k leaves at chunk k + D
                for (int k = 0; k < K; ++k) {
                    live |= stage_sc(k + SCS - 1) ? 1u << (SCS - 1) : 0u;
                    const bool has_in = k < P.nchunk, has_out = k >= D;
                    const int is = nin % SL, os = nout % SL;
                    if (has_in) wait_bar(&in_full[is], (nin / SL) & 1);
                    if (has_out) wait_bar(&out_empty[os], ((nout / SL) & 1) ^ 1);
                    const double * const bin = in_ring + is * SLOT + lane_off;    // read while elements enter (has_in)
                    double * const bout = out_ring + os * SLOT + lane_off;        // written once elements leave (has_out)
                    const bool odd = D > 1 && (k & 1);   // the chunk starts halfway round the window
                    if (live & 1u) {
                        const int slot = sc_used % SCS;
                        wait_bar(&scbar[q * SCS + slot], (sc_used / SCS) & 1);
                        ++sc_used;
                        const double2 * sc[B];
#pragma unroll
                        for (int b = 0; b < B; ++b)
                            sc[b] = ((lane_mask >> b) & 1u ? sc_ring + slot * SCLEN + (HI2LO ? B - 1 - b : b) * Geo::kSkewLen * CH : ident) + c_lane;
                        if (odd) stage_steps<HI2LO, NCOL, B, E, E % (2 * B), T::ROWD, CH, Geo::kSkewLen * CH, SUBS, true>(win, bin, bout, has_in, has_out, sc);
                        else     stage_steps<HI2LO, NCOL, B, E, 0, T::ROWD, CH, Geo::kSkewLen * CH, SUBS, true>(win, bin, bout, has_in, has_out, sc);
                    } else {
                        const double2 * const none[B] = {};
                        if (odd) stage_steps<HI2LO, NCOL, B, E, E % (2 * B), T::ROWD, CH, Geo::kSkewLen * CH, SUBS, false>(win, bin, bout, has_in, has_out, none);
                        else     stage_steps<HI2LO, NCOL, B, E, 0, T::ROWD, CH, Geo::kSkewLen * CH, SUBS, false>(win, bin, bout, has_in, has_out, none);
                    }
                    live >>= 1;
                    __syncwarp();
                    if (lane == 0) {
                        if (has_in) tc::mbar_arrive(&in_empty[is]);
                        if (has_out) tc::mbar_arrive(&out_full[os]);
                    }
                    nin += has_in; nout += has_out;
                }
            }
        }
        // every staged copy was waited for above unless a wait ran out: then wait (bounded) here
        for (; sc_used != sc_issued; ++sc_used) {
            const long long t0 = clock64();
            while (!tc::mbar_try_wait(&scbar[q * SCS + sc_used % SCS], (sc_used / SCS) & 1) && clock64() - t0 < (1LL << 24)) {}
        }
    } else if (warp <= W) {   // (== W: the compiler's layout takes 0.5 % longer at sph degree 4095)
        // ---------------- loading warp ----------------
        unsigned n0 = 0;           // chunks of earlier passes
        for (;;) {
            const int id = next_unit();
            if (id < 0) break;
            const RotChain chain = pipe ? L.chains[id] : RotChain{id, 0, 0, 1};
            const RotTask task = group(chain.task);
            const RotField & F = L.fields[task.field];
            const TaskGeo<KIND, NC, W, B> G(F, task);
            if (lane == 0 && G.nsw > 0 && (chain.first >= G.npass || chain.stride < 1))
                atomicCAS(&g_rot_status, 0, 4);   // a schedule that does not match this launch shape
            const MV mv(F, task, G.mlast, lane);
            for (int r = chain.first; r < G.npass; r += chain.stride) {
                const Pass<KIND, HI2LO, W, B, E> P(G.N, G.nsw, G.npass, G.jpar, G.jlo, r, r == 0 && F.in != F.out);
                const double * const src = r == 0 ? F.in : F.out;
                const int * const prev = (pipe && r > 0) ? L.prog + chain.prog0 + r - 1 : nullptr;
                const bool prev_local = !pipe && r > 0;
                ++seq;
                int seen = -0x7fffffff - 1;          // the predecessor's progress as last read
                unsigned long long seen_local = 0;
                // wait until the predecessor has finished the positions chunk i loads
                auto wait_chunk = [&](int i) {
                    if (!prev && !prev_local) return;
                    const int pmin = P.pmin(i), pmax = pmin + E - 1;
                    const int need = HI2LO ? -max(pmin, 0) : min(pmax, P.emax);
                    if (prev) {
                        if (seen < need) { if (lane == 0) seen = wait_progress(prev, need); seen = __shfl_sync(0xffffffffu, seen, 0); }
                    } else {
                        const unsigned long long want = local_word(seq - 1, need);
                        if (seen_local < want) { if (lane == 0) seen_local = wait_local(&s_local, want); seen_local = __shfl_sync(0xffffffffu, seen_local, 0); }
                    }
                    __syncwarp();
                };
                // the copies land in the slot by themselves: up to SL chunks are on their way
                auto fetch = [&](int i) {
                    const unsigned n = n0 + i;
                    const int pmin = P.pmin(i);
                    wait_bar(&empt[n % SL], ((n / SL) & 1) ^ 1);
                    const uint32_t slot = tc::smem_addr(rings + (size_t) (n % SL) * SLOT);
#pragma unroll 1
                    for (int ph = 0; ph < MV::PH; ++ph) {
                        const bool ok = mv.row_ok(ph, pmin, P.emax);
                        const double * g = src + mv.at(ph, pmin);
                        uint32_t sa = slot + 8u * mv.slot_at(ph);
#pragma unroll 4
                        for (int v = 0; v < MV::NV; ++v, g += mv.step(), sa += 8u * MV::SLOT_STEP) {
                            const bool valid = ok && mv.seg_ok(ph, v);
                            copy_async8(sa, valid ? g : src, valid);
                        }
                    }
                    copy_async_arrive(&full[n % SL]);
                };
                wait_chunk(0);
                // hi2lo: the positions above this pass's range are final once the predecessor has
                // finished the first chunk's (they belong to earlier passes only)
                if (HI2LO && pipe && lane == 0 && r + 1 < G.npass) publish_progress(L.prog + chain.prog0 + r, -(P.emax + 1));
                for (int i = 0; i < P.nchunk; ++i) { wait_chunk(i); fetch(i); }
                n0 += P.nchunk;
            }
        }
        asm volatile("cp.async.wait_all;\n" ::: "memory");
    } else {
        // ---------------- storing warp ----------------
        unsigned n = 0;
        uint64_t * const bfull = full + W * SL, * const bempt = empt + W * SL;
        const double * const ring = rings + (size_t) W * SL * SLOT;
        for (;;) {
            const int id = next_unit();
            if (id < 0) break;
            const RotChain chain = pipe ? L.chains[id] : RotChain{id, 0, 0, 1};
            const RotTask task = group(chain.task);
            const RotField & F = L.fields[task.field];
            const TaskGeo<KIND, NC, W, B> G(F, task);
            const MV mv(F, task, G.mlast, lane);
            // publish every 16 positions for short columns, every 64 for long ones (and at the end): a
            // successor trailing by a little more loses little of a long pass
            const int every = max(1, (F.N >= 2048 ? 64 : 16) / E);
            for (int r = chain.first; r < G.npass; r += chain.stride) {
                const Pass<KIND, HI2LO, W, B, E> P(G.N, G.nsw, G.npass, G.jpar, G.jlo, r, r == 0 && F.in != F.out);
                ++seq;
                int since = 0;
                for (int i = 0; i < P.nchunk; ++i, ++n) {
                    const int pmin = P.pmin(i);
                    wait_bar(&bfull[n % SL], (n / SL) & 1);
                    const double * const slot = ring + (n % SL) * SLOT;
#pragma unroll 1
                    for (int ph = 0; ph < MV::PH; ++ph) {
                        if (!mv.row_ok(ph, pmin, P.emax)) continue;
                        double * g = F.out + mv.at(ph, pmin);
                        const double * x = slot + mv.slot_at(ph);
#pragma unroll 4
                        for (int v = 0; v < MV::NV; ++v, g += mv.step(), x += MV::SLOT_STEP)
                            if (mv.seg_ok(ph, v)) __stcg(g, *x);
                    }
                    __syncwarp();
                    if (lane == 0) tc::mbar_arrive(&bempt[n % SL]);
                    if (r + 1 == G.npass || (++since < every && i + 1 < P.nchunk)) continue;   // no pass follows the last
                    since = 0;
                    __syncwarp();
                    if (lane == 0) {
                        const int v = i + 1 == P.nchunk ? 0x7fffffff : HI2LO ? -pmin : pmin + E - 1;
                        if (pipe) publish_progress(L.prog + chain.prog0 + r, v);
                        else      publish_local(&s_local, local_word(seq, v));
                    }
                }
            }
        }
    }
}

template <int KIND, int NC, bool HI2LO, int W, int B, int E, int MINB>
cudaError_t launch_cfg(const RotLaunch & L, int max_ctas, int per_sm_most, cudaStream_t st) {
    using SH = Shape<KIND, NC, W, B, E>;
    auto kern = rot_kernel<KIND, NC, HI2LO, W, B, E, MINB>;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    // resident CTAs of the whole device, asked for once per device
    static std::atomic<int> resident[16] = {};   // SMs x 256 + CTAs per SM
    int room = dev < 16 ? resident[dev].load(std::memory_order_acquire) : 0;
    if (room == 0) {
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) SH::bytes);
        if (e != cudaSuccess) return e;
        int sms = 0, per_sm = 1;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, SH::WARPS * 32, SH::bytes) != cudaSuccess || per_sm < 1) per_sm = 1;
        room = sms * 256 + per_sm;
        if (dev < 16) resident[dev].store(room, std::memory_order_release);
    }
    int ctas = (room >> 8) * (per_sm_most > 0 ? std::min(per_sm_most, room & 255) : room & 255);
    if (max_ctas > 0 && ctas > max_ctas) ctas = max_ctas;
    const int work = L.chains ? L.nchains : L.ntasks * SH::SPLIT;   // queue entries: pipeline entries or groups
    if (ctas > work) ctas = work;
    if (ctas <= 0) return cudaSuccess;
    if (!L.chains) e = cudaMemsetAsync(L.counter, 0, sizeof(int) * kCounterWords, st);   // with chains: launch_shape
    if (e != cudaSuccess) return e;
    kern<<<ctas, SH::WARPS * 32, SH::bytes, st>>>(L);
    count_launch();
    e = cudaGetLastError();
    if (e != cudaSuccess) {
        cudaFuncAttributes fa{};
        cudaFuncGetAttributes(&fa, kern);
        std::fprintf(stderr, "rot_kernel launch failed (%s): regs %d, static smem %zu, dyn smem %zu, max threads %d, params %zu B\n",
                     cudaGetErrorString(e), fa.numRegs, fa.sharedSizeBytes, SH::bytes, fa.maxThreadsPerBlock, sizeof(RotLaunch));
    }
    return e;
}

// ---------------------------------------------------------------------------
// The same sweeps with the columns of a task resident in shared memory, for chains short enough
// to fit.  One CTA per group of orders, one lane per sequence (order, column, chain); the warps
// take the task's blocks of B sweeps in turn and run down the columns in place, warp g + 1 behind
// warp g.  Nothing is streamed between stages or passes, so a column's sweeps follow each other at
// a distance of 2B + E positions whatever their number, and the loop is short enough for the
// instruction cache.  Each (sin, cos) load feeds one sequence instead of two, so a chip full of
// tasks runs faster in rot_kernel (launch_rotations has the rule).
// ---------------------------------------------------------------------------
template <int KIND>
struct RT {
    static constexpr int CH = KT<KIND>::CH, STEP = KT<KIND>::STEP, ES = KT<KIND>::ES, NC = KT<KIND>::SEQ;
    static constexpr int ORD = 32 / (CH * NC);                  // orders of a CTA
    static constexpr int SPLIT = KT<KIND>::ORD / ORD;           // CTAs of a task of the list
    static constexpr int W = 8, B = 8, E = 8, D = 2 * B / E, SCS = 3;
    static constexpr int ROW = 33;                              // doubles of a position: 32 lanes and a pad
    static constexpr int SCLEN = B * E * CH, IDLEN = E * CH;
    static constexpr size_t pair_bytes = sizeof(double2) * ((size_t) W * SCS * SCLEN + IDLEN);
    // positions -1 .. chain_len rounded up to whole chunks
    __host__ __device__ static int rows(int N) { return (Geo::chain_len(KIND, N, 0) + E - 1) / E * E + E; }
    __host__ __device__ static size_t bytes(int N) { return pair_bytes + sizeof(double) * (size_t) rows(N) * ROW; }
};

template <int KIND, bool HI2LO>
__global__ void __launch_bounds__(RT<KIND>::W * 32, 2)
rot_resident_kernel(const __grid_constant__ RotLaunch L) {
    using R = RT<KIND>;
    constexpr int CH = R::CH, STEP = R::STEP, ES = R::ES, NC = R::NC, ORD = R::ORD, W = R::W, B = R::B, E = R::E, D = R::D,
                  SCS = R::SCS, ROW = R::ROW, SCLEN = R::SCLEN;
    extern __shared__ __align__(16) double smem[];
    double2 * const pairs = reinterpret_cast<double2 *>(smem);
    double2 * const ident = pairs + W * SCS * SCLEN;
    double * const col = reinterpret_cast<double *>(ident + R::IDLEN) + ROW;   // position p of lane l at col[p * ROW + l]
    __shared__ __align__(8) uint64_t scbar[W * SCS];
    __shared__ int prog[W], s_gave_up;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    allow_next();
    wait_for_previous();
    if (L.lead > L.lead0) copy_lead(L);
    const RotTask task = L.tasks[blockIdx.x / R::SPLIT];
    const RotField & F = L.fields[task.field];
    const int N = F.N, mlast = Geo::last_order(KIND, F.M);
    const int mbase = task.mbase + STEP * ORD * (R::SPLIT - 1 - (int) (blockIdx.x % R::SPLIT));
    if (mbase > mlast) return;
    int jlo, jhi;
    const int nsw = Geo::task_sweeps(KIND, F.M, mbase, F.blk, &jlo, &jhi, F.spin, ORD);
    const int jpar = KIND == TRI ? 0 : (KIND == SPIN ? ((mbase + F.spin) & 1) : (mbase & 1));
    if (nsw == 0 && F.in == F.out) return;

    if (threadIdx.x < W) prog[threadIdx.x] = -1;
    if (threadIdx.x == 0) {
        s_gave_up = 0;
        s_giveup = GiveUp{&s_gave_up, 0};
        for (int i = 0; i < W * SCS; ++i) tc::mbar_init(&scbar[i], 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    for (int i = threadIdx.x; i < R::IDLEN; i += blockDim.x) ident[i] = make_double2(0.0, 1.0);
    // columns in: segment s is a column (order s / SEGC), its doubles in memory order
    constexpr int SEGC = NC / ES;                 // columns of an order
    const int rowsN = R::rows(N), len = N * ES;
    // positions outside the chains (and the second chain's last one of an odd column): zero
    for (int i = threadIdx.x; i < ROW; i += blockDim.x) col[i - ROW] = 0.0;
    for (int i = N / CH * ROW + threadIdx.x; i < (rowsN - 1) * ROW; i += blockDim.x) col[i] = 0.0;
    __syncthreads();
    auto column_at = [&](int s, long long * at) -> bool {
        const int o = s / SEGC, m = mbase + STEP * o;
        long long c;
        if (KIND == TRI || KIND == RECT) c = m;
        else if (KIND == SPIN) c = 2LL * m - (task.side ? 0 : 1);
        else c = 2LL * m - 1 + s % SEGC;
        *at = c * ES * F.lda;
        return m <= mlast && c >= 0 && c < F.M;
    };
    auto place = [&](int s, int x) -> int {       // double x of segment s
        const int row = x / ES, h = ES == 2 ? x % 2 : s % SEGC;
        return row / CH * ROW + (s / SEGC * NC + h) * CH + row % CH;
    };
    const int nblk = (nsw + B - 1) / B;
    double2 * const sc_ring = pairs + warp * SCS * SCLEN;
    uint64_t * const bars = scbar + warp * SCS;
    unsigned sc_issued = 0, sc_used = 0;
    // the warp's block: its lowest sweep, highest chunk, steps of a chunk, pairs
    int i0 = 0, chi = 0, K = 0, nk = 0;
    const double2 * rows = nullptr;
    unsigned live = 0;          // bit i: the pairs of chunk k + i are staged
    auto stage_sc = [&](int k) -> bool {
        const int kappa = HI2LO ? chi + D - k : k;
        if (k >= K || kappa >= nk) return false;
        if (lane == 0) {
            uint64_t * const bar = &bars[sc_issued % SCS];
            tc::mbar_arrive_expect_tx(bar, (uint32_t) (SCLEN * sizeof(double2)));
            tc::bulk_g2s(sc_ring + (sc_issued % SCS) * SCLEN, rows + kappa * Geo::skew_chunk(KIND), (uint32_t) (SCLEN * sizeof(double2)), bar);
        }
        ++sc_issued;
        return true;
    };
    auto begin = [&](int g) {
        i0 = (jlo - jpar) / STEP + (HI2LO ? nblk - 1 - g : g) * B;
        // chunk c covers positions cE .. cE + E - 1 (hi2lo, from the highest with a rotation down)
        // or cE - 1 .. cE + E - 2 (lo2hi, from 0 up), aligned as the skewed table is
        const int last = Geo::chain_len(KIND, N, 0) - 1;
        const int emax = max(0, min(last, Geo::top(KIND, N, jpar + STEP * i0, 0) + 1));
        chi = HI2LO ? emax / E : (emax + 1) / E;
        K = chi + 1 + D;
        const int beta = i0 / Geo::kSkewRows;
        nk = beta < Geo::skew_blocks(KIND, N, jpar) ? Geo::skew_chunks(KIND, N, jpar, beta) : 0;
        rows = F.sc + Geo::skew_at(KIND, N, jpar, beta);
        live = 0;
#pragma unroll
        for (int i = 0; i + 1 < SCS; ++i) live |= stage_sc(i) ? 1u << i : 0u;
    };
    if (warp < nblk) begin(warp);                 // its first pairs land while the columns do
    // a warp's columns together, so that their loads are in flight at the same time
    constexpr int SW = ORD * SEGC / W;
    static_assert(ORD * SEGC % W == 0, "the columns must split evenly over the warps");
    {
        const double * from[SW];
#pragma unroll
        for (int i = 0; i < SW; ++i) {
            long long at;
            from[i] = column_at(warp + i * W, &at) ? F.in + at : nullptr;
        }
#pragma unroll 2
        for (int x = lane; x < len; x += 32) {
            double v[SW];
#pragma unroll
            for (int i = 0; i < SW; ++i) v[i] = from[i] ? __ldcg(from[i] + x) : 0.0;
#pragma unroll
            for (int i = 0; i < SW; ++i) col[place(warp + i * W, x)] = v[i];
        }
    }
    __syncthreads();

    const int c_lane = lane % CH, m_lane = mbase + STEP * (lane / (CH * NC));
    const int me_lane = KIND == SPIN ? abs(m_lane - F.spin) : m_lane;
    const int jcut = F.blk > 0 ? m_lane - STEP * (((m_lane - jpar) / STEP) % F.blk) : jpar;
    for (int g = warp; g < nblk; g += W) {
        unsigned lane_mask = 0;
#pragma unroll
        for (int b = 0; b < B; ++b) {
            const int j = jpar + STEP * (HI2LO ? i0 + B - 1 - b : i0 + b);
            if (j <= me_lane - STEP && j >= jcut) lane_mask |= 1u << b;
        }
        double win[2 * B];
#pragma unroll
        for (int x = 0; x < 2 * B; ++x) win[x] = 0.0;
        // The warp's word: block g, and how far down the columns it is final (hi2lo: every chunk >= c
        // as 2048 - c, lo2hi: every chunk <= c as c + 1).  Chunks above a block's own in hi2lo order
        // have not been touched by the blocks before it either.
        volatile int * const mine = &prog[warp];
        const int * const before = &prog[(warp + W - 1) % W];
        if (lane == 0) *mine = g * 4096 + (HI2LO ? 2048 - (chi + 1) : 0);
        int seen = -2;
        for (int k = 0; k < K; ++k) {
            live |= stage_sc(k + SCS - 1) ? 1u << (SCS - 1) : 0u;
            const bool has_in = k <= chi, has_out = k >= D;
            const int cin = HI2LO ? chi - k : k, cout = HI2LO ? cin + D : cin - D;
            if (has_in && g > 0) {
                const int need = (g - 1) * 4096 + (HI2LO ? 2048 - cin : cin + 1);
                if (seen < need) seen = wait_word(before, need);
            }
            // position of the chunk's first step, and the way the steps go
            const double * const bin = col + (HI2LO ? cin * E + E - 1 : cin * E - 1) * ROW + lane;
            double * const bout = col + (HI2LO ? cout * E + E - 1 : cout * E - 1) * ROW + lane;
            const bool odd = D > 1 && (k & 1);
            if (live & 1u) {
                const int slot = sc_used % SCS;
                wait_bar(&bars[slot], (sc_used / SCS) & 1);
                ++sc_used;
                const double2 * sc[B];
#pragma unroll
                for (int b = 0; b < B; ++b)
                    sc[b] = ((lane_mask >> b) & 1u ? sc_ring + slot * SCLEN + (HI2LO ? B - 1 - b : b) * E * CH : ident) + c_lane;
                if (odd) resident_steps<HI2LO, CH, B, E, E % (2 * B), ROW, true>(win, bin, bout, has_in, has_out, sc);
                else     resident_steps<HI2LO, CH, B, E, 0, ROW, true>(win, bin, bout, has_in, has_out, sc);
            } else {
                const double2 * const none[B] = {};
                if (odd) resident_steps<HI2LO, CH, B, E, E % (2 * B), ROW, false>(win, bin, bout, has_in, has_out, none);
                else     resident_steps<HI2LO, CH, B, E, 0, ROW, false>(win, bin, bout, has_in, has_out, none);
            }
            live >>= 1;
            __syncwarp();
            if (lane == 0 && has_out) publish_word(&prog[warp], g * 4096 + (k + 1 == K ? 4095 : HI2LO ? 2048 - cout : cout + 1));
        }
        if (g + W < nblk) begin(g + W);
    }
    for (; sc_used != sc_issued; ++sc_used) {     // only after a wait that ran out: no copy may outlive the CTA
        const long long t0 = clock64();
        while (!tc::mbar_try_wait(&bars[sc_used % SCS], (sc_used / SCS) & 1) && clock64() - t0 < (1LL << 24)) {}
    }
    __syncthreads();
    for (int s = warp; s < ORD * SEGC; s += W) {
        long long at;
        if (!column_at(s, &at)) continue;
#pragma unroll 4
        for (int x = lane; x < len; x += 32) __stcg(F.out + at + x, col[place(s, x)]);
    }
}

// Resident CTAs cover a field's whole columns, so they take it when its chains fit.
template <int KIND>
bool resident_fits(const RotLaunch & L) {
    for (int f = 0; f < L.nfields; ++f)
        if (RT<KIND>::bytes(L.fields[f].N) + 1024 > 232448 || Geo::chain_len(KIND, L.fields[f].N, 0) / RT<KIND>::E > 2000) return false;
    return true;
}

template <int KIND, bool HI2LO>
cudaError_t launch_resident(const RotLaunch & L, cudaStream_t st) {
    using R = RT<KIND>;
    auto kern = rot_resident_kernel<KIND, HI2LO>;
    int nmax = 0;
    for (int f = 0; f < L.nfields; ++f) nmax = std::max(nmax, L.fields[f].N);
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    static std::atomic<bool> ready[16] = {};
    if (dev >= 16 || !ready[dev].load(std::memory_order_acquire)) {
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448 - 1024);
        if (e != cudaSuccess) return e;
        if (dev < 16) ready[dev].store(true, std::memory_order_release);
    }
    count_launch();
    return launch_overlapped(kern, dim3(L.ntasks * R::SPLIT), R::W * 32, R::bytes(nmax), st, L);
}

}  // namespace

// Launch shapes: 0 .. 4 rot_kernel with W stage warps x B sweeps per warp, chunk E; 5
// rot_resident_kernel.
//   0: 8 x 8 x 16    1: 8 x 8 x 8    2: 4 x 8 x 8, one CTA per SM
// with one sequence a lane (half the orders a group, twice the groups):
//   3: 8 x 8 x 8, one CTA per SM    4: 4 x 8 x 16, two CTAs per SM
// Shape 4 is the heads' (one pass of at most 31 sweeps): two CTAs with chunks of 16 fit because a ring
// holds half the columns, and a stage's 16 steps have no second copy for the other half of its window.
// us a launch, against 4 x 8 x 8 with both sequences a lane, two CTAs per SM: sph 4095 x 16 fields 4667 /
// 4804, 2047 x 8 657 / 729, 1023 x 8 201 / 231, disk 1500 x 6 589 / 735, tri 767 x 12 180 / 200; whole
// sweeps through the pipeline sph 1024 269 / 395, disk 700 355 / 543.
template <int KIND, bool HI2LO>
cudaError_t launch_kind(int cfg, const RotLaunch & L, int max_ctas, cudaStream_t st) {
    constexpr int NC = order_sequences(KIND);
    if (cfg == 5 && resident_fits<KIND>(L)) return launch_resident<KIND, HI2LO>(L, st);
    if (cfg == 1) return launch_cfg<KIND, NC, HI2LO, 8, 8, 8, 1>(L, max_ctas, 0, st);
    if (cfg == 2) return launch_cfg<KIND, NC, HI2LO, 4, 8, 8, 2>(L, max_ctas, 1, st);
    if (cfg == 3) return launch_cfg<KIND, 1, HI2LO, 8, 8, 8, 1>(L, max_ctas, 1, st);
    if (cfg == 4) return launch_cfg<KIND, 1, HI2LO, 4, 8, 16, 2>(L, max_ctas, 0, st);
    return launch_cfg<KIND, NC, HI2LO, 8, 8, 16, 1>(L, max_ctas, 0, st);
}

int g_rot_cfg = -2;

// A configuration is a launch shape 0 .. 5 plus 8 x a pass-pipeline mode 0 .. 2
// (schedule_passes).  FT_B200_ROT_CFG forces one (as does ft_b200_set_rotation_config);
// otherwise -1 (chosen per launch shape).
constexpr int kPipeModes = 3;
bool valid_config(int cfg) { return cfg >= 0 && (cfg & 7) <= 5 && cfg < 8 * kPipeModes; }

int rotation_config() {
    if (g_rot_cfg == -2) {
        const char * e = std::getenv("FT_B200_ROT_CFG");
        const int v = e ? std::atoi(e) : -1;
        g_rot_cfg = (e && e[0] >= '0' && e[0] <= '9' && valid_config(v)) ? v : -1;
    }
    return g_rot_cfg;
}

void set_rotation_config(int cfg) { g_rot_cfg = valid_config(cfg) ? cfg : -1; }

struct RotSchedule {
    std::vector<RotTask> tasks;                          // host copy of the device list (same order)
    struct Units { RotChain * d_chains = nullptr; int * d_words = nullptr; int n = 0, nprog = 0; };   // words: counter, progress
    std::map<std::tuple<int, int, int>, Units> lists;    // (sweeps per pass and split, heads only, mode) -> queue
    std::mutex mu;
};

RotSchedule * rot_schedule_new(const std::vector<RotTask> & tasks) {
    RotSchedule * s = new RotSchedule();
    s->tasks = tasks;
    return s;
}

void rot_schedule_free(RotSchedule * s) {
    if (!s) return;
    for (auto & kv : s->lists) cudaFree(kv.second.d_chains);   // the words are in the same allocation
    delete s;
}

bool rotation_plan_skew(ft_rotation_plan * RP) {
    if (RP->d_skew) { cudaFree(RP->d_skew); RP->d_skew = nullptr; }
    const long long len = std::max(1LL, Geo::skew_len(RP->kind, RP->n));
    cudaError_t e = cudaMalloc(&RP->d_skew, sizeof(double2) * len);
    if (e != cudaSuccess) {
        RP->d_skew = nullptr;
        set_error(e == cudaErrorMemoryAllocation ? FT_B200_ENOMEM : FT_B200_ECUDA, std::string("cudaMalloc(skewed table): ") + cudaGetErrorString(e));
        return false;
    }
    const dim3 grid((unsigned) std::max(1, Geo::skew_blocks(RP->kind, RP->n, 0)), (unsigned) Geo::skew_parities(RP->kind));
    skew_table_kernel<<<grid, 256>>>(RP->d_sc, RP->d_skew, RP->kind, RP->n);
    count_launch();
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e != cudaSuccess) {
        set_error(FT_B200_ECUDA, std::string("skew_table_kernel: ") + cudaGetErrorString(e));
        return false;
    }
    return true;
}

int rotation_status(int value) {
    int v = 0;
    if (cudaMemcpyFromSymbol(&v, g_rot_status, sizeof(int)) != cudaSuccess) return -1;
    if (v != value && cudaMemcpyToSymbol(g_rot_status, &value, sizeof(int)) != cudaSuccess) return -1;
    return v;
}

namespace {

// Sweeps per pass (W x B) of each launch shape.
int shape_pass(int cfg) {
    static const int wb[6] = {64, 64, 32, 64, 32, 64};
    return (cfg >= 0 && cfg < 6) ? wb[cfg] : 64;
}
// Groups that a shape makes of a task of the list (Shape::SPLIT).
int shape_split(int cfg, int kind) { return cfg == 3 || cfg == 4 ? order_sequences(kind) : 1; }

// The queue of the pass pipeline for L's tasks with passes of wb sweeps, built on first use;
// null when the stream is capturing then (the upload synchronises) or on an allocation
// failure.  One entry per pass, pass-major (every task's pass r before any task's pass r + 1,
// tasks in list order, longest first), so a pass's predecessor is always pulled first: a
// pass rarely waits long for it, but consecutive passes of a task run far apart in time, so
// its columns leave L2 between them when the matrix is large.  (Splitting each task into a
// few entries that take every D-th pass side by side, which keeps the columns in L2, measured
// slower at every size: a CTA whose entry waits for its task's previous pass cannot take
// other work meanwhile.)
// mode 2 (bounded): pass-major over only the longest tasks whose columns fit in half the L2
// (so consecutive passes of a task still find them there), then every other task as one
// entry running all its passes, longest first: the long tasks no longer end the launch alone,
// and the short ones fill in at the end.
const RotSchedule::Units * schedule_passes(RotSchedule * S, int kind, const RotLaunch & L, int wb, int split, int mode, cudaStream_t st) {
    const int blk = L.fields[0].blk;
    std::lock_guard<std::mutex> lk(S->mu);
    const auto key = std::make_tuple(wb * 8 + split, blk > 0 ? 1 : 0, mode);
    auto it = S->lists.find(key);
    if (it != S->lists.end()) return it->second.d_chains ? &it->second : nullptr;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) return nullptr;
    const int nt = (int) S->tasks.size() * split, orders = Geo::task_orders(kind) / split;   // groups, and their orders
    std::vector<int> npass(nt, 0), prog0(nt, 0);
    int nprog = 0, maxp = 0;
    for (int t = 0; t < nt; ++t) {
        const RotTask & T = S->tasks[t / split];
        const RotField & F = L.fields[T.field];
        const int mbase = T.mbase + Geo::step(kind) * orders * (t % split);
        int jlo, jhi;
        const int nsw = mbase > Geo::last_order(kind, F.M) ? 0 : Geo::task_sweeps(kind, F.M, mbase, F.blk, &jlo, &jhi, F.spin, orders);
        npass[t] = (nsw + wb - 1) / wb;
        prog0[t] = nprog;
        nprog += npass[t];
        maxp = std::max(maxp, npass[t]);
    }
    // tasks pipelined pass by pass: all (mode 1), or the longest ones (the list is longest first)
    // whose columns fit in half the L2 (mode 2)
    int npipe = nt;
    if (mode == 2) {
        int dev = 0, l2 = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, dev);
        const int seqs = (kind == TRI || kind == RECT) ? 1 : 2;   // doubles per order and row
        const long long cols = (long long) orders * seqs;
        const long long foot = cols * (long long) L.fields[0].N * (long long) sizeof(double);
        npipe = (int) std::min<long long>(nt, std::max<long long>(1, (l2 / 2) / std::max<long long>(foot, 1)));
    }
    std::vector<RotChain> q;   // entry: pass r of task t alone (stride npass), or all of its passes
    for (int r = 0; r < maxp; ++r)
        for (int t = 0; t < npipe; ++t)
            if (r < npass[t]) q.push_back(RotChain{t, prog0[t], r, npass[t]});
    for (int t = npipe; t < nt; ++t)
        if (npass[t] > 0) q.push_back(RotChain{t, prog0[t], 0, 1});
    RotSchedule::Units U;
    U.n = (int) q.size();
    U.nprog = nprog;
    if (U.n > 0) {
        const size_t list = (sizeof(RotChain) * q.size() + 255) & ~(size_t) 255;
        if (cudaMalloc(&U.d_chains, list + sizeof(int) * (size_t) (kProgLead + nprog)) != cudaSuccess ||
            cudaMemcpy(U.d_chains, q.data(), sizeof(RotChain) * q.size(), cudaMemcpyHostToDevice) != cudaSuccess) {
            cudaFree(U.d_chains);
            U = RotSchedule::Units{};
        } else {
            U.d_words = reinterpret_cast<int *>(reinterpret_cast<char *>(U.d_chains) + list);
        }
    }
    S->lists[key] = U;
    return U.d_chains ? &S->lists[key] : nullptr;
}

cudaError_t launch_with(int kind, bool hi2lo, int cfg, const RotLaunch & L, int max_ctas, cudaStream_t st) {
    switch (kind) {
        case SPH:  return hi2lo ? launch_kind<SPH, true>(cfg, L, max_ctas, st) : launch_kind<SPH, false>(cfg, L, max_ctas, st);
        case TRI:  return hi2lo ? launch_kind<TRI, true>(cfg, L, max_ctas, st) : launch_kind<TRI, false>(cfg, L, max_ctas, st);
        case DISK: return hi2lo ? launch_kind<DISK, true>(cfg, L, max_ctas, st) : launch_kind<DISK, false>(cfg, L, max_ctas, st);
        case SPIN: return hi2lo ? launch_kind<SPIN, true>(cfg, L, max_ctas, st) : launch_kind<SPIN, false>(cfg, L, max_ctas, st);
        case RECT: return hi2lo ? launch_kind<RECT, true>(cfg, L, max_ctas, st) : launch_kind<RECT, false>(cfg, L, max_ctas, st);
    }
    return cudaErrorInvalidValue;
}

bool resident_fits(int kind, const RotLaunch & L) {
    switch (kind) {
        case SPH:  return resident_fits<SPH>(L);
        case TRI:  return resident_fits<TRI>(L);
        case DISK: return resident_fits<DISK>(L);
        case SPIN: return resident_fits<SPIN>(L);
        case RECT: return resident_fits<RECT>(L);
    }
    return false;
}

// One launch in configuration cfg: shape cfg & 7, through the pass pipeline in mode cfg >> 3
// (schedule_passes) when the task list has a schedule (else, and in mode 0, each CTA runs
// every pass of its tasks).  The progress words are the call's own (prog_call) when it has
// them, else the schedule's.
cudaError_t launch_shape(int kind, bool hi2lo, int cfg, const RotLaunch & L, int max_ctas, cudaStream_t st,
                         RotSchedule * sched, int * prog_call = nullptr, int prog_cap = 0) {
    const int shape = cfg & 7, mode = cfg >> 3;
    if (shape == 5 && resident_fits(kind, L)) return launch_with(kind, hi2lo, shape, L, max_ctas, st);   // no queue
    const RotSchedule::Units * U = (mode > 0 && sched) ? schedule_passes(sched, kind, L, shape_pass(shape), shape_split(shape, kind), mode, st) : nullptr;
    // a call with words of its own too few for this queue runs whole tasks per CTA instead
    if (!U || (prog_call && U->nprog > prog_cap)) return launch_with(kind, hi2lo, shape, L, max_ctas, st);
    int * const words = prog_call ? prog_call - kProgLead : U->d_words;
    static thread_local RotLaunch P;
    P = L;
    P.chains = U->d_chains;
    P.nchains = U->n;
    P.counter = words;
    P.prog = words + kProgLead;
    P.counter0 = (int) 0x80808080;   // the fill also puts the progress words below any position
    const cudaError_t e = cudaMemsetAsync(words, 0x80, sizeof(int) * (size_t) (kProgLead + U->nprog), st);
    if (e != cudaSuccess) return e;
    return launch_with(kind, hi2lo, shape, P, max_ctas, st);
}

// Configuration without measurements (in-place launches, capturing streams, the spin and tetrahedral
// sweeps).  Measured per launch in us, one field in place, resident / 8 x 8 x 8 with one sequence a
// lane (tri, rect: 4 x 8 x 8) / 8 x 8 x 16, the last two through the pass pipeline:
//   sph 301 60 / 70 / 98, 600 141 / 141 / 204, 767 203 / 182 / 266, 1024 320 / 288 / 365,
//       1200 425 / 414 / 455, 1500 - / 710 / 603, 2048 - / 1670 / 1210
//   disk 301 142 / 158 / 200, 400 210 / 182 / 275, 700 555 / 375 / 505, 1024 - / 890 / 803
//   spin 512 147 / 155 / 202, 767 273 / 307 / 340, 1024 530 / 560 / 491
//   tri 301 133 / 134 / 138, 400 208 / 164 / 180, 1001 - / 450 / 475, 2048 - / 2400 / 1500
//   rect 301 58 / 72 / 73, 512 107 / 111 / 114, 767 199 / 162 / 173, 1024 316 / 235 / 240
// A launch of few passes is bound by the longest task's passes following each other, and a stage
// follows the one before at 2B + E steps, a step taking a warp four cycles per FP64 instruction.
// Resident columns have no passes, and win until a CTA's own work, which grows with the cube of n,
// takes over: chains of 300 positions, more where their CTAs fill the chip.  Then one sequence a
// lane halves a step, at half the rotations per (sin, cos) load, until about 400 passes of 64
// sweeps give every SM enough of them for throughput to count.
int default_config(int kind, const RotLaunch & L, RotSchedule * sched, cudaStream_t st) {
    if (L.nfields > 0 && L.fields[0].blk > 0) return 4;   // at most 31 sweeps a column: one pass
    const bool pair = order_sequences(kind) == 2;
    int len = 0;
    for (int f = 0; f < L.nfields; ++f) len = std::max(len, Geo::chain_len(kind, L.fields[f].N, 0));
    const int ctas = L.ntasks * order_sequences(kind);    // of the resident kernel
    const RotSchedule::Units * const U =
        sched && len > (pair && ctas >= 148 ? 400 : 300) ? schedule_passes(sched, kind, L, shape_pass(0), 1, 1, st) : nullptr;
    if (!U) return 5;             // whole tasks: resident where they fit, else 8 x 8 x 16
    if (pair) return U->n <= 400 ? 8 + 3 : 8;
    return U->n <= 300 ? 8 + 2 : 8;
}

// The autotuner's choices, by launch shape: family, direction, heads only or all sweeps,
// fields, tasks, and the first field's N and M (the tasks of a shape are the same).
std::mutex g_tune_mu;
std::map<std::string, int> g_tuned;

std::string shape_key(int kind, bool hi2lo, const RotLaunch & L) {
    char k[160];
    std::snprintf(k, sizeof k, "%d/%d/%d/%d/%d/%d/%d", kind, hi2lo ? 1 : 0, L.fields[0].blk > 0 ? 1 : 0, L.nfields,
                  L.ntasks, L.fields[0].N, L.fields[0].M);
    return k;
}

bool autotune_enabled() {
    static const bool on = [] {
        const char * e = std::getenv("FT_B200_AUTOTUNE");
        return !(e && e[0] == '0');
    }();
    return on;
}

// Times every configuration once (after one untimed launch) with CUDA events on the
// launch stream, on a copy of L whose fields read and write only dead[f] (memory whose
// contents the caller no longer needs, at least the field's N x M at its leading
// dimension); returns the fastest, or -1 if a launch or an event failed.  The rotation
// kernel's cost does not depend on the values, and every configuration computes the same
// results bit for bit (each element meets its rotations in the same order).
int tune(int kind, bool hi2lo, const RotLaunch & L, double * const * dead, int max_ctas, cudaStream_t st,
         RotSchedule * sched, int * prog_call, int prog_cap) {
    static thread_local RotLaunch S;
    S = L;
    for (int f = 0; f < L.nfields; ++f) { S.fields[f].in = dead[f]; S.fields[f].out = dead[f]; }
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    if (cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess) {
        if (e0) cudaEventDestroy(e0);
        return -1;
    }
    int best = -1;
    float best_ms = 0.0f;
    // every shape, each also through the pass pipeline when the list has a schedule (it
    // spreads a task's passes over SMs: worth it when there are few tasks, not when the
    // columns would leave L2 between passes)
    for (int cfg = 0; cfg < 8 * kPipeModes; ++cfg) {
        if ((cfg & 7) > 5) continue;
        // head sweeps are one pass in every shape: the pipeline's queue is the task list again
        if ((cfg >> 3) && (!sched || L.fields[0].blk > 0)) continue;
        if (launch_shape(kind, hi2lo, cfg, S, max_ctas, st, sched, prog_call, prog_cap) != cudaSuccess) { best = -1; break; }
        if (cudaEventRecord(e0, st) != cudaSuccess) { best = -1; break; }
        if (launch_shape(kind, hi2lo, cfg, S, max_ctas, st, sched, prog_call, prog_cap) != cudaSuccess) { best = -1; break; }
        float ms = 0.0f;
        if (cudaEventRecord(e1, st) != cudaSuccess || cudaEventSynchronize(e1) != cudaSuccess ||
            cudaEventElapsedTime(&ms, e0, e1) != cudaSuccess) { best = -1; break; }
        if (best < 0 || ms < best_ms) { best = cfg; best_ms = ms; }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    return best;
}

}  // namespace

cudaError_t launch_rotations(int kind, bool hi2lo, const RotLaunch & L, int max_ctas, cudaStream_t st,
                             double * const * dead, RotSchedule * sched, int * prog_call, int prog_cap) {
    if (L.ntasks <= 0) return cudaSuccess;
    int cfg = rotation_config();
    if (cfg < 0) {
        cfg = -1;
        if (autotune_enabled() && L.nfields > 0) {
            const std::string key = shape_key(kind, hi2lo, L);
            int known = -1;
            {
                std::lock_guard<std::mutex> lk(g_tune_mu);
                auto it = g_tuned.find(key);
                if (it != g_tuned.end()) known = it->second;
            }
            cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
            if (known >= 0) {
                cfg = known;
            } else if (dead && cudaStreamIsCapturing(st, &cs) == cudaSuccess && cs == cudaStreamCaptureStatusNone) {
                const int t = tune(kind, hi2lo, L, dead, max_ctas, st, sched, prog_call, prog_cap);
                if (t >= 0) {
                    std::lock_guard<std::mutex> lk(g_tune_mu);
                    g_tuned[key] = t;
                    cfg = t;
                }
            }
        }
    }
    if (cfg < 0) cfg = default_config(kind, L, sched, st);
    return launch_shape(kind, hi2lo, cfg, L, max_ctas, st, sched, prog_call, prog_cap);
}


}  // namespace ftb
