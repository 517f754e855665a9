// Device kernels of the multi-RHS block solve: k <= 32 right-hand sides of one system,
// each running the reference's BiCGSTAB (AFIIM/src/bicgstab.cpp:168-275) with its own
// scalars and termination, sharing every sparse product.
//
// Vectors are n x k, row-major (entry (i, j) at i*k + j), so the k values a gathered
// column index needs are contiguous. Work mapping: a lane group of L lanes (a power of two)
// takes one row and each lane owns VW consecutive right-hand sides (lane l: columns l*VW ..
// l*VW + VW - 1; VW = 1, 2 or 4, loaded as one or two 16-byte pairs); a warp holds 32/L row
// groups. The vector updates walk the rows in grid-stride order with VW = 1 and L = next power of
// two >= k; the sparse products walk chunks of consecutive rows of about equal work and take their
// (L, VW) from the solver's shape (the row groups per warp and the load width), which never changes
// a product. Sparse products: the group's entries are loaded L at a time (coalesced) and handed
// to every lane one by one, so each right-hand side's row sum is formed left to right in storage
// order with rounded products (the reference's arithmetic, bit for bit).
// Reductions are per right-hand side: lanes of equal j are combined within the warp and
// the CTA in a fixed tree, the CTA writes k partials, and the last CTA (ticket) adds them
// in a fixed order and runs each right-hand side's scalar step.
#pragma once

#include "fiim_batch.cuh"
#include "fiim_kernels.cuh"

namespace fiim {
namespace bk {

using bt::BState;

struct Shape {
    long n;
    int k;        // right-hand sides
};

// Per-RHS reduction over the CTA and the grid; every thread calls it (uniformly). A thread
// holds the partials of its VW right-hand sides (lane % L) * VW + u, u < VW.
template <int L, int VW, int NR, class Fin>
__device__ __forceinline__ void rhs_reduce(double (&v)[VW][NR], int k, double *__restrict__ partials, BState &bs,
                                           const Fin &fin) {
    __shared__ double sm[kWarps][32][NR];
    __shared__ int last;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    // combine the row groups of the warp (lanes with the same right-hand sides)
#pragma unroll
    for (int u = 0; u < VW; ++u)
#pragma unroll
        for (int j = 0; j < NR; ++j)
#pragma unroll
            for (int o = L; o < 32; o <<= 1) v[u][j] += __shfl_xor_sync(0xffffffffu, v[u][j], o);
    if (lane < L)
#pragma unroll
        for (int u = 0; u < VW; ++u)
#pragma unroll
            for (int j = 0; j < NR; ++j) sm[w][lane * VW + u][j] = v[u][j];
    __syncthreads();
    if (threadIdx.x < k) {
        const int jj = threadIdx.x;
#pragma unroll
        for (int j = 0; j < NR; ++j) {
            double s = 0.0;
#pragma unroll
            for (int q = 0; q < kWarps; ++q) s += sm[q][jj][j];
            partials[((size_t)blockIdx.x * 32 + jj) * NR + j] = s;
        }
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned t = atomicAdd(bs.ticket, 1u);
        last = (t == gridDim.x - 1);
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    // warp w adds the CTAs w, w + 8, ... of lane j's right-hand side; the warps are added in order
    // (one thread a right-hand side over every CTA was a serial chain of 600 L2 loads; with the
    // updates' loads ahead of their stores, 150 us less an iteration at n = 200,003, k = 32)
    double tot[NR];
#pragma unroll
    for (int j = 0; j < NR; ++j) tot[j] = 0.0;
    if (lane < k)
#pragma unroll 8
        for (int c = w; c < (int)gridDim.x; c += kWarps)
#pragma unroll
            for (int j = 0; j < NR; ++j) tot[j] += __ldcg(partials + ((size_t)c * 32 + lane) * NR + j);
#pragma unroll
    for (int j = 0; j < NR; ++j) sm[w][lane][j] = tot[j];
    __syncthreads();
    if (threadIdx.x < k) {
#pragma unroll
        for (int j = 0; j < NR; ++j) {
            tot[j] = 0.0;
#pragma unroll
            for (int q = 0; q < kWarps; ++q) tot[j] += sm[q][lane][j];
        }
        if (!bs.done[lane] || !Fin::GATED) fin.finish(bs, lane, tot);
    }
    __syncthreads();
    if (threadIdx.x == 0) *bs.ticket = 0u;
}

// ---------------------------------------------------------------- epilogues
// emit_pre(at, s, q, red) finishes entry `at` of the n x k output block from its row sum s and
// its operand q = pre(at, row), which can be loaded before the sum is ready;
// emit2(at, s0, s1, red0, red1) finishes the two consecutive entries at, at + 1 (at even)
// with the same arithmetic per entry, reading and writing both as one 16-byte pair (the
// sparse products with two or four right-hand sides per lane).
#define FIIM_BEPI(nr, reduces, gated)            \
    static constexpr int NR = nr;                \
    static constexpr bool REDUCES = reduces;     \
    static constexpr bool GATED = gated

__device__ __forceinline__ void st2(double *p, double a, double b) { *reinterpret_cast<double2 *>(p) = make_double2(a, b); }
__device__ __forceinline__ double2 ld2(const double *__restrict__ p) { return __ldg(reinterpret_cast<const double2 *>(p)); }

struct KEpiStore {
    FIIM_BEPI(1, false, true);
    double *y;
    __device__ double pre(size_t, long) const { return 0.0; }
    __device__ void emit_pre(size_t at, double s, double, double (&)[NR]) const { y[at] = s; }
    __device__ void emit2(size_t at, double s0, double s1, double (&)[NR], double (&)[NR]) const { st2(y + at, s0, s1); }
    __device__ void finish(BState &, int, const double *) const {}
};
struct KEpiScale {                 // y = d o (M x), d per row
    FIIM_BEPI(1, false, true);
    double *y;
    const double *__restrict__ d;
    int k;
    __device__ double pre(size_t, long row) const { return __ldg(d + row); }
    __device__ void emit_pre(size_t at, double s, double di, double (&)[NR]) const { y[at] = __dmul_rn(di, s); }
    __device__ void emit2(size_t at, double s0, double s1, double (&)[NR], double (&)[NR]) const {
        const double di = __ldg(d + at / k);
        st2(y + at, __dmul_rn(di, s0), __dmul_rn(di, s1));
    }
    __device__ void finish(BState &, int, const double *) const {}
};
struct KEpiNorm {
    FIIM_BEPI(1, true, true);
    double *y;
    __device__ double pre(size_t, long) const { return 0.0; }
    __device__ void emit_pre(size_t at, double s, double, double (&r)[NR]) const { y[at] = s; r[0] += s * s; }
    __device__ void emit2(size_t at, double s0, double s1, double (&ra)[NR], double (&rb)[NR]) const {
        st2(y + at, s0, s1);
        ra[0] += s0 * s0;
        rb[0] += s1 * s1;
    }
    __device__ void finish(BState &bs, int j, const double *t) const { bs.pc2[j] = t[0]; }
};
struct KEpiAlpha {
    FIIM_BEPI(1, true, true);
    double *y;
    const double *__restrict__ r0;
    __device__ double pre(size_t at, long) const { return __ldg(r0 + at); }
    __device__ void emit_pre(size_t at, double s, double q, double (&r)[NR]) const {
        y[at] = s;
        r[0] += q * s;
    }
    __device__ void emit2(size_t at, double s0, double s1, double (&ra)[NR], double (&rb)[NR]) const {
        st2(y + at, s0, s1);
        const double2 q = ld2(r0 + at);
        ra[0] += q.x * s0;
        rb[0] += q.y * s1;
    }
    __device__ void finish(BState &bs, int j, const double *t) const { bt::BFinAlpha{}.finish(bs, j, t); }
};
struct KEpiOmega {
    FIIM_BEPI(2, true, true);
    double *y;
    const double *__restrict__ sv;
    __device__ double pre(size_t at, long) const { return __ldg(sv + at); }
    __device__ void emit_pre(size_t at, double s, double q, double (&r)[NR]) const {
        y[at] = s;
        r[0] += s * q;
        r[1] += s * s;
    }
    __device__ void emit2(size_t at, double s0, double s1, double (&ra)[NR], double (&rb)[NR]) const {
        st2(y + at, s0, s1);
        const double2 q = ld2(sv + at);
        ra[0] += s0 * q.x;
        ra[1] += s0 * s0;
        rb[0] += s1 * q.y;
        rb[1] += s1 * s1;
    }
    __device__ void finish(BState &bs, int j, const double *t) const { bs.omega[j] = t[0] / t[1]; }
};
struct KEpiInit {
    FIIM_BEPI(1, true, true);
    const double *__restrict__ b;
    double *p, *r0, *r;
    __device__ double pre(size_t at, long) const { return b[at]; }
    __device__ void emit_pre(size_t at, double s, double bi, double (&red)[NR]) const {
        const double pi = __dadd_rn(bi, __dmul_rn(-1.0, s));
        p[at] = pi;
        r0[at] = pi;
        r[at] = pi;
        red[0] += pi * pi;
    }
    __device__ void emit2(size_t at, double s0, double s1, double (&ra)[NR], double (&rb)[NR]) const {
        const double2 q = ld2(b + at);
        const double p0 = __dadd_rn(q.x, __dmul_rn(-1.0, s0)), p1 = __dadd_rn(q.y, __dmul_rn(-1.0, s1));
        st2(p + at, p0, p1);
        st2(r0 + at, p0, p1);
        st2(r + at, p0, p1);
        ra[0] += p0 * p0;
        rb[0] += p1 * p1;
    }
    __device__ void finish(BState &bs, int j, const double *t) const { bt::BFinInit{}.finish(bs, j, t); }
};
struct KEpiRestart : KEpiInit {
    __device__ void finish(BState &bs, int j, const double *t) const { bt::BFinRestart{}.finish(bs, j, t); }
};
struct KEpiResid {
    FIIM_BEPI(2, true, false);
    const double *__restrict__ b;
    __device__ double pre(size_t at, long) const { return b[at]; }
    __device__ void emit_pre(size_t at, double s, double bi, double (&red)[NR]) const {
        const double ri = bi - s;
        red[0] += ri * ri;
        red[1] += bi * bi;
    }
    __device__ void emit2(size_t at, double s0, double s1, double (&ra)[NR], double (&rb)[NR]) const {
        const double2 q = ld2(b + at);
        const double ri0 = q.x - s0, ri1 = q.y - s1;
        ra[0] += ri0 * ri0;
        ra[1] += q.x * q.x;
        rb[0] += ri1 * ri1;
        rb[1] += q.y * q.y;
    }
    __device__ void finish(BState &bs, int j, const double *t) const {
        bs.ts[j] = t[0];
        bs.tt[j] = t[1];
    }
};

__device__ __forceinline__ double wide(double v) { return v; }
__device__ __forceinline__ double wide(float v) { return (double)v; }

// ---------------------------------------------------------------- SpMM
// chunk[ch] .. chunk[ch + 1] are the rows of chunk ch (BlockSolver::set_chunks), one a warp: as many
// as the chip holds of the one-value-a-lane kernels (4 CTAs an SM below, 6 in k_spmm), so that each
// warp has one run of consecutive rows and all end together. Rows dealt one by one left the warps
// with the long rows of a power-law matrix running on alone, and two or four chunks a warp were
// 5 to 40% slower than one. k_spmm with DEAL takes matrices of even rows: a chunk is one step of the
// warp, and they are dealt out in order.
#define FIIM_CHUNKS(ch)                                                                       \
    for (int ch = (int)(((long)blockIdx.x * kThreads + threadIdx.x) >> 5); ch < nch;          \
         ch += (int)(((long)gridDim.x * kThreads) >> 5))

// X's VW values of one gathered row for a lane, from a 16-byte aligned address when VW > 1
// (VW > 1 needs an even k and VW | k, so that row * k + l * VW is a multiple of VW).
template <int VW>
__device__ __forceinline__ void gather(const double *__restrict__ p, double (&x)[VW]) {
    if constexpr (VW == 1) {
        x[0] = __ldg(p);
    } else {
#pragma unroll
        for (int u = 0; u < VW; u += 2) {
            const double2 d = __ldg(reinterpret_cast<const double2 *>(p + u));
            x[u] = d.x;
            x[u + 1] = d.y;
        }
    }
}

template <int L, int VW, typename V, typename Epi, bool DEAL>
static __global__ void __launch_bounds__(kThreads, VW == 1 ? (DEAL ? 8 : 6) : 1)
k_spmm(CsrView<V> M, Shape sh, const int *__restrict__ chunk, int nch, const double *__restrict__ X, Epi epi, BState bs,
       double *__restrict__ partials) {
    if (Epi::GATED && bs.g->active <= 0) return;
    double red[VW][Epi::NR];
#pragma unroll
    for (int u = 0; u < VW; ++u)
#pragma unroll
        for (int q = 0; q < Epi::NR; ++q) red[u][q] = 0.0;
    const int lane_ = threadIdx.x & 31, j_ = lane_ % L, grp_ = lane_ / L;
    FIIM_CHUNKS(ch)
    for (long base = DEAL ? ch * (32L / L) : __ldg(chunk + ch),
              last_ = DEAL ? min(base + 32 / L, (long)M.n) : __ldg(chunk + ch + 1); base < last_; base += 32 / L) {
        const long row = base + grp_;
        const bool live = row < last_;
        const int j0 = j_ * VW;            // this lane's first right-hand side
        int beg = 0, len = 0;
        if (live) {
            beg = __ldg(M.rp + row);
            len = __ldg(M.rp + row + 1) - beg;
        }
        // every group of the warp walks the longest row of the warp (uniform shuffles), and
        // within a trip only as many entries as the longest remaining row part holds
        const int trips = __reduce_max_sync(0xffffffffu, (len + L - 1) / L);
        double s[VW];
#pragma unroll
        for (int u = 0; u < VW; ++u) s[u] = 0.0;
        for (int t = 0; t < trips; ++t) {
            const int q = t * L + j_;
            int c = 0;
            double a = 0.0;
            if (q < len) {
                c = ldi(M.ci + beg + q);
                a = wide(ldm(M.v + beg + q));
            }
            const int ne = (int)__reduce_max_sync(0xffffffffu, (unsigned)max(0, min(L, len - t * L)));
#pragma unroll 4
            for (int e = 0; e < ne; ++e) {
                const int ce = __shfl_sync(0xffffffffu, c, grp_ * L + e);
                const double ae = __shfl_sync(0xffffffffu, a, grp_ * L + e);
                if (t * L + e < len && j0 < sh.k) {
                    double xv[VW];
                    gather<VW>(X + (size_t)ce * sh.k + j0, xv);
#pragma unroll
                    for (int u = 0; u < VW; ++u) s[u] = __dadd_rn(s[u], __dmul_rn(ae, xv[u]));
                }
            }
        }
        if (live && j0 < sh.k) {
            const size_t at = (size_t)row * sh.k + j0;
            bool all = true;   // every right-hand side of this lane still running
            if constexpr (Epi::GATED)
#pragma unroll
                for (int u = 0; u < VW; ++u) all = all && !bs.done[j0 + u];
            if (VW > 1 && all) {
#pragma unroll
                for (int u = 0; u < VW; u += 2) epi.emit2(at + u, s[u], s[u + 1], red[u], red[u + 1]);
            } else {
#pragma unroll
                for (int u = 0; u < VW; ++u)
                    if (!(Epi::GATED && bs.done[j0 + u])) epi.emit_pre(at + u, s[u], epi.pre(at + u, row), red[u]);
            }
        }
    }
    if constexpr (Epi::REDUCES) rhs_reduce<L, VW, Epi::NR>(red, sh.k, partials, bs, epi);
}

// 17 to 32 right-hand sides, one a lane: a warp walks its chunk's entries as one stream, whatever
// rows they belong to. What bounds the product is the gathers (8 k bytes an entry, from L2) and the
// instructions around them, so: the gathers of eight entries are in flight before the first is
// added, across row ends; entries reach the lanes through 512 bytes of shared memory a warp, one
// broadcast each with the column already times k (three shuffles and a product before); eight
// entries of one row are added without looking for its end; the next 32 entries are loaded while
// these are added, and a row's epilogue operand when the row begins. Row sums in storage order, as
// everywhere. Power-law matrix, n = 200,003, 2.9 M entries, 32 right-hand sides: A X 445 -> 152 us,
// M X (FP32 factors) 176 -> 133, an iteration 1.53 -> 0.60 ms with the shorter reductions and
// updates of this file.
// Its int positions run up to two tiles past a run's end, so a matrix whose entries come that close to 2^31
// keeps k_spmm, whose positions start at a row. (Positions compared by what is left, here, took 1.2% more:
// 6.68 -> 6.76 ms for the ten iterations of the system above.)
inline bool streams(long nnz) { return nnz <= INT_MAX - 64; }

template <typename V, typename Epi>
static __global__ void __launch_bounds__(kThreads, 4)
k_spmm_stream(CsrView<V> M, Shape sh, const int *__restrict__ chunk, int nch, const double *__restrict__ X, Epi epi, BState bs,
              double *__restrict__ partials) {
    if (Epi::GATED && bs.g->active <= 0) return;
    constexpr int AHEAD = 8;
    const unsigned full = 0xffffffffu;
    __shared__ longlong2 tile[kWarps][32];   // a warp's 32 entries: the value's bits, column * k
    const int lane = (int)threadIdx.x & 31;
    longlong2 *const mytile = tile[threadIdx.x >> 5];
    const double *const Xl = X + lane;
    const bool mine = lane < sh.k, out = mine && !(Epi::GATED && bs.done[lane]);
    double red[1][Epi::NR];
#pragma unroll
    for (int q = 0; q < Epi::NR; ++q) red[0][q] = 0.0;
    FIIM_CHUNKS(ch) {
        const int r0 = __ldg(chunk + ch), r1 = __ldg(chunk + ch + 1);
        int row = r0, held = r0;   // rows held .. held + 31 end where the lanes say
        int ends = held + lane < r1 ? __ldg(M.rp + held + lane + 1) : 0;
        const int e0 = __ldg(M.rp + r0), e1 = __ldg(M.rp + r1);
        int end = __shfl_sync(full, ends, 0);
        double s = 0.0, op = out ? epi.pre((size_t)row * sh.k + lane, row) : 0.0;
        auto finish_row = [&] {
            if (out) epi.emit_pre((size_t)row * sh.k + lane, s, op, red[0]);
            s = 0.0;
            if (++row - held == 32) {
                held = row;
                ends = held + lane < r1 ? __ldg(M.rp + held + lane + 1) : 0;
            }
            end = __shfl_sync(full, ends, row - held);
            op = out && row < r1 ? epi.pre((size_t)row * sh.k + lane, row) : 0.0;
        };
        int c = e0 + lane < e1 ? ldi(M.ci + e0 + lane) : 0;
        V a = e0 + lane < e1 ? ldm(M.v + e0 + lane) : V(0);
        for (int t = e0; t < e1; t += 32) {
            __syncwarp();   // the last tile is read
            mytile[lane] = make_longlong2(__double_as_longlong(wide(a)), (long long)c * sh.k);
            __syncwarp();
            if (t + 32 + lane < e1) {
                c = ldi(M.ci + t + 32 + lane);
                a = ldm(M.v + t + 32 + lane);
            }
            const int m = min(32, e1 - t);
            for (int u0 = 0; u0 < m; u0 += AHEAD) {
                double xv[AHEAD], au[AHEAD];
#pragma unroll
                for (int u = 0; u < AHEAD; ++u) {   // past the last entry: an older one, not added
                    const longlong2 e = mytile[u0 + u];
                    au[u] = __longlong_as_double(e.x);
                    xv[u] = mine ? __ldg(Xl + e.y) : 0.0;
                }
                while (t + u0 == end) finish_row();
                if (t + u0 + AHEAD <= end) {   // all of one row
#pragma unroll
                    for (int u = 0; u < AHEAD; ++u) s = __dadd_rn(s, __dmul_rn(au[u], xv[u]));
                } else {
#pragma unroll
                    for (int u = 0; u < AHEAD; ++u)
                        if (u0 + u < m) {
                            if (u > 0)
                                while (t + u0 + u == end) finish_row();
                            s = __dadd_rn(s, __dmul_rn(au[u], xv[u]));
                        }
                }
            }
        }
        while (row < r1) finish_row();
    }
    if constexpr (Epi::REDUCES) rhs_reduce<32, 1, Epi::NR>(red, sh.k, partials, bs, epi);
}

// ---------------------------------------------------------------- updates (n x k)
struct KFinS {
    static constexpr bool GATED = true;
    __device__ void finish(BState &bs, int j, const double *t) const { bt::BFinS{}.finish(bs, j, t); }
};
struct KFinControl {
    static constexpr bool GATED = true;
    __device__ void finish(BState &bs, int j, const double *t) const { bt::BFinControl{}.finish(bs, j, t); }
};

// Four rows' operands are read before any result is written (the compiler must assume the vectors
// alias), each thread's terms still added in row order.
constexpr int kRows = 4;
#define FIIM_ROWS_BY_4(KP)                                                                    \
    const int lane_ = threadIdx.x & 31, j_ = lane_ % (KP), grp_ = lane_ / (KP);               \
    const long nw_ = ((long)gridDim.x * kThreads) >> 5, gw_ = ((long)blockIdx.x * kThreads + threadIdx.x) >> 5; \
    const bool run_ = j_ < sh.k && !bs.done[j_];                                              \
    for (long row0 = gw_ * (32 / (KP)) + grp_; run_ && row0 < sh.n; row0 += kRows * nw_ * (32 / (KP)))
#define FIIM_ROW(KP, u) (row0 + (u) * nw_ * (32 / (KP)))

template <int KP>
static __global__ void __launch_bounds__(kThreads)
k_kupdate_s(Shape sh, const double *__restrict__ r, const double *__restrict__ v, const double *__restrict__ x,
            double *__restrict__ s, BState bs, double *__restrict__ partials) {
    if (bs.g->active <= 0) return;
    double red[1][2] = {{0.0, 0.0}};
    FIIM_ROWS_BY_4(KP) {
        const double a = -bs.alpha[j_];
        double ri[kRows], xi[kRows], vi[kRows];
#pragma unroll
        for (int u = 0; u < kRows; ++u) {
            const long row = FIIM_ROW(KP, u);
            const size_t at = (size_t)row * sh.k + j_;
            const bool in = row < sh.n;
            ri[u] = in ? r[at] : 0.0;
            xi[u] = in ? x[at] : 0.0;
            vi[u] = in ? v[at] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < kRows; ++u) {
            const long row = FIIM_ROW(KP, u);
            if (row < sh.n) s[(size_t)row * sh.k + j_] = __dadd_rn(ri[u], __dmul_rn(a, vi[u]));
            red[0][0] += ri[u] * ri[u];
            red[0][1] += xi[u] * xi[u];
        }
    }
    rhs_reduce<KP, 1, 2>(red, sh.k, partials, bs, KFinS{});
}

template <int KP>
static __global__ void __launch_bounds__(kThreads)
k_kupdate_xr(Shape sh, const double *__restrict__ pc, const double *__restrict__ sc, const double *__restrict__ s,
             const double *__restrict__ t, const double *__restrict__ r0, double *__restrict__ x,
             double *__restrict__ r, BState bs, double *__restrict__ partials) {
    if (bs.g->active <= 0) return;
    double red[1][1] = {{0.0}};
    FIIM_ROWS_BY_4(KP) {
        const double a = bs.alpha[j_], om = bs.omega[j_];
        double xi[kRows], pi[kRows], ci[kRows], si[kRows], ti[kRows], qi[kRows];
#pragma unroll
        for (int u = 0; u < kRows; ++u) {
            const long row = FIIM_ROW(KP, u);
            const size_t at = (size_t)row * sh.k + j_;
            const bool in = row < sh.n;
            xi[u] = in ? x[at] : 0.0;
            pi[u] = in ? pc[at] : 0.0;
            ci[u] = in ? sc[at] : 0.0;
            si[u] = in ? s[at] : 0.0;
            ti[u] = in ? t[at] : 0.0;
            qi[u] = in ? r0[at] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < kRows; ++u) {
            const long row = FIIM_ROW(KP, u);
            if (row >= sh.n) break;
            const size_t at = (size_t)row * sh.k + j_;
            x[at] = __dadd_rn(__dadd_rn(xi[u], __dmul_rn(a, pi[u])), __dmul_rn(om, ci[u]));
            const double ri = __dadd_rn(si[u], __dmul_rn(-om, ti[u]));
            r[at] = ri;
            red[0][0] += qi[u] * ri;
        }
    }
    rhs_reduce<KP, 1, 1>(red, sh.k, partials, bs, KFinControl{});
}

template <int KP>
static __global__ void __launch_bounds__(kThreads)
k_kupdate_p(Shape sh, const double *__restrict__ r, const double *__restrict__ v, double *__restrict__ p, BState bs,
            cudaGraphConditionalHandle h, int cond) {
    if (cond && blockIdx.x == 0 && threadIdx.x == 0) {
        const int loops = ++bs.g->loops;
        if (bs.g->active > 0 && loops > bs.g->nmax + 2) bs.g->active = -1;
        cudaGraphSetConditional(h, bs.g->active > 0 ? 1u : 0u);
    }
    if (bs.g->active <= 0) return;
    FIIM_ROWS_BY_4(KP) {
        const double b = bs.beta[j_], c = __dmul_rn(-b, bs.omega[j_]);
        double ri[kRows], vi[kRows], pi[kRows];
#pragma unroll
        for (int u = 0; u < kRows; ++u) {
            const long row = FIIM_ROW(KP, u);
            const size_t at = (size_t)row * sh.k + j_;
            const bool in = row < sh.n;
            ri[u] = in ? r[at] : 0.0;
            vi[u] = in ? v[at] : 0.0;
            pi[u] = in ? p[at] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < kRows; ++u) {
            const long row = FIIM_ROW(KP, u);
            if (row >= sh.n) break;
            p[(size_t)row * sh.k + j_] = __dadd_rn(__dadd_rn(__dmul_rn(c, vi[u]), __dmul_rn(b, pi[u])), ri[u]);
        }
    }
}

}  // namespace bk
}  // namespace fiim
