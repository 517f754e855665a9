// PDFIIM factor construction on the GPU: the same G, D^{-1} and H as the host construction
// (fiim_pdfiim.cpp), and so as the reference's pdfiim (PDFIIM/src/parPrec.cpp:95-588) for
// pattern 'B', bit for bit. One warp builds one row i at a time:
//   * the row's pattern, an insertion-ordered set, lives in the warp's shared memory; a
//     row of A or A^T is merged into it 32 entries at a time, the absent columns appended in
//     column order (the same order as one-by-one insertion, since a row's columns are
//     distinct);
//   * the dense LU with partial pivoting of the pattern's B (Golub & Van Loan Alg. 3.4.1,
//     first largest pivot) eliminates one row per lane; every product and difference is
//     rounded separately, as the host code compiled without contraction;
//   * the triangular solves, the filter norms and the D^{-1} sums add in the host's sequential
//     order; products and independent sums are spread over the lanes;
//   * kept entries are sorted by index through their ranks.
// One pass over the rows leaves every row's entries and D^{-1} in the next free places; running
// totals of the counts and a transpose, all on the device, put them in order, and the second call
// copies them from there into the caller's arrays. A row whose pattern outgrows the warp's shared
// memory (CAP members in a solve, 4 CAP in the set; 2048 at the largest CAP) is listed and built
// again with a larger CAP; past the largest CAP the call returns FIIM_EARG and the host
// construction serves.

#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstring>
#include <memory>
#include <new>
#include <type_traits>
#include <vector>

#include "fiim_b200.h"
#include "fiim_internal.h"
#include "fiim_kernels.cuh"

namespace fiim {
namespace pg {

struct CsrD {
    const int *rp, *ci;
    const double *v;
};

struct Params {
    int prefill, lfill, postfill, warpsize;
    double ftol;
    char filttype;
};

struct Out {
    int *gcnt, *hcnt;           // kept entries + unit diagonal, per row
    double *D;
    long *at;                   // a row's first entry in ej / ev: g's, then h's
    int *ej;
    double *ev;
    unsigned long long *used;   // entries asked for so far
    unsigned long long room;    // entries ej and ev hold
    int *overflow, *noverflow;  // rows left for a larger CAP
};

template <int CAP>
struct WarpSmem {
    // Set capacity: 4 CAP, and 2048 at the largest CAP, where a warpsize cap keeps the solve
    // small while wide rows (random columns, hundreds of entries) still grow the set.
    static constexpr int SET = CAP >= 128 ? 2048 : 4 * CAP;
    int list[SET];
    int inds[CAP];
    int piv[CAP];
    int rank[CAP];
    double g[CAP], h[CAP];
    double B[CAP * CAP];
};

__device__ __forceinline__ unsigned lanemask_lt() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

template <int CAP>
struct RowBuilder {
    WarpSmem<CAP> &s;
    const CsrD &A, &At;
    const int i, lane;
    int size = 0;
    bool over = false;

    __device__ RowBuilder(WarpSmem<CAP> &s_, const CsrD &A_, const CsrD &At_, int i_)
        : s(s_), A(A_), At(At_), i(i_), lane((int)(threadIdx.x & 31)) {}

    // Columns < i of row j of M, appended in column order where absent.
    __device__ void push_row_below(const CsrD &M, int j) {
        if (over) return;
        const int beg = M.rp[j], end = M.rp[j + 1];
        for (int base = beg; base < end; base += 32) {
            const int k = base + lane;
            const int c = k < end ? M.ci[k] : INT_MAX;
            const bool valid = c < i;
            bool present = false;
            if (valid)
                for (int q = 0; q < size; ++q)
                    if (s.list[q] == c) {
                        present = true;
                        break;
                    }
            const unsigned add = __ballot_sync(0xffffffffu, valid && !present);
            if (valid && !present) {
                const int at = size + __popc(add & lanemask_lt());
                if (at < WarpSmem<CAP>::SET) s.list[at] = c;
            }
            size += __popc(add);
            if (size > WarpSmem<CAP>::SET) over = true;
            __syncwarp();
            if (!__all_sync(0xffffffffu, valid) || over) break;
        }
    }

    __device__ int pos_of(int c, int len) const {
        for (int q = 0; q < len; ++q)
            if (s.inds[q] == c) return q;
        return -1;
    }

    // x at the pattern's members from -(row i of M), columns below i; a column stored twice
    // counts as its last entry does.
    __device__ void assemble(const CsrD &M, double *x, int len) {
        const int beg = M.rp[i], end = M.rp[i + 1];
        for (int base = beg; base < end; base += 32) {
            const int k = base + lane;
            const int c = k < end ? M.ci[k] : INT_MAX;
            const int q = c < i ? pos_of(c, len) : -1;
            const unsigned same = __match_any_sync(0xffffffffu, q);
            if (q >= 0 && (same >> lane) == 1u) x[q] = -M.v[k];
            __syncwarp();
        }
    }

    // LU with partial pivoting of B (len x len, row-major), then B g = g, B^T h = h.
    __device__ void factor_solve(int len) {
        double *B = s.B;
        for (int k = 0; k < len; ++k) {
            // First row of largest |B(r, k)|, r >= k, as a sequential scan from r = k finds it
            // (a NaN at (k, k) keeps row k, a NaN below is never taken).
            int p = len;
            if constexpr (CAP <= 32) {
                // One row a lane: the largest upper word decides, and the lower words only where
                // several lanes share it (upper words of non-negative doubles order as they do).
                const double v = lane >= k && lane < len ? fabs(B[lane * len + k]) : nan("");
                const bool in = !isnan(v);
                const unsigned hi = in ? (unsigned)__double2hiint(v) : 0u;
                const unsigned top = __reduce_max_sync(0xffffffffu, hi);   // every lane, before any test
                unsigned at = __ballot_sync(0xffffffffu, in && hi == top);
                if (at & (at - 1u)) {   // the same in every lane
                    const bool tie = at >> lane & 1u;
                    const unsigned lo = tie ? (unsigned)__double2loint(v) : 0u;
                    const unsigned low = __reduce_max_sync(0xffffffffu, lo);
                    at = __ballot_sync(0xffffffffu, tie && lo == low);
                }
                if (at) p = __ffs(at) - 1;
            } else {
                double best = -1.0;
                for (int r = k + lane; r < len; r += 32) {
                    const double v = fabs(B[r * len + k]);
                    if (v > best) {
                        best = v;
                        p = r;
                    }
                }
                for (int o = 16; o > 0; o >>= 1) {
                    const double ob = __shfl_xor_sync(0xffffffffu, best, o);
                    const int op = __shfl_xor_sync(0xffffffffu, p, o);
                    if (ob > best || (ob == best && op < p)) {
                        best = ob;
                        p = op;
                    }
                }
            }
            if (isnan(B[k * len + k])) p = k;
            if (lane == 0) s.piv[k] = p;
            __syncwarp();
            if (B[p * len + k] == 0.0) continue;
            if (p != k)
                for (int c = lane; c < len; c += 32) {
                    const double t = B[k * len + c];
                    B[k * len + c] = B[p * len + c];
                    B[p * len + c] = t;
                }
            __syncwarp();
            const double d = B[k * len + k];
            for (int r = k + 1 + lane; r < len; r += 32) {
                const double l = B[r * len + k] / d;
                B[r * len + k] = l;
                // four entries of the row in flight: the compiler cannot tell the rows apart
                double *Br = B + r * len;
                const double *Bk = B + k * len;
                int c = k + 1;
                for (; c + 4 <= len; c += 4) {
                    double q[4], p[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        q[u] = Br[c + u];
                        p[u] = Bk[c + u];
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u) Br[c + u] = __dsub_rn(q[u], __dmul_rn(l, p[u]));
                }
                for (; c < len; ++c) Br[c] = __dsub_rn(Br[c], __dmul_rn(l, Bk[c]));
            }
            __syncwarp();
        }
        solve_pair(len);
    }

    // B g = g and B^T h = h with the factors of factor_solve, both at once. Each unknown's sum is
    // subtracted in ascending order of the other unknown's index, as a sequential solve does. The
    // forward solves go column by column over the lanes, which is that order. A backward solve
    // needs its row's products lowest index first, so the lanes form them and one lane
    // subtracts them: lane 0 for g, lane 1 for h, whose chains are as long. (Lane 0 doing all four
    // solves alone was three quarters of the kernel.) The products lie in the set's list, which is
    // written again after the solve.
    __device__ void solve_pair(int len) {
        static_assert(WarpSmem<CAP>::SET * sizeof(int) >= 2 * CAP * sizeof(double), "two rows of products");
        const double *B = s.B;
        double *g = s.g, *h = s.h, *pg = reinterpret_cast<double *>(s.list), *ph = pg + CAP;
        const int *piv = s.piv;
        if (lane == 0)
            for (int k = 0; k < len; ++k)
                if (piv[k] != k) {
                    const double t = g[k];
                    g[k] = g[piv[k]];
                    g[piv[k]] = t;
                }
        __syncwarp();
        for (int c = 0; c < len; ++c) {
            const double gc = g[c], hc = h[c] / B[c * len + c];
            __syncwarp();
            if (lane == 0) h[c] = hc;
            for (int r = c + 1 + lane; r < len; r += 32) {
                g[r] = __dsub_rn(g[r], __dmul_rn(B[r * len + c], gc));
                h[r] = __dsub_rn(h[r], __dmul_rn(B[c * len + r], hc));
            }
            __syncwarp();
        }
        for (int r = len - 1; r >= 0; --r) {
            for (int c = r + 1 + lane; c < len; c += 32) {
                pg[c] = __dmul_rn(B[r * len + c], g[c]);
                ph[c] = __dmul_rn(B[c * len + r], h[c]);
            }
            __syncwarp();
            if (lane < 2) {
                const double *p = lane ? ph : pg;
                double acc = lane ? h[r] : g[r];
                int c = r + 1;
                for (; c + 4 <= len; c += 4) {
                    double q[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) q[u] = p[c + u];
#pragma unroll
                    for (int u = 0; u < 4; ++u) acc = __dsub_rn(acc, q[u]);
                }
                for (; c < len; ++c) acc = __dsub_rn(acc, p[c]);
                if (lane) h[r] = acc;
                else g[r] = acc / B[r * len + r];
            }
            __syncwarp();
        }
        if (lane == 0)
            for (int k = len - 1; k >= 0; --k)
                if (piv[k] != k) {
                    const double t = h[k];
                    h[k] = h[piv[k]];
                    h[piv[k]] = t;
                }
        __syncwarp();
    }
};

__device__ double filter_norm(char filttype, const double *x, int len) {
    double nrm = 1.0;
    if (filttype == '1') {
        for (int j = 0; j < len; ++j) nrm = __dadd_rn(nrm, fabs(x[j]));
        nrm = nrm / (double)(len + 1);
    } else if (filttype == '2') {
        for (int j = 0; j < len; ++j) nrm = __dadd_rn(nrm, __dmul_rn(x[j], x[j]));
        nrm = sqrt(nrm);
    } else {
        for (int j = 0; j < len; ++j) nrm = (nrm < fabs(x[j])) ? fabs(x[j]) : nrm;
    }
    return nrm;
}

// Rows rows[0..nrows) (or 1..n-1 when rows == NULL), one warp each.
template <int CAP>
static __global__ void __launch_bounds__(256)
k_pdfiim_rows(int n, const int *__restrict__ rows, int nrows, CsrD A, CsrD At, Params P, Out o) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    WarpSmem<CAP> &s = reinterpret_cast<WarpSmem<CAP> *>(smem_raw)[w];
    const long wid = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long nw = ((long)gridDim.x * blockDim.x) >> 5;
    const long total = rows ? nrows : (long)n - 1;
    const double floor_diag = fmax(1e-4, P.ftol);
    for (long t = wid; t < total; t += nw) {
        const int i = rows ? rows[t] : (int)(t + 1);
        RowBuilder<CAP> rb(s, A, At, i);
        // Level 1 and the pre-fill levels (parPrec.cpp:144-177), newest member first.
        rb.push_row_below(At, i);
        rb.push_row_below(A, i);
        for (int k = 2; k <= P.prefill && !rb.over; ++k) {
            const int len = rb.size;
            for (int q = len - 1; q >= 0 && !rb.over; --q) {
                const int jind = s.list[q];
                rb.push_row_below(At, jind);
                rb.push_row_below(A, jind);
            }
        }
        int tlen = 0;
        double ng = 0.0, nh = 0.0;
        for (int k = 1; k <= P.lfill && !rb.over; ++k) {
            ng = 0.0;
            int len = rb.size;
            tlen = len;
            if (len == 0) break;
            if (P.warpsize != -1)
                for (int j = len; j >= P.warpsize; --j) rb.size--;   // drop the newest members
            len = rb.size;
            tlen = len;
            if (len > CAP) {
                rb.over = true;
                break;
            }
            __syncwarp();
            for (int j = lane; j < len; j += 32) s.inds[j] = s.list[j];
            for (int q = lane; q < len * len; q += 32) s.B[q] = 0.0;
            for (int j = lane; j < len; j += 32) {
                s.g[j] = 0.0;
                s.h[j] = 0.0;
            }
            __syncwarp();
            // B = A restricted to the pattern (one row per lane, in storage order), with the
            // diagonal floor.
            for (int j = lane; j < len; j += 32) {
                const int row = s.inds[j];
                s.B[j * len + j] = floor_diag;
                for (int kk = A.rp[row]; kk < A.rp[row + 1] && A.ci[kk] < i; ++kk) {
                    const int q = rb.pos_of(A.ci[kk], len);
                    if (q >= 0) s.B[j * len + q] = A.v[kk];
                }
                if (s.B[j * len + j] == 0.0) s.B[j * len + j] = floor_diag;
            }
            __syncwarp();
            rb.assemble(At, s.g, len);   // g from A^T row i, h from A row i
            rb.assemble(A, s.h, len);
            __syncwarp();
            rb.factor_solve(len);
            const double norm = lane < 2 ? filter_norm(P.filttype, lane ? s.h : s.g, len) : 0.0;
            ng = __shfl_sync(0xffffffffu, norm, 0);
            nh = __shfl_sync(0xffffffffu, norm, 1);
            // New set: kept g entries in order, then kept h entries not yet in it.
            rb.size = 0;
            int c = 0, c2 = 0;
            for (int base = 0; base < len; base += 32) {
                const int j = base + lane;
                const bool kg = j < len && fabs(s.g[j]) >= P.ftol * ng;
                const unsigned m = __ballot_sync(0xffffffffu, kg);
                if (kg) s.list[rb.size + __popc(m & lanemask_lt())] = s.inds[j];
                rb.size += __popc(m);
                c += __popc(m);
            }
            for (int base = 0; base < len; base += 32) {
                const int j = base + lane;
                const bool kh = j < len && fabs(s.h[j]) >= P.ftol * nh;
                const bool kg = j < len && fabs(s.g[j]) >= P.ftol * ng;
                const unsigned mh = __ballot_sync(0xffffffffu, kh);
                const unsigned m = __ballot_sync(0xffffffffu, kh && !kg);
                if (kh && !kg) s.list[rb.size + __popc(m & lanemask_lt())] = s.inds[j];
                rb.size += __popc(m);
                c2 += __popc(mh);
            }
            __syncwarp();
            if ((c == 0 && c2 == 0) || c2 == P.warpsize) break;
            // The last level's growth reaches nothing the result depends on.
            if (k == P.lfill) break;
            // Next level set from the first |set| members of the solved pattern (parPrec.cpp:366-385).
            const int kept = rb.size;
            for (int j = 0; j < kept && !rb.over; ++j) {
                const int jind = s.inds[j];
                rb.push_row_below(At, jind);
                rb.push_row_below(A, jind);
            }
            for (int m = 2; m <= P.postfill && !rb.over; ++m) {
                const int len2 = rb.size;
                for (int q = len2 - 1; q >= 0 && !rb.over; --q) {
                    const int jind = s.list[q];
                    rb.push_row_below(At, jind);
                    rb.push_row_below(A, jind);
                }
            }
            if (rb.size == kept) break;
        }
        if (rb.over) {
            if (lane == 0) o.overflow[atomicAdd(o.noverflow, 1)] = i;
            __syncwarp();
            continue;
        }
        // Kept entries sorted by index (ranks), unit diagonal last (parPrec.cpp:460-500).
        int cnt[2] = {0, 0};
        for (int which = 0; which < 2; ++which) {
            const double *x = which == 0 ? s.g : s.h;
            const double nrm = which == 0 ? ng : nh;
            for (int j = lane; j < tlen; j += 32) {
                int r = -1;
                if (fabs(x[j]) >= P.ftol * nrm) {
                    r = 0;
                    for (int q = 0; q < tlen; ++q)
                        if (fabs(x[q]) >= P.ftol * nrm && s.inds[q] < s.inds[j]) ++r;
                }
                s.rank[j] = r;
            }
            int kc = 0;
            for (int base = 0; base < tlen; base += 32) {
                const int j = base + lane;
                kc += __popc(__ballot_sync(0xffffffffu, j < tlen && fabs(x[j]) >= P.ftol * nrm));
            }
            cnt[which] = kc;
            __syncwarp();
            if (which == 0)   // the ranks are used below: g's aside, in the list
                for (int j = lane; j < tlen; j += 32) s.list[j] = s.rank[j];
            __syncwarp();
        }
        // Entries to the next free places: g's and h's kept ones, each with its unit diagonal.
        const int gn = cnt[0] + 1, hn = cnt[1] + 1;
        unsigned long long at = 0;
        if (lane == 0) at = atomicAdd(o.used, (unsigned long long)(gn + hn));
        at = __shfl_sync(0xffffffffu, at, 0);
        if (lane == 0) {
            o.gcnt[i] = gn;
            o.hcnt[i] = hn;
            o.at[i] = (long)at;
        }
        if (at + gn + hn > o.room) {   // counted; the host makes room and runs the rows again
            __syncwarp();
            continue;
        }
        for (int which = 0; which < 2; ++which) {
            const double *x = which == 0 ? s.g : s.h;
            const int *rank = which == 0 ? s.list : s.rank;
            const long off = (long)at + (which == 0 ? 0 : gn);
            for (int j = lane; j < tlen; j += 32)
                if (rank[j] >= 0) {
                    o.ej[off + rank[j]] = s.inds[j];
                    o.ev[off + rank[j]] = x[j];
                }
            if (lane == 0) {
                o.ej[off + cnt[which]] = i;
                o.ev[off + cnt[which]] = 1.0;
            }
        }
        __syncwarp();
        // D^{-1}_i = 1 / sum_j h_j (A g)_j over the kept patterns (parPrec.cpp:502-532): each lane
        // takes entries of h, walks the row of A beside g's sorted entries and leaves its products
        // where the sequential sum takes them; one lane adds them.
        const int *gj = o.ej + at, *hj = gj + gn;
        const double *gv = o.ev + at, *hv = gv + gn;
        auto walk = [&](int j, auto hit) {
            const int hr = hj[j], end = A.rp[hr + 1];
            int kk = A.rp[hr], cc = 0;
            while (kk < end && cc < gn) {
                const int c = A.ci[kk], gc = gj[cc];
                if (c == gc) hit(kk, cc);
                if (c <= gc) ++kk;
                if (c >= gc) ++cc;
            }
        };
        double sum = 0.0;
        for (int base = 0; base < hn; base += 32) {
            const int j = base + lane;
            int hits = 0;
            if (j < hn) walk(j, [&](int, int) { ++hits; });
            int before = hits;
            for (int q = 1; q < 32; q <<= 1) {
                const int u = __shfl_up_sync(0xffffffffu, before, q);
                if (lane >= q) before += u;
            }
            const int all = __shfl_sync(0xffffffffu, before, 31);
            before -= hits;
            const bool fits = all <= CAP * CAP;   // B is free by now
            if (fits && j < hn) {
                const double hvj = hv[j];
                int put = before;
                walk(j, [&](int kk, int cc) { s.B[put++] = __dmul_rn(__dmul_rn(hvj, A.v[kk]), gv[cc]); });
            }
            __syncwarp();
            if (lane == 0) {
                if (fits) {
                    for (int q = 0; q < all; ++q) sum = __dadd_rn(sum, s.B[q]);
                } else {
                    for (int jj = base; jj < min(base + 32, hn); ++jj) {
                        const double hvj = hv[jj];
                        walk(jj, [&](int kk, int cc) {
                            sum = __dadd_rn(sum, __dmul_rn(__dmul_rn(hvj, A.v[kk]), gv[cc]));
                        });
                    }
                }
            }
            __syncwarp();
        }
        if (lane == 0) o.D[i] = 1.0 / sum;
        __syncwarp();
    }
}

// ---------------------------------------------------------------- transposes and offsets
// Counts, then their running totals over chunks of kScan (chunk sums, the sums' totals in one
// CTA, the chunks again), then entries to their rows in whatever order the threads arrive, then
// each row's entries to their ranks: the order a sequential counting sort gives.
constexpr int kScan = 4 * 1024;

static __global__ void __launch_bounds__(kThreads) k_count(long nnz, const int *__restrict__ c, int *cnt) {
    FIIM_FOR_ROWS(k, nnz) { atomicAdd(cnt + c[k], 1); }
}

__device__ __forceinline__ long block_scan(long v, long *all) {   // exclusive over 1,024 threads
    __shared__ long sm[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    long x = v;
    for (int o = 1; o < 32; o <<= 1) {
        const long u = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += u;
    }
    if (lane == 31) sm[w] = x;
    __syncthreads();
    if (w == 0) {
        long t = sm[lane];
        for (int o = 1; o < 32; o <<= 1) {
            const long u = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += u;
        }
        sm[lane] = t;
    }
    __syncthreads();
    const long out = x - v + (w ? sm[w - 1] : 0);
    *all = sm[31];
    __syncthreads();
    return out;
}

// sums[b]: the counts of chunk b.
static __global__ void __launch_bounds__(1024) k_scan_sums(int n, const int *__restrict__ cnt, long *sums) {
    long v = 0, all;
    for (int u = 0; u < 4; ++u) {
        const long i = (long)blockIdx.x * kScan + threadIdx.x * 4 + u;
        if (i < n) v += cnt[i];
    }
    block_scan(v, &all);
    if (threadIdx.x == 0) sums[blockIdx.x] = all;
}
// sums[b]: the counts before chunk b; sums[nb]: all of them. One CTA.
static __global__ void __launch_bounds__(1024) k_scan_top(int nb, long *sums) {
    long base = 0;
    for (int b0 = 0; b0 < nb; b0 += 1024) {
        const int b = b0 + (int)threadIdx.x;
        long all;
        const long before = block_scan(b < nb ? sums[b] : 0, &all);
        if (b < nb) sums[b] = base + before;
        base += all;
    }
    if (threadIdx.x == 0) sums[nb] = base;
}
// ptr[i], i <= n: the counts before i; next[i] the same, for the scatter (may be null).
static __global__ void __launch_bounds__(1024)
k_scan_write(int n, const int *__restrict__ cnt, const long *__restrict__ sums, int *ptr, int *next) {
    int c[4];
    long v = 0, all;
    for (int u = 0; u < 4; ++u) {
        const long i = (long)blockIdx.x * kScan + threadIdx.x * 4 + u;
        c[u] = i < n ? cnt[i] : 0;
        v += c[u];
    }
    long at = sums[blockIdx.x] + block_scan(v, &all);
    for (int u = 0; u < 4; ++u) {
        const long i = (long)blockIdx.x * kScan + threadIdx.x * 4 + u;
        if (i < n) {
            ptr[i] = (int)at;
            if (next) next[i] = (int)at;
        }
        at += c[u];
        if (i == n - 1) ptr[n] = (int)at;
    }
}

// Entries of a CSR matrix to their columns' lists: (position in the matrix, row).
static __global__ void __launch_bounds__(kThreads)
k_to_columns(int n, const int *__restrict__ rp, const int *__restrict__ ci, int *next, int *key, int *row) {
    FIIM_FOR_ROWS(r, n) {
        for (int k = rp[r]; k < rp[r + 1]; ++k) {
            const int q = atomicAdd(next + ci[k], 1);
            key[q] = k;
            row[q] = (int)r;
        }
    }
}
// Task i's g entries (rows ej, column i) counted by row, and then to their rows' lists.
static __global__ void __launch_bounds__(kThreads) k_count_g(int n, Out o, int *cnt) {
    FIIM_FOR_ROWS(i, n) {
        for (int q = 0; q < o.gcnt[i]; ++q) atomicAdd(cnt + o.ej[o.at[i] + q], 1);
    }
}
static __global__ void __launch_bounds__(kThreads) k_g_to_rows(int n, Out o, int *next, int *key, double *val) {
    FIIM_FOR_ROWS(i, n) {
        for (int q = 0; q < o.gcnt[i]; ++q) {
            const int at = atomicAdd(next + o.ej[o.at[i] + q], 1);
            key[at] = (int)i;
            val[at] = o.ev[o.at[i] + q];
        }
    }
}
// Task i's h entries are row i of H.
static __global__ void __launch_bounds__(kThreads) k_h_rows(int n, Out o, const int *__restrict__ Hi, int *Hj, double *Hv) {
    const int lane = (int)threadIdx.x & 31;
    for (long i = ((long)blockIdx.x * kThreads + threadIdx.x) >> 5; i < n; i += ((long)gridDim.x * kThreads) >> 5)
        for (int q = lane; q < o.hcnt[i]; q += 32) {
            Hj[Hi[i] + q] = o.ej[o.at[i] + o.gcnt[i] + q];
            Hv[Hi[i] + q] = o.ev[o.at[i] + o.gcnt[i] + q];
        }
}
// The lists ptr[c] .. ptr[c + 1] to ascending keys (distinct within a list): entry q moves to the
// place its key has among the list's. val null: the value is vals[key]. A warp per list, which compares
// every entry with every other; lists past kLong are noted for k_sort_long.
constexpr int kLong = 1024;
struct Lists {
    const int *ptr, *key, *idx;      // idx: what goes to oj (may be key)
    const double *val, *vals;
    int *oj;
    double *ov;
};
__device__ __forceinline__ void place(const Lists &l, int b, int e, int q) {
    const int key = l.key[q];
    int rank = 0;
    for (int p = b; p < e; ++p) rank += l.key[p] < key;
    l.oj[b + rank] = l.idx[q];
    l.ov[b + rank] = l.val ? l.val[q] : l.vals[key];
}
static __global__ void __launch_bounds__(kThreads) k_rank(int n, Lists l, int *longs, int *nlongs) {
    const int lane = (int)threadIdx.x & 31;
    for (long c = ((long)blockIdx.x * kThreads + threadIdx.x) >> 5; c < n; c += ((long)gridDim.x * kThreads) >> 5) {
        const int b = l.ptr[c], e = l.ptr[c + 1];
        if (e - b > kLong) {
            if (lane == 0) longs[atomicAdd(nlongs, 1)] = (int)c;
            continue;
        }
        for (int q = b + lane; q < e; q += 32) place(l, b, e, q);
    }
}
// The noted lists, a CTA each: a radix sort (Knuth, TAOCP 3, 5.2.5) of the entries' places by their keys, eight bits
// a pass from the lowest, `passes` of them. A pass counts the digits, then takes 1,024 entries at a time in order; a
// warp's entries of one digit are ranked by their lanes, the warps' counts added up in order. Places go back and
// forth between the lists' own outputs: oj's ints (after the last pass) and ov's storage. Linear in the list: with a
// column of 1.5 M entries over a band a construction takes 39 ms, 23 of them without the column; comparing every
// pair over the whole grid took 1,034 (0.4 M entries: 14 against 86).
static __global__ void __launch_bounds__(1024)
k_sort_long(Lists l, int passes, const int *__restrict__ longs, const int *__restrict__ nlongs) {
    __shared__ int base[256], part[32][256];   // next place of each digit; a tile's, by warp
    const unsigned tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    for (int k = (int)blockIdx.x; k < *nlongs; k += (int)gridDim.x) {
        const int b = l.ptr[longs[k]];
        const unsigned len = (unsigned)(l.ptr[longs[k] + 1] - b);
        const int *key = l.key + b, *from = nullptr;
        for (int p = 0; p < passes; ++p) {
            int *to = (passes - p) & 1 ? l.oj + b : reinterpret_cast<int *>(l.ov + b);
            auto entry = [&](unsigned r) { return from ? from[r] : (int)r; };
            auto digit = [&](int q) { return key[q] >> 8 * p & 255; };
            if (tid < 256) base[tid] = 0;
            __syncthreads();
            for (unsigned r = tid; r < len; r += 1024) atomicAdd(base + digit(entry(r)), 1);
            __syncthreads();
            if (w == 0) {
                int c[8], sum = 0;
                for (int u = 0; u < 8; ++u) {
                    c[u] = sum;
                    sum += base[8 * lane + u];
                }
                int before = sum;
                for (int o = 1; o < 32; o <<= 1) {
                    const int u = __shfl_up_sync(0xffffffffu, before, o);
                    if ((int)lane >= o) before += u;
                }
                before -= sum;
                for (int u = 0; u < 8; ++u) base[8 * lane + u] = before + c[u];
            }
            __syncthreads();
            for (unsigned t = 0; t < len; t += 1024) {
                const unsigned r = t + tid;
                const bool live = r < len;
                const int q = live ? entry(r) : 0, d = live ? digit(q) : 256;
                for (int u = 0; u < 8; ++u) part[w][lane + 32 * u] = 0;
                __syncwarp();
                const unsigned same = __match_any_sync(0xffffffffu, d);
                const int rank = __popc(same & lanemask_lt());
                if (live && rank == 0) part[w][d] = __popc(same);
                __syncthreads();
                if (tid < 256) {
                    int at = base[tid];
                    for (int v = 0; v < 32; ++v) {
                        const int c = part[v][tid];
                        part[v][tid] = at;
                        at += c;
                    }
                    base[tid] = at;
                }
                __syncthreads();
                if (live) to[part[w][d] + rank] = q;
                __syncwarp();
            }
            __syncthreads();
            from = to;
        }
        for (unsigned r = tid; r < len; r += 1024) {
            const int q = from[r];
            l.ov[b + r] = l.val ? l.val[b + q] : l.vals[key[q]];
            l.oj[b + r] = l.idx[b + q];
        }
        __syncthreads();
    }
}

template <int CAP>
int launch_rows(int n, const int *rows, int nrows, const CsrD &A, const CsrD &At, const Params &P, const Out &o,
                cudaStream_t st) {
    constexpr int warps = CAP <= 32 ? 8 : (CAP <= 64 ? 4 : 1);
    constexpr size_t smem = sizeof(WarpSmem<CAP>) * warps;
    auto kern = k_pdfiim_rows<CAP>;
    FIIM_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 0;
    FIIM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * warps, smem));
    const long total = rows ? nrows : (long)n - 1;
    const long need = (total + warps - 1) / warps;
    const int grid = (int)std::max<long>(1, std::min<long>(need, (long)std::max(per_sm, 1) * num_sms()));
    kern<<<grid, 32 * warps, smem, st>>>(n, rows, nrows, A, At, P, o);
    FIIM_CUDA(cudaGetLastError());
    return FIIM_OK;
}

// One device allocation carved into pieces.
struct Slab {
    char *p = nullptr;
    size_t used = 0, size = 0;
    Slab() = default;
    Slab(const Slab &) = delete;
    Slab &operator=(const Slab &) = delete;
    ~Slab() { release(); }
    void release() {
        if (p) cudaFree(p);
        p = nullptr;
        used = size = 0;
    }
    bool fits(size_t bytes) {
        release();
        size = bytes;
        if (cudaMalloc(&p, bytes) == cudaSuccess) return true;
        size = 0;
        cudaGetLastError();
        p = nullptr;
        return false;
    }
    int reserve(size_t bytes) {
        if (fits(bytes)) return FIIM_OK;
        return set_error(FIIM_ENOMEM, "device allocation of %zu bytes for the factor construction failed", bytes);
    }
    template <typename T>
    static size_t need(size_t count) {
        return Arena::need(sizeof(T) * std::max<size_t>(count, 1));
    }
    template <typename T>
    T *take(size_t count) {
        char *at = p + used;
        used += need<T>(count);
        return reinterpret_cast<T *>(at);
    }
};

// Factors built by the thread's last first call, until the second call copies them out (or another
// first call replaces them, or the thread ends): on the device up to kHeldMost bytes, which a caller that
// only asks for the sizes leaves there; larger ones in host memory, device = -1.
constexpr size_t kHeldMost = size_t(512) << 20;
struct BuiltGpu {
    int n = 0, device = -1;
    long nG = 0, nH = 0;
    Slab mem;
    std::unique_ptr<char[]> host;
    int *Gi = nullptr, *Gj = nullptr, *Hi = nullptr, *Hj = nullptr;
    double *Gv = nullptr, *Hv = nullptr, *D = nullptr;
    void clear() {
        mem.release();
        host.reset();
        n = 0;
    }
    // The arrays' places in one piece of memory that starts at p; its size.
    size_t carve(char *p, int rows) {
        size_t used = 0;
        auto take = [&](auto *&at, size_t count) {
            using T = std::remove_reference_t<decltype(*at)>;
            at = reinterpret_cast<T *>(p + used);
            used += Slab::need<T>(count);
        };
        take(Gi, (size_t)rows + 1);
        take(Hi, (size_t)rows + 1);
        take(D, (size_t)rows);
        take(Gj, (size_t)nG);
        take(Gv, (size_t)nG);
        take(Hj, (size_t)nH);
        take(Hv, (size_t)nH);
        return used;
    }
    int to_host(int dev);
    int order_on_host(const Out &o, int rows, cudaStream_t st);
};
thread_local BuiltGpu g_built_gpu;

constexpr int kCaps[3] = {32, 64, 128};

int run_cap(int cap, int n, const int *rows, int nrows, const CsrD &A, const CsrD &At, const Params &P, const Out &o,
            cudaStream_t st) {
    if (cap == 32) return launch_rows<32>(n, rows, nrows, A, At, P, o, st);
    if (cap == 64) return launch_rows<64>(n, rows, nrows, A, At, P, o, st);
    return launch_rows<128>(n, rows, nrows, A, At, P, o, st);
}

// ptr[0..n] (and next, if not null) from cnt[0..n) on st; sums: n / kScan + 2 longs of scratch.
int scan(int n, const int *cnt, long *sums, int *ptr, int *next, cudaStream_t st) {
    const int nb = (n + kScan - 1) / kScan;
    k_scan_sums<<<nb, 1024, 0, st>>>(n, cnt, sums);
    k_scan_top<<<1, 1024, 0, st>>>(nb, sums);
    k_scan_write<<<nb, 1024, 0, st>>>(n, cnt, sums, ptr, next);
    FIIM_CUDA(cudaGetLastError());
    return FIIM_OK;
}

// keys: what the lists' keys stay below.
int rank_lists(int n, const Lists &l, long keys, int *longs, int *nlongs, cudaStream_t st) {
    FIIM_CUDA(cudaMemsetAsync(nlongs, 0, sizeof(int), st));
    k_rank<<<grid_for(k_rank, kWarps, n), kThreads, 0, st>>>(n, l, longs, nlongs);
    int passes = 1;
    while (passes < 4 && keys > 1L << 8 * passes) ++passes;
    k_sort_long<<<num_sms(), 1024, 0, st>>>(l, passes, longs, nlongs);
    FIIM_CUDA(cudaGetLastError());
    return FIIM_OK;
}

int build_gpu(int n, const int *Ai, const int *Aj, const double *Av, const Params &P, BuiltGpu &out) {
    out.clear();
    int dev = -1;
    FIIM_TRY(check_device(&dev));
    const long nnz = Ai[n];
    cudaStream_t st = nullptr;
    FIIM_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    struct StreamGuard {
        cudaStream_t s;
        ~StreamGuard() {
            cudaStreamSynchronize(s);
            cudaStreamDestroy(s);
        }
    };
    Slab mem, entries;
    StreamGuard guard{st};   // after the slabs: synchronized before they go
    const int nb = (n + kScan - 1) / kScan;
    FIIM_TRY(mem.reserve(2 * Slab::need<int>(n + 1) + 2 * Slab::need<int>(nnz) + 2 * Slab::need<double>(nnz) +
                         7 * Slab::need<int>(n) + Slab::need<double>(n) + Slab::need<long>(n) + Slab::need<long>(nb + 1) +
                         3 * Slab::need<long>(1)));
    int *dAi = mem.take<int>(n + 1), *dTi = mem.take<int>(n + 1), *dAj = mem.take<int>(nnz), *dTj = mem.take<int>(nnz);
    double *dAv = mem.take<double>(nnz), *dTv = mem.take<double>(nnz), *dD = mem.take<double>(n);
    int *gcnt = mem.take<int>(n), *hcnt = mem.take<int>(n), *ovf = mem.take<int>(n), *rows2 = mem.take<int>(n),
        *cnt = mem.take<int>(n), *next = mem.take<int>(n), *longs = mem.take<int>(n);
    long *at = mem.take<long>(n), *sums = mem.take<long>(nb + 1);
    unsigned long long *used = mem.take<unsigned long long>(1);
    int *novf = mem.take<int>(1), *nlongs = mem.take<int>(1);
    // Room for four entries per entry of A and row; a construction that keeps more is counted, given exactly
    // what it needs, and run again. Where the device has not that much left, the first run only counts.
    // A^T's lists are made in the same room.
    auto entry_bytes = [](size_t count) { return Slab::need<int>(count) + Slab::need<double>(count); };
    unsigned long long room = 4ULL * (unsigned long long)(nnz + n), asked = 0;
    if (!entries.fits(entry_bytes(room))) {
        room = (unsigned long long)nnz;
        FIIM_TRY(entries.reserve(entry_bytes(room)));
    }
    int *key = entries.take<int>(nnz), *row = entries.take<int>(nnz);
    Stager &stager = thread_stager(dev);
    FIIM_TRY(stager.copy(dAi, Ai, sizeof(int) * (n + 1), st));
    if (nnz > 0) {
        FIIM_TRY(stager.copy(dAj, Aj, sizeof(int) * nnz, st));
        FIIM_TRY(stager.copy(dAv, Av, sizeof(double) * nnz, st));
    }
    // A^T: rows ascend within each column's list.
    FIIM_CUDA(cudaMemsetAsync(cnt, 0, sizeof(int) * n, st));
    k_count<<<grid_for(k_count, kThreads, nnz), kThreads, 0, st>>>(nnz, dAj, cnt);
    FIIM_TRY(scan(n, cnt, sums, dTi, next, st));
    k_to_columns<<<grid_for(k_to_columns, kThreads, n), kThreads, 0, st>>>(n, dAi, dAj, next, key, row);
    FIIM_TRY(rank_lists(n, Lists{dTi, key, row, nullptr, dAv, dTj, dTv}, nnz, longs, nlongs, st));
    const CsrD A{dAi, dAj, dAv}, At{dTi, dTj, dTv};
    // Every row's entries and D^{-1}, in one pass: they go to the next free places, which are then
    // put in order.
    Out o{gcnt, hcnt, dD, at, nullptr, nullptr, used, 0, ovf, novf};
    for (;;) {
        entries.used = 0;
        o.ej = entries.take<int>(room);
        o.ev = entries.take<double>(room);
        o.room = room;
        const unsigned long long two = 2;   // row 0: the unit entries of g and h
        const int one = 1, zero[2] = {0, 0};
        const double unit[2] = {1.0, 1.0}, d0 = 1.0 / Av[0];   // D = 1 / (first stored entry of row 0)
        const long at0 = 0;
        FIIM_CUDA(cudaMemcpyAsync(used, &two, sizeof two, cudaMemcpyHostToDevice, st));
        FIIM_CUDA(cudaMemcpyAsync(gcnt, &one, sizeof one, cudaMemcpyHostToDevice, st));
        FIIM_CUDA(cudaMemcpyAsync(hcnt, &one, sizeof one, cudaMemcpyHostToDevice, st));
        FIIM_CUDA(cudaMemcpyAsync(at, &at0, sizeof at0, cudaMemcpyHostToDevice, st));
        FIIM_CUDA(cudaMemcpyAsync(o.ej, zero, sizeof zero, cudaMemcpyHostToDevice, st));
        FIIM_CUDA(cudaMemcpyAsync(o.ev, unit, sizeof unit, cudaMemcpyHostToDevice, st));
        FIIM_CUDA(cudaMemcpyAsync(dD, &d0, sizeof d0, cudaMemcpyHostToDevice, st));
        const int *rows = nullptr;
        int nrows = n - 1;
        for (int c = 0; c < 3 && n > 1; ++c) {   // rows that outgrow a CAP run again at the next one
            FIIM_CUDA(cudaMemsetAsync(novf, 0, sizeof(int), st));
            FIIM_TRY(run_cap(kCaps[c], n, rows, nrows, A, At, P, o, st));
            int no = 0;
            FIIM_CUDA(cudaMemcpyAsync(&no, novf, sizeof(int), cudaMemcpyDeviceToHost, st));
            FIIM_CUDA(cudaStreamSynchronize(st));
            if (no == 0) break;
            std::vector<int> left(no);   // on st, as the kernel that reads rows2: no stream orders another's copies
            FIIM_CUDA(cudaMemcpyAsync(left.data(), ovf, sizeof(int) * no, cudaMemcpyDeviceToHost, st));
            FIIM_CUDA(cudaStreamSynchronize(st));
            std::sort(left.begin(), left.end());
            if (c == 2)
                return set_error(FIIM_EARG, "row %d's pattern outgrows %d members; use the host construction "
                                            "(fiim_pdfiim_build) or a warpsize cap", left[0], kCaps[2]);
            FIIM_CUDA(cudaMemcpyAsync(rows2, left.data(), sizeof(int) * no, cudaMemcpyHostToDevice, st));
            FIIM_CUDA(cudaStreamSynchronize(st));   // before the host rows go
            rows = rows2;
            nrows = no;
        }
        FIIM_CUDA(cudaMemcpyAsync(&asked, used, sizeof asked, cudaMemcpyDeviceToHost, st));
        FIIM_CUDA(cudaStreamSynchronize(st));
        if (asked <= room) break;
        room = asked;
        FIIM_TRY(entries.reserve(entry_bytes(room)));
    }
    // H: the tasks' h lists one after another; G: the tasks' g lists, columns, turned into rows.
    if (asked > 2ULL * 0x7fffffffULL) return set_error(FIIM_EARG, "factors too large for int32 CSR");
    FIIM_TRY(scan(n, hcnt, sums, dTi, nullptr, st));   // A^T is done with
    FIIM_CUDA(cudaMemcpyAsync(&out.nH, sums + nb, sizeof(long), cudaMemcpyDeviceToHost, st));
    FIIM_CUDA(cudaStreamSynchronize(st));
    out.nG = (long)asked - out.nH;
    if (out.nG > 0x7fffffffL || out.nH > 0x7fffffffL) return set_error(FIIM_EARG, "factors too large for int32 CSR");
    Slab lists;
    if (!out.mem.fits(out.carve(nullptr, n)) || !lists.fits(Slab::need<int>(out.nG) + Slab::need<double>(out.nG))) {
        out.mem.release();
        return out.order_on_host(o, n, st);   // A, A^T and the entries are all the device has to hold
    }
    const size_t held = out.carve(out.mem.p, n);
    FIIM_CUDA(cudaMemcpyAsync(out.Hi, dTi, sizeof(int) * (n + 1), cudaMemcpyDeviceToDevice, st));
    k_h_rows<<<grid_for(k_h_rows, kWarps, n), kThreads, 0, st>>>(n, o, out.Hi, out.Hj, out.Hv);
    FIIM_CUDA(cudaMemsetAsync(cnt, 0, sizeof(int) * n, st));
    k_count_g<<<grid_for(k_count_g, kThreads, n), kThreads, 0, st>>>(n, o, cnt);
    FIIM_TRY(scan(n, cnt, sums, out.Gi, next, st));
    int *gkey = lists.take<int>(out.nG);
    double *gval = lists.take<double>(out.nG);
    k_g_to_rows<<<grid_for(k_g_to_rows, kThreads, n), kThreads, 0, st>>>(n, o, next, gkey, gval);
    FIIM_TRY(rank_lists(n, Lists{out.Gi, gkey, gkey, gval, nullptr, out.Gj, out.Gv}, n, longs, nlongs, st));
    FIIM_CUDA(cudaMemcpyAsync(out.D, dD, sizeof(double) * n, cudaMemcpyDeviceToDevice, st));
    FIIM_CUDA(cudaStreamSynchronize(st));
    out.n = n;
    out.device = dev;
    return held > kHeldMost ? out.to_host(dev) : FIIM_OK;
}

int BuiltGpu::to_host(int dev) {
    host.reset(new (std::nothrow) char[mem.size]);
    if (!host) return set_error(FIIM_ENOMEM, "host allocation of %zu bytes for the factors failed", mem.size);
    FIIM_TRY(thread_stager(dev).copy_out(host.get(), mem.p, mem.size));
    carve(host.get(), n);
    mem.release();
    device = -1;
    return FIIM_OK;
}

// The tasks' lists put in order in host memory, by counting sorts; o's arrays are on the device, st is done.
int BuiltGpu::order_on_host(const Out &o, int rows, cudaStream_t st) {
    const size_t count = (size_t)(nG + nH);
    std::unique_ptr<int[]> cg(new (std::nothrow) int[rows]), ch(new (std::nothrow) int[rows]), ej(new (std::nothrow) int[count]);
    std::unique_ptr<long[]> at(new (std::nothrow) long[rows]);
    std::unique_ptr<double[]> ev(new (std::nothrow) double[count]);
    const size_t bytes = carve(nullptr, rows);
    host.reset(new (std::nothrow) char[bytes]);
    if (!cg || !ch || !ej || !at || !ev || !host)
        return set_error(FIIM_ENOMEM, "host allocation of %zu bytes for the factors failed", bytes + 12 * count);
    carve(host.get(), rows);
    FIIM_CUDA(cudaMemcpyAsync(cg.get(), o.gcnt, sizeof(int) * rows, cudaMemcpyDeviceToHost, st));
    FIIM_CUDA(cudaMemcpyAsync(ch.get(), o.hcnt, sizeof(int) * rows, cudaMemcpyDeviceToHost, st));
    FIIM_CUDA(cudaMemcpyAsync(at.get(), o.at, sizeof(long) * rows, cudaMemcpyDeviceToHost, st));
    FIIM_CUDA(cudaMemcpyAsync(ej.get(), o.ej, sizeof(int) * count, cudaMemcpyDeviceToHost, st));
    FIIM_CUDA(cudaMemcpyAsync(ev.get(), o.ev, sizeof(double) * count, cudaMemcpyDeviceToHost, st));
    FIIM_CUDA(cudaMemcpyAsync(D, o.D, sizeof(double) * rows, cudaMemcpyDeviceToHost, st));
    FIIM_CUDA(cudaStreamSynchronize(st));
    std::fill(Gi, Gi + rows + 1, 0);
    Hi[0] = 0;
    for (int i = 0; i < rows; ++i) {
        for (long q = at[i]; q < at[i] + cg[i]; ++q) Gi[ej[q] + 1]++;
        Hi[i + 1] = Hi[i] + ch[i];
        std::copy_n(ej.get() + at[i] + cg[i], ch[i], Hj + Hi[i]);
        std::copy_n(ev.get() + at[i] + cg[i], ch[i], Hv + Hi[i]);
    }
    for (int i = 0; i < rows; ++i) Gi[i + 1] += Gi[i];
    for (int i = 0; i < rows; ++i)   // Gi[r]: row r's next place, until all are shifted back by one row
        for (long q = at[i]; q < at[i] + cg[i]; ++q) {
            const int place = Gi[ej[q]]++;
            Gj[place] = i;
            Gv[place] = ev[q];
        }
    for (int r = rows; r > 0; --r) Gi[r] = Gi[r - 1];
    Gi[0] = 0;
    n = rows;
    device = -1;
    return FIIM_OK;
}

// The second call: straight into the caller's arrays.
int copy_out(const BuiltGpu &b, double *Gv, int *Gj, int *Gi, double *D, double *Hv, int *Hj, int *Hi) {
    const size_t n = (size_t)b.n, g = (size_t)b.nG, h = (size_t)b.nH;
    const struct {
        void *to;
        const void *from;
        size_t bytes;
    } parts[] = {{Gi, b.Gi, sizeof(int) * (n + 1)}, {Gj, b.Gj, sizeof(int) * g}, {Gv, b.Gv, sizeof(double) * g},
                 {Hi, b.Hi, sizeof(int) * (n + 1)}, {Hj, b.Hj, sizeof(int) * h}, {Hv, b.Hv, sizeof(double) * h},
                 {D, b.D, sizeof(double) * n}};
    if (b.device < 0) {
        for (const auto &p : parts) copy_parallel(p.to, p.from, p.bytes);
        return FIIM_OK;
    }
    int was = -1, rc = FIIM_OK;
    FIIM_CUDA(cudaGetDevice(&was));
    FIIM_CUDA(cudaSetDevice(b.device));
    Stager &stager = thread_stager(b.device);
    for (const auto &p : parts)
        if (rc == FIIM_OK) rc = stager.copy_out(p.to, p.from, p.bytes);
    cudaSetDevice(was);
    return rc;
}

}  // namespace pg
}  // namespace fiim

extern "C" int fiim_pdfiim_build_gpu(int n, const int *Ai, const int *Aj, const double *Av, int prefill, int lfill,
                                     int postfill, double ftol, int warpsize, char filttype, char patt, int *nnzG,
                                     int *nnzH, double *Gv, int *Gj, int *Gi, double *D, double *Hv, int *Hj,
                                     int *Hi) {
    using fiim::pg::g_built_gpu;
    if (!Gv) {
        if (n <= 0 || !Ai || !Aj || !Av || !nnzG || !nnzH) return fiim::set_error(FIIM_EARG, "null argument or n <= 0");
        if (patt != 'B') return fiim::set_error(FIIM_EARG, "only the two-sided pattern 'B' is served");
        if (warpsize == 0 || warpsize < -1) return fiim::set_error(FIIM_EARG, "warpsize is -1 or positive");
        const fiim::pg::Params P{prefill, lfill, postfill, warpsize, ftol, filttype};
        const int rc = fiim::pg::build_gpu(n, Ai, Aj, Av, P, g_built_gpu);
        if (rc != FIIM_OK) {
            g_built_gpu.clear();
            return rc;
        }
        *nnzG = (int)g_built_gpu.nG;
        *nnzH = (int)g_built_gpu.nH;
        return FIIM_OK;
    }
    if (g_built_gpu.n <= 0 || g_built_gpu.n != n || !Gj || !Gi || !D || !Hv || !Hj || !Hi)
        return fiim::set_error(FIIM_EARG, "call first with Gv == NULL, then with every output");
    const int rc = fiim::pg::copy_out(g_built_gpu, Gv, Gj, Gi, D, Hv, Hj, Hi);
    g_built_gpu.clear();
    return rc;
}
