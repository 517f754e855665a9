// Set-up kernels of the sliced forms of a CSR matrix (fiim_kernels.cuh: k_spmv_dia): which
// diagonals each slice of rows shares, the slice records and values, and which slices are the
// same as another one. Every kernel walks the matrix the same way: one warp per slice, R rows a
// lane, all rows advancing together by ascending diagonal d = col - row (a warp minimum over
// the rows' next diagonals), so a slice's records come out sorted without sorting. A slice's
// columns and values are contiguous in the CSR arrays, so the lanes' walks share cache lines.
// A walk reads the matrix once: at 128^3, 60-90 us for H (22.7 M entries), where the host
// analysis it replaces took 0.2-0.3 s with its copy of the columns.
#pragma once

#include <climits>

#include "fiim_kernels.cuh"

namespace fiim {
namespace sl {

// What a walk of a matrix found (device, read back once).
struct Stats {
    unsigned long long ndiag;        // diagonals over all slices
    unsigned long long uniq_ndiag;   // ... over the slices that are the first of their kind
    int max_m;                       // most diagonals of a slice
    int refused;                     // a row not sorted by column, or a slice past `most`
    int pad;                         // an entry holds the padding pattern
    int uniq;                        // different slices
    int bad;                         // verify / place: the copy does not hold these values
};

// Shared blocks serve slices of which at most half differ: otherwise the class numbers cost a load
// in front of every block and most blocks are read once. k_spmv_cls counts the blocks' values, whole
// quads of diagonals, in ints.
__host__ __device__ inline bool sharing(const Stats &st, int R, int nsl) {
    return 2L * st.uniq <= nsl && 32L * R * (long)st.uniq_ndiag < (1L << 31);
}

struct Args {
    int n, nsl;
    int most;                        // scan: diagonals of one slice at most
    const int *__restrict__ rp;
    const int *__restrict__ ci;
    const void *vals;                // nnz values of B's width
    const int2 *__restrict__ pos;    // first row and rows of each slice (null: one segment)
    Stats *stats;
    int *m;                          // scan: diagonals per slice
    unsigned long long *hash;        // scan: hash of a slice's record and values
    unsigned long long *keys;        // count: table of the hashes met (k_insert), 0 empty
    unsigned mask;
    // the copy (write, verify, place)
    int *rec;
    int rs;
    void *dv;
    const int *cls;                  // class of each slice (null: its own index)
    const int *k0;                   // first diagonal of each class's block (write)
    const int *rep;                  // the class's first slice (write; null: every slice writes)
    const int *list;                 // place: the slices to walk, nsl of them (null: all)
};

enum { kScan, kCount, kWrite, kVerify, kPlace };   // count: a scan that leaves only the different slices' number

template <typename B>
__device__ __forceinline__ B pad_bits() {
    if constexpr (sizeof(B) == 8) return (B)kDiaPad;
    else if constexpr (sizeof(B) == 4) return (B)kDiaPad32;
    else return (B)kDiaPad16;
}

// The place of hash h in an open-addressing table (0 empty), claimed if nobody did: (claimed, place). The table
// holds more places than hashes, so an empty or equal one exists.
struct Claim {
    bool first;
    unsigned at;
};
__device__ __forceinline__ Claim claim(unsigned long long *keys, unsigned mask, unsigned long long h) {
    unsigned at = (unsigned)h & mask;
    for (;;) {
        const unsigned long long was = atomicCAS(keys + at, 0ULL, h);
        if (was == 0ULL || was == h) return Claim{was == 0ULL, at};
        at = (at + 1) & mask;
    }
}
__device__ __forceinline__ int quads(int m) { return (m + kDiaQuad - 1) & -kDiaQuad; }   // shared blocks hold whole quads

// LANES: lane l owns the rows first + l + 32 j (shared blocks), else first + R l + j.
template <int R, typename B, int MODE, bool LANES>
static __global__ void __launch_bounds__(kThreads) k_walk(Args a) {
    constexpr int SH = 32 * R;
    constexpr bool SCAN = MODE == kScan || MODE == kCount;
    const unsigned full = 0xffffffffu;
    const int lane = (int)threadIdx.x & 31;
    auto slot_of = [&](int j) { return LANES ? lane + 32 * j : R * lane + j; };   // row - first
    const B *vals = static_cast<const B *>(a.vals);
    B *dv = static_cast<B *>(a.dv);
    unsigned long long sum_m = 0;
    int max_m = 0;
    for (int at = (int)blockIdx.x * kWarps + ((int)threadIdx.x >> 5); at < a.nsl; at += (int)gridDim.x * kWarps) {
        const int s = MODE == kPlace && a.list ? __ldg(a.list + at) : at;
        // refused already: random matrices end at once (one lane's read, so the warp agrees)
        if (SCAN && __shfl_sync(full, *(volatile int *)&a.stats->refused, 0)) break;
        const int c = a.cls ? __ldg(a.cls + s) : s;
        if (MODE == kWrite && a.rep && __ldg(a.rep + s) != s) continue;
        int first = s * SH, rows = min(SH, a.n - s * SH);
        if (a.pos) {
            const int2 q = __ldg(a.pos + s);
            first = q.x;
            rows = q.y;
        }
        int *rec = SCAN ? nullptr : a.rec + (long)c * a.rs;
        int k0 = 0, m_have = 0;
        if (MODE == kWrite) k0 = __ldg(a.k0 + s);
        if (MODE == kVerify || MODE == kPlace) {
            k0 = rec[0];
            m_have = rec[1] & kDiaCountMask;
        }
        int e[R], end[R], cur[R];
#pragma unroll
        for (int j = 0; j < R; ++j) {
            const int row = first + slot_of(j);
            e[j] = end[j] = 0;
            if (slot_of(j) < rows) {
                e[j] = __ldg(a.rp + row);
                end[j] = __ldg(a.rp + row + 1);
            }
            cur[j] = e[j] < end[j] ? __ldg(a.ci + e[j]) - row : INT_MAX;
        }
        unsigned long long h = 0;
        int k = 0, dlo = 0, dhi = 0;
        bool refused = false, pad = false, bad = false;
        for (;;) {
            int d = cur[0];
#pragma unroll
            for (int j = 1; j < R; ++j) d = min(d, cur[j]);
            d = __reduce_min_sync(full, d);
            if (d == INT_MAX) break;
            if (k == (SCAN ? a.most : a.rs - kDiaRecHead) || (MODE >= kVerify && k == m_have)) {
                if (SCAN) refused = true;
                else bad = true;
                break;
            }
            if (k == 0) dlo = d;
            dhi = d;
            if (MODE == kWrite && lane == 0) rec[kDiaRecHead + k] = d;
            if (MODE >= kVerify && rec[kDiaRecHead + k] != d) {   // uniform in the warp
                bad = true;
                break;
            }
            if (SCAN) h = mix64(h ^ (unsigned)d);
#pragma unroll
            for (int j = 0; j < R; ++j) {
                B o = pad_bits<B>();
                if (cur[j] == d) {
                    o = vals[e[j]];
                    if (dia_is_pad(o, pad_bits<B>())) pad = true;
                    const int row = first + slot_of(j);
                    const int nd = ++e[j] < end[j] ? __ldg(a.ci + e[j]) - row : INT_MAX;
                    if (nd <= d) refused = true;
                    cur[j] = nd;
                }
                const long slot = (long)(k0 + k) * SH + R * lane + j;
                if (SCAN) h = mix64(h ^ (unsigned long long)o);
                if (MODE == kWrite || MODE == kPlace) dv[slot] = o;
                if (MODE == kVerify && dv[slot] != o) bad = true;
            }
            ++k;
        }
        if (MODE == kWrite && a.cls)   // shared blocks hold whole quads
            for (int kk = k; kk < ((k + kDiaQuad - 1) & -kDiaQuad); ++kk)
#pragma unroll
                for (int j = 0; j < R; ++j) dv[(long)(k0 + kk) * SH + R * lane + j] = pad_bits<B>();
        const int clamp = rows < SH || (long)first + dlo < 0 || (long)first + SH - 1 + dhi > a.n - 1 ? kDiaClamp : 0;
        if (MODE >= kVerify && (k != m_have || rec[1] != (k | clamp))) bad = true;
        refused = __any_sync(full, refused);
        pad = __any_sync(full, pad);
        bad = __any_sync(full, bad);
        if (SCAN) {
            h = mix64(h ^ ((unsigned long long)(lane + 1) << 32));
            for (int o = 16; o > 0; o >>= 1) h += __shfl_xor_sync(full, h, o);
            h = mix64(h ^ (unsigned)(k | clamp));
        }
        if (lane == 0) {
            if (SCAN) {
                if (h == 0ULL) h = 1ULL;   // 0 marks an empty slot of the table
                if (refused) atomicExch(&a.stats->refused, 1);
            }
            if (MODE == kScan) {
                a.m[s] = k;
                a.hash[s] = h;
                sum_m += (unsigned)k;
                max_m = max(max_m, k);
            }
            if (MODE == kCount && claim(a.keys, a.mask, h).first) {
                ++max_m;
                sum_m += (unsigned)quads(k);
            }
            if (MODE == kWrite) {
                rec[0] = k0;
                rec[1] = k | clamp;
                rec[2] = (k + kDiaQuad - 1) / kDiaQuad;
            }
            if (pad) atomicExch(&a.stats->pad, 1);
            if (MODE >= kVerify && (bad || refused || pad)) atomicExch(&a.stats->bad, 1);
        }
    }
    if (MODE == kScan && lane == 0 && max_m) {
        atomicAdd(&a.stats->ndiag, sum_m);
        atomicMax(&a.stats->max_m, max_m);
    }
    if (MODE == kCount && lane == 0 && max_m) {   // the slices this warp met first
        atomicAdd(&a.stats->uniq, max_m);
        atomicAdd(&a.stats->uniq_ndiag, sum_m);
    }
}

// The packed slices (one row a lane; fiim_kernels.cuh, k_spmv_pack): first, the records from the
// scan's counts at the offsets k0, then the values. PLACE writes the values of a matrix whose
// records are there already, and sets *bad when its columns are not those the records describe.
template <bool PLACE>
static __global__ void __launch_bounds__(kThreads)
k_pack(Args a, int4 *hdr, int2 *rec) {
    const unsigned full = 0xffffffffu;
    const int lane = (int)threadIdx.x & 31;
    const double *vals = static_cast<const double *>(a.vals);
    double *dv = static_cast<double *>(a.dv);
    for (int s = (int)blockIdx.x * kWarps + ((int)threadIdx.x >> 5); s < a.nsl; s += (int)gridDim.x * kWarps) {
        const int row = s * 32 + lane;
        const int k0 = PLACE ? hdr[s].x : a.k0[s], m = PLACE ? hdr[s].y : a.m[s];
        const int v0 = __ldg(a.rp + s * 32);
        int e = 0, end = 0;
        if (row < a.n) {
            e = __ldg(a.rp + row);
            end = __ldg(a.rp + row + 1);
        }
        int cur = e < end ? __ldg(a.ci + e) - row : INT_MAX, at = v0;
        bool bad = PLACE && hdr[s].z != v0;
        int dlo = 0, dhi = 0;
        for (int k = 0;; ++k) {
            const int d = __reduce_min_sync(full, cur);
            if (d == INT_MAX) {
                if (k != m) bad = true;
                break;
            }
            if (k == m) {
                bad = true;
                break;
            }
            if (k == 0) dlo = d;
            dhi = d;
            const unsigned mask = __ballot_sync(full, cur == d);
            if (!PLACE && lane == 0) rec[k0 + k] = make_int2(d, (int)mask);
            if (PLACE) {
                const int2 q = rec[k0 + k];
                if (q.x != d || q.y != (int)mask) {   // uniform in the warp
                    bad = true;
                    break;
                }
            }
            if (cur == d) {
                dv[at + __popc(mask & ((1u << lane) - 1u))] = vals[e];
                cur = ++e < end ? __ldg(a.ci + e) - row : INT_MAX;
                if (cur <= d) bad = true;   // not sorted: the next minimum would go back
            }
            at += __popc(mask);
        }
        // a chunk past the last record gathers at d = 0, so the slice's own rows count too
        const bool edge = s * 32 + min(dlo, 0) < 0 || s * 32 + 31 + max(dhi, 0) > a.n - 1;
        if (!PLACE && lane == 0) hdr[s] = make_int4(k0, m, v0, (at - v0) << 1 | (int)edge);
        if (__any_sync(full, bad) && lane == 0) atomicExch(&a.stats->bad, 1);
    }
}

// Open-addressing table of slice hashes: each distinct hash keeps the smallest slice index that
// holds it, so the classes do not depend on the order the threads arrive in.
static __global__ void __launch_bounds__(kThreads)
k_insert(int nsl, const unsigned long long *__restrict__ hash, unsigned long long *keys, int *first, unsigned mask,
         int *slot) {
    FIIM_FOR_ROWS(s, nsl) {
        const unsigned at = claim(keys, mask, hash[s]).at;
        atomicMin(first + at, (int)s);
        slot[s] = (int)at;
    }
}

// rep[s]: the first slice with s's hash; counts the distinct ones and their diagonals.
static __global__ void __launch_bounds__(kThreads)
k_reps(int nsl, const int *__restrict__ first, const int *__restrict__ slot, const int *__restrict__ m, int *rep,
       Stats *stats) {
    int c = 0;
    unsigned long long d = 0;
    FIIM_FOR_ROWS(s, nsl) {
        rep[s] = first[slot[s]];
        if (rep[s] == (int)s) {
            ++c;
            d += (unsigned)quads(m[s]);
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        c += __shfl_xor_sync(0xffffffffu, c, o);
        d += __shfl_xor_sync(0xffffffffu, d, o);
    }
    if ((threadIdx.x & 31) == 0 && c) {
        atomicAdd(&stats->uniq, c);
        atomicAdd(&stats->uniq_ndiag, d);
    }
}

// Whether a count of the slices in the values a copy with own blocks now holds (for R = 1, 2 where nsl[R - 1]
// is not 0) finds what would be shared: then the copy is not the form build_dia would choose for them.
static __global__ void k_recheck(int2 nsl, const Stats *__restrict__ count, Stats *copy) {
    for (int R = 1; R <= 2; ++R) {
        const Stats &st = count[R - 1];
        const int k = R == 1 ? nsl.x : nsl.y;
        if (k && !st.refused && !st.pad && sharing(st, R, k)) copy->bad = 1;
    }
}

// In slice order, over the slices that write (all, or with rep those that are their own
// representative): id[s] = how many came before, k0[s] = their diagonals. One CTA.
static __global__ void __launch_bounds__(1024)
k_offsets(int nsl, const int *__restrict__ m, const int *__restrict__ rep, int *__restrict__ id, int *__restrict__ k0) {
    __shared__ int sc[32], sd[32], tc, td;
    const int t = (int)threadIdx.x, lane = t & 31, w = t >> 5;
    int basec = 0, based = 0;
    for (int s0 = 0; s0 < nsl; s0 += 1024) {
        const int s = s0 + t;
        const int c = s < nsl && (!rep || rep[s] == s), d = c ? (rep ? quads(m[s]) : m[s]) : 0;
        int ic = c, dd = d;
        for (int o = 1; o < 32; o <<= 1) {
            const int uc = __shfl_up_sync(0xffffffffu, ic, o), ud = __shfl_up_sync(0xffffffffu, dd, o);
            if (lane >= o) {
                ic += uc;
                dd += ud;
            }
        }
        if (lane == 31) {
            sc[w] = ic;
            sd[w] = dd;
        }
        __syncthreads();
        if (w == 0) {
            int xc = sc[lane], xd = sd[lane];
            for (int o = 1; o < 32; o <<= 1) {
                const int uc = __shfl_up_sync(0xffffffffu, xc, o), ud = __shfl_up_sync(0xffffffffu, xd, o);
                if (lane >= o) {
                    xc += uc;
                    xd += ud;
                }
            }
            sc[lane] = xc;
            sd[lane] = xd;
            if (lane == 31) {
                tc = xc;
                td = xd;
            }
        }
        __syncthreads();
        if (s < nsl) {
            id[s] = basec + (w ? sc[w - 1] : 0) + ic - c;
            k0[s] = based + (w ? sd[w - 1] : 0) + dd - d;
        }
        basec += tc;
        based += td;
        __syncthreads();
    }
}

// The class of each slice, and each class's first slice.
static __global__ void __launch_bounds__(kThreads)
k_classes(int nsl, const int *__restrict__ rep, const int *__restrict__ id, int *__restrict__ cls, int *__restrict__ first) {
    FIIM_FOR_ROWS(s, nsl) {
        cls[s] = id[rep[s]];
        if (rep[s] == (int)s) first[id[s]] = (int)s;
    }
}

}  // namespace sl
}  // namespace fiim
