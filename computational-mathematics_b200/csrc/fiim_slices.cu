// Building and refreshing the sliced-diagonal copy of a matrix (fiim_kernels.cuh, k_spmv_dia)
// on the device. The copy holds one record and one block of values per DIFFERENT slice: a
// stencil with constant coefficients has a few dozen where the grid's lines are whole or simple
// fractions of slices (128^3 convection-diffusion: A 18, G 40, H 22 of 32,768 slices of 64 rows,
// 0.07 to 0.12 MB of blocks, which stay in L1), and hundreds where they are not (97^3: 403, 638 and
// 481 of 14,261, 1.7 to 2.7 MB, which come from L2). Its products then read the vectors and
// little else: an iteration at 96, 97, 100, 127 and 128 a side takes 89, 95, 91, 78 and 74 ps a row,
// against 131, 133, 133, 114 and 114 with a block a slice. Slices count as the same when their diagonals, their values bit
// for bit (padding included) and their clamp flag agree; equality is found by a 64-bit hash
// and then checked on every slice, so a hash collision costs the sharing, never a product.

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "fiim_b200.h"
#include "fiim_internal.h"
#include "fiim_kernels.cuh"
#include "fiim_slices.cuh"

namespace fiim {

bool dia_wanted() {
    // FIIM_SPMV=rows / staged / warp keep a CSR-stream form; FIIM_DIA=0 never builds the copy.
    const char *force = std::getenv("FIIM_SPMV"), *off_env = std::getenv("FIIM_DIA");
    return !((force && std::strcmp(force, "dia") != 0) || (off_env && std::strcmp(off_env, "0") == 0));
}

// FIIM_DIA_SHARE=0 stores every slice's own record and values.
static bool share_wanted() {
    const char *e = std::getenv("FIIM_DIA_SHARE");
    return !(e && e[0] == '0' && e[1] == 0);
}

int dia_rows_per_lane(int vbytes) {
    if (vbytes == 8) {
        const char *e = std::getenv("FIIM_DIA_R");
        return (e && (e[0] == '1' || e[0] == '2') && e[1] == 0) ? e[0] - '0' : 0;   // 0: by the matrix
    }
    return vbytes == 4 ? 2 : 4;
}

void release_dia(DevCsr &M) {
    if (M.dia_mem) cudaFree(M.dia_mem);
    if (M.dscan) cudaFree(M.dscan);
    M.dscan = nullptr;
    M.dia_fit = 0;
    M.dia_pad = false;
    M.dia_mem = nullptr;
    M.dia_bytes = 0;
    M.drec = M.dcls = M.dfirst = nullptr;
    M.dpos = nullptr;
    M.dstat = nullptr;
    M.dvals = nullptr;
    M.dvbytes = 0;
    M.dsh = 0;
    M.dseg = false;
    M.dia = 0;
    M.nsl = M.dncls = 0;
    M.drs = 0;
    M.ndiag = 0;
    M.pack = 0;
    M.khdr = nullptr;
    M.krec = nullptr;
}

static int col_hash(DevCsr &M, cudaStream_t s, unsigned long long *h) {
    *h = 0;
    if (M.nnz <= 0 || !M.dhash) return FIIM_OK;
    FIIM_CUDA(cudaMemsetAsync(M.dhash, 0, sizeof(unsigned long long), s));
    k_col_hash<<<grid_for(k_col_hash, kThreads, M.nnz), kThreads, 0, s>>>(M.nnz, M.ci, M.dhash);
    FIIM_CUDA(cudaGetLastError());
    FIIM_CUDA(cudaMemcpyAsync(h, M.dhash, sizeof(unsigned long long), cudaMemcpyDeviceToHost, s));
    FIIM_CUDA(cudaStreamSynchronize(s));
    return FIIM_OK;
}

template <int R, typename B, int MODE, bool LANES>
static cudaError_t walk_as(const sl::Args &a, cudaStream_t s) {
    auto kern = sl::k_walk<R, B, MODE, LANES>;
    kern<<<grid_for(kern, kWarps, a.nsl), kThreads, 0, s>>>(a);
    return cudaGetLastError();
}

// The walk for R rows a lane of values of vbytes bytes (FP64: 1 or 2, FP32: 2, BF16: 4).
template <int MODE, bool LANES>
static cudaError_t walk(int R, int vbytes, const sl::Args &a, cudaStream_t s) {
    if (vbytes == 4) return walk_as<2, unsigned, MODE, LANES>(a, s);
    if (vbytes == 2) return walk_as<4, unsigned short, MODE, LANES>(a, s);
    return R == 2 ? walk_as<2, unsigned long long, MODE, LANES>(a, s)
                  : walk_as<1, unsigned long long, MODE, LANES>(a, s);
}

namespace {
// Device scratch of one build, freed on every way out.
struct Scratch {
    void *p = nullptr;
    size_t used = 0;
    ~Scratch() {
        if (p) cudaFree(p);
    }
    int reserve(size_t bytes) {
        if (cudaMalloc(&p, bytes) == cudaSuccess) return FIIM_OK;
        cudaGetLastError();
        p = nullptr;
        return FIIM_ENOMEM;
    }
    template <typename T>
    T *take(size_t count) {
        char *at = static_cast<char *>(p) + used;
        used += Arena::need(sizeof(T) * count);
        return reinterpret_cast<T *>(at);
    }
};
}  // namespace

// The walk's arguments for the copy M holds.
static sl::Args copy_args(const DevCsr &M, const void *vals) {
    sl::Args a{};
    a.n = (int)M.n;
    a.nsl = M.nsl;
    a.rp = M.rp;
    a.ci = M.ci;
    a.vals = vals;
    a.pos = M.dpos;
    a.stats = reinterpret_cast<sl::Stats *>(M.dstat);
    a.rec = M.drec;
    a.rs = M.drs;
    a.dv = M.dvals;
    a.cls = M.dcls;
    return a;
}

static cudaError_t pack(bool place, const sl::Args &a, int4 *hdr, int2 *rec, cudaStream_t s) {
    auto go = [&](auto kern) {
        kern<<<grid_for(kern, kWarps, a.nsl), kThreads, 0, s>>>(a, hdr, rec);
        return cudaGetLastError();
    };
    return place ? go(sl::k_pack<true>) : go(sl::k_pack<false>);
}

// The packed slices of M, where they are worth it: fewer bytes than the CSR streams, and at least
// one slot in kPackFill of the slices' diagonals holds an entry (a product takes as many
// instructions for an empty slot as for an entry).
static int build_pack(DevCsr &M, cudaStream_t s, const void *vals, int nsl, const sl::Stats &st, int *m, int *id,
                      int *k0) {
    constexpr double kPackFill = 3.0;
    const double bytes = (double)M.nnz * 8 + 8.0 * (double)st.ndiag + 16.0 * nsl;
    const double csr = (double)M.nnz * (8 + (M.narrow ? 2 : 4)) + 4.0 * (M.n + 1);
    if (st.refused || !(bytes < csr) || 32.0 * (double)st.ndiag > kPackFill * (double)M.nnz) return FIIM_OK;
    const size_t b_hdr = Arena::need(sizeof(int4) * nsl), b_rec = Arena::need(sizeof(int2) * st.ndiag),
                 b_st = Arena::need(sizeof(sl::Stats)),
                 b_v = Arena::need(8UL * (M.nnz + 32));   // a lane past the last value reads one further
    char *mem = nullptr;
    if (cudaMalloc(&mem, b_hdr + b_rec + b_st + b_v) != cudaSuccess) {
        cudaGetLastError();
        return FIIM_OK;   // no room for the copy: the CSR streams serve
    }
    M.dia_mem = mem;
    M.dia_bytes = b_hdr + b_rec + b_st + b_v;
    M.khdr = reinterpret_cast<int4 *>(mem);
    M.krec = reinterpret_cast<int2 *>(mem + b_hdr);
    M.dstat = mem + b_hdr + b_rec;
    M.dvals = mem + b_hdr + b_rec + b_st;
    M.dvbytes = 8;
    M.dsh = 32;
    M.nsl = nsl;
    M.ndiag = (long)st.ndiag;
    FIIM_CUDA(cudaMemsetAsync(M.dstat, 0, sizeof(sl::Stats), s));
    sl::k_offsets<<<1, 1024, 0, s>>>(nsl, m, nullptr, id, k0);
    FIIM_CUDA(cudaGetLastError());
    sl::Args a = copy_args(M, vals);
    a.m = m;
    a.k0 = k0;
    FIIM_CUDA(pack(false, a, M.khdr, M.krec, s));
    int bad = 0;
    FIIM_CUDA(cudaMemcpyAsync(&bad, &a.stats->bad, sizeof(int), cudaMemcpyDeviceToHost, s));
    FIIM_CUDA(cudaStreamSynchronize(s));   // before the scratch goes
    if (bad) release_dia(M);
    else M.pack = 1;
    return FIIM_OK;
}

int build_dia(DevCsr &M, cudaStream_t s, int vbytes, const void *vals, const std::vector<int> *segments) {
    release_dia(M);
    M.dia_tried = false;
    M.hseg_sl.clear();
    if (!dia_wanted()) return FIIM_OK;
    const int n = (int)M.n;
    const long nnz = M.nnz;
    if (n <= 0 || nnz <= 0 || (long)M.hrp.size() != (long)n + 1) return FIIM_OK;
    const std::vector<int> whole = {0, n};
    const std::vector<int> &seg = segments ? *segments : whole;
    if (seg.size() < 2 || seg.front() != 0 || seg.back() != n) return set_error(FIIM_EARG, "segments must cover the rows");
    FIIM_TRY(col_hash(M, s, &M.dia_cols));
    M.dia_tried = true;
    const bool segmented = seg.size() > 2;
    // Slices of up to 32 R rows, never straddling a segment: first row, rows (only kept for
    // several segments), and each segment's first slice.
    std::vector<int2> pos;
    std::vector<int> seg_sl;
    auto slices = [&](int R) -> int {
        const int sh = 32 * R;
        if (!segmented) {
            seg_sl = {0, (n + sh - 1) / sh};
            return seg_sl[1];
        }
        pos.clear();
        seg_sl.assign(1, 0);
        for (size_t q = 0; q + 1 < seg.size(); ++q) {
            for (int r = seg[q]; r < seg[q + 1]; r += sh) pos.push_back(make_int2(r, std::min(sh, seg[q + 1] - r)));
            seg_sl.push_back((int)pos.size());
        }
        return (int)pos.size();
    };
    const long most = (n + 31) / 32 + (long)seg.size();   // slices at one row a lane, at most
    unsigned table = 64;
    while (table < 2 * (unsigned long)most) table <<= 1;
    Scratch tmp;
    if (tmp.reserve(Arena::need(sizeof(sl::Stats)) + 5 * Arena::need(sizeof(int) * most) + Arena::need(sizeof(int2) * most) +
                    Arena::need(8 * most) + Arena::need(12UL * table) + 256) != FIIM_OK)
        return FIIM_OK;   // no room: the CSR streams serve
    sl::Stats *d_st = tmp.take<sl::Stats>(1), st{};
    int *m = tmp.take<int>(most), *slot = tmp.take<int>(most), *rep = tmp.take<int>(most), *id = tmp.take<int>(most),
        *k0 = tmp.take<int>(most);
    int2 *d_pos = tmp.take<int2>(most);
    unsigned long long *hash = tmp.take<unsigned long long>(most), *keys = tmp.take<unsigned long long>(table);
    int *firsts = tmp.take<int>(table);   // 12 bytes a table entry with its key
    const bool share_on = share_wanted();
    // Diagonals, hashes and classes of the slices for R rows a lane; one read-back.
    auto scan = [&](int R, int nsl, int limit = kDiaMaxDiags) -> int {
        if (segmented) FIIM_CUDA(cudaMemcpyAsync(d_pos, pos.data(), sizeof(int2) * nsl, cudaMemcpyHostToDevice, s));
        FIIM_CUDA(cudaMemsetAsync(d_st, 0, sizeof(sl::Stats), s));
        FIIM_CUDA(cudaMemsetAsync(keys, 0, 8UL * table, s));
        FIIM_CUDA(cudaMemsetAsync(firsts, 0x7f, 4UL * table, s));
        sl::Args a{};
        a.n = n;
        a.nsl = nsl;
        a.most = limit;
        a.rp = M.rp;
        a.ci = M.ci;
        a.vals = vals;
        a.pos = segmented ? d_pos : nullptr;
        a.stats = d_st;
        a.m = m;
        a.hash = hash;
        FIIM_CUDA((walk<sl::kScan, true>(R, vbytes, a, s)));
        if (share_on) {
            const int g = grid_for(sl::k_insert, kThreads, nsl);
            sl::k_insert<<<g, kThreads, 0, s>>>(nsl, hash, keys, firsts, table - 1, slot);
            FIIM_CUDA(cudaGetLastError());
            sl::k_reps<<<g, kThreads, 0, s>>>(nsl, firsts, slot, m, rep, d_st);
            FIIM_CUDA(cudaGetLastError());
        }
        FIIM_CUDA(cudaMemcpyAsync(&st, d_st, sizeof st, cudaMemcpyDeviceToHost, s));
        FIIM_CUDA(cudaStreamSynchronize(s));
        return FIIM_OK;
    };
    // Kept only when its slices, each with its own values, would move fewer bytes than the CSR
    // streams they replace.
    auto record_ints = [&] { return st.max_m <= 16 - kDiaRecHead ? 16 : 32; };
    auto smaller = [&](int R, int nsl) {
        const double dia = (double)vbytes * 32 * R * (double)st.ndiag + 4.0 * record_ints() * nsl;
        const double csr = (double)nnz * (vbytes + (M.narrow ? 2 : 4)) + 4.0 * (n + 1);
        const bool fits = !st.refused && st.max_m <= kDiaMaxDiags && dia < csr && 32.0 * R * (double)st.ndiag < 2147483648.0;
        if (fits) M.dia_fit |= R;
        if (st.pad) M.dia_pad = true;
        return fits && !st.pad;
    };
    auto sharing = [&](int R, int nsl) { return share_on && sl::sharing(st, R, nsl); };
    // FP64 slices that share take two rows a lane (k_spmv_cls). The others take two when their
    // 32-row slices average more diagonals than one chunk of the kernel holds (H at 128^3: 11
    // diagonals, 32.9 against 41.6 us a product; A and G, 7 diagonals, were slower with two).
    int R = dia_rows_per_lane(vbytes), nsl = 0;
    const int asked = R;
    bool dia = true;
    if (R) {
        nsl = slices(R);
        FIIM_TRY(scan(R, nsl));
        dia = smaller(R, nsl);
    } else {
        R = 2;
        nsl = slices(R);
        FIIM_TRY(scan(R, nsl));
        const bool two = smaller(R, nsl);
        if (!two || !sharing(R, nsl)) {
            R = 1;
            nsl = slices(R);
            FIIM_TRY(scan(R, nsl, kPackMax));
            dia = smaller(R, nsl);
            if (dia && two && !sharing(R, nsl) && (long)st.ndiag > 8L * nsl) {
                R = 2;
                nsl = slices(R);
                FIIM_TRY(scan(R, nsl));
            }
        }
    }
    if (!dia) {
        const char *pe = std::getenv("FIIM_PACK");   // 0: the CSR streams instead of packed slices
        if (pe && pe[0] == '0' && pe[1] == 0) return FIIM_OK;
        // FP64 single systems only: with FP32 factors the CSR streams read 6 bytes an entry and the
        // packed product's instructions weigh more (mixed solve 12.4 against 11.8 ms at 880,000 rows).
        if (segmented || vbytes != 8) return FIIM_OK;
        if (R != 1 || asked == 1) {   // scanned for the copy's limit of diagonals
            nsl = slices(1);
            FIIM_TRY(scan(1, nsl, kPackMax));
        }
        return build_pack(M, s, vals, nsl, st, m, id, k0);
    }
    const int sh = 32 * R, rs = record_ints();
    for (bool share = sharing(R, nsl);; share = false) {
        const int ncls = share ? st.uniq : nsl;
        const long ndiag = share ? (long)st.uniq_ndiag : (long)st.ndiag;
        const size_t b_rec = Arena::need(sizeof(int) * (size_t)rs * ncls),
                     b_cls = share ? Arena::need(sizeof(int) * nsl) : 0, b_first = share ? Arena::need(sizeof(int) * ncls) : 0,
                     b_pos = segmented ? Arena::need(sizeof(int2) * nsl) : 0, b_st = Arena::need(sizeof(sl::Stats)),
                     b_v = Arena::need((size_t)vbytes * sh * ndiag), all = b_rec + b_cls + b_pos + b_st + b_v + b_first;
        char *mem = nullptr;
        if (cudaMalloc(&mem, all) != cudaSuccess) {
            cudaGetLastError();
            return FIIM_OK;   // no room for the copy: the CSR streams serve
        }
        M.dia_mem = mem;
        M.dia_bytes = all;
        M.drec = reinterpret_cast<int *>(mem);
        M.dcls = share ? reinterpret_cast<int *>(mem + b_rec) : nullptr;
        M.dpos = segmented ? reinterpret_cast<int2 *>(mem + b_rec + b_cls) : nullptr;
        M.dstat = mem + b_rec + b_cls + b_pos;
        M.dvals = mem + b_rec + b_cls + b_pos + b_st;
        M.dfirst = share ? reinterpret_cast<int *>(mem + b_rec + b_cls + b_pos + b_st + b_v) : nullptr;
        M.dvbytes = vbytes;
        M.dsh = sh;
        M.nsl = nsl;
        M.dncls = ncls;
        M.drs = rs;
        M.ndiag = ndiag;
        M.hseg_sl = seg_sl;
        M.dseg = segmented;
        FIIM_CUDA(cudaMemsetAsync(M.drec, 0, sizeof(int) * (size_t)rs * ncls, s));
        FIIM_CUDA(cudaMemsetAsync(M.dstat, 0, sizeof(sl::Stats), s));
        if (segmented) FIIM_CUDA(cudaMemcpyAsync(M.dpos, d_pos, sizeof(int2) * nsl, cudaMemcpyDeviceToDevice, s));
        sl::k_offsets<<<1, 1024, 0, s>>>(nsl, m, share ? rep : nullptr, id, k0);
        FIIM_CUDA(cudaGetLastError());
        if (share) {
            sl::k_classes<<<grid_for(sl::k_classes, kThreads, nsl), kThreads, 0, s>>>(nsl, rep, id, M.dcls, M.dfirst);
            FIIM_CUDA(cudaGetLastError());
        }
        sl::Args a = copy_args(M, vals);
        a.k0 = k0;
        a.rep = share ? rep : nullptr;
        FIIM_CUDA((share ? walk<sl::kWrite, true>(R, vbytes, a, s) : walk<sl::kWrite, false>(R, vbytes, a, s)));
        if (share) {
            FIIM_CUDA((walk<sl::kVerify, true>(R, vbytes, a, s)));
            FIIM_CUDA(cudaMemcpyAsync(&st.bad, &a.stats->bad, sizeof(int), cudaMemcpyDeviceToHost, s));
        }
        FIIM_CUDA(cudaStreamSynchronize(s));   // before the scratch goes
        if (!share || !st.bad) break;
        release_dia(M);   // two different slices hash alike: every slice keeps its own block
    }
    M.dia = 1;
    return FIIM_OK;
}

// Enqueues the new values `vals` of M's matrix into the copy, and the check that it then holds them;
// stats.bad tells afterwards whether it does and build_dia would choose this form for them. Shared
// blocks take the values of their first slices, and every slice is checked against its block (slices
// that were alike and are alike still share; laying the copy out again for new constant coefficients
// made a drop-in call at 110^3 with five iterations 13.8 ms, this way it takes 10.0). For slices with
// their own blocks whose columns would allow shared ones, the different slices are counted again, which
// reads the matrix once for each number of rows a lane that fits. ok = false: not enqueued, the form
// has to be chosen anew.
static int enqueue_refresh(DevCsr &M, const void *vals, cudaStream_t s, bool *ok) {
    // which numbers of rows a lane, sharing, would be chosen before what the copy is now
    const int better = M.dia_fit & (!M.dcls ? 3 : M.dsh == 32 ? 2 : 0);
    const bool recount = better && M.dvbytes == 8 && !M.dseg && share_wanted();
    const int nsl[2] = {(int)((M.n + 31) / 32), (int)((M.n + 63) / 64)};
    unsigned table = 64;
    while (table < 2U * (unsigned)nsl[0]) table <<= 1;
    const size_t b_st = Arena::need(2 * sizeof(sl::Stats)), b_keys = Arena::need(8UL * table);
    *ok = !M.dia_pad;
    if (recount && !M.dscan && cudaMalloc(&M.dscan, b_st + 2 * b_keys) != cudaSuccess) {
        cudaGetLastError();
        M.dscan = nullptr;
        *ok = false;
    }
    if (!*ok) return FIIM_OK;
    sl::Args a = copy_args(M, vals);
    FIIM_CUDA(cudaMemsetAsync(M.dstat, 0, sizeof(sl::Stats), s));
    if (M.pack) {
        FIIM_CUDA(pack(true, a, M.khdr, M.krec, s));
    } else if (M.dcls) {
        sl::Args first = a;
        first.nsl = M.dncls;
        first.list = M.dfirst;
        FIIM_CUDA((walk<sl::kPlace, true>(M.dsh / 32, M.dvbytes, first, s)));
        FIIM_CUDA((walk<sl::kVerify, true>(M.dsh / 32, M.dvbytes, a, s)));
    } else {
        FIIM_CUDA((walk<sl::kPlace, false>(M.dsh / 32, M.dvbytes, a, s)));
    }
    if (!recount) return FIIM_OK;
    FIIM_CUDA(cudaMemsetAsync(M.dscan, 0, b_st + 2 * b_keys, s));
    char *mem = static_cast<char *>(M.dscan);
    sl::Stats *count = reinterpret_cast<sl::Stats *>(mem);
    a.most = kDiaMaxDiags;
    a.mask = table - 1;
    a.cls = nullptr;
    for (int R = 1; R <= 2; ++R) {
        if (!(better & R)) continue;
        a.nsl = nsl[R - 1];
        a.stats = count + (R - 1);
        a.keys = reinterpret_cast<unsigned long long *>(mem + b_st + (R - 1) * b_keys);
        FIIM_CUDA((walk<sl::kCount, true>(R, 8, a, s)));
    }
    sl::k_recheck<<<1, 1, 0, s>>>(make_int2(better & 1 ? nsl[0] : 0, better & 2 ? nsl[1] : 0), count,
                                  reinterpret_cast<sl::Stats *>(M.dstat));
    FIIM_CUDA(cudaGetLastError());
    return FIIM_OK;
}

int refresh_dia(DevCsr &M, cudaStream_t s) {
    if (!dia_wanted()) return FIIM_OK;
    if (!M.dia && !M.pack) {   // not built for the previous columns: decide again only if they changed
        unsigned long long h = 0;
        FIIM_TRY(col_hash(M, s, &h));
        if (M.dia_tried && h == M.dia_cols && !M.dia_fit) return FIIM_OK;   // whatever the values
        return build_dia(M, s, 8, M.v);
    }
    bool ok = false;
    FIIM_TRY(enqueue_refresh(M, M.v, s, &ok));
    if (!ok) return build_dia(M, s, 8, M.v);
    sl::Stats st{};
    FIIM_CUDA(cudaMemcpyAsync(&st, M.dstat, sizeof st, cudaMemcpyDeviceToHost, s));
    FIIM_CUDA(cudaStreamSynchronize(s));
    if (!st.bad) return FIIM_OK;
    return build_dia(M, s, 8, M.v);
}

int refresh_dia_async(DevCsr &M, cudaStream_t copy_s, cudaStream_t aux, cudaEvent_t done, int *h_bad) {
    FIIM_CUDA(cudaEventRecord(done, copy_s));
    FIIM_CUDA(cudaStreamWaitEvent(aux, done, 0));
    bool ok = false;
    *h_bad = 1;
    FIIM_TRY(enqueue_refresh(M, M.v, aux, &ok));
    if (!ok) return FIIM_OK;
    FIIM_CUDA(cudaMemcpyAsync(h_bad, &reinterpret_cast<sl::Stats *>(M.dstat)->bad, sizeof(int), cudaMemcpyDeviceToHost, aux));
    return FIIM_OK;
}

}  // namespace fiim
