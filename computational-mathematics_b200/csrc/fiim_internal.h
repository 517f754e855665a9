// Internal declarations shared by the host-side translation units.
#pragma once

#include <cuda_runtime.h>
#include <cuda_bf16.h>

#include <cstdarg>
#include <cstdlib>
#include <algorithm>
#include <cstddef>
#include <map>
#include <mutex>
#include <vector>

#include "fiim_b200.h"

namespace fiim {

int set_error(int code, const char *fmt, ...);
const char *last_error();
int check_device(int *dev_out);
int num_sms();

#define FIIM_CUDA(call)                                                                   \
    do {                                                                                  \
        cudaError_t e_ = (call);                                                          \
        if (e_ != cudaSuccess) {                                                          \
            cudaGetLastError();                                                           \
            return ::fiim::set_error(FIIM_ECUDA, "%s: %s (%s:%d)", #call,                 \
                                     cudaGetErrorString(e_), __FILE__, __LINE__);         \
        }                                                                                 \
    } while (0)

#define FIIM_TRY(call)                      \
    do {                                    \
        int rc_ = (call);                   \
        if (rc_ != FIIM_OK) return rc_;     \
    } while (0)

// One device allocation carved into 256-byte aligned pieces.
struct Arena {
    void *base = nullptr;
    size_t cap = 0, used = 0;
    int reserve(size_t bytes);   // ensure capacity (reallocates only to grow); resets use
    void *take(size_t bytes);    // nullptr when exhausted
    void release();
    static size_t need(size_t bytes);
};

// Forms of the solver's SpMV. All give the same bits. The CSR-stream forms differ in how a
// row block's streams reach shared memory: through registers, pipelined by one block
// (kFormRows, fiim_kernels.cuh), by bulk copies into two buffers (kFormBulk, fiim_pipe.cuh),
// or per warp (kFormWarp); kFormDia and kFormPack read a sliced copy of the values instead.
constexpr int kFormRows = 0, kFormBulk = 1, kFormWarp = 2, kFormDia = 3, kFormPack = 4;

// A CSR matrix resident on the device. v holds FP64 values; v32 / v16 are optional
// FP32 / BF16 copies for the mixed-precision inner solve.
struct DevCsr {
    long n = 0, nnz = 0;
    int *rp = nullptr, *ci = nullptr;
    double *v = nullptr;
    float *v32 = nullptr;
    __nv_bfloat16 *v16 = nullptr;
    int tile = 2048;             // entries per row block of the CSR-stream SpMV
    int form = 0;                // CSR-stream SpMV form, one of the kForm* constants
    int *rb = nullptr;           // row-block first rows (device), nblk + 1 entries
    int *eb = nullptr;           // row-block first entries (device), nblk + 1 entries
    int *cb = nullptr;           // row-block base columns of the narrow column stream
    short *cd = nullptr;         // narrow column stream: column - block base (device)
    int *wide = nullptr;         // device flag written by the narrow-stream builder
    int narrow = 0;              // 1: the CSR-stream SpMV reads cd / cb instead of ci
    int nblk = 0;
    // Sliced-diagonal copy (kFormDia; fiim_kernels.cuh, k_spmv_dia), in its own allocation.
    int dia = 0;                 // 1: built and current
    int nsl = 0;                 // slices of dsh rows
    int dncls = 0;               // different slices: records and value blocks held
    int dsh = 0;                 // rows a slice: 32 R, R rows a lane (dia_rows_per_lane)
    int drs = 0;                 // ints per slice record (16 or 32): first diagonal, count, offsets
    long ndiag = 0;              // diagonals over the blocks held (dsh slots each)
    int *drec = nullptr;         // dncls records
    int *dcls = nullptr;         // the record of each slice (null: its own)
    int *dfirst = nullptr;       // the first slice of each record (with dcls)
    int2 *dpos = nullptr;        // first row and rows of each slice (several segments only)
    char *dstat = nullptr;       // device counters of the check (fiim_slices.cuh, Stats)
    void *dvals = nullptr;       // dsh * ndiag values of dvbytes bytes each (FP64, FP32 or BF16)
    int dvbytes = 0;
    void *dia_mem = nullptr;
    size_t dia_bytes = 0;        // size of that allocation
    // Packed slices (kFormPack; fiim_kernels.cuh, k_spmv_pack), in the same allocation with dvals:
    // nsl slices of 32 rows.
    int pack = 0;                // 1: built and current (then dia is 0)
    int4 *khdr = nullptr;        // per slice: first record, records, first value
    int2 *krec = nullptr;        // offset and row mask of each slice's diagonals (ndiag of them)
    bool dia_tried = false;      // the copy was considered for the columns hashed in dia_cols
    int dia_fit = 0;             // R set: for these columns, R rows a lane move fewer bytes than the CSR streams
    bool dia_pad = false;        // refused for a value that holds the padding pattern
    void *dscan = nullptr;       // scratch of the class count that a refresh repeats (its own allocation)
    unsigned long long dia_cols = 0;
    unsigned long long *dhash = nullptr;   // device scratch of the column hash (in the arena)
    std::vector<int> hseg_sl;    // first slice of each segment (host), segments + 1 entries
    bool dseg = false;           // built with several segments: only the batched kernel reads it
    std::vector<int> hrp;        // row offsets on the host (row blocks, tuning key)
    bool rows_same = false;      // the last upload_csr found the same row offsets as before
    std::vector<long> sig;       // tuning-cache key: n, nnz, sampled row offsets
};

// Row blocks of a CSR matrix: consecutive rows, at most max_rows of them, whose entries
// total at most tile; a row with more than tile entries forms a block by itself.
void build_row_blocks(const std::vector<int> &rp, int tile, int max_rows, std::vector<int> &rb);

// A run of entries [b, e) of a CSR matrix, walked a step at a time. Positions are unsigned and the end is told
// by what is left, so nothing wraps, however close the end is to the last entry an int can count.
struct EntryRun {
    unsigned at, left;
    __host__ __device__ EntryRun(int b, int e) : at((unsigned)b), left(e > b ? (unsigned)(e - b) : 0u) {}
    __host__ __device__ bool more() const { return left > 0; }
    __host__ __device__ bool has(int k) const { return (unsigned)k < left; }   // entry k of the step
    __host__ __device__ void next(int step) {
        at += (unsigned)step;
        left = left > (unsigned)step ? left - (unsigned)step : 0u;
    }
};

// Host CSR (owning), used for symmetric expansion and transposes.
struct HostCsr {
    int n = 0;
    std::vector<int> rp, ci;
    std::vector<double> v;
};

// Set-up helpers shared by the FP64 and mixed-precision solvers (fiim_solver.cu).
void signature(DevCsr &M, const int *host_rp);
size_t csr_bytes(long n, long nnz);
int carve_csr(Arena &ar, DevCsr &M, long n, long nnz);
// Copies between pageable memory and the device through a ring of pinned buffers: all host
// threads copy one chunk to or from a pinned buffer while the other chunks' DMA runs, which moves
// pageable data several times faster than a copy from pageable memory (staged by the driver one
// page run at a time). Pinned memory and small copies go straight to cudaMemcpyAsync. copy: the
// source is read completely before it returns, the DMA may still be in flight on s; copy_out
// returns with the destination written, and waits for nothing but its own stream.
// One ring per thread and device (thread_stager), kept while the thread lives: pinning the
// buffers costs more than most copies. 32 MB each, given back when the thread ends.
struct Stager {
    static constexpr int kBufs = 4;
    static constexpr size_t kChunk = size_t(8) << 20;
    static constexpr size_t kMinStaged = size_t(4) << 20;
    void *buf[kBufs] = {};
    cudaEvent_t ev[kBufs] = {};
    bool pending[kBufs] = {};
    int next = 0;
    cudaStream_t out = nullptr;
    int copy(void *dst, const void *src, size_t bytes, cudaStream_t s);
    int copy_out(void *dst, const void *src, size_t bytes);
    bool ready();                // the pinned buffers (false: no pinned memory)
    void release();
    ~Stager() { release(); }
};
Stager &thread_stager(int device);
void copy_parallel(void *to, const void *from, size_t len);   // memcpy by all host threads

int upload_csr_async(DevCsr &M, long nnz_cap, int n, const int *rp, const int *ci, const double *v, bool device_src,
                     cudaStream_t s, Stager *stager = nullptr);
int check_fill_launch(DevCsr &M, int fill, cudaStream_t s, unsigned long long *d_count, unsigned long long *h_count);
int check_fill_finish(DevCsr &M, int fill, unsigned long long outside, cudaStream_t s);
int upload_csr(DevCsr &M, long nnz_cap, int n, const int *rp, const int *ci, const double *v, int fill,
               bool device_src, cudaStream_t s, unsigned long long *d_count, unsigned long long *h_count);
int set_tile(DevCsr &M, int tile, cudaStream_t s);
// Builds the narrow column stream (cd, cb) of M's row blocks (eb) when every block allows it.
int build_narrow(DevCsr &M, cudaStream_t s);
// The sliced-diagonal copy of M (fiim_kernels.cuh, k_spmv_dia; fiim_slices.cu). build_dia lays
// it out for the nnz device values `vals` of vbytes bytes (8, 4 or 2) and sets M.dia = 1 when
// M's rows are sorted by column, every slice (32 R rows, R = dia_rows_per_lane; slices never
// straddle a boundary of `segments`, ascending row starts from 0 to n, one segment when null)
// has at most kDiaMaxDiags diagonals, no entry holds the padding pattern and the copy moves
// fewer bytes than the CSR streams; otherwise M keeps the CSR streams. Slices with the same
// diagonals and values share one record and block (FIIM_DIA_SHARE=0: none do).
// refresh_dia, after new FP64 values M.v (and possibly new columns) with the same row offsets,
// keeps or re-places the values where the copy allows it and build_dia would choose the same form
// for them (the slices' classes are counted again), and builds it again otherwise.
// refresh_dia_async enqueues the same on `aux`, after the copies issued on `copy_s` before the
// call, so it runs while later copies do; once `aux` is done, *h_bad (pinned) is 0 when the
// copy holds the new values, else they are not to be used and refresh_dia decides again.
// release_dia frees the copy; dia_wanted is false under FIIM_DIA=0 or FIIM_SPMV=rows / staged /
// warp.
bool dia_wanted();
// Rows a lane of the sliced-diagonal copy for values of vbytes bytes: 2 for FP32, 4 for BF16;
// for FP64 0, which lets build_dia choose 1 or 2 by the matrix (FIIM_DIA_R=1 or 2 forces one).
int dia_rows_per_lane(int vbytes);
int build_dia(DevCsr &M, cudaStream_t s, int vbytes, const void *vals, const std::vector<int> *segments = nullptr);
int refresh_dia(DevCsr &M, cudaStream_t s);
int refresh_dia_async(DevCsr &M, cudaStream_t copy_s, cudaStream_t aux, cudaEvent_t done, int *h_bad);
void release_dia(DevCsr &M);
void expand_sym_upper(int n, const int *rp, const int *ci, const double *v, HostCsr &out);
void transpose_upper(int n, const int *rp, const int *ci, const double *v, HostCsr &out);

// Launch a 256-thread kernel with programmatic stream serialization (programmatic
// dependent launch: the kernel's CTAs may be scheduled while the previous kernel in the
// stream finishes; the kernels wait for it with griddepcontrol.wait before touching its
// results). FIIM_PDL=0 launches without the attribute.
inline bool pdl_enabled() {
    static const bool on = [] {
        const char *e = std::getenv("FIIM_PDL");
        return !(e && e[0] == '0' && e[1] == 0);
    }();
    return on;
}

template <typename... KArgs, typename... Args>
cudaError_t launch_k(void (*kern)(KArgs...), int grid, size_t smem, cudaStream_t s, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
}

// Resident blocks per SM of a kernel launched with 256 threads, cached by kernel address.
template <typename K>
int occupancy(K kernel) {
    constexpr int kBlockThreads = 256;
    static std::mutex mu;
    static std::map<const void *, int> occ;
    std::lock_guard<std::mutex> lk(mu);
    auto it = occ.find((const void *)kernel);
    if (it != occ.end()) return it->second;
    int b = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kernel, kBlockThreads, 0) != cudaSuccess || b < 1) {
        cudaGetLastError();
        b = 4;
    }
    occ[(const void *)kernel] = b;
    return b;
}

// Grid: enough blocks for the work, capped at one full wave of resident blocks.
template <typename K>
int grid_for(K kernel, long units_per_block, long units) {
    const long need = std::max<long>(1, (units + units_per_block - 1) / units_per_block);
    return (int)std::min<long>(need, (long)occupancy(kernel) * num_sms());
}

// The grid of the sliced-diagonal products whose sums steer the iteration, for one row a lane (four
// CTAs per SM, at most one 32-row slice a warp when the matrix is small). A property of the sums'
// tree, not of a kernel's occupancy: such products are launched on it whatever that is.
inline int dia_grid(long n) {
    return (int)std::min<long>((n + 32 * 8 - 1) / (32 * 8), 4L * num_sms());
}


}  // namespace fiim
