// Device-resident objects behind the opaque handles of the C ABI, and the
// internal launch functions shared between translation units.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <vector>

#include "common.h"

#define CTBB_CUDA(call)                                                                        \
    do {                                                                                       \
        cudaError_t err__ = (call);                                                            \
        if (err__ != cudaSuccess)                                                              \
            return ::ctbb::fail(err__ == cudaErrorMemoryAllocation ? CTBB_ERR_OOM : CTBB_ERR_CUDA, \
                                "%s:%d %s: %s", __FILE__, __LINE__, #call,                     \
                                cudaGetErrorString(err__));                                    \
    } while (0)

#define CTBB_TRY(call)                        \
    do {                                      \
        ctbb_status st__ = (call);            \
        if (st__ != CTBB_OK) return st__;     \
    } while (0)

struct ctbb_ctx {
    // Objects (matrices, reconstructions, batches) created on this context;
    // ctbb_gpu_destroy defers the teardown until the last of them is freed.
    std::atomic<int> refs{0};
    std::atomic<bool> closing{false};
    int device = 0;
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    int sm_count = 148;
    size_t smem_per_block_optin = 0;
    // Reusable FP64 reduction scratch (partial sums), sized on demand.
    double* d_partials = nullptr;
    size_t partials_cap = 0;
    // Work-queue head for the grouped ICD kernel.
    unsigned long long* d_queue = nullptr;
    int* d_flags = nullptr;  // device-side error flags
};

// Second layout of a sinogram, for the bulk-staged kernels with many updates in
// flight (bulk_layout_pays): views fastest but for groups of 2 channels x 2 rows,
//   (((channel >> 1) * row groups + (row >> 1)) * stride + view) * 4, then the
//   channel's and the row's low bits.
// What bounds those launches is not bytes but requests: a voxel meets a few
// neighbouring channels and two rows per view, and its channels drift slowly from
// view to view, so in the raw data's order (row fastest) neighbouring entries each
// lie in another 128-byte line. Here a line holds 8 views of a group and a 32-byte
// sector two: the 16 entry pairs of a warp's load touch 5.7 lines and 12.0 sectors
// instead of 15.0 and 16.4 (mean of 40 columns of the 512 x 512 x 64 benchmark; on
// 2.3 mm voxels 6.9 and 9.9; groups of 4 rows of one channel: 6.7 and 13.1, 9.7 and
// 13.7). A slice's first view still adds a constant to every index of a column.
// Channels and rows are padded to whole groups, views to whole lines; padding holds
// zeros. stride 0: the raw data's order, also where there is one row or channel or
// the index would not fit 31 bits.
struct SinoLayout {
    int nr = 0, nch = 0, nrb = 0, ncb = 0;
    uint32_t stride = 0;  // views, padded

    static SinoLayout raw() { return SinoLayout(); }
    static SinoLayout grouped(uint64_t nch, uint64_t nr, uint64_t views) {
        SinoLayout l;
        const uint64_t nrb = (nr + 1) / 2, ncb = (nch + 1) / 2, stride = (views + 7) / 8 * 8;
        if (nr < 2 || nch < 2 || ncb * nrb * stride * 4 >= 2147483648ull) return l;
        l.nr = (int)nr;
        l.nch = (int)nch;
        l.nrb = (int)nrb;
        l.ncb = (int)ncb;
        l.stride = (uint32_t)stride;
        return l;
    }
    bool is_raw() const { return stride == 0; }
    // Elements of a sinogram (grouped layouts).
    uint64_t size() const { return (uint64_t)ncb * nrb * stride * 4; }
    __host__ __device__ uint32_t at(uint32_t view, uint32_t ch, uint32_t row) const {
        return (((ch >> 1) * (uint32_t)nrb + (row >> 1)) * stride + view) * 4 + (ch & 1) * 2 + (row & 1);
    }
    // Index of the raw data's element q = row + nr * (channel + nch * view).
    __host__ __device__ uint32_t from_raw(uint32_t q) const {
        const uint32_t t = q / (uint32_t)nr, v = t / (uint32_t)nch;
        return at(v, t - v * (uint32_t)nch, q - t * (uint32_t)nr);
    }
    // The same element in a layout of another stride.
    __host__ __device__ uint32_t restride(uint32_t a, const SinoLayout& to) const {
        const uint32_t g = a >> 2, line = g / stride;
        return (line * to.stride + (g - line * stride)) * 4 + (a & 3);
    }
    // From an odd row to the next row of the same view and channel (from an even one: 1).
    uint32_t row_step() const { return stride * 4 - 1; }
    bool operator==(const SinoLayout& o) const { return nr == o.nr && nch == o.nch && stride == o.stride; }
};

// Stored system matrix: per voxel column c = i + nx*j, entries sorted by
// q = row + Nrows*(channel + n_channels*view). colptr[c] is the first entry of
// column c; vptr[c*(nvsm+1) + v] is the offset (relative to colptr[c]) of the
// first entry of SSM view v, so a view window [v0, v1) is one contiguous run.
struct ctbb_ssm {
    ctbb_ctx* ctx = nullptr;
    // Unique for the life of the process: what a reconstruction keeps about a
    // matrix (captured launches, entry counts) is keyed by it, since a later
    // matrix may be allocated at the same addresses.
    uint64_t id = next_id();
    static uint64_t next_id() {
        static std::atomic<uint64_t> n{0};
        return ++n;
    }
    ctbb_geom_c geom{};
    uint64_t ncol = 0, nvsm = 0, nnz = 0, max_col_nnz = 0;
    int64_t* d_colptr = nullptr;  // [ncol + 1]
    uint32_t* d_vptr = nullptr;   // [ncol * (nvsm + 1)]
    int32_t* d_idx = nullptr;     // [nnz]
    float* d_w32 = nullptr;       // [nnz] (CTBB_SSM_FP32 held)
    __half* d_w16 = nullptr;      // [nnz] (CTBB_SSM_FP16 held)
    // Entry pairs (built on first use from idx + w16, ssm_build_pairs):
    // {q, w0 | w1 << 16} for two entries at consecutive sinogram indices,
    // w1 = 0 for a lone entry; same column / per-view offset layout.
    int64_t* d_pcolptr = nullptr;  // [ncol + 1]
    uint32_t* d_pvptr = nullptr;   // [ncol * (nvsm + 1)]
    uint2* d_pairs = nullptr;      // [npairs]
    uint64_t npairs = 0;
    bool pairs_checked = false;  // build tried (pairs kept only where they pay)
    bool pairs_pay = false;      // and kept
    SinoLayout pair_lay;         // of the pairs' indices; entries keep the raw data's order
    uint64_t pairs_id = 0;       // changes with the pairs and with their layout
    int weights = 0;
    int ffs = 0;
    double build_ms = 0.0;
    uint64_t bytes = 0;
};

// Device-resident ICD state. The sequential (parity) mode keeps the image
// and the sinogram estimate y_hat = A x in FP64 like icd_iteration.cpp:47-48;
// the grouped mode keeps an FP32 image and the FP32 error sinogram e = y - A x.
struct ctbb_recon {
    ctbb_ctx* ctx = nullptr;
    ctbb_geom_c geom{};
    uint64_t nvox = 0, data_size = 0;
    std::vector<uint64_t> slice_indices;
    int32_t* d_start = nullptr;  // [nz] first data view of each slice's SSM window
    float* d_raw = nullptr;      // y
    double* d_x64 = nullptr;     // sequential-mode image
    double* d_est64 = nullptr;   // sequential-mode A x (FP64); also FP64 refresh accumulator
    float* d_x32 = nullptr;      // grouped-mode image
    float* d_e32 = nullptr;      // grouped-mode y - A x
    SinoLayout bulk_lay;         // the second layout of this scan
    bool e_bulk = false;         // d_e32 is in it (else in the raw data's order)
    int rep = 0;                 // 0: x64/est64 current, 1: x32/e32 current
    // Sum over voxels inside the FOV of in-range matrix entries (cached per matrix).
    uint64_t entries_ssm = 0;
    double entries = 0.0;
    // Grouped-mode visiting order: packed (column * nz + slice) per item,
    // built once per lattice spacing.
    uint32_t* d_order = nullptr;
    uint64_t n_order = 0;
    int order_P = 0;
    // Where each slice stack (same-parity slices of one cell) starts in the
    // order, n_stacks + 1 entries (the last is n_order).
    uint32_t* d_stacks = nullptr;
    uint64_t n_stacks = 0;
    // Learned warm start: per-voxel priority (size of the warm-start step)
    // and the visiting order restricted to the highest-priority voxels.
    float* d_prio = nullptr;
    uint32_t* d_prio_order = nullptr;
    uint64_t n_prio_order = 0;
    uint32_t* d_prio_stacks = nullptr;
    uint64_t n_prio_stacks = 0;
    int prio_P = 0;
    // Grouped iteration captured in a CUDA graph, and the launch it encodes.
    cudaGraphExec_t icd_graph = nullptr;
    std::vector<unsigned char> icd_graph_key;
};

struct ctbb_cnn;

namespace ctbb {

// Reference counting of a context by the objects created on it.
void ctx_retain(ctbb_ctx* ctx);
void ctx_release(ctbb_ctx* ctx);

ctbb_status ensure_partials(ctbb_ctx* ctx, size_t n);

// ssm.cu
ctbb_status ssm_validate_geometry(const ctbb_geom_c& g);
// The pair form with its indices in `lay`; no pairs where they do not pay.
ctbb_status ssm_build_pairs(ctbb_ssm* s, const SinoLayout& lay);

// recon.cu
// Refuses a matrix of another geometry or context.
ctbb_status check_pair(const ctbb_recon* rc, const ctbb_ssm* ssm);
// Grouped mode: the error sinogram in the second layout or in the raw data's order.
ctbb_status arrange_error(ctbb_recon* rc, bool bulk);
ctbb_status recon_to_grouped(ctbb_recon* rc, const ctbb_ssm* ssm);
ctbb_status recon_to_sequential(ctbb_recon* rc, const ctbb_ssm* ssm);
ctbb_status forward_project_f64(ctbb_recon* rc, const ctbb_ssm* ssm, bool from_x32, double* d_out);
ctbb_status cost_f64(ctbb_recon* rc, const ctbb_ssm* ssm, bool exact, double* out);

// icd_seq.cu
ctbb_status launch_icd_sequential(ctbb_recon* rc, const ctbb_ssm* ssm, int n_iter, float* ms);

// icd_grouped.cu
ctbb_status launch_icd_grouped(ctbb_recon* rc, const ctbb_ssm* ssm, const ctbb_icd_opts& o,
                               float* ms, double* entries, uint64_t* items, double* scattered = nullptr);
int stage_capacity(const ctbb_ctx* ctx, int nw, int wbytes);
int default_warps_in_flight(const ctbb_recon* rc);
int lattice_spacing(const ctbb_recon* rc, const ctbb_icd_opts& o);
uint64_t requested_items(const ctbb_recon* rc, const ctbb_icd_opts& o);
uint64_t max_items_in_flight(uint64_t n_items, int nz, int T);
ctbb_status inrange_entries(ctbb_recon* rc, const ctbb_ssm* ssm, double* out);

// rotate.cu
ctbb_status rotate_volume(ctbb_ctx* ctx, const ctbb_geom_c& g, const double* tube_angles_deg,
                          const uint64_t* slice_indices, const float* d_in, float* d_out, int direction);

// cnn_tc.cu
ctbb_status conv_mid_tc(ctbb_ctx* ctx, int nx, int ny, int nz, const __nv_bfloat16* in, const __nv_bfloat16* wt,
                        const float* bias, const __nv_bfloat16* residual, const __nv_bfloat16* mask, int relu,
                        __nv_bfloat16* out, int* err);

// cnn.cu
ctbb_status cnn_predict_correction(ctbb_cnn* c, const float* x_dev, int nx, int ny, int nz, float* d_dev);
ctbb_status apply_correction(ctbb_ctx* ctx, uint64_t n, float* x_dev, const float* d_dev, float* prio_dev);
ctbb_ctx* cnn_ctx(const ctbb_cnn* c);
ctbb_status cnn_check_flag(ctbb_cnn* c);

}  // namespace ctbb
