// Sequential-order ICD (parity mode).
//
// Reproduces icd_iteration.cpp:149-274: voxels visited y-outer, x, z-inner;
// for each voxel alpha = sum a^2 and beta = sum a (y - y_hat) over the
// in-range entries of its column (:198-212), the penalty update
// (penalties.cpp:61-139), the positivity clamp (:233-234), x += delta and
// y_hat += delta * a (:240-249). The image and y_hat are FP64, weights and
// raw data FP32, products formed with the reference's float/double mixing.
//
// What bounds it: each update depends on the previous one, so an iteration takes
// (voxels) x (latency of one update), and a column of tens of thousands of
// entries keeps one SM's load/store unit busy for most of that. One cluster of up
// to 16 CTAs of 8 warps walks the voxels. Every data view belongs to one warp of
// the cluster, so the estimates a warp reads were last written by itself and no
// barrier orders them; a warp keeps its share of the column (index, weight,
// estimate) in registers from the gather to the update, so the update only
// stores. Left on the critical path: one round trip of estimate loads, one
// cluster barrier for alpha and beta, the penalty (every CTA evaluates it from the
// same sums and its own copy of the voxel's neighbours) and two CTA barriers; the
// next voxel's entries are fetched meanwhile. Only the summation order of
// alpha/beta differs from the reference's OpenMP reduction. Compiled with
// -fmad=false.
#include <algorithm>

#include "gpu_internal.h"

namespace {

struct SeqParams {
    int nx, ny, nz, nch, nr, nvsm, readings, penalty;
    uint64_t nvsm1;
    double cvx, cvy, vx, vy, fov_limit, lambda, delta;
};

__device__ __forceinline__ double W8(int i) {
    const double r2 = 1.0 / 1.41421356237309504880168872420969807;  // penalties.cpp:15, :33-40
    return (i == 1 || i == 3 || i == 4 || i == 6) ? 1.0 : r2;
}

// Flat index of neighbour l (0-7) of voxel q; size_t arithmetic: indices below
// zero wrap and fail `< array_size`.
__device__ __forceinline__ size_t neighbour(int q, size_t nx, int l) {
    const size_t row = l < 3 ? (size_t)q - nx : l < 5 ? (size_t)q : (size_t)q + nx;
    const int d = l < 3 ? l - 1 : l < 5 ? 2 * (l - 3) - 1 : l - 6;
    return row + (size_t)(int64_t)d;
}

// penalties.cpp:61-85 by one warp: lanes 0-7 hold a neighbour's value, every lane
// adds the eight terms in the reference's order.
__device__ double quadratic_update_warp(double alpha, double beta, double lambda, double xq, double xn, bool valid) {
    const int lane = threadIdx.x & 31;
    const double term = valid ? W8(lane) * (xn - xq) : 0.0;
    const unsigned vmask = __ballot_sync(0xffffffffu, valid);
    double sum = 0.0;
    for (int i = 0; i < 8; ++i) {
        const double v = __shfl_sync(0xffffffffu, term, i);
        if (vmask & (1u << i)) sum += v;
    }
    double ws = 0.0;
    for (int i = 0; i < 8; ++i) ws += W8(i);
    return (beta + lambda * sum) / (alpha + lambda * ws);
}

// penalties.cpp:88-154 (bisection on func) evaluated by one warp: lanes 0-7
// compute the eight neighbour terms of func in parallel and every lane then
// adds them in the order i = 0..7, so each f(d) (and hence the bisection
// path) is bit-identical to the serial evaluation. f(a) is a pure function of
// a, so it is carried along instead of being re-evaluated each step.
__device__ double edge_update_warp(double alpha, double beta, double lambda, double delta, double xq, double xn,
                                   bool valid) {
    const int lane = threadIdx.x & 31;
    if (alpha == 0.0) return 0.0;
    const double wl = lane < 8 ? W8(lane) : 0.0;
    const unsigned vmask = __ballot_sync(0xffffffffu, valid);
    double a = beta / alpha, b = beta / alpha;
    for (int i = 0; i < 8; ++i) {
        const double d = __shfl_sync(0xffffffffu, xn, i) - xq;
        if (vmask & (1u << i)) {
            if (d < a) a = d;
            if (d > b) b = d;
        }
    }
    auto f = [&](double du) {
        double term = 0.0;
        if (valid) {
            const double t = du - (xn - xq);
            const double g = 1.0 - 1.0 / (1.0 + fabs(t / delta));
            term = (t >= 0) ? wl * g : -(wl * g);
        }
        double sum = 0.0;
        for (int i = 0; i < 8; ++i) {
            const double v = __shfl_sync(0xffffffffu, term, i);
            if (vmask & (1u << i)) sum = sum + v;
        }
        return 2 * alpha * du - 2 * beta + lambda * sum;
    };
    double fa = f(a);
    double c = (a + b) / 2.0;
    for (int it = 0; it < 1000000; ++it) {
        c = (a + b) / 2.0;
        const double fc = f(c);
        if (fc == 0 || (b - a) / 2 < 0.00000001) return c;
        const int sc = fc < 0 ? -1 : 1, sa = fa < 0 ? -1 : 1;
        if (sc == sa) {
            a = c;
            fa = fc;
        } else {
            b = c;
        }
    }
    return c;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

constexpr int kSeqWarps = 8;     // warps per CTA
constexpr int kSeqCluster = 16;  // CTAs per cluster at most
constexpr int kSeqR = 8;         // entries a lane keeps in registers

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void st_remote2d(uint32_t addr, uint32_t rank, double a, double b) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(r), "d"(a), "d"(b) : "memory");
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// A voxel of the reference's visiting order (y outer, x, z inner).
struct SeqVoxel {
    int i, j, k;  // j == ny: past the last
};

// `vb` consecutive data views form a block; block g belongs to warp g mod (warps of
// the cluster), and a view window holds at most one block of each warp.
__global__ void __launch_bounds__(32 * kSeqWarps) icd_seq_kernel(
    SeqParams P, const int64_t* __restrict__ colptr, const uint32_t* __restrict__ vptr,
    const int32_t* __restrict__ idx, const float* __restrict__ w, const float* __restrict__ raw,
    const int32_t* __restrict__ start, double* est, double* x, int cluster, int vb) {
    __shared__ double2 s_warp[kSeqWarps];
    __shared__ double2 s_cta[2][kSeqCluster];
    __shared__ double s_upd;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    uint32_t rank;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    const int nwarps = cluster * kSeqWarps, self = wid * cluster + (int)rank;
    const size_t nxs = (size_t)P.nx;
    const size_t nvox = (size_t)P.nx * P.ny * P.nz;

    auto inside = [&](int i, int j) {
        const double y = (j - P.cvy) * P.vy, xx = (i - P.cvx) * P.vx;
        return (xx * xx + y * y) < P.fov_limit;  // icd_iteration.cpp:181
    };
    auto settle = [&](SeqVoxel& v) {  // the first column at or after (i, j) inside the FOV
        while (v.j < P.ny && !inside(v.i, v.j))
            if (++v.i == P.nx) {
                v.i = 0;
                ++v.j;
            }
    };
    auto next = [&](SeqVoxel v) {
        if (v.j >= P.ny) return v;
        if (++v.k == P.nz) {
            v.k = 0;
            if (++v.i == P.nx) {
                v.i = 0;
                ++v.j;
            }
            settle(v);
        }
        return v;
    };
    // This warp's entries [b, e) of a voxel's in-range column, and the sinogram offset.
    auto range = [&](const SeqVoxel& v, int64_t& b, int64_t& e, int& off) {
        b = e = 0;
        off = 0;
        if (v.j >= P.ny) return;
        const int s = __ldg(start + v.k);
        const int v0 = max(0, -s), v1 = min(P.nvsm, P.readings - s);
        if (v1 <= v0) return;
        const int first = (s + v0) / vb;
        const int g = first + (self - first % nwarps + nwarps) % nwarps;
        const int va = max(v0, g * vb - s), ve = min(v1, (g + 1) * vb - s);
        off = s * P.nch * P.nr;
        if (va >= ve) return;
        const uint64_t col = (uint64_t)v.i + nxs * v.j;
        const int64_t cb = __ldg(colptr + col);
        b = cb + __ldg(vptr + col * P.nvsm1 + va);
        e = cb + __ldg(vptr + col * P.nvsm1 + ve);
    };
    int qi[kSeqR];
    float wi[kSeqR];
    auto fetch = [&](int64_t b, int64_t e, int off) {
#pragma unroll
        for (int r = 0; r < kSeqR; ++r) {
            const int64_t m = b + lane + 32 * r;
            qi[r] = -1;
            wi[r] = 0.f;
            if (m < e) {
                qi[r] = __ldg(idx + m) + off;
                wi[r] = __ldg(w + m);
            }
        }
    };

    SeqVoxel cur = {0, 0, 0};
    settle(cur);
    SeqVoxel nx1 = next(cur);
    int64_t b, e, b1, e1;
    int off, off1;
    range(cur, b, e, off);
    fetch(b, e, off);
    range(nx1, b1, e1, off1);
    cluster_arrive();  // every CTA runs before another writes to it
    cluster_wait();
    int par = 0;
    for (; cur.j < P.ny; par ^= 1) {
        const int q = (int)((uint64_t)cur.i + nxs * cur.j + nxs * P.ny * cur.k);
        // The voxel and its in-plane neighbours (written by this very warp).
        double xq = 0.0, xn = 0.0;
        bool valid = false;
        if (wid == 0) {
            xq = x[q];
            if (lane < 8) {
                const size_t n = neighbour(q, nxs, lane);
                valid = n < nvox;
                if (valid) xn = x[n];
            }
        }
        double ev[kSeqR];
        float rv[kSeqR];
#pragma unroll
        for (int r = 0; r < kSeqR; ++r) {
            ev[r] = qi[r] >= 0 ? est[qi[r]] : 0.0;
            rv[r] = qi[r] >= 0 ? __ldg(raw + qi[r]) : 0.f;
        }
        double alpha = 0.0, beta = 0.0;
#pragma unroll
        for (int r = 0; r < kSeqR; ++r) {
            const float ww = wi[r] * wi[r];  // float product (:208)
            alpha += (double)ww;
            beta += (double)wi[r] * ((double)rv[r] - ev[r]);
        }
        for (int64_t m = b + 32 * kSeqR + lane; m < e; m += 32) {
            const float wm = __ldg(w + m);
            const int index = __ldg(idx + m) + off;
            const float ww = wm * wm;
            alpha += (double)ww;
            beta += (double)wm * ((double)__ldg(raw + index) - est[index]);
        }
        alpha = warp_sum(alpha);
        beta = warp_sum(beta);
        if (lane == 0) s_warp[wid] = make_double2(alpha, beta);
        __syncthreads();
        if (wid == 0) {
            double2 t = lane < kSeqWarps ? s_warp[lane] : make_double2(0.0, 0.0);
#pragma unroll
            for (int o = kSeqWarps / 2; o > 0; o >>= 1) {
                t.x += __shfl_xor_sync(0xffffffffu, t.x, o);
                t.y += __shfl_xor_sync(0xffffffffu, t.y, o);
            }
            t.x = __shfl_sync(0xffffffffu, t.x, 0);
            t.y = __shfl_sync(0xffffffffu, t.y, 0);
            if (lane < cluster) st_remote2d(smem_addr(&s_cta[par][rank]), (uint32_t)lane, t.x, t.y);
            __syncwarp();
        }
        cluster_arrive();
        // While the sums travel: where the voxel after next keeps its entries.
        const SeqVoxel nx2 = next(nx1);
        int64_t b2, e2;
        int off2;
        range(nx2, b2, e2, off2);
        int qn[kSeqR];
        float wn[kSeqR];
#pragma unroll
        for (int r = 0; r < kSeqR; ++r) {
            const int64_t m = b1 + lane + 32 * r;
            qn[r] = -1;
            wn[r] = 0.f;
            if (m < e1) {
                qn[r] = __ldg(idx + m) + off1;
                wn[r] = __ldg(w + m);
            }
        }
        cluster_wait();
        if (wid == 0) {
            double2 t = lane < cluster ? s_cta[par][lane] : make_double2(0.0, 0.0);
            const double A = warp_sum(t.x), B = warp_sum(t.y);
            double upd = P.penalty == CTBB_PENALTY_QUADRATIC
                             ? quadratic_update_warp(A, B, P.lambda, xq, xn, valid)
                             : edge_update_warp(A, B, P.lambda, P.delta, xq, xn, valid);
            if (upd + xq < 0) upd = -xq;
            if (lane == 0) {
                x[q] = xq + upd;  // every CTA stores the same value
                s_upd = upd;
            }
            __syncwarp();
        }
        __syncthreads();
        const double upd = s_upd;
#pragma unroll
        for (int r = 0; r < kSeqR; ++r)
            if (qi[r] >= 0) est[qi[r]] = ev[r] + upd * (double)wi[r];
        for (int64_t m = b + 32 * kSeqR + lane; m < e; m += 32) {
            const int index = __ldg(idx + m) + off;
            est[index] += upd * (double)__ldg(w + m);
        }
        __syncwarp();
        cur = nx1;
        nx1 = nx2;
        b = b1;
        e = e1;
        off = off1;
        b1 = b2;
        e1 = e2;
        off1 = off2;
#pragma unroll
        for (int r = 0; r < kSeqR; ++r) {
            qi[r] = qn[r];
            wi[r] = wn[r];
        }
    }
    cluster_arrive();  // no CTA leaves while another may still write to it
    cluster_wait();
}

// The largest cluster (a power of two up to kSeqCluster) the device can place.
ctbb_status seq_cluster(int* out) {
    CTBB_CUDA(cudaFuncSetAttribute(icd_seq_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    for (int c = kSeqCluster; c > 1; c /= 2) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(c);
        cfg.blockDim = dim3(32 * kSeqWarps);
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = c;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, icd_seq_kernel, &cfg) == cudaSuccess && n > 0) {
            *out = c;
            return CTBB_OK;
        }
        cudaGetLastError();
    }
    *out = 1;
    return CTBB_OK;
}

}  // namespace

namespace ctbb {

ctbb_status launch_icd_sequential(ctbb_recon* rc, const ctbb_ssm* ssm, int n_iter, float* ms) {
    const ctbb_geom_c& g = rc->geom;
    SeqParams P;
    P.nx = (int)g.num_voxels_x;
    P.ny = (int)g.num_voxels_y;
    P.nz = (int)g.num_voxels_z;
    P.nch = (int)g.n_channels;
    P.nr = (int)g.Nrows_projection;
    P.nvsm = (int)ssm->nvsm;
    P.nvsm1 = ssm->nvsm + 1;
    P.readings = (int)g.Readings;
    P.penalty = g.penalty;
    P.cvx = g.center_voxel_x;
    P.cvy = g.center_voxel_y;
    P.vx = g.voxel_size_x;
    P.vy = g.voxel_size_y;
    P.fov_limit = (g.acquisition_fov / 2.0) * (g.acquisition_fov / 2.0);  // icd_iteration.cpp:154
    P.lambda = g.lambda;
    P.delta = g.delta;
    cudaStream_t st = rc->ctx->stream;
    cudaEvent_t e0, e1;
    CTBB_CUDA(cudaEventCreate(&e0));
    CTBB_CUDA(cudaEventCreate(&e1));
    CTBB_CUDA(cudaEventRecord(e0, st));
    int cluster = 1;
    CTBB_TRY(seq_cluster(&cluster));
    // Views per block: a window of nvsm views touches at most (warps) blocks.
    const int warps = cluster * kSeqWarps;
    const int vb = std::max(1, (P.nvsm + warps - 2) / (warps - 1));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(cluster);
    cfg.blockDim = dim3(32 * kSeqWarps);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cluster;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    for (int it = 0; it < n_iter; ++it)
        CTBB_CUDA(cudaLaunchKernelEx(&cfg, icd_seq_kernel, P, (const int64_t*)ssm->d_colptr,
                                     (const uint32_t*)ssm->d_vptr, (const int32_t*)ssm->d_idx,
                                     (const float*)ssm->d_w32, (const float*)rc->d_raw, (const int32_t*)rc->d_start,
                                     rc->d_est64, rc->d_x64, cluster, vb));
    CTBB_CUDA(cudaEventRecord(e1, st));
    CTBB_CUDA(cudaEventSynchronize(e1));
    cudaEventElapsedTime(ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    return CTBB_OK;
}

}  // namespace ctbb
