// From what the caller hands over to the stored values on the device (tgbm_input.h).
#include "tgbm_input.h"

#include <cub/cub.cuh>

#include <algorithm>

namespace tgbm {

// Stored values per row and the largest column that holds one.  A warp takes a row, lanes over the columns.
template <typename T>
static __global__ void __launch_bounds__(256)
k_dense_count(const T *__restrict__ x, int n, int c, int *__restrict__ count, int *__restrict__ max_col) {
    const int lane = threadIdx.x & 31;
    int top = -1;
    for (int r = (blockIdx.x * 256 + threadIdx.x) >> 5; r < n; r += gridDim.x * 8) {
        const T *row = x + (size_t)r * c;
        int cnt = 0;
        for (int j0 = 0; j0 < c; j0 += 32) {
            const bool stored = j0 + lane < c && row[j0 + lane] != T(0);   // a NaN is stored
            const unsigned m = __ballot_sync(0xffffffffu, stored);
            cnt += __popc(m);
            if (m) top = max(top, j0 + 31 - __clz(m));
        }
        if (lane == 0) count[r] = cnt;
    }
    __shared__ int s_top;
    if (threadIdx.x == 0) s_top = -1;
    __syncthreads();
    if (lane == 0 && top >= 0) atomicMax(&s_top, top);
    __syncthreads();
    if (threadIdx.x == 0 && s_top >= 0) atomicMax(max_col, s_top);
}

// The CSR of the matrix; row_ptr is the exclusive scan of the counts above.
template <typename T>
static __global__ void __launch_bounds__(256)
k_dense_fill(const T *__restrict__ x, int n, int c, const int *__restrict__ row_ptr, int *__restrict__ col, float *__restrict__ val) {
    const int lane = threadIdx.x & 31;
    for (int r = (blockIdx.x * 256 + threadIdx.x) >> 5; r < n; r += gridDim.x * 8) {
        const T *row = x + (size_t)r * c;
        int at = row_ptr[r];
        for (int j0 = 0; j0 < c; j0 += 32) {
            const T v = j0 + lane < c ? row[j0 + lane] : T(0);
            const bool stored = v != T(0);
            const unsigned m = __ballot_sync(0xffffffffu, stored);
            if (stored) {
                const int p = at + __popc(m & ((1u << lane) - 1u));
                col[p] = j0 + lane;
                val[p] = (float)v;
            }
            at += __popc(m);
        }
    }
}

static __global__ void k_to_float(const double *__restrict__ x, size_t n, float *__restrict__ out) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) out[i] = (float)x[i];
}

// column ids and row pointers of a matrix without missing values, for the paths that want them
static __global__ void k_full_col(int *__restrict__ col, size_t n, int c) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) col[i] = (int)((unsigned)i % (unsigned)c);
}
static __global__ void k_full_row_ptr(int *__restrict__ row_ptr, int n, int c) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i <= n; i += gridDim.x * blockDim.x) row_ptr[i] = i * c;
}

static __global__ void k_widen_ids(const uint16_t *__restrict__ in, size_t n, int *__restrict__ out) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) out[i] = in[i];
}

// The largest and smallest column index are found on the device, at HBM speed, instead of by a pass over the host copy.
void DeviceRows::upload(const DataSet &ds, cudaStream_t stream, int num_sms, int up_threads) {
    const int N = ds.n_rows;
    if (ds.is_dense()) {
        upload_dense(ds, stream, num_sms, up_threads);
        return;
    }
    nnz = (size_t)ds.rp[N];
    val.alloc(std::max<size_t>(nnz, 1));
    const int cols = N > 0 ? ds.rp[1] : 0;
    if (upload_csr_values(val.p, ds.vv, ds.rp, ds.ci, N, cols, stream, up_threads)) {
        full_cols = cols;
        max_col = cols - 1;
        return;
    }
    row_ptr.alloc(N + 1); col.alloc(std::max<size_t>(nnz, 1));
    upload_h2d(row_ptr.p, ds.rp, sizeof(int) * (size_t)(N + 1), stream, up_threads);
    {
        DevBuf<uint16_t> narrow;
        narrow.alloc(std::max<size_t>(nnz, 1));
        if (upload_ids16(narrow.p, ds.ci, nnz, up_threads)) {
            k_widen_ids<<<(int)std::min<size_t>((nnz + 255) / 256, (size_t)num_sms * 16), 256, 0, stream>>>(narrow.p, nnz, col.p);
            TGBM_CUDA(cudaStreamSynchronize(stream));
        } else {
            upload_h2d(col.p, ds.ci, sizeof(int) * nnz, stream, up_threads);
        }
    }
    if (nnz) {
        DevBuf<int> d_mm;
        d_mm.alloc(2);
        size_t tb = 0, tb2 = 0;
        TGBM_CUDA(cub::DeviceReduce::Max(nullptr, tb, col.p, d_mm.p, (long long)nnz, stream));
        TGBM_CUDA(cub::DeviceReduce::Min(nullptr, tb2, col.p, d_mm.p + 1, (long long)nnz, stream));
        DevBuf<unsigned char> tmp;
        tmp.alloc(std::max<size_t>(std::max(tb, tb2), 1));
        TGBM_CUDA(cub::DeviceReduce::Max(tmp.p, tb, col.p, d_mm.p, (long long)nnz, stream));
        TGBM_CUDA(cub::DeviceReduce::Min(tmp.p, tb2, col.p, d_mm.p + 1, (long long)nnz, stream));
        int h_mm[2] = {0, 0};
        TGBM_CUDA(cudaMemcpyAsync(h_mm, d_mm.p, sizeof(h_mm), cudaMemcpyDeviceToHost, stream));
        TGBM_CUDA(cudaStreamSynchronize(stream));
        max_col = h_mm[0]; min_col = h_mm[1];
    }
}

void DeviceRows::upload_dense(const DataSet &ds, cudaStream_t stream, int num_sms, int up_threads) {
    const int N = ds.n_rows, C = ds.dense_cols;
    const size_t cells = (size_t)N * C;
    DevBuf<double> xd;
    DevBuf<float> xf;
    const int grid = num_sms * 8;
    DevBuf<int> count, top;
    int h_top = -1, h_nnz = 0;
    row_ptr.alloc(N + 1);
    if (cells) {
        if (ds.dense_f64) xd.alloc(cells); else xf.alloc(cells);
        upload_h2d(ds.dense_f64 ? (void *)xd.p : (void *)xf.p, ds.dense, (ds.dense_f64 ? 8 : 4) * cells, stream, up_threads);
        count.alloc(N + 1); top.alloc(1);
        TGBM_CUDA(cudaMemsetAsync(top.p, 0xff, sizeof(int), stream));
        TGBM_CUDA(cudaMemsetAsync(count.p + N, 0, sizeof(int), stream));
        if (ds.dense_f64) k_dense_count<<<grid, 256, 0, stream>>>(xd.p, N, C, count.p, top.p);
        else k_dense_count<<<grid, 256, 0, stream>>>(xf.p, N, C, count.p, top.p);
        size_t tb = 0;
        TGBM_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tb, count.p, row_ptr.p, N + 1, stream));
        DevBuf<unsigned char> tmp;
        tmp.alloc(std::max<size_t>(tb, 1));
        TGBM_CUDA(cub::DeviceScan::ExclusiveSum(tmp.p, tb, count.p, row_ptr.p, N + 1, stream));
        TGBM_CUDA(cudaMemcpyAsync(&h_top, top.p, sizeof(int), cudaMemcpyDeviceToHost, stream));
        TGBM_CUDA(cudaMemcpyAsync(&h_nnz, row_ptr.p + N, sizeof(int), cudaMemcpyDeviceToHost, stream));
        TGBM_CUDA(cudaStreamSynchronize(stream));
    } else {
        row_ptr.zero(stream);
    }
    nnz = (size_t)h_nnz;
    max_col = h_top;
    if (cells && nnz == cells) {
        full_cols = C;
        row_ptr.release();
        if (ds.dense_f64) {
            val.alloc(cells);
            k_to_float<<<grid, 256, 0, stream>>>(xd.p, cells, val.p);
            TGBM_CUDA(cudaStreamSynchronize(stream));
        } else {
            val.take(xf);
        }
        return;
    }
    col.alloc(std::max<size_t>(nnz, 1)); val.alloc(std::max<size_t>(nnz, 1));
    if (nnz) {
        if (ds.dense_f64) k_dense_fill<<<grid, 256, 0, stream>>>(xd.p, N, C, row_ptr.p, col.p, val.p);
        else k_dense_fill<<<grid, 256, 0, stream>>>(xf.p, N, C, row_ptr.p, col.p, val.p);
    }
    TGBM_CUDA(cudaStreamSynchronize(stream));
}

// column ids and row pointers of a matrix without missing values
void DeviceRows::need_csr(int N, cudaStream_t stream, int num_sms) {
    if (!full_cols || col.p) return;
    row_ptr.alloc(N + 1); col.alloc(std::max<size_t>(nnz, 1));
    k_full_row_ptr<<<std::min((N + 256) / 256, num_sms * 8), 256, 0, stream>>>(row_ptr.p, N, full_cols);
    if (nnz) k_full_col<<<(int)std::min<size_t>((nnz + 255) / 256, (size_t)num_sms * 16), 256, 0, stream>>>(col.p, nnz, full_cols);
}

}  // namespace tgbm
