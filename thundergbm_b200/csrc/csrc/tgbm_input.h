// From what the caller hands over to the stored values on the device.
//
// Three forms arrive: a CSR, a CSR whose rows all hold the columns 0 .. C - 1 in order (a dense matrix in CSR clothing;
// its column ids and row pointers say nothing and are not sent), and a row-major float or double matrix whose zeros are
// not stored.  A matrix without zeros is the second form at once; otherwise its CSR is made on the device, in two passes
// at HBM speed.
#pragma once
#include "tgbm_device.cuh"

namespace tgbm {

struct DeviceRows {
    DevBuf<int> row_ptr, col;   // empty while full_cols > 0, until need_csr()
    DevBuf<float> val;
    size_t nnz = 0;
    int full_cols = 0;          // > 0: every row stores the columns 0 .. full_cols - 1
    int max_col = -1, min_col = 0;   // over the stored values

    // up_threads: host threads that may stage a pageable source
    void upload(const DataSet &ds, cudaStream_t stream, int num_sms, int up_threads);
    void need_csr(int n_rows, cudaStream_t stream, int num_sms);   // row_ptr and col of a matrix without missing values
    void release() { row_ptr.release(); col.release(); val.release(); }

private:
    void upload_dense(const DataSet &ds, cudaStream_t stream, int num_sms, int up_threads);
};

}  // namespace tgbm
