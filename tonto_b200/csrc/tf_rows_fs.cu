// tf_rows_fs.cu — lane-group kernels of the (fs| and (fp| classes (tf_rows.cuh).
#include "tf_rows.cuh"

namespace tf {

int launch_rows_fs(int key, const RowArgs& a, cudaStream_t s) {
  switch (key) {
    TF_ROWS_CASE(3, 0, 1, 1) TF_ROWS_CASE(3, 0, 2, 0) TF_ROWS_CASE(3, 0, 2, 1) TF_ROWS_CASE(3, 0, 2, 2)
    TF_ROWS_CASE(3, 0, 3, 0)
    TF_ROWS_CASE(3, 1, 1, 0) TF_ROWS_CASE(3, 1, 1, 1) TF_ROWS_CASE(3, 1, 2, 0) TF_ROWS_CASE(3, 1, 2, 1)
    TF_ROWS_CASE(3, 1, 2, 2) TF_ROWS_CASE(3, 1, 3, 0) TF_ROWS_CASE(3, 1, 3, 1)
    default: return 0;
  }
}

}  // namespace tf
