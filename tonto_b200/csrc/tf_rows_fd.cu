// tf_rows_fd.cu — lane-group kernels of the (fd| classes (tf_rows.cuh).
#include "tf_rows.cuh"

namespace tf {

int launch_rows_fd(int key, const RowArgs& a, cudaStream_t s) {
  switch (key) {
    TF_ROWS_CASE(3, 2, 1, 0) TF_ROWS_CASE(3, 2, 1, 1) TF_ROWS_CASE(3, 2, 2, 0) TF_ROWS_CASE(3, 2, 2, 1)
    TF_ROWS_CASE(3, 2, 2, 2) TF_ROWS_CASE(3, 2, 3, 0) TF_ROWS_CASE(3, 2, 3, 1) TF_ROWS_CASE(3, 2, 3, 2)
    default: return 0;
  }
}

}  // namespace tf
