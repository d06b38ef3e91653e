// tf_rows_d.cu — lane-group kernels of the classes up to d shells (tf_rows.cuh).
#include "tf_rows.cuh"

namespace tf {

int launch_rows_d(int key, const RowArgs& a, cudaStream_t s) {
  switch (key) {
    TF_ROWS_CASE(1, 1, 1, 1)
    TF_ROWS_CASE(2, 1, 1, 1) TF_ROWS_CASE(2, 1, 2, 0) TF_ROWS_CASE(2, 1, 2, 1)
    TF_ROWS_CASE(2, 2, 1, 0) TF_ROWS_CASE(2, 2, 1, 1) TF_ROWS_CASE(2, 2, 2, 0) TF_ROWS_CASE(2, 2, 2, 1)
    TF_ROWS_CASE(2, 2, 2, 2)
    default: return 0;
  }
}

}  // namespace tf
