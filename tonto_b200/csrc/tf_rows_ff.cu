// tf_rows_ff.cu — lane-group kernels of the (ff| classes (tf_rows.cuh).
#include "tf_rows.cuh"

namespace tf {

int launch_rows_ff(int key, const RowArgs& a, cudaStream_t s) {
  switch (key) {
    TF_ROWS_CASE(3, 3, 1, 0) TF_ROWS_CASE(3, 3, 1, 1) TF_ROWS_CASE(3, 3, 2, 0) TF_ROWS_CASE(3, 3, 2, 1)
    TF_ROWS_CASE(3, 3, 2, 2) TF_ROWS_CASE(3, 3, 3, 0) TF_ROWS_CASE(3, 3, 3, 1) TF_ROWS_CASE(3, 3, 3, 2)
    TF_ROWS_CASE(3, 3, 3, 3)
    default: return 0;
  }
}

}  // namespace tf
