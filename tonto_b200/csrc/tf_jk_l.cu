// tf_jk_l.cu — thread kernels of the larger classes, for lists long enough (dispatch_jk) (tf_thread.cuh).
#include "tf_thread.cuh"

namespace tf {

int launch_jk_l(int key, const JKArgs& a, cudaStream_t s, bool fp32, int variant) {
  switch (key) {
    TF_JK_CASE(launch_jk_f64, 1, 1, 1, 1)
    TF_JK_CASE(launch_jk_f64, 2, 1, 2, 0)
    TF_JK_CASE(launch_jk_f64, 2, 2, 1, 0)
    TF_JK_CASE(launch_jk_f64, 3, 0, 1, 1)
    TF_JK_CASE(launch_jk_f64, 3, 1, 1, 0)
    default: return 0;
  }
}

}  // namespace tf
