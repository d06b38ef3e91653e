// tf_jk_l2.cu — thread kernels of the larger classes, for lists long enough (dispatch_jk) (tf_thread.cuh).
#include "tf_thread.cuh"

namespace tf {

int launch_jk_l2(int key, const JKArgs& a, cudaStream_t s, bool fp32, int variant) {
  switch (key) {
    TF_JK_CASE(launch_jk_f64, 3, 0, 2, 0)
    TF_JK_CASE(launch_jk_f64, 3, 0, 3, 0)
    TF_JK_CASE(launch_jk_f64, 3, 2, 1, 0)
    TF_JK_CASE(launch_jk_f64, 3, 3, 1, 0)
    default: return 0;
  }
}

}  // namespace tf
