// tf_jk_f.cu — thread kernels of the classes with an f shell (tf_thread.cuh).
#include "tf_thread.cuh"

namespace tf {

int launch_jk_f(int key, const JKArgs& a, cudaStream_t s, bool fp32, int variant) {
  switch (key) {
    TF_JK_CASE(launch_jk_f64, 3, 0, 0, 0)
    TF_JK_CASE(launch_jk_f64, 3, 0, 1, 0)
    TF_JK_CASE(launch_jk_f64, 3, 1, 0, 0)
    TF_JK_CASE(launch_jk_f64, 3, 2, 0, 0)
    TF_JK_CASE(launch_jk_f64, 3, 3, 0, 0)
    default: return 0;
  }
}

}  // namespace tf
