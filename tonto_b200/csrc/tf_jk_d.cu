// tf_jk_d.cu — thread kernels of the heavier classes up to d shells (tf_thread.cuh).
#include "tf_thread.cuh"

namespace tf {

int launch_jk_d(int key, const JKArgs& a, cudaStream_t s, bool fp32, int variant) {
  switch (key) {
    TF_JK_CASE(launch_jk, 2, 0, 1, 1)
    TF_JK_CASE(launch_jk, 2, 0, 2, 0)
    TF_JK_CASE(launch_jk, 2, 1, 0, 0)
    TF_JK_CASE(launch_jk, 2, 1, 1, 0)
    TF_JK_CASE(launch_jk, 2, 2, 0, 0)
    default: return 0;
  }
}

}  // namespace tf
