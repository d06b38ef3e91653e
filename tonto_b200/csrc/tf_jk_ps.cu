// tf_jk_ps.cu — thread kernels of the |ps) kets (tf_thread.cuh).
#include "tf_thread.cuh"

namespace tf {

int launch_jk_ps(int key, const JKArgs& a, cudaStream_t s, bool fp32, int variant) {
  switch (key) {
    TF_JK_CASE(launch_jk, 1, 0, 1, 0)
    TF_JK_CASE(launch_jk, 1, 1, 1, 0)
    TF_JK_CASE(launch_jk, 2, 0, 1, 0)
    default: return 0;
  }
}

}  // namespace tf
