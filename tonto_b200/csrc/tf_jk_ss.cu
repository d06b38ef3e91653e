// tf_jk_ss.cu — thread kernels of the |ss) kets (tf_thread.cuh).
#include "tf_thread.cuh"

namespace tf {

int launch_jk_ss(int key, const JKArgs& a, cudaStream_t s, bool fp32, int variant) {
  switch (key) {
    TF_JK_CASE(launch_jk, 0, 0, 0, 0)
    TF_JK_CASE(launch_jk, 1, 0, 0, 0)
    TF_JK_CASE(launch_jk, 1, 1, 0, 0)
    TF_JK_CASE(launch_jk, 2, 0, 0, 0)
    default: return 0;
  }
}

}  // namespace tf
