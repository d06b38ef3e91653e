// tf_jk_ss.cu — thread kernels of the |ss) kets (tf_thread.cuh).
#include "tf_thread.cuh"

namespace tf {

bool launch_jk_ss(int key, const JKArgs& a, cudaStream_t s, bool fp32, int variant) {
  switch (key) {
    case class_key(0, 0, 0, 0): launch_jk<0, 0, 0, 0>(a, s, fp32, variant); return true;
    case class_key(1, 0, 0, 0): launch_jk<1, 0, 0, 0>(a, s, fp32, variant); return true;
    case class_key(1, 1, 0, 0): launch_jk<1, 1, 0, 0>(a, s, fp32, variant); return true;
    case class_key(2, 0, 0, 0): launch_jk<2, 0, 0, 0>(a, s, fp32, variant); return true;
    default: return false;
  }
}

}  // namespace tf
