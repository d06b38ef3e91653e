// tf_jk_d.cu — thread kernels of the heavier classes up to d shells (tf_thread.cuh).
#include "tf_thread.cuh"

namespace tf {

bool launch_jk_d(int key, const JKArgs& a, cudaStream_t s, bool fp32, int variant) {
  switch (key) {
    case class_key(2, 0, 1, 1): launch_jk<2, 0, 1, 1>(a, s, fp32, variant); return true;
    case class_key(2, 0, 2, 0): launch_jk<2, 0, 2, 0>(a, s, fp32, variant); return true;
    case class_key(2, 1, 0, 0): launch_jk<2, 1, 0, 0>(a, s, fp32, variant); return true;
    case class_key(2, 1, 1, 0): launch_jk<2, 1, 1, 0>(a, s, fp32, variant); return true;
    case class_key(2, 2, 0, 0): launch_jk<2, 2, 0, 0>(a, s, fp32, variant); return true;
    default: return false;
  }
}

}  // namespace tf
