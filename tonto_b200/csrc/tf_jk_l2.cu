// tf_jk_l2.cu — thread kernels of the larger classes, for lists long enough (dispatch_jk) (tf_thread.cuh).
#include "tf_thread.cuh"

namespace tf {

bool launch_jk_l2(int key, const JKArgs& a, cudaStream_t s, bool fp32, int variant) {
  switch (key) {
    case class_key(3, 0, 2, 0): launch_jk_f64<3, 0, 2, 0>(a, s, fp32, variant); return true;
    case class_key(3, 0, 3, 0): launch_jk_f64<3, 0, 3, 0>(a, s, fp32, variant); return true;
    case class_key(3, 2, 1, 0): launch_jk_f64<3, 2, 1, 0>(a, s, fp32, variant); return true;
    case class_key(3, 3, 1, 0): launch_jk_f64<3, 3, 1, 0>(a, s, fp32, variant); return true;
    default: return false;
  }
}

}  // namespace tf
