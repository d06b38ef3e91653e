// tf_jk_l.cu — thread kernels of the larger classes, for lists long enough (dispatch_jk) (tf_thread.cuh).
#include "tf_thread.cuh"

namespace tf {

bool launch_jk_l(int key, const JKArgs& a, cudaStream_t s, bool fp32, int variant) {
  switch (key) {
    case class_key(1, 1, 1, 1): launch_jk_f64<1, 1, 1, 1>(a, s, fp32, variant); return true;
    case class_key(2, 1, 2, 0): launch_jk_f64<2, 1, 2, 0>(a, s, fp32, variant); return true;
    case class_key(2, 2, 1, 0): launch_jk_f64<2, 2, 1, 0>(a, s, fp32, variant); return true;
    case class_key(3, 0, 1, 1): launch_jk_f64<3, 0, 1, 1>(a, s, fp32, variant); return true;
    case class_key(3, 1, 1, 0): launch_jk_f64<3, 1, 1, 0>(a, s, fp32, variant); return true;
    default: return false;
  }
}

}  // namespace tf
