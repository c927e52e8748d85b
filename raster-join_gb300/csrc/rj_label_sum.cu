// rj_label_sum.cu -- the label pass with a summed aggregate (rj_label_core.cuh).
#include "rj_label_core.cuh"

namespace rj {

LabelKernel label_points_sum(int shape, int ni, int nf) { return label_kernel_cols<true>(shape, ni, nf); }

}  // namespace rj
