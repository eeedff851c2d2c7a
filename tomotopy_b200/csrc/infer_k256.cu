// infer_k256.cu -- k_infer_reg for K <= 256 (infer.cuh says why the kernels are apart).
#include "infer_reg.cuh"

namespace tmtk {

template <bool WT>
static void launch(const InferArgs& a, int num_sms, cudaStream_t st)
{
    if (a.K <= 32) launch_infer_reg_g<1, 3, WT>(a, num_sms, st);
    else if (a.K <= 64) launch_infer_reg_g<1, 4, WT>(a, num_sms, st);
    else if (a.K <= 124) launch_infer_reg_g<1, 5, WT>(a, num_sms, st);     // (lane 31 without topics)
    else launch_infer_reg_g<2, 5, WT>(a, num_sms, st);
}

void launch_infer_k256(const InferArgs& a, int num_sms, cudaStream_t st)
{
    if (a.wt) launch<true>(a, num_sms, st);
    else launch<false>(a, num_sms, st);
}

} // namespace tmtk
