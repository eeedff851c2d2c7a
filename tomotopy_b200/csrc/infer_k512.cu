// infer_k512.cu -- k_infer_reg for K in 257..512 (infer.cuh says why the kernels are apart).
#include "infer_reg.cuh"

namespace tmtk {

template <bool WT>
static void launch(const InferArgs& a, int num_sms, cudaStream_t st)
{
    if (a.K <= 384) launch_infer_reg_g<3, 5, WT>(a, num_sms, st);
    else launch_infer_reg_g<4, 5, WT>(a, num_sms, st);
}

void launch_infer_k512(const InferArgs& a, int num_sms, cudaStream_t st)
{
    if (a.wt) launch<true>(a, num_sms, st);
    else launch<false>(a, num_sms, st);
}

} // namespace tmtk
