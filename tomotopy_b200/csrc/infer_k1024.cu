// infer_k1024.cu -- k_infer_reg for K in 513..1024 (infer.cuh says why the kernels are apart).
#include "infer_reg.cuh"

namespace tmtk {

template <bool WT>
static void launch(const InferArgs& a, int num_sms, cudaStream_t st)
{
    // (exact widths above 512 topics: shorter chains and smaller arrays, so more documents
    // an SM; 6,000 documents of 80 tokens, 60 sweeps at K = 520, one width for 513..1024
    // and now: 39.0 -> 29.5 ms, with word priors 54.1 -> 38)
    if (a.K <= 640) launch_infer_reg_g<5, 5, WT>(a, num_sms, st);
    else if (a.K <= 768) launch_infer_reg_g<6, 5, WT>(a, num_sms, st);
    else if (a.K <= 896) launch_infer_reg_g<7, 5, WT>(a, num_sms, st);
    else launch_infer_reg_g<8, 5, WT>(a, num_sms, st);
}

void launch_infer_k1024(const InferArgs& a, int num_sms, cudaStream_t st)
{
    if (a.wt) launch<true>(a, num_sms, st);
    else launch<false>(a, num_sms, st);
}

} // namespace tmtk
