// infer_doc.cuh -- what the inference kernels share.
#pragma once
#include <type_traits>
#include "infer.cuh"

namespace tmtk {

// A finished document's theta and FP64 ll over the cells it touched.  dlen: its
// length (weight sum); own: K zeroed ints, zeroed again on return; count(k): its n_dk.
template <bool WT, class F>
__device__ __forceinline__ void finish_doc(const InferArgs& a, uint32_t sl, uint64_t b, uint32_t L, float dlen, int lane,
                                           int* own, F count)
{
    using CT = typename std::conditional<WT, float, int>::type;
    const CT* nkw = reinterpret_cast<const CT*>(a.nkw);
    const CT* nkv = reinterpret_cast<const CT*>(a.nk);
    const int K = (int)a.K;
    double acc = 0;
    const float denom = __fadd_rn(dlen, a.asum_f);
    for (int k = lane; k < K; k += 32) {
        const CT n = count(k);
        if (a.theta) a.theta[(uint64_t)sl * K + k] = __fdiv_rn(__fadd_rn((float)n, __ldg(a.alpha + k)), denom);
        if (n != CT(0)) {
            const double gk = (double)__ldg(nkv + k);
            const double es = a.esum ? (double)__ldg(a.esum + k) : a.veta_d;
            acc += lgamma(gk + es) - lgamma(gk + (double)n + es);
            const double al = (double)__ldg(a.alpha + k);
            acc += lgamma((double)n + al) - lgamma(al);
        }
    }
    uint32_t rb = 0;
    while (rb < L) {            // word cells: per run, each distinct topic once
        const uint32_t v = a.words[b + rb];
        uint32_t re = rb + 1;
        for (;;) {
            const uint32_t j = re + lane;
            const bool diff = j >= L || a.words[b + j] != v;
            const unsigned mm = __ballot_sync(FULL, diff);
            if (mm) { re += __ffs(mm) - 1; break; }
            re += 32;
        }
        if (v < a.V) {
            for (uint32_t j = rb + lane; j < re; j += 32) atomicAdd(&own[a.z[b + j]], 1);
            __syncwarp();
            const float wr = WT ? a.wt[b + rb] : 1.f;    // the run's weight
            const float* pe = nullptr;
            if (a.pidx) {
                const int p = a.pidx[v];
                if (p >= 0) pe = a.pval + (uint64_t)p * K;
            }
            for (uint32_t j = rb + lane; j < re; j += 32) {
                const int k = a.z[b + j];
                const int c = atomicExch(&own[k], 0);
                if (c) {
                    const CT gk = __ldg(nkw + (uint64_t)v * K + k);
                    const double ek = pe ? (double)pe[k] : (double)a.eta;
                    double after;
                    if constexpr (WT) after = lgamma(((double)gk + (double)__fmul_rn((float)c, wr)) + ek);
                    else after = lgamma((double)(gk + c) + ek);
                    acc += after - (gk != CT(0) ? lgamma((double)gk + ek) : (pe ? lgamma(ek) : a.lg_eta));
                }
            }
            __syncwarp();
        }
        rb = re;
    }
    acc = warp_sum(acc);
    if (lane == 0 && a.ll) a.ll[sl] = acc - (lgamma((double)dlen + a.asum_d) - a.lg_asum);
    __syncwarp();
}

} // namespace tmtk
