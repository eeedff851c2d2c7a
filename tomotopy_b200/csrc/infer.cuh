// infer.cuh -- inference of unseen documents against a frozen model:
// tomotopy's LDAModel::_infer<together = false> (LDAModel.hpp:920-953).
//
// Each document gets a private copy of the model with its own tokens added,
// z0 ~ Discrete(alpha), then sequential Gibbs sweeps.  Only the document's
// cells differ from the frozen model, so one warp keeps them on chip:
//   A_k = (float)n_dk[k] + alpha_k
//   R_k = 1 / ((float)(n_k[k] + n_dk[k]) + V*eta)
//   B_k = (float)(n_kw[k,v] + own[k]) + eta   (own: the document's other tokens of word v)
//   weight A_k * (B_k * R_k), drawn with the blocked two-pass draw of the training sweep.
// Documents are sorted by word id (prepareDoc, LDAModel.hpp:716-722), so the
// tokens of one word form a run and `own` is that run's topic histogram.
//
// The kernel works on "slots" and is resumable: one launch advances each
// listed slot through sweeps [it_begin, it_end); z and n_dk persist in device
// memory between launches.  Draws use the absolute (token, sweep) counter, so
// a document's result does not depend on how its sweeps are split across
// launches or on which other documents share them.
#pragma once
#include <algorithm>
#include <cmath>
#include <cstring>
#include "common.cuh"
#include "philox.cuh"

namespace tmtk {

struct InferArgs {
    // frozen model
    const int32_t* nkw;          // K x V column-major
    const int32_t* nk;
    const float* alpha;
    const float* acum;           // sequential float cumsum of alpha
    uint32_t K, V;
    float eta, veta, asum_f;
    double veta_d, asum_d, lg_asum, lg_eta;
    uint64_t key;                // seed ^ 'INFR'
    // tokens, addressed by the slots
    const uint32_t* words;       // sorted within each document
    uint16_t* z;
    // slots
    const uint64_t* tok_begin;   // first token of each slot; with tok_len == NULL, tok_begin[s+1] ends slot s
    const uint32_t* tok_len;
    const uint64_t* keys;        // per-slot draw key; NULL: 0
    const uint32_t* it_begin;    // per-slot sweep range of this launch; NULL: the uniform values below
    const uint32_t* it_end;
    const uint32_t* it_total;
    uint32_t u_begin, u_end, u_total;
    int32_t* ndk;                // slot x K counts kept between launches; NULL when every slot finishes here
    float* theta;                // slot x K, written when a slot finishes (may be NULL)
    double* ll;                  // slot, written when a slot finishes (may be NULL)
    const uint32_t* work;        // slots advanced by this launch; NULL: 0 .. n_work-1
    uint32_t n_work;
    uint32_t* counter;           // zeroed before the launch
    // weighted counts (TermWeight IDF / PMI): nkw, nk and ndk hold floats;
    // wt[token] is the token's weight, the same for every token of one word
    // within a document (IDF: the word's weight; PMI: a function of the word's
    // count in the document)
    const float* wt;
    // word priors (etaByTopicWord): pidx[v] >= 0 names row pidx[v] of pval
    // (K floats); esum[k] replaces V*eta; z0 draws from pcum (the rows'
    // cumulative sums) or ecum (a column of eta).  pidx == NULL: no priors.
    const int32_t* pidx;
    const float* pval;
    const float* esum;
    const float* pcum;
    const float* ecum;
    // no n_k or n_kw with a document's tokens added is larger; infinity if one may be
    // negative or not a number (count_bound)
    double count_max;
};

// The bound on counts of which k_max_count found `bits` the largest.
inline double count_bound(uint32_t bits, bool weighted)
{
    if (!weighted) return bits > 0x7FFFFFFFu ? INFINITY : (double)bits;
    if (bits > 0x7F800000u) return INFINITY;
    float f;
    std::memcpy(&f, &bits, sizeof(f));
    return (double)f;
}

constexpr double kMaxTokenWeight = 65536.0;      // what the callers accept

constexpr uint32_t kInferRegMaxK = 1024;     // k_infer_reg; above it k_infer_slots
constexpr int kInferRegWarps = 4;            // its warps (documents) per block: one per SM sub-partition

// warps per block so that 16 * KP bytes of state per warp fit in 200 KB; 0: too large
inline uint32_t infer_warps(uint32_t K)
{
    const uint32_t per_warp = 16 * round4(K);
    return std::min(8u, (200u * 1024u) / per_warp);
}

// the largest of n counts, or of non-negative floats by their bits; negative ones (and
// NaN) as larger than all others (out must be 0 before)
static __global__ void k_max_count(const int32_t* __restrict__ c, uint64_t n, uint32_t* __restrict__ out)
{
    uint32_t m = 0;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        m = max(m, (uint32_t)c[i]);
    m = __reduce_max_sync(FULL, m);
    if ((threadIdx.x & 31) == 0 && m) atomicMax(out, m);
}

// One launch for this K (the counter must be zeroed first); a.wt != NULL: weighted
// counts.  The kernels are in modules of their own by K: the driver loads a
// module whole when its first kernel is launched.  With the training kernels in one module they
// made a process's first upload 49 ms; now 16 (build.py), and the first inference 3 to 4.
void launch_infer(const InferArgs& a, int num_sms, cudaStream_t st);
void launch_infer_k256(const InferArgs& a, int num_sms, cudaStream_t st);     // K <= 256
void launch_infer_k512(const InferArgs& a, int num_sms, cudaStream_t st);     // 257..512
void launch_infer_k1024(const InferArgs& a, int num_sms, cudaStream_t st);    // 513..1024

} // namespace tmtk
