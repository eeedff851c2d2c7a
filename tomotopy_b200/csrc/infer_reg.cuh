// infer_reg.cuh -- inference of unseen documents for K <= kInferRegMaxK, included by
// infer_k256.cu, infer_k512.cu and infer_k1024.cu.  k_infer_slots (infer.cu) is the
// kernel of larger K; infer.cuh states the computation.  Both give the same
// results, bit for bit.
//
// What bounds it: a document is one warp's chain of draws (its tokens times its
// sweeps), so a call lasts as long as its longest documents and the figure that
// counts is cycles per draw: ~700 at K = 100 (2,300 before), ~1,800 at K = 1000
// (3,900 before), most of it the latency of dependent shuffles and shared-memory
// accesses.  Lane l owns topics 128 j + 4 l + i (j < CH); A_k, R_k and the counts
// sit in shared memory, padded with zeros to 128 CH.  A draw's critical path is the reads
// of A and R, one fma chain of 4 CH steps, the lane scan's shuffles, the total's
// broadcast, the choice of a topic and the update of its entry.  Up to CH = 4
// every lane forms the prefix sums of its own topics while the scan's shuffles are
// in flight, so the lane that is hit knows its topic already; above, the hit lane
// hands its weights to the warp for a second scan (32 prefix sums a lane would
// cost more than they save).  The next token's removal is formed beside the scan,
// and (integer counts, CH <= 4) so are A and R of one token more for the topic that
// gained one last, so that an addition only copies its entry.  The next token's
// column of the frozen n_kw is loaded during the current draw.
// One document of 250 tokens, K = 100, 50 sweeps: 14.4 -> 4.8 ms; 4,096 documents
// 312 -> 137 ms; 1,024 documents at K = 1000 146 -> 69 ms.

#pragma once
#include <algorithm>
#include "infer_doc.cuh"

namespace tmtk {

// resident blocks per SM (registers a thread may use), as many as leave the draws
// (nearly) without spills and as the arrays' shared memory admits
template <int CH, int MODE>
struct InferRegBlocks {
    static constexpr int value = CH <= 1 ? 5 : CH <= 2 ? 6 : CH <= 4 ? 4 : CH <= 5 ? (MODE == 2 ? 3 : 4)
                                 : CH <= 7 ? 3 : 2;
};

//   CH: blocks of four topics per lane (K <= 128 CH); STEPS: steps of the lane scan,
//       the lanes that hold topics being the first 2^STEPS at most
//   WT: weighted counts (TermWeight IDF / PMI)
//   MODE 0: K a multiple of 4 and the launch's fast conditions (launch_infer_reg_g);
//        1: the fast conditions, columns loaded by the element;
//        2: any (word priors, counts of 2^23 and more, extreme V eta)
template <int CH, int STEPS, bool WT, int MODE>
__global__ void __launch_bounds__(kInferRegWarps * 32, InferRegBlocks<CH, MODE>::value)
k_infer_reg(InferArgs a)
{
    using CT = typename std::conditional<WT, float, int>::type;
    using G4 = typename std::conditional<WT, float4, int4>::type;
    constexpr int T = 4 * CH;
    constexpr int KW = 128 * CH;
    constexpr bool GEN = MODE == 2;
    constexpr bool kWide = CH > 4;
    // integer counts up to CH = 4: A and R of one token more are kept for every topic
    constexpr bool kPlus = !WT && !kWide;
    constexpr int kArrays = kPlus ? 6 : 4;
    extern __shared__ __align__(16) float s_dyn[];
    const int K = (int)a.K;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // per block and topic: {n_k (int bits, or float), alpha, eta sum, -}
    float4* s_st = reinterpret_cast<float4*>(s_dyn);
    // per warp: A, R, counts, the current run's other tokens per topic and, with
    // kPlus, A and R of one token more -- kArrays arrays of KW words, one address with offsets
    float* s_A = s_dyn + 4 * KW + warp * kArrays * KW;
    float* s_R = s_A + KW;
    CT* s_n = reinterpret_cast<CT*>(s_A + 2 * KW);
    int* s_own = reinterpret_cast<int*>(s_A + 3 * KW);
    float* s_Ap = s_A + (kPlus ? 4 : 0) * KW;
    float* s_Rp = s_A + (kPlus ? 5 : 0) * KW;
    // two batches of 32 tokens: {topic | kind << 16 | run << 18, uniform, weight,
    // word}; a draw leaves its topic in the first.  run: the tokens of its word from
    // it on, 0 when they go on past the batch.  kind: what follows the token -- 1: the next
    // one is of the same word (a run goes on); else 3: the next one starts a run;
    // else 2: a run ends here; else 0
    __shared__ __align__(16) float4 s_tok_all[kInferRegWarps][64];
    __shared__ __align__(16) float s_xs_all[kInferRegWarps][kWide ? T : 4];
    float4* s_tok = s_tok_all[warp];
    float* s_xs = s_xs_all[warp];
    const CT* nkw = reinterpret_cast<const CT*>(a.nkw);
    const CT* nkv = reinterpret_cast<const CT*>(a.nk);
    CT* ndk_s = reinterpret_cast<CT*>(a.ndk);
    const unsigned lt = (1u << lane) - 1u;
    const int left = K - 4 * lane;
    const int nh = left <= 0 ? 0 : 4 * (left >> 7) + min(left & 127, 4);     // this lane's topics
    const int last_lane = ((K - 1) >> 2) & 31;                               // the lane of topic K - 1
    const float eta = a.eta;
    auto topic_of = [&](int t) { return 128 * (t >> 2) + 4 * lane + (t & 3); };
    // place of topic k in the per-warp arrays: with CH > 4 block j is turned by j
    // lanes, so that one lane's topics sit in different banks
    auto at = [&](int k) { return kWide ? (k & ~127) | ((k + 4 * (k >> 7)) & 127) : k; };
    const int my4 = 4 * lane;
    const bool vec = MODE == 0 || (GEN && kWide && (K & 3) == 0);    // 16-byte column loads
    auto blk = [&](int jj) { return 128 * jj + (kWide ? ((my4 + 4 * jj) & 127) : my4); };
    // the denominators lie in recip_mid's range in the fast modes (launch_infer_reg_g):
    // V eta in [1e-30, 1e30] and counts below 1e31 above it
    auto recip = [](float x) -> float { return GEN ? __frcp_rn(x) : recip_mid(x); };
    // (float)n of a count: in the fast modes below 2^23, where 2^23 + n is exact in
    // the float whose mantissa holds n (the conversion unit does one warp in 8 cycles)
    auto to_f = [](CT n) -> float {
        if constexpr (WT || GEN) return (float)n;
        else return __fsub_rn(__int_as_float(n | 0x4B000000), 8388608.f);
    };
    // A and R of a topic with count n (e: its entry)
    auto eval = [&](const float4& e, CT n, float& A, float& R) {
        if constexpr (WT) {
            A = __fadd_rn(n, e.y);
            R = recip(__fadd_rn(__fadd_rn(e.x, n), e.z));
        } else {
            A = __fadd_rn(to_f(n), e.y);
            R = recip(__fadd_rn(to_f(__float_as_int(e.x) + n), e.z));
        }
    };
    auto less = [&](CT n, float wt) -> CT {     // a token removed
        if constexpr (WT) return fmaxf(__fsub_rn(n, wt), 0.f);
        else return n - 1;
    };
    auto more = [&](CT n, float wt) -> CT {
        if constexpr (WT) return __fadd_rn(n, wt);
        else return n + 1;
    };
    float lm[5];                             // 1 in the lanes at or above 2^i, else 0
#pragma unroll
    for (int i = 0; i < 5; ++i) lm[i] = lane >= (1 << i) ? 1.f : 0.f;
    // a scan step: for finite sums fma(y, 1, x) rounds as x + y and fma(y, 0, x) is x
    auto scan_step = [&](float x, int i) {
        if constexpr (GEN) return hs_up(x, 1 << i);
        else return __fmaf_rn(__shfl_up_sync(FULL, x, 1 << i), lm[i], x);
    };
    for (int k = threadIdx.x; k < KW; k += blockDim.x) {
        float4 e = make_float4(0.f, 0.f, 1.f, 0.f);
        if (k < K) {
            const CT nk = __ldg(nkv + k);
            if constexpr (WT) e.x = nk;
            else e.x = __int_as_float(nk);
            e.y = __ldg(a.alpha + k);
            e.z = a.esum ? __ldg(a.esum + k) : a.veta;
        }
        s_st[k] = e;
    }
    for (int k = lane; k < KW; k += 32) {
        s_A[k] = s_R[k] = 0.f;
        s_n[k] = CT(0);
        s_own[k] = 0;
    }
    for (int i = lane; i < 64; i += 32) s_tok[i] = make_float4(0.f, 0.f, 0.f, 0.f);   // (read ahead: any word)
    __syncthreads();

    // predicated stores (a store under `if` is a branch on every draw's chain):
    // count, A and R of a topic ...
    auto put = [](bool p, float* at_a, CT n, float A, float R) {
        float nb;
        if constexpr (WT) nb = n;
        else nb = __int_as_float(n);
        asm volatile("{\n .reg .pred p;\n setp.ne.s32 p, %0, 0;\n @p st.shared.f32 [%1], %3;\n"
                     " @p st.shared.f32 [%1+%5], %4;\n @p st.shared.f32 [%1+%6], %2;\n}"
                     :: "r"((int)p), "r"((uint32_t)__cvta_generic_to_shared(at_a)), "f"(nb), "f"(A), "f"(R),
                        "n"(4 * KW), "n"(8 * KW) : "memory");
    };
    // ... and its A and R of one token more
    auto put_plus = [](bool p, float* at_a, float A, float R) {
        asm volatile("{\n .reg .pred p;\n setp.ne.s32 p, %0, 0;\n @p st.shared.f32 [%1+%4], %2;\n"
                     " @p st.shared.f32 [%1+%5], %3;\n}"
                     :: "r"((int)p), "r"((uint32_t)__cvta_generic_to_shared(at_a)), "f"(A), "f"(R),
                        "n"(16 * KW), "n"(20 * KW) : "memory");
    };
    auto put_i = [](bool p, void* at, int v) {
        asm volatile("{\n .reg .pred p;\n setp.ne.s32 p, %0, 0;\n @p st.shared.s32 [%1], %2;\n}"
                     :: "r"((int)p), "r"((uint32_t)__cvta_generic_to_shared(at)), "r"(v) : "memory");
    };
    auto add_own = [](bool p, float* at_a, int v) {
        asm volatile("{\n .reg .pred p;\n setp.ne.s32 p, %0, 0;\n @p red.shared.add.s32 [%1+%3], %2;\n}"
                     :: "r"((int)p), "r"((uint32_t)__cvta_generic_to_shared(at_a)), "r"(v), "n"(12 * KW) : "memory");
    };

    for (;;) {
        uint32_t q = 0;
        if (lane == 0) q = atomicAdd(a.counter, 1u);
        q = __shfl_sync(FULL, q, 0);
        if (q >= a.n_work) break;
        const uint32_t sl = a.work ? a.work[q] : q;
        const uint64_t b = a.tok_begin[sl];
        const uint32_t L = a.tok_len ? a.tok_len[sl] : (uint32_t)(a.tok_begin[sl + 1] - b);
        const uint64_t dk = a.keys ? a.keys[sl] : 0;
        const uint32_t klo = (uint32_t)dk, khi = (uint32_t)(dk >> 32);
        const uint32_t it0 = a.it_begin ? a.it_begin[sl] : a.u_begin;
        const uint32_t it1 = a.it_end ? a.it_end[sl] : a.u_end;
        const uint32_t itT = a.it_total ? a.it_total[sl] : a.u_total;
        const uint32_t* words = a.words + b;
        uint16_t* z = a.z + b;
        const float* wts = WT ? a.wt + b : nullptr;
        int nvalid = 0;
        float wsum = 0.f;                    // WT: the document's weight sum, in token order
        __syncwarp();
        if (it0 == 0) {
            // z0 ~ Discrete(alpha), added to the document's counts
            for (int k = lane; k < KW; k += 32) s_n[k] = CT(0);
            __syncwarp();
            for (uint32_t j = lane; j < L; j += 32) {
                const uint32_t w = words[j];
                uint16_t zz = 0xFFFF;
                if (w < a.V) {
                    const float u = tmt::u01(tmt::philox_u32(j, 0xFFFFFFFFu, klo, khi, a.key));
                    const float* cum = a.acum;
                    if (GEN && a.pidx) {
                        const int p = a.pidx[w];
                        cum = p >= 0 ? a.pcum + (uint64_t)p * K : a.ecum;
                    }
                    const float r = __fmul_rn(u, cum[K - 1]);
                    uint32_t lo = 0, hi = K - 1;
                    while (lo < hi) {
                        const uint32_t mid = (lo + hi) >> 1;
                        if (r < cum[mid]) hi = mid; else lo = mid + 1;
                    }
                    zz = (uint16_t)lo;
                    if constexpr (!WT) atomicAdd(s_n + at((int)lo), 1);
                    ++nvalid;
                }
                z[j] = zz;
            }
            if constexpr (WT) {
                __syncwarp();
                if (lane == 0)
                    for (uint32_t j = 0; j < L; ++j)
                        if (words[j] < a.V) {
                            const float wj = wts[j];
                            CT& n = s_n[at(z[j])];
                            n = __fadd_rn(n, wj);
                            wsum = __fadd_rn(wsum, wj);
                        }
            }
        } else {
            for (int k = lane; k < K; k += 32) s_n[at(k)] = ndk_s[(uint64_t)sl * K + k];
            for (uint32_t j = lane; j < L; j += 32) nvalid += words[j] < a.V;
            if (WT && lane == 0)
                for (uint32_t j = 0; j < L; ++j)
                    if (words[j] < a.V) wsum = __fadd_rn(wsum, wts[j]);
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) nvalid += __shfl_xor_sync(FULL, nvalid, o);
        if (WT) wsum = __shfl_sync(FULL, wsum, 0);
        __syncwarp();
        const uint32_t Lv = (uint32_t)nvalid;    // words are sorted: the sampled tokens come first
        for (int k = lane; k < K; k += 32) {
            float A, R;
            eval(s_st[k], s_n[at(k)], A, R);
            s_A[at(k)] = A;
            s_R[at(k)] = R;
            if constexpr (kPlus) {
                eval(s_st[k], more(s_n[k], 0.f), A, R);
                s_Ap[k] = A;
                s_Rp[k] = R;
            }
        }

        // a batch's tokens, one per lane, loaded a batch ahead of their staging
        uint32_t w1 = 0, z1 = 0;
        float wt1 = 0.f;
        auto fetch = [&](uint32_t base) {
            const uint32_t j = base + lane;
            if (j < Lv) {
                w1 = words[j];
                z1 = z[j];
                if (WT) wt1 = wts[j];
                const bool same = j + 1 < Lv && words[j + 1] == w1;
                const bool starts = j + 2 < Lv && words[j + 1] == words[j + 2];
                const bool ends = j > 0 && words[j - 1] == w1;
                z1 |= (same ? 1u : starts ? 3u : ends ? 2u : 0u) << 16;
            }
            const unsigned stops = __ballot_sync(FULL, j >= Lv || ((z1 >> 16) & 3) != 1) >> lane;
            if (j < Lv) z1 |= (uint32_t)__ffs(stops) << 18;
        };
        auto stage = [&](uint32_t base, uint32_t it) {
            const uint32_t j = base + lane;
            const float u = tmt::u01(tmt::philox_u32(j, it, klo, khi, a.key));
            if (j < Lv) s_tok[j & 63] = make_float4(__int_as_float((int)z1), u, wt1, __int_as_float((int)w1));
        };
        auto topic = [](const float4& t) { return __float_as_int(t.x) & 0xFFFF; };
        auto kind_of = [](const float4& t) { return (__float_as_int(t.x) >> 16) & 3; };
        uint32_t staged = 0;                 // tokens staged so far
        auto clear_own = [&]() {
#pragma unroll
            for (int jj = 0; jj < CH; ++jj) *reinterpret_cast<int4*>(s_own + blk(jj)) = make_int4(0, 0, 0, 0);
            __syncwarp();
        };
        // the run that starts at token j: its other tokens' topics into s_own (zero before)
        auto start_run = [&](uint32_t j, const float4& t) {
            if (const int run = __float_as_int(t.x) >> 18) {
                const int zi = topic(s_tok[(j + 1 + lane) & 63]);
                add_own(lane < run - 1, s_A + at(min(zi, K - 1)), 1);
                __syncwarp();
                return;
            }
            for (uint32_t i0 = j;; i0 += 32) {
                const uint32_t i = i0 + lane;
                bool in = false;
                int zi = 0;
                if (i < staged) {
                    const float4 e = s_tok[i & 63];
                    in = __float_as_int(e.w) == __float_as_int(t.w);
                    zi = topic(e);
                } else if (i < Lv) {
                    in = words[i] == (uint32_t)__float_as_int(t.w);
                    zi = z[i];
                }
                if (in && i > j) atomicAdd(&s_own[at(zi)], 1);
                if (__ballot_sync(FULL, !in)) break;
            }
            __syncwarp();
        };
        // (a lane's blocks past K are never loaded and stay 0)
        auto load_col = [&](float word, G4 (&g)[CH]) {
            const CT* col = nkw + (uint64_t)(uint32_t)__float_as_int(word) * (uint32_t)K + my4;
            if (vec) {
#pragma unroll
                for (int jj = 0; jj < CH; ++jj)
                    if (128 * jj + my4 < K) g[jj] = __ldg(reinterpret_cast<const G4*>(col + 128 * jj));
            } else {
#pragma unroll
                for (int jj = 0; jj < CH; ++jj) {
                    const int k0 = 128 * jj + my4;
                    if (k0 < K) g[jj].x = __ldg(col + 128 * jj);
                    if (k0 + 1 < K) g[jj].y = __ldg(col + 128 * jj + 1);
                    if (k0 + 2 < K) g[jj].z = __ldg(col + 128 * jj + 2);
                    if (k0 + 3 < K) g[jj].w = __ldg(col + 128 * jj + 3);
                }
            }
        };

        int kp = -1;                         // kPlus: the topic this lane last added to, its plus entry not yet renewed
        for (uint32_t it = it0; it < it1 && Lv; ++it) {
            fetch(0);
            stage(0, it);
            staged = min(32u, Lv);
            fetch(32);
            __syncwarp();
            float4 tok = s_tok[0];
            G4 ga[CH], gb[CH];               // the columns of even and odd tokens
#pragma unroll
            for (int jj = 0; jj < CH; ++jj) {
                ga[jj].x = ga[jj].y = ga[jj].z = ga[jj].w = CT(0);
                gb[jj] = ga[jj];
            }
            load_col(tok.w, ga);
            // the prior column of a word, NULL if it has none
            auto prior_of = [&](float word) -> const float* {
                if (!GEN || !a.pidx) return nullptr;
                const int p = __ldg(a.pidx + (uint32_t)__float_as_int(word));
                return p >= 0 ? a.pval + (uint64_t)p * K : nullptr;
            };
            const float* pe_next = GEN && kWide ? prior_of(tok.w) : nullptr;     // (of the coming token)
            bool in_run = kind_of(tok) == 1;
            {
                // the first token leaves its topic
                const int zo = topic(tok);
                const CT n = less(s_n[at(zo)], tok.z);
                float A, R;
                eval(s_st[zo], n, A, R);
                const float A0 = s_A[at(zo)], R0 = s_R[at(zo)];
                __syncwarp();
                put(lane == 0, s_A + at(zo), n, A, R);
                if constexpr (kPlus) put_plus(lane == 0, s_A + zo, A0, R0);
                __syncwarp();
                if (in_run) start_run(0, tok);
            }
            for (uint32_t base = 0; base < Lv; base += 32) {
              if (staged < Lv) {
                  // the next batch's tokens into the other half of the ring; the one
                  // after it on its way
                  stage(staged, it);
                  staged = min(staged + 32, Lv);
                  fetch(staged);
                  __syncwarp();
              }
              const uint32_t end = min(base + 32, Lv);
              // one token: its column in g, the next one's into gn
              auto step = [&](uint32_t jt, G4 (&g)[CH], G4 (&gn)[CH]) {
                const float4 nt = s_tok[(jt + 1) & 63];
                load_col(nt.w, gn);
                const bool more_tokens = jt + 1 < Lv;
                const int zn = min(topic(nt), K - 1);    // the topic the next token leaves (if there is one)
                const int kind = kind_of(tok);
                const float u = tok.y, wt = tok.z;
                // The word's prior column, if any.  With CH > 4 it is looked up a token ahead
                // and loaded at once (6,000 documents of 80 tokens, 60 sweeps, priors: K = 1000
                // 57 -> 50 ms); below, the lookup costs more than its latency (K = 100, 64
                // documents: 10.1 against 11.3 ms).
                const float* pe = nullptr;
                if (GEN && !kWide) pe = prior_of(tok.w);
                float w[T];                          // CH > 4: the etas; then, in pass 1, the weights
                if constexpr (GEN && kWide) {
                    pe = pe_next;
                    pe_next = prior_of(nt.w);
#pragma unroll
                    for (int t = 0; t < T; ++t) w[t] = eta;
                    if (pe && vec) {
#pragma unroll
                        for (int jj = 0; jj < CH; ++jj)
                            if (128 * jj + my4 < K) {
                                const float4 e = __ldg(reinterpret_cast<const float4*>(pe + 128 * jj + my4));
                                w[4 * jj] = e.x;
                                w[4 * jj + 1] = e.y;
                                w[4 * jj + 2] = e.z;
                                w[4 * jj + 3] = e.w;
                            }
                    } else if (pe) {
#pragma unroll
                        for (int t = 0; t < T; ++t)
                            if (topic_of(t) < K) w[t] = __ldg(pe + topic_of(t));
                    }
                }
                auto ek = [&](int t) -> float {
                    if constexpr (GEN && kWide) return w[t];
                    else return GEN && pe && topic_of(t) < K ? __ldg(pe + topic_of(t)) : eta;
                };
                // the run's other tokens of the word (zero outside a run)
                if (CH <= 2 || in_run)
#pragma unroll
                for (int jj = 0; jj < CH; ++jj) {
                    const int4 o = *reinterpret_cast<const int4*>(s_own + blk(jj));
                    if constexpr (WT) {
                        g[jj].x = __fadd_rn(g[jj].x, __fmul_rn((float)o.x, wt));
                        g[jj].y = __fadd_rn(g[jj].y, __fmul_rn((float)o.y, wt));
                        g[jj].z = __fadd_rn(g[jj].z, __fmul_rn((float)o.z, wt));
                        g[jj].w = __fadd_rn(g[jj].w, __fmul_rn((float)o.w, wt));
                    } else {
                        g[jj].x += o.x;
                        g[jj].y += o.y;
                        g[jj].z += o.z;
                        g[jj].w += o.w;
                    }
                }
                // pass 1: fma chain over this lane's topics; w: A_k for CH <= 4
                // turned into the weights, above B_k R_k
                float s = 0.f;
#pragma unroll
                for (int jj = 0; jj < CH; ++jj) {
                    const float4 A4 = *reinterpret_cast<const float4*>(s_A + blk(jj));
                    const float4 R4 = *reinterpret_cast<const float4*>(s_R + blk(jj));
                    w[4 * jj] = __fmul_rn(__fadd_rn(to_f(g[jj].x), ek(4 * jj)), R4.x);
                    w[4 * jj + 1] = __fmul_rn(__fadd_rn(to_f(g[jj].y), ek(4 * jj + 1)), R4.y);
                    w[4 * jj + 2] = __fmul_rn(__fadd_rn(to_f(g[jj].z), ek(4 * jj + 2)), R4.z);
                    w[4 * jj + 3] = __fmul_rn(__fadd_rn(to_f(g[jj].w), ek(4 * jj + 3)), R4.w);
                    s = __fmaf_rn(A4.x, w[4 * jj], s);
                    s = __fmaf_rn(A4.y, w[4 * jj + 1], s);
                    s = __fmaf_rn(A4.z, w[4 * jj + 2], s);
                    s = __fmaf_rn(A4.w, w[4 * jj + 3], s);
                    if constexpr (!kWide) {
                        w[4 * jj] = __fmul_rn(A4.x, w[4 * jj]);
                        w[4 * jj + 1] = __fmul_rn(A4.y, w[4 * jj + 1]);
                        w[4 * jj + 2] = __fmul_rn(A4.z, w[4 * jj + 2]);
                        w[4 * jj + 3] = __fmul_rn(A4.w, w[4 * jj + 3]);
                    }
                }
                float x = s;
#pragma unroll
                for (int i = 0; i < STEPS; ++i) x = scan_step(x, i);
                const float total = __shfl_sync(FULL, x, (1 << STEPS) - 1);
                const float E = GEN ? up1_or_0(x) : __fmul_rn(__shfl_up_sync(FULL, x, 1), lm[0]);
                // the next token's removal, should this draw leave its topic alone
                float Az = 0.f, Rz = 0.f, Az0 = 0.f, Rz0 = 0.f;
                CT nz = CT(0);
                if constexpr (!kWide) {
                    nz = less(s_n[zn], nt.z);
                    eval(s_st[zn], nz, Az, Rz);
                    Az0 = s_A[zn];
                    Rz0 = s_R[zn];
                }
                if constexpr (kPlus) {
                    // the topic added to last: its A and R of one token more
                    const int k = max(kp, 0);
                    float A1, R1;
                    eval(s_st[k], s_n[k] + 1, A1, R1);
                    put_plus(kp >= 0, s_A + k, A1, R1);
                }
                const float r = __fmul_rn(u, total);
                const bool in = nh > 0 && r < __fadd_rn(E, s);
                int knew = 0;                        // the new topic (in the lane that keeps it)
                bool keep;
                if constexpr (!kWide) {
                    // prefix sums of this lane's own weights (Hillis-Steele order)
#pragma unroll
                    for (int off = 1; off < T; off <<= 1) {
#pragma unroll
                        for (int t = T - 1; t >= off; --t) w[t] = __fadd_rn(w[t], w[t - off]);
                    }
                    int found = T - 1;
#pragma unroll
                    for (int t = T - 2; t >= 0; --t)
                        if (r < __fadd_rn(E, w[t])) found = t;
                    found = in ? min(found, nh - 1) : max(nh - 1, 0);
                    knew = topic_of(found);
                    __syncwarp();                    // (the plus entries are renewed)
                    // the topic this lane would draw with the token added -- and the next
                    // one removed, if it leaves the same topic
                    const bool same = more_tokens && knew == zn;
                    CT nx = more(s_n[knew], wt);
                    float Ax, Rx;
                    if constexpr (kPlus) {
                        Ax = s_Ap[knew];
                        Rx = s_Rp[knew];
                    } else {
                        if (same) nx = less(nx, nt.z);
                        eval(s_st[knew], nx, Ax, Rx);
                    }
                    // the first lane that r falls in; topic K - 1 when rounding left it
                    // at or above the total
                    unsigned m = __ballot_sync(FULL, in);
                    if (m == 0) m = 1u << last_lane;
                    keep = (m & (0u - m)) == lt + 1u;
                    __syncwarp();                    // every lane has read its entries
                    // (integer counts: an addition and a removal of one topic leave it as it was)
                    put(keep && !(kPlus && same), s_A + knew, nx, Ax, Rx);
                    put(keep && more_tokens && !same, s_A + zn, nz, Az, Rz);
                    if constexpr (kPlus) {
                        put_plus(keep && more_tokens && !same, s_A + zn, Az0, Rz0);
                        kp = keep && !same ? knew : -1;
                    }
                } else {
                    const unsigned m = __ballot_sync(FULL, in);
                    knew = K - 1;
                    if (m) {
                        // pass 2: position among lane h's topics
                        const int h = __ffs(m) - 1;
                        const float Eh = __shfl_sync(FULL, E, h);
                        if (lane == h) {
#pragma unroll
                            for (int jj = 0; jj < CH; ++jj)
                                *reinterpret_cast<float4*>(s_xs + 4 * jj) =
                                    make_float4(w[4 * jj], w[4 * jj + 1], w[4 * jj + 2], w[4 * jj + 3]);
                        }
                        const int mh = K - 4 * h;
                        const int nhh = 4 * (mh >> 7) + min(mh & 127, 4);
                        const int k = 128 * (lane >> 2) + 4 * h + (lane & 3);
                        __syncwarp();
                        float x2 = 0.f;
                        if (lane < nhh) x2 = __fmul_rn(s_A[at(k)], s_xs[lane]);
#pragma unroll
                        for (int i = 0; i < 5; ++i) x2 = scan_step(x2, i);
                        const unsigned mb = __ballot_sync(FULL, lane < nhh && r < __fadd_rn(Eh, x2));
                        const int found = mb ? __ffs(mb) - 1 : nhh - 1;
                        knew = 128 * (found >> 2) + 4 * h + (found & 3);
                    }
                    // lane 0 forms the addition, lane 1 the next token's removal
                    const bool both = more_tokens && knew == zn;
                    const int kx = lane == 1 && more_tokens ? zn : knew;
                    const CT n = s_n[at(kx)];
                    CT nx = lane == 1 ? less(n, nt.z) : more(n, wt);
                    if (both) nx = less(more(n, wt), nt.z);
                    float Ax, Rx;
                    eval(s_st[kx], nx, Ax, Rx);
                    keep = lane == 0;
                    __syncwarp();                    // every lane has read its entries
                    put(lane == 0 || (lane == 1 && more_tokens && !both), s_A + at(kx), nx, Ax, Rx);
                }
                put_i(keep, &s_tok[jt & 63].x, knew);
                add_own(keep && kind == 1, s_A + at(knew), 1);
                add_own(lane == 0 && kind == 1, s_A + at(zn), -1);
                if (kind >= 2) {
                    if (in_run) clear_own();
                    if (kind == 3) start_run(jt + 1, nt);
                }
                in_run = kind & 1;
                __syncwarp();
                tok = nt;
              };
#pragma unroll 1
              for (uint32_t jt = base; jt < end; jt += 2) {      // (base is even)
                  step(jt, ga, gb);
                  if (jt + 1 < end) step(jt + 1, gb, ga);
              }
              if (base + lane < end) z[base + lane] = (uint16_t)__float_as_int(s_tok[(base + lane) & 63].x);
              __syncwarp();
            }
        }
        if (it1 < itT) {            // keep the document's counts for the next launch
            for (int k = lane; k < K; k += 32) ndk_s[(uint64_t)sl * K + k] = s_n[at(k)];
            continue;
        }
        // finished: theta, FP64 ll over the touched cells
        finish_doc<WT>(a, sl, b, L, WT ? wsum : (float)nvalid, lane, s_own, [&](int k) -> CT { return s_n[at(k)]; });
    }
}

template <int CH, int STEPS, bool WT, int MODE>
inline void launch_infer_reg_t(const InferArgs& a, int num_sms, cudaStream_t st)
{
    auto kern = k_infer_reg<CH, STEPS, WT, MODE>;
    const uint32_t smem = (4 + kInferRegWarps * (!WT && CH <= 4 ? 6 : 4)) * 4 * 128 * CH;     // (k_infer_reg's s_dyn)
    CK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 0;
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kInferRegWarps * 32, smem));
    if (per_sm < 1) throw CudaError("infer kernel does not fit on an SM");
    const uint32_t grid = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>((uint64_t)per_sm * num_sms,
                                                                          (a.n_work + kInferRegWarps - 1) / kInferRegWarps));
    kern<<<grid, kInferRegWarps * 32, smem, st>>>(a);
    CK(cudaGetLastError());
}

template <int CH, int STEPS, bool WT>
inline void launch_infer_reg_g(const InferArgs& a, int num_sms, cudaStream_t st)
{
    // The fast modes' conditions: scalar eta, counts exact in to_f, denominators in
    // recip's range.  (Their general forms cost a draw at k = 100 about 50 of 450
    // cycles.)  Element loads where columns are not 16-byte aligned.
    // (No weight or sum of weights can overflow: A B R below 1e36 / K.  With V eta at
    // most 1e30 this also keeps weighted counts below 1e31, inside recip's range.)
    const double most = WT ? a.count_max : 8388608.0;
    const bool finite = (most + (double)a.asum_f) * (most + (double)a.eta) < 1e32 * (double)a.veta;
    const bool exact = WT || a.count_max < 8388608.0;
    if (a.pidx || !exact || !finite || !(a.veta >= 1e-30f && a.veta <= 1e30f))
        launch_infer_reg_t<CH, 5, WT, 2>(a, num_sms, st);
    else if (a.K & 3) launch_infer_reg_t<CH, STEPS, WT, 1>(a, num_sms, st);
    else launch_infer_reg_t<CH, STEPS, WT, 0>(a, num_sms, st);
}

} // namespace tmtk
