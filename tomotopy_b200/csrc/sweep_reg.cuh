// sweep_reg.cuh -- the training sweep for K <= 512 (K <= kRegMaxK): the
// document's row in registers.  Included by engine.cu inside its namespace,
// after SweepArgs; k_sweep_doc there, the kernel of K > 1024, states the sampler
// (k_sweep_wide is the one between).  All compute the same draws, bit for bit.
//
// What bounds it: a document is a chain of draws, each token waiting for the
// one before, so a launch of few or long documents lasts (longest document) x
// (cycles per draw), and one of many short ones is bound by instructions.
// The layout serves the chain: lane l owns topics 128 j + 4 l + i (j < CH) and
// keeps their counts, alphas and weights in registers, so a draw's critical
// path is one fma chain of 4 CH steps, the five shuffles of the lane scan, the
// total's broadcast, one vote and the hit lane's own increment -- no shared
// memory and no second scan: every lane forms the prefix sums of its own
// topics while the scan's shuffles are in flight, and the lane that is hit
// already knows its topic.  What does not depend on the draw is done for 32
// tokens at a time, one per lane (words, assignments, uniforms, the own
// topic's weight, and the count deltas of the tokens that moved), a batch or
// two ahead of the draws; the words' table columns are loaded kRing - 1 tokens
// ahead.  (Products with a 0/1 vector in place of the own topic's selects, and split
// merges through per-warp buffers in place of shared-memory atomics, measured slower.)
// The sampling kernels of one sweep, k_sweep_doc and this kernel: K = 20, 1.5M tokens 1.33 ->
// 0.45 ms; K = 100, 27.5M tokens 8.5 -> 4.7 ms; IDF weights, K = 200, 8M tokens 12.6 -> 4.6 ms
// (2.5 of them the launch of the 10,000-token documents).

constexpr uint32_t kRegMaxK = 512;
constexpr uint64_t kRegFloatLen = 1ull << 24;    // counts below are exact as floats
constexpr uint64_t kRegMaxLen = 1ull << 31;      // positions are 32 bits; from here on k_sweep_doc
constexpr int kRegWarps = 4;         // warps per block without split documents: one per SM sub-partition

// resident blocks per SM (registers a thread may use): as many as leave the
// token loop without spills (6 blocks of 80 registers with CH = 1 spilled 40 bytes:
// K = 100, 27.5M tokens, 10 sweeps 59-61 against 55 ms with 5; split documents at
// 2 blocks of 8 warps spilled 40-140 with CH = 2 and 3: K = 333 26.9 against 25.4 ms)
template <int CH, bool SPLIT>
struct RegBlocks {
    static constexpr int value = SPLIT ? (CH <= 1 ? 2 : 1)
                                       : CH <= 1 ? 5 : CH <= 2 ? 4 : 3;
};

//   CH: blocks of four topics per lane (K <= 128 CH)
//   STEPS: steps of the lane scan, the lanes that hold topics being the first
//       2^STEPS at most (the skipped steps would add zeros)
//   WT: weighted counts (TermWeight IDF / PMI)
//   SPLIT: the launch's first n_long documents are sampled a block each in
//       kSweepWarps slices (see kSplitStep); integer counts
//   OPT: per-document masks or alphas may be set
//   BIG: documents of kRegFloatLen tokens and more: integer counts are held as integers
//       (a conversion per topic and draw; as floats they need none)
template <int CH, int STEPS, bool WT, bool SPLIT, bool OPT, bool BIG>
__global__ void __launch_bounds__((SPLIT ? kSweepWarps : kRegWarps) * 32, RegBlocks<CH, SPLIT>::value)
k_sweep_reg(SweepArgs a)
{
    static_assert(!(SPLIT && WT), "split documents have integer counts");
    static_assert(!(BIG && WT), "weighted counts are floats");
    using CT = typename std::conditional<WT, float, int>::type;
    using FT = typename std::conditional<BIG, int, float>::type;
    constexpr int T = 4 * CH;            // topics per lane
    constexpr int kRing = CH <= 2 ? 4 : 2;
    constexpr int kWarps = SPLIT ? kSweepWarps : kRegWarps;
    extern __shared__ __align__(16) int smem[];
    const int K = (int)a.K;
    const int KP = (int)round4(a.K);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    // the batch's tokens, one 16-byte broadcast read each: {topic, own weight,
    // uniform, token weight}; the draw's topic replaces the first
    __shared__ __align__(16) float4 s_tok_all[kWarps][33];
    // the words' columns (their index in 16-byte units) of two batches
    __shared__ uint32_t s_col_all[kWarps][64];
    float4* s_tok = s_tok_all[warp];
    uint32_t* s_col = s_col_all[warp];
    for (int i = lane; i < 64; i += 32) s_col[i] = 0;    // (read ahead of what is written: any column)
    __syncwarp();
    int* s_dnk = smem;                   // n_k deltas of the block (integer counts): its rows' changes
    int* s_dlt = smem + KP;              // SPLIT: three step buffers of the document's row changes
    __shared__ uint32_t s_q;
    if (!WT) {
        for (int k = threadIdx.x; k < K; k += blockDim.x) s_dnk[k] = 0;
        __syncthreads();
    }
    const unsigned lt = (1u << lane) - 1u;
    // this lane's number of topics
    const int left = K - 4 * lane;
    const int nh = left <= 0 ? 0 : 4 * (left >> 7) + min(left & 127, 4);
    const unsigned last_bit = 1u << (((K - 1) >> 2) & 31);   // the lane of topic K - 1
    float lm[5];                         // 1 in the lanes at or above 2^i, else 0
#pragma unroll
    for (int i = 0; i < 5; ++i) lm[i] = lane >= (1 << i) ? 1.f : 0.f;
    const float eta = a.eta, veta = a.veta;
    const uint32_t iter = a.iter_ptr ? *a.iter_ptr : a.iter;

    FT fn[T];                            // counts of this lane's topics
    float al[T], mk[OPT ? T : 1];        // their alphas, mask (1 / 0)
    auto topic_of = [&](int t) { return 128 * (t >> 2) + 4 * lane + (t & 3); };
    auto load_alpha = [&](const float* alpha) {
#pragma unroll
        for (int t = 0; t < T; ++t) {
            const int k = topic_of(t);
            al[t] = k < K ? __ldg(alpha + k) : 0.f;
        }
    };
    load_alpha(a.alpha);
    auto set_doc = [&](uint64_t d) {
        if constexpr (OPT) {
            if (a.arow) load_alpha(a.alpha_rows + (uint64_t)a.arow[d] * K);
            const uint32_t* dm = a.mask ? a.mask + d * (uint64_t)a.mw : nullptr;
#pragma unroll
            for (int t = 0; t < T; ++t) {
                const int k = topic_of(t);
                mk[t] = (dm && k < K) ? (float)((__ldg(dm + (k >> 5)) >> (k & 31)) & 1u) : 1.f;
            }
        }
    };

    // --- a token batch's three stages (one token per lane) ---
    uint32_t w2 = 0, z2 = 0, w1 = 0, z1 = 0, w0 = 0, z0 = 0;
    float wt2 = 0.f, wt1 = 0.f, wt0 = 0.f;
    CT nkw1 = CT(0);
    float ri1 = 0.f, u0 = 0.f, po0 = 0.f;
    // The current document's (or slice's) tokens are [0, len) from token tok0;
    // positions and lengths are below 2^31 (kRegMaxLen).
    uint64_t tok0 = 0;
    uint32_t col_at = 0, col_end = 0;    // s_col: the current batch's first entry, the next one's end (mod 64)
    unsigned vm1 = 0, vm0 = 0;           // the lanes whose word is sampled
    // stage 2: a token's word, assignment and weight; lanes past `end` hold word 0xFFFFFFFF
    auto fetch_token = [&](uint32_t base, uint32_t end) {
        w2 = 0xFFFFFFFFu;
        z2 = 0;
        if (base + lane < end) {
            const uint64_t i = tok0 + (base + lane);
            w2 = a.words[i];
            z2 = a.z[i];
            if (WT) wt2 = a.wt[i];
        }
    };
    // stage 1: the own topic's count and reciprocal (weighted: n_k) in the snapshot
    auto fetch_own = [&]() {
        w1 = w2;
        z1 = z2;
        wt1 = wt2;
        nkw1 = CT(0);
        ri1 = 0.f;
        vm1 = __ballot_sync(FULL, w1 < a.V);
        if (w1 < a.V) {
            // (32 bits: V K below 2^34; the counts' 12 bytes an entry end a device's memory before)
            s_col[(col_end + __popc(vm1 & lt)) & 63] = w1 * (uint32_t)(KP >> 2);
            nkw1 = __ldg(reinterpret_cast<const CT*>(a.nkw) + (uint64_t)w1 * K + z1);
            ri1 = __ldg((WT ? reinterpret_cast<const float*>(a.nk) : a.rm1) + z1);
        }
        col_end += __popc(vm1);
    };
    // stage 0: the token's uniform and its own topic's word weight with the
    // token removed from n_kw and n_k
    auto form_own = [&](uint32_t base) {
        w0 = w1;
        z0 = z1;
        wt0 = wt1;
        vm0 = vm1;
        const uint64_t gi = tok0 + (base + lane) + a.tok_offset;
        u0 = tmt::u01(tmt::philox_u32((uint32_t)gi, (uint32_t)(gi >> 32), tmt::kStreamSweep, iter, a.seed));
        float eo = eta;
        if (a.pr.idx && w0 < a.V) {
            const float* pe = prior_col(a.pr, w0, K);
            if (pe) eo = __ldg(pe + z0);
        }
        if constexpr (WT) {
            const float so = a.pr.idx && w0 < a.V ? __ldg(a.pr.esum + z0) : veta;
            float co = __fsub_rn(nkw1, wt0), no = __fsub_rn(ri1, wt0);
            co = co > 0.f ? co : 0.f;
            no = no > 0.f ? no : 0.f;
            po0 = __fmul_rn(__fadd_rn(co, eo), __fdiv_rn(1.0f, __fadd_rn(no, so)));
        } else {
            po0 = __fmul_rn(__fadd_rn((float)(nkw1 - 1), eo), ri1);
        }
    };

    float4 pv[kRing][CH];                // columns of the word table: token j in pv[j % kRing]
    const float4* phi4 = reinterpret_cast<const float4*>(a.phi) + lane;
    auto load_col = [&](uint32_t col, float4 (&p)[CH]) {
        const float4* ph = phi4 + col;
#pragma unroll
        for (int jj = 0; jj < CH; ++jj)
            if (4 * lane + 128 * jj < KP) p[jj] = __ldg(ph + 32 * jj);
    };
    // (a lane's blocks past K are never loaded and stay 0)
#pragma unroll
    for (int q = 0; q < kRing; ++q)
#pragma unroll
        for (int jj = 0; jj < CH; ++jj) pv[q][jj] = make_float4(0.f, 0.f, 0.f, 0.f);

    // One draw: the token t4 = {topic, own weight, uniform, weight} at s_tok[j]
    // with column p; updates fn and leaves the new topic in s_tok[j].
    auto draw = [&](const float4 t4, int j, const float4 (&p)[CH]) {
        float A[T], w[T];
        float own_w = 0.f, s = 0.f;
        const float po = t4.y, u = t4.z, wt = t4.w;
        // the own topic's place among this lane's, if 128 j + i
        const int zr = __float_as_int(t4.x) - 4 * lane;
#pragma unroll
        for (int t = 0; t < T; ++t) {
            const bool own = zr == 128 * (t >> 2) + (t & 3);
            if (own) {
                if constexpr (WT) fn[t] = fmaxf(__fsub_rn(fn[t], wt), 0.f);
                else fn[t] -= FT(1);
            }
            A[t] = __fadd_rn((float)fn[t], al[t]);
            if constexpr (OPT) A[t] = __fmul_rn(A[t], mk[t]);
            const float4 q = p[t >> 2];
            const float pt = (t & 3) == 0 ? q.x : (t & 3) == 1 ? q.y : (t & 3) == 2 ? q.z : q.w;
            // the own topic is left out of the chain (its product is 0) and added last
            // (products with a 0/1 vector in place of the selects measured slower)
            s = __fmaf_rn(A[t], own ? 0.f : pt, s);
            w[t] = __fmul_rn(A[t], own ? po : pt);
            if (own) own_w = w[t];
        }
        s = __fadd_rn(s, own_w);
        float x = s;
#pragma unroll
        for (int i = 0; i < STEPS; ++i) x = hs_step(x, 1 << i, lm[i]);
        const float total = __shfl_sync(FULL, x, (1 << STEPS) - 1);
        const float E = __fmul_rn(__shfl_up_sync(FULL, x, 1), lm[0]);
        // the prefix sums of this lane's own weights (Hillis-Steele order)
#pragma unroll
        for (int off = 1; off < T; off <<= 1) {
#pragma unroll
            for (int t = T - 1; t >= off; --t) w[t] = __fadd_rn(w[t], w[t - off]);
        }
        const float r = __fmul_rn(u, total);
        const bool q = r < __fadd_rn(E, s);
        int found = T - 1;
#pragma unroll
        for (int t = T - 2; t >= 0; --t)
            if (r < __fadd_rn(E, w[t])) found = t;
        found = q ? min(found, nh - 1) : nh - 1;
        // the first lane that r falls in; topic K - 1 when rounding left it at
        // or above the total.  With CH = 1 that topic's lane is the last one
        // with topics, and lanes past it do not count.
        unsigned m = __ballot_sync(FULL, q);
        if (CH == 1) m |= last_bit;
        else if (m == 0) m = last_bit;
        const bool hit = (m & (0u - m)) == lt + 1u;
        const int sel = hit ? found : -1;
#pragma unroll
        for (int t = 0; t < T; ++t)
            if (sel == t) fn[t] += WT ? FT(wt) : FT(1);
        // (predicated: a store under `if` is a branch on the draw's chain)
        asm volatile("{\n .reg .pred p;\n setp.ne.s32 p, %0, 0;\n @p st.shared.s32 [%1], %2;\n}"
                     :: "r"((int)hit), "r"((uint32_t)__cvta_generic_to_shared(s_tok + j)), "r"(topic_of(found))
                     : "memory");
    };

    bool primed = false;                 // pv holds the first kRing - 1 columns of the coming draws
    // The draws of the batch in stage 0 (n token positions from base), then its
    // assignments and count deltas.  SPLIT: `sub` positions at a time, and
    // step_done() after each part that ends a step (dlt: the step's row changes).
    auto process = [&](uint32_t base, uint32_t n, uint32_t sub, bool last, int*& dlt, auto&& step_done) {
        const bool valid = w0 < a.V;
        const int rank = __popc(vm0 & lt), cnt = __popc(vm0);
        if (valid) s_tok[rank] = make_float4(__int_as_float((int)z0), po0, u0, wt0);
        __syncwarp();
        uint32_t coming = s_col[(col_at + kRing - 1) & 63];
        float4 tok = s_tok[0];
        // one token: the column of the token kRing - 1 ahead and the next token, then the draw
        auto step = [&](int j, int slot) {
            load_col(coming, pv[(slot + kRing - 1) % kRing]);
            coming = s_col[(col_at + j + kRing) & 63];
            const float4 cur = tok;
            tok = s_tok[j + 1];
            draw(cur, j, pv[slot]);
        };
        uint32_t lo = 0;
        int j = 0;
        for (;;) {
            const uint32_t hi = SPLIT ? min(lo + sub, n) : n;
            const int end = SPLIT && hi < 32 ? __popc(vm0 & ((1u << hi) - 1u)) : cnt;
            const int count = end - j;
            if (!primed) {
#pragma unroll
                for (int q = 0; q < kRing - 1; ++q) load_col(s_col[(col_at + j + q) & 63], pv[q]);
            }
#pragma unroll 1
            for (; j + kRing <= end; j += kRing) {
#pragma unroll
                for (int q = 0; q < kRing; ++q) step(j + q, q);
            }
#pragma unroll
            for (int q = 0; q < kRing - 1; ++q)
                if (j + q < end) step(j + q, q);
            j = end;
            primed = count % kRing == 0 && (primed || count > 0);
            __syncwarp();
            if (valid && (!SPLIT || ((uint32_t)lane >= lo && (uint32_t)lane < hi))) {
                const uint32_t znew = (uint32_t)__float_as_int(s_tok[rank].x);
                a.z[tok0 + (base + lane)] = (uint16_t)znew;
                if (znew != z0) {
                    if constexpr (WT) {
                        const unsigned long long q = (unsigned long long)wq_of(wt0);
                        unsigned long long* dw = reinterpret_cast<unsigned long long*>(a.dkw) + (uint64_t)w0 * K;
                        atomicAdd(dw + z0, 0ull - q);
                        atomicAdd(dw + znew, q);
                    } else {
                        int32_t* col = a.nkw_next + (uint64_t)w0 * K;
                        atomicSub(col + z0, 1);
                        atomicAdd(col + znew, 1);
                        if (SPLIT && dlt) {
                            atomicSub(&dlt[z0], 1);
                            atomicAdd(&dlt[znew], 1);
                        }
                    }
                }
            }
            __syncwarp();
            if (!SPLIT) break;
            if (dlt && (hi < n || last)) dlt = step_done();
            lo = hi;
            if (lo >= n) break;
        }
        col_at += cnt;
        if (cnt == 0) primed = false;    // (the batch after it was not yet in s_col)
    };

    // The document's (or slice's) len > 0 tokens from `begin`, in batches of at most
    // 32.  SPLIT with steps of m positions (dlt != NULL): a batch is 32
    // positions when m divides 32 (its parts are the steps), else it ends where a
    // step ends; step_done() follows each step and returns the next one's delta buffer.
    auto run = [&](uint64_t begin, uint32_t len, uint32_t m, int* dlt, auto&& step_done) {
        tok0 = begin;
        const bool parts = !SPLIT || !dlt || (m < 32 && 32 % m == 0);
        const uint32_t sub = SPLIT && dlt && parts ? m : 32;
        uint32_t stop = parts ? len : min(m, len);           // of the batch fetched last
        auto batch_end = [&](uint32_t base) {
            if (SPLIT && base >= stop) stop = min(stop + m, len);
            return min(base + 32, stop);
        };
        // a batch that ends inside a step ends none (SPLIT without parts)
        auto ends_step = [&](uint32_t end) { return parts || end == stop; };
        col_at = col_end = 0;
        primed = false;
        uint32_t b0 = 0, b1 = batch_end(0);                  // batch 0 is [b0, b1), batch 1 [b1, b2)
        bool last0 = ends_step(b1);
        fetch_token(0, b1);
        fetch_own();
        uint32_t b2 = b1 < len ? batch_end(b1) : len;
        bool last1 = ends_step(b2);
        fetch_token(b1, b2);
        for (;;) {
            form_own(b0);
            fetch_own();
            const uint32_t b3 = b2 < len ? batch_end(b2) : len;
            const bool last2 = ends_step(b3);
            fetch_token(b2, b3);
            process(b0, b1 - b0, sub, last0, dlt, step_done);
            if (b1 >= len) break;
            b0 = b1; b1 = b2; b2 = b3;
            last0 = last1; last1 = last2;
        }
    };

    // Phase 1: split documents, one per block, as kSweepWarps slices side by
    // side.  Every warp keeps the whole row (counts as of the step's start plus
    // its own changes) in registers; all changes of step s go to buffer s % 3,
    // which every warp adds to its integer copy after the step's barrier.
    // Three buffers need one barrier a step: buffer (s + 1) % 3 is cleared
    // during step s, after the barrier that ended step s - 1 -- its readers,
    // after step s - 2, all passed that barrier.
    if constexpr (SPLIT) {
        for (;;) {
            __syncthreads();
            if (threadIdx.x == 0) s_q = atomicAdd(a.long_counter, 1u);
            for (int k = threadIdx.x; k < 3 * KP; k += blockDim.x) s_dlt[k] = 0;
            __syncthreads();
            const uint32_t q = s_q;
            if (q >= a.n_long) break;
            const uint64_t d = a.doc_order[a.pos_begin + q];
            set_doc(d);
            int* grow = reinterpret_cast<int*>(a.ndk) + d * (uint64_t)K;
            int cn[T];
#pragma unroll
            for (int t = 0; t < T; ++t) {
                const int k = topic_of(t);
                cn[t] = k < K ? grow[k] : 0;
                fn[t] = (FT)cn[t];
            }
            __syncthreads();             // every warp has the row before any of them could write it back
            const uint64_t b = a.doc_off[d];
            const uint32_t L = (uint32_t)(a.doc_off[d + 1] - b);
            const uint32_t sb = (uint32_t)((uint64_t)warp * L / nwarps), se = (uint32_t)((uint64_t)(warp + 1) * L / nwarps);
            const uint32_t m = a.split_step;
            const uint32_t steps = ((L + nwarps - 1) / nwarps + m - 1) / m;   // the longest slice's steps
            uint32_t st = 0;
            int buf = 0;                 // st % 3
            auto merge = [&]() -> int* {
                __syncthreads();         // every slice's changes of this step are in its buffer
                const int* d0 = s_dlt + buf * KP;
#pragma unroll
                for (int t = 0; t < T; ++t) {
                    const int k = topic_of(t);
                    if (k < K) cn[t] += d0[k];
                    fn[t] = (FT)cn[t];
                }
                buf = buf == 2 ? 0 : buf + 1;
                ++st;
                int* nx = s_dlt + (buf == 2 ? 0 : buf + 1) * KP;
                for (int k = threadIdx.x; k < KP; k += blockDim.x) nx[k] = 0;
                return s_dlt + buf * KP;
            };
            if (sb < se) run(b + sb, se - sb, m, s_dlt, merge);
            while (st < steps) merge();  // slices one token shorter can have one step less
            if (warp == 0) {
#pragma unroll
                for (int t = 0; t < T; ++t) {
                    const int k = topic_of(t);
                    if (k < K) {
                        const int change = cn[t] - grow[k];
                        if (change) atomicAdd(&s_dnk[k], change);
                        grow[k] = cn[t];
                    }
                }
            }
        }
    }

    // Phase 2: the other documents (or shared rows), one per warp, in order.
    for (;;) {
        uint32_t q = 0;
        if (lane == 0) q = atomicAdd(a.doc_counter, 1u);
        q = __shfl_sync(FULL, q, 0);
        const uint64_t pos = a.pos_begin + (SPLIT ? a.n_long : 0) + q;
        if (pos >= a.pos_end) break;
        const uint64_t d = a.doc_order[pos];
        set_doc(d);
        CT* grow = reinterpret_cast<CT*>(a.ndk) + d * (uint64_t)K;
#pragma unroll
        for (int t = 0; t < T; ++t) {
            const int k = topic_of(t);
            fn[t] = k < K ? (FT)grow[k] : FT(0);
        }
        auto none = [] () -> int* { return nullptr; };
        const uint64_t un_end = a.unit_off ? a.unit_off[d + 1] : 1;
        for (uint64_t un = a.unit_off ? a.unit_off[d] : 0; un < un_end; ++un) {
            const uint64_t dd = a.unit_off ? a.unit_docs[un] : d;
            const uint64_t b = a.doc_off[dd];
            const uint32_t len = (uint32_t)(a.doc_off[dd + 1] - b);
            if (len) run(b, len, 0, nullptr, none);
        }
#pragma unroll
        for (int t = 0; t < T; ++t) {
            const int k = topic_of(t);
            if (k < K) {
                if constexpr (!WT) {
                    const int change = (int)fn[t] - grow[k];
                    if (change) atomicAdd(&s_dnk[k], change);
                }
                grow[k] = (CT)fn[t];
            }
        }
    }
    if (!WT) {
        __syncthreads();
        for (int k = threadIdx.x; k < K; k += blockDim.x)
            if (s_dnk[k]) atomicAdd(&a.nk_next[k], s_dnk[k]);
    }
}
