// sweep_wide.cuh -- the training sweep for K <= kWideMaxK with many topics (launch_sweep):
// one warp a document, its row in shared memory, a word's column in registers.
// Included by engine.cu inside its namespace, after SweepArgs; k_sweep_doc there
// states the sampler.  Both compute the same draws, bit for bit.
//
// What bounds it: at K = 1000 a draw reads a 4 KB row through shared memory and, for
// 60% of the tokens, a new 4 KB column from L2; its chain is 32 fma steps, two
// scans and the row's update, ~2,000 cycles with 24 warps an SM.  k_sweep_doc spent
// 281 warp instructions a token and waited for each new column.  Here the next
// token's column is loaded as soon as the hit lane has handed its part of the
// current one to the second scan, so the second scan and the update hide the load
// (a second buffer in registers hid it too, but at 16 warps an SM: K = 1000, 24M tokens,
// 10 sweeps with the state read back 198 against 186 ms); token scalars, own-topic weights and count deltas are formed for 32 tokens
// at a time (as in k_sweep_reg); the row's updates are predicated stores; the
// row is padded with zeros to 128 CH topics and CH is exact, so the fma chain has no
// guards.  The sampling kernels of one sweep, k_sweep_doc's faster variant and this kernel: K = 1000,
// 24M tokens 15.7 -> 14.2 ms, 4.6 -> 3.4 of it the launch of the longest documents; 204M
// tokens, where that launch weighs little, 90.6 -> 90.4 ms, but without the tuner's sweeps
// of a slower variant.

constexpr uint32_t kWideMaxK = 1024;
constexpr int kWideWarps = 4;
constexpr int kWideBlocks = 6;       // resident per SM

//   CH: blocks of four topics per lane (128 (CH - 1) < K <= 128 CH, 2 < CH <= 8)
//   NT: the counts' type -- uint16_t (documents below 65,536 tokens), int, or
//       float for weighted counts (TermWeight IDF / PMI)
//   OPT: per-document masks or alphas may be set
template <int CH, typename NT, bool OPT>
__global__ void __launch_bounds__(kWideWarps * 32, kWideBlocks)
k_sweep_wide(SweepArgs a)
{
    constexpr bool WT = std::is_same<NT, float>::value;
    using CT = typename std::conditional<WT, float, int>::type;
    constexpr int KW = 128 * CH;
    extern __shared__ __align__(16) float s_dyn[];
    const int K = (int)a.K;
    const int KP = (int)round4(a.K);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // block: alpha, n_k deltas; warp: A, counts
    float* s_alpha = s_dyn;
    int* s_dnk = reinterpret_cast<int*>(s_dyn + KW);
    float* s_A = s_dyn + 2 * KW + warp * KW;
    NT* s_n = reinterpret_cast<NT*>(s_dyn + (2 + kWideWarps) * KW) + warp * KW;
    __shared__ __align__(16) float4 s_tok_all[kWideWarps][33];   // as in k_sweep_reg
    __shared__ uint32_t s_col_all[kWideWarps][64];
    __shared__ __align__(16) float s_xs_all[kWideWarps][4 * CH];
    float4* s_tok = s_tok_all[warp];
    uint32_t* s_col = s_col_all[warp];
    float* s_xs = s_xs_all[warp];
    for (int i = lane; i < 64; i += 32) s_col[i] = 0;
    for (int k = threadIdx.x; k < KW; k += blockDim.x) {
        s_alpha[k] = k < K ? a.alpha[k] : 0.f;
        s_dnk[k] = 0;
    }
    for (int k = lane; k < KW; k += 32) {
        s_A[k] = 0.f;
        s_n[k] = NT(0);
    }
    __syncthreads();
    const unsigned lt = (1u << lane) - 1u;
    float lm[5];                         // 1 in the lanes at or above 2^i, else 0
#pragma unroll
    for (int i = 0; i < 5; ++i) lm[i] = lane >= (1 << i) ? 1.f : 0.f;
    const float eta = a.eta, veta = a.veta;
    const uint32_t iter = a.iter_ptr ? *a.iter_ptr : a.iter;

    const float* alpha = nullptr;        // the document's own alphas, if any
    const uint32_t* dmask = nullptr;
    // A of topic k with count n
    auto weight = [&](CT n, int k) -> float {
        float f;
        if constexpr (std::is_same<NT, uint16_t>::value) f = __fsub_rn(__int_as_float(n | 0x4B000000), 8388608.f);   // (float)n
        else f = (float)n;
        float x = __fadd_rn(f, OPT && alpha ? __ldg(alpha + k) : s_alpha[k]);
        if (OPT && dmask) x = __fmul_rn(x, (float)((__ldg(dmask + (k >> 5)) >> (k & 31)) & 1u));
        return x;
    };
    auto less = [](CT n, float wt) -> CT {
        if constexpr (WT) return fmaxf(__fsub_rn(n, wt), 0.f);
        else return n - 1;
    };
    auto more = [](CT n, float wt) -> CT {
        if constexpr (WT) return __fadd_rn(n, wt);
        else return n + 1;
    };

    // --- a token batch's three stages (as in k_sweep_reg, whose comments hold) ---
    uint32_t w2 = 0, z2 = 0, w1 = 0, z1 = 0, w0 = 0, z0 = 0;
    float wt2 = 0.f, wt1 = 0.f, wt0 = 0.f;
    CT nkw1 = CT(0);
    float ri1 = 0.f, u0 = 0.f, po0 = 0.f;
    uint64_t tok0 = 0;
    uint32_t col_at = 0, col_end = 0;
    unsigned vm1 = 0, vm0 = 0;
    auto fetch_token = [&](uint64_t base, uint64_t end) {
        w2 = 0xFFFFFFFFu;
        z2 = 0;
        if (base + lane < end) {
            const uint64_t i = tok0 + base + lane;
            w2 = a.words[i];
            z2 = a.z[i];
            if (WT) wt2 = a.wt[i];
        }
    };
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
    auto form_own = [&](uint64_t base) {
        w0 = w1;
        z0 = z1;
        wt0 = wt1;
        vm0 = vm1;
        const uint64_t gi = tok0 + base + lane + a.tok_offset;
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

    float4 p[CH];                        // the column `have` of the word table
#pragma unroll
    for (int jj = 0; jj < CH; ++jj) p[jj] = make_float4(0.f, 0.f, 0.f, 0.f);
    uint32_t have = 0xFFFFFFFFu;
    const bool last_block = 4 * lane + 128 * (CH - 1) < KP;
    const float4* phi4 = reinterpret_cast<const float4*>(a.phi) + lane;
    auto load_col = [&](uint32_t col) {
        have = col;
#pragma unroll
        for (int jj = 0; jj < CH; ++jj)
            if (jj < CH - 1 || last_block) p[jj] = __ldg(phi4 + col + 32 * jj);
    };
    const uint32_t sA32 = (uint32_t)__cvta_generic_to_shared(s_A), sn32 = (uint32_t)__cvta_generic_to_shared(s_n),
                   st32 = (uint32_t)__cvta_generic_to_shared(s_tok);
    float Ao = 0.f;                      // the current token's topic's A without it (its slot of the row is 0)

    // One draw: token t (at s_tok[j]) with the column in p; nt: the next one, whose
    // topic it then leaves (`next`: there is one in this batch) and whose column, nx, is
    // loaded as soon as p is free.
    auto draw = [&](const float4& t, const float4& nt, int j, bool next, uint32_t nx) {
        const int zo = __float_as_int(t.x);
        const float po = t.y, u = t.z, wt = t.w;
        const float own_w = __fmul_rn(Ao, po);
        float s = 0.f;
#pragma unroll
        for (int jj = 0; jj < CH; ++jj) {
            const float4 A4 = *reinterpret_cast<const float4*>(s_A + 128 * jj + 4 * lane);
            s = __fmaf_rn(A4.x, p[jj].x, s);
            s = __fmaf_rn(A4.y, p[jj].y, s);
            s = __fmaf_rn(A4.z, p[jj].z, s);
            s = __fmaf_rn(A4.w, p[jj].w, s);
        }
        s = __fadd_rn(s, lane == ((zo >> 2) & 31) ? own_w : 0.f);
        float x = s;
#pragma unroll
        for (int i = 0; i < 5; ++i) x = hs_step(x, 1 << i, lm[i]);
        const float total = __shfl_sync(FULL, x, 31);
        const float E = __fmul_rn(__shfl_up_sync(FULL, x, 1), lm[0]);
        const float r = __fmul_rn(u, total);
        const unsigned m = __ballot_sync(FULL, r < __fadd_rn(E, s));
        const int h = m ? __ffs(m) - 1 : 0;
        if (lane == h) {                 // its part of the column, for the second scan
#pragma unroll
            for (int jj = 0; jj < CH; ++jj) *reinterpret_cast<float4*>(s_xs + 4 * jj) = p[jj];
        }
        if (nx != have) load_col(nx);
        // the hit lane's topics: their prefix sums across the warp
        const float Eh = __shfl_sync(FULL, E, h);
        const int mh = K - 4 * h;
        const int nh = 4 * (mh >> 7) + min(mh & 127, 4);
        const int k = 128 * (lane >> 2) + 4 * h + (lane & 3);
        const float Ah = lane < nh ? s_A[k] : 0.f;
        __syncwarp();
        // (the own topic's slot is 0 in the row: its weight is added)
        float x2 = 0.f;
        if (lane < nh) x2 = k == zo ? own_w : __fmul_rn(Ah, s_xs[lane]);
#pragma unroll
        for (int i = 0; i < 5; ++i) x2 = hs_step(x2, 1 << i, lm[i]);
        const unsigned mb = __ballot_sync(FULL, lane < nh && r < __fadd_rn(Eh, x2));
        const int found = mb ? __ffs(mb) - 1 : nh - 1;
        // (no lane hit: rounding left r at or above the total)
        const int knew = m ? 128 * (found >> 2) + 4 * h + (found & 3) : K - 1;
        // the row: zo's slot back, the new topic's count, the next token's topic
        // left; every lane forms them, lane 0 stores in this order (topics may coincide)
        const int zn = next ? __float_as_int(nt.x) : knew;
        const CT nk = more((CT)s_n[knew], wt);
        CT nz = (CT)s_n[zn];
        const float Ak = weight(nk, knew);
        nz = less(zn == knew ? nk : nz, nt.w);
        const float Az = weight(nz, zn);
        __syncwarp();
        // (predicated: a branch would sit on the draw's chain)
        const int n_to = next ? 1 : 0;
        float nkb, nzb;
        if constexpr (WT) {
            nkb = nk;
            nzb = nz;
        } else {
            nkb = __int_as_float(nk);
            nzb = __int_as_float(nz);
        }
        if constexpr (sizeof(NT) == 2)
            asm volatile("{\n .reg .pred p, q;\n .reg .b16 a, b;\n setp.eq.s32 p, %0, 0;\n setp.ne.and.s32 q, %1, 0, p;\n"
                         " cvt.u16.u32 a, %8;\n cvt.u16.u32 b, %9;\n"
                         " @p st.shared.f32 [%2], %5;\n @p st.shared.f32 [%3], %6;\n @p st.shared.u16 [%10], a;\n"
                         " @q st.shared.f32 [%4], 0f00000000;\n @q st.shared.u16 [%11], b;\n @p st.shared.s32 [%12], %7;\n}"
                         :: "r"(lane), "r"(n_to), "r"(sA32 + 4 * zo), "r"(sA32 + 4 * knew), "r"(sA32 + 4 * zn), "f"(Ao),
                            "f"(Ak), "r"(knew), "r"(__float_as_int(nkb)), "r"(__float_as_int(nzb)), "r"(sn32 + 2 * knew),
                            "r"(sn32 + 2 * zn), "r"(st32 + 16 * j) : "memory");
        else
            asm volatile("{\n .reg .pred p, q;\n setp.eq.s32 p, %0, 0;\n setp.ne.and.s32 q, %1, 0, p;\n"
                         " @p st.shared.f32 [%2], %5;\n @p st.shared.f32 [%3], %6;\n @p st.shared.f32 [%10], %8;\n"
                         " @q st.shared.f32 [%4], 0f00000000;\n @q st.shared.f32 [%11], %9;\n @p st.shared.s32 [%12], %7;\n}"
                         :: "r"(lane), "r"(n_to), "r"(sA32 + 4 * zo), "r"(sA32 + 4 * knew), "r"(sA32 + 4 * zn), "f"(Ao),
                            "f"(Ak), "r"(knew), "f"(nkb), "f"(nzb), "r"(sn32 + 4 * knew), "r"(sn32 + 4 * zn),
                            "r"(st32 + 16 * j) : "memory");
        Ao = Az;
        __syncwarp();
    };

    auto process = [&](uint64_t base) {
        const bool valid = w0 < a.V;
        const int rank = __popc(vm0 & lt), cnt = __popc(vm0);
        if (valid) s_tok[rank] = make_float4(__int_as_float((int)z0), po0, u0, wt0);
        __syncwarp();
        if (cnt) {
            float4 tok = s_tok[0];
            {
                // the batch's first token leaves its topic
                const int zo = __float_as_int(tok.x);
                const CT n = less((CT)s_n[zo], tok.w);
                Ao = weight(n, zo);
                __syncwarp();
                if (lane == 0) {
                    s_n[zo] = (NT)n;
                    s_A[zo] = 0.f;
                }
                __syncwarp();
            }
            if (s_col[col_at & 63] != have) load_col(s_col[col_at & 63]);
#pragma unroll 1
            for (int j = 0; j < cnt; ++j) {
                const float4 cur = tok;
                tok = s_tok[j + 1];
                draw(cur, tok, j, j + 1 < cnt, s_col[(col_at + j + 1) & 63]);
            }
        }
        if (valid) {
            const uint32_t znew = (uint32_t)__float_as_int(s_tok[rank].x);
            a.z[tok0 + base + lane] = (uint16_t)znew;
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
                    atomicSub(&s_dnk[z0], 1);
                    atomicAdd(&s_dnk[znew], 1);
                }
            }
        }
        __syncwarp();
        col_at += cnt;
    };

    for (;;) {
        uint32_t q = 0;
        if (lane == 0) q = atomicAdd(a.doc_counter, 1u);
        q = __shfl_sync(FULL, q, 0);
        const uint64_t pos = a.pos_begin + q;
        if (pos >= a.pos_end) break;
        const uint64_t d = a.doc_order[pos];
        if constexpr (OPT) {
            alpha = a.arow ? a.alpha_rows + (uint64_t)a.arow[d] * K : nullptr;
            dmask = a.mask ? a.mask + d * (uint64_t)a.mw : nullptr;
        }
        CT* grow = reinterpret_cast<CT*>(a.ndk) + d * (uint64_t)K;
        for (int k = lane; k < K; k += 32) {
            const CT n = grow[k];
            s_n[k] = (NT)n;
            s_A[k] = weight(n, k);
        }
        __syncwarp();
        const uint64_t un_end = a.unit_off ? a.unit_off[d + 1] : 1;
        for (uint64_t un = a.unit_off ? a.unit_off[d] : 0; un < un_end; ++un) {
            const uint64_t dd = a.unit_off ? a.unit_docs[un] : d;
            tok0 = a.doc_off[dd];
            const uint64_t len = a.doc_off[dd + 1] - tok0;
            if (!len) continue;
            col_at = col_end = 0;
            fetch_token(0, len);
            fetch_own();
            fetch_token(32, len);
            for (uint64_t b = 0; b < len; b += 32) {
                form_own(b);
                fetch_own();
                fetch_token(b + 64, len);
                process(b);
            }
        }
        __syncwarp();
        for (int k = lane; k < K; k += 32) grow[k] = (CT)s_n[k];
        __syncwarp();
    }
    if (!WT) {
        __syncthreads();
        for (int k = threadIdx.x; k < K; k += blockDim.x)
            if (s_dnk[k]) atomicAdd(&a.nk_next[k], s_dnk[k]);
    }
}
