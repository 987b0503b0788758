// lg_attn_deep.cuh -- split-KV flash-decode for full-attention layers of long-context sessions.
//
// The decode step's attention kernel (lg_attn_kernel) gives every tile of 128 keys its own CTA and
// lets the last CTA of a KV head merge all tiles: right at a few thousand keys, but at 32K keys that
// is 257 one-tile CTAs per head, one per SM at a time with its load and its math back to back, and a
// 2 MB merge by a single CTA.  Here a CTA walks a SPAN of G consecutive tiles of 64 keys with an
// online softmax (running max / sum per query, accumulators in registers), the next tile's copies run
// under the math, and the merge runs over spans, G times fewer partials.
//
// Spans, like tiles, lie on ABSOLUTE position boundaries (span s = keys [s*G*64, (s+1)*G*64)), G is a
// property of the session (the cache length), and a tile that lies wholly behind a query is an exact
// no-op for that query (weights 0, rescale 1).  So a query row's result depends on its own
// position only -- not on the verify width or on which other rows share the launch -- which keeps the
// speculative stream byte-identical to plain decoding.
#pragma once
#include "lg_kernels.cuh"
#include "lg_attn_cluster.cuh"         // kv_at

#define LG_DEEP_S 64

// dynamic smem (1024-byte aligned): K | V tile [HD/64][64][64] f16 swizzled | Qhi | Qlo [NQ16][HD+8] f16 | scores 2 x [NQ16][64] f32
//               | Phi | Plo [NQ16][72] f16 | m, l, alpha [NQ16][3] | new K / V rows [2 LG_MAXM][HD] f16
// Bound by the instruction chain of a tile between its four block barriers; the copies run under it.  128 registers, so that two CTAs
// share an SM (left alone, head size 256 takes 221 and one fits) -- up to 16 query rows: at head size 256 the shared memory of 17 to 32
// (E4B-class, widths 5 to 8: 134 KB) leaves room for one.  12B-class layer, 32768 positions, 4 x 16 query rows (268 MB of
// cache): 105 us with the merge by a last CTA and plain copies, 65 + 8 us now, 0.64 of the copy rate.
template <int HD>
__global__ void __launch_bounds__(LG_ATTN_THREADS, 2)
lg_attn_deep_kernel(const __grid_constant__ CUtensorMap tmk, const __grid_constant__ CUtensorMap tmv, LgAttnArgs a) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ float s_qn[HD], s_kn[HD];
    __shared__ __align__(8) uint64_t kbar, vbar;
    pdl_launch();
    LG_STAMP_KIND(a.tag, 5);
    if (threadIdx.x == 0) { mbar_init(&kbar, 1); mbar_init(&vbar, 1); }
    if (!a.q_ready)
        for (int i = threadIdx.x; i < HD; i += LG_ATTN_THREADS) { s_qn[i] = a.q_norm[i]; s_kn[i] = a.k_norm ? a.k_norm[i] : 1.0f; }
    if (!a.early_kv) pdl_wait();
    const int called_off = !a.early_kv && a.skip ? __ldcg(a.skip) : 0;      // read beside the position
    constexpr int S = LG_DEEP_S, LDH = HD + 8, LDP = S + 8, PER = HD / 64, HALF = HD / 2, NW = LG_ATTN_THREADS / 32;
    const int G = a.G;
    const int kvh = blockIdx.x, gqa = a.H / a.Hkv, nq = gqa * a.M, nq16 = (nq + 15) & ~15;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int pos0 = __ldcg(a.pos);
    if (called_off) return;
    const int p_last = pos0 + a.M - 1 + a.qpos_off;
    if (p_last < 0) return;
    const int t_hi = p_last / S, SP = blockIdx.y, slot = SP % a.n_slots;      // last tile; this CTA's span
    const int T0 = SP * G, T1 = min(T0 + G - 1, t_hi);
    if (T0 > t_hi) return;
    const bool writes_kv = a.owns_kv && !a.q_ready;

    unsigned char *smem = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    __half *sk = (__half *)smem, *sv = sk + (size_t)S * HD;
    __half *qhi = sv + (size_t)S * HD, *qlo = qhi + (size_t)nq16 * LDH;
    float *sc = (float *)(qlo + (size_t)nq16 * LDH), *sc2 = sc + (size_t)nq16 * S;    // scores: lower / upper half of the head dims
    __half *phi = (__half *)(sc2 + (size_t)nq16 * S), *plo = phi + (size_t)nq16 * LDP;
    float *row_m = (float *)(plo + (size_t)nq16 * LDP), *row_l = row_m + nq16, *row_a = row_l + nq16;
    __half *kvnew = (__half *)(row_a + nq16);                   // the block's own K / V rows (row 2 tok + isv)

    // one thread sends a tile's boxes; rows past the last position arrive as the cache holds them and meet zero weights
    auto load_rows = [&](int T, const CUtensorMap *map, __half *dst, uint64_t *bar) {
        mbar_expect_tx(bar, (uint32_t)S * HD * 2);
        const int y = (int)(((long long)T * S) % a.seq);
        #pragma unroll
        for (int c = 0; c < HD / 64; c++) tma_load_2d(dst + (size_t)c * S * 64, map, kvh * HD + c * 64, y, bar);
    };
    if (threadIdx.x == 0) { load_rows(T0, &tmk, sk, &kbar); load_rows(T0, &tmv, sv, &vbar); }
    if (a.early_kv) pdl_wait();
    __syncthreads();                                            // the norm weights and the barriers are in place

    // the block's own K / V rows that fall into this span (norm + rope, f16 RNE): to the cache, and set aside for the tile.  Their
    // loads go out with those of the warp's first query row.
    auto store_q = [&](int qi, const float (&v0)[PER], const float (&v1)[PER]) {
        #pragma unroll
        for (int e = 0; e < PER; e++) {
            int i = lane * PER + e;
            __half h0 = __float2half_rn(v0[e]), h1 = __float2half_rn(v1[e]);
            qhi[(size_t)qi * LDH + i] = h0; qhi[(size_t)qi * LDH + i + HALF] = h1;
            qlo[(size_t)qi * LDH + i] = __float2half_rn(v0[e] - __half2float(h0));
            qlo[(size_t)qi * LDH + i + HALF] = __float2half_rn(v1[e] - __half2float(h1));
        }
    };
    {
        auto q_src = [&](int qi) {
            const int tok = qi / gqa, hq = kvh * gqa + qi % gqa;
            return a.q_ready ? a.qkv + ((size_t)tok * a.H + hq) * HD : a.qkv + (size_t)tok * a.ld + (size_t)hq * HD;
        };
        float qv0[2][PER], qv1[2][PER]; float2 qcs[2][PER];
        float kv0[2][PER], kv1[2][PER]; float2 kcs[2][PER];
        bool hask[2];
        #pragma unroll
        for (int u = 0; u < 2; u++) {
            const int qi = warp + u * NW;
            if (qi < nq) head_load<HD>(q_src(qi), a.q_ready ? nullptr : a.rope + (size_t)(qi / gqa) * HALF, lane, qv0[u], qv1[u], qcs[u]);
        }
        #pragma unroll
        for (int u = 0; u < 2; u++) {
            const int j = warp + u * NW, tok = j >> 1, isv = j & 1, TT = (pos0 + tok) / S;
            hask[u] = writes_kv && j < 2 * a.M && TT >= T0 && TT <= T1;
            if (hask[u])
                head_load<HD>(a.qkv + (size_t)tok * a.ld + (size_t)(a.H + ((isv && a.has_v) ? a.Hkv : 0) + kvh) * HD,
                              isv ? nullptr : a.rope + (size_t)tok * HALF, lane, kv0[u], kv1[u], kcs[u]);
        }
        #pragma unroll
        for (int u = 0; u < 2; u++) {
            const int qi = warp + u * NW;
            if (qi < nq) {
                if (!a.q_ready) head_finish<HD>(s_qn, true, a.eps, lane, qv0[u], qv1[u], qcs[u]);
                store_q(qi, qv0[u], qv1[u]);
            }
        }
        #pragma unroll
        for (int u = 0; u < 2; u++) {
            if (!hask[u]) continue;
            const int j = warp + u * NW, tok = j >> 1, isv = j & 1, p = pos0 + tok;
            head_finish<HD>(isv ? nullptr : s_kn, !isv, a.eps, lane, kv0[u], kv1[u], kcs[u]);
            __half *dst = (isv ? a.vc : a.kc) + (size_t)(p % a.seq) * a.kv_dim + (size_t)kvh * HD;
            #pragma unroll
            for (int e = 0; e < PER; e++) {
                const __half h0 = __float2half_rn(kv0[u][e]), h1 = __float2half_rn(kv1[u][e]);
                dst[lane * PER + e] = h0; dst[lane * PER + e + HALF] = h1;
                kvnew[(size_t)j * HD + lane * PER + e] = h0; kvnew[(size_t)j * HD + lane * PER + e + HALF] = h1;
            }
        }
        for (int qi = warp + 2 * NW; qi < nq; qi += NW) {
            float v0[PER], v1[PER];
            if (a.q_ready) {
                const float *src = q_src(qi);
                #pragma unroll
                for (int e = 0; e < PER; e++) { v0[e] = src[lane * PER + e]; v1[e] = src[lane * PER + e + HALF]; }
            } else {
                head_norm_rope<HD>(q_src(qi), s_qn, a.rope + (size_t)(qi / gqa) * HALF, a.eps, lane, v0, v1);
            }
            store_q(qi, v0, v1);
        }
        for (int qi = nq + warp; qi < nq16; qi += NW) {
            float z[PER];
            #pragma unroll
            for (int e = 0; e < PER; e++) z[e] = 0.0f;
            store_q(qi, z, z);
        }
    }
    for (int r = threadIdx.x; r < nq16; r += LG_ATTN_THREADS) { row_m[r] = -INFINITY; row_l[r] = 0.0f; row_a[r] = 1.0f; }
    // rows past the last query only pad the 16-row tiles: their probabilities stay zero, the softmax skips them
    for (int i = threadIdx.x; i < (nq16 - nq) * LDP; i += LG_ATTN_THREADS) {
        phi[(size_t)nq * LDP + i] = __float2half_rn(0.0f); plo[(size_t)nq * LDP + i] = __float2half_rn(0.0f);
    }

    const int g = lane >> 2, t = lane & 3;
    // Both products run "transposed": keys (scores) or head dims (P V) are the 16-row side of the tensor-core tile and
    // the queries its 8-column side, so a block of up to 8 query rows costs one column tile, not a half-empty 16-row tile.
    constexpr int MTW = HD / 16 / NW;                            // 16-dim row tiles of O^T per warp
    static_assert(S == 64 && NW == 8 && HD % (16 * NW) == 0, "four 16-key row tiles x two halves of the head dims over eight warps");
    const int nq8 = (nq + 7) >> 3;                               // 8-query column tiles (at most 4)
    float o[MTW][4][4];                                          // O^T accumulators [dim tile][query tile][frag], kept across the span's tiles
    #pragma unroll
    for (int mt = 0; mt < MTW; mt++)
        #pragma unroll
        for (int n = 0; n < 4; n++) o[mt][n][0] = o[mt][n][1] = o[mt][n][2] = o[mt][n][3] = 0.0f;

    // a tile's rows of the block's own positions go over whatever the copy brought for them; rows of V behind the block become zeros
    // (a cache that was used before may hold infinities there, and the product takes every row of the tile)
    auto patch = [&](int T, __half *tile, int isv) {
        for (int tok = warp; tok < a.M; tok += NW) {
            const int p = pos0 + tok;
            if (p / S != T) continue;
            #pragma unroll
            for (int e = 0; e < PER; e++) {
                *kv_at<S>(tile, p - T * S, lane * PER + e) = kvnew[(size_t)(2 * tok + isv) * HD + lane * PER + e];
                *kv_at<S>(tile, p - T * S, lane * PER + e + HALF) = kvnew[(size_t)(2 * tok + isv) * HD + lane * PER + e + HALF];
            }
        }
    };
    uint32_t parity = 0;
    for (int T = T0; T <= T1; T++, parity ^= 1) {
        __syncthreads();                                         // Q and the new rows are in place; the previous tile's V and P are no longer read
        if (T > T0 && threadIdx.x == 0) { fence_async_shared(); load_rows(T, &tmv, sv, &vbar); }
        if (!mbar_wait(&kbar, parity) && a.err && lane == 0) atomicOr(a.err, LG_ERR_MBAR_TIMEOUT);
        if (writes_kv && pos0 + a.M > T * S && pos0 < (T + 1) * S) { patch(T, sk, 0); __syncthreads(); }
        if (T == T0 + 2) LG_STAMP(a.tag, 1);

        // scores S^T = K Q^T: warp w holds keys [16 (w & 3), +16) as the tile's rows and half (w >> 2) of the head dims,
        // 8 queries per column tile; the two halves land in two buffers the softmax adds.  A key that a query does not see is -inf in
        // both: rows behind the block arrive as the cache holds them, and -inf plus what a NaN or an infinity of an earlier use makes is NaN
        {
            float c0[4][4], c1[4][4];
            #pragma unroll
            for (int n = 0; n < 4; n++)
                #pragma unroll
                for (int f = 0; f < 4; f++) c0[n][f] = c1[n][f] = 0.0f;
            const int kt = warp & 3, dh = warp >> 2;
            const int krow = kt * 16 + (lane & 7) + ((lane >> 3) & 1) * 8, kcol = dh * (HD / 2) + (lane >> 4) * 8;
            #pragma unroll 2
            for (int k0 = 0; k0 < HD / 2; k0 += 16) {
                uint32_t ka[4];                                  // A operand: 16 keys x 16 dims
                ldsm_x4(ka, kv_at<S>(sk, krow, kcol + k0));
                #pragma unroll
                for (int n = 0; n < 4; n++) {
                    if (n >= nq8) break;
                    uint32_t bq[4];                              // B operands: 8 queries x 16 dims, hi (bq[0..1]) and lo (bq[2..3])
                    const __half *qp = ((lane >> 4) ? qlo : qhi) + (size_t)(n * 8 + (lane & 7)) * LDH + dh * (HD / 2) + k0 + ((lane >> 3) & 1) * 8;
                    ldsm_x4(bq, qp);
                    mma_f16(c0[n], ka, bq[0], bq[1]); mma_f16(c1[n], ka, bq[2], bq[3]);
                }
            }
            float *dst = dh ? sc2 : sc;
            #pragma unroll
            for (int n = 0; n < 4; n++) {
                if (n >= nq8) break;
                #pragma unroll
                for (int e = 0; e < 2; e++) {
                    const int qi = n * 8 + t * 2 + e;
                    const int pj = pos0 + qi / gqa + a.qpos_off;
                    #pragma unroll
                    for (int h2 = 0; h2 < 2; h2++) {
                        const int key = kt * 16 + g + h2 * 8, p = T * S + key;
                        const float v = c0[n][h2 * 2 + e] + c1[n][h2 * 2 + e];
                        dst[(size_t)qi * S + key] = qi < nq && p <= pj ? v : -INFINITY;
                    }
                }
            }
        }
        __syncthreads();
        if (T < T1 && threadIdx.x == 0) { fence_async_shared(); load_rows(T + 1, &tmk, sk, &kbar); }     // K is free: the next tile's under softmax and value product
        if (T == T0 + 2) LG_STAMP(a.tag, 2);

        // online softmax, one warp per query row: new running max, the tile's weights against it, the rescale
        // of what was accumulated before (exactly 1 when the tile adds nothing for this row)
        for (int qi = warp; qi < nq; qi += NW) {
            const float s0 = sc[(size_t)qi * S + lane] + sc2[(size_t)qi * S + lane], s1 = sc[(size_t)qi * S + lane + 32] + sc2[(size_t)qi * S + lane + 32];
            const float m_old = row_m[qi];
            const float m_new = fmaxf(m_old, warp_max(fmaxf(s0, s1)));
            const float e0 = s0 == -INFINITY ? 0.0f : expf(s0 - m_new), e1 = s1 == -INFINITY ? 0.0f : expf(s1 - m_new);
            const __half h0 = __float2half_rn(e0), h1 = __float2half_rn(e1);
            phi[(size_t)qi * LDP + lane] = h0; phi[(size_t)qi * LDP + lane + 32] = h1;
            plo[(size_t)qi * LDP + lane] = __float2half_rn(e0 - __half2float(h0));
            plo[(size_t)qi * LDP + lane + 32] = __float2half_rn(e1 - __half2float(h1));
            const float sum = warp_sum(e0 + e1);
            if (lane == 0) {
                const float alpha = (m_old == m_new) ? 1.0f : expf(m_old - m_new);     // m_old = -inf < m_new: 0
                row_a[qi] = alpha;
                row_l[qi] = row_l[qi] * alpha + sum;
                row_m[qi] = m_new;
            }
        }
        if (!mbar_wait(&vbar, parity) && a.err && lane == 0) atomicOr(a.err, LG_ERR_MBAR_TIMEOUT);
        if (writes_kv && pos0 + a.M > T * S && pos0 < (T + 1) * S) patch(T, sv, 1);
        if (p_last + 1 < (T + 1) * S)
            for (int i = threadIdx.x; i < (T * S + S - 1 - p_last) * (HD / 8); i += LG_ATTN_THREADS)
                *(uint4 *)kv_at<S>(sv, p_last + 1 - T * S + i / (HD / 8), i % (HD / 8) * 8) = make_uint4(0, 0, 0, 0);
        __syncthreads();
        if (T == T0 + 2) LG_STAMP(a.tag, 3);

        // O^T = alpha O^T + V^T P^T: warp w holds MTW tiles of 16 head dims as rows, 8 queries per column tile
        {
            #pragma unroll
            for (int n = 0; n < 4; n++) {
                if (n >= nq8) break;
                const float a0 = row_a[n * 8 + t * 2], a1 = row_a[n * 8 + t * 2 + 1];
                #pragma unroll
                for (int mt = 0; mt < MTW; mt++) { o[mt][n][0] *= a0; o[mt][n][1] *= a1; o[mt][n][2] *= a0; o[mt][n][3] *= a1; }
            }
            #pragma unroll
            for (int k0 = 0; k0 < S; k0 += 32) {
                uint32_t ph[4][4], pl[4][4];                    // B operands: 8 queries x keys k0, +8, +16, +24 (hi and lo halves of P)
                #pragma unroll
                for (int n = 0; n < 4; n++) {
                    if (n >= nq8) break;
                    ldsm_x4(ph[n], phi + (size_t)(n * 8 + (lane & 7)) * LDP + k0 + (lane >> 3) * 8);
                    ldsm_x4(pl[n], plo + (size_t)(n * 8 + (lane & 7)) * LDP + k0 + (lane >> 3) * 8);
                }
                #pragma unroll
                for (int mt = 0; mt < MTW; mt++) {
                    const int d0 = (warp * MTW + mt) * 16;
                    uint32_t va[4], vb[4];                      // A operands (transposed loads): 16 dims x keys k0..k0+15, k0+16..k0+31
                    ldsm_x4_t(va, kv_at<S>(sv, k0 + (lane & 7) + (lane >> 4) * 8, d0 + ((lane >> 3) & 1) * 8));
                    ldsm_x4_t(vb, kv_at<S>(sv, k0 + 16 + (lane & 7) + (lane >> 4) * 8, d0 + ((lane >> 3) & 1) * 8));
                    #pragma unroll
                    for (int n = 0; n < 4; n++) {
                        if (n >= nq8) break;
                        mma_f16(o[mt][n], va, ph[n][0], ph[n][1]); mma_f16(o[mt][n], va, pl[n][0], pl[n][1]);
                        mma_f16(o[mt][n], vb, ph[n][2], ph[n][3]); mma_f16(o[mt][n], vb, pl[n][2], pl[n][3]);
                    }
                }
            }
        }
        if (T == T0 + 2) LG_STAMP(a.tag, 4);
    }

    // the span's partial (max, sum, accumulators) of every query row
    #pragma unroll
    for (int n = 0; n < 4; n++) {
        if (n >= nq8) break;
        #pragma unroll
        for (int e = 0; e < 2; e++) {
            const int qi = n * 8 + t * 2 + e;
            if (qi >= nq) continue;
            const int tok = qi / gqa, hq = kvh * gqa + qi % gqa;
            float *pp = a.part + (((size_t)slot * a.M + tok) * a.H + hq) * HD;
            #pragma unroll
            for (int mt = 0; mt < MTW; mt++) {
                const int d0 = (warp * MTW + mt) * 16;
                pp[d0 + g] = o[mt][n][e];
                pp[d0 + g + 8] = o[mt][n][2 + e];
            }
            if (warp == 0 && g == 0) a.part_ml[((size_t)slot * a.M + tok) * a.H + hq] = make_float2(row_m[qi], row_l[qi]);
        }
    }
}

// Merge of the spans.  One CTA per (query row, 128 output dims): a warp owns every eighth span, a lane 4 dims.  Bound by one
// round of loads: the partials (1 MB per KV head at 64 spans x 16 queries) are read by M H hd / 128 CTAs at once, where the last
// CTA of the span kernel used to read them alone.  E4B-class, 8192 positions: attention of a verify step of width 1 / 4 / 8 356 / 742 /
// 1295 us before, 291 / 457 / 724 with this merge and the tiled copies.  Which sums a span enters, and in which order, follows
// from its absolute index alone; spans behind a query add exact zeros.
#define LG_MERGE_DIMS 128
#define LG_MERGE_UNROLL 8
__global__ void __launch_bounds__(256) lg_attn_merge_kernel(LgAttnArgs a) {
    __shared__ float s_red[8], s_sum[8];
    __shared__ float4 s_acc[8][LG_MERGE_DIMS / 4];
    pdl_launch();
    const int lane = threadIdx.x & 31, part = threadIdx.x >> 5;          // a warp per eighth of the spans
    const int tok = blockIdx.y, hq = blockIdx.x, d4 = blockIdx.z * LG_MERGE_DIMS + lane * 4;
    pdl_wait();
    const int called_off = a.skip ? __ldcg(a.skip) : 0;
    const int S = LG_DEEP_S, G = a.G, pos0 = __ldcg(a.pos);
    if (called_off) return;
    const int pj = pos0 + tok + a.qpos_off, p_last = pos0 + a.M - 1 + a.qpos_off;
    if (p_last < 0) return;
    const int s_hi = p_last / S / G, i1 = pj >= 0 ? pj / S / G : -1;      // last span of the block, of the query
    const size_t row = (size_t)tok * a.H + hq, slot = (size_t)a.M * a.H;
    // largest score maximum over all spans of the query
    float mx = -INFINITY;
    for (int s = threadIdx.x; s <= s_hi; s += 256) {
        const float2 v = __ldcg(a.part_ml + (s % a.n_slots) * slot + row);
        if (s <= i1 && v.y > 0.0f) mx = fmaxf(mx, v.x);
    }
    mx = warp_max(mx);
    if (lane == 0) s_red[part] = mx;
    __syncthreads();
    #pragma unroll
    for (int w = 0; w < 8; w++) mx = fmaxf(mx, s_red[w]);
    float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float lsum = 0.0f;
    for (int s = part; s <= s_hi; s += 8 * LG_MERGE_UNROLL) {
        float4 v[LG_MERGE_UNROLL]; float2 m[LG_MERGE_UNROLL];
        #pragma unroll
        for (int j = 0; j < LG_MERGE_UNROLL; j++)
            if (s + 8 * j <= s_hi) {
                const size_t at = ((s + 8 * j) % a.n_slots) * slot + row;
                m[j] = __ldcg(a.part_ml + at);
                v[j] = __ldcg((const float4 *)(a.part + at * a.hd + d4));
            }
        #pragma unroll
        for (int j = 0; j < LG_MERGE_UNROLL; j++)
            if (s + 8 * j <= s_hi) {
                const int sp = s + 8 * j;
                const float w = (sp <= i1 && m[j].y > 0.0f) ? expf(m[j].x - mx) : 0.0f;
                lsum = fmaf(w, m[j].y, lsum);
                acc.x = fmaf(w, v[j].x, acc.x); acc.y = fmaf(w, v[j].y, acc.y);
                acc.z = fmaf(w, v[j].z, acc.z); acc.w = fmaf(w, v[j].w, acc.w);
            }
    }
    s_acc[part][lane] = acc;
    if (lane == 0) s_sum[part] = lsum;
    __syncthreads();
    if (part >= LG_MERGE_DIMS / 32) return;
    // warp `part` finishes 32 dims: the eight partial sums in order
    float y = 0.0f, l = 0.0f;
    #pragma unroll
    for (int w = 0; w < 8; w++) { y += ((const float *)s_acc[w])[part * 32 + lane]; l += s_sum[w]; }
    y = l > 0.0f ? y * (1.0f / l) : 0.0f;
    const int d = blockIdx.z * LG_MERGE_DIMS + part * 32 + lane;
    if (a.out_f32) a.out_f32[row * a.hd + d] = y;
    if (a.out_h) a.out_h[(size_t)tok * a.ld_h + hq * a.hd + d] = __float2half_rn(y);
    if (a.out.q) quant_group_store(y, lane, tok, (hq * a.hd + d) >> 5, a.out);
}

inline size_t attn_deep_smem(int nq, int hd) {
    size_t nq16 = (size_t)((nq + 15) & ~15), ldh = hd + 8, S = LG_DEEP_S;
    return 1024 + 2 * S * hd * 2 + 2 * nq16 * ldh * 2 + 2 * nq16 * S * 4 + 2 * nq16 * (S + 8) * 2 + nq16 * 12 + (size_t)2 * LG_MAXM * hd * 2;
}
