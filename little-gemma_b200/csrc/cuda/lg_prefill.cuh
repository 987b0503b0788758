// lg_prefill.cuh -- the wide (prompt) matmul on the 5th-generation tensor cores.
//
// out[tok][row] = sum_k W[row][k] * X[tok][k] for a block of up to LG_PF_MAXN prompt tokens at once.
// W is the same tile-major q4 matrix the decode step streams (16 rows x 64 columns per 512-byte
// tile, nibbles stored as two's-complement q-8); X is an f16 row-major activation block.  The
// weights are expanded to f16 on the fly -- d*(q-8) rounded once to f16, i.e. the f16 rounding of
// the exact dequantised value -- and the multiply-accumulate runs as tcgen05.mma (kind::f16, f32 accumulate).
//
// Persistent: a CTA takes work items (128 weight rows x one token tile x one k slice) blockIdx.x, + gridDim.x, ...  Token
// tiles are equal shares of the block (a.nt <= 256 tokens each, a multiple of 16), the items of one row block side by side,
// so its weights leave HBM once and the other token tiles find them in L2.  Per step of two k blocks (128 columns):
//   warp DQ     (one thread) streams the raw q4 tiles + scales, one tiled copy each (8 row tiles x 2 positions);
//   warp DQ + 1 (one thread) loads the X block [nt tokens x 64] twice with tiled TMA copies (128-byte swizzle);
//   warps 0..DQ-1 expand: three groups of four warps take the steps in turn, a warp the two row tiles of its 32 tensor-memory
//               lanes, and write the f16 A operand straight into tensor memory.  A tile's lane order -- lane (g, t) holds columns
//               4t..4t+3 and 16+4t..16+4t+3 of rows g and g+8 -- is the register order of tcgen05.st.16x256b: nothing is shuffled;
//   warp DQ + 2 issues eight tcgen05.mma (M = 128, N = the tile's tokens, K = 16), A from tensor memory, B from shared memory,
//               and commits the stage back to both producers;
//   warps 0..DQ-1 then read the accumulator with tcgen05.ld (lane quarter = warp % 4, the columns shared out over the groups) and
//               store f32 rows, or apply GeGLU on interleaved gate/up rows and store the f16 input of the down projection.
// Tensor memory: columns [0, 256) accumulator, [256, 448) three A stages of 64 columns.
// What bounds it: the issuing warp (0.32 us per k block of 128 rows x 240 tokens where the products alone take 0.25) and, per item,
// the epilogue; gate/up keeps the tensor pipe busy for 67 % of the active cycles.  12B-class q4_0, 928 tokens in one block: gate/up + GeGLU 168 us (1305 TFLOP/s), down 76 (1432), o 29 (1010),
// qkv 51 (1139).  Against A expanded into shared memory, one CTA per 128 rows x 256 tokens and 16 bulk copies per weight stage
// (four launches): 355, 109, 109 (with k slices) and 96 us.  On the way: one copy per row tile instead of a tiled copy kept the copy thread
// at 115 cycles a copy and every k block at 0.53 us whatever the tile; a barrier pair per k block and operand cost 0.10 us.
// k slices leave their partial sums in separate planes of `out` (matrices with few rows would otherwise fill a fraction of the
// SMs); the consumer adds the planes.
// Every mbarrier wait is bounded; a timeout raises LG_ERR_MBAR_TIMEOUT, the role stops waiting, drains its own copies, and the
// CTA frees its tensor memory and returns.
#pragma once
#include <cuda.h>
#include "lg_kernels.cuh"

#define LG_PF_BM 128
#define LG_PF_BK 64
#define LG_PF_NT 256            // most tokens of a tile (accumulator columns)
#define LG_PF_GROUPS 3          // groups of four expand warps, on steps in turn
#define LG_PF_STAGES 3          // operand stages (A in tensor memory, X in shared memory) behind one pair of barriers: one per group,
                                // so that a stage's phases are observed in order by the same threads
#define LG_PF_SMEM_MAX 232448   // 227 KB: the most dynamic shared memory a CTA can have
#define LG_PF_DQ_WARPS (4 * LG_PF_GROUPS)
#define LG_PF_THREADS ((LG_PF_DQ_WARPS + 3) * 32)
#define LG_PF_MAXN 1024         // tokens of a block: at most the spare rows of a sliding-window ring (RING_SPARE)
#define LG_PF_MAX_RAW 15

enum { LG_PF_STORE = 0, LG_PF_GEGLU = 1 };

struct LgPfGemmArgs {
    int nkp, n_row_tiles;
    int n_tok;                  // valid tokens of the block
    int nt, tok_tiles;          // tokens per tile (the X copy's box), tiles
    int kslices;
    int rs;                     // raw stages: a multiple of LG_PF_GROUPS
    float *out; int ldo;        // STORE: out[slice][tok][ldo]
    size_t part_stride;         // floats between the planes of two k slices
    int n_rows;                 // rows >= n_rows are padding and are not stored
    __half *act; int ld_act;    // GEGLU: act[tok][ld_act], element j = gelu(gate_j) * up_j
    int *err;
};

// raw stage: 8 row tiles x 2 tile positions of nibbles, then their scales, then (q4_K) their {d,dmin}
__host__ __device__ constexpr int pf_raw_stage_bytes(int fmt) { return 8 * 2 * (512 + 64 + (fmt == LG_FMT_Q4_K ? 64 : 0)); }
// raw stages: as many as fit beside the X stages, at most 15 -- the bytes in flight from HBM per SM
__host__ __device__ constexpr int pf_raw_stages(int nt, int fmt) {
    const int n = (LG_PF_SMEM_MAX - 1024 - 512 - LG_PF_STAGES * nt * 256) / pf_raw_stage_bytes(fmt);
    return (n > LG_PF_MAX_RAW ? LG_PF_MAX_RAW : n) / LG_PF_GROUPS * LG_PF_GROUPS;
}
__host__ __device__ constexpr size_t pf_smem_bytes(int nt, int fmt) {
    return 1024 + (size_t)LG_PF_STAGES * nt * 256 + (size_t)pf_raw_stages(nt, fmt) * pf_raw_stage_bytes(fmt) + 512;
}
static_assert(pf_raw_stages(LG_PF_NT, LG_FMT_Q4_K) >= LG_PF_GROUPS, "a raw stage per group");

// two stored nibbles (bytes b0,b1 of `n`, already q = stored ^ 8) -> half2 (q0-8, q1-8) * d
__device__ __forceinline__ uint32_t pf_pair_q4_0(uint32_t n, uint32_t sel, __half2 d2) {
    uint32_t v;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(v) : "r"(n), "r"(0x64646464u), "r"(sel));        // (1024+q0, 1024+q1)
    __half2 h = __hsub2(*(__half2 *)&v, __half2half2(__ushort_as_half((unsigned short)0x6408)));   // - 1032
    h = __hmul2(h, d2);
    return *(uint32_t *)&h;
}
// q4_K: d*sc*q - dmin*m with the two products rounded to f16 first
__device__ __forceinline__ uint32_t pf_pair_q4_K(uint32_t n, uint32_t sel, __half2 dsc2, __half2 negdm2) {
    uint32_t v;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(v) : "r"(n), "r"(0x64646464u), "r"(sel));
    __half2 h = __hsub2(*(__half2 *)&v, __half2half2(__ushort_as_half((unsigned short)0x6400)));   // - 1024 = q
    h = __hfma2(h, dsc2, negdm2);
    return *(uint32_t *)&h;
}

// a CTA's work item `it`: token tiles fastest, then row blocks, then k slices
struct PfItem { int rt0, tok0, n, slice, kb_lo, nkb; };
__device__ __forceinline__ PfItem pf_item(const LgPfGemmArgs &a, int it) {
    PfItem w;
    const int tt = it % a.tok_tiles, rest = it / a.tok_tiles, row_blocks = (a.n_row_tiles + 7) >> 3;
    w.rt0 = (rest % row_blocks) * 8; w.slice = rest / row_blocks;
    w.tok0 = tt * a.nt; w.n = min(a.nt, a.n_tok - w.tok0);
    w.kb_lo = (int)((long long)a.nkp * w.slice / a.kslices);
    w.nkb = (int)((long long)a.nkp * (w.slice + 1) / a.kslices) - w.kb_lo;
    return w;
}
// a ring position and the parity of the pass it is in
struct PfRing {
    int s = 0; uint32_t ph = 0;
    __device__ __forceinline__ void next(int n) { if (++s == n) { s = 0; ph ^= 1; } }
};

template <int FMT, int EPI>
__global__ void __launch_bounds__(LG_PF_THREADS, 1) lg_pf_gemm_kernel(const __grid_constant__ CUtensorMap tmx, const __grid_constant__ CUtensorMap tmq,
                                                                       const __grid_constant__ CUtensorMap tms, const __grid_constant__ CUtensorMap tmd, LgPfGemmArgs a) {
    extern __shared__ unsigned char pf_smem_raw[];
    constexpr int ST = LG_PF_STAGES, NG = LG_PF_GROUPS, RAW = pf_raw_stage_bytes(FMT), DQ = LG_PF_DQ_WARPS;
    static_assert(ST == NG, "a stage belongs to one expand group");
    constexpr int RAW_SC = 16 * 512, RAW_DD = RAW_SC + 16 * 64;
    const int RS = a.rs, B_BYTES = a.nt * 128;
    unsigned char *sB = (unsigned char *)(((uintptr_t)pf_smem_raw + 1023) & ~(uintptr_t)1023), *sRaw = sB + ST * 2 * B_BYTES;
    uint64_t *bars = (uint64_t *)(sRaw + RS * RAW);
    // full[s]: the group's four warps + the bytes of the X copies; empty[s]: one commit frees both operands
    uint64_t *raw_full = bars, *raw_empty = raw_full + RS, *full = raw_empty + RS, *empty = full + ST, *acc_full = empty + ST, *acc_empty = acc_full + 1;
    uint32_t *tmem_slot = (uint32_t *)(acc_empty + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_items = ((a.n_row_tiles + 7) >> 3) * a.tok_tiles * a.kslices;

    if (threadIdx.x == 0) {
        for (int i = 0; i < RS; i++) { mbar_init(raw_full + i, 1); mbar_init(raw_empty + i, 4); }
        for (int i = 0; i < ST; i++) { mbar_init(full + i, 5); mbar_init(empty + i, 1); }
        mbar_init(acc_full, 1); mbar_init(acc_empty, DQ);
    }
    if (warp == DQ + 2) {        // tensor memory: 256 accumulator columns, 3 x 64 columns of weights
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot, tmem_a = tmem + LG_PF_NT;
    pdl_launch();                // only now: a dependant must not take tensor memory a CTA of this grid still waits for

    if (warp == DQ) {
        // ---------------- raw weight producer ----------------
        if (lane == 0) {
            bool ok = true;
            PfRing q;
            int issued = 0;
            for (int it = blockIdx.x; it < n_items && ok; it += gridDim.x) {
                const PfItem w = pf_item(a, it);
                for (int k = 0; k < w.nkb; k += 2) {
                    if (issued >= RS && !mbar_wait(raw_empty + q.s, q.ph ^ 1)) { atomicOr(a.err, LG_ERR_MBAR_TIMEOUT | 2); ok = false; break; }
                    // boxes of 8 row tiles x 2 positions; what lies past the matrix arrives as zeros, what lies past the slice unused
                    unsigned char *st = sRaw + q.s * RAW;
                    mbar_expect_tx(raw_full + q.s, RAW);
                    tma_load_2d(st, &tmq, (w.kb_lo + k) * 128, w.rt0, raw_full + q.s);
                    tma_load_2d(st + RAW_SC, &tms, (w.kb_lo + k) * 16, w.rt0, raw_full + q.s);
                    if (FMT == LG_FMT_Q4_K) tma_load_2d(st + RAW_DD, &tmd, (w.kb_lo + k) * 16, w.rt0, raw_full + q.s);
                    issued++;
                    q.next(RS);
                }
            }
            if (!ok)      // drain: the copies already issued must land before the CTA's shared memory is released
                for (int r = max(0, issued - RS); r < issued; r++) mbar_wait(raw_full + r % RS, (r / RS) & 1);
        }
    } else if (warp == DQ + 1) {
        // ---------------- activation producer ----------------
        if (lane == 0) {
            pdl_wait();
            bool ok = true;
            PfRing q;
            int issued = 0;
            for (int it = blockIdx.x; it < n_items && ok; it += gridDim.x) {
                const PfItem w = pf_item(a, it);
                for (int k = 0; k < w.nkb; k += 2) {
                    if (issued >= ST && !mbar_wait(empty + q.s, q.ph ^ 1)) { atomicOr(a.err, LG_ERR_MBAR_TIMEOUT | 4); ok = false; break; }
                    const int np = min(2, w.nkb - k);
                    mbar_expect_tx(full + q.s, np * B_BYTES);
                    for (int h = 0; h < np; h++)
                        tma_load_2d(sB + (2 * q.s + h) * B_BYTES, &tmx, (w.kb_lo + k + h) * LG_PF_BK, w.tok0, full + q.s);
                    issued++;
                    q.next(ST);
                }
            }
            if (!ok)      // drain; the group's warps may never arrive: the waits are bounded, and far longer than any copy
                for (int r = max(0, issued - ST); r < issued; r++) mbar_wait(full + r % ST, (r / ST) & 1);
        }
    } else if (warp == DQ + 2) {
        // ---------------- MMA issuer ----------------
        // The whole warp walks the loop and one elected thread issues (a lane-0 branch around the loop cost 10 %).  It never waits
        // in a long item: what it does between two steps' products bounds the kernel (a wait that is over costs about 100
        // cycles, a step's products 1024), so the next step's barrier is looked at before this step's products are issued.
        bool ok = true, ready = false;
        PfRing q;
        uint32_t aph = 0;                            // parity of the accumulator's next release
        const uint64_t bdesc0 = umma_desc_k128(smem_u32(sB));
        const uint32_t bstep = (uint32_t)B_BYTES >> 4;
        for (int it = blockIdx.x; it < n_items && ok; it += gridDim.x) {
            const PfItem w = pf_item(a, it);
            const uint32_t idesc = (1u << 4) | ((uint32_t)((w.n + 15) >> 4) << 18) | ((uint32_t)(LG_PF_BM >> 4) << 24);
            if (it != (int)blockIdx.x) {
                ok = mbar_wait(acc_empty, aph);
                aph ^= 1;
            }
            for (int k = 0; k < w.nkb; k += 2) {
                if (ok && !ready) ok = mbar_wait(full + q.s, q.ph);
                if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t ad = tmem_a + q.s * 64, done = smem_u32(empty + q.s);
                const uint64_t bd = bdesc0 + 2 * q.s * bstep;
                q.next(ST);
                ready = mbar_test(full + q.s, q.ph);
                if (elect_one()) {
                    #pragma unroll
                    for (int j = 0; j < 4; j++) umma_f16_ta(tmem, ad + 8 * j, bd + 2 * j, idesc, k | j);
                    if (k + 1 < w.nkb) {
                        #pragma unroll
                        for (int j = 0; j < 4; j++) umma_f16_ta(tmem, ad + 32 + 8 * j, bd + bstep + 2 * j, idesc, 1);
                    }
                    umma_commit_u32(done);
                }
                __syncwarp();
            }
            if (!ok && lane == 0) atomicOr(a.err, LG_ERR_MBAR_TIMEOUT | 8);
            if (elect_one()) umma_commit(acc_full);  // arrives when every MMA above has completed
            __syncwarp();
        }
    } else {
        // ---------------- expand q4 -> f16 A operand in tensor memory, then the epilogue ----------------
        const int g = lane >> 2, lq = warp & 3, grp = warp >> 2;        // lane quarter, expand group
        const uint32_t raw0 = smem_u32(sRaw) + lane * 16;
        const uint32_t rsc0 = smem_u32(sRaw) + RAW_SC + g * 8, rdd0 = smem_u32(sRaw) + RAW_DD + g * 8;
        const uint32_t lanes = (uint32_t)(lq * 32) << 16;
        bool ok = true;
        int step = 0;                                // steps of the items before this one and of this one so far
        int rs = grp; uint32_t rph = 0, sph = 1;     // this group's raw stage and its parity; parity of the operand stage's release
        uint32_t cph = 0;
        for (int it = blockIdx.x; it < n_items && ok; it += gridDim.x) {
            const PfItem w = pf_item(a, it);
            for (int k = 0; k < w.nkb; k += 2, step++) {
                if (step % NG != grp) continue;
                const int np = min(2, w.nkb - k);
                if (!mbar_wait(raw_full + rs, rph)) { ok = false; atomicOr(a.err, LG_ERR_MBAR_TIMEOUT | 32); }
                if (ok && step >= ST && !mbar_wait(empty + grp, sph)) { ok = false; atomicOr(a.err, LG_ERR_MBAR_TIMEOUT | 64); }
                sph ^= 1;
                if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                #pragma unroll
                for (int h = 0; h < 2; h++) {
                    if (h >= np) break;
                    #pragma unroll
                    for (int j = 0; j < 2; j++) {
                        const int ti = lq * 2 + j;                                         // row tile of the CTA's 8
                        const uint32_t roff = rs * RAW + ti * 1024 + h * 512, soff = rs * RAW + ti * 128 + h * 64;
                        uint4 wv; uint2 sc, dd = make_uint2(0, 0);
                        asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(wv.x), "=r"(wv.y), "=r"(wv.z), "=r"(wv.w) : "r"(raw0 + roff));
                        asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(sc.x), "=r"(sc.y) : "r"(rsc0 + soff));
                        if (FMT == LG_FMT_Q4_K) asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(dd.x), "=r"(dd.y) : "r"(rdd0 + soff));
                        uint32_t v[16];                                                    // [16 columns][row g: 2, row g + 8: 2]
                        #pragma unroll
                        for (int sbk = 0; sbk < 2; sbk++)
                            #pragma unroll
                            for (int h8 = 0; h8 < 2; h8++) {
                                const uint32_t word = sbk ? (h8 ? wv.w : wv.z) : (h8 ? wv.y : wv.x);
                                const uint32_t sw = sbk ? sc.y : sc.x;
                                const uint32_t lo = (word & 0x0F0F0F0Fu) ^ 0x08080808u, hi = ((word >> 4) & 0x0F0F0F0Fu) ^ 0x08080808u;
                                uint32_t *vl = v + 8 * sbk + 2 * h8, *vh = vl + 4;
                                if (FMT == LG_FMT_Q4_0) {
                                    uint32_t dbits;                                        // the row's scale in both halves
                                    asm("prmt.b32 %0, %1, %1, %2;" : "=r"(dbits) : "r"(sw), "r"(h8 ? 0x3232u : 0x1010u));
                                    const __half2 d2 = *(const __half2 *)&dbits;
                                    vl[0] = pf_pair_q4_0(lo, 0x4140u, d2); vl[1] = pf_pair_q4_0(lo, 0x4342u, d2);
                                    vh[0] = pf_pair_q4_0(hi, 0x4140u, d2); vh[1] = pf_pair_q4_0(hi, 0x4342u, d2);
                                } else {
                                    const uint32_t sm = h8 ? (sw >> 16) : (sw & 0xffff);
                                    const float2 dm = __half22float2(*(const __half2 *)(h8 ? &dd.y : &dd.x));
                                    const __half2 dsc2 = __float2half2_rn(dm.x * (float)(sm & 0xff));
                                    const __half2 ndm2 = __float2half2_rn(-dm.y * (float)(sm >> 8));
                                    vl[0] = pf_pair_q4_K(lo, 0x4140u, dsc2, ndm2); vl[1] = pf_pair_q4_K(lo, 0x4342u, dsc2, ndm2);
                                    vh[0] = pf_pair_q4_K(hi, 0x4140u, dsc2, ndm2); vh[1] = pf_pair_q4_K(hi, 0x4342u, dsc2, ndm2);
                                }
                            }
                        tmem_st_16x256b_x4(tmem_a + grp * 64 + h * 32 + lanes + ((uint32_t)j << 20), v);
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(raw_empty + rs);
                tmem_wait_st();
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(full + grp);
                rs += NG;
                if (rs >= RS) { rs = grp; rph ^= 1; }
            }

            // ---------------- epilogue: lane l of warp w holds accumulator row 32 (w % 4) + l ----------------
            if (ok && !mbar_wait(acc_full, cph)) { ok = false; atomicOr(a.err, LG_ERR_MBAR_TIMEOUT | 128); }
            cph ^= 1;
            if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int lrow = lq * 32 + lane, rt = w.rt0 + (lrow >> 4);       // row within the CTA's 128
            float *outp = a.out + (size_t)w.slice * a.part_stride + (size_t)w.tok0 * a.ldo + w.rt0 * 16 + lrow;
            const bool row_ok = rt < a.n_row_tiles && w.rt0 * 16 + lrow < a.n_rows;
            for (int c0 = grp * 32; c0 < w.n; c0 += NG * 32) {               // uniform per warp
                uint32_t v[32];
                tmem_ld32(tmem + lanes + c0, v);
                if (EPI == LG_PF_STORE) {
                    if (row_ok) {
                        #pragma unroll
                        for (int j = 0; j < 32; j++)
                            if (c0 + j < w.n) outp[(size_t)(c0 + j) * a.ldo] = __uint_as_float(v[j]);
                    }
                } else {
                    // tile rows 0-7 are gate rows, rows 8-15 the matching up rows: lane l pairs with lane l + 8.  Of two tokens
                    // the gate lane takes the even one and the up lane the odd one: one exchange, one GeLU and one store each.
                    const int r16 = lrow & 15, upper = r16 >> 3;
                    __half *ap = a.act + (size_t)(w.tok0 + c0 + upper) * a.ld_act + rt * 8 + (r16 & 7);
                    #pragma unroll
                    for (int j = 0; j < 32; j += 2) {
                        const float e = __uint_as_float(v[j]), o = __uint_as_float(v[j + 1]);
                        const float got = __shfl_xor_sync(0xffffffffu, upper ? e : o, 8);
                        const float gate = upper ? got : e, up = upper ? o : got;
                        if (rt < a.n_row_tiles && c0 + j + upper < w.n)
                            ap[(size_t)j * a.ld_act] = __float2half_rn(__fmul_rn(gelu_tanh(gate), up));
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(acc_empty);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == DQ + 2) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(512) : "memory");
    }
}

// y = gelu_tanh(sum of the planes of gate) * up as f16 rows (per-layer-embedding gate of a prompt block)
__global__ void lg_pf_geglu_rows(const float *__restrict__ gate, const float *__restrict__ up, int ld_g, int ld_u, int n,
                                 __half *__restrict__ out, int ld_out, int n_parts, size_t part_stride) {
    pdl_launch(); pdl_wait();
    const int tok = blockIdx.y;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float v = gate[(size_t)tok * ld_g + i];
        for (int p = 1; p < n_parts; p++) v += gate[(size_t)p * part_stride + (size_t)tok * ld_g + i];
        out[(size_t)tok * ld_out + i] = __float2half_rn(__fmul_rn(gelu_tanh(v), up[(size_t)tok * ld_u + i]));
    }
}

// Media positions of a prompt block: x[tok] = rows[ridx[tok]] where ridx[tok] >= 0 (the row replaces the token embedding as it is)
__global__ void lg_inject_rows(float *__restrict__ x, int ldx, const float *__restrict__ rows, const int *__restrict__ ridx, int n) {
    pdl_launch(); pdl_wait();
    const int tok = blockIdx.x, r = ridx[tok];
    if (r < 0) return;
    for (int i = threadIdx.x; i < n; i += blockDim.x) x[(size_t)tok * ldx + i] = rows[(size_t)r * n + i];
}

// The residual update and the norm of a prompt block's rows, one CTA per token with the row in registers (V groups of four
// elements a thread), n a multiple of 4 and at most 4 V blockDim.x: x += rmsnorm(sum of the planes of add) * add_w, x *= out_scale;
// yh = rmsnorm(x) * norm_w, or x itself, as f16.  Bound by memory traffic and the two sums over the block; 928 rows of 3840: 33 us with the row in shared
// memory and three barriers per sum, 14 us now.
struct LgPfNormArgs {
    float *x;
    const float *add; int n_parts; size_t part_stride; int ld_add;
    const float *add_w; float out_scale;
    const float *norm_w;
    __half *yh;
    int n; float eps;
};
__device__ __forceinline__ float pf_block_sum(float v, float *red) {        // red: one float per warp, a buffer of its own per sum
    v = warp_sum(v);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    const int nw = blockDim.x >> 5;
    return warp_sum((int)(threadIdx.x & 31) < nw ? red[threadIdx.x & 31] : 0.0f);
}
template <int V>
__global__ void __launch_bounds__(512) lg_pf_norm_kernel(LgPfNormArgs a) {
    __shared__ float red[2][32];
    const int tok = blockIdx.x, n4 = a.n >> 2;
    float4 aw[V], nw[V], x[V], o[V];
    pdl_launch();
    #pragma unroll
    for (int k = 0; k < V; k++) {                          // the weights do not depend on the previous kernel
        const int i = threadIdx.x + k * blockDim.x;
        aw[k] = nw[k] = x[k] = o[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (i < n4 && a.add) aw[k] = ((const float4 *)a.add_w)[i];
        if (i < n4 && a.norm_w) nw[k] = ((const float4 *)a.norm_w)[i];
    }
    pdl_wait();
    float4 *row = (float4 *)(a.x + (size_t)tok * a.n);
    const float *src = a.add + (size_t)tok * a.ld_add;
    float ss = 0.0f;
    #pragma unroll
    for (int k = 0; k < V; k++) {
        const int i = threadIdx.x + k * blockDim.x;
        if (i >= n4) continue;
        x[k] = row[i];
        if (!a.add) continue;
        for (int p = 0; p < a.n_parts; p++) {
            const float4 t = ((const float4 *)(src + (size_t)p * a.part_stride))[i];
            o[k].x += t.x; o[k].y += t.y; o[k].z += t.z; o[k].w += t.w;
        }
        ss += o[k].x * o[k].x + o[k].y * o[k].y + o[k].z * o[k].z + o[k].w * o[k].w;
    }
    if (a.add) {
        const float s = 1.0f / sqrtf(pf_block_sum(ss, red[0]) / (float)a.n + a.eps);
        auto upd = [&](float x, float o, float w) { return __fmul_rn(__fadd_rn(x, __fmul_rn(__fmul_rn(o, s), w)), a.out_scale); };
        #pragma unroll
        for (int k = 0; k < V; k++) {
            const int i = threadIdx.x + k * blockDim.x;
            if (i >= n4) continue;
            x[k] = make_float4(upd(x[k].x, o[k].x, aw[k].x), upd(x[k].y, o[k].y, aw[k].y), upd(x[k].z, o[k].z, aw[k].z), upd(x[k].w, o[k].w, aw[k].w));
            row[i] = x[k];
        }
    }
    if (!a.yh) return;
    float s = 1.0f;
    if (a.norm_w) {
        ss = 0.0f;
        #pragma unroll
        for (int k = 0; k < V; k++) ss += x[k].x * x[k].x + x[k].y * x[k].y + x[k].z * x[k].z + x[k].w * x[k].w;
        s = 1.0f / sqrtf(pf_block_sum(ss, red[1]) / (float)a.n + a.eps);
    }
    auto y = [&](float x, float w) { return a.norm_w ? __fmul_rn(__fmul_rn(x, s), w) : x; };
    #pragma unroll
    for (int k = 0; k < V; k++) {
        const int i = threadIdx.x + k * blockDim.x;
        if (i >= n4) continue;
        const __half2 h0 = __floats2half2_rn(y(x[k].x, nw[k].x), y(x[k].y, nw[k].y)), h1 = __floats2half2_rn(y(x[k].z, nw[k].z), y(x[k].w, nw[k].w));
        ((uint2 *)(a.yh + (size_t)tok * a.n))[i] = make_uint2(*(const uint32_t *)&h0, *(const uint32_t *)&h1);
    }
}

// f32 rows -> f16 rows (the B operand of the wide matmul)
__global__ void lg_f32_to_f16_rows(const float *__restrict__ src, int ld_src, __half *__restrict__ dst, int ld_dst, int n) {
    pdl_launch(); pdl_wait();
    const int tok = blockIdx.y;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        dst[(size_t)tok * ld_dst + i] = __float2half_rn(src[(size_t)tok * ld_src + i]);
}

// ---------------------------------------------------------------------------------------------
// attention of a prompt block: all query rows of the block in one launch per layer
// ---------------------------------------------------------------------------------------------
// Step 1 (lg_pf_qkv_prep_kernel): per token, per-head RMSNorm + NeoX RoPE of the raw projection
// rows.  Queries go to an f16 hi + lo pair [kv head][tok][query heads of it][hd]; K (norm + rope) and V (plain norm) rows go
// to the f16 cache of the owning layer (round to nearest even) at row (pos % seq).  The cache ring
// of a sliding-window layer has at least as many spare rows as a block has tokens, so writing the whole block
// first does not overwrite a row an earlier query of the block still attends to.
struct LgPfPrepArgs {
    const float *qkv; int ld;            // [n][ld] = [q (H*hd) | k (Hkv*hd) | v (Hkv*hd)], the sum of n_parts planes
    int n_parts; size_t part_stride;
    int has_v, owns_kv;
    const float *q_norm, *k_norm; float eps;
    const float2 *rope;                  // [n][hd/2]
    __half *kc, *vc; int seq, kv_dim;
    int H, Hkv;
    const int *pos;                      // position of the block's first token
    __half *q_hi, *q_lo;                 // [Hkv][n][H / Hkv][hd]
};

// One head vector per warp, PER consecutive elements of each half a lane; the norm weights do not depend on the previous kernel
// and are fetched before the wait.  Bound by its memory traffic (928 tokens of a 12B-class layer: 53 MB); wide loads and stores
// instead of one element at a time: 22 -> 15 us.
template <int N> struct PfVec;
template <> struct PfVec<1> { typedef float F; typedef uint16_t H; };
template <> struct PfVec<2> { typedef float2 F; typedef uint32_t H; };
template <> struct PfVec<4> { typedef float4 F; typedef uint2 H; };
template <int N> __device__ __forceinline__ void pf_load(const float *p, float (&v)[N]) { *(typename PfVec<N>::F *)v = *(const typename PfVec<N>::F *)p; }
template <int N> __device__ __forceinline__ void pf_store(__half *p, const __half (&h)[N]) { *(typename PfVec<N>::H *)p = *(const typename PfVec<N>::H *)h; }

template <int HD>
__global__ void __launch_bounds__(256) lg_pf_qkv_prep_kernel(LgPfPrepArgs a) {
    constexpr int PER = HD / 64, HALF = HD / 2;
    const int tok = blockIdx.x, lane = threadIdx.x & 31, j = blockIdx.y * 8 + (threadIdx.x >> 5), i0 = lane * PER;
    const int jj = j - a.H, isv = jj >= a.Hkv, kvh = isv ? jj - a.Hkv : jj;
    const bool live = j < a.H + (a.owns_kv ? 2 * a.Hkv : 0);
    const float *w = j < a.H ? a.q_norm : isv ? nullptr : a.k_norm;
    alignas(16) float w0[PER], w1[PER], v0[PER], v1[PER];
    #pragma unroll
    for (int e = 0; e < PER; e++) w0[e] = w1[e] = 1.0f;
    pdl_launch();
    if (live && w) { pf_load(w + i0, w0); pf_load(w + i0 + HALF, w1); }
    pdl_wait();
    if (!live) return;
    const int p = *a.pos + tok;
    const float *src = a.qkv + (size_t)tok * a.ld + (size_t)(j < a.H ? j : a.H + ((isv && a.has_v) ? a.Hkv : 0) + kvh) * HD + i0;
    pf_load(src, v0); pf_load(src + HALF, v1);
    float2 cs[PER];
    #pragma unroll
    for (int e = 0; e < PER; e++) cs[e] = isv ? make_float2(1.0f, 0.0f) : a.rope[(size_t)tok * HALF + i0 + e];
    for (int q = 1; q < a.n_parts; q++) {                                   // the k-slice planes, in order
        alignas(16) float t0[PER], t1[PER];
        pf_load(src + (size_t)q * a.part_stride, t0); pf_load(src + (size_t)q * a.part_stride + HALF, t1);
        #pragma unroll
        for (int e = 0; e < PER; e++) { v0[e] += t0[e]; v1[e] += t1[e]; }
    }
    float ss = 0.0f;
    #pragma unroll
    for (int e = 0; e < PER; e++) ss += v0[e] * v0[e] + v1[e] * v1[e];
    const float sc = 1.0f / sqrtf(warp_sum(ss) / (float)HD + a.eps);
    alignas(8) __half h0[PER], h1[PER];
    #pragma unroll
    for (int e = 0; e < PER; e++) {
        float x = __fmul_rn(__fmul_rn(v0[e], sc), w0[e]), y = __fmul_rn(__fmul_rn(v1[e], sc), w1[e]);
        if (!isv) {
            const float r0 = __fsub_rn(__fmul_rn(x, cs[e].x), __fmul_rn(y, cs[e].y));
            y = __fadd_rn(__fmul_rn(x, cs[e].y), __fmul_rn(y, cs[e].x));
            x = r0;
        }
        v0[e] = x; v1[e] = y;
        h0[e] = __float2half_rn(x); h1[e] = __float2half_rn(y);
    }
    if (j < a.H) {
        const int gqa = a.H / a.Hkv;
        const size_t qrow = (((size_t)(j / gqa) * gridDim.x + tok) * gqa + j % gqa) * HD + i0;
        pf_store(a.q_hi + qrow, h0); pf_store(a.q_hi + qrow + HALF, h1);
        #pragma unroll
        for (int e = 0; e < PER; e++) { h0[e] = __float2half_rn(v0[e] - __half2float(h0[e])); h1[e] = __float2half_rn(v1[e] - __half2float(h1[e])); }
        pf_store(a.q_lo + qrow, h0); pf_store(a.q_lo + qrow + HALF, h1);
    } else {
        __half *dst = (isv ? a.vc : a.kc) + (size_t)(p % a.seq) * a.kv_dim + (size_t)kvh * HD + i0;
        pf_store(dst, h0); pf_store(dst + HALF, h1);
    }
}

// Step 2 (lg_pf_attn_kernel): one CTA = one KV head x 128 query rows (the TMEM lanes; 128 / gqa consecutive tokens x the gqa
// query heads of that KV head), longest rows first.  It walks the keys of its causal / sliding window in tiles of 64 with an
// online softmax, S = Q K^T and O += P V on tcgen05 (f16 operands, f32 accumulation in tensor memory), Q and P as f16 hi + lo
// pairs like the decode kernel, scale 1.0.
//   warp 4  copies the two query blocks, then key and value tiles in the order the products take them, through three slots;
//           rows behind the last position written so far hold whatever was there: their values are zeroed in the last tile;
//   warp 5  issues the products: S(i + 1) into one of two 64-column buffers while tile i is in its softmax, then O += P(i) V
//           with P from tensor memory and V as it lies in the cache (an MN-major operand);
//   warps 0-3  one query row per thread: scores from tensor memory, softmax in f32, the weights back over the scores.  O is
//           rescaled only when a row's maximum has grown by more than LG_PFA_SLACK since the one in use (until then weights
//           are merely larger than 1), which needs the previous product to have finished.
// Scores of two tiles may be finished before the first one's weights are used, so the buffers have barriers of their own.
// What bounds it: the products of a row block's tiles and the softmax between them, about 1.8 us a tile of 64 keys at head size 256
// (the products alone: 1.1 us).  In a serialised launch list: 12B-class layer, 928 tokens from position 0, 36.6 us (mma.sync, 32 rows
// per CTA: 165); E4B-class layer, 48 tokens behind 701, 26 us on 4 CTAs.  The weights by ex2.approx of log2(e) s - m: 35.6 and 24.4 us,
// but up to 2 % more error in a row's weights (scores within 0 .. 300 +- 16) and none below 2^-126; expf stays.
struct LgPfAttnArgs {
    int seq, H, Hkv, n;
    int window;                          // <= 0: full causal
    const int *pos;
    __half *out; int ld_out;             // [n][ld_out], head hq at column hq*hd
    int *err;
};
#define LG_PFA_Q 128
#define LG_PFA_S 64
#define LG_PFA_SLOTS 3
#define LG_PFA_THREADS 192
#define LG_PFA_SLACK 5.5f
template <int HD> constexpr size_t pf_attn_smem() { return 1024 + (size_t)HD / 64 * (2 * LG_PFA_Q + LG_PFA_SLOTS * LG_PFA_S) * 128 + 256; }

template <int HD>
__global__ void __launch_bounds__(LG_PFA_THREADS, 1)
lg_pf_attn_kernel(const __grid_constant__ CUtensorMap tmqh, const __grid_constant__ CUtensorMap tmql, const __grid_constant__ CUtensorMap tmk,
                  const __grid_constant__ CUtensorMap tmv, LgPfAttnArgs a) {
    extern __shared__ __align__(16) unsigned char pfa_smem[];
    constexpr int NB = HD / 64, S = LG_PFA_S, SL = LG_PFA_SLOTS, Q_BLK = LG_PFA_Q * 128, T_BLK = S * 128, SLOT = NB * T_BLK;
    constexpr uint32_t TCOLS = 2 * S + HD <= 256 ? 256 : 512;            // scores / weights twice 64 columns, output HD
    unsigned char *sQ = (unsigned char *)(((uintptr_t)pfa_smem + 1023) & ~(uintptr_t)1023), *sT = sQ + 2 * NB * Q_BLK;
    uint64_t *qfull = (uint64_t *)(sT + SL * SLOT), *full = qfull + 1, *empty = full + SL, *sfull = empty + SL /* two */,
             *pready = sfull + 2 /* two */, *odone = pready + 2 /* two */, *vfix = odone + 2;
    uint32_t *tmem_slot = (uint32_t *)(vfix + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        mbar_init(qfull, 1); mbar_init(vfix, 1);
        for (int i = 0; i < SL; i++) { mbar_init(full + i, 1); mbar_init(empty + i, 1); }
        for (int i = 0; i < 2; i++) { mbar_init(sfull + i, 1); mbar_init(pready + i, 4); mbar_init(odone + i, 1); }
    }
    if (warp == 5) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(tmem_slot)), "r"(TCOLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot, tO = tmem + 2 * S;
    pdl_launch();                        // only now: a dependant must not take tensor memory a CTA of this grid still waits for
    pdl_wait();

    const int kvh = blockIdx.y, gqa = a.H / a.Hkv, qb = LG_PFA_Q / gqa;                 // qb tokens per CTA
    const int t0 = (gridDim.x - 1 - blockIdx.x) * qb, nt = min(qb, a.n - t0);           // its valid tokens
    const int pos0 = *a.pos, p_last = pos0 + t0 + nt - 1;
    const int k_first = (a.window > 0 ? max(0, pos0 + t0 - a.window + 1) : 0) / S * S;
    const int n_tiles = (p_last - k_first) / S + 1;
    const int v_stale = pos0 + a.n - (k_first + (n_tiles - 1) * S);                     // first unwritten row of the last tile

    if (warp == 4) {
        bool ok = true;
        int issued = 0;
        PfRing q;
        if (lane == 0) {
            mbar_expect_tx(qfull, 2 * NB * Q_BLK);
            const int row = (kvh * a.n + t0) * gqa;
            for (int c = 0; c < NB; c++) {
                tma_load_2d(sQ + c * Q_BLK, &tmqh, c * 64, row, qfull);
                tma_load_2d(sQ + (NB + c) * Q_BLK, &tmql, c * 64, row, qfull);
            }
            // K0, K1, V0, K2, V1, ..
            for (int u = 0; u < 2 * n_tiles; u++) {
                const bool is_v = u == 2 * n_tiles - 1 || (u >= 2 && !(u & 1));
                const int i = u == 0 ? 0 : is_v ? (u == 2 * n_tiles - 1 ? n_tiles - 1 : u / 2 - 1) : (u + 1) / 2;
                if (issued >= SL && !mbar_wait(empty + q.s, q.ph ^ 1)) { atomicOr(a.err, LG_ERR_MBAR_TIMEOUT | 4); ok = false; break; }
                mbar_expect_tx(full + q.s, SLOT);
                const int r = (k_first + i * S) % a.seq;
                for (int c = 0; c < NB; c++) tma_load_2d(sT + q.s * SLOT + c * T_BLK, is_v ? &tmv : &tmk, kvh * HD + c * 64, r, full + q.s);
                issued++;
                if (u != 2 * n_tiles - 1) q.next(SL);
            }
            if (!ok) {           // own copies in flight land before the CTA ends
                mbar_wait(qfull, 0);
                for (int r = max(0, issued - SL); r < issued; r++) mbar_wait(full + r % SL, (r / SL) & 1);
            }
        }
        if (v_stale < S) {
            const int slot = __shfl_sync(0xffffffffu, q.s, 0), ph = __shfl_sync(0xffffffffu, (int)q.ph, 0);
            ok = __shfl_sync(0xffffffffu, (int)ok, 0) && mbar_wait(full + slot, ph);
            if (__all_sync(0xffffffffu, ok)) {
                for (int c = lane; c < NB * (S - v_stale) * 8; c += 32) {       // a row's 16-byte chunks stay within its 128 bytes
                    const int b = c / ((S - v_stale) * 8), rest = c % ((S - v_stale) * 8);
                    *(uint4 *)(sT + slot * SLOT + b * T_BLK + v_stale * 128 + rest * 16) = make_uint4(0, 0, 0, 0);
                }
                fence_async_shared();
                __syncwarp();
                if (lane == 0) mbar_arrive(vfix);
            }
        }
    } else if (warp == 5) {
        // f32 accumulator, f16 x f16; N = keys of a tile / value columns
        const uint32_t fmt = (1u << 4) | ((uint32_t)(LG_PFA_Q >> 4) << 24);
        const uint32_t idS = fmt | ((uint32_t)(S >> 3) << 17), idO = fmt | ((uint32_t)(HD >> 3) << 17) | LG_UMMA_B_MN;
        const uint64_t qd = umma_desc_k128(smem_u32(sQ)), kd0 = umma_desc_k128(smem_u32(sT)), vd0 = umma_desc_mn128(smem_u32(sT), T_BLK);
        PfRing q;
        bool ok = mbar_wait(qfull, 0);
        auto scores = [&](int i) {
            if (!__all_sync(0xffffffffu, mbar_wait(full + q.s, q.ph))) return false;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t tS = tmem + (i & 1) * S;
            const uint64_t kd = kd0 + q.s * (SLOT >> 4);
            if (elect_one()) {
                #pragma unroll
                for (int part = 0; part < 2; part++)
                    #pragma unroll
                    for (int c = 0; c < NB; c++)
                        #pragma unroll
                        for (int j = 0; j < 4; j++)
                            umma_f16(tS, qd + (part * NB + c) * (Q_BLK >> 4) + 2 * j, kd + c * (T_BLK >> 4) + 2 * j, idS, part | c | j);
                umma_commit(empty + q.s);
                umma_commit(sfull + (i & 1));
            }
            __syncwarp();
            q.next(SL);
            return true;
        };
        ok = __all_sync(0xffffffffu, ok) && scores(0);
        for (int i = 0; i < n_tiles && ok; i++) {
            if (i + 1 < n_tiles) ok = scores(i + 1);
            ok = ok && mbar_wait(pready + (i & 1), (i >> 1) & 1) && mbar_wait(full + q.s, q.ph);
            if (ok && i == n_tiles - 1 && v_stale < S) ok = mbar_wait(vfix, 0);
            if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t tP = tmem + (i & 1) * S;
            const uint64_t vd = vd0 + q.s * (SLOT >> 4);
            if (elect_one()) {
                #pragma unroll
                for (int j = 0; j < 4; j++) umma_f16_ta(tO, tP + 8 * j, vd + j * 128, idO, i | j);
                #pragma unroll
                for (int j = 0; j < 4; j++) umma_f16_ta(tO, tP + 32 + 8 * j, vd + j * 128, idO, 1u);
                umma_commit(empty + q.s);
                umma_commit(odone + (i & 1));
            }
            __syncwarp();
            q.next(SL);
        }
        if (!ok && lane == 0) atomicOr(a.err, LG_ERR_MBAR_TIMEOUT | 8);
    } else {
        const int r = threadIdx.x, tok = t0 + r / gqa, hq = kvh * gqa + r % gqa;
        const bool rv = r / gqa < nt;
        const int pj = rv ? pos0 + tok : -1, lo = rv && a.window > 0 ? max(0, pj - a.window + 1) : 0;       // keys lo .. pj
        // every row of the warp sees keys all_lo .. all_hi
        const int all_lo = __reduce_max_sync(0xffffffffu, lo), all_hi = __reduce_min_sync(0xffffffffu, pj);
        const uint32_t lanes = (uint32_t)(warp * 32) << 16;
        float m = -INFINITY, l = 0.0f;
        bool ok = true;
        for (int i = 0; i < n_tiles; i++) {
            const int k0 = k_first + i * S;
            ok = __all_sync(0xffffffffu, mbar_wait(sfull + (i & 1), (i >> 1) & 1));
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t tS = tmem + lanes + (i & 1) * S;
            uint32_t s0[32], s1[32];
            tmem_ld32(tS, s0);
            tmem_ld32(tS + 32, s1);
            float mx = -INFINITY;
            if (k0 < all_lo || k0 + S - 1 > all_hi) {
                #pragma unroll
                for (int j = 0; j < 32; j++) {
                    const int k = k0 + j;
                    if (k < lo || k > pj) s0[j] = 0xff800000u;
                    if (k + 32 < lo || k + 32 > pj) s1[j] = 0xff800000u;
                }
            }
            #pragma unroll
            for (int j = 0; j < 32; j++) mx = fmaxf(mx, fmaxf(__uint_as_float(s0[j]), __uint_as_float(s1[j])));
            const bool grow = mx > m + LG_PFA_SLACK;             // from -inf: as soon as the row sees a key
            if (__any_sync(0xffffffffu, grow)) {
                const float m_new = fmaxf(m, mx), alpha = m == -INFINITY ? 0.0f : expf(m - m_new);
                if (i) {
                    ok = __all_sync(0xffffffffu, mbar_wait(odone + ((i - 1) & 1), ((i - 1) >> 1) & 1));
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    for (int c = 0; c < HD; c += 32) {
                        uint32_t o[32];
                        tmem_ld32(tO + lanes + c, o);
                        #pragma unroll
                        for (int j = 0; j < 32; j++) o[j] = __float_as_uint(__uint_as_float(o[j]) * alpha);
                        tmem_st32(tO + lanes + c, o);
                    }
                    tmem_wait_st();
                }
                l *= alpha; m = m_new;
            }
            const float mu = m == -INFINITY ? 0.0f : m;          // nothing seen yet: every weight is e^-inf
            #pragma unroll
            for (int half = 0; half < 2; half++) {
                uint32_t hi[16], lw[16];
                #pragma unroll
                for (int j = 0; j < 16; j++) {
                    const float x = __uint_as_float(half ? s1[2 * j] : s0[2 * j]), y = __uint_as_float(half ? s1[2 * j + 1] : s0[2 * j + 1]);
                    const float p = expf(x - mu), w = expf(y - mu);
                    l += p + w;
                    const __half2 h = __floats2half2_rn(p, w);
                    const float2 f = __half22float2(h);
                    const __half2 d = __floats2half2_rn(p - f.x, w - f.y);
                    hi[j] = *(const uint32_t *)&h; lw[j] = *(const uint32_t *)&d;
                }
                tmem_st16(tS + 16 * half, hi);
                tmem_st16(tS + 32 + 16 * half, lw);
            }
            tmem_wait_st();
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(pready + (i & 1));
        }
        ok = __all_sync(0xffffffffu, ok && mbar_wait(odone + ((n_tiles - 1) & 1), ((n_tiles - 1) >> 1) & 1));
        if (!ok && lane == 0) atomicOr(a.err, LG_ERR_MBAR_TIMEOUT | 32);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const float inv = l > 0.0f ? 1.0f / l : 0.0f;
        if (ok)
            for (int c = 0; c < HD; c += 32) {
                uint32_t o[32];
                tmem_ld32(tO + lanes + c, o);
                if (rv) {
                    uint4 *dst = (uint4 *)(a.out + (size_t)tok * a.ld_out + (size_t)hq * HD + c);
                    #pragma unroll
                    for (int j = 0; j < 4; j++) {
                        auto two = [&](int k) { const __half2 h = __floats2half2_rn(__uint_as_float(o[8 * j + k]) * inv, __uint_as_float(o[8 * j + k + 1]) * inv); return *(const uint32_t *)&h; };
                        dst[j] = make_uint4(two(0), two(2), two(4), two(6));
                    }
                }
                __syncwarp();
            }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
    __syncthreads();
    if (warp == 5) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(TCOLS) : "memory");
    }
}
