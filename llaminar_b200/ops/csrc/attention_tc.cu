// Paged causal GQA prefill attention on the 5th-generation tensor cores (head_dim 128).
//
// One CTA = two slots of 128 query rows that share a K/V head: two query heads of its group, or two query tiles where the group
// is odd.  Both slots walk the same keys in tiles of 128 (two 64-token pages); each goes through
//   S = Q K^T          tcgen05.mma, M = 128 query rows, N = 128 keys, K = head_dim, fp32 accumulator in TMEM
//   softmax            one thread per query row (== TMEM lane): the 128 scores of a tile pass through its registers once, so row
//                      maximum and row sum need no exchange; P = exp2(...) goes back as bf16 into the columns of S
//   O += P V           tcgen05.mma, M = 128 query rows, N = head_dim, K = 128 keys, A = P from TMEM.  O stays in TMEM and is
//                      rescaled only when a row's maximum rises by more than 2^RESCALE_STEP (P then stays below that; a bf16 P and
//                      fp32 sums have the same relative error at either scale).
// While the softmax warps of one slot work, the tensor core has the other slot's products: that, one copy of K and V for both
// slots, and the absence of shared-memory passes over P and V are what the split is for.  What bounds it: the chain S -> softmax ->
// P V of a slot; the exponentials alone (16 per clock and SM) are 2048 clocks per tile of both slots, the products as many.
// K and V pages arrive by TMA.  Every operand is a 128-byte-swizzled tile; V is read as it lies in the page (rows of head_dim
// values), as an MN-major B operand.
//
// Measured (32 query / 8 key heads, us; in brackets one 128-row tile per CTA with V transposed by loader warps and O in registers, then
// the mma.sync kernel of attention.cu): 2048 rows 62 (128, 246), 4096 rows 164 (374, 785; now 837 TFLOP/s, 1004 with 64 heads),
// 8 x 1020 rows 125 (287, 424), 500 rows behind 7000 tokens 120 (155, 414), 37 rows 8.8 (11.2, 10.5).
//
// Roles (384 threads): warps 0-3 and 4-7 softmax and output of slot 0 and 1, warp 8 TMA, warp 9 TMEM allocation + MMA issue; warps 10
// and 11 complete the third warpgroup, which hands most of its registers to the other two.
// Every mbarrier wait is bounded; on a timeout the kernel raises the status word and tears down cleanly.
//
// Replaces flash_attention_2_pipelined_kernel of the reference (src/v2/kernels/cuda/attention/CUDAFlashAttentionKernels.cu:348).
#include "launch.h"
#include "ops.h"
#include "tc_tile.cuh"

namespace llm {
namespace atc {
using namespace tc5;

constexpr int D = 128, BQ = 128, BK = 128, PAGE = 64, SLOTS = 2;
constexpr int THREADS = 384;
constexpr int REGS_LAUNCH = 168, REGS_SOFTMAX = 232, REGS_OTHER = 40;       // per thread; three warpgroups
static_assert(2 * REGS_SOFTMAX + REGS_OTHER <= 3 * REGS_LAUNCH, "a warpgroup would wait for registers that nobody gives back");
constexpr float RESCALE_STEP = 8.f;

// shared-memory map (offsets from a 1024-byte aligned base): atoms of 128 rows x 64 values, two (d halves) per tile
constexpr int OFF_Q = 0;                           // a tile per slot
constexpr int OFF_K = OFF_Q + SLOTS * 2 * ATOM;    // two tiles
constexpr int OFF_V = OFF_K + 2 * 2 * ATOM;        // two tiles
constexpr int SMEM_BYTES = OFF_V + 2 * 2 * ATOM + 1024;
// TMEM columns: per slot 128 of S (P in the first 64 of them), then per slot 128 of O
constexpr uint32_t COL_O = SLOTS * BK;

constexpr uint32_t IDESC_S = instr_desc(BK), IDESC_O = instr_desc(D) | (1u << 16);        // bit 16: B is MN-major

LLM_DEVICE void cp_async16(uint32_t dst, const void* src) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory"); }
LLM_DEVICE void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// One row's attention over keys [k0, k1) alone, by a warp: lane i has values 4i .. 4i + 3 of q and of the unscaled result o.
// `row_of(key, kv)`: the key's K (0) or V (1) row.
template <bool CAP, class F>
LLM_DEVICE void exact_row(const __nv_bfloat16* q, int k0, int k1, const ScoreScale& score, F&& row_of, float& m, float& l, float (&o)[4]) {
    const int lane = threadIdx.x & 31;
    auto four = [&](const __nv_bfloat16* x, float (&f)[4]) {
        const uint2 v = __ldcg(reinterpret_cast<const uint2*>(x + lane * 4));
        f[0] = bf16_lo(v.x); f[1] = bf16_hi(v.x); f[2] = bf16_lo(v.y); f[3] = bf16_hi(v.y);
    };
    float a[4];
    four(q, a);
    m = -INFINITY; l = 0.f;
    o[0] = o[1] = o[2] = o[3] = 0.f;
#pragma unroll 4
    for (int key = k0; key < k1; ++key) {
        float k[4], v[4];
        four(row_of(key, 0), k);
        four(row_of(key, 1), v);
        const float s = warp_sum(a[0] * k[0] + a[1] * k[1] + a[2] * k[2] + a[3] * k[3]);
        const float x = CAP ? score.capped(s) : score.linear(s), top = fmaxf(m, x);
        if (top == -INFINITY) continue;                    // a score of -inf: probability 0
        const float c = exp2f(m - top), e = exp2f(x - top);
        m = top;
        l = l * c + e;
#pragma unroll
        for (int i = 0; i < 4; ++i) o[i] = o[i] * c + e * v[i];
    }
}

// Four values a lane of a row's unscaled result, on to the output: the sink's share of the denominator, the output gate
LLM_DEVICE void finish_row(const AttnPrefillParams& p, size_t at, int head, float m, float l, float (&o)[4]) {
    const int lane = threadIdx.x & 31;
    if (p.sink) l += exp2f(p.sink[head] * LOG2E - m);
    float inv = l > 0.f ? 1.f / l : 0.f;
    if (p.gate && p.gate_heads) inv *= __fdividef(1.f, 1.f + __expf(-__bfloat162float(p.gate[at * p.gate_row + head])));
    if (p.gate && !p.gate_heads) {
        const uint2 g = *reinterpret_cast<const uint2*>(p.gate + at * p.gate_row + head * D + lane * 4);
        o[0] *= __fdividef(1.f, 1.f + __expf(-bf16_lo(g.x))); o[1] *= __fdividef(1.f, 1.f + __expf(-bf16_hi(g.x)));
        o[2] *= __fdividef(1.f, 1.f + __expf(-bf16_lo(g.y))); o[3] *= __fdividef(1.f, 1.f + __expf(-bf16_hi(g.y)));
    }
    *reinterpret_cast<uint2*>(p.out + (at * p.n_heads + head) * D + lane * 4) = make_uint2(pack_bf16(o[0] * inv, o[1] * inv), pack_bf16(o[2] * inv, o[3] * inv));
}

enum Bar { K_FULL = 0, K_EMPTY = 2, V_FULL = 4, V_EMPTY = 6, Q_FULL = 8, S_FULL = 9, P_FULL = 11, O_FULL = 13, N_BARS = 15 };

template <bool CAP>                                // scores are soft-capped
__global__ void __launch_bounds__(THREADS, 1) paged_attn_prefill_tc_kernel(const __grid_constant__ CUtensorMap map_kv, const AttnPrefillTcParams p, int* status) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t s_bars[N_BARS];
    __shared__ uint32_t s_tmem;
    __shared__ int s_abort[2];       // [1] stays 0 here (tc_common.cuh: restarts the wait clock when set)
    pdl_wait();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int splits = max(1, p.splits), seq = blockIdx.z / splits, split = blockIdx.z - seq * splits;
    const int kvh = blockIdx.y, G = p.n_heads / p.n_kv_heads;
    const int q_start = p.cu_q[seq], q_len = p.cu_q[seq + 1] - q_start;
    // slot z of this sequence and K/V head: query tile z / G, head z % G of the group.  The last query tiles see the most keys: they
    // go first so that the grid ends with the short CTAs.
    const int n_slots = (q_len + BQ - 1) / BQ * G;
    const int first = 2 * ((int)gridDim.x - 1 - (int)blockIdx.x);
    if (first >= n_slots) return;                          // uniform for the CTA, before any barrier or allocation
    const bool both = first + 1 < n_slots;
    const int ctx = p.ctx_lens[seq];                       // tokens already in the cache before this chunk
    const int q_lo = first / G * BQ, q_hi = min(((both ? first + 1 : first) / G + 1) * BQ, q_len);
    const int kv_end = ctx + q_hi;                         // keys the CTA's rows can see
    const int tile_lo = first_key(ctx + q_lo, p.window, p.chunk) / BK;        // tile of the first key that its first row sees
    const int tile_hi = (kv_end + BK - 1) / BK, n_pages = (kv_end + PAGE - 1) / PAGE;
    const int per = (tile_hi - tile_lo + splits - 1) / splits, tile0 = tile_lo + split * per, nt = min(tile_hi, tile0 + per) - tile0;
    // where this CTA's first slot parks its results, if the keys are shared out
    const size_t part = (((size_t)(seq * p.n_kv_heads + kvh) * gridDim.x + first / 2) * 2 * splits + split) * BQ;
    if (nt <= 0) {                                         // fewer tiles than splits
        for (int i = threadIdx.x; i < 2 * BQ; i += THREADS)
            *reinterpret_cast<float2*>(p.part_ml + (part + (size_t)(i / BQ) * splits * BQ + i % BQ) * 2) = make_float2(-INFINITY, 0.f);
        return;
    }
    const int* btab = p.block_table + (size_t)seq * p.max_pages;
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t bars = smem_u32(s_bars);
    auto bar = [&](int i) { return bars + i * 8; };

    if (tid == 0) {
        s_abort[0] = 0; s_abort[1] = 0;
        for (int i = 0; i < N_BARS; ++i) mbar_init(bar(i), i == Q_FULL ? (both ? 8 : 4) : i == P_FULL || i == P_FULL + 1 ? 4 : 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_proxy_async();
    }
    if (warp == 9) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    volatile int* abort_flag = s_abort;

    if (warp < 8) {
        // ------------------------------ softmax + output: one thread per query row (== TMEM lane) ------------------------------
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS_SOFTMAX));       // a row's 128 scores stay in registers
        const int slot = warp >> 2, row = tid & 127;
        if (slot == 0 || both) {
            const int q0 = (first + slot) / G * BQ, head = kvh * G + (first + slot) % G;
            const int rows = min(BQ, q_len - q0);
            const uint32_t sQ = base + OFF_Q + slot * 2 * ATOM;
#pragma unroll 4
            for (int idx = row; idx < BQ * 16; idx += 128) {
                const int r = idx >> 4, u = idx & 15;
                const uint32_t dst = atom_addr(sQ + (u >> 3) * ATOM, r, u & 7);
                if (r < rows) cp_async16(dst, p.q + ((size_t)(q_start + q0 + r) * p.n_heads + head) * D + u * 8);
                else st_shared_v4(dst, make_uint4(0, 0, 0, 0));
            }
            cp_async_wait_all();
            fence_proxy_async();
            __syncwarp();
            mbar_arrive_if(bar(Q_FULL), lane == 0);

            const int lim = ctx + min(q0 + row, q_len - 1) + 1;           // this row sees keys < lim, and >= low
            const int low = first_key(lim - 1, p.window, p.chunk);
            const uint32_t t_lane = tmem + ((uint32_t)((warp & 3) * 32) << 16);
            const uint32_t t_s = t_lane + slot * BK, t_o = t_lane + COL_O + slot * D;
            const ScoreScale score(p.scale, p.softcap);
            const float sl2 = score.mul;
            float m = -INFINITY, l = 0.f;
            bool ok = true;
            for (int j = 0; j < nt; ++j) {
                ok = mbar_wait_warp(bar(S_FULL + slot), j & 1, abort_flag);
                if (!ok) break;
                tc_fence_after();
                uint32_t s[4][32];
#pragma unroll
                for (int c = 0; c < 4; ++c) tmem_ld32_issue(t_s + c * 32, s[c]);
#pragma unroll
                for (int c = 0; c < 4; ++c) tmem_wait_ld(s[c]);
                const int key0 = (tile0 + j) * BK;
                if (__any_sync(0xffffffffu, key0 + BK > lim || key0 < low)) {
                    const int hi = lim - key0, lo = low - key0;
#pragma unroll
                    for (int c = 0; c < 4; ++c)
#pragma unroll
                        for (int i = 0; i < 32; ++i) s[c][i] = c * 32 + i < hi && c * 32 + i >= lo ? s[c][i] : 0xff800000u;       // -inf
                }
                float mx4[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    mx4[c] = __uint_as_float(s[c][0]);
#pragma unroll
                    for (int i = 1; i < 32; ++i) mx4[c] = fmaxf(mx4[c], __uint_as_float(s[c][i]));
                }
                const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
                float top;
                if constexpr (CAP) top = mx == -INFINITY ? mx : score.capped(mx);          // the cap keeps the order
                else top = mx * sl2;
                const bool raise = top > m + RESCALE_STEP;                // also the first keys, where m is -inf
                const float factor = raise ? ex2(m - top) : 1.f;
                if (raise) m = top;
                // S of this tile was issued behind the last tile's P V and both are complete: O may be changed
                if (j > 0 && __any_sync(0xffffffffu, raise)) {
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        uint32_t r[32];
                        tmem_ld_n<32>(t_o + c * 32, r);
#pragma unroll
                        for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * factor);
                        tmem_st32(t_o + c * 32, r);
                    }
                }
                const float mb = m == -INFINITY ? 0.f : m;
                const float c2 = -2.f * score.cap, c1 = score.cap - mb;
                auto prob = [&](uint32_t r) {
                    const float x = __uint_as_float(r);
                    if constexpr (CAP) return x == -INFINITY ? 0.f : ex2(fmaf(c2, __fdividef(1.f, 1.f + ex2(x * sl2)), c1));
                    else return ex2(fmaf(x, sl2, -mb));
                };
                float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    uint32_t w[16];
#pragma unroll
                    for (int i = 0; i < 32; i += 2) {
                        const float p0 = prob(s[c][i]), p1 = prob(s[c][i + 1]);
                        sum[(i >> 1) & 1] += p0;
                        sum[2 + ((i >> 1) & 1)] += p1;
                        w[i >> 1] = pack_bf16(p0, p1);
                    }
                    tmem_st_n<16>(t_s + c * 16, w);
                }
                l = l * factor + ((sum[0] + sum[1]) + (sum[2] + sum[3]));
                tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                mbar_arrive_if(bar(P_FULL + slot), lane == 0);
            }
            ok = ok && mbar_wait_warp(bar(O_FULL + slot), 0, abort_flag);
            const float sum_l = l;
            float odd[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};       // NaN once a value of the row's O is not finite
            if (ok && splits > 1) {
                tc_fence_after();
                const size_t at = part + (size_t)slot * splits * BQ + row;
                float4* dst = reinterpret_cast<float4*>(p.part_o + at * D);
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    uint32_t r[32];
                    tmem_ld_n<32>(t_o + c * 32, r);
#pragma unroll
                    for (int i = 0; i < 32; ++i) odd[i & 7] = fmaf(__uint_as_float(r[i]), 0.f, odd[i & 7]);
#pragma unroll
                    for (int u = 0; u < 8; ++u)
                        dst[c * 8 + u] = make_float4(__uint_as_float(r[4 * u]), __uint_as_float(r[4 * u + 1]), __uint_as_float(r[4 * u + 2]), __uint_as_float(r[4 * u + 3]));
                }
                *reinterpret_cast<float2*>(p.part_ml + at * 2) = make_float2(m, l);
            } else if (ok) {
                tc_fence_after();
                if (p.sink) l += exp2f(p.sink[head] * LOG2E - m);
                float inv = l > 0.f ? 1.f / l : 0.f;
                const size_t at = (size_t)(q_start + q0 + row);
                if (row < rows && p.gate && p.gate_heads) inv *= __fdividef(1.f, 1.f + __expf(-__bfloat162float(p.gate[at * p.gate_row + head])));
                __nv_bfloat16* dst = p.out + (at * p.n_heads + head) * D;
                const __nv_bfloat16* gate = p.gate && !p.gate_heads ? p.gate + at * p.gate_row + head * D : nullptr;
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    uint32_t r[32];
                    tmem_ld_n<32>(t_o + c * 32, r);
#pragma unroll
                    for (int i = 0; i < 32; ++i) odd[i & 7] = fmaf(__uint_as_float(r[i]), 0.f, odd[i & 7]);
                    if (row < rows) {
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            float o[8];
#pragma unroll
                            for (int i = 0; i < 8; ++i) o[i] = __uint_as_float(r[8 * u + i]);
                            if (gate) {
                                const uint4 g = *reinterpret_cast<const uint4*>(gate + c * 32 + 8 * u);
                                const uint32_t gw[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
                                for (int i = 0; i < 4; ++i) {
                                    o[2 * i] *= __fdividef(1.f, 1.f + __expf(-bf16_lo(gw[i])));
                                    o[2 * i + 1] *= __fdividef(1.f, 1.f + __expf(-bf16_hi(gw[i])));
                                }
                            }
                            uint4 v;
                            v.x = pack_bf16(o[0] * inv, o[1] * inv); v.y = pack_bf16(o[2] * inv, o[3] * inv);
                            v.z = pack_bf16(o[4] * inv, o[5] * inv); v.w = pack_bf16(o[6] * inv, o[7] * inv);
                            *reinterpret_cast<uint4*>(dst + c * 32 + 8 * u) = v;
                        }
                    }
                }
            }
            // A masked key has P = 0, and 0 times an infinity or NaN in its V row (a later token, or what the page held before) is
            // NaN.  Rows that are not finite although their scores are, and that have such a key in their tiles, are computed again
            // over their own keys alone.
            const float any = ((odd[0] + odd[1]) + (odd[2] + odd[3])) + ((odd[4] + odd[5]) + (odd[6] + odd[7]));
            unsigned again = __ballot_sync(0xffffffffu, ok && row < rows && any != 0.f && fabsf(sum_l) <= 3.4e38f);
            if (again) __syncwarp();                               // the stores above come before the ones below
#pragma unroll 1
            for (; again; again &= again - 1) {
                const int src = __ffs(again) - 1, i = (warp & 3) * 32 + src;
                const int t0 = tile0 * BK, t1 = t0 + nt * BK, k0 = max(t0, __shfl_sync(0xffffffffu, low, src)), k1 = max(k0, min(t1, __shfl_sync(0xffffffffu, lim, src)));
                auto row_of = [&](int key, int kv) {
                    const size_t page = LLM_CHECK_INDEX(btab[min(key / PAGE, n_pages - 1)], p.n_pages);
                    return p.kv + (((page * 2 + kv) * p.n_kv_heads + kvh) * PAGE + key % PAGE) * D;
                };
                float zero = 0.f;
#pragma unroll 1
                for (int key = t0; key < t1; ++key) {
                    if (key == k0) { key = k1; if (key >= t1) break; }
                    const uint2 v = __ldcg(reinterpret_cast<const uint2*>(row_of(key, 1) + lane * 4));
                    zero += (bf16_lo(v.x) + bf16_hi(v.x)) * 0.f + (bf16_lo(v.y) + bf16_hi(v.y)) * 0.f;
                }
                if (!__any_sync(0xffffffffu, zero != 0.f)) continue;
                const size_t at = (size_t)(q_start + q0 + i);
                float rm, rl, o[4];
                exact_row<CAP>(p.q + (at * p.n_heads + head) * D, k0, k1, score, row_of, rm, rl, o);
                if (splits > 1) {
                    const size_t mine = part + (size_t)slot * splits * BQ + i;
                    *reinterpret_cast<float4*>(p.part_o + mine * D + lane * 4) = make_float4(o[0], o[1], o[2], o[3]);
                    if (lane == 0) *reinterpret_cast<float2*>(p.part_ml + mine * 2) = make_float2(rm, rl);
                } else finish_row(p, at, head, rm, rl, o);
            }
        }
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS_OTHER));
        if (warp == 8) {
            // ------------------------------ K and V tiles: page by page, half a head at a time ------------------------------
            if (elect_one()) {
                bool ok = true;
                auto load = [&](int j, int kv, int full, int empty) {
                    const int b = j & 1;
                    ok = mbar_wait(bar(empty + b), ((j >> 1) & 1) ^ 1, abort_flag);
                    if (!ok) return;
                    mbar_arrive_expect_tx(bar(full + b), 2 * ATOM);
                    const uint32_t dst = base + (kv ? OFF_V : OFF_K) + b * 2 * ATOM;
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        // a page past the end repeats the last one (its keys are masked)
                        const int page = LLM_CHECK_INDEX(btab[min(2 * (tile0 + j) + h, n_pages - 1)], p.n_pages);
                        const int y = ((page * 2 + kv) * p.n_kv_heads + kvh) * PAGE;
                        tma_load_2d(dst + h * (ATOM / 2), &map_kv, 0, y, bar(full + b));
                        tma_load_2d(dst + ATOM + h * (ATOM / 2), &map_kv, 64, y, bar(full + b));
                    }
                };
                for (int j = 0; j < nt && ok; ++j) {
                    load(j, 0, K_FULL, K_EMPTY);
                    if (ok) load(j, 1, V_FULL, V_EMPTY);
                }
            }
        } else if (warp == 9 && elect_one()) {
            // ------------------------------ MMA issue ------------------------------
            auto issue_s = [&](int slot, int j) {
                const uint32_t q = base + OFF_Q + slot * 2 * ATOM, k = base + OFF_K + (j & 1) * 2 * ATOM;
#pragma unroll
                for (int ks = 0; ks < 8; ++ks)
                    mma_f16(tmem + slot * BK, smem_desc_sw128(q + (ks >> 2) * ATOM) + 2 * (ks & 3), smem_desc_sw128(k + (ks >> 2) * ATOM) + 2 * (ks & 3), IDESC_S, ks > 0 ? 1u : 0u);
                mma_commit(bar(S_FULL + slot));
            };
            bool ok = mbar_wait(bar(Q_FULL), 0, abort_flag) && mbar_wait(bar(K_FULL), 0, abort_flag);
            if (ok) {
                tc_fence_after();
                issue_s(0, 0);
                if (both) issue_s(1, 0);
                mma_commit(bar(K_EMPTY));
            }
            for (int j = 0; j < nt && ok; ++j) {
                const bool more = j + 1 < nt;
                ok = mbar_wait(bar(V_FULL + (j & 1)), (j >> 1) & 1, abort_flag) && (!more || mbar_wait(bar(K_FULL + ((j + 1) & 1)), ((j + 1) >> 1) & 1, abort_flag));
                for (int slot = 0; slot < (both ? 2 : 1) && ok; ++slot) {
                    ok = mbar_wait(bar(P_FULL + slot), j & 1, abort_flag);
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t v = base + OFF_V + (j & 1) * 2 * ATOM;
#pragma unroll
                    for (int ks = 0; ks < 8; ++ks)      // 16 keys: 8 TMEM columns of P, 16 rows of the V tile
                        mma_f16_ts(tmem + COL_O + slot * D, tmem + slot * BK + ks * 8, smem_desc_mn_sw128(v + ks * 16 * 128, ATOM), IDESC_O, j > 0 || ks > 0 ? 1u : 0u);
                    if (more) issue_s(slot, j + 1);     // behind the P V that reads P from the same columns
                    else mma_commit(bar(O_FULL + slot));
                }
                if (ok) {
                    mma_commit(bar(V_EMPTY + (j & 1)));
                    if (more) mma_commit(bar(K_EMPTY + ((j + 1) & 1)));
                }
            }
        }
    }

    // ------------------------------ teardown ------------------------------
    tc_fence_before();
    __syncthreads();
    teardown(abort_flag, tid, status);
    if (warp == 9) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
}

// The splits' results of a query row, a warp per row and head: rescaled to the largest maximum, summed up in split order.
__global__ void __launch_bounds__(128) paged_attn_prefill_merge_kernel(const AttnPrefillTcParams p, int pairs) {
    pdl_trigger();
    pdl_wait();
    const int lane = threadIdx.x & 31, G = p.n_heads / p.n_kv_heads, head = blockIdx.y, kvh = head / G, seq = blockIdx.z;
    const int q_start = p.cu_q[seq], q_len = p.cu_q[seq + 1] - q_start;
    const int r = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (r >= q_len) return;
    const int z = r / BQ * G + head % G;                    // the row's slot
    const size_t part = (((size_t)(seq * p.n_kv_heads + kvh) * pairs * 2 + z) * p.splits) * BQ + r % BQ;
    float m = -INFINITY;
    for (int s = 0; s < p.splits; ++s) m = fmaxf(m, __ldcg(p.part_ml + (part + (size_t)s * BQ) * 2));
    float l = 0.f, o[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (int s = 0; s < p.splits; ++s) {
        const float2 ml = __ldcg(reinterpret_cast<const float2*>(p.part_ml + (part + (size_t)s * BQ) * 2));
        const float c = ml.x == -INFINITY ? 0.f : exp2f(ml.x - m);
        if (ml.x == -INFINITY && ml.y == 0.f) continue;     // no keys there
        const float4 v = __ldcg(reinterpret_cast<const float4*>(p.part_o + (part + (size_t)s * BQ) * D) + lane);
        l += c * ml.y;
        o[0] += c * v.x; o[1] += c * v.y; o[2] += c * v.z; o[3] += c * v.w;
    }
    finish_row(p, (size_t)(q_start + r), head, m, l, o);
}

static int pairs_of(int n_heads, int n_kv_heads, int max_q_len) { return ((max_q_len + BQ - 1) / BQ * (n_heads / n_kv_heads) + 1) / 2; }

}  // namespace atc

// A pair of query tiles walks its keys at 1.5 us per tile of 128 whatever else the GPU does: where the pairs leave SMs without a CTA, the
// keys are shared out, at least four tiles to a split (500 rows behind 7000 tokens, 32 / 8 heads: 116 -> 76 us;
// 16 rows behind 7000: 105 -> 28.5; 200 rows of two sequences behind 6000: 97 -> 65).
int attn_prefill_tc_splits(int n_heads, int n_kv_heads, int n_seqs, int max_q_len, int max_kv_len, long long part_o, long long part_ml) {
    if (n_kv_heads < 1 || n_heads % n_kv_heads || n_seqs < 1 || max_q_len < 1) return 1;
    const long long ctas = (long long)atc::pairs_of(n_heads, n_kv_heads, max_q_len) * n_kv_heads * n_seqs, slots = 2 * ctas;
    long long s = 148 / ctas;
    const long long by_keys = max_kv_len / (4 * atc::BK), by_o = part_o / (slots * atc::BQ * atc::D), by_ml = part_ml / (slots * atc::BQ * 2);
    if (s > by_keys) s = by_keys;
    if (s > by_o) s = by_o;
    if (s > by_ml) s = by_ml;
    if (s > 16) s = 16;
    return s < 2 ? 1 : (int)s;
}

cudaError_t launch_attn_prefill_tc(const AttnPrefillTcParams& p, int n_seqs, int max_q_len, int* status, cudaStream_t st) {
    if (n_seqs == 0 || max_q_len == 0) return cudaSuccess;
    if (p.head_dim != atc::D || p.n_heads % p.n_kv_heads) return cudaErrorInvalidValue;
    // the cache as a matrix of head_dim columns: 64 rows per page, K or V, and head
    CUtensorMap map;
    if (!tc5::make_map(&map, p.kv, atc::D, (uint64_t)p.n_pages * 2 * p.n_kv_heads * atc::PAGE, atc::D, atc::PAGE)) return cudaErrorInvalidValue;
    const int splits = p.splits > 1 ? p.splits : 1;
    const dim3 grid(atc::pairs_of(p.n_heads, p.n_kv_heads, max_q_len), p.n_kv_heads, n_seqs * splits);
    if (splits > 1 && (!p.part_o || !p.part_ml || ((reinterpret_cast<uintptr_t>(p.part_o) | reinterpret_cast<uintptr_t>(p.part_ml)) & 15))) return cudaErrorInvalidValue;
    auto go = [&](auto kernel, bool& once) -> cudaError_t {
        if (!once) {
            cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, atc::SMEM_BYTES);
            if (e != cudaSuccess) return e;
            once = true;
        }
        return launch_pdl(kernel, grid, dim3(atc::THREADS), atc::SMEM_BYTES, st, map, p, status);
    };
    static bool plain = false, capped = false;
    const cudaError_t e = p.softcap > 0.f ? go(atc::paged_attn_prefill_tc_kernel<true>, capped) : go(atc::paged_attn_prefill_tc_kernel<false>, plain);
    if (e != cudaSuccess || splits == 1) return e;
    return launch_pdl(atc::paged_attn_prefill_merge_kernel, dim3((max_q_len + 3) / 4, p.n_heads, n_seqs), dim3(128), 0, st, p, (int)grid.x);
}

LLM_DEFINE_BOUNDS_STATUS_READER(bounds_status_attention_tc)

}  // namespace llm
