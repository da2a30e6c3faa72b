// Streaming grouped GEMV of the routed experts for decode steps: the work list of `moe_route` (up to four pairs of one expert per item)
// against the experts' packed matrices, int8 activations and dp4a as in gemv.cu.
//
// What bounded the register-path kernel (gemv.cu, `items`): a CTA per item and 128-row tile whose eight warps each had one chunk of
// loads in flight, behind a prologue that normalised and quantised the item's rows again for every tile.  Here the flattened (item, tile,
// chunk) work is shared evenly between one persistent CTA per SM: a producer thread fetches the chunks by bulk copy into a ring of
// shared-memory slots (it starts while the rows are quantised), rows are quantised once per item and CTA, and a tile split between CTAs is
// finished by the one that holds its first chunk, which adds the others' parked sums in CTA order.  The weighted sum of the experts is
// a launch of its own: inside this one it was a serial tail of the last CTA of every tile.
// Measured (128 experts of 768 x 2048, Q4_K, 8 tokens x 8 experts, one of eight layers in turn): gate | up 34.7 us (55.2 on the register
// path), down and sum 26.2 us (35.6); what bounds it now is the dp4a arithmetic of four rows per chunk and the rows' quantisation.
#include <cuda.h>

#include "formats.cuh"
#include "gemv.h"
#include "launch.h"
#include "tc_common.cuh"

namespace llm {
namespace ms {
using namespace tc5;

constexpr int M = 4, N_WARPS = 16, THREADS = (N_WARPS + 1) * 32, N_COMPUTE = N_WARPS * 32;       // + the producer warp
constexpr uint32_t TICKET_SPIN = 1u << 20;

struct Extra {
    float* partials;           // [grid][4][128] sums parked by the CTAs that do not finish a split tile
    unsigned* tickets;         // [items][n_tiles] arrivals at a split tile, zero between launches
    int* status;               // STATUS_TIMEOUT is written here when a bounded wait gives up
    int slots;                 // ring slots (4 or 8)
};

LLM_DEVICE void bar_compute() { asm volatile("bar.sync 1, %0;" ::"n"(N_COMPUTE) : "memory"); }
LLM_DEVICE void bar_rows() { asm volatile("bar.sync 2, 128;" ::: "memory"); }

// A CTA's range of the flattened chunks, unit by unit (a unit = the part of one tile inside the range).
struct Unit { int vt, kb0, nkb, first_cta, last_cta; };          // vt = item * n_tiles + tile
struct Walk {
    int k_blocks, total, G, pos, end;
    LLM_DEVICE void init(int kb, int n_units, int grid, int cta) {
        k_blocks = kb; total = kb * n_units;
        G = min(grid, max(1, total / 4));      // at least four chunks per CTA
        pos = cta < G ? (int)(((unsigned)cta * (unsigned)total) / (unsigned)G) : 0;
        end = cta < G ? (int)(((unsigned)(cta + 1) * (unsigned)total) / (unsigned)G) : 0;
    }
    // 32-bit arithmetic: the launcher refuses problems with (chunks + 1) * grid >= 2^32
    LLM_DEVICE int cta_of(int x) const { return (int)(((unsigned)(x + 1) * (unsigned)G - 1u) / (unsigned)total); }
    LLM_DEVICE bool next(Unit& u) {
        if (pos >= end) return false;
        u.vt = pos / k_blocks;
        u.kb0 = pos - u.vt * k_blocks;
        u.nkb = min(k_blocks - u.kb0, end - pos);
        u.first_cta = cta_of(u.vt * k_blocks);
        u.last_cta = cta_of(u.vt * k_blocks + k_blocks - 1);
        pos += u.nkb;
        return true;
    }
};

// The item's four rows, RMS-normalised (NORM) and quantised to int8 per 32 columns, at acts[m * k_blocks + kb].  Run by the compute warps.
template <int NORM>
LLM_DEVICE void quantise_rows(const GemvParams& p, const MoeItem& item, ActBlk* acts, float* s_ss) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // four warps per row
    const int m = warp >> 2, part = (warp & 3) * 32 + lane;
    const size_t row = (size_t)(item.slot[m] / p.x_div) * p.x_stride;
    float rms = 1.f;
    if (NORM) {
        const float4* x4 = reinterpret_cast<const float4*>(static_cast<const float*>(p.x) + row);
        float ss = 0.f;
#pragma unroll 4
        for (int i = part; i < p.k / 4; i += 128) {
            const float4 v = __ldcg(x4 + i);
            ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
        }
        ss = warp_sum(ss);
        if (lane == 0) s_ss[warp] = ss;
        bar_compute();
        rms = rsqrtf((s_ss[4 * m] + s_ss[4 * m + 1] + s_ss[4 * m + 2] + s_ss[4 * m + 3]) / p.k + p.eps);
    }
#pragma unroll 4
    for (int qd = part; qd < p.k / 4; qd += 128) {          // 4 columns per thread, 8 lanes per 32-column block
        float v0, v1, v2, v3;
        if (NORM) {
            const float4 v = __ldcg(reinterpret_cast<const float4*>(static_cast<const float*>(p.x) + row) + qd);
            const float4 g = reinterpret_cast<const float4*>(p.norm_w)[qd];
            v0 = v.x * rms * g.x; v1 = v.y * rms * g.y; v2 = v.z * rms * g.z; v3 = v.w * rms * g.w;
        } else {
            const uint2 v = __ldcg(reinterpret_cast<const uint2*>(static_cast<const __nv_bfloat16*>(p.x) + row) + qd);
            v0 = bf16_lo(v.x); v1 = bf16_hi(v.x); v2 = bf16_lo(v.y); v3 = bf16_hi(v.y);
        }
        float amax = fmaxf(fmaxf(fabsf(v0), fabsf(v1)), fmaxf(fabsf(v2), fabsf(v3)));
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 4));
        const float d = amax * (1.0f / 127.0f);
        const float inv = amax > 0.f ? 127.0f / amax : 0.f;
        const int q0 = __float2int_rn(v0 * inv), q1 = __float2int_rn(v1 * inv);
        const int q2 = __float2int_rn(v2 * inv), q3 = __float2int_rn(v3 * inv);
        int s = q0 + q1 + q2 + q3;
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        ActBlk& ab = acts[m * p.k_blocks + (qd >> 6)];
        const int qi = qd & 63;
        ab.a[qi] = (q0 & 0xff) | ((q1 & 0xff) << 8) | ((q2 & 0xff) << 16) | ((q3 & 0xff) << 24);
        if ((qi & 7) == 0) ab.d[qi >> 3] = d;
        if ((qi & 3) == 0) ab.ds16[qi >> 2] = d * s;
    }
    bar_compute();
}

// NORM = 1: gate | up of the normalised residual rows, SwiGLU, bf16 rows out[pair].  NORM = 0: down projection of bf16 rows, fp32
// rows out[pair].
template <int FMT, int NORM>
__global__ void __launch_bounds__(THREADS, 1) moe_stream_kernel(const GemvParams p, const Extra e) {
    constexpr int CHUNK = FmtTraits<FMT>::CHUNK;
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ __align__(8) uint64_t s_full[8], s_empty[8];
    __shared__ int s_abort[2], s_flag, s_go[2];
    pdl_trigger();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int R = e.slots;
    uint8_t* ring = smem;                                                        // R slots of CHUNK bytes
    ActBlk* acts = reinterpret_cast<ActBlk*>(smem + (size_t)R * CHUNK);          // [M][k_blocks]
    float* s_red = reinterpret_cast<float*>(acts + (size_t)M * p.k_blocks);      // [2][4][M][128]
    uint32_t* s_grid = reinterpret_cast<uint32_t*>(s_red + 2 * 4 * M * 128);     // IQ3_S only
    const uint32_t full_bar = smem_u32(s_full), empty_bar = smem_u32(s_empty), ring_addr = smem_u32(ring);
    if (tid == 0) {
        s_abort[0] = 0; s_abort[1] = 0;
        for (int s = 0; s < R; ++s) { mbar_init(full_bar + s * 8, 1); mbar_init(empty_bar + s * 8, 4); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_proxy_async();
    }
    if (FMT == FMT_IQ3_S) {
        for (int i = tid; i < 512; i += THREADS) s_grid[i] = g_iq3s_grid[i];
    }
    __syncthreads();
    pdl_wait();                                  // the work list and the rows are the previous kernels'
    volatile int* abort_flag = s_abort;
    Walk it;
    it.init(p.k_blocks, __ldcg(p.n_items) * p.n_tiles, gridDim.x, blockIdx.x);
    Unit u;

    if (warp == N_WARPS) {
        // ---------------- producer: one bulk copy per chunk ----------------
        if (elect_one()) {
            int cc = 0;
            bool ok = true;
            while (ok && it.next(u)) {
                const int item = u.vt / p.n_tiles, tile = u.vt - item * p.n_tiles;
                const uint8_t* src = p.w + (size_t)__ldcg(&p.items[item].expert) * p.expert_stride + ((size_t)tile * p.k_blocks + u.kb0) * CHUNK;
                for (int c = 0; c < u.nkb && ok; ++c, ++cc) {
                    const int slot = cc % R, phase = (cc / R) & 1;
                    ok = mbar_wait(empty_bar + slot * 8, phase ^ 1, abort_flag);
                    if (!ok) break;
                    mbar_arrive_expect_tx(full_bar + slot * 8, CHUNK);
                    bulk_load(ring_addr + slot * CHUNK, src + (size_t)c * CHUNK, CHUNK, full_bar + slot * 8);
                }
            }
        }
    } else {
        // ---------------- compute warps: warp (g, q) has rows 32 g .. 32 g + 31 of the tile and every fourth chunk ----------------
        const int g = warp & 3, q = warp >> 2;
        const int act_stride = p.k_blocks * (int)sizeof(ActBlk);
        float acc[M];
#pragma unroll
        for (int m = 0; m < M; ++m) acc[m] = 0.f;
        int cc = 0, ui = 0, cur = -1;
        MoeItem work{};
        bool ok = true;
        // A wait that gives up sets the CTA's abort flag; from then on this warp skips the work but still walks the units, because
        // the named barriers below have no time limit of their own and every compute warp has to reach them.
        while (it.next(u)) {
            const int item = u.vt / p.n_tiles, tile = u.vt - item * p.n_tiles;
            if (item != cur) {                       // every warp is past the last unit's dot products (barrier below)
                cur = item;
                // (written by the kernel before, like the rows: L2-coherent loads)
                work.m = __ldcg(&p.items[item].m);
#pragma unroll
                for (int m = 0; m < M; ++m) work.slot[m] = __ldcg(&p.items[item].slot[m]);
                quantise_rows<NORM>(p, work, acts, s_red + (ui & 1) * (4 * M * 128));
            }
            for (int c = 0; c < u.nkb; ++c, ++cc) {
                if ((cc & 3) != q || !ok) continue;
                const int slot = cc % R, phase = (cc / R) & 1;
                ok = mbar_wait_warp(full_bar + slot * 8, phase, abort_flag);
                if (!ok) continue;
                const uint8_t* chunk = ring + (size_t)slot * CHUNK;
                if constexpr (FMT == FMT_IQ3_S) DotBlock<FMT, M, LdShared>::run(chunk, g, lane, acts + u.kb0 + c, act_stride, acc, s_grid);
                else DotBlock<FMT, M, LdShared>::run(chunk, g, lane, acts + u.kb0 + c, act_stride, acc);
                __syncwarp();                        // every lane has its bytes in registers
                mbar_arrive_if(empty_bar + slot * 8, lane == 0);
            }
            // ---- the unit is done: add up the four chunk phases of every row ----
            float* red = s_red + (ui & 1) * (4 * M * 128);
            const int r = g * 32 + lane;
#pragma unroll
            for (int m = 0; m < M; ++m) { red[(q * M + m) * 128 + r] = acc[m]; acc[m] = 0.f; }
            if (tid == 0) s_go[ui & 1] = abort_flag[0] ? 0 : 1;       // one reading of the flag for all row threads (they meet at barriers below)
            bar_compute();
            const bool go = s_go[ui & 1] != 0;
            ++ui;
            if (tid >= 128 || !go) continue;
            float v[M];
#pragma unroll
            for (int m = 0; m < M; ++m) v[m] = red[m * 128 + tid] + red[(M + m) * 128 + tid] + red[(2 * M + m) * 128 + tid] + red[(3 * M + m) * 128 + tid];
            if (u.first_cta != u.last_cta) {
                if ((int)blockIdx.x != u.first_cta) {
                    // park and tell the finisher (every thread's stores, then one release from thread 0)
                    float* mine = e.partials + (size_t)blockIdx.x * (M * 128);
#pragma unroll
                    for (int m = 0; m < M; ++m) __stcg(&mine[m * 128 + tid], v[m]);
                    bar_rows();
                    if (tid == 0) { __threadfence(); red_release_gpu_add(&e.tickets[u.vt], 1u); }
                    continue;
                }
                // finisher: the others hold later chunks of the tile but reach them at the START of their ranges
                const unsigned want = (unsigned)(u.last_cta - u.first_cta);
                if (tid == 0) {
                    int got = 0;
                    for (uint32_t i = 0; i < TICKET_SPIN; ++i) {
                        if (ld_acquire_gpu(&e.tickets[u.vt]) >= want) { got = 1; break; }
                        if (i > 64) { if (abort_flag[0]) break; __nanosleep(64); }
                    }
                    if (!got) abort_flag[0] = 1;
                    s_flag = got;
                }
                bar_rows();
                const bool got = s_flag != 0;
                if (got) for (int cta = u.first_cta + 1; cta <= u.last_cta; ++cta) {
                    const float* theirs = e.partials + (size_t)cta * (M * 128);
#pragma unroll
                    for (int m = 0; m < M; ++m) v[m] += __ldcg(&theirs[m * 128 + tid]);
                }
                bar_rows();                                          // everybody has read the count's verdict and the slots
                if (tid == 0) e.tickets[u.vt] = 0u;
                if (!got) continue;
            }
            // ---- a finished tile ----
            if (NORM) {
                // a 32-row group holds 16 gate rows followed by the 16 matching up rows: pair lanes l and l + 16
                const int col = tile * 64 + (tid >> 5) * 16 + (lane & 15);
#pragma unroll
                for (int m = 0; m < M; ++m) {
                    const float other = __shfl_xor_sync(0xffffffffu, v[m], 16);
                    if (lane < 16 && col < p.n / 2 && m < work.m)
                        static_cast<__nv_bfloat16*>(p.out)[(size_t)work.slot[m] * p.out_stride + col] = __float2bfloat16(silu(v[m]) * other);
                }
            } else {
                const int row = tile * 128 + tid;
                if (row < p.n) {
#pragma unroll
                    for (int m = 0; m < M; ++m)
                        if (m < work.m) static_cast<float*>(p.out)[(size_t)work.slot[m] * p.out_stride + row] = v[m];
                }
            }
        }
    }
    __syncthreads();
    if (*abort_flag) {
        if (tid == 0 && e.status) atomicExch(e.status, (int)STATUS_TIMEOUT);
        for (int i = 0; i < 2000; ++i) __nanosleep(100);      // let bulk copies still in flight land before the shared memory is handed on
    }
}

// h[t] += sum over the locally owned pairs of the token, in slot order, of weight * y[pair]
__global__ void __launch_bounds__(128) moe_combine_pairs_kernel(const MoeCombine c, int d) {
    pdl_trigger();
    pdl_wait();
    const int t = blockIdx.x, i = blockIdx.y * 128 + threadIdx.x;
    if (i >= d) return;
    constexpr int AHEAD = 8;
    float sum = 0.f;
    float* h = c.h + (size_t)t * c.h_stride + i;
    const float old = __ldcg(h);
    for (int j0 = 0; j0 < c.top_k; j0 += AHEAD) {
        float w[AHEAD], y[AHEAD];
        bool mine[AHEAD];
#pragma unroll
        for (int j = 0; j < AHEAD; ++j) {
            const int pr = t * c.top_k + min(j0 + j, c.top_k - 1);
            mine[j] = j0 + j < c.top_k && (unsigned)(__ldcg(c.ids + pr) - c.e0) < (unsigned)c.n_local;
            w[j] = __ldcg(c.wts + pr);
            y[j] = mine[j] ? __ldcg(c.yslot + (size_t)pr * c.y_stride + i) : 0.f;
        }
#pragma unroll
        for (int j = 0; j < AHEAD; ++j)
            if (mine[j]) sum += w[j] * y[j];
    }
    *h = old + sum;
}

template <int FMT>
static cudaError_t launch_f(const GemvParams& p, int grid, Extra e, cudaStream_t st) {
    constexpr int CHUNK = FmtTraits<FMT>::CHUNK;
    auto bytes = [&](int slots) { return (size_t)slots * CHUNK + (size_t)M * p.k_blocks * sizeof(ActBlk) + 2 * 4 * M * 128 * sizeof(float) + 512 * sizeof(uint32_t); };
    e.slots = bytes(8) <= 216 * 1024 ? 8 : 4;
    const size_t smem = bytes(e.slots);
    if (smem > 216 * 1024) return cudaErrorNotSupported;
    auto go = [&](auto kernel, bool& once) -> cudaError_t {
        if (!once) {
            const cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
            if (err != cudaSuccess) return err;
            once = true;
        }
        return launch_pdl(kernel, dim3(grid), dim3(THREADS), smem, st, p, e);
    };
    static bool norm = false, plain = false;
    return p.norm_w ? go(moe_stream_kernel<FMT, 1>, norm) : go(moe_stream_kernel<FMT, 0>, plain);
}

}  // namespace ms

// cudaErrorNotSupported: the call is not one this kernel takes (the caller falls back to launch_gemv).
cudaError_t launch_moe_stream(const GemvParams& p, int z_max, float* partials, size_t partials_floats, unsigned* tickets, size_t n_tickets, int* status, cudaStream_t st) {
    if (!p.items || !p.n_items || p.tp || !partials || !tickets || p.x_div < 1) return cudaErrorNotSupported;
    if (p.epi == EPI_SWIGLU ? !p.norm_w : p.epi != EPI_MOE_COMBINE || p.norm_w) return cudaErrorNotSupported;
    if ((reinterpret_cast<uintptr_t>(p.w) | p.expert_stride) & 15) return cudaErrorNotSupported;
    // 16-byte loads of the rows and gains
    if (p.norm_w ? ((reinterpret_cast<uintptr_t>(p.x) | reinterpret_cast<uintptr_t>(p.norm_w)) & 15) || p.x_stride % 4 : (reinterpret_cast<uintptr_t>(p.x) & 7) || p.x_stride % 4)
        return cudaErrorNotSupported;
    const unsigned long long units = (unsigned long long)z_max * p.n_tiles;
    const int grid = sm_count();
    if (units > n_tickets || (units * p.k_blocks + 1) * grid >= (1ull << 32) || (size_t)grid * ms::M * 128 > partials_floats) return cudaErrorNotSupported;
    const ms::Extra e{partials, tickets, status, 0};
    cudaError_t err = cudaErrorInvalidValue;
    switch (p.fmt) {
        case FMT_Q4_K: err = ms::launch_f<FMT_Q4_K>(p, grid, e, st); break;
        case FMT_Q5_K: err = ms::launch_f<FMT_Q5_K>(p, grid, e, st); break;
        case FMT_Q6_K: err = ms::launch_f<FMT_Q6_K>(p, grid, e, st); break;
        case FMT_Q8_0: err = ms::launch_f<FMT_Q8_0>(p, grid, e, st); break;
        case FMT_Q4_0: err = ms::launch_f<FMT_Q4_0>(p, grid, e, st); break;
        case FMT_IQ3_S: err = ms::launch_f<FMT_IQ3_S>(p, grid, e, st); break;
    }
    if (err != cudaSuccess || p.epi != EPI_MOE_COMBINE) return err;
    return launch_pdl(ms::moe_combine_pairs_kernel, dim3(p.moe.tokens, (p.n + 127) / 128), dim3(128), 0, st, p.moe, p.n);
}

}  // namespace llm
