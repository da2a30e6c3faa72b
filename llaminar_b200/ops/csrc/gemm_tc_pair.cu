// Large-row variant of the tcgen05 dequant GEMM: out[M, N] = x[M, K] * dequant(W)[N, K]^T for prompts (129 rows and more) and for the
// grouped expert GEMMs.  A pair of CTAs (a cluster of two, tcgen05 cta_group::2) computes 256 weight rows x up to 256 tokens.
//
// What bounds a tile of 128 weight rows on its own is not the tensor core: its 256 tokens x 64 columns of activations (32 KB) have to
// come from L2 for every 512 clocks of MMAs, on all SMs at once some 11 TB/s at full rate, and shared memory carries them twice more,
// beside the weights.  So here
//   * the pair shares the activations: each CTA loads half of the tokens, the MMA reads both halves;
//   * the weights never pass through shared memory: eight warps per CTA fetch packed blocks into registers half a chunk ahead, convert
//     them and store them into tensor memory, from where the MMA takes its A operand (lane == weight row);
//   * a slot of the operand ring is one 64-column atom: the activations in shared memory, the weights in 32 TMEM columns, one full and
//     one empty barrier for both.  Warps 0-3 and 4-7 take alternate 256-column chunks; each set owns four of the eight slots, so that
//     every waiter meets each barrier on every revolution and the 1-bit parities stay exact;
//   * the CTAs are persistent.  The one accumulator (256 columns, the ring has the other 256) is read into registers at once and handed
//     back; stores to memory run under the next tile's MMAs, and the chunk of the next tile that each set converts before it turns to
//     the epilogue keeps the tensor core going meanwhile;
//   * the number of tokens of a tile is a run-time value (a multiple of 32): launches choose it so that the last wave is full, ragged
//     tiles and small experts multiply no more than their rows rounded up to 32.
// Measured, us (before: one CTA per 128 weight rows x 256 tokens, weights and activations in shared memory, one tile per CTA):
//   24576 x 4096 Q4_K, 2048 rows 279 (400; now 1479 TFLOP/s), 8160 rows 1083 (1635); 51200 x 5120 Q4_K, 2048 rows 674 (960), 8160 rows
//   2700 (3856); 4096 x 12288 Q6_K, 2048 rows 187 (225); 24576 x 4096 Q8_0, 500 rows 105 (146), 2048 rows 351 (518); 24576 x 4096 Q5_K,
//   2048 rows 337 (445); 24576 x 4096 Q4_K, 160 rows 53 (162).  Sixteen dequantising warps instead of eight: 287 for the first.
// Roles (384 threads): warps 0-7 dequantisation and epilogue, warp 8 TMA, warp 9 TMEM allocation and, in the first CTA of the pair, MMA
// issue; warps 10 and 11 complete the third warpgroup, which hands most of its registers to the other two.
// The loads carry no multicast.  Every wait is bounded; on a timeout the status word is raised and both CTAs tear down.
#include <cuda.h>

#include "formats_half.cuh"
#include "gemm_tc.h"
#include "gemv.h"
#include "launch.h"
#include "tc_tile.cuh"

namespace llm {
namespace tcp {
using namespace tc5;

constexpr int SLOTS = 8, SLOT_BYTES = 128 * 128;        // 128 tokens (half a tile) x 64 columns
constexpr int DEQUANT_WARPS = 8, THREADS = (DEQUANT_WARPS + 4) * 32, SMEM_BYTES = SLOTS * SLOT_BYTES + 1024;
constexpr int REGS_LAUNCH = 168, REGS_DEQUANT = 232, REGS_OTHER = 40;       // per thread; three warpgroups
static_assert(2 * REGS_DEQUANT + REGS_OTHER <= 3 * REGS_LAUNCH, "a warpgroup would wait for registers that nobody gives back");
constexpr uint32_t COL_A = 256;                          // TMEM: accumulator [0, 256), slot i of the weights at 256 + 32 i
constexpr int MAX_GROUPS = 256;
constexpr int RASTER = 8;                                // token tiles that are walked together, so that weights and activations both stay in L2

LLM_DEVICE uint32_t cluster_rank() { uint32_t r; asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
LLM_DEVICE uint32_t in_cta(uint32_t addr, uint32_t rank) { uint32_t r; asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank)); return r; }
LLM_DEVICE void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// An arrival in either CTA of the pair.  What it announces is tensor memory, written or read by tcgen05 instructions that have completed
// and are fenced.  A release would hold it back until the loads of the next chunk have come in as well.
LLM_DEVICE void arrive_cluster_if(uint32_t bar, bool pred) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %1, 0;\n\t@p mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];\n\t}" ::"r"(bar), "r"((uint32_t)pred) : "memory");
}
// 64 columns of this CTA's half of the tokens; the bytes are counted by the barrier of the pair's first CTA
LLM_DEVICE void tma_load_pair(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar) : "memory");
}
LLM_DEVICE void mma_pair_ts(uint32_t d, uint32_t a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(d), "r"(a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// completion of all MMAs so far, told to the barrier at this offset in both CTAs
LLM_DEVICE void commit_pair(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3) : "memory");
}

// One tile of the pair: 256 weight rows from 128 * n0, `cols` tokens (a multiple of 32) from row0, of which those below row_hi exist.
struct Tile { int n0, row0, row_hi, cols, group; };
struct Tiles {
    int n_pairs, m_tiles, bt, m;
    const int *rows, *firsts;            // grouped: first row and first tile of every group (shared memory), else nullptr
    int groups;
    LLM_DEVICE int count() const { return n_pairs * m_tiles; }
    LLM_DEVICE Tile at(int t) const {
        Tile u;
        if (firsts) {
            const int j = t / n_pairs;
            int lo = 0, hi = groups;
            while (hi - lo > 1) {
                const int mid = (lo + hi) >> 1;
                if (firsts[mid] <= j) lo = mid; else hi = mid;
            }
            u.n0 = 2 * (t - j * n_pairs);
            u.group = lo;
            u.row0 = rows[lo] + (j - firsts[lo]) * bt;
            u.row_hi = rows[lo + 1];
        } else {
            const int per = RASTER * n_pairs, q = t / per, r = t - q * per, h = min(RASTER, m_tiles - q * RASTER);
            u.n0 = 2 * (r / h);
            u.group = 0;
            u.row0 = (q * RASTER + r % h) * bt;
            u.row_hi = m;
        }
        u.cols = min(bt, (u.row_hi - u.row0 + 31) & ~31);
        return u;
    }
};

// RESID: the residual epilogue, else store or SwiGLU (one kernel with all of them was 2 to 5 % slower from Q6_K)
template <int FMT, bool RESID>
__global__ void __launch_bounds__(THREADS, 1) gemm_pair_kernel(const __grid_constant__ CUtensorMap tmap_x, const GemmTcParams p, const int bt) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t s_full[SLOTS], s_empty[SLOTS], s_acc_full, s_acc_empty;
    __shared__ uint32_t s_tmem;
    __shared__ int s_abort[2];           // [1] stays 0 here (tc_common.cuh)
    __shared__ int s_rows[MAX_GROUPS + 1], s_firsts[MAX_GROUPS + 1];
    __shared__ uint32_t s_grid[FMT == FMT_IQ3_S ? 512 : 1];
    pdl_wait();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t rank = cluster_rank();
    const int pair = blockIdx.x >> 1, n_clusters = gridDim.x >> 1;
    const int k_blocks = p.k / 256, n_tiles = (p.n + 127) / 128;
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t full_bar = smem_u32(s_full), empty_bar = smem_u32(s_empty), accf_bar = smem_u32(&s_acc_full), acce_bar = smem_u32(&s_acc_empty);

    if (tid == 0) {
        s_abort[0] = 0; s_abort[1] = 0;
        for (int s = 0; s < SLOTS; ++s) { mbar_init(full_bar + s * 8, 9); mbar_init(empty_bar + s * 8, 1); }       // full: four warps of each CTA, the bytes
        mbar_init(accf_bar, 1);
        mbar_init(acce_bar, 2 * DEQUANT_WARPS);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_proxy_async();
    }
    if (FMT == FMT_IQ3_S) {
        for (int i = tid; i < 512; i += THREADS) s_grid[i] = g_iq3s_grid[i];
    }
    if (p.groups > 0) {
        for (int i = tid; i <= p.groups; i += THREADS) { s_rows[i] = p.group_row_off[i]; s_firsts[i] = p.group_tile_off[i]; }
    }
    if (warp == DEQUANT_WARPS + 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();                      // the other CTA's barriers are initialised, its tensor memory is allocated
    tc_fence_after();
    pdl_trigger();                       // not before the allocation: CTAs of the next kernel must not come between
    const uint32_t tmem = s_tmem;
    volatile int* abort_flag = s_abort;
    const Tiles tiles{(n_tiles + 1) / 2, p.groups > 0 ? s_firsts[p.groups] : (p.m + bt - 1) / bt, bt, p.m, s_rows, p.groups > 0 ? s_firsts : nullptr, p.groups};
    const int count = tiles.count(), mine = count > pair ? (count - pair + n_clusters - 1) / n_clusters : 0;       // tiles of this pair
    auto tile = [&](int i) { return tiles.at(pair + i * n_clusters); };

    if (warp < DEQUANT_WARPS) {
        // ------------------------------ dequantisation and epilogue ------------------------------
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS_DEQUANT));
        const int g = warp & 3, set = warp >> 2;
        const uint32_t t_lane = tmem + ((uint32_t)(g * 32) << 16);
        const uint32_t acce_first = in_cta(acce_bar, 0);

        auto epilogue = [&](int i) -> bool {
            const Tile t = tile(i);
            if (!mbar_wait_warp(accf_bar, i & 1, abort_flag)) return false;
            tc_fence_after();
            uint32_t r[4][32];           // blocks set, set + 2, ... of 32 tokens
#pragma unroll
            for (int b = 0; b < 4; ++b)
                if ((set + 2 * b) * 32 < t.cols) tmem_ld32_issue(t_lane + (set + 2 * b) * 32, r[b]);
#pragma unroll
            for (int b = 0; b < 4; ++b) tmem_wait_ld(r[b]);
            tc_fence_before();
            __syncwarp();
            arrive_cluster_if(acce_first, lane == 0);
            const int tile_n = t.n0 + (int)rank, n_row = tile_n * 128 + g * 32 + lane;
            if (tile_n >= n_tiles) return true;                    // the pair's second half past an odd number of tiles
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                const int c0 = (set + 2 * b) * 32, m0 = t.row0 + c0;
                if (c0 >= t.cols) break;
                if (!RESID && p.epi == EPI_SWIGLU) {
                    // rows of a 32-row group: 16 gate rows, then the 16 matching up rows.  Lanes l and l + 16 hold one output column;
                    // the lower lane finishes the even tokens and the upper lane the odd ones, so one exchange serves two.
                    const int col = tile_n * 64 + g * 16 + (lane & 15);
                    const bool lower = lane < 16;
                    __nv_bfloat16* o = static_cast<__nv_bfloat16*>(p.out) + (size_t)(m0 + (lower ? 0 : 1)) * p.out_stride + col;
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        const float even = __uint_as_float(r[b][2 * j]), odd = __uint_as_float(r[b][2 * j + 1]);
                        const float got = __shfl_xor_sync(0xffffffffu, lower ? odd : even, 16);
                        const float gate = lower ? even : got, up = lower ? got : odd;
                        if (col < p.n / 2 && m0 + 2 * j + (lower ? 0 : 1) < t.row_hi) o[(size_t)(2 * j) * p.out_stride] = __float2bfloat16(silu(gate) * up);
                    }
                    continue;
                }
                if (n_row >= p.n) continue;
                const float bias = p.bias ? p.bias[n_row] : 0.f;
                if constexpr (RESID) {
                    // one addition to every element, made in L2: read, added and written here they were a chain of sixteen trips
                    // to L2 (4096 x 4096 Q4_K, 1024 rows: 42 us, 34 so; 4096 rows: 172 and 128)
                    float* h = static_cast<float*>(p.out) + (size_t)m0 * p.out_stride + n_row;
#pragma unroll
                    for (int j = 0; j < 32; ++j)
                        if (m0 + j < t.row_hi)
                            asm volatile("red.relaxed.gpu.global.add.f32 [%0], %1;" ::"l"(h + (size_t)j * p.out_stride), "f"(__uint_as_float(r[b][j]) + bias) : "memory");
                    continue;
                }
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                    if (m0 + j >= t.row_hi) continue;
                    const size_t at = (size_t)(m0 + j) * p.out_stride + n_row;
                    const float v = __uint_as_float(r[b][j]) + bias;
                    if (p.out_f32) static_cast<float*>(p.out)[at] = v;
                    else static_cast<__nv_bfloat16*>(p.out)[at] = __float2bfloat16(v);
                }
            }
            return true;
        };

        const uint32_t t_slot = t_lane + COL_A + set * 128, full_first = in_cta(full_bar, 0) + set * 32, empty = empty_bar + set * 32;
        bool ok = true;
        uint32_t parity = 1;
        // the 64 columns of this lane's row into slot `k` of the set, once it is free, and on to the MMA warp
        auto put = [&](int k, const uint32_t (&o)[32]) {
            if (ok) ok = mbar_wait_warp(empty + k * 8, parity, abort_flag);
            if (!ok) return;
            tc_fence_after();
            tmem_st32(t_slot + k * 32, o);
            tmem_wait_st();
            tc_fence_before();
            arrive_cluster_if(full_first + k * 8, lane == 0);
        };
        // Chunks of this set: every second one of the pair's sequence (tile by tile, k_blocks each).  A set converts its first chunk of
        // a tile before it turns to the epilogue of the tile before.
        int i = 0, kb = set, done = 0, left = 0;
        bool inside = false;             // this set has converted a chunk of tile i; `left`: the tile before that
        auto settle = [&]() { while (kb >= k_blocks) { kb -= k_blocks; ++i; } };
        auto chunk_at = [&](int i, int kb) {
            const Tile t = tile(i);
            return p.w + (size_t)t.group * p.w_group_stride + ((size_t)min(t.n0 + (int)rank, n_tiles - 1) * k_blocks + kb) * FmtTraits<FMT>::CHUNK;
        };
        settle();
        using Half = HalfChunk<FMT>;
        typename Half::Regs regs[2];
        const uint8_t* chunk = i < mine ? chunk_at(i, kb) : nullptr;
#pragma unroll
        for (int h = 0; h < 2; ++h)
            if (chunk) regs[h] = Half::load(chunk, g, lane, h);
#pragma unroll 1
        for (int u = 0; ok; ++u) {
            const int due = i >= mine ? mine : inside ? i : left;
#pragma unroll 1
            for (; done < due && ok; ++done) ok = epilogue(done);
            if (i >= mine || !ok) break;
            const int was = i;
            kb += 2;
            settle();
            chunk = i < mine ? chunk_at(i, kb) : nullptr;
            parity = (u & 1) ^ 1;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint32_t o[32];
                Half::template atom<0>(regs[h], h, o, s_grid);
                put(2 * h, o);
                Half::template atom<1>(regs[h], h, o, s_grid);
                put(2 * h + 1, o);
                if (chunk) regs[h] = Half::load(chunk, g, lane, h);      // this set's next chunk, on its way while the other half is converted
            }
            inside = i == was;
            if (!inside) left = was;
        }
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS_OTHER));
        if (warp == DEQUANT_WARPS && elect_one()) {
            // ------------------------------ activations: this CTA's half of the tokens ------------------------------
            const uint32_t full_first = in_cta(full_bar, 0);
            bool ok = true;
            int gc = 0;
            for (int i = 0; i < mine && ok; ++i) {
                const Tile t = tile(i);
                const int y = t.row0 + (int)rank * (t.cols / 2);
                for (int kb = 0; kb < k_blocks && ok; ++kb, ++gc) {
                    for (int a = 0; a < 4; ++a) {
                        const int slot = (gc & 1) * 4 + a;
                        ok = mbar_wait(empty_bar + slot * 8, ((gc >> 1) & 1) ^ 1, abort_flag);
                        if (!ok) break;
                        if (rank == 0) mbar_arrive_expect_tx(full_bar + slot * 8, bt * 128);          // both halves
                        tma_load_pair(smem_base + slot * SLOT_BYTES, &tmap_x, kb * 256 + a * 64, y, full_first + slot * 8);
                    }
                }
            }
            // the last commits have arrived here before this CTA may leave
            for (int c = gc > 2 ? gc - 2 : 0; c < gc && ok; ++c)
                for (int a = 0; a < 4 && ok; ++a) ok = mbar_wait(empty_bar + ((c & 1) * 4 + a) * 8, (c >> 1) & 1, abort_flag);
        } else if (warp == DEQUANT_WARPS + 1 && rank == 0 && elect_one()) {
            // ------------------------------ MMA issue for both CTAs ------------------------------
            bool ok = true;
            int gc = 0;
            for (int i = 0; i < mine && ok; ++i) {
                const Tile t = tile(i);
                // bf16 x bf16 -> fp32, both K-major, M = 256, N = t.cols
                const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(t.cols >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
                ok = mbar_wait(acce_bar, (i & 1) ^ 1, abort_flag);
                for (int kb = 0; kb < k_blocks && ok; ++kb, ++gc) {
#pragma unroll
                    for (int a = 0; a < 4; ++a) {
                        const int slot = (gc & 1) * 4 + a;
                        if (ok) ok = mbar_wait(full_bar + slot * 8, (gc >> 1) & 1, abort_flag);
                        if (!ok) break;
                        tc_fence_after();
                        const uint64_t bdesc = smem_desc_sw128(smem_base + slot * SLOT_BYTES);
                        const uint32_t a_tmem = tmem + COL_A + slot * 32;
#pragma unroll
                        for (int k4 = 0; k4 < 4; ++k4) mma_pair_ts(tmem, a_tmem + k4 * 8, bdesc + 2 * k4, idesc, (kb > 0 || a > 0 || k4 > 0) ? 1u : 0u);
                        commit_pair(empty_bar + slot * 8);
                    }
                }
                if (ok) commit_pair(accf_bar);
            }
        }
    }

    // ------------------------------ teardown: nobody leaves while the other CTA may still reach it ------------------------------
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    cluster_sync();
    if (abort_flag[0]) {
        if (tid == 0 && p.status) atomicExch(p.status, (int)STATUS_TIMEOUT);
        for (int i = 0; i < 2000; ++i) __nanosleep(100);      // let copies still in flight land before the memory is reused
    }
    __syncthreads();
    cluster_sync();
    if (warp == DEQUANT_WARPS + 1) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
}

template <int FMT, bool RESID>
static cudaError_t launch_one(const GemmTcParams& p, int bt, cudaStream_t st) {
    static bool attr_set = false;
    if (!attr_set) {
        const cudaError_t e = raise_smem(gemm_pair_kernel<FMT, RESID>, SMEM_BYTES);
        if (e != cudaSuccess) return e;
        attr_set = true;
    }
    CUtensorMap map;
    if (!make_map(&map, p.x, p.k, p.m, p.k, bt / 2)) return cudaErrorInvalidValue;
    const long long pairs = ((p.n + 127) / 128 + 1) / 2, tiles = pairs * ((p.m + bt - 1) / bt + p.groups);
    const int clusters = (int)(tiles < sm_count() / 2 ? tiles : sm_count() / 2);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * clusters); cfg.blockDim = dim3(THREADS); cfg.dynamicSmemBytes = SMEM_BYTES; cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = pdl_enabled() ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, gemm_pair_kernel<FMT, RESID>, map, p, bt);
}
template <int FMT>
static cudaError_t launch_fmt(const GemmTcParams& p, int bt, cudaStream_t st) {
    return p.epi == EPI_RESID ? launch_one<FMT, true>(p, bt, st) : launch_one<FMT, false>(p, bt, st);
}

}  // namespace tcp

// Tokens of a tile: the multiple of 32 (at most 256) with the shortest run of tiles on the busiest pair.  A chunk takes as long as its
// MMAs (1.5 us with 256 tokens) or as its conversion (1.1 us from Q4_K and Q4_0, 1.4 us from the others), whichever is longer, a tile
// some of that time more for its start and end.
int gemm_pair_tokens(int fmt, int m, int n, int k) {
    const int pairs = ((n + 127) / 128 + 1) / 2, kb = k / 256, slots = sm_count() / 2;
    const double least_chunk = fmt == FMT_Q4_K || fmt == FMT_Q4_0 ? 0.7 : 0.9;
    int best = 256;
    double least = 0.;
    for (int bt = 256; bt >= 32; bt -= 32) {
        const double waves = (double)(((long long)pairs * ((m + bt - 1) / bt) + slots - 1) / slots), chunk = bt / 256.;
        const double cost = waves * (kb * (chunk > least_chunk ? chunk : least_chunk) + 0.5 + chunk);
        if (bt == 256 || cost < 0.97 * least) { least = cost; best = bt; }
    }
    return best;
}

cudaError_t launch_gemm_tc_pair(const GemmTcParams& p, int bt, cudaStream_t st) {
    if (bt < 32 || bt > 256 || bt % 32 || p.groups > tcp::MAX_GROUPS) return cudaErrorInvalidValue;
    switch (p.fmt) {
        case FMT_Q4_K: return tcp::launch_fmt<FMT_Q4_K>(p, bt, st);
        case FMT_Q5_K: return tcp::launch_fmt<FMT_Q5_K>(p, bt, st);
        case FMT_Q6_K: return tcp::launch_fmt<FMT_Q6_K>(p, bt, st);
        case FMT_Q8_0: return tcp::launch_fmt<FMT_Q8_0>(p, bt, st);
        case FMT_Q4_0: return tcp::launch_fmt<FMT_Q4_0>(p, bt, st);
        case FMT_IQ3_S: return tcp::launch_fmt<FMT_IQ3_S>(p, bt, st);
    }
    return cudaErrorInvalidValue;
}

}  // namespace llm
