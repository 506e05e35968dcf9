// GEMMs on the 5th-generation tensor cores: D(M x N) = A(M x K) B(N x K)^T, both operands bf16 and K-major, f32
// accumulation in tensor memory, D stored as f32 (row-major, ldd) for the rows < M and columns < N.
//
// Two kinds:
//  * split-BF16 (three products): A = A_hi + A_lo, B = B_hi + B_lo, D = A_hi B_hi + A_hi B_lo + A_lo B_hi. The
//    reverse pass's weight cotangent (backward_age_sums, OpenSPS src/physics/opensps_csp_batch.f90:5226-5300) and
//    the SSP operator's template GEMM (template_columns, src/physics/opensps_ssp_batch.f90:3247-3385) use it.
//  * one product, bf16 or f16 operands: the emulator's training GEMMs (forward in f16; input cotangents and
//    weight gradients in bf16).
//
// Groups and split-K: the tile index runs over (group, K split, M tile, N tile). Group g reads the A rows from
// g * a_grp, the B rows from g * b_grp and writes D from g * d_grp (elements); K split s covers the K blocks
// [s * nkb / ksplit, (s + 1) * nkb / ksplit) and writes its partial sums from s * d_split. The emulator's five
// ensemble members are the groups; the weight gradients (K = the minibatch) are split over K.
//
// Slabs (mtab): the operator's fold of models whose weights lie in two metallicity slabs z, z + 1 of every age. An M tile
// holds rows of one z; a K block is 64 columns of an age's two slabs (slab2 columns, contiguous in A's rows at age slab2
// and in B's at age age_cols + z slab2 / 2), so that the other slabs' columns, all zero in A, are neither read nor
// multiplied.
//
// Tile 128 x 256 x 64, or 256 x 256 x 64 by a CTA pair (three products, gemm_pairs), persistent CTAs over tiles; warp 0 =
// TMA producer, warp 1 = MMA issuer and TMEM owner,
// warps 2..5 = epilogue (one accumulator row per thread); TMEM double-buffered. Two smem stages of 96 KB (split), three
// of 64 KB (split, a CTA of a pair) or four of 48 KB (plain). Every mbarrier wait is bounded (status word, no hang).
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <algorithm>
#include <cstdint>
#include "sm103_ptx.cuh"
#include "csp_kernels.h"

namespace sps {

constexpr int G_BM = 128, G_BN = 256, G_BK = 64;
constexpr int G_A_BYTES = G_BM * G_BK * 2, G_B_BYTES = G_BN * G_BK * 2;
constexpr int G_THREADS = 6 * 32;

template <int NPROD, int CTAS = 1>
struct GemmCfg {
    static constexpr int B_BYTES = G_B_BYTES / CTAS;     // a pair's CTA holds half of the tile's B rows
    static constexpr int STAGE_BYTES = NPROD == 3 ? 2 * G_A_BYTES + 2 * B_BYTES : G_A_BYTES + B_BYTES;
    static constexpr int STAGES = NPROD == 3 ? (CTAS == 2 ? 3 : 2) : 4;
    static constexpr int SMEM = STAGES * STAGE_BYTES + 256 + 1024;
};

struct GemmTile {
    int g, s, m0, n0, rows, z;   // rows: of D from m0 that this tile stores (an end); z: its slab (GemmArgs::mtab)
};
template <bool SLABS, int CTAS>
__device__ __forceinline__ GemmTile gemm_tile(const GemmArgs &g, int tile, int mt_n, int nt_n, int rank) {
    GemmTile t;
    t.m0 = (tile % mt_n * CTAS + rank) * G_BM;
    t.rows = g.M;
    t.z = 0;
    if constexpr (SLABS) {
        const int4 e = __ldg(g.mtab + tile % mt_n);
        t.m0 = e.x; t.rows = e.y; t.z = e.z;
    }
    int r = tile / mt_n;
    t.n0 = (r % nt_n) * G_BN;
    r /= nt_n;
    t.s = r % g.ksplit;
    t.g = r / g.ksplit;
    return t;
}

// CTAS = 2: a CTA pair takes 256 x 256, half of A's and of B's rows in each CTA's shared memory (CTA 0 issues the MMAs).
template <int NPROD, bool SLABS, int CTAS>
__global__ void __launch_bounds__(G_THREADS, 1)
gemm_bf16_kernel(const __grid_constant__ CUtensorMap tm_a_hi, const __grid_constant__ CUtensorMap tm_a_lo,
                 const __grid_constant__ CUtensorMap tm_b_hi, const __grid_constant__ CUtensorMap tm_b_lo,
                 GemmArgs g) {
    using C = GemmCfg<NPROD, CTAS>;
    constexpr int NS = C::STAGES;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + NS * C::STAGE_BYTES);
    uint64_t *full = bars, *empty = bars + NS, *tfull = bars + 2 * NS, *tempty = bars + 2 * NS + 2;
    uint64_t *mma_done = bars + 2 * NS + 4;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 2 * NS + 5);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = CTAS == 2 ? (int)cluster_ctarank() : 0, tile0 = blockIdx.x / CTAS, tile_step = gridDim.x / CTAS;
    const int mt_n = SLABS ? g.n_mtiles : (g.M + CTAS * G_BM - 1) / (CTAS * G_BM), nt_n = (g.N + G_BN - 1) / G_BN;
    const int n_tiles = mt_n * nt_n * g.ksplit * g.groups;
    // (SLABS: K blocks of an age's two slabs, kpa of them, the last of tail_steps steps of 16 columns)
    const int kpa = SLABS ? (g.slab2 + G_BK - 1) / G_BK : 1, nkb = SLABS ? g.ages * kpa : (g.K + G_BK - 1) / G_BK;
    const int tail_steps = SLABS ? (g.slab2 - (kpa - 1) * G_BK + 15) / 16 : G_BK / 16;
    int *status = g.status;

    if (threadIdx.x == 0) {
        for (int s = 0; s < NS; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(&tfull[b], 1); mbar_init(&tempty[b], CTAS * 4); }
        mbar_init(mma_done, 1);
        fence_mbar_init();
    }
    if (warp == 1) {
        if constexpr (CTAS == 2) { tmem_alloc_pair(tmem_slot, 512); tmem_relinquish_pair(); }
        else { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
    }
    tc_fence_before();
    __syncthreads();
    if constexpr (CTAS == 2) cluster_sync();      // (the barriers of both CTAs are ready)
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            int s = 0; uint32_t ph = 0;
            int last_fill[NS];
            for (int i = 0; i < NS; ++i) last_fill[i] = -1;
            bool ok = true;
            for (int tile = tile0; tile < n_tiles && ok; tile += tile_step) {
                const GemmTile t = gemm_tile<SLABS, CTAS>(g, tile, mt_n, nt_n, rank);
                const int arow = (int)(t.g * g.a_grp) + t.m0;
                const int brow = (int)(t.g * g.b_grp) + g.b_row0 + t.n0 + rank * (G_BN / CTAS);
                const int kb0 = t.s * nkb / g.ksplit, kb1 = (t.s + 1) * nkb / g.ksplit;
                for (int kb = kb0; kb < kb1; ++kb) {
                    if (!mbar_wait(&empty[s], ph ^ 1u, status, ERR_TIMEOUT_PRODUCER)) { ok = false; break; }
                    uint8_t *st = smem + s * C::STAGE_BYTES;
                    // (a pair's copies, of both CTAs, complete on CTA 0's barrier, whose phase its producer arms for all)
                    if (rank == 0) mbar_arrive_expect_tx(&full[s], CTAS * C::STAGE_BYTES);
                    if (NPROD == 3) {
                        int xa = kb * G_BK, xb = xa;
                        if constexpr (SLABS) {
                            const int age = kb / kpa, off = (kb - age * kpa) * G_BK;
                            xa = age * g.slab2 + off;
                            xb = age * g.age_cols + t.z * (g.slab2 / 2) + off;
                        }
                        uint8_t *b_hi = st + 2 * G_A_BYTES, *b_lo = b_hi + C::B_BYTES;
                        if constexpr (CTAS == 2) {
                            const uint32_t bar = cluster_addr(&full[s], 0);
                            tma_load_2d_pair(st, &tm_a_hi, xa, arow, bar);
                            tma_load_2d_pair(st + G_A_BYTES, &tm_a_lo, xa, arow, bar);
                            tma_load_2d_pair(b_hi, &tm_b_hi, xb, brow, bar);
                            tma_load_2d_pair(b_lo, &tm_b_lo, xb, brow, bar);
                        } else {                  // (B's box is 128 rows, a pair's half)
                            tma_load_2d(st, &tm_a_hi, xa, arow, &full[s]);
                            tma_load_2d(st + G_A_BYTES, &tm_a_lo, xa, arow, &full[s]);
                            tma_load_2d(b_hi, &tm_b_hi, xb, brow, &full[s]);
                            tma_load_2d(b_hi + G_B_BYTES / 2, &tm_b_hi, xb, brow + G_BN / 2, &full[s]);
                            tma_load_2d(b_lo, &tm_b_lo, xb, brow, &full[s]);
                            tma_load_2d(b_lo + G_B_BYTES / 2, &tm_b_lo, xb, brow + G_BN / 2, &full[s]);
                        }
                    } else {
                        tma_load_2d(st, &tm_a_hi, kb * G_BK, arow, &full[s]);
                        tma_load_2d(st + G_A_BYTES, &tm_b_hi, kb * G_BK, brow, &full[s]);
                    }
                    last_fill[s] = (int)ph;
                    if (++s == NS) { s = 0; ph ^= 1u; }
                }
            }
            for (int i = 0; i < NS; ++i)
                if (last_fill[i] >= 0 && rank == 0) mbar_wait(&full[i], (uint32_t)last_fill[i], status, ERR_TIMEOUT_PRODUCER, false);
        }
    } else if (warp == 1) {
        if (lane == 0 && rank == 0) {
            auto mma = [](uint32_t d, uint64_t da, uint64_t db, uint32_t id, uint32_t accum) {
                if constexpr (CTAS == 2) mma_bf16_pair(d, da, db, id, accum);
                else mma_bf16(d, da, db, id, accum);
            };
            auto commit = [](uint64_t *bar) {
                if constexpr (CTAS == 2) mma_commit_pair(bar);
                else mma_commit(bar);
            };
            int s = 0; uint32_t ph = 0;
            int acc = 0; uint32_t aph = 0;
            bool ok = true;
            for (int tile = tile0; tile < n_tiles && ok; tile += tile_step) {
                const GemmTile t = gemm_tile<SLABS, CTAS>(g, tile, mt_n, nt_n, rank);
                const int kb0 = t.s * nkb / g.ksplit, kb1 = (t.s + 1) * nkb / g.ksplit;
                if (!mbar_wait(&tempty[acc], aph ^ 1u, status, ERR_TIMEOUT_MMA)) { ok = false; break; }
                tc_fence_after();
                const uint32_t d = tmem_base + acc * G_BN;
                const uint32_t idesc = (NPROD == 1 && g.f16) ? idesc_f16_f32(G_BM, G_BN) : idesc_bf16_f32(CTAS * G_BM, G_BN);
                for (int kb = kb0; kb < kb1; ++kb) {
                    if (!mbar_wait(&full[s], ph, status, ERR_TIMEOUT_MMA)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t sa = smem_u32(smem + s * C::STAGE_BYTES);
#pragma unroll
                    for (int k = 0; k < G_BK / 16; ++k) {
                        if (SLABS && k >= tail_steps && kb % kpa == kpa - 1) break;
                        const uint32_t off = k * 32;
                        const uint32_t first = (kb > kb0 || k > 0) ? 1u : 0u;
                        if (NPROD == 3) {
                            const uint32_t a_hi = sa, a_lo = sa + G_A_BYTES, b_hi = sa + 2 * G_A_BYTES, b_lo = b_hi + C::B_BYTES;
                            mma(d, sw128_desc(a_hi + off), sw128_desc(b_hi + off), idesc, first);
                            mma(d, sw128_desc(a_hi + off), sw128_desc(b_lo + off), idesc, 1u);
                            mma(d, sw128_desc(a_lo + off), sw128_desc(b_hi + off), idesc, 1u);
                        } else {
                            mma(d, sw128_desc(sa + off), sw128_desc(sa + G_A_BYTES + off), idesc, first);
                        }
                    }
                    commit(&empty[s]);
                    if (++s == NS) { s = 0; ph ^= 1u; }
                }
                if (!ok) break;
                commit(&tfull[acc]);
                if (++acc == 2) { acc = 0; aph ^= 1u; }
            }
            commit(mma_done);
            mbar_wait(mma_done, 0, status, ERR_TIMEOUT_MMA, false);
        }
    } else {
        // epilogue: warp w reads TMEM lanes 32 (w % 4) .. : one row of D per thread
        const int q = warp & 3;
        int acc = 0; uint32_t aph = 0;
        for (int tile = tile0; tile < n_tiles; tile += tile_step) {
            const GemmTile t = gemm_tile<SLABS, CTAS>(g, tile, mt_n, nt_n, rank);
            mbar_wait(&tfull[acc], aph, status, ERR_TIMEOUT_EPILOGUE);
            named_bar_sync(1, 128);
            if (*(volatile int *)status != 0) break;
            tc_fence_after();
            const int row = t.m0 + q * 32 + lane;
            const uint32_t trow = tmem_base + ((uint32_t)(q * 32) << 16) + acc * G_BN;
            float *dbase = g.D + t.g * g.d_grp + t.s * g.d_split;
            for (int c = 0; c < G_BN; c += 32) {
                if (t.n0 + c >= g.N) break;
                float v[32];
                tmem_ld32(trow + c, v);
                if (row < t.rows) {
                    float *dst = dbase + (size_t)row * g.ldd + t.n0 + c;
                    if (t.n0 + c + 32 <= g.N && ((g.ldd | g.d_grp | g.d_split) & 3) == 0) {
#pragma unroll
                        for (int i = 0; i < 32; i += 4)
                            *reinterpret_cast<float4 *>(dst + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
                    } else {
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            if (t.n0 + c + i < g.N) dst[i] = v[i];
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                if constexpr (CTAS == 2) mbar_arrive_cluster(cluster_addr(&tempty[acc], 0));
                else mbar_arrive(&tempty[acc]);
            }
            if (++acc == 2) { acc = 0; aph ^= 1u; }
        }
    }
    tc_fence_before();
    __syncthreads();
    // (a pair's CTAs leave together: CTA 0's MMAs read CTA 1's shared memory, CTA 1 arrives on CTA 0's barriers)
    if constexpr (CTAS == 2) cluster_sync();
    if (warp == 1) {
        tc_fence_after();
        if constexpr (CTAS == 2) tmem_dealloc_pair(tmem_base, 512);
        else tmem_dealloc(tmem_base, 512);
    }
}

int gemm_bk() { return G_BK; }
int gemm_bm() { return G_BM; }
int gemm_bn() { return G_BN; }
int gemm_box_n() { return G_BN / 2; }

static long long gemm_tiles(long long rows, int tile) { return (rows + tile - 1) / tile; }

// K splits for a GEMM of tiles_mn output tiles over nkb K blocks: the fewest giving at least two waves over the SMs
// with the last wave at least 85% full (else the fullest last wave), each split keeping 8 or more K blocks.
int gemm_choose_ksplit(int tiles_mn, int nkb, int num_sms) {
    int best = 1;
    double best_eff = -1.0;
    const int cap = std::max(1, std::min(64, nkb / 8));
    for (int ks = 1; ks <= cap; ++ks) {
        const long long tiles = (long long)tiles_mn * ks, waves = (tiles + num_sms - 1) / num_sms;
        const double eff = (double)tiles / (double)(waves * num_sms);
        if (tiles >= 2LL * num_sms && eff >= 0.85) return ks;
        if (eff > best_eff + 1e-9) { best_eff = eff; best = ks; }
    }
    return best;
}

template <int NPROD, bool SLABS = false, int CTAS = 1>
static cudaError_t launch_gemm(const GemmPlan &pl, const GemmArgs &g, cudaStream_t st) {
    if (g.M <= 0 || g.N <= 0 || g.K <= 0 || g.groups <= 0 || g.ksplit <= 0) return cudaSuccess;
    const int nkb = SLABS ? g.ages * ((g.slab2 + G_BK - 1) / G_BK) : (g.K + G_BK - 1) / G_BK;
    if (g.ksplit > nkb) return cudaErrorInvalidValue;          // every split needs a K block
    if ((reinterpret_cast<uintptr_t>(g.D) & 15) != 0) return cudaErrorInvalidValue;
    using C = GemmCfg<NPROD, CTAS>;
    auto kern = gemm_bf16_kernel<NPROD, SLABS, CTAS>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
    if (e != cudaSuccess) return e;
    const long long tiles = (SLABS ? g.n_mtiles : gemm_tiles(g.M, CTAS * G_BM)) * gemm_tiles(g.N, G_BN) * g.ksplit * g.groups;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(CTAS * std::min<long long>(tiles, pl.num_sms / CTAS)));
    cfg.blockDim = dim3(G_THREADS);
    cfg.dynamicSmemBytes = C::SMEM;
    cfg.stream = st;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = CTAS;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = CTAS > 1 ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, pl.tm_a_hi, pl.tm_a_lo, pl.tm_b_hi, pl.tm_b_lo, g);
}

// Pairs where their waves cost less: an MMA of 256 x 256 over two SMs takes 147 cycles against 200 for 128 x 256 in one
// (each SM reads 8 KB of operands from shared memory instead of 12), but the pairs' tiles are coarser. Measured, one CTA
// -> pairs: the operator's templates at 1024 models (2048 x 5994 x 2752) 152 -> 142 us (8.8 TB/s of operands from L2 to
// shared memory), at 100 models 56 -> 49; the reverse pass's weights at 2000 models 38.5 -> 34.5 and 60 -> 52.
static bool gemm_pairs(const GemmPlan &pl, const GemmArgs &g) {
    const long long rest = gemm_tiles(g.N, G_BN) * g.ksplit * g.groups, pairs = std::max(pl.num_sms / 2, 1);
    const long long one = (gemm_tiles(g.M, G_BM) * rest + pl.num_sms - 1) / pl.num_sms;
    const long long two = (gemm_tiles(g.M, 2 * G_BM) * rest + pairs - 1) / pairs;
    return pl.num_sms >= 2 && two * 147 < one * 200;
}

cudaError_t run_gemm_bf16x3(const GemmPlan &pl, const GemmArgs &g, cudaStream_t st) {
    if (g.mtab) return launch_gemm<3, true>(pl, g, st);
    return gemm_pairs(pl, g) ? launch_gemm<3, false, 2>(pl, g, st) : launch_gemm<3>(pl, g, st);
}
cudaError_t run_gemm_bf16(const GemmPlan &pl, const GemmArgs &g, cudaStream_t st) { return launch_gemm<1>(pl, g, st); }

}  // namespace sps
