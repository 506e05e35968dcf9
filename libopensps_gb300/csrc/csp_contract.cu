// The CSP contraction with its fused per-pixel epilogue, on the 5th-generation tensor cores.
//
//   spec(p, m) = S( [ young(p, m) (T_birth (1 - frac_obrun) + frac_obrun) + old(p, m) T_dust3 ]
//                   (T_diffuse (1 - frac_nodust) + frac_nodust) T_igm(p, m) )
//   young / old(p, m) = sum_k basis(p, k) w(k, m) over the ages <= / > dust_tesc (k = age x metallicity)
//
// (OpenSPS compute_csp_batch stages 3-7: age_sums_w src/physics/opensps_csp_batch.f90:2269-2324, attenuate_batch
// :3576-3660, apply_igm_z :4205-4299, smoothing src/spectra/opensps_smoothing.f90:553-633.) The nebular lines are in
// the basis already (they are linear in the weights: the basis holds each young SSP with its lines).
//
// Matrix form: D(pixels x models) = basis(pixels x K) . W(models x K)^T, both operands K-major bf16 split into hi and
// lo parts (x = x_hi + x_lo); D = A_hi B_hi + A_hi B_lo + A_lo B_hi, accumulated in f32 in tensor memory. Tile: 128
// pixels x BN models x 64 K per stage; the 128 pixel rows of a tile are 120 output pixels with a halo of 4 on each
// side for the smoothing; BN is the largest tile (256 models, 128 with two accumulators) or a narrower one of a smaller
// batch, with the stages that fit (contract_tile); a CTA pair takes two pixel tiles by BN models in one MMA (with an odd
// count of pixel tiles the last pair's second CTA multiplies zeros and stores nothing). The 16-column K steps past a
// range's last column are left out (81 steps of 84 for 107 ages x 12 metallicities). One CTA per SM, persistent over
// tiles (model tile outer, pixel tile inner, so that the CTAs running together share the weights of a model tile in L2).
// Warp roles: warp 0 = TMA producer, warp 1 = MMA issuer (and TMEM owner; in a pair CTA 0's), the others = epilogue in
// groups of four (group g takes the models of the g-th part of the columns; in a group, warp w reads TMEM lanes
// 32 (w % 4) ..): four groups (with two the epilogue was the longer part of a pair's tile, 1820 us at 65536 models
// against 1591). Accumulators are double-buffered in TMEM so that the epilogue of a tile overlaps the MMAs of the next.
//
// Epilogue of a chunk of 8 models, per group: phase 1, thread = pixel row: the attenuated, IGM-absorbed spectrum
// of the chunk's models into a staging tile; phase 2, thread = 4 consecutive output pixels of one model: the velocity
// smoothing (taps in registers) and the store.
//
// NACC = 1: one accumulator (no birth-cloud or old-star screen in the batch: young and old are only ever summed).
// NACC = 2: young and old accumulators (the K range is ordered young block first, then old block).
// Nebular emission's escaping ionizing light (frac_obrun above 0, nebular_kernels step 2 of OpenSPS,
// src/physics/opensps_csp_batch.f90:2726-2750): the basis holds the nebular ages' ionizing pixels absorbed (zero), and
// extra K blocks after the old block hold those ages' unabsorbed ionizing spectra against the weights times each
// model's escaping fraction; the ion young blocks accumulate into the young sums and the ion old blocks into the old
// ones. Only the pixel tiles that reach an ionizing pixel run them.
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <algorithm>
#include <cstdint>
#include "sm103_ptx.cuh"
#include "csp_kernels.h"

namespace sps {

constexpr int BM = 128;          // pixel rows per tile (MMA M)
constexpr int BK = 64;           // K per stage (one 128-byte swizzled row of bf16)
constexpr int HALO = 4;          // smoothing halo (taps -4 .. 4)
constexpr int OUT_ROWS = BM - 2 * HALO;
constexpr int MAX_STAGES = 4;    // stages of a tile of few models (2 at the full tile)
constexpr int TROW = BM + 4;     // staging row (floats): 16-byte aligned rows, and room for the phase-2 reads

template <int NACC, int CTAS>
struct ContractCfg {
    static constexpr int BN = (NACC == 1) ? 256 : 128;           // most models per tile (MMA N)
    static constexpr int A_BYTES = BM * BK * 2;                   // one of A_hi / A_lo
    static constexpr int STAGE_SMEM = 2 * (2 * A_BYTES + 2 * BN * BK * 2);   // the stages' shared memory
    static constexpr int ACC_COLS = NACC * BN;                    // TMEM columns of one accumulator set
    static constexpr int TMEM_COLS = 2 * ACC_COLS;                // double-buffered (= 512)
    static constexpr int EPI_GROUPS = 4;
    static constexpr int EPI_WARPS = 4 * EPI_GROUPS;
    static constexpr int NTHREADS = (2 + EPI_WARPS) * 32;
    static constexpr int CHUNK = 8;                               // models per epilogue chunk
    static constexpr int STAGE_T_FLOATS = CHUNK * TROW;           // per group
    static constexpr int PAR_FLOATS = 2 * CHUNK * MODEL_PAR_FLOATS;   // per group, double-buffered
    static constexpr int EPI_BYTES = EPI_GROUPS * (STAGE_T_FLOATS + PAR_FLOATS) * 4;
    static constexpr int SMEM_BYTES = STAGE_SMEM + EPI_BYTES + 256 + 1024;
    // a CTA's stage of tiles of bn models (a pair's CTAs hold half of the models each), and the stages that fit
    static constexpr __host__ __device__ int stage_bytes(int bn) { return 2 * A_BYTES + 2 * (bn / CTAS) * BK * 2; }
    static constexpr __host__ __device__ int stages(int bn) {
        return STAGE_SMEM / stage_bytes(bn) < MAX_STAGES ? STAGE_SMEM / stage_bytes(bn) : MAX_STAGES;
    }
};

// 2^x by the SFU (relative error ~2^-22; flushes results below the smallest normal to zero).
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// 8 consecutive f32 columns of this warp's 32 TMEM lanes.
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float *v) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}

template <int NACC, int CTAS>
__global__ void __launch_bounds__(ContractCfg<NACC, CTAS>::NTHREADS, 1)
csp_contract_kernel(const __grid_constant__ CUtensorMap tm_a_hi, const __grid_constant__ CUtensorMap tm_a_lo,
                    const __grid_constant__ CUtensorMap tm_b_hi, const __grid_constant__ CUtensorMap tm_b_lo,
                    ContractArgs args) {
    using C = ContractCfg<NACC, CTAS>;
    constexpr int EPI_GROUPS = C::EPI_GROUPS, EPI_WARPS = C::EPI_WARPS, CHUNK = C::CHUNK;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t *stage_base = smem;
    float *epi_base = reinterpret_cast<float *>(smem + C::STAGE_SMEM);
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + C::STAGE_SMEM + C::EPI_BYTES);
    uint64_t *full = bars;                     // [MAX_STAGES]
    uint64_t *empty = bars + MAX_STAGES;       // [MAX_STAGES]
    uint64_t *tfull = bars + 2 * MAX_STAGES;   // [2]
    uint64_t *tempty = bars + 2 * MAX_STAGES + 2;
    uint64_t *mma_done = bars + 2 * MAX_STAGES + 4;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 2 * MAX_STAGES + 5);
    const int bn = args.bn, nstage = C::stages(bn);
    const uint32_t stage_bytes = (uint32_t)C::stage_bytes(bn), b_bytes = (uint32_t)(bn / CTAS * BK * 2);
    const uint32_t rank = CTAS == 2 ? cluster_ctarank() : 0u;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // tiles of CTAS pixel tiles (a pair's CTA takes the one of its rank) by bn models, taken by CTA (pair)
    const int n_ptiles = (args.n_ptiles + CTAS - 1) / CTAS;
    const int n_tiles = n_ptiles * args.n_mtiles, tile0 = blockIdx.x / CTAS, tile_step = gridDim.x / CTAS;
    const int nkb = args.nkb_young + args.nkb_old;
    const int nkb_ion = args.nkb_ion_young + args.nkb_ion_old;
    // K blocks of pixel tile pt: the escaping-light blocks only where the tile reaches an ionizing pixel
    auto tile_nkb = [&](int pt) { return (nkb_ion > 0 && pt * CTAS * OUT_ROWS - HALO < args.ion_pix) ? nkb + nkb_ion : nkb; };
    int *status = args.status;

    if (threadIdx.x == 0) {
        for (int s = 0; s < nstage; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(&tfull[b], 1); mbar_init(&tempty[b], CTAS * EPI_WARPS); }
        mbar_init(mma_done, 1);
        fence_mbar_init();
    }
    if (warp == 1) {
        if constexpr (CTAS == 2) { tmem_alloc_pair(tmem_slot, C::TMEM_COLS); tmem_relinquish_pair(); }
        else { tmem_alloc(tmem_slot, C::TMEM_COLS); tmem_relinquish(); }
    }
    if (warp == 0 && lane == 0) {
        tma_prefetch_desc(&tm_a_hi); tma_prefetch_desc(&tm_a_lo);
        tma_prefetch_desc(&tm_b_hi); tma_prefetch_desc(&tm_b_lo);
    }
    tc_fence_before();
    __syncthreads();
    if constexpr (CTAS == 2) cluster_sync();      // (the barriers of both CTAs are ready)
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        if (lane == 0) {
            int s = 0; uint32_t ph = 0;
            int last_fill[MAX_STAGES];          // parity of the last fill issued into each stage, -1: none
#pragma unroll
            for (int i = 0; i < MAX_STAGES; ++i) last_fill[i] = -1;
            bool ok = true;
            for (int tile = tile0; tile < n_tiles && ok; tile += tile_step) {
                const int mt = tile / n_ptiles, pt = tile % n_ptiles;
                const int p0 = (pt * CTAS + (int)rank) * OUT_ROWS - HALO, m0 = mt * bn + (int)rank * (bn / CTAS);
                const int kbn = tile_nkb(pt);
                for (int kb = 0; kb < kbn; ++kb) {
                    if (!mbar_wait(&empty[s], ph ^ 1u, status, ERR_TIMEOUT_PRODUCER)) { ok = false; break; }
                    uint8_t *st = stage_base + s * stage_bytes;
                    if constexpr (CTAS == 2) {
                        // both CTAs' copies complete on CTA 0's barrier, whose phase its producer arms for all of them
                        const uint32_t bar = cluster_addr(&full[s], 0);
                        if (rank == 0) mbar_arrive_expect_tx(&full[s], 2 * stage_bytes);
                        tma_load_2d_pair(st, &tm_a_hi, kb * BK, p0, bar);
                        tma_load_2d_pair(st + C::A_BYTES, &tm_a_lo, kb * BK, p0, bar);
                        tma_load_2d_pair(st + 2 * C::A_BYTES, &tm_b_hi, kb * BK, m0, bar);
                        tma_load_2d_pair(st + 2 * C::A_BYTES + b_bytes, &tm_b_lo, kb * BK, m0, bar);
                    } else {
                        mbar_arrive_expect_tx(&full[s], stage_bytes);
                        tma_load_2d(st, &tm_a_hi, kb * BK, p0, &full[s]);
                        tma_load_2d(st + C::A_BYTES, &tm_a_lo, kb * BK, p0, &full[s]);
                        tma_load_2d(st + 2 * C::A_BYTES, &tm_b_hi, kb * BK, m0, &full[s]);
                        tma_load_2d(st + 2 * C::A_BYTES + b_bytes, &tm_b_lo, kb * BK, m0, &full[s]);
                    }
#pragma unroll
                    for (int i = 0; i < MAX_STAGES; ++i)
                        if (i == s) last_fill[i] = (int)ph;
                    if (++s == nstage) { s = 0; ph ^= 1u; }
                }
            }
            // Drain: every copy this thread issued must have landed before the CTA may exit (CTA 0 waits for a pair's, and
            // CTA 1 for CTA 0 at the cluster barrier below).
#pragma unroll
            for (int i = 0; i < MAX_STAGES; ++i)
                if (last_fill[i] >= 0 && rank == 0) mbar_wait(&full[i], (uint32_t)last_fill[i], status, ERR_TIMEOUT_PRODUCER, false);
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer (CTA 0 of a pair)
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
            const uint32_t idesc = idesc_bf16_f32(CTAS * BM, bn);
            bool ok = true;
            for (int tile = tile0; tile < n_tiles && ok; tile += tile_step) {
                if (!mbar_wait(&tempty[acc], aph ^ 1u, status, ERR_TIMEOUT_MMA)) { ok = false; break; }
                tc_fence_after();
                const uint32_t d_base = tmem_base + acc * C::ACC_COLS;
                const int kbn = tile_nkb(tile % n_ptiles);
                for (int kb = 0; kb < kbn; ++kb) {
                    if (!mbar_wait(&full[s], ph, status, ERR_TIMEOUT_MMA)) { ok = false; break; }
                    tc_fence_after();
                    // the accumulator of block kb: young / old blocks, then the escaping light's young / old blocks
                    // (which always add to sums their own range has begun: a young ion block exists only with young
                    // ages, an old one only with old ages)
                    const bool ion_old = kb >= nkb + args.nkb_ion_young;
                    const int which = (NACC == 2 && ((kb >= args.nkb_young && kb < nkb) || ion_old)) ? 1 : 0;
                    const uint32_t d = d_base + which * C::BN;
                    const int kfirst = kb >= nkb ? -1 : (which == 0) ? 0 : args.nkb_young;
                    const uint32_t sa = smem_u32(stage_base + s * stage_bytes);
                    const uint32_t a_hi = sa, a_lo = sa + C::A_BYTES;
                    const uint32_t b_hi = sa + 2 * C::A_BYTES, b_lo = b_hi + b_bytes;
                    // (the last block of a range holds only its last columns' K steps)
                    const int r = kb < args.nkb_young ? 0 : kb < nkb ? 1 : kb < nkb + args.nkb_ion_young ? 2 : 3;
                    const int rend = r == 0 ? args.nkb_young : r == 1 ? nkb : r == 2 ? nkb + args.nkb_ion_young : nkb + nkb_ion;
                    const int ksteps = kb + 1 == rend ? (int)((args.ktail >> (8 * r)) & 0xffu) : BK / 16;
                    auto step = [&](int k) {
                        const uint32_t off = k * 32;
                        const uint32_t accum = (kb > kfirst || k > 0) ? 1u : 0u;
                        mma(d, sw128_desc(a_hi + off), sw128_desc(b_hi + off), idesc, accum);
                        mma(d, sw128_desc(a_hi + off), sw128_desc(b_lo + off), idesc, 1u);
                        mma(d, sw128_desc(a_lo + off), sw128_desc(b_hi + off), idesc, 1u);
                    };
                    if (ksteps == BK / 16) {
#pragma unroll
                        for (int k = 0; k < BK / 16; ++k) step(k);
                    } else {
                        for (int k = 0; k < ksteps; ++k) step(k);
                    }
                    commit(&empty[s]);          // frees the stage once these MMAs have read it
                    if (++s == nstage) { s = 0; ph ^= 1u; }
                }
                if (!ok) break;
                commit(&tfull[acc]);            // accumulator ready for the epilogue
                if (++acc == 2) { acc = 0; aph ^= 1u; }
            }
            // Every MMA issued by this thread must be complete before the TMEM is released.
            commit(mma_done);
            mbar_wait(mma_done, 0, status, ERR_TIMEOUT_MMA, false);
        }
    } else {
        // ------------------------------------------------------------------ epilogue (warps 2 ..)
        const int ew = warp - 2;
        const int g = ew >> 2;                  // group: its part of the columns
        const int wg = ew & 3;                  // warp within the group
        const int q = warp & 3;                 // TMEM lane quarter this warp may access
        const int r = q * 32 + lane;            // pixel row of the tile (phase 1)
        const int et = wg * 32 + lane;          // 0..127 within the group
        const int bar_id = 1 + g;
        float *stageT = epi_base + g * (C::STAGE_T_FLOATS + C::PAR_FLOATS);
        float *parbuf = stageT + C::STAGE_T_FLOATS;
        const bool vec_store = (args.ld_spec & 1) == 0;
        const int group_cols = bn / EPI_GROUPS;          // models per epilogue group
        int acc = 0; uint32_t aph = 0;
        int pb = 0;
        for (int tile = tile0; tile < n_tiles; tile += tile_step) {
            const int mt = tile / n_ptiles, pt = tile % n_ptiles;
            const int p0 = (pt * CTAS + (int)rank) * OUT_ROWS - HALO, m0 = mt * bn;
            const int p = p0 + r;
            const bool inpix = (p >= 0 && p < args.nspec);
            // per-pixel data of this thread's row (phase 1)
            float ltab2 = 0.f, curve_u = 1.f, ia[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            float4 tcv = make_float4(0.f, 0.f, 0.f, 0.f);   // the curve tables T0..T3 (models' own tabulated curves)
            if (inpix) {
                const float4 *px = reinterpret_cast<const float4 *>(args.pix + (size_t)p * PIX_FLOATS);
                const float4 v0 = px[0], v1 = px[1];
                ltab2 = v0.x; curve_u = v0.y; ia[0] = v0.z; ia[1] = v0.w;
                ia[2] = v1.x; ia[3] = v1.y; ia[4] = v1.z; ia[5] = v1.w;
                if (args.tab_curve) tcv = px[PIX_T / 4];
            }
            const bool igm_pix = inpix && p < args.jtop;

            mbar_wait(&tfull[acc], aph, status, ERR_TIMEOUT_EPILOGUE);
            // the group agrees on whether to go on (a thread that gave up set the status first)
            named_bar_sync(bar_id, 128);
            if (*(volatile int *)status != 0) break;
            tc_fence_after();
            const uint32_t t_row = tmem_base + ((uint32_t)(q * 32) << 16) + acc * C::ACC_COLS;

            for (int c = 0; c < group_cols / CHUNK; ++c) {
                const int col0 = g * group_cols + c * CHUNK;      // first model of the chunk in the tile
                // model parameters of the chunk (double-buffered)
                float *par = parbuf + pb * CHUNK * MODEL_PAR_FLOATS;
                for (int i = et; i < CHUNK * MODEL_PAR_FLOATS / 4; i += 128) {
                    const int mm = m0 + col0 + (i * 4) / MODEL_PAR_FLOATS;
                    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (mm < args.n_models)
                        v = reinterpret_cast<const float4 *>(args.mpar + (size_t)mm * MODEL_PAR_FLOATS)[(i * 4) % MODEL_PAR_FLOATS / 4];
                    reinterpret_cast<float4 *>(par)[i] = v;
                }
                float y[CHUNK];
                tmem_ld8(t_row + col0, y);
                float o[CHUNK];
                if constexpr (NACC == 2) {
                    tmem_ld8(t_row + C::BN + col0, o);
                    if (args.nkb_young == 0) {
#pragma unroll
                        for (int j = 0; j < CHUNK; ++j) y[j] = 0.f;
                    }
                    if (args.nkb_old == 0) {
#pragma unroll
                        for (int j = 0; j < CHUNK; ++j) o[j] = 0.f;
                    }
                }
                if (c == group_cols / CHUNK - 1) {
                    // all of this group's accumulator columns have been read: hand them back to the MMA warp
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        if constexpr (CTAS == 2) mbar_arrive_cluster(cluster_addr(&tempty[acc], 0));
                        else mbar_arrive(&tempty[acc]);
                    }
                }
                named_bar_sync(bar_id, 128);
                // ---- phase 1: thread = pixel row r, the chunk's models
#pragma unroll
                for (int j = 0; j < CHUNK; ++j) {
                    const float *mp = par + j * MODEL_PAR_FLOATS;
                    const float4 d0 = *reinterpret_cast<const float4 *>(mp);          // kd2, 1-fnd, fnd, index
                    const float curve = pix_curve(args.uniform_index, args.tab_curve, curve_u, ltab2, tcv,
                                                  make_float4(mp[MP_CS1], mp[MP_CS1 + 1], mp[MP_CS1 + 2], 0.f), d0.w);
                    float ss;
                    if constexpr (NACC == 2) {
                        if (args.young && inpix && r >= HALO && r < BM - HALO && m0 + col0 + j < args.n_models) {
                            // the parts: young and old age sums before dust (compute_csp_batch_parts)
                            args.young[(size_t)(m0 + col0 + j) * args.ld_spec + p] = y[j];
                            args.old[(size_t)(m0 + col0 + j) * args.ld_spec + p] = o[j];
                        }
                        const float4 d1 = *reinterpret_cast<const float4 *>(mp + 4);  // kd1, d1 index, 1-fo, fo
                        const float kd3 = mp[MP_KD3];
                        const float tb = (d1.x != 0.f) ? ex2(d1.x * ex2(d1.y * ltab2)) : 1.f;
                        const float to = (kd3 != 0.f) ? ex2(kd3 * curve) : 1.f;
                        ss = (y[j] * tb * d1.z + y[j] * d1.w) + o[j] * to;
                    } else {
                        ss = y[j];
                    }
                    float tot = ss * fmaf(ex2(d0.x * curve), d0.y, d0.z);
                    if (igm_pix) {
                        const float4 g0 = *reinterpret_cast<const float4 *>(mp + MP_IGM_ON);   // on, jmax, kcap, kd3
                        if (g0.x != 0.f) {
                            float arg;
                            if (p < __float_as_int(g0.y)) {
                                arg = g0.z;
                            } else {
                                const float4 g1 = *reinterpret_cast<const float4 *>(mp + MP_IGM_KB);   // kb0..kb3
                                const float2 g2 = *reinterpret_cast<const float2 *>(mp + MP_IGM_KB + 4);  // kb4, kb5
                                arg = ia[0] * g1.x + ia[1] * g1.y + ia[2] * g1.z + ia[3] * g1.w + ia[4] * g2.x +
                                      ia[5] * g2.y;
                            }
                            tot *= ex2(arg);
                        }
                    }
                    stageT[j * TROW + r] = tot;
                }
                named_bar_sync(bar_id, 128);
                // ---- phase 2: warp wg takes its quarter of the chunk's models; lane l the output rows 4 + 4l .. 7 + 4l (no
                // spectra when a per-model epilogue forms them from the young and old sums)
                if (args.spec != nullptr && lane < OUT_ROWS / 4) {
                    const int row0 = HALO + 4 * lane;
                    const int pq = p0 + row0;                      // first output pixel of this lane
#pragma unroll 1
                    for (int jj = 0; jj < CHUNK / 4; ++jj) {
                        const int j = wg * (CHUNK / 4) + jj;
                        const int mm = m0 + col0 + j;
                        if (mm >= args.n_models || pq >= args.nspec) continue;
                        const float *mp = par + j * MODEL_PAR_FLOATS;
                        const float *row = stageT + j * TROW + row0 - HALO;   // 16-byte aligned
                        const float4 w0 = *reinterpret_cast<const float4 *>(row);
                        const float4 w1 = *reinterpret_cast<const float4 *>(row + 4);
                        const float4 w2 = *reinterpret_cast<const float4 *>(row + 8);
                        const float win[12] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w, w2.x, w2.y, w2.z, w2.w};
                        float out[4] = {win[4], win[5], win[6], win[7]};
                        const int R = __float_as_int(mp[MP_SMOOTH_R]);
                        if (R >= 0 && pq + 3 >= args.sm_lo && pq <= args.sm_hi) {
                            const float4 ta = *reinterpret_cast<const float4 *>(mp + MP_TAPS);
                            const float4 tb = *reinterpret_cast<const float4 *>(mp + MP_TAPS + 4);
                            const float tc = mp[MP_TAPS + 8];
                            const float tap[9] = {ta.x, ta.y, ta.z, ta.w, tb.x, tb.y, tb.z, tb.w, tc};
#pragma unroll
                            for (int u = 0; u < 4; ++u) {
                                const int pu = pq + u;
                                if (pu < args.sm_lo || pu > args.sm_hi) continue;
                                float s = 0.f;
#pragma unroll
                                for (int d = 0; d < 9; ++d) s = fmaf(tap[d], win[u + d], s);
                                out[u] = s;
                            }
                        }
                        float *dst = args.spec + (size_t)mm * args.ld_spec + pq;
                        if (vec_store && pq + 3 < args.nspec) {
                            reinterpret_cast<float2 *>(dst)[0] = make_float2(out[0], out[1]);
                            reinterpret_cast<float2 *>(dst)[1] = make_float2(out[2], out[3]);
                        } else {
#pragma unroll
                            for (int u = 0; u < 4; ++u)
                                if (pq + u < args.nspec) dst[u] = out[u];
                        }
                    }
                }
                pb ^= 1;
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
        if constexpr (CTAS == 2) tmem_dealloc_pair(tmem_base, C::TMEM_COLS);
        else tmem_dealloc(tmem_base, C::TMEM_COLS);
    }
}

// ---------------------------------------------------------------------------------------------- host side
template <int NACC, int CTAS>
static cudaError_t launch_contract(const ContractPlan &pl, const ContractArgs &a, cudaStream_t st) {
    using C = ContractCfg<NACC, CTAS>;
    auto kern = csp_contract_kernel<NACC, CTAS>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES);
    if (e != cudaSuccess) return e;
    const int n_tiles = (a.n_ptiles + CTAS - 1) / CTAS * a.n_mtiles;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(CTAS * std::min(n_tiles, pl.num_sms / CTAS));
    cfg.blockDim = dim3(C::NTHREADS);
    cfg.dynamicSmemBytes = C::SMEM_BYTES;
    cfg.stream = st;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = CTAS;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = CTAS > 1 ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, pl.tm_a_hi, pl.tm_a_lo, pl.tm_b_hi, pl.tm_b_lo, a);
}

// The tile by its measured cost: a first wave of tiles takes what the K loop's latency and an epilogue that nothing
// overlaps add up to (first: us at width 0, us per model of width), a further wave what the tables give (us at bn = 32,
// 64 ..). CTA pairs (one accumulator): an MMA of 256 pixels by bn models over two SMs reads a CTA's share of both
// operands from shared memory once, 8 KB at bn = 256 against 12 KB by one CTA, whose 12 KB at about 64 bytes a cycle
// take 1.5 times the multiplications' 128 cycles; below 160 models the A operand's share is the bound either way. Two
// accumulators (at most 128 models a tile, so that they fit TMEM twice) run on single CTAs: pairs measured 450 us at 9001
// models against 429. The widest tile is not always the cheapest: a batch may fill its last wave badly, or hold fewer
// models than a tile.
// Measured, one CTA per 256 (128) models and eight epilogue warps -> with the rule and sixteen: 38.7 -> 20 us at one
// model, 80 -> 51 at 1000, 317 -> 239 at 9001, 1951 -> 1591 at 65536 (1.90 PFLOP/s of the
// pixels' products, 2.0 with the halo rows'). The costs are those of 1296 columns of K. Every tile gives the same
// bits: an output's products are summed in the same order.
ContractTile contract_tile(int nacc, int n_models, int n_ptiles, int num_sms) {
    struct Shape { int nacc, ctas, bn0; double first0, first1; double further[8]; };
    static const Shape shapes[3] = {
        {1, 2, 160, 14.0, 0.112, {0, 0, 0, 0, 14.0, 15.0, 16.6, 18.7}},
        {1, 1, 32, 13.5, 0.117, {12.4, 12.7, 13.1, 13.5, 16.3, 17.7, 19.5, 21.4}},
        {2, 1, 32, 20.7, 0.125, {14.5, 15.0, 16.4, 17.0, 0, 0, 0, 0}},
    };
    ContractTile best = {0, 1};
    double best_t = 1e300;
    for (const Shape &s : shapes) {
        if (s.nacc != nacc || num_sms < s.ctas) continue;
        const int most = nacc == 1 ? ContractCfg<1, 1>::BN : ContractCfg<2, 1>::BN;
        for (int bn = most; bn >= s.bn0; bn -= 32) {
            const long long tiles = (long long)((n_models + bn - 1) / bn) * ((n_ptiles + s.ctas - 1) / s.ctas);
            const long long waves = (tiles + num_sms / s.ctas - 1) / (num_sms / s.ctas);
            const double t = s.first0 + s.first1 * bn + (double)(waves - 1) * s.further[bn / 32 - 1];
            if (t < best_t) { best_t = t; best = {bn, s.ctas}; }
        }
    }
    return best;
}
int contract_out_rows() { return OUT_ROWS; }
int contract_halo() { return HALO; }
int contract_bk() { return BK; }
int contract_bm() { return BM; }

cudaError_t run_contract(int nacc, const ContractPlan &pl, const ContractArgs &a, cudaStream_t st) {
    if (nacc == 2) return a.ctas == 1 ? launch_contract<2, 1>(pl, a, st) : cudaErrorInvalidValue;
    return a.ctas == 2 ? launch_contract<1, 2>(pl, a, st) : launch_contract<1, 1>(pl, a, st);
}

}  // namespace sps
