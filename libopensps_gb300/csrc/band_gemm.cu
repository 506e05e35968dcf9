// Band fluxes and AB magnitudes as a tensor-core GEMM: fband(m, b) = sum_j Fobs(m, j) C(j, b).
//
// compute_magnitudes_columns (OpenSPS src/spectra/opensps_batch_photometry.f90:53-180): each model's rest-frame
// spectrum resampled to the observed frame at its redshift, divided by lambda (observed_frame_z :819-903), then the
// trapezoid filter integrals regrouped by pixel, C(j, b) = band(j, b) (wtl(j - 1) + wtl(j)) (the split-K product
// :1002-1044, prepare_batch_grid :375-392), then magnitudes_from_fluxes :185-232 (AB, distance term, NaN for bands
// not computed). The division by lambda is folded into the band matrix (C(j, b) / lambda(j), formed in FP64 on the
// host), so the A operand is the resampled spectrum itself.
//
// Per CTA: 128 models (MMA M). K = the pixels that any band reaches, 64 per stage. The A operand (observed frame
// of 128 models x 64 pixels) is built by warps 0..15 in shared memory from the spectra, in the 128-byte swizzled
// K-major layout, split into bf16 hi and lo; the B operand (band matrix, hi and lo, bands x pixels) comes by TMA.
// fband = A_hi B_hi + A_hi B_lo + A_lo B_hi in f32 in tensor memory; all the warps form the magnitudes.
// Warp roles: warps 0..15 build the A operand (8 model rows each: two CTAs of 17 warps per SM at 56 registers, against
// 9 warps of 16 rows at 92), warp 16 issues the band matrix's TMA and the MMAs.
// Two stages with mbarriers: a builder warp signals its rows of stage s on full_a[s] and goes on to the next stage as
// soon as the MMAs that read that buffer have completed (empty[s], a tcgen05 commit), so that the warps do not wait
// for one another between stages. The band matrix comes up to three blocks ahead in slots of its own.
// The pixel blocks split over the CTAs of a cluster (band_gemm_ksplit); each leaves its partial fluxes in its shared
// memory, and the CTAs read one another's to form the magnitudes, a share of the rows each, in split order: no scratch
// in memory and no second kernel.
// Bound by the builders' instructions and their latencies (a warp's 8 rows of a block take 300; without any load three
// quarters of the time are left). 20001 models: 111 us, 144 unsplit, when 5 SMs had two of the 157 tiles; 9001: 49 us
// against 57 and a second kernel; 1000: 18 us against 15 and 5; 65536: 277, as before.
#include <cuda_runtime.h>
#include <algorithm>
#include <cuda_bf16.h>
#include <cfloat>
#include <cmath>
#include <cstdint>
#include "sm103_ptx.cuh"
#include "csp_kernels.h"

namespace sps {

constexpr int BG_M = 128;
constexpr int BG_K = 64;
constexpr int BG_BUILD_WARPS = 16;
constexpr int BG_BUILD_THREADS = BG_BUILD_WARPS * 32;
constexpr int BG_MMA_WARP = BG_BUILD_WARPS;             // TMA of the band matrix and the MMAs
constexpr int BG_THREADS = BG_BUILD_THREADS + 32;
constexpr int BG_A_BYTES = BG_M * BG_K * 2;   // 16 KB
constexpr int BG_AHEAD = 1;                             // row pairs whose loads are in flight while one is converted
constexpr int BG_MAX_SPLIT = 16, BG_MIN_BLOCKS = 4, BG_SETUP = 3, BG_FEW_TILES = 32;   // (band_gemm_ksplit)

struct BandGemmSmem {
    static int b_bytes(int npad) { return npad * BG_K * 2; }
    static int total(int npad, int slots) { return 4 * BG_A_BYTES + slots * 2 * b_bytes(npad) + 256 + 1024; }
    static constexpr int SM_BYTES = 232448, OTHER = 1024 + 6144;   // (OTHER per CTA: the system's, the static arrays)
    // Band-matrix slots: three, unless a second CTA fits the SM with two only, or not even one CTA with three.
    static int slots(int npad) {
        if (2 * (total(npad, 3) + OTHER) <= SM_BYTES) return 3;
        if (2 * (total(npad, 2) + OTHER) <= SM_BYTES) return 2;
        return total(npad, 3) + OTHER <= SM_BYTES ? 3 : 2;
    }
    static bool two_ctas(int npad) { return 2 * (total(npad, slots(npad)) + OTHER) <= SM_BYTES; }   // (per SM)
};

// 2^x by the SFU
__device__ __forceinline__ float bg_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// AB magnitude of an FP32 band flux (NaN when not positive): -2.5 log10 f in FP32 (the flux carries FP32's precision
// already; an FP64 logarithm per band was most of the epilogue's time on GB300's narrow FP64 pipe), then the zero
// point and the model's distance term in FP64.
__device__ __forceinline__ double band_mag(float f, double zp, double dist) {
    if (!(f > 0.f)) return __longlong_as_double(0x7ff8000000000000LL);
    return (double)(-2.5f * log10f(f)) - zp + dist;
}

__global__ void __launch_bounds__(BG_THREADS, 2)
band_gemm_kernel(const __grid_constant__ CUtensorMap tm_c_hi, const __grid_constant__ CUtensorMap tm_c_lo,
                 BandGemmArgs a) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int npad = a.npad;
    const int b_bytes = npad * BG_K * 2;
    constexpr int stage_bytes = 2 * BG_A_BYTES;      // two stages of the A operand (hi, lo), then the B slots (hi, lo)
    uint8_t *bslots = smem + 2 * stage_bytes;
    const int nb = a.slots;
    uint64_t *bars = reinterpret_cast<uint64_t *>(bslots + nb * 2 * b_bytes);
    uint64_t *full_a = bars;         // [2] the builder warps' rows of a stage (16 arrivals)
    uint64_t *empty = bars + 2;      // [2] the MMAs that read a stage have completed
    uint64_t *full_b = bars + 4;     // [3] the band matrix's TMA of a slot
    uint64_t *bar_done = bars + 7;   // every MMA has completed
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 8);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.x * BG_M;
    // this CTA's pixel blocks: split blockIdx.y of gridDim.y
    const int kb0 = (int)((long long)blockIdx.y * a.nkb / gridDim.y), kb1 = (int)((long long)(blockIdx.y + 1) * a.nkb / gridDim.y);
    const int nst = kb1 - kb0;
    const bool split = gridDim.y > 1;
    int *status = a.status;
    const uint32_t tcols = npad <= 32 ? 32 : (npad <= 64 ? 64 : (npad <= 128 ? 128 : 256));
    __shared__ float4 zsm[BG_M];     // the observed-frame shift of the CTA's models (w = 2: no model in this row)
    // per row, for the interior case: observed pixel j reads rest pixels j - d and j - d + 1; a lane's five, of its
    // four observed pixels, lie in the two aligned float4 that begin at rest pixel p = j - d - mis (mis: the row's
    // place in a float4, the same for every lane, whose first pixels differ by multiples of four). x = d + mis,
    // y = the largest p whose eight rest pixels and four observed ones lie inside the grid (interior: p <= y, as
    // unsigned), z = 4 x the row's offset from the CTA's first model's + mis, w = t; a row without a model has none
    __shared__ int4 rsh[BG_M];

    if (tid == 0) {
        for (int s = 0; s < 2; ++s) { mbar_init(&full_a[s], BG_BUILD_WARPS); mbar_init(&empty[s], 1); }
        for (int s = 0; s < 3; ++s) mbar_init(&full_b[s], 1);
        mbar_init(bar_done, 1);
        fence_mbar_init();
        tma_prefetch_desc(&tm_c_hi);
        tma_prefetch_desc(&tm_c_lo);
    }
    if (warp == 0) { tmem_alloc(tmem_slot, tcols); tmem_relinquish(); }
    for (int i = tid; i < BG_M; i += BG_THREADS) {
        const float4 zs = (m0 + i < a.n_models) ? a.zinfo[m0 + i] : make_float4(0.f, 0.f, 0.f, 2.f);
        zsm[i] = zs;
        // the interior interpolation's first rest pixel: n0 + 1 below the observed one unless the shift is whole
        const int kind = zs.w == 1.f ? 1 : (zs.w == 0.f ? 0 : 2);
        const int d = kind == 1 ? __float_as_int(zs.x) + (zs.y > 0.f ? 1 : 0) : 0;
        const float *row = a.spec + (size_t)(m0 + i) * a.ld_spec;
        const int mis = (int)((((long long)(reinterpret_cast<uintptr_t>(row) >> 2)) + a.j0 - d) & 3);
        const int last = min(a.nspec - 8, a.nspec - 4 - (d + mis));
        rsh[i] = kind == 2 || last < 0 ? make_int4(1 << 30, 0, 0, 0)
                                       : make_int4(d + mis, last, 4 * i * a.ld_spec + mis, __float_as_int(kind == 1 ? zs.y : 0.f));
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == BG_MMA_WARP) {
        // ---------------------------------------------------------------- band matrix TMA and MMAs (one thread)
        if (lane == 0) {
            const uint32_t idesc = idesc_bf16_f32(BG_M, npad);
            // block li's band matrix in slot li mod nb, nb blocks ahead of its MMAs (issued when the block's A operand
            // was asked for, its latency was a third of the time of each block)
            auto fetch = [&](int li, int slot) {
                uint8_t *bs = bslots + slot * 2 * b_bytes;
                mbar_arrive_expect_tx(&full_b[slot], 2 * b_bytes);
                tma_load_2d(bs, &tm_c_hi, (kb0 + li) * BG_K, 0, &full_b[slot]);
                tma_load_2d(bs + b_bytes, &tm_c_lo, (kb0 + li) * BG_K, 0, &full_b[slot]);
            };
            int fetched = 0;                              // blocks whose copies were issued
            for (; fetched < min(nb, nst); ++fetched) fetch(fetched, fetched);
            bool ok = true;
            int slot = 0, bpar = 0, done = 0;             // done: blocks whose copies have landed
            for (int li = 0; li < nst; ++li) {
                const int s = li & 1;
                if (!mbar_wait(&full_a[s], (li >> 1) & 1, status, ERR_TIMEOUT_BAND) ||
                    !mbar_wait(&full_b[slot], bpar, status, ERR_TIMEOUT_BAND)) { ok = false; break; }
                ++done;
                tc_fence_after();
                const uint32_t ahi = smem_u32(smem + s * stage_bytes), alo = ahi + BG_A_BYTES;
                const uint32_t bhi = smem_u32(bslots + slot * 2 * b_bytes), blo = bhi + b_bytes;
#pragma unroll
                for (int k = 0; k < BG_K / 16; ++k) {
                    const uint32_t o = k * 32;
                    mma_bf16(tmem, sw128_desc(ahi + o), sw128_desc(bhi + o), idesc, (li > 0 || k > 0) ? 1u : 0u);
                    mma_bf16(tmem, sw128_desc(ahi + o), sw128_desc(blo + o), idesc, 1u);
                    mma_bf16(tmem, sw128_desc(alo + o), sw128_desc(bhi + o), idesc, 1u);
                }
                mma_commit(&empty[s]);
                // the slot of block li - 1 is free once its MMAs have completed: the block nb after it
                if (li >= 1 && fetched < nst) {
                    if (!mbar_wait(&empty[s ^ 1], ((li - 1) >> 1) & 1, status, ERR_TIMEOUT_BAND)) { ok = false; break; }
                    fetch(fetched, slot == 0 ? nb - 1 : slot - 1);
                    ++fetched;
                }
                if (++slot == nb) { slot = 0; bpar ^= 1; }
            }
            // every MMA issued completes on bar_done (the epilogue's wait, and the TMEM's release below), after the
            // copies still in flight have landed
            for (; done < fetched; ++done) {              // (none unless a wait gave up)
                mbar_wait(&full_b[done % nb], (uint32_t)(done / nb) & 1u, status, ERR_TIMEOUT_BAND, false);
            }
            mma_commit(bar_done);
            if (!ok) mbar_wait(bar_done, 0, status, ERR_TIMEOUT_BAND, false);
        }
    } else {
        // ---------------------------------------------------------------- A operand builders (warps 0..15)
        const float dl2 = a.dl2, inv_em1 = a.inv_em1;
        // each warp builds 8 model rows, two at a time: lane l takes row parity l / 16 and pixels 4 (l % 16) ..
        // 4 (l % 16) + 3 of the stage
        const int q = lane & 15, hr = lane >> 4;
        const int row0 = warp * 8 + hr;
        // an interior row pair's loads are two aligned float4 a lane (five scalar loads touched each line five times:
        // L1 at 75 % of its peak, now 27), and BG_AHEAD pairs are in flight while one is converted, across the stages
        // (split in two, none ahead: 85 us at 9001 models; one: 62; two or three: 64 to 66)
        float4 va[4], vb[4];
        const float *rows = a.spec + (size_t)m0 * a.ld_spec;
        auto interior = [&](int li, int i) {                 // (of a lane's pixels of block li in its row of pair i)
            const int2 rs = *reinterpret_cast<const int2 *>(&rsh[row0 + 2 * i]);
            return (unsigned)(a.j0 + (kb0 + li) * BG_K + 4 * q - rs.x) <= (unsigned)rs.y;
        };
        // (the zeros: without them the old values stay live through the condition, and spill)
        auto load = [&](int li, int i) {
            va[i] = vb[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (li < nst && interior(li, i)) {
                const int4 rs = rsh[row0 + 2 * i];
                const float4 *sp = reinterpret_cast<const float4 *>(rows + ((rs.z >> 2) + a.j0 + (kb0 + li) * BG_K + 4 * q - rs.x));
                va[i] = __ldg(sp);
                vb[i] = __ldg(sp + 1);
            }
        };
#pragma unroll
        for (int i = 0; i < BG_AHEAD; ++i) load(0, i);
        for (int li = 0; li < nst; ++li) {
            const int s = li & 1, kb = kb0 + li;
            uint8_t *st = smem + s * stage_bytes;
            const int j = a.j0 + kb * BG_K + 4 * q;          // first observed pixel of this lane
            // the stage's A buffer is free once the MMAs of stage li - 2 have completed
            if (li >= 2 && !mbar_wait(&empty[s], ((li - 2) >> 1) & 1, status, ERR_TIMEOUT_BAND)) break;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                load(li + (i + BG_AHEAD) / 4, (i + BG_AHEAD) % 4);
                const int r = row0 + 2 * i;
                float f[4];
                if (interior(li, i)) {
                    // v = s(c) + t (s(c + 1) - s(c)), t = 0 for whole shifts and the rest frame (v = s(c) exactly
                    // for finite spectra); NaN -> 0 and negatives -> 0 in one fmaxf
                    const int2 rs = *reinterpret_cast<const int2 *>(&rsh[r].z);
                    const float t = __int_as_float(rs.y);
                    const bool m1 = rs.x & 1, m2 = rs.x & 2;
                    const float w0 = m2 ? va[i].z : va[i].x, w1 = m2 ? va[i].w : va[i].y, w2 = m2 ? vb[i].x : va[i].z,
                                w3 = m2 ? vb[i].y : va[i].w, w4 = m2 ? vb[i].z : vb[i].x, w5 = m2 ? vb[i].w : vb[i].y;
                    const float sv[5] = {m1 ? w1 : w0, m1 ? w2 : w1, m1 ? w3 : w2, m1 ? w4 : w3, m1 ? w5 : w4};
#pragma unroll
                    for (int u = 0; u < 4; ++u) f[u] = fmaxf(fmaf(t, sv[u + 1] - sv[u], sv[u]), 0.f);
                } else {
                    // the general case: no model, pixels past the grid's end, or intervals outside the grid (they
                    // extrapolate from the first / last one, the reference's clamped find_interval: position
                    // t = (e^(x dlnl) - 1) / (e^dlnl - 1), x pixels from the interval start)
                    const float4 zs = zsm[r];
                    const float *sp = a.spec + (size_t)(m0 + r) * a.ld_spec;
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int ju = j + u;
                        float v = 0.f;
                        if (zs.w == 1.f) {
                            const int n0 = __float_as_int(zs.x);
                            const int il = ju - n0 - ((zs.y > 0.f) ? 1 : 0);
                            const int cc = min(max(il, 0), a.nspec - 2);
                            const float tt = (cc == il) ? zs.y : (bg_ex2(((float)(ju - cc) - zs.z) * dl2) - 1.f) * inv_em1;
                            const float x0 = __ldg(sp + cc), x1 = __ldg(sp + cc + 1);
                            v = fmaf(tt, x1 - x0, x0);
                        } else if (zs.w == 0.f && ju < a.nspec) {
                            v = __ldg(sp + ju);
                        }
                        f[u] = fmaxf(v, 0.f);
                    }
                }
                // bf16 hi and lo parts, four pixels = 8 bytes of the row's 128-byte swizzled line
                const __nv_bfloat162 h01 = __floats2bfloat162_rn(f[0], f[1]), h23 = __floats2bfloat162_rn(f[2], f[3]);
                const float2 g01 = __bfloat1622float2(h01), g23 = __bfloat1622float2(h23);
                const __nv_bfloat162 l01 = __floats2bfloat162_rn(f[0] - g01.x, f[1] - g01.y);
                const __nv_bfloat162 l23 = __floats2bfloat162_rn(f[2] - g23.x, f[3] - g23.y);
                const uint32_t off = r * 128 + ((((uint32_t)q >> 1) ^ (r & 7)) << 4) + ((q & 1) << 3);
                uint2 hv, lv;
                hv.x = *reinterpret_cast<const uint32_t *>(&h01); hv.y = *reinterpret_cast<const uint32_t *>(&h23);
                lv.x = *reinterpret_cast<const uint32_t *>(&l01); lv.y = *reinterpret_cast<const uint32_t *>(&l23);
                *reinterpret_cast<uint2 *>(st + off) = hv;
                *reinterpret_cast<uint2 *>(st + BG_A_BYTES + off) = lv;
            }
            // this warp's rows of the stage, visible to the tensor core's (async) reads
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(&full_a[s]);
        }
        mbar_wait(bar_done, 0, status, ERR_TIMEOUT_BAND, false);
        tc_fence_after();

        // the CTA's fluxes from TMEM into shared memory, over the stages (no copy is in flight into them: bar_done came
        // after the last): warps w and w + 4 read lane quarter w % 4 (one model per thread), columns 32 (w / 4) + 64 i
        if (warp < 8 && *(volatile int *)status == 0) {
            const int r = (warp & 3) * 32 + lane;
            const uint32_t trow = tmem + ((uint32_t)((warp & 3) * 32) << 16);
            float *dst = reinterpret_cast<float *>(smem) + r * (npad + 1);   // (odd pitch: a column without conflicts)
            for (int c0 = (warp >> 2) * 32; c0 < npad; c0 += 64) {
                float v[32];
                tmem_ld32(trow + c0, v);
#pragma unroll
                for (int i = 0; i < 32; ++i)
                    if (c0 + i < npad) dst[c0 + i] = v[i];
            }
        }
    }
    // the magnitudes: the cluster's CTAs share the tile's rows, each summing its rows' partial fluxes in split order
    __syncwarp();
    if (split) cluster_sync();
    else __syncthreads();
    if (*(volatile int *)status == 0) {
        const int ks = (int)gridDim.y, r0 = BG_M * (int)blockIdx.y / ks, r1 = BG_M * ((int)blockIdx.y + 1) / ks;
        const int tot = (min(r1, a.n_models - m0) - r0) * a.nbands;
        for (int i = tid; i < tot; i += BG_THREADS) {
            const int r = r0 + i / a.nbands, b = i % a.nbands, m = m0 + r;
            const float *src = reinterpret_cast<const float *>(smem) + r * (npad + 1) + b;
            float v = 0.f;
            if (split)
                for (int k = 0; k < ks; ++k) v += ld_cluster_f32(cluster_addr(src, (uint32_t)k));
            else
                v = *src;
            if (a.fband) a.fband[(size_t)m * a.nbands + b] = (double)v;
            if (a.mags) {
                double mg = __longlong_as_double(0x7ff8000000000000LL);
                if (a.do_band == nullptr || a.do_band[b] != 0) mg = band_mag(v, a.zp, a.dist[m]);
                a.mags[(size_t)m * a.nbands + b] = mg;
            }
        }
    }
    __syncwarp();
    if (split) cluster_sync();   // (no CTA leaves while another reads its fluxes)
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, tcols);
    }
}

int band_gemm_npad(int nbands) { return (nbands + 15) / 16 * 16 < 32 ? 32 : (nbands + 15) / 16 * 16; }

// Splits of the pixel blocks over a cluster's CTAs. Few tiles (at most 4096 models): up to two CTAs per SM. More: the
// split with the least time on the busiest SM, where every CTA takes BG_SETUP blocks' time besides its blocks' (its setup,
// the pipeline's fill, its magnitudes).
// Up to 80 bands an SM's CTAs run two at a time: a pair takes 3.1 us a pixel block, a CTA alone 2.3 (a builder warp's own
// latencies bound it, and two CTAs hide part of them). Measured, us at splits of 1 .. 6: 113, 64, 60, 49, 68, 67 at 9001
// models; 145, 132, 111, 114, 110, 116 at 20001; 120 and 90 at 1 and 2 at 16384.
// Above 80 bands one CTA fills an SM: 1, 2 or 4 CTAs by the waves of clusters (of four, one in twenty's places is lost to
// the GPCs' sizes; other sizes lose more). 100 bands, us at splits of 1 .. 8: 124, 76, 61, 52, 72, 66, 84, 76 at 4500 models;
// 146, 89, 115, 97, 117, 133, 151, 136 at 9001; 150, 158, 166, 174 .. at 16384; 278, 295, 311, 294 .. at 30000; 543, 517,
// 612, 613 .. at 65536 (priced as pairs of CTAs: 77, 97, 159, 279, 518).
static int band_gemm_ksplit(int n_models, int nkb, int npad, int num_sms) {
    const int tiles = (n_models + BG_M - 1) / BG_M;
    // (clusters beyond the portable eight only where two of their CTAs share an SM)
    const bool two = BandGemmSmem::two_ctas(npad);
    const int most = std::max(1, std::min(nkb / BG_MIN_BLOCKS, two ? BG_MAX_SPLIT : 8));
    if (tiles <= BG_FEW_TILES) return std::min((2 * num_sms + tiles - 1) / tiles, most);
    int best = 1;
    long long best_cost = 0;
    for (int ks = 1; ks <= std::min(most, two ? 8 : 4); ks = two ? ks + 1 : 2 * ks) {
        const long long blocks = (nkb + ks - 1) / ks + BG_SETUP;
        long long cost;
        if (two) {
            const long long ctas = ((long long)tiles * ks + num_sms - 1) / num_sms;     // of the busiest SM
            cost = (ctas / 2 * 31 + ctas % 2 * 23) * blocks;
        } else {
            const int at_once = std::max(1, (ks == 4 ? num_sms * 19 / 20 : num_sms) / ks);   // clusters
            cost = (tiles + at_once - 1) / at_once * blocks;
        }
        if (ks == 1 || cost < best_cost) { best = ks; best_cost = cost; }
    }
    return best;
}

// Loads the band GEMM's module on the current device (CUDA loads modules lazily, on first use), so that a later
// launch loads nothing.
cudaError_t band_gemm_load() {
    cudaFuncAttributes fa;
    cudaError_t e = cudaFuncGetAttributes(&fa, band_gemm_kernel);
    return e;
}

cudaError_t run_band_gemm(const BandGemmArgs &a_in, const CUtensorMap &tm_hi, const CUtensorMap &tm_lo,
                          cudaStream_t st) {
    if (a_in.n_models <= 0 || a_in.nkb <= 0) return cudaSuccess;
    BandGemmArgs a = a_in;
    a.slots = BandGemmSmem::slots(a.npad);
    a.dl2 = (float)(a.dlnl * 1.4426950408889634);
    a.inv_em1 = (float)(1.0 / std::expm1(a.dlnl));   // (on the host: each CTA's warps took 7 us for it on the FP64 pipe)
    const int ks = band_gemm_ksplit(a.n_models, a.nkb, a.npad, a.num_sms);
    const int smem = BandGemmSmem::total(a.npad, a.slots);
    cudaError_t e = cudaFuncSetAttribute(band_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    if (ks > 8 && (e = cudaFuncSetAttribute(band_gemm_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1)) != cudaSuccess)
        return e;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((a.n_models + BG_M - 1) / BG_M, ks);
    cfg.blockDim = dim3(BG_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 1;
    at[0].val.clusterDim.y = (unsigned)ks;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = ks > 1 ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, band_gemm_kernel, tm_hi, tm_lo, a);
}

}  // namespace sps
