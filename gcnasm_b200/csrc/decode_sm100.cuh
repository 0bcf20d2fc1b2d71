// Skinny-M ("decode") A8W8 GEMM for sm_100a: C[M,N] = A[M,K] . W[N,K]^T with M <= 64.
//
// The reference runs its one 256x256x128 tile for every M (opus_fmm/flatmm_a8w8_gfx950.cc:684-687,
// out-of-range rows clamped at :268, stores predicated at :537-541); for M <= 64 that wastes the
// machine, and the job is purely a weight stream.  Here the operands are swapped: a 128(N) x 128(K)
// weight tile is the UMMA M-side operand and the block of 16, 32 or 64 tokens (what lies behind the last one
// is anything) is the UMMA N-side operand, so D[n][token] lands in TMEM with one weight row per lane.  One CTA owns one 128-row
// weight panel (optionally one K slice of it) and streams it through a deep TMA ring; HBM is the bound.
//
// Weights are accepted row-major [N,K] (128-byte swizzled tiles) or in the reference's pre-shuffled
// flat layout [N/16][K/16][16][16] (shuffle_b, flatmm_a8w8_gfx950.cc:638-681).  A flat 16x16 block is
// two 8x16-byte UMMA core matrices back to back, so the TMA box {256 B, 8 slabs, 8 k-chunks} arrives
// in shared memory as [k-chunk][slab][256 B]: a canonical un-swizzled K-major operand with
// LBO = 2048 (next core matrix along K) and SBO = 128 (next 8 rows).  No re-layout pass is needed.
//
// Block scales (A: per token per 128 K, [K/128][M]; W: per 128x128 block, [N/128][K/128]) follow
// gemm_a8w8_blockscale_host.cc:66-90: every K group gets a fresh TMEM buffer and is folded into
// register accumulators as acc += partial * (sfa[g][token] * sfb[nblk][g]).
//
// MX scales: the tensor core applies them, so a CTA's whole K range accumulates in one TMEM buffer; the E8M0 atoms of the weight
// panel and of the token block travel with their stage.  The 128 x 128 single-CTA tile has at most one CTA per 128 weight rows; here a
// panel's K is split over a cluster (mx_skinny_kblocks() says from which K on that pays).
#pragma once

#include "gemm_sm100.cuh"

namespace b200 {

struct DecodeParams {
    CUtensorMap tmap_w;          // weights: 3-D [batch][N][K] swizzled, or the 4-D flat view
    CUtensorMap tmap_x;          // tokens:  3-D [batch][M][K], box 128 x M, 128-byte swizzle (what lies in a stage behind the M tokens is anything)
    void* c;
    float* partial;              // split-K workspace [splits][batch][M][N] fp32, or null: the splits of a panel are a cluster
    const float* sfa;            // MX: the atoms (bytes), as are sfb and, in atoms and bytes, the strides
    const float* sfb;
    const float* scale_a;
    const float* scale_b;
    long long ldc, c_batch;
    long long sfa_stride, sfb_stride, sfa_batch, sfb_batch;
    int m, n, k, batch;
    int tiles_n, kblocks, splits, kb_per_split;
    int out_dtype;
    int inputs_ready;            // the weights are not written by work still in flight on the stream (b200_gemm_flags)
    int* status;
};

// Shared-memory bytes for the staged scales of one CTA.  16-token blocks already reach the ten-stage cap of the ring
// with 34 KB; wider token blocks get one more ring stage from a 24 KB area (config 4: 56 groups x 64 tokens = 14 KB).
__host__ __device__ constexpr int decode_sf_bytes(int mt) { return mt <= 16 ? 34 * 1024 : 24 * 1024; }

template <int MT_, int MODE_, int BLAYOUT_>
struct DecodeCfg {
    static constexpr int MT = MT_, MODE = MODE_, BLAYOUT = BLAYOUT_;
    static constexpr int BNW = 128, BK = 128;
    static constexpr int W_BYTES = BNW * BK;
    static constexpr int X_BYTES = MT * BK;
    static constexpr int SF_BYTES = MODE == MODE_MX ? 1024 : 0;     // MX: the atom of the weight rows, then that of the tokens
    static constexpr int STAGE_BYTES = ((W_BYTES + X_BYTES + SF_BYTES + 1023) / 1024) * 1024;
    // combined scales [K groups of this CTA][MT]; problems whose groups do not fit are split along K by the launcher
    static constexpr int SF_SMEM = MODE == MODE_MX ? 0 : decode_sf_bytes(MT_);
    static constexpr int STAGES_RAW = (225 * 1024 - 1024 - SF_SMEM) / STAGE_BYTES;
    static constexpr int STAGES = STAGES_RAW > 10 ? 10 : STAGES_RAW;
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + SF_SMEM + 1024;
    // Block-scale mode gives every K group its own TMEM buffer (a fresh accumulator per group), but hands the
    // buffers over in BATCHES of GB groups: one hand-off between the MMA issuer and the epilogue warps costs on
    // the order of a microsecond (commit -> barrier -> TMEM loads -> barrier), far more than the tiny MMAs of a
    // group, so it is paid once per GB groups.  Two batch sets ping-pong: TMEM holds 2 x GB x MT columns.
    static constexpr int GB = 4;
    static constexpr int NBUF = 2;
    static constexpr int SF_COL = MT;                               // MX: scale columns behind the one accumulator
    static constexpr int TMEM_COLS = MODE == MODE_MX ? (MT + 8 <= 32 ? 32 : (MT + 8 <= 64 ? 64 : 128)) : (NBUF * GB * MT < 32 ? 32 : NBUF * GB * MT);
    static constexpr int THREADS = 192;
    static constexpr int MAX_SF_FLOATS = SF_SMEM / 4;
    static_assert(MT == 16 || MT == 32 || MT == 64, "token block is 16, 32 or 64");
};

template <class Cfg>
__global__ void __launch_bounds__(Cfg::THREADS, 1) decode_a8w8_sm100_kernel(const __grid_constant__ DecodeParams p) {
    constexpr int MT = Cfg::MT, BK = Cfg::BK, BNW = Cfg::BNW, STAGES = Cfg::STAGES, MODE = Cfg::MODE;

    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem_gen + STAGES * Cfg::STAGE_BYTES);
    const uint32_t bar_full0 = smem_base + STAGES * Cfg::STAGE_BYTES;
    const uint32_t bar_empty0 = bar_full0 + STAGES * 8;
    const uint32_t bar_accf0 = bar_empty0 + STAGES * 8;
    constexpr int NBUF = Cfg::NBUF;
    const uint32_t bar_acce0 = bar_accf0 + NBUF * 8;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 2 * NBUF);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    float* sf_smem = reinterpret_cast<float*>(smem_gen + STAGES * Cfg::STAGE_BYTES + 1024);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;

    // work item: (batch, n tile, k split)
    int w = blockIdx.x;
    const int split = w % p.splits;
    w /= p.splits;
    const int ni = w % p.tiles_n;
    const int b = w / p.tiles_n;
    const int kb0 = split * p.kb_per_split;
    const int kb1 = (kb0 + p.kb_per_split < p.kblocks) ? kb0 + p.kb_per_split : p.kblocks;
    const int nkb = kb1 - kb0;
    // C takes 16-byte stores (c_batch and ldc are in elements; the columns a store starts at are multiples of 4, of 32 without splits)
    const bool c_vec = (reinterpret_cast<uintptr_t>(p.c) & 15) == 0 && (p.ldc * (p.out_dtype == OUT_BF16 ? 2 : 4)) % 16 == 0 &&
                       (p.c_batch * (p.out_dtype == OUT_BF16 ? 2 : 4)) % 16 == 0;

    // Consecutive decode GEMMs of a serving step are launched with programmatic serialization: this kernel may
    // start while its predecessor is still draining.  When the caller has vouched for the weights
    // (B200_GEMM_INPUTS_READY: resident, not written by anything still in flight) the first ring of weight tiles is
    // requested right away; otherwise the weights, like everything that may be the predecessor's output (tokens,
    // token scales) and every write to C, come after pdl_wait(), and that first ring is only prefetched into L2 before it:
    // HBM streams while the predecessor (the activation quantiser of the same layer, as a rule) still runs.  With the
    // quantiser in front, 16 tokens: 2560 x 7168 10.4 -> 9.8 us, 7168 x 2048 9.3 -> 8.4; nothing where every SM streams for
    // long (18432 x 7168).
    pdl_launch_dependents();
    const int first = nkb < STAGES ? nkb : STAGES;
    const uint32_t load_bytes = Cfg::W_BYTES + p.m * BK + Cfg::SF_BYTES;
    // MX: atom (kb, 128-row block) of an image [batch][K/128][rows/128][512 B]
    auto mx_atom = [&](const float* image, long long batch_bytes, long long blocks, int kb, int blk) {
        return reinterpret_cast<const uint8_t*>(image) + b * batch_bytes + (static_cast<long long>(kb) * blocks + blk) * 512;
    };
    auto request_weights = [&](int i) {
        const uint32_t sw = smem_base + i * Cfg::STAGE_BYTES;
        const uint32_t full = bar_full0 + i * 8;
        mbar_arrive_expect_tx(full, load_bytes);
        if constexpr (Cfg::BLAYOUT == BL_NK)
            tma_load_3d(sw, &p.tmap_w, full, (kb0 + i) * BK, ni * BNW, b);
        else
            tma_load_4d(sw, &p.tmap_w, full, 0, ni * (BNW / 16), (kb0 + i) * (BK / 16), b);
        if constexpr (MODE == MODE_MX)
            bulk_load(sw + Cfg::W_BYTES + Cfg::X_BYTES, mx_atom(p.sfb, p.sfb_batch, p.sfb_stride, kb0 + i, ni), 512, full);
    };
    if (threadIdx.x == 2 * 32 && !p.inputs_ready) {
        for (int i = 0; i < first; ++i) {
            if constexpr (Cfg::BLAYOUT == BL_NK)
                tma_prefetch_3d(&p.tmap_w, (kb0 + i) * BK, ni * BNW, b);
            else
                tma_prefetch_4d(&p.tmap_w, 0, ni * (BNW / 16), (kb0 + i) * (BK / 16), b);
        }
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(bar_full0 + s * 8, 1);
            mbar_init(bar_empty0 + s * 8, 1);
        }
        for (int s = 0; s < NBUF; ++s) {
            mbar_init(bar_accf0 + s * 8, 1);
            mbar_init(bar_acce0 + s * 8, 4);
        }
        *abort_flag = 0;
        fence_barrier_init();
        fence_proxy_async_smem();
        if (p.inputs_ready)
            for (int i = 0; i < first; ++i) request_weights(i);
    }
    if (warp == 1) {
        tmem_alloc<1>(smem_u32(tmem_slot), Cfg::TMEM_COLS);
        tmem_relinquish<1>();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_wait();
    if (threadIdx.x == 0) {
        for (int i = 0; i < first; ++i) {
            if (!p.inputs_ready) request_weights(i);
            tma_load_3d(smem_base + i * Cfg::STAGE_BYTES + Cfg::W_BYTES, &p.tmap_x, bar_full0 + i * 8, (kb0 + i) * BK, 0, b);
            if constexpr (MODE == MODE_MX)
                bulk_load(smem_base + i * Cfg::STAGE_BYTES + Cfg::W_BYTES + Cfg::X_BYTES + 512, mx_atom(p.sfa, p.sfa_batch, p.sfa_stride, kb0 + i, 0),
                          512, bar_full0 + i * 8);
        }
    }

    if (warp == 0) {
        if (lane == 0) {
            // ------------------------------ TMA producer ------------------------------
            for (int i = first; i < nkb; ++i) {
                const int kb = kb0 + i;
                const uint32_t s = i % STAGES;
                const uint32_t ph = (i / STAGES) & 1;
                if (!mbar_wait_poll<false, 64>(bar_empty0 + s * 8, ph ^ 1, abort_flag, p.status, KSTAT_TIMEOUT_EMPTY)) break;
                const uint32_t sw = smem_base + s * Cfg::STAGE_BYTES;
                const uint32_t sx = sw + Cfg::W_BYTES;
                const uint32_t full = bar_full0 + s * 8;
                mbar_arrive_expect_tx(full, load_bytes);
                if constexpr (Cfg::BLAYOUT == BL_NK)
                    tma_load_3d(sw, &p.tmap_w, full, kb * BK, ni * BNW, b);
                else
                    tma_load_4d(sw, &p.tmap_w, full, 0, ni * (BNW / 16), kb * (BK / 16), b);
                tma_load_3d(sx, &p.tmap_x, full, kb * BK, 0, b);
                if constexpr (MODE == MODE_MX) {
                    bulk_load(sx + Cfg::X_BYTES, mx_atom(p.sfb, p.sfb_batch, p.sfb_stride, kb, ni), 512, full);
                    bulk_load(sx + Cfg::X_BYTES + 512, mx_atom(p.sfa, p.sfa_batch, p.sfa_stride, kb, 0), 512, full);
                }
            }
        }
    } else if (warp == 1) {
        {
            // ------------------------------ UMMA issuer (the warp; an elected lane issues) ------------
            const bool elected = elect_one() != 0;
            constexpr uint32_t idesc = make_idesc_f8(BNW, MT);
            uint32_t phase = 0;
            bool ok = true;
            if constexpr (MODE != MODE_BLOCK) {
                // the single accumulator buffer is free at kernel start
            }
            constexpr int GBATCH = (MODE == MODE_BLOCK) ? Cfg::GB : 1;
            for (int i0 = 0; i0 < nkb && ok; i0 += GBATCH, ++phase) {
                const int gb = (nkb - i0 < GBATCH) ? nkb - i0 : GBATCH;       // groups in this batch
                const uint32_t set = phase % NBUF;
                if constexpr (MODE == MODE_BLOCK) {
                    const uint32_t aph = (phase / NBUF) & 1;
                    if (!role_all<true>(mbar_wait<false, 0>(bar_acce0 + set * 8, aph ^ 1, abort_flag, p.status, KSTAT_TIMEOUT_ACC_E))) {
                        ok = false;
                        break;
                    }
                }
                for (int j = 0; j < gb && ok; ++j) {
                    const int i = i0 + j;
                    const uint32_t s = i % STAGES;
                    const uint32_t ph = (i / STAGES) & 1;
                    const uint32_t sw = smem_base + s * Cfg::STAGE_BYTES;
                    const uint32_t sx = sw + Cfg::W_BYTES;
                    constexpr uint32_t LBO = (BNW / 16) * 256;
                    // The descriptors are formed before the wait, and the wait suspends the warp.  Formed behind it, polling with 20 ns of
                    // sleep / so, us: block scales, 16 tokens, 7168 x 2048 6.4 / 6.2, 2560 x 7168 8.0 / 7.75, 18432 x 7168 22.1 / 21.9; unscaled,
                    // 64 tokens, 2048 x 7168 8.4 / 8.1; MX, 64 tokens, 7168 x 2048 8.0 / 7.75.
                    uint64_t dw0 = Cfg::BLAYOUT == BL_NK ? make_smem_desc(sw, 16, 1024, kSwizzle128B) : make_smem_desc(sw, LBO, 128, kSwizzleNone);
                    uint64_t dx0 = make_smem_desc(sx, 16, 1024, kSwizzle128B);
                    uint64_t dsf0 = make_smem_desc(sx + Cfg::X_BYTES, 0, 128, kSwizzleNone);                 // MX
                    asm volatile("" : "+l"(dw0), "+l"(dx0), "+l"(dsf0));
                    if (!role_all<true>(mbar_wait<false, 0>(bar_full0 + s * 8, ph, abort_flag, p.status, KSTAT_TIMEOUT_FULL))) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    if (!elected) continue;
                    const uint32_t tacc = (MODE == MODE_BLOCK) ? tmem_base + (set * Cfg::GB + j) * MT : tmem_base;
                    const uint32_t tsf = tmem_base + Cfg::SF_COL;
                    if constexpr (MODE == MODE_MX) {
                        tmem_cp_sf<1>(tsf, dsf0);
                        tmem_cp_sf<1>(tsf + 4, dsf0 + 32);
                    }
#pragma unroll
                    for (int k = 0; k < BK / 32; ++k) {
                        const uint64_t dw = dw0 + (Cfg::BLAYOUT == BL_NK ? k * 2u : (k * 2 * LBO) >> 4), dx = dx0 + k * 2;
                        const uint32_t accum = (MODE == MODE_BLOCK) ? (k > 0 ? 1u : 0u) : ((i > 0 || k > 0) ? 1u : 0u);
                        if constexpr (MODE == MODE_MX) umma_mxf8<1>(tacc, dw, dx, make_idesc_mxf8(BNW, MT, k, k), accum, tsf, tsf + 4);
                        else umma_f8<1>(tacc, dw, dx, idesc, accum);
                    }
                    umma_commit<1>(bar_empty0 + s * 8);
                }
                if (!ok) break;
                if constexpr (MODE == MODE_BLOCK) {
                    if (elected) umma_commit<1>(bar_accf0 + set * 8);
                } else {
                    if (i0 + gb >= nkb && elected) umma_commit<1>(bar_accf0);
                }
            }
        }
    } else {
        // ---------------------------------- epilogue ----------------------------------
        const int quad = warp & 3;
        const int et = (warp - 2) * 32 + lane;             // 0..127 over the four epilogue warps
        const int n_row = ni * BNW + quad * 32 + lane;
        const uint32_t tmem_lane = static_cast<uint32_t>(quad * 32) << 16;
        float acc[MT];
#pragma unroll
        for (int j = 0; j < MT; ++j) acc[j] = 0.0f;
        bool ok = true;

        if constexpr (MODE == MODE_BLOCK) {
            // stage this CTA's combined scales: sf_smem[i*MT + j] = sfa[kb0+i][j] * sfb[ni][kb0+i] (the product the
            // promotion multiplies by, formed once here instead of once per thread and group)
            const float* sfa_g = p.sfa + b * p.sfa_batch;
            const float* sfb_g = p.sfb + b * p.sfb_batch + static_cast<long long>(ni) * p.sfb_stride;
            // (U independent element loads in flight per thread: with one element per round trip this loop cost
            // 0.35 us per 128 x MT elements, 10 us of a 37 us launch at MT = 64.  Eight in flight cover a config-4 panel
            // in 1, 2 and 4 round trips at MT = 16, 32, 64; the wider token blocks therefore keep 16 and 28 in flight --
            // the accumulators are not live yet, so the registers are there.)
            constexpr int U = MT <= 16 ? 8 : (MT <= 32 ? 16 : 28);
            const int total = nkb * MT;
            for (int base = et; base < total; base += 128 * U) {
                float va[U], vb[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int idx = base + u * 128;
                    va[u] = 0.0f;
                    vb[u] = 0.0f;
                    if (idx < total) {
                        const int i = idx / MT, j = idx - i * MT;
                        if (j < p.m) {
                            va[u] = __ldg(sfa_g + static_cast<long long>(kb0 + i) * p.sfa_stride + j);
                            vb[u] = __ldg(sfb_g + kb0 + i);
                        }
                    }
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int idx = base + u * 128;
                    if (idx < total) sf_smem[idx] = va[u] * vb[u];
                }
            }
            asm volatile("bar.sync 1, 128;" ::: "memory");   // epilogue warps only

            // packed accumulators (token pairs); the TMEM loads of group j+1 run behind the FMAs of group j
            unsigned long long acc2[MT / 2];
#pragma unroll
            for (int j = 0; j < MT / 2; ++j) acc2[j] = 0ull;
            float vbuf[2][MT];
            uint32_t phase = 0;
            for (int i0 = 0; i0 < nkb && ok; i0 += Cfg::GB, ++phase) {
                const int gb = (nkb - i0 < Cfg::GB) ? nkb - i0 : Cfg::GB;
                const uint32_t set = phase % NBUF;
                const uint32_t aph = (phase / NBUF) & 1;
                if (!mbar_wait(bar_accf0 + set * 8, aph, abort_flag, p.status, KSTAT_TIMEOUT_ACC_F)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t tset = tmem_base + tmem_lane + set * Cfg::GB * MT;
#pragma unroll
                for (int c = 0; c < MT / 16; ++c) tmem_ld16(tset + c * 16, &vbuf[0][c * 16]);
#pragma unroll
                for (int j = 0; j < Cfg::GB; ++j) {
                    if (j < gb) {
                        tmem_ld_wait();                                  // group j is in vbuf[j & 1]
                        if (j + 1 < gb) {
#pragma unroll
                            for (int c = 0; c < MT / 16; ++c) tmem_ld16(tset + (j + 1) * MT + c * 16, &vbuf[(j + 1) & 1][c * 16]);
                        } else {
                            // the whole batch has left TMEM: the set goes back to the MMA issuer
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) mbar_arrive(bar_acce0 + set * 8);
                        }
                        const float4* s4 = reinterpret_cast<const float4*>(sf_smem + (i0 + j) * MT);
#pragma unroll
                        for (int jj = 0; jj < MT; jj += 4) {
                            const float4 sc = s4[jj / 4];
                            acc2[jj / 2] = ffma2(pack_f32x2(vbuf[j & 1][jj], vbuf[j & 1][jj + 1]), pack_f32x2(sc.x, sc.y), acc2[jj / 2]);
                            acc2[jj / 2 + 1] = ffma2(pack_f32x2(vbuf[j & 1][jj + 2], vbuf[j & 1][jj + 3]), pack_f32x2(sc.z, sc.w), acc2[jj / 2 + 1]);
                        }
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < MT / 2; ++j) unpack_f32x2(acc2[j], acc[2 * j], acc[2 * j + 1]);
        } else {
            if (nkb > 0) {
                if (mbar_wait(bar_accf0, 0, abort_flag, p.status, KSTAT_TIMEOUT_ACC_F)) {
                    tc_fence_after();
#pragma unroll
                    for (int c = 0; c < MT / 16; ++c) tmem_ld16(tmem_base + tmem_lane + c * 16, &acc[c * 16]);
                    tmem_ld_wait();
                    float tscale = 1.0f;
                    if (p.scale_a) tscale *= __ldg(p.scale_a);
                    if (p.scale_b) tscale *= __ldg(p.scale_b);
#pragma unroll
                    for (int j = 0; j < MT; ++j) acc[j] *= tscale;
                } else {
                    ok = false;
                }
            }
        }

        // Every MMA of this CTA has completed, so the ring is free.  (A split that gave up leaves anything there: nobody adds it.)
        if (p.splits > 1 && !p.partial) {
            float* mine = reinterpret_cast<float*>(smem_gen) + quad * 32 + lane;      // partial sums [token][weight row]
#pragma unroll
            for (int j = 0; j < MT; ++j) mine[j * BNW] = acc[j];
        } else if (ok && p.splits == 1 && c_vec && ni * BNW + quad * 32 + 32 <= p.n) {
            // a thread holds one column of the output: the warp turns its 32 columns round in shared memory and stores 16 bytes
            // per lane, 64 (128) contiguous bytes per token.  One two-byte store per token and thread, written out token by token,
            // was most of what a 64-token call took longer than one of 1 token whatever K (18432 x 7168, in a graph, 64 tokens:
            // 24.9 -> 23.4 us, K = 3584 15.4 -> 13.7; 32 tokens 23.05 -> 22.35; 16 22.1 -> 21.8; one token the same; on another GPU of the
            // kind 64 tokens 25.6 -> 24.15).
            uint8_t* mine = smem_gen + quad * (MT * 128);
            const int pieces = p.out_dtype == OUT_BF16 ? 4 : 8;                       // 16-byte pieces per token
            if (p.out_dtype == OUT_BF16) {
                __nv_bfloat16* t = reinterpret_cast<__nv_bfloat16*>(mine) + lane;
#pragma unroll
                for (int j = 0; j < MT; ++j) t[j * 32] = __float2bfloat16_rn(acc[j]);
            } else {
                float* t = reinterpret_cast<float*>(mine) + lane;
#pragma unroll
                for (int j = 0; j < MT; ++j) t[j * 32] = acc[j];
            }
            __syncwarp();
            const size_t esz = p.out_dtype == OUT_BF16 ? 2 : 4;
            uint8_t* dst = reinterpret_cast<uint8_t*>(p.c) + (static_cast<size_t>(b) * p.c_batch + ni * BNW + quad * 32) * esz;
#pragma unroll 4
            for (int q = lane; q < p.m * pieces; q += 32)
                *reinterpret_cast<uint4*>(dst + static_cast<size_t>(q / pieces) * p.ldc * esz + (q % pieces) * 16) =
                    *reinterpret_cast<const uint4*>(mine + q * 16);
        } else if (ok && n_row < p.n) {
            float* part = p.partial ? p.partial + ((static_cast<size_t>(split) * p.batch + b) * p.m) * p.n + n_row : nullptr;
            const size_t o = static_cast<size_t>(b) * p.c_batch + n_row;
#pragma unroll
            for (int j = 0; j < MT; ++j) {
                if (j >= p.m) break;
                if (p.splits > 1) part[static_cast<size_t>(j) * p.n] = acc[j];
                else if (p.out_dtype == OUT_BF16) reinterpret_cast<__nv_bfloat16*>(p.c)[o + static_cast<size_t>(j) * p.ldc] = __float2bfloat16_rn(acc[j]);
                else reinterpret_cast<float*>(p.c)[o + static_cast<size_t>(j) * p.ldc] = acc[j];
            }
        }
    }

    // The K splits of one weight panel are the CTAs of a cluster: each leaves its partial sums in its own shared memory and,
    // one barrier later, CTA r sums rows r, r + splits, ... over all of them, in the order of K.  (The partials in a global
    // workspace, summed by a second kernel, with the quantiser in front, 16 tokens: 7168 x 2048 10.1 -> 8.4 us, 4096 x 7168
    // 14.4 -> 11.5, 2560 x 7168 12.7 -> 9.8.)
    if (p.splits > 1 && !p.partial) {
        __syncwarp();
        cluster_arrive();
        cluster_wait();
        // A split that gave up (an expired wait) has no sums to add: the panel is left unwritten then, as without a cluster.
        // Asked for first and looked at after the first row's sums, whose loads cover it.
        const uint32_t gave_up = lane < p.splits ? ld_shared_cluster_u32(mapa_shared(smem_u32(tmem_slot + 1), lane)) : 0u;
        // a lane sums four neighbouring columns: a quarter of the remote loads (MX, 64 x 2048 x 2048 with eight splits 6.35 -> 6.04 us)
        const int col = ni * BNW + lane * 4;
        const bool whole = c_vec && col + 4 <= p.n;
        for (int j = split + warp * p.splits; j < p.m; j += p.splits * (Cfg::THREADS / 32)) {
            const uint32_t row = smem_base + static_cast<uint32_t>(j * BNW + lane * 4) * 4;
            float sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 8
            for (int s = 0; s < p.splits; ++s) {
                const float4 v = ld_shared_cluster_f32x4(mapa_shared(row, s));
                sum[0] += v.x;
                sum[1] += v.y;
                sum[2] += v.z;
                sum[3] += v.w;
            }
            if (__any_sync(0xFFFFFFFFu, gave_up != 0u)) break;
            const size_t o = static_cast<size_t>(b) * p.c_batch + static_cast<size_t>(j) * p.ldc + col;
            if (whole && p.out_dtype == OUT_BF16) {
                *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(p.c) + o) = make_uint2(pack_bf16x2(sum[0], sum[1]), pack_bf16x2(sum[2], sum[3]));
            } else if (whole) {
                *reinterpret_cast<float4*>(reinterpret_cast<float*>(p.c) + o) = make_float4(sum[0], sum[1], sum[2], sum[3]);
            } else {
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    if (col + c < p.n) {
                        if (p.out_dtype == OUT_BF16) reinterpret_cast<__nv_bfloat16*>(p.c)[o + c] = __float2bfloat16_rn(sum[c]);
                        else reinterpret_cast<float*>(p.c)[o + c] = sum[c];
                    }
                }
            }
        }
        __syncwarp();              // (the lanes of a ragged panel part above; the barrier wants the warp together)
        cluster_arrive();          // no CTA leaves while another one reads its partials
        cluster_wait();
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc<1>(tmem_base, Cfg::TMEM_COLS);
    }
}

// Sums the split-K partials [splits][rows] -> C (fixed order, so the result is deterministic).
__global__ void decode_splitk_reduce_kernel(const float* __restrict__ partial, void* __restrict__ c, int splits,
                                            long long per_split, int m, int n, long long ldc, long long c_batch,
                                            int out_dtype) {
    const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= per_split) return;
    float s = 0.0f;
    for (int k = 0; k < splits; ++k) s += partial[k * per_split + i];
    const long long mn = static_cast<long long>(m) * n;
    const long long b = i / mn;
    const long long r = i - b * mn;
    const long long row = r / n, col = r - row * n;
    const long long o = b * c_batch + row * ldc + col;
    if (out_dtype == OUT_BF16) reinterpret_cast<__nv_bfloat16*>(c)[o] = __float2bfloat16_rn(s);
    else reinterpret_cast<float*>(c)[o] = s;
}

}  // namespace b200
